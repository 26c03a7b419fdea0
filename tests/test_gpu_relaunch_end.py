"""The relaunch option at a launch's end: free lanes that still wait for more
when the tickets run out.  Launches long enough that lanes draw several
photons, in every kernel whose last photons move between warps; the tallies
are those of relaunch 1."""
import numpy as np
import pytest

import cudamcfl_gb300 as mc
from tests import cases
from tests.test_gpu_walk import _plain

DET = mc.Detector(0.0, 0.0, 0.05, 0.05, 30, 30)


def _runs(ctx, kind, relaunch):
    ctx.set_option("relaunch", relaunch)
    if kind == "layered":
        case = cases.layered(300000)
        med = case.engine_medium(ctx)
        r = ctx.run(med, case.run_desc(31, 32))
        med.free()
        return [r.Rd, r.Tt, r.fhd, np.array(list(r.stats_exc.values()))]
    if kind == "indices":
        case = cases.mismatch(300000, 2000)
        med = case.engine_medium(ctx)
        r = ctx.run(med, case.run_desc(31, 32))
        med.free()
        return [r.Rd, r.Tt, r.fhd, r.flR128, r.flT128, np.array(list(r.stats_exc.values()))]
    lab, bulks, geo = _plain(13, 6, 7)
    meds = [ctx.medium(lab, bulks, **geo) for _ in range(2)]
    runs = [mc.run_desc(n, det=DET, seed_exc=40 + i) for i, n in enumerate((300000, 1, 20011))]
    res, _ = mc.batch_run(ctx, meds[0] if kind == "plain" else [meds[0], meds[1], meds[0]], runs)
    for m in meds:
        m.free()
    return [a for r in res for a in (r["Rd"], r["Tt"], np.array(list(r["stats"].values())))]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "plain media in one launch", "indices", "layered"])
def test_tallies_do_not_depend_on_relaunch(kind, gpu_ctx):
    try:
        want = _runs(gpu_ctx, kind, 1)
        for relaunch in (2, 8, 31, 32):
            got = _runs(gpu_ctx, kind, relaunch)
            assert all(np.array_equal(a, b) for a, b in zip(got, want)), relaunch
    finally:
        gpu_ctx.set_option("relaunch", 1)
