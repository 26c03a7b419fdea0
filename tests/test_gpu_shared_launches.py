"""Plain media (walk kernel) beside media of several indices (transport
kernel).  A launch over several media runs the walk kernel when all of them are
plain and the transport kernel otherwise, so the kernel of a plain request
depends on the requests beside it, and a served photon may be parked by one
kernel and resumed by the other.  Strict math gives every request the tallies
of its run alone; fast math gives them to plain media, whose pass the two
kernels round alike (media of several indices: the compiler may contract
the mixed-media form of their reflections in another way)."""
import numpy as np
import pytest

import cudamcfl_gb300 as mc

VOX = (0.1, 0.1, 0.05)
TDET = (0.1, -0.05, 2, 2, 0.25, 0.25, 0.15, 0, 20, 150000)


def _media():
    """One grid, plain and with labels of several indices, one of them free of
    scattering."""
    rng = np.random.default_rng(3)
    lab = rng.integers(1, 4, size=(14, 20, 24)).astype(np.uint8)
    lab[:7, :10] = 1
    out, b = mc.outer_bulk(1.0), mc.bulk_from_mci_columns
    plain = [out, b(1.4, 0.1, 100.0, g=0.9), b(1.4, 0.3, 60.0, 1.0, 0.05, 0.02, 0.1, 0.8), b(1.4, 0.4, 40.0, g=0.75), out]
    indices = [out, b(1.37, 0.2, 60.0, g=0.8), b(1.52, 0.5, 40.0, 2.0, 0.1, 0.04, 0.2, 0.7), b(1.4, 0.05, 0.0, g=0.9),
               out]
    return lab, plain, indices


def _desc(photons, i, timed, fluence):
    return mc.run_desc(photons, source=(0.1 * i, 0.0, 0.0), det=mc.Detector(0.0, 0.0, 0.05, 0.05, 30, 30), seed_exc=40 + i,
                       tdet=TDET if timed else None, fluence=fluence)


def _assert_equal(got, one, timed, fluence=False):
    for k in ("Rd", "Tt") + (("time_xyt",) if timed else ()) + (("fhd",) if fluence else ()):
        assert np.array_equal(np.ravel(got[k]), getattr(one, k).ravel()), k
    assert got["stats"] == one.stats_exc


@pytest.fixture(params=[mc.MATH_EXACT, mc.MATH_FAST], ids=["strict", "fast"])
def ctx(request, mcfl_lib):
    c = mc.Context(math=request.param)
    yield c
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("timed", [False, True])
def test_batched_plain_run_beside_another_medium_equals_alone(timed, ctx):
    lab, plain, indices = _media()
    p, q = ctx.medium(lab, plain, voxel_cm=VOX), ctx.medium(lab, indices, voxel_cm=VOX)
    runs = [_desc(n, i, timed, 0) for i, n in enumerate((200011, 30000, 9001, 5000))]
    alone = [ctx.run(m, rd) for m, rd in zip((p, q, p, q), runs)]
    for mixed_variant in range(3):
        ctx.set_option("mixed_variant", mixed_variant)
        got, _ = mc.batch_run(ctx, [p, q, p, q], runs)
        for i in (0, 1, 2, 3) if ctx.get_option("math") == mc.MATH_EXACT else (0, 2):
            _assert_equal(got[i], alone[i], timed)
    p.free()
    q.free()


# slices of 37 passes: photons of the long plain request are in flight (parked and resumed) while requests of several
# indices come and go beside it
@pytest.mark.gpu
@pytest.mark.parametrize("timed", [False, True])
@pytest.mark.parametrize("slice_passes", [37, 1000])
def test_served_plain_request_beside_another_medium_equals_alone(slice_passes, timed, ctx):
    lab, plain, indices = _media()
    reqs = [(plain, _desc(60011, 0, timed, 1)), (plain, _desc(300, 1, timed, 0)), (indices, _desc(500, 2, timed, 1)),
            (plain, _desc(700, 3, timed, 1)), (indices, _desc(2000, 4, timed, 0))]
    srv = mc.Server(ctx, max_jobs=2, slice_passes=slice_passes)
    try:
        ids = [srv.submit(lab, bulks, VOX, rd) for bulks, rd in reqs]
        for i in ids:
            assert srv.wait(i, 120000) == 0
        got = [srv.result(i) for i in ids]
        assert srv.metrics()["slices"] > 4
    finally:
        srv.close()
    for (bulks, rd), r in zip(reqs, got):
        if bulks is indices and ctx.get_option("math") != mc.MATH_EXACT:
            continue
        med = ctx.medium(lab, bulks, voxel_cm=VOX)
        _assert_equal(r, ctx.run(med, rd), timed, fluence=bool(rd.fluence))
        med.free()
