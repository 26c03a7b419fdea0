"""The walk kernel (plain media) at the sizes where it can go wrong, against
the CPU oracle bit for bit (strict math) or against itself under another
launch shape (fast math, whose roundings are fixed so that a photon's walk
does not depend on what the other lanes of its warp do)."""
import ctypes

import numpy as np
import pytest

import cudamcfl_gb300 as mc
from tests import cases
from tests.test_gpu_parity import _compare


def _plain(nx, ny, nz, seed=1, hx=None, labels=(1, 2, 3), g3=0.75, mua3=0.4):
    """Three labels of one refractive index over an odd grid; oracle and
    engine geometry."""
    rng = np.random.default_rng(seed)
    lab = rng.choice(np.array(labels, dtype=np.uint8), p=None, size=(nz, ny, nx)).astype(np.uint8)
    lab[: nz // 2, : ny // 2] = 1
    bulks = [mc.outer_bulk(1.0), mc.bulk_from_mci_columns(1.4, 0.1, 100.0, g=0.9),
             mc.bulk_from_mci_columns(1.4, 0.3, 60.0, 1.0, 0.05, 0.02, 0.1, 0.8),
             mc.bulk_from_mci_columns(1.4, mua3, 40.0, g=g3), mc.outer_bulk(1.0)]
    hx = hx or 0.05 * nx
    return lab, bulks, dict(half_x=float(np.float32(hx)), half_y=float(np.float32(0.05 * ny)),
                            thickness=float(np.float32(0.05 * nz)), vox_per_cm=(10.0, 10.0, 20.0))


def _oracle(oracle, table, lab, bulks, geo, photons, per_voxel, source=(0.0, 0.0, 0.0), start_weight=0):
    from oracle import pyoracle
    sim = pyoracle.sim_from_arrays(lab, bulks, photons=photons, per_voxel=per_voxel,
                                   det=(0.05, 0.05, 30, 30, 0.0, 0.0), source=source, start_weight=start_weight,
                                   **dict(geo, vox_per_cm=list(geo["vox_per_cm"])))
    return sim, oracle.run_photon(sim, table, 21, 22, libm=False)


def _run(ctx, lab, bulks, geo, sim, photons, per_voxel, source=(0.0, 0.0, 0.0), fluence=1):
    med = ctx.medium(lab, bulks, **geo)
    try:
        return ctx.run(med, mc.run_desc(photons, source=source, det=mc.Detector(0.0, 0.0, 0.05, 0.05, 30, 30),
                                        photons_per_voxel=per_voxel, fluence=fluence, seed_exc=21, seed_fl=22,
                                        start_weight=sim.start_weight))
    finally:
        med.free()


# grid sizes around the label tiles' edges (multiples of 4 and one off), photon counts around a warp, a queue, one
# photon per spread warp, and the launch's end shared among warps
@pytest.mark.gpu
@pytest.mark.parametrize("shape,photons,per_voxel", [((5, 7, 3), 1, 1), ((8, 8, 4), 17, 1), ((9, 11, 5), 33, 2),
                                                     ((13, 6, 7), 2000, 1), ((4, 21, 9), 60000, 1)])
def test_plain_media_bit_identical_to_oracle(shape, photons, per_voxel, gpu_ctx, oracle, table32768):
    lab, bulks, geo = _plain(*shape)
    sim, ref = _oracle(oracle, table32768, lab, bulks, geo, photons, per_voxel)
    try:
        for variant, block in ((0, 256), (1, 256), (2, 128), (0, 32), (0, 96)):
            gpu_ctx.set_option("variant", variant)
            gpu_ctx.set_option("block", block)
            _compare(_run(gpu_ctx, lab, bulks, geo, sim, photons, per_voxel), ref)
    finally:
        gpu_ctx.set_option("variant", 0)
        gpu_ctx.set_option("block", 256)


# media next to plain ones, which the host must tell apart: an extent beyond the grid, a voxel of the media outside, an
# isotropic label, a drop above half of the weight, a drop of zero
@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["wide_extent", "outside_label", "isotropic", "black", "clear"])
def test_media_that_are_not_plain_bit_identical_to_oracle(kind, gpu_ctx, oracle, table32768):
    lab, bulks, geo = _plain(9, 10, 6, hx=0.7 if kind == "wide_extent" else None,
                             g3=0.0 if kind == "isotropic" else 0.75,
                             mua3={"black": 70.0, "clear": 0.0}.get(kind, 0.4))
    if kind == "outside_label":
        lab[4, 6, 5] = 4
        lab[3, 7, 7] = 0
    sim, ref = _oracle(oracle, table32768, lab, bulks, geo, 4000, 3)
    _compare(_run(gpu_ctx, lab, bulks, geo, sim, 4000, 3), ref)


# starts that the first pass made ahead must leave to the event code
@pytest.mark.gpu
@pytest.mark.parametrize("source,start_weight", [((0.0, 0.0, 0.29999), 0), ((0.2, -0.1, 0.1), 300000),
                                                 ((0.0, 0.0, 0.0), 430000), ((5.0, 0.0, 0.0), 0)])
def test_starts_bit_identical_to_oracle(source, start_weight, gpu_ctx, oracle, table32768):
    lab, bulks, geo = _plain(9, 10, 6)
    sim, ref = _oracle(oracle, table32768, lab, bulks, geo, 3000, 0, source, start_weight)
    res = _run(gpu_ctx, lab, bulks, geo, sim, 3000, 0, source)
    _compare(res, ref, emission=False)


@pytest.mark.gpu
@pytest.mark.parametrize("cap", [1, 2, 3, 40])
def test_pass_cap_equals_branching_pass(cap, gpu_ctx):
    """Photons stopped by the pass cap: the same tallies as the per-test
    branching pass counts."""
    lab, bulks, geo = _plain(12, 12, 8)
    med = gpu_ctx.medium(lab, bulks, **geo)
    nv, xy = lab.size, 30 + 30 * 30
    rd = mc.run_desc(5000, det=mc.Detector(0.0, 0.0, 0.05, 0.05, 30, 30), fluence=1, seed_exc=3)
    got = []
    try:
        gpu_ctx.set_option("step_cap", cap)
        for form in (0, 1):
            gpu_ctx.set_option("pass_form", form)
            out, keep = mc._alloc_out(xy, nv, images=False, fluence=True)
            rc = mc.load().mcfl_run(gpu_ctx.handle, med.handle, ctypes.byref(rd), ctypes.byref(out))
            assert rc == mc.E_CAPPED
            got.append((keep["Rd"], keep["Tt"], keep["fhd"], np.array(list(out.stats_exc), dtype=np.uint64)))
    finally:
        gpu_ctx.set_option("step_cap", 1 << 24)
        gpu_ctx.set_option("pass_form", 0)
        med.free()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert got[0][3][mc.STAT_NAMES.index("capped")] > 0


@pytest.mark.gpu
@pytest.mark.parametrize("timed", [False, True])
def test_fast_walk_does_not_depend_on_the_launch(timed, mcfl_lib):
    """Fast math: the same tallies for every launch shape, in batches and
    through the server's slices (photons parked and resumed)."""
    ctx = mc.Context(math=mc.MATH_FAST)
    lab, bulks, geo = _plain(20, 18, 12)
    vox = (0.1, 0.1, 0.05)
    tdet = (0.1, -0.05, 2, 2, 0.25, 0.25, 0.15, 0, 20, 150000) if timed else None
    runs = [mc.run_desc(7001 + 900 * i, source=(0.1 * i, 0.0, 0.0), det=mc.Detector(0.0, 0.0, 0.05, 0.05, 30, 30),
                        seed_exc=40 + i, tdet=tdet) for i in range(3)]
    keys = ("Rd", "Tt") + (("time_xyt",) if timed else ())
    med, med2 = ctx.medium(lab, bulks, voxel_cm=vox), ctx.medium(lab, bulks, voxel_cm=vox)

    def alone(rd):
        r = ctx.run(med, rd)
        return [getattr(r, k).ravel() for k in keys] + [np.array(list(r.stats_exc.values()), dtype=np.uint64)]

    ref = [alone(rd) for rd in runs]
    for opts in (dict(block=64), dict(blocks_per_sm=1), dict(variant=1), dict(relaunch=5)):
        for k, v in opts.items():
            ctx.set_option(k, v)
        for rd, want in zip(runs, ref):
            assert all(np.array_equal(a, b) for a, b in zip(alone(rd), want)), opts
        for k, v in (("block", 256), ("blocks_per_sm", 0), ("variant", 0), ("relaunch", 1)):
            ctx.set_option(k, v)
    for media_of in (med, [med, med2, med]):
        res, _ = mc.batch_run(ctx, media_of, runs)
        for r, want in zip(res, ref):
            got = [r[k].ravel() for k in keys] + [np.array(list(r["stats"].values()), dtype=np.uint64)]
            assert all(np.array_equal(a, b) for a, b in zip(got, want))
    for slice_passes in (37, 64, 1000):
        srv = mc.Server(ctx, max_jobs=4, slice_passes=slice_passes)
        try:
            ids = [srv.submit(lab, bulks, vox, rd) for rd in runs]
            for i, want in zip(ids, ref):
                assert srv.wait(i, 120000) == 0
                r = srv.result(i)
                got = [r[k].ravel() for k in keys] + [np.array(list(r["stats"].values()), dtype=np.uint64)]
                assert all(np.array_equal(a, b) for a, b in zip(got, want)), slice_passes
        finally:
            srv.close()
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["tiny_timed", "layered", "blocks_exact"])
def test_last_photons_gathered_bit_identical_to_oracle(name, gpu_ctx, oracle, table32768):
    """Launches long enough that the last photons move between warps: timed,
    layered and voxel-boundary stepping."""
    make = {"tiny_timed": lambda: cases.timed(60000, 2, 0, cases.tiny), "layered": lambda: cases.layered(60000),
            "blocks_exact": lambda: cases.exact(cases.blocks)(40000, 2)}[name]
    case = make()
    ref = oracle.run_photon(case.oracle_sim(), table32768, 31, 32, libm=False)
    med = case.engine_medium(gpu_ctx)
    res = gpu_ctx.run(med, case.run_desc(31, 32))
    med.free()
    _compare(res, ref, emission=name != "layered")


# hitting densities summed over a photon's passes in a voxel (few voxel columns under the source) and added pass by pass
@pytest.mark.gpu
@pytest.mark.parametrize("timed", [False, True])
@pytest.mark.parametrize("width", [0.0, 0.5, 2.0, 3.9])
def test_hitting_density_equals_branching_pass(width, timed, gpu_ctx):
    lab, bulks, geo = _plain(40, 40, 8)
    med = gpu_ctx.medium(lab, bulks, **geo)
    tdet = (0.1, -0.05, 2, 2, 0.25, 0.25, 0.15, 0, 20, 150000) if timed else None
    rd = mc.run_desc(20011, det=mc.Detector(0.0, 0.0, 0.05, 0.05, 30, 30), fluence=1, seed_exc=5, tdet=tdet,
                     kind=mc.SOURCE_WIDEFIELD if width else mc.SOURCE_GAUSS_BEAM, width=width, height=width)
    got = []
    try:
        for form in (0, 1):
            gpu_ctx.set_option("pass_form", form)
            got.append(gpu_ctx.run(med, rd))
    finally:
        gpu_ctx.set_option("pass_form", 0)
        med.free()
    assert np.array_equal(got[0].fhd, got[1].fhd) and got[0].fhd.any()
    assert np.array_equal(got[0].Rd, got[1].Rd) and got[0].stats_exc == got[1].stats_exc
