"""The walk kernel's forms against runs that it does not make: the transport
kernel's pass forms and the CPU oracle."""
import numpy as np
import pytest

import cudamcfl_gb300 as mc
from tests.test_gpu_parity import _compare
from tests.test_gpu_walk import _oracle, _plain, _run

TDET = (0.1, -0.05, 2, 2, 0.25, 0.25, 0.15, 0, 20, 150000)


def _desc(photons, width, timed, per_voxel=0):
    return mc.run_desc(photons, det=mc.Detector(0.0, 0.0, 0.05, 0.05, 30, 30), fluence=1, seed_exc=5, seed_fl=6,
                       photons_per_voxel=per_voxel, tdet=TDET if timed else None, width=width, height=width,
                       kind=mc.SOURCE_WIDEFIELD if width else mc.SOURCE_GAUSS_BEAM)


# The pass form is an option of untimed launches alone, so the other side of a timed run is the untimed one of the same
# seeds in the transport kernel's branching pass: the time of flight draws no random numbers.  Few voxel columns under
# the source (hitting densities summed over a photon's passes in a voxel) and more than 1024 of them (added pass by pass).
@pytest.mark.gpu
@pytest.mark.parametrize("width", [0.0, 0.5, 2.0, 3.9])
def test_timed_hitting_density_equals_untimed_branching_pass(width, gpu_ctx):
    lab, bulks, geo = _plain(40, 40, 8)
    med = gpu_ctx.medium(lab, bulks, **geo)
    timed = gpu_ctx.run(med, _desc(20011, width, True))
    try:
        gpu_ctx.set_option("pass_form", 1)
        ref = gpu_ctx.run(med, _desc(20011, width, False))
    finally:
        gpu_ctx.set_option("pass_form", 0)
        med.free()
    assert timed.time_xyt.any() and ref.time_xyt is None
    assert timed.fhd.any() and np.array_equal(timed.fhd, ref.fhd)
    assert np.array_equal(timed.Rd, ref.Rd) and np.array_equal(timed.Tt, ref.Tt)
    assert timed.stats_exc == ref.stats_exc


# fast math: the walk kernel states the roundings that the transport kernel's compiler chose for plain media
@pytest.mark.gpu
@pytest.mark.parametrize("width,per_voxel", [(0.0, 3), (3.9, 0)])
@pytest.mark.parametrize("variant", [0, 1, 2])
def test_fast_walk_equals_transport_kernel(variant, width, per_voxel, mcfl_lib):
    ctx = mc.Context(math=mc.MATH_FAST, variant=variant)
    lab, bulks, geo = _plain(40, 40, 8)
    med = ctx.medium(lab, bulks, **geo)
    rd = _desc(100003, width, False, per_voxel)
    want = ctx.run(med, rd)
    for option, value in (("pass_form", 1), ("phd_agg", 1), ("phd_agg", 2)):
        ctx.set_option(option, value)
        got = ctx.run(med, rd)
        ctx.set_option(option, 0)
        for k in ("Rd", "Tt", "fhd") + (("flR128", "flT128") if per_voxel else ()):
            assert np.array_equal(getattr(got, k), getattr(want, k)), (option, value, k)
        assert got.stats_exc == want.stats_exc and got.stats_fl == want.stats_fl
    med.free()
    ctx.close()


# photons that start outside the slab: below it they cross it without a step draw, above it their first step may end
# above it too
@pytest.mark.gpu
@pytest.mark.parametrize("source", [(0.0, 0.0, 0.35), (0.1, 0.0, 0.3), (0.0, 0.1, -0.02)])
def test_sources_outside_the_slab_bit_identical_to_oracle(source, gpu_ctx, oracle, table32768):
    lab, bulks, geo = _plain(9, 10, 6)
    sim, ref = _oracle(oracle, table32768, lab, bulks, geo, 3000, 0, source)
    _compare(_run(gpu_ctx, lab, bulks, geo, sim, 3000, 0, source), ref, emission=False)
