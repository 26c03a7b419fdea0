"""The label tiles of the walk kernel: built for the launches that read them
and no others, the L2 window over the array that the launch's kernel reads,
and a run without room for tiles taken by the transport kernel."""
import numpy as np
import pytest

import cudamcfl_gb300 as mc
from tests.test_gpu_walk import _plain

DET = mc.Detector(0.0, 0.0, 0.05, 0.05, 30, 30)
TDET = (0.1, -0.05, 2, 2, 0.25, 0.25, 0.15, 0, 20, 150000)


def _tile_bytes(nx, ny, nz):
    return 16 * (nx + 1) * (ny // 4 + 1) * (nz // 4 + 1)


def _desc(**more):
    return mc.run_desc(500, det=DET, seed_exc=3, fluence=1, **more)


# options of a launch, whether the run is timed, and whether it reads tiles (a timed launch has one form, the walk
# kernel's; FP64 and voxel-boundary stepping have none)
@pytest.mark.gpu
@pytest.mark.parametrize("math,options,more,walk",
                         [(mc.MATH_FAST, {}, {}, True), (mc.MATH_EXACT, dict(variant=2), {}, True),
                          (mc.MATH_FAST, dict(pass_form=1), {}, False), (mc.MATH_FAST, dict(phd_agg=1), {}, False),
                          (mc.MATH_EXACT, dict(phd_agg=2), {}, False), (mc.MATH_F64, {}, {}, False),
                          (mc.MATH_FAST, dict(pass_form=1), dict(tdet=TDET), True),
                          (mc.MATH_FAST, {}, dict(exact_stepping=1), False)])
@pytest.mark.parametrize("tiles_first", [False, True])
def test_tiles_and_window_follow_the_kernel(math, options, more, walk, tiles_first, mcfl_lib):
    nx, ny, nz = 21, 18, 11
    lab, bulks, geo = _plain(nx, ny, nz)
    ctx = mc.Context(math=math, l2_window=1, **options)
    med = ctx.medium(lab, bulks, **geo)
    created = med.nbytes
    if tiles_first:  # from a run in the first form, fast math
        for k, v in dict(math=mc.MATH_FAST, pass_form=0, phd_agg=0).items():
            ctx.set_option(k, v)
        ctx.run(med, _desc())
        assert med.nbytes == created + _tile_bytes(nx, ny, nz)
        ctx.set_option("math", math)
        for k, v in options.items():
            ctx.set_option(k, v)
    ctx.run(med, _desc(**more))
    tiles = _tile_bytes(nx, ny, nz) if walk or tiles_first else 0
    stepping = 2 * lab.size if more.get("exact_stepping") else 0
    assert med.nbytes == created + tiles + stepping
    assert ctx.get_option("l2_window_bytes") == (_tile_bytes(nx, ny, nz) if walk else lab.size)
    mc.batch_run(ctx, med, [mc.run_desc(100, det=DET, **more)] * 2, images=False)
    assert ctx.get_option("l2_window_bytes") == (_tile_bytes(nx, ny, nz) if walk else lab.size)
    med.free()
    ctx.close()


@pytest.mark.gpu
def test_run_without_room_for_tiles_goes_on(mcfl_lib):
    """Tiles of a grid one voxel thick are four times its labels (the padding
    voxel takes a tile of its own).  Tiles in place are given back to a run
    whose buffers need the room, and a run with no room for them goes through
    the transport kernel, with the same tallies."""
    torch = pytest.importorskip("torch")
    n = 8192
    tiles = _tile_bytes(n, n, 1)  # 256 MiB; the hitting density and its normalised image 512 MiB each
    lab = np.ones((1, n, n), dtype=np.uint8)
    bulks = [mc.outer_bulk(1.0), mc.bulk_from_mci_columns(1.4, 0.1, 100.0, g=0.9), mc.outer_bulk(1.0)]
    ctx = mc.Context(math=mc.MATH_FAST)
    med = ctx.medium(lab, bulks, half_x=4.0, half_y=4.0, thickness=0.5, vox_per_cm=(n / 8.0, n / 8.0, 2.0))
    created = med.nbytes

    def run(fluence):
        r = ctx.run(med, mc.run_desc(2000, det=DET, seed_exc=3, fluence=fluence), images=False)
        return r.Rd, np.array(list(r.stats_exc.values()), dtype=np.uint64)

    want = run(0)
    assert med.nbytes == created + tiles
    torch.cuda.synchronize()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (900 << 20), dtype=torch.uint8, device="cuda")
    for fluence, room in ((1, False), (0, False), (1, True)):
        if room:
            del hold
            torch.cuda.empty_cache()
        got = run(fluence)
        assert med.nbytes == created + (tiles if room else 0)
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
    med.free()
    ctx.close()
