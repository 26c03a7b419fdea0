"""The work users of this engine have it do, as cases that can be timed.

A case goes through the package's public calls (Context.medium, Context.run,
batch_run, Server) with the options a user's program sets; whatever it does
not set keeps its default.  Media are seeded and synthetic: a slab with
spheres and cylinders of other labels burned into a background, as the media
of the benchmark (config1: 50^3 voxels and one sphere; config2: 200 x 200 x
100 voxels, 8 labels and a fluorophore map).

Every tally is a whole number that the photon's random stream and the
single-precision arithmetic of its walk decide, and the floating images are
those whole numbers over a constant.
"""
import math

import numpy as np

import cudamcfl_gb300 as mc
from cudamcfl_gb300 import media

MATH = {"exact": mc.MATH_EXACT, "fast": mc.MATH_FAST}

# Transport passes of one photon in these media (background mua 0.1/cm, mus
# 100/cm, g 0.9, n 1.4, slab of 2 cm), about: excitation from a beam on the
# face, emission from inside; and the floating-point operations of a pass.
PASSES_EXC, PASSES_FL, FLOPS = 700, 850, 60


def listed():
    return [
        # a first look at a medium: the default context (strict IEEE math), a couple of thousand photons, both
        # phases; latency of one call
        dict(name="look_exact", kind="run", medium="sphere", math="exact", nx=50, ny=50, nz=50, photons=1999,
             emission=2000),
        # the same look with the fast math, excitation images only, on a small odd grid
        dict(name="look_fast", kind="run", medium="inclusions", math="fast", nx=37, ny=41, nz=29, photons=20011,
             emission=0, fluence=0),
        # config1 at its budget of 1e6 photons: the plain method's ordinary run, both phases
        dict(name="sphere_1e6", kind="run", medium="sphere", math="fast", nx=50, ny=50, nz=50, photons=1000000,
             emission=250000),
        # the same kind of run in strict IEEE math, for results that are compared bit by bit
        dict(name="inclusions_exact", kind="run", medium="inclusions", math="exact", nx=96, ny=96, nz=64,
             photons=1000000, emission=500000),
        # config2 at a fifth of its excitation budget, with the options the autotuner picks for it: the headline
        dict(name="voxels_two_phase", kind="run", medium="inclusions", math="fast", nx=200, ny=200, nz=100,
             photons=20000000, emission=20000000, variant=1, relaunch=2),
        # tissue whose labels differ in refractive index, one of them free of scattering
        dict(name="indices", kind="run", medium="indices", math="fast", nx=121, ny=117, nz=83, photons=2000000,
             emission=1000000),
        # wide-field illumination of a large grid, with the photon hitting density
        dict(name="widefield_large", kind="run", medium="inclusions", math="fast", nx=256, ny=256, nz=128,
             photons=4000000, emission=0, source="wide"),
        # time-resolved reflectance
        dict(name="time_resolved", kind="run", medium="inclusions", math="fast", nx=128, ny=128, nz=64,
             photons=2000000, emission=0, timed=1),
        # layered medium with an inclusion (bulk method 1)
        dict(name="layered", kind="layered", math="fast", grid=20, photons=1000003),
        # a raster of beams over one medium, uneven budgets, each with its own images
        dict(name="raster", kind="batch", medium="sphere", math="fast", nx=50, ny=50, nz=50, runs=30, media=1,
             lo=20000, hi=1000000),
        # voxel-boundary stepping, both phases
        dict(name="boundary_stepping", kind="run", medium="inclusions", math="fast", nx=160, ny=160, nz=80,
             photons=1000000, emission=1000000, stepping=1),
        # requests with media of their own, queued at the server
        dict(name="served", kind="serve", medium="inclusions", math="fast", nx=128, ny=128, nz=64, runs=10,
             lo=100000, hi=2000000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "layered", "batch", "batch", "serve"])
    if kind == "layered":
        return dict(kind="layered", math=rng.choice(["fast", "exact"]), grid=rng.randrange(8, 33),
                    photons=_log(rng, 2000, 4000000), timed=rng.choice([0, 1]))
    c = dict(kind=kind, medium=rng.choice(["sphere", "inclusions", "inclusions", "indices"]),
             math=rng.choice(["fast", "fast", "exact"]), nx=_log(rng, 24, 256), ny=_log(rng, 24, 256),
             nz=_log(rng, 20, 128))
    if kind == "run":
        c["stepping"] = int(rng.random() < 0.2)
        c["timed"] = int(rng.random() < 0.2)
        c["source"] = rng.choice(["beam", "beam", "wide"])
        c["photons"] = _log(rng, 1000, 3000000 if c["stepping"] or c["math"] == "exact" else 8000000)
        c["emission"] = rng.choice([0, 1]) * _log(rng, 1000, c["photons"] + 1000)
        if c["math"] == "fast" and rng.random() < 0.5:
            c["variant"], c["relaunch"] = rng.randrange(3), rng.choice([1, 2])
        return c
    c["runs"] = rng.randrange(2, 31 if kind == "batch" else 13)
    c["media"] = rng.choice([1, 3, 5]) if kind == "batch" else 1
    c["lo"] = _log(rng, 1000, 100000)
    c["hi"] = c["lo"] * rng.randrange(2, 11)
    if kind == "serve":
        c["nx"], c["ny"], c["nz"] = min(c["nx"], 160), min(c["ny"], 160), min(c["nz"], 96)
    return c


# ------------------------------------------------------------------ media

def _medium(case, seed):
    """labels, bulks, voxel size and fluorophore map of a 4 x 4 x 2 cm slab."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    vox = (4.0 / nx, 4.0 / ny, 2.0 / nz)
    rng = np.random.default_rng([seed, nx, ny, nz])
    lab = np.ones((nz, ny, nx), dtype=np.uint8)
    if case["medium"] == "sphere":
        centre = (float(rng.uniform(-0.2, 0.2)), float(rng.uniform(-0.2, 0.2)), 1.0)
        media.add_sphere(lab, vox, centre, 0.25, 2)
        bulks = [mc.outer_bulk(1.0), mc.bulk_from_mci_columns(1.4, 0.1, 100.0, g=0.9),
                 mc.bulk_from_mci_columns(1.4, 0.1, 100.0, 1.0, 0.05, 0.05, 0.1, 0.9), mc.outer_bulk(1.0)]
        return lab, bulks, vox, None
    n_labels = 8
    indices = case["medium"] == "indices"
    bulks = [mc.outer_bulk(1.0), mc.bulk_from_mci_columns(1.4, 0.1, 100.0, g=0.9)]
    for i in range(2, n_labels + 1):
        n = float(rng.uniform(1.33, 1.52)) if indices else 1.4
        mus = 0.0 if indices and i == n_labels else float(rng.uniform(50.0, 150.0))
        fl = 1.0 if mus else 0.0
        bulks.append(mc.bulk_from_mci_columns(n, float(rng.uniform(0.02, 0.5)), mus, fl,
                                              fl * float(rng.uniform(0.01, 0.1)), fl * float(rng.uniform(0.005, 0.05)),
                                              fl * float(rng.uniform(0.05, 0.2)), float(rng.uniform(0.8, 0.95))))
    bulks.append(mc.outer_bulk(1.0))
    fmap = np.zeros(lab.shape, dtype=np.float32)
    fval = rng.random(size=lab.shape, dtype=np.float32)
    for k in range(int(rng.integers(6, 16))):
        label = n_labels if indices and k == 0 else int(rng.integers(2, n_labels + 1))
        c = (float(rng.uniform(-1.5, 1.5)), float(rng.uniform(-1.5, 1.5)), float(rng.uniform(0.3, 1.7)))
        if rng.uniform() < 0.5:
            media.add_sphere(lab, vox, c, float(rng.uniform(0.1, 0.5)), label, fmap, fval)
        else:
            media.add_cylinder(lab, vox, c, rng.normal(size=3), float(rng.uniform(0.05, 0.3)),
                               float(rng.uniform(0.3, 1.5)), label, fmap, fval)
    return lab, bulks, vox, fmap


def _layers(case, seed):
    rng = np.random.default_rng([seed, case["grid"]])
    n2 = float(rng.uniform(1.33, 1.5))
    layers = mc.layers_from_mci_columns(1.0, [(1.4, 0.1, 90.0, 0, 0, 0, 0, 0.9, 0.3),
                                              (n2, 0.3, 60.0, 0, 0, 0, 0, 0.8, 0.7)], 1.0)
    return layers, mc.inclusion_from_mci_columns(0.1, -0.05, 0.4, 0.2, 1.4, 0.8, 70.0, g=0.85)


DETECTOR = (0.0, 0.0, 0.04, 0.04, 100, 100)  # 100 x 100 pixels of 0.04 cm
TIMED = (0.1, -0.05, 3, 2, 0.25, 0.25, 0.15, 0, 40, 150000)  # 3 x 2 discs on the entry face, 40 bins over 0.15 ns


def _context(case):
    options = {k: case[k] for k in ("variant", "relaunch") if k in case}
    return mc.Context(math=MATH[case["math"]], **options)


def _desc(case, photons, seed, **more):
    wide = dict(kind=mc.SOURCE_WIDEFIELD, width=4.0, height=4.0) if case.get("source") == "wide" else {}
    if case.get("timed"):
        more["tdet"] = TIMED
    return mc.run_desc(photons, det=mc.Detector(*DETECTOR), seed_exc=2 * seed + 1, seed_fl=2 * seed + 2,
                       exact_stepping=case.get("stepping", 0), **wide, **more)


def _budgets(case, rng):
    return [int(b) for b in np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), case["runs"]))]


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng([seed, 77])
    if kind == "serve":  # media, budgets and sources as they reach the server, one after another
        reqs = []
        for i, b in enumerate(_budgets(case, rng)):
            c = dict(case, nx=max(24, case["nx"] - 16 * (i % 4)), nz=max(20, case["nz"] - 8 * (i % 3)),
                     source="wide" if i % 2 else "beam")
            reqs.append((_medium(c, seed + 1000 * i), _desc(c, b, seed + 1000 * i)))
        ctx = _context(case)
        return {"server": mc.Server(ctx, max_jobs=64), "ctx": ctx, "kind": kind, "requests": reqs}
    ctx = _context(case)
    if kind == "layered":
        layers, incl = _layers(case, seed)
        med = ctx.medium_layered(layers, incl, case["grid"])
        rd = _desc(case, case["photons"], seed, source=(0.05, 0.02, 0.0), fluence=1)
        return {"medium": med, "ctx": ctx, "kind": kind, "desc": rd}
    if kind == "batch":
        meds = []
        for k in range(case["media"]):
            lab, bulks, vox, _ = _medium(case, seed + 1000 * k)
            meds.append(ctx.medium(lab, bulks, voxel_cm=vox))
        side = math.ceil(math.sqrt(case["runs"]))
        runs = [_desc(case, b, seed + i, source=(3.0 * (i % side + 0.5) / side - 1.5, 3.0 * (i // side + 0.5) / side - 1.5, 0.0))
                for i, b in enumerate(_budgets(case, rng))]
        media_of = meds[0] if len(meds) == 1 else [meds[i % len(meds)] for i in range(len(runs))]
        return {"medium": media_of, "ctx": ctx, "kind": kind, "runs": runs}
    lab, bulks, vox, fmap = _medium(case, seed)
    per_voxel = 0
    if case["emission"]:  # photons per emitting voxel, from the emission photons wanted in all
        bright = np.array([b.albedof < 1 for b in bulks])[lab]
        if fmap is not None:
            bright &= fmap > 0
        per_voxel = max(1, case["emission"] // max(1, int(bright.sum())))
    med = ctx.medium(lab, bulks, voxel_cm=vox, fluor_map=fmap)
    rd = _desc(case, case["photons"], seed, photons_per_voxel=per_voxel, fluence=case.get("fluence", 1))
    return {"medium": med, "ctx": ctx, "kind": kind, "desc": rd}


def _whole(a):
    """64-bit tallies as the signed type every array library sums."""
    return a.view(np.int64) if a.dtype == np.uint64 else a


def _counters(stats):
    return np.array([list(s.values()) for s in stats], dtype=np.uint64).view(np.int64)


def run(state):
    kind = state["kind"]
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(lab, bulks, vox, rd, fluor_map=fmap) for (lab, bulks, vox, fmap), rd in state["requests"]]
        for i in ids:
            mc.check(srv.wait(i))
        res = [srv.result(i) for i in ids]
        out = {"%s%d" % (k, i): _whole(r[k]) for i, r in enumerate(res) for k in ("Rd", "Tt")}
        out["stats"] = _counters([r["stats"] for r in res])
        return out
    if kind == "batch":
        res, _ = mc.batch_run(state["ctx"], state["medium"], state["runs"], images=False)
        out = {"%s%d" % (k, i): _whole(r[k]) for i, r in enumerate(res) for k in ("Rd", "Tt")}
        out["stats"] = _counters([r["stats"] for r in res])
        return out
    r = state["ctx"].run(state["medium"], state["desc"])
    out = {k: _whole(v) for k in ("Rd", "Tt", "R", "T", "fhd", "phd", "flR", "flT", "flR128", "flT128", "time_xyt")
           if (v := getattr(r, k)) is not None}
    out["stats"] = _counters([r.stats_exc, r.stats_fl])
    out["energy"] = np.array(r.energy_exc)
    return out


def work(case):
    pixels = DETECTOR[4] * (DETECTOR[5] + 1)
    if case["kind"] in ("batch", "serve"):
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])  # of a log-uniform budget
        grid = case["nx"] * case["ny"] * case["nz"]
        media_read = case["runs"] if case["kind"] == "serve" else case["media"]
        return {"bytes": media_read * grid + case["runs"] * 2 * 8 * pixels,
                "flops": case["runs"] * mean * PASSES_EXC * FLOPS}
    if case["kind"] == "layered":
        return {"bytes": 16 * 16 * case["grid"] ** 3 + 4 * 8 * pixels,
                "flops": case["photons"] * PASSES_EXC * FLOPS}
    grid, em = case["nx"] * case["ny"] * case["nz"], case["emission"]
    tallies = 16 * grid if em or case.get("fluence", 1) else 0
    return {"bytes": grid + tallies + (4 * grid if em and case["medium"] != "sphere" else 0) +
            (4 + (6 if em else 0)) * 8 * pixels,
            "flops": (case["photons"] * PASSES_EXC + em * PASSES_FL) * FLOPS}


def exact(case, seed):
    """None: a tally counts where single-precision walks end.  A walk of
    several hundred scatterings in 64 bits parts from it after a few dozen, so
    no other arithmetic gives the same whole numbers."""
    return None
