"""The work that a user of this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values; prepare() makes what a user's program holds before the call (the
scene resident on the device, rays, a batch), run() is one pass through the public entry points, and
exact() gives the result of the per-ray cases in 64-bit numpy.  The kinds:

  phase    Context.run_phase of the stellar emission, then the instruments (and, where the scene
           keeps it, the absorbed luminosity per cell) read back: a simulation without dust emission
  dust     the phases of a panchromatic simulation with dust self-absorption and dust emission
           (MonteCarloSimulation), then its frame, dust temperatures and absorbed totals
  batch    one Batch.run over several parameter variants of one model, every frame read back: what a
           fit evaluates in a generation
  tau      Context.optical_depth: optical depth maps and checks
  paths    Context.trace_paths_noalloc: the cells and lengths along rays, into the caller's device buffers

Grids depend on the case alone and are kept for the process (a user builds one grid and runs many
simulations on it); packets, rays, dust optical depth and viewing angles come from the seed.
"""
import functools
import math
import random

import numpy as np
import torch

from skirt7_b200 import _abi as A
from skirt7_b200 import models, runtime
from skirt7_b200.scene import DEG, KPC, MPC, CartesianDustGrid, FullInstrument

EXT = (-20 * KPC, -20 * KPC, -2 * KPC, 20 * KPC, 20 * KPC, 2 * KPC)


def listed():
    return [
        # a quick look at a small model before the real run: few packets, where launches and latency count
        dict(name="quick_look", kind="phase", grid="cartesian", nx=40, ny=40, nz=20, nl=1, packets=10000, npix=60,
             fp64=False, absorb=True, full=False),
        # the plain oligochromatic simulation (benchmark configuration 1) with its default packet count
        dict(name="oligo_cartesian", kind="phase", grid="cartesian", nx=100, ny=100, nz=50, nl=1, packets=1000000,
             npix=300, fp64=False, absorb=True, full=False),
        # the same kind of run with the 64-bit traversal, on a grid of odd sizes and three bands
        dict(name="cartesian_fp64", kind="phase", grid="cartesian", nx=101, ny=97, nz=33, nl=3, packets=77777,
             npix=255, fp64=True, absorb=False, full=False),
        # a small tree simulation with every flux component recorded (FullInstrument)
        dict(name="octree_full_instrument", kind="phase", grid="octree", level=7, fraction=1e-4, nl=8, packets=30001,
             npix=64, fp64=False, absorb=False, full=True),
        # the headline: panchromatic octree disk, 50 wavelengths, three 512 x 512 frames (2,986,747 leaves)
        dict(name="octree_pan", kind="phase", grid="octree", level=10, fraction=1e-6, nl=50, packets=400000, npix=512,
             fp64=False, absorb=False, full=False),
        # the stellar phase on a k-d tree with the absorbed luminosity kept, odd packet count
        dict(name="kdtree_absorption", kind="phase", grid="kdtree", level=26, fraction=3e-6, nl=10, packets=333333,
             npix=256, fp64=False, absorb=True, full=False),
        # a full panchromatic simulation: stellar phase, dust self-absorption, dust emission
        dict(name="kdtree_dust_emission", kind="dust", grid="kdtree", level=26, fraction=3e-6, nl=40, packets=100000,
             npix=512),
        # a clumpy model on a small Voronoi grid
        dict(name="voronoi_small", kind="phase", grid="voronoi", sites=20000, nl=1, packets=100000, npix=100,
             fp64=False, absorb=False, full=False),
        # the clumpy Voronoi configuration, 10^6 sites
        dict(name="voronoi_clumpy", kind="phase", grid="voronoi", sites=1000000, nl=1, packets=2000000, npix=300,
             fp64=False, absorb=False, full=False),
        # one generation of a fit: parameter variants on grids of different sizes in one launch
        dict(name="fit_batch", kind="batch", variants=24, nmin=32, nmax=128, packets=100000, npix=256),
        # optical depths along many lines of sight
        dict(name="optical_depth", kind="tau", grid="cartesian", nx=100, ny=100, nz=50, rays=200000, fp64=True),
        # the cells along rays, as a user inspects a grid with
        dict(name="trace_paths", kind="paths", grid="cartesian", nx=100, ny=100, nz=50, rays=20000, fp64=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["cartesian", "cartesian", "octree", "octree", "kdtree", "voronoi", "dust", "batch", "tau",
                       "paths"])
    npix = _log(rng, 32, 512)
    if what == "cartesian":
        return dict(kind="phase", grid="cartesian", nx=_log(rng, 8, 128), ny=_log(rng, 8, 128), nz=_log(rng, 4, 64),
                    nl=rng.randint(1, 3), packets=_log(rng, 1000, 700000), npix=npix, fp64=rng.random() < 0.25,
                    absorb=rng.random() < 0.6, full=rng.random() < 0.25)
    if what in ("octree", "kdtree"):
        level = rng.randint(6, 9) if what == "octree" else rng.randint(15, 26)
        return dict(kind="phase", grid=what, level=level, fraction=10 ** rng.uniform(-5.3, -3.5),
                    nl=rng.randint(2, 50), packets=_log(rng, 500, 100000), npix=min(npix, 256),
                    fp64=rng.random() < 0.15, absorb=rng.random() < 0.4, full=rng.random() < 0.25)
    if what == "voronoi":
        return dict(kind="phase", grid="voronoi", sites=_log(rng, 3000, 200000), nl=1, packets=_log(rng, 1000, 1000000),
                    npix=npix, fp64=rng.random() < 0.15, absorb=rng.random() < 0.4, full=False)
    if what == "dust":
        return dict(kind="dust", grid="kdtree", level=rng.randint(15, 26), fraction=10 ** rng.uniform(-5.3, -3.5),
                    nl=rng.randint(12, 48), packets=_log(rng, 1000, 60000), npix=npix)
    if what == "batch":
        return dict(kind="batch", variants=rng.randint(2, 24), nmin=rng.randint(16, 48), nmax=rng.randint(49, 128),
                    packets=_log(rng, 2000, 100000), npix=min(npix, 256))
    return dict(kind=what, grid="cartesian", nx=_log(rng, 8, 128), ny=_log(rng, 8, 128), nz=_log(rng, 4, 64),
                rays=_log(rng, 100, 200000 if what == "tau" else 20000), fp64=rng.random() < 0.7)


# ---------------------------------------------------------------------------------------------
# grids and scenes

@functools.lru_cache(maxsize=None)
def _tree(grid, level, fraction):
    model = models.pan_disk(nlambda=2, inclinations=(60,), npix=32)
    kd = grid == "kdtree"
    return runtime.build_tree(model, A.GRID_BINTREE if kd else A.GRID_OCTREE, EXT, minLevel=6 if kd else 2,
                              maxLevel=level, maxMassFraction=fraction, sampleCount=100, seed=4357)


@functools.lru_cache(maxsize=None)
def _voronoi(nsites):
    """80 % of the sites from the dust disk, 20 % uniform in the box."""
    rng = np.random.default_rng(77)
    lo, hi = np.array(EXT[:3]), np.array(EXT[3:])
    base = models.clumpy_disk(clumps=1).dustComps[0].geometry.geometry
    d = np.zeros((0, 3))
    nd = int(0.8 * nsites)
    while len(d) < nd:
        q = models.sample_expdisk(base, nsites, rng).reshape(-1, 3)
        d = np.concatenate([d, q[np.all((q > lo) & (q < hi), axis=1)]])
    return runtime.build_voronoi(np.concatenate([d[:nd], lo + rng.random((nsites - nd, 3)) * (hi - lo)]), EXT)


def _full_instrument(case, inclination):
    return FullInstrument(scatteringLevels=3, distance=10 * MPC, inclination=inclination, pixelsX=case["npix"],
                          pixelsY=case["npix"], fieldOfViewX=40 * KPC, fieldOfViewY=40 * KPC, instrumentName="full")


def _model(case, seed):
    rng = random.Random(seed)
    tau, turn = math.exp(rng.uniform(-0.4, 0.4)), rng.uniform(-2, 2)
    nl = case["nl"]
    if case["grid"] == "cartesian":
        m = models.oligo_disk(N=(case["nx"], case["ny"], case["nz"]), tauV=tau, inclination=(80 + turn) * DEG,
                              npix=case["npix"], wavelengths=[(0.45 + 0.1 * i) * 1e-6 for i in range(nl)],
                              write_absorption=case["absorb"])
    elif case["grid"] == "voronoi":
        m = models.clumpy_disk(tauV=5 * tau, seed=seed % 1000, wavelengths=[(0.45 + 0.1 * i) * 1e-6 for i in range(nl)],
                               npix=case["npix"])
        m.dustGrid = _voronoi(case["sites"])
        m.writeAbsorption = case["absorb"]
    elif case["kind"] == "dust":
        m = models.pan_disk(nlambda=nl, lmin=0.1e-6, lmax=1000e-6, inclinations=(60 + turn,), npix=case["npix"],
                            tauV=tau, point_fraction=0.1, dust_emission=True, write_absorption=True)
        m.dustGrid = _tree("kdtree", case["level"], case["fraction"])
        return m
    else:
        m = models.pan_disk(nlambda=nl, inclinations=(0, 60 + turn, 88), npix=case["npix"], tauV=tau,
                            write_absorption=case["absorb"])
        m.dustGrid = _tree(case["grid"], case["level"], case["fraction"])
    if case["full"]:
        m.instruments.append(_full_instrument(case, (30 + turn) * DEG))
    return m


def _disk_density(case, seed):
    """Densities of an exponential disk at the cell centres, with a factor of its own per cell."""
    g = CartesianDustGrid(EXT[0], EXT[3], EXT[1], EXT[4], EXT[2], EXT[5], case["nx"], case["ny"], case["nz"])
    x, y, z = (0.5 * (v[1:] + v[:-1]) for v in (g.xv, g.yv, g.zv))
    R = np.hypot(x[:, None], y[None, :])[:, :, None]
    f = np.exp(-R / (6 * KPC) - np.abs(z) / (0.25 * KPC)) * np.random.default_rng(seed).uniform(0.5, 2, R.shape[:2] + z.shape)
    return g, (f * 1.5 / (models.KAPPA_V_DEFAULT * 0.5 * KPC)).reshape(1, -1)


def _rays(case, seed):
    """Origins anywhere in the box, isotropic directions."""
    rng = np.random.default_rng(seed)
    n = case["rays"]
    lo, hi = np.array(EXT[:3]), np.array(EXT[3:])
    r = lo + (0.001 + 0.998 * rng.random((n, 3))) * (hi - lo)
    cost, phi = rng.uniform(-1, 1, n), rng.uniform(0, 2 * math.pi, n)
    st = np.sqrt(1 - cost ** 2)
    return r, np.ascontiguousarray(np.stack([st * np.cos(phi), st * np.sin(phi), cost], 1))


@functools.lru_cache(maxsize=None)
def _stream():
    """The stream of the calls into device buffers: one for the program, as they share the library's scratch."""
    return torch.cuda.Stream()


def _capacity(case):
    return case["rays"] * (case["nx"] + case["ny"] + case["nz"])


def _precision(case):
    return A.PREC_FP64 if case["fp64"] else A.PREC_FP32


def _host_frames(ctx, pinned):
    """Page-locked buffers that the instruments are read into, as a program that steps keeps them;
    a single small run reads into fresh arrays."""
    if not pinned:
        return [None] * len(ctx.model.instruments)
    out = []
    for ins in ctx.model.instruments:
        n = ctx.nlambda * (ins.pixelsX * ins.pixelsY)
        out.append((torch.zeros(n, dtype=torch.float64, pin_memory=True).numpy(), np.zeros(ctx.nlambda)))
    return out


# ---------------------------------------------------------------------------------------------
# the passes

def prepare(case, seed):
    kind = case["kind"]
    if kind == "phase":
        ctx = runtime.Context(_model(case, seed))
        return dict(case=case, ctx=ctx, seed=seed, out=_host_frames(ctx, case["grid"] == "octree" and not case["full"]))
    if kind == "dust":
        sim = runtime.MonteCarloSimulation(_model(case, seed), case["packets"], seed=seed, selfAbsorption=True, cycles=1)
        sim.setup()
        return dict(case=case, sim=sim)
    if kind == "batch":
        rng = random.Random(seed)
        ctxs, npp = [], []
        sizes = random.Random(case["variants"])
        for _ in range(case["variants"]):
            p = (rng.uniform(3, 9) * KPC, rng.uniform(0.1, 0.5) * KPC, math.exp(rng.uniform(math.log(0.2), math.log(4))),
                 rng.uniform(75, 90) * DEG, rng.uniform(0, 0.5))
            ctxs.append(runtime.Context(models.fit_variant(p, sizes.randint(case["nmin"], case["nmax"]), npix=case["npix"])))
            npp.append(int(case["packets"] * math.exp(sizes.uniform(-1, 0.5))))
        return dict(case=case, ctxs=ctxs, npp=npp, seed=seed,
                    batch=runtime.Batch(max_slots=32, max_items=64, max_ells=256))
    g, rho = _disk_density(case, seed)
    m = models.oligo_disk(N=(2, 2, 2), npix=16)
    m.dustGrid, m.rho = g, rho
    s = dict(case=case, ctx=runtime.Context(m), rays=_rays(case, seed))
    if kind == "paths":
        s["capacity"] = _capacity(case)
        s["rays"] = tuple(torch.from_numpy(v).cuda() for v in s["rays"])
        s["segments"] = (torch.zeros(case["rays"] + 1, dtype=torch.int64, device="cuda"),
                         torch.zeros(s["capacity"], dtype=torch.int32, device="cuda"),
                         torch.zeros(s["capacity"], dtype=torch.float64, device="cuda"))
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "phase":
        ctx = state["ctx"]
        ctx.reset_tallies()
        ctx.run_phase(A.PHASE_STELLAR, np.arange(case["nl"]), case["packets"], seed=state["seed"],
                      precision=_precision(case))
        got = [ctx.read_instrument(i, out=out) for i, out in enumerate(state["out"])]
        if case["absorb"]:
            got.append(ctx.read_absorption()[0])
        return got
    if kind == "dust":
        sim = state["sim"]
        sim.ctx.reset_tallies()
        sim.runstellaremission()
        sim.rundustselfabsorption()
        sim.rundustemission()
        return dict(frame=sim.ctx.read_instrument(0), temperature=sim.ctx.calc_dust_emission(),
                    absorbed=sim.ctx.absorbed_totals())
    if kind == "batch":
        for ctx in state["ctxs"]:
            ctx.reset_tallies()
        state["batch"].run(A.PHASE_STELLAR, [(ctx, [0, 1, 2], n, 0, n, state["seed"] + i)
                                             for i, (ctx, n) in enumerate(zip(state["ctxs"], state["npp"]))])
        state["batch"].sync()
        return [ctx.read_instrument(0)[0] for ctx in state["ctxs"]]
    r, k = state["rays"]
    if kind == "tau":
        return state["ctx"].optical_depth(r, k, precision=_precision(case))
    off, cells, ds = state["segments"]
    state["ctx"].trace_paths_noalloc(r.data_ptr(), k.data_ptr(), case["rays"], cells.data_ptr(), ds.data_ptr(),
                                     off.data_ptr(), state["capacity"], precision=_precision(case),
                                     stream=_stream().cuda_stream)
    return off, cells, ds


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    """Bytes: the grid (cell densities and what locates a cell) read once, the results written once.
    Flops: about 20 per cell step of the walks (exit distances of three axes, the step, its optical
    depth), with the mean number of cells a walk crosses and about 16 walks per packet (peel-offs,
    paths, re-walks)."""
    kind = case["kind"]
    if kind in ("tau", "paths"):
        cells = case["nx"] * case["ny"] * case["nz"]
        crossed = 0.12 * (case["nx"] + case["ny"] + 4 * case["nz"])
        out = case["rays"] * (8 if kind == "tau" else 8 + 12 * crossed)
        return dict(bytes=8 * cells + 48 * case["rays"] + out, flops=20 * crossed * case["rays"])
    if kind == "batch":
        side = 0.5 * (case["nmin"] + case["nmax"])
        packets = 3 * 0.85 * case["packets"] * case["variants"]
        return dict(bytes=case["variants"] * (4 * side ** 3 + 24 * case["npix"] ** 2),
                    flops=20 * packets * 11 * 0.4 * side)
    nl = case["nl"]
    if case["grid"] == "cartesian":
        cells, steps = case["nx"] * case["ny"] * case["nz"], 1.8 * (case["nx"] + case["ny"] + case["nz"])
    elif case["grid"] == "voronoi":
        cells, steps = case["sites"], 6 * case["sites"] ** (1 / 3)
    else:
        cells = 3 / case["fraction"]
        steps = (9 if case["grid"] == "octree" else 3.5) * cells ** (1 / 3)
    frames = 8 * nl * case["npix"] ** 2 * (3 if case["grid"] in ("octree", "kdtree") and kind == "phase" else 1)
    if kind == "dust":
        packets = 3.43 * nl * case["packets"]
        return dict(bytes=32 * cells + frames + 5 * 8 * nl * cells, flops=20 * steps * packets)
    out = frames + (8 * nl * cells if case["absorb"] else 0) + (9 * 8 * nl * case["npix"] ** 2 if case["full"] else 0)
    per = 4 if case["grid"] == "cartesian" else 32 if case["grid"] != "voronoi" else 260
    return dict(bytes=per * cells + out, flops=20 * steps * nl * case["packets"])


def exact(case, seed):
    """The per-ray cases by sorting every ray's plane crossings, in 64 bits."""
    if case["kind"] not in ("tau", "paths"):
        return None
    g, rho = _disk_density(case, seed)
    r, k = _rays(case, seed)
    planes = (g.xv, g.yv, g.zv)
    n = [len(v) - 1 for v in planes]
    tau, counts, cells, lengths = [], [], [], []
    for a in range(0, len(r), 20000):
        rr, kk = r[a:a + 20000], k[a:a + 20000]
        t = [(v[None, :] - rr[:, i:i + 1]) / kk[:, i:i + 1] for i, v in enumerate(planes)]
        end = np.min([x.max(1) for x in t], axis=0)
        cross = np.concatenate([np.zeros((len(rr), 1))] + t, axis=1)
        cross = np.sort(np.clip(cross, 0, end[:, None]), axis=1)
        ds = np.diff(cross, axis=1)
        mid = 0.5 * (cross[:, 1:] + cross[:, :-1])
        idx = []
        for i, v in enumerate(planes):
            p = (rr[:, i:i + 1] + mid * kk[:, i:i + 1] - v[0]) / (v[1] - v[0])
            idx.append(np.clip(p.astype(np.int64), 0, n[i] - 1))
        m = idx[2] + n[2] * (idx[1] + n[1] * idx[0])
        if case["kind"] == "tau":
            tau.append((models.KAPPA_V_DEFAULT * rho[0][m] * ds).sum(1))
        else:
            on = ds > 0
            counts.append(on.sum(1))
            cells.append(m[on].astype(np.int32))
            lengths.append(ds[on])
    if case["kind"] == "tau":
        return np.concatenate(tau)
    off = np.concatenate([[0], np.cumsum(np.concatenate(counts))]).astype(np.int64)
    cells, lengths = np.concatenate(cells), np.concatenate(lengths)
    rest = (0, _capacity(case) - len(cells))
    return off, np.pad(cells, rest), np.pad(lengths, rest)
