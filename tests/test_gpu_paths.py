"""Kernel variants at the sizes where they can go wrong: edges of tiles, remainders, ties, extremes."""
import ctypes

import numpy as np
import pytest

from ekgsim_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

ECG_TOL = 1e-4  # the engine's bar against the FP64 oracle (rel-L2 over leads x steps)


@pytest.fixture(scope="module")
def engine():
    from ekgsim_gb300.engine import Engine
    e = Engine(0)
    yield e
    e.close()


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("shape,delays", [
    ((8, 8, 8), [1, 2, 2]),           # one tile
    ((9, 16, 17), [1, 2, 2]),         # one cell over a tile, exact tiles
    ((1, 70, 3), [0.3, 3, 1]),        # a strip through many tiles
    ((24, 23, 25), [0, 2, 1]),        # a zero delay: ties within a step
    ((24, 23, 25), [1e-9, 40, 0.7]),  # lags below the resolution of a time's high word
    ((31, 33, 32), [1.37, 0.71, 2.9]),
    ((40, 40, 9), [300, 0.5, 2]),     # most of a round's horizon empty
])
def test_activation_tiles(engine, shape, delays):
    """Activation times bit-exact against the oracle, through the heart's set-up and in caller-owned buffers:
    random layers with holes, two stimuli, tiles cut by the grid's edge."""
    import torch
    from ekgsim_gb300 import _lib as L
    from ekgsim_gb300.engine import Heart
    rng = np.random.Generator(np.random.PCG64(shape[0] * 100 + shape[2]))
    grid = rng.integers(0, 4, size=shape).astype(np.int32)
    grid[0, 0, 0] = -1
    grid[-1, shape[1] // 2, -1] = -3
    tm = synth.transfer_matrix(3, delays)
    ref, _ = O.activation(grid, tm)
    h = Heart.create(engine, grid, tm, np.array([[90.0, 95.0, 100.0]]), "3D4", 0.0, 10.0, 1.0)
    assert np.array_equal(h.activation().view(np.int64), ref.view(np.int64))
    h.close()
    layers = torch.from_numpy(grid).cuda()
    at = torch.full(shape, -7.0, dtype=torch.float64, device="cuda")
    t = np.ascontiguousarray(tm, dtype=np.float64)
    torch.cuda.synchronize()
    L.check(L.load().ekg_activation_noalloc(*shape, ctypes.c_void_p(layers.data_ptr()), t.shape[0], L.dptr(t),
                                            ctypes.c_void_p(at.data_ptr()), None))
    assert np.array_equal(at.cpu().numpy().view(np.int64), ref.view(np.int64))


@pytest.mark.parametrize("n,sims,moved", [(12, 2, 1), (20, 11, 3), (28, 33, 2)])
def test_resting_potential_rows(engine, n, sims, moved):
    """The resting-potential constant of the moved leads with fewer 8-AP parts in a layer than segments
    (12^3), rows that are no multiple of a warp or a block's rows, and a row over 64."""
    from ekgsim_gb300.engine import Heart, layer_aps, move_leads
    spec = synth.small_spec(n, n_leads=4, seed=5)
    grid, tm = synth.ellipsoid_heart(spec), synth.transfer_matrix(3, spec.delays)
    rng = np.random.Generator(np.random.PCG64(n))
    leads = synth.leads(spec, rng)[:, ::-1].copy()
    base = [[k0] + list(synth.BASE_AP[1:]) for k0 in (-86.0, -80.0, -90.0)]
    h = Heart.create(engine, grid, tm, leads, "3D4", 0.0, 200.0, 1.0)
    h.set_eval(base, synth.K_MIN, synth.K_MAX, [5, 6, 7, 8], list(synth.analytic_target(4, 200, 3)), mid_position=0.6)
    genes = np.zeros((sims, 12 + 8))
    genes[:, :12] = synth.GENE_MIN[:12] + (synth.GENE_MAX - synth.GENE_MIN)[:12] * rng.random((sims, 12))
    genes[:, 12:12 + 2 * moved] = rng.uniform(-20, 20, size=(sims, 2 * moved))
    ecg = h.eval_batch(genes, want_ecg=True)[2]
    at, layer = O.activation(grid, tm)
    for i in {0, sims // 2, sims - 1}:
        lk = layer_aps(h._cfg, 3, genes[i, :12])[0]
        ref = O.run(layer, at, lk, move_leads(leads, genes[i, 12:].reshape(-1, 2)), "3D4", 0.0, 200.0, 1.0)
        assert rel_l2(ecg[i], ref) <= ECG_TOL, i
    h.close()


@pytest.mark.parametrize("kind,sims,moved,nhood", [
    ("ellipsoid", 1, 1, "3D4"), ("ellipsoid", 4, 3, "3D4"), ("ellipsoid", 2, 2, "cube"),
    ("few times", 3, 2, "3D4"),  # thousands of voxels in an AP: the block's range in many parts
    ("few times", 1, 3, "cube"),
])
def test_few_simulations_operand(engine, kind, sims, moved, nhood):
    """The moved-lead operand of one to four simulations (a thread per voxel, then one per AP): odd and even
    numbers of moved leads, APs of one voxel up to thousands, both neighbourhoods."""
    from ekgsim_gb300.engine import Heart, layer_aps, move_leads
    rng = np.random.Generator(np.random.PCG64(sims * 10 + moved))
    if kind == "ellipsoid":
        spec = synth.small_spec(24, n_leads=4, seed=9)
        grid, tm = synth.ellipsoid_heart(spec), synth.transfer_matrix(3, spec.delays)
        at, layer = O.activation(grid, tm)
        given = None
    else:
        grid = rng.integers(1, 4, size=(17, 20, 19)).astype(np.int32)
        grid[rng.random(grid.shape) < 0.05] = 0
        tm = synth.transfer_matrix(3, [1, 2, 2])
        layer = grid.copy()
        given = at = np.where(grid > 0, np.floor(np.arange(20) / 10)[None, :, None] * 7.0 + 3.0, 0.0)
    leads = np.array(grid.shape) / 2 + 30.0 * np.array([[1.0, 0.2, 0.1], [-0.3, 1.0, 0.4], [0.2, -0.5, -1.0], [0.6, 0.7, 0.5]])
    h = Heart.create(engine, grid, tm, leads, nhood, 0.0, 150.0, 1.0, activation=given)
    h.set_eval([synth.BASE_AP] * 3, synth.K_MIN, synth.K_MAX, [5, 6, 7, 8], list(synth.analytic_target(4, 150, 3)),
               mid_position=0.6)
    genes = np.zeros((sims, 12 + 8))
    genes[:, :12] = synth.GENE_MIN[:12] + (synth.GENE_MAX - synth.GENE_MIN)[:12] * rng.random((sims, 12))
    genes[:, 12:12 + 2 * moved] = rng.uniform(-8, 8, size=(sims, 2 * moved))
    for _ in range(2):  # a single simulation takes the batched form from its second call on
        ecg = h.eval_batch(genes, want_ecg=True)[2]
    for i in range(sims):
        lk = layer_aps(h._cfg, 3, genes[i, :12])[0]
        ref = O.run(layer, at, lk, move_leads(leads, genes[i, 12:].reshape(-1, 2)), nhood, 0.0, 150.0, 1.0)
        assert rel_l2(ecg[i], ref) <= ECG_TOL, i
    h.close()


def small_heart(engine, n, n_leads, steps, free, seed):
    from ekgsim_gb300.engine import Heart
    spec = synth.small_spec(n, n_leads=n_leads, seed=seed)
    grid, tm = synth.ellipsoid_heart(spec), synth.transfer_matrix(3, spec.delays)
    rng = np.random.Generator(np.random.PCG64(seed))
    leads = synth.leads(spec, rng)[:, ::-1].copy()
    h = Heart.create(engine, grid, tm, leads, "3D4", 0.0, float(steps), 1.0)
    h.set_eval([synth.BASE_AP] * 3, synth.K_MIN, synth.K_MAX, free, list(synth.analytic_target(n_leads, steps, 3)),
               mid_position=0.6)
    return h, O.activation(grid, tm), leads, rng


def check_sims(h, act, leads, rng, sims, moved, free, steps):
    from ekgsim_gb300.engine import layer_aps, move_leads
    at, layer = act
    nk, nl = 3 * len(free), len(leads)
    lo, hi = np.array(synth.K_MIN)[free], np.array(synth.K_MAX)[free]
    genes = np.zeros((sims, nk + 2 * nl))
    genes[:, :nk] = np.tile(lo, 3) + np.tile(hi - lo, 3) * rng.random((sims, nk))
    genes[:, nk:nk + 2 * moved] = rng.uniform(-15, 15, size=(sims, 2 * moved))
    ecg = h.eval_batch(genes, want_ecg=True)[2]
    for i in {0, sims // 2, sims - 1}:
        lk = layer_aps(h._cfg, 3, genes[i, :nk])[0]
        ref = O.run(layer, at, lk, move_leads(leads, genes[i, nk:].reshape(-1, 2)), "3D4", 0.0, float(steps), 1.0)
        assert rel_l2(ecg[i], ref) <= ECG_TOL, i


@pytest.mark.parametrize("n_leads,steps", [(1, 61), (4, 300), (5, 97), (12, 257), (13, 64), (17, 129)])
def test_band_contraction_leads(engine, n_leads, steps):
    """Upstrokes that differ per simulation: every compiled number of leads per block, a block with few of its
    leads, steps that are no multiple of a pass or of the probes of a run's end."""
    free = [1, 5, 6, 7, 8]
    h, act, leads, rng = small_heart(engine, 22, n_leads, steps, free, seed=n_leads)
    check_sims(h, act, leads, rng, 9, min(2, n_leads), free, steps)
    h.close()


@pytest.mark.parametrize("sims,moved,steps", [
    (3, 2, 1400),    # as many steady entries per layer as there can be
    (467, 3, 300),   # outputs of the steady sums: thousands, no multiple of a warp's four
    (33, 1, 128),    # a group of 16 simulations with one of them
    (4000, 1, 64),   # inputs and criteria too large for the pass's own copies
])
def test_steady_sums_and_static_leads(engine, sims, moved, steps):
    """Batched passes with moved and static leads: the steady sums' two passes, the static leads' groups."""
    free = [5, 6, 7, 8]
    h, act, leads, rng = small_heart(engine, 20, 5, steps, free, seed=sims)
    check_sims(h, act, leads, rng, sims, moved, free, steps)
    h.close()


def test_fresh_result_pages(engine):
    """Results into memory that was never touched, at an odd offset in its pages: what goes into touched memory."""
    import mmap
    from ekgsim_gb300 import _lib as L
    h, act, leads, rng = small_heart(engine, 40, 2, 50, [5, 6, 7, 8], seed=1)
    want = h.activation()
    fresh = mmap.mmap(-1, want.nbytes + 4096)
    base = ctypes.addressof(ctypes.c_char.from_buffer(fresh))
    L.check(L.load().ekg_heart_activation(h._h, ctypes.cast(base + 1000, ctypes.POINTER(ctypes.c_double))))
    got = np.frombuffer(ctypes.string_at(base, len(fresh)), dtype=np.uint8)
    assert np.array_equal(got[1000:1000 + want.nbytes], want.reshape(-1).view(np.uint8))
    assert not got[:1000].any() and not got[1000 + want.nbytes:].any()
    h.close()


@pytest.mark.parametrize("shape,holes", [
    ((1, 1, 1), 0), ((1, 31, 33), 0), ((1, 32, 32), 0), ((25, 41, 1), 0), ((9, 17, 23), 0.2), ((31, 33, 35), 0.5),
])
def test_ap_order(engine, shape, holes):
    """De-duplicated APs in caller-given times whose bytes all differ: one voxel, one under, at and over the sort's
    tile of 1024, several tiles.  The numbering is that of first appearance in raster order."""
    from ekgsim_gb300.engine import Heart
    rng = np.random.Generator(np.random.PCG64(shape[1] * 100 + shape[2]))
    grid = rng.integers(1, 4, size=shape).astype(np.int32)
    if holes:
        grid[rng.random(shape) < holes] = 0
    values = np.concatenate([[1.0, 1.0 + 2.0**-52, 3.0e5], rng.random(200) * 10.0 ** rng.integers(-3, 5, size=200)])
    at = np.where(grid != 0, values[rng.integers(0, values.size, size=shape)], 0.0)
    h = Heart.create(engine, grid, synth.transfer_matrix(3, [1, 2, 2]), np.array([[90.0, 95.0, 100.0]]), "3D4", 0.0, 10.0,
                     1.0, activation=at)
    seen, want = {}, np.full(grid.size, -1, dtype=np.int64)
    for i, (g, t) in enumerate(zip(grid.reshape(-1), at.reshape(-1))):
        if g:
            want[i] = seen.setdefault((int(g), float(t)), len(seen))
    assert h.info.n_aps == len(seen)
    got = h.ap_index().reshape(-1)
    assert np.array_equal(got[want >= 0], want[want >= 0])
    h.close()


@pytest.mark.parametrize("layers", [11, 12, 31])
def test_noalloc_lag_tables(engine, layers):
    """Activation times in caller-owned buffers with the largest lag table that goes with a launch, and longer ones."""
    import torch
    from ekgsim_gb300 import _lib as L
    rng = np.random.Generator(np.random.PCG64(layers))
    grid = rng.integers(0, layers + 1, size=(17, 12, 20)).astype(np.int32)
    grid[3, 3, 3], grid[0, 0, 0] = layers, -1
    tm = synth.transfer_matrix(layers, list(rng.random(layers) * 3 + 0.1))
    ref, _ = O.activation(grid, tm)
    d = torch.from_numpy(grid).cuda()
    at = torch.full(grid.shape, -7.0, dtype=torch.float64, device="cuda")
    t = np.ascontiguousarray(tm, dtype=np.float64)
    torch.cuda.synchronize()
    L.check(L.load().ekg_activation_noalloc(*grid.shape, ctypes.c_void_p(d.data_ptr()), t.shape[0], L.dptr(t),
                                            ctypes.c_void_p(at.data_ptr()), None))
    assert np.array_equal(at.cpu().numpy().view(np.int64), ref.view(np.int64))
