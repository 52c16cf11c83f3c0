"""Compiled variants that a dispatch picks by size, on both sides of its limits."""
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


@pytest.mark.parametrize("mode", [1, 2, 3, 4])
@pytest.mark.parametrize("sims,steps", [
    (3, 1024),    # the most steps that a block keeps in registers
    (3, 1025),
    (2, 1500),
    (300, 1025),  # a warp per simulation and lead
])
def test_criteria_long_leads(engine, sims, steps, mode):
    """Criteria and peak positions of long simulations: the FP64 comparison of the engine's own ECG with the
    target, which is longer than the simulation for one lead and shorter for the others."""
    from ekgsim_gb300.engine import Heart
    spec = synth.small_spec(20, n_leads=4, seed=3)
    grid, tm = synth.ellipsoid_heart(spec), synth.transfer_matrix(3, spec.delays)
    rng = np.random.Generator(np.random.PCG64(steps))
    leads = synth.leads(spec, rng)[:, ::-1].copy()
    h = Heart.create(engine, grid, tm, leads, "3D4", 0.0, float(steps), 1.0)
    whole = synth.analytic_target(4, steps + 50, 9)
    target = [whole[0], whole[1][:steps], whole[2][:steps - 1], whole[3][:steps - 130]]
    offs = [0.5, 1.0, 0.25, 2.0]
    h.set_eval([synth.BASE_AP] * 3, synth.K_MIN, synth.K_MAX, [5, 6, 7, 8], target, target_offsets=offs,
               mid_position=0.6, comparison_mode=mode, peak=True)
    genes = np.stack([synth.genes_for(spec, r, 0) for r in range(sims)])
    crit, _, ecg = h.eval_batch(genes, want_ecg=True)
    for s in {0, sims // 2, sims - 1}:
        for l in range(4):
            ref = O.clamp(O.compare(mode, ecg[s, l], target[l], offs[l]))
            assert crit[s, 2 * l] == pytest.approx(ref, rel=1e-9, abs=1e-12), (s, l)
            assert crit[s, 2 * l + 1] == abs(int(np.argmax(ecg[s, l])) - int(np.argmax(target[l]))), (s, l)
    h.close()


def test_strip_with_many_stimuli():
    """A strip of 65,536 tiles with a stimulus in each has its activation times after a few rounds: nothing is
    queued for a front that would run along all of it (that took 0.36 s; a few milliseconds without)."""
    import time
    import torch
    from ekgsim_gb300 import _lib as L
    shape = (8, 8, 8 * 65536)
    d = torch.ones(shape, dtype=torch.int32, device="cuda")
    d[0, 0, ::8] = -1
    at = torch.empty(shape, dtype=torch.float64, device="cuda")
    tm = np.ascontiguousarray(synth.transfer_matrix(1, [1.0]))
    rounds, took = ctypes.c_int32(0), []
    for _ in range(3):
        torch.cuda.synchronize()
        t = time.perf_counter()
        L.check(L.load().ekg_activation_noalloc(*shape, ctypes.c_void_p(d.data_ptr()), tm.shape[0], L.dptr(tm),
                                                ctypes.c_void_p(at.data_ptr()), ctypes.byref(rounds)))
        took.append(time.perf_counter() - t)
    assert rounds.value < 20
    assert min(took) < 0.1
    grid = np.ones((8, 8, 8 * 4), dtype=np.int32)
    grid[0, 0, ::8] = -1
    ref, _ = O.activation(grid, tm)
    got = at.cpu().numpy()
    for tile, like in ((0, 0), (1, 1), (30000, 1), (65534, 2)):  # two tiles each: the first, inner ones, the last
        assert np.array_equal(got[:, :, 8 * tile:8 * tile + 16].view(np.int64),
                              ref[:, :, 8 * like:8 * like + 16].view(np.int64))


def steady_entries(at, k1, steps):
    """Steady prefixes that a layer with these activation times keeps: one per group of the 128-step tiles before
    the first one in which the whole layer is steady (at most seven groups), and the whole layer."""
    t_plus = 30.0 * np.log(2.0) / k1
    starts = np.arange(0, steps, 128)
    steady = [j for j, t0 in enumerate(starts) if at.max() < t0 - t_plus]
    first = steady[0] if steady else len(starts)
    size = max(1, (first + 6) // 7)
    return -(-first // size) + (first < len(starts))


@pytest.mark.parametrize("entries,latest,steps", [
    (4, 370.0, 700),    # the most that the smaller variant of the steady sums takes
    (5, 500.0, 800),
    (8, 880.0, 1400),   # as many as there can be
    (7, 1700.0, 850),   # no tile in which the whole layer is steady
    (8, 1700.0, 2100),  # groups of two tiles
])
def test_steady_entries(engine, entries, latest, steps):
    """Batched passes on hearts whose activation times spread over many 128-step tiles."""
    from ekgsim_gb300.engine import Heart, layer_aps, move_leads
    spec = synth.small_spec(20, n_leads=4, seed=6)
    grid, tm = synth.ellipsoid_heart(spec), synth.transfer_matrix(3, spec.delays)
    rng = np.random.Generator(np.random.PCG64(steps))
    layer = np.abs(grid).astype(np.int32)
    at = np.where(layer > 0, rng.uniform(1.0, latest - 60.0, size=grid.shape), 0.0)
    for a in (1, 2, 3):
        z, y, x = (v[0] for v in np.nonzero(layer == a))
        at[z, y, x] = latest
        assert steady_entries(at[layer == a], synth.BASE_AP[1], steps) == entries
    leads = synth.leads(spec, rng)[:, ::-1].copy()
    h = Heart.create(engine, grid, tm, leads, "3D4", 0.0, float(steps), 1.0, activation=at)
    h.set_eval([synth.BASE_AP] * 3, synth.K_MIN, synth.K_MAX, [5, 6, 7, 8], list(synth.analytic_target(4, steps, 3)),
               mid_position=0.6)
    for sims, moved in ((7, 2), (150, 3)):
        genes = np.zeros((sims, 12 + 8))
        genes[:, :12] = synth.GENE_MIN[:12] + (synth.GENE_MAX - synth.GENE_MIN)[:12] * rng.random((sims, 12))
        genes[:, 0:12:4] = synth.K_MIN[5]  # the batched form takes such times with a small k5 only
        genes[:, 12:12 + 2 * moved] = rng.uniform(-15, 15, size=(sims, 2 * moved))
        ecg = h.eval_batch(genes, want_ecg=True)[2]
        aps = np.stack([layer_aps(h._cfg, 3, g[:12])[0] for g in genes])
        assert h.benchmark(aps, np.stack([move_leads(leads, g[12:].reshape(-1, 2)) for g in genes]), 1, 1)["batched"]
        for i in (0, sims - 1):
            lk = aps[i]
            ref = O.run(layer, at, lk, move_leads(leads, genes[i, 12:].reshape(-1, 2)), "3D4", 0.0, float(steps), 1.0)
            assert np.linalg.norm(ecg[i] - ref) <= ECG_TOL * np.linalg.norm(ref), (sims, i)
    h.close()


@pytest.mark.parametrize("case", ["one voxel", "ragged", "plane", "zero lag", "unreachable", "128^3"])
def test_activation_in_callers_buffers(engine, case):
    """The heart's set-up and the call that allocates nothing: the same times, and the oracle's."""
    import torch
    from ekgsim_gb300 import _lib as L
    from ekgsim_gb300.engine import Heart
    rng = np.random.Generator(np.random.PCG64(7))
    tm = synth.transfer_matrix(3, [1, 2, 2])
    if case == "one voxel":
        grid = np.array([[[-1]]], dtype=np.int32)
    elif case == "ragged":
        grid = rng.integers(0, 4, size=(13, 17, 11)).astype(np.int32)
        grid[6, 8, 5] = -2
    elif case == "plane":
        grid = rng.integers(1, 4, size=(1, 37, 29)).astype(np.int32)
        grid[0, 3, 4] = -1
    elif case == "zero lag":
        grid = rng.integers(1, 4, size=(12, 10, 14)).astype(np.int32)
        grid[0, 0, 0] = -1
        tm[2, 3] = 0.0
    elif case == "unreachable":
        grid = np.zeros((10, 10, 10), dtype=np.int32)
        grid[1, 1, 1] = -1
        grid[5:9, 5:9, 5:9] = 2
    else:
        grid = synth.ellipsoid_heart(synth.config(1)["spec"]).astype(np.int32)
    ref, _ = O.activation(grid, tm)
    h = Heart.create(engine, grid, tm, np.array([[200.0, 210.0, 220.0]]), "3D4", 0.0, 10.0, 1.0)
    assert np.array_equal(h.activation().view(np.int64), ref.view(np.int64))
    h.close()
    d = torch.from_numpy(np.ascontiguousarray(grid)).cuda()
    at = torch.full(grid.shape, -7.0, dtype=torch.float64, device="cuda")
    t = np.ascontiguousarray(tm, dtype=np.float64)
    torch.cuda.synchronize()
    L.check(L.load().ekg_activation_noalloc(*grid.shape, ctypes.c_void_p(d.data_ptr()), t.shape[0], L.dptr(t),
                                            ctypes.c_void_p(at.data_ptr()), None))
    assert np.array_equal(at.cpu().numpy().view(np.int64), ref.view(np.int64))
