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
