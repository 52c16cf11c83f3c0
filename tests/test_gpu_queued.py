"""Calls beside evaluations that are queued on the device."""
import time

import numpy as np
import pytest

from ekgsim_gb300 import synth

pytestmark = pytest.mark.gpu


def test_activation_times_beside_a_queued_generation():
    """Activation times are handed over while a queued generation still runs, not behind it."""
    from ekgsim_gb300.engine import Engine, Heart
    e = Engine(0)
    spec = synth.small_spec(96, n_leads=12, seed=2)
    grid, tm = synth.ellipsoid_heart(spec), synth.transfer_matrix(3, spec.delays)
    rng = np.random.Generator(np.random.PCG64(2))
    leads = synth.leads(spec, rng)[:, ::-1].copy()
    h = Heart.create(e, grid, tm, leads, "3D4", 0.0, 600.0, 1.0)
    h.set_eval([synth.BASE_AP] * 3, synth.K_MIN, synth.K_MAX, [5, 6, 7, 8], list(synth.analytic_target(12, 600, 3)),
               mid_position=0.6)
    sims = 5000
    genes = np.zeros((sims, 36))
    genes[:, :12] = synth.GENE_MIN[:12] + (synth.GENE_MAX - synth.GENE_MIN)[:12] * rng.random((sims, 12))
    genes[:, 12:] = rng.uniform(-20, 20, size=(sims, 24))
    out = h.eval_batch(genes)
    want = h.activation()

    def timed(f):
        t = time.perf_counter()
        f()
        return time.perf_counter() - t

    whole = min(timed(lambda: h.eval_batch(genes, out=out)) for _ in range(3))
    alone = min(timed(h.activation) for _ in range(3))
    beside, left = [], []
    for _ in range(3):
        ticket = h.eval_batch_submit(genes, out)
        t = time.perf_counter()
        got = h.activation()
        beside.append(time.perf_counter() - t)
        left.append(timed(lambda: h.eval_batch_wait(ticket)))
        assert np.array_equal(got.view(np.int64), want.view(np.int64))
    assert alone < whole / 8, (alone, whole)  # the generation is long enough to tell
    assert min(beside) < whole / 4 and max(left) > whole / 8, (alone, whole, beside, left)
    h.close()
    e.close()
