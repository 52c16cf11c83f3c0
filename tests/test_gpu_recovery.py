"""Evaluations on the device after one that did not fit.  The larger batch asks for more than any GPU holds, so
that the allocation is refused at once and nothing of it runs."""
import numpy as np
import pytest

from ekgsim_gb300 import synth

pytestmark = pytest.mark.gpu

TOO_MUCH = 400e9  # bytes


@pytest.mark.parametrize("form,free,n_leads,steps,dt", [
    ("every pass's buffers", [5, 6, 7, 8], 64, 20000, 2.0**-6),
    ("per-simulation buffers", [1, 5, 6, 7, 8], 24, 800, 1.0),
])
def test_batch_after_one_that_does_not_fit(form, free, n_leads, steps, dt):
    """A batch, the same batch from its captured graph, one that is refused for memory, the first one again: the
    same bits, and what the larger one gave up is allocated anew."""
    from ekgsim_gb300.engine import Engine, EkgError, Heart
    e = Engine(0)
    spec = synth.small_spec(24 if dt < 1 else 96, n_leads=n_leads, seed=4)
    grid, tm = synth.ellipsoid_heart(spec), synth.transfer_matrix(3, spec.delays)
    rng = np.random.Generator(np.random.PCG64(n_leads))
    leads = synth.leads(spec, rng)[:, ::-1].copy()
    h = Heart.create(e, grid, tm, leads, "3D4", 0.0, steps * dt, dt)
    h.set_eval([synth.BASE_AP] * 3, synth.K_MIN, synth.K_MAX, free, list(synth.analytic_target(n_leads, steps, 3)),
               mid_position=0.6)
    lo, hi = np.array(synth.K_MIN)[free], np.array(synth.K_MAX)[free]

    def genes(sims):
        return np.concatenate([np.tile(lo, 3) + np.tile(hi - lo, 3) * rng.random((sims, 3 * len(free))),
                               np.zeros((sims, 2 * n_leads))], axis=1)

    few = genes(3)
    want = [h.eval_batch(few, want_ecg=True) for _ in range(3)]
    info = h.info
    if 1 in free:  # field and band values of every simulation
        per_sim = 4.0 * n_leads * info.n_aps + 4.0 * (info.n_aps / 512) * n_leads * steps
    else:          # ECGs, in FP64 and as float-float
        per_sim = 16.0 * n_leads * steps
    many = genes(int(TOO_MUCH / per_sim) + 1)
    with pytest.raises(EkgError) as err:
        h.eval_batch(many, want_ecg=False)
    assert err.value.code == -2
    for _ in range(3):
        got = h.eval_batch(few, want_ecg=True)
        for a, b, c in zip(want[0], want[2], got):
            assert np.array_equal(a, c) and np.array_equal(b, c)
    h.close()
    e.close()


@pytest.mark.parametrize("want_ecg", [False, True])
def test_batch_after_one_that_failed_half_way(want_ecg):
    """A batch with more moved rows (65,544) than a grid has: its first kernels are queued when CUDA refuses the
    launch.  The batch after it waits for them and gives what it gave before."""
    from ekgsim_gb300.engine import Engine, EkgError, Heart
    e = Engine(0)
    spec = synth.small_spec(24, n_leads=12, seed=4)
    grid, tm = synth.ellipsoid_heart(spec), synth.transfer_matrix(3, spec.delays)
    rng = np.random.Generator(np.random.PCG64(5))
    leads = synth.leads(spec, rng)[:, ::-1].copy()
    h = Heart.create(e, grid, tm, leads, "3D4", 0.0, 40.0, 1.0)
    h.set_eval([synth.BASE_AP] * 3, synth.K_MIN, synth.K_MAX, [5, 6, 7, 8], list(synth.analytic_target(12, 40, 3)),
               mid_position=0.6)
    genes = np.zeros((5462, 36))
    genes[:, :12] = synth.GENE_MIN[:12] + (synth.GENE_MAX - synth.GENE_MIN)[:12] * rng.random((5462, 12))
    genes[:, 12:] = rng.uniform(-10, 10, size=(5462, 24))
    want = h.eval_batch(genes[:9], want_ecg=want_ecg)
    for _ in range(2):
        with pytest.raises(EkgError) as err:
            h.eval_batch(genes, want_ecg=want_ecg)
        assert err.value.code == -4
        for a, b in zip(want, h.eval_batch(genes[:9], want_ecg=want_ecg)):
            assert np.array_equal(a, b)
    h.close()
    e.close()
