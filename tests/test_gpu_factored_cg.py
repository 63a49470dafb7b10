"""The matrix-free CG of basic RBMs on the factors of O (spins x activations)
against the oracle's CG on the O store itself, at the edges of the kernel's
tiles: 64 samples x 32 hidden units, 64 sites x 16 hidden units, 256-sample
stages, at most eight sample chunks."""
import numpy as np
import pytest

import oracle as O
import rbmnqs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,L,alpha,N,precision", [
    ("kitaev", 5, 1, 257, 0),   # 50 sites, 50 hidden units, one sample past a stage
    ("kitaev", 6, 1, 65, 0),    # 72 sites, one sample past a row tile, a single chunk
    ("kitaev", 7, 1, 2049, 1),  # 98 sites, chunks of two stages, the last one short
    ("toric", 8, 2, 64, 1),     # 128 sites, 256 hidden units: the largest
    ("kitaev", 7, 2, 300, 0),   # 196 hidden units: remainder of 4 in both tilings
])
def test_factored_cg_matches_oracle(model, L, alpha, N, precision):
    """25 CG iterations from a warm start.  Both sides do the same recurrence
    in FP64 and differ by the order of the sums (1e-15 per product, growing
    with the iterations): 1e-8 on the iterate, as for the operator form."""
    its = 25
    gm = rbmnqs.Model.kitaev(L) if model == "kitaev" else rbmnqs.Model.toric(L)
    cfg = rbmnqs.default_config(rbm_type=0, alpha=alpha, n_chains=N, samples_per_chain=1, warmup=3, seed=9,
                                precision=precision, max_iterations=its)
    s = rbmnqs.Session(gm, cfg)
    P = s.n_params
    assert P > 2048
    rng = np.random.default_rng(P)
    w = rng.normal(0, 0.03, P) + 1j * rng.normal(0, 0.03, P)
    lr, r1, r2, rd = O.Decay(1e-2), O.Decay(1, 1e-4, 0.9), O.Decay(1e-3, 1e-6, 0.9), O.Decay(1e-2)
    x = np.zeros(P, np.complex128)
    for _ in range(2):  # the second solve starts from the first one's solution
        s.set_weights(w)
        s.sample()
        E, Om = s.samples()
        st = s.optimize()
        d, F, diag = O.sr_moments(Om, E)
        lrv, r1v, r2v, rdv = lr.get(), r1.get(), r2.get(), rd.get()
        x, it, _ = O.cg_solve(Om, d, F, x, r1v, r2v, rdv, diag, max_iterations=its)
        assert st["iterations"] == it == its
        step = (w - s.get_weights()) / lrv
        assert np.linalg.norm(step - x) < 1e-8 * np.linalg.norm(x)
        x = x * lrv  # the update scales the stored solution (warm start)
