"""S of an FP32 session on both sides of the line between the FP64 and the
tensor-core Gram, N P^2 = 2e7."""
import numpy as np
import pytest

import oracle as O
import rbmnqs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,kind,alpha,N,fp64", [
    (2, 1, 1, 2, True),       # the fewest samples
    (2, 1, 2, 65, True),      # one tile of S, a ragged sample count
    (4, 1, 4, 1130, True),    # P = 133: 1.999e7
    (4, 1, 4, 1131, False),   # 2.0006e7
])
def test_gram_route_matches_oracle(L, kind, alpha, N, fp64):
    """FP64 sums of FP32 O against the oracle on the same O: 1e-10, as for the
    FP64 Gram; the FP16x3 Gram: 1e-5."""
    cfg = rbmnqs.default_config(rbm_type=kind, alpha=alpha, n_chains=N, samples_per_chain=1, warmup=3, seed=3,
                                precision=0)
    s = rbmnqs.Session(rbmnqs.Model.kitaev(L), cfg)
    P = s.n_params
    assert (N * P * P <= 2e7) == fp64
    rng = np.random.default_rng(N)
    s.set_weights(rng.normal(0, 0.1, P) + 1j * rng.normal(0, 0.1, P))
    s.sample()
    s.optimize()
    E, Om = s.samples()
    S = s.sr_moments()[3]
    So = O.sr_matrix(Om, O.sr_moments(Om, E)[0])
    assert np.linalg.norm(S - So) <= (1e-10 if fp64 else 1e-5) * np.linalg.norm(So)
    assert np.array_equal(S, S.conj().T)
