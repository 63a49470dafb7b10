"""E_loc and O_k of symmetric machines in FP32 (psi ratios as products over
tables of the flipped row tuples) against the oracle: every group width and
number of groups per lane, remainders, four-site flips, field terms, and the
ranges outside the products (saturated and opposed activations, weights whose
factors leave FP32), which fall back to ln cosh sums."""
import numpy as np
import pytest

import oracle as O
import rbmnqs

pytestmark = pytest.mark.gpu


def check(model, L, alpha, std=0.05, hid=0.0, scale=None, B=37, h=0.0, seed=0):
    rng = np.random.default_rng(seed + 10 * L + alpha)
    symm = 0.5 if model == "kitaev" else 1.0
    om = O.Model.kitaev(L, h=h) if model == "kitaev" else O.Model.toric(L)
    gm = rbmnqs.Model.kitaev(L, h=h, symmetry=symm) if model == "kitaev" else rbmnqs.Model.toric(L, symmetry=symm)
    mach = O.Machine(om, "symmetry", alpha, symm=symm)
    cfg = rbmnqs.default_config(rbm_type=1, alpha=alpha, n_chains=8, precision=0)
    s = rbmnqs.Session(gm, cfg)
    P, nv, nh = s.n_params, s.n_vb, s.n_hidden
    w = rng.normal(0, std, P) + 1j * rng.normal(0, std, P)
    w[nv:nv + nh] += hid
    if scale is not None:
        w[nv + nh] = scale
    mach.set_params(w)
    s.set_weights(w)
    down = rng.integers(0, 2, (B, s.n)).astype(np.uint64)
    spins = np.zeros((B, 4), np.uint64)
    for i in range(s.n):
        spins[:, i // 32] |= down[:, i] << np.uint64(i % 32)
    spins = spins.astype(np.uint32)
    _, eo, Oo = O.eval_batch(mach, om, spins)
    _, eg, Og = s.eval_batch(spins, logpsi=False)
    # a product of up to 512 factors, each with a few roundings of 6e-8:
    # 3e-6 typical, 2e-5 allowed, on the scale of the energies
    assert np.all(np.abs(eg - eo) < 2e-5 * np.maximum(np.abs(eo), np.median(np.abs(eo)) + 1))
    assert np.max(np.abs(Og - Oo)) < 1e-5 * max(1.0, np.max(np.abs(Oo)))


@pytest.mark.parametrize("model,L,alpha", [
    ("kitaev", 2, 1), ("kitaev", 3, 3), ("kitaev", 5, 3), ("kitaev", 7, 3), ("kitaev", 7, 5),  # one hidden unit a group
    ("kitaev", 2, 2), ("kitaev", 5, 2), ("kitaev", 8, 2), ("toric", 3, 1),                     # two
    ("kitaev", 4, 4), ("kitaev", 5, 4), ("kitaev", 6, 4), ("kitaev", 8, 4), ("toric", 4, 2),   # four
])
def test_products_match_oracle(model, L, alpha):
    check(model, L, alpha)


def test_field_terms():
    check("kitaev", 3, 2, h=0.3)


@pytest.mark.parametrize("hid", [-4.0, 4.0, -12.0 + 0.5j, 25.0])
def test_saturated_activations(hid):
    check("kitaev", 4, 4, std=0.05, hid=hid)


def test_opposed_activations():
    """Hidden biases of +-12: a lane's product leaves FP32 on either side."""
    check("kitaev", 4, 4, hid=np.array([12.0, -12.0, 12.0, -12.0]))


@pytest.mark.parametrize("scale", [2.5, -16.0, 9.0 + 1.0j])
def test_large_weights(scale):
    check("kitaev", 3, 2, std=0.02, scale=scale)
