"""E_loc of symmetric FP32 machines far from trained weights: saturated
activations that a flip cancels or carries to the other side, single weights
and whole rows beyond the range of the products, mixed hidden units.  Every
psi ratio counts with a bound on its own rounding, so that a wrong one cannot
hide behind the energy's scale."""
import numpy as np
import pytest

import oracle as O
import rbmnqs

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


def terms_of(om, bits, o):
    """(flipped sites, matrix element) of operator o's off-diagonal entries
    from the configuration bits (1: down)."""
    k, sites, m = int(om.k[o]), om.sites[o], om.op_matrix(o)
    loc = sum(int(bits[sites[i]]) << i for i in range(k))
    return [([int(sites[i]) for i in range(k) if (loc ^ c) >> i & 1], m[loc, c])
            for c in range(1 << k) if c != loc and m[loc, c] != 0]


def ratio_and_bound(mach, spins, flipped, flips):
    """psi'/psi and its relative rounding error: z = exp(-2 theta) and q, each
    rounded once, enter as z + q with the condition number (|z| + |q|) / |z +
    q| = cosh(Re theta') / |cosh theta'|; an addition (u) and a complex
    multiplication (sqrt(5) u) an entry, the warp's tree of products, and exp
    (30 u together).  The ln cosh sums outside the products' range round theta
    once: u |theta| |tanh theta - tanh theta'|."""
    r = np.exp(O.log_psi_over_psi(mach, spins, flips))
    t, t1 = O.theta(mach, spins), O.theta(mach, flipped)
    cond = np.abs((1 + np.exp(-2 * np.abs(t1.real))) /
                  (1 + np.exp(-2 * np.abs(t1.real) - 2j * np.sign(t1.real) * t1.imag)))
    b = np.sum(cond + 3.3) + 30 + np.sum(np.abs(t) * np.abs(np.tanh(t) - np.tanh(t1)))
    return r, U * b


def check(L, alpha, hid=0.0, std=0.02, rows=(), B=12, h=0.0, seed=0):
    """rows: (site, hidden unit, weight).  No zz bonds: without a field the
    energy is its psi ratios alone.  The first configurations are all up, all
    down and one spin off, where every term carries theta the same way."""
    rng = np.random.default_rng(seed + 10 * L + alpha)
    J = (-1.0, -1.0, 0.0)
    om, gm = O.Model.kitaev(L, J=J, h=h), rbmnqs.Model.kitaev(L, J=J, h=h, symmetry=0.5)
    mach = O.Machine(om, "symmetry", alpha, symm=0.5)
    s = rbmnqs.Session(gm, rbmnqs.default_config(rbm_type=1, alpha=alpha, n_chains=8, precision=0))
    nv, nh, n = s.n_vb, s.n_hidden, s.n
    w = rng.normal(0, std, s.n_params) + 1j * rng.normal(0, std, s.n_params)
    w[nv:nv + nh] += hid
    for j, k, v in rows:
        w[nv + nh + n * k + j] = v
    mach.set_params(w)
    s.set_weights(w)
    bits = rng.integers(0, 2, (B, n))
    bits[0], bits[1], bits[2] = 0, 1, np.arange(n) == 3
    spins = O.spins_from_bits(bits)
    _, eo, Oo = O.eval_batch(mach, om, spins)
    _, eg, Og = s.eval_batch(spins, logpsi=False)
    for b in range(B):
        tol = 1e-14 * om.n_ops * h
        for o in range(om.n_ops):
            for flips, val in terms_of(om, bits[b], o):
                fb = bits[b].copy()
                fb[flips] ^= 1
                r, bound = ratio_and_bound(mach, spins[b], O.spins_from_bits(fb[None])[0], flips)
                tol += np.abs(val * r) * bound
        assert abs(eg[b] - eo[b]) <= tol, (b, eg[b], eo[b], tol)
    assert np.max(np.abs(Og - Oo)) < 1e-5 * max(1.0, np.max(np.abs(Oo)))


@pytest.mark.parametrize("hid,row", [
    ([12, 12], (0, 0, 7)), ([6, 6], (0, 0, 9)), ([10, 10], (0, 0, 12)), ([40, -25], (0, 1, 10)),
    ([20, 20], (0, 0, -10)), ([-20, -20], (0, 0, 10)), ([17, 17], (0, 0, 14.9 + 0.3j)),
])
def test_flip_cancels_a_saturated_activation(hid, row):
    check(3, 2, hid=np.array(hid, float), rows=[row])


@pytest.mark.parametrize("alpha", [1, 2, 3, 4])
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("theta", [10, 14, 19, 24, 30])
def test_saturated_activation_to_zero_and_across(theta, sign, alpha):
    """Both orientations.  One row that carries theta to zero, near it and to
    the other side, and two rows that do so together; one and two-site flips."""
    for f in (1.0, -1.0, 0.5, 0.6, 0.97):
        hid, w = sign * theta * (1 - f / 2 if f > 0 else 1), f * sign * theta / 2
        check(3, alpha, hid=hid, rows=[(0, alpha - 1, w)], B=4)
        check(3, alpha, hid=hid, rows=[(0, alpha - 1, w / 2), (1, alpha - 1, w / 2 + 0.1j)], B=4, h=0.2)


@pytest.mark.parametrize("std", [1.0, 1.5, 2.0])
def test_wide_weights(std):
    check(3, 2, std=std)
    check(4, 4, std=std, B=3)


@pytest.mark.parametrize("v", [16.0, -22.0, 14.9])
def test_rows_beyond_the_factors(v):
    check(3, 2, hid=np.array([8.0, -3.0]), rows=[(0, 0, v), (4, 1, -v)])


def test_mixed_hidden_units():
    """Entries far above and far below one in the same lane, whose partial
    products leave FP32 while the whole stays inside."""
    check(8, 4, hid=np.array([15.0, -15.0, 11.0, -11.0]), B=3,
          rows=[(j, k, (7.5, -7.5, 5.5, -5.5)[k]) for j in (0, 5) for k in range(4)])
    check(4, 4, hid=np.array([22.0, 22.0, -22.0, 22.0]), B=4, rows=[(0, 2, 11.0), (3, 0, -11.0)])
