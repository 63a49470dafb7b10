"""The screened Metropolis sweep decides every proposal as the exact ln|cosh|
sums do: FP32 chains equal those of a session that sweeps by the sums alone (one
with learned proposals of which it makes none), FP64 chains equal the oracle's.
Group widths of one, two and four hidden units, remainders, p in shared memory
and in L2, bond proposals, refreshes of z, weights beyond the screen's range."""
import numpy as np
import pytest

import oracle as O
import rbmnqs

pytestmark = pytest.mark.gpu


def weights(P, std, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(0, std, P) + 1j * rng.normal(0, std, P)


def model(name, L):
    return rbmnqs.Model.kitaev(L) if name == "kitaev" else rbmnqs.Model.toric(L)


@pytest.mark.parametrize("name,L,kind,alpha,std", [
    ("kitaev", 8, 1, 4, 0.02), ("kitaev", 8, 1, 4, 0.08),  # four hidden units a group
    ("kitaev", 8, 1, 3, 0.05),                              # one, remainder of the lanes
    ("toric", 8, 1, 3, 0.05),                               # two
    ("kitaev", 8, 0, 3, 0.03),                              # basic, p in L2
    ("kitaev", 8, 1, 4, 0.6),                               # beyond the range of z
])
def test_fp32_chains_equal_the_exact_sums(name, L, kind, alpha, std):
    """128 sites without bond proposals: both sessions draw the same proposals.
    Twelve sweeps (a refresh of z after eight), then a second epoch from the
    persistent chains."""
    out = []
    for proposal in (0, 1):
        cfg = rbmnqs.default_config(rbm_type=kind, alpha=alpha, n_chains=150, samples_per_chain=3, warmup=9, step=1,
                                    bond_flips=0.0, seed=5, precision=0, reinit_chains=0, max_iterations=2,
                                    proposal=proposal, learned_steps=0, learned_train=0)
        s = rbmnqs.Session(model(name, L), cfg)
        s.set_weights(weights(s.n_params, std, 3))
        a = s.sample()["acceptance"]
        c0 = s.sample_configs()
        s.sample()
        out.append((a, c0, s.sample_configs(), s.spins()))
    assert out[0][0] == out[1][0]
    for x, y in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("name,L,kind,alpha,std,bond", [
    ("kitaev", 8, 1, 4, 0.03, 0.5), ("kitaev", 7, 1, 3, 0.03, 0.3), ("toric", 4, 1, 1, 0.05, 0.0),
    ("toric", 8, 0, 2, 0.02, 0.0),   # p in L2
    ("kitaev", 5, 0, 1, 0.05, 0.5),  # p in shared memory
    ("kitaev", 2, 1, 1, 0.1, 0.5), ("kitaev", 4, 1, 2, 1.5, 0.5),
])
def test_fp64_chains_equal_the_oracle(name, L, kind, alpha, std, bond):
    chains, spc, warm = 12, 2, 10
    om = O.Model.kitaev(L) if name == "kitaev" else O.Model.toric(L)
    symm = 0.5 if name == "kitaev" else 1.0
    mach = O.Machine(om, "symmetry" if kind else "basic", alpha, symm=symm)
    w = weights(mach.n_params, std, 4)
    mach.set_params(w)
    cfg = rbmnqs.default_config(rbm_type=kind, alpha=alpha, n_chains=chains, samples_per_chain=spc, warmup=warm,
                                step=1, bond_flips=bond, seed=21, precision=1, max_iterations=2)
    s = rbmnqs.Session(model(name, L), cfg)
    s.set_weights(w)
    s.sample()
    E, _ = s.samples(with_O=False)
    Eo = O.metropolis(mach, om, chains, spc, warmup=warm, bond_flips=bond, seed=21, epoch=0)[0]
    # the same chains give the same configurations; one different spin would
    # change an energy by far more than the FP64 rounding of its terms
    assert np.all(np.abs(E - Eo) < 1e-9 * np.maximum(1.0, np.abs(Eo)))
