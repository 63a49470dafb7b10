"""The screened sweep where its two computations of a proposal differ most:
saturated hidden units of one sign (totals of 1e4, whose float spacing exceeds
the rest of the margin), activations near a zero of cosh in many entries at
once, wide weights, which it leaves to the sums' kernel.  FP32 chains equal
those of a session that sweeps by the sums alone, FP64 chains the oracle's; an
FP64 session that sweeps in many launches equals one that does so in one."""
import numpy as np
import pytest

import oracle as O
import rbmnqs

pytestmark = pytest.mark.gpu


def weights(s, std, hid, seed=3):
    rng = np.random.default_rng(seed)
    w = rng.normal(0, std, s.n_params) + 1j * rng.normal(0, std, s.n_params)
    w[s.n_vb:s.n_vb + s.n_hidden] += hid
    return w


def run(L, alpha, std, hid, up=False, **kw):
    cfg = rbmnqs.default_config(rbm_type=1, alpha=alpha, seed=5, reinit_chains=0, max_iterations=2, **kw)
    s = rbmnqs.Session(rbmnqs.Model.kitaev(L), cfg)
    s.set_weights(weights(s, std, hid))
    if up:
        s.set_spins(np.zeros((cfg.n_chains, 4), np.uint32))
    a = s.sample()["acceptance"]
    return a, s.sample_configs(), s.spins()


def same(x, y):
    assert x[0] == y[0] and np.array_equal(x[1], y[1]) and np.array_equal(x[2], y[2])


@pytest.mark.parametrize("std,hid", [
    (0.02, -5.0), (0.02, -8.0), (0.02, -10.0), (0.02, 9.0), (0.05, 0.0), (0.1, 0.0), (0.3, 0.0),
    (0.02, 1.56j), (0.02, 1.3j - 0.02), (0.002, -9.0 + 1.2j),
])
def test_fp32_chains_equal_the_exact_sums(std, hid):
    """Ten million proposals, from all spins up, where the entries of a hidden
    unit are equal."""
    kw = dict(n_chains=4096, samples_per_chain=2, warmup=18, step=1, bond_flips=0.0, precision=0)
    same(run(8, 4, std, hid, up=True, proposal=0, **kw),
         run(8, 4, std, hid, up=True, proposal=1, learned_steps=0, learned_train=0, **kw))


@pytest.mark.parametrize("L,alpha,std,hid,bond", [
    (8, 4, 0.02, -8.0, 0.5), (8, 4, 0.02, -10.0, 0.0), (4, 3, 0.05, -9.0, 0.5), (4, 3, 0.03, 1.5j, 0.0),
    (4, 2, 0.3, 0.0, 0.5), (3, 1, 1.0, 0.0, 0.5),
])
def test_fp64_chains_equal_the_oracle(L, alpha, std, hid, bond):
    chains, spc, warm = 24, 2, 14
    om = O.Model.kitaev(L)
    mach = O.Machine(om, "symmetry", alpha, symm=0.5)
    cfg = rbmnqs.default_config(rbm_type=1, alpha=alpha, n_chains=chains, samples_per_chain=spc, warmup=warm, step=1,
                                bond_flips=bond, seed=21, precision=1, max_iterations=2)
    s = rbmnqs.Session(rbmnqs.Model.kitaev(L), cfg)
    w = weights(s, std, hid, 4)
    mach.set_params(w)
    s.set_weights(w)
    s.sample()
    E, _ = s.samples(with_O=False)
    Eo = O.metropolis(mach, om, chains, spc, warmup=warm, bond_flips=bond, seed=21, epoch=0)[0]
    assert np.all(np.abs(E - Eo) < 1e-9 * np.maximum(1.0, np.abs(Eo)))


@pytest.mark.parametrize("L,alpha,std", [(8, 4, 0.03), (4, 3, 0.05), (4, 2, 0.5)])
def test_fp64_launches_of_one_sweep_equal_one_launch(L, alpha, std):
    """A learned-proposal session that makes no learned moves."""
    kw = dict(n_chains=300, samples_per_chain=10, warmup=3, step=1, bond_flips=0.0, precision=1)
    same(run(L, alpha, std, 0.0, proposal=0, **kw),
         run(L, alpha, std, 0.0, proposal=1, learned_steps=0, learned_train=0, **kw))


@pytest.mark.parametrize("precision,chains", [(0, 600), (1, 100)])
def test_a_launch_left_to_the_sums_and_back(precision, chains):
    """Persistent chains through captured epochs whose weights the screen takes,
    then not, then again."""
    out = []
    for proposal in (0, 1):
        cfg = rbmnqs.default_config(rbm_type=1, alpha=4, n_chains=chains, samples_per_chain=3, warmup=0, step=1, seed=5,
                                    bond_flips=0.0, reinit_chains=0, max_iterations=2, precision=precision,
                                    proposal=proposal, learned_steps=0, learned_train=0)
        s = rbmnqs.Session(rbmnqs.Model.kitaev(8), cfg)
        got = []
        for std, hid in ((0.02, 0.0), (0.6, 0.0), (0.03, 0.0), (0.02, -9.0), (0.02, 0.5)):
            s.set_weights(weights(s, std, hid))
            st, _ = s.epoch()
            got.append((st["acceptance"], s.sample_configs(), s.spins()))
        out.append(got)
    for x, y in zip(*out):
        same(x, y)


@pytest.mark.parametrize("warmup,spc,chains,screened", [(0, 1, 16384, True), (0, 1, 2100, False), (2, 1, 2100, False),
                                                         (3, 1, 2100, True)])
def test_launches_of_few_sweeps_take_the_sums(warmup, spc, chains, screened):
    """The launch shape of a session that sweeps by the sums (learned proposals), or not."""
    shape = []
    for proposal in (0, 1):
        cfg = rbmnqs.default_config(rbm_type=1, alpha=4, n_chains=chains, samples_per_chain=spc, warmup=warmup, step=1,
                                    seed=5, precision=0, proposal=proposal)
        shape.append(rbmnqs.Session(rbmnqs.Model.kitaev(8), cfg).sweep_shape()[0])
    assert (shape[0] != shape[1]) == screened
