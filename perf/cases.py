"""Performance cases: the calls a program that trains or evaluates neural
quantum states makes, over the sizes the library supports.

A case is a dict of plain values; its "kind" says which call it is:

  epoch     one training epoch of one session: weights in, Session.epoch(),
            weights and chain configurations out
  batch     the same for several independent trainings in one Batch.epoch()
  evaluate  Session.eval_batch() on given configurations
  ratio     Session.log_psi_over_psi() on given configurations and flips
  solve     rbmnqs.sr_solve_noalloc() on the caller's device buffers

Sessions of precision 0 compute psi ratios, E_loc and O_k in FP32; their
results are handed on in that precision (complex64).  Sessions of precision 1
and the linear solves hand on FP64.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "rbm-nqs_b200"))
import rbmnqs  # noqa: E402


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # a notebook-sized lattice: an epoch is a chain of short launches
        dict(name="epoch_8", kind="epoch", model="kitaev", cells=2, rbm="symmetry", alpha=2, chains=64, spc=4,
             warmup=3, step=1, bond=0.5, std=0.1),
        # 32-spin Kitaev training, the everyday size
        dict(name="epoch_32", kind="epoch", model="kitaev", cells=4, rbm="symmetry", alpha=4, chains=4096, spc=1,
             warmup=63, step=1, bond=0.5, std=0.05),
        # the same lattice in the reference's arithmetic (FP64 throughout)
        dict(name="epoch_32_fp64", kind="epoch", model="kitaev", cells=4, rbm="symmetry", alpha=3, chains=500, spc=2,
             warmup=15, step=2, bond=0.5, std=0.05, precision=1),
        # RBM + Pfaffian training, inverse rebuilt every 32 accepted moves
        dict(name="epoch_32_pfaffian", kind="epoch", model="kitaev", cells=4, rbm="symmetry", alpha=2, chains=2048,
             spc=1, warmup=63, step=1, bond=0.5, std=0.05, pfaffian=1, refresh=32),
        # a basic RBM with more parameters than samples (matrix-free solver), ragged sizes
        dict(name="epoch_98_basic", kind="epoch", model="kitaev", cells=7, rbm="basic", alpha=2, chains=1000, spc=1,
             warmup=30, step=1, bond=0.3, std=0.03, max_iterations=60),
        # the 128-spin lattice, persistent chains, 16 samples per chain: the largest single training
        dict(name="epoch_128", kind="epoch", model="kitaev", cells=8, rbm="symmetry", alpha=4, chains=16384, spc=16,
             warmup=0, step=1, bond=0.0, std=0.02),
        # the same lattice with learned proposals trained alongside
        dict(name="epoch_128_learned", kind="epoch", model="kitaev", cells=8, rbm="symmetry", alpha=4, chains=8192,
             spc=8, warmup=0, step=1, bond=0.0, std=0.02, learned=1),
        # a scan of toric-code trainings advanced together, up to 33152 parameters each
        dict(name="batch_toric", kind="batch", cells_from=3, cells_to=8, copies=2, alpha=2, chains=1024, warmup=63,
             std=0.03, max_iterations=100),
        # exact enumeration of 2^18 states instead of sampling (small-lattice validation)
        dict(name="epoch_full_18", kind="epoch", model="kitaev", cells=3, rbm="symmetry", alpha=3, full=1, std=0.06),
        # energies and amplitudes of given configurations (measuring a trained state)
        dict(name="evaluate_128", kind="evaluate", cells=8, rbm="symmetry", alpha=4, batch=16384, std=0.02,
             derivatives=0),
        # with the log-derivatives, for an optimiser outside the library
        dict(name="evaluate_32", kind="evaluate", cells=4, rbm="symmetry", alpha=4, batch=3001, std=0.05,
             derivatives=1),
        # the SR solve alone on a caller's device buffers
        dict(name="solve_133", kind="solve", params=133, samples=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _std(rng, n):
    """A weight spread for n sites that gives hidden units of order one, as after training."""
    return round(rng.uniform(0.15, 0.35) / math.sqrt(n), 4)


def draw(rng):
    kind = rng.choice(["epoch"] * 5 + ["evaluate"] * 2 + ["batch", "ratio", "solve"])
    if kind == "epoch":
        form = rng.choice(["plain", "plain", "plain", "fp64", "pfaffian", "learned", "full"])
        cells = rng.randint(2, 8)
        if form in ("fp64", "pfaffian"):
            cells = rng.randint(2, 4)
        if form == "full":
            cells = rng.randint(2, 3)
        n = 2 * cells * cells
        rbm = rng.choice(["symmetry", "symmetry", "basic"])
        c = dict(kind="epoch", model="kitaev", cells=cells, rbm=rbm, alpha=rng.randint(1, min(4, 512 // n)),
                 std=_std(rng, n))
        if form == "full":
            if rbm == "basic" and cells == 3:
                c["alpha"] = 1
            return dict(c, full=1)
        matrix_free = rbm == "basic" and n * n * c["alpha"] > 2000
        c.update(chains=_log_int(rng, 64, 1500 if matrix_free or form != "plain" else 12000),
                 spc=1 if matrix_free else rng.randint(1, 8), warmup=rng.randint(0, 24), step=rng.randint(1, 2),
                 bond=rng.choice([0.0, 0.3, 0.5]))
        if matrix_free:
            c["max_iterations"] = rng.randint(20, 80)
        if form == "fp64":
            c["precision"] = 1
        if form == "pfaffian":
            c.update(pfaffian=1, refresh=rng.choice([8, 16, 32]), alpha=min(2, c["alpha"]))
        if form == "learned":
            c["learned"] = 1
        return c
    if kind == "batch":
        lo = rng.randint(2, 5)
        return dict(kind="batch", cells_from=lo, cells_to=min(8, lo + rng.randint(0, 3)), copies=rng.randint(1, 3),
                    alpha=rng.randint(1, 2), chains=_log_int(rng, 100, 1000), warmup=rng.randint(3, 50), std=0.03,
                    max_iterations=rng.randint(20, 80))
    if kind == "evaluate":
        cells = rng.randint(2, 8)
        der = rng.randint(0, 1)
        return dict(kind="evaluate", cells=cells, rbm=rng.choice(["symmetry", "basic"]) if cells <= 5 else "symmetry",
                    alpha=rng.randint(1, min(4, 256 // (cells * cells))),
                    batch=_log_int(rng, 16, 800 if der else 14000),
                    std=_std(rng, 2 * cells * cells), derivatives=der)
    if kind == "ratio":
        cells = rng.randint(2, 8)
        return dict(kind="ratio", cells=cells, alpha=rng.randint(1, 2), batch=_log_int(rng, 100, 30000),
                    flips=rng.randint(1, 4), std=_std(rng, 2 * cells * cells))
    return dict(kind="solve", params=rng.randint(8, 256), samples=_log_int(rng, 300, 8000))


# ---------------------------------------------------------------- prepare --
def _weights(n_params, std, seed, n_neural=None):
    """Complex Gaussian weights of a trained state's size (pair parameters of a Pfaffian: std 1e-2)."""
    rng = np.random.default_rng(seed)
    w = rng.normal(0, std, n_params) + 1j * rng.normal(0, std, n_params)
    if n_neural is not None and n_neural < n_params:
        m = n_params - n_neural
        w[n_neural:] = rng.normal(0, 1e-2, m) + 1j * rng.normal(0, 1e-2, m)
    return w


def _configs(n, batch, seed):
    """Random configurations as the library packs them: bit i of word i / 32 set <=> site i down."""
    down = np.random.default_rng(seed + 1).integers(0, 2, (batch, n)).astype(np.uint64)
    words = np.zeros((batch, 4), np.uint64)
    for i in range(n):
        words[:, i // 32] |= down[:, i] << np.uint64(i % 32)
    return words.astype(np.uint32), 1.0 - 2.0 * down.astype(np.float64)


def _session(model, c, seed, **kw):
    cfg = rbmnqs.default_config(rbm_type=1 if c.get("rbm") == "symmetry" else 0, alpha=c["alpha"], seed=1 + seed,
                                precision=c.get("precision", 0), reinit_chains=0, reg2=(1e-4, 1e-4, 1.0), **kw)
    return rbmnqs.Session(model, cfg)


def _solve_inputs(c, seed, device):
    """Centred-problem inputs of an SR solve: O [N][P], its mean, its variance and a force in its range."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    N, P = c["samples"], c["params"]
    scale = torch.logspace(0, -1.5, P, dtype=torch.float64)
    re, im = (torch.randn(N, P, generator=g, dtype=torch.float64) for _ in range(2))
    O = (torch.complex(re, im) * scale + torch.complex(scale, -scale)).to(device)
    E = torch.complex(torch.randn(N, generator=g, dtype=torch.float64),
                      0.1 * torch.randn(N, generator=g, dtype=torch.float64)).to(device)
    d = O.mean(0)
    diag = ((O - d).abs() ** 2).sum(0) / (N - 1)
    F = ((O - d).conj() * (E - E.mean())[:, None]).mean(0)
    return O.contiguous(), d.contiguous(), diag.contiguous(), F.contiguous()


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve":
        O, d, diag, F = _solve_inputs(c, seed, "cuda")
        return dict(case=c, O=O, d=d, diag=diag, F=F, x=torch.zeros_like(F))
    if kind == "batch":
        sessions, weights = [], []
        for L in range(c["cells_from"], c["cells_to"] + 1):
            model = rbmnqs.Model.toric(L)
            for k in range(c["copies"]):
                s = _session(model, c, 1000 * seed + 10 * L + k, n_chains=c["chains"], samples_per_chain=1,
                             warmup=c["warmup"], step=1, bond_flips=0.0, max_iterations=c["max_iterations"])
                sessions.append(s)
                weights.append(_weights(s.n_params, c["std"], 1000 * seed + 10 * L + k))
        return dict(case=c, sessions=sessions, batch=rbmnqs.Batch(sessions), weights=weights)
    if kind == "ratio":
        s = _session(rbmnqs.Model.toric(c["cells"]), c, seed, n_chains=64)
        w = _weights(s.n_params, c["std"], seed)
        s.set_weights(w)
        spins, _ = _configs(s.n, c["batch"], seed)
        return dict(case=c, session=s, spins=spins, flips=_flips(c, seed))
    model = rbmnqs.Model.kitaev(c["cells"], symmetry=0.5)
    if kind == "evaluate":
        s = _session(model, c, seed, n_chains=64)
        s.set_weights(_weights(s.n_params, c["std"], seed))
        spins, _ = _configs(s.n, c["batch"], seed)
        return dict(case=c, session=s, spins=spins)
    kw = dict(max_iterations=c.get("max_iterations", 0))
    if c.get("full"):
        kw.update(sampler_type=1, n_chains=64)
    else:
        kw.update(n_chains=c["chains"], samples_per_chain=c["spc"], warmup=c["warmup"], step=c["step"],
                  bond_flips=c["bond"])
    if c.get("pfaffian"):
        kw.update(pfaffian=1, pfaffian_symmetry=0.5, pfaffian_refresh=c["refresh"], gram=1)
    if c.get("learned"):
        kw.update(proposal=1, learned_steps=1, learned_train=2, learned_lr=1e-3)
    s = _session(model, c, seed, **kw)
    return dict(case=c, session=s, weights=_weights(s.n_params, c["std"], seed, s.n_neural))


# -------------------------------------------------------------------- run --
def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "solve":
        state["x"].zero_()
        ptr = {k: state[k].data_ptr() for k in ("O", "d", "diag", "F", "x")}
        rbmnqs.sr_solve_noalloc(ptr["O"], c["samples"], c["params"], c["params"], ptr["d"], float(c["samples"]),
                                ptr["F"], ptr["x"], 1e-3, 1e-3, 0.0, ptr["diag"], rtol=1e-22,
                                stream=torch.cuda.current_stream().cuda_stream)
        return state["x"]
    if kind == "batch":
        for s, w in zip(state["sessions"], state["weights"]):
            s.set_weights(w)
        stats, _ = state["batch"].epoch()
        return dict(energy=np.array([x["energy"] for x in stats], np.complex64),
                    weights=[s.get_weights().astype(np.complex64) for s in state["sessions"]])
    s = state["session"]
    if kind == "ratio":
        return s.log_psi_over_psi(state["spins"], state["flips"]).astype(np.complex64)
    if kind == "evaluate":
        logpsi, eloc, O = s.eval_batch(state["spins"], O=bool(c["derivatives"]))
        out = dict(logpsi=logpsi.astype(np.complex64), eloc=eloc.astype(np.complex64))
        if O is not None:
            out["O"] = O.astype(np.complex64)
        return out
    s.set_weights(state["weights"])
    stats, _ = s.epoch()
    w = s.get_weights()
    t = np.complex128 if c.get("precision") else np.complex64
    out = dict(energy=np.array([stats["energy"]], t), weights=w.astype(t))
    if not c.get("full"):
        out["spins"] = s.spins().view(np.int32)
    return out


# ------------------------------------------------------------------- work --
def _sizes(model, cells, rbm, alpha):
    """(sites, theta entries, parameters, off-diagonal terms of H)."""
    n = 2 * cells * cells
    nh = alpha if rbm == "symmetry" else alpha * n
    n_vb = 1 if rbm == "symmetry" else n
    return n, alpha * n, n_vb + nh + n * nh, n if model == "kitaev" else n // 2


def _epoch_work(model, cells, rbm, alpha, chains, spc, sweeps, bond, max_it, pfaffian=0, full=0):
    n, T, P, terms = _sizes(model, cells, rbm, alpha)
    N = 2 ** n if full else chains * spc
    # a psi ratio is one complex multiply-add and one complex product per theta entry
    flops = 16.0 * T * (N * terms + (0 if full else chains * sweeps * n / (1 + bond)))
    if pfaffian:
        flops += chains * sweeps * n / (1 + bond) * 16.0 * n
    # S or its products with a vector: the solver's part
    flops += 16.0 * N * P * max_it if P > 2048 else 4.0 * N * P * (P + 1)
    return 32.0 * P + 32.0 * (0 if full else chains), flops


def work(case):
    c, kind = case, case["kind"]
    if kind == "solve":
        N, P = c["samples"], c["params"]
        return dict(bytes=16.0 * N * P + 16.0 * 5 * P, flops=4.0 * N * P * (P + 1))
    if kind == "batch":
        parts = [_epoch_work("toric", L, "basic", c["alpha"], c["chains"], 1, c["warmup"] + 1, 0.0,
                             c["max_iterations"]) for L in range(c["cells_from"], c["cells_to"] + 1)]
        return dict(bytes=c["copies"] * sum(p[0] for p in parts), flops=c["copies"] * sum(p[1] for p in parts))
    if kind == "ratio":
        n, T, P, _ = _sizes("toric", c["cells"], "basic", c["alpha"])
        return dict(bytes=c["batch"] * (16.0 + 4.0 * c["flips"] + 16.0) + 16.0 * P,
                    flops=c["batch"] * T * (4.0 * n + 16.0))
    if kind == "evaluate":
        n, T, P, terms = _sizes("kitaev", c["cells"], c["rbm"], c["alpha"])
        out = 32.0 + (16.0 * P if c["derivatives"] else 0.0)
        return dict(bytes=c["batch"] * (16.0 + out) + 16.0 * P, flops=c["batch"] * T * (16.0 * terms + 4.0 * n))
    sweeps = 0 if c.get("full") else c["warmup"] + c["spc"] * c["step"]
    b, f = _epoch_work(c["model"], c["cells"], c["rbm"], c["alpha"], c.get("chains", 0), c.get("spc", 0), sweeps,
                       c.get("bond", 0.0), c.get("max_iterations", 0) or 100, c.get("pfaffian", 0), c.get("full", 0))
    return dict(bytes=b, flops=f)


# ------------------------------------------------------------------ exact --
def _flips(c, seed):
    rng = np.random.default_rng(seed + 2)
    n = 2 * c["cells"] * c["cells"]
    return np.argsort(rng.random((c["batch"], n)), axis=1)[:, : c["flips"]].astype(np.int32)


def _honeycomb(L):
    """Bonds (a, b, type) of the L x L honeycomb torus and the permutations
    (translations, each followed by its 180-degree rotation)."""
    def site(i, j, b):
        return 2 * ((i % L) + L * (j % L)) + b

    cells = [(i, j) for j in range(L) for i in range(L)]
    bonds = []
    for i, j in cells:
        bonds += [(site(i, j, 0), site(i, j, 1), 0), (site(i, j, 0), site(i - 1, j, 1), 1),
                  (site(i, j, 0), site(i, j - 1, 1), 2)]
    n, perm = 2 * L * L, []
    for di, dj in cells:
        t = [site(i + di, j + dj, b) for i, j in cells for b in (0, 1)]
        perm += [t, [n - 1 - x for x in t]]
    return bonds, np.array(perm)


def _lncosh(x):
    """Principal ln cosh, entry by entry, without overflow."""
    x = torch.where(x.real < 0, -x, x)
    return x.real - math.log(2.0) + torch.log((1 + torch.exp(-2 * x.real)) * torch.cos(x.imag)
                                              + 1j * (1 - torch.exp(-2 * x.real)) * torch.sin(x.imag))


def exact(case, seed):
    c, kind = case, case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "solve":
        O, d, diag, F = _solve_inputs(c, seed, dev)
        A = O.mH @ O / c["samples"] - torch.outer(d.conj(), d)
        A += torch.diag(1e-3 * diag + 1e-3 * diag.max()).to(A.dtype)
        return torch.linalg.solve(A, F)
    if kind not in ("evaluate", "ratio"):
        return None  # sampled, so there is no value in closed form
    cells = c["cells"]
    n = 2 * cells * cells
    sym = c.get("rbm") == "symmetry"
    nv, nh = (1, c["alpha"]) if sym else (n, c["alpha"] * n)
    w = torch.from_numpy(_weights(nv + nh + n * nh, c["std"], seed)).to(dev)
    v, h, W = w[:nv], w[nv:nv + nh], w[nv + nh:].reshape(nh, n).T  # W[site, hidden]
    sig = torch.from_numpy(_configs(n, c["batch"], seed)[1]).to(dev)
    vis = v.expand(n) if sym else v
    if sym:
        bonds, perm = _honeycomb(cells)
        perm = torch.from_numpy(perm).to(dev)
        # theta entry (symmetry s, hidden k): its weight of site f is W[P_s(f), k]
        big = W[perm].permute(1, 0, 2).reshape(n, -1)
        hid = h.repeat(len(perm))
    else:
        bonds = _honeycomb(cells)[0]
        big, hid = W, h
    theta = sig.to(big.dtype) @ big + hid
    lnc = _lncosh(theta)
    if kind == "ratio":
        out = torch.zeros(c["batch"], dtype=w.dtype, device=dev)
        t2 = theta.clone()
        flips = torch.from_numpy(_flips(c, seed)).to(dev).long()
        for q in range(c["flips"]):
            f = flips[:, q]
            s = sig.gather(1, f[:, None])[:, 0]
            out -= 2 * s * vis[f]
            t2 -= 2 * s[:, None] * big[f]
        return out + (_lncosh(t2) - lnc).sum(1)
    eloc = torch.zeros(c["batch"], dtype=w.dtype, device=dev)
    step = max(1, (1 << 24) // theta.shape[1])
    for a, b, kind_ab in bonds:
        sa, sb = sig[:, a], sig[:, b]
        if kind_ab == 2:
            eloc -= sa * sb
            continue
        for lo in range(0, c["batch"], step):
            r = slice(lo, lo + step)
            t2 = theta[r] - 2 * sa[r, None] * big[a] - 2 * sb[r, None] * big[b]
            ratio = torch.exp(-2 * (sa[r] * vis[a] + sb[r] * vis[b]) + (_lncosh(t2) - lnc[r]).sum(1))
            eloc[r] -= ratio if kind_ab == 0 else -(sa[r] * sb[r]) * ratio
    out = dict(logpsi=(sig * vis).sum(1) + lnc.sum(1), eloc=eloc)
    if c["derivatives"]:
        t = torch.tanh(theta)
        if sym:
            inv = torch.argsort(perm, dim=1)
            ts = t.reshape(c["batch"], len(perm), nh)
            dW = torch.einsum("bsj,bsk->bkj", sig[:, inv].to(t.dtype), ts)
            out["O"] = torch.cat([sig.sum(1, keepdim=True).to(t.dtype), ts.sum(1), dW.reshape(c["batch"], -1)], 1)
        else:
            dW = t[:, :, None] * sig[:, None, :]
            out["O"] = torch.cat([sig.to(t.dtype), t, dW.reshape(c["batch"], -1)], 1)
    return out
