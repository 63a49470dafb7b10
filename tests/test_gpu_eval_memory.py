"""eval_batch's device memory: an FP32 O leaves in pieces, and an allocation that
fails leaves the session as it was."""
import numpy as np
import pytest

import oracle as O
import rbmnqs

pytestmark = pytest.mark.gpu


def session(alpha=4, precision=0):
    s = rbmnqs.Session(rbmnqs.Model.kitaev(4), rbmnqs.default_config(rbm_type=1, alpha=alpha, n_chains=8,
                                                                     precision=precision))
    rng = np.random.default_rng(1)
    s.set_weights(rng.normal(0, 0.05, s.n_params) + 1j * rng.normal(0, 0.05, s.n_params))
    return s


def spins(B):
    return O.random_spins(np.random.default_rng(2), B, 32)


def test_log_derivatives_in_pieces():
    """40001 x 133 entries: two pieces of 2^21 and a remainder."""
    s = session()
    c = spins(40001)
    _, _, a = s.eval_batch(c, logpsi=False, eloc=False)
    for r in (slice(0, 100), slice(15700, 15900), slice(31500, 31600), slice(39990, 40001)):
        assert np.array_equal(a[r], s.eval_batch(c[r], logpsi=False, eloc=False)[2])


def test_failed_allocation_leaves_the_session_usable():
    torch = pytest.importorskip("torch")
    s, c = session(), spins(16000)
    ref = session().eval_batch(c, logpsi=False)  # kept buffer of 50 MB
    small = s.eval_batch(c[:10], logpsi=False)
    hold = []
    for piece in (1 << 30, 1 << 26, 1 << 23):
        while torch.cuda.mem_get_info()[0] > piece + (1 << 22):
            try:
                hold.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                break
    try:
        with pytest.raises(rbmnqs.RbmNqsError):
            s.eval_batch(c, logpsi=False)
    finally:
        del hold
        torch.cuda.empty_cache()
    for n in (10, 16000):
        _, e, d = s.eval_batch(c[:n], logpsi=False)
        assert np.array_equal(e, ref[1][:n]) and np.array_equal(d, ref[2][:n])
    assert np.array_equal(small[1], ref[1][:10])
