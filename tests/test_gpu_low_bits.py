"""Ops whose target bit already is the lowest of its group: Z order is key order
then, and tiles are not merged.  A gate moves its target to the lowest bit, so
the same gate again takes that path; both routes, both amplitude types, tiles
whose last group is ragged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 30


def _state(n, dtype, seed):
    from bass_b200.state import SparseState
    rng = np.random.default_rng(seed)
    # runs of neighbouring keys too, so that groups have one to four entries
    base = rng.integers(0, 2 ** (N - 2), size=n, dtype=np.uint64) << np.uint64(2)
    x = np.unique(np.concatenate([base, base + rng.integers(0, 4, size=n, dtype=np.uint64)]))
    x = np.sort(rng.permutation(x)[:n])
    a = rng.standard_normal(len(x)) + 1j * rng.standard_normal(len(x))
    a = (a / np.linalg.norm(a)).astype(dtype)
    st = SparseState(N, n, dtype=dtype, _capacity=4 * n + 16)
    st.load(x, a)
    return st, x, a


@pytest.mark.parametrize("n", [3, 507, 5001, 330001, 620001])
def test_lowest_bits_match_oracle(pkg, orc, n):
    from bass_b200 import _native as nat
    from bass_b200.gates import haar_random_unitary
    G1, G2 = haar_random_unitary(2, seed=5), haar_random_unitary(4, seed=6)
    for op in ("gate1", "gate2", "gate2 swapped"):
        st, x, a = _state(n, np.complex128, n)
        n = len(x)
        k = (3 * n) // 2
        for _ in range(2):
            if op == "gate1":
                st._apply_1q(G1, 0, nat.trunc(k, k))
                x, a = orc.apply_1q(x, a, G1, 0)
            else:
                q1, q2 = (1, 0) if op == "gate2" else (0, 1)
                st._apply_2q(G2, q1, q2, nat.trunc(k, k))
                x, a = orc.apply_2q_sorted(x, a, G2, q1, q2)
            x, a, _, _ = orc.select_topk(x, a, k)
            o = np.argsort(x)
            x, a = x[o], a[o]
            assert np.array_equal(st.x, x) and np.array_equal(st.alpha, a), op
        rho = st._rdm_2q(1, 0)
        assert abs(np.trace(rho) - np.sum(np.abs(a) ** 2)) < 1e-9


@pytest.mark.parametrize("n", [507, 5001, 330001, 620001])
def test_lowest_bits_complex64(pkg, n):
    """complex64: the same gate on a qubit that is merged and on the same
    entries with that qubit renamed to the lowest bit."""
    from bass_b200 import _native as nat
    from bass_b200.gates import haar_random_unitary
    G = haar_random_unitary(2, seed=7)
    st, x, a = _state(n, np.complex64, n + 1)
    n = len(x)
    st._apply_1q(G, 0, nat.trunc(n, n))
    low = st.x, st.alpha
    # bit 0 <-> bit 20
    swap = lambda v: (v & ~np.uint64(1 | 1 << 20)) | ((v >> np.uint64(20)) & np.uint64(1)) | ((v & np.uint64(1)) << np.uint64(20))
    st.load(swap(x), a)
    st._apply_1q(G, 20, nat.NO_TRUNC)
    hx, ha = swap(st.x), st.alpha
    o = np.argsort(hx)
    hx, ha = hx[o], ha[o]
    at = np.searchsorted(hx, low[0])
    assert np.array_equal(hx[at], low[0]) and np.array_equal(ha[at], low[1])
