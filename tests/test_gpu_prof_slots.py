"""Profile counts: an op's entries are counted in the slots of the kernels that
read and write them, and nowhere else."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EVAL, CHIP, WRITE = 0, 2, 3   # passes of an op kind's slots


@pytest.mark.parametrize("n,read,wrote", [(400, CHIP, CHIP), (5000, CHIP, CHIP), (400000, CHIP, CHIP), (620000, EVAL, WRITE)])
@pytest.mark.parametrize("op,kind", [("gate1", 0), ("gate2", 2), ("topk", 4)])
def test_entries_are_counted_where_they_move(pkg, n, read, wrote, op, kind):
    from bass_b200 import _native as nat
    from bass_b200.gates import haar_random_unitary
    from bass_b200.state import SparseState
    rng = np.random.default_rng(n)
    x = np.unique(rng.integers(0, 2 ** 34, size=n + 100, dtype=np.uint64))[:n]
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    k = (2 * n) // 3
    st = SparseState(34, n, _capacity=4 * n + 16)
    st.load(x, a / np.linalg.norm(a))
    L = st._eng.L
    L.bass_profile_enable(1)
    try:
        if op == "gate1":
            st._apply_1q(haar_random_unitary(2, seed=1), 20, nat.trunc(k, k))
        elif op == "gate2":
            st._apply_2q(haar_random_unitary(4, seed=1), 20, 3, nat.trunc(k, k))
        else:
            st._topk(nat.trunc(k, k))
        c = st._eng.check_errors()
    finally:
        L.bass_profile_enable(0)
        ms, cnt = np.zeros(48), np.zeros(48, np.int64)
        L.bass_profile_collect(nat._host(ms), nat._host(cnt), 48)
    want_in, want_out = np.zeros(5, np.int64), np.zeros(5, np.int64)
    want_in[read], want_out[wrote] = n, k
    assert st.nnz == k
    assert c["prof_in"][5 * kind:5 * kind + 5].tolist() == want_in.tolist()
    assert c["prof_out"][5 * kind:5 * kind + 5].tolist() == want_out.tolist()
