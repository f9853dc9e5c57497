"""A small state under a large bound: a workspace sized for many more entries
than the state holds (a state of large capacity with few entries left, or a
caller that passes one workspace to every call).  The op is done on chip all
the same, and its result is the oracle's, at the edges of what one block and
the first launch's blocks hold.  The same ops also run while another stream
keeps the GPU busy, when the first launch may have to be called off."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHIP, EVAL, WRITE = 2, 0, 3          # passes of an op kind's profile slots
FIRST = 64 * 508                     # entries the first launch's blocks hold
FIRST_TOPK = 148 * 508               # ... of a truncation: a block per SM
N = 36


def _state(n, seed, dtype=np.complex128):
    from bass_b200.state import SparseState
    rng = np.random.default_rng(seed)
    x = np.unique(rng.integers(0, 2 ** N, size=n + 64, dtype=np.uint64))
    x = np.sort(rng.permutation(x)[:n])
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    a = (a / np.linalg.norm(a)).astype(dtype)
    st = SparseState(N, 1 << 20, dtype=dtype, _capacity=1 << 20)
    st.load(x, a)
    st._cur.nmax = st._cur.cap       # as after gates that were not truncated
    return st, x, a


def _gates():
    from bass_b200.gates import haar_random_unitary
    return haar_random_unitary(2, seed=2), haar_random_unitary(4, seed=3)


def _run(st, op, k):
    from bass_b200 import _native as nat
    G1, G2 = _gates()
    tr = nat.trunc(k, k)
    if op == "gate1":
        st._apply_1q(G1, 30, tr)
    elif op == "gate2":
        st._apply_2q(G2, 30, 7, tr)
    elif op == "topk":
        st._topk(tr)
    else:
        eng = st._eng
        eng.set_ctrl("pr_cur", 1e300)
        nat.check(eng.L.bass_rotate_step(st._cur.ptr, st._tmp.ptr, nat._host(nat.host_c128(G1)), 30, k, 0, eng.ctrl_ptr,
                                         eng.ws_ptr, eng.ws_bytes, eng.stream), "rotate")
        st._touch()


def _want(orc, x, a, op, k):
    G1, G2 = _gates()
    if op == "gate1":
        x, a = orc.apply_1q(x, a, G1, 30)
    elif op == "gate2":
        x, a = orc.apply_2q_sorted(x, a, G2, 30, 7)
    elif op == "rot":
        x, a = orc.rotate_1q(x, a, 30, G1)
    x, a, kept, _ = orc.select_topk(x, a, k)
    if op == "rot":                  # the accepted candidate, renormalised
        a = a * (1.0 / np.sqrt(kept))
    o = np.argsort(x)
    return x[o], a[o]


@pytest.mark.parametrize("op,kind", [("gate1", 0), ("rot", 1), ("gate2", 2), ("topk", 4)])
@pytest.mark.parametrize("n", [3, 508, 509, FIRST, FIRST + 1, FIRST_TOPK, FIRST_TOPK + 1])
def test_small_state_under_a_large_bound(pkg, orc, n, op, kind):
    from bass_b200 import _native as nat
    k = max(1, (2 * n) // 3)
    st, x, a = _state(n, n)
    L = st._eng.L
    L.bass_profile_enable(1)
    try:
        _run(st, op, k)
        c = st._eng.check_errors()
    finally:
        L.bass_profile_enable(0)
        ms, cnt = np.zeros(48), np.zeros(48, np.int64)
        L.bass_profile_collect(nat._host(ms), nat._host(cnt), 48)
    wx, wa = _want(orc, x, a, op, k)
    assert np.array_equal(st.x, wx) and np.array_equal(st.alpha, wa)
    want = np.zeros(5, np.int64)
    want[CHIP if n <= (FIRST_TOPK if op == "topk" else FIRST) else EVAL] = n
    assert c["prof_in"][5 * kind:5 * kind + 5].tolist() == want.tolist()


@pytest.mark.parametrize("op", ["gate1", "rot", "gate2", "topk"])
@pytest.mark.parametrize("n", [400, 20000])
def test_beside_other_work(pkg, orc, n, op):
    """Another stream's kernels hold most of the GPU: whether the first launch
    gets its blocks together or is called off, the result is the same."""
    import torch
    k = (2 * n) // 3
    m = torch.randn(8192, 8192, device="cuda")
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    x = a = None
    for _ in range(6):
        st, x, a = _state(n, 1)
        torch.cuda.synchronize()
        with torch.cuda.stream(other):
            for _ in range(3):
                m @ m
        _run(st, op, k)
        got = st.x, st.alpha
        st._eng.check_errors()
        wx, wa = _want(orc, x, a, op, k)
        assert np.array_equal(got[0], wx) and np.array_equal(got[1], wa)
    torch.cuda.synchronize()
