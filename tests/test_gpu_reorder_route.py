"""The reorder pass of a 2-qubit gate is routed by the entries that the gate can
take, not by the four times as many children that its workspace holds: on chip
up to the same size as the gate's small tiles, against the oracle at the edges;
a state larger than the workspace allows is refused as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHIP, EVAL, PERM = 2, 0, 3
N = 34


def _state(n, dtype):
    from bass_b200.state import SparseState
    rng = np.random.default_rng(n)
    x = np.unique(rng.integers(0, 2 ** N, size=n + 100, dtype=np.uint64))
    x = np.sort(rng.permutation(x)[:n])
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    a = (a / np.linalg.norm(a)).astype(dtype)
    st = SparseState(N, n, dtype=dtype, _capacity=4 * n)
    st.load(x, a)
    return st, x, a


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("n,route", [(508, CHIP), (509, CHIP), (75185, CHIP), (150001, CHIP), (300000, CHIP),
                                     (302000, EVAL)])
def test_reorder_route(pkg, orc, n, route, dtype):
    from bass_b200 import _native as nat
    from bass_b200.gates import haar_random_unitary
    st, x, a = _state(n, dtype)
    G = haar_random_unitary(4, seed=3)
    L = st._eng.L
    L.bass_profile_enable(1)
    try:
        st._apply_2q(G, 20, 7, nat.trunc(4 * n, 4 * n))
        c = st._eng.check_errors()
    finally:
        L.bass_profile_enable(0)
        ms, cnt = np.zeros(48), np.zeros(48, np.int64)
        L.bass_profile_collect(nat._host(ms), nat._host(cnt), 48)
    want = np.zeros(5, np.int64)
    want[route] = n
    assert c["prof_in"][5 * PERM:5 * PERM + 5].tolist() == want.tolist()
    if dtype == np.complex128:
        wx, wa = orc.apply_2q_sorted(x, a, G, 20, 7)
        o = np.argsort(wx)
        assert np.array_equal(st.x, wx[o]) and np.array_equal(st.alpha, wa[o])


def test_too_many_entries_are_refused(pkg):
    from bass_b200 import _native as nat
    from bass_b200.gates import haar_random_unitary
    st, _, _ = _state(3000, np.complex128)
    eng = st._eng
    G = haar_random_unitary(4, seed=3)
    small = int(eng.L.bass_workspace_bytes(1000, 4000, N))   # a quarter of its 4000 and a little more
    nat.check(eng.L.bass_gate_2q(st._cur.ptr, st._tmp.ptr, st._tmp2.ptr, nat._host(nat.host_c128(G)), 20, 7,
                                 nat.trunc(100, 100), eng.ctrl_ptr, eng.ws_ptr, small, eng.stream), "gate")
    with pytest.raises(nat.BassError):
        eng.check_errors()
