"""Gates, rotation steps and truncations on both routes of the op kernels (a
chip op holds every tile on the GPU's SMs, larger states are staged), at the
edges of their tiles and against the oracle, bit for bit: one block and the
first size beyond it, ragged last tiles, runs of equal |a|^2 across the cut,
and a sample that misses the threshold on either side."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _haar(rng, d):
    q, r = np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))
    return q * (np.diag(r) / np.abs(np.diag(r)))


def _keys(rng, N, n):
    x = np.unique(rng.integers(0, 2 ** N, size=n + n // 2 + 64, dtype=np.uint64))
    return np.sort(rng.permutation(x)[:n])


def _state(N, x, a):
    from bass_b200.state import SparseState
    st = SparseState(N, len(x), dtype=a.dtype, _capacity=4 * len(x) + 16)
    st.load(x, a)
    return st


def _check(st, ox, oa):
    o = np.argsort(ox)
    assert np.array_equal(st.x, ox[o]) and np.array_equal(st.alpha, oa[o])


# 1-qubit tiles of 508 at most, whole grid 592 of them; staged tiles of 2040
SIZES = [1, 2, 507, 508, 509, 1017, 4099, 150001, 300736, 300737, 2040 * 160, 2040 * 160 + 1]


@pytest.mark.parametrize("op", ["gate1", "gate2", "topk"])
@pytest.mark.parametrize("n", SIZES)
def test_op_matches_oracle(pkg, orc, n, op):
    from bass_b200 import _native as nat
    rng = np.random.default_rng(n)
    N = 34 if n > 10 else 5
    x = _keys(rng, N, n)
    a = rng.standard_normal(len(x)) + 1j * rng.standard_normal(len(x))
    a /= np.linalg.norm(a)
    k = max(1, (2 * n) // 3)
    st = _state(N, x, a)
    tr = nat.trunc(k, k, 0, 0)
    if op == "gate1":
        G, q = _haar(rng, 2), int(rng.integers(N))
        st._apply_1q(G, q, tr)
        ox, oa = orc.apply_1q(x, a, G, q)
    elif op == "gate2":
        G = _haar(rng, 4)
        q1, q2 = (int(v) for v in rng.permutation(N)[:2])
        st._apply_2q(G, q1, q2, tr)
        ox, oa = orc.apply_2q_sorted(x, a, G, q1, q2)
    else:
        st._topk(tr)
        ox, oa = x, a
    before = len(ox)
    ox, oa, kept, total = orc.select_topk(ox, oa, k)
    _check(st, ox, oa)
    c = st._eng.read_ctrl()
    if before > k:
        assert float(c["last_kept"]) == kept and float(c["last_total"]) == total


@pytest.mark.parametrize("levels", [1, 3])
@pytest.mark.parametrize("n", [400, 3000, 310000])
def test_equal_probabilities_are_cut_by_key(pkg, orc, n, levels):
    """More children of equal |a|^2 than are ranked one by one: the smallest
    true keys stay."""
    from bass_b200 import _native as nat
    rng = np.random.default_rng(n + levels)
    N = 30
    x = _keys(rng, N, n)
    a = (2.0 ** -rng.integers(0, levels, size=len(x))).astype(np.complex128) / 1024
    for k in (n // 7, n // 2 + 3):
        st = _state(N, x, a)
        st._topk(nat.trunc(k, k, 0, 0))
        ox, oa, _, _ = orc.select_topk(x, a, k)
        _check(st, ox, oa)


def _fmix64(z):
    z = z.copy()
    with np.errstate(over="ignore"):
        z ^= z >> np.uint64(33)
        z *= np.uint64(0xff51afd7ed558ccd)
        z ^= z >> np.uint64(33)
        z *= np.uint64(0xc4ceb9fe1a85ec53)
        z ^= z >> np.uint64(33)
    return z


@pytest.mark.parametrize("sampled", [1e-9, 1e3])
def test_a_sample_that_misses_the_threshold(pkg, orc, sampled):
    """The staged route's bracket comes from entries at hashed places; here
    exactly those are far below (above) the others, so the first bracket does
    not hold the threshold, and the result is still the exact one."""
    from bass_b200 import _native as nat
    rng = np.random.default_rng(3)
    N, n, k, S = 36, 400000, 180000, 16384
    x = _keys(rng, N, n)
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    s = np.arange(S, dtype=np.uint64)
    lo, hi = s * np.uint64(n) // np.uint64(S), (s + np.uint64(1)) * np.uint64(n) // np.uint64(S)
    a[(lo + _fmix64(s + np.uint64(1)) % (hi - lo)).astype(np.int64)] *= sampled
    a /= np.linalg.norm(a)
    st = _state(N, x, a)
    st._topk(nat.trunc(k, k, 0, 0))
    ox, oa, kept, total = orc.select_topk(x, a, k)
    _check(st, ox, oa)
    c = st._eng.read_ctrl()
    assert float(c["last_kept"]) == kept and float(c["last_total"]) == total


@pytest.mark.parametrize("n", [400, 5000, 320000])
def test_probabilities_of_one_and_above(pkg, orc, n):
    """An unnormalised state: |a|^2 of 1 and above takes the integer path of the
    exact sums."""
    from bass_b200 import _native as nat
    rng = np.random.default_rng(n)
    N = 33
    x = _keys(rng, N, n)
    a = 3.0 * (rng.standard_normal(n) + 1j * rng.standard_normal(n))
    k, q, G = n, 9, _haar(rng, 2)
    st = _state(N, x, a)
    st._apply_1q(G, q, nat.trunc(k, k, 0, 0))
    ox, oa = orc.apply_1q(x, a, G, q)
    ox, oa, kept, total = orc.select_topk(ox, oa, k)
    _check(st, ox, oa)
    c = st._eng.read_ctrl()
    assert float(c["last_kept"]) == kept and float(c["last_total"]) == total


@pytest.mark.parametrize("angle", [0.0, 0.4])
@pytest.mark.parametrize("n", [300, 6000, 330000])
def test_rotation_step_sums(pkg, orc, n, angle):
    """A rotation step's retained mass and decision, with and without a
    truncation (at angle 0 every second child is dropped, so nothing is cut
    although twice the entries would not fit)."""
    from bass_b200 import _native as nat
    rng = np.random.default_rng(n)
    N, q = 35, 30
    x = _keys(rng, N, n)
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    a[rng.permutation(n)[:n // 2]] *= 1e-9       # a part far below the rest
    a /= np.linalg.norm(a)
    U = np.array([[np.cos(angle), -np.sin(angle)], [np.sin(angle), np.cos(angle)]], complex)
    ox, oa = orc.rotate_1q(x, a, q, U)
    if len(ox) > n:
        ox, oa, kept, _ = orc.select_topk(ox, oa, n)
    else:
        kept = orc.sum_p(oa)
    pr = kept * kept / orc.sum_p2(oa)
    for limit, accepted in ((pr * 1.5, 1), (pr * 0.5, 0)):
        st = _state(N, x, a)
        eng = st._eng
        eng.set_ctrl("pr_cur", limit)
        nat.check(eng.L.bass_rotate_step(st._cur.ptr, st._tmp.ptr, nat._host(nat.host_c128(U)), q, n, 0, eng.ctrl_ptr,
                                         eng.ws_ptr, eng.ws_for(n, 2), eng.stream), "rotate")
        c = eng.check_errors()
        assert int(c["accept"][q]) == accepted and float(c["frac"][q]) == kept
        st._touch()
        if accepted:
            assert float(c["pr_cur"]) == pr
            o = np.argsort(ox)
            assert np.array_equal(st.x, ox[o])
        else:
            assert np.array_equal(st.x, x) and np.array_equal(st.alpha, a)
