"""The chip route and the staged route give the same bits.  A state of 80,000
entries is done on chip when the workspace bounds it tightly and staged when it
does not; the chip route's complex128 results are checked against the oracle
elsewhere.  Inputs: Gaussian, runs of equal |a|^2 across the cut, |a|^2 of 1 and
above, infinities and NaN, entries that make the sample miss the threshold on
either side, and keys at an 8-byte offset (per-entry tile loads)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, n, S = 36, 80000, 16384
KINDS = {"gate1": 0, "rot": 1, "gate2": 2, "topk": 4}
SLOTS = {"gate1": 2, "gate2": 4, "topk": 1, "rot": 2}


def _fmix64(z):
    with np.errstate(over="ignore"):
        for m in (0xff51afd7ed558ccd, 0xc4ceb9fe1a85ec53):
            z = z ^ (z >> np.uint64(33))
            z = z * np.uint64(m)
        return z ^ (z >> np.uint64(33))


def _input(what, dtype):
    rng = np.random.default_rng(7)
    x = np.unique(rng.integers(0, 2 ** N, size=n, dtype=np.uint64))
    # half of the entries have their partner on qubit 30
    x = np.unique(np.concatenate([x[:n // 3], x[:n // 3] ^ np.uint64(1 << 30), x[n // 3:]]))
    x = np.sort(rng.permutation(x)[:n])
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    a /= np.linalg.norm(a)
    some = rng.permutation(n)[:9]
    if what == "ties":
        a = (2.0 ** -rng.integers(4, 7, size=n)).astype(complex)
    elif what == "large":
        a *= 1000.0
    elif what == "inf":
        a[some] = np.inf
    elif what == "nan":
        a[some] = np.nan
    elif what in ("low sample", "high sample"):
        s = np.arange(S, dtype=np.uint64)
        lo, hi = s * np.uint64(n) // np.uint64(S), (s + np.uint64(1)) * np.uint64(n) // np.uint64(S)
        a[(lo + _fmix64(s + np.uint64(1)) % (hi - lo)).astype(np.int64)] *= 1e-9 if what == "low sample" else 1e3
        a /= np.linalg.norm(a)
    return x, a.astype(dtype)


def _bits(v):
    return np.ascontiguousarray(v).view(np.uint8)


def _run(x, a, op, k, bound, offset):
    from bass_b200 import _native as nat
    from bass_b200.gates import haar_random_unitary
    from bass_b200.state import SparseState
    G1, G2 = haar_random_unitary(2, seed=2), haar_random_unitary(4, seed=3)
    st = SparseState(N, 1 << 17, dtype=a.dtype, _capacity=1 << 20)
    st.load(x, a)
    eng, cur = st._eng, st._cur
    keep = None
    if offset:                       # the same entries, keys 8 bytes into a buffer
        torch = eng.torch
        kb = torch.zeros(cur.cap + 1, dtype=torch.int64, device=eng.device)
        kx = torch.from_numpy(x.view(np.int64).copy()).to(eng.device)
        ka = torch.from_numpy(a.view(np.float32 if a.dtype == np.complex64 else np.float64).copy()).to(eng.device)
        P = ctypes.c_void_p
        nat.check(eng.L.bass_state_import_typed(cur.ptr, P(kb.data_ptr() + 8), P(cur.amps.data_ptr()), cur.cap,
                                                P(kx.data_ptr()), P(ka.data_ptr()), n, eng.nq, cur.amp_type, eng.ws_ptr,
                                                eng.ws_bytes, eng.ctrl_ptr, eng.stream), "import")
        keep = kb, kx, ka
        st._rekeyed()
    cur.nmax = n if bound == "tight" else cur.cap
    tr = nat.trunc(k, k)
    L = eng.L
    L.bass_profile_enable(1)
    try:
        if op == "gate1":
            st._apply_1q(G1, 30, tr)
        elif op == "gate2":
            st._apply_2q(G2, 30, 7, tr)
        elif op == "topk":
            st._topk(tr)
        else:
            eng.set_ctrl("pr_cur", 1e300)
            nat.check(L.bass_rotate_step(cur.ptr, st._tmp.ptr, nat._host(nat.host_c128(G1)), 30, k, 0, eng.ctrl_ptr,
                                         eng.ws_ptr, eng.ws_for(cur.nmax, 2), eng.stream), "rotate")
            st._touch()
        c = eng.check_errors()
    finally:
        L.bass_profile_enable(0)
        ms, cnt = np.zeros(48), np.zeros(48, np.int64)
        L.bass_profile_collect(nat._host(ms), nat._host(cnt), 48)
    staged = int(c["prof_in"][5 * KINDS[op]]) == n
    out = [st.x, _bits(st.alpha)] + [_bits(c[f]) for f in ("last_kept", "last_total", "pr_cur", "frac", "accept")]
    del keep
    return staged, out


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("op", list(KINDS))
@pytest.mark.parametrize("what", ["plain", "ties", "large", "inf", "nan", "low sample", "high sample", "offset"])
def test_routes_agree(pkg, what, op, dtype):
    x, a = _input(what, dtype)
    k = 36000
    chip, c = _run(x, a, op, k, "tight", what == "offset")
    staged, s = _run(x, a, op, k, "large", what == "offset")
    assert staged and not chip
    for u, v in zip(c, s):
        assert np.array_equal(u, v)
