"""Segmented ops on both routes in one launch: states that their blocks hold on
chip beside states that are staged, bit for bit against the single-state calls;
with workspaces that bound the states tightly (no staged launches when all fit)
and with larger ones."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 34
MIXES = {
    "staged": [150001, 98304, 200000],
    "mixed": [3, 508, 120000, 700, 5000, 260000, 1],
    "chip": [400, 2000, 30001, 64],
    "many": [2048 + 7 * i for i in range(148)],
}
CALL = {"gate1": "bass_gate_1q_batch", "gate2": "bass_gate_2q_batch", "topk": "bass_topk_batch",
        "rot": "bass_rotate_step_batch"}
SLOTS = {"gate1": 2, "gate2": 4, "topk": 1, "rot": 2}


def _state(n, seed, dtype):
    from bass_b200.state import SparseState
    rng = np.random.default_rng(seed)
    # pairs of neighbours among the keys, so that groups of every size occur
    x = np.unique(rng.integers(0, 2 ** N, size=n // 2 + 8, dtype=np.uint64))
    x = np.unique(np.concatenate([x, x ^ np.uint64(1 << 20)]))
    x = np.sort(rng.permutation(x)[:n])
    a = rng.standard_normal(len(x)) + 1j * rng.standard_normal(len(x))
    a = (a / np.linalg.norm(a)).astype(dtype)
    st = SparseState(N, n, dtype=dtype, _capacity=2 * n + 16)
    st.load(x, a)
    return st


def _gates():
    from bass_b200.gates import haar_random_unitary
    return haar_random_unitary(2, seed=2), haar_random_unitary(4, seed=3)


def _segmented(sts, op, bound):
    from bass_b200 import _native as nat
    import torch
    G1, G2 = _gates()
    o = np.zeros(len(sts), dtype=nat.SEG_OP_DTYPE)
    for r, s in zip(o, sts):
        eng, n = s._eng, s.k
        r["in"], r["tmp"], r["out"] = (nat._ptr(d.desc) for d in (s._cur, s._tmp, s._tmp2))
        r["ctrl"], r["ws"] = nat._ptr(eng.ctrl), nat._ptr(eng.ws)
        r["ws_bytes"] = eng.ws_for(n, SLOTS[op]) if bound == "tight" else eng.ws_bytes
        r["k_cond"] = r["k_keep"] = max(1, (2 * n) // 3)
    o["q1"], o["q2"] = 20, 7
    g = nat.host_c128(G2 if op == "gate2" else G1).view(np.float64).reshape(-1)
    o["G"][:, :len(g)] = g
    L = sts[0]._eng.L
    nb = int(L.bass_batch_ws_bytes(len(sts)))
    bws = torch.empty(nb, dtype=torch.uint8, device="cuda")
    nat.check(getattr(L, CALL[op])(ctypes.c_void_p(o.ctypes.data), len(sts), ctypes.c_void_p(bws.data_ptr()), nb,
                                   sts[0]._eng.stream), op)
    torch.cuda.synchronize()
    for s in sts:
        if op != "rot":
            nat.swap(s._cur, s._tmp2)
        s._cur.nmax = s._cur.cap
        s._rekeyed()


def _single(st, op):
    from bass_b200 import _native as nat
    G1, G2 = _gates()
    k = max(1, (2 * st.k) // 3)
    tr = nat.trunc(k, k)
    if op == "gate1":
        st._apply_1q(G1, 20, tr)
    elif op == "gate2":
        st._apply_2q(G2, 20, 7, tr)
    elif op == "topk":
        st._topk(tr)
    else:
        eng = st._eng
        nat.check(eng.L.bass_rotate_step(st._cur.ptr, st._tmp.ptr, nat._host(nat.host_c128(G1)), 20, k, 0, eng.ctrl_ptr,
                                         eng.ws_ptr, eng.ws_bytes, eng.stream), "rotate")
        st._touch()


@pytest.mark.parametrize("bound", ["tight", "large"])
@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("op", list(CALL))
@pytest.mark.parametrize("mix", list(MIXES))
def test_segments_match_single_states(pkg, mix, op, dtype, bound):
    sts = [_state(n, 100 + i, dtype) for i, n in enumerate(MIXES[mix])]
    for i, s in enumerate(sts):      # rotation steps: some accepted, some rejected
        s._eng.set_ctrl("pr_cur", 1e300 if i % 2 else 0.0)
    _segmented(sts, op, bound)
    for i, (n, s) in enumerate(zip(MIXES[mix], sts)):
        if mix == "many" and i % 30:
            continue
        w = _state(n, 100 + i, dtype)
        w._eng.set_ctrl("pr_cur", 1e300 if i % 2 else 0.0)
        _single(w, op)
        assert np.array_equal(s.x, w.x) and np.array_equal(s.alpha, w.alpha), (i, n)
        a, b = s._eng.check_errors(), w._eng.check_errors()
        for f in ("last_kept", "last_total", "pr_cur", "gamma_running", "amp_updates", "n_trunc"):
            assert a[f] == b[f], (i, n, f)
        assert a["accept"][20] == b["accept"][20] and a["frac"][20] == b["frac"][20]
