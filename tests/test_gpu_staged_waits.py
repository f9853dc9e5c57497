"""The staged route's bounded waits: with wait_limit < 0 its tile loads give up
at once, which every later launch of the op sees (nothing is written, the
output's descriptor stays as it was, the barrier word is reset), the error is
reported, and with the default limit the same op on the same input is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["gate1", "gate2", "topk", "rot"])
def test_staged_op_gives_up_and_recovers(pkg, orc, op):
    from bass_b200 import _native as nat
    from bass_b200.gates import haar_random_unitary
    from bass_b200.state import SparseState
    N, n, k = 32, 620000, 400000
    rng = np.random.default_rng(5)
    x = np.unique(rng.integers(0, 2 ** N, size=n + 200, dtype=np.uint64))[:n]
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    a /= np.linalg.norm(a)
    G1, G2 = haar_random_unitary(2, seed=2), haar_random_unitary(4, seed=3)
    st = SparseState(N, n, _capacity=n + 16)
    eng = st._eng
    tr = nat.trunc(k, k)

    def run():
        if op == "gate1":
            st._apply_1q(G1, 7, tr)
        elif op == "gate2":
            st._apply_2q(G2, 7, 20, tr)
        elif op == "topk":
            st._topk(tr)
        else:
            nat.check(eng.L.bass_rotate_step(st._cur.ptr, st._tmp.ptr, nat._host(nat.host_c128(G1)), 7, k, 0,
                                             eng.ctrl_ptr, eng.ws_ptr, eng.ws_bytes, eng.stream), "rotate")
            st._touch()

    st.load(x, a)
    eng.set_ctrl("pr_cur", 1e300)
    eng.set_ctrl("wait_limit", -1)
    before = st._cur.read_desc(), [int(d.read_desc()["nnz"]) for d in (st._tmp, st._tmp2)]
    run()
    with pytest.raises(nat.BassError, match="wait gave up"):
        eng.raise_on_error()
    if op == "rot":                  # the state is still the one before the step
        assert bytes(st._cur.read_desc()) == bytes(before[0])
    else:
        assert int(st._cur.read_desc()["nnz"]) in before[1]
    c = eng.read_ctrl()
    assert int(c["sync_counter"]) == 0 and int(c["n_trunc"]) == 0
    eng.set_ctrl("wait_limit", 0)
    st.load(x, a)
    run()
    ox, oa = {"gate1": lambda: orc.apply_1q(x, a, G1, 7), "gate2": lambda: orc.apply_2q_sorted(x, a, G2, 7, 20),
              "topk": lambda: (x, a), "rot": lambda: orc.rotate_1q(x, a, 7, G1)}[op]()
    ox, oa, kept, _ = orc.select_topk(ox, oa, k)
    if op == "rot":
        oa = oa * (1.0 / np.sqrt(kept))
    o = np.argsort(ox)
    assert np.array_equal(st.x, ox[o]) and np.array_equal(st.alpha, oa[o])
    assert int(eng.read_ctrl()["error"]) == 0
