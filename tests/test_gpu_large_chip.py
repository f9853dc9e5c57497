"""States of 300,737 to 603,840 entries: gates and truncations are done on chip in
tiles of 1020, at the edges of that range and with ragged last tiles, against
the oracle; rotation steps stay on the staged route."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["gate1", "gate2", "topk", "rot"])
@pytest.mark.parametrize("n", [300737, 411111, 603840, 603841])
def test_large_chip_tiles(pkg, orc, n, op):
    from bass_b200 import _native as nat
    from bass_b200.gates import haar_random_unitary
    from bass_b200.state import SparseState
    N = 34
    rng = np.random.default_rng(n)
    x = np.unique(rng.integers(0, 2 ** N, size=n, dtype=np.uint64))
    x = np.unique(np.concatenate([x[:n // 3], x[:n // 3] ^ np.uint64(1 << 20), x[n // 3:]]))
    x = np.unique(np.concatenate([x, rng.integers(0, 2 ** N, size=n // 2, dtype=np.uint64)]))
    x = np.sort(rng.permutation(x)[:n])
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    a /= np.linalg.norm(a)
    k = (2 * n) // 3
    st = SparseState(N, n, _capacity=n + 16)
    st.load(x, a)
    eng, tr = st._eng, nat.trunc(k, k)
    G1, G2 = haar_random_unitary(2, seed=2), haar_random_unitary(4, seed=3)
    if op == "gate1":
        st._apply_1q(G1, 20, tr)
        ox, oa = orc.apply_1q(x, a, G1, 20)
    elif op == "gate2":
        st._apply_2q(G2, 20, 7, tr)
        ox, oa = orc.apply_2q_sorted(x, a, G2, 20, 7)
    elif op == "topk":
        st._topk(tr)
        ox, oa = x, a
    else:
        eng.set_ctrl("pr_cur", 1e300)
        nat.check(eng.L.bass_rotate_step(st._cur.ptr, st._tmp.ptr, nat._host(nat.host_c128(G1)), 20, k, 0, eng.ctrl_ptr,
                                         eng.ws_ptr, eng.ws_for(n, 2), eng.stream), "rotate")
        st._touch()
        ox, oa = orc.rotate_1q(x, a, 20, G1)
    ox, oa, kept, total = orc.select_topk(ox, oa, k)
    c = eng.check_errors()
    if op == "rot":
        oa = oa * (1.0 / np.sqrt(kept))
        assert float(c["frac"][20]) == kept
    else:
        assert float(c["last_kept"]) == kept and float(c["last_total"]) == total
    o = np.argsort(ox)
    assert np.array_equal(st.x, ox[o]) and np.array_equal(st.alpha, oa[o])
