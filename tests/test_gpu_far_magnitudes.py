"""The staged route on states whose |a|^2 all lie outside the sample's fine bins
(below 2^-64: the tail of a small-angle circuit, or a state that is not
renormalised; 1 and above): the bracket still leaves only children near the
threshold undecided, and the result is the oracle's.

The bracket spans four deviations of a rank among 16,384 sampled entries on
either side (2 x 3.1 per cent of the entries) plus the bins of its edges: at most
a quarter of a power of two each, which holds at most 0.37 ln(2) / 4 = 6.4 per
cent of exponentially distributed children.  A quarter of the children is more
than their sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C_OUT, C_DEF, C_STAGED = 2, 3, 4   # words of the workspace's op counters


@pytest.mark.parametrize("op,n,scale", [(op, 620001, s) for op in ("gate1", "gate2", "topk")
                                        for s in (2.0 ** -30, 2.0 ** -200, 2.0 ** 14)]
                         + [("rot", 310001, 2.0 ** -30), ("rot", 310001, 2.0 ** 14)])
def test_bracket_outside_the_fine_bins(pkg, orc, op, n, scale):
    import torch
    from bass_b200 import _native as nat
    from bass_b200.gates import haar_random_unitary
    from bass_b200.state import SparseState
    N = 36
    rng = np.random.default_rng(n)
    x = np.unique(rng.integers(0, 2 ** N, size=n + n // 8, dtype=np.uint64))
    x = np.sort(rng.permutation(x)[:n])
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    a = a / np.linalg.norm(a) * scale
    k = (2 * n) // 3
    st = SparseState(N, n, _capacity=n + 16)
    st.load(x, a)
    eng, tr = st._eng, nat.trunc(k, k)
    G1, G2 = haar_random_unitary(2, seed=2), haar_random_unitary(4, seed=3)
    if op == "gate1":
        st._apply_1q(G1, 30, tr)
        ox, oa = orc.apply_1q(x, a, G1, 30)
    elif op == "gate2":
        st._apply_2q(G2, 30, 7, tr)
        ox, oa = orc.apply_2q_sorted(x, a, G2, 30, 7)
    elif op == "topk":
        st._topk(tr)
        ox, oa = x, a
    else:
        eng.set_ctrl("pr_cur", 1e300)
        nat.check(eng.L.bass_rotate_step(st._cur.ptr, st._tmp.ptr, nat._host(nat.host_c128(G1)), 30, k, 0,
                                         eng.ctrl_ptr, eng.ws_ptr, eng.ws_for(n, 2), eng.stream), "rotate")
        st._touch()
        ox, oa = orc.rotate_1q(x, a, 30, G1)
    eng.check_errors()
    cn = eng.ws[:64].view(torch.int64).cpu().numpy()
    assert cn[C_OUT] == len(ox)
    assert cn[C_DEF] <= k <= cn[C_STAGED]
    assert cn[C_STAGED] - cn[C_DEF] <= len(ox) // 4
    if op == "rot":
        return   # (its PR is a quotient of sums that these magnitudes leave no digits of)
    ox, oa, kept, total = orc.select_topk(ox, oa, k)
    o = np.argsort(ox)
    assert np.array_equal(st.x, ox[o]) and np.array_equal(st.alpha, oa[o])
