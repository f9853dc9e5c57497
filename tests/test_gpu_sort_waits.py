"""The sort's bounded waits follow the control block's limit, and one that gives
up is reported.  With wait_limit < 0 the first block at the first grid barrier
of a sort of several tiles gives up after one poll, so every kernel returns and
the context stays usable."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sort(eng, nat, k, a, bits, ctrl):
    import torch
    P = nat.ctypes.c_void_p
    tk = torch.from_numpy(k.view(np.int64).copy()).cuda()
    ta = torch.from_numpy(a.view(np.float64).copy()).cuda()
    nat.check(eng.L.bass_radix_sort_u64(P(tk.data_ptr()), P(ta.data_ptr()), len(k), bits, eng.ws_ptr, eng.ws_bytes,
                                        ctrl, eng.stream), "sort")
    return tk.cpu().numpy().view(np.uint64), ta.cpu().numpy().view(np.complex128)


@pytest.mark.parametrize("bits", [8, 40])
@pytest.mark.parametrize("n", [4097, 100001])
def test_a_sort_that_gives_up_says_so(pkg, n, bits):
    from bass_b200 import _native as nat
    rng = np.random.default_rng(n + bits)
    k = rng.integers(0, 2 ** bits, size=n, dtype=np.uint64)
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    eng = nat.Engine(max_n=n, num_qubits=40)
    eng.set_ctrl("wait_limit", -1)
    _sort(eng, nat, k, a, bits, eng.ctrl_ptr)
    with pytest.raises(nat.BassError, match="wait gave up"):
        eng.raise_on_error()
    # the same workspace sorts again, with a control block and without one
    eng.set_ctrl("wait_limit", 0)
    o = np.argsort(k, kind="stable")
    for ctrl in (eng.ctrl_ptr, None):
        gk, ga = _sort(eng, nat, k, a, bits, ctrl)
        assert np.array_equal(gk, k[o]) and np.array_equal(ga, a[o])
    assert int(eng.read_ctrl()["error"]) == 0


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
def test_an_export_that_gives_up_says_so(pkg, dtype):
    from bass_b200 import _native as nat
    from bass_b200.state import SparseState
    n = 30001
    x = np.arange(n, dtype=np.uint64) * np.uint64(7)
    a = (np.ones(n) / np.sqrt(n)).astype(dtype)
    st = SparseState(30, n, dtype=dtype, _capacity=n + 16)
    st.load(x, a)
    st._eng.set_ctrl("wait_limit", -1)
    st._cur.export()
    with pytest.raises(nat.BassError, match="wait gave up"):
        st._eng.raise_on_error()
    st._eng.set_ctrl("wait_limit", 0)
    gx, ga = st._cur.export()
    assert np.array_equal(gx, x) and np.array_equal(ga, a)
