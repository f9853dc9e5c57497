"""The moment passes' bounded tile waits follow the control block's limit: one
that gives up is reported (after its copies have landed), and with the default
limit the same moments are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("n", [300, 30001])
def test_rdm_gives_up_and_recovers(pkg, n, dtype):
    from bass_b200 import _native as nat
    from bass_b200.state import SparseState
    N = 20
    rng = np.random.default_rng(n)
    x = np.sort(rng.permutation(2 ** N)[:n]).astype(np.uint64)
    a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    a = (a / np.linalg.norm(a)).astype(dtype)
    st = SparseState(N, n, dtype=dtype, _capacity=n + 16)
    st.load(x, a)
    eng = st._eng

    def rdm():
        nat.check(eng.L.bass_rdm_1q(st._cur.ptr, N, nat.ctypes.c_void_p(nat._ptr(eng.rho)), eng.ctrl_ptr, eng.ws_ptr,
                                    eng.ws_bytes, eng.stream), "rdm")
        return eng.rho[:4 * N].cpu().numpy().reshape(N, 4)

    eng.set_ctrl("wait_limit", -1)
    rdm()
    with pytest.raises(nat.BassError, match="wait gave up"):
        eng.raise_on_error()
    eng.set_ctrl("wait_limit", 0)
    r = rdm()
    assert int(eng.read_ctrl()["error"]) == 0
    p = np.abs(a.astype(np.complex128)) ** 2
    for q in range(N):
        one = (x >> np.uint64(q)) & np.uint64(1) == 1
        assert abs(r[q, 0] - p[~one].sum()) < 1e-12 and abs(r[q, 1] - p[one].sum()) < 1e-12
