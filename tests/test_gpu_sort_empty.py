"""The export of an empty state: nothing is written, and a caller that expects
the other amplitude type is refused as it is for any other state."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 5])
def test_export_of_the_wrong_type_is_refused(pkg, n):
    import torch
    from bass_b200 import _native as nat
    from bass_b200.state import SparseState
    st = SparseState(12, 64)
    st.load(np.arange(n, dtype=np.uint64), np.ones(n, np.complex128))
    eng = st._eng
    P = nat.ctypes.c_void_p
    for amp_type, refused in ((nat.AMP_C128, False), (nat.AMP_C64, True)):
        ok = torch.full((8,), -1, dtype=torch.int64, device=eng.device)
        oa = torch.zeros(16, dtype=torch.float64, device=eng.device)
        nat.check(eng.L.bass_state_export_typed(st._cur.ptr, P(ok.data_ptr()), P(oa.data_ptr()), 12, amp_type,
                                                eng.ws_ptr, eng.ws_bytes, eng.ctrl_ptr, eng.stream), "export")
        err = eng.L.bass_error(eng.ctrl_ptr, eng.stream)
        assert bool(err & (1 << nat.ERR_ARG)) == refused
        want = [-1] * 8 if refused else list(range(n)) + [-1] * (8 - n)
        assert ok.cpu().tolist() == want
