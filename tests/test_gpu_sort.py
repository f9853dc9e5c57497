"""The radix sort and the sorted export at the edges of their tiles: one tile
of 4096 entries and the first sizes beyond it, ragged ends, odd and even pass
counts, equal keys (the order among them is kept)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 8, 9, 24, 40, 64])
@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 8192, 12289, 700001])
def test_radix_sort_is_stable(pkg, n, bits):
    import torch
    from bass_b200 import _native as nat
    rng = np.random.default_rng(n * 100 + bits)
    k = rng.integers(0, 2 ** bits, size=n, dtype=np.uint64) if bits < 64 else \
        rng.integers(0, 2 ** 64, size=n, dtype=np.uint64)
    k[n // 2:] = k[:n - n // 2]        # every key twice
    a = np.arange(2 * n, dtype=np.float64).view(np.complex128)   # the source position tells equal keys apart
    eng = nat.Engine(max_n=max(n, 16), num_qubits=40)
    tk = torch.from_numpy(k.view(np.int64).copy()).cuda()
    ta = torch.from_numpy(a.view(np.float64).copy()).cuda()
    P = nat.ctypes.c_void_p
    nat.check(eng.L.bass_radix_sort_u64(P(tk.data_ptr()), P(ta.data_ptr()), n, bits, eng.ws_ptr, eng.ws_bytes,
                                        eng.ctrl_ptr, eng.stream), "sort")
    o = np.argsort(k, kind="stable")
    assert np.array_equal(tk.cpu().numpy().view(np.uint64), k[o])
    assert np.array_equal(ta.cpu().numpy().view(np.complex128), a[o])


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64])
@pytest.mark.parametrize("n", [1, 4096, 4097, 50001])
def test_export_order_and_scale(pkg, n, dtype):
    """Export after a permuting gate and a pending renormalisation: true keys
    ascending, every amplitude its own entry's, scaled."""
    from bass_b200 import _native as nat
    from bass_b200.state import SparseState
    rng = np.random.default_rng(n)
    x = np.unique(rng.integers(0, 2 ** 33, size=n + n // 4 + 8, dtype=np.uint64))
    x = np.sort(rng.permutation(x)[:n])
    a = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(dtype)
    st = SparseState(33, n, dtype=dtype, _capacity=2 * n + 16)
    st.load(x, a)
    # X on qubit 20: a relabelling that leaves the device order permuted
    st._apply_1q(np.array([[0, 1], [1, 0]], complex), 20, nat.NO_TRUNC)
    y = x ^ np.uint64(1 << 20)
    o = np.argsort(y)
    assert np.array_equal(st.x, y[o]) and np.array_equal(st.alpha, a[o])
    norm = st._norm2()
    st._renorm()
    b = a.astype(np.complex128)
    r = 1.0 / np.sqrt(norm)
    want = (b.real * r + 1j * (b.imag * r)).astype(dtype)
    assert np.array_equal(st.x, y[o]) and np.array_equal(st.alpha, want[o])
