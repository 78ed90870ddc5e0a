"""Layout kernels by 16-byte words against the same moves by element and numpy: bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def B():
    from alpha2_b200.backend import CudaBackend
    return CudaBackend(0)


# rows of whole words and not, in both element sizes; one row, one column
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("shape", [(2, 5, 3, 32), (1, 7, 2, 4), (3, 4, 5, 6), (2, 3, 4, 1), (4, 129, 8, 8), (1, 1, 1, 16)])
def test_head_split_and_merge(B, dtype, shape):
    x = np.arange(np.prod(shape), dtype=np.float32).reshape(shape) % 251      # exact in bf16
    t = B.transpose(B.upload(x, dtype), 1, 2)
    assert np.array_equal(np.array(t.data), x.transpose(0, 2, 1, 3))
    assert np.array_equal(np.array(B.transpose(t, 1, 2).data), x)
    assert np.array_equal(np.array(B.transpose(B.upload(x, dtype), 0, 2).data), x.transpose(2, 1, 0, 3))


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("rows,cols,c0,c1", [(5, 96, 32, 64), (3, 24, 0, 8), (4, 24, 8, 24), (7, 24, 3, 11), (2, 10, 1, 3),
                                             (1, 8, 0, 8), (9, 12, 4, 8)])
def test_columns(B, dtype, rows, cols, c0, c1):
    from alpha2_b200 import _lib as L
    from alpha2_b200._lib import AlphaCudaError, check
    x = np.arange(rows * cols, dtype=np.float32).reshape(rows, cols) % 251
    a, out, back = B.upload(x, dtype), B.zeros((rows, c1 - c0), dtype), B.zeros((rows, cols), dtype)
    check(B.lib.alpha_slice_cols(a.ptr, out.ptr, rows, cols, c0, c1, L.DTYPE_CODE[dtype]))
    check(B.lib.alpha_scatter_cols(out.ptr, back.ptr, rows, cols, c0, c1, L.DTYPE_CODE[dtype]))
    want = np.zeros_like(x)
    want[:, c0:c1] = x[:, c0:c1]
    assert np.array_equal(np.array(out.data), x[:, c0:c1]) and np.array_equal(np.array(back.data), want)
    with pytest.raises(AlphaCudaError):
        check(B.lib.alpha_slice_cols(a.ptr, out.ptr, rows, cols, c0, c1, L.I32))


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("rows,d", [(3, 64), (5, 8), (4, 6), (1, 1)])
def test_qkv_slices(B, dtype, rows, d):
    from alpha2_b200 import _lib as L
    from alpha2_b200._lib import check
    x = np.arange(rows * 3 * d, dtype=np.float32).reshape(rows, 3 * d) % 251
    a, parts = B.upload(x, dtype), [B.zeros((rows, d), dtype) for _ in range(3)]
    check(B.lib.alpha_slice_qkv(a.ptr, *(p.ptr for p in parts), rows, d, L.DTYPE_CODE[dtype]))
    for i, p in enumerate(parts):
        assert np.array_equal(np.array(p.data), x[:, i * d:(i + 1) * d])
