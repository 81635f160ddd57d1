"""The torch views of device matrices that the library allocated have their arrays' lengths and types: a product of
int32 matrices holds int64 values, a transposed int32 matrix int32 ones."""
import numpy as np
import pytest

import casgemm
from matrices import from_coo


@pytest.mark.parametrize("val_type,value_bytes,typestr", [(casgemm.VAL_F64, 8, "<f8"), (casgemm.VAL_I32, 8, "<i8"),
                                                          (casgemm.VAL_I32, 4, "<i4")])
def test_value_view(monkeypatch, val_type, value_bytes, typestr):
    """On the CPU: what torch would be told of the values' array."""
    import torch
    monkeypatch.setattr(torch, "as_tensor", lambda v, device: v.__cuda_array_interface__)
    cc = casgemm.CasCsr(4, 5, 3, 4096, 8192, 12288, 4, val_type, 1, 1)
    cc.value_bytes = value_bytes
    rp, cols, vals = casgemm.device_tensors(cc)
    assert (rp["typestr"], rp["shape"], cols["typestr"], cols["shape"]) == ("<i8", (5,), "<i4", (3,))
    assert (vals["typestr"], vals["shape"], vals["data"][0]) == (typestr, (3,), 12288)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.int32, np.float64])
def test_transposed_and_product(ctx, dtype):
    rng = np.random.default_rng(3)
    A = from_coo(300, 500, *np.nonzero(rng.random((300, 500)) < 0.05), dtype=dtype)
    A.vals[:] = rng.integers(1, 9, A.nnz)
    dA = casgemm.DeviceCsr.upload(A)
    B = ctx.transpose_device(dA)
    want = A.transpose()
    rp, cols, vals = casgemm.device_tensors(B)
    assert str(vals.dtype) == ("torch.float64" if dtype is np.float64 else "torch.int32")
    np.testing.assert_array_equal(rp.cpu().numpy(), want.row_ptrs)
    np.testing.assert_array_equal(cols.cpu().numpy(), want.cols)
    np.testing.assert_array_equal(vals.cpu().numpy(), want.vals)
    if dtype is np.int32:
        with pytest.raises(ValueError):
            ctx.digest(B)
    dB = casgemm.DeviceCsr.upload(want)
    C, _ = ctx.spgemm_device(dA, dB, "hybacc")
    assert str(casgemm.device_tensors(C)[2].dtype) == ("torch.float64" if dtype is np.float64 else "torch.int64")
    assert int(casgemm.device_tensors(C)[2].sum()) == ctx.spgemm(A, want, "hybacc").csr.vals.sum()
    ctx.free(C)
    ctx.free(B)
