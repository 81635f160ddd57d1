"""GPU: a program that makes a memory pool of its own current on the device has the library's results and scratch
from there, as cudaMallocAsync's, and the default pool's use does not grow."""
import pytest

import casgemm
import oracle

pytestmark = pytest.mark.gpu


def _attr(cudart, pool, name):
    err, v = cudart.cudaMemPoolGetAttribute(pool, getattr(cudart.cudaMemPoolAttr, "cudaMemPoolAttr" + name))
    assert int(err) == 0
    return int(v)


@pytest.mark.parametrize("op", ["product", "host", "transpose"])
def test_own_pool_is_followed(op):
    from cuda.bindings import driver, runtime as cudart
    A = casgemm.gen_g500(12, 8, 5)
    dA = casgemm.DeviceCsr.upload(A)
    default = cudart.cudaDeviceGetDefaultMemPool(0)[1]
    props = cudart.cudaMemPoolProps()
    props.allocType = cudart.cudaMemAllocationType.cudaMemAllocationTypePinned
    props.location.type = cudart.cudaMemLocationType.cudaMemLocationTypeDevice
    props.location.id = 0
    err, pool = cudart.cudaMemPoolCreate(props)
    assert int(err) == 0
    with casgemm.Context(0) as ctx:
        C, _ = ctx.spgemm_device(dA, dA, "hybacc")  # under the default pool, with a workspace for the next
        want = ctx.digest(C)
        ctx.free(C)
        before = _attr(cudart, default, "UsedMemCurrent")
        cudart.cudaMemPoolSetAttribute(default, cudart.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh,
                                       driver.cuuint64_t(0))
        assert int(cudart.cudaDeviceSetMemPool(0, pool)[0]) == 0
        try:
            for _ in range(2):
                if op == "transpose":
                    B = ctx.transpose_device(dA)
                    held, size = _attr(cudart, pool, "UsedMemCurrent"), 12 * B.num_nnz
                    ctx.free(B)
                elif op == "product":
                    C, _ = ctx.spgemm_device(dA, dA, "hybacc")
                    held, size = _attr(cudart, pool, "UsedMemCurrent"), 12 * C.num_nnz
                    assert ctx.digest(C) == want
                    ctx.free(C)
                else:
                    out = ctx.spgemm(A, A, "hybacc")
                    held, size = _attr(cudart, pool, "UsedMemHigh"), 12 * out.csr.nnz
                    assert oracle.csr_digest(out.csr.row_ptrs, out.csr.cols, out.csr.vals)[0] == want
                assert held >= size
                assert _attr(cudart, default, "UsedMemHigh") <= before
        finally:
            assert int(cudart.cudaDeviceSetMemPool(0, default)[0]) == 0
        C, _ = ctx.spgemm_device(dA, dA, "hybacc")
        assert ctx.digest(C) == want
        ctx.free(C)
    assert _attr(cudart, pool, "UsedMemCurrent") == 0
    assert int(cudart.cudaMemPoolDestroy(pool)[0]) == 0
