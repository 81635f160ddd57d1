"""GPU: memory that the library holds idle serves its own allocations before one of them fails.

In a process of its own, with the device's memory filled up to 256 MB: a context that has run a product of some 600 MB
of scratch keeps that as its workspace, and another context's transpose needs more than what is free.
"""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
MB = 1 << 20


def idle_workspace():
    import torch
    from cuda.bindings import runtime as cudart

    import casgemm
    A = casgemm.gen_g500(15, 16, 3)
    dA = casgemm.DeviceCsr.upload(A)
    one, two = casgemm.Context(0), casgemm.Context(0)

    def digest():
        C, _ = one.spgemm_device(dA, dA, "hybacc")
        try:
            return one.digest(C)
        finally:
            one.free(C)

    want = [digest() for _ in range(3)][0]
    kept = one.stats()["symb_bins"]["dense"] * 65536  # the bitmaps of the dense rows, among the scratch
    assert kept > 400 * MB, kept
    need = 256 * MB + kept // 2
    n, nnz = 1 << 16, need // 28  # a transpose holds B (12 bytes an entry) and two keys (16)
    cols = (torch.arange(nnz, device="cuda", dtype=torch.int64) * 40503 % n).to(torch.int32)
    rp = torch.arange(n + 1, device="cuda", dtype=torch.int64) * nnz // n
    vals = torch.arange(nnz, device="cuda", dtype=torch.float64)
    T = casgemm.DeviceCsr(n, n, nnz, rp.data_ptr(), cols.data_ptr(), vals.data_ptr(), keep=(rp, cols, vals))
    torch.cuda.synchronize()
    pool = cudart.cudaDeviceGetDefaultMemPool(0)[1]
    cudart.cudaMemPoolTrimTo(pool, 0)
    fill = torch.empty(torch.cuda.mem_get_info()[0] - 256 * MB, dtype=torch.uint8, device="cuda")
    B = two.transpose_device(T)
    brp, bcols, bvals = casgemm.device_tensors(B)
    assert int(brp[-1]) == nnz and float(bvals.sum()) == float(vals.sum())
    two.free(B)
    del fill, brp, bcols, bvals, cols, rp, vals, T
    torch.cuda.empty_cache()
    assert [digest() for _ in range(3)] == [want] * 3
    print("ok")


@pytest.mark.gpu
def test_idle_workspace_of_another_context():
    p = subprocess.run([sys.executable, os.path.abspath(__file__)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.strip().endswith("ok"), p.stdout + p.stderr


if __name__ == "__main__":
    ROOT = os.path.dirname(HERE)
    sys.path[:0] = [HERE, ROOT, os.path.join(ROOT, "contention-aware-spgemm_b200"), os.path.join(ROOT, "oracle")]
    idle_workspace()
