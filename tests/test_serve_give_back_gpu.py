"""GPU: a server sizes a request although what its slots hold idle fills the device.

In a process of its own: after a request with some 450 MB of scratch, the device's memory is filled up to 64 MB, and a
request of 2^24 rows needs 128 MB to be sized.
"""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
MB = 1 << 20


def submit_on_a_full_device():
    import torch
    from cuda.bindings import runtime as cudart

    import casgemm
    A = casgemm.gen_g500(15, 16, 3)
    dA = casgemm.DeviceCsr.upload(A)
    m = 1 << 24
    rp = torch.ones(m + 1, dtype=torch.int64, device="cuda")
    rp[0] = 0
    one_c = torch.zeros(1, dtype=torch.int32, device="cuda")
    one_v = torch.ones(1, dtype=torch.float64, device="cuda")
    tall = casgemm.DeviceCsr(m, A.num_row, 1, rp.data_ptr(), one_c.data_ptr(), one_v.data_ptr(), keep=(rp, one_c, one_v))
    torch.cuda.synchronize()
    with casgemm.Server(slots=1) as srv:
        results = [srv.wait(srv.submit(dA, dA)) for _ in range(3)]
        assert all(r["status"] == 0 for r in results)
        cudart.cudaMemPoolTrimTo(cudart.cudaDeviceGetDefaultMemPool(0)[1], 0)
        fill = torch.empty(torch.cuda.mem_get_info()[0] - 64 * MB, dtype=torch.uint8, device="cuda")
        tall_id = srv.submit(tall, dA)
        del fill
        torch.cuda.empty_cache()
        srv.wait(tall_id)  # computed while the device was full or not: its status is either
        again = srv.wait(srv.submit(dA, dA))
        assert (again["status"], again["digest"]) == (0, results[0]["digest"])
    print("ok")


@pytest.mark.gpu
def test_submit_on_a_full_device():
    p = subprocess.run([sys.executable, os.path.abspath(__file__)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.strip().endswith("ok"), p.stdout + p.stderr


if __name__ == "__main__":
    ROOT = os.path.dirname(HERE)
    sys.path[:0] = [HERE, ROOT, os.path.join(ROOT, "contention-aware-spgemm_b200"), os.path.join(ROOT, "oracle")]
    submit_on_a_full_device()
