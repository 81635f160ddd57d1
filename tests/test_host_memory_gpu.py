"""GPU: a product whose C finds no host memory fails once, and is not computed a second time.

In a process of its own that limits its address space after the device's memory is in hand: the call reports host
memory, has launched fewer kernels than a whole product, and works again under the old limit.
"""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def no_host_memory():
    import ctypes
    import resource

    import casgemm
    A = casgemm.gen_g500(13, 16, 2)
    dA = casgemm.DeviceCsr.upload(A)
    with casgemm.Context(0) as ctx:
        def call(on_device):
            cc = casgemm.CasCsr()
            cc.on_device, cc.col_bytes = on_device, 4
            before = ctx.stats()["kernel_launches"]
            st = ctx.lib.cas_spgemm(ctx.h, casgemm.ACCUM["hybacc"], ctypes.byref(dA.c), ctypes.byref(dA.c),
                                    ctypes.byref(cc), None)
            text = ctx.lib.cas_last_error(ctx.h).decode() if st else ""
            got = (st, text, ctx.stats()["kernel_launches"] - before, cc.num_nnz)
            if st == 0:
                ctx.free(cc)
            return got

        ctx.set_tuning(out_blocks=1)
        whole = [call(1) for _ in range(3)][-1]
        assert whole[0] == 0 and 12 * whole[3] > 100 << 20, whole
        pages = int(open("/proc/self/statm").read().split()[0])
        old = resource.getrlimit(resource.RLIMIT_AS)
        resource.setrlimit(resource.RLIMIT_AS, (pages * resource.getpagesize() + (32 << 20), old[1]))
        failed = call(0)
        resource.setrlimit(resource.RLIMIT_AS, old)
        assert failed[0] == 2 and "host allocation" in failed[1], failed
        assert failed[2] < whole[2], (failed, whole)
        assert call(0)[0] == 0
    print("ok")


@pytest.mark.gpu
def test_one_try():
    p = subprocess.run([sys.executable, os.path.abspath(__file__)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.strip().endswith("ok"), p.stdout + p.stderr


if __name__ == "__main__":
    ROOT = os.path.dirname(HERE)
    sys.path[:0] = [HERE, ROOT, os.path.join(ROOT, "contention-aware-spgemm_b200"), os.path.join(ROOT, "oracle")]
    no_host_memory()
