"""CPU: the kernel that the benchmark's roofline names for a bin is the one that the library launches."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402
import casgemm  # noqa: E402

IDX = "k_numc_esc_idx<256,%s,keys in registers>"


@pytest.mark.parametrize("bin_name,ncol,form,fused,warp,rows,want", [
    ("fused", 1 << 21, 2, 148, 0, 0, "k_numc_rank<256,4,5120,fused>"),
    ("fused", 1 << 21, 2, 147, 0, 0, IDX % "5120,11,fused"),  # fewer rows than SMs
    ("fused", (1 << 21) + 1, 2, 9000, 0, 0, IDX % "5120,11,fused"),
    ("fused", 1 << 17, 1, 9000, 0, 0, "k_numc_esc_idx<256,5120,11,fused>"),
    ("fused", 1 << 17, 0, 9000, 0, 0, "k_numc_esc_msd<256,5120,11,fused>"),
    ("esc1k", 1 << 18, 2, 0, 1184, 5000, "k_numc_warp + k_numc_rank<128,12,1024>"),
    ("esc1k", 1 << 18, 2, 0, 1183, 5000, "k_numc_rank<128,12,1024>"),
    ("esc1k", 1 << 18, 2, 0, 5000, 1183, "k_numc_rank<128,12,1024>"),
    ("esc1k", (1 << 18) + 1, 2, 0, 5000, 5000, "k_numc_rank<128,12,1024>"),
    ("esc1k", 1 << 18, 1, 0, 5000, 5000, "k_numc_esc_msd<256,1024,9>"),
    ("esc5k", 1 << 20, 2, 0, 0, 10, "k_numc_rank<256,4,5120>"),
    ("esc5k", 1 << 22, 2, 0, 0, 10, IDX % "4800,11"),
    ("esc8k", 1 << 22, 2, 0, 0, 10, "k_numc_esc_idx<256,8192,11>"),
    ("esc4k", 1 << 22, 2, 0, 0, 10, "k_numc_esc_msd<256,4096,10>"),
    ("hash256", 1 << 20, 2, 0, 5000, 5000, "k_numc_warp + k_numc_hash<256,9>"),
    ("hash256", (1 << 20) + 1, 2, 0, 5000, 5000, "k_numc_hash<256,9>"),
    ("hash256", 1 << 22, 2, 0, 5000, 5000, "k_numc_hash<256,9>"),
    ("hash256", 1 << 15, 1, 0, 5000, 5000, "k_numc_hash<256,9>"),
    ("hash1k", 1 << 16, 2, 0, 0, 9, "k_numc_dense<512>"), ("hash1k", 1 << 17, 2, 0, 0, 9, "k_numc_hash<256,11>"),
    ("hash4k", 1 << 18, 0, 0, 0, 9, "k_numc_dense<512>"), ("hash4k", 1 << 19, 2, 0, 0, 9, "k_numc_hash<512,13>"),
    ("dense", 1 << 25, 2, 0, 0, 9, "k_numc_dense<512>"), ("tiny", 9, 2, 0, 0, 9, "k_numc_tiny<256>")])
def test_names(bin_name, ncol, form, fused, warp, rows, want):
    assert bench.numc_kernel(bin_name, ncol, form, fused, warp, rows, 148) == want


def test_warp_rows():
    lens = np.array([1, 32, 33, 128, 129, 200])  # entries of A's rows, each of a B row of 4 products
    A = casgemm.Csr(6, 300, np.concatenate([[0], lens.cumsum()]), np.concatenate([np.arange(n) for n in lens]).astype(np.int32),
                    np.ones(lens.sum()))
    B = casgemm.Csr(300, 4, np.arange(301) * 4, np.tile(np.arange(4, dtype=np.int32), 300), np.ones(1200))
    assert bench.warp_rows(A, B) == 3  # 128, 132 and 512 products; 4, 516 and 800 are not
