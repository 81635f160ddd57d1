"""GPU: the workspace that a context keeps for its products' scratch.

Products of growing and shrinking sizes on one context, dense and split rows among them, several contexts on several
threads, and a context's stream changed between products.
"""
import threading

import numpy as np
import pytest

import casgemm
import oracle

pytestmark = pytest.mark.gpu

GRAPHS = [(8, 4), (12, 16), (9, 2), (14, 8), (13, 16), (6, 2), (14, 8)]


def digest_of(ctx, dA):
    C, _ = ctx.spgemm_device(dA, dA, "hybacc")
    try:
        return ctx.digest(C)
    finally:
        ctx.free(C)


@pytest.fixture(scope="module")
def graphs(ctx):
    out = []
    for s, ef in GRAPHS:
        A = casgemm.gen_g500(s, ef, 40 + s)
        rp, cols, vals, _ = oracle.oracle_spgemm(A, A, "hybacc")
        out.append((casgemm.DeviceCsr.upload(A), oracle.csr_digest(rp, cols, vals)[0]))
    return out


def test_sizes_grow_and_shrink(graphs):
    with casgemm.Context(0) as ctx:
        for _ in range(2):
            for dA, ref in graphs:
                assert digest_of(ctx, dA) == ref


def test_contexts_on_threads(graphs):
    bad = []

    def work(k):
        with casgemm.Context(0) as ctx:
            for i in range(2 * len(graphs)):
                dA, ref = graphs[(i + k) % len(graphs)]
                if digest_of(ctx, dA) != ref:
                    bad.append((k, i))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_stream_changes(graphs):
    import torch
    with casgemm.Context(0) as ctx:
        streams = [torch.cuda.Stream().cuda_stream, None, torch.cuda.Stream().cuda_stream]
        for i, (dA, ref) in enumerate(graphs):
            ctx.set_stream(streams[i % 3])
            assert digest_of(ctx, dA) == ref
        ctx.set_stream(None)
