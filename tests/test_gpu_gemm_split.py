"""The GEMM whose last wave is cut along K keeps partial tiles in a workspace.  Products that may run at once must
not share one: on several streams, on the per-thread default streams, in graphs that replay beside eager calls.  A
product's slices are added in a fixed order, so every result must equal the first one bit for bit; one that shared
its workspace would mix partial tiles, or run out of its bounded waits."""
import os
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

M, N, K = 4096, 3584, 4096


@pytest.fixture(scope="module")
def product():
    import ctypes as C

    import mini_nccl_b200 as mn
    from mini_nccl_b200.ops import gemm_bf16

    first, slices, per = C.c_int(), C.c_int(), C.c_int()
    L = mn.lib()
    assert L.mncclGemmSplitPlan(M, N, K, L.mncclGemmMaxPairs(), C.byref(first), C.byref(slices), C.byref(per)) == 1
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    want = gemm_bf16(a, b)
    os.environ["MINI_NCCL_GEMM_SPLIT_K"] = "0"
    try:
        whole = gemm_bf16(a, b)
    finally:
        del os.environ["MINI_NCCL_GEMM_SPLIT_K"]
    torch.cuda.synchronize()
    assert not torch.equal(want, whole), "the sums are taken in another order when the last wave is split"
    return a, b, want, whole


def _check(outs, want):
    from mini_nccl_b200.ops import gemm_status

    torch.cuda.synchronize()
    assert gemm_status() == 0, "a bounded wait ran out inside the GEMM"
    for i, o in enumerate(outs):
        assert torch.equal(o, want), i


def test_products_on_more_streams_than_workspaces(product):
    from mini_nccl_b200.ops import gemm_bf16

    a, b, want, _ = product
    streams = [torch.cuda.Stream() for _ in range(11)]
    outs = [torch.zeros_like(want) for _ in range(3 * len(streams))]
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        gemm_bf16(a, b, out=o, stream=streams[i % len(streams)])
    _check(outs, want)


def test_products_on_the_per_thread_default_streams(product):
    from mini_nccl_b200.ops import gemm_bf16

    a, b, want, _ = product
    outs = [torch.zeros_like(want) for _ in range(6)]
    torch.cuda.synchronize()

    def work(mine):
        torch.cuda.set_device(want.device)
        for o in mine:
            gemm_bf16(a, b, out=o, stream=2)     # cudaStreamPerThread

    threads = [threading.Thread(target=work, args=(outs[k::2],)) for k in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    _check(outs, want)


def test_the_first_cuda_call_of_a_thread(product):
    """A thread that has made no CUDA call has no context yet; the product is its first."""
    from mini_nccl_b200.ops import gemm_bf16

    a, b, want, _ = product
    out = torch.zeros_like(want)
    torch.cuda.synchronize()
    failed = []

    def work():
        try:
            gemm_bf16(a, b, out=out, stream=0)
        except RuntimeError as e:
            failed.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not failed, failed
    _check([out], want)


def _capture(a, b, out, stream):
    from mini_nccl_b200.ops import gemm_bf16

    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream), torch.cuda.graph(g, stream=stream):
        gemm_bf16(a, b, out=out)
    return g


def test_captured_products_replay_beside_eager_ones(product):
    """Captured on a stream that never ran the product: split all the same, in a workspace of the graph's own."""
    from mini_nccl_b200.ops import gemm_bf16

    a, b, want, _ = product
    cap = torch.cuda.Stream()
    outs = [torch.zeros_like(want) for _ in range(4)]
    graphs = [_capture(a, b, outs[k], cap) for k in range(2)]     # two graphs from one stream
    elsewhere = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(4):
        for k in range(2):
            with torch.cuda.stream(elsewhere[k]):
                graphs[k].replay()
        gemm_bf16(a, b, out=outs[2], stream=cap)
        gemm_bf16(a, b, out=outs[3])
    _check(outs, want)


def test_products_of_one_capture_on_two_streams(product):
    from mini_nccl_b200.ops import gemm_bf16

    a, b, want, _ = product
    cap, side = torch.cuda.Stream(), torch.cuda.Stream()
    outs = [torch.zeros_like(want) for _ in range(4)]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(cap), torch.cuda.graph(g, stream=cap):
        side.wait_stream(cap)
        for k in range(2):
            gemm_bf16(a, b, out=outs[2 * k], stream=cap)
            gemm_bf16(a, b, out=outs[2 * k + 1], stream=side)
        cap.wait_stream(side)
    for _ in range(3):
        g.replay()
    _check(outs, want)


def test_workspaces_of_graphs_are_bounded_and_given_back(product):
    a, b, want, whole = product
    cap = torch.cuda.Stream()
    outs = [torch.zeros_like(want) for _ in range(10)]
    graphs = [_capture(a, b, o, cap) for o in outs]
    for g in graphs:
        g.replay()
    torch.cuda.synchronize()
    g = None
    split = [torch.equal(o, want) for o in outs]
    assert split == [True] * 8 + [False] * 2 and all(torch.equal(o, whole) for o in outs[8:])
    graphs.clear()                                               # destroys them
    torch.cuda.synchronize()
    again = [torch.zeros_like(want) for _ in range(3)]
    graphs = [_capture(a, b, o, cap) for o in again]
    for g in graphs:
        g.replay()
    _check(again, want)
