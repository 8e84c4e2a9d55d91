"""The GEMM for small products (swapped operands, K over the CTAs of a cluster) and the persistent kernels'
store to rows that start anywhere.  Operands are small integers, so every partial sum is exact in fp32
whatever the order or the number of slices: results must equal the fp32 product bit for bit (bf16: its one
rounding)."""
import ctypes as C

import pytest
import torch


def _plan(M, N, K, out=0):
    import mini_nccl_b200 as mn

    tn, slices, deep = C.c_int(0), C.c_int(0), C.c_int(0)
    used = mn.lib().mncclGemmSmallPlan(M, N, K, out, 148, C.byref(tn), C.byref(slices), C.byref(deep))
    return (tn.value, slices.value, bool(deep.value)) if used else None


def test_plan_covers_the_kernel_variants_and_leaves_large_products_alone():
    plans = [_plan(M, N, K) for M in (1, 16, 17, 40, 128, 300, 777) for N in (64, 300, 1003, 4096, 14336) for K in (64, 200, 1544, 4096, 14336)]
    plans = [p for p in plans if p]
    assert {p[0] for p in plans} == {16, 32, 64, 128} and {p[1] for p in plans} == {1, 2, 4, 8} and {p[2] for p in plans} == {False, True}
    for M, N, K in ((4096, 14336, 4096), (4096, 3584, 4096), (4096, 4096, 1792), (2048, 2048, 2048), (8192, 4096, 512)):
        assert _plan(M, N, K) is None


def _ints(rows, cols, seed, pad=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-3, 4, (rows, cols + pad), generator=g, device="cuda").to(torch.bfloat16)[:, :cols]


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1, 1, 8), (1, 129, 64), (15, 64, 72), (16, 14336, 136), (17, 4096, 4096), (33, 300, 14336),
                                   (64, 256, 8192), (65, 1003, 1544), (127, 1024, 1024), (129, 640, 320), (300, 300, 14336),
                                   (777, 1003, 1544), (512, 512, 512), (256, 4096, 4096), (5, 50257, 128)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_small_products_exact(M, N, K, out_dtype):
    from mini_nccl_b200.ops import gemm_bf16, gemm_status

    assert _plan(M, N, K, 1 if out_dtype == torch.float32 else 0), "this shape was meant for the small kernel"
    a, b = _ints(M, K, M * 7 + K, pad=8), _ints(N, K, N * 3 + K)
    guard = torch.full((M + 1, N + 3), 7.0, dtype=out_dtype, device="cuda")
    gemm_bf16(a, b, out=guard[:M, :N])
    torch.cuda.synchronize()
    assert gemm_status() == 0
    assert torch.equal(guard[:M, :N], (a.float() @ b.float().t()).to(out_dtype))
    assert torch.all(guard[M] == 7) and torch.all(guard[:, N:] == 7), "wrote outside the result"


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,ffn,hidden", [(128, 16, 512), (128, 1792, 512), (256, 272, 1024), (384, 3584, 4096)])
def test_swiglu_and_reduce_scatter_of_few_tokens(tokens, ffn, hidden):
    """One rank's tensor-parallel MLP on the kernels for small products, and (3584 x 4096) on the persistent
    ones with the last wave's tiles cut along K."""
    import mini_nccl_b200 as mn
    from mini_nccl_b200.ops import AllGatherGemm, GemmReduceScatter, gemm_status, interleave_gate_up

    comm = mn.Communicator(1, 0)
    try:
        g = torch.Generator(device="cuda").manual_seed(tokens + ffn)
        x = torch.randn(tokens, hidden, generator=g, device="cuda").to(torch.bfloat16)
        wg, wu = ((torch.randn(ffn, hidden, generator=g, device="cuda") * 0.05).to(torch.bfloat16) for _ in range(2))
        ag = AllGatherGemm(comm, tokens, hidden)
        ag.local_shard.copy_(x)
        act = ag(interleave_gate_up(wg, wu), swiglu=True)
        gt, ut = x.float() @ wg.float().t(), x.float() @ wu.float().t()
        ref = gt * torch.sigmoid(gt) * ut
        # one rounding to bf16 (2^-9 relative) of an fp32 value; the sums' order moves it by far less
        assert torch.all((act.float() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-4 * ref.abs().max())
        rs = GemmReduceScatter(comm, tokens, hidden)
        a, b = _ints(tokens, ffn, 5), _ints(hidden, ffn, 6)
        assert torch.equal(rs(a, b), (a.float() @ b.float().t()).to(torch.bfloat16))
        assert gemm_status() == 0
    finally:
        comm.destroy()


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("M,N,K,out_dtype", [(300, 1003, 136, torch.bfloat16), (513, 515, 72, torch.float32), (4096, 3593, 4096, torch.bfloat16)])
def test_persistent_kernels_store_rows_that_start_anywhere(mode, M, N, K, out_dtype):
    from mini_nccl_b200.ops import gemm_bf16, gemm_status
    from mini_nccl_b200.ops.gemm import set_pair_mode

    a, b = _ints(M, K, 1), _ints(N, K, 2)
    guard = torch.full((M + 1, N + 2), 7.0, dtype=out_dtype, device="cuda")
    set_pair_mode(mode)
    try:
        gemm_bf16(a, b, out=guard[:M, :N])
        torch.cuda.synchronize()
    finally:
        set_pair_mode(-1)
    assert gemm_status() == 0
    assert torch.equal(guard[:M, :N], (a.float() @ b.float().t()).to(out_dtype))
    assert torch.all(guard[M] == 7) and torch.all(guard[:, N:] == 7), "wrote outside the result"
