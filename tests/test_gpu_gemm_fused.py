"""The fused GEMM + collective kernels themselves, with one rank, through the test-suite's own copy of the library (the
public entry points leave a single rank to the plain GEMM).  GEMM -> reduce-scatter: every tile is rounded to bf16 into
the staging, announced by a flag, read back and written out, in alternating halves from call to call.  all-gather ->
GEMM: the producer looks for the counter of every row block, as for rows a peer delivers.  Operands are small
integers, so sums are exact in fp32 and results must equal the fp32 product rounded once."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hooks():
    from mini_nccl_b200 import _lib

    L = _lib.hooks_lib()
    vp, i = C.c_void_p, C.c_int
    L.mnccl_test_gemm_rs_fused.argtypes = [vp, vp, vp, i, i, i, vp, vp, vp, vp]
    L.mnccl_test_ag_gemm_fused.argtypes = [vp, vp, vp, i, i, i, vp, vp, vp, i, vp]
    L.mncclGemmRsStageBytes.restype = L.mncclGemmRsFlagWords.restype = L.mncclAgGemmReadyWords.restype = C.c_size_t
    L.mncclAgGemmReadyWords.argtypes = [i]
    yield L
    L.mncclGemmSetPairMode(-1)


def _operands(M, N, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a, b = (torch.randint(-3, 4, (r, K), generator=g, device="cuda").to(torch.bfloat16) for r in (M, N))
    return a, b, a.float() @ b.float().t()


def _status(L):
    st = C.c_uint32()
    assert L.mncclGemmStatus(C.byref(st)) == 0
    return st.value


def _words(n):
    return torch.zeros(max(n, 4), dtype=torch.int32, device="cuda")


# one tile; a ragged N; more tiles than CTAs, pairs of 128-row tiles and an odd number of them; the TP=8 shape
SHAPES = [(128, 64, 64), (128, 264, 200), (384, 1000, 512), (512, 1024, 384), (2560, 2048, 256), (4096, 4096, 1792)]


@pytest.mark.parametrize("pair", [0, 1], ids=["single_cta", "cta_pair"])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_reduce_scatter(hooks, M, N, K, pair):
    hooks.mncclGemmSetPairMode(pair)
    stage = torch.zeros(hooks.mncclGemmRsStageBytes(M, N, 1), dtype=torch.uint8, device="cuda")
    flags, state = _words(hooks.mncclGemmRsFlagWords(M, N, 1)), _words(4)
    stream = torch.cuda.current_stream().cuda_stream
    for call in range(3):                                        # epochs and staging halves
        a, b, want = _operands(M, N, K, call)
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        rc = hooks.mnccl_test_gemm_rs_fused(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, stage.data_ptr(), flags.data_ptr(),
                                            state.data_ptr(), stream)
        assert rc == 0 and _status(hooks) == 0
        assert torch.equal(out, want.to(torch.bfloat16)), call
        assert state.tolist()[:2] == [call + 1, 0], "epoch stored, ticket cleared"
    assert int(flags.max()) == 3


@pytest.mark.parametrize("swiglu", [False, True], ids=["plain", "swiglu"])
@pytest.mark.parametrize("pair", [0, 1], ids=["single_cta", "cta_pair"])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_all_gather_gemm(hooks, M, N, K, pair, swiglu):
    if swiglu and N % 32:
        N = N // 32 * 32
    hooks.mncclGemmSetPairMode(pair)
    ready, bar, state = _words(hooks.mncclAgGemmReadyWords(M)), _words(4096), _words(4)
    stream = torch.cuda.current_stream().cuda_stream
    for call in range(3):
        a, b, want = _operands(M, N, K, call)
        ready[:M // 128] += 4                                    # four quarters of every row block have arrived
        out = torch.full((M, N // 2 if swiglu else N), float("nan"), dtype=torch.bfloat16, device="cuda")
        if swiglu:
            b = (b.float() / 8).to(torch.bfloat16)               # exact; keeps silu away from its flat ends
            want = a.float() @ b.float().t()
        rc = hooks.mnccl_test_ag_gemm_fused(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, ready.data_ptr(), bar.data_ptr(),
                                            state.data_ptr(), int(swiglu), stream)
        assert rc == 0 and _status(hooks) == 0
        if swiglu:
            h = want.double().view(M, N // 32, 2, 16)
            act = (h[:, :, 0] * torch.sigmoid(h[:, :, 0]) * h[:, :, 1]).reshape(M, N // 2)
            # one rounding to bf16 (2^-9 of the value, here 2^-8 with room for __expf and the fp32 product)
            assert torch.all((out.double() - act).abs() <= act.abs() * 2.0 ** -8 + 1e-30), call
        else:
            assert torch.equal(out, want.to(torch.bfloat16)), call
        assert state.tolist()[:2] == [call + 1, 0]
