"""The one-rank AllReduce kernels at the sizes and alignments where their work split can go wrong: units of
32 bytes, tiles of 256 threads x 2 or 4 units, the last count % unit elements, buffers that are only
element-aligned, host buffers around the chunk pipeline's boundaries.  The result is one product rounded
once, so it must equal PyTorch's bit for bit."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

F32, BF16, F16, F64, I8, I32, I64 = (torch.float32, torch.bfloat16, torch.float16, torch.float64, torch.int8, torch.int32,
                                     torch.int64)


@pytest.fixture(scope="module")
def comm():
    import mini_nccl_b200 as mn

    c = mn.Communicator(1, 0)
    yield c
    c.destroy()


def _values(n, dtype):
    return torch.randint(-100, 100, (n,), device="cuda", dtype=dtype) if not dtype.is_floating_point else torch.randn(n, device="cuda").to(dtype)


@pytest.mark.parametrize("src,dst", [(F32, F32), (BF16, BF16), (BF16, F32), (F32, BF16), (F16, F16), (F64, F64), (I8, I8), (I32, I32), (I64, I64)])
def test_every_remainder_and_alignment(comm, src, dst):
    unit = 32 // max(torch.tensor([], dtype=src).element_size(), torch.tensor([], dtype=dst).element_size())
    tile = 256 * (2 if src == dst else 4) * unit
    for count in (1, unit - 1, unit, unit + 1, tile - 1, tile, tile + 1, 3 * tile + unit + 1):
        for off_in, off_out in ((0, 0), (unit // 2, unit // 2), (1, 0), (0, 1)):
            x = _values(count + off_in, src)[off_in:]
            guard = torch.full((count + off_out + 64,), 7, dtype=dst, device="cuda")
            y = guard[off_out:off_out + count]
            for scale in (1.0, 0.375) if src.is_floating_point else (1.0,):
                comm.all_reduce(x, "sum", out=y, scale=scale)
                wide = torch.float64 if dst == F64 else torch.float32
                want = (x.to(wide) * scale).to(dst) if src.is_floating_point else x
                assert torch.equal(y, want), (count, off_in, off_out, scale)
                assert torch.all(guard[:off_out] == 7) and torch.all(guard[off_out + count:] == 7), "wrote outside the result"


@pytest.mark.parametrize("mib,extra", [(0, 1000), (16, -1), (16, 0), (33, 777), (150, 5)])
@pytest.mark.parametrize("scale", [1.0, 0.5])
def test_host_buffers_around_the_pipeline_boundaries(comm, mib, extra, scale):
    n = (mib << 18) + extra
    x, y = torch.randn(n, pin_memory=True), torch.zeros(n, pin_memory=True)
    d = torch.zeros(n, device="cuda")
    for _ in range(2):                                     # the second call meets the slots of the first
        y.zero_()
        comm.all_reduce(x, "sum", out=y, scale=scale)      # host -> host
        comm.all_reduce(x, "sum", out=d, scale=scale)      # host -> device
        torch.cuda.synchronize()
        assert torch.equal(y, x * scale) and torch.equal(d.cpu(), x * scale)
    y.zero_()
    comm.all_reduce(d, "sum", out=y, scale=scale)          # device -> host
    torch.cuda.synchronize()
    assert torch.equal(y, x * scale * scale)


@pytest.mark.parametrize("offset", [0, 1])
def test_local_sum_of_unaligned_and_ragged_buffers(offset):
    import ctypes as C

    import mini_nccl_b200 as mn

    fn = mn.lib().mncclLocalAllReduceNoAlloc
    fn.restype, fn.argtypes = C.c_int, [C.POINTER(C.c_void_p), C.POINTER(C.c_void_p), C.c_int, C.c_size_t, C.c_int, C.c_int, C.c_void_p]
    for n, count in ((2, 1), (3, 513), (4, 16383)):
        ins = [torch.randn(count + offset, device="cuda")[offset:] for _ in range(n)]
        outs = [torch.zeros(count + offset, device="cuda")[offset:] for _ in range(n)]
        want = ins[0].clone()
        for t in ins[1:]:
            want += t                                      # the same order, fp32: the same bits
        sp, rp = (C.c_void_p * n)(*[t.data_ptr() for t in ins]), (C.c_void_p * n)(*[t.data_ptr() for t in outs])
        assert fn(sp, rp, n, count, mn.FLOAT32, mn.SUM, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert all(torch.equal(o, want) for o in outs), (n, count)
