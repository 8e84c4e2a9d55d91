"""Pinned host buffers on one GPU: the reference's programs hand pinned host memory to
ncclAllReduce (src/main.cpp:35, tests/perf_test.cpp:78-79).  From 16 MB up the copy engines move such
buffers in chunks through a ring of four slots (host -> device, kernel, device -> host as a pipeline), below
that the kernel reads and writes them itself; the result must equal a plain PyTorch fp32 computation."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comm():
    import mini_nccl_b200 as mn

    c = mn.Communicator(1, 0)
    yield c
    c.destroy()


def test_host_in_host_out_scaled(comm):
    n = (5 << 20) + 777                       # 20 MB: five chunks of 4 MB and a ragged tail
    x = torch.randn(n).pin_memory()
    y = torch.zeros(n).pin_memory()
    before = comm.stats()["pipelined_calls"]
    comm.all_reduce(x, "sum", out=y, scale=0.5)
    torch.cuda.synchronize()
    assert torch.equal(y, x * 0.5)
    assert comm.stats()["pipelined_calls"] == before + 1


@pytest.mark.parametrize("n,pipelined", [(3 << 20, 0), ((10 << 20) + 3, 1)], ids=["kernel", "ring"])
def test_host_in_place(comm, n, pipelined):
    x = torch.randn(n).pin_memory()
    ref = x.clone()
    before = comm.stats()["pipelined_calls"]
    comm.all_reduce(x, "sum", scale=2.0)
    torch.cuda.synchronize()
    assert torch.equal(x, ref * 2.0)
    assert comm.stats()["pipelined_calls"] == before + pipelined


def test_host_to_device_and_back_with_cast(comm):
    n = (4 << 20) + 64
    x = torch.randn(n).pin_memory()
    d = torch.zeros(n, dtype=torch.bfloat16, device="cuda")
    comm.all_reduce(x, "sum", out=d)          # pinned fp32 -> device bf16
    torch.cuda.synchronize()
    assert torch.equal(d.cpu(), x.to(torch.bfloat16))
    h = torch.zeros(n).pin_memory()
    comm.all_reduce(d, "sum", out=h)          # device bf16 -> pinned fp32
    torch.cuda.synchronize()
    assert torch.equal(h, x.to(torch.bfloat16).float())


def test_small_host_buffer_takes_the_direct_kernel(comm):
    x = torch.randn(1000).pin_memory()
    y = torch.zeros(1000).pin_memory()
    before = comm.stats()["pipelined_calls"]
    comm.all_reduce(x, "sum", out=y)
    torch.cuda.synchronize()
    assert torch.equal(y, x)
    assert comm.stats()["pipelined_calls"] == before


@pytest.mark.parametrize("scale", [3.0, 1.0], ids=["kernel", "copy_engines_only"])
@pytest.mark.parametrize("n,pipelined", [(3 << 20, 0), ((10 << 20) + 3, 1)], ids=["direct", "ring"])
def test_host_pipeline_in_cuda_graph(comm, n, pipelined, scale):
    x = torch.randn(n).pin_memory()
    y = torch.zeros(n).pin_memory()
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        comm.all_reduce(x, "sum", out=y, scale=scale)   # a warm-up outside capture
        s.synchronize()
        before = comm.stats()["pipelined_calls"]
        with torch.cuda.graph(g, stream=s):
            comm.all_reduce(x, "sum", out=y, scale=scale)
    assert comm.stats()["pipelined_calls"] == before + pipelined
    for _ in range(2):
        y.zero_()
        x.neg_()                                         # a replay moves what is there now
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, x * scale)


def _filled(n, value):
    return torch.full((n,), float(value)).pin_memory()


@pytest.mark.parametrize("scale,mib", [(2.0, 40), (1.0, 160)], ids=["kernel", "copy_engines_only"])
def test_calls_on_two_streams_do_not_share_the_ring_at_once(comm, scale, mib):
    """Host buffers large enough that the ring of device slots wraps, on two streams that nothing orders: each call
    has to wait for the one before it to be through with the slots."""
    n = (mib << 20) // 4 + 13
    xs = [_filled(n, 1 + k) for k in range(2)]
    ys = [[torch.zeros(n).pin_memory() for _ in range(2)] for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    before = comm.stats()["pipelined_calls"]
    for it in range(2):
        for k, s in enumerate(streams):
            comm.all_reduce(xs[k], "sum", out=ys[k][it], scale=scale, stream=s)
    torch.cuda.synchronize()
    assert comm.stats()["pipelined_calls"] == before + 4
    for k in range(2):
        for it in range(2):
            assert torch.equal(ys[k][it], xs[k] * scale), (k, it)


def test_replay_beside_eager_calls(comm):
    """A captured pipelined call has a ring of its own: its replays run beside eager calls of the communicator."""
    n = (40 << 20) // 4 + 5
    x, y = _filled(n, 3), torch.zeros(n).pin_memory()
    ex, ey = _filled(n, 5), torch.zeros(n).pin_memory()
    cap, other = torch.cuda.Stream(), torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    before = comm.stats()["pipelined_calls"]
    with torch.cuda.stream(cap), torch.cuda.graph(g, stream=cap):
        comm.all_reduce(x, "sum", out=y, scale=3.0)
    assert comm.stats()["pipelined_calls"] == before + 1, "the captured call is pipelined, without a warm-up"
    for _ in range(3):
        with torch.cuda.stream(cap):
            g.replay()
        comm.all_reduce(ex, "sum", out=ey, scale=0.5, stream=other)
    torch.cuda.synchronize()
    assert torch.equal(y, x * 3.0) and torch.equal(ey, ex * 0.5)


def test_an_eager_call_between_the_calls_of_a_capture(comm):
    """The side streams of a captured call stay in the capture until it ends; eager calls do not meet them."""
    n = (20 << 20) // 4
    x, y, z = _filled(n, 1), torch.zeros(n).pin_memory(), torch.zeros(n).pin_memory()
    ex, ey = _filled(n, 7), torch.zeros(n).pin_memory()
    cap, other = torch.cuda.Stream(), torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(cap), torch.cuda.graph(g, stream=cap, capture_error_mode="relaxed"):
        comm.all_reduce(x, "sum", out=y, scale=2.0)
        comm.all_reduce(ex, "sum", out=ey, scale=2.0, stream=other)
        comm.all_reduce(x, "sum", out=z, scale=4.0)
    other.synchronize()
    assert torch.equal(ey, ex * 2.0)
    assert float(y[0]) == 0.0
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, x * 2.0) and torch.equal(z, x * 4.0)


def test_rings_of_graphs_are_bounded_and_reused():
    import mini_nccl_b200 as mn

    comm = mn.Communicator(1, 0)
    n = (16 << 20) // 4
    x = _filled(n, 1)
    try:
        def capture(scale):
            y = torch.zeros(n).pin_memory()
            g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            with torch.cuda.stream(s), torch.cuda.graph(g, stream=s):
                comm.all_reduce(x, "sum", out=y, scale=scale)
            return g, y

        live = [capture(float(k + 2)) for k in range(5)]
        assert comm.stats()["pipelined_calls"] == 4, "the fifth live graph holds a plain kernel"
        for g, _ in live:
            g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(y, x * float(k + 2)) for k, (_, y) in enumerate(live))
        g = None
        del live                                             # destroys the graphs: their rings are free again
        again = [capture(9.0) for _ in range(4)]
        assert comm.stats()["pipelined_calls"] == 8
        again[3][0].replay()
        torch.cuda.synchronize()
        assert torch.equal(again[3][1], x * 9.0)
        again = None
    finally:
        comm.destroy()


def test_staging_is_sized_for_the_message_and_grows():
    import mini_nccl_b200 as mn

    comm = mn.Communicator(1, 0)
    try:
        comm.all_reduce(_filled(1 << 20, 1).cuda())
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        for mib, most in ((32, 20), (200, 68), (32, 68)):            # four slots of an eighth, of 16 MB at most
            n = (mib << 20) // 4
            x, y = torch.randn(n).pin_memory(), torch.zeros(n).pin_memory()
            for scale in (1.0, 2.0):
                comm.all_reduce(x, "sum", out=y, scale=scale)
                torch.cuda.synchronize()
                assert torch.equal(y, x * scale)
            assert free - torch.cuda.mem_get_info()[0] <= most << 20, mib
        big = (160 << 20) // 4                                        # a later, larger call of one capture: a ring of its own
        x, y, z = torch.randn(big).pin_memory(), torch.zeros(big).pin_memory(), torch.zeros(big).pin_memory()
        g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.stream(s), torch.cuda.graph(g, stream=s):
            comm.all_reduce(x[:big // 8], "sum", out=y[:big // 8], scale=3.0)
            comm.all_reduce(x, "sum", out=z, scale=5.0)
        for _ in range(2):
            g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y[:big // 8], x[:big // 8] * 3.0) and torch.equal(z, x * 5.0)
    finally:
        comm.destroy()


def test_an_idle_ring_grows_inside_a_capture():
    """A ring that a destroyed graph gave back may be too small for the next capture: it grows there."""
    import mini_nccl_b200 as mn

    comm = mn.Communicator(1, 0)
    try:
        before = comm.stats()["pipelined_calls"]
        for mib in (20, 160, 20):
            x, y = torch.randn(mib << 18).pin_memory(), torch.zeros(mib << 18).pin_memory()
            g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            with torch.cuda.stream(s), torch.cuda.graph(g, stream=s):
                comm.all_reduce(x, "sum", out=y, scale=2.0)
            for _ in range(2):
                g.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, x * 2.0), mib
            del g
        assert comm.stats()["pipelined_calls"] == before + 3
    finally:
        comm.destroy()


def test_the_pipeline_starts_where_the_user_says():
    import mini_nccl_b200 as mn

    comm = mn.Communicator(1, 0)
    try:
        x, y = torch.randn(1 << 20).pin_memory(), torch.zeros(1 << 20).pin_memory()   # 4 MiB
        for knob, pipelined in ((None, 0), (1 << 20, 1), (0, 0), (8 << 20, 0)):
            if knob is not None:
                comm.set_knob("HOST_PIPELINE_MIN_BYTES", knob)
            before = comm.stats()["pipelined_calls"]
            comm.all_reduce(x, "sum", out=y.zero_(), scale=0.5)
            torch.cuda.synchronize()
            assert torch.equal(y, x * 0.5) and comm.stats()["pipelined_calls"] == before + pipelined, knob
    finally:
        comm.destroy()
