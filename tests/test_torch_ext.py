"""The PyTorch extension of the binding and the ctypes calls that stand in for it where it cannot be built."""
import subprocess
import sys
from pathlib import Path

import pytest

torch = pytest.importorskip("torch")

ROOT = Path(__file__).resolve().parent.parent


def _run(code, env=None, cwd=ROOT):
    import os

    e = dict(os.environ, PYTHONPATH=str(ROOT))
    e.update(env or {})
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=str(cwd), timeout=240, env=e)
    assert r.returncode == 0, r.stdout + r.stderr
    return r


def test_pytorch_without_cuda_uses_ctypes(free_port):
    """A PyTorch without CUDA has no c10_cuda to link against: build() passes the extension over and the network
    plane works through ctypes (two ranks on host memory)."""
    code = """
import sys, torch
import mini_nccl_b200.build as b
from mini_nccl_b200 import _ext_file
_ext_file.torch_dir = lambda: None
assert b.build_torch_ext() is None
import mini_nccl_b200 as mn
from mini_nccl_b200 import _lib
assert type(_lib.ext()).__name__ == "Calls"
rank = int(sys.argv[1])
comm = mn.Communicator(2, rank, "127.0.0.1")
x = torch.arange(1000, dtype=torch.float32) + rank
y = torch.empty_like(x)
assert comm.all_reduce(x, "sum", out=y) is y
assert torch.equal(y, torch.arange(1000, dtype=torch.float32) * 2 + 1)
assert comm.all_reduce(x, "max") is x and torch.equal(x, torch.arange(1000, dtype=torch.float32) + 1)
for bad, error in ((lambda: comm.all_reduce(x[::2]), ValueError), (lambda: comm.all_reduce(x, out=y[:3]), ValueError),
                   (lambda: comm.all_reduce(x.bool()), TypeError), (lambda: comm.all_reduce([1.0]), TypeError)):
    try:
        bad()
    except error:
        continue
    raise AssertionError(error)
comm.destroy()
"""
    import os

    env = dict(os.environ, PYTHONPATH=str(ROOT), MINI_NCCL_BOOTSTRAP_PORT=str(free_port), CUDA_VISIBLE_DEVICES="")
    procs = [subprocess.Popen([sys.executable, "-c", code, str(r)], cwd=str(ROOT), env=env, stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                              text=True) for r in range(2)]
    outs = [p.communicate(timeout=120)[0] for p in procs]
    assert [p.returncode for p in procs] == [0, 0], outs


def test_no_build_is_honoured():
    """MINI_NCCL_NO_BUILD=1: a missing extension is not compiled; its calls go through ctypes, and a warning says so."""
    _run("""
import warnings
import mini_nccl_b200.build as b
from mini_nccl_b200 import _ext_file, _lib
def never(*a, **k): raise AssertionError("built although MINI_NCCL_NO_BUILD=1")
b.build_torch_ext = never
_lib.lib()
_ext_file.DIR = _ext_file.DIR / "nowhere"   # the extension's file is missing
with warnings.catch_warnings(record=True) as w:
    warnings.simplefilter("always")
    assert type(_lib.ext()).__name__ == "Calls"
assert any("MINI_NCCL_NO_BUILD" in str(x.message) for x in w)
""", {"MINI_NCCL_NO_BUILD": "1"})


def test_without_a_compiler_the_calls_go_through_ctypes(tmp_path):
    _run("""
import os, warnings, torch
from pathlib import Path
import mini_nccl_b200.build as b
from mini_nccl_b200 import _ext_file, _lib
_ext_file.DIR = b.BUILD = Path(%r)
_lib.lib()
os.environ["PATH"] = ""                     # no g++
with warnings.catch_warnings(record=True) as w:
    warnings.simplefilter("always")
    assert type(_lib.ext()).__name__ == "Calls"
assert any("g++" in str(x.message) for x in w)
""" % str(tmp_path))


def test_the_file_is_that_of_this_pytorch_python_and_source(tmp_path):
    _run("""
import importlib.machinery, torch
from pathlib import Path
from mini_nccl_b200 import _ext_file as f, _lib
path = f.torch_ext_path()
assert torch.__version__ in path.name and path.name.endswith(importlib.machinery.EXTENSION_SUFFIXES[0])
assert Path(_lib.ext().__file__) == path, "the file loaded is the one of this name"
tmp = Path(%r)
other = tmp / "torch"
(other / "lib").mkdir(parents=True)
(other / "lib" / "libc10_cuda.so").touch()
(other / "version.py").write_text("__version__ = '9.9.9'\\n")
real = f.torch_dir
f.torch_dir = lambda: other
assert "9.9.9" in f.torch_ext_path().name, "another PyTorch, another file"
f.torch_dir = real
src = f.CSRC
f.CSRC = tmp / "csrc"
(f.CSRC / "torch").mkdir(parents=True)
(f.CSRC / "torch" / "ext.cpp").write_text((src / "torch" / "ext.cpp").read_text() + "// edited")
assert f.torch_ext_path() not in (None, path), "an edited source, another file"
""" % str(tmp_path))


def test_processes_that_start_together_build_it_once_and_never_see_half_a_file(tmp_path):
    """A stand-in compiler that writes its output in two halves, a moment apart; three processes find the file
    missing at the same time."""
    fake = tmp_path / "bin" / "g++"
    fake.parent.mkdir()
    fake.write_text('#!/bin/sh\necho run >> "%s/runs"\nwhile [ "$1" != "-o" ]; do shift; done\nprintf first > "$2"\nsleep 1\n'
                    'printf second >> "$2"\n' % tmp_path)
    fake.chmod(0o755)
    code = """
import sys, threading
from pathlib import Path
import mini_nccl_b200.build as b
from mini_nccl_b200 import _ext_file
_ext_file.DIR = b.BUILD = Path(%r)
path, seen, done = _ext_file.torch_ext_path(), [], threading.Event()
def watch():
    while not done.is_set():
        if path.exists(): seen.append(path.read_text())
t = threading.Thread(target=watch); t.start()
assert b.build_torch_ext() == path
done.set(); t.join()
assert path.read_text() == "firstsecond" and set(seen) <= {"firstsecond"}, set(seen)
""" % str(tmp_path)
    import os

    env = dict(os.environ, PYTHONPATH=str(ROOT), PATH=f"{fake.parent}:{os.environ['PATH']}")
    procs = [subprocess.Popen([sys.executable, "-c", code], env=env, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
             for _ in range(3)]
    outs = [p.communicate(timeout=120)[0] for p in procs]
    assert [p.returncode for p in procs] == [0, 0, 0], outs
    assert (tmp_path / "runs").read_text() == "run\n"
    assert [p.suffix for p in tmp_path.glob("_torch_ext*")] == [".so"]


@pytest.mark.gpu
def test_ctypes_calls_give_what_the_extension_gives():
    import mini_nccl_b200 as mn
    from mini_nccl_b200 import _lib
    from mini_nccl_b200._ctypes_calls import Calls
    from mini_nccl_b200.ops import AllGatherGemm, GemmReduceScatter

    calls, ext = Calls(mn.lib()), _lib.ext()
    assert type(ext).__name__ == "module"
    comm = mn.Communicator(1, 0)
    try:
        g = torch.Generator(device="cuda").manual_seed(3)
        a, b = (torch.randn(256, 192, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
        x = torch.randn(4097, generator=g, device="cuda")
        for out in (None, torch.empty(4097, device="cuda"), torch.empty(4097, dtype=torch.bfloat16, device="cuda")):
            got = []
            for c in (ext, calls):
                src, dst = x.clone(), None if out is None else out.clone()
                assert c.all_reduce(comm._h.value, src, dst, None, 0, 0.5, 0, None) == 0
                got.append(src if dst is None else dst)
            assert torch.equal(*got)
        for dtype in (None, torch.float32):
            assert torch.equal(ext.gemm(a, b, None, dtype, None), calls.gemm(a, b, None, dtype, torch.cuda.current_stream()))
        rs, ag = GemmReduceScatter(comm, 256, 256), AllGatherGemm(comm, 256, 192)
        ag.local_shard.copy_(a)
        want_rs, want_ag, want_act = rs(a, b), ag(b), ag(b, swiglu=True)
        rs._call, ag._call = calls.gemm_rs, calls.ag_gemm
        assert torch.equal(rs(a, b), want_rs) and torch.equal(ag(b), want_ag) and torch.equal(ag(b, swiglu=True), want_act)
        for c in (ext, calls):
            for error, bad in ((TypeError, lambda: c.gemm(a.float(), b, None, None, None)), (ValueError, lambda: c.gemm(a, b[:, :8], None, None, None)),
                               (ValueError, lambda: c.gemm(a, b, a, None, None)), (ValueError, lambda: c.gemm(a.t(), b.t(), None, None, None)),
                               (ValueError, lambda: c.gemm_rs(comm._h.value, a[:8], b, None, None, rs._workspace)),
                               (TypeError, lambda: c.ag_gemm(comm._h.value, 0, b.float(), None, None, False, ag._workspace))):
                with pytest.raises(error):
                    bad()
    finally:
        comm.destroy()
