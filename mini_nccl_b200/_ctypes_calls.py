"""The calls of the PyTorch extension (csrc/torch/ext.cpp) through ctypes, with the same arguments, results and
errors: for a PyTorch without CUDA, against which the extension cannot be built, and wherever else it is missing.
About 8 us slower per call."""
from __future__ import annotations

import ctypes as C

import torch

_CODES = {torch.int8: 0, torch.uint8: 1, torch.int32: 2, torch.int64: 4, torch.float16: 6, torch.float32: 7, torch.float64: 8,
          torch.bfloat16: 9}
_CODES.update({getattr(torch, name): code for name, code in (("uint32", 3), ("uint64", 5)) if hasattr(torch, name)})


def _stream(stream) -> int:
    if stream is None:
        return torch.cuda.current_stream().cuda_stream if torch.cuda.is_available() else 0
    return stream.cuda_stream if hasattr(stream, "cuda_stream") else int(stream)


def _tensor(t, name):
    if not isinstance(t, torch.Tensor):
        raise TypeError(f"{name} must be a torch tensor")
    return t


def _bf16(*tensors):
    return all(t.dtype == torch.bfloat16 for t in tensors)


def all_reduce(lib, comm, tensor, out, wire_dtype, op, scale, algo, stream):
    out = _tensor(tensor, "tensor") if out is None else _tensor(out, "out")
    if not tensor.is_contiguous() or not out.is_contiguous():
        raise ValueError("all_reduce needs contiguous tensors")
    if out.numel() != tensor.numel():
        raise ValueError("size mismatch")
    if wire_dtype is not None and not isinstance(wire_dtype, torch.dtype):
        raise TypeError("wire_dtype must be a torch dtype")
    wire = wire_dtype if wire_dtype is not None else (out.dtype if tensor.dtype == out.dtype else torch.bfloat16)
    if not {tensor.dtype, out.dtype, wire} <= _CODES.keys():
        raise TypeError("unsupported dtype")
    return lib.mncclAllReduceEx(tensor.data_ptr(), _CODES[tensor.dtype], out.data_ptr(), _CODES[out.dtype], _CODES[wire], tensor.numel(),
                                op, float(scale), algo, comm, _stream(stream))


def gemm(lib, a, b, out, out_dtype, stream):
    if not _bf16(_tensor(a, "a"), _tensor(b, "b")):
        raise TypeError("gemm_bf16 needs bf16 operands")
    if a.dim() != 2 or b.dim() != 2 or a.shape[1] != b.shape[1]:
        raise ValueError("shapes: a [M, K], b [N, K]")
    if a.stride(1) != 1 or b.stride(1) != 1:
        raise ValueError("operands need a unit inner stride")
    (M, K), N = a.shape, b.shape[0]
    if out is None:
        if out_dtype is not None and not isinstance(out_dtype, torch.dtype):
            raise TypeError("out_dtype must be a torch dtype")
        out = torch.empty((M, N), dtype=out_dtype or torch.bfloat16, device=a.device)
    if _tensor(out, "out").dtype not in (torch.bfloat16, torch.float32) or tuple(out.shape) != (M, N) or out.stride(1) != 1:
        raise ValueError("out must be [M, N] bf16 or fp32 with a unit inner stride")
    rc = lib.mncclGemmBf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, a.stride(0), b.stride(0), out.stride(0),
                           1 if out.dtype == torch.float32 else 0, _stream(stream))
    if rc != 0:
        raise RuntimeError(f"mncclGemmBf16 failed with code {rc}")
    return out


def _error(lib, comm) -> int:
    e = C.c_int()
    rc = lib.mncclCommGetAsyncError(comm, C.byref(e))
    return rc if rc != 0 else e.value


def _pointers(address):
    return C.cast(C.c_void_p(address), C.POINTER(C.c_void_p))


def _bytes(address):
    return C.cast(C.c_void_p(address), C.c_char_p)


def gemm_rs(lib, comm, a, b, out, stream, workspace):
    M, N, rank, ranks, stage, flags, state, handle, handle_bytes = workspace
    _tensor(a, "a"), _tensor(b, "b")
    if a.dim() != 2 or b.dim() != 2 or a.shape[0] != M or b.shape[0] != N or a.shape[1] != b.shape[1]:
        raise ValueError("shape mismatch")
    if not _bf16(a, b) or a.stride(1) != 1 or b.stride(1) != 1:
        raise TypeError("bf16 operands with a unit inner stride")
    if out is None:
        out = torch.empty((M // ranks, N), dtype=torch.bfloat16, device=a.device)
    s, e = _stream(stream), _error(lib, comm)
    if e != 0:
        return e
    rc = lib.mncclGemmReduceScatterBf16Comm(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, a.shape[1], a.stride(0), b.stride(0),
                                            out.stride(0), rank, ranks, _pointers(stage), _pointers(flags), state,
                                            _bytes(handle), handle_bytes, s)
    if rc != 0:
        raise RuntimeError(f"mncclGemmReduceScatterBf16 failed with code {rc}")
    return out


def ag_gemm(lib, comm, n_comm_ctas, b, out, stream, swiglu, workspace):
    M, K, rank, ranks, xg, ready, bar, state, handle, handle_bytes = workspace
    if not _bf16(_tensor(b, "b")) or b.dim() != 2 or b.shape[1] != K or b.stride(1) != 1:
        raise TypeError("b must be bf16 [N, K] with a unit inner stride")
    N = b.shape[0]
    if swiglu and N % 32:
        raise ValueError("SwiGLU in the epilogue needs N a multiple of 32")
    n_out = N // 2 if swiglu else N
    if out is None:
        out = torch.empty((M, n_out), dtype=torch.bfloat16, device=b.device)
    if tuple(_tensor(out, "out").shape) != (M, n_out) or out.dtype != torch.bfloat16 or out.stride(1) != 1:
        raise ValueError(f"out must be bf16 [{M}, {n_out}] with a unit inner stride")
    s, e = _stream(stream), _error(lib, comm)
    if e != 0:
        return e
    rc = lib.mncclAllGatherGemmBf16Comm(_pointers(xg), b.data_ptr(), out.data_ptr(), M, N, K, K, b.stride(0), out.stride(0), rank, ranks,
                                        _pointers(ready), _pointers(bar), state, n_comm_ctas, 1 if swiglu else 0, _bytes(handle),
                                        handle_bytes, s)
    if rc != 0:
        raise RuntimeError(f"all-gather->GEMM kernel failed with code {rc}")
    return out


class Calls:
    """The extension's functions, bound to a loaded library."""

    def __init__(self, lib):
        from functools import partial

        for f in (all_reduce, gemm, gemm_rs, ag_gemm):
            setattr(self, f.__name__, partial(f, lib))
