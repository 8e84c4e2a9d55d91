"""bf16 GEMM on the Blackwell tensor cores (tcgen05.mma, accumulators in tensor memory, operands
staged by TMA): ``C = A @ B.T`` with ``A [M, K]`` and ``B [N, K]`` row-major, the layout of an
``nn.Linear`` weight.  Fails loudly when the native kernel is missing: there is no fallback."""
from __future__ import annotations

import ctypes as C

from .._lib import ext, lib

_gemm = None   # the extension's entry point, looked up on the first call


def _native():
    L = lib()
    if not hasattr(L, "mncclGemmBf16"):
        raise RuntimeError("libmini_nccl.so was built without the sm_100a GEMM (csrc/kernels/gemm_sm100.cu)")
    return L


def gemm_bf16(a, b, out=None, out_dtype=None, stream=None):
    """``out[M, N] = a[M, K] @ b[N, K].T``; ``a`` and ``b`` bf16 with a unit inner stride."""
    global _gemm
    if _gemm is None:
        _native()
        _gemm = ext().gemm
    return _gemm(a, b, out, out_dtype, stream)


def gemm_status() -> int:
    """Error word of the GEMM kernels on the current device (0 = every bounded wait completed); clears it."""
    st = C.c_uint32()
    rc = _native().mncclGemmStatus(C.byref(st))
    if rc != 0:
        raise RuntimeError(f"mncclGemmStatus failed with code {rc}")
    return st.value


def set_pair_mode(mode: int) -> None:
    """-1: automatic; 0: single-CTA 128 x 256 tiles; 1: CTA pairs (tcgen05 cta_group::2, 256 x 256 tiles)."""
    _native().mncclGemmSetPairMode(int(mode))


def gemm_plan(M: int, N: int, ctas: int = 148, narrow: bool = True):
    """``(tile_n, pair)``: the tile width the single-CTA kernel would use for an ``M x N`` product on
    ``ctas`` CTAs and whether the CTA-pair kernel would be taken instead.  Host logic only; needs no GPU."""
    import ctypes as C

    tile_n, pair = C.c_int(0), C.c_int(0)
    _native().mncclGemmPlan(int(M), int(N), int(ctas), 1 if narrow else 0, C.byref(tile_n), C.byref(pair))
    return tile_n.value, bool(pair.value)
