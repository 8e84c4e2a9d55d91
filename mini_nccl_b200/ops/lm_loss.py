"""Output projection and mean cross-entropy of a language model as one autograd node.

``F.cross_entropy(F.linear(x, weight).float(), targets)`` on the kernels of csrc/kernels/lm_loss.cu and the
tcgen05 GEMM.  Two things made the plain operators slow: a vocabulary that is not a multiple of eight (50257) leaves
the rows of the logits unaligned, and the library's only kernels for such rows run the products at a fifth of the
tensor cores' rate; and the logits went through memory thirteen times.  Here their rows are padded in memory and the
loss touches them once forward and once backward: 8192 tokens, 1024 features, 50257 classes 21.1 -> 8.2 ms forward
and backward, 32000 classes 3.4 -> 1.7 ms.

One product stays with the library where the vocabulary is not a multiple of eight, the gradient of the activations.
The GEMM would take it from 5.3 to 0.6 ms (8192 tokens, 1024 features, 50257 classes) and is closer to a 64-bit
reference (1.7e-3 of the norm against 3.0e-3: the library's sum over the classes is split and rounded), but that
difference grows through a deep decoder's backward pass: with 24 layers single gradients moved by up to 1.1 times their
bucket's root mean square, two to three times what two runs of the same code differ by."""
from __future__ import annotations

import torch
import torch.nn.functional as F

from .._lib import lib
from .gemm import gemm_bf16

_MAX_ROWS = 65535 * 64   # mncclLmLossBackward and mncclTransposeBf16


def _reference(x, weight, targets):
    logits = F.linear(x, weight)
    return F.cross_entropy(logits.float().view(-1, logits.size(-1)), targets.view(-1))


def _eight(n):
    return (n + 7) // 8 * 8


def _check(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what} failed with code {rc}")


def _rows(t):
    """``t`` as the kernels read it: dense rows that start on 16 bytes (saved-tensor hooks may hand back any copy)."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _transposed(t, stream):
    rows, cols = t.shape
    out = torch.empty((cols, _eight(rows)), dtype=t.dtype, device=t.device)
    _check(lib().mncclTransposeBf16(t.data_ptr(), t.stride(0), rows, cols, out.data_ptr(), out.stride(0), stream),
           "mncclTransposeBf16")
    return out[:, :rows]


class _LmHeadCrossEntropy(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, targets):
        V = weight.shape[0]
        rows, w, t = _rows(x.detach()).view(-1, x.shape[-1]), _rows(weight.detach()), targets.view(-1).contiguous()
        T = rows.shape[0]
        logits = torch.empty((T, _eight(V)), dtype=x.dtype, device=x.device)
        gemm_bf16(rows, w, out=logits[:, :V])
        # gather checks the indices, as the loss does; -100 marks rows that count for nothing
        picked = logits[:, :V].gather(1, torch.where(t == -100, 0, t).unsqueeze(1))
        lse, row_loss = torch.empty((2, T), dtype=torch.float32, device=x.device)
        mean = torch.empty(2, dtype=torch.float32, device=x.device)
        _check(lib().mncclLmLossForward(logits.data_ptr(), logits.stride(0), T, V, t.data_ptr(), picked.data_ptr(), lse.data_ptr(),
                                        row_loss.data_ptr(), mean.data_ptr(), torch.cuda.current_stream().cuda_stream),
               "mncclLmLossForward")
        ctx.save_for_backward(x, weight, t, logits, lse, mean)
        return mean[0].clone()

    @staticmethod
    def backward(ctx, grad):
        x, weight, t, logits, lse, mean = ctx.saved_tensors
        want_x, want_w = ctx.needs_input_grad[:2]
        if torch.is_grad_enabled():   # create_graph: the gradient itself is differentiated, by the plain operators
            ins = [x.view_as(x), weight.view_as(weight)]
            picks = [i for i, want in enumerate((want_x, want_w)) if want]
            got = torch.autograd.grad(_reference(ins[0], ins[1], t), [ins[i] for i in picks], grad, create_graph=True)
            out = dict(zip(picks, got))
            return out.get(0), out.get(1), None
        stream = torch.cuda.current_stream().cuda_stream
        V = weight.shape[0]
        rows, logits, grad = _rows(x).view(-1, x.shape[-1]), _rows(logits), grad.contiguous()
        T = rows.shape[0]
        d = torch.empty((T, _eight(V)), dtype=x.dtype, device=x.device) if want_x else None
        dt = torch.empty((V, _eight(T)), dtype=x.dtype, device=x.device) if want_w else None
        _check(lib().mncclLmLossBackward(logits.data_ptr(), logits.stride(0), T, V, t.data_ptr(), lse.data_ptr(), grad.data_ptr(),
                                         mean.data_ptr(), d.data_ptr() if want_x else None, _eight(V),
                                         dt.data_ptr() if want_w else None, _eight(T), stream), "mncclLmLossBackward")
        dx = None
        if want_x and V % 8 == 0:
            dx = gemm_bf16(d, _transposed(_rows(weight), stream)).view(x.shape)
        elif want_x:   # dense rows, as the library always had them
            dx = torch.mm(d[:, :V].contiguous(), _rows(weight)).view(x.shape)
        del d
        dw = gemm_bf16(dt[:, :T], _transposed(rows, stream)) if want_w else None
        return dx, dw, None


def _plain(t):
    return type(t) in (torch.Tensor, torch.nn.Parameter) and t.layout == torch.strided


def _native(x, weight, targets):
    """Whether the kernels take the call: bf16 matrices and 64-bit indices on the current GPU, with nothing active
    that looks at or transforms the single operators (autocast, tracing, vmap, forward-mode, modes)."""
    if not (x.is_cuda and _plain(x) and _plain(weight) and _plain(targets)):
        return False
    if not (x.dtype == weight.dtype == torch.bfloat16 and targets.dtype == torch.int64):
        return False
    if not (x.device == weight.device == targets.device and x.device.index == torch.cuda.current_device()):
        return False
    if x.dim() < 2 or weight.dim() != 2 or x.shape[-1] != weight.shape[1] or x.shape[:-1] != targets.shape:
        return False
    T, (V, d) = targets.numel(), weight.shape
    if T == 0 or V < 8 or d < 8 or d % 8 != 0 or max(T, V) > _MAX_ROWS:
        return False
    if torch.is_autocast_enabled() or torch.jit.is_tracing() or torch.compiler.is_compiling():
        return False
    if torch._C._are_functorch_transforms_active() or torch._C._len_torch_function_stack() or torch._C._len_torch_dispatch_stack():
        return False
    return all(torch.autograd.forward_ad.unpack_dual(t).tangent is None for t in (x, weight))


def _pays(T, V, d):
    """The node costs about 100 us more host time than the plain operators (forward and backward, measured with the
    GPU idle), so small losses stay with those.  4096 x 8192 logits, d = 512: 436 us plain, 269 here; 1024 x 16384:
    252 against 301.  Unaligned rows cost the plain products so much that these change over earlier: 1024 x 8191,
    d = 512: 365 against 272; d = 128: 239 against 268."""
    return T * V >= 32_000_000 or (V % 8 != 0 and T * V * d >= 4_000_000_000)


def lm_head_cross_entropy(x, weight, targets):
    """Mean cross-entropy of ``F.linear(x, weight)`` (logits rounded to x's type, loss in fp32) against class indices
    ``targets`` (``-100``: ignored).  ``x [..., d]``, ``weight [V, d]``, ``targets [...]``; differentiable in both."""
    if _pays(targets.numel(), *weight.shape) and _native(x, weight, targets):
        return _LmHeadCrossEntropy.apply(x, weight, targets)
    return _reference(x, weight, targets)
