"""Output projection and cross-entropy as one node against plain PyTorch in 64 bits.

Operands are small multiples of 1/8 and d <= 128, so the logits are exact in bf16 (at most 256 steps of 1/8) and
both sides see the same ones.  The oracle rounds the logits' gradient to bf16 where the node does, so what is left
is fp32 arithmetic in the loss (1e-5) and the rounding of a gradient to bf16: at most 2^-8 of each element, and
so of the 2-norm (logits' gradients that fp32 pushes over a rounding boundary are one in some thousands)."""
import pytest
import torch
import torch.nn.functional as F

from mini_nccl_b200.ops.lm_loss import _LmHeadCrossEntropy, _native, _pays, _reference, lm_head_cross_entropy

GRAD_REL = 2.0 ** -8
node = _LmHeadCrossEntropy.apply   # whatever the size


def _case(shape, V, d, seed=0, device="cuda", ignored=0.0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randint(-2, 3, (*shape, d), generator=g).to(torch.bfloat16) * 0.5
    w = torch.randint(-1, 2, (V, d), generator=g).to(torch.bfloat16) * 0.25
    t = torch.randint(0, V, shape, generator=g)
    t[torch.rand(shape, generator=g) < ignored] = -100
    return x.to(device).requires_grad_(), w.to(device).requires_grad_(), t.to(device)


def _exact(x, w, t, scale=1.0):
    x, w, t = x.detach().double().cpu(), w.detach().double().cpu(), t.reshape(-1).cpu()
    logits = (x.view(-1, x.shape[-1]) @ w.t()).requires_grad_()
    loss = F.cross_entropy(logits, t)
    d = torch.autograd.grad(loss, logits, torch.tensor(scale, dtype=torch.float64))[0].to(torch.bfloat16).double()
    return loss.detach(), (d @ w).view(x.shape), d.t() @ x.view(-1, x.shape[-1])


def _rel(got, want):
    return float((got.double().cpu() - want).norm() / want.norm().clamp_min(1e-30))


def _close(loss, dx, dw, want):
    assert abs(float(loss) - float(want[0])) <= 1e-5 * max(1.0, abs(float(want[0])))
    # the activations' gradient over a number of classes that is no multiple of eight is the library's product, which
    # may round the partial sums of its slices and their running total as well as the result
    assert _rel(dx, want[1]) <= GRAD_REL * (1 if dw.shape[0] % 8 == 0 else 3) and _rel(dw, want[2]) <= GRAD_REL


def test_cpu_takes_the_plain_operators():
    x, w, t = _case((3, 5), 33, 16, device="cpu")
    assert not _native(x, w, t)
    assert torch.equal(lm_head_cross_entropy(x, w, t), _reference(x, w, t))
    assert _pays(8192, 50257, 1024) and _pays(1024, 8191, 512) and not _pays(1024, 8191, 128) and not _pays(1024, 16384, 1024)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,V,d", [((1,), 8, 8), ((2, 3), 9, 8), ((64,), 64, 64), ((65,), 63, 72), ((5, 13), 65, 16),
                                       ((3, 43), 2047, 128), ((4, 64), 2049, 128), ((300,), 8200, 64), ((2, 333), 50257, 128),
                                       ((1024,), 512, 128)])
@pytest.mark.parametrize("ignored", [0.0, 0.3])
def test_loss_and_gradients(shape, V, d, ignored):
    x, w, t = _case(shape, V, d, seed=V + d, ignored=ignored)
    if bool((t == -100).all()):
        t.view(-1)[0] = 0
    assert _native(x, w, t)
    loss = node(x, w, t)
    assert loss.dtype == torch.float32 and loss.dim() == 0
    (loss * 3.0).backward()
    _close(loss.detach(), x.grad, w.grad, _exact(x, w, t, 3.0))


@pytest.mark.gpu
def test_what_autograd_may_do_with_the_node():
    x, w, t = _case((3, 43), 1003, 64, seed=5, ignored=0.1)
    want = _exact(x, w, t)
    loss = node(x, w, t)
    first = torch.autograd.grad(loss, [x, w], retain_graph=True)
    second = torch.autograd.grad(loss, [x, w])
    assert all(torch.equal(a, b) for a, b in zip(first, second))
    _close(loss.detach(), *first, want)

    with torch.autograd.graph.saved_tensors_hooks(lambda s: s.cpu(), lambda s: s.cuda()):   # loses views and strides
        loss = node(x, w, t)
    assert all(torch.equal(a, b) for a, b in zip(first, torch.autograd.grad(loss, [x, w])))

    for one in (x, w):   # the other one is frozen
        ins = [s if s is one else s.detach() for s in (x, w)]
        got, = torch.autograd.grad(node(*ins, t), [one])
        assert torch.equal(got, first[0 if one is x else 1])

    strided = x.detach().transpose(0, 1).contiguous().transpose(0, 1).requires_grad_()
    assert torch.equal(torch.autograd.grad(node(strided, w, t), [strided])[0], first[0])

    def second_order(f):
        gx, = torch.autograd.grad(f(x, w, t), [x], create_graph=True)
        return torch.autograd.grad((gx.float() ** 2).sum() * 1e4, [x, w])

    # one path, the plain operators', from the roundings of the first gradient on: those differ by 2^-8 at most
    for got, ref in zip(second_order(node), second_order(_reference)):
        assert _rel(got, ref.double().cpu()) <= 2 * GRAD_REL


@pytest.mark.gpu
def test_rows_that_all_count_for_nothing_and_values_that_are_not_finite():
    x, w, t = _case((70,), 129, 16, seed=3)
    nothing = torch.full_like(t, -100)
    for f in (node, _reference):
        loss = f(x, w, nothing)
        assert torch.isnan(loss) and not any(g.any() for g in torch.autograd.grad(loss, [x, w]))
    for bad in (float("nan"), float("inf"), -float("inf")):
        xb = x.detach().clone()
        xb[7, 3] = bad
        xb.requires_grad_()
        got, ref = (torch.autograd.grad(f(xb, w, t), [xb])[0] for f in (node, _reference))
        assert torch.equal(torch.isnan(got), torch.isnan(ref))


@pytest.mark.gpu
def test_calls_that_stay_with_the_plain_operators():
    x, w, t = _case((4, 16), 640, 64)
    assert _native(x, w, t)
    assert not _native(x.float(), w.float(), t) and not _native(x.half(), w.half(), t) and not _native(x, w, t.reshape(-1))
    assert not _native(x[..., :60], w[:, :60], t) and not _native(x, w, torch.zeros(4, 16, dtype=torch.uint8, device="cuda"))
    with torch.autocast("cuda", dtype=torch.float16):
        assert not _native(x, w, t)
    with torch.autograd.forward_ad.dual_level():
        assert not _native(torch.autograd.forward_ad.make_dual(x.detach(), torch.ones_like(x)), w, t)
    seen = []
    torch.func.vmap(lambda s: (seen.append(_native(s, w, t[0])), s)[1])(x.detach())
    assert seen == [False]


@pytest.mark.gpu
def test_targets_that_cannot_be_viewed_as_one_row_are_refused_by_both():
    x, w, t = _case((4, 16), 640, 64)
    apart = torch.cat((t, t), dim=1)[:, :16]
    for f in (node, _reference):
        with pytest.raises(RuntimeError, match="view"):
            f(x, w, apart)
    every_other = torch.stack((t, t), dim=-1)[..., 0]            # strided, but one row all the same
    assert torch.equal(node(x, w, every_other), node(x, w, t))
