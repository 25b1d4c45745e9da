"""The eager C++ route against the torch.library route (what a traced graph runs) over the forms that both accept:
broadcast prefixes, operand types, storage orders, offsets and paddings, subsets of gradients."""
import random

import pytest
import torch

import openfold3_triangle_kernel_b200 as tk
from openfold3_triangle_kernel_b200 import _cabi
from openfold3_triangle_kernel_b200.synthetic import trimul_weights

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


class _NoEagerRoute:
    """`_native` without its eager entry points: every call declines and goes through torch.library."""

    def __init__(self, module):
        self._module = module

    def __getattr__(self, name):
        if name in ("attention", "trimul", "pair_block"):
            return lambda *a, **k: None
        return getattr(self._module, name)


def _stored(t, rng, offsets=True):
    """`t`'s values in another storage: permuted, padded rows, strided outer dimension, odd offset, expanded."""
    kind = rng.choice(("plain", "permuted", "padded", "outer", "expanded") + (("offset",) if offsets else ()))
    if kind == "offset":
        flat = torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)
        flat[1:].copy_(t.reshape(-1))
        return flat[1:].view(t.shape)
    if kind == "permuted":
        order = list(range(t.ndim))
        rng.shuffle(order)
        return t.permute(order).contiguous().permute([order.index(i) for i in range(t.ndim)])
    if kind == "padded":
        wide = torch.zeros(*t.shape[:-1], t.shape[-1] + 8, device="cuda", dtype=t.dtype)
        wide[..., :t.shape[-1]] = t
        return wide[..., :t.shape[-1]]
    if kind == "outer" and t.ndim > 1:
        both = torch.stack([t, t], 1)
        return both[:, 1]
    if kind == "expanded" and t.ndim > 2:
        return t.narrow(0, 0, 1).expand(t.shape)
    return t.clone()


def _both(monkeypatch, call):
    eager = call()
    with monkeypatch.context() as m:
        traced = _NoEagerRoute(_cabi.native())
        m.setattr(_cabi, "native", lambda: traced)
        return eager, call()


def _check(results, tol):
    for i, (a, b) in enumerate(zip(*results)):
        assert a.shape == b.shape and a.dtype == b.dtype, i
        assert torch.equal(torch.isfinite(a), torch.isfinite(b)), i
        a, b = (torch.where(torch.isfinite(x), x, 0).double() for x in (a, b))
        assert (a - b).norm() <= tol * b.norm() + 1e-12, (i, float((a - b).norm() / b.norm()))


@pytest.mark.parametrize("seed", range(24))
def test_attention_routes_agree(seed, monkeypatch):
    rng, gen = random.Random(seed), torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()  # noqa: E731
    prefix = rng.choice(((1,), (2,), (2, 3), (1, 2, 1)))
    O, H, N, D = rng.choice((1, 2, 5)), rng.choice((1, 3, 4)), rng.choice((1, 16, 31, 70)), rng.choice((1, 16, 20, 32, 48, 64))
    part = lambda: rng.choice((prefix, prefix[-1:], tuple(rng.choice((1, p)) for p in prefix), ()))  # noqa: E731
    q, k, v = (_stored(rn(*prefix, O, H, N, D), rng, offsets=False) for _ in range(3))  # (both routes refuse an offset)
    bias = _stored(rn(*part(), 1, H, N, N).to(rng.choice((torch.bfloat16, torch.float32))), rng)
    mask = None
    if rng.random() < 0.7:
        dt = rng.choice((torch.float32, torch.bfloat16, torch.float16))
        drop = rng.choice((-float("inf"), torch.finfo(dt).min))
        keep = torch.rand(*part(), O, 1, 1, N, device="cuda", generator=gen) < 0.8
        mask = _stored(torch.where(keep, 0.0, drop).to(dt), rng)
    grad = [rng.random() < 0.6 for _ in range(4)]
    d_out = _stored(rn(*prefix, O, N, H, D), rng, offsets=False)

    def call():
        x = [t.detach().requires_grad_(r) for t, r in zip((q, k, v, bias), grad)]
        out, lse = tk.turbo_attention(*x[:3], pair_bias=x[3], res_mask=mask, return_lse=True)
        wanted = [t for t, r in zip(x, grad) if r]
        return [out, lse, *(torch.autograd.grad(out, wanted, d_out) if wanted else ())]

    # the kernels are the same; a broadcast bias sums its gradient in fp32 on one route and in bf16 (2^-9 a step, over at
    # most six batch entries) on the other
    _check(_both(monkeypatch, call), 6 * 2.0 ** -9)


@pytest.mark.parametrize("seed", range(16))
def test_trimul_routes_agree(seed, monkeypatch):
    rng, gen = random.Random(seed), torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()  # noqa: E731
    prefix = rng.choice(((1,), (2,), (2, 2)))
    N, C = rng.choice((1, 7, 8, 24, 33)), rng.choice((32, 64, 96, 128))
    z, d_out = _stored(rn(*prefix, N, N, C), rng), _stored(rn(*prefix, N, N, C), rng)
    dt = rng.choice((torch.float32, torch.bfloat16, torch.float64))
    w = {n: t.cuda().to(dt) for n, t in trimul_weights(C, seed).items()}
    w = {n: _stored(t, rng) if t.ndim == 1 else t.t().contiguous().t() for n, t in w.items()}
    mask = None
    if rng.random() < 0.7:
        keep = torch.rand(*rng.choice((prefix, (1,), ())), N, N, device="cuda", generator=gen) < 0.8
        mask = _stored(keep.to(rng.choice((torch.bool, torch.float32, torch.bfloat16, torch.float16))), rng)
    grad = {n: rng.random() < 0.5 for n in ("z", *w)}
    direction = rng.choice(("outgoing", "incoming"))

    def call():
        x = {n: t.detach().requires_grad_(grad[n]) for n, t in (("z", z), *w.items())}
        out = tk.turbo_trimul(x["z"], direction, mask, **{n: x[n] for n in w})
        wanted = [t for n, t in x.items() if grad[n]]
        return [out, *(torch.autograd.grad(out, wanted, d_out) if wanted else ())]

    # the same products and sums, row padding aside: fp32 sums in another order behind one bf16 rounding
    _check(_both(monkeypatch, call), 2.0 ** -9)
