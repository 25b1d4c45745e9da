"""The eager C++ route of the operators: ragged lengths without padded copies, operand types and strides, and calls
without gradients (which keep no intermediates) equal to calls with them."""
import pytest
import torch

import openfold3_triangle_kernel_b200 as tk
from oracle import attention_oracle as ao
from oracle import trimul_oracle as to
from oracle.inputs import attention_inputs, trimul_inputs

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("direction", ["outgoing", "incoming"])
@pytest.mark.parametrize("N", [1, 7, 8, 9, 63, 65, 130])
def test_trimul_any_length(N, direction):
    t = trimul_inputs(2, N, 64, seed=N, mask_mode="trailing10")
    d_out = torch.randn(2, N, N, 64, generator=torch.Generator().manual_seed(N)).bfloat16()
    z = t["z"].cuda().requires_grad_(True)
    w = {k: v.cuda().requires_grad_(True) for k, v in t["weights"].items()}
    for mask in (t["mask"].cuda(), t["mask"].cuda().bool(), t["mask"].cuda().half().transpose(1, 2).contiguous().transpose(1, 2)):
        out = tk.turbo_trimul(z, direction, mask, **w)
        with torch.no_grad():
            assert torch.equal(tk.turbo_trimul(z, direction, mask, **w), out)
    out.backward(d_out.cuda())
    ref = to.trimul_forward_backward(t["z"], direction, t["mask"], t["weights"], d_out)
    assert ao.rel_l2(out.detach().cpu(), ref["out"]) <= 1e-2
    assert ao.rel_l2(z.grad.cpu(), ref["dz"]) <= 2e-2
    for k in ("p_in_weight", "g_out_weight", "norm_in_bias", "norm_out_weight"):
        assert ao.rel_l2(w[k].grad.cpu(), ref["d_" + k]) <= 2.5e-2, k


@pytest.mark.parametrize("N", [1, 24, 37])
def test_absent_mask_equals_a_mask_that_keeps_everything(N):
    a = attention_inputs(2, 3, 2, N, 32, seed=N, mask_mode="none")
    t = trimul_inputs(1, N, 32, seed=N, mask_mode="none")
    d_att = torch.randn(2, 3, N, 2, 32, generator=torch.Generator().manual_seed(N)).bfloat16().cuda()
    d_tri = torch.randn(1, N, N, 32, generator=torch.Generator().manual_seed(N)).bfloat16().cuda()

    def attention(mask):
        x = [a[n].cuda().requires_grad_(True) for n in ("q", "k", "v", "pair_bias")]
        out = tk.turbo_attention(*x[:3], pair_bias=x[3], res_mask=mask)
        with torch.no_grad():
            assert torch.equal(tk.turbo_attention(*x[:3], pair_bias=x[3], res_mask=mask), out)
        return [out, *torch.autograd.grad(out, x, d_att)]

    def trimul(mask):
        z = t["z"].cuda().requires_grad_(True)
        w = {k: v.cuda().requires_grad_(True) for k, v in t["weights"].items()}
        out = tk.turbo_trimul(z, "outgoing", mask, **w)
        with torch.no_grad():
            assert torch.equal(tk.turbo_trimul(z, "outgoing", mask, **w), out)
        return [out, *torch.autograd.grad(out, [z, *w.values()], d_tri)]

    for fn, keep in ((attention, torch.zeros(2, 3, 1, 1, N, device="cuda")), (trimul, torch.ones(1, N, N, device="cuda"))):
        for got, want in zip(fn(None), fn(keep)):
            assert torch.equal(got, want)


# every subset of the four inputs that can ask for a gradient: the kernels of the others are left out
@pytest.mark.parametrize("wanted", range(1, 16))
def test_attention_gradient_subsets(wanted):
    a = attention_inputs(1, 5, 2, 40, 32, seed=8)
    d_out = torch.randn(1, 5, 40, 2, 32, generator=torch.Generator().manual_seed(8)).bfloat16().cuda()

    def grads(mask):
        x = [a[n].cuda().requires_grad_(bool(mask >> i & 1)) for i, n in enumerate(("q", "k", "v", "pair_bias"))]
        out = tk.turbo_attention(*x[:3], pair_bias=x[3], res_mask=a["res_mask"].cuda())
        out.backward(d_out)
        return [t.grad for t in x]

    for i, (got, full) in enumerate(zip(grads(wanted), grads(15))):
        assert (got is not None) == bool(wanted >> i & 1)
        assert got is None or torch.equal(got, full)


def _entry_points():
    """name -> (call, differentiable inputs) of the three entry points at a small size"""
    from openfold3_triangle_kernel_b200.pair_block import pair_stack_block
    from oracle.pair_block_oracle import block_params
    a = attention_inputs(1, 9, 2, 24, 32, seed=1)
    x = [a[n].cuda().requires_grad_(True) for n in ("q", "k", "v", "pair_bias")]
    t = trimul_inputs(1, 24, 64, seed=2)
    z = t["z"].cuda().requires_grad_(True)
    w = {k: v.cuda().requires_grad_(True) for k, v in t["weights"].items()}
    blk = {k: {n: v.cuda().requires_grad_(True) for n, v in m.items()} for k, m in block_params(64, 4, 16, seed=3).items()}
    mask = t["mask"].cuda()
    return {"attention": (lambda: tk.turbo_attention(*x[:3], pair_bias=x[3], res_mask=a["res_mask"].cuda()), x),
            "trimul": (lambda: tk.turbo_trimul(z, "incoming", mask, **w), [z, *w.values()]),
            "block": (lambda: pair_stack_block(z, mask, blk, 4), [z, *(v for m in blk.values() for v in m.values())])}


@pytest.mark.parametrize("name", ["attention", "trimul", "block"])
def test_second_derivative_is_refused(name):
    call, leaves = _entry_points()[name]
    want = torch.autograd.grad(call().float().square().sum(), leaves)
    out = call()
    got = torch.autograd.grad(out.float().square().sum(), leaves, create_graph=True)   # allowed: first derivatives
    for g, r in zip(got, want):
        assert torch.equal(g, r)
    for g in got:   # a penalty on any of them, alone or next to a term that has a derivative
        with pytest.raises(RuntimeError, match="no second derivative"):
            torch.autograd.grad(out.float().sum() + g.float().square().sum(), leaves[:1], retain_graph=True)
        with pytest.raises(RuntimeError, match="no second derivative"):
            g.float().square().sum().backward(retain_graph=True)
    # the incoming gradient is an input of the backward as well
    d_out = torch.ones_like(out).requires_grad_(True)
    g, = torch.autograd.grad(call(), leaves[:1], d_out, create_graph=True)
    with pytest.raises(RuntimeError, match="no second derivative"):
        torch.autograd.grad(g.float().sum(), d_out)


class _Tagged(torch.Tensor):
    """A subclass that sees what is called on it (default behaviour: results are of the subclass, too)."""
    calls = []

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        cls.calls.append(str(func))
        return super().__torch_function__(func, types, args, kwargs or {})


@pytest.mark.parametrize("which", range(9))
def test_tensor_subclasses_take_the_route_they_can_see(which):
    from openfold3_triangle_kernel_b200.pair_block import pair_stack_block
    from oracle.pair_block_oracle import block_params
    a = attention_inputs(1, 4, 2, 16, 32, seed=4)
    t = trimul_inputs(1, 16, 64, seed=4)
    blk = {k: {n: v.cuda() for n, v in m.items()} for k, m in block_params(64, 4, 16, seed=4).items()}
    x = [a[n].cuda() for n in ("q", "pair_bias", "res_mask")] + [t["z"].cuda(), t["mask"].cuda(),
         t["weights"]["g_out_weight"].cuda(), t["z"].cuda(), t["mask"].cuda(), blk["tri_att_end"]["w_q"]]
    plain = list(x)
    x[which] = x[which].as_subclass(_Tagged)

    def call(x):
        if which < 3:
            return tk.turbo_attention(x[0], a["k"].cuda(), a["v"].cuda(), pair_bias=x[1], res_mask=x[2])
        if which < 6:
            w = {n: v.cuda() for n, v in t["weights"].items()}
            return tk.turbo_trimul(x[3], "outgoing", x[4], **{**w, "g_out_weight": x[5]})
        return pair_stack_block(x[6], x[7], {**blk, "tri_att_end": {**blk["tri_att_end"], "w_q": x[8]}}, 4)

    _Tagged.calls.clear()
    out = call(x)
    assert type(out) is _Tagged and any("tpf_b200" in c for c in _Tagged.calls)
    # (the block's subclass route is the composition of the operators, which rounds between its steps)
    assert ao.rel_l2(out.as_subclass(torch.Tensor).cpu(), call(plain).cpu()) <= (1e-2 if which >= 6 else 0)
    # parameters are tensors as far as the operators are concerned
    assert type(call([torch.nn.Parameter(v) if v.is_floating_point() and i not in (2, 4, 7) else v
                      for i, v in enumerate(plain)])) is torch.Tensor


class _Named(torch.nn.Parameter):
    """A parameter class that carries something of its own and overrides nothing."""


class _Watched(torch.nn.Parameter):
    calls = []

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        cls.calls.append(str(func))
        with torch._C.DisableTorchFunctionSubclass():
            return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("cls,native", [(torch.nn.Parameter, True), (_Named, True), (_Watched, False)])
def test_parameter_classes_take_the_native_route_unless_they_watch(cls, native):
    from openfold3_triangle_kernel_b200 import _cabi
    from oracle.pair_block_oracle import block_params
    own = lambda t: cls(t.cuda())  # noqa: E731
    lib = _cabi.native()
    a = attention_inputs(1, 4, 2, 16, 32, seed=4)
    t = trimul_inputs(1, 16, 64, seed=4)
    order = ("p_in_weight", "g_in_weight", "p_out_weight", "g_out_weight", "norm_in_weight", "norm_in_bias",
             "norm_out_weight", "norm_out_bias")
    weights = tuple(own(t["weights"][n]) for n in order)
    z, mask = t["z"].cuda(), t["mask"].cuda()
    blk = block_params(64, 4, 16, seed=4)
    parts = [tuple(own(blk[m][n]) for n in order) for m in ("tri_mul_out", "tri_mul_in")]
    parts += [tuple(own(blk[m][n]) for n in ("ln_w", "ln_b", "w_z", "w_q", "w_k", "w_v", "w_g", "w_o"))
              for m in ("tri_att_start", "tri_att_end")]
    for out in (lib.attention(a["q"].cuda(), a["k"].cuda(), a["v"].cuda(), own(a["pair_bias"]), a["res_mask"].cuda(), False),
                lib.trimul(z, False, mask, weights), lib.pair_block(z, mask, *parts, 4)):
        assert (out is not None) == native
    got = tk.turbo_trimul(z, "outgoing", mask, **dict(zip(order, weights)))
    assert torch.equal(got, tk.turbo_trimul(z, "outgoing", mask, **{n: w.detach().as_subclass(torch.Tensor)
                                                                    for n, w in zip(order, weights)}))


def _shifted(t):
    """The same values one element behind a 16-byte boundary, as a parameter inside a flat buffer has them."""
    flat = torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)
    flat[1:].copy_(t.reshape(-1))
    return flat[1:].view(t.shape)


@pytest.mark.parametrize("N,C", [(16, 32), (17, 64), (24, 96), (33, 128)])
def test_tensors_that_start_between_16_byte_boundaries(N, C):
    from openfold3_triangle_kernel_b200.pair_block import pair_stack_block
    from oracle.pair_block_oracle import block_params
    t = trimul_inputs(1, N, C, seed=N)
    blk = block_params(C, 2, 16, seed=N)
    d_out = torch.randn(1, N, N, C, generator=torch.Generator().manual_seed(N)).bfloat16()

    def run(place):
        z = place(t["z"].cuda()).requires_grad_(True)
        mask = place(t["mask"].cuda())
        w = {k: place(v.cuda()).requires_grad_(True) for k, v in t["weights"].items()}
        b = {k: {n: place(v.cuda()).requires_grad_(True) for n, v in m.items()} for k, m in blk.items()}
        out = tk.turbo_trimul(z, "outgoing", mask, **w)
        res = [out, *torch.autograd.grad(out, [z, *w.values()], place(d_out.cuda()))]
        out = pair_stack_block(z, mask, b, 2)
        res += [out, *torch.autograd.grad(out, [z, *(v for m in b.values() for v in m.values())], place(d_out.cuda()))]
        # the operators behind a traced graph
        pad = (-N) % 8
        zp = place(torch.nn.functional.pad(t["z"].cuda(), (0, 0, 0, pad, 0, pad))).requires_grad_(True)
        mp = place(torch.nn.functional.pad(t["mask"].cuda(), (0, pad, 0, pad)))
        order = ("p_in_weight", "g_in_weight", "p_out_weight", "g_out_weight", "norm_in_weight", "norm_in_bias",
                 "norm_out_weight", "norm_out_bias")
        op = torch.ops.tpf_b200.trimul_fwd(zp, mp, *(w[n] for n in order), False)[0]
        res += [op, *torch.autograd.grad(op.float().square().sum(), [zp, *w.values()])]
        return res

    for got, want in zip(run(_shifted), run(lambda x: x.clone())):
        assert torch.equal(got, want)


# Enough rows for the projections that keep all weights in shared memory (113 row tiles and more), with a ragged last
# row tile; 145 tiles at N = 136, one round of 148 row tiles and a second one at N = 184.
@pytest.mark.parametrize("N,C", [(119, 128), (136, 32), (136, 64), (120, 96), (184, 128)])
def test_trimul_resident_weights(N, C):
    t = trimul_inputs(1, N, C, seed=N, mask_mode="trailing10")
    d_out = torch.randn(1, N, N, C, generator=torch.Generator().manual_seed(N)).bfloat16()
    z = t["z"].cuda().requires_grad_(True)
    w = {k: v.cuda().requires_grad_(True) for k, v in t["weights"].items()}
    out = tk.turbo_trimul(z, "outgoing", t["mask"].cuda(), **w)
    out.backward(d_out.cuda())
    ref = to.trimul_forward_backward(t["z"], "outgoing", t["mask"], t["weights"], d_out)
    assert ao.rel_l2(out.detach().cpu(), ref["out"]) <= 1e-2
    assert ao.rel_l2(z.grad.cpu(), ref["dz"]) <= 2e-2
    for k in ("p_in_weight", "g_in_weight", "g_out_weight", "norm_in_bias"):
        assert ao.rel_l2(w[k].grad.cpu(), ref["d_" + k]) <= 2.5e-2, k


@pytest.mark.parametrize("N,D,bias_type,mask_type", [(3, 16, torch.float32, torch.float16), (37, 32, torch.bfloat16, torch.bfloat16),
                                                     (66, 40, torch.float32, torch.float32), (64, 64, torch.bfloat16, torch.float32)])
def test_attention_operand_types_and_strides(N, D, bias_type, mask_type):
    a = attention_inputs(2, N, 2, N, D, seed=N, mask_mode="trailing15")
    q, k, v = (a[n].cuda().requires_grad_(True) for n in ("q", "k", "v"))
    base = a["pair_bias"].to(bias_type).cuda().permute(0, 1, 3, 4, 2).contiguous().requires_grad_(True)  # [B,1,N,N,H]
    bias = base.permute(0, 1, 4, 2, 3)
    mask = a["res_mask"].to(mask_type).cuda()
    d_out = torch.randn(2, N, N, 2, D, generator=torch.Generator().manual_seed(N)).bfloat16()
    out = tk.turbo_attention(q, k, v, pair_bias=bias, res_mask=mask)
    with torch.no_grad():
        assert torch.equal(tk.turbo_attention(q, k, v, pair_bias=bias, res_mask=mask), out)
    out.backward(d_out.cuda())
    ref = ao.attention_forward_backward(a["q"], a["k"], a["v"], a["pair_bias"], a["res_mask"], d_out)
    for name, got in (("out", out), ("dq", q.grad), ("dk", k.grad), ("dv", v.grad),
                      ("dbias", base.grad.permute(0, 1, 4, 2, 3))):
        assert ao.rel_l2(got.detach().cpu(), ref[name]) <= 1e-2, name
    # gradients that nobody asked for are not computed; the ones that are do not change
    q2 = a["q"].cuda().requires_grad_(True)
    tk.turbo_attention(q2, k.detach(), v.detach(), pair_bias=bias.detach(), res_mask=mask).backward(d_out.cuda())
    assert torch.equal(q2.grad, q.grad)


# Ragged ends of the gradient tiles (32-row blocks, 128-row tiles, strips of 384 keys), and more planes per CTA than the
# backward kernel keeps records of, or than the forward kernel has buffers for (900 and 1800 one-tile planes).
@pytest.mark.parametrize("O,N,D", [(2, 31, 32), (2, 33, 16), (3, 96, 32), (2, 129, 64), (2, 385, 16), (2, 416, 32), (450, 20, 32),
                                   (900, 50, 16)])
def test_attention_gradient_tiles(O, N, D):
    a = attention_inputs(1, O, 2, N, D, seed=N, mask_mode="trailing15")
    q, k, v, bias = (a[n].cuda().requires_grad_(True) for n in ("q", "k", "v", "pair_bias"))
    d_out = torch.randn(1, O, N, 2, D, generator=torch.Generator().manual_seed(N)).bfloat16()
    tk.turbo_attention(q, k, v, pair_bias=bias, res_mask=a["res_mask"].cuda()).backward(d_out.cuda())
    ref = ao.attention_forward_backward(a["q"], a["k"], a["v"], a["pair_bias"], a["res_mask"], d_out)
    for name, got in (("dq", q.grad), ("dk", k.grad), ("dv", v.grad), ("dbias", bias.grad)):
        assert ao.rel_l2(got.cpu(), ref[name]) <= 1e-2, name


@pytest.mark.parametrize("N,C,H,D", [(1, 64, 4, 16), (9, 128, 4, 32), (65, 32, 2, 16), (130, 96, 3, 32), (40, 64, 8, 16),
                                     (119, 128, 4, 32)])
def test_pair_block_any_length(N, C, H, D):
    from openfold3_triangle_kernel_b200.pair_block import pair_stack_block
    from oracle.pair_block_oracle import block_params, pair_block_forward
    g = torch.Generator().manual_seed(N)
    z = torch.randn(2, N, N, C, generator=g).bfloat16()
    mask = torch.ones(2, N, N)
    if N > 4:
        mask[0, N - 3:] = 0
        mask[0, :, N - 3:] = 0
    d_out = torch.randn(2, N, N, C, generator=g).bfloat16() * mask.unsqueeze(-1).bfloat16()
    params = block_params(C, H, D, seed=N)
    zr = z.double().requires_grad_(True)
    pr = {k: {n: t.double().requires_grad_(True) for n, t in v.items()} for k, v in params.items()}
    ref = pair_block_forward(zr, mask, pr, H, dtype=torch.float64)
    ref.backward(d_out.double())
    pd = {k: {n: t.cuda().requires_grad_(True) for n, t in v.items()} for k, v in params.items()}
    zz = z.cuda().requires_grad_(True)
    out = pair_stack_block(zz, mask.cuda(), pd, H)
    with torch.no_grad():
        assert torch.equal(pair_stack_block(zz, mask.cuda().bool(), pd, H), out)
    out.backward(d_out.cuda())
    valid = mask.bool().unsqueeze(-1)
    pick = lambda t: torch.where(valid, t.detach().cpu().double(), 0.0)  # noqa: E731
    assert ao.rel_l2(pick(out), pick(ref)) <= 1e-2
    assert ao.rel_l2(pick(zz.grad), pick(zr.grad)) <= 2e-2
    for k, v in pd.items():
        for n, t in v.items():
            want = pr[k][n].grad
            if want.norm() > 1e-6 * N:   # N = 1: a softmax over one key has no gradient in q, k and the bias
                assert ao.rel_l2(t.grad.cpu(), want) <= 4e-2, (k, n)


# D = 16 is the fused block, D = 64 its composition of the operators
@pytest.mark.parametrize("D", [16, 64])
def test_pair_block_counts_its_attention_calls(D):
    from openfold3_triangle_kernel_b200.attention import invocation_count
    from openfold3_triangle_kernel_b200.pair_block import pair_stack_block
    from oracle.pair_block_oracle import block_params
    z = torch.zeros(1, 16, 16, 64, device="cuda", dtype=torch.bfloat16)
    params = {k: {n: t.cuda() for n, t in v.items()} for k, v in block_params(64, 2, D, seed=1).items()}
    before = invocation_count()
    pair_stack_block(z, torch.ones(1, 16, 16, device="cuda"), params, 2)
    assert invocation_count() == before + 2


# Gates of the attention modules that are nearly closed (logits -10 .. -16): the gate's own value counts, since the output
# projection scales it back up.  One LayerNorm channel is constant and alone carries the gate logits, which bf16 holds
# exactly.  A gate that is off by a factor scales the gradients that belong to its column of w_o and its rows of w_v and
# w_g by that factor; what the bf16 intermediates leave of that measure (about 1 % here, open gates included) bounds it.
@pytest.mark.parametrize("N,C,H,D", [(40, 64, 4, 16), (33, 128, 4, 32)])
def test_pair_block_closed_gates(N, C, H, D):
    from openfold3_triangle_kernel_b200.pair_block import pair_stack_block
    from oracle.pair_block_oracle import block_params, pair_block_forward
    g = torch.Generator().manual_seed(N)
    z = torch.randn(1, N, N, C, generator=g).bfloat16()
    mask = torch.ones(1, N, N)
    params = block_params(C, H, D, seed=N)
    logits = (-10.0 - 6.0 * torch.rand(H * D, generator=g)).bfloat16().float()
    nodes = ("tri_att_start", "tri_att_end")
    for k in nodes:
        p = params[k]
        p["ln_w"][0], p["ln_b"][0] = 0.0, 1.0
        p["w_g"].zero_()
        p["w_g"][:, 0] = logits
        p["w_o"].mul_(10 * torch.exp(-logits))
    d_out = torch.randn(1, N, N, C, generator=g).bfloat16()
    pr = {k: {n: t.double().requires_grad_(k in nodes) for n, t in v.items()} for k, v in params.items()}
    pair_block_forward(z.double(), mask, pr, H, dtype=torch.float64).backward(d_out.double())
    pd = {k: {n: t.cuda().requires_grad_(k in nodes) for n, t in v.items()} for k, v in params.items()}
    pair_stack_block(z.cuda(), mask.cuda(), pd, H).backward(d_out.cuda())
    for k in nodes:
        for n in ("w_o", "w_v", "w_g"):
            got, want = pd[k][n].grad.cpu().double(), pr[k][n].grad
            if n == "w_o":
                got, want = got.T, want.T
            factor = (got * want).sum(1) / (want * want).sum(1)
            assert (factor - 1).abs().max() <= 2.5e-2, (k, n, float((factor - 1).abs().max()))
