"""The forward of TriMul with its norms inside the projection and output kernels (C = 64 and 128), at the edges of its
128-row tiles, 64-row copies and padded lines: against the fp64 oracle, and the forward that keeps nothing against the one
with a backward behind it.

Tolerance: eight roundings to bf16 lie between the inputs and a result (four weights, a, b, x, the result), independent and
2^-9 in the root mean square (2^-8 at most): 2^-9 sqrt(8) = 5.5e-3.
"""
import pytest
import torch

import openfold3_triangle_kernel_b200 as tk
from openfold3_triangle_kernel_b200 import _cabi as C
from oracle import trimul_oracle as to
from oracle.attention_oracle import rel_l2
from oracle.inputs import trimul_inputs

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]


@pytest.mark.parametrize("B,N,channels,direction,mask,shift", [
    (1, 1, 128, "outgoing", "pair", 0.0),      # one row of 64, most of it padding
    (1, 8, 64, "incoming", "pair", 0.0),       # half a tile
    (3, 8, 128, "outgoing", "half", 0.0),      # a tile that spans batch entries
    (2, 20, 64, "outgoing", "pair", 0.0),      # padded lines shorter than a 64-row copy
    (3, 33, 128, "incoming", "bool", 0.0),
    (1, 64, 128, "outgoing", "none", 0.0),     # the caller's rows as they are
    (2, 72, 64, "incoming", "pair", 0.0),
    (1, 131, 128, "outgoing", "pair", 0.0),    # 64-row copies and lines that end inside one
    (2, 259, 64, "outgoing", "pair", 0.0),     # seven or eight tiles a CTA
    (1, 40, 128, "incoming", "pair", 40.0),    # rows whose mean is forty times their spread
])
def test_forward_at_tile_edges(B, N, channels, direction, mask, shift):
    t = trimul_inputs(B, N, channels, seed=N)
    z = (t["z"].float() + shift).bfloat16()
    g = torch.Generator().manual_seed(N)
    w = {n: x + 0.2 * torch.randn(x.shape, generator=g) if x.ndim == 1 else x for n, x in t["weights"].items()}
    m = t["mask"]
    m = {"pair": m, "half": (m * 0.75).half(), "bool": m.bool(), "none": None}[mask]
    dm = None if m is None else m.cuda()
    with torch.no_grad():
        got = tk.turbo_trimul(z.cuda(), direction, dm, **{n: x.cuda() for n, x in w.items()})
    kept = tk.turbo_trimul(z.cuda(), direction, dm, **{n: x.cuda().requires_grad_(True) for n, x in w.items()}).detach()
    torch.cuda.synchronize()
    assert C.device_status() == 0
    assert torch.equal(got, kept)
    ref = to.trimul_forward_backward(z, direction, torch.ones(B, N, N) if m is None else m.float(), w,
                                     torch.zeros_like(z))["out"]
    assert rel_l2(got.cpu(), ref) <= 5.5e-3


# A CTA keeps the row sums of four tiles at C = 128 and of eight at C = 64, on 148 SMs: 800 tiles are five or six a CTA, 841
# the same with padded lines, 1250 and 1301 are eight or nine.
@pytest.mark.parametrize("N,channels,direction,mask", [
    (320, 128, "outgoing", "pair"), (325, 128, "incoming", "bool"), (400, 64, "incoming", "pair"),
    (403, 64, "outgoing", "none")])
def test_forward_with_rings_used_again(N, channels, direction, mask):
    t = trimul_inputs(1, N, channels, seed=N)
    g = torch.Generator().manual_seed(N)
    w = {n: x + 0.2 * torch.randn(x.shape, generator=g) if x.ndim == 1 else x for n, x in t["weights"].items()}
    m = {"pair": t["mask"], "bool": t["mask"].bool(), "none": None}[mask]
    dm = None if m is None else m.cuda()
    z = t["z"].cuda()
    with torch.no_grad():
        got = tk.turbo_trimul(z, direction, dm, **{n: x.cuda() for n, x in w.items()})
    kept = tk.turbo_trimul(z, direction, dm, **{n: x.cuda().requires_grad_(True) for n, x in w.items()}).detach()
    torch.cuda.synchronize()
    assert C.device_status() == 0
    assert torch.equal(got, kept)
    ref = to.trimul_forward(t["z"], direction, torch.ones(1, N, N) if m is None else m.float(), w)
    assert rel_l2(got.cpu(), ref) <= 5.5e-3


def test_passes_over_different_inputs_do_not_leak_into_one_another():
    """The block at C = 64 with more row tiles than CTAs: its residual is the z tile in shared memory, whose slot the next
    tile's copy takes.  Read after that copy had begun, it gave other values in some passes, and only where the
    passes before had left other data."""
    from openfold3_triangle_kernel_b200.pair_block import pair_stack_block
    from oracle.pair_block_oracle import block_params
    N = 400
    params = {k: {n: v.cuda() for n, v in m.items()} for k, m in block_params(64, 4, 16, seed=5).items()}
    mask = torch.ones(1, N, N, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(5)
    zs = [torch.randn(1, N, N, 64, generator=g, device="cuda").bfloat16() for _ in range(5)]
    first = None
    with torch.no_grad():
        for _ in range(10):
            outs = [pair_stack_block(z, mask, params, 4) for z in zs]
            first = first or outs
            assert all(torch.equal(a, b) for a, b in zip(outs, first))
    assert C.device_status() == 0


@pytest.mark.parametrize("B,N,channels,shift", [
    (3, 8, 128, 0.0),     # a tile that spans batch entries, the last one half full
    (1, 40, 64, 40.0),    # rows whose mean is forty times their spread
    (1, 40, 128, 40.0),
    (1, 152, 128, 0.0),   # a second tile for some CTAs
])
def test_rows_kept_for_the_backward(B, N, channels, shift):
    """The normalised rows and their statistics, which the projection kernel writes beside a and b.  A value is rounded
    to bf16 once (half of a unit in the eighth bit: 2^-8 of it at most); fp32 sums of squares leave (shift / spread)^2 2^-24
    times a few in the variance, 1e-4."""
    t = trimul_inputs(B, N, channels, seed=N)
    z = (t["z"].float() + shift).bfloat16().cuda()
    g = torch.Generator().manual_seed(N)
    w = {n: (x + 0.2 * torch.randn(x.shape, generator=g) if x.ndim == 1 else x).cuda() for n, x in t["weights"].items()}
    order = ("p_in_weight", "g_in_weight", "p_out_weight", "g_out_weight", "norm_in_weight", "norm_in_bias",
             "norm_out_weight", "norm_out_bias")
    kept = C.native().trimul_fwd(z, t["mask"].cuda(), [w[n] for n in order], False)
    x = z.double().reshape(-1, channels)
    mean, var = x.mean(1), x.var(1, unbiased=False)
    ref = (x - mean[:, None]) / (var + 1e-5).sqrt()[:, None] * w["norm_in_weight"].double() + w["norm_in_bias"].double()
    assert ((kept[1].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-4 * (1 + ref.abs())).all()
    assert ((kept[2].double() - mean).abs() <= 1e-6 * (1 + mean.abs())).all()
    assert ((kept[3].double() * (var + 1e-5).sqrt() - 1).abs() <= 2e-4).all()


@pytest.mark.parametrize("channels,kernels", [(32, 6), (64, 5), (96, 6), (128, 5)])
def test_a_forward_with_a_backward_behind_it_reads_z_twice(channels, kernels):
    """Weights, [norm,] projection, contraction, output norm, output: at C = 64 and 128 the norm of z is not a pass of its
    own."""
    t = trimul_inputs(1, 21, channels, seed=1)
    w = {n: x.cuda().requires_grad_(True) for n, x in t["weights"].items()}
    n0 = C.load().tpf_launch_count()
    tk.turbo_trimul(t["z"].cuda().bfloat16(), "outgoing", t["mask"].cuda(), **w)
    assert C.load().tpf_launch_count() - n0 == kernels
