"""The forward of TriMul with its norms inside the projection and output kernels (C = 64 and 128), at the edges of its
128-row tiles, 64-row copies and padded lines: against the fp64 oracle, and the forward that keeps nothing against the one
with a backward behind it.

Tolerance: eight roundings to bf16 lie between the inputs and a result (four weights, a, b, x, the result), 2^-9 at most and
independent: 2^-9 sqrt(8) = 5.5e-3.
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
    (1, 131, 128, "outgoing", "pair", 0.0),    # 64-row copies and lines that end inside one; a second tile for some CTAs
    (2, 259, 64, "outgoing", "pair", 0.0),     # more tiles of a CTA than it keeps row sums of
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
