"""The stages of a row-sharded TriMul on one GPU, one shard after the other: the results and the state kept for the backward
are the unsharded operator's bit for bit, and no stage launches more kernels than its part of the whole call has."""
import pytest
import torch

import openfold3_triangle_kernel_b200 as tk
from openfold3_triangle_kernel_b200 import _cabi as C
from openfold3_triangle_kernel_b200.dap import CudaTrimulStages
from oracle.inputs import trimul_inputs

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA device")]

ORDER = ("p_in_weight", "g_in_weight", "p_out_weight", "g_out_weight", "norm_in_weight", "norm_in_bias",
         "norm_out_weight", "norm_out_bias")


@pytest.mark.parametrize("channels", [32, 64, 96, 128])
@pytest.mark.parametrize("direction", ["outgoing", "incoming"])
def test_stages_of_two_shards(channels, direction):
    B, N, P = 2, 64, 2
    t = trimul_inputs(B, N, channels, seed=channels, mask_mode="trailing10")
    g = torch.Generator().manual_seed(channels)
    w = {n: (x + 0.2 * torch.randn(x.shape, generator=g) if x.ndim == 1 else x).cuda() for n, x in t["weights"].items()}
    z, mask = t["z"].bfloat16().cuda(), t["mask"].cuda()
    incoming = direction == "incoming"
    whole = C.native().trimul_fwd(z, mask, [w[n] for n in ORDER], incoming)
    out, zln, mean_in, rstd_in, a_cm, b_cm, gate, x_cm, xln, mean_out, rstd_out = whole

    be, launches = CudaTrimulStages(), C.load().tpf_launch_count
    shards = []
    for r in range(P):
        rows = slice(r * N // P, (r + 1) * N // P)
        n0 = launches()
        shards.append(be.proj_fwd(z[:, rows].contiguous(), mask[:, rows].contiguous(), w, incoming))
        # the weights' layouts, the norm where it is a kernel of its own, the projection
        assert launches() - n0 <= (2 if channels % 64 == 0 else 3)
    cat = lambda name: torch.cat([s[name] for s in shards], 2)  # noqa: E731
    x = be.contract(cat("a_cm"), cat("b_cm"), incoming)
    for r in range(P):
        n0 = launches()
        be.out_fwd(shards[r], x[:, :, r * N // P:(r + 1) * N // P])
        assert launches() - n0 <= 3  # the weights' layouts, the norm, the output projection
    torch.cuda.synchronize()
    assert C.device_status() == 0

    assert torch.equal(out, tk.turbo_trimul(z, direction, mask, **w))
    assert torch.equal(torch.cat([s["out"] for s in shards], 1), out)
    assert torch.equal(x.reshape(x_cm.shape), x_cm)
    for name, ref in (("a_cm", a_cm), ("b_cm", b_cm)):
        assert torch.equal(cat(name).reshape(ref.shape), ref), name
    for name, ref in (("zln", zln), ("mean_in", mean_in), ("rstd_in", rstd_in), ("gate", gate), ("xln", xln),
                      ("mean_out", mean_out), ("rstd_out", rstd_out)):
        got = torch.cat([s[name].reshape(B, N // P, N, -1) for s in shards], 1)
        assert torch.equal(got, ref.reshape(got.shape)), name


def test_forward_workspace_does_not_grow_with_the_rows():
    """A rank's shard holds a part of the rows only, and nothing of the workspace belongs to one of them."""
    size = C.load().tpf_trimul_fwd_workspace_bytes
    for channels in (32, 64, 96, 128):
        assert size(1, 8, channels) == size(4, 1536, channels)
