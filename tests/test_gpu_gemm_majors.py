"""The tensor-core GEMM's TMA form over every pair of operand layouts (each operand's contiguous dimension is K or the
other one), at the edges of its tiles and chunks; and the reductions that share a backward launch."""
import numpy as np
import pytest
import torch

from oracle import mlp_oracle as MO
from pramana_b200.mlp import MlpNetwork, gemm_bf16

pytestmark = pytest.mark.gpu


# K of one MMA step, one chunk, one more than the deepest pipeline; M and N of one row, around one tile of each
# width, and (the last two) enough tiles for every SM at 128 x 128 and at 128 x 256
@pytest.mark.parametrize("m,n,k", [(8, 8, 8), (128, 64, 64), (136, 72, 72), (120, 56, 1), (64, 136, 584),
                                   (1672, 1672, 136), (2184, 2568, 200)])
@pytest.mark.parametrize("a_k", [True, False])
@pytest.mark.parametrize("b_k", [True, False])
def test_layouts(m, n, k, a_k, b_k):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    lead = 8 * (k // 8 + 1)  # a row stride beyond the row, so that K itself may be any size
    a = torch.randn(m, lead, device="cuda", generator=g).to(torch.bfloat16)[:, :k]
    b = torch.randn(n, lead, device="cuda", generator=g).to(torch.bfloat16)[:, :k]
    at, bt = a if a_k else a.t().contiguous(), b if b_k else b.t().contiguous()
    mask = torch.randn(m, n, device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(n, device="cuda", generator=g)
    cf = torch.empty(m, n, device="cuda")
    cb = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    gemm_bf16(at, bt, alpha=0.5, bias=bias, relu=True, mask=mask, out_f32=cf, out_bf16=cb, m=m, n=n, k=k,
              a_strides=(lead, 1) if a_k else (1, m), b_strides=(1, lead) if b_k else (n, 1))
    torch.cuda.synchronize()
    want = torch.relu(0.5 * (a.double() @ b.double().t()) + bias)
    want = torch.where(mask.float() > 0, want, torch.zeros_like(want))
    scale = 0.5 * (a.double().abs() @ b.double().abs().t()) + bias.abs()
    assert torch.all((cf.double() - want).abs() <= 1e-5 * scale)
    assert torch.equal(cb, cf.to(torch.bfloat16))


# rows around one staging of the column sums (1,544 rows of 32 columns in eight 24 KB stages; fewer stages, fewer
# rows) and one row; the loss's 148 partial sums
@pytest.mark.parametrize("rows", [1, 127, 129, 1543, 1545, 3100])
def test_bias_gradients_and_loss(rows):
    widths = [8, 72, 40]
    rng = np.random.default_rng(rows)
    x = rng.uniform(-1, 1, size=(rows, 8)).astype(np.float32)
    t = rng.standard_normal((rows, 40)).astype(np.float32)
    net = MlpNetwork(widths, max_batch=rows, seed=3)
    loss, grad = net.loss_grad(x, t)
    want_loss, want = MO.loss_grad(net.get_params(), widths, x, t, bf16_points=True)
    assert abs(loss - want_loss) <= 1e-3 * want_loss
    offs, _ = MO.layout(widths)
    for (w0, b0), end in zip(offs, [offs[1][0], len(want)]):
        for lo, hi in ((w0, b0), (b0, end)):
            assert np.linalg.norm(grad[lo:hi] - want[lo:hi]) <= 1e-2 * np.linalg.norm(want[lo:hi])
