"""GPU: one row through the one-launch decode route, whose CTAs load x (and what is folded into it) before they use any:
short and full passes, quads that are not aligned, columns that are not a multiple of four, each type and prologue."""
import pytest
import torch

from oracle import bqq_oracle as O
from tests.helpers import oracle_forward_t, synth_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize('cw,Q', [(1, 32), (16, 32), (17, 32), (64, 32), (127, 32), (33, 30), (40, 28), (65, 31)])
def test_one_row_prepared_in_the_decode_kernel(cw, Q, dtype):
    from bqq_b200.bqq_modules import BinaryQuadratic
    Y, Z, A, _, _ = synth_layer(2, 2, cw, 32, Q, 32, 1, seed=cw)
    n = cw * Q
    bq = BinaryQuadratic(Y.float(), Z.float(), A).cuda()
    gen = torch.Generator(device='cuda').manual_seed(5)
    wide = torch.randn(1, 4 * n + 64, generator=gen, device='cuda').to(dtype)
    w = torch.rand(n + 1, generator=gen, device='cuda') + 0.5
    tol = {torch.float32: 1e-4, torch.bfloat16: 5e-3, torch.float16: 1e-3}[dtype]

    def check(y, x):
        assert O.max_rel_err(y.float().cpu().numpy(), oracle_forward_t(Y, Z, A, None, x.float().cpu())) < tol

    with torch.no_grad():
        for skip in (0, 1, 8):                               # 1: no quad of x is aligned
            x, g2 = wide[:, skip:skip + n], wide[:, skip:skip + 2 * n]
            check(bq(x), x)
            for ws in (w[:n], w[1:]):
                check(bq.forward_fused(x, rms_weight=ws), torch.nn.functional.rms_norm(x.float(), (n,), ws, 1e-5))
            check(bq.forward_fused(g2, swiglu=True), torch.nn.functional.silu(g2[:, :n].float()) * g2[:, n:].float())
