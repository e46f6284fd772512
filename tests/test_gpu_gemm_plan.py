"""GPU: the prefill GEMM where its tile width, row halves and K split change: few tiles with a long K (the sums of a tile meet
in a cluster), odd numbers of pieces per CTA, tile borders that cut row patches, every element type."""
import pytest
import torch

from oracle import bqq_oracle as O
from tests.helpers import oracle_forward_t, synth_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('rw,cw,M', [(2, 160, 129), (5, 64, 200), (12, 60, 333), (40, 90, 150), (9, 33, 700), (37, 40, 300),
                                     (1, 96, 260)])
def test_split_and_tile_rules(rw, cw, M):
    from bqq_b200.bqq_modules import BinaryQuadratic, check_status
    Y, Z, A, bias, X = synth_layer(2, rw, cw, 40, 32, 32, M, seed=rw + cw + M, bias=True)      # P = 40: borders cut row patches
    bq = BinaryQuadratic(Y.float(), Z.float(), A, bias=bias).cuda()
    for dt, tol in ((torch.float32, 1e-4), (torch.bfloat16, 1e-3 + 2 ** -8), (torch.float16, 1e-3 + 2 ** -10)):
        Xd = X.to(dt)
        with torch.no_grad():
            y = bq(Xd.cuda())
            again = bq(Xd.cuda())
        assert torch.equal(y, again)                        # the exchange adds in a fixed order
        assert O.max_rel_err(y.float().cpu().numpy(), oracle_forward_t(Y, Z, A, bias, Xd)) < tol
    check_status()


@pytest.mark.parametrize('rw,cw,M,dtype', [(1100, 32, 300, torch.bfloat16), (900, 40, 2100, torch.float16), (520, 64, 256, torch.float32)])
def test_pairs_and_panels(rw, cw, M, dtype):
    """W of more than 64 MB: column panels of one wave each, and CTA pairs where the row tiles are even."""
    from bqq_b200.bqq_modules import BinaryQuadratic, check_status
    Y, Z, A, _, X = synth_layer(1, rw, cw, 32, 32, 8, M, seed=rw, x_dtype=dtype)
    bq = BinaryQuadratic(Y.float(), Z.float(), A).cuda()
    with torch.no_grad():
        y = bq(X.cuda()).float()
        W = bq.get_weight(torch.float32)
        ref = X.cuda().double() @ W.double().T
    tol = 1e-4 if dtype == torch.float32 else 1e-3 + (2 ** -8 if dtype == torch.bfloat16 else 2 ** -10)
    assert ((y - ref).abs().max() / ref.abs().max()).item() < tol
    check_status()


@pytest.mark.parametrize('cw', [4, 33, 65])
@pytest.mark.parametrize('M', [130, 700])
def test_rows_staged_from_any_place(cw, M):
    """x whose rows are not aligned to four elements, or not a multiple of a block's columns, takes the staging kernel."""
    from bqq_b200.bqq_modules import BinaryQuadratic
    Y, Z, A, _, X = synth_layer(2, 3, cw, 32, 32, 32, M, seed=cw + M)
    bq = BinaryQuadratic(Y.float(), Z.float(), A).cuda()
    for dt, tol in ((torch.float32, 1e-4), (torch.bfloat16, 1e-3 + 2 ** -8), (torch.float16, 1e-3 + 2 ** -10)):
        Xd = X.to(dt)
        ref = oracle_forward_t(Y, Z, A, None, Xd)
        for skip, pitch in ((0, 0), (1, 3), (8, 8), (4, 5)):
            wide = torch.zeros(M, cw * 32 + 16 + pitch, dtype=dt, device='cuda')
            wide[:, skip:skip + cw * 32] = Xd.cuda()
            with torch.no_grad():
                y = bq(wide[:, skip:skip + cw * 32])
            assert O.max_rel_err(y.float().cpu().numpy(), ref) < tol
