"""GPU: the fused rebuild-and-multiply route (9 to 128 rows, and patch geometries the decode kernel pads badly) at the edges
of its tiles: rows of x around the operand width, row blocks that do not fill a tile, several chunks of K and items per
CTA, more bit layers than a stage holds, every element type; a row shard gives the bits of the whole layer."""
import pytest
import torch

from oracle import bqq_oracle as O
from tests.helpers import oracle_forward_t, synth_layer

pytestmark = pytest.mark.gpu


def _run(bq, X):
    with torch.no_grad():
        return bq(X.cuda())


@pytest.mark.parametrize('shape', [(2, 3, 5, 32, 32, 32), (9, 5, 7, 32, 32, 32), (1, 3, 5, 96, 40, 33), (3, 4, 6, 64, 64, 64),
                                   (2, 7, 3, 40, 128, 16), (2, 9, 40, 32, 32, 32)])
@pytest.mark.parametrize('M', [4, 5, 8, 9, 12, 13, 16, 17, 33, 64, 65, 128])
def test_fused_against_oracle(shape, M):
    from bqq_b200.bqq_modules import BinaryQuadratic, check_status
    Y, Z, A, bias, X = synth_layer(*shape, M, seed=sum(shape) + M, bias=True)
    bq = BinaryQuadratic(Y.float(), Z.float(), A, bias=bias).cuda()
    for dt, tol in ((torch.float32, 1e-4), (torch.bfloat16, 1e-3 + 2 ** -8), (torch.float16, 1e-3 + 2 ** -10)):
        Xd = X.to(dt)
        ref = oracle_forward_t(Y, Z, A, bias, Xd)
        y = _run(bq, Xd)
        assert y.dtype == dt and O.max_rel_err(y.float().cpu().numpy(), ref) < tol
        assert torch.equal(_run(bq, Xd), y)                  # reproducible, scratch left as it was
    check_status()


@pytest.mark.parametrize('rw,cw,M', [(1200, 12, 16), (160, 70, 100), (2400, 4, 33)])
def test_fused_many_items(rw, cw, M):
    """Several items per CTA and tiles completed by any of them; sampled row patches against the oracle."""
    from bqq_b200.bqq_modules import BinaryQuadratic, shard_rows
    Y, Z, A, _, X = synth_layer(2, rw, cw, 32, 32, 32, M, seed=rw, x_dtype=torch.bfloat16)
    bq = BinaryQuadratic(Y.float(), Z.float(), A).cuda()
    y = _run(bq, X)
    rows = sorted({0, 3, 4, rw // 2 + 1, rw - 1})
    a, b, c, d = O.split_coefficients(A[:, rows].numpy())
    ref = O.forward(Y[:, rows].numpy(), Z[:, rows].numpy(), a, b, c, d, X.float().numpy())
    got = y.float().cpu().reshape(M, rw, 32)[:, rows].reshape(M, -1).numpy()
    assert O.max_rel_err(got, ref) < 1e-3 + 2 ** -8
    if M <= 16:
        parts = [_run(shard_rows(bq, k, 2).cuda(), X) for k in range(2)]
        assert torch.equal(torch.cat(parts, -1), y)


@pytest.mark.parametrize('cw,Q,M', [(530, 32, 20), (530, 31, 3), (131, 128, 17), (40, 31, 74), (2, 36, 128)])
def test_fused_rows_of_every_length(cw, Q, M):
    """x staged by either preparation (rows of up to 16384 columns and longer ones), quads aligned or not."""
    from bqq_b200.bqq_modules import BinaryQuadratic
    Y, Z, A, _, X = synth_layer(1, 2, cw, 96, Q, 33, M, seed=cw + M)
    bq = BinaryQuadratic(Y.float(), Z.float(), A).cuda()
    for dt, tol in ((torch.float32, 1e-4), (torch.bfloat16, 1e-3 + 2 ** -8), (torch.float16, 1e-3 + 2 ** -10)):
        Xd = X.to(dt)
        ref = oracle_forward_t(Y, Z, A, None, Xd)
        assert O.max_rel_err(_run(bq, Xd).float().cpu().numpy(), ref) < tol
        wide = torch.zeros(M, cw * Q + 3, dtype=dt, device='cuda')
        wide[:, 1:1 + cw * Q] = Xd.cuda()
        assert O.max_rel_err(_run(bq, wide[:, 1:1 + cw * Q]).float().cpu().numpy(), ref) < tol
