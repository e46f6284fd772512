"""GPU: the native calls of the module (csrc/bqq_torch.cpp) against the interpreter's route, which still takes every case
that is not plain: strided and leading dimensions, replaced buffers and parameters, types, autograd."""
import pytest
import torch

from oracle import bqq_oracle as O
from tests.helpers import oracle_forward_t, synth_layer

pytestmark = pytest.mark.gpu


def _layer(seed=1, bias=True):
    from bqq_b200.bqq_modules import BinaryQuadratic
    Y, Z, A, b, X = synth_layer(2, 3, 5, 32, 32, 32, 20, seed=seed, bias=bias)
    return BinaryQuadratic(Y.float(), Z.float(), A, bias=b).cuda(), (Y, Z, A, b), X.cuda()


@pytest.mark.parametrize('rows', [1, 3, 20])
def test_native_and_python_routes_agree(rows):
    from bqq_b200 import _bqq_torch
    bq, _, X = _layer()
    wide = torch.zeros(20, 200, device='cuda')
    wide[:, 8:168] = X
    with torch.no_grad():
        bq(X), bq(X[:16])                                    # packs the planes and sizes the scratch of both routes
        for x in (X[:rows], wide[:rows, 8:168], X[:rows].reshape(1, rows, 160), X[:rows].bfloat16(), X[:rows].half()):
            y = _bqq_torch.forward(bq.__dict__, x)
            assert y is not None and y.shape == (*x.shape[:-1], 96) and y.dtype == x.dtype
            assert torch.equal(y, bq(x.clone()))
        res = torch.randn(rows, 96, device='cuda')
        w = torch.rand(160, device='cuda')
        f = _bqq_torch.forward_fused(bq.__dict__, X[:rows], w, 1e-5, False, res)
        assert (f is None) == (rows > 16)
        if f is not None:
            ref = bq(torch.nn.functional.rms_norm(X[:rows], (160,), w, 1e-5)) + res
            assert O.max_rel_err(f.cpu().numpy(), ref.cpu().numpy()) < 1e-4
        # not plain: a transposed X, an unpacked module, another width
        assert _bqq_torch.forward(bq.__dict__, X[:rows].t().contiguous().t()) is None or rows == 1
        assert _bqq_torch.forward({}, X) is None
        assert _bqq_torch.forward(bq.__dict__, X[:, :32].contiguous()) is None
    if any(p.requires_grad for p in bq.parameters()):
        assert _bqq_torch.forward(bq.__dict__, X) is None    # autograd: the Python route raises


def test_changed_buffers_and_parameters_are_seen():
    bq, (Y, Z, A, b), X = _layer(seed=2)
    with torch.no_grad():
        bq(X[:1])
        bq.Y.copy_(~Y.cuda())                                # in place: the version counter moves
        y = bq(X[:1])
        assert O.max_rel_err(y.cpu().numpy(), oracle_forward_t(~Y, Z, A, b, X[:1].cpu())) < 1e-4
        bq.a = torch.nn.Parameter(bq.a.data * 2)             # another tensor under the same name
        bq.bias = None
        A2 = A.clone()
        A2[..., 0] *= 2
        y = bq(X[:1])
        assert O.max_rel_err(y.cpu().numpy(), oracle_forward_t(~Y, Z, A2, None, X[:1].cpu())) < 1e-4
