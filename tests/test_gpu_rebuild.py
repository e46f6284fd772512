"""GPU: dense weights rebuilt from the planes where the work split changes: more bit layers than one stage holds, an odd
number of super-groups, padded col patches, several blocks per patch, coefficients of every type and of extreme size."""
import numpy as np
import pytest
import torch

from oracle import bqq_oracle as O
from tests.helpers import synth_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape', [(1, 1, 1, 32, 32, 32), (8, 3, 5, 32, 32, 32), (9, 2, 3, 32, 32, 32),
                                   (17, 2, 2, 40, 48, 40), (3, 5, 13, 64, 64, 64), (2, 160, 9, 32, 32, 32),
                                   (1, 2, 7, 128, 128, 64)])
@pytest.mark.parametrize('dtype', [torch.float32, torch.bfloat16])
def test_weight_across_stage_borders(shape, dtype):
    from bqq_b200.bqq_modules import BinaryQuadratic
    bw, rw, cw, P, Q, r = shape
    Y, Z, A, _, _ = synth_layer(bw, rw, cw, P, Q, r, 1, seed=sum(shape))
    bq = BinaryQuadratic(Y.float(), Z.float(), A).cuda()
    a, b, c, d = O.split_coefficients(A.numpy())
    Wref = O.dense_weight(Y.numpy(), Z.numpy(), a, b, c, d)
    W = bq.get_weight(dtype)
    assert tuple(W.shape) == (rw * P, cw * Q)
    eps = 1e-5 if dtype == torch.float32 else 2 ** -8
    assert np.abs(W.float().cpu().numpy() - Wref).max() <= eps * max(1.0, np.abs(Wref).max())


@pytest.mark.parametrize('scale', [1e-9, 1.0, 1e9])
@pytest.mark.parametrize('coef_dtype', [torch.float32, torch.bfloat16])
def test_weight_coefficient_range(scale, coef_dtype):
    from bqq_b200.bqq_modules import BinaryQuadratic
    Y, Z, A, _, _ = synth_layer(2, 3, 6, 32, 32, 32, 1, seed=5)
    bq = BinaryQuadratic(Y.float(), Z.float(), A * scale).cuda()
    for n in 'abcd':
        setattr(bq, n, torch.nn.Parameter(getattr(bq, n).data.to(coef_dtype)))
    a, b, c, d = (getattr(bq, n).data.float().cpu().numpy() for n in 'abcd')
    Wref = O.dense_weight(Y.numpy(), Z.numpy(), a, b, c, d)
    W = bq.get_weight(torch.float32).cpu().numpy()
    assert np.abs(W - Wref).max() <= 1e-5 * np.abs(Wref).max()
