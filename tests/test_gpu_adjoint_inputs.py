"""The parameter fields that the mass adjoint takes: several types at once, lazy negatives, refusals."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def test_field_types(cuda_device):
    import torch
    import fame_b200 as F
    N = 2
    m = F.MassBackend(torch.as_tensor(O.material_smooth_exp(N), device=cuda_device), N)
    X = torch.as_tensor(np.stack([O.start_vector(s, 3 * m.NF) for s in (1, 2)], 1), device=cuda_device)
    g = torch.as_tensor(np.random.default_rng(4).normal(size=m.NF), device=cuda_device)
    g32, gi = g.float(), (4 * g).to(torch.int64)
    neg = torch._neg_view(g)
    want = F.grad.mass_adjoint(m, X, [g, g32.double(), gi.double(), -g])
    assert np.array_equal(F.grad.mass_adjoint(m, X, [g, g32, gi, neg]), want)
    assert np.array_equal(F.grad.mass_adjoint(m, X, [neg]), want[:, 3:])
    for bad in ([g32], [gi], [g32, gi], [torch.complex(g, g)], [g[:-1]], [g.cpu()]):
        with pytest.raises(ValueError):
            F.grad.mass_adjoint(m, X, bad)
