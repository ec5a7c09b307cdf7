"""A bounded device-side wait that gives up is reported by the call whose result it spoils: the
expiry is made by the self-test entry (barriers armed for bytes that no copy delivers)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

PASS_B, DENSITY, GRAM_SCHMIDT = 0, 1, 2


def _mass(N):
    import torch
    import fame_b200 as F
    return F.MassBackend(torch.as_tensor(O.material_separable_cos(N, 12.0), device="cuda"), N)


def _expire(m, kernel):
    from fame_b200 import _lib as L
    m.ctx.bind()
    assert L.lib.fame_selftest_expired_wait(m.h, kernel, 1024) == L.FAME_OK


@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 6, 7])
def test_adjoint_reports_an_expired_wait(cuda_device, N):
    import torch
    import fame_b200 as F
    m = _mass(N)
    X = torch.as_tensor(O.start_vector(3, 3 * m.NF), device="cuda").reshape(-1, 1)
    g = [torch.ones(m.NF, dtype=torch.float64, device="cuda")]
    ref = F.grad.mass_adjoint(m, X, g)
    _expire(m, DENSITY)
    with pytest.raises(F.FameError) as e:
        F.grad.mass_adjoint(m, X, g)
    assert e.value.status == F._lib.FAME_ERR_CUDA
    assert np.array_equal(F.grad.mass_adjoint(m, X, g), ref)  # cleared, and the context is usable


@pytest.mark.parametrize("kernel", [PASS_B, GRAM_SCHMIDT])
def test_lanczos_reports_an_expired_wait(cuda_device, kernel):
    import fame_b200 as F
    m = _mass(2)
    sysq = F.build_q_system(m, F.configs.P_GOLDEN, F.configs.Q_PHYS)
    op, _ = F.make_explicit_krinv_compact(sysq, 1e-10, 3000)
    v0 = F.start_vector(7, sysq.nr)
    args = (op, None, None, sysq.nr, 4, 1e-8, 30, 24, v0)
    ref = F.Lanczos(*args)[1]
    _expire(m, kernel)
    with pytest.raises(F.FameError) as e:
        F.Lanczos(*args)
    assert e.value.status == F._lib.FAME_ERR_CUDA
    assert np.array_equal(F.Lanczos(*args)[1], ref)


def test_selftest_refuses_other_arguments(cuda_device):
    from fame_b200 import _lib as L
    m = _mass(1)
    for kernel, limit in ((3, 16), (-1, 16), (0, 0), (1, 1 << 21)):
        assert L.lib.fame_selftest_expired_wait(m.h, kernel, limit) == L.FAME_ERR_INVALID


def test_every_context_hears_of_a_fault_once(cuda_device):
    """The fault word is the device's: the context whose check clears it need not be the one whose
    work was spoiled, so the others report it at their next synchronisation too, once; a context
    made afterwards does not, and calls that check their own run are not refused for it."""
    import torch
    import fame_b200 as F
    m = _mass(2)
    m.ctx.sync()
    other, third = F.Context(0), F.Context(0)
    _expire(m, PASS_B)
    for ctx in (other, m.ctx):  # the first of them clears the word
        with pytest.raises(F.FameError) as e:
            ctx.sync()
        assert e.value.status == F._lib.FAME_ERR_CUDA
        ctx.sync()
    late = F.Context(0)
    late.sync()
    # a healthy call of a context that has not synchronised since is not refused
    m3 = F.MassBackend(torch.as_tensor(O.material_separable_cos(2, 12.0), device="cuda"), 2, ctx=third)
    X = torch.as_tensor(O.start_vector(3, 3 * m.NF), device="cuda").reshape(-1, 1)
    g = [torch.ones(m.NF, dtype=torch.float64, device="cuda")]
    assert np.array_equal(F.grad.mass_adjoint(m3, X, g), F.grad.mass_adjoint(m, X, g))
    with pytest.raises(F.FameError):
        third.sync()
    third.sync()


def test_rayleigh_ritz_reports_an_expired_wait(cuda_device):
    import torch
    import fame_b200 as F
    m = _mass(2)
    sysq = F.build_q_system(m, F.configs.P_GOLDEN, F.configs.Q_PHYS)
    Y = torch.stack([F.start_vector(s, sysq.nr) for s in (1, 2, 3)], 0).t()
    _expire(m, PASS_B)
    with pytest.raises(F.FameError) as e:
        F.rayleigh_ritz(sysq, Y)
    assert e.value.status == F._lib.FAME_ERR_CUDA
    assert F.rayleigh_ritz(sysq, Y)[0].shape == (3,)
