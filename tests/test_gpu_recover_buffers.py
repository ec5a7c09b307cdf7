"""Recovery where the caller's buffers or streams are not the plain ones: outputs that overlap the
input, a mass handle made on another stream, and materials the chain on 1/E does not invert."""
import ctypes as C

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _system(N, E):
    import torch
    import fame_b200 as F
    return F.build_q_system(F.MassBackend(torch.as_tensor(E, device="cuda"), N), F.configs.P_REFERENCE,
                            F.configs.Q_TRACKING)


def _recover(sg, Y, X, MX):
    from fame_b200 import _lib as L
    rr = (C.c_double * 1)()
    sg.ctx.bind()
    st = L.lib.fame_recover_eigvecs(sg.h, sg.mass.h, C.c_void_p(Y.data_ptr()), 1, C.c_double(1e-12), 3000,
                                    L.FAME_PREC_FP64, C.c_void_p(X.data_ptr()), C.c_void_p(MX.data_ptr()), None, rr)
    return st, rr[0]


@pytest.mark.parametrize("N", [1, 2, 3, 4])
@pytest.mark.parametrize("which", ["X", "MX", "tail"])
def test_outputs_over_the_input(cuda_device, N, which):
    """One vector recovered over its own input; bound: the PCG's residual of 1e-12 times the
    material's contrast of 11, as in test_gpu_exact_inverse.py."""
    import torch
    sg = _system(N, O.material_smooth_exp(N))
    y = torch.as_tensor(O.start_vector(5, sg.nr), device="cuda")
    X, MX = (torch.empty(sg.ndof, dtype=torch.complex128, device="cuda") for _ in range(2))
    assert _recover(sg, y, X, MX)[0] == 0
    A, B = (torch.empty(sg.ndof, dtype=torch.complex128, device="cuda") for _ in range(2))
    buf = A if which == "X" else B
    at = buf[sg.ndof - sg.nr:] if which == "tail" else buf[:sg.nr]
    at.copy_(y)
    st, rr = _recover(sg, at, A, B)
    assert st == 0 and rr <= 1e-12
    for got, ref in ((A, X), (B, MX)):
        assert float(torch.linalg.norm(got - ref) / torch.linalg.norm(ref)) < 2e-11


def test_material_that_is_not_inverted_runs_no_chain(cuda_device):
    """Contrast 4001 (16 ulp times that is above the tolerance): left to the PCG alone, which
    writes nothing before it has converged."""
    import torch
    from fame_b200 import _lib as L
    N = 3
    sg = _system(N, O.material_separable_cos(N, 4000.0))
    y = torch.as_tensor(O.start_vector(5, sg.nr), device="cuda")
    X, MX = (torch.full((sg.ndof,), 7.0, dtype=torch.complex128, device="cuda") for _ in range(2))
    rr = (C.c_double * 1)()
    sg.ctx.bind()
    st = L.lib.fame_recover_eigvecs(sg.h, sg.mass.h, C.c_void_p(y.data_ptr()), 1, C.c_double(1e-12), 2,
                                    L.FAME_PREC_FP64, C.c_void_p(X.data_ptr()), C.c_void_p(MX.data_ptr()), None, rr)
    assert st == L.FAME_ERR_NOT_CONVERGED
    assert bool((X == 7.0).all()) and bool((MX == 7.0).all())


def test_mass_made_on_another_stream(cuda_device):
    """The chains wait for the mass handle's tables although another stream fills them."""
    import torch
    import fame_b200 as F
    N = 3
    E = torch.as_tensor(O.material_smooth_exp(N), device="cuda")
    ref = _system(N, O.material_smooth_exp(N))
    y = torch.as_tensor(O.start_vector(5, ref.nr), device="cuda").reshape(-1, 1)
    X0, _, _ = F.recover_original_eigenvectors(y, ref)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)  # the set-up below is queued behind this
        m = F.MassBackend(E, N)
    sg = F.build_q_system(m, F.configs.P_REFERENCE, F.configs.Q_TRACKING)
    X, _, info = F.recover_original_eigenvectors(y, sg)
    assert info["iterations"] == [1] and np.isfinite(info["relativeResiduals"][0])
    assert torch.equal(X, X0)
