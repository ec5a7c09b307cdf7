"""The nested K_r^{-1} with its inner PCG kept by request: its options and counts are the PCG's, in
both precision forms, on a material that the product on 1/eps inverts to within tolM."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _systems(N, cuda_device):
    import torch
    import fame_b200 as F
    E = O.material_separable_cos(N, 12.0)
    S = O.build_q_system(N, F.configs.P_GOLDEN, F.configs.Q_PHYS, E)
    return S, F.build_q_system(F.MassBackend(torch.as_tensor(E, device=cuda_device), N), F.configs.P_GOLDEN,
                               F.configs.Q_PHYS)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_inner_pcg_matches_the_oracle(cuda_device, precision):
    """tolKr 1e-12, tolM 1e-12: within 1e-10 of the explicit oracle form, as the nested form without
    the request (test_gpu_solver.py)."""
    import torch
    import fame_b200 as F
    S, sg = _systems(2, cuda_device)
    rng = np.random.default_rng(6)
    b = rng.standard_normal(S.nr) + 1j * rng.standard_normal(S.nr)
    y_exact = O.make_explicit_krinv_compact(S, 1e-14, 5000)[0](b)
    op, stats = F.make_nested_krinv_instrumented(sg, 4.0, 1e-12, 1e-12, maxitKr=2000, maxitM=4000,
                                                 precision=precision, inner_pcg=True)
    y = op(torch.as_tensor(b, device=cuda_device)).cpu().numpy()
    assert np.linalg.norm(y - y_exact) < 1e-10 * np.linalg.norm(y_exact)
    st = stats()
    assert st.inverseCalls == 1 and st.massSolveCalls > 0 and st.totalMassIterations > 2 * st.massSolveCalls
    if precision == "mixed":
        assert st.fp32Iterations == st.totalMassIterations and st.refineSteps >= st.massSolveCalls
    else:
        assert st.fp32Iterations == 0 and st.refineSteps == 0


def test_inner_iteration_limit_is_an_error_again(cuda_device):
    """maxitM 1 does not reach tolM: the inner solve's error with the PCG kept, no effect otherwise."""
    import torch
    import fame_b200 as F
    S, sg = _systems(3, cuda_device)
    b = torch.as_tensor(O.start_vector(5, S.nr), device=cuda_device)
    op, _ = F.make_nested_krinv_instrumented(sg, maxitM=1, inner_pcg=True)
    with pytest.raises(F.FameError) as e:
        op(b)
    assert e.value.status == F._lib.FAME_ERR_NOT_CONVERGED and "Nested M solve" in str(e.value)
    op, stats = F.make_nested_krinv_instrumented(sg, maxitM=1)
    op(b)
    assert stats().totalMassIterations == stats().massSolveCalls


def test_unknown_kinds_stay_refused(cuda_device):
    import fame_b200 as F
    _, sg = _systems(1, cuda_device)
    for kind in (-1, 3, 7):
        o = F.core._opts(kind=kind)
        with pytest.raises(F.FameError) as e:
            F.KrInv(sg, o)
        assert e.value.status == F._lib.FAME_ERR_INVALID


@pytest.mark.parametrize("N", [1, 2, 3])
@pytest.mark.parametrize("inner_pcg", [False, True])
def test_negative_preconditioner_scale(cuda_device, N, inner_pcg):
    """epsC < 0 breaks the outer PCG down after one step, in both inner forms: that step is the
    solution on eps = 1, where K_r is |q|^2 (accepted on its residual), and the breakdown's error on
    any other material."""
    import torch
    import fame_b200 as F
    b = None
    for E, ok in ((np.ones((2 * N) ** 6), True), (O.material_separable_cos(N, 12.0), False)):
        sg = F.build_q_system(F.MassBackend(torch.as_tensor(E, device=cuda_device), N), F.configs.P_GOLDEN,
                              F.configs.Q_PHYS)
        b = torch.as_tensor(O.start_vector(5, sg.nr), device=cuda_device)
        op, _ = F.make_nested_krinv_instrumented(sg, epsC=-1.0, inner_pcg=inner_pcg)
        if ok:
            y = op(b)
            ref = b / sg.sigmaR
            assert float(torch.linalg.norm(y - ref) / torch.linalg.norm(ref)) < 1e-9
        else:
            with pytest.raises(F.FameError) as e:
                op(b)
            assert e.value.status == F._lib.FAME_ERR_NOT_CONVERGED
