"""The forms of the larger grids (2N = 8, 10, 12, 14 have tile shapes and launch bounds of their own)
against plain torch in complex128: recovery, the nested K_r^{-1}, the mass adjoint, and Gram-Schmidt
over more row tiles than a launch has blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(N):
    import fame_b200 as F
    E = F.configs.material_separable_cos(N, delta=12.0)
    return E, F.build_q_system(F.MassBackend(E, N), F.configs.P_GOLDEN, F.configs.Q_PHYS)


def _mass(x, E, N):
    """fftn(E .* ifftn(x)) for every NF block of x."""
    import torch
    n = 2 * N
    return torch.cat([torch.fft.fftn(E.view((n,) * 6) * torch.fft.ifftn(b.view((n,) * 6))).reshape(-1)
                      for b in x.view(-1, n ** 6)])


def _V(sg, y):
    import torch
    y1, y2 = y[:sg.NF], y[sg.NF:]
    return torch.cat([sg.V11 * y1 + sg.V12 * y2, sg.V21 * y1 + sg.V22 * y2, sg.V31 * y1 + sg.V32 * y2])


def _VH(sg, w):
    import torch
    a, b, c = w.view(3, -1)
    return torch.cat([sg.V11.conj() * a + sg.V21.conj() * b + sg.V31.conj() * c,
                      sg.V12.conj() * a + sg.V22.conj() * b + sg.V32.conj() * c])


@pytest.mark.parametrize("N", [4, 5, 6, 7])
def test_recovery(cuda_device, N):
    """X and M X to rounding: a few ulp times the material's contrast of 13 (bound 1e-13)."""
    import torch
    import fame_b200 as F
    E, sg = _system(N)
    Y = torch.stack([F.start_vector(s, sg.nr) for s in (3, 4)], 0).t()
    X, MX, info = F.recover_original_eigenvectors(Y, sg)
    assert info["iterations"] == [1, 1] and max(info["relativeResiduals"]) <= 1e-12
    for j in range(2):
        b = _V(sg, Y[:, j].contiguous())
        x = _mass(b, 1.0 / E, N)
        s = 1.0 / torch.sqrt(torch.vdot(x, b).real)
        for got, ref in ((X[:, j], x * s), (MX[:, j], b * s)):
            assert float(torch.linalg.norm(got - ref) / torch.linalg.norm(ref)) < 1e-13


@pytest.mark.parametrize("N", [4, 5, 6, 7])
def test_nested_exact(cuda_device, N):
    """K_r y = b to the outer tolerance: ||b - V^* M^{-1} V y|| <= (1e-8 + rounding) ||b||; the check's
    own products carry a few ulp times the contrast, far below a tenth of that."""
    import torch
    import fame_b200 as F
    E, sg = _system(N)
    b = F.start_vector(11, sg.nr)
    op, stats = F.make_nested_krinv_instrumented(sg, tolKr=1e-8, maxitKr=4000)
    y = op(b)
    st = stats()
    assert st.massSolveCalls == st.totalMassIterations > 0
    r = b - _VH(sg, _mass(_V(sg, y), 1.0 / E, N))
    assert float(torch.linalg.norm(r) / torch.linalg.norm(b)) < 1.1e-8


@pytest.mark.parametrize("N,modes,params", [(5, 3, 2), (6, 2, 1), (7, 1, 1), (7, 3, 2)])
def test_adjoint(cuda_device, N, modes, params):
    """sum_y g(y) NF sum_c |ifftn(x_c)(y)|^2 with g of random sign: 1e-13 of the sum of magnitudes."""
    import torch
    import fame_b200 as F
    E, _ = _system(N)
    m = F.MassBackend(E, N)
    X = torch.stack([F.start_vector(20 + j, 3 * m.NF) for j in range(modes)], 0).t()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(N)
    g = [torch.randn(m.NF, dtype=torch.float64, device="cuda", generator=gen) for _ in range(params)]
    out = F.grad.mass_adjoint(m, X, g)
    n = 2 * N
    for j in range(modes):
        d = sum(torch.fft.ifftn(c.view((n,) * 6)).abs().square().reshape(-1) for c in X[:, j].contiguous().view(3, -1))
        for t in range(params):
            ref, size = float((g[t] * d).sum()) * m.NF, float((g[t].abs() * d).sum()) * m.NF
            assert abs(out[j, t] - ref) < 1e-13 * size


@pytest.mark.parametrize("N", [3, 4])
def test_gram_schmidt_over_many_tiles(cuda_device, N):
    """729 and 4096 tiles of 128 rows on at most 365 blocks: the fused passes (p = 40) and the
    two-kernel form they are compared with (p = 70, the columns past 64) give the same smallest
    eigenvalues (tol 1e-10, tolCG 1e-12, bound 1e-9), with orthonormal vectors."""
    import torch
    import fame_b200 as F
    _, sg = _system(N)
    op, _ = F.make_explicit_krinv_compact(sg, 1e-12, 3000)
    v0 = F.start_vector(7, sg.nr)
    Y, th, _, info = F.Lanczos(op, None, None, sg.nr, 3, 1e-10, 100, 40, v0)
    ref = F.Lanczos(op, None, None, sg.nr, 3, 1e-10, 100, 70, v0)[1]
    assert info["converged"]
    assert np.max(np.abs(np.sort(th) - np.sort(ref)) / np.sort(ref)) < 1e-9
    G = (Y.conj().t() @ Y).cpu().numpy()
    assert np.max(np.abs(G - np.eye(3))) < 1e-12
