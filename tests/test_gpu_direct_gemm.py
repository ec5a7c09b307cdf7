"""FP64 direct-grid reconstruction: the matrix-instruction GEMMs at grid sizes around the edges
of their 8-wide blocks and 48-wide tiles, on every 2N, against NumPy's factorised sum."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,sizes", [(1, (1, 1, 1)), (1, (7, 8, 9)), (2, (8, 47, 1)), (2, (48, 49, 50)),
                                     (3, (9, 5, 97)), (3, (96, 3, 41)), (4, (17, 33, 2)), (5, (11, 7, 5)),
                                     (6, (3, 10, 4))])
@pytest.mark.parametrize("ncomp", [1, 3])
def test_direct_grid_sizes(cuda_device, N, sizes, ncomp):
    """Sums of (2N)^6 terms in three FP64 contractions of (2N)^2: relative 1e-13 of the field's norm."""
    import torch
    import fame_b200 as F
    n, NF = 2 * N, (2 * N) ** 6
    rng = np.random.default_rng(N)
    sg = F.build_q_system(F.MassBackend(torch.as_tensor(O.material_smooth_exp(N), device=cuda_device), N),
                          F.configs.P_GOLDEN, F.configs.Q_PHYS)
    P, k = F.configs.P_GOLDEN, sg.kLift
    c = rng.standard_normal(ncomp * NF) + 1j * rng.standard_normal(ncomp * NF)
    axes = [[rng.uniform(-1, 1, size=s) for s in sizes] for _ in range(ncomp)]
    u = F.reconstruct_fields_direct_grid(torch.as_tensor(c, device=cuda_device), sg,
                                         [tuple(torch.as_tensor(a, device=cuda_device) for a in ax) for ax in axes])
    xi = np.concatenate([np.arange(N), np.arange(-N, 0)]).astype(float)
    for comp in range(ncomp):
        T = []
        for d in range(3):
            q = P[d, d] * (xi + k[d])[None, :] + P[d + 3, d] * (xi + k[d + 3])[:, None]  # [j_hi, j_lo]
            T.append(np.exp(1j * axes[comp][d][:, None, None] * q[None]))
        C = c[comp * NF:(comp + 1) * NF].reshape((n,) * 6)  # j6 j5 j4 j3 j2 j1
        t = np.tensordot(C, T[0], axes=([2, 5], [1, 2]))    # j6 j5 j3 j2 x
        t = np.tensordot(t, T[1], axes=([1, 3], [1, 2]))    # j6 j3 x y
        t = np.tensordot(t, T[2], axes=([0, 1], [1, 2]))    # x y z
        ref = t.transpose(2, 1, 0).reshape(-1)
        assert np.linalg.norm(u[comp].cpu().numpy() - ref) < 1e-13 * np.linalg.norm(ref)


@pytest.mark.parametrize("N,sizes,ncomp", [(1, (1, 1, 1), 1), (1, (5, 3, 2), 3), (1, (131072 + 67, 1, 1), 1),
                                           (2, (4, 64, 65), 1), (2, (65, 257, 2), 2), (3, (63, 5, 31), 3),
                                           (4, (3, 33, 1), 1), (5, (66, 2, 33), 2), (6, (7, 9, 5), 1)])
def test_direct_grid_tensor_core_chain(cuda_device, N, sizes, ncomp):
    """Tensor-core contractions whose intermediates are written as split panels: groups of 4 points
    of x and tiles of 64, padded k (n2 = 4, 36, 100), two column tiles (y = 257), more than one slab
    of x (N = 1, 131139 points).  Against the FP64 contractions, relative 4e-6: three chained FP32
    sums of at most 288 truncated products with a bias of at most 288/4 steps of 2^-24 each would
    be 1.3e-5; coefficients of random sign leave a third of it at most."""
    import torch
    import fame_b200 as F
    NF = (2 * N) ** 6
    rng = np.random.default_rng(N)
    sg = F.build_q_system(F.MassBackend(torch.as_tensor(O.material_smooth_exp(N), device=cuda_device), N),
                          F.configs.P_GOLDEN, F.configs.Q_PHYS)
    c = torch.as_tensor(rng.standard_normal(ncomp * NF) + 1j * rng.standard_normal(ncomp * NF), device=cuda_device)
    axes = [tuple(torch.as_tensor(rng.uniform(-1, 1, size=s), device=cuda_device) for s in sizes) for _ in range(ncomp)]
    ref = F.reconstruct_fields_direct_grid(c, sg, axes)
    for _ in range(2):
        u = F.reconstruct_fields_direct_grid(c, sg, axes, tensor_cores=True)
        for comp in range(ncomp):
            assert torch.linalg.norm(u[comp] - ref[comp]) < 4e-6 * torch.linalg.norm(ref[comp])


@pytest.mark.parametrize("axis", [1, 2])
def test_direct_grid_axis_longer_than_one_launch(cuda_device, axis):
    """y or z axes with more column tiles (48 points) than one launch's 65535: the points at both
    ends of each launch against the 64 terms in NumPy, relative 1e-12 (phases of up to 5 radians)."""
    import torch
    import fame_b200 as F
    N, n, edge = 1, 2, 65535 * 48
    P = np.asarray(F.configs.P_GOLDEN)
    sg = F.build_q_system(F.MassBackend(torch.as_tensor(O.material_smooth_exp(N), device=cuda_device), N), P,
                          F.configs.Q_PHYS)
    rng = np.random.default_rng(axis)
    c = rng.standard_normal(64) + 1j * rng.standard_normal(64)
    axes = [rng.uniform(-1, 1, size=edge + 100 if d == axis else 1) for d in range(3)]
    u = F.reconstruct_field_direct_grid(torch.as_tensor(c, device=cuda_device), sg,
                                        [torch.as_tensor(a, device=cuda_device) for a in axes]).cpu().numpy()
    xi = np.array([0.0, -1.0])
    j = np.arange(64)
    k = np.asarray(sg.kLift)
    q = np.zeros((3, 64))
    for ell in range(6):
        q += P[ell][:, None] * (xi[(j >> ell) & 1] + k[ell])[None, :]
    at = np.concatenate([np.arange(50), np.arange(edge - 50, edge + 100)])
    for i in at:
        r = np.array([axes[d][i if d == axis else 0] for d in range(3)])
        ref = np.sum(c * np.exp(1j * (r @ q)))
        assert abs(u[i] - ref) < 1e-12 * np.linalg.norm(c) * 8
