"""FP64 Taylor moments as matrix products: every column-tile and center-tile shape of the
dispatch (orders 0..12, 1..40 centers, mode counts that leave ragged slices) against the
oracle's moments evaluated with NumPy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _numpy_taylor(c, Q, R, p, ptr, ids):
    import math
    al = [(a, b, d) for a in range(p + 1) for b in range(p + 1 - a) for d in range(p + 1 - a - b)]
    u = np.zeros(R.shape[0], dtype=complex)
    pw = [[Q[:, d] ** k for k in range(p + 1)] for d in range(3)]
    M = np.stack([pw[0][a] * pw[1][b] * pw[2][e] for a, b, e in al], 1)
    coef = np.array([1j ** (a + b + e) / (math.factorial(a) * math.factorial(b) * math.factorial(e)) for a, b, e in al])
    for k in range(len(ptr) - 1):
        i = ids[ptr[k]:ptr[k + 1]]
        if i.size == 0:
            continue
        cen = 0.5 * (R[i].min(0) + R[i].max(0))
        g = coef * ((c * np.exp(1j * (Q @ cen))) @ M)
        D = R[i] - cen
        dw = [[D[:, d] ** k2 for k2 in range(p + 1)] for d in range(3)]
        u[i] = np.stack([dw[0][a] * dw[1][b] * dw[2][e] for a, b, e in al], 1) @ g
    return u


# orders: 1..57 column tiles; centers: both thresholds of the row tiles (2/3, 8/9, 16/17, 32/33)
@pytest.mark.parametrize("p,nB,NF", [(0, 3, 1), (1, 3, 31), (2, 8, 33), (3, 9, 200), (4, 16, 1000), (5, 17, 129),
                                     (6, 2, 5000), (7, 32, 700), (8, 33, 2049), (9, 5, 300), (10, 40, 4097),
                                     (10, 9, 257), (11, 8, 300), (11, 20, 300), (12, 3, 100), (12, 12, 100),
                                     (12, 33, 515), (10, 1, 20000)])
def test_taylor_moments_shapes(cuda_device, p, nB, NF):
    """Sums of NF terms of size <= |q|^p |r|^p / p! with |q| <= 3, |r| <= 1: relative 1e-12 of the field's norm."""
    import torch
    import fame_b200 as F
    rng = np.random.default_rng(100 * p + nB)
    Q = rng.uniform(-3, 3, size=(NF, 3))
    c = rng.standard_normal(NF) + 1j * rng.standard_normal(NF)
    R = rng.uniform(-1, 1, size=(37 * nB + 5, 3))
    order = rng.permutation(R.shape[0])
    cuts = np.sort(rng.choice(np.arange(1, R.shape[0]), size=nB - 1, replace=False))
    ptr = np.concatenate([[0], cuts, [R.shape[0]]]).astype(np.int64)
    if nB > 4:
        ptr[3] = ptr[2]  # an empty block
    dev = cuda_device
    Qd = torch.as_tensor(Q.T.copy(), device=dev).t()
    Rd = torch.as_tensor(R.T.copy(), device=dev).t()
    u = F.taylor_on_blocks(torch.as_tensor(c, device=dev), Qd, Rd, p,
                           (torch.as_tensor(ptr, device=dev), torch.as_tensor(order.astype(np.int64), device=dev)))
    ref = _numpy_taylor(c, Q, R, p, ptr, order)
    assert np.linalg.norm(u.cpu().numpy() - ref) < 1e-12 * np.linalg.norm(ref)


def test_phase_reduction_at_large_arguments(cuda_device):
    """Phases beyond the two-term reduction's range (2^19 pi/2) and at multiples of pi/2, order 0:
    the moment is c e^{i q.r}, exact to the rounding of q.r itself (bound 1e-12 for products
    computed from exactly representable factors)."""
    import torch
    import fame_b200 as F
    vals = np.array([0.0, 0.5, 2.0 ** 19, 2.0 ** 20, 2.0 ** 24 + 1, 3.0, 12345.0, 823549.0, 823550.0])
    for v in vals:
        Q = np.array([[v, 0.0, 0.0]] * 2)
        R = np.concatenate([np.full((4, 3), s) for s in (1.0, -1.0, 0.5, -0.25)])
        ptr = np.arange(0, 17, 4).astype(np.int64)
        u = F.taylor_on_blocks(torch.tensor([1.0 + 0j, 0.5j], device=cuda_device, dtype=torch.complex128),
                               torch.as_tensor(Q.T.copy(), device=cuda_device).t(),
                               torch.as_tensor(R.T.copy(), device=cuda_device).t(), 0,
                               (torch.as_tensor(ptr, device=cuda_device),
                                torch.arange(16, device=cuda_device, dtype=torch.int64)))
        ref = (1 + 0.5j) * np.exp(1j * v * R[:, 0])
        assert np.max(np.abs(u.cpu().numpy() - ref)) < 1e-12


def test_phase_accuracy_around_multiples_of_half_pi(cuda_device):
    """e^{ix} at and within a few ulp of multiples of pi/2 and of the octant boundaries between them,
    up to and past the end of the reduction (2^19 pi/2), against 80-bit sin and cos: absolute error
    below 3e-16 (half an ulp each of the reduced argument, of the result and of the polynomials'
    last products, 5.6e-17 at most).  One point per block makes the block's center the point, and
    at order 0 the field is the phase."""
    import torch
    import fame_b200 as F
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no 80-bit reference")
    rng = np.random.default_rng(9)
    k = np.unique(np.concatenate([np.arange(300), 2 ** np.arange(0, 20), rng.integers(1, 2 ** 19, 900),
                                  2 ** 19 - np.arange(12)]))
    half_pi = (np.longdouble(np.pi) + np.longdouble(1.2246467991473532e-16)) / 2
    x = np.concatenate([k * half_pi, (k + 0.5) * half_pi]).astype(np.float64)
    x = np.concatenate([x, np.nextafter(x, np.inf), np.nextafter(x, -np.inf), x * (1 + 3 * 2.0 ** -52),
                        rng.uniform(-40, 40, 2000), [823549.0, np.nextafter(823549.0, 0), 1e6, 1e300]])
    x = np.concatenate([x, -x])
    assert x.size < 65536
    M = x.size
    R = np.zeros((3, M))
    R[0] = x
    Q = np.zeros((3, 2))
    Q[0] = 1.0
    u = F.taylor_on_blocks(torch.tensor([1.0, 0.0], device=cuda_device, dtype=torch.complex128),
                           torch.as_tensor(Q, device=cuda_device).t(), torch.as_tensor(R, device=cuda_device).t(), 0,
                           (torch.arange(M + 1, device=cuda_device, dtype=torch.int64),
                            torch.arange(M, device=cuda_device, dtype=torch.int64))).cpu().numpy()
    xl = x.astype(np.longdouble)
    small = np.abs(x) < 2.0 ** 60  # the 80-bit functions reduce arguments up to 2^63
    err = np.maximum(np.abs(u.real - np.cos(xl)), np.abs(u.imag - np.sin(xl)))[small]
    assert float(err.max()) < 3e-16
    ref = np.stack([np.cos(x), np.sin(x)])[:, ~small]
    assert np.max(np.abs(np.stack([u.real, u.imag])[:, ~small] - ref)) < 3e-16
