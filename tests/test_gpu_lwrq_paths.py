"""LWRQ paths beside the axis-block material: general cut matrices, a zero row, windows smaller
than the Gaussian and ragged tile edges, and eigenvalue guesses far from the field's own (the
residual's second pass), against the oracle; the refusals."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu

KEYS = ("lambdaCrop", "lambda3D", "eta3D", "etaUsing6DLambda", "deltaLambda", "VLWRQ", "nuLWRQ", "croppedMass")


def _fields(n, h, seed, noise):
    """A smooth transverse plane wave per component (small residual) plus noise."""
    rng = np.random.default_rng(seed)
    m = 2 * n + 3
    x = (np.arange(m) - (n + 1)) * h
    out = []
    for c in range(3):
        k = rng.uniform(-3, 3, 3)
        f = np.exp(1j * (k[0] * x[:, None, None] + k[1] * x[None, :, None] + k[2] * x[None, None, :]))
        out.append(f * (1 + 0.3 * c) + noise * (rng.standard_normal((m,) * 3) + 1j * rng.standard_normal((m,) * 3)))
    return out


def _P(kind):
    import fame_b200 as F
    if kind == "block":
        return F.configs.P_REFERENCE
    rng = np.random.default_rng(3)
    P = rng.uniform(-1, 1, size=(6, 3))
    if kind == "zero_row":
        P = np.vstack([np.eye(3), np.zeros((1, 3)), np.diag([1.3, 0.7, 1.9])[1:]])
    return P


@pytest.mark.parametrize("n", [1, 2, 7, 16, 19])
@pytest.mark.parametrize("kind", ["block", "general", "zero_row"])
@pytest.mark.parametrize("material", [("exp", 4.0, 1.2), ("cos", 12.0)])
def test_lwrq_against_oracle(cuda_device, n, kind, material):
    """FP64 sums of (2n+1)^3 terms: 1e-11 relative (the residuals are formed from sums that lose
    at most two bits, or directly)."""
    import fame_b200 as F
    h, P = 0.05, _P(kind)
    for noise, lam6 in ((0.0, 1e-3), (0.0, 1.0), (0.5, 0.05), (0.0, 1e4)):
        u = _fields(n, h, 10 * n, noise)
        ref, sref = O.compute_yee_lwrq_metrics(*u, lam6, P, n, h, material, save_spatial=True)
        dev = [torch.as_tensor(f.reshape(-1, order="F"), device=cuda_device) for f in u]
        met, sp = F.compute_yee_lwrq_metrics(dev, lam6, P, n, h, material, save_spatial=True)
        for k in KEYS:
            np.testing.assert_allclose(met[k], ref[k], rtol=1e-11, err_msg=k)
        # the spread of rho about lambda3D carries rho's rounding
        for k in ("relativeDeviation_z0", "relativeDeviation_x0"):
            np.testing.assert_allclose(sp[k], sref[k], rtol=1e-10, atol=1e-12)
        # lambda6D = lambda3D: both residuals agree
        met2, none = F.compute_yee_lwrq_metrics(dev, ref["lambda3D"], P, n, h, material)
        np.testing.assert_allclose(met2["eta3D"], ref["eta3D"], rtol=1e-11)
        assert none is None


def test_lwrq_refusals(cuda_device):
    import fame_b200 as F
    n = 4
    m = 2 * n + 3
    zero = [torch.zeros(m ** 3, dtype=torch.complex128, device=cuda_device) for _ in range(3)]
    with pytest.raises(F.FameError) as e:  # no mass
        F.compute_yee_lwrq_metrics(zero, 0.05, F.configs.P_GOLDEN, n, 0.05, ("cos", 12.0))
    assert e.value.status == F._lib.FAME_ERR_INVALID
    part = [z.clone() for z in zero]
    for p in part:  # mass in one corner only: empty windows elsewhere
        p.view(m, m, m)[:4, :4, :4] = 1.0
    with pytest.raises(F.FameError) as e:
        F.compute_yee_lwrq_metrics(part, 0.05, F.configs.P_GOLDEN, n, 0.05, ("cos", 12.0))
    assert e.value.status == F._lib.FAME_ERR_NONFINITE
    bad = [torch.full_like(z, float("nan")) for z in zero]
    with pytest.raises(F.FameError) as e:
        F.compute_yee_lwrq_metrics(bad, 0.05, F.configs.P_GOLDEN, n, 0.05, ("cos", 12.0))
    assert e.value.status == F._lib.FAME_ERR_INVALID


@pytest.mark.parametrize("n", [1, 4, 9, 20])
def test_slices_in_both_layouts(cuda_device, n):
    """Python hands the slices out as C-contiguous arrays; the C entry's column-major slices hold
    the same values."""
    import ctypes as C
    import torch
    import fame_b200 as F
    from fame_b200 import _lib as L
    m, q = 2 * n + 3, 2 * n + 1
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    us = [torch.complex(torch.randn(m ** 3, dtype=torch.float64, device="cuda", generator=g),
                        torch.randn(m ** 3, dtype=torch.float64, device="cuda", generator=g)) for _ in range(3)]
    P = np.asarray(F.configs.P_GOLDEN, dtype=np.float64)
    _, sp = F.compute_yee_lwrq_metrics(us, 0.05, P, n, 0.0125, ("cos", 12.0), save_spatial=True)
    cols = [np.empty((q, q), order="F") for _ in range(2)]
    ctx = F.core.default_context()
    out = (C.c_double * 10)()
    dp = C.POINTER(C.c_double)
    F._lib.call("fame_yee_lwrq_metrics", ctx.bind(), *[C.c_void_p(u.data_ptr()) for u in us], n, 0.0125,
                (C.c_double * 18)(*P.reshape(6, 3).ravel(order="F")), 1, 12.0, 0.0, 0.05, out,
                *[a.ctypes.data_as(dp) for a in cols])
    for a, key in zip(cols, ("relativeDeviation_z0", "relativeDeviation_x0")):
        assert sp[key].flags.c_contiguous and sp[key].shape == (q, q)
        assert np.array_equal(sp[key], a)
