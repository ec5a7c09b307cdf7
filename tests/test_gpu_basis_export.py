"""Exported basis diagonals at destinations other than a tensor's start: a complex128 array needs
no more than a double's alignment, and what a device copy reaches (host memory) is reached."""
import ctypes as C

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", range(14))
def test_destinations(cuda_device, which):
    import torch
    import fame_b200 as F
    from fame_b200 import _lib as L
    N = 2
    E = O.material_smooth_exp(N)
    sg = F.build_q_system(F.MassBackend(torch.as_tensor(E, device=cuda_device), N), F.configs.P_REFERENCE,
                          F.configs.Q_TRACKING)
    S = O.build_q_system(N, F.configs.P_REFERENCE, F.configs.Q_TRACKING, E)
    words = (2 if which < 9 else 1) * sg.NF
    bufs = [torch.zeros(8 * words + 16, dtype=torch.uint8, device=cuda_device) for _ in range(3)]
    bufs.append(torch.zeros(8 * words + 16, dtype=torch.uint8).pin_memory())
    got = []
    for buf, off in zip(bufs, (0, 8, 4, 8)):
        sg.ctx.bind()
        assert L.lib.fame_basis_get(sg.h, which, C.c_void_p(buf.data_ptr() + off)) == L.FAME_OK
        sg.ctx.sync()
        h = buf.cpu().numpy()
        assert not h[:off].any() and not h[off + 8 * words:].any()
        got.append(h[off:off + 8 * words].tobytes())
    assert all(g == got[0] for g in got)
    v = np.frombuffer(got[0], dtype=np.complex128 if which < 9 else np.float64)
    if which < 6:
        ref = np.asarray([S.V11, S.V21, S.V31, S.V12, S.V22, S.V32][which]).reshape(-1)
        assert np.linalg.norm(v - ref) < 1e-12 * np.linalg.norm(ref)
