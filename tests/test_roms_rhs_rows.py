"""The ROMS-form 3D right-hand side at the edges of its strips (29 columns) and row runs (8 rows a warp),
FP64 bit for bit against the oracle, FP32 to the rounding of its sums."""
import ctypes

import numpy as np
import pytest

import roms_oracle as ro


@pytest.mark.gpu
@pytest.mark.parametrize("I,J,N", [(6, 6, 5), (29, 8, 6), (30, 9, 5), (31, 32, 7), (58, 33, 5), (59, 40, 6), (88, 65, 5)])
def test_rhs3d_strips(I, J, N):
    import torch
    from sailfish_b200 import configs
    from sailfish_b200._lib import lib
    from sailfish_b200.model import Model
    cfg = configs.basin(I - 2, J - 2, N, 2e3, [], dt=120.0, ndtfast=1, hflat=300.0)
    g = cfg["grid"]
    r = np.random.default_rng(I + J)
    f = lambda n, lo, hi: r.uniform(lo, hi, (n, J, I)).astype(np.float32).astype(np.float64)
    u, v, Hu, Hv, Hz = f(N + 1, -1, 1), f(N + 1, -1, 1), f(N + 1, -1e4, 1e4), f(N + 1, -1e4, 1e4), f(N, 1, 9)
    got = {}
    for prec in ("fp64", "fp32"):
        m = Model(g, cfg["boundary"], 120.0, 1, precision=prec, semantics="roms")
        T = [torch.tensor(a, dtype=m.tdtype, device="cuda") for a in (u, v, Hu, Hv, Hz)]
        out = [torch.full((N + 1, J, I), 7.0, dtype=m.tdtype, device="cuda") for _ in range(2)]
        p = lambda a: ctypes.c_void_p(a.data_ptr())
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert lib.sf_roms_rhs3d(m.ctx.ptr, *[p(a) for a in T + out], st) == 0
        torch.cuda.synchronize()
        got[prec] = [a.double().cpu().numpy() for a in out]
    want = [np.zeros((N + 1) * J * I) for _ in range(2)]
    g.Hz = Hz
    ro.rhs3d(g, u.reshape(-1), v.reshape(-1), Hu.reshape(-1), Hv.reshape(-1), *want)
    for a, b, w in zip(got["fp64"], got["fp32"], want):
        np.testing.assert_array_equal(a.reshape(-1), w)
        # six products of magnitude up to 4e4 (fluxes) and fomn Hz, some 20 roundings
        scale = 6 * 4e4 + 2 * 9 * np.abs(g.fomn).max()
        assert np.abs(b.reshape(-1) - w).max() <= 20 * 2.0 ** -24 * scale
