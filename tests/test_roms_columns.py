"""The ROMS-form column solve at every remainder of its level chunks (8, 4, 2, 1 in FP32; 6, 4, 2, 1 in
FP64) and on rows that end inside a block: FP64 bit for bit against the oracle, FP32 within the
rounding of its N-level recurrences of the FP64 result."""
import ctypes

import numpy as np
import pytest

import roms_oracle as ro


@pytest.mark.gpu
@pytest.mark.parametrize("N", [5, 6, 7, 8, 9, 10, 12, 13, 15, 16, 17, 33, 64])
def test_column_solve_levels(N):
    import torch
    from sailfish_b200 import configs
    from sailfish_b200._lib import lib
    from sailfish_b200.model import Model
    cfg = configs.basin(21, 17, N, 2e3, [], dt=120.0, ndtfast=1, hflat=300.0)
    g = cfg["grid"]
    r = np.random.default_rng(N)
    J, I = g.J, g.I
    f = lambda *s, lo, hi: r.uniform(lo, hi, s).astype(np.float32).astype(np.float64)
    Hz = f(N, J, I, lo=2.0, hi=20.0)
    z_r = np.cumsum(Hz, 0) - 0.5 * Hz - Hz.sum(0)
    z_r = z_r.astype(np.float32).astype(np.float64)
    u, v = f(N + 1, J, I, lo=-0.5, hi=0.5), f(N + 1, J, I, lo=-0.5, hi=0.5)
    ru = [f(N + 1, J, I, lo=-2e3, hi=2e3) for _ in range(3)]
    rv = [f(N + 1, J, I, lo=-2e3, hi=2e3) for _ in range(3)]
    Akv, W = f(N + 1, J, I, lo=1e-5, hi=1e-1), f(N + 1, J, I, lo=-5e2, hi=5e2)
    DU, DV = f(J, I, lo=-5e4, hi=5e4), f(J, I, lo=-5e4, hi=5e4)
    got = {}
    for prec in ("fp64", "fp32"):
        m = Model(g, cfg["boundary"], 120.0, 1, precision=prec, semantics="roms")
        t = lambda a: torch.tensor(a, dtype=m.tdtype, device="cuda")
        p = lambda a: ctypes.c_void_p(a.data_ptr())
        F = [t(a) for a in (u, v, *ru, *rv)]
        bars = [torch.full((J, I), 7.0, dtype=m.tdtype, device="cuda") for _ in range(4)]
        G = [t(a) for a in (Hz, Akv, z_r, W)]
        D = [torch.tensor(a.ravel(), device="cuda") for a in (DU, DV)]
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert lib.sf_roms_step3d_uv(m.ctx.ptr, *[p(a) for a in F + bars + G + D], 4, 0, 1.0, 120.0, st) == 0
        torch.cuda.synchronize()
        got[prec] = [a.double().cpu().numpy() for a in F[:2] + bars]
    S = ro.State(J, I)
    S.DU_avg1[...], S.DV_avg1[...] = DU, DV
    uo, vo = u.copy().reshape(-1), v.copy().reshape(-1)
    ro.roms_step3d(g, S, uo, vo, [a.reshape(-1) for a in ru], [a.reshape(-1) for a in rv],
                   ro.ab3_coefficients(4), Hz.reshape(-1), Akv.reshape(-1), z_r.reshape(-1), W.reshape(-1), 120.0, 1.0)
    want = [uo.reshape(N + 1, J, I), vo.reshape(N + 1, J, I), S.ubar[1], S.vbar[1], S.ubar_p, S.vbar_p]
    for k, (a, b) in enumerate(zip(got["fp64"], want)):
        np.testing.assert_array_equal(a, b, err_msg=str(k))
    # FP32: N levels of elimination and of back substitution, some ten roundings each
    for k, (a, b) in enumerate(zip(got["fp32"], want)):
        assert np.abs(a - b).max() <= 20 * N * 2.0 ** -24 * np.abs(b).max(), k
