"""set_maxflux + omega in FP64 at the sizes between which its forms change (more blocks than two per SM; 37, 40
and 56 levels): the same bits for every chunk length, fused or as two entries."""
import ctypes

import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("Lm,Mm,N", [(280, 275, 6), (280, 275, 37), (280, 275, 38), (150, 170, 37), (40, 30, 56), (280, 275, 57)])
def test_forms_agree(Lm, Mm, N):
    import torch
    from sailfish_b200 import configs
    from sailfish_b200._lib import lib
    from sailfish_b200.model import Model
    cfg = configs.basin(Lm, Mm, N, 2e3, [], dt=120.0, ndtfast=1, hflat=300.0)
    m = Model(cfg["grid"], cfg["boundary"], 120.0, 1, precision="fp64", semantics="roms")
    gen = torch.Generator(device="cuda").manual_seed(N)
    for n in ("u", "v", "Hz", "z_w"):
        a = getattr(m, n)
        a.copy_(2.0 * torch.rand(a.shape, generator=gen, device="cuda", dtype=a.dtype) - (1.0 if n in "uv" else -1.0))
    m.z_w.copy_(m.z_w.cumsum(0))
    p = lambda a: ctypes.c_void_p(a.data_ptr())
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    c, outs = m.ctx.ptr, []
    for chunk in (0, 4, 5, 8):
        for fused in (True, False):
            assert lib.sf_ctx_tune(c, 0, chunk) == 0
            for n in ("Huon", "Hvom", "W"):
                getattr(m, n).zero_()
            if fused:
                assert lib.sf_maxflux_omega(c, p(m.u), p(m.v), p(m.Huon), p(m.Hvom), p(m.Hz), p(m.W), p(m.z_w), None, None,
                                            None, st) == 0
            else:
                assert lib.sf_set_maxflux(c, p(m.u), p(m.v), p(m.Huon), p(m.Hvom), p(m.Hz), st) == 0
                assert lib.sf_omega(c, p(m.W), p(m.Huon), p(m.Hvom), p(m.z_w), st) == 0
            torch.cuda.synchronize()
            outs.append([getattr(m, n).clone() for n in ("Huon", "Hvom", "W")])
    assert all(float(a.abs().max()) > 0 for a in outs[0])
    for o in outs[1:]:
        for a, b in zip(outs[0], o):
            assert torch.equal(a, b)
