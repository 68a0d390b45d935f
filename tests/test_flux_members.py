"""set_maxflux + omega in FP32: a member of an ensemble gives the bits of its basin alone (the chunked form on both
sides)."""
import ctypes

import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("N", [(5, 16), (32, 33), (50, 64)])
def test_members_equal_single_basins(N):
    import torch
    from sailfish_b200 import configs, ensemble
    from sailfish_b200._lib import lib
    from sailfish_b200.model import Model
    cfgs = [configs.basin(40 + 21 * k, 31 - 8 * k, n, 2e3, [], dt=120.0, ndtfast=1, hflat=300.0) for k, n in enumerate(N)]
    p = lambda a: ctypes.c_void_p(a.data_ptr())

    def run(m):
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert lib.sf_maxflux_omega(m.ctx.ptr, p(m.u), p(m.v), p(m.Huon), p(m.Hvom), p(m.Hz), p(m.W), p(m.z_w), None, None,
                                    None, st) == 0
        torch.cuda.synchronize()

    e = ensemble.Ensemble([(c["grid"], c["boundary"]) for c in cfgs], 120.0, 1, "fp32", semantics="roms")
    alone = []
    for k, c in enumerate(cfgs):
        g = c["grid"]
        m = Model(g, c["boundary"], 120.0, 1, precision="fp32", semantics="roms")
        gen = torch.Generator(device="cuda").manual_seed(g.N)
        f = lambda n, s, o: s * torch.rand(n, g.J, g.I, generator=gen, device="cuda") + o
        for n, a in dict(u=f(g.N + 1, 2.0, -1.0), v=f(g.N + 1, 2.0, -1.0), Hz=f(g.N, 8.0, 1.0),
                         z_w=f(g.N + 1, 8.0, 1.0).cumsum(0)).items():
            getattr(m, n).copy_(a.reshape(getattr(m, n).shape))
            e.member(n, k).copy_(a.reshape(e.member(n, k).shape))
        run(m)
        alone.append(m)
    run(e)
    for k, m in enumerate(alone):
        for n in ("Huon", "Hvom", "W"):
            assert torch.equal(getattr(m, n).reshape(-1), e.member(n, k).reshape(-1)), (k, n)
