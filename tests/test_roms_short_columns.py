"""The ROMS-form column solve of ensembles, whose form follows the members' largest N (up to 16 levels, and
more): each member equals the same basin alone, bit for bit, though alone it may take the other form."""
import ctypes

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("N", [(5, 16), (7, 17), (16, 64)])
def test_members_equal_single_basins(N, prec):
    import torch
    from sailfish_b200 import configs, ensemble
    from sailfish_b200._lib import check, lib
    from sailfish_b200.model import Model
    cfgs = [configs.basin(19 + 9 * k, 23 - 6 * k, n, 2e3, [], dt=120.0, ndtfast=1, hflat=300.0) for k, n in enumerate(N)]
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    st = lambda: ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

    def solve(m, rs):
        check(lib.sf_roms_step3d_uv(m.ctx.ptr, p(m.u), p(m.v), *[p(t) for t in rs], p(m.ubar[1]), p(m.vbar[1]),
                                    p(m.ubar[2]), p(m.vbar[2]), p(m.Hz), p(m.AKv), p(m.z_r), p(m.W), p(m.DU_avg1),
                                    p(m.DV_avg1), 5, 0, 1.0, 120.0, st()), "sf_roms_step3d_uv")

    e = ensemble.Ensemble([(c["grid"], c["boundary"]) for c in cfgs], 120.0, 1, prec, semantics="roms")
    ers = [torch.zeros_like(e.ru) for _ in range(6)]
    alone = []
    for k, c in enumerate(cfgs):
        g = c["grid"]
        m = Model(g, c["boundary"], 120.0, 1, precision=prec, semantics="roms")
        r = np.random.default_rng(10 * k + g.N)
        f = lambda n, lo, hi: torch.tensor(r.uniform(lo, hi, (n, g.J, g.I)), device="cuda")
        Hz = f(g.N, 2.0, 20.0)
        data = dict(u=f(g.N + 1, -0.5, 0.5), v=f(g.N + 1, -0.5, 0.5), Hz=Hz, z_r=Hz.cumsum(0) - 0.5 * Hz,
                    AKv=f(g.N + 1, 1e-5, 1e-1), W=f(g.N + 1, -5e2, 5e2), DU_avg1=f(1, -5e4, 5e4), DV_avg1=f(1, -5e4, 5e4))
        rs = []
        for n, a in data.items():
            getattr(m, n).copy_(a.reshape(getattr(m, n).shape))
            e.member(n, k).copy_(a.reshape(e.member(n, k).shape))
        for q in range(6):
            a = f(g.N + 1, -2e3, 2e3)
            rs.append(a.to(m.tdtype))
            o = e.ctx.off3[k]
            ers[q][o:o + a.numel()] = a.to(m.tdtype).reshape(-1)
        solve(m, rs)
        alone.append(m)
    solve(e, ers)
    torch.cuda.synchronize()
    for k, m in enumerate(alone):
        for n in ("u", "v"):
            assert torch.equal(getattr(m, n).reshape(-1), e.member(n, k).reshape(-1)), (k, n)
        o, s2 = e.ctx.off2[k], m.grid.s2
        for n in ("ubar", "vbar"):
            for slot in (1, 2):
                assert torch.equal(getattr(m, n)[slot].reshape(-1), getattr(e, n)[slot][o:o + s2]), (k, n, slot)
