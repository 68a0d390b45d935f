"""set_maxflux + omega at every remainder of its level chunks: FP64 the same bits for every chunk length
(0: one level at a time), fused or as two entries, on a single grid and on a member of an ensemble."""
import ctypes

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("N", [5, 6, 7, 8, 9, 10, 13, 17, 32, 33, 50, 64])
def test_chunk_lengths_agree(N):
    import torch
    from sailfish_b200 import configs, ensemble
    from sailfish_b200._lib import lib
    from sailfish_b200.model import Model
    cfg = configs.basin(26, 19, N, 2e3, [], dt=120.0, ndtfast=1, hflat=300.0)
    g = cfg["grid"]
    r = np.random.default_rng(N)
    f = lambda n, lo, hi: r.uniform(lo, hi, (n, g.J, g.I))
    data = dict(u=f(N + 1, -1, 1), v=f(N + 1, -1, 1), Hz=f(N, 1, 9), z_w=np.cumsum(f(N + 1, 1, 9), 0))
    p = lambda a: ctypes.c_void_p(a.data_ptr())
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    outs = []

    def run(m, put, get, chunk, fused):
        for n, a in data.items():
            put(n, torch.tensor(a, device="cuda"))
        assert lib.sf_ctx_tune(m.ctx.ptr, 0, chunk) == 0
        c = m.ctx.ptr
        if fused:
            assert lib.sf_maxflux_omega(c, p(m.u), p(m.v), p(m.Huon), p(m.Hvom), p(m.Hz), p(m.W), p(m.z_w), None, None,
                                        None, st) == 0
        else:
            assert lib.sf_set_maxflux(c, p(m.u), p(m.v), p(m.Huon), p(m.Hvom), p(m.Hz), st) == 0
            assert lib.sf_omega(c, p(m.W), p(m.Huon), p(m.Hvom), p(m.z_w), st) == 0
        torch.cuda.synchronize()
        outs.append([get(n).clone() for n in ("Huon", "Hvom", "W")])

    for chunk in (0, 4, 5, 8):
        for fused in (True, False):
            m = Model(g, cfg["boundary"], 120.0, 1, precision="fp64", semantics="roms")
            run(m, lambda n, a: getattr(m, n).copy_(a), lambda n: getattr(m, n), chunk, fused)
    other = configs.basin(31, 12, 5, 2e3, [], dt=120.0, ndtfast=1, hflat=300.0)
    for chunk in (0, 4):
        e = ensemble.Ensemble([(other["grid"], other["boundary"]), (g, cfg["boundary"])], 120.0, 1, "fp64", semantics="roms")
        run(e, lambda n, a: e.member(n, 1).copy_(a), lambda n: e.member(n, 1), chunk, True)
    for o in outs[1:]:
        for a, b in zip(outs[0], o):
            assert torch.equal(a, b)
