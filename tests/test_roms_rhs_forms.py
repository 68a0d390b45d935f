"""The forms of the ROMS-form 3D right-hand side: by strips (8 rows a warp; 32 from 2^20 points; ensembles as the
barotropic phases) and by points, which basins of few columns take, the same bits; by points in FP64 against
the oracle."""
import ctypes

import numpy as np
import pytest

import roms_oracle as ro


def _run(m, put):
    import torch
    from sailfish_b200._lib import check, lib
    p = lambda a: ctypes.c_void_p(a.data_ptr())
    put(m)
    for n in ("ru", "rv"):
        getattr(m, n).fill_(7.0)
    check(lib.sf_roms_rhs3d(m.ctx.ptr, p(m.u), p(m.v), p(m.Huon), p(m.Hvom), p(m.Hz), p(m.ru), p(m.rv),
                            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "sf_roms_rhs3d")
    torch.cuda.synchronize()


def _data(g, k):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(100 * k + g.I)
    f = lambda n, s, o: s * torch.rand(n, g.J, g.I, generator=gen, device="cuda", dtype=torch.float64) + o
    return dict(u=f(g.N + 1, 2.0, -1.0), v=f(g.N + 1, 2.0, -1.0), Huon=f(g.N + 1, 2e4, -1e4), Hvom=f(g.N + 1, 2e4, -1e4),
                Hz=f(g.N, 8.0, 1.0))


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("sizes", [((5, 60, 6), (58, 400, 9)),         # strips; the first alone by points
                                   ((6, 300, 7), (58, 9, 5)),          # points; the second alone by strips
                                   ((6, 6000, 9), (5, 90, 5)),         # points, four threads a column
                                   ((1100, 960, 5), (90, 31, 6))])     # 8 rows a warp; the first alone 32
def test_members_equal_single_basins(sizes, prec):
    import torch
    from sailfish_b200 import configs, ensemble
    from sailfish_b200.model import Model
    cfgs = [configs.basin(I - 2, J - 2, N, 2e3, [], dt=120.0, ndtfast=1, hflat=300.0) for I, J, N in sizes]
    data = [_data(c["grid"], k) for k, c in enumerate(cfgs)]

    def put_members(e):
        for k, d in enumerate(data):
            for n, a in d.items():
                t = e.member(n, k)
                t.copy_(a.reshape(t.shape))

    e = ensemble.Ensemble([(c["grid"], c["boundary"]) for c in cfgs], 120.0, 1, prec, semantics="roms")
    _run(e, put_members)
    for k, c in enumerate(cfgs):
        def put(m):
            for n, a in data[k].items():
                t = getattr(m, n)
                t.copy_(a.reshape(t.shape))

        m = Model(c["grid"], c["boundary"], 120.0, 1, precision=prec, semantics="roms")
        _run(m, put)
        for n in ("ru", "rv"):
            assert torch.equal(getattr(m, n).reshape(-1), e.member(n, k).reshape(-1)), (k, n)


@pytest.mark.gpu
@pytest.mark.parametrize("I,J,N", [(5, 5, 5), (6, 47, 6), (12, 40, 5), (6, 6000, 9), (5, 53000, 7)])
def test_point_form_bit_exact(I, J, N):
    from sailfish_b200 import configs
    from sailfish_b200.model import Model
    cfg = configs.basin(I - 2, J - 2, N, 2e3, [], dt=120.0, ndtfast=1, hflat=300.0)
    g = cfg["grid"]
    d = _data(g, 3)

    def put(m):
        for n, a in d.items():
            t = getattr(m, n)
            t.copy_(a.reshape(t.shape))

    m = Model(g, cfg["boundary"], 120.0, 1, precision="fp64", semantics="roms")
    _run(m, put)
    want = [np.zeros((N + 1) * J * I) for _ in range(2)]
    h = {n: a.cpu().numpy() for n, a in d.items()}
    g.Hz = h["Hz"]
    ro.rhs3d(g, *[h[n].reshape(-1) for n in ("u", "v", "Huon", "Hvom")], *want)
    for n, w in zip(("ru", "rv"), want):
        np.testing.assert_array_equal(getattr(m, n).cpu().numpy().reshape(-1), w, err_msg=n)
