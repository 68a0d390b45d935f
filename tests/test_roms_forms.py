"""The forms of the ROMS-form barotropic substep (one launch on tiles, two by strips, four by points) against each
other, bit for bit in both precisions, and the point form against the oracle: which form runs follows the
grid's shape and the number of substeps, and members of an ensemble take the form of the whole."""
import ctypes

import numpy as np
import pytest

import roms_oracle as ro

# columns x rows: wide (tiles; phases by strips, in FP64 by points), narrow and long (points), narrow and shorter
# (tiles; points in an ensemble with the longer), a small basin (tiles and strips)
WIDE, LONG, THIN, PLAIN = (1000, 700), (5, 12000), (28, 4000), (300, 200)


def _basin(I, J):
    from sailfish_b200 import configs
    return configs.basin(I - 2, J - 2, 5, 2e3, [], dt=30.0, ndtfast=1, hflat=400.0)


def _load(m, k, g, put):
    import torch
    i = torch.arange(g.I, device="cuda", dtype=torch.float64)[None, :]
    j = torch.arange(g.J, device="cuda", dtype=torch.float64)[:, None]
    put("zeta", 0.05 * torch.sin(j / 17.0 + k) * torch.cos(i / 5.0))
    put("ubar", 0.02 * torch.cos(j / 11.0) * torch.sin(i / 7.0 + k))
    put("vbar", 0.02 * torch.sin(j / 13.0 + k) * torch.cos(i / 3.0))
    put("sustr", 1e-4 * torch.cos(j / 19.0) + 0 * i)
    put("svstr", 5e-5 * torch.sin(i / 9.0) + 0 * j)


def _single(I, J, prec, nd=20):
    from sailfish_b200.model import Model
    cfg = _basin(I, J)
    m = Model(cfg["grid"], cfg["boundary"], 300.0, nd, precision=prec, semantics="roms")
    m.rdrag2 = 3e-3

    def put(n, a):
        f = getattr(m, n)
        for t in (f if n in m.NAMES2 else [f]):
            t.copy_(a.reshape(t.shape))

    _load(m, 0, cfg["grid"], put)
    return m


def _ensemble(sizes, prec, nd=20):
    from sailfish_b200 import ensemble
    cfgs = [_basin(*s) for s in sizes]
    e = ensemble.Ensemble([(c["grid"], c["boundary"]) for c in cfgs], 300.0, nd, prec, semantics="roms")
    e.rdrag2 = 3e-3
    for k, c in enumerate(cfgs):
        o, s2 = e.ctx.off2[k], c["grid"].s2

        def put(n, a):
            f = getattr(e, n)
            for t in (f if n in e.NAMES2 else [f]):
                t[o:o + s2] = a.reshape(-1)

        _load(e, 0, c["grid"], put)
    return e


def _loop(m):
    import torch
    s = m.state2d()
    m._roms_loop(s, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    m._sync_slots(s)


FIELDS = ("zeta", "ubar", "vbar")
SUMS = ("Zt_avg1", "DU_avg1", "DV_avg1", "DU_avg2", "DV_avg2")


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("size", [WIDE, LONG, THIN, PLAIN, (640, 420), (1200, 900)])
def test_runs_equal_single_steps(size, prec):
    """15 steps in one call (two groups of six fused where tiles run) and in 15 calls."""
    import torch
    a, b = _single(*size, prec), _single(*size, prec)
    a.step2d(15)
    for _ in range(15):
        b.step2d(1)
    torch.cuda.synchronize()
    assert a.slots == b.slots
    for n in FIELDS + ("rzeta", "rubar", "rvbar"):
        assert torch.equal(getattr(a, n), getattr(b, n)), n
    assert float(a.vbar.abs().max()) > 0 and bool(torch.isfinite(a.zeta).all())


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,prec", [((WIDE, LONG, PLAIN), "fp32"), ((WIDE, (5, 6000), PLAIN), "fp64"),
                                        ((LONG, THIN), "fp32"), ((LONG, THIN), "fp64")])
def test_members_equal_single_basins(sizes, prec):
    """2D steps and a loop with its averages: the ensembles with the wide basin go by tiles (their long member alone
    by points), the others by points (their other member alone by tiles)."""
    import torch
    e = _ensemble(sizes, prec)
    e.step2d(9)
    _loop(e)
    for k, size in enumerate(sizes):
        m = _single(*size, prec)
        m.step2d(9)
        _loop(m)
        torch.cuda.synchronize()
        o, s2 = e.ctx.off2[k], size[0] * size[1]
        assert m.slots == e.slots
        for n in FIELDS:
            for t in (0, 1):
                assert torch.equal(getattr(m, n)[m.slots[t]].reshape(-1), getattr(e, n)[e.slots[t]][o:o + s2]), (size, n, t)
        for n in SUMS:
            assert torch.equal(getattr(m, n).reshape(-1), getattr(e, n)[o:o + s2]), (size, n)


@pytest.mark.gpu
@pytest.mark.parametrize("I,J", [(5, 12000), (640, 420)])
def test_point_form_bit_exact(I, J):
    """FP64 at sizes whose phases go by points (the first's loop too) against the oracle."""
    import torch
    m = _single(I, J, "fp64")
    g = m.grid
    G = dict(h=g.h, pm=g.pm, pn=g.pn, on_u=g.on_u, om_v=g.om_v, fomn=g.fomn)
    S = ro.State(g.J, g.I)
    for k in range(2):
        for n in FIELDS:
            getattr(S, n)[k][...] = getattr(m, n)[k].cpu().numpy().reshape(g.J, g.I)
    su, sv = (getattr(m, n).cpu().numpy().reshape(g.J, g.I) for n in ("sustr", "svstr"))
    m.step2d(9)
    ro.main2d(G, S, 9, m.dtfast, su, sv, 3e-3)
    _loop(m)
    ro.barotropic_loop(G, S, m.nfast, m.W1, m.W2, m.dtfast, su, sv, 3e-3)
    torch.cuda.synchronize()
    for n in FIELDS:
        for k in range(2):
            np.testing.assert_array_equal(getattr(m, n)[m.slots[k]].cpu().numpy().reshape(g.J, g.I), getattr(S, n)[k], err_msg=n)
    for n in SUMS:
        np.testing.assert_array_equal(getattr(m, n).cpu().numpy().reshape(g.J, g.I), getattr(S, n), err_msg=n)


def _launches(m):
    """Kernel nodes of a captured loop."""
    import torch
    _loop(m)
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        _loop(m)
    n = ctypes.c_size_t()
    assert ctypes.CDLL("libcuda.so.1").cuGraphGetNodes(ctypes.c_void_p(g.raw_cuda_graph()), None, ctypes.byref(n)) == 0
    return n.value


@pytest.mark.gpu
@pytest.mark.parametrize("size,prec,nd,want", [
    (PLAIN, "fp32", 1, None), (PLAIN, "fp32", 4, None), (PLAIN, "fp32", 5, None), (PLAIN, "fp32", 9, None),
    (PLAIN, "fp32", 10, None), (PLAIN, "fp64", 30, None), (LONG, "fp32", 9, 4), (WIDE, "fp64", 9, None)])
def test_loop_launches_counted(size, prec, nd, want):
    """Model.loop_launches, which the bench counts with, against the launches that a loop makes; want: launches of
    every substep, where none runs fused."""
    m = _single(*size, prec, nd)
    assert m.loop_launches == _launches(m)
    if want:
        assert m.loop_launches == want * m.nfast + 1
