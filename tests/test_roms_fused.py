"""The fused ROMS-form substep (predictor and corrector in one launch, runs of six substeps) against
the oracle in FP64, bit for bit, at the edges of its tiles (27 columns x 9 rows), with the tile
count on both sides of the switch of its two forms (200 in FP64), and where the caller's slots end."""
import numpy as np
import pytest

import roms_oracle as ro


def _case(I, J):
    from sailfish_b200 import configs
    cfg = configs.basin(I - 2, J - 2, 5, 2e3, [], dt=30.0, ndtfast=1, hflat=400.0)
    g = cfg["grid"]
    r = np.random.default_rng(I * 1000 + J)
    smooth = lambda a: a * (np.sin(g.x / 9e3 + r.uniform(0, 6)) * np.cos(g.y / 7e3 + r.uniform(0, 6)))
    G = dict(h=g.h, pm=g.pm, pn=g.pn, on_u=g.on_u, om_v=g.om_v, fomn=g.fomn)
    S = ro.State(g.J, g.I)
    for k in range(2):
        S.zeta[k][...] = smooth(0.05)
        ro._ring(S.zeta[k])
        S.ubar[k][1:-1, 2:-1] = smooth(0.02)[1:-1, 2:-1]
        S.vbar[k][2:-1, 1:-1] = smooth(0.02)[2:-1, 1:-1]
    return cfg, g, G, S, smooth(1e-4), smooth(1e-4)


@pytest.mark.gpu
@pytest.mark.parametrize("I,J", [(6, 6), (27, 9), (28, 10), (29, 11), (54, 18), (57, 20), (82, 29),
                                 (330, 140), (541, 127)])
def test_fused_substeps_bit_exact(I, J):
    import torch
    from sailfish_b200.model import Model
    cfg, g, G, S, su, sv = _case(I, J)
    m = Model(g, cfg["boundary"], 300.0, 20, precision="fp64", semantics="roms")
    m.set_forcing(su, sv, 3e-3)
    one = Model(g, cfg["boundary"], 300.0, 20, precision="fp64", semantics="roms")
    one.set_forcing(su, sv, 3e-3)
    for x in (m, one):
        for n in ("zeta", "ubar", "vbar"):
            a = np.zeros((3, g.J, g.I))
            a[0], a[1] = getattr(S, n)
            x.load({n: a})
    # 2D steps: one call of 15 (two groups of six fused) against the oracle, and the slots and
    # the scratch level of 15 single calls
    m.step2d(15)
    for _ in range(15):
        one.step2d(1)
    ro.main2d(G, S, 15, m.dtfast, su, sv, 3e-3)
    torch.cuda.synchronize()
    assert m.slots == one.slots
    for n in ("zeta", "ubar", "vbar", "rzeta", "rubar", "rvbar"):
        assert torch.equal(getattr(m, n), getattr(one, n)), n
        for k in range(2):
            np.testing.assert_array_equal(getattr(m, n)[m.slots[k]].cpu().numpy(), getattr(S, n)[k], err_msg=n)
    # the loop with its averages
    st = m.state2d()
    import ctypes
    m._roms_loop(st, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    m._sync_slots(st)
    ro.barotropic_loop(G, S, m.nfast, m.W1, m.W2, m.dtfast, su, sv, 3e-3)
    torch.cuda.synchronize()
    assert m.nfast >= 14
    for n in ("zeta", "ubar", "vbar"):
        for k in range(2):
            np.testing.assert_array_equal(getattr(m, n)[m.slots[k]].cpu().numpy(), getattr(S, n)[k], err_msg=n)
    for n in ("Zt_avg1", "DU_avg1", "DV_avg1", "DU_avg2", "DV_avg2"):
        np.testing.assert_array_equal(getattr(m, n).cpu().numpy().reshape(g.J, g.I), getattr(S, n), err_msg=n)
