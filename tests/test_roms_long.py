"""ROMS-form 2D steps on basins with more rows than 65,535 tiles of 9 (the fused substep) or 65,535 blocks
of 32 rows (the two phases) hold: a run of steps in one call equals as many single calls, bit for bit."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("I,J", [(26, 589830), (5, 2097190)])
def test_long_basins_run(I, J):
    import torch
    from sailfish_b200 import configs
    from sailfish_b200.model import Model
    cfg = configs.basin(I - 2, J - 2, 5, 2e3, [], dt=30.0, ndtfast=1, hflat=400.0)
    g = cfg["grid"]
    out = []
    for calls in ((8,), (1,) * 8):
        m = Model(g, cfg["boundary"], 300.0, 20, precision="fp32", semantics="roms")
        j = torch.arange(J, device="cuda", dtype=torch.float64)[:, None]
        z = (0.05 * torch.sin(j / 37.0) * torch.cos(torch.arange(I, device="cuda") / 3.0)).float()
        for k in range(3):
            m.zeta[k].copy_(z.view(m.zeta[k].shape))
        m.sustr.fill_(1e-4)
        m.rdrag2 = 3e-3
        for n in calls:
            m.step2d(n)
        torch.cuda.synchronize()
        out.append([getattr(m, n)[m.slots[1]] for n in ("zeta", "ubar", "vbar")])
        assert float(out[-1][2].abs().max()) > 0
    for a, b in zip(*out):
        assert torch.equal(a, b)
