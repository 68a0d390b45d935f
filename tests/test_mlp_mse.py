"""sf_mlp_mse over its range of valid columns, none included (a zero gradient and no loss), on buffers on and
off 16-byte boundaries; columns past the valid ones may hold anything."""
import ctypes

import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n,nvalid", [(16, 0), (48, 1), (112, 63), (1040, 98), (16, 128)])
def test_valid_columns(n, nvalid, shift):
    import torch
    from sailfish_b200._lib import lib
    gen = torch.Generator(device="cuda").manual_seed(n + nvalid)
    new = lambda: torch.full((n * 128 + 4,), float("nan"), device="cuda")[shift:shift + n * 128].view(n, 128)
    Y, T, dY = new(), new(), new()
    for a in (Y, T):
        a[:, :nvalid] = torch.randn(n, nvalid, generator=gen, device="cuda")
    loss = torch.full((1,), 3.0, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    assert lib.sf_mlp_mse(n, nvalid, p(Y), p(T), p(dY), p(loss), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert torch.equal(dY[:, nvalid:], torch.zeros(n, 128 - nvalid, device="cuda"))
    if nvalid == 0:
        assert float(loss) == 3.0
        return
    d = (Y - T)[:, :nvalid]
    # one rounding each of the difference, the product with 2 (none) and the quotient (by a tensor: torch
    # divides by a number by multiplying with its reciprocal)
    assert torch.equal(dY[:, :nvalid], torch.div(2.0 * d, torch.full_like(d, n * nvalid)))
    want = 3.0 + float((d.double() ** 2).mean())
    # FP32 sums of at most n nvalid positive terms, each within 2 roundings, and the atomics onto 3
    assert abs(float(loss) - want) <= (n * nvalid + 150) * 2.0 ** -24 * want
