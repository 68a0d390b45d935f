"""The fused training passes (one launch for the forward, three for the backward) against the
layer-by-layer ones, which buffers off 16-byte boundaries take: the forward pass and dW bit for bit
(the same products, sums and epilogues), db to the rounding of a sum taken in another order."""
import ctypes

import pytest


def _passes(torch, lib, P, n, X, dY, shift):
    """Y, acts, pre, dW, db of one forward and backward pass; every FP32 buffer `shift` elements
    into its allocation."""
    def buf(*shape):
        m = 1
        for s in shape:
            m *= s
        return torch.full((m + 4,), float("nan"), device="cuda")[shift:shift + m].view(*shape)

    p = lambda t: ctypes.c_void_p(t.data_ptr())
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    tX, tdY, Y, acts, pre, work = buf(n, 128), buf(n, 128), buf(n, 128), buf(4, n, 128), buf(5, n, 128), buf(2, n, 128)
    tX.copy_(X)
    tdY.copy_(dY)
    dW, db = [buf(128, 128) for _ in range(5)], [buf(128) for _ in range(5)]
    ptrs = lambda ts: (ctypes.c_void_p * 5)(*[t.data_ptr() for t in ts])
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert lib.sf_mlp_forward(ctypes.byref(P), n, p(tX), p(Y), p(acts), p(pre), p(err), st) == 0, lib.sf_mlp_last_error()
    assert lib.sf_mlp_backward(ctypes.byref(P), n, p(tX), p(acts), p(pre), p(tdY), ptrs(dW), ptrs(db), p(work),
                               p(err), st) == 0, lib.sf_mlp_last_error()
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    return Y, acts, pre, dW, db


@pytest.mark.gpu
@pytest.mark.parametrize("act", ["gelu", "relu"])
@pytest.mark.parametrize("n", [16, 112, 128, 144, 1040, 2176])   # one tile, remainders, many tiles
def test_fused_passes_match_layer_by_layer(n, act):
    import torch
    from sailfish_b200._lib import MLP_ACT, MlpParams, lib
    gen = torch.Generator(device="cuda").manual_seed(n)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    W = [(r(128, 128) / 128 ** 0.5).to(torch.bfloat16) for _ in range(5)]
    b = [0.05 * r(128) for _ in range(5)]
    P = MlpParams()
    for l in range(5):
        P.W[l], P.b[l] = W[l].data_ptr(), b[l].data_ptr()
    P.act = MLP_ACT[act]
    X, dY = r(n, 128), 1e-2 * r(n, 128)
    fused = _passes(torch, lib, P, n, X, dY, 0)
    plain = _passes(torch, lib, P, n, X, dY, 1)
    for a, c in zip(fused[:3], plain[:3]):
        assert torch.equal(a, c)
    for a, c in zip(fused[3], plain[3]):   # dW: the rows summed in the same order
        assert torch.equal(a, c)
    G = dY.double()   # db: FP32 sums of n values in any order, bound 2 n 2^-24 sum |G|
    for l in range(4, -1, -1):
        if l < 4:
            z = plain[2][l].double().requires_grad_()
            y = torch.nn.functional.gelu(z, approximate="tanh") if act == "gelu" else z.relu()
            G = torch.autograd.grad(y, z, G)[0]
        # 1.02: the G here is not the passes' own to the last BF16 rounding
        bound = 1.02 * 2 * n * 2.0 ** -24 * G.abs().sum(0) + 1e-30
        assert ((fused[4][l] - plain[4][l]).double().abs() <= bound).all(), l
        G = G.float().to(torch.bfloat16).double() @ W[l].double()
