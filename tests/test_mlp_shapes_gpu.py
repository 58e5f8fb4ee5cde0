"""The surrogate network's layer products at ragged batch and layer sizes
(remainders of the 32 x 32 output tiles and 32-deep K slices, one partial
tile, unaligned operands) against the FP64 oracle."""
import numpy as np
import pytest
import torch

from augurv2_b200 import hlrb as H
from oracle import batched as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,h1,h2,Bn,pad", [(8, 8, 8, 1, 0), (16, 24, 40, 31, 0), (40, 32, 64, 33, 4), (136, 72, 256, 65, 0),
                                            (64, 264, 128, 512, 8), (24, 16, 8, 7, 0)])
def test_forward_backward_match_fp64_at_ragged_sizes(D, h1, h2, Bn, pad):
    sur = H.MlpSurrogate(D, h1, h2, seed=D + Bn)
    gen = torch.Generator("cuda").manual_seed(Bn)
    # rows of x `pad` elements longer than the layer; dy starts 4 bytes off a
    # 16-byte boundary, so its groups are loaded element by element
    x = torch.randn(Bn, D + pad, device="cuda", generator=gen)
    dy_mem = torch.randn(Bn * D + 1, device="cuda", generator=gen)
    dy = dy_mem[1:]
    sc = sur._scratch(Bn)
    L = H.N.lib()
    H.N.check(L.ab_mlp_forward(H.C.byref(sur.desc), Bn, H.N.ptr(x), D + pad, H.N.ptr(sc["out"]), D, H.N.ptr(sc["act"]), None))
    H.N.check(L.ab_mlp_backward(H.C.byref(sur.desc), Bn, H.N.ptr(x), D + pad, dy.data_ptr(), H.N.ptr(sc["act"]),
                                H.N.ptr(sur.gw), H.N.ptr(sc["bsc"]), None))
    torch.cuda.synchronize()
    wmat, w = sur.wb.double().cpu().numpy(), sur.w.double().cpu().numpy()
    x64 = x[:, :D].double().cpu().numpy()
    Y, _ = B.mlp_forward(wmat, w, x64, D, h1, h2, D)
    out = sc["out"].double().cpu().numpy()
    assert np.max(np.abs(out - Y)) <= 1e-4 * max(1.0, np.max(np.abs(Y)))
    # the oracle's loss gradient at the target that gives this dy (FP64 outputs
    # differ from the device's by rounding only)
    t64 = Y - dy.double().cpu().numpy().reshape(Bn, D) * (0.5 * Bn * D)
    _, g = B.mlp_loss_grad(wmat, w, x64, t64, D, h1, h2, D)
    gd = sur.gw.double().cpu().numpy()
    n1, n2 = h1 * D, h2 * h1
    offs = [0, n1, n1 + h1, n1 + h1 + n2, n1 + h1 + n2 + h2, n1 + h1 + n2 + h2 + D * h2, len(g)]
    for a, b in zip(offs[:-1], offs[1:]):
        assert np.max(np.abs(gd[a:b] - g[a:b])) <= 1e-4 * np.max(np.abs(g[a:b])), (a, b)


@pytest.mark.parametrize("D,h1,h2,C,pad", [(8, 8, 8, 1, 0), (16, 256, 256, 128, 0), (40, 32, 64, 129, 4), (136, 72, 264, 256, 0),
                                           (136, 72, 264, 257, 8), (512, 256, 256, 33, 0), (1600, 24, 16, 130, 0), (1600, 24, 16, 101, 0), (320, 32, 64, 129, 0), (256, 8, 24, 4, 8)])
@pytest.mark.parametrize("dense", [False, True])
def test_surrogate_prediction_matches_fp64(D, h1, h2, C, pad, dense):
    # both kernels of the one-launch network, four and eight rows a cluster,
    # remainders of the rows, of the features and of the lanes; FP32 sums of at
    # most 1,600 terms against FP64 stay within 1600 * 2^-24 = 1e-4
    sur = H.MlpSurrogate(D, h1, h2, seed=D + C)
    gen = torch.Generator("cuda").manual_seed(C)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    for t in (sur.mu, sur.a, sur.h, sur.o):
        t.copy_(rnd(D))
    sur.inv_s.copy_(0.5 + rnd(D).abs())
    sur.dense = dense
    if dense:
        sur.M.copy_(rnd(D, D) / D ** 0.5)
    mem, out = rnd(C, D + pad), torch.full((C, D), float("nan"), device="cuda")
    theta = mem[:, :D]
    sur.predict(theta, out)
    torch.cuda.synchronize()
    d64 = lambda t: t.double().cpu().numpy()
    dt = d64(theta) - d64(sur.mu)
    Y, _ = B.mlp_forward(d64(sur.wb), d64(sur.w), dt * d64(sur.inv_s), D, h1, h2, D)
    want = d64(sur.a) + d64(sur.h) * dt + d64(sur.o) * Y + (dt @ d64(sur.M) if dense else 0.0)
    assert np.max(np.abs(d64(out) - want)) <= 1e-4 * np.max(np.abs(want))


@pytest.mark.parametrize("D,h1,h2", [(64, 256, 256), (512, 264, 40)])
def test_passes_agree_across_their_kernels(D, h1, h2):
    # the same rows in batches on both sides of each kernel's limit, and the
    # forward pass with and without kept activations: FP32 sums of at most 512
    # terms in two orders stay within 2 * 512 * 2^-24 = 6e-5 of one another,
    # through three layers within 2e-4 of the largest output
    sur = H.MlpSurrogate(D, h1, h2, seed=D)
    gen = torch.Generator("cuda").manual_seed(D)
    x = torch.randn(300, D, device="cuda", generator=gen)
    sur.M.copy_(torch.randn(D, D, device="cuda", generator=gen) / D ** 0.5)
    L = H.N.lib()
    for dense in (False, True):
        sur.dense = dense
        full = sur.predict(x, torch.empty_like(x)).clone()
        for C in (1, 128, 129, 256, 257):
            got = sur.predict(x[:C], torch.empty(C, D, device="cuda"))
            again = sur.predict(x[:C], torch.empty(C, D, device="cuda"))
            assert torch.equal(got, again)
            assert float((got - full[:C]).abs().max()) <= 2e-4 * float(full.abs().max())
    for Bn in (5, 200, 300):
        sc = sur._scratch(Bn)
        y = torch.empty(Bn, D, device="cuda")
        for act, out in ((sc["act"], sc["out"]), (None, y)):
            H.N.check(L.ab_mlp_forward(H.C.byref(sur.desc), Bn, H.N.ptr(x), D, H.N.ptr(out), D, H.N.ptr(act), None))
        torch.cuda.synchronize()
        assert float((y - sc["out"]).abs().max()) <= 2e-4 * float(y.abs().max())
