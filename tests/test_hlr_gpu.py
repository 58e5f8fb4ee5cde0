"""GPU parity of the HLR log-density / gradient and of the HMC, NUTS, MWG and
reflective-slice transitions against the CPU oracle (itself pinned to the reference's own
kernels).

Tolerances: the data terms run in FP32 with compensated sums, so block
log-densities agree with the FP64 oracle within 1e-5 relative and each
gradient component within 1e-5 of the scale sum_n |r_n x_nk| (plus the prior
term); transitions start from the same state and substreams and agree to
1e-4 relative when the accept decision (a comparison of nearly equal
binary64 values, which FP32 data terms can flip) agrees.
"""
import numpy as np
import pytest
import torch

from augurv2_b200 import hlr as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def orc():
    return O.Oracle("oracle")


def make(N, D, seed, has_b, vprior, compat, x_dtype="f32"):
    X, y, beta, s2 = O.hlr_synthetic(N, D, seed, has_b=has_b)
    if x_dtype == "bf16":
        X = torch.as_tensor(X, dtype=torch.float32).to(torch.bfloat16).to(torch.float32).numpy().astype(np.float64)
    om = O.HlrModel(X, y, has_b=has_b, vprior=vprior, compat=compat)
    gd = H.HlrData(X, y, has_b=has_b, vprior=vprior, compat=compat, x_dtype=x_dtype)
    return X, y, beta, s2, om, gd


@pytest.mark.parametrize("N,D,has_b,vprior,compat,xd", [
    (1000, 10, False, "invgamma", True, "f32"),
    (777, 33, True, "exponential", True, "f32"),
    (2500, 300, True, "exponential", False, "f32"),
    (3000, 64, False, "invgamma", False, "bf16"),
    (5, 1, True, "exponential", True, "f32"),
])
def test_ll_grad_matches_fp64_oracle(orc, N, D, has_b, vprior, compat, xd):
    X, y, beta, s2, om, gd = make(N, D, 3, has_b, vprior, compat, xd)
    rng = np.random.default_rng(1)
    C = 6
    pars = np.zeros((C, D + 2))
    pars[:, :D] = beta + 0.3 * rng.standard_normal((C, D))
    pars[:, D] = 0.2 * rng.standard_normal(C) if has_b else 0.0
    pars[:, D + 1] = 0.5 + rng.random(C)
    blocks = [list(range(D)), [D + 1], [D + 1] + ([D] if has_b else []) + list(range(D))]
    if has_b:
        blocks.append([D])
    for idx in blocks:
        ll, g = H.ll_grad(gd, pars, idx)
        for c in range(C):
            l_ref = O.hlr_ll(orc, om, pars[c], idx)
            g_ref = O.hlr_grad(orc, om, pars[c], idx)
            assert abs(ll[c] - l_ref) <= 1e-5 * abs(l_ref) + 1e-9, (idx[:3], c, ll[c], l_ref)
            t = X @ pars[c, :D] + (pars[c, D] if has_b else 0.0)
            r = np.abs(y - 1.0 / (1.0 + np.exp(-t)))
            scale_th = np.abs(X).T @ r + np.abs(pars[c, :D]) / pars[c, D + 1]
            for j, i in enumerate(idx):
                if i < D:
                    tol = 1e-5 * scale_th[i] + 1e-9
                elif i == D:
                    tol = 1e-5 * (r.sum() + abs(pars[c, D]) / pars[c, D + 1]) + 1e-9
                else:
                    tol = 1e-9 * max(1.0, abs(g_ref[j]))
                assert abs(g[c, j] - g_ref[j]) <= tol, (idx[:3], c, j, g[c, j], g_ref[j])


def run_one(gd, sched, par, it, seed, C=1):
    ch = H.HlrChains(gd, sched, C=C, init=par, seed=seed, iter0=it)
    ch.run(1)
    return ch.state(), ch.stats.cpu().numpy()


@pytest.mark.parametrize("has_b,vprior,block", [(False, "invgamma", ["theta"]),
                                                (True, "exponential", ["v", "b", "theta"])])
def test_hmc_transition_matches_oracle(orc, has_b, vprior, block):
    X, y, beta, s2, om, gd = make(1000, 10, 4, has_b, vprior, True)
    D = 10
    idx = H.block_indices(block, D)
    par = np.concatenate([beta, [0.1 if has_b else 0.0], [max(s2, 0.5)]])
    agree = 0
    for it in range(8):
        p_ref = par.copy()
        acc, L, prop = O.hlr_hmc(orc, om, p_ref, idx, 0.1, 0.01, 11, it)
        got, st = run_one(gd, [{"kind": "HMC", "block": block, "simlen": 0.1, "eps": 0.01}], par, it, 11)
        if int(st[0, 0, 0]) == acc:
            agree += 1
            np.testing.assert_allclose(got[0], p_ref, rtol=1e-4, atol=1e-6)
        par = p_ref
    assert agree >= 7


@pytest.mark.parametrize("N,D,xd,C,kind", [
    (7, 14, "f32", 1, "HMC"), (257, 15, "bf16", 2, "NUTS"), (600, 30, "f32", 1, "NUTS"), (1000, 31, "bf16", 1, "HMC"),
    (1025, 41, "bf16", 2, "NUTS"), (1023, 33, "f32", 150, "HMC"), (2049, 100, "f32", 1, "HMC"), (900, 300, "bf16", 1, "HMC")])
def test_chain_paths_match_oracle(orc, N, D, xd, C, kind):
    """The chain engine's ways through the data (16 and 32 columns, wide; X in
    shared memory as f32 or bf16, or too large for it; one or two chains per
    SM; remainders of a chunk of rows): a transition of the first and the last
    chain equals the oracle's."""
    X, y, beta, s2, om, gd = make(N, D, N + D, True, "exponential", True, xd)
    block = ["v", "b", "theta"]
    idx = H.block_indices(block, D)
    par = np.concatenate([0.5 * beta, [0.1], [1.0]])
    eps = 0.3 / np.sqrt(N + 10.0)
    sched = [{"kind": kind, "block": block, "eps": eps, "simlen": 5 * eps, "max_depth": 3}]
    ch = H.HlrChains(gd, sched, C=C, init=par, seed=17)
    ch.run(2)                                    # the second iteration starts from the first's gradient
    got, st = ch.state(), ch.stats.cpu().numpy()
    one = H.HlrChains(gd, sched, C=C, init=par, seed=17)
    one.run(1)
    one.run(1)
    np.testing.assert_array_equal(got, one.state())
    for c in {0, C - 1}:
        p = par.copy()
        tally = 0
        for it in range(2):
            if kind == "HMC":
                tally += O.hlr_hmc(orc, om, p, idx, 5 * eps, eps, 17, it, chain=c)[0]
            else:
                tally += O.hlr_nuts(orc, om, p, idx, eps, 17, it, max_depth=3, chain=c)[0]
        assert int(st[c, 0, 0 if kind == "HMC" else 1]) == tally
        np.testing.assert_allclose(got[c], p, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("N,D,xd,C", [(9, 3, "f32", 1), (1000, 10, "bf16", 2), (1500, 20, "f32", 150), (300, 33, "f32", 1),
                                      (9001, 9, "f32", 2), (900, 120, "bf16", 150), (4000, 60, "f32", 1)])
def test_slice_and_metropolis_moves_on_every_path(orc, N, D, xd, C):
    """Reflective-slice and Metropolis moves with X in shared memory (f32,
    bf16) or too large for it, 16, 32 and more columns, one or more chains an
    SM: the first and the last chain's moves equal the oracle's.  A component
    a launch, so that every chain starts from the oracle's state; an FP32
    data term may flip one decision of the lot."""
    X, y, beta, s2, om, gd = make(N, D, N + D, True, "exponential", True, xd)
    theta = H.block_indices(["theta"], D)
    eps = 0.4 / np.sqrt(N + 10.0)
    par = np.concatenate([beta, [0.1], [max(s2, 0.5)]])
    agree = total = 0
    for it in range(4):
        for comp in ({"kind": "RSlice", "block": ["theta"], "simlen": 4 * eps, "eps": eps},
                     {"kind": "MWG", "var": "b", "scale": 0.05}, {"kind": "MWG", "var": "v", "scale": 0.3}):
            got, st = run_one(gd, [comp], par, it, 31, C)
            refs = {}
            for c in {0, C - 1}:
                p = par.copy()
                if comp["kind"] == "RSlice":
                    moved = O.hlr_rslice(orc, om, p, theta, 4 * eps, eps, 31, it, chain=c)[0]
                else:
                    moved = O.hlr_mwg(orc, om, p, D if comp["var"] == "b" else D + 1, comp["scale"], 31, it, chain=c)
                refs[c] = p
                total += 1
                if int(st[c, 0, 0]) == moved:
                    agree += 1
                    np.testing.assert_allclose(got[c], p, rtol=1e-4, atol=1e-6)
            par = refs[0]
    assert agree >= total - 1


@pytest.mark.parametrize("N,D,xd", [(1, 1, "f32"), (255, 7, "bf16"), (257, 8, "f32"), (511, 9, "bf16"), (513, 14, "f32"),
                                    (700, 15, "bf16"), (769, 16, "f32"), (300, 22, "bf16"), (1025, 24, "f32"), (256, 30, "bf16"),
                                    (1030, 31, "f32"), (90, 254, "bf16"), (60, 255, "f32"), (60, 600, "f32")])
def test_ll_and_gradient_at_the_edges_of_the_row_walk(orc, N, D, xd):
    """Rows and columns around the groups in which the evaluation loads them,
    with and without the gradient (two rows at a time without), the variance
    alone: the same density with and without, within 1e-5 of its terms'
    magnitudes of the oracle's, and gradients that do not depend on columns of
    zeros beside them."""
    X, y, beta, s2, om, gd = make(N, D, N + D, True, "exponential", True, xd)
    rng = np.random.default_rng(D)
    par = np.concatenate([beta + 0.2 * rng.standard_normal(D), [0.2], [0.7]])
    pars = np.stack([par, par * 0.5, par])
    pars[:, D + 1] = [0.7, 1.3, 0.7]
    L, C_ = H.N.lib(), len(pars)
    for idx in ([D + 1, D] + list(range(D)), list(range(D)), [D + 1]):
        ll, g = H.ll_grad(gd, pars, idx)
        pt = torch.as_tensor(pars).cuda()
        ih = np.ascontiguousarray(idx, np.int32)
        only = torch.zeros(C_, dtype=torch.float64, device="cuda")
        H.N.check(L.ab_hlr_ll_grad(H.C.byref(gd.c), H.N.ptr(torch.as_tensor(ih).cuda()), ih.ctypes.data_as(H.C.c_void_p), len(ih),
                                   C_, H.N.ptr(pt), H.N.ptr(only), None, H.N.stream_ptr()))
        np.testing.assert_array_equal(only.cpu().numpy(), ll)
        np.testing.assert_array_equal(g[0], g[2])
        for c in range(2):
            p = pars[c]
            t = X @ p[:D] + p[D]
            l_ref = O.hlr_ll(orc, om, p, idx)
            size = np.abs(y * t).sum() + np.logaddexp(0.0, t).sum() if idx != [D + 1] else 0.0
            assert abs(ll[c] - l_ref) <= 1e-5 * size + 1e-9 * max(1.0, abs(l_ref))
    if D <= 30:
        # columns of zeros up to the walk's width change no bit of the others' sums
        W = 14 if D <= 14 else 30
        wide = H.HlrData(np.hstack([X, np.zeros((N, W - D))]), y, has_b=True, vprior="exponential", compat=True, x_dtype=xd)
        wp = np.hstack([pars[:, :D], np.zeros((len(pars), W - D)), pars[:, D:]])
        gw = H.ll_grad(wide, wp, list(range(D)) + [W])[1]
        np.testing.assert_array_equal(H.ll_grad(gd, pars, list(range(D)) + [D])[1], gw)


@pytest.mark.parametrize("N,D,xd,C", [(200, 300, "bf16", 1), (200, 300, "bf16", 150), (1600, 28, "f32", 150), (700, 300, "f32", 2)])
def test_nuts_with_rows_or_stacks_in_shared_memory(orc, N, D, xd, C):
    """NUTS where shared memory holds X but not the walk's stacks, the stacks
    but not X, or both, for fewer and more chains than SMs: the first and the
    last chain's trees and states equal the oracle's."""
    X, y, beta, s2, om, gd = make(N, D, N + D, True, "exponential", True, xd)
    block = ["v", "b", "theta"]
    idx = H.block_indices(block, D)
    par = np.concatenate([0.5 * beta, [0.1], [1.0]])
    eps = 0.2 / np.sqrt(N + 10.0)
    got, st = run_one(gd, [{"kind": "NUTS", "block": block, "eps": eps, "max_depth": 3}], par, 0, 23, C)
    for c in {0, C - 1}:
        p = par.copy()
        depth = O.hlr_nuts(orc, om, p, idx, eps, 23, 0, max_depth=3, chain=c)[0]
        assert int(st[c, 0, 1]) == depth
        np.testing.assert_allclose(got[c], p, rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("compat", [True, False])
@pytest.mark.parametrize("vprior", ["exponential", "invgamma"])
@pytest.mark.parametrize("v", [1e-158, 1e-156, 3e-155, 1e-100, 1e150])
def test_variance_gradient_at_the_ends_of_the_range(v, vprior, compat):
    """The prior's derivative in the variance where 1 / v^2 is out of binary64's
    range and the derivative is not: some coefficients zero, some far below
    the root of v, an inverse-gamma scale as small."""
    D = 7
    s0 = v * v * 2.0 ** 90
    gd = H.HlrData(np.ones((3, D)), np.array([0, 1, 1]), has_b=True, vprior=vprior, lam=0.5, a0=2.0, s0=s0, compat=compat)
    par = np.zeros((1, D + 2))
    par[0, 2], par[0, D] = 0.25 * v * 2.0 ** 60, -3.0 * v
    par[0, D + 1] = v
    _, g = H.ll_grad(gd, par, [D + 1])
    q = np.array([par[0, 2], par[0, D]]) / v
    want = (D + 1) * (-0.5 * v if compat else -0.5 / v) + 0.5 * (q * q).sum()
    want += -0.5 if vprior == "exponential" else -3.0 / v + s0 / v / v
    np.testing.assert_allclose(g[0, 0], want, rtol=1e-12)


def test_hmc_many_chains_distinct_streams(orc):
    X, y, beta, s2, om, gd = make(400, 5, 6, False, "invgamma", True)
    D = 5
    par = np.concatenate([beta, [0.0], [1.0]])
    C = 16
    ch = H.HlrChains(gd, [{"kind": "HMC", "block": ["theta"], "simlen": 0.2, "eps": 0.02}], C=C, init=par, seed=5)
    ch.run(1)
    got = ch.state()
    idx = list(range(D))
    for c in range(0, C, 5):
        p_ref = par.copy()
        acc, L, prop = O.hlr_hmc(orc, om, p_ref, idx, 0.2, 0.02, 5, 0, chain=c)
        np.testing.assert_allclose(got[c], p_ref, rtol=1e-4, atol=1e-6)
    assert len({tuple(np.round(r, 12)) for r in got}) > 1


def test_nuts_transition_matches_oracle(orc):
    X, y, beta, s2, om, gd = make(300, 4, 8, True, "exponential", True)
    D = 4
    block = ["v", "b", "theta"]
    idx = H.block_indices(block, D)
    par = np.concatenate([beta, [0.1], [max(s2, 0.5)]])
    agree = 0
    for it in range(8):
        p_ref = par.copy()
        depth, leaves, ovf = O.hlr_nuts(orc, om, p_ref, idx, 0.05, 13, it, max_depth=10)
        got, st = run_one(gd, [{"kind": "NUTS", "block": block, "eps": 0.05, "max_depth": 10}], par, it, 13)
        if int(st[0, 0, 1]) == depth and np.allclose(got[0], p_ref, rtol=1e-4, atol=1e-6):
            agree += 1
        par = p_ref
    assert agree >= 7


def test_mwg_matches_oracle(orc):
    X, y, beta, s2, om, gd = make(500, 6, 9, True, "exponential", True)
    D = 6
    par = np.concatenate([beta, [0.3], [1.3]])
    for which, name in [(D + 1, "v"), (D, "b")]:
        p = par.copy()
        for it in range(6):
            p_ref = p.copy()
            acc = O.hlr_mwg(orc, om, p_ref, which, 0.5, 21, it)
            got, st = run_one(gd, [{"kind": "MWG", "var": name, "scale": 0.5}], p, it, 21)
            assert int(st[0, 0, 0]) == acc
            np.testing.assert_allclose(got[0], p_ref, rtol=1e-12)
            p = p_ref


@pytest.mark.parametrize("block,simlen,eps", [(["theta"], 0.5, 0.05), (["v", "b", "theta"], 1.0, 0.08)])
def test_rslice_matches_oracle(orc, block, simlen, eps):
    """Reflective slice (h_augur_mcmc_refl_slice): the same move or stay,
    the same number of reflections, and the same end point (1e-4) as the
    oracle, itself equal to the reference's kernel bit for bit."""
    X, y, beta, s2, om, gd = make(400, 5, 17, True, "exponential", True)
    D = 5
    idx = H.block_indices(block, D)
    par = np.concatenate([beta, [0.1], [max(s2, 0.5)]])
    agree, refl_total = 0, 0
    for it in range(10):
        p_ref = par.copy()
        moved, L, refl = O.hlr_rslice(orc, om, p_ref, idx, simlen, eps, 19, it)
        got, st = run_one(gd, [{"kind": "RSlice", "block": block, "simlen": simlen, "eps": eps}], par, it, 19)
        refl_total += refl
        if int(st[0, 0, 0]) == moved and int(st[0, 0, 2]) == refl and \
                np.allclose(got[0], p_ref, rtol=1e-4, atol=1e-6):
            agree += 1
        par = p_ref
    assert agree >= 9
    assert refl_total > 0


def test_schedule_composition_runs():
    X, y, beta, s2, om, gd = make(800, 8, 10, True, "exponential", True)
    sched = [{"kind": "MWG", "var": "v", "scale": 1.0}, {"kind": "MWG", "var": "b", "scale": 1.0},
             {"kind": "HMC", "block": ["theta"], "simlen": 0.5, "eps": 0.05}]
    ch = H.HlrChains(gd, sched, C=8, init=np.concatenate([beta, [0.0], [1.0]]), seed=1)
    ch.run(20)
    s = ch.state()
    assert np.isfinite(s).all() and (s[:, 9] > 0).all()
    st = ch.stats.cpu().numpy()
    assert (st[:, 2, 0] > 0).all()
