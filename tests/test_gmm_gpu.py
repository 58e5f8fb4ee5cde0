"""GPU parity of the Gaussian-mixture path against the CPU oracle.

Contract: the Cholesky / inverse / quadratic-form arithmetic repeats the
reference's operation order in binary64, so given the same weights, means,
covariances and uniforms the assignments z equal the reference's bit for bit
(exp/log of CUDA versus the C library could differ in a last bit, which
would only matter for a uniform within 1e-16 of a boundary); the
statistics are exact counts and binary64 sums in another order (1e-12
relative); conjugate draws agree to 1e-9 relative given the same statistics.
"""
import numpy as np
import pytest
import torch

from augurv2_b200 import _native as N
from augurv2_b200.gmm import GmmGibbs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def orc():
    return O.Oracle("oracle")


def hmodel(N_, K, d, seed):
    Y, z, mus, covs, pis = O.gmm_synthetic(N_, K, d, seed)
    om = O.GmmModel(Y, K, np.zeros(d), 25 * np.eye(d), False, alpha=np.ones(K), df=d + 2, scale0=np.eye(d))
    return Y, z, mus, covs, pis, om


@pytest.mark.parametrize("N_,K,d", [(3000, 16, 32), (2000, 4, 5), (500, 3, 2), (400, 5, 40)])
def test_disc_z_bit_exact(orc, N_, K, d):
    Y, z, mus, covs, pis, om = hmodel(N_, K, d, 1 + d)
    g = GmmGibbs(Y, K, np.zeros(d), 25 * np.eye(d), alpha=np.ones(K), df=d + 2, mu=mus, cov=covs, pis=pis, seed=4)
    L = N.lib()
    N.check(L.ab_gmm_prep(K, d, N.ptr(g.cov), N.ptr(g.Linv), N.ptr(g.hdet), N.stream_ptr()), "prep")
    N.check(L.ab_gmm_disc_z(N_, d, K, 0, N.ptr(g.Y), N.ptr(g.pis), N.ptr(g.mu), N.ptr(g.Linv), N.ptr(g.hdet),
                            N.ptr(g.z), 4, 6, 0, N.stream_ptr()), "disc_z")
    got = g.z.cpu().numpy()
    ref = O.gmm_disc_z(orc, om, pis, mus, covs, 4, 6)
    np.testing.assert_array_equal(got, ref)


def test_stats_and_conj_draws(orc):
    N_, K, d = 2500, 6, 8
    Y, z, mus, covs, pis, om = hmodel(N_, K, d, 3)
    g = GmmGibbs(Y, K, np.zeros(d), 25 * np.eye(d), alpha=np.ones(K), df=d + 2, mu=mus, cov=covs, pis=pis, z=z, seed=9)
    L = N.lib()
    st = N.stream_ptr()
    N.check(L.ab_gmm_stats(N_, d, K, N.ptr(g.Y), N.ptr(g.z), N.ptr(g.mu), N.ptr(g.cnt), N.ptr(g.sum), N.ptr(g.obs),
                           N.ptr(g.scratch), st), "stats")
    cnt, s, obs = O.gmm_stats(orc, om, z, mus)
    np.testing.assert_array_equal(g.cnt.cpu().numpy(), cnt)
    np.testing.assert_allclose(g.sum.cpu().numpy(), s, rtol=1e-12, atol=1e-9)
    np.testing.assert_allclose(g.obs.cpu().numpy(), obs, rtol=1e-12, atol=1e-9)
    # conjugate draws from the oracle's exact statistics
    g.cnt.copy_(torch.as_tensor(cnt)); g.sum.copy_(torch.as_tensor(s)); g.obs.copy_(torch.as_tensor(obs))
    N.check(L.ab_gmm_conj_pis(K, N.ptr(g.alpha), N.ptr(g.cnt), N.ptr(g.pis), 9, 2, 0, st), "pis")
    np.testing.assert_allclose(g.pis.cpu().numpy(), O.gmm_conj_pis(orc, om, cnt, 9, 2), rtol=1e-12)
    N.check(L.ab_gmm_conj_mu(K, d, 0, N.ptr(g.mu0), N.ptr(g.cov0), N.ptr(g.cnt), N.ptr(g.sum), N.ptr(g.cov),
                             N.ptr(g.mu), 9, 2, 0, st), "mu")
    np.testing.assert_allclose(g.mu.cpu().numpy(), O.gmm_conj_mu(orc, om, cnt, s, covs, 9, 2), rtol=1e-9, atol=1e-9)
    N.check(L.ab_gmm_conj_cov(K, d, d + 2, N.ptr(g.scale0), N.ptr(g.cnt), N.ptr(g.obs), N.ptr(g.cov), 9, 2, 0, st),
            "cov")
    np.testing.assert_allclose(g.cov.cpu().numpy(), O.gmm_conj_cov(orc, om, cnt, obs, 9, 2), rtol=1e-9, atol=1e-12)


@pytest.mark.parametrize("K,d", [(16, 32), (3, 5)])
def test_conj_cov_in_two_calls_equals_one(K, d):
    """ab_gmm_bartlett + ab_gmm_conj_cov_chi (the sweep's split, the first on
    a side stream) give ab_gmm_conj_cov's draw bit for bit."""
    rng = np.random.default_rng(K + d)
    cnt = torch.as_tensor(rng.integers(0, 5000, size=K).astype(np.int32)).cuda()
    a = rng.standard_normal((K, d, d))
    obs = torch.as_tensor(np.einsum("kij,klj->kil", a, a) * 50.0).cuda()
    scale0 = torch.eye(d, dtype=torch.float64, device="cuda")
    one = torch.zeros((K, d, d), dtype=torch.float64, device="cuda")
    two = torch.zeros_like(one)
    chi = torch.zeros((K, d), dtype=torch.float64, device="cuda")
    L = N.lib()
    st = N.stream_ptr()
    N.check(L.ab_gmm_conj_cov(K, d, d + 2, N.ptr(scale0), N.ptr(cnt), N.ptr(obs), N.ptr(one), 5, 3, 0, st), "cov")
    N.check(L.ab_gmm_bartlett(K, d, d + 2, N.ptr(cnt), N.ptr(chi), 5, 3, 0, st), "bartlett")
    N.check(L.ab_gmm_conj_cov_chi(K, d, d + 2, N.ptr(scale0), N.ptr(cnt), N.ptr(obs), N.ptr(chi), N.ptr(two), 5, 3,
                                  0, st), "cov_chi")
    torch.cuda.synchronize()
    assert torch.equal(one, two)
    assert torch.isfinite(one).all()


@pytest.mark.parametrize("d", [1, 2, 15, 16, 17, 31, 32, 33, 62, 64])
def test_factorisations_at_the_edges_of_the_dimension_ranges(orc, d):
    """Component tables and conjugate draws at the smallest and largest d and
    around the d (16, 32) at which the kernels change, counts of zero and one
    among them; tables also where the pivots leave the range of the short
    reciprocal root (covariances scaled by 2^-930 and 2^930)."""
    K = 3
    rng = np.random.default_rng(d)
    A = rng.standard_normal((K, d, d + 3))
    covs = np.einsum("kij,klj->kil", A, A) / (d + 3) + 0.1 * np.eye(d)
    L = N.lib()
    st = N.stream_ptr()
    for scale in (1.0, 2.0 ** -930, 2.0 ** 930):
        cov_t = torch.as_tensor(covs * scale).cuda()
        Linv = torch.full((K, d, d), float("nan"), dtype=torch.float64, device="cuda")
        hdet = torch.zeros(K, dtype=torch.float64, device="cuda")
        N.check(L.ab_gmm_prep(K, d, N.ptr(cov_t), N.ptr(Linv), N.ptr(hdet), st), "prep")
        ref = np.linalg.inv(np.linalg.cholesky(covs)) / np.sqrt(scale)
        got = Linv.cpu().numpy()
        assert np.all(got[:, np.triu_indices(d, 1)[0], np.triu_indices(d, 1)[1]] == 0.0)
        np.testing.assert_allclose(got, ref, rtol=1e-9, atol=1e-9 * np.abs(ref).max())
        if scale == 1.0:
            np.testing.assert_allclose(hdet.cpu().numpy(), 0.5 * np.linalg.slogdet(covs)[1], rtol=1e-9, atol=1e-9)
    cnt = np.array([0, 1, 900], np.int32)
    s = rng.standard_normal((K, d)) * cnt[:, None]
    obs = covs * cnt[:, None, None]
    om = O.GmmModel(rng.standard_normal((4, d)), K, np.zeros(d), 25 * np.eye(d), False, alpha=np.ones(K), df=d + 2,
                    scale0=np.eye(d))
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()
    cnt_t, s_t, obs_t, cov_t = dev(cnt), dev(s), dev(obs), dev(covs)
    mu0, cov0, scale0 = dev(np.zeros(d)), dev(25 * np.eye(d)), dev(np.eye(d))
    mu = torch.zeros((K, d), dtype=torch.float64, device="cuda")
    cov = torch.zeros((K, d, d), dtype=torch.float64, device="cuda")
    N.check(L.ab_gmm_conj_mu(K, d, 0, N.ptr(mu0), N.ptr(cov0), N.ptr(cnt_t), N.ptr(s_t), N.ptr(cov_t), N.ptr(mu), 9, 2, 0,
                             st), "mu")
    np.testing.assert_allclose(mu.cpu().numpy(), O.gmm_conj_mu(orc, om, cnt, s, covs, 9, 2), rtol=1e-9, atol=1e-9)
    N.check(L.ab_gmm_conj_cov(K, d, d + 2, N.ptr(scale0), N.ptr(cnt_t), N.ptr(obs_t), N.ptr(cov), 9, 2, 0, st), "cov")
    want = O.gmm_conj_cov(orc, om, cnt, obs, 9, 2)
    np.testing.assert_allclose(cov.cpu().numpy(), want, rtol=1e-9, atol=1e-9 * np.abs(want).max())


def _tables(A):
    """augur_mat_cholesky then augur_mat_lower_trmi of the matrices A [K][d][d]
    in the reference's order of operations (numpy's are IEEE binary64)."""
    L = A.copy()
    K, d, _ = L.shape
    for j in range(d):
        s = np.zeros(K)
        for k in range(j):
            s = s + L[:, j, k] * L[:, j, k]
        L[:, j, j] = np.sqrt(L[:, j, j] - s)
        r = 1.0 / L[:, j, j]
        for i in range(j + 1, d):
            s = np.zeros(K)
            for k in range(j):
                s = s + L[:, i, k] * L[:, j, k]
            L[:, i, j] = r * (L[:, i, j] - s)
    M = np.zeros_like(L)
    for c in range(d):
        for m in range(c, d):
            b = np.full(K, 1.0 if c == m else 0.0)
            for i in range(c, m):
                b = b - L[:, m, i] * M[:, i, c]
            M[:, m, c] = b / L[:, m, m]
    return M


def _device_tables(A):
    K, d, _ = A.shape
    cov = torch.as_tensor(np.ascontiguousarray(A)).cuda()
    Linv = torch.full((K, d, d), float("nan"), dtype=torch.float64, device="cuda")
    hdet = torch.zeros(K, dtype=torch.float64, device="cuda")
    N.check(N.lib().ab_gmm_prep(K, d, N.ptr(cov), N.ptr(Linv), N.ptr(hdet), N.stream_ptr()), "prep")
    return Linv.cpu().numpy()


def test_roots_reciprocals_and_quotients_are_correctly_rounded():
    """Component tables of diagonal matrices (a reciprocal of a root an entry)
    and of 2 x 2 blocks (a quotient each) equal IEEE arithmetic bit for bit:
    random values of a wide range, values beside powers of four (whose roots
    are beside powers of two), beside squares, and beyond the short steps'
    range."""
    rng = np.random.default_rng(8)
    K, d = 64, 64
    n = K * d
    j = np.arange(1.0, 33.0)
    edges = np.concatenate([4.0 ** e * np.concatenate([1.0 - j * 2.0 ** -53, 1.0 + j * 2.0 ** -52, [1.0]])
                            for e in (-440, -60, -1, 0, 1, 2, 60, 440)])
    sq = rng.integers(2 ** 26, 2 ** 27, 2000).astype(np.float64) ** 2
    edges = np.concatenate([edges, sq, np.nextafter(sq, 0.0), np.nextafter(sq, np.inf), 2.0 ** rng.uniform(-1000, -900, 500),
                            2.0 ** rng.uniform(900, 1000, 500)])
    pool = [np.resize(edges, -(-len(edges) // n) * n).reshape(-1, K, d)]
    pool.append(np.exp2(rng.uniform(-40, 40, (40, K, d))))
    for x in np.concatenate(pool):
        A = np.zeros((K, d, d))
        A[:, np.arange(d), np.arange(d)] = x
        got = _device_tables(A)
        np.testing.assert_array_equal(got[:, np.arange(d), np.arange(d)], 1.0 / np.sqrt(x))
        assert np.count_nonzero(got) == n
    i = 2 * np.arange(d // 2)
    for rep in range(40):
        A = np.zeros((K, d, d))
        a, c = np.exp2(rng.uniform(-20, 20, (2, K, d // 2)))
        if rep < 8:
            a = np.nextafter(4.0 ** rng.integers(-3, 4, a.shape), 0.0)
        b = np.sqrt(a * c) * rng.uniform(-0.999, 0.999, a.shape)
        if rep < 8:
            c = np.nextafter(4.0 ** rng.integers(-3, 4, a.shape), 0.0) + (b / np.sqrt(a)) ** 2
        A[:, i, i], A[:, i + 1, i], A[:, i, i + 1], A[:, i + 1, i + 1] = a, b, b, c
        got = _device_tables(A)
        r0 = 1.0 / np.sqrt(a)
        l10 = r0 * b
        l11 = np.sqrt(c - l10 * l10)
        np.testing.assert_array_equal(got[:, i, i], r0)
        np.testing.assert_array_equal(got[:, i + 1, i + 1], 1.0 / l11)
        np.testing.assert_array_equal(got[:, i + 1, i], -(l10 * r0) / l11)
    # zero over an infinite pivot is zero
    np.testing.assert_array_equal(_device_tables(np.diag([1.0, np.inf])[None]), [[[1.0, 0.0], [0.0, 0.0]]])


@pytest.mark.parametrize("d", [1, 7, 16, 33])
def test_component_tables_bit_exact(d):
    """Tables of covariances, and of correlation-like ones whose diagonal is
    just below 1, equal the reference's order of operations bit for bit."""
    rng = np.random.default_rng(d)
    K = 48
    A = rng.standard_normal((K, d, d + 3))
    cov = np.einsum("kij,klj->kil", A, A) / (d + 3) + 0.1 * np.eye(d)
    sd = np.sqrt(np.einsum("kii->ki", cov))
    cor = 0.5 * cov / (sd[:, :, None] * sd[:, None, :])
    cor[:, np.arange(d), np.arange(d)] = np.nextafter(1.0, 0.0)
    for m in (cov, cor):
        np.testing.assert_array_equal(_device_tables(m), _tables(m))


@pytest.mark.parametrize("N_,K,d", [(300_000, 16, 32), (250_000, 3, 40), (1, 2, 3), (900, 16, 2)])
def test_stats_sizes(orc, N_, K, d):
    """Statistics at sizes where a CTA's chunk spans several shared-memory
    sub-chunks (N = 3e5 at d = 32), the widest d of the pass, a single point,
    and many components with few points each; a label outside [0, K) is not
    counted."""
    rng = np.random.default_rng(N_ + d)
    Y = rng.standard_normal((N_, d)).astype(np.float32) * 3
    z = rng.integers(0, K, size=N_).astype(np.int32)
    mus = rng.standard_normal((K, d))
    om = O.GmmModel(Y.astype(np.float64), K, np.zeros(d), 25 * np.eye(d), False, alpha=np.ones(K), df=d + 2,
                    scale0=np.eye(d))
    g = GmmGibbs(Y, K, np.zeros(d), 25 * np.eye(d), alpha=np.ones(K), df=d + 2, mu=mus, z=z, seed=1)
    if N_ > 10:
        g.z[N_ // 2] = K + 3                     # not a component: skipped
    L = N.lib()
    N.check(L.ab_gmm_stats(N_, d, K, N.ptr(g.Y), N.ptr(g.z), N.ptr(g.mu), N.ptr(g.cnt), N.ptr(g.sum), N.ptr(g.obs),
                           N.ptr(g.scratch), N.stream_ptr()), "stats")
    keep = np.ones(N_, bool)
    if N_ > 10:
        keep[N_ // 2] = False
    cnt = np.bincount(z[keep], minlength=K)
    s = np.zeros((K, d))
    obs = np.zeros((K, d, d))
    Y64 = Y.astype(np.float64)
    for k in range(K):
        m = keep & (z == k)
        s[k] = Y64[m].sum(0)
        c = Y64[m] - mus[k]
        obs[k] = c.T @ c
    np.testing.assert_array_equal(g.cnt.cpu().numpy(), cnt)
    np.testing.assert_allclose(g.sum.cpu().numpy(), s, rtol=1e-12, atol=1e-9)
    np.testing.assert_allclose(g.obs.cpu().numpy(), obs, rtol=1e-12, atol=1e-8)


@pytest.mark.parametrize("N_,K,d", [(1, 1, 1), (1023, 3, 2), (1024, 64, 16), (1025, 3, 16), (2048, 5, 17), (513, 2, 32), (129, 4, 33),
                                    (6143, 64, 2), (12_289, 64, 2), (14_337, 64, 2), (131_072, 3, 1), (131_073, 3, 1), (3000, 7, 62)])
@pytest.mark.parametrize("same", [False, True])
def test_stats_of_few_points(N_, K, d, same):
    """The pass without the points' order, one and more shares of them, up to
    the number of partial sums and points from which the ordered pass takes over:
    small integers, so without any rounding; each output wanted and not; labels
    outside [0, K), empty components, all points in one."""
    rng = np.random.default_rng(N_ + d)
    Y = rng.integers(-4, 5, (N_, d))
    z = np.full(N_, K - 1) if same else rng.integers(-1, max(1, K - 1), N_)
    mus = rng.integers(-2, 3, (K, d))
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a), dtype=dt).cuda()
    Yt, zt, mt = t(Y, torch.float32), t(z, torch.int32), t(mus, torch.float64)
    L = N.lib()
    want_cnt = np.bincount(z[z >= 0], minlength=K)
    want_sum = np.zeros((K, d))
    np.add.at(want_sum, z[z >= 0], Y[z >= 0])
    want_obs = np.stack([(Y[z == k] - mus[k]).T @ (Y[z == k] - mus[k]) for k in range(K)])
    for ws, wo in ((True, True), (True, False), (False, True), (False, False)):
        cnt = torch.full((K,), 77, dtype=torch.int32, device="cuda")
        s = torch.full((K, d), 7.0, dtype=torch.float64, device="cuda")
        obs = torch.full((K, d, d), 7.0, dtype=torch.float64, device="cuda")
        scratch = torch.full((int(L.ab_gmm_stats_scratch_bytes(d, K)),), 0x5b, dtype=torch.uint8, device="cuda")
        N.check(L.ab_gmm_stats(N_, d, K, N.ptr(Yt), N.ptr(zt), N.ptr(mt) if wo else None, N.ptr(cnt), N.ptr(s) if ws else None,
                               N.ptr(obs) if wo else None, N.ptr(scratch), N.stream_ptr()), "stats")
        np.testing.assert_array_equal(cnt.cpu().numpy(), want_cnt)
        np.testing.assert_array_equal(s.cpu().numpy(), want_sum if ws else 7.0)
        np.testing.assert_array_equal(obs.cpu().numpy(), want_obs if wo else 7.0)


SLAB = 1 << 20     # points the statistics take at a time


@pytest.mark.parametrize("N_,K,d", [(SLAB, 3, 2), (SLAB + 1, 3, 2), (2 * SLAB + 700, 5, 3)])
def test_stats_of_several_slabs(N_, K, d):
    """Statistics of exactly one, and of more, slabs of points: counts and, as
    the points are small integers, sums and scatter matrices without any
    rounding, over stale outputs; the last component appears only in the
    last points and one label is not a component."""
    rng = np.random.default_rng(N_ % 1000 + d)
    Y = rng.integers(-4, 5, (N_, d))
    z = rng.integers(0, K - 1, N_)
    z[-1] = K - 1
    z[N_ // 3] = -1
    mus = rng.integers(-2, 3, (K, d))
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a), dtype=dt).cuda()
    Yt, zt, mt = t(Y, torch.float32), t(z, torch.int32), t(mus, torch.float64)
    cnt = torch.full((K,), 77, dtype=torch.int32, device="cuda")
    s = torch.full((K, d), 7.0, dtype=torch.float64, device="cuda")
    obs = torch.full((K, d, d), 7.0, dtype=torch.float64, device="cuda")
    L = N.lib()
    scratch = torch.full((int(L.ab_gmm_stats_scratch_bytes(d, K)),), 0x5b, dtype=torch.uint8, device="cuda")
    N.check(L.ab_gmm_stats(N_, d, K, N.ptr(Yt), N.ptr(zt), N.ptr(mt), N.ptr(cnt), N.ptr(s), N.ptr(obs), N.ptr(scratch),
                           N.stream_ptr()), "stats")
    for k in range(K):
        y = Y[z == k]
        c = y - mus[k]
        assert int(cnt[k]) == len(y)
        np.testing.assert_array_equal(s[k].cpu().numpy(), y.sum(0))
        np.testing.assert_array_equal(obs[k].cpu().numpy(), c.T @ c)


def test_sweep_of_several_slabs_equals_one_stream():
    """A sweep of more points than a slab and 1024 chi-square sums (more than
    run at once) beside the scatter pass equals the same draws made one after
    the other on one stream."""
    N_, K, d = SLAB + 50_000, 64, 16
    rng = np.random.default_rng(5)
    mus = 4.0 * rng.standard_normal((K, d))
    z = rng.integers(0, K, N_).astype(np.int32)
    Y = (mus[z] + rng.standard_normal((N_, d))).astype(np.float32)
    mk = lambda: GmmGibbs(Y, K, np.zeros(d), 25 * np.eye(d), alpha=np.ones(K), df=d + 2, mu=mus, z=z, seed=6)
    a, b = mk(), mk()
    L = N.lib()
    st = N.stream_ptr()
    for it in range(2):
        a.sweep(1)
        p = N.ptr
        N.check(L.ab_gmm_stats(N_, d, K, p(b.Y), p(b.z), None, p(b.cnt), p(b.sum), None, p(b.scratch), st))
        N.check(L.ab_gmm_conj_pis(K, p(b.alpha), p(b.cnt), p(b.pis), 6, it, 0, st))
        N.check(L.ab_gmm_conj_mu(K, d, 0, p(b.mu0), p(b.cov0), p(b.cnt), p(b.sum), p(b.cov), p(b.mu), 6, it, 0, st))
        N.check(L.ab_gmm_stats(N_, d, K, p(b.Y), p(b.z), p(b.mu), p(b.cnt), None, p(b.obs), p(b.scratch), st))
        N.check(L.ab_gmm_conj_cov(K, d, d + 2, p(b.scale0), p(b.cnt), p(b.obs), p(b.cov), 6, it, 0, st))
        N.check(L.ab_gmm_prep(K, d, p(b.cov), p(b.Linv), p(b.hdet), st))
        N.check(L.ab_gmm_disc_z_screened(N_, d, K, 0, p(b.Y), p(b.pis), p(b.mu), p(b.Linv), p(b.hdet), p(b.z), 6, it, 0,
                                         p(b.zscratch), st))
        for name in ("pis", "mu", "cov", "z", "cnt"):
            assert torch.equal(getattr(a, name), getattr(b, name)), (it, name)


def test_hmvgmm_sweeps_per_sweep_contract(orc):
    N_, K, d = 1500, 4, 5
    Y, z, mus, covs, pis, om = hmodel(N_, K, d, 11)
    g = GmmGibbs(Y, K, np.zeros(d), 25 * np.eye(d), alpha=np.ones(K), df=d + 2, mu=mus, cov=covs, pis=pis, z=z,
                 seed=3)
    for it in range(4):
        prev = g.state()
        g.sweep(1)
        st = g.state()
        # the oracle sweep from the GPU's previous state
        p, m, c, zz = prev["pis"].copy(), prev["mu"].copy(), prev["cov"].copy(), prev["z"].copy()
        O.gmm_sweep(orc, om, p, m, c, zz, 3, it)
        np.testing.assert_allclose(st["pis"], p, rtol=1e-10)
        np.testing.assert_allclose(st["mu"], m, rtol=1e-8, atol=1e-8)
        np.testing.assert_allclose(st["cov"], c, rtol=1e-8, atol=1e-10)
        # z bit-exact given the GPU's own new parameters
        z_ref = O.gmm_disc_z(orc, om, st["pis"], st["mu"], st["cov"], 3, it)
        np.testing.assert_array_equal(st["z"], z_ref)


@pytest.mark.parametrize("move", ["conj", "eslice", "mwg"])
def test_mvgmm_moves(orc, move):
    rng = np.random.default_rng(5)
    K, d, N_ = 3, 2, 300
    centres = np.array([[0.0, 2.0], [2.0, -2.0], [-2.0, -2.0]])
    covs = 0.1 * np.eye(d)
    Y = (centres[np.arange(N_) % K] + rng.standard_normal((N_, d)) * np.sqrt(0.1)).astype(np.float32).astype(np.float64)
    pis = np.full(K, 1.0 / K)
    om = O.GmmModel(Y, K, np.zeros(d), np.eye(d), True)
    mu0 = centres + 0.3 * rng.standard_normal((K, d))
    z0 = (np.arange(N_) % K).astype(np.int32)
    g = GmmGibbs(Y, K, np.zeros(d), np.eye(d), pis=pis, covs=covs, mu=mu0, z=z0, move=move,
                 prop_cov=0.05 * np.eye(d), seed=2)
    for it in range(3):
        prev = g.state()
        g.sweep(1)
        st = g.state()
        if move == "conj":
            m = prev["mu"].copy()
            cnt, s, _ = O.gmm_stats(orc, om, prev["z"], m)
            m = O.gmm_conj_mu(orc, om, cnt, s, covs, 2, it)
        elif move == "eslice":
            m = O.gmm_eslice(orc, om, prev["mu"], covs, prev["z"], 2, it)
        else:
            m = O.gmm_mwg(orc, om, prev["mu"], covs, prev["z"], 0.05 * np.eye(d), 2, it)
        np.testing.assert_allclose(st["mu"], m, rtol=1e-9, atol=1e-9)
        np.testing.assert_array_equal(st["z"], O.gmm_disc_z(orc, om, pis, st["mu"], covs, 2, it))


@pytest.mark.parametrize("move", ["eslice", "mwg"])
@pytest.mark.parametrize("N_,K,d", [(1, 2, 1), (6, 3, 1), (300, 3, 17), (1000, 64, 4), (700, 4, 33), (300, 2, 64),
                                    (9000, 5, 6)])
def test_mean_moves_at_ragged_sizes(orc, move, N_, K, d):
    """Fewer points than CTAs that add them, empty components, the widest d,
    the d at which the kernels change, labels outside [0, K): the moved means
    equal the oracle's, which evaluates every point at every candidate."""
    rng = np.random.default_rng(N_ + d)
    centres = rng.standard_normal((K, d)) * 2
    A = rng.standard_normal((d, d + 2))
    covs = A @ A.T / (d + 2) + 0.1 * np.eye(d)
    z = rng.integers(0, max(1, K - 1), N_).astype(np.int32)          # the last component is empty
    Y = (centres[z] + rng.standard_normal((N_, d))).astype(np.float32)
    om = O.GmmModel(Y.astype(np.float64), K, 0.1 * np.ones(d), 4 * np.eye(d), True)
    mu = centres + 0.1 * rng.standard_normal((K, d))
    prop = 0.02 * (np.eye(d) + 0.3)
    g = GmmGibbs(Y, K, 0.1 * np.ones(d), 4 * np.eye(d), pis=np.full(K, 1.0 / K), covs=covs, mu=mu, z=z, move=move,
                 prop_cov=prop, seed=2)
    for it in range(3):
        prev = g.mu.cpu().numpy()
        g.z.copy_(torch.as_tensor(z))
        g.sweep(1)
        want = O.gmm_eslice(orc, om, prev, covs, z, 2, it) if move == "eslice" else O.gmm_mwg(orc, om, prev, covs, z, prop, 2, it)
        np.testing.assert_allclose(g.mu.cpu().numpy(), want, rtol=1e-9, atol=1e-9)


@pytest.mark.parametrize("move", ["eslice", "mwg"])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_mean_moves_beside_a_point_that_is_not_finite(orc, move, value):
    """A component with such a point has no finite density anywhere: its mean
    stays where it is, as in the oracle; the other component moves."""
    N_, K = 200, 2
    for d in (1, 3):
        rng = np.random.default_rng(d)
        z = (np.arange(N_) % K).astype(np.int32)
        Y = rng.standard_normal((N_, d)).astype(np.float32)
        Y[4, d - 1] = value
        om = O.GmmModel(Y.astype(np.float64), K, np.zeros(d), 4 * np.eye(d), True)
        cov, prop = np.eye(d), 0.02 * np.eye(d)
        g = GmmGibbs(Y, K, np.zeros(d), 4 * np.eye(d), pis=np.full(K, 0.5), covs=cov, mu=np.zeros((K, d)), z=z, move=move,
                     prop_cov=prop, seed=5)
        moved = 0
        for it in range(6):
            prev = g.mu.cpu().numpy()
            g.z.copy_(torch.as_tensor(z))
            g.sweep(1)
            got = g.mu.cpu().numpy()
            want = O.gmm_eslice(orc, om, prev, cov, z, 5, it) if move == "eslice" else O.gmm_mwg(orc, om, prev, cov, z, prop, 5, it)
            np.testing.assert_array_equal(got[0], prev[0])
            np.testing.assert_allclose(got, want, rtol=1e-9, atol=1e-9)
            moved += bool((got[1] != prev[1]).any())
        assert moved > 0


def test_bench_shape_properties():
    """K=16, d=32, N=2e5 (the benchmark shape): statistics sum to N, the
    covariances stay symmetric positive definite, assignments recover most
    of the generating components' structure."""
    K, d, N_ = 16, 32, 200000
    Y, z, mus, covs, pis = O.gmm_synthetic(N_, K, d, 0)
    g = GmmGibbs(Y, K, np.zeros(d), 25 * np.eye(d), alpha=np.ones(K), df=d + 2, mu=mus, cov=covs, pis=pis, z=z,
                 seed=1)
    g.sweep(3)
    st = g.state()
    assert int(g.cnt.sum()) == N_
    for k in range(K):
        c = st["cov"][k]
        np.testing.assert_allclose(c, c.T, rtol=0, atol=1e-12)
        assert np.linalg.eigvalsh(c).min() > 0
    assert abs(st["pis"].sum() - 1) < 1e-12
