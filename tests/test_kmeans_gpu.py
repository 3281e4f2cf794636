"""GPU parity of the k-means assign / accumulate / update kernels against the CPU restatement of
src/pq_kmeans.c, through the C ABI. Codes must be bit-identical."""
import ctypes as C

import os

import numpy as np
import pytest

from tests import _cpu

pytestmark = pytest.mark.gpu


def oracle_assign(libs, X, Cn):
    idx = np.empty(len(X), np.int32); dist = np.empty(len(X), np.float32)
    libs.oracle.ibo_kmeans_assign(X, len(X), X.shape[1], Cn, len(Cn), idx, dist.ctypes.data, 2)
    return idx, dist


@pytest.mark.parametrize("N,D,K", [(100000, 8, 256), (5000, 2, 16), (3333, 5, 100), (4097, 16, 64), (1000, 32, 7),
                                   (700, 3, 1000), (64, 8, 1), (1, 8, 256)])
def test_assign_codes_bit_exact(backend, cpu_libs, N, D, K):
    rng = np.random.default_rng(N + D + K)
    X = (rng.standard_normal((N, D)) * 0.02).astype(np.float32)
    Cn = (rng.standard_normal((K, D)) * 0.02).astype(np.float32)
    m = min(N, K); Cn[:m] = X[:m]
    got, gd = backend.kmeans_assign(X, Cn, want_dist=True)
    want, wd = oracle_assign(cpu_libs, X, Cn)
    assert np.array_equal(got, want)
    assert np.array_equal(gd, wd)                               # same roundings, same distance bits


@pytest.mark.parametrize("D", [2, 4, 5, 8, 12])
def test_assign_near_ties_and_exact_ties(backend, cpu_libs, D):
    """Points on the bisector of two centroids decide on the last bit; duplicated centroids are exact
    ties that the lowest index must win; NaN rows fall to centroid 0."""
    rng = np.random.default_rng(40 + D)
    K = 8
    Cn = (rng.standard_normal((K, D)) * 0.02).astype(np.float32)
    Cn[5] = Cn[2]                                               # exact duplicate
    mid = (Cn[0].astype(np.float64) + Cn[1]) / 2
    d = Cn[1].astype(np.float64) - Cn[0]; d /= np.linalg.norm(d)
    noise = rng.standard_normal((50000, D)) * 0.002
    noise -= (noise @ d)[:, None] * d
    X = (mid + noise).astype(np.float32)
    X[10] = Cn[2]; X[11] = np.nan
    got = backend.kmeans_assign(X, Cn)
    want, _ = oracle_assign(cpu_libs, X, Cn)
    assert np.array_equal(got, want)
    assert got[10] == 2 and got[11] == 0
    assert 0 < int((got == 0).sum()) < len(X)


def _lloyd_gpu(be, X, C0, iters, teacher=None):
    N, D = X.shape; K = len(C0)
    dX = be.upload(X); dC = be.upload(C0)
    di, dd = be.alloc(N * 4), be.alloc(N * 4)
    ds, dc, dn = be.alloc(K * D * 4), be.alloc(K * 4), be.alloc(8)
    hist = []
    for it in range(iters):
        if teacher is not None:
            be.write(dC, teacher[it])
        be._check(be.lib.ibcu_kmeans_lloyd_iter(be.ctx, dX.ptr, N, D, dC.ptr, K, di.ptr, dd.ptr, ds.ptr, dc.ptr, dn.ptr))
        be.sync()
        hist.append(dict(idx=be.download(di, np.int32, N), sums=be.download(ds, np.float32, K * D).reshape(K, D),
                         counts=be.download(dc, np.int32, K), inertia=float(be.download(dn, np.float64, 1)[0]),
                         C=be.download(dC, np.float32, K * D).reshape(K, D)))
    return hist


def _lloyd_cpu(libs, X, C0, iters):
    N, D = X.shape; K = len(C0)
    Cn = C0.copy(); hist = []
    for it in range(iters):
        before = Cn.copy()
        idx = np.empty(N, np.int32); sums = np.empty((K, D), np.float32); counts = np.empty(K, np.int32)
        inertia = C.c_double()
        libs.oracle.ibo_kmeans_lloyd_iter(X, N, D, Cn, K, idx, sums, counts, C.byref(inertia), 2)
        hist.append(dict(idx=idx, sums=sums, counts=counts, inertia=inertia.value, C=Cn.copy(), C_in=before))
    return hist


def test_lloyd_teacher_forced_and_free_running(backend, cpu_libs):
    """10 Lloyd iterations from C0 = X[:K]. Teacher-forced (the CPU's centroids fed in each iteration):
    codes and counts bit-exact, sums / centroids / inertia within float tolerance. Free-running: the
    trajectory may drift by summation order; the mismatch count is reported and bounded loosely."""
    rng = np.random.default_rng(77)
    N, D, K, iters = 200000, 8, 256, 10
    X = (rng.standard_normal((N, D)) * 0.02).astype(np.float32)
    C0 = X[:K].copy()
    cpu = _lloyd_cpu(cpu_libs, X, C0, iters)
    forced = _lloyd_gpu(backend, X, C0, iters, teacher=[h["C_in"] for h in cpu])
    for it, (g, c) in enumerate(zip(forced, cpu)):
        assert np.array_equal(g["idx"], c["idx"]), it
        assert np.array_equal(g["counts"], c["counts"]), it
        assert np.allclose(g["sums"], c["sums"], rtol=1e-4, atol=1e-5), it
        assert np.allclose(g["C"], c["C"], rtol=1e-4, atol=1e-6), it
        assert abs(g["inertia"] - c["inertia"]) <= 1e-6 * c["inertia"], it
    free = _lloyd_gpu(backend, X, C0, iters)
    mism = int((free[-1]["idx"] != cpu[-1]["idx"]).sum())
    print(f"free-running: {mism} of {N} codes differ after {iters} iterations; "
          f"max centroid diff {np.max(np.abs(free[-1]['C'] - cpu[-1]['C'])):.3e}")
    assert mism <= N // 100
    assert abs(free[-1]["inertia"] - cpu[-1]["inertia"]) <= 1e-4 * cpu[-1]["inertia"]
    # determinism: the same run again gives the same bits
    again = _lloyd_gpu(backend, X, C0, iters)
    assert np.array_equal(again[-1]["C"], free[-1]["C"]) and np.array_equal(again[-1]["idx"], free[-1]["idx"])


def test_empty_cluster_keeps_its_centroid(backend, cpu_libs):
    rng = np.random.default_rng(5)
    X = (rng.standard_normal((5000, 4)) * 0.02).astype(np.float32)
    C0 = X[:16].copy(); C0[7] = 100.0                            # nobody is near centroid 7
    g = _lloyd_gpu(backend, X, C0, 1)[0]
    c = _lloyd_cpu(cpu_libs, X, C0, 1)[0]
    assert g["counts"][7] == 0 and np.array_equal(g["C"][7], C0[7])
    assert np.array_equal(g["idx"], c["idx"]) and np.array_equal(g["counts"], c["counts"])
    assert np.allclose(g["C"], c["C"], rtol=1e-4, atol=1e-6)


def test_update_rounding_matches(backend, cpu_libs):
    """Given the same sums and counts the centroid move is bit-identical (reciprocal then multiply)."""
    rng = np.random.default_rng(6)
    K, D = 256, 8
    sums = rng.standard_normal((K, D)).astype(np.float32); counts = rng.integers(0, 50, K).astype(np.int32)
    C0 = rng.standard_normal((K, D)).astype(np.float32)
    want = C0.copy(); shift = cpu_libs.oracle.ibo_kmeans_update(want, K, D, sums, counts)
    be = backend
    dC, ds, dc, dsh = be.upload(C0), be.upload(sums), be.upload(counts), be.alloc(4)
    be._check(be.lib.ibcu_kmeans_update(be.ctx, dC.ptr, K, D, ds.ptr, dc.ptr, dsh.ptr)); be.sync()
    assert np.array_equal(be.download(dC, np.float32, K * D).reshape(K, D), want)
    assert abs(float(be.download(dsh, np.float32, 1)[0]) - shift) <= 1e-4 * shift


def test_full_size_properties(backend):
    """Benchmark-size properties (4 Mi points): every code is a valid index, assigning twice is idempotent,
    counts sum to N, and a point equal to a centroid gets that centroid (or an equal-valued earlier one)."""
    rng = np.random.default_rng(1234)
    N, D, K = 1 << 22, 8, 256
    X = (rng.standard_normal((N, D)) * 0.02).astype(np.float32)
    C0 = X[:K].copy()
    h = _lloyd_gpu(backend, X, C0, 1)[0]
    assert h["idx"].min() >= 0 and h["idx"].max() < K
    assert int(h["counts"].sum()) == N and np.array_equal(np.bincount(h["idx"], minlength=K), h["counts"])
    assert np.array_equal(h["idx"][:K], np.arange(K))
    # sums against a float64 bincount
    for d in range(0, D, 3):
        ref = np.bincount(h["idx"], weights=X[:, d].astype(np.float64), minlength=K)
        assert np.allclose(h["sums"][:, d], ref, rtol=1e-4, atol=1e-5)


def test_full_size_codes_against_the_reference(backend, cpu_libs):
    """The benchmark configuration itself: 4 Mi points x 8, K = 256, centroids = the first 256 points, then
    one more assignment with the centroids of one CPU update (teacher-forced): codes bit-equal to the
    unmodified reference's ib_kmeans_assign run on its own thread pool (src/pq_kmeans.c:399-413), or to
    the restatement where the reference library did not travel."""
    rng = np.random.default_rng(1234)
    N, D, K = 1 << 22, 8, 256
    X = (rng.standard_normal((N, D)) * 0.02).astype(np.float32)
    Cn = X[:K].copy()
    want = np.empty(N, np.int32)
    pool = None
    if cpu_libs.ref is not None:
        pool = cpu_libs.ref.ib_pool_create(min(32, os.cpu_count() or 1))
    for step in range(2):
        if cpu_libs.ref is not None:
            assert cpu_libs.ref.ib_kmeans_assign(X, N, D, Cn, K, want, pool) == 0
        else:
            cpu_libs.oracle.ibo_kmeans_assign(X, N, D, Cn, K, want, None, 2)
        got = backend.kmeans_assign(X, Cn)
        bad = np.flatnonzero(got != want)
        assert bad.size == 0, (step, bad[:10], got[bad[:10]], want[bad[:10]])
        # centroids of the next iteration from the reference's own codes (float64 means rounded to FP32: any
        # centroid set will do for a teacher-forced check)
        cnt = np.bincount(want, minlength=K)
        for d in range(D):
            s = np.bincount(want, weights=X[:, d].astype(np.float64), minlength=K)
            Cn[:, d] = np.where(cnt > 0, s / np.maximum(cnt, 1), Cn[:, d]).astype(np.float32)
    if pool:
        cpu_libs.ref.ib_pool_destroy(pool)


@pytest.mark.parametrize("D", [4, 8, 16])
@pytest.mark.parametrize("N,K", [(1, 1), (127, 7), (128, 32), (129, 33), (148 * 128 + 1, 200), (40001, 256), (6000, 130), (300, 16)])
def test_tensor_core_assign_and_sums_at_the_edges(backend, cpu_libs, D, N, K):
    """Tiles of 128 points and groups of 8 centroids, padded: last rows, first and last group, one centroid; codes and distances are the
    checker's bits, and the sums a Lloyd iteration leaves are those of the codes (FP32 sums of at most N terms)."""
    rng = np.random.default_rng(N * 31 + K + D)
    X = (rng.standard_normal((N, D)) * 0.02).astype(np.float32)
    Cn = (rng.standard_normal((K, D)) * 0.02).astype(np.float32)
    m = min(N, K) // 2
    Cn[K - m:] = X[:m]
    if K > 20:
        Cn[K - 1] = Cn[K - 9]                                    # exact ties between two groups
    got, gd = backend.kmeans_assign(X, Cn, want_dist=True)
    want, wd = oracle_assign(cpu_libs, X, Cn)
    assert np.array_equal(got, want) and np.array_equal(gd, wd)
    h = _lloyd_gpu(backend, X, Cn, 1)[0]
    assert np.array_equal(h["idx"], want)
    assert np.array_equal(h["counts"], np.bincount(want, minlength=K))
    for d in range(D):
        ref = np.bincount(want, weights=X[:, d].astype(np.float64), minlength=K)
        mag = np.bincount(want, weights=np.abs(X[:, d]).astype(np.float64), minlength=K)
        assert np.all(np.abs(h["sums"][:, d] - ref) <= 2.0 ** -24 * (N + 16) * mag)
    assert abs(h["inertia"] - wd.astype(np.float64).sum()) <= 1e-12 * wd.astype(np.float64).sum()


@pytest.mark.parametrize("D", [4, 8, 16])
def test_tensor_core_filter_hands_over_what_it_cannot_decide(backend, cpu_libs, D):
    """Near ties across groups, NaN and Inf in points and centroids (centroid 0 among them: the reference's scan starts from it and a NaN
    there is never replaced), squares that overflow or vanish."""
    rng = np.random.default_rng(90 + D)
    K, N = 72, 20000
    Cn = (rng.standard_normal((K, D)) * 0.02).astype(np.float32)
    mid = (Cn[3].astype(np.float64) + Cn[60]) / 2
    d = Cn[60].astype(np.float64) - Cn[3]; d /= np.linalg.norm(d)
    noise = rng.standard_normal((N, D)) * 0.002
    noise -= (noise @ d)[:, None] * d
    X = (mid + noise).astype(np.float32)
    X[5, 1] = np.nan; X[6, 0] = np.inf; X[7, 2] = -np.inf
    X[8] *= np.float32(1e20); X[9] *= np.float32(1e-22); X[10] = 0
    for scale, bad in ((1.0, None), (1.0, (0, np.nan)), (1.0, (70, np.nan)), (1.0, (9, np.inf)), (1e-20, None), (3e18, None), (2e19, None)):
        Cs, Xs = Cn * np.float32(scale), X * np.float32(scale)
        if bad:
            Cs[bad[0], 1] = bad[1]
        got, gd = backend.kmeans_assign(Xs, Cs, want_dist=True)
        want, wd = oracle_assign(cpu_libs, Xs, Cs)
        assert np.array_equal(got, want), (scale, bad)
        assert np.array_equal(gd, wd, equal_nan=True), (scale, bad)


def test_tensor_core_assign_points_far_from_small_centroids(backend, cpu_libs):
    """Points up to 2^20 times longer than every centroid, on all sides, with padded centroids in the last group."""
    rng = np.random.default_rng(17)
    for D in (4, 8, 16):
        Cn = (rng.standard_normal((41, D)) * 0.02).astype(np.float32)
        X = rng.standard_normal((6000, D)).astype(np.float32) * np.exp2(rng.integers(-8, 14, (6000, 1))).astype(np.float32)
        got, gd = backend.kmeans_assign(X, Cn, want_dist=True)
        want, wd = oracle_assign(cpu_libs, X, Cn)
        assert np.array_equal(got, want) and np.array_equal(gd, wd)


@pytest.mark.parametrize("D,K", [(4, 256), (4, 7), (8, 256), (8, 100), (8, 264), (16, 256), (16, 12), (3, 20)])
@pytest.mark.parametrize("off_x,off_c", [(4, 0), (0, 4), (8, 12)])
def test_arrays_at_any_float(backend, cpu_libs, D, K, off_x, off_c):
    """Points or centroids that start at a float but not at 16 bytes (a caller's own offset into a registered range): same codes,
    distances and counts, no 16-byte load of them anywhere."""
    rng = np.random.default_rng(D * 1000 + K + off_x)
    N, be = 3001, backend
    X = (rng.standard_normal((N, D)) * 0.02).astype(np.float32)
    Cn = (rng.standard_normal((K, D)) * 0.02).astype(np.float32)
    dX, dC = be.alloc(X.nbytes + 16), be.alloc(Cn.nbytes + 16)
    be.write(dX, X, off_x); be.write(dC, Cn, off_c)
    di, dd, ds, dc, dn = be.alloc(N * 4), be.alloc(N * 4), be.alloc(K * D * 4), be.alloc(K * 4), be.alloc(8)
    want, wd = oracle_assign(cpu_libs, X, Cn)
    for call in ("assign", "lloyd"):
        if call == "assign":
            be._check(be.lib.ibcu_kmeans_assign(be.ctx, dX.ptr + off_x, N, D, dC.ptr + off_c, K, di.ptr, dd.ptr))
        else:
            be._check(be.lib.ibcu_kmeans_lloyd_iter(be.ctx, dX.ptr + off_x, N, D, dC.ptr + off_c, K, di.ptr, dd.ptr, ds.ptr, dc.ptr, dn.ptr))
        be.sync()
        assert np.array_equal(be.download(di, np.int32, N), want), call
        assert np.array_equal(be.download(dd, np.float32, N), wd), call
    assert np.array_equal(be.download(dc, np.int32, K), np.bincount(want, minlength=K))


def _iteration_sums(X, codes, K, tables):
    """The sums of a fused iteration, bit for bit: tile t of 128 points goes to block t % 148 as its tile i. Rows of a quarter of a tile that share a
    cluster are summed in index order in FP32, and the sums added, tile after tile, to that quarter's table for i % 3 (twelve tables) or its only
    one (four). A block's tables are joined in double in order, blocks in double by eight interleaved groups."""
    N, D = X.shape
    nb = min((N + 127) // 128, 148)
    p = np.arange(N)
    group, inv = np.unique((p // 32) * K + codes, return_inverse=True)       # (tile, quarter, cluster), ascending
    tile, q, k = group // K // 4, group // K % 4, group % K
    i, b = tile // nb, tile % nb
    key = (b * tables + (q + 4 * (i % 3) if tables == 12 else q)) * K + k
    out = np.empty((K, D), np.float32)
    for d in range(D):
        s = np.zeros(len(group), np.float32)
        np.add.at(s, inv, X[:, d])                           # one after the other, in index order
        t = np.zeros(nb * tables * K, np.float32)
        np.add.at(t, key, s)
        t = t.reshape(nb, tables, K).astype(np.float64)
        total = t[:, 0].copy()
        for w in range(1, tables):
            total += t[:, w]
        part = total.astype(np.float32).astype(np.float64)
        g = np.zeros((8, K))
        for blk in range(nb):
            g[blk % 8] += part[blk]
        out[:, d] = ((g[0] + g[1]) + (g[2] + g[3])) + ((g[4] + g[5]) + (g[6] + g[7]))
    return out


@pytest.mark.parametrize("N,D,K,tables", [
    (148 * 128 * 26 + 1, 4, 256, 12), (148 * 128 * 26 + 1, 4, 200, 12), (148 * 128 * 14 - 77, 8, 256, 12), (148 * 128 * 25 + 4000, 8, 40, 12),
    (148 * 128 * 26 + 1, 16, 64, 12), (148 * 128 * 26 + 1, 16, 200, 4), (148 * 128 * 27 - 5, 16, 256, 4), (148 * 128 * 200 + 40, 4, 8, 12),
])
def test_fused_iteration_at_length(backend, cpu_libs, N, D, K, tables):
    """Every ring of the kernel wrapped (more than twelve tiles a block; shared tables from tile 4 on): codes, distances and counts are the
    checker's, the sums are the stated order's bits and within what a chain of one add per tile may err, and iterations launched without a
    wait between them give what waited-for ones give."""
    rng = np.random.default_rng(N + D + K)
    X = (rng.standard_normal((N, D), dtype=np.float32) * np.float32(0.02))
    X[rng.random(N) < 0.4] *= np.float32(0.1)                # a crowd around the origin: few clusters take many points
    X[rng.random(N) < 0.2] = X[5]                             # and one point over and over
    Cn = X[:K].copy()
    Cn[0] = 0
    h = _lloyd_gpu(backend, X, Cn, 3)
    want, wd = oracle_assign(cpu_libs, X, Cn)
    assert np.array_equal(h[0]["idx"], want)
    assert np.array_equal(h[0]["counts"], np.bincount(want, minlength=K))
    assert abs(h[0]["inertia"] - wd.astype(np.float64).sum()) <= 1e-11 * wd.astype(np.float64).sum()
    assert np.array_equal(h[0]["sums"], _iteration_sums(X, want, K, tables))
    assert np.array_equal(h[1]["sums"], _iteration_sums(X, h[1]["idx"], K, tables))
    adds = 31 + -(-N // (128 * 148)) // (tables // 4) + 1 + 2           # within a quarter, tiles of a table, the block's sum and the total rounded
    for d in range(D):
        ref = np.bincount(want, weights=X[:, d].astype(np.float64), minlength=K)
        mag = np.bincount(want, weights=np.abs(X[:, d]).astype(np.float64), minlength=K)
        assert np.all(np.abs(h[0]["sums"][:, d] - ref) <= adds * 2.0 ** -24 * mag)
    be = backend
    dX, dC = be.upload(X), be.upload(Cn)
    di, dd, ds, dc, dn = be.alloc(N * 4), be.alloc(N * 4), be.alloc(K * D * 4), be.alloc(K * 4), be.alloc(8)
    for _ in range(3):
        be._check(be.lib.ibcu_kmeans_lloyd_iter(be.ctx, dX.ptr, N, D, dC.ptr, K, di.ptr, dd.ptr, ds.ptr, dc.ptr, dn.ptr))
    be.sync()
    assert np.array_equal(be.download(di, np.int32, N), h[2]["idx"])
    assert np.array_equal(be.download(dd, np.float32, N), oracle_assign(cpu_libs, X, h[1]["C"])[1])
    assert np.array_equal(be.download(dC, np.float32, K * D).reshape(K, D), h[2]["C"])
    assert np.array_equal(be.download(ds, np.float32, K * D).reshape(K, D), h[2]["sums"])
    for b in (dX, dC, di, dd, ds, dc, dn):
        b.free(); be._bufs.remove(b)


@pytest.mark.parametrize("D,K", [(4, 256), (4, 130), (8, 250), (8, 33), (16, 256), (16, 49)])
def test_many_points_the_filter_cannot_decide(backend, cpu_libs, D, K):
    """Warps in which few, about the limit, or all rows are undecided: equal centroids, points on a grid (ties between any groups), with NaN and
    Inf centroids among them, and a NaN centroid 0, from which the reference's scan never gets away."""
    rng = np.random.default_rng(D * K)
    N = 41000                                                # past 37888 points, where every one of these goes to the tensor cores
    base = (rng.standard_normal((N, D)) * 0.02).astype(np.float32)
    grid = (np.round(base / 0.02) * 0.02).astype(np.float32)
    for name, X in [("zeros", np.zeros_like(base)), ("grid", grid)] + [(f, np.where(rng.random((N, 1)) < f, 0, base).astype(np.float32)) for f in (0.02, 0.3, 0.5, 0.7)]:
        Cn = X[:K].copy()
        Cn[K // 2] = 0; Cn[1] = 0                            # the same centroid in two groups
        for bad in (None, (K - 1, np.nan), (2, np.inf), (0, np.nan)):
            Cs = Cn.copy()
            if bad:
                Cs[bad[0], D - 1] = bad[1]
            want, wd = oracle_assign(cpu_libs, X, Cs)
            got, gd = backend.kmeans_assign(X, Cs, want_dist=True)
            assert np.array_equal(got, want) and np.array_equal(gd, wd, equal_nan=True), (name, bad)
            h = _lloyd_gpu(backend, X, Cs, 1)[0]
            assert np.array_equal(h["idx"], want), (name, bad)
            assert np.array_equal(h["counts"], np.bincount(want, minlength=K)), (name, bad)


@pytest.mark.parametrize("D", [4, 8, 16])
def test_fused_iteration_on_what_the_filter_cannot_decide(backend, cpu_libs, D):
    """Near ties across groups, NaN, Inf, squares that overflow or vanish, and points up to 2^20 times longer than every centroid, through an iteration,
    which takes the tensor cores at every size: codes and distances are the checker's."""
    rng = np.random.default_rng(300 + D)
    be, K, N = backend, 72, 9000
    Cn = (rng.standard_normal((K, D)) * 0.02).astype(np.float32)
    d = Cn[60].astype(np.float64) - Cn[3]; d /= np.linalg.norm(d)
    noise = rng.standard_normal((N, D)) * 0.002
    near = ((Cn[3].astype(np.float64) + Cn[60]) / 2 + noise - (noise @ d)[:, None] * d).astype(np.float32)
    near[5, 1] = np.nan; near[6, 0] = np.inf; near[7, 2] = -np.inf
    near[8] *= np.float32(1e20); near[9] *= np.float32(1e-22); near[10] = 0
    far = rng.standard_normal((N, D)).astype(np.float32) * np.exp2(rng.integers(-8, 14, (N, 1))).astype(np.float32)
    cases = [(far, Cn[:41], 1.0, None)] + [(near, Cn, s, b) for s, b in ((1.0, None), (1.0, (0, np.nan)), (1.0, (70, np.nan)), (1.0, (9, np.inf)), (1e-20, None), (3e18, None), (2e19, None))]
    for X, C0, scale, bad in cases:
        Xs, Cs = X * np.float32(scale), C0 * np.float32(scale)
        if bad:
            Cs[bad[0], 1] = bad[1]
        k = len(Cs)
        bufs = [be.upload(Xs), be.upload(Cs), be.alloc(N * 4), be.alloc(N * 4), be.alloc(k * D * 4), be.alloc(k * 4), be.alloc(8)]
        dX, dC, di, dd, ds, dc, dn = bufs
        be._check(be.lib.ibcu_kmeans_lloyd_iter(be.ctx, dX.ptr, N, D, dC.ptr, k, di.ptr, dd.ptr, ds.ptr, dc.ptr, dn.ptr))
        want, wd = oracle_assign(cpu_libs, Xs, Cs)
        assert np.array_equal(be.download(di, np.int32, N), want), (scale, bad)
        assert np.array_equal(be.download(dd, np.float32, N), wd, equal_nan=True), (scale, bad)
        for b in bufs:
            b.free(); be._bufs.remove(b)
