"""The DP kernels pair by pair against the FP64 oracle: every precision
(FP32, compensated FP32, FP64) on every kernel (round-striped; anti-diagonal
with a warp, two warps or a CTA per pair; a lane per pair; band-relative
with a warp per pair), across
query/candidate shapes, bands and windows.
FP64 values must be bit-identical, compensated within 1e-9, FP32 within the
FP32 error bound (n+m+8)*2^-24, LCSS counts exact."""
import numpy as np
import pytest

from cudaruntime1_gb300 import datagen as G

pytestmark = pytest.mark.gpu


def _setup(nq, nc, lo, hi, seed):
    import torch
    ql = G.uniform_lengths(nq, lo, hi, seed)
    cl = G.uniform_lengths(nc, lo, hi, seed + 1)
    qp, qo = G.random_walks(nq, ql, seed + 2)
    cp, co = G.random_walks(nc, cl, seed + 3)
    # nearby pairs too: candidates 0..nq-1 are noisy copies of the queries, resampled
    for i in range(min(nq, nc)):
        src = np.linspace(0, ql[i] - 1, cl[i]).round().astype(int)
        cp[co[i]:co[i + 1]] = qp[qo[i] + src] + 0.3 * np.random.default_rng(i).standard_normal((cl[i], 2)).astype(np.float32)
    rng = np.random.default_rng(seed + 4)
    pairs = np.stack([rng.integers(0, nq, 600), rng.integers(0, nc, 600)], 1).astype(np.int32)
    pairs[:nq, 0] = np.arange(nq)
    pairs[:nq, 1] = np.arange(nq)
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in
           dict(qp=qp, qo=qo, cp=cp, co=co, pr=pairs).items()}
    return qp, qo, cp, co, pairs, dev, int(ql.max()), int(cl.max())


CASES = [
    ("dtw", dict(band_pct=10, cost=0), 16, 120),
    ("dtw", dict(band_pct=10, cost=0), 64, 512),
    ("dtw", dict(band_pct=30, cost=1), 8, 60),
    ("dtw", dict(band_pct=-1, cost=0), 2, 40),
    ("frechet", dict(), 2, 30),
    ("frechet", dict(), 20, 90),
    ("lcss", dict(epsilon=1.0, delta=5), 10, 150),
    ("lcss", dict(epsilon=0.5, delta=-1), 2, 28),
    # full rows past 31*4+1 columns: anti-diagonal passes with R = 8 and 16
    ("dtw", dict(band_pct=-1, cost=0), 130, 480),
    ("frechet", dict(), 130, 240),
    ("lcss", dict(epsilon=0.5, delta=200), 130, 300),
]


@pytest.mark.parametrize("measure,kw,lo,hi", CASES)
def test_dp_pairs_all_kernels(tsim, cuda_ctx, oracle, measure, kw, lo, hi):
    import torch
    from cudaruntime1_gb300 import api
    qp, qo, cp, co, pairs, dev, mq, mc = _setup(12, 80, lo, hi, 31 + lo + hi)
    okw = dict(kw)
    if "epsilon" in okw:
        okw["eps"] = okw.pop("epsilon")
    want = np.array([oracle.pair(measure, qp[qo[a]:qo[a + 1]], cp[co[b]:co[b + 1]], **okw)
                     for a, b in pairs])
    n_ = np.diff(qo)[pairs[:, 0]]
    m_ = np.diff(co)[pairs[:, 1]]
    fp32 = {}
    for kernel in (1, 2, 3, 4, 5, 6):
        for precision in ((0,) if measure == "lcss" else (0, 1, 2)):
            o32 = torch.full((len(pairs),), float("nan"), dtype=torch.float32, device="cuda")
            o64 = torch.full((len(pairs),), float("nan"), dtype=torch.float64, device="cuda")
            ctx = cuda_ctx
            api.dp_pairs(ctx, measure, precision, kernel, dev["qp"].data_ptr(), dev["qo"].data_ptr(),
                         mq, dev["cp"].data_ptr(), dev["co"].data_ptr(), mc, dev["pr"].data_ptr(),
                         len(pairs), o32.data_ptr(), o64.data_ptr(), **kw)
            torch.cuda.synchronize()
            got = (o32 if precision == 0 else o64).cpu().numpy().astype(np.float64)
            if precision == 0:
                fp32[kernel] = o32.cpu().numpy()
            w = want ** 2 if measure == "frechet" else want  # kernels report Frechet squared
            tag = (measure, kernel, precision)
            assert np.array_equal(np.isfinite(got), np.isfinite(w)), tag
            f = np.isfinite(w)
            if measure == "lcss":
                assert np.array_equal(got, w), tag
                continue
            rel = np.abs(got[f] - w[f]) / np.maximum(w[f], 1e-30)
            if precision == 2:
                ok = np.array_equal(got[f], w[f]) if measure != "frechet" else rel.max() <= 1e-15
                assert ok, (tag, rel.max())
            elif precision == 1:  # DTW: 4u from the FP32 costs; Frechet: double-float
                lim = 4.5 * 2.0 ** -24 if measure == "dtw" else 1e-9
                assert rel.max() <= lim, (tag, rel.max(), np.argmax(rel), pairs[f][np.argmax(rel)])
            else:
                bound = (n_[f] + m_[f] + 8) * 2.0 ** -24 * 1.01 + 1e-12
                assert np.all(rel <= bound), (tag, rel.max(), np.argmax(rel / bound))
    # the same cells with the same operations: FP32 values agree to the bit
    # between the warp-per-pair, lane-per-pair and band-relative kernels
    for kernel in (5, 6):
        assert np.array_equal(fp32[2].view(np.uint32), fp32[kernel].view(np.uint32)), \
            (measure, kernel)


@pytest.mark.parametrize("m,kernel", [(31, 2), (32, 2), (33, 2), (63, 4), (64, 4), (65, 4),
                                      (255, 3), (256, 3), (257, 3)])
@pytest.mark.parametrize("measure", ["dtw", "frechet", "lcss"])
def test_dp_full_rows_as_wide_as_the_lanes(tsim, cuda_ctx, oracle, measure, m, kernel):
    """Full rows of as many columns as a warp, two warps or a CTA has lanes
    (one row per lane), queries of several rounds of lanes: a group's first
    diagonal is outside the matrix, not the end of the row above it."""
    import torch
    from cudaruntime1_gb300 import api
    cp, co = G.random_walks(40, m, 900 + m, start_range=2.0)
    qp, qo = G.random_walks(4, [m + 2, 2 * m + 5, 3 * m, 4 * m + 1], 901 + m, start_range=2.0)
    pairs = np.stack(np.meshgrid(np.arange(4), np.arange(40), indexing="ij"), -1).reshape(-1, 2)
    kw, okw = (dict(epsilon=2.0), dict(eps=2.0)) if measure == "lcss" else ({}, {})
    want = np.array([oracle.pair(measure, qp[qo[a]:qo[a + 1]], cp[co[b]:co[b + 1]], **okw)
                     for a, b in pairs])
    want = want ** 2 if measure == "frechet" else want
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
           (qp, np.asarray(qo), cp, np.asarray(co), pairs.astype(np.int32))]
    for precision in (0,) if measure == "lcss" else (0, 1):
        out = torch.full((len(pairs),), float("nan"), device="cuda",
                         dtype=(torch.float32, torch.float64)[precision])
        api.dp_pairs(cuda_ctx, measure, precision, kernel, dev[0].data_ptr(), dev[1].data_ptr(),
                     4 * m + 1, dev[2].data_ptr(), dev[3].data_ptr(), m, dev[4].data_ptr(),
                     len(pairs), out.data_ptr(), out.data_ptr(), **kw)
        torch.cuda.synchronize()
        got = out.cpu().numpy().astype(np.float64)
        # FP32: 4 roundings a cost and one per cell of a path of at most 5 m cells
        lim = 0.0 if measure == "lcss" else ((5 * m + 8) * 2.0 ** -24 * 1.01 if precision == 0
                                             else 4.5 * 2.0 ** -24)
        assert np.all(np.abs(got - want) <= lim * want), (precision, np.abs(got - want).max())


# the edges of a lane's rows, of a half warp's, a warp's and several strips of
# rows, and of the staged side; (320, 260): several strips either way round
STRIP_SHAPES = [(1, 1), (1, 40), (33, 2), (31, 32), (64, 65), (127, 129), (128, 128), (16, 511),
                (257, 255), (256, 300), (320, 260), (513, 40), (700, 600)]


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("measure,kw", [("dtw", dict(cost=0)), ("dtw", dict(cost=1)),
                                        ("frechet", {})])
def test_dp_full_rows_by_strips(tsim, cuda_ctx, measure, kw, many):
    """Full rows, the kernel chosen by the library, against the round-striped
    one: the same cells with the same operations, so the same bits; a few
    pairs (a warp each) and more than eight per SM (two to a warp, where one
    side is short)."""
    import torch
    from cudaruntime1_gb300 import api
    for shape in STRIP_SHAPES:
        nc = 1400 if many else 37
        if many and max(shape) > 520:
            continue
        lens = np.full(nc, shape[1])
        lens[::3] = np.maximum(1, shape[1] - np.arange(len(lens[::3])) % 7)  # ragged
        qp, qo = G.random_walks(2, [shape[0], max(1, shape[0] - 1)], 77, start_range=10.0)
        cp, co = G.random_walks(nc, lens, 78, start_range=10.0)
        pairs = np.stack(np.meshgrid(np.arange(2), np.arange(nc), indexing="ij"), -1)
        dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
               (qp, np.asarray(qo), cp, np.asarray(co), pairs.reshape(-1, 2).astype(np.int32))]
        for precision in (0, 1):
            out = []
            for kernel in (1, 0):
                o = torch.full((2 * nc,), float("nan"), device="cuda",
                               dtype=(torch.float32, torch.float64)[precision])
                api.dp_pairs(cuda_ctx, measure, precision, kernel, dev[0].data_ptr(),
                             dev[1].data_ptr(), shape[0], dev[2].data_ptr(), dev[3].data_ptr(),
                             shape[1], dev[4].data_ptr(), 2 * nc, o.data_ptr(), o.data_ptr(), **kw)
                torch.cuda.synchronize()
                out.append(o.cpu().numpy())
            assert np.array_equal(out[0], out[1]), (shape, precision)


def test_frechet_fp64_rescore_of_long_pairs(tsim, cuda_ctx, oracle):
    """The exact FP64 re-score over one and several strips of rows: bit for
    bit the oracle's values."""
    lens = np.concatenate([np.arange(120, 140), np.arange(250, 262), [32, 500, 513]])
    cp, co = G.random_walks(len(lens), lens, 5, start_range=10.0)
    qp, qo = G.random_walks(4, [90, 128, 257, 520], 6, start_range=10.0)
    db = tsim.Database(cuda_ctx, cp, co)
    want_ids, want = oracle.knn("frechet", qp, qo, cp, co, 20)
    import torch
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (qp, np.asarray(qo, np.int64))]
    ids = torch.empty(4 * 20, dtype=torch.int32, device="cuda")
    d, d64 = torch.empty(80, device="cuda"), torch.empty(80, dtype=torch.float64, device="cuda")
    for flags in (tsim.api.FLAG_FP64_RESCORE, tsim.api.FLAG_FP64_RESCORE | tsim.api.FLAG_ALWAYS_PRUNE):
        tsim.knn_device(cuda_ctx, db, dev[0].data_ptr(), dev[1].data_ptr(), 4, 520, ids.data_ptr(),
                        d.data_ptr(), d64.data_ptr(), "frechet", 20, flags=flags)
        cuda_ctx.synchronize()
        assert np.array_equal(ids.cpu().numpy().reshape(4, 20), want_ids)
        assert np.array_equal(d64.cpu().numpy().reshape(4, 20), want)
    db.close()


@pytest.mark.parametrize("steps", [1, 16, 100])
def test_frechet_fp64_among_close_costs(tsim, cuda_ctx, oracle, steps):
    """Pairs whose optimum is one of several FP64 costs that FP32 cannot tell
    apart -- a few, up to 64, more -- with cells below and above them, over
    one to 32 words of rows, more rows than that, and columns around the
    32-column blocks: bit for bit the oracle's values."""
    rng = np.random.default_rng(steps)

    def walks(lens, near, far, unit, levels):
        x = [np.where(rng.random(n) < 0.6, near + rng.integers(0, levels, n) * unit,
                      rng.choice(far, n)) for n in lens]
        for w in x:
            w[0] = w[-1] = near
        off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
        x = np.concatenate(x)
        return np.stack([x, np.zeros_like(x)], 1).astype(np.float32), off

    # 0 and 2 are as far from 1; 0.2 is near 0 and far from 2, 1.8 the reverse
    qp, qo = walks([1, 31, 32, 33, 64, 257, 1024, 1025], 0.0, [2.0], 2.0 ** -26, steps)
    cp, co = walks([1, 2, 31, 32, 33, 63, 64, 65, 96, 300, 1023, 1024, 1025, 1500], 1.0, [0.2, 1.8],
                   2.0 ** -23, 3)
    db = tsim.Database(cuda_ctx, cp, co)
    want_ids, want = oracle.knn("frechet", qp, qo, cp, co, 14)
    import torch
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (qp, qo)]
    ids = torch.empty(8 * 14, dtype=torch.int32, device="cuda")
    d = torch.empty(8 * 14, device="cuda")
    d64 = torch.empty(8 * 14, dtype=torch.float64, device="cuda")
    tsim.knn_device(cuda_ctx, db, dev[0].data_ptr(), dev[1].data_ptr(), 8, 1025, ids.data_ptr(),
                    d.data_ptr(), d64.data_ptr(), "frechet", 14, flags=tsim.api.FLAG_FP64_RESCORE)
    cuda_ctx.synchronize()
    assert np.array_equal(ids.cpu().numpy().reshape(8, 14), want_ids)
    assert np.array_equal(d64.cpu().numpy().reshape(8, 14), want)
    db.close()


@pytest.mark.parametrize("delta", [0, 1, 3, 15, 16, 20, 31])
def test_lcss_window_bit_vectors(tsim, cuda_ctx, oracle, delta):
    """Windowed LCSS, the kernel chosen by the library, against the oracle:
    dense and sparse matches, one-point sides, rows and columns past the
    other side's window, gaps of more than 64 columns between matches; and
    within kNN, where the queries' window boxes skip columns."""
    import torch
    from cudaruntime1_gb300 import api
    cl = np.array([1, 2, 31, 32, 33, 64, 100, 200, 400] * 4)
    cp, co = G.random_walks(len(cl), cl, 41, start_range=4.0)
    qp, qo = G.random_walks(6, [1, 30, 64, 65, 129, 390], 42, start_range=4.0)
    far = qp[qo[5]:qo[6]].copy()  # a copy of the longest query, far away but for its ends
    far[8:-8] += 1e4
    cp = np.concatenate([cp, far])
    co = np.concatenate([co, [co[-1] + len(far)]])
    nc = len(co) - 1
    pairs = np.stack(np.meshgrid(np.arange(6), np.arange(nc), indexing="ij"), -1).reshape(-1, 2)
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
           (qp, np.asarray(qo), cp, np.asarray(co), pairs.astype(np.int32))]
    for eps in (0.25, 3.0):
        out = torch.full((len(pairs),), float("nan"), device="cuda")
        api.dp_pairs(cuda_ctx, "lcss", 0, 0, dev[0].data_ptr(), dev[1].data_ptr(), 390,
                     dev[2].data_ptr(), dev[3].data_ptr(), 400, dev[4].data_ptr(), len(pairs),
                     out.data_ptr(), epsilon=eps, delta=delta)
        torch.cuda.synchronize()
        want = np.array([oracle.pair("lcss", qp[qo[a]:qo[a + 1]], cp[co[b]:co[b + 1]], eps=eps,
                                     delta=delta) for a, b in pairs])
        assert np.array_equal(out.cpu().numpy(), want), eps
        db = tsim.Database(cuda_ctx, cp, co)
        ids, d, _ = tsim.knn(cuda_ctx, db, qp, qo, "lcss", 12, epsilon=eps, delta=delta,
                             flags=api.FLAG_ALWAYS_PRUNE)
        wi, wd = oracle.knn("lcss", qp, qo, cp, co, 12, eps=eps, delta=delta)
        assert np.array_equal(ids, wi) and np.array_equal(d, wd)
        db.close()


@pytest.mark.parametrize("stated,most", [(100, 200), (128, 128), (250, 60)])
@pytest.mark.parametrize("measure,kw", [("dtw", {}), ("dtw", dict(cost=1)), ("frechet", {})])
def test_full_rows_of_queries_longer_than_stated(tsim, cuda_ctx, oracle, measure, kw, stated, most):
    """Full rows, queries past the stated longest length -- by a point, past
    one strip of rows, past several -- against candidates that fit the
    staging: pair values are the bits of the round-striped kernel (given the
    true length), kNN answers the oracle's."""
    import torch
    from cudaruntime1_gb300 import api
    ql = [stated, stated + 1, 129, 257, 300, 513, 700, 40]
    cl = np.random.default_rng(3).integers(30, most + 1, 300)
    cl[0] = most
    qp, qo = G.random_walks(8, ql, 95, start_range=10.0)
    cp, co = G.random_walks(300, cl, 96, start_range=10.0)
    pairs = np.stack(np.meshgrid(np.arange(8), np.arange(300), indexing="ij"), -1).reshape(-1, 2)
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
           (qp, np.asarray(qo), cp, np.asarray(co), pairs.astype(np.int32))]
    for count in (300, len(pairs)):
        for precision in (0, 1):
            out = []
            for kernel, longest in ((1, max(ql)), (0, stated)):
                o = torch.full((count,), float("nan"), device="cuda",
                               dtype=(torch.float32, torch.float64)[precision])
                api.dp_pairs(cuda_ctx, measure, precision, kernel, dev[0].data_ptr(),
                             dev[1].data_ptr(), longest, dev[2].data_ptr(), dev[3].data_ptr(), most,
                             dev[4][len(pairs) - count:].data_ptr(), count, o.data_ptr(),
                             o.data_ptr(), **kw)
                torch.cuda.synchronize()
                out.append(o.cpu().numpy())
            assert np.array_equal(out[0], out[1]), (count, precision)
    db = tsim.Database(cuda_ctx, cp, co)
    want_ids, want = oracle.knn(measure, qp, qo, cp, co, 10, **kw)
    ids = torch.empty(80, dtype=torch.int32, device="cuda")
    d, d64 = torch.empty(80, device="cuda"), torch.empty(80, dtype=torch.float64, device="cuda")
    for flags in (0, tsim.api.FLAG_ALWAYS_PRUNE):
        tsim.knn_device(cuda_ctx, db, dev[0].data_ptr(), dev[1].data_ptr(), 8, stated,
                        ids.data_ptr(), d.data_ptr(), d64.data_ptr(), measure, 10,
                        flags=flags | tsim.api.FLAG_FP64_RESCORE, **kw)
        cuda_ctx.synchronize()
        assert np.array_equal(ids.cpu().numpy().reshape(8, 10), want_ids)
        assert np.array_equal(d64.cpu().numpy().reshape(8, 10), want)
    db.close()


@pytest.mark.parametrize("measure", ["dtw", "frechet"])
@pytest.mark.parametrize("longest", [1710, 1712])
def test_compensated_full_rows_past_one_cta_an_sm(tsim, cuda_ctx, measure, longest):
    """Compensated full rows of more pairs than one block an SM holds, on both
    sides of the length from which they are round-striped: the same bits, for
    pairs of every length, as from fewer pairs."""
    import torch
    from cudaruntime1_gb300 import api
    qp, qo = G.random_walks(2, [longest, 33], 99, start_range=10.0)
    cp, co = G.random_walks(12, [longest, 1, 2, 31, 32, 33, 64, 100, 255, 256, 257, 300], 100,
                            start_range=10.0)
    pairs = np.stack(np.meshgrid(np.arange(2), np.arange(12), indexing="ij"), -1).reshape(-1, 2)
    pairs = np.concatenate([pairs] + [pairs[13:]] * 60).astype(np.int32)  # short ones again and again
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
           (qp, np.asarray(qo), cp, np.asarray(co), pairs)]
    out = []
    for count in (len(pairs), 24):
        o = torch.full((len(pairs),), float("nan"), dtype=torch.float64, device="cuda")
        api.dp_pairs(cuda_ctx, measure, 1, 0, dev[0].data_ptr(), dev[1].data_ptr(), longest,
                     dev[2].data_ptr(), dev[3].data_ptr(), longest, dev[4].data_ptr(), count, 0,
                     o.data_ptr())
        torch.cuda.synchronize()
        out.append(o.cpu().numpy())
    assert len(pairs) > 608 and np.array_equal(out[0][:24], out[1][:24])
    assert np.array_equal(out[0][24:], np.tile(out[1][13:24], 60))


@pytest.mark.parametrize("band", [0, 1, 2])
@pytest.mark.parametrize("cost", [0, 1])
def test_dp_pairs_with_rows_the_band_leaves_empty(tsim, cuda_ctx, oracle, band, cost):
    """Narrow bands of sides of very different lengths, where some rows (or
    columns) admit no cell and the pair has no path: the oracle's infinities on
    every kernel, few pairs and enough for a lane each, and its answer in kNN."""
    import torch
    from cudaruntime1_gb300 import api
    ql = [2, 9, 20, 31, 40, 60, 200]
    cl = np.concatenate([np.arange(2, 22), [40, 60, 100, 200, 399]] * 30)
    qp, qo = G.random_walks(7, ql, 103, start_range=10.0)
    cp, co = G.random_walks(len(cl), cl, 104, start_range=10.0)
    pairs = np.stack(np.meshgrid(np.arange(7), np.arange(len(cl)), indexing="ij"), -1).reshape(-1, 2)
    want = np.array([oracle.pair("dtw", qp[qo[a]:qo[a + 1]], cp[co[b]:co[b + 1]], band_pct=band,
                                 cost=cost) for a, b in pairs])
    assert np.isinf(want).any() and np.isfinite(want).any()
    lens = np.diff(qo)[pairs[:, 0]] + np.diff(co)[pairs[:, 1]]
    many = np.tile(pairs, (12, 1))
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
           (qp, np.asarray(qo), cp, np.asarray(co), many.astype(np.int32))]
    for count in (len(pairs), len(many)):
        for kernel in range(7):
            o = torch.full((count,), float("nan"), device="cuda")
            api.dp_pairs(cuda_ctx, "dtw", 0, kernel, dev[0].data_ptr(), dev[1].data_ptr(), 200,
                         dev[2].data_ptr(), dev[3].data_ptr(), 399, dev[4].data_ptr(), count,
                         o.data_ptr(), band_pct=band, cost=cost)
            torch.cuda.synchronize()
            got = o.cpu().numpy().astype(np.float64).reshape(-1, len(pairs))
            fin = np.isfinite(want)
            assert np.array_equal(np.isfinite(got), np.broadcast_to(fin, got.shape)), (count, kernel)
            # 4 roundings a cost and one per cell of the path
            lim = (lens[fin] + 8) * 2.0 ** -24 * 1.01 * want[fin]
            assert np.all(np.abs(got[:, fin] - want[fin]) <= lim), (count, kernel)
    cp, co = G.random_walks(6000, G.uniform_lengths(6000, 4, 20, 105), 106, start_range=10.0)
    qp, qo = G.random_walks(20, [13, 20, 40, 70] * 5, 107, start_range=10.0)
    db = tsim.Database(cuda_ctx, cp, co)
    want_ids, want = oracle.knn("dtw", qp, qo, cp, co, 10, band_pct=band, cost=cost)
    for flags in (0, api.FLAG_NO_PRUNE):
        ids, d, _ = tsim.knn(cuda_ctx, db, qp, qo, "dtw", 10, band_pct=band, cost=cost, flags=flags)
        assert np.array_equal(ids, want_ids), flags
        assert np.array_equal(np.isfinite(d), np.isfinite(want)), flags
    db.close()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("measure,kw", [("dtw", dict(cost=0)), ("dtw", dict(cost=1)), ("frechet", {})])
def test_full_rows_with_points_that_are_not_finite(tsim, cuda_ctx, measure, kw, bad):
    """The strips' own points at infinity beside a trajectory's: the same pairs
    have a finite value as on the round-striped kernel, and the same bits;
    strips of a pair and of two pairs a warp."""
    import torch
    from cudaruntime1_gb300 import api
    for longest, nc in ((40, 30), (120, 700), (300, 30)):
        ql, cl = G.uniform_lengths(4, 2, longest, 61), G.uniform_lengths(nc, 2, longest, 62)
        qp, qo = G.random_walks(4, ql, 63, start_range=10.0)
        cp, co = G.random_walks(nc, cl, 64, start_range=10.0)
        rng = np.random.default_rng(65)
        for q in (0, 1):  # one in the middle; the last one
            qp[qo[q] + (ql[q] // 2 if q else ql[q] - 1), q] = bad
        for c in range(0, nc, 3):
            cp[co[c] + rng.integers(0, cl[c]), rng.integers(0, 2)] = bad if c % 2 else np.inf
        pairs = np.stack(np.meshgrid(np.arange(4), np.arange(nc), indexing="ij"), -1)
        dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in
               (qp, qo, cp, co, pairs.reshape(-1, 2).astype(np.int32))]
        for precision in (0, 1):
            out = []
            for kernel in (1, 0):
                o = torch.zeros(4 * nc, device="cuda",
                                dtype=(torch.float32, torch.float64)[precision])
                api.dp_pairs(cuda_ctx, measure, precision, kernel, dev[0].data_ptr(),
                             dev[1].data_ptr(), int(ql.max()), dev[2].data_ptr(),
                             dev[3].data_ptr(), int(cl.max()), dev[4].data_ptr(), 4 * nc,
                             o.data_ptr(), o.data_ptr(), **kw)
                torch.cuda.synchronize()
                out.append(o.cpu().numpy())
            fin = np.isfinite(out[0])
            assert fin.any() and not fin.all()
            assert np.array_equal(fin, np.isfinite(out[1])), (longest, precision)
            assert np.array_equal(out[0][fin], out[1][fin]), (longest, precision)


@pytest.mark.parametrize("lo,hi,band,npairs", [
    (480, 520, 100, 20), (480, 520, 100, 900), (300, 620, 100, 20), (500, 900, 60, 50),
    (900, 1100, 30, 3000), (2, 90, 60, 40), (2, 140, 60, 2000), (600, 1510, 3, 1500),
    (1500, 1502, 3, 1000), (1, 60, 5, 300)])
@pytest.mark.parametrize("precision", [0, 1])
def test_dp_pairs_picks_a_kernel_for_any_band(tsim, cuda_ctx, lo, hi, band, npairs, precision):
    """The kernel chosen by the library for banded pairs against the
    round-striped one: the same bits, wide bands and narrow ones, few pairs
    and many."""
    import torch
    from cudaruntime1_gb300 import api
    ql, cl = G.uniform_lengths(9, lo, hi, 71), G.uniform_lengths(40, lo, hi, 72)
    ql[0], cl[0] = hi, hi
    qp, qo = G.random_walks(9, ql, 73)
    cp, co = G.random_walks(40, cl, 74)
    rng = np.random.default_rng(75)
    pairs = np.stack([rng.integers(0, 9, npairs), rng.integers(0, 40, npairs)], 1).astype(np.int32)
    pairs[0] = 0
    dev = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (qp, qo, cp, co, pairs)]
    out = []
    for kernel in (1, 0):
        o = torch.zeros(npairs, device="cuda", dtype=(torch.float32, torch.float64)[precision])
        api.dp_pairs(cuda_ctx, "dtw", precision, kernel, dev[0].data_ptr(), dev[1].data_ptr(), hi,
                     dev[2].data_ptr(), dev[3].data_ptr(), hi, dev[4].data_ptr(), npairs,
                     o.data_ptr(), o.data_ptr(), band_pct=band)
        torch.cuda.synchronize()
        out.append(o.cpu().numpy())
    assert np.array_equal(out[0], out[1])
