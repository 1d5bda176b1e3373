"""Exact kNN on the GPU against the FP64 brute-force oracle: ids bit-exact
(ties by candidate index), FP64 distances bit-identical, float distances
within 1e-5 relative (they are the FP64 values rounded once)."""
import numpy as np
import pytest

from cudaruntime1_gb300 import datagen as G

pytestmark = pytest.mark.gpu
REL_TOL = 1e-5


def _db(nc, lo, hi, seed, step="normal"):
    lens = G.uniform_lengths(nc, lo, hi, seed)
    return G.random_walks(nc, lens, seed + 1, step=step)


def _device_knn(tsim, ctx, db, qp, qo, measure, k, **kw):
    import torch
    qpt = torch.from_numpy(qp).cuda()
    qot = torch.from_numpy(np.asarray(qo, np.int64)).cuda()
    nq = len(qo) - 1
    ids = torch.empty(nq * k, dtype=torch.int32, device="cuda")
    d = torch.empty(nq * k, dtype=torch.float32, device="cuda")
    d64 = torch.empty(nq * k, dtype=torch.float64, device="cuda")
    maxq = int(np.max(np.diff(qo)))
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    st = tsim.knn_device(ctx, db, qpt.data_ptr(), qot.data_ptr(), nq, maxq, ids.data_ptr(),
                         d.data_ptr(), d64.data_ptr(), measure, k, stats=True, **kw)
    torch.cuda.synchronize()
    return (ids.cpu().numpy().reshape(nq, k), d.cpu().numpy().reshape(nq, k),
            d64.cpu().numpy().reshape(nq, k), st)


CASES = [
    ("dtw", dict(band_pct=10, cost=0)),
    ("dtw", dict(band_pct=-1, cost=0)),
    ("dtw", dict(band_pct=20, cost=1)),
    ("lcss", dict(epsilon=0.5, delta=5)),
    ("lcss", dict(epsilon=0.25, delta=-1)),
    ("frechet", dict()),
    ("hausdorff", dict()),
]


@pytest.mark.parametrize("pruned", [False, True])
@pytest.mark.parametrize("measure,kw", CASES)
def test_knn_matches_fp64_oracle(tsim, cuda_ctx, oracle, measure, kw, pruned):
    cp, co = _db(700, 16, 120, 100)
    ql = G.uniform_lengths(9, 16, 120, 7)
    qp, qo = G.random_walks(9, ql, 8)
    k = 10
    db = tsim.Database(cuda_ctx, cp, co)
    okw = dict(kw)
    if "epsilon" in okw:
        okw["eps"] = okw.pop("epsilon")
    want_ids, want_d = oracle.knn(measure, qp, qo, cp, co, k, **okw)
    if pruned:  # the bound stages, which a request this small skips by default
        kw = dict(kw, flags=tsim.api.FLAG_ALWAYS_PRUNE)
    ids, d, d64, st = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, k, **kw)
    assert np.array_equal(ids, want_ids), (ids, want_ids)
    if measure == "lcss":
        assert np.array_equal(d.astype(np.float64), want_d)
    else:
        fin = np.isfinite(want_d)
        assert np.array_equal(np.isfinite(d64), fin)
        rel = np.abs(d.astype(np.float64)[fin] - want_d[fin]) / np.maximum(want_d[fin], 1e-30)
        assert rel.max() <= REL_TOL
        # DTW's compensated re-score (FP32 costs within 4 2^-24, path sum
        # compensated) and the other measures' FP32 values (FP64 only for
        # near-ties) are all within a few 2^-24 of FP64
        rel64 = np.abs(d64[fin] - want_d[fin]) / np.maximum(want_d[fin], 1e-30)
        assert rel64.max() <= 1e-6, rel64.max()
        # forced FP64 re-score: bit-identical to the FP64 oracle
        kw64 = dict(kw, flags=kw.get("flags", 0) | tsim.api.FLAG_FP64_RESCORE)
        ids2, _, d64b, st2 = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, k, **kw64)
        assert np.array_equal(ids2, want_ids)
        assert np.array_equal(d64b, want_d)
        assert st2["rescored_fp64"] >= np.isfinite(want_d).sum()
    # the host-pointer entry point gives the same answer
    ids_h, d_h, _ = tsim.knn(cuda_ctx, db, qp, qo, measure, k, **kw)
    assert np.array_equal(ids_h, ids) and np.array_equal(d_h, d)
    db.close()


def test_knn_edge_cases(tsim, cuda_ctx, oracle):
    # fewer candidates than k; single-point trajectories; duplicates (ties)
    cp, co = _db(5, 1, 6, 300)
    qp, qo = G.random_walks(3, [1, 4, 6], 301)
    db = tsim.Database(cuda_ctx, cp, co)
    for measure, kw, okw in [("dtw", dict(band_pct=10), dict(band_pct=10)),
                             ("frechet", {}, {}),
                             ("lcss", dict(epsilon=30.0, delta=2), dict(eps=30.0, delta=2))]:
        want_ids, want_d = oracle.knn(measure, qp, qo, cp, co, 8, **okw)
        ids, d, d64, _ = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 8, **kw)
        assert np.array_equal(ids, want_ids), (measure, ids, want_ids)
    db.close()
    # exact duplicates in the database: ties broken by index
    base, bo = G.random_walks(4, 30, 400)
    cp = np.concatenate([base, base[bo[1]:bo[2]], base[bo[1]:bo[2]]])
    co = np.concatenate([bo, [bo[-1] + 30, bo[-1] + 60]])
    db = tsim.Database(cuda_ctx, cp, co)
    qp = base[bo[1]:bo[2]].copy()
    qo = np.array([0, 30])
    for measure in ("dtw", "frechet", "lcss"):
        want_ids, _ = oracle.knn(measure, qp, qo, cp, co, 6)
        ids, _, _, _ = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 6)
        assert np.array_equal(ids, want_ids), (measure, ids, want_ids)
        assert list(ids[0][:3]) == [1, 4, 5]
    db.close()


def test_knn_longer_queries_than_candidates(tsim, cuda_ctx, oracle):
    cp, co = _db(300, 10, 40, 500)
    qp, qo = G.random_walks(4, [200, 150, 90, 300], 501)
    db = tsim.Database(cuda_ctx, cp, co)
    for measure, kw, okw in [("dtw", dict(band_pct=30), dict(band_pct=30)),
                             ("lcss", dict(epsilon=1.0, delta=4), dict(eps=1.0, delta=4))]:
        want_ids, want_d = oracle.knn(measure, qp, qo, cp, co, 5, **okw)
        ids, d, d64, _ = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 5, **kw)
        assert np.array_equal(ids, want_ids), measure
    db.close()


def test_context_destroyed_before_database(tsim):
    """Destroying a context releases its databases' device memory and
    detaches them; closing such a database afterwards is safe and using it is
    an error, whatever order Python collects the objects in."""
    ctx = tsim.Context(0)
    cp, co = _db(50, 8, 20, 700)
    db = tsim.Database(ctx, cp, co)
    qp, qo = G.random_walks(1, 10, 701)
    ids, _, _ = tsim.knn(ctx, db, qp, qo, "dtw", 3)
    ctx2 = tsim.Context(0)
    with pytest.raises(tsim._lib.TsimError):
        tsim.knn(ctx2, db, qp, qo, "dtw", 3)  # wrong context
    ctx.close()
    db.close()
    ctx2.close()


def test_host_calls_two_contexts_growing_requests(tsim, oracle):
    """Host-pointer kNN on two contexts of one thread, interleaved, with
    requests that grow (each context's device staging is its own and grows
    with the request); a NULL point array is an argument error."""
    import ctypes as C
    cp, co = _db(200, 8, 40, 720)
    ctxs = [tsim.Context(0), tsim.Context(0)]
    dbs = [tsim.Database(c, cp, co) for c in ctxs]
    for i, nq in enumerate([1, 3, 40, 2, 90]):
        qp, qo = G.random_walks(nq, G.uniform_lengths(nq, 4, 60, 730 + i), 740 + i)
        want_ids, _ = oracle.knn("dtw", qp, qo, cp, co, 4, band_pct=20)
        for c, db in zip(ctxs, dbs):
            ids, _, _ = tsim.knn(c, db, qp, qo, "dtw", 4, band_pct=20)
            assert np.array_equal(ids, want_ids), (nq, ids, want_ids)
    h = C.c_void_p()
    off = np.array([0, 3], np.int64)
    st = ctxs[0].L.tsim_db_create(ctxs[0].h, None, off.ctypes.data, 1, C.byref(h))
    assert st == tsim._lib.TSIM_ERR_INVALID_ARG and not h.value
    for db in dbs:
        db.close()
    for c in ctxs:
        c.close()


def test_euclidean_knn_prefix_rule_and_long_pairs(tsim, cuda_ctx, oracle):
    """Lock-step Euclidean: candidates of length 64 and a few of 1,100 points
    (> 1024: the FP64 accumulation branch) against queries of 1,100 points;
    a candidate is compared with the query's first m points."""
    rng = np.random.default_rng(9)
    lens = np.where(rng.random(600) < 0.02, 1100, 64)
    lens[:3] = 1100
    cp, co = G.random_walks(600, lens, 901, step="student_t")
    qp, qo = G.random_walks(5, 1100, 902, step="student_t")
    # plant near matches: candidate 1 = query 0 plus noise, candidate 7 = query 1 prefix
    cp[co[1]:co[2]] = qp[qo[0]:qo[0] + 1100] + 0.01
    cp[co[7]:co[8]] = qp[qo[1]:qo[1] + lens[7]] + 0.02
    db = tsim.Database(cuda_ctx, cp, co)
    want_ids, want_d = oracle.knn("euclidean", qp, qo, cp, co, 10)
    ids, d, d64, st = _device_knn(tsim, cuda_ctx, db, qp, qo, "euclidean", 10)
    assert np.array_equal(ids, want_ids)
    assert ids[0][0] == 1 and ids[1][0] == 7
    fin = np.isfinite(want_d)
    assert np.max(np.abs(d[fin] - want_d[fin]) / want_d[fin]) <= REL_TOL
    ids2, _, d64b, _ = _device_knn(tsim, cuda_ctx, db, qp, qo, "euclidean", 10,
                                   flags=tsim.api.FLAG_FP64_RESCORE)
    assert np.array_equal(ids2, want_ids) and np.array_equal(d64b, want_d)
    db.close()


def test_query_batches(tsim, cuda_ctx, oracle):
    """More query x candidate pairs than one batch holds: the queries are
    processed in slices with the same results."""
    cp, co = _db(70000, 8, 24, 950)
    qp, qo = G.random_walks(300, G.uniform_lengths(300, 8, 24, 951), 952)
    db = tsim.Database(cuda_ctx, cp, co)
    sel = [0, 137, 299]
    ids, d, d64, _ = _device_knn(tsim, cuda_ctx, db, qp, qo, "frechet", 4)
    for q in sel:
        sub_o = np.array([0, qo[q + 1] - qo[q]])
        wi, wd = oracle.knn("frechet", qp[qo[q]:qo[q + 1]], sub_o, cp, co, 4)
        assert np.array_equal(ids[q], wi[0]), q
    db.close()


@pytest.mark.parametrize("measure,kw", [("dtw", dict(band_pct=10)), ("lcss", dict(epsilon=0.5, delta=5)),
                                        ("hausdorff", {})])
def test_pruning_never_changes_the_answer(tsim, cuda_ctx, measure, kw):
    """TSIM_FLAG_NO_PRUNE refines every pair; the pruned pipeline must return
    the same ids and distances."""
    cp, co = _db(1500, 20, 90, 1200)
    qp, qo = G.random_walks(6, G.uniform_lengths(6, 20, 90, 1201), 1202)
    db = tsim.Database(cuda_ctx, cp, co)
    ids, d, _, st = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 10,
                                flags=tsim.api.FLAG_ALWAYS_PRUNE, **kw)
    ids2, d2, _, st2 = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 10,
                                   flags=tsim.api.FLAG_NO_PRUNE, **kw)
    assert np.array_equal(ids, ids2) and np.array_equal(d, d2)
    assert st2["pairs_refined"] >= 6 * 1500 and st["pairs_refined"] < st2["pairs_refined"]
    db.close()


def test_graph_replay_follows_inputs(tsim, cuda_ctx, oracle):
    """Repeated requests of one shape replay a captured CUDA graph; the graph
    re-reads its input buffers, so changed query points give the new answer."""
    import torch
    cp, co = _db(900, 20, 60, 1300)
    qp, qo = G.random_walks(24, G.uniform_lengths(24, 20, 60, 1301), 1302)
    db = tsim.Database(cuda_ctx, cp, co)
    stream = torch.cuda.Stream()
    cuda_ctx.set_stream(stream.cuda_stream)
    qpt = torch.from_numpy(qp).cuda()
    qot = torch.from_numpy(qo).cuda()
    k = 5
    ids = torch.empty(24 * k, dtype=torch.int32, device="cuda")
    d = torch.empty(24 * k, dtype=torch.float32, device="cuda")
    want, _ = oracle.knn("dtw", qp, qo, cp, co, k, band_pct=10)
    cuda_ctx.counters(reset=True)
    for it in range(4):  # eager, capture, replay, replay
        tsim.knn_device(cuda_ctx, db, qpt.data_ptr(), qot.data_ptr(), 24, 60, ids.data_ptr(),
                        d.data_ptr(), None, "dtw", k, band_pct=10)
        stream.synchronize()
        assert np.array_equal(ids.cpu().numpy().reshape(24, k), want), it
    launches = cuda_ctx.counters(reset=True)["launches"]
    assert launches > 0
    qp2 = qp[::-1].copy()  # new query points in the same buffer
    qpt.copy_(torch.from_numpy(qp2))
    stream.synchronize()
    tsim.knn_device(cuda_ctx, db, qpt.data_ptr(), qot.data_ptr(), 24, 60, ids.data_ptr(),
                    d.data_ptr(), None, "dtw", k, band_pct=10)
    stream.synchronize()
    want2, _ = oracle.knn("dtw", qp2, qo, cp, co, k, band_pct=10)
    assert np.array_equal(ids.cpu().numpy().reshape(24, k), want2)
    cuda_ctx.set_stream(None)
    db.close()


@pytest.mark.parametrize("measure,kw", [("dtw", dict(band_pct=-1, cost=0)), ("frechet", dict())])
def test_knn_full_rows_long_candidates(tsim, cuda_ctx, oracle, measure, kw):
    """Full-row DP of candidates longer than 31*4+1 points: anti-diagonal
    passes with 8 and 16 rows per lane-group, with early abandon."""
    cp, co = _db(600, 130, 480, 300)
    ql = G.uniform_lengths(6, 130, 480, 301)
    qp, qo = G.random_walks(6, ql, 302)
    db = tsim.Database(cuda_ctx, cp, co)
    want_ids, want_d = oracle.knn(measure, qp, qo, cp, co, 10, **kw)
    ids, d, d64, st = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 10, **kw)
    assert np.array_equal(ids, want_ids)
    rel = np.abs(d.astype(np.float64) - want_d) / np.maximum(want_d, 1e-30)
    assert rel.max() <= REL_TOL
    db.close()


@pytest.mark.parametrize("measure,kw", [("dtw", dict(band_pct=10)), ("lcss", dict(epsilon=0.5, delta=20))])
def test_knn_mixed_query_lengths_one_call(tsim, cuda_ctx, oracle, measure, kw):
    """Queries of 512, 600 and 1,100 points in one call: their sparse tables
    share a stride sized for the longest, although a 512-row table is larger
    than a 600-row one (rows are grouped in blocks beyond 512)."""
    cp, co = _db(1500, 40, 200, 400)
    qp, qo = G.random_walks(4, [512, 600, 300, 1100], 401)
    db = tsim.Database(cuda_ctx, cp, co)
    okw = dict(kw)
    if "epsilon" in okw:
        okw["eps"] = okw.pop("epsilon")
    want_ids, want_d = oracle.knn(measure, qp, qo, cp, co, 10, **okw)
    ids, d, _, _ = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 10,
                               flags=tsim.api.FLAG_ALWAYS_PRUNE, **kw)
    assert np.array_equal(ids, want_ids)
    db.close()


@pytest.mark.parametrize("pruned", [False, True])
def test_knn_k64_with_many_ties(tsim, cuda_ctx, oracle, pruned):
    """k at its maximum (64) over a database in which every trajectory occurs
    eight times: the block selections (radix passes over the packed keys,
    ties broken by candidate index) against the oracle."""
    base, bo = _db(60, 12, 70, 900)
    reps = 8
    parts, offs = [], [0]
    for r in range(reps):
        for t in range(60):
            seg = base[bo[t]:bo[t + 1]]
            parts.append(seg)
            offs.append(offs[-1] + len(seg))
    cp = np.concatenate(parts)
    co = np.array(offs, np.int64)
    ql = G.uniform_lengths(6, 12, 70, 901)
    qp, qo = G.random_walks(6, ql, 902)
    db = tsim.Database(cuda_ctx, cp, co)
    k = 64
    for measure, kw, okw in [("dtw", dict(band_pct=20), dict(band_pct=20)),
                             ("lcss", dict(epsilon=1.5, delta=-1), dict(eps=1.5, delta=-1)),
                             ("hausdorff", {}, {})]:
        want_ids, want_d = oracle.knn(measure, qp, qo, cp, co, k, **okw)
        if pruned:
            kw = dict(kw, flags=tsim.api.FLAG_ALWAYS_PRUNE)
        ids, d, _, _ = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, k, **kw)
        assert np.array_equal(ids, want_ids), (measure, pruned)
    db.close()


def test_frechet_fp64_window_and_tiny_values(tsim, cuda_ctx, oracle):
    """The exact FP64 Frechet re-score (FP64 costs only in the window around
    the FP32 optimum) against the oracle, bit for bit: exact duplicates (value
    0), near-duplicates whose optimum is below 1e-20 (every cell in FP64) and
    offsets that keep it in the window."""
    base, bo = G.random_walks(6, 40, 1200)
    parts, offs = [], [0]
    rng = np.random.default_rng(1201)
    for t in range(6):
        seg = base[bo[t]:bo[t + 1]].astype(np.float64)
        for scale in (0.0, 1e-12, 1e-3, 0.5):
            v = seg + scale * rng.standard_normal(seg.shape)
            parts.append(v.astype(np.float32))
            offs.append(offs[-1] + len(seg))
    cp = np.concatenate(parts)
    co = np.array(offs, np.int64)
    qp = np.concatenate([base[bo[t]:bo[t + 1]] for t in (0, 3)])
    qo = np.array([0, 40, 80], np.int64)
    db = tsim.Database(cuda_ctx, cp, co)
    k = 8
    want_ids, want_d = oracle.knn("frechet", qp, qo, cp, co, k)
    for flags in (tsim.api.FLAG_FP64_RESCORE,
                  tsim.api.FLAG_FP64_RESCORE | tsim.api.FLAG_ALWAYS_PRUNE):
        ids, _, d64, _ = _device_knn(tsim, cuda_ctx, db, qp, qo, "frechet", k, flags=flags)
        assert np.array_equal(ids, want_ids)
        assert np.array_equal(d64, want_d)
    db.close()


@pytest.mark.parametrize("pruned", [False, True])
def test_plain_small_workload_full_size(tsim, cuda_ctx, oracle, pruned):
    """The small plain workload at its own size: 8 queries x 1,024 candidates,
    every trajectory 128 points (N(0,1) random walks), all five measures with
    the full DP (no band, no LCSS window), top-10 -- ids bit-exact against
    the FP64 brute-force oracle, LCSS counts exact, distances within 1e-5."""
    from cudaruntime1_gb300 import datagen as G
    cp, co = G.random_walks(1024, 128, 11 + 3)
    qp, qo = G.random_walks(8, 128, 11 + 4)
    db = tsim.Database(cuda_ctx, cp, co)
    runs = [("dtw", dict(band_pct=-1, cost=0)), ("lcss", dict(epsilon=0.5, delta=-1)),
            ("frechet", {}), ("hausdorff", {}), ("euclidean", {})]
    for measure, kw in runs:
        okw = dict(kw)
        if "epsilon" in okw:
            okw["eps"] = okw.pop("epsilon")
        want_ids, want_d = oracle.knn(measure, qp, qo, cp, co, 10, **okw)
        if pruned:
            kw = dict(kw, flags=tsim.api.FLAG_ALWAYS_PRUNE)
        ids, d, d64, st = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 10, **kw)
        assert np.array_equal(ids, want_ids), measure
        if measure == "lcss":
            assert np.array_equal(d.astype(np.float64), want_d)
        else:
            rel = np.abs(d.astype(np.float64) - want_d) / np.maximum(want_d, 1e-30)
            assert rel.max() <= REL_TOL, (measure, rel.max())
        assert st["pairs"] == 8 * 1024
    db.close()


@pytest.mark.parametrize("measure,kw", [("dtw", dict(band_pct=10, cost=0)),
                                        ("dtw", dict(band_pct=-1, cost=1)),
                                        ("lcss", dict(epsilon=0.5, delta=8)),
                                        ("frechet", {})])
def test_dp_kernel_choices_agree(tsim, cuda_ctx, oracle, measure, kw):
    """Rounds of many pairs run a lane per pair (dp_lane.cu), DTW and Frechet
    rounds start on the band-relative kernel (dp_wave.cu); with
    TSIM_FLAG_NO_LANE_DP / TSIM_FLAG_NO_WAVE_DP they run on the row-group
    kernels instead.  Every choice gives the same ids and distance bits,
    brute force (36,000 pairs, past the lane kernel's gate) and pruned, and
    the ids equal the FP64 oracle's."""
    cp, co = _db(3000, 16, 300, 91)
    ql = G.uniform_lengths(12, 16, 300, 92)
    qp, qo = G.random_walks(12, ql, 93)
    db = tsim.Database(cuda_ctx, cp, co)
    okw = {("eps" if k == "epsilon" else k): v for k, v in kw.items()}
    want_ids, _ = oracle.knn(measure, qp, qo, cp, co, 10, **okw)
    off = tsim.api.FLAG_NO_LANE_DP | tsim.api.FLAG_NO_WAVE_DP
    for extra in (0, tsim.api.FLAG_ALWAYS_PRUNE):
        base = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 10, flags=extra | off, **kw)
        assert np.array_equal(base[0], want_ids), (measure, extra)
        for choice in (0, tsim.api.FLAG_NO_LANE_DP, tsim.api.FLAG_NO_WAVE_DP):
            got = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 10, flags=extra | choice, **kw)
            assert np.array_equal(got[0], base[0]), (measure, extra, choice)
            assert np.array_equal(got[1].view(np.uint32), base[1].view(np.uint32)), \
                (measure, extra, choice)
            if measure != "lcss":  # the FP64 re-scored distances
                assert np.array_equal(got[2].view(np.uint64), base[2].view(np.uint64)), \
                    (measure, extra, choice)
    db.close()


@pytest.mark.parametrize("offset", [0.0, 3e5])
@pytest.mark.parametrize("nc,k", [(300, 40), (5000, 3), (9000, 10)])
def test_euclidean_segment_means(tsim, cuda_ctx, oracle, nc, k, offset):
    """The segment-mean bound: ragged candidates down to one point (empty
    segments), queries of the same, a longer and a too short length, several
    seed candidates a chunk and one, coordinates far from the origin (whose
    sums round coarsely): the oracle's ids, and the distances of a request
    that refines every pair."""
    lens = np.random.default_rng(nc).integers(1, 70, nc)
    lens[::5] = 64
    cp, co = G.random_walks(nc, lens, 31, step="student_t", start_range=20.0)
    qp, qo = G.random_walks(9, [64, 1, 3, 8, 63, 65, 200, 64, 9], 32, step="student_t",
                            start_range=20.0)
    cp, qp = (cp + np.float32(offset)).astype(np.float32), (qp + np.float32(offset)).astype(np.float32)
    db = tsim.Database(cuda_ctx, cp, co)
    want_ids, want_d = oracle.knn("euclidean", qp, qo, cp, co, k)
    ids, d, d64, _ = _device_knn(tsim, cuda_ctx, db, qp, qo, "euclidean", k,
                                 flags=tsim.api.FLAG_ALWAYS_PRUNE)
    ids2, d2, d642, _ = _device_knn(tsim, cuda_ctx, db, qp, qo, "euclidean", k,
                                    flags=tsim.api.FLAG_NO_PRUNE)
    assert np.array_equal(ids, want_ids)
    assert np.array_equal(ids, ids2) and np.array_equal(d, d2) and np.array_equal(d64, d642)
    db.close()


@pytest.mark.parametrize("pruned", [False, True])
def test_hausdorff_point_counts(tsim, cuda_ctx, oracle, pruned):
    """Sides around the kernel's points per lane, its sample's smallest side
    and the targets staged at a time: the oracle's ids and distances."""
    sizes = [1, 2, 31, 32, 33, 63, 64, 65, 127, 130, 255, 257, 300, 511, 512, 513, 515, 1030]
    cp, co = G.random_walks(3 * len(sizes), sizes * 3, 51, start_range=30.0)
    qp, qo = G.random_walks(6, [1, 33, 64, 161, 513, 1100], 52, start_range=30.0)
    db = tsim.Database(cuda_ctx, cp, co)
    flags = tsim.api.FLAG_ALWAYS_PRUNE if pruned else tsim.api.FLAG_NO_PRUNE
    ids, d, _ = tsim.knn(cuda_ctx, db, qp, qo, "hausdorff", 7, flags=flags)
    want_ids, want = oracle.knn("hausdorff", qp, qo, cp, co, 7)
    assert np.array_equal(ids, want_ids)
    # one rounded squared distance (8 2^-24), its root and the result's rounding
    assert np.all(np.abs(d - want) <= 8 * 2.0 ** -24 * want)
    db.close()


@pytest.mark.parametrize("band,cost", [(0, 0), (1, 0), (10, 0), (10, 1), (45, 0), (100, 0)])
def test_dtw_row_bounds(tsim, cuda_ctx, oracle, band, cost):
    """The row side of LB_Keogh: queries shorter, longer and far longer than
    the candidates, two-point sides, bands from the diagonal to the whole
    matrix (windows of one block to more than 15): the oracle's ids, and the
    distances of a request that refines every pair."""
    lens = np.random.default_rng(7).integers(2, 90, 500)
    lens[::9] = 300
    lens[5::50] = 700
    cp, co = G.random_walks(500, lens, 61, start_range=15.0)
    qp, qo = G.random_walks(6, [2, 3, 40, 300, 301, 900], 62, start_range=15.0)
    db = tsim.Database(cuda_ctx, cp, co)
    kw = dict(band_pct=band, cost=cost)
    ids, d, _ = tsim.knn(cuda_ctx, db, qp, qo, "dtw", 5, flags=tsim.api.FLAG_ALWAYS_PRUNE, **kw)
    ids2, d2, _ = tsim.knn(cuda_ctx, db, qp, qo, "dtw", 5, flags=tsim.api.FLAG_NO_PRUNE, **kw)
    want_ids, _ = oracle.knn("dtw", qp, qo, cp, co, 5, **kw)
    assert np.array_equal(ids, want_ids)
    assert np.array_equal(ids, ids2) and np.array_equal(d, d2)
    db.close()


@pytest.mark.parametrize("least", [1, 2])
@pytest.mark.parametrize("measure,kw,longest", [
    ("dtw", dict(band_pct=31), (100, 100)), ("dtw", dict(band_pct=32), (100, 100)),
    ("dtw", dict(band_pct=63), (100, 90)), ("dtw", dict(band_pct=64), (90, 100)),
    ("dtw", dict(band_pct=100), (33, 400)), ("dtw", dict(band_pct=100), (400, 65)),
    ("frechet", dict(band_pct=45), (300, 70)), ("dtw", dict(), (64, 2050)),
    ("frechet", dict(), (2050, 40)), ("lcss", dict(delta=40), (90, 120))])
def test_known_lengths(tsim, cuda_ctx, oracle, least, measure, kw, longest):
    """A request whose lengths are known launches no kernel for pairs that
    cannot be left over: the same results as with a longest query length
    alone, trajectories of one point among them or not."""
    rng = np.random.default_rng(9)
    cl, ql = rng.integers(least, longest[1] + 1, 300), rng.integers(least, longest[0] + 1, 8)
    cl[:6] = ql[:2] = least
    cl[6:9], ql[2] = longest[1], longest[0]
    cp, co = G.random_walks(300, cl, 71, start_range=10.0)
    qp, qo = G.random_walks(8, ql, 72, start_range=10.0)
    db = tsim.Database(cuda_ctx, cp, co)
    want_ids, _ = oracle.knn(measure, qp, qo, cp, co, 5, **kw)
    for flags in (tsim.api.FLAG_ALWAYS_PRUNE, tsim.api.FLAG_NO_PRUNE):
        ids, d, _ = tsim.knn(cuda_ctx, db, qp, qo, measure, 5, flags=flags, **kw)
        ids2, d2, _, _ = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 5, flags=flags, **kw)
        assert np.array_equal(ids, want_ids)
        assert np.array_equal(ids, ids2) and np.array_equal(d, d2)
    db.close()


@pytest.mark.parametrize("band,cost", [(0, 0), (4, 0), (12, 1), (40, 0), (60, 1)])
def test_dtw_from_both_ends(tsim, cuda_ctx, oracle, band, cost):
    """Banded DTW's latency rounds, each pair from both ends to the middle:
    sums of lengths odd and even, halves around blocks of 16 anti-diagonals,
    anti-diagonals of up to 32 cells, up to 64 and more, two-point sides."""
    cp, co = G.random_walks(20, [2, 3, 4, 14, 15, 16, 17, 18, 30, 31, 32, 33, 34, 35, 63, 64, 65, 66,
                                 120, 200], 81, start_range=10.0)
    qp, qo = G.random_walks(10, [2, 3, 16, 17, 18, 33, 34, 65, 66, 170], 82, start_range=10.0)
    db = tsim.Database(cuda_ctx, cp, co)
    kw = dict(band_pct=band, cost=cost)
    want_ids, want = oracle.knn("dtw", qp, qo, cp, co, 20, **kw)
    fin = np.isfinite(want)
    for flags in (0, tsim.api.FLAG_ALWAYS_PRUNE):
        ids, d, _ = tsim.knn(cuda_ctx, db, qp, qo, "dtw", 20, flags=flags, **kw)
        assert np.array_equal(ids, want_ids)
        assert np.array_equal(np.isfinite(d), fin)
        # costs within 4 2^-24, their compensated sum, the result's rounding
        assert np.all(np.abs(d[fin] - want[fin]) <= 5 * 2.0 ** -24 * want[fin])
    db.close()


@pytest.mark.parametrize("kw", [dict(band_pct=10), dict(band_pct=10, cost=1), dict(band_pct=-1)])
def test_dtw_on_a_database_beyond_l2(tsim, cuda_ctx, kw):
    """Round 1 ahead of LB_Keogh, whose points come from HBM (108 MB of them):
    the answer of a request that refines every pair, bit for bit."""
    lens = np.random.default_rng(3).integers(400, 500, 30000)
    lens[:200] = np.arange(2, 202)
    cp, co = G.random_walks(30000, lens, 91, start_range=20.0)
    qp, qo = G.random_walks(3, [2, 100, 700], 92, start_range=20.0)
    db = tsim.Database(cuda_ctx, cp, co)
    ids, d, _ = tsim.knn(cuda_ctx, db, qp, qo, "dtw", 10, flags=tsim.api.FLAG_ALWAYS_PRUNE, **kw)
    ids2, d2, _ = tsim.knn(cuda_ctx, db, qp, qo, "dtw", 10, flags=tsim.api.FLAG_NO_PRUNE, **kw)
    assert np.array_equal(ids, ids2) and np.array_equal(d, d2)
    db.close()


@pytest.mark.parametrize("band", [10, -1])
@pytest.mark.parametrize("cost", [0, 1])
def test_distances_alone_and_in_a_batch(tsim, cuda_ctx, cost, band):
    """DTW's distances do not depend on how many queries share the
    call, nor on the kernels chosen: the bits of each query alone, of a few
    together, and of all of them with the row-group kernels."""
    rng = np.random.default_rng(97)
    cp, co = _db(3000, 16, 300, 97)
    qp, qo = G.random_walks(24, G.uniform_lengths(24, 16, 300, 98), 99)
    for c in range(480):  # near copies, whose costs span more bits than a pair of floats holds
        src = np.linspace(qo[c % 24], qo[c % 24 + 1] - 1, co[c + 1] - co[c]).round().astype(int)
        scale = 2.0 ** rng.uniform(-16, 3, (len(src), 1))
        cp[co[c]:co[c + 1]] = qp[src] + scale * rng.standard_normal((len(src), 2))
    db = tsim.Database(cuda_ctx, cp, co)
    kw = dict(band_pct=band, cost=cost)
    for flags in (0, tsim.api.FLAG_ALWAYS_PRUNE):
        want = _device_knn(tsim, cuda_ctx, db, qp, qo, "dtw", 10, flags=flags, **kw)
        off = _device_knn(tsim, cuda_ctx, db, qp, qo, "dtw", 10,
                          flags=flags | tsim.api.FLAG_NO_WAVE_DP, **kw)
        assert np.array_equal(off[0], want[0])
        assert np.array_equal(off[2].view(np.uint64), want[2].view(np.uint64))
        for q0, q1 in [(q, q + 1) for q in range(0, 24, 3)] + [(1, 4), (5, 9)]:
            got = _device_knn(tsim, cuda_ctx, db, qp[qo[q0]:qo[q1]], qo[q0:q1 + 1] - qo[q0], "dtw",
                              10, flags=flags, **kw)
            assert np.array_equal(got[0], want[0][q0:q1])
            assert np.array_equal(got[1].view(np.uint32), want[1][q0:q1].view(np.uint32))
            assert np.array_equal(got[2].view(np.uint64), want[2][q0:q1].view(np.uint64))
    db.close()


@pytest.mark.parametrize("count,length", [(6010 * 256, 2), (33000, 381), (33000, 382), (33000, 383)])
def test_shared_memory_around_48_kib(tsim, cuda_ctx, count, length):
    """Databases whose seed keys, or whose longest candidate's copies, take
    about 48 KiB of a block's shared memory: the answer of a request that
    refines every pair."""
    cp, co = G.random_walks(count, length, 17)
    qp, qo = G.random_walks(2, 30, 18)
    db = tsim.Database(cuda_ctx, cp, co)
    ids, d, _ = tsim.knn(cuda_ctx, db, qp, qo, "dtw", 10, band_pct=20)
    ids2, d2, _ = tsim.knn(cuda_ctx, db, qp, qo, "dtw", 10, band_pct=20,
                           flags=tsim.api.FLAG_NO_PRUNE)
    assert np.array_equal(ids, ids2) and np.array_equal(d, d2)
    db.close()


@pytest.mark.parametrize("delta", [-1, 6])
@pytest.mark.parametrize("eps", [1e-45, 0.5, 3e38])
def test_lcss_without_a_finite_extent(tsim, cuda_ctx, oracle, eps, delta):
    """LCSS queries with NaNs or infinities among their points, alone on an
    axis, or everywhere, and the smallest and largest epsilon: the oracle's
    counts."""
    cp, co = G.random_walks(400, G.uniform_lengths(400, 3, 60, 5), 6, start_range=4.0)
    cp[co[7]:co[8]], cp[co[9]:co[10], 0] = np.nan, np.inf
    ql = [40] * 9
    qp, qo = G.random_walks(9, ql, 7, start_range=4.0)
    bad = [(0, np.nan), (0, np.inf), (1, -np.inf), (slice(None), np.nan), (slice(None), np.inf)]
    for q, (axis, v) in enumerate(bad):
        qp[qo[q]:qo[q + 1], axis] = v
    qp[qo[5] + 3, 0], qp[qo[6] + 5, 1], qp[qo[7], 0], qp[qo[7] + 1, 0] = np.inf, np.nan, -np.inf, np.inf
    cp[co[20]:co[21]] = qp[qo[8]:qo[9]][:co[21] - co[20]][:1]  # equal points: they match at any epsilon
    db = tsim.Database(cuda_ctx, cp, co)
    want_ids, want = oracle.knn("lcss", qp, qo, cp, co, 10, eps=eps, delta=delta)
    for flags in (0, tsim.api.FLAG_ALWAYS_PRUNE, tsim.api.FLAG_NO_PRUNE):
        ids, d, _ = tsim.knn(cuda_ctx, db, qp, qo, "lcss", 10, epsilon=eps, delta=delta, flags=flags)
        assert np.array_equal(d, want), flags
        assert np.array_equal(ids, want_ids), flags
    db.close()


@pytest.mark.parametrize("measure,kw", [("dtw", dict(band_pct=10)), ("dtw", dict(cost=1)),
                                        ("frechet", {}), ("hausdorff", {}), ("euclidean", {})])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_candidates_without_a_finite_distance(tsim, cuda_ctx, oracle, measure, kw, bad):
    """Fewer candidates at a finite distance than neighbours asked for, the
    others with a point at infinity or a NaN, and queries of which one has no
    finite distance at all: the oracle's answer among the finite ones, then
    the others at infinity, the lowest indices first."""
    if measure == "frechet" and np.isnan(bad):
        pytest.skip("a maximum passes over a NaN cost: such a pair's distance is finite")
    cp, co = G.random_walks(300, 40, 15, start_range=10.0)
    qp, qo = G.random_walks(9, 40, 16, start_range=10.0)
    good = np.array([5, 100, 101, 200, 255, 299])
    rng = np.random.default_rng(17)
    for c in np.setdiff1d(np.arange(300), good):
        cp[co[c] + rng.choice([0, 20, 39]), 1] = bad
    qp[qo[8] + 20, 0] = bad
    gp = np.concatenate([cp[co[c]:co[c + 1]] for c in good])
    want_ids, want = oracle.knn(measure, qp[:qo[8]], qo[:9], gp, np.arange(7) * 40, 6, **kw)
    db = tsim.Database(cuda_ctx, cp, co)
    for flags in (0, tsim.api.FLAG_ALWAYS_PRUNE, tsim.api.FLAG_FP64_RESCORE):
        ids, d, _ = tsim.knn(cuda_ctx, db, qp, qo, measure, 10, flags=flags, **kw)
        assert np.array_equal(ids[:8, :6], good[want_ids]), flags
        assert np.all(np.abs(d[:8, :6] - want) <= 1e-5 * want), flags
        assert np.all(np.isposinf(d[:8, 6:])) and np.all(np.isposinf(d[8])), flags
        assert np.all(ids[:8, 6:] == np.setdiff1d(np.arange(300), good)[:4]), flags
        assert np.array_equal(ids[8], np.arange(10)), flags
    db.close()


@pytest.mark.parametrize("cost", [0, 1])
def test_dtw_row_bounds_of_corners_that_are_no_number(tsim, cuda_ctx, cost):
    """Banded DTW where most corner cells are NaN and no threshold exists: the
    row side of LB_Keogh keeps what the column side keeps, the candidates of a
    request that refines every pair."""
    cp, co = G.random_walks(300, 40, 19, start_range=10.0)
    qp, qo = G.random_walks(3, 40, 20, start_range=10.0)
    cp[co[:-1][np.arange(300) % 60 != 7]] = np.nan
    db = tsim.Database(cuda_ctx, cp, co)
    ids, d, _ = tsim.knn(cuda_ctx, db, qp, qo, "dtw", 10, band_pct=10, cost=cost,
                         flags=tsim.api.FLAG_ALWAYS_PRUNE)
    ids2, d2, _ = tsim.knn(cuda_ctx, db, qp, qo, "dtw", 10, band_pct=10, cost=cost,
                           flags=tsim.api.FLAG_NO_PRUNE)
    assert np.array_equal(ids, ids2) and np.array_equal(d, d2)
    db.close()


@pytest.mark.parametrize("nq", [1, 4, 5, 40])
@pytest.mark.parametrize("delta", [-1, 3, 20, 31])
def test_lcss_dense_and_sparse_queries(tsim, oracle, nq, delta):
    """LCSS of one query, a few and many, alternately matching nearly every
    point and few: lists shorter and longer than a block's tile, and enough
    densely matching pairs for a lane each (74,000 of 40 queries, one stream),
    one-point sides among them: the oracle's counts, with and without the lanes."""
    ctx = tsim.Context(0)
    ctx.set_concurrency(1)
    cl = G.uniform_lengths(6000, 20, 60, 21)
    cl[:40] = 1
    cp, co = G.random_walks(6000, cl, 22, start_range=10.0)
    ql = np.resize([60, 50, 30, 55, 1, 45], nq)
    qp, qo = G.random_walks(nq, ql, 23, start_range=10.0)
    for q in range(1, nq, 2):  # every other query far away but for its ends
        qp[qo[q] + 3:max(qo[q] + 3, qo[q + 1] - 3)] += 1e4
    db = tsim.Database(ctx, cp, co)
    for eps in (0.5, 20.0):
        want_ids, want = oracle.knn("lcss", qp, qo, cp, co, 5, eps=eps, delta=delta)
        for flags in (0, tsim.api.FLAG_ALWAYS_PRUNE,
                      tsim.api.FLAG_ALWAYS_PRUNE | tsim.api.FLAG_NO_LANE_DP):
            ids, d, _ = tsim.knn(ctx, db, qp, qo, "lcss", 5, epsilon=eps, delta=delta,
                                 flags=flags)
            assert np.array_equal(d, want), (eps, flags)
            assert np.array_equal(ids, want_ids), (eps, flags)
    db.close()
    ctx.close()


@pytest.mark.parametrize("nq", [5, 20, 43])
@pytest.mark.parametrize("measure,kw", [("dtw", dict(band_pct=20)), ("lcss", dict(epsilon=0.5, delta=3)),
                                        ("frechet", {}), ("hausdorff", {}), ("euclidean", {})])
def test_first_bound_queries_a_block(tsim, measure, kw, nq):
    """Requests whose first bound takes one query a block, a few and eight, the
    last block with fewer: the answer of a request that refines every pair."""
    ctx = tsim.Context(0)
    ctx.set_concurrency(1)
    cp, co = G.random_walks(33000, G.uniform_lengths(33000, 8, 24, 31), 32, start_range=60.0)
    qp, qo = G.random_walks(nq, 24, 33, start_range=60.0)
    db = tsim.Database(ctx, cp, co)
    ids, d, _ = tsim.knn(ctx, db, qp, qo, measure, 10, **kw)
    ids2, d2, _ = tsim.knn(ctx, db, qp, qo, measure, 10, flags=tsim.api.FLAG_NO_PRUNE, **kw)
    assert np.array_equal(ids, ids2) and np.array_equal(d, d2)
    db.close()
    ctx.close()


@pytest.mark.parametrize("measure,kw", [("lcss", dict(epsilon=0.5, delta=40)),
                                        ("lcss", dict(epsilon=0.5, delta=-1)),
                                        ("lcss", dict(epsilon=2.0, delta=12)),
                                        ("dtw", dict(band_pct=-1, cost=0))])
def test_dp_kernel_choices_agree_past_strips_and_bit_vectors(tsim, cuda_ctx, oracle, measure, kw):
    """LCSS without bit vectors (a lane or a warp a pair), with them, and DTW's
    full rows: what the kernel choices still differ in where strips and bit
    vectors come first."""
    cp, co = _db(3000, 8, 150, 94)
    qp, qo = G.random_walks(14, G.uniform_lengths(14, 8, 150, 95), 96)
    db = tsim.Database(cuda_ctx, cp, co)
    okw = {("eps" if k == "epsilon" else k): v for k, v in kw.items()}
    want_ids, _ = oracle.knn(measure, qp, qo, cp, co, 10, **okw)
    for extra in (0, tsim.api.FLAG_ALWAYS_PRUNE, tsim.api.FLAG_NO_PRUNE):
        base = None
        for choice in (0, tsim.api.FLAG_NO_LANE_DP, tsim.api.FLAG_NO_WAVE_DP,
                       tsim.api.FLAG_NO_LANE_DP | tsim.api.FLAG_NO_WAVE_DP):
            got = _device_knn(tsim, cuda_ctx, db, qp, qo, measure, 10, flags=extra | choice, **kw)
            assert np.array_equal(got[0], want_ids), (extra, choice)
            base = base or got
            assert np.array_equal(got[1].view(np.uint32), base[1].view(np.uint32)), (extra, choice)
    db.close()
