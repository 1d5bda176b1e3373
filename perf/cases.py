"""The work that users of this engine have it do, through its public entry
points: exact kNN of all five measures over resident databases, the serving
loop, values of explicit pairs, and the reference-named batch calls.

Trajectories are seeded random walks (start uniform in [0,100)^2, N(0,1) or
Student-t(3) steps), the data of the engine's own workloads; the
reference-named calls take the reference generator's shapes (candidates are
noisy resampled copies of the queries).  Walks are summed in 2^-30 fixed
point, so that the same seed gives the same bits whatever order a sum runs in.

A case's ``op`` is the entry point:

  knn    ``knn_device``: device pointers in and out, asynchronous; or ``knn``:
         host arrays end to end (``host``)
  serve  ``Server.submit`` / ``wait`` of single-query requests, all at once
  pairs  ``dp_pairs``: values of every (query, candidate) pair, kernel chosen
         by the library
  ref    the reference's batch calls: host arrays, one value per query
"""
import math

import numpy as np
import torch

import cudaruntime1_gb300 as T
from cudaruntime1_gb300 import api
from cudaruntime1_gb300 import datagen as G

POINT = 8  # bytes of a point
FLOPS = {"dtw": 8, "lcss": 6, "frechet": 7, "hausdorff": 6, "euclidean": 6}  # per cell or point pair
BOUND_FLOPS = 10  # one O(1) lower bound of a pair
SERVED = ("dtw", "lcss", "frechet", "hausdorff", "euclidean")
SERVED_PARAMS = {"dtw": dict(band_pct=10, cost=api.COST_SQEUCLID),
                 "lcss": dict(epsilon=0.25, delta=20), "frechet": {}, "hausdorff": {},
                 "euclidean": {}}
SERVED_MOST = {"frechet": 256}  # the longest query a measure is asked with


# --------------------------------------------------------------------- cases
def listed():
    return [
        # an application asking for the neighbours of a handful of fixes: the
        # smallest calls, host arrays in and out, launches and latency count
        knn("small_dtw", "dtw", 8, 1024, 128, 128, host=True, band_pct=-1),
        knn("small_hausdorff", "hausdorff", 8, 1024, 128, 128, host=True),
        # one interactive query of an odd length against a mid-sized database
        knn("one_query_dtw", "dtw", 1, 16384, 64, 512, qlo=333, qhi=333, host=True, band_pct=10),
        # the batched workload: uneven lengths, 10 % band, device-resident
        knn("batched_dtw", "dtw", 64, 16384, 64, 512, band_pct=10),
        # counts under an index window; lengths lognormal, as recorded tracks are
        knn("batched_lcss", "lcss", 256, 65536, 32, 1024, lens="lognormal", epsilon=0.25, delta=20),
        # discrete Frechet of tracks of up to 256 fixes, with the FP64 re-score of every top-10
        knn("batched_frechet", "frechet", 256, 65536, 32, 1024, lens="lognormal", qlo=32, qhi=256,
            fp64=True),
        # bulk joins over a large database with heavy-tailed steps
        knn("large_hausdorff", "hausdorff", 1024, 262144, 32, 256, step="student_t"),
        # ... lock-step, one candidate in a hundred long enough for FP64 sums
        knn("large_euclidean", "euclidean", 1024, 262144, 256, 256, step="student_t", qlo=2048,
            qhi=2048, long_len=2048),
        # the serving loop with its queue full: mixed measures, ragged queries
        dict(name="serve_mixed", op="serve", nc=1000000, lo=50, hi=500, nreq=60, qlo=16, qhi=2048,
             k=10, slots=32),
        # a program written for the reference: its DTW and Hausdorff batch calls
        dict(name="ref_dtw", op="ref", measure="dtw", nt=1024, n=128, m=128),
        dict(name="ref_hausdorff", op="ref", measure="hausdorff", nt=1024, n=128, m=128),
        # the DP alone at saturation: a distance matrix of queries x candidates
        dict(name="pairs_dtw", op="pairs", measure="dtw", nq=64, nc=2048, lo=64, hi=512,
             precision=0, band_pct=10, cost=0),
    ]


def knn(name, measure, nq, nc, lo, hi, *, lens="uniform", step="normal", qlo=0, qhi=0, k=10,
        host=False, band_pct=-1, cost=0, epsilon=0.5, delta=-1, fp64=False, long_len=0):
    """A kNN case; candidates of lo .. hi points, queries of qlo .. qhi (0: the
    candidates' lengths); long_len: 1 % of the candidates have that many."""
    c = dict(name=name, op="knn", measure=measure, nq=nq, nc=nc, lo=lo, hi=hi, lens=lens,
             step=step, qlo=qlo, qhi=qhi, k=k, host=host, fp64=fp64, long_len=long_len)
    if measure == "dtw":
        c.update(band_pct=band_pct, cost=cost)
    if measure == "lcss":
        c.update(epsilon=epsilon, delta=delta)
    return c


def draw(rng):
    top = max(_weight(c) for c in listed())
    while True:
        c = _draw(rng)
        c.pop("name", None)
        if _weight(c) <= top:
            return c


def _weight(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw(rng):
    kind = rng.choice(["small", "one", "dtw", "lcss", "frechet", "hausdorff", "euclidean", "serve",
                       "ref", "pairs"])
    k = rng.choice([1, 5, 10, 10, 10, 32])
    if kind == "small":
        lo = _logint(rng, 16, 128)
        return knn("", rng.choice(SERVED), rng.randint(1, 16), _logint(rng, 64, 2048), lo,
                   rng.choice([lo, rng.randint(lo, 160)]), k=k, host=True,
                   band_pct=rng.choice([-1, 10]), delta=rng.choice([-1, 10]))
    if kind == "one":
        measure = rng.choice(["dtw", "frechet", "hausdorff"])
        q = _logint(rng, 32, 256 if measure == "frechet" else 900)
        return knn("", measure, rng.randint(1, 3),
                   _logint(rng, 4096, 65536), rng.randint(16, 100), rng.randint(200, 512), qlo=q,
                   qhi=q, k=k, host=True, band_pct=10)
    if kind == "dtw":
        return knn("", "dtw", _logint(rng, 8, 96), _logint(rng, 4096, 32768), rng.randint(16, 90),
                   rng.randint(200, 600), k=k, band_pct=rng.randint(5, 20), cost=rng.choice([0, 0, 1]))
    if kind == "lcss":
        return knn("", "lcss", _logint(rng, 16, 256), _logint(rng, 8192, 65536), 32, 1024,
                   lens="lognormal", k=k, epsilon=rng.choice([0.25, 0.5]), delta=rng.randint(10, 30))
    if kind == "frechet":
        return knn("", "frechet", _logint(rng, 16, 256), _logint(rng, 8192, 65536), 32, 1024,
                   lens="lognormal", qlo=32, qhi=256, k=k, fp64=rng.choice([True, False]))
    if kind == "hausdorff":
        return knn("", "hausdorff", _logint(rng, 64, 1024), _logint(rng, 16384, 262144),
                   rng.randint(16, 48), rng.randint(128, 256), step="student_t", k=k)
    if kind == "euclidean":
        n = _logint(rng, 64, 256)
        q = rng.choice([n, 2048])
        return knn("", "euclidean", _logint(rng, 64, 1024), _logint(rng, 16384, 262144), n, n,
                   step="student_t", qlo=q, qhi=q, k=k, long_len=2048 if q == 2048 else 0)
    if kind == "serve":
        return dict(op="serve", nc=_logint(rng, 100000, 800000), lo=rng.randint(30, 60),
                    hi=rng.randint(300, 500), nreq=rng.randint(15, 60), qlo=16,
                    qhi=rng.choice([512, 1024, 2048]), k=10, slots=rng.choice([16, 32]))
    if kind == "ref":
        return dict(op="ref", measure=rng.choice(SERVED), nt=_logint(rng, 64, 1500),
                    n=rng.randint(32, 160), m=rng.randint(32, 160))
    measure = rng.choice(["dtw", "dtw", "lcss", "frechet"])
    return dict(op="pairs", measure=measure, nq=_logint(rng, 8, 64), nc=_logint(rng, 256, 2048),
                lo=rng.randint(16, 96), hi=rng.randint(200, 512),
                precision=0 if measure == "lcss" else rng.choice([0, 0, 1]),
                **{"dtw": dict(band_pct=rng.randint(5, 20), cost=0), "frechet": {},
                   "lcss": dict(epsilon=0.5, delta=rng.randint(10, 30))}[measure])


# -------------------------------------------------------------------- inputs
def _lengths(gen, count, lo, hi, lens):
    if lens == "lognormal":
        x = torch.randn(count, generator=gen, device="cuda", dtype=torch.float64)
        return torch.exp(math.log(200.0) + 0.6 * x).round().clamp(lo, hi).to(torch.int64)
    return torch.randint(lo, hi + 1, (count,), generator=gen, device="cuda")


def _walks(gen, lens, step="normal"):
    """Random walks of the given lengths: points float32 [total, 2], offsets int64."""
    off = torch.zeros(len(lens) + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=off[1:])
    total = int(off[-1])
    pts = torch.empty(total, 2, device="cuda")
    for xy in range(2):  # one coordinate at a time: a scan along a contiguous row
        s = torch.randn(total, generator=gen, device="cuda")
        if step == "student_t":
            chi2 = torch.zeros_like(s)
            for _ in range(3):
                chi2 += torch.randn(total, generator=gen, device="cuda").square_()
            s *= chi2.div_(3).rsqrt_()
        q = (s.double() * 2.0 ** 30).round_().to(torch.int64)
        start = torch.randint(0, 100 << 30, (len(lens),), generator=gen, device="cuda")
        q[off[:-1]] = 0
        q = torch.cumsum(q, 0)
        q += torch.repeat_interleave(start - q[off[:-1]], lens, output_size=total)
        pts[:, xy] = q.double() * 2.0 ** -30
    return pts, off


def _inputs(case, seed):
    """(query points, query offsets, candidate points, candidate offsets) on the GPU."""
    gen = torch.Generator("cuda").manual_seed(seed)
    lens, step = case.get("lens", "uniform"), case.get("step", "normal")
    lo, hi = case["lo"], case["hi"]
    cl = _lengths(gen, case["nc"], lo, hi, lens)
    if case.get("long_len"):
        cl[torch.rand(case["nc"], generator=gen, device="cuda") < 0.01] = case["long_len"]
    nq = case.get("nq") or case["nreq"]
    ql = _lengths(gen, nq, case.get("qlo") or lo, case.get("qhi") or hi, lens)
    return _walks(gen, ql, step) + _walks(gen, cl, step)


def _ref_inputs(case, seed):
    t1 = G.ref_base_trajectories(case["nt"], case["n"], seed)
    return t1, G.ref_similar_trajectories(t1, case["nt"], case["n"], case["m"] if
                                          case["measure"] != "euclidean" else case["n"], 2.0, seed + 1)


def _params(case):
    return {k: case[k] for k in ("band_pct", "cost", "epsilon", "delta") if k in case}


def prepare(case, seed):
    T.build()
    if case["op"] == "ref":
        t1, t2 = _ref_inputs(case, seed)
        return dict(case=case, t1=t1, t2=t2)
    qp, qo, cp, co = _inputs(case, seed)
    torch.cuda.synchronize()
    ctx = T.Context(0)
    s = dict(case=case, ctx=ctx, kw=_params(case), cp=cp, co=co,
             maxq=int((qo[1:] - qo[:-1]).max()), maxc=int((co[1:] - co[:-1]).max()))
    if case["op"] == "pairs":
        nq, nc = case["nq"], case["nc"]
        pair = torch.stack(torch.meshgrid(torch.arange(nq), torch.arange(nc), indexing="ij"), -1)
        s.update(qp=qp, qo=qo, pairs=pair.reshape(-1, 2).to(torch.int32).cuda(),
                 out=torch.empty(nq * nc, dtype=(torch.float32, torch.float64)[case["precision"]],
                                 device="cuda"))
        torch.cuda.synchronize()
        return s
    s["db"] = T.Database(ctx, device_pts=cp.data_ptr(), device_off=co.data_ptr(), count=case["nc"],
                         max_len=s["maxc"])
    if case["op"] == "serve":
        hp, ho = qp.cpu().numpy(), qo.cpu().numpy()
        s["requests"] = []
        for i in range(case["nreq"]):
            m = SERVED[i % 5]
            n = min(int(ho[i + 1] - ho[i]), SERVED_MOST.get(m, case["qhi"]))
            s["requests"].append((m, hp[ho[i]:ho[i] + n].copy(), np.array([0, n], np.int64)))
        s["server"] = T.Server(ctx, s["db"], slots=case["slots"], hbm_budget_bytes=8 << 30)
        return s
    if case["host"]:
        s.update(qp=qp.cpu().numpy(), qo=qo.cpu().numpy())
        return s
    if case["fp64"]:
        s["kw"]["flags"] = api.FLAG_FP64_RESCORE
    shape = (case["nq"], case["k"])
    s.update(qp=qp, qo=qo, ids=torch.empty(shape, dtype=torch.int32, device="cuda"),
             dists=torch.empty(shape, device="cuda"),
             dists64=torch.empty(shape, dtype=torch.float64, device="cuda") if case["fp64"] else None)
    torch.cuda.synchronize()
    return s


# ----------------------------------------------------------------------- run
def run(s):
    case = s["case"]
    if case["op"] == "ref":
        return {"values": _run_ref(case, s["t1"], s["t2"])}
    if case["op"] == "pairs":
        f64 = case["precision"] > 0
        api.dp_pairs(s["ctx"], case["measure"], case["precision"], 0, s["qp"].data_ptr(),
                     s["qo"].data_ptr(), s["maxq"], s["cp"].data_ptr(), s["co"].data_ptr(),
                     s["maxc"], s["pairs"].data_ptr(), len(s["pairs"]),
                     0 if f64 else s["out"].data_ptr(), s["out"].data_ptr() if f64 else 0, **s["kw"])
        return {"values": s["out"]}
    if case["op"] == "serve":
        srv = s["server"]
        tickets = [srv.submit(p, o, m, case["k"], **SERVED_PARAMS[m]) for m, p, o in s["requests"]]
        got = [srv.wait(t) for t in tickets]
        return {"ids": np.concatenate([g[0] for g in got]), "dists": np.concatenate([g[1] for g in got])}
    if case["host"]:
        ids, dists, _ = T.knn(s["ctx"], s["db"], s["qp"], s["qo"], case["measure"], case["k"],
                              stats=False, **s["kw"])
        return {"ids": ids, "dists": dists}
    d64 = s["dists64"]
    T.knn_device(s["ctx"], s["db"], s["qp"].data_ptr(), s["qo"].data_ptr(), case["nq"], s["maxq"],
                 s["ids"].data_ptr(), s["dists"].data_ptr(), None if d64 is None else d64.data_ptr(),
                 case["measure"], case["k"], **s["kw"])
    out = {"ids": s["ids"], "dists": s["dists"]}
    return out if d64 is None else dict(out, dists64=d64)


def _run_ref(case, t1, t2):
    nt, n, m = case["nt"], case["n"], case["m"]
    if case["measure"] == "dtw":
        return api.launch_dtw_batch_gpu_knn(t1, t2, nt, n, m)[0]
    if case["measure"] == "lcss":
        return api.launch_lcss_batch_gpu_wavefront_knn(t1, t2, nt, n, m, 0.5)[0]
    if case["measure"] == "frechet":
        return api.launch_frechet_batch_gpu_wavefront(t1, t2, nt, n, m)[0]
    if case["measure"] == "hausdorff":
        return api.run_hausdorff_rtree_gpu_pipeline(t1, nt, n, t2, nt, m, 10)[0]
    return api.launch_euclidean_batch_gpu_rtree_exact(t1, t2, nt, n)[0]


# ---------------------------------------------------------------------- work
def _mean_len(case, lo, hi):
    return 235.0 if case.get("lens") == "lognormal" else (lo + hi) / 2


def _cells(case, n, m):
    """DP cells or point pairs of an n x m pair."""
    if case["measure"] == "euclidean":
        return min(n, m)
    if case["measure"] == "hausdorff":
        return 2 * n * m
    pct, delta = case.get("band_pct", -1), case.get("delta", -1)
    width = 0.02 * pct * m if pct >= 0 else (2 * delta + 1 if delta >= 0 else m)
    return n * min(m, width)


def work(case):
    """Every trajectory read once and every result written once; one O(1)
    bound per pair (no candidate can be left out without one) and the exact
    values of the neighbours returned."""
    if case["op"] == "ref":
        nt, n, m = case["nt"], case["n"], case["m"]
        c = 50 if case["measure"] == "euclidean" else 10
        bound = BOUND_FLOPS * (m if case["measure"] in ("dtw", "lcss", "frechet") else 1)
        return {"bytes": nt * (POINT * (n + m) + 4),
                "flops": nt * (nt * bound + min(c, nt) * _cells(case, n, m) * FLOPS[case["measure"]])}
    nc, lo, hi = case["nc"], case["lo"], case["hi"]
    mc = _mean_len(case, lo, hi) + (0.01 * case["long_len"] if case.get("long_len") else 0)
    mq = _mean_len(case, case.get("qlo") or lo, case.get("qhi") or hi)
    nq = case.get("nq") or case["nreq"]
    if case["op"] == "pairs":
        return {"bytes": POINT * (nq * mq + nc * mc) + nq * nc * (8 + 4 * (1 + case["precision"])),
                "flops": nq * nc * _cells(case, mq, mc) * FLOPS[case["measure"]]}
    if case["op"] == "serve":
        per = sum(_cells(dict(SERVED_PARAMS[m], measure=m), mq, mc) * FLOPS[m] for m in SERVED) / 5
    else:
        per = _cells(case, mq, mc) * FLOPS[case["measure"]]
    return {"bytes": POINT * (nq * mq + nc * mc) + nq * case["k"] * (16 if case.get("fp64") else 8),
            "flops": nq * (nc * BOUND_FLOPS + case["k"] * per)}


# --------------------------------------------------------------------- exact
INF = float("inf")
MOST_CELLS = 4e11  # past this a 64-bit evaluation takes too long


def exact(case, seed):
    """The distances in 64 bits, from the definitions (ids have no such value);
    None where that would take too long."""
    if case["op"] == "serve":
        return None
    if case["op"] == "ref":
        return {"values": _ref64(case, *_ref_inputs(case, seed))}
    qp, qo, cp, co = _inputs(case, seed)
    q, c = _padded(qp, qo), _padded(cp, co)
    if case["op"] == "pairs":
        if case["nq"] * case["nc"] * 2.0 * q[0].shape[1] * c[0].shape[1] > MOST_CELLS:
            return None
        qi = torch.arange(case["nq"], device="cuda").repeat_interleave(case["nc"])
        ci = torch.arange(case["nc"], device="cuda").repeat(case["nq"])
        return {"values": _pair_values(case, q, c, qi, ci)}
    d = _knn64(case, q, c)
    if d is None:
        return None
    out = {"ids": None, "dists": d}
    return dict(out, dists64=d) if case["fp64"] else out


def _padded(p, off):
    """Points as float64 [count, longest, 2] (rows past the end repeat the
    last point), lengths."""
    n = off[1:] - off[:-1]
    at = torch.arange(int(n.max()), device="cuda")
    at = torch.minimum(at[None], n[:, None] - 1) + off[:-1, None]
    return p.double()[at], n


def _boxes(s):
    return s[0].amin(1), s[0].amax(1)


def _bounds(case, q, c):
    """A lower bound (LCSS: none) of every pair's distance (Frechet, Hausdorff,
    Euclidean: squared)."""
    (q0, q1), (c0, c1) = _boxes(q), _boxes(c)
    if case["measure"] == "hausdorff":
        e = torch.maximum((q0[:, None] - c0[None]).abs(), (q1[:, None] - c1[None]).abs())
        return e.amax(-1).square()
    gap = torch.maximum(q0[:, None] - c1[None], c0[None] - q1[:, None]).clamp(min=0)
    gap = gap.square().sum(-1)
    first = (q[0][:, None, 0] - c[0][None, :, 0]).square().sum(-1)
    last = (q[0][:, None, -1] - c[0][None, :, -1]).square().sum(-1)
    if case["measure"] == "frechet":
        return torch.maximum(torch.maximum(first, last), gap)
    L = torch.maximum(q[1][:, None], c[1][None])
    if case["cost"]:
        first, last, gap = first.sqrt(), last.sqrt(), gap.sqrt()
    return torch.where(L > 1, first + last + (L - 2).clamp(min=0) * gap, first)


def _knn64(case, q, c):
    k, nq, nc, measure = case["k"], case["nq"], case["nc"], case["measure"]
    if measure == "euclidean":
        return _euclid64(q, c, k)
    best = []
    for a in range(0, nq, 32):
        qa = (q[0][a:a + 32], q[1][a:a + 32])
        nb = len(qa[1])
        vals = torch.full((nb, nc), INF, dtype=torch.float64, device="cuda")
        if measure == "lcss":
            take = torch.ones_like(vals, dtype=torch.bool)
        else:  # the candidates whose bound is not above the k-th of the best by bound
            lb = _bounds(case, qa, c)
            s = lb.topk(min(nc, 4 * k), largest=False).indices
            qi = torch.arange(nb, device="cuda").repeat_interleave(s.shape[1])
            v = _pair_values(case, qa, c, qi, s.reshape(-1)).reshape(s.shape)
            take = lb <= v.topk(min(k, v.shape[1]), largest=False).values[:, -1:] * (1 + 1e-9)
        qi, ci = take.nonzero(as_tuple=True)
        cells = float((qa[1][qi].double() * c[1][ci].double()).sum())
        if cells * (nq / nb) > MOST_CELLS / 4:
            return None
        v = _pair_values(case, qa, c, qi, ci)
        vals[qi, ci] = -v if measure == "lcss" else v
        best.append(vals.topk(k, largest=False, sorted=True).values)
    best = torch.cat(best)
    if measure == "lcss":
        return -best
    return best.sqrt() if measure != "dtw" else best


def _euclid64(q, c, k):
    """|q|^2 + |c|^2 - 2 q.c picks the nearest, whose distances are then summed directly."""
    n, m = q[1], c[1]
    L = c[0].shape[1]
    live = torch.arange(L, device="cuda") < m[:, None]
    cz = torch.where(live[..., None], c[0], 0.0).reshape(len(m), -1)
    qz = torch.zeros(len(n), L, 2, dtype=torch.float64, device="cuda")
    qz[:, :min(L, q[0].shape[1])] = q[0][:, :L]
    pre = qz.square().sum(-1).cumsum(1)
    d = pre[:, m - 1] + cz.square().sum(1)
    for a in range(0, len(m), 65536):
        d[:, a:a + 65536] -= 2 * (qz.reshape(len(n), -1) @ cz[a:a + 65536].T)
    d[n[:, None] < m[None]] = INF
    s = d.topk(min(len(m), k + 8), largest=False).indices
    e = torch.empty(s.shape, dtype=torch.float64, device="cuda")
    for a in range(0, len(n), 64):
        t = s[a:a + 64]
        x = (qz[a:a + 64, None] - c[0][t]).square().sum(-1)
        e[a:a + 64] = torch.where(live[t], x, 0.0).sum(-1)
    e[torch.gather(d, 1, s) == INF] = INF
    return e.sort(1).values[:, :k].sqrt()


def _pair_values(case, q, c, qi, ci):
    """Values of the pairs (Frechet, Hausdorff: squared; LCSS: counts)."""
    out = torch.empty(len(qi), dtype=torch.float64, device="cuda")
    if len(qi) == 0:
        return out
    n, m = q[1][qi], c[1][ci]
    order = torch.argsort(n + m, descending=True)
    hausdorff = case["measure"] == "hausdorff"
    at = 0
    while at < len(order):
        head = order[at]
        per = int(n[head] + m[head]) ** 2 // 2 if hausdorff else int(n[head] + m[head])
        o = order[at:at + max(1, int(6e7) // per)]
        A, B = q[0][qi[o]][:, :int(n[o].max())], c[0][ci[o]][:, :int(m[o].max())]
        if hausdorff:  # repeats of a last point change no minimum and no maximum
            d = (A[:, :, None, 0] - B[:, None, :, 0]).square()
            d += (A[:, :, None, 1] - B[:, None, :, 1]).square()
            out[o] = torch.maximum(d.amin(2).amax(1), d.amin(1).amax(1))
        else:
            out[o] = _dp64(case, A, B, n[o], m[o])
        at += len(o)
    return out


def _dp64(case, A, B, n, m):
    """The dynamic program over anti-diagonals, pairs by falling n + m."""
    P, N, M = len(n), A.shape[1], B.shape[1]
    measure, pct, delta = case["measure"], case.get("band_pct", -1), case.get("delta", -1)
    lcss = measure == "lcss"
    edge = 0.0 if lcss else INF
    rev = torch.zeros(P, M + 2 * N, 2, dtype=torch.float64, device="cuda")
    rev[:, N:N + M] = B.flip(1)
    i = torch.arange(N, device="cuda")
    ends = (n + m - 2).tolist()
    W = None
    if measure == "dtw" and pct >= 0:
        W = ((pct * torch.maximum(n, m) + 99) // 100 * (torch.minimum(n, m) - 1))[:, None]
    one = torch.full((P, N + 1), edge, dtype=torch.float64, device="cuda")  # column 0: row -1
    two = one.clone()
    if not lcss:
        two[:, 0] = 0.0  # D(-1,-1)
    out = torch.empty(P, dtype=torch.float64, device="cuda")
    live = P
    for t in range(N + M - 1):
        r = N + M - 1 - t
        d = A[:live] - rev[:live, r:r + N]
        j = t - i
        inside = (j >= 0) & (j < m[:live, None]) & (i < n[:live, None])
        if W is not None:
            inside &= (i * (m[:live, None] - 1) - j * (n[:live, None] - 1)).abs() <= W[:live]
        up, left, diag = one[:live, :-1], one[:live, 1:], two[:live, :-1]
        if lcss:
            hit = (d.float().abs() < case["epsilon"]).all(-1)
            if delta >= 0:
                hit &= (i - j).abs() <= delta
            v = torch.where(hit, diag + 1, torch.maximum(up, left))
            v = torch.where(inside, v, 0.0)
        else:
            cost = d[..., 0].square() + d[..., 1].square()
            if measure == "dtw" and case.get("cost", 0):
                cost = cost.sqrt()
            least = torch.minimum(torch.minimum(up, left), diag)
            v = torch.maximum(cost, least) if measure == "frechet" else cost + least
            v = torch.where(inside, v, INF)
        two = one
        one = torch.nn.functional.pad(v, (1, 0), value=edge)
        while live and ends[live - 1] == t:  # the shortest of the pairs end here
            first = live
            while first and ends[first - 1] == t:
                first -= 1
            rows = torch.arange(first, live, device="cuda")
            out[first:live] = one[rows, n[first:live]]
            live = first
        if not live:
            break
    return out


def _ref64(case, t1, t2):
    """The reference's batch semantics: the K best candidates by its bound,
    then the best of their values."""
    nt, n, measure = case["nt"], case["n"], case["measure"]
    a = torch.from_numpy(t1).cuda().double().reshape(nt, n, 2)
    b = torch.from_numpy(t2).cuda().double().reshape(nt, -1, 2)
    m = b.shape[1]
    K = min(50 if measure == "euclidean" else 10, nt)
    if measure in ("hausdorff", "euclidean"):  # nearest bounding boxes, ties by index
        gap = torch.maximum(a.amin(1)[:, None] - b.amax(1)[None], b.amin(1)[None] - a.amax(1)[:, None])
        key = gap.clamp(min=0).square().sum(-1)
    else:  # the r = 5 envelope of the query at each candidate position
        at = torch.arange(m, device="cuda") * n // m
        win = (at[:, None] + torch.arange(-5, 6, device="cuda")).clamp(0, n - 1)
        lo, hi = a[:, win].amin(2), a[:, win].amax(2)
        key = torch.empty(nt, nt, dtype=torch.float64, device="cuda")
        for s in range(0, nt, 64):
            l, h = lo[s:s + 64, None], hi[s:s + 64, None]
            if measure == "lcss":
                inside = (b[None].float() > l.float() - 0.5) & (b[None].float() < h.float() + 0.5)
                key[s:s + 64] = -inside.all(-1).sum(-1).double()
            else:
                d = torch.maximum(l - b[None], b[None] - h).clamp(min=0).square().sum(-1).sqrt()
                key[s:s + 64] = d.sum(-1) if measure == "dtw" else d.amax(-1)
    ci = torch.argsort(key, stable=True, dim=1)[:, :K].reshape(-1)
    qi = torch.arange(nt, device="cuda").repeat_interleave(K)
    if measure == "euclidean":
        v = (a[qi] - b[ci]).square().sum((1, 2)).reshape(nt, K)
        return v.amin(1).sqrt()
    full = dict(case, epsilon=0.5, delta=-1, band_pct=-1, cost=1)
    lens = (a, torch.full((nt,), n, device="cuda")), (b, torch.full((nt,), m, device="cuda"))
    v = _pair_values(full, *lens, qi, ci).reshape(nt, K)
    if measure == "lcss":
        return v.amax(1) / min(n, m)
    return v.amin(1) if measure == "dtw" else v.amin(1).sqrt()
