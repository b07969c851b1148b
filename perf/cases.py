"""The measured work of this framework: searches, index building and their real sizes.

A case is one call (or the few calls) that a user's program makes through the public entry points
of ``mestrado_gb300``: single and batched searches in the plain FP32 and the precision form, the
re-ranked and the refined search, the flat PQ search, parallel2's ``core_gpu``, quantizer training
and base encoding. Sizes follow the benchmark's workloads (1M / 1,024 lists, 10M / 65,536 lists,
100M / 262,144 Zipf lists, the 1B workload's long lists with refinement codes); ``draw`` gives more
of the same ranges.

Inputs are synthetic, as the benchmark's are: vectors of a Gaussian mixture (d = 128, component
means uniform in [0, 120], sigma 20, byte-valued). The indexes are drawn from the law that a trained
one follows, without training it: list centroids scattered about their mixture component, list sizes
log-normal (a trained index's are uneven), PQ centroids with the variance that 256 centroids keep of
a Gaussian sub-vector, uniform codes. Queries come from the components of rows drawn at random, so
that long lists and heavy components are probed most.
"""
import math

import numpy as np
import torch

from mestrado_gb300 import gpu_build
from mestrado_gb300.engine import GpuIndex, GpuPQ

D = 128


def listed():
    return [
        # one online query against the 1M drop-in index: latency of the smallest call
        dict(name="query_1", kind="search", nq=1, n=1_000_000, C=1024, m=8, w=16, k=100, mixed=False, ncomp=1024),
        # a front-end's small batch against the 10M index, tensor-core coarse stage, the scan form left to the engine
        dict(name="queries_37", kind="search", nq=37, n=10_000_000, C=65_536, m=8, w=32, k=10, mixed=True, ncomp=4096),
        # the drop-in workload: 10,000 queries, re-rank of the 100 best by the raw vectors
        dict(name="drop_in_rerank", kind="rerank", nq=10_000, n=1_000_000, C=1024, m=8, w=16, k=100, kl=100, ncomp=1024),
        # the 10M workload in the plain form (the default of every entry point) ...
        dict(name="batch_10M_plain", kind="device", nq=10_000, n=10_000_000, C=65_536, m=8, w=32, k=100, mixed=False, ncomp=4096),
        # ... and in the precision form
        dict(name="batch_10M_mixed", kind="device", nq=10_000, n=10_000_000, C=65_536, m=8, w=32, k=100, mixed=True, ncomp=4096),
        # uneven batch through the host entry point, plain form: the 100M workload's shape at 1/5 scale
        dict(name="uneven_20M_plain", kind="uneven", nq=8192, n=20_000_000, C=65_536, m=16, w=256, k=1000, mixed=False, ncomp=65_536),
        # the headline: the 100M workload's uneven batch, precision form, replayed as a CUDA graph
        dict(name="uneven_100M_mixed", kind="graph", nq=32_768, n=100_000_000, C=262_144, m=16, w=256, k=1000, mixed=True, ncomp=262_144),
        # the 1B workload's search on a 1/32 slice: long lists, refinement re-rank of the 1,000 best
        dict(name="refine_long_lists", kind="refine", nq=2000, n=32_000_000, C=16_384, m=8, w=64, k=100, kl=1000, ncomp=1024),
        # exhaustive PQ search of a flat codebook, a small batch
        dict(name="flat_pq", kind="flat", nq=50, n=1_000_000, m=8, k=100),
        # parallel2's core: residuals and probes from the caller
        dict(name="core_residuals", kind="core", nq=500, n=1_000_000, C=1024, m=8, w=8, k=100, ncomp=1024),
        # quantizers of the 1M workload, its 100,000 training vectors
        dict(name="train", kind="train", n=100_000, C=1024, m=8, niter=10, ncomp=1024),
        # base vectors assigned and encoded for an m = 16 index, one odd-sized block of the base
        dict(name="encode", kind="encode", n=500_003, C=16_384, m=16, ncomp=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "rerank", "device", "device", "uneven", "graph", "refine", "flat", "core",
                       "train", "encode"])
    m = rng.choice([8, 16])
    if kind == "search":
        C = rng.choice([1024, 4096, 16_384, 65_536])
        return dict(kind=kind, nq=_log(rng, 1, 300), n=_log(rng, 300 * C, 600 * C), C=C, m=m, w=_log(rng, 4, 64),
                    k=rng.choice([1, 10, 100]), mixed=rng.random() < 0.5, ncomp=min(C, 4096))
    if kind == "rerank":
        return dict(kind=kind, nq=_log(rng, 100, 10_000), n=_log(rng, 200_000, 1_000_000), C=1024, m=m,
                    w=_log(rng, 4, 16), k=rng.choice([1, 10, 100]), kl=rng.choice([100, 200]), ncomp=1024)
    if kind == "device":
        C = rng.choice([4096, 16_384, 65_536])
        return dict(kind=kind, nq=_log(rng, 500, 10_000), n=_log(rng, 150 * C, 300 * C), C=C, m=m, w=_log(rng, 8, 48),
                    k=rng.choice([10, 100]), mixed=rng.random() < 0.5, ncomp=4096)
    if kind in ("uneven", "graph"):
        C = rng.choice([16_384, 65_536])
        return dict(kind=kind, nq=_log(rng, 300, 8192), n=_log(rng, 150 * C, 380 * C), C=C, m=m, w=_log(rng, 32, 256),
                    k=rng.choice([100, 1000]), mixed=rng.random() < 0.6, ncomp=C)
    if kind == "refine":
        return dict(kind=kind, nq=_log(rng, 100, 2000), n=_log(rng, 8_000_000, 32_000_000), C=16_384, m=8,
                    w=_log(rng, 16, 64), k=rng.choice([10, 100]), kl=rng.choice([400, 1000]), ncomp=1024)
    if kind == "flat":
        return dict(kind=kind, nq=_log(rng, 1, 200), n=_log(rng, 10_000, 1_000_000), m=m, k=rng.choice([1, 10, 100]))
    if kind == "core":
        return dict(kind=kind, nq=_log(rng, 10, 1000), n=_log(rng, 200_000, 1_000_000), C=1024, m=m,
                    w=_log(rng, 1, 12), k=rng.choice([10, 100]), ncomp=1024)
    if kind == "train":
        C = rng.choice([256, 1024])
        return dict(kind=kind, n=_log(rng, 20_000, 100_000), C=C, m=m, niter=rng.randint(4, 10), ncomp=C)
    return dict(kind=kind, n=_log(rng, 30_000, 500_000), C=rng.choice([1024, 16_384]), m=m, ncomp=4096)


# -- inputs ---------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device="cuda")


def _vectors(g, means, comp):
    """Byte-valued mixture vectors of the given components."""
    return (means[comp] + 20.0 * _normal(g, len(comp), D)).clamp_(0, 255).round_()


def _index_parts(case, g):
    """Centroids, PQ, list offsets, ids and codes (device tensors; offsets on the host) and queries."""
    n, C, m, nq = case["n"], case["C"], case["m"], case["nq"]
    zipf = case["kind"] in ("uneven", "graph")
    means = 120.0 * torch.rand((case["ncomp"], D), generator=g, device="cuda")
    if zipf:  # components of Zipf-distributed weight hold centroids in proportion to it
        cdf = torch.cumsum(torch.arange(1, case["ncomp"] + 1, device="cuda", dtype=torch.float64) ** -1.1, 0)
        u = torch.rand(C, generator=g, device="cuda", dtype=torch.float64) * cdf[-1]
        comp = torch.searchsorted(cdf, u).clamp_(max=case["ncomp"] - 1)
    else:
        comp = torch.arange(C, device="cuda") % case["ncomp"]
    spread = 7.0 if zipf else 4.5 if C > case["ncomp"] else 1.0
    coa = means[comp] + spread * _normal(g, C, D)
    ds = D // m
    keep = {8: 0.84, 16: 0.67, 32: 0.5}[ds]  # deviation that 256 centroids keep of a ds-dimensional Gaussian
    pq = 20.0 * keep * _normal(g, m, 256, ds)
    cum = torch.cumsum(torch.exp(0.7 * _normal(g, C).double()), 0)
    label = torch.searchsorted(cum, torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * cum[-1])
    label = label.clamp_(max=C - 1).to(torch.int32)
    rows_of = label[torch.randint(0, n, (nq,), generator=g, device="cuda")].long()
    queries = _vectors(g, means, comp[rows_of])
    off = np.zeros(C + 1, np.int64)
    np.cumsum(torch.bincount(label, minlength=C).cpu().numpy(), out=off[1:])
    ids = torch.sort(label, stable=True).indices.to(torch.int32)
    del label
    codes = torch.randint(0, 256, (n, m), generator=g, device="cuda", dtype=torch.uint8)
    return coa, pq, off, ids, codes, queries


def _uneven(case, seed):
    r = np.random.default_rng(int(seed))
    nq, w, k = case["nq"], case["w"], case["k"]
    wq = np.clip(np.exp(r.uniform(0.0, math.log(w), nq)).round(), 1, w).astype(np.int32)
    ks = np.array([x for x in (1, 10, 100, 1000) if x <= k], np.int32)
    kq = r.permutation(ks[-1 - np.arange(nq) % len(ks)])  # the same result count whatever the seed
    wq[0] = w
    return wq, kq


def _refined(g):
    return 9.0 * _normal(g, 8, 256, 16)


def _decoded(coa, pq, off, codes, lo, hi, dtype=torch.float32):
    """Rows lo..hi (list order) rebuilt from their codes: y_l + c1(codes)."""
    lists = torch.from_numpy(np.searchsorted(off, np.arange(lo, hi), side="right") - 1).cuda()
    m = pq.shape[0]
    c1 = torch.cat([pq[s].to(dtype)[codes[lo:hi, s].long()] for s in range(m)], 1)
    return coa[lists].to(dtype) + c1


def _base(g, coa, pq, off, ids, codes):
    """Raw vectors whose codes the index holds (row id = base id)."""
    base = torch.empty((len(ids), D), device="cuda")
    for lo in range(0, len(ids), 1 << 18):
        hi = min(len(ids), lo + (1 << 18))
        x = _decoded(coa, pq, off, codes, lo, hi) + 12.0 * _normal(g, hi - lo, D)
        base[ids[lo:hi].long()] = x.clamp_(0, 255).round_()
    return base


def prepare(case, seed):
    g, kind, st = _gen(seed), case["kind"], dict(kind=case["kind"], case=case)
    if kind in ("train", "encode"):
        means = 120.0 * torch.rand((case["ncomp"], D), generator=g, device="cuda")
        comp = torch.randint(0, case["ncomp"], (case["n"],), generator=g, device="cuda")
        st["x"] = _vectors(g, means, comp)
        if kind == "encode":
            st["coa"] = means[torch.arange(case["C"], device="cuda") % case["ncomp"]] + 4.5 * _normal(g, case["C"], D)
            st["pq"] = 20.0 * (0.84 if case["m"] == 16 else 0.67) * _normal(g, case["m"], 256, D // case["m"])
        return st
    if kind == "flat":
        ds = D // case["m"]
        pq = (60.0 + 35.0 * _normal(g, case["m"], 256, ds)).clamp_(0, 255).cpu().numpy()
        codes = torch.randint(0, 256, (case["n"], case["m"]), generator=g, device="cuda", dtype=torch.uint8).cpu().numpy()
        st["queries"] = (60.0 + 40.0 * _normal(g, case["nq"], D)).clamp_(0, 255).round_().cpu().numpy()
        st["index"] = GpuPQ(pq, codes)
        return st
    coa, pq, off, ids, codes, q = _index_parts(case, g)
    nq, w, k = case["nq"], case["w"], case["k"]
    more = {}
    st["graph"] = None  # goes before the index that it replays on
    if kind == "refine":
        more = dict(pq2=_refined(g).cpu().numpy(),
                    d_codes2=torch.randint(0, 256, (case["n"], 8), generator=g, device="cuda", dtype=torch.uint8))
    base = _base(g, coa, pq, off, ids, codes).cpu().numpy() if kind == "rerank" else None
    coa_h, pq_h = coa.cpu().numpy(), pq.cpu().numpy()
    st["index"] = ix = GpuIndex.from_device(coa_h, pq_h, off, ids, codes, **more)
    if kind == "rerank":
        ix.set_base(base)
    if kind == "core":
        order = torch.topk(torch.cdist(q.double(), coa.double()), w, largest=False).indices
        rid = order.reshape(-1).to(torch.int32).cpu().numpy()
        st["residual"] = (q[:, None, :] - coa[order]).reshape(-1, D).cpu().numpy()
        found = np.minimum(np.diff(off)[rid.reshape(nq, w)].sum(1), k)
        start = np.zeros(nq, np.int32)
        start[1:] = np.cumsum(found)[:-1]
        st.update(rid=rid, start=start, nout=int(found.sum()))
    elif kind in ("search", "uneven"):
        st["queries"] = q.cpu().numpy()
        if kind == "uneven":
            st["wq"], st["kq"] = _uneven(case, seed)
    else:  # device buffers
        total = nq * k
        if kind == "graph":
            wq, kq = _uneven(case, seed)
            total = int(kq.sum())
            st["off"] = torch.from_numpy(np.concatenate([[0], np.cumsum(kq)[:-1]]).astype(np.int64)).cuda()
            st["wq"], st["kq"] = torch.from_numpy(wq).cuda(), torch.from_numpy(kq).cuda()
        st["q"] = q
        st["ids"] = torch.empty(total, dtype=torch.int32, device="cuda")
        st["dis"] = torch.empty(total, dtype=torch.float32, device="cuda")
        if kind == "graph":
            torch.cuda.synchronize()
            stream = torch.cuda.Stream()
            st["graph"] = ix.capture_graph(q.data_ptr(), nq, k, w, st["ids"].data_ptr(), st["dis"].data_ptr(),
                                           mixed_coarse=case["mixed"], mixed_scan=case["mixed"],
                                           d_w_ptr=st["wq"].data_ptr(), d_k_ptr=st["kq"].data_ptr(),
                                           d_off_ptr=st["off"].data_ptr(), stream_ptr=stream.cuda_stream)
    return st


# -- one pass -------------------------------------------------------------


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "train":
        return gpu_build.train_quantizers(st["x"], case["C"], case["m"], niter=case["niter"], seed=3)
    if kind == "encode":
        return gpu_build.encode_base(st["x"], st["coa"], st["pq"])
    ix = st["index"]
    if kind == "flat":
        return ix.pq_search(st["queries"], case["k"])
    if kind == "core":
        return ix.core_gpu(st["residual"], st["rid"], st["start"], st["nout"], case["k"], case["w"])
    if kind == "search":
        return ix.search(st["queries"], case["k"], case["w"], mixed_coarse=case["mixed"],
                         mixed_scan="auto" if case["mixed"] else False)
    if kind == "uneven":
        return ix.search_batched(st["queries"], st["wq"], st["kq"], mixed_coarse=case["mixed"],
                                 mixed_scan=case["mixed"])[:2]
    if kind == "graph":
        st["graph"].launch(torch.cuda.current_stream().cuda_stream)
        return st["ids"], st["dis"]
    mixed = case.get("mixed", False)
    ix.search_device(st["q"].data_ptr(), case["nq"], case["k"], case["w"], st["ids"].data_ptr(), st["dis"].data_ptr(),
                     kl=case.get("kl"), rerank=kind == "rerank", refine=kind == "refine",
                     stream_ptr=torch.cuda.current_stream().cuda_stream,
                     mixed_coarse=mixed or kind == "refine", mixed_scan=mixed)
    return st["ids"], st["dis"]


# -- what a pass cannot do without ---------------------------------------


def work(case):
    """Bytes: queries, centroids, the probed lists' codes (at most all of them, once) and the results.
    Operations: the query x centroid product, the probes' distance tables, the code look-ups."""
    kind, n, m = case["kind"], case["n"], case["m"]
    if kind == "train":
        per = 2.0 * n * (case["C"] * D + 256 * D)
        return dict(bytes=4.0 * (n * D + case["C"] * D + 256 * D), flops=case["niter"] * per)
    if kind == "encode":
        return dict(bytes=4.0 * n * D + n * (4.0 + m), flops=2.0 * n * (case["C"] * D + 256 * D))
    nq, k = case["nq"], case["k"]
    if kind == "flat":
        return dict(bytes=4.0 * nq * D + n * m + 8.0 * nq * k, flops=2.0 * nq * 256 * D + float(nq) * n * m)
    C, w = case["C"], case["w"]
    if kind in ("uneven", "graph"):  # log-uniform probe counts, k over its powers of ten
        w = (w - 1) / math.log(w)
        k = {1000: 277.75, 100: 37.0}.get(k, k)
    rows = nq * w * (n / C) * math.exp(0.49)  # lists are met in proportion to their length
    flops = 2.0 * nq * w * 256 * D + rows * m + (0.0 if kind == "core" else 2.0 * nq * C * D)
    moved = 4.0 * (nq * D * (w if kind == "core" else 1) + C * D) + min(rows, n) * m + 8.0 * nq * k
    if kind == "rerank":
        moved += min(nq * case["kl"], n) * 4.0 * D
        flops += 2.0 * nq * case["kl"] * D
    if kind == "refine":
        moved += min(nq * case["kl"], n) * 16.0
        flops += 4.0 * nq * case["kl"] * D
    return dict(bytes=moved, flops=flops)


# -- the same results in 64 bits -----------------------------------------


def _adc64(res, lists, beg, length, codes, pq, keep):
    """ADC distances of a block of queries in 64 bits: res (b, w, D) residuals, lists (b, w) probes
    (-1: none); the `keep` best per query, ascending, with their rows (inf, -1 past the last)."""
    b, w = lists.shape
    m, ds = pq.shape[0], pq.shape[2]
    tab = ((res.view(b, w, m, 1, ds) - pq[None, None]) ** 2).sum(-1).reshape(-1)  # (b, w, m, 256)
    safe = lists.clamp(min=0)
    ln = torch.where(lists >= 0, length[safe], torch.zeros_like(lists)).reshape(-1)
    first = beg[safe].reshape(-1)
    total = int(ln.sum())
    pair = torch.repeat_interleave(torch.arange(b * w, device="cuda"), ln)
    start = torch.cumsum(ln, 0) - ln
    row = first[pair] + torch.arange(total, device="cuda") - start[pair]
    dist = torch.zeros(total, dtype=torch.float64, device="cuda")
    for s in range(m):
        dist += tab[(pair * m + s) * 256 + codes[row, s].long()]
    per = ln.view(b, w).sum(1)
    q = pair // w
    at = torch.arange(total, device="cuda") - (torch.cumsum(per, 0) - per)[q]
    width = max(int(per.max()), keep)
    full = torch.full((b, width), math.inf, dtype=torch.float64, device="cuda")
    rows = torch.full((b, width), -1, dtype=torch.int64, device="cuda")
    full[q, at] = dist
    rows[q, at] = row
    best, i = torch.topk(full, keep, dim=1, largest=False)
    return best, torch.gather(rows, 1, i)


def exact(case, seed):
    kind = case["kind"]
    if kind == "encode":
        return None  # whole numbers only
    g = _gen(seed)
    if kind == "train":
        return _train64(case, g)
    if kind == "flat":
        ds = D // case["m"]
        pq = (60.0 + 35.0 * _normal(g, case["m"], 256, ds)).clamp_(0, 255).double()
        codes = torch.randint(0, 256, (case["n"], case["m"]), generator=g, device="cuda", dtype=torch.uint8)
        q = (60.0 + 40.0 * _normal(g, case["nq"], D)).clamp_(0, 255).round_().double()
        zero = torch.zeros((1, 1), dtype=torch.int64, device="cuda")
        beg, ln = zero[0], zero[0] + case["n"]
        dis = torch.cat([_adc64(x[None, None], zero, beg, ln, codes, pq, case["k"])[0] for x in q])
        return dis.T.contiguous(), None
    nq, w, k = case["nq"], case["w"], case["k"]
    mean_w = (w - 1) / math.log(w) if kind in ("uneven", "graph") else w
    if nq * mean_w * case["n"] / case["C"] * case["m"] > 3e10:
        return None
    coa, pq, off, ids, codes, q = _index_parts(case, g)
    if kind == "refine":
        pq2 = _refined(g).double()
        codes2 = torch.randint(0, 256, (case["n"], 8), generator=g, device="cuda", dtype=torch.uint8)
    base = _base(g, coa, pq, off, ids, codes) if kind == "rerank" else None
    coa, pq, q = coa.double(), pq.double(), q.double()
    beg, length = torch.from_numpy(off[:-1]).cuda(), torch.from_numpy(np.diff(off)).cuda()
    wq = kq = None
    if kind in ("uneven", "graph"):
        wq, kq = (torch.from_numpy(v).cuda().long() for v in _uneven(case, seed))
    cn = (coa * coa).sum(1)
    keep = case.get("kl", k)
    step = max(1, min(512, int(6e7 / (mean_w * max(case["n"] / case["C"], 256) * 4))))
    out = []
    for q0 in range(0, nq, step):
        x = q[q0:q0 + step]
        order = torch.topk(cn[None, :] - 2.0 * (x @ coa.T), w, largest=False).indices
        if wq is not None:
            order[torch.arange(w, device="cuda")[None, :] >= wq[q0:q0 + step, None]] = -1
            order = order[:, :int(wq[q0:q0 + step].max())]
        res = x[:, None, :] - coa[order.clamp(min=0)]
        best, rows = _adc64(res, order, beg, length, codes, pq, keep)
        if kind == "rerank":
            v = base[ids[rows.clamp(min=0)].long()].double()
            best = ((x[:, None, :] - v) ** 2).sum(-1)
        elif kind == "refine":
            r = rows.clamp(min=0)
            lists = torch.searchsorted(torch.from_numpy(off).cuda(), r, right=True) - 1
            for b0 in range(0, len(x), 32):
                rb, lb = r[b0:b0 + 32], lists[b0:b0 + 32]
                e = x[b0:b0 + 32, None, :] - coa[lb]
                e = e - torch.cat([pq[s][codes[rb, s].long()] for s in range(case["m"])], 2)
                e = e - torch.cat([pq2[s][codes2[rb, s].long()] for s in range(8)], 2)
                best[b0:b0 + 32] = (e * e).sum(-1)
        if kind in ("rerank", "refine"):
            best = torch.where(rows >= 0, best, torch.full_like(best, math.inf))
            best = torch.sort(best, 1).values[:, :k]
        if kq is not None:
            best = best[torch.arange(k, device="cuda")[None, :] < kq[q0:q0 + step, None]]
        elif kind == "core":  # packed: min(k, candidates) results per query
            best = best[rows >= 0]
        out.append(best)
    dis = torch.cat(out)
    return None, dis if kind in ("search", "core", "uneven", "graph") else dis.reshape(-1)


def _mix64(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _hash4(a, b, c, d):
    with np.errstate(over="ignore"):
        a, b, c, d = (np.asarray(v, np.uint64) for v in (a, b, c, d))
        return _mix64(a ^ _mix64(b ^ _mix64(c ^ _mix64(d))))


def _kmeans64(x, k, niter, seed):
    """Lloyd's k-means in 64 bits from one pseudo-random point of each of k slices of x; an empty
    cluster takes a pseudo-random point."""
    n, c = len(x), np.arange(k)
    step = n // k
    cent = x[torch.from_numpy((c * step + (_hash4(seed, 0x1D17, c, 0) % np.uint64(step)).astype(np.int64))).cuda()]
    for it in range(niter):
        a = torch.cat([((cent * cent).sum(1)[None, :] - 2.0 * (b @ cent.T)).argmin(1) for b in x.split(1 << 16)])
        count = torch.bincount(a, minlength=k)
        new = torch.zeros_like(cent).index_add_(0, a, x) / count.clamp(min=1)[:, None]
        again = torch.from_numpy((_hash4(seed, 0xE317, it, c) % np.uint64(n)).astype(np.int64)).cuda()
        cent = torch.where(count[:, None] > 0, new, x[again])
    return cent


def _train64(case, g):
    means = 120.0 * torch.rand((case["ncomp"], D), generator=g, device="cuda")
    comp = torch.randint(0, case["ncomp"], (case["n"],), generator=g, device="cuda")
    x = _vectors(g, means, comp).double()
    coa = _kmeans64(x, case["C"], case["niter"], 3)
    a = torch.cat([((coa * coa).sum(1)[None, :] - 2.0 * (b @ coa.T)).argmin(1) for b in x.split(1 << 16)])
    res = (x - coa[a]).view(len(x), case["m"], D // case["m"])
    pq = [_kmeans64(res[:, s].contiguous(), 256, case["niter"], 3 + 1 + 1 + s) for s in range(case["m"])]
    return coa, torch.stack(pq)
