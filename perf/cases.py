"""The work that users of the scan path have it do, as timed cases.

Each case is one call (or one table encoding) through the public Python entry
points of fvgb300 at sizes taken from this repository's benchmark and tests, or
generic ones. Inputs are synthetic, made on the GPU from the seed alone:
Gaussian mixtures as in the benchmark configurations (integer-valued rows in
[0, 255], unit vectors, unbounded rows), and Zipf-sized posting lists. The
IVF tables are built here with plain torch, so they do not depend on the
library's own encoders.

`exact` evaluates the same search with torch in 64 bits: brute force for the
flat scans, and for the IVF scans the probed lists, the approximate distances
of their codes, the shortlist and its rerank.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "flashvector-gpu_gb300"))

from fvgb300 import scan  # noqa: E402
from fvgb300.index import BUILD_FP16, GpuVectorIndex, IndexConfig  # noqa: E402
from fvgb300.ivf import IvfTable, build_rabitq  # noqa: E402

DEV = "cuda"
SENTINEL = 1e30  # distance of an unfilled result slot


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one query against the buffer of live inserts (or a small collection): launch latency
        dict(name="flat_1q", path="flat", data="int", n=10_000, dim=128, queries=1, k=10, metric="l2", allowed=1.0),
        # exact search of a batch: the benchmark's exact fp32 configuration
        dict(name="flat_batch", path="flat", data="int", n=100_000, dim=128, queries=1000, k=10, metric="l2",
             allowed=1.0),
        # exact cosine search with a filter at ragged sizes, a long result list
        dict(name="flat_cos_ragged", path="flat", data="free", n=30_011, dim=99, queries=77, k=100, metric="cosine",
             allowed=0.5),
        # the headline configuration: embedding search of a full batch, half the rows filtered out
        dict(name="fp16_batch", path="fp16", data="unit", n=1_000_000, dim=768, queries=1024, k=10, metric="ip",
             allowed=0.5),
        # one interactive query against the same table
        dict(name="fp16_1q", path="fp16", data="unit", n=1_000_000, dim=768, queries=1, k=10, metric="ip",
             allowed=1.0),
        # short rows, a long result list, nothing a multiple of a tile
        dict(name="fp16_l2_ragged", path="fp16", data="free", n=200_003, dim=100, queries=333, k=100, metric="l2",
             allowed=1.0),
        # the largest job: all-neighbours style batch over a short-row fp8 table
        dict(name="fp8_batch", path="fp8", data="free", n=10_000_000, dim=96, queries=10_000, k=100, metric="l2",
             allowed=1.0),
        # product-quantised lists of Zipf sizes under a 10% filter, reranked
        dict(name="ivf_pq_batch", path="ivf", mode="pq", n=1_000_000, dim=128, queries=2000, k=10, metric="l2",
             allowed=0.1, nlist=4096, nprobe=32, rerank=400, m_pq=32),
        # binary codes over the same kind of lists, unfiltered
        dict(name="ivf_rabitq_batch", path="ivf", mode="rabitq", n=1_000_000, dim=128, queries=2000, k=10,
             metric="l2", allowed=1.0, nlist=4096, nprobe=32, rerank=400, m_pq=0),
        # a few served requests against byte codes of long rows
        dict(name="ivf_sq8_few", path="ivf", mode="sq8", n=300_000, dim=768, queries=8, k=10, metric="ip",
             allowed=1.0, nlist=1024, nprobe=64, rerank=100, m_pq=0),
        # the engine's blocking search on host buffers, with deleted rows and live inserts present
        dict(name="engine_fp16", path="engine", data="int", n=50_000, dim=128, queries=500, k=10, metric="l2",
             added=2_000, deleted=500),
        # encoding a table: fp16 rows and norms of an embedding set
        dict(name="encode_fp16", path="encode", data="unit", precision="fp16", n=500_000, dim=768),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["flat", "flat", "fp16", "fp16", "fp8", "ivf", "ivf", "ivf", "engine", "encode"])
    metric = rng.choice(["l2", "l2", "ip", "cosine"])
    if path == "flat":
        dim, queries = _log(rng, 8, 512), _log(rng, 1, 2000)
        n = _log(rng, 1000, min(200_000, max(2000, 12e9 / (dim * queries))))
        return dict(path=path, data=rng.choice(["int", "free"]), n=n, dim=dim, queries=queries, k=_log(rng, 1, 128),
                    metric=metric, allowed=rng.choice([1.0, 0.5, 0.1]))
    if path == "fp16":
        dim, queries = _log(rng, 32, 1024), _log(rng, 1, 1024)
        n = _log(rng, 10_000, min(2_000_000, 700e6 / dim))
        return dict(path=path, data=rng.choice(["unit", "free"]), n=n, dim=dim, queries=queries, k=_log(rng, 1, 100),
                    metric=metric, allowed=rng.choice([1.0, 0.5]))
    if path == "fp8":
        dim, queries = _log(rng, 32, 512), _log(rng, 1, 8000)
        n = _log(rng, 50_000, min(6_000_000, 800e6 / dim, max(60_000, 8e12 / (dim * queries))))
        return dict(path=path, data=rng.choice(["unit", "free"]), n=n, dim=dim, queries=queries, k=_log(rng, 1, 100),
                    metric=metric, allowed=rng.choice([1.0, 0.5]))
    if path == "ivf":
        mode = rng.choice(["pq", "sq8", "rabitq"])
        sub, m_pq = rng.choice([4, 8]), rng.choice([16, 24, 32])
        dim = sub * m_pq if mode == "pq" else _log(rng, 48, 768 if mode == "sq8" else 512)
        n = _log(rng, 20_000, min(1_000_000, 230e6 / dim))
        nlist = _log(rng, 32, max(64, min(4096, n / 100)))
        nprobe = _log(rng, 1, min(64, nlist))
        k = _log(rng, 1, 50)
        return dict(path=path, mode=mode, n=n, dim=dim, queries=_log(rng, 1, 1000), k=k, metric=metric,
                    allowed=rng.choice([1.0, 0.5, 0.1]), nlist=nlist, nprobe=nprobe, rerank=_log(rng, max(k, 2), 512),
                    m_pq=m_pq if mode == "pq" else 0)
    if path == "engine":
        n = _log(rng, 5_000, 100_000)
        return dict(path=path, data=rng.choice(["int", "free"]), n=n, dim=_log(rng, 32, 512),
                    queries=_log(rng, 1, 500), k=_log(rng, 1, 50), metric=rng.choice(["l2", "ip"]),
                    added=rng.choice([0, _log(rng, 1, 4000)]), deleted=rng.choice([0, n // 100]))
    dim = _log(rng, 32, 1024)
    return dict(path=path, data="free", precision=rng.choice(["fp16", "fp8", "rabitq"]),
                n=_log(rng, 10_000, min(2_000_000, 380e6 / dim)), dim=dim)


# ---------------------------------------------------------------- inputs
def _gen(seed, stream):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 7919 + stream)
    return g


def _mixture(case, seed, count, stream):
    """`count` rows of the case's Gaussian mixture (stream 1: the base, 2: the queries, 3: live inserts)."""
    data, dim = case["data"], case["dim"]
    comps, sigma = {"int": (1024, 20.0), "unit": (4096, 0.3), "free": (4096, 0.5)}[data]
    g = _gen(seed, 0)
    centers = torch.rand((comps, dim), generator=g, device=DEV) * 255 if data == "int" else torch.randn(
        (comps, dim), generator=g, device=DEV)
    if data == "unit":
        centers /= centers.norm(dim=1, keepdim=True)
    g = _gen(seed, stream)
    out = torch.empty((count, dim), dtype=torch.float32, device=DEV)
    for s in range(0, count, 1 << 20):
        e = min(count, s + (1 << 20))
        x = torch.randn((e - s, dim), generator=g, device=DEV).mul_(sigma)
        x += centers[torch.randint(0, comps, (e - s,), generator=g, device=DEV)]
        if data == "int":
            x.round_().clamp_(0.0, 255.0)
        elif data == "unit":
            x /= x.norm(dim=1, keepdim=True)
        out[s:e] = x
    return out


def _allowed(case, seed):
    """bool[n] of the rows that the filter lets through, or None."""
    if case["allowed"] >= 1.0:
        return None
    return torch.rand((case["n"],), generator=_gen(seed, 5), device=DEV) < case["allowed"]


def _mask_words(allowed):
    """The filter as packed 32-bit words, least significant bit first."""
    if allowed is None:
        return None
    pad = (-allowed.numel()) % 32
    bits = torch.nn.functional.pad(allowed, (0, pad)).view(-1, 32).to(torch.int64)
    words = (bits << torch.arange(32, device=DEV)).sum(1)
    return torch.where(words >= 2 ** 31, words - 2 ** 32, words).to(torch.int32)


def _hadamard(p):
    h = torch.ones((1, 1), dtype=torch.float64, device=DEV)
    while h.shape[0] < p:
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
    return h / math.sqrt(p)


def _rotation(signs, p, dtype):
    """The RaBitQ rotation (three rounds of signs and Walsh-Hadamard) as a matrix for row vectors."""
    m, h = torch.eye(p, dtype=torch.float64, device=DEV), _hadamard(p)
    for r in range(3):
        m = (m * signs.view(3, p)[r].double()) @ h
    return m.to(dtype)


def _ivf_lists(case, seed):
    """Rows in Zipf(1.1)-sized lists around scattered centres, and queries around the same centres."""
    n, dim, nlist = case["n"], case["dim"], case["nlist"]
    rng = np.random.default_rng([seed, 3])
    w = np.arange(1, nlist + 1, dtype=np.float64) ** -1.1
    floor = min(64, n // (2 * nlist))
    sizes = np.floor(floor + (n - floor * nlist) * w / w.sum()).astype(np.int64)
    sizes[0] += n - sizes.sum()
    sizes = torch.from_numpy(sizes[rng.permutation(nlist)]).to(DEV)
    g = _gen(seed, 1)
    comps = torch.rand((1024, dim), generator=g, device=DEV) * 255
    cent = comps[torch.randint(0, 1024, (nlist,), generator=g, device=DEV)]
    cent = cent + 20.0 * torch.randn((nlist, dim), generator=g, device=DEV)
    assign = torch.repeat_interleave(torch.arange(nlist, device=DEV), sizes)
    assign = assign[torch.randperm(n, generator=g, device=DEV)]
    rows = torch.randn((n, dim), generator=g, device=DEV).mul_(8.0).add_(cent[assign]).round_().clamp_(0.0, 255.0)
    g = _gen(seed, 2)
    li = assign[torch.randint(0, n, (case["queries"],), generator=g, device=DEV)]
    q = (cent[li] + 8.0 * torch.randn((case["queries"], dim), generator=g, device=DEV)).round_().clamp_(0.0, 255.0)
    vec_ids = torch.argsort(assign, stable=True)
    offsets = torch.zeros(nlist + 1, dtype=torch.int64, device=DEV)
    offsets[1:] = torch.cumsum(sizes, 0)
    return rows, cent, assign, q, offsets, vec_ids


def _pq_codebooks(res, m, g):
    """Codewords of each sub-space: sampled residuals and three rounds of k-means on a sample."""
    sub = res.shape[1] // m
    pick = torch.randint(0, res.shape[0], (8192,), generator=g, device=DEV)
    x = res[pick].view(-1, m, sub).permute(1, 0, 2).contiguous()
    cb = x[:, :256].clone()
    for _ in range(3):
        near = torch.cdist(x, cb).argmin(2)
        hot = torch.nn.functional.one_hot(near, 256).to(torch.float32)
        count = hot.sum(1)
        cb = torch.where(count[..., None] > 0, hot.transpose(1, 2) @ x / count.clamp_min(1)[..., None], cb)
    return cb.contiguous()


def _ivf_table(case, seed):
    """The tables of a built IVF index (codes by row id) as torch tensors."""
    n, dim, mode = case["n"], case["dim"], case["mode"]
    rows, cent, assign, q, offsets, vec_ids = _ivf_lists(case, seed)
    t = dict(centroids=cent, offsets=offsets.to(torch.int32), vec_ids=vec_ids.to(torch.int32))
    if mode == "rabitq":
        p = max(32, 1 << (dim - 1).bit_length())
        signs = torch.randint(0, 2, (3 * p,), generator=_gen(seed, 4), device=DEV).to(torch.float32) * 2 - 1
        rot = _rotation(signs, p, torch.float32)[:dim].contiguous()
        bits, meta = torch.empty((n, p // 32), dtype=torch.int32, device=DEV), torch.empty((n, 4), device=DEV)
        shift = torch.arange(32, device=DEV)
        for s in range(0, n, 1 << 18):
            x = rows[s:s + (1 << 18)]
            r = x - cent[assign[s:s + (1 << 18)]]
            y = r @ rot
            on = y >= 0
            w = (on.view(-1, p // 32, 32).to(torch.int64) << shift).sum(2)
            bits[s:s + (1 << 18)] = torch.where(w >= 2 ** 31, w - 2 ** 32, w).to(torch.int32)
            r2 = r.square().sum(1)
            meta[s:s + (1 << 18)] = torch.stack([r2, r2 / y.abs().sum(1).clamp_min(1e-12), on.sum(1).float(),
                                                 x.square().sum(1)], 1)
        t.update(padded_dim=p, rot_signs=signs, rot_centroids=cent @ rot, rabitq_bits=bits, rabitq_meta=meta)
        return rows, q, t
    res = rows - cent[assign]
    if mode == "sq8":
        mins = res.min(0).values
        scales = ((res.max(0).values - mins) / 255.0).clamp_min(1e-8)
        codes = ((res - mins) / scales).round_().clamp_(0, 255).to(torch.uint8)
        t.update(sq_mins=mins, sq_scales=scales, sq_codes=codes)
        return rows, q, t
    m = case["m_pq"]
    cb = _pq_codebooks(res, m, _gen(seed, 4))
    codes = torch.empty((n, m), dtype=torch.uint8, device=DEV)
    for s in range(0, n, 1 << 16):
        x = res[s:s + (1 << 16)].view(-1, m, dim // m).permute(1, 0, 2)
        d = cb.square().sum(2)[:, None, :] - 2.0 * torch.bmm(x, cb.transpose(1, 2))
        codes[s:s + (1 << 16)] = d.argmin(2).to(torch.uint8).t()
    t.update(codebooks=cb, pq_codes=codes)
    return rows, q, t


def prepare(case, seed):
    path = case["path"]
    if path == "ivf":
        rows, q, t = _ivf_table(case, seed)
        table = IvfTable(case["mode"], t, vectors=rows, list_major=True)
        return dict(case=case, table=table, q=q, mask=_mask_words(_allowed(case, seed)))
    x = _mixture(case, seed, case["n"], 1)
    if path == "encode":
        s = dict(case=case, x=x)
        if case["precision"] == "rabitq":
            s["cent"] = x[:256].clone()
            s["assign"] = torch.randint(0, 256, (case["n"],), generator=_gen(seed, 4), device=DEV, dtype=torch.int32)
        return s
    q = _mixture(case, seed, case["queries"], 2)
    if path == "engine":
        idx = GpuVectorIndex(IndexConfig(dim=case["dim"], metric=case["metric"], build_flags=BUILD_FP16))
        torch.cuda.synchronize()
        idx.build_device(x)
        if case["deleted"]:
            idx.delete_ids(_deleted(case, seed).cpu().numpy())
        if case["added"]:
            idx.add_vectors(_mixture(case, seed, case["added"], 3).cpu().numpy())
        return dict(case=case, index=idx, q=q.cpu().numpy())
    mask = _mask_words(_allowed(case, seed))
    if path == "flat":
        return dict(case=case, x=x, q=q, mask=mask)
    table = scan.Fp16Table(x) if path == "fp16" else scan.Fp8Table(x)
    return dict(case=case, table=table, q=q, mask=mask)


def _deleted(case, seed):
    return torch.randperm(case["n"], generator=_gen(seed, 6), device=DEV)[: case["deleted"]]


# ---------------------------------------------------------------- one pass
def _answer(res):
    """The two halves of a (queries, k) result array, as views of it."""
    return dict(ids=res[..., 0], distances=res.view(torch.float32)[..., 1])


def run(state):
    c = state["case"]
    path = c["path"]
    if path == "flat":
        return _answer(scan.flat_scan(state["x"], state["q"], c["k"], c["metric"], mask=state["mask"]))
    if path == "fp16":
        return _answer(scan.fp16_search(state["table"], state["q"], c["k"], c["metric"], mask=state["mask"]))
    if path == "fp8":
        return _answer(scan.fp8_search(state["table"], state["q"], c["k"], c["metric"], mask=state["mask"]))
    if path == "ivf":
        return _answer(state["table"].search(state["q"], c["k"], c["nprobe"], c["rerank"], c["metric"],
                                             mask=state["mask"]))
    if path == "engine":
        ids, dist = state["index"].batch_search_fp16_tc(state["q"], c["queries"], c["k"])
        return dict(ids=ids.view(np.int32), distances=dist)
    if c["precision"] == "fp16":
        rows, norms = scan.encode_fp16(state["x"])
        return dict(rows=rows, norms=norms)
    if c["precision"] == "fp8":
        rows, scales, norms = scan.encode_fp8(state["x"])
        return dict(rows=rows, scales=scales, norms=norms)
    t = build_rabitq(state["x"], state["cent"], state["assign"])
    return dict(bits=t["rabitq_bits"], meta=t["rabitq_meta"])


def work(case):
    n, dim, path = case["n"], case["dim"], case["path"]
    if path == "encode":
        pad = {"fp16": 2 * (-(-dim // 16) * 16) + 4, "fp8": -(-(dim + 3) // 16) * 16 + 8,
               "rabitq": max(32, 1 << (dim - 1).bit_length()) // 8 + 16}[case["precision"]]
        return dict(bytes=n * (4 * dim + pad), flops=3 * n * dim)
    nq, k = case["queries"], case["k"]
    io = nq * (4 * dim + 8 * k)
    if path == "ivf":
        code = {"pq": case["m_pq"], "sq8": dim, "rabitq": max(32, 1 << (dim - 1).bit_length()) // 8 + 16}[case["mode"]]
        share = case["nprobe"] / case["nlist"] * case["allowed"]
        touched = n * case["allowed"] * (1 - (1 - case["nprobe"] / case["nlist"]) ** nq)
        rerank = min(n * case["allowed"], nq * min(case["rerank"], n * share))
        return dict(bytes=io + 4 * case["nlist"] * dim + touched * (code + 4) + rerank * 4 * dim,
                    flops=nq * (2 * case["nlist"] * dim + share * n * 2 * code + 3 * case["rerank"] * dim))
    elem = {"flat": 4, "fp16": 2, "fp8": 1, "engine": 2}[path]
    extra = case.get("added", 0)
    return dict(bytes=io + n * dim * elem + 4 * extra * dim + (n / 8 if case.get("allowed", 1.0) < 1 else 0),
                flops=2 * nq * (n + extra) * dim)


# ---------------------------------------------------------------- 64 bits
def _distances64(q, x, metric):
    """Distances of q [b, d] to x [b, c, d], in 64 bits."""
    q, x = q.double()[:, None, :], x.double()
    if metric == "l2":
        return (q - x).square_().sum(2)
    dot = (q * x).sum(2)
    if metric == "ip":
        return -dot
    return 1.0 - dot / (q.square().sum(2).sqrt() * x.square().sum(2).sqrt() + 1e-8)


def _brute(x, q, k, metric, allowed):
    """The k smallest distances of each query, ascending: candidates by 32-bit products, then 64-bit distances."""
    n, nq = x.shape[0], q.shape[0]
    want = min(n, k + 64)
    best_d = torch.full((nq, want), math.inf, device=DEV)
    best_i = torch.full((nq, want), -1, dtype=torch.int64, device=DEV)
    qq = q / q.norm(dim=1, keepdim=True) if metric == "cosine" else q
    step = max(4096, min(250_000, int(2.5e9 / nq)))
    for s in range(0, n, step):
        xs = x[s:s + step]
        if metric == "cosine":
            xs = xs / xs.norm(dim=1, keepdim=True)
        d = qq @ xs.t()
        if metric == "l2":
            d.mul_(-2.0).add_(xs.square().sum(1))
        else:
            d.neg_()
        if allowed is not None:
            d.masked_fill_(~allowed[s:s + step], math.inf)
        v, i = torch.topk(d, min(want, d.shape[1]), dim=1, largest=False)
        v, i = torch.cat([best_d, v], 1), torch.cat([best_i, i + s], 1)
        best_d, at = torch.topk(v, want, dim=1, largest=False)
        best_i = torch.gather(i, 1, at)
    out = torch.full((nq, k), SENTINEL, dtype=torch.float64, device=DEV)
    rows = max(1, int(4e8 / (want * x.shape[1])))
    for s in range(0, nq, rows):
        i = best_i[s:s + rows]
        d = _distances64(q[s:s + rows], x[i.clamp_min(0)], metric)
        d.masked_fill_(torch.isinf(best_d[s:s + rows]), SENTINEL)
        d = torch.sort(d, dim=1).values[:, :k]
        out[s:s + rows, : d.shape[1]] = d
    return out


def _ivf_exact(case, seed):
    rows, q, t = _ivf_table(case, seed)
    n, dim, mode, k = case["n"], case["dim"], case["mode"], case["k"]
    allowed = _allowed(case, seed)
    cent, offsets, ids = t["centroids"].double(), t["offsets"].cpu().numpy(), t["vec_ids"].long()
    qd = q.double()
    ok = None if allowed is None else allowed[ids]
    codes = t[{"pq": "pq_codes", "sq8": "sq_codes", "rabitq": "rabitq_bits"}[mode]][ids]
    if mode == "rabitq":
        p = t["padded_dim"]
        rq = qd @ _rotation(t["rot_signs"], p, torch.float64)[:dim]
        rc, meta = t["rot_centroids"].double(), t["rabitq_meta"][ids].double()
        byte = (torch.arange(256, device=DEV)[:, None] >> torch.arange(8, device=DEV)) & 1
        codes = codes.contiguous().view(torch.uint8)
    d2 = (qd.square().sum(1)[:, None] + cent.square().sum(1) - 2.0 * qd @ cent.t())
    probes = torch.topk(d2, case["nprobe"], dim=1, largest=False).indices
    probes_h = probes.cpu().numpy()
    out = torch.full((case["queries"], k), SENTINEL, dtype=torch.float64, device=DEV)
    for i in range(case["queries"]):
        pos, of = [], []
        for j, l in enumerate(probes_h[i]):
            pos.append(np.arange(offsets[l], offsets[l + 1]))
            of.append(np.full(offsets[l + 1] - offsets[l], j))
        pos = torch.from_numpy(np.concatenate(pos)).to(DEV)
        of = torch.from_numpy(np.concatenate(of)).to(DEV)
        if ok is not None:
            keep = ok[pos]
            pos, of = pos[keep], of[keep]
        if not pos.numel():
            continue
        r = qd[i] - cent[probes[i]]
        if mode == "pq":
            m = case["m_pq"]
            lut = (r.view(-1, m, 1, dim // m) - t["codebooks"].double()[None]).square().sum(3)
            at = (of[:, None] * m + torch.arange(m, device=DEV)) * 256 + codes[pos].long()
            est = lut.view(-1)[at].sum(1)
        elif mode == "sq8":
            est = torch.empty(pos.numel(), dtype=torch.float64, device=DEV)
            for s in range(0, pos.numel(), 1 << 18):
                rec = codes[pos[s:s + (1 << 18)]].double() * t["sq_scales"].double() + t["sq_mins"].double()
                est[s:s + (1 << 18)] = (r[of[s:s + (1 << 18)]] - rec).square_().sum(1)
        else:
            diff = rq[i] - rc[probes[i]]
            lo, hi = diff.min(1, keepdim=True).values, diff.max(1, keepdim=True).values
            u = ((diff - lo) * 15.0 / (hi - lo).clamp_min(1e-12)).round().clamp(0, 15)
            lut = torch.einsum("lbe,ve->lbv", u.view(-1, p // 8, 8), byte.double())
            at = (of[:, None] * (p // 8) + torch.arange(p // 8, device=DEV)) * 256 + codes[pos].long()
            s_bu = lut.view(-1)[at].sum(1)
            m = meta[pos]
            x = ((hi - lo) / 15.0)[of, 0] * (2 * s_bu - u.sum(1)[of]) + lo[of, 0] * (2 * m[:, 2] - p)
            est = d2[i][probes[i]][of] + m[:, 0] - 2.0 * m[:, 1] * x
            if case["metric"] == "ip":
                est = -0.5 * (qd[i].square().sum() + m[:, 3] - est)
        if case["rerank"] != 1:
            short = torch.topk(est, min(max(case["rerank"], k), est.numel()), largest=False).indices
            est = _distances64(q[i][None], rows[ids[pos[short]]][None], case["metric"])[0]
        est = torch.sort(est).values[:k]
        out[i, : est.numel()] = est
    return dict(ids=None, distances=out)


def exact(case, seed):
    path = case["path"]
    if path == "ivf":
        # the loop over queries touches every probed code in 64 bits
        heavy = case["queries"] * (1 + case["n"] * case["allowed"] * case["dim"] / 4e7)
        return None if heavy > 20_000 else _ivf_exact(case, seed)
    x = _mixture(case, seed, case["n"], 1)
    if path == "encode":
        norms = torch.cat([x[s:s + 65536].double().square().sum(1) for s in range(0, case["n"], 65536)])
        if case["precision"] == "rabitq":
            return None  # codes and sums of the library's own rotation
        return dict(rows=None, norms=norms) if case["precision"] == "fp16" else dict(rows=None, scales=None, norms=norms)
    q = _mixture(case, seed, case["queries"], 2)
    if path == "engine":
        allowed = torch.ones(case["n"] + case["added"], dtype=torch.bool, device=DEV)
        if case["deleted"]:
            allowed[_deleted(case, seed)] = False
        if case["added"]:
            x = torch.cat([x, _mixture(case, seed, case["added"], 3)])
        return dict(ids=None, distances=_brute(x, q, case["k"], case["metric"], allowed))
    return dict(ids=None, distances=_brute(x, q, case["k"], case["metric"], _allowed(case, seed)))
