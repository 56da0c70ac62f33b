"""Kernels at the sizes where their tiles, remainders and dispatch rules end,
against the oracle (bit for bit unless a test says otherwise)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 257, 1000])
@pytest.mark.parametrize("dim,pd,offset", [(1, 16, 0), (3, 16, 0), (4, 16, 0), (32, 32, 0), (33, 48, 0), (100, 112, 0),
                                           (64, 96, 0), (64, 64, 1)])
def test_encode_fp16_row_and_column_remainders(cuda, oracle_mod, n, dim, pd, offset):
    """32-row warps and 32-column chunks, padding wider than the rows' last
    chunk, and rows that do not start on a 16-byte boundary (offset floats)."""
    from fvgb300 import scan

    torch = cuda
    rng = np.random.default_rng(n * 131 + dim)
    x = (rng.standard_normal((n, dim)) * np.exp(rng.uniform(-8, 8, (n, 1)))).astype(np.float32)
    buf = torch.empty(n * dim + offset, device="cuda")
    xd = buf[offset:].view(n, dim)
    xd.copy_(torch.from_numpy(x))
    codes, norms = scan.encode_fp16(xd, pd)
    ref_codes, ref_norms = oracle_mod.encode_fp16_padded(x)
    got = codes.cpu().numpy().view(np.uint16)
    assert np.array_equal(got[:, :dim], ref_codes[:, :dim])
    assert not got[:, dim:].any()
    assert np.array_equal(norms.cpu().numpy().view(np.uint32), ref_norms.view(np.uint32))


@pytest.mark.parametrize("metric", ["l2", "ip", "cosine"])
@pytest.mark.parametrize(
    "n,dim,nq,k",
    [(200, 96, 3, 100), (256, 64, 129, 1), (1000, 100, 33, 10), (4097, 128, 300, 12), (20_001, 70, 5, 100),
     (33_000, 200, 257, 25), (140_003, 48, 64, 60), (140_003, 264, 1, 10)],
)
@pytest.mark.parametrize("fp8,masked", [(False, False), (False, True), (True, True)])
def test_bounded_scan_equals_unbounded(cuda, metric, n, dim, nq, k, fp8, masked):
    """The scan bounded by the minima pass (every width of a minimum, sampled
    and whole bases, one and several query blocks, partial last tiles, bases
    too small for it) returns what the scan without a bound returns."""
    from fvgb300 import datasets, scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(n + dim + k)
    x = torch.randn((n, dim), generator=g, device="cuda")
    q = torch.randn((nq, dim), generator=g, device="cuda")
    t = scan.Fp8Table(x) if fp8 else scan.Fp16Table(x)
    search = scan.fp8_search if fp8 else scan.fp16_search
    mask = torch.from_numpy(datasets.bernoulli_mask_words(n, 0.3, 7).view(np.int32)).cuda() if masked else None
    with scan.tuned(tc_prepass=0):
        ref = search(t, q, k, metric, mask=mask)
    # (one tile and a 400-row shortlist: its range heaps report an overflow)
    status = scan.device_status()
    got = search(t, q, k, metric, mask=mask)
    torch.cuda.synchronize()
    assert scan.device_status() == status
    assert torch.equal(got, ref)


@pytest.mark.parametrize("nq,k", [(1, 10), (130, 10)])
def test_select_with_more_keys_than_foreseen(cuda, nq, k):
    """The sampled tiles (every 32nd) hold only far rows, so the bound admits
    nearly every row and the selection meets full range heaps, more keys than
    its block holds: it falls back to their k-th key, same answer."""
    from fvgb300 import scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(3)
    n = 64 * 32 * 256 + 77
    x = torch.randn((n, 32), generator=g, device="cuda")
    x[(torch.arange(n, device="cuda") // 256) % 32 == 0] *= 100.0
    q = torch.randn((nq, 32), generator=g, device="cuda")
    t = scan.Fp16Table(x)
    with scan.tuned(tc_prepass=0):
        ref = scan.fp16_search(t, q, k, "l2")
    with scan.tuned(tc_prepass_stride=32):
        got = scan.fp16_search(t, q, k, "l2")
    torch.cuda.synchronize()
    assert scan.device_status() == 0
    assert torch.equal(got, ref)


@pytest.mark.parametrize("n", [1, 2, 3, 33, 64, 100, 127, 128, 129, 255, 256, 257, 1000, 1024, 2048, 2049, 4096])
def test_block_sort_sizes(cuda, n):
    """The block sort around its warp (128 keys) and barrier strides."""
    from fvgb300 import scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(n)
    keys = torch.randint(-50, 50, (n,), generator=g, device="cuda").float()
    vals = torch.randperm(n, generator=g, device="cuda").to(torch.int32)
    ko, vo = scan.bitonic_sort(keys, vals)
    order = np.lexsort((vals.cpu().numpy(), keys.cpu().numpy()))
    assert np.array_equal(ko.cpu().numpy(), keys.cpu().numpy()[order])
    assert np.array_equal(vo.cpu().numpy(), vals.cpu().numpy()[order])


@pytest.mark.parametrize("metric", ["l2", "ip", "cosine"])
@pytest.mark.parametrize("nq", [1, 8, 9, 16, 17, 33, 64, 77, 129])
@pytest.mark.parametrize("n,dim,k", [(1, 1, 1), (127, 31, 32), (129, 32, 33), (700, 36, 128), (1500, 101, 129),
                                     (5000, 64, 256)])
def test_flat_query_tiles_and_list_lengths(cuda, oracle_mod, metric, nq, n, dim, k):
    """Every query-tile width with its remainder, row and dimension
    remainders, list lengths around the 32 and 128 keys of a merge; integer
    rows give many equal distances (ties -> lower slot)."""
    from fvgb300 import datasets, scan

    torch = cuda
    rng = np.random.default_rng(n * 7 + nq)
    base = np.rint(rng.uniform(-3, 3, (n, dim))).astype(np.float32)
    queries = rng.standard_normal((nq, dim), dtype=np.float32) if nq % 2 else base[rng.integers(0, n, nq)]
    mask = datasets.bernoulli_mask_words(n, 0.6, 3) if nq > 8 else None
    md = None if mask is None else torch.from_numpy(mask.view(np.int32)).cuda()
    res = scan.flat_scan(torch.from_numpy(base).cuda(), torch.from_numpy(queries).cuda(), k, metric, mask=md)
    r = res.cpu().numpy()
    ref = oracle_mod.exact_knn(base, queries, k, metric, mask=mask)
    assert np.array_equal(r[..., 0].view(np.uint32), ref["id"])
    assert np.array_equal(r[..., 1].view(np.uint32), ref["distance"].view(np.uint32))


@pytest.mark.parametrize("metric", ["l2", "ip", "cosine"])
@pytest.mark.parametrize("data", ["normal", "integers", "shifted", "outliers", "tiny", "huge", "duplicates", "broken",
                                  "sorted"])
@pytest.mark.parametrize("n,dim,nq,k,masked", [(2048, 8, 32, 1, False), (2305, 33, 130, 10, True),
                                               (9001, 100, 65, 256, False), (40_003, 256, 48, 100, True)])
def test_filtered_flat_scan_equals_plain(cuda, metric, data, n, dim, nq, k, masked):
    """The exact scan behind the tensor-core filter returns the plain scan's
    answer bit for bit: ordinary rows, ties, a common offset, rows far outside
    the others' scale, values near the ends of fp32, equal rows, zero and
    non-finite rows and queries, rows in order of distance."""
    from fvgb300 import datasets, scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(n + dim)
    x = torch.randn((n, dim), generator=g, device="cuda")
    q = torch.randn((nq, dim), generator=g, device="cuda")
    if data == "integers":
        x, q = (x * 3).round(), (q * 3).round()
    elif data == "shifted":
        x, q = x + 300.0, q + 300.0
    elif data == "outliers":
        x[::97] *= 5000.0
        q[::7] *= 5000.0
    elif data == "tiny":
        x, q = x * 1e-21, q * 1e-21
    elif data == "huge":
        x, q = x * 1e17, q * 1e17
    elif data == "duplicates":
        x = x[torch.randint(0, 40, (n,), generator=g, device="cuda")]
    elif data == "broken":
        x[5], x[n - 1, 0], x[7], q[3], q[4, 0], q[5, -1] = 0.0, float("nan"), float("inf"), 0.0, float("nan"), -float("inf")
    elif data == "sorted":
        x = x[torch.argsort((x - q[0]).square().sum(1))]
    mask = torch.from_numpy(datasets.bernoulli_mask_words(n, 0.5, 9).view(np.int32)).cuda() if masked else None
    ids = torch.randperm(4 * n, generator=g, device="cuda")[:n].to(torch.int32) if masked else None
    with scan.tuned(flat_tc=0):
        ref = scan.flat_scan(x, q, k, metric, mask=mask, vec_ids=ids)
    with scan.tuned(flat_tc=1):
        got = scan.flat_scan(x, q, k, metric, mask=mask, vec_ids=ids)
    torch.cuda.synchronize()
    assert torch.equal(got, ref)


def _ivf_case(oracle_mod, n, dim, nlist, m_pq, seed, skew):
    rng = np.random.default_rng(seed)
    cent = rng.uniform(-2, 2, (nlist, dim)).astype(np.float32)
    w = np.arange(1, nlist + 1, dtype=np.float64) ** -skew
    assign = rng.choice(nlist, n, p=w / w.sum()).astype(np.uint32)
    x = (cent[assign] + np.float32(0.6) * rng.standard_normal((n, dim))).astype(np.float32)
    q = (cent[rng.integers(0, nlist, 21)] + np.float32(0.6) * rng.standard_normal((21, dim))).astype(np.float32)
    t = oracle_mod.build_ivf(x, nlist=nlist, m_pq=m_pq, iters=2, seed=seed)
    return x, q, t


@pytest.mark.parametrize("mode", ["pq", "sq8", "rabitq"])
@pytest.mark.parametrize("n,dim,nlist,m_pq,nprobe,rerank,skew", [
    (3000, 64, 200, 16, 200, 33, 1.2),   # several chunks of 32 lists, many empty or of a few postings
    (6000, 48, 33, 12, 33, 300, 0.5),    # one list over a chunk; PQ codes without 16-byte rows
    (9000, 128, 12, 32, 9, 1, 1.0),      # lists on both sides of the PQ table threshold, no rerank
    (2500, 256, 40, 64, 17, 128, 0.8),
    (700, 20, 7, 5, 7, 64, 0.0),         # ragged rows
])
@pytest.mark.parametrize("masked", [False, True])
def test_ivf_list_sequences(cuda, oracle_mod, mode, n, dim, nlist, m_pq, nprobe, rerank, skew, masked):
    """The walk over many lists as one sequence: empty lists, lists shorter than
    a warp, chunk borders, both code layouts, one CTA per query and ranges."""
    from fvgb300 import datasets, scan
    from fvgb300.ivf import IvfTable

    torch = cuda
    x, q, t = _ivf_case(oracle_mod, n, dim, nlist, m_pq, n + dim, skew)
    mask = datasets.bernoulli_mask_words(n, 0.3, 5) if masked else None
    fn = {"pq": oracle_mod.ivf_pq_search, "sq8": oracle_mod.ivf_sq_search, "rabitq": oracle_mod.ivf_rabitq_search}[mode]
    ref = fn(t, x, q, 12, nprobe, rerank, mask=mask)
    md = None if mask is None else torch.from_numpy(mask.view(np.int32)).cuda()
    for list_major in (False, True):
        table = IvfTable(mode, t, vectors=x, list_major=list_major)
        for split in (0, 3, -1):
            with scan.tuned(ivf_split=split):
                r = table.search(torch.from_numpy(q).cuda(), 12, nprobe, rerank, mask=md).cpu().numpy()
            assert np.array_equal(r[..., 0].view(np.uint32), ref["id"])
            assert np.array_equal(r[..., 1].view(np.uint32), ref["distance"].view(np.uint32))
    assert scan.device_status() == 0


@pytest.mark.parametrize("n", [1, 7, 8, 9, 65, 1000])
@pytest.mark.parametrize("dim,pad,offset", [(1, 0, 0), (4, 0, 0), (13, 0, 0), (14, 16, 0), (96, 0, 0), (96, 0, 1),
                                            (157, 0, 0), (260, 32, 0)])
def test_encode_fp8_row_and_column_remainders(cuda, n, dim, pad, offset):
    """Groups of eight rows, rows that end inside a word, a row's last digit at
    its last column (13), wider padding, and rows off a 16-byte boundary
    (offset floats): codes, digits and scales as from the definition, and the
    norms to the last bit of a compensated sum (2^-23 of relative error)."""
    from fvgb300 import scan

    torch = cuda
    rng = np.random.default_rng(n * 131 + dim)
    x = (rng.standard_normal((n, dim)) * np.exp(rng.uniform(-3, 3, (n, 1)))).astype(np.float32)
    x[n // 2] = 0.0
    buf = torch.empty(n * dim + offset, device="cuda")
    xd = buf[offset:].view(n, dim)
    xd.copy_(torch.from_numpy(x))
    pd = scan.fp8_padded_dim(dim) + pad
    codes, scales, norms = scan.encode_fp8(xd, pd)
    nrm = norms.cpu().numpy()
    exact = (x.astype(np.float64) ** 2).sum(1)
    # each square and the final sum rounded once
    assert np.all(np.abs(nrm - exact) <= exact * 2.0 ** -23)
    s = scales.cpu().numpy()
    assert np.all(s == s[0])
    b = int(np.log2(s[0]))
    if nrm.max() > 0:
        assert np.ldexp(np.float32(896.0), 2 * b - 2) < nrm.max() <= np.ldexp(np.float32(896.0), 2 * b)
    to_e4m3 = lambda v: torch.from_numpy(np.ascontiguousarray(v, dtype=np.float32)).cuda().to(torch.float8_e4m3fn)
    want = np.zeros((n, pd), dtype=np.uint8)
    want[:, :dim] = to_e4m3(np.ldexp(x, -b)).view(torch.uint8).cpu().numpy()
    r = np.ldexp(nrm, -1 - 2 * b).astype(np.float32)
    for i in range(3):
        c = to_e4m3(r)
        want[:, dim + i] = c.view(torch.uint8).cpu().numpy()
        r = (r - c.float().cpu().numpy()).astype(np.float32)
    assert np.array_equal(codes.cpu().numpy().view(np.uint8), want)


@pytest.mark.parametrize("n", [1, 3, 9, 500])
@pytest.mark.parametrize("dim", [5, 32, 33, 64, 100, 129, 256, 500, 777, 1024, 1100])
def test_rabitq_encoder_row_lengths(cuda, oracle_mod, n, dim):
    """Every padded length held in registers, the first that is not, batches of
    rows that are not full, and a residual of zero."""
    from fvgb300.ivf import build_rabitq

    torch = cuda
    rng = np.random.default_rng(dim * 7 + n)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    cent = rng.standard_normal((6, dim)).astype(np.float32)
    x[0] = cent[2]  # a zero residual
    assign = rng.integers(0, 6, n).astype(np.int32)
    assign[0] = 2
    ref = oracle_mod.rabitq_encode(x, cent, assign)
    got = build_rabitq(torch.from_numpy(x).cuda(), torch.from_numpy(cent).cuda(), torch.from_numpy(assign).cuda())
    torch.cuda.synchronize()
    for key in ("rot_centroids", "rabitq_bits", "rabitq_meta"):
        assert np.array_equal(got[key].cpu().numpy().view(np.uint32), ref[key].view(np.uint32)), key


@pytest.mark.parametrize("dim,offset", [(16, 0), (48, 0), (64, 0), (100, 0), (37, 0), (128, 4), (130, 0)])
@pytest.mark.parametrize("nq,nlist", [(3, 11), (520, 40)])
def test_ivf_sq8_row_staging(cuda, oracle_mod, dim, offset, nq, nlist):
    """Rows copied ahead (few queries, or rows off a 16-byte boundary by their
    length or the table's start) and rows staged in turn: last chunks of every
    width, lists shorter than a warp, lanes without a second row."""
    from fvgb300.ivf import IvfTable

    torch = cuda
    x, q, t = _ivf_case(oracle_mod, 2200, dim, nlist, max(d for d in (1, 2, 4) if dim % d == 0), dim + nq, 1.0)
    q = np.resize(q, (nq, dim)).astype(np.float32)
    ref = oracle_mod.ivf_sq_search(t, x, q, 10, 9, 40)
    for list_major in (False, True):
        table = IvfTable("sq8", t, vectors=x, list_major=list_major)
        if offset:
            name = "codes_lm" if list_major else "codes"
            codes = getattr(table, name)
            buf = torch.empty(codes.numel() + offset, dtype=torch.uint8, device="cuda")
            buf[offset:].copy_(codes.reshape(-1).view(torch.uint8))
            setattr(table, name, buf[offset:].view(codes.shape))
            table._build_structs()
        r = table.search(torch.from_numpy(q).cuda(), 10, 9, 40).cpu().numpy()
        assert np.array_equal(r[..., 0].view(np.uint32), ref["id"])
        assert np.array_equal(r[..., 1].view(np.uint32), ref["distance"].view(np.uint32))


@pytest.mark.parametrize("stride", [2, 3, 16])
def test_sample_stride_that_does_not_fit(cuda, stride):
    """A stride whose minima would not fit the scan's scratch (many queries, few
    ranges) is raised until they do; the answer stays the unbounded scan's."""
    from fvgb300 import scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(stride)
    x = torch.randn((300_000, 32), generator=g, device="cuda")
    q = torch.randn((2500, 32), generator=g, device="cuda")
    t = scan.Fp16Table(x)
    with scan.tuned(tc_prepass=0):
        ref = scan.fp16_search(t, q, 5, "l2")
    with scan.tuned(tc_prepass_stride=stride):
        got = scan.fp16_search(t, q, 5, "l2")
    torch.cuda.synchronize()
    assert scan.device_status() == 0
    assert torch.equal(got, ref)


def _fp_table(scan, precision, x):
    return scan.Fp16Table(x) if precision == "fp16" else scan.Fp8Table(x, per_vector=precision == "fp8_rows")


@pytest.mark.parametrize("precision,broken", [("fp16", "nan"), ("fp16", "overflow"), ("fp8", "nan"), ("fp8_rows", "nan")])
@pytest.mark.parametrize("k", [1, 10])
def test_bound_ignores_columns_without_a_distance(cuda, precision, broken, k):
    """Whole groups of columns whose distance is NaN (NaN rows; finite rows
    beyond fp16's range against queries with zeros) are no rows near the query:
    the bounded scan still returns what the scan without a bound returns."""
    from fvgb300 import scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn((10_000, 128), generator=g, device="cuda")
    q = torch.randn((70, 128), generator=g, device="cuda")
    if broken == "nan":
        x[1024:4096] = float("nan")
    else:
        x[1024:4096] = 1e6
        q[:, ::3] = 0.0
    t = _fp_table(scan, precision, x)
    search = scan.fp16_search if precision == "fp16" else scan.fp8_search
    with scan.tuned(tc_prepass=0):
        ref = search(t, q, k, "l2")
    got = search(t, q, k, "l2")
    torch.cuda.synchronize()
    assert (ref[..., 0] != -1).all()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("precision", ["fp8", "fp8_rows"])
@pytest.mark.parametrize("rows", ["all", "some"])
def test_cosine_bound_with_norms_that_overflow(cuda, precision, rows):
    """Cosine rows and queries whose product of squared norms overflows fp32
    have the distance 1, whatever their angle: the bounded scan ranks them so too."""
    from fvgb300 import scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn((10_000, 64), generator=g, device="cuda")
    q = torch.randn((70, 64), generator=g, device="cuda") * 1e10
    if rows == "all":
        x *= 1e10
    else:
        x[1000:3000] *= 1e10
    t = _fp_table(scan, precision, x)
    with scan.tuned(tc_prepass=0):
        ref = scan.fp8_search(t, q, 10, "cosine")
    got = scan.fp8_search(t, q, 10, "cosine")
    torch.cuda.synchronize()
    assert (ref[..., 0] != -1).all()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("metric", ["ip", "cosine", "l2"])
@pytest.mark.parametrize("k", [1, 10, 100])
def test_bound_of_products_that_overflow(cuda, metric, k):
    """One coordinate beyond fp16's range makes a product infinite, and the row
    nearer than any other: a bound that is itself infinite admits those rows."""
    from fvgb300 import scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn((20_000, 96), generator=g, device="cuda")
    q = torch.randn((70, 96), generator=g, device="cuda")
    x[::5, 3] = 1e6
    q[::2, 3] = q[::2, 3].abs() + 0.1
    t = scan.Fp16Table(x)
    with scan.tuned(tc_prepass=0):
        ref = scan.fp16_search(t, q, k, metric)
    scan.device_status()
    got = scan.fp16_search(t, q, k, metric)
    torch.cuda.synchronize()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("metric", ["l2", "ip", "cosine"])
def test_filtered_flat_scan_survives_a_wait_that_runs_out(cuda, metric):
    """A tensor-core pass that gives up a wait (a 1 ns limit) has not seen every
    row: the plain scan answers the call, which is exact and reports nothing."""
    from fvgb300 import scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn((20_000, 64), generator=g, device="cuda")
    q = torch.randn((200, 64), generator=g, device="cuda")
    with scan.tuned(flat_tc=0):
        ref = scan.flat_scan(x, q, 10, metric)
    scan.device_status()
    with scan.tuned(flat_tc=1, tc_wait_limit_ns=1):
        got = scan.flat_scan(x, q, 10, metric)
        torch.cuda.synchronize()
    assert scan.device_status() == 0
    assert torch.equal(got, ref)


@pytest.mark.parametrize("offset", [0, 8, 16])
def test_filtered_flat_scan_in_a_callers_arena(cuda, offset):
    """A caller's arena that starts on an 8-byte boundary serves the plain scan,
    one on a 16-byte boundary the filtered one: the same answer."""
    import ctypes as C

    from fvgb300 import _lib, scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn((20_000, 64), generator=g, device="cuda")
    q = torch.randn((200, 64), generator=g, device="cuda")
    with scan.tuned(flat_tc=0):
        ref = scan.flat_scan(x, q, 10, "l2")
    arena = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    handle = C.c_void_p(stream.cuda_stream)
    _lib.call("fv_set_stream_scratch", handle, C.c_void_p(arena.data_ptr() + offset), arena.numel() - offset)
    try:
        with scan.tuned(flat_tc=1):
            scan.profile_enable(True)
            scan.profile_summary()
            got = scan.flat_scan(x, q, 10, "l2", stream=stream)
            stream.synchronize()
            ran = scan.profile_summary()
    finally:
        scan.profile_enable(False)
        _lib.call("fv_release_stream_scratch", handle)
    assert ("flat_tc_prep" in ran) == (offset % 16 == 0)
    assert torch.equal(got, ref)


@pytest.mark.parametrize("path", ["flat", "ivf"])
def test_scans_while_knobs_change(cuda, oracle_mod, path):
    """Another thread sets the knobs that the tensor-core passes of an exact scan
    or a coarse probe are planned by: each call keeps the plan that its scratch
    was taken for."""
    import threading

    from fvgb300 import scan
    from fvgb300.ivf import IvfTable

    torch = cuda
    if path == "flat":
        g = torch.Generator(device="cuda").manual_seed(8)
        x = torch.randn((20_000, 200), generator=g, device="cuda")
        q = torch.randn((150, 200), generator=g, device="cuda")
        search = lambda: scan.flat_scan(x, q, 10, "l2")
    else:
        x, q, t = _ivf_case(oracle_mod, 6000, 200, 400, 8, 3, 0.5)
        table = IvfTable("sq8", t, vectors=x)
        q = torch.from_numpy(np.resize(q, (150, 200)).astype(np.float32)).cuda()
        search = lambda: table.search(q, 10, 9, 40)
    with scan.tuned(flat_tc=0, ivf_tc_coarse=0):
        ref = search()
    stop = threading.Event()

    def turn():
        i = 0
        while not stop.is_set():
            scan.tune_set("tc.pair", (-1, 0)[i % 2])
            scan.tune_set("tc.prepass_stride", (0, 2, 7)[i % 3])
            scan.tune_set("tc.prepass", (-1, 0)[i % 5 == 0])
            i += 1

    with scan.tuned(flat_tc=1, ivf_tc_coarse=1, tc_pair=-1, tc_prepass_stride=0, tc_prepass=-1):
        thread = threading.Thread(target=turn)
        thread.start()
        try:
            got = [search() for _ in range(300)]
        finally:
            stop.set()
            thread.join()
    torch.cuda.synchronize()
    assert all(torch.equal(r, ref) for r in got)


def test_filtered_flat_scan_and_captured_graphs(cuda):
    """A capture that finds no memory for the filter takes the plain scan; a graph
    that holds the filter's memory keeps it when a larger call asks for more; and
    a filtered call leaves the arena that another graph holds alone."""
    import ctypes as C

    from fvgb300 import _lib, scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn((20_000, 64), generator=g, device="cuda")
    q = torch.randn((200, 64), generator=g, device="cuda")
    x2 = torch.randn((60_000, 128), generator=g, device="cuda")
    q2 = torch.randn((500, 128), generator=g, device="cuda")
    table, q16 = scan.Fp16Table(x[:2000].clone()), q[:10].clone()
    with scan.tuned(flat_tc=0):
        ref, ref2 = scan.flat_scan(x, q, 10, "l2"), scan.flat_scan(x2, q2, 10, "l2")
    ref16 = scan.fp16_search(table, q16, 10, "l2")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    outs = [torch.zeros_like(r) for r in (ref, ref, ref16)]
    flat = lambda out: scan.flat_scan(x, q, 10, "l2", out=out, stream=stream)
    fp16 = lambda: scan.fp16_search(table, q16, 10, "l2", out=outs[2], stream=stream)
    try:
        with scan.tuned(flat_tc=0):
            flat(outs[0])  # the arena fits the plain scan (and the tensor-core scan)
        fp16()
        with scan.tuned(flat_tc=1):
            plain = scan.Graph.capture(lambda: flat(outs[0]), stream)
            fp16_graph = scan.Graph.capture(fp16, stream)
            flat(outs[1])
            filtered = scan.Graph.capture(lambda: flat(outs[1]), stream)
            assert filtered.kernels > plain.kernels
            got2 = scan.flat_scan(x2, q2, 10, "l2", stream=stream)  # grows the filter's memory
            noise = torch.full((1 << 26,), 7, dtype=torch.int32, device="cuda")
            for o in outs:
                o.zero_()
            torch.cuda.synchronize()
            for graph in (plain, fp16_graph, filtered):
                graph.launch(stream)
            stream.synchronize()
        del noise
        assert torch.equal(got2, ref2)
        assert torch.equal(outs[0], ref) and torch.equal(outs[1], ref) and torch.equal(outs[2], ref16)
    finally:
        stream.synchronize()
        _lib.call("fv_release_stream_scratch", C.c_void_p(stream.cuda_stream))


@pytest.mark.parametrize("dim,rerank", [(3750, 7000), (3751, 7000), (3752, 7000), (10_918, 100), (10_919, 100)])
def test_ivf_sq8_staging_at_the_shared_memory_limit(cuda, oracle_mod, dim, rerank):
    """Rows and shortlists with which the staging takes the last bytes of a
    block's shared memory: the call runs (unstaged where it must)."""
    from fvgb300.ivf import IvfTable

    torch = cuda
    x, q, t = _ivf_case(oracle_mod, 600, dim, 4, 1, dim, 0.5)
    ref = oracle_mod.ivf_sq_search(t, x, q[:3], 10, 4, rerank)
    r = IvfTable("sq8", t, vectors=x).search(torch.from_numpy(q[:3]).cuda(), 10, 4, rerank).cpu().numpy()
    assert np.array_equal(r[..., 0].view(np.uint32), ref["id"])
    assert np.array_equal(r[..., 1].view(np.uint32), ref["distance"].view(np.uint32))


@pytest.mark.parametrize("precision", ["fp16", "fp8", "fp8_rows"])
@pytest.mark.parametrize("n,dim,nq,k,overfetch,splits", [(20_000, 96, 300, 100, 0, 0), (33_000, 64, 2500, 256, 0, 0),
                                                         (131_000, 64, 300, 100, 1, 6), (4000, 300, 70, 150, 1, 4)])
def test_certain_bound_over_rows_in_order(cuda, precision, n, dim, nq, k, overfetch, splits):
    """All rows near a query in one range, whose list holds fewer than the
    answer: the query is scanned again without its bound, and the slots are
    filled (and the overflow reported) as the scan without a bound does."""
    from fvgb300 import scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(n + k)
    x = torch.randn((n, dim), generator=g, device="cuda")
    q = torch.randn((nq, dim), generator=g, device="cuda") * 0.05
    x = x[torch.argsort(x.square().sum(1))]
    t = _fp_table(scan, precision, x)
    opts = scan.options(overfetch=overfetch, splits=splits)
    search = lambda: (scan.fp16_search if precision == "fp16" else scan.fp8_search)(t, q, k, "l2", opts=opts)
    scan.device_status()
    with scan.tuned(tc_prepass=0):
        ref = search()
    status = scan.device_status()
    got = search()
    torch.cuda.synchronize()
    assert scan.device_status() == status
    assert (ref[..., 0] != -1).all()
    assert torch.equal(got, ref)


@pytest.mark.parametrize("metric", ["l2", "ip", "cosine"])
@pytest.mark.parametrize("n,dim,nq,k,clusters", [(255, 64, 9, 1, 3), (257, 64, 9, 1, 3), (2047, 32, 140, 3, 11),
                                                 (20_001, 96, 64, 10, 50), (70_003, 300, 130, 10, 90),
                                                 (400_010, 40, 200, 12, 200)])
@pytest.mark.parametrize("precision,masked", [("fp16", False), ("fp16", True), ("fp8", True), ("fp8_rows", True)])
def test_bounded_scan_of_rows_in_clusters(cuda, metric, n, dim, nq, k, clusters, precision, masked):
    """Rows stored by cluster: the bound's sample (runs of 8 rows spread over the
    base, partial last tiles, bases of less than one tile) and the ranges (every
    so many tiles) give the answer of the scan without a bound."""
    from fvgb300 import datasets, scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(n + dim)
    c = torch.randn((clusters, dim), generator=g, device="cuda")
    own = torch.randint(0, clusters, (n,), generator=g, device="cuda").sort().values
    x = torch.randn((n, dim), generator=g, device="cuda") * 0.3 + c[own]
    q = torch.randn((nq, dim), generator=g, device="cuda") * 0.3 + c[torch.arange(nq, device="cuda") % clusters]
    t = _fp_table(scan, precision, x)
    search = scan.fp16_search if precision == "fp16" else scan.fp8_search
    mask = torch.from_numpy(datasets.bernoulli_mask_words(n, 0.3, 7).view(np.int32)).cuda() if masked else None
    scan.device_status()
    with scan.tuned(tc_prepass=0):
        ref = search(t, q, k, metric, mask=mask)
    got = search(t, q, k, metric, mask=mask)
    torch.cuda.synchronize()
    assert scan.device_status() == 0
    assert torch.equal(got, ref)


def test_select_with_more_keys_than_foreseen_by_runs(cuda):
    """The sampled runs (every 32nd run of 8 rows) hold only far rows, so the
    bound admits nearly every row: full range lists, and a selection that falls
    back to their k-th key, same answer."""
    from fvgb300 import scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(3)
    n = 64 * 32 * 256 + 77
    x = torch.randn((n, 32), generator=g, device="cuda")
    x[(torch.arange(n, device="cuda") // 8) % 32 == 0] *= 100.0
    q = torch.randn((130, 32), generator=g, device="cuda")
    t = scan.Fp16Table(x)
    with scan.tuned(tc_prepass=0):
        ref = scan.fp16_search(t, q, 10, "l2")
    with scan.tuned(tc_prepass_stride=32):
        got = scan.fp16_search(t, q, 10, "l2")
    torch.cuda.synchronize()
    assert scan.device_status() == 0
    assert torch.equal(got, ref)


@pytest.mark.parametrize("metric", ["l2", "ip", "cosine"])
@pytest.mark.parametrize("data", ["normal", "integers", "sorted", "nan row", "inf rows", "far rows", "masked far row",
                                  "zero row"])
def test_filtered_flat_scan_answers_by_itself(cuda, metric, data):
    """The filter proves nearly every query of a call, rows that are not finite or
    far outside the others' scale among the base or not: the plain scan of the
    flagged queries takes a small part of the plain scan's time (a twentieth as
    a rule; the limit is a half)."""
    from fvgb300 import scan

    torch = cuda
    n, dim, nq = 60_000, 128, 512
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn((n, dim), generator=g, device="cuda")
    q = torch.randn((nq, dim), generator=g, device="cuda")
    mask = None
    if data == "integers":
        x, q = (x * 20).round(), (q * 20).round()
    elif data == "sorted":
        x = x[torch.argsort((x - q[0]).square().sum(1))]
    elif data == "nan row":
        x[777, 3] = float("nan")
    elif data == "inf rows":
        x[777, 3], x[20_001] = float("inf"), -float("inf")
    elif data == "far rows":
        x[777] *= 1000.0
        x[20_001:20_020] *= 3e6
    elif data == "masked far row":
        x[777] *= 1000.0
        mask = torch.full(((n + 31) // 32,), -1, dtype=torch.int32, device="cuda")
        mask[777 // 32] &= ~(1 << (777 % 32))
    elif data == "zero row":
        x[777] = 0.0
    run = lambda: scan.flat_scan(x, q, 10, metric, mask=mask)
    res = {}
    for knob in (0, 1):
        with scan.tuned(flat_tc=knob):
            run()
            torch.cuda.synchronize()
            scan.profile_enable(True)
            try:
                scan.profile_summary()
                out = run()
                torch.cuda.synchronize()
                res[knob] = out, scan.profile_summary()
            finally:
                scan.profile_enable(False)
    assert torch.equal(res[1][0], res[0][0])
    assert "flat_tc_prep" in res[1][1] and "flat_tc_prep" not in res[0][1]
    assert res[1][1]["flat_f32_scan"]["ms"] < 0.5 * res[0][1]["flat_f32_scan"]["ms"]


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 63, 65])
@pytest.mark.parametrize("dim,pd", [(127, 128), (128, 144), (129, 144), (132, 144), (120, 272), (256, 256), (300, 304),
                                    (511, 512), (512, 512), (768, 768), (1031, 1040)])
def test_encode_fp16_chunks(cuda, oracle_mod, n, dim, pd):
    """Rows of several 128-dimension chunks, full and partial, as 16-byte loads and
    single values, two rows a warp (from 512 dimensions) and eight: the norms'
    sums go on across chunks; padding that reaches a chunk past the row."""
    from fvgb300 import scan

    torch = cuda
    rng = np.random.default_rng(n * 131 + dim)
    x = (rng.standard_normal((n, dim)) * np.exp(rng.uniform(-8, 8, (n, 1)))).astype(np.float32)
    codes, norms = scan.encode_fp16(torch.from_numpy(x).cuda(), pd)
    ref_codes, ref_norms = oracle_mod.encode_fp16_padded(x)
    got = codes.cpu().numpy().view(np.uint16)
    assert np.array_equal(got[:, :dim], ref_codes[:, :dim])
    assert not got[:, dim:].any()
    assert np.array_equal(norms.cpu().numpy().view(np.uint32), ref_norms.view(np.uint32))


@pytest.mark.parametrize("n", [1, 3, 8, 200])
@pytest.mark.parametrize("dim", [255, 256, 263, 768, 1000])
def test_encode_fp8_rows_a_warp(cuda, n, dim):
    """One row a warp gives the codes, scale and norms, bit for bit, that two
    (the same rows at the head of a table of 20,000) and eight (of 100,000) give."""
    from fvgb300 import scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(n + dim)
    x = torch.randn((n, dim), generator=g, device="cuda")
    few = scan.encode_fp8(x)
    for total in (20_000, 100_000):
        big = torch.zeros((total, dim), device="cuda")
        big[:n] = x
        many = scan.encode_fp8(big)
        for a, b in zip(few, many):
            assert torch.equal(a, b[:n])


@pytest.mark.parametrize("precision", ["fp16", "fp8", "fp8_rows"])
@pytest.mark.parametrize("scale", [1.0, 1e-9, 1e9])
def test_cosine_bound_with_rows_of_zeros(cuda, precision, scale):
    """Zero rows (distance 1) among the base, queries of any scale and a zero
    query: the bounded scan returns what the scan without a bound returns, also
    where the zero rows are among the answer."""
    from fvgb300 import scan

    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(12)
    x = torch.randn((9_000, 64), generator=g, device="cuda")
    x[::7] = 0.0
    q = torch.randn((150, 64), generator=g, device="cuda") * scale
    q[::10] = -x[1].abs() * scale
    x[1::2] = x[1::2].abs()
    q[5] = 0.0
    t = _fp_table(scan, precision, x)
    search = scan.fp16_search if precision == "fp16" else scan.fp8_search
    with scan.tuned(tc_prepass=0):
        ref = search(t, q, 10, "cosine")
    got = search(t, q, 10, "cosine")
    torch.cuda.synchronize()
    assert torch.equal(got, ref)
