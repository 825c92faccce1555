"""Kernels at the sizes where their tiling can go wrong -- edges of tiles and
passes, remainders, the smallest and largest of a range -- against the oracle
(bit for bit) or a plain restatement of the same operation."""
import numpy as np
import pytest
import torch

import pyoracle
from helpers import make_queries, oracle_of, tiny_index
from mvr import PREC_BF16, SEM_BASIC, SEM_PP, Index, build, exhaustive

pytestmark = pytest.mark.gpu


def gpu_index(ix):
    return Index.from_arrays(ix["item_n_vec"], ix["centroid"], ix["vq_code"], ix["ivf_off"],
                             ix["ivf_size"], ix["ivf_ids"], ix["weight"], ix["n_bit"],
                             ix["residual"])


# doc lengths around the exact rerank's 32-token rows and 128-token tiles
LENGTHS = [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 160, 255, 256, 257, 300]


@pytest.mark.parametrize("n_bit", [1, 2, 4, 8])
def test_exact_rerank_edges(n_bit):
    """Query widths around the 16- and 32-token passes, shortlists around the
    docs-per-CTA windows (4 to 64), one query and enough for the widest window."""
    ix = tiny_index(n_doc=160, n_centroid=32, n_bit=n_bit, seed=50 + n_bit,
                    lengths=(LENGTHS * 10)[:160])
    o = oracle_of(ix)
    with gpu_index(ix) as g:
        for nq, sem in ((1, SEM_PP), (15, SEM_PP), (16, SEM_BASIC), (17, SEM_PP), (32, SEM_BASIC),
                        (33, SEM_PP), (48, SEM_PP), (49, SEM_BASIC), (64, SEM_PP)):
            q, off = make_queries(ix, 2, nq, seed=nq)
            for ptk in (3, 4, 9, 65, 160):
                r = o.search(q, off, 3, 8, ptk, sem)
                s, i = g.search(q, 3, 8, ptk, tok_off=off, semantics=sem)
                np.testing.assert_array_equal(i, r[1])
                np.testing.assert_array_equal(s, r[0])
        q, off = make_queries(ix, 700, (1, 64), seed=3)
        r = o.search(q, off, 3, 8, 130)
        s, i = g.search(q, 3, 8, 130, tok_off=off)
        np.testing.assert_array_equal(i, r[1])
        np.testing.assert_array_equal(s, r[0])


def top_scan(q, cen, nprobe):
    """The canonical scores' top nprobe per token, by the oracle's assignment
    with every chosen centroid's row removed in turn."""
    left = [np.arange(len(cen))] * len(q)
    out = np.zeros((len(q), nprobe), np.int64)
    for k in range(nprobe):
        for t in range(len(q)):
            j = int(pyoracle.assign(q[t:t + 1], cen[left[t]])[0])  # lowest id on ties
            out[t, k] = left[t][j]
            left[t] = np.delete(left[t], j)
    return out


def unit(x):
    return (x / np.linalg.norm(x, axis=1, keepdims=True)).astype(np.float32)


def hostile(kind, n, c, rng):
    """(vectors, centroids) for which the tensor-core scan's lists or bound give out."""
    x, cen = unit(rng.standard_normal((n, 128))), unit(rng.standard_normal((c, 128)))
    if kind == "rising":   # every centroid beats all before it
        cen = (np.linspace(0.1, 1.0, c)[:, None] * unit(np.ones((1, 128)) + 0 * cen[:1])).astype(np.float32)
        x = np.abs(x)
    elif kind == "equal":  # one centroid many times over
        cen = np.repeat(cen[:1], c, axis=0)
    elif kind == "zero":
        x[: n // 2] = 0
    elif kind == "scale":  # sizes over which a BF16 rounding is larger than unit scores
        x *= np.float32(10.0) ** rng.integers(-12, 12, (n, 1)).astype(np.float32)
        cen *= np.float32(3000.0)
    elif kind == "huge":   # norms that overflow FP32: the bound is not finite
        x[: n // 2] *= np.float32(3e37)
    return x, cen


@pytest.mark.parametrize("n,c", [(1, 1), (1, 63), (127, 64), (128, 65), (129, 1000), (300, 4096),
                                 (5000, 129)])
def test_assign_edges(n, c):
    rng = np.random.default_rng(n + c)
    x, cen = unit(rng.standard_normal((n, 128))), unit(rng.standard_normal((c, 128)))
    code, _ = build.assign(torch.from_numpy(x).cuda(), torch.from_numpy(cen).cuda())
    np.testing.assert_array_equal(code.cpu().numpy(), pyoracle.assign(x, cen).astype(np.int64))


@pytest.mark.parametrize("kind", ["rising", "equal", "zero", "scale", "huge"])
@pytest.mark.parametrize("n,c", [(3, 300), (200, 2000)])
def test_assign_hostile(kind, n, c):
    x, cen = hostile(kind, n, c, np.random.default_rng(n))
    code, _ = build.assign(torch.from_numpy(x).cuda(), torch.from_numpy(cen).cuda())
    np.testing.assert_array_equal(code.cpu().numpy(), pyoracle.assign(x, cen).astype(np.int64))


@pytest.mark.parametrize("kind", ["plain", "rising", "equal", "zero", "scale"])
@pytest.mark.parametrize("nprobe", [1, 2, 3, 4, 7, 8, 9, 16, 17, 32])
def test_probe_edges(kind, nprobe):
    """Probe lists of the plain path: ids of an exact scan, for list widths at and
    beside the powers of two, one query (many splits) and a batch (few)."""
    base = tiny_index(n_doc=60, n_centroid=33, n_bit=2, seed=7)
    rng = np.random.default_rng(nprobe)
    n_cent = 700
    q, cen = hostile(kind, 40, n_cent, rng)
    code = pyoracle.assign(base["tokens"], cen)
    off, size, ids = pyoracle.ivf_build(code, base["item_n_vec"], n_cent)
    ix = dict(base, centroid=cen, vq_code=code, ivf_off=off, ivf_size=size, ivf_ids=ids)
    want = top_scan(q[:5], cen, nprobe)
    with gpu_index(ix) as g:
        t = g.trace(q[:5], 5, nprobe, 20)
        np.testing.assert_array_equal(t["probe_id"].astype(np.int64), want)
        t = g.trace(q, 5, nprobe, 20)
        np.testing.assert_array_equal(t["probe_id"][:5].astype(np.int64), want)
        o = oracle_of(ix)
        many = np.tile(q, (160, 1))
        toff = np.arange(0, len(many) + 1, 40).astype(np.uint64)
        r = o.search(q, toff[:2], 5, nprobe, 20)
        s, i = g.search(many, 5, nprobe, 20, tok_off=toff)
        for k in (0, 77, 159):
            np.testing.assert_array_equal(i[k], r[1][0])
            np.testing.assert_array_equal(s[k], r[0][0])


@pytest.mark.parametrize("n,n_bit,shift", [(1, 1, 0), (3, 2, 1), (1000, 2, 0), (777, 4, 3),
                                           (4097, 8, 0)])
def test_residual_quantiles_edges(n, n_bit, shift):
    """Order statistics of ties, signed zeros and wide exponents, from arrays at any
    4-byte offset, against a sort."""
    rng = np.random.default_rng(n)
    vec = rng.standard_normal((n, 128)).astype(np.float32) * np.float32(10.0) ** rng.integers(-9, 3, (n, 1)).astype(np.float32)
    vec[:, ::7] = np.float32(0.25)
    cen = np.zeros((5, 128), np.float32)
    cen[1:, ::7] = np.float32(0.25)
    cen[2] = -cen[2]
    code = rng.integers(0, 5, n).astype(np.int32)

    def at(a):
        t = torch.empty(a.size + shift, device="cuda")
        t[shift:] = torch.from_numpy(a.reshape(-1)).cuda()
        return t[shift:].view(a.shape)
    cut, w = build.residual_quantiles(at(vec), at(cen), torch.from_numpy(code).cuda(), n_bit)
    e = np.sort((vec - cen[code]).reshape(-1))
    nb = 1 << n_bit
    np.testing.assert_array_equal(cut, [e[int(np.floor((i + 1) / nb * e.size))] for i in range(nb - 1)])
    np.testing.assert_array_equal(w, [e[int(np.floor((i / nb + 0.5 / nb) * e.size))] for i in range(nb)])


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_maxsum_edges(dtype):
    """Max over each doc's columns, sum over each query's tokens: widths around 32 on
    both sides, empty docs, NaN and infinities, against the torch form."""
    lens = np.array([0, 1, 31, 32, 33, 64, 100, 0, 5], np.int64)
    off = np.cumsum([0, 1, 31, 32, 33, 64, 0, 100])
    g = torch.Generator(device="cuda").manual_seed(3)
    s = torch.randn((int(off[-1]), int(lens.sum())), device="cuda", generator=g, dtype=dtype)
    s[5, 40] = float("nan")
    s[70, 200] = float("inf")
    s[71, :] = -float("inf")
    q_off = torch.from_numpy(off).cuda()
    got = exhaustive._maxsum(s, q_off, lens)
    want = exhaustive._maxsum(s.cpu(), q_off.cpu(), lens)
    # sums of up to 100 terms of size ~3 in another order: 100 ulps of 512 at most
    tol = 100 * 512 * torch.finfo(dtype).eps
    torch.testing.assert_close(got.cpu(), want, rtol=0, atol=tol, equal_nan=True)


@pytest.mark.parametrize("ptk", [1, 511, 512, 513, 700, 3999, 4000, 5000])
def test_shortlist_cut_edges(ptk):
    """The shortlist's cut among equal scores (every key of the boundary bin differs in
    its id alone), in the middle of distinct ones, and at the candidate count."""
    rng = np.random.default_rng(1)
    cen = unit(rng.standard_normal((40, 128)))
    code = np.concatenate([np.zeros(3000, np.uint32), rng.integers(1, 40, 1000).astype(np.uint32)])
    lens = np.ones(4000, np.uint32)
    off, size, ids = pyoracle.ivf_build(code, lens, 40)
    ix = dict(item_n_vec=lens, centroid=cen, vq_code=code, ivf_off=off, ivf_size=size, ivf_ids=ids,
              weight=np.array([-0.05, 0.05], np.float32), n_bit=1,
              residual=rng.integers(0, 256, 4000 * 16).astype(np.uint8))
    q = unit(cen[0] + 0.3 * rng.standard_normal((3, 128)))
    r = oracle_of(ix).search_one(q, 1, 32, ptk)
    with gpu_index(ix) as g:
        t = g.trace(q, 1, 32, ptk)
    o = np.argsort(r["short_id"])
    np.testing.assert_array_equal(t["cand_id"], r["cand_id"])
    np.testing.assert_array_equal(t["short_id"], r["short_id"][o])
    np.testing.assert_array_equal(t["short_approx"], r["short_approx"][o])


@pytest.mark.parametrize("n_bit", [1, 2, 4, 8])
@pytest.mark.parametrize("sem", [SEM_PP, SEM_BASIC], ids=["pp", "basic"])
def test_exact_search_through_bf16_cut(n_bit, sem):
    """Exact FP32 searches long enough to leave docs out by their BF16 scores return the
    oracle's results: queries of several norms (large ones, and small ones whose
    error is the accumulator's), ragged widths, and corpora of duplicates that all tie."""
    rng = np.random.default_rng(n_bit)
    ix = tiny_index(n_doc=700, n_centroid=48, n_bit=n_bit, seed=60 + n_bit)
    dup = tiny_index(n_doc=300, n_centroid=16, n_bit=n_bit, seed=61, lengths=[7] * 300)
    for k in ("vq_code", "residual"):  # every doc the same tokens
        per = np.asarray(dup[k]).reshape(300, -1)
        dup[k] = np.repeat(per[:1], 300, axis=0).reshape(np.asarray(dup[k]).shape)
    dup["ivf_off"], dup["ivf_size"], dup["ivf_ids"] = pyoracle.ivf_build(
        dup["vq_code"], dup["item_n_vec"], 16)
    for x, ptk in ((ix, 400), (dup, 250)):
        o = oracle_of(x)
        q, off = make_queries(x, 140, (17, 64), seed=4)
        scale = np.repeat(10.0 ** rng.integers(-6, 5, 140), np.diff(off.astype(np.int64)))
        with gpu_index(x) as g:
            for qq in (q, (q * scale[:, None]).astype(np.float32)):
                for k in (1, 10, 60):
                    r = o.search(qq, off, k, 8, ptk, sem)
                    s, i = g.search(qq, k, 8, ptk, tok_off=off, semantics=sem)
                    np.testing.assert_array_equal(i, r[1])
                    np.testing.assert_array_equal(s, r[0])


@pytest.mark.parametrize("n_bit", [1, 2, 4, 8])
def test_bf16_rescore_cut(n_bit):
    """BF16 searches: a batch whose re-scored lists are long enough to be cut by the
    bound on the BF16 error returns what batches too small for the cut return."""
    ix = tiny_index(n_doc=900, n_centroid=48, n_bit=n_bit, seed=80 + n_bit)
    for width in ((1, 32), (20, 64)):
        q, off = make_queries(ix, 140, width, seed=5)
        scale = np.repeat(10.0 ** np.random.default_rng(n_bit).integers(-6, 5, 140),
                          np.diff(off.astype(np.int64)))
        with gpu_index(ix) as g:
            for qq in (q, (q * scale[:, None]).astype(np.float32)):
                for k, r, ptk in ((1, 300, 400), (10, 400, 400), (100, 130, 300)):
                    g.set_rescore(r)
                    for sem in (SEM_PP, SEM_BASIC):
                        g.set_batch(20)  # 20 x 400 docs: no cut
                        s0, i0 = g.search(qq, k, 8, ptk, tok_off=off, semantics=sem | PREC_BF16)
                        g.set_batch(140)  # 140 x 130 docs or more: cut
                        s1, i1 = g.search(qq, k, 8, ptk, tok_off=off, semantics=sem | PREC_BF16)
                        np.testing.assert_array_equal(i1, i0)
                        np.testing.assert_array_equal(s1, s0)


@pytest.mark.parametrize("n_bit", [1, 2, 4, 8])
@pytest.mark.parametrize("n_query,width", [(1, (32, 32)), (3, (1, 31)), (6, (30, 36)), (150, (1, 32))])
def test_bf16_maxsim_edges(n_bit, n_query, width):
    """The BF16 MaxSim at its docs per CTA, doc lengths around its 128-token tiles and
    query widths around its 32 columns: the k docs it picks have, one by one, exact
    scores within twice the BF16 error of the exact k best.  With |x| <= X = max |c| +
    sqrt(128) max |w|, rounding q, c and w to BF16 (2^-9 each) moves a dot product by at
    most 2^-8 |q| X, rounding a sum c + w by as much again; 2^-11 covers the products
    of these and the FP32 accumulation from an offset of up to 4 |q| X."""
    lengths = (LENGTHS * 20)[:300]
    ix = tiny_index(n_doc=300, n_centroid=48, n_bit=n_bit, seed=90 + n_bit, lengths=lengths)
    q, off = make_queries(ix, n_query, width, seed=6)
    X = np.linalg.norm(ix["centroid"], axis=1).max() + np.sqrt(128) * np.abs(ix["weight"]).max()
    o, k = oracle_of(ix), 20
    with gpu_index(ix) as g:
        g.set_rescore(k)  # the BF16 pass alone chooses
        for ptk in (20, 129, 300):
            want = o.search(q, off, k, 8, ptk, SEM_PP)[0]
            got, ids = g.search(q, k, 8, ptk, tok_off=off, semantics=SEM_PP | PREC_BF16)
            for b in range(n_query):
                n = np.linalg.norm(q[int(off[b]):int(off[b + 1])].astype(np.float64), axis=1).sum()
                assert len(set(ids[b])) == k
                assert (got[b] >= want[b] - 2 * n * X * (2.0**-7 + 2.0**-11)).all()
                if ptk == k:
                    np.testing.assert_array_equal(got[b], want[b])


@pytest.mark.parametrize("n_bit", [1, 2, 4, 8])
def test_exact_search_through_bf16_cut_narrow(n_bit):
    """As test_exact_search_through_bf16_cut, queries of up to 32 tokens (1 to 32 wide)."""
    ix = tiny_index(n_doc=700, n_centroid=48, n_bit=n_bit, seed=95 + n_bit, lengths=(LENGTHS * 50)[:700])
    o = oracle_of(ix)
    q, off = make_queries(ix, 140, (1, 32), seed=8)
    scale = np.repeat(10.0 ** np.random.default_rng(n_bit).integers(-6, 5, 140),
                      np.diff(off.astype(np.int64)))
    with gpu_index(ix) as g:
        for qq in (q, (q * scale[:, None]).astype(np.float32)):
            for k in (1, 10, 100):
                for sem in (SEM_PP, SEM_BASIC):
                    r = o.search(qq, off, k, 8, 400, sem)
                    s, i = g.search(qq, k, 8, 400, tok_off=off, semantics=sem)
                    np.testing.assert_array_equal(i, r[1])
                    np.testing.assert_array_equal(s, r[0])


@pytest.mark.parametrize("n_bit", [1, 2, 4, 8])
@pytest.mark.parametrize("n_query,width", [(1, (1, 1)), (1, (33, 33)), (5, (15, 18)), (16, (1, 64))])
def test_exact_rerank_small_grids(n_bit, n_query, width):
    """The exact rerank at one, two and a few docs per CTA (32- and 128-token tiles)."""
    ix = tiny_index(n_doc=300, n_centroid=48, n_bit=n_bit, seed=70 + n_bit,
                    lengths=(LENGTHS * 20)[:300])
    o = oracle_of(ix)
    q, off = make_queries(ix, n_query, width, seed=7)
    with gpu_index(ix) as g:
        for ptk in (1, 37, 74, 300):
            for sem in (SEM_PP, SEM_BASIC):
                k = min(ptk, 40)
                r = o.search(q, off, k, 8, ptk, sem)
                s, i = g.search(q, k, 8, ptk, tok_off=off, semantics=sem)
                np.testing.assert_array_equal(i, r[1])
                np.testing.assert_array_equal(s, r[0])


@pytest.mark.parametrize("n_query", [255, 256, 300, 520])
def test_host_queries_scored_in_pieces(n_query):
    """Host-buffer calls large enough to be copied and scored in pieces, whose plans take
    more splits of the centroids than the whole would: the results of small calls."""
    rng = np.random.default_rng(n_query)
    n_doc, n_tok, n_cen = 2000, 8, 8192
    code = rng.integers(0, n_cen, n_doc * n_tok).astype(np.uint32)
    lengths = np.full(n_doc, n_tok, np.uint32)
    ivf_off, ivf_size, ivf_ids = pyoracle.ivf_build(code, lengths, n_cen)
    cen = unit(rng.standard_normal((n_cen, 128)))
    q = unit(rng.standard_normal((n_query * 32, 128))).reshape(n_query, 32, 128)
    with Index.from_arrays(lengths, cen, code, ivf_off, ivf_size, ivf_ids,
                           np.array([-0.1, -0.03, 0.03, 0.1], np.float32), 2,
                           rng.integers(0, 256, n_doc * n_tok * 32).astype(np.uint8)) as g:
        s, i = g.search(q, 10, 4, 100)  # the first call sizes the workspace
        for b in range(0, n_query, 100):
            s1, i1 = g.search(q[b:b + 100], 10, 4, 100)
            np.testing.assert_array_equal(i[b:b + 100], i1)
            np.testing.assert_array_equal(s[b:b + 100], s1)


def buckets(ix):
    """[n_vec, 128] bucket of every residual value."""
    b = ix["n_bit"]
    r = np.asarray(ix["residual"]).reshape(-1, 128 * b // 8, 1)
    return ((r >> (8 - b * (np.arange(8 // b) + 1))) & ((1 << b) - 1)).reshape(-1, 128)


def with_buckets(ix, bk, weight):
    b = ix["n_bit"]
    v = bk.reshape(-1, 128 * b // 8, 8 // b) << (8 - b * (np.arange(8 // b) + 1))
    return dict(ix, residual=v.sum(2).astype(np.uint8).reshape(np.asarray(ix["residual"]).shape),
                weight=np.asarray(weight, np.float32))


@pytest.mark.parametrize("n_bit", [1, 2, 4, 8])
@pytest.mark.parametrize("width", [(17, 32), (20, 64)], ids=["narrow", "wide"])
@pytest.mark.parametrize("large", [1e2, 1e4, 1e6])
def test_bf16_cut_with_an_unused_large_weight(n_bit, width, large):
    """A bucket weight far above the others that no token uses: FP32 searches cut by their
    BF16 scores, and BF16 searches whose re-scored docs are cut, return the oracle's
    results (the scores' offset has to follow the tokens, as the cut's bound does)."""
    ix = tiny_index(n_doc=700, n_centroid=48, n_bit=n_bit, seed=110 + n_bit)
    last = (1 << n_bit) - 1
    bk = buckets(ix)
    ix = with_buckets(ix, np.where(bk == last, last - 1, bk), np.append(ix["weight"][:-1], large))
    o = oracle_of(ix)
    q, off = make_queries(ix, 140, width, seed=9)
    with gpu_index(ix) as g:
        g.set_rescore(400)
        for k in (1, 10, 60):
            r = o.search(q, off, k, 8, 400, SEM_PP)
            for prec in (0, PREC_BF16):
                s, i = g.search(q, k, 8, 400, tok_off=off, semantics=SEM_PP | prec)
                np.testing.assert_array_equal(i, r[1])
                np.testing.assert_array_equal(s, r[0])


@pytest.mark.parametrize("n_bit", [4, 8])
@pytest.mark.parametrize("kind", ["weight", "centroid"])
@pytest.mark.parametrize("large", [30.0, 1e3, 1e5])
def test_bf16_scores_beside_a_large_token(n_bit, kind, large):
    """BF16 scores of ordinary docs where one doc holds a token many times their norm:
    within the rounding of their own values.  Rounding q, c, w and a sum c + w to BF16
    moves a dot product by at most 2^-9 |q| (|x| + |c| + |w| + |x|), and the FP32
    accumulation by 2^-13 |q| |x|: less than 2^-7 |q| (|c| + |w|) together."""
    ix = tiny_index(n_doc=300, n_centroid=48, n_bit=n_bit, seed=120 + n_bit)
    tok0 = np.concatenate([[0], np.cumsum(ix["item_n_vec"].astype(np.int64))])
    bk, cen, weight = buckets(ix), ix["centroid"].copy(), ix["weight"].copy()
    if kind == "weight":  # a bucket that one value of doc 0 alone uses
        last = (1 << n_bit) - 1
        bk = np.where(bk == last, last - 1, bk)
        bk[0, 5], weight[last] = last, large
        ix = with_buckets(ix, bk, weight)
    else:                 # a centroid that doc 0's first token alone has
        cen = np.concatenate([cen, cen[:1] * np.float32(large)])
        code = np.asarray(ix["vq_code"]).copy()
        code[0] = 48
        off, size, ids = pyoracle.ivf_build(code, ix["item_n_vec"], 49)
        ix = dict(ix, centroid=cen, vq_code=code, ivf_off=off, ivf_size=size, ivf_ids=ids)
    c = cen[ix["vq_code"]].astype(np.float64)
    w = ix["weight"].astype(np.float64)[bk]
    norm = np.linalg.norm(c, axis=1) + np.linalg.norm(w, axis=1)
    with gpu_index(ix) as g:
        for nq in (20, 32):
            q, _ = make_queries(ix, 1, nq, seed=nq)
            t = g.trace(q, 10, 8, 250, SEM_PP | PREC_BF16)
            q = q.astype(np.float64)
            dots = q @ (c + w).T
            for d, got in zip(t["short_id"], t["short_exact"]):
                s = slice(tok0[d], tok0[d + 1])
                tol = np.linalg.norm(q, axis=1).sum() * norm[s].max() * 2.0**-7
                assert abs(got - dots[:, s].max(1).sum()) <= tol


@pytest.mark.parametrize("n_query", [410, 700, 1184])
def test_probe_lists_at_their_memory_limit(n_query):
    """Probe launches whose lists the memory limit leaves fewer splits or makes smaller
    (32 probes of 16,384 centroids): the results of small calls."""
    rng = np.random.default_rng(n_query)
    n_doc, n_tok, n_cen = 2000, 8, 16384
    code = rng.integers(0, n_cen, n_doc * n_tok).astype(np.uint32)
    lengths = np.full(n_doc, n_tok, np.uint32)
    ivf_off, ivf_size, ivf_ids = pyoracle.ivf_build(code, lengths, n_cen)
    q = unit(rng.standard_normal((n_query * 32, 128))).reshape(n_query, 32, 128)
    with Index.from_arrays(lengths, unit(rng.standard_normal((n_cen, 128))), code, ivf_off, ivf_size,
                           ivf_ids, np.array([-0.1, -0.03, 0.03, 0.1], np.float32), 2,
                           rng.integers(0, 256, n_doc * n_tok * 32).astype(np.uint8)) as g:
        d = torch.from_numpy(q).cuda()  # (host queries would be scored in smaller pieces)
        ds = torch.empty((n_query, 10), device="cuda")
        di = torch.empty((n_query, 10), dtype=torch.int32, device="cuda")
        g.search_device(d.data_ptr(), None, n_query, 32, 10, 32, 100, ds.data_ptr(), di.data_ptr())
        s, i = ds.cpu().numpy(), di.cpu().numpy().view(np.uint32)
        for b in range(0, n_query, 100):
            s1, i1 = g.search(q[b:b + 100], 10, 32, 100)
            np.testing.assert_array_equal(i[b:b + 100], i1)
            np.testing.assert_array_equal(s[b:b + 100], s1)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_exhaustive_of_nothing(dtype):
    """No queries, queries without tokens, docs that are all empty, no docs: the results
    of the torch form on the CPU."""
    g = torch.Generator().manual_seed(4)
    doc, q = (torch.randn((n, 128), generator=g, dtype=dtype) for n in (40, 6))
    none = doc[:0]
    pieces = [(0, [0, 0, 0], none), (3, [7, 0, 33], doc), (6, [], none), (6, [0], none)]
    for qq, off in ((q, [0, 2, 2, 6]), (none, [0]), (none, [0, 0, 0])):
        want = exhaustive.exhaustive_topk_stream(qq, off, pieces, 5, dtype)
        got = exhaustive.exhaustive_topk_stream(qq.cuda(), off, [(d, n, x.cuda()) for d, n, x in pieces], 5, dtype)
        np.testing.assert_array_equal(got[1], want[1])
        # 6 terms of size ~30, products summed in another order: 128 * 6 ulps of 64
        np.testing.assert_allclose(got[0], want[0], rtol=0, atol=128 * 6 * 64 * torch.finfo(dtype).eps)


def test_exhaustive_of_a_padded_piece():
    """Tokens behind the last doc's count for no doc, on the GPU as on the CPU."""
    g = torch.Generator(device="cuda").manual_seed(6)
    s = torch.randn((70, 301), device="cuda", generator=g, dtype=torch.float64)
    q_off, lens = torch.tensor([0, 33, 70]), np.array([40, 0, 200])
    got = exhaustive._maxsum(s, q_off.cuda(), lens)
    want = exhaustive._maxsum(s[:, :240].cpu(), q_off, lens)
    # up to 37 terms of size ~4 in another order: 37 ulps of 256
    torch.testing.assert_close(got.cpu(), want, rtol=0, atol=37 * 256 * torch.finfo(s.dtype).eps)


@pytest.mark.parametrize("n_query", [15, 520])
def test_stage_times_of_one_batch(n_query):
    """Timed host calls of one batch: the query copy is stage 0 (it cannot be faster than
    the bus), the stages add up to the device time, and a query's time is its batch's.  Without stage
    times the larger call is copied in four pieces: stage 0 is the first."""
    rng = np.random.default_rng(n_query)
    n_doc, n_tok, n_cen = 2000, 8, 1024
    code = rng.integers(0, n_cen, n_doc * n_tok).astype(np.uint32)
    lengths = np.full(n_doc, n_tok, np.uint32)
    ivf_off, ivf_size, ivf_ids = pyoracle.ivf_build(code, lengths, n_cen)
    q = unit(rng.standard_normal((n_query * 32, 128))).reshape(n_query, 32, 128)
    least = q.nbytes / 64e9  # 64 GB/s: what PCIe 5 x16 carries at most
    with Index.from_arrays(lengths, unit(rng.standard_normal((n_cen, 128))), code, ivf_off, ivf_size,
                           ivf_ids, np.array([-0.1, -0.03, 0.03, 0.1], np.float32), 2,
                           rng.integers(0, 256, n_doc * n_tok * 32).astype(np.uint8)) as g:
        s0, i0 = g.search(q, 10, 4, 100)
        for _ in range(3):
            s, i, st = g.search(q, 10, 4, 100, with_stats=True, with_stages=True)
            stages = st["stage_time_s"]
            np.testing.assert_array_equal(i, i0)
            np.testing.assert_array_equal(s, s0)
            assert st["n_batch"] == 1 and (stages[:, 0] >= least).all()
            np.testing.assert_allclose(stages.sum(1), st["query_time_s"], rtol=0, atol=50e-6)
            np.testing.assert_allclose(st["query_time_s"], st["device_ms"] * 1e-3, rtol=0, atol=50e-6)
            _, _, st = g.search(q, 10, 4, 100, with_stats=True)
            assert st["stage_ms"][0] * 1e-3 >= (least if n_query == 15 else least / 4)
            assert abs(sum(st["stage_ms"]) - st["device_ms"]) <= 0.05


def test_assign_beside_pending_work():
    """assign on a side stream while the current one still has to read a freed block as
    large as assign's workspace: the block keeps its values, the codes are the oracle's."""
    import ctypes as C

    from mvr._lib import check, lib
    rng = np.random.default_rng(9)
    x, cen = unit(rng.standard_normal((5000, 128))), unit(rng.standard_normal((1000, 128)))
    dx, dc = torch.from_numpy(x).cuda(), torch.from_numpy(cen).cuda()
    n = C.c_size_t()
    check(lib().mvr_assign_work_bytes(5000, 1000, C.byref(n)))
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    block = torch.full((n.value,), 171, dtype=torch.uint8, device="cuda")
    torch.cuda._sleep(500_000_000)  # some 0.3 s
    kept = block.clone()
    del block
    code, _ = build.assign(dx, dc, stream=side)
    np.testing.assert_array_equal(code.cpu().numpy(), pyoracle.assign(x, cen).astype(np.int64))
    assert bool((kept == 171).all())


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_assign_centroids_at_any_offset(shift):
    """Centroids that start at any 4-byte offset (rows of a larger buffer)."""
    rng = np.random.default_rng(shift)
    x, cen = unit(rng.standard_normal((700, 128))), unit(rng.standard_normal((300, 128)))
    buf = torch.zeros(300 * 128 + shift, device="cuda")
    buf[shift:] = torch.from_numpy(cen.reshape(-1)).cuda()
    code, score = build.assign(torch.from_numpy(x).cuda(), buf[shift:].view(300, 128))
    same, s = build.assign(torch.from_numpy(x).cuda(), torch.from_numpy(cen).cuda())
    np.testing.assert_array_equal(code.cpu().numpy(), pyoracle.assign(x, cen).astype(np.int64))
    assert torch.equal(code, same) and torch.equal(score, s)


@pytest.mark.parametrize("n_bit", [1, 2, 4, 8])
@pytest.mark.parametrize("sem", [SEM_PP, SEM_BASIC], ids=["pp", "basic"])
def test_bf16_cut_of_equal_docs(n_bit, sem):
    """Queries of 17 to 32 tokens, which are cut at every code width: a corpus of docs that
    all tie, and one of distinct docs; by the launches, the cut did run."""
    ix = tiny_index(n_doc=300, n_centroid=16, n_bit=n_bit, seed=130 + n_bit, lengths=[7] * 300)
    dup = dict(ix)
    for k in ("vq_code", "residual"):
        per = np.asarray(ix[k]).reshape(300, -1)
        dup[k] = np.repeat(per[:1], 300, axis=0).reshape(np.asarray(ix[k]).shape)
    dup["ivf_off"], dup["ivf_size"], dup["ivf_ids"] = pyoracle.ivf_build(
        dup["vq_code"], dup["item_n_vec"], 16)
    q, off = make_queries(ix, 140, (17, 32), seed=4)
    for x in (ix, dup):
        o = oracle_of(x)
        with gpu_index(x) as g:
            for k in (1, 60):
                r = o.search(q, off, k, 8, 250, sem)
                s, i, cut = g.search(q, k, 8, 250, tok_off=off, semantics=sem, with_stats=True)
                np.testing.assert_array_equal(i, r[1])
                np.testing.assert_array_equal(s, r[0])
                *_, plain = g.search(q, k, 8, 230, tok_off=off, semantics=sem, with_stats=True)
                # 140 x 250 docs are cut, 140 x 230 are not: the BF16 MaxSim and the cut
                assert cut["gpu_launches"] == plain["gpu_launches"] + 2
