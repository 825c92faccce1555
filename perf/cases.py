"""What this framework's performance is measured on: the calls that a user's
program makes, over the range of sizes and options in which it makes them.

Three groups, by use:
  search     one query for a waiting client, a handful of queries, whole
             evaluation sets; the reference's two methods (true doc lengths and
             padded docs) in FP32, and the FP8 and BF16 paths; every residual
             code width; uniform and ragged queries; host and device buffers;
  build      the index builder's training (k-means, cutoffs, weights) and its
             encoding of a chunk of tokens;
  read back  decoded tokens of an index, and the exhaustive MaxSim that recall
             is measured against.

Indexes are drawn, not trained, so that preparing one takes a second: a corpus
of docs that each mix 5 to 15 of up to 20,000 latent means (lognormal lengths,
mean 70), 1 to 13 centroids beside each mean as k-means leaves them, a token's
centroid one of its mean's, and uniform residual buckets, which is what
quantile cutoffs give.  Query tokens are noisy copies of a random doc's means.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("multi-vector-retrieval-gpu_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from mvr import PREC_BF16, PREC_FP8, SEM_BASIC, Index, build, exhaustive  # noqa: E402

DIM = 128
_PREC = {"fp32": 0, "fp8": PREC_FP8, "bf16": PREC_BF16}


def _search(name, n_doc, n_centroid, n_bit, n_query, tok_lo, tok_hi, nprobe, probe_topk, k,
            precision, io, basic=False, graphs=False, len_hi=180):
    return dict(name=name, kind="search", n_doc=n_doc, n_centroid=n_centroid, n_bit=n_bit,
                n_query=n_query, tok_lo=tok_lo, tok_hi=tok_hi, nprobe=nprobe,
                probe_topk=probe_topk, k=k, precision=precision, io=io, basic=basic,
                graphs=graphs, len_hi=len_hi)


def listed():
    return [
        # one query at a time on a small corpus, host buffers, the reference's FP32 method:
        # its own command-line search, and any interactive use
        _search("one_fp32_small", 10_000, 8192, 2, 1, 32, 32, 4, 200, 10, "fp32", "host"),
        # one query of a serving process on a 1M-doc index: device buffers, FP8, the call
        # recorded as a graph
        _search("one_fp8_1m", 1_000_000, 65_536, 2, 1, 32, 32, 8, 1500, 10, "fp8", "device",
                graphs=True),
        # a handful of queries of different lengths that arrived together (37 users of one server)
        _search("few_ragged_fp8", 250_000, 32_768, 2, 37, 8, 32, 8, 1000, 10, "fp8", "host"),
        # bulk search of a 1M-doc index, the FP8 path: two full device batches
        _search("bulk_fp8_1m", 1_000_000, 65_536, 2, 2368, 32, 32, 8, 1500, 10, "fp8", "device"),
        # an evaluation set through the reference's FP32 method on the same index
        _search("bulk_fp32_1m", 1_000_000, 65_536, 2, 400, 32, 32, 8, 1500, 10, "fp32", "host"),
        # long docs, 4-bit codes, queries of up to 64 tokens
        _search("long_fp8_b4", 300_000, 65_536, 4, 600, 33, 64, 8, 1500, 10, "fp8", "host",
                len_hi=300),
        # the reference's wide setting (16 lists, 1400 docs, 100 results), BF16, 1-bit codes
        _search("wide_bf16_b1", 200_003, 16_384, 1, 500, 32, 32, 16, 1400, 100, "bf16", "device"),
        # the reference's padded method on 8-bit codes, 100 results
        _search("basic_fp32_b8", 50_000, 16_384, 8, 200, 20, 32, 4, 400, 100, "fp32", "host",
                basic=True),
        # the builder's training: k-means over a sample, then cutoffs and bucket weights
        dict(name="train", kind="train", n_vec=300_007, n_centroid=8192, n_bit=2, n_iter=4),
        # the builder's encoding of one chunk of a large corpus
        dict(name="encode", kind="encode", n_vec=1_000_003, n_centroid=65_536, n_bit=2,
             assign="tc"),
        # decoded tokens of an index, for a program that scores docs itself
        dict(name="decode", kind="decode", n_doc=100_000, n_centroid=16_384, n_bit=2,
             n_ids=40_009),
        # the exhaustive ground truth that recall is measured against
        dict(name="exhaustive", kind="exhaustive", n_doc=20_001, n_query=64, n_tok=32, k=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: two of three are searches."""
    kind = rng.choice(["search"] * 8 + ["train", "encode", "decode", "exhaustive"])
    n_bit = rng.choice([1, 2, 2, 2, 4, 4, 8])
    if kind == "search":
        precision = rng.choice(["fp32", "fp8", "fp8", "bf16"])
        n_doc = _log_int(rng, 8_000, 1_000_000)
        # 16 sqrt(tokens) rounded down to a power of two, the reference's rule, or half of it
        n_centroid = build.n_centroid_default(70 * n_doc) >> rng.choice([0, 0, 1])
        n_centroid = min(65_536, n_centroid) + rng.choice([0, 0, 17])
        k = rng.choice([1, 10, 10, 100])
        lo = rng.choice([4, 8, 32, 32, 64])
        hi = rng.choice([x for x in (lo, 32, 64) if x >= lo])
        # fewer queries where a query costs more (FP32, long queries)
        most = (1200 if precision != "fp32" else 300) * 32 // hi
        return dict(kind="search", n_doc=n_doc, n_centroid=n_centroid, n_bit=n_bit,
                    n_query=_log_int(rng, 1, most), tok_lo=lo, tok_hi=hi,
                    nprobe=rng.choice([2, 4, 8, 8, 16]),
                    probe_topk=max(k, _log_int(rng, 100, 2000)), k=k, precision=precision,
                    io=rng.choice(["host", "device"]), basic=rng.random() < 0.2,
                    graphs=rng.random() < 0.2, len_hi=rng.choice([180, 180, 300]))
    if kind == "train":
        n = _log_int(rng, 20_000, 300_000)
        return dict(kind=kind, n_vec=n, n_centroid=_log_int(rng, 256, min(8192, n // 16)),
                    n_bit=rng.choice([2, 2, 4]), n_iter=rng.choice([1, 2, 4]))
    if kind == "encode":
        assign = rng.choice(["tc", "fp32"])
        return dict(kind=kind, n_vec=_log_int(rng, 5_000, 1_000_000 if assign == "tc" else 200_000),
                    n_centroid=_log_int(rng, 1000, 65_536 if assign == "tc" else 16_384),
                    n_bit=n_bit, assign=assign)
    if kind == "decode":
        return dict(kind=kind, n_doc=_log_int(rng, 5_000, 100_000), n_centroid=16_384,
                    n_bit=n_bit, n_ids=_log_int(rng, 1, 100_000))
    return dict(kind=kind, n_doc=_log_int(rng, 1_000, 20_000), n_query=_log_int(rng, 1, 64),
                n_tok=rng.choice([8, 32]), k=rng.choice([1, 10, 100]))


# ---------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _unit(x):
    return torch.nn.functional.normalize(x, dim=1)


def _randn(g, *shape):
    return torch.randn(shape, device="cuda", generator=g)


def _rand(g, *shape):
    return torch.rand(shape, device="cuda", generator=g)


def _weights(n_bit):
    """Bucket weights: the mid quantiles of a token's distance from its centroid, per dimension."""
    p = (torch.arange(1 << n_bit, dtype=torch.float64) + 0.5) / (1 << n_bit)
    return (torch.erfinv(2 * p - 1) * math.sqrt(2) * 0.45 / math.sqrt(DIM)).float().cuda()


def _corpus(g, n_doc, n_latent, len_hi):
    """(latent means, doc lengths, clusters of each doc, how many of them, doc of each token)"""
    latent = _unit(_randn(g, n_latent, DIM))
    sigma = math.sqrt(math.log(1.25))  # mean 70, sd 35
    lens = torch.exp(math.log(70.0) - sigma * sigma / 2 + sigma * _randn(g, n_doc))
    lens = lens.round().clamp_(8, len_hi).long()
    n_mix = torch.randint(5, 16, (n_doc,), device="cuda", generator=g)
    mix = torch.randint(0, n_latent, (n_doc, 15), device="cuda", generator=g)
    doc = torch.repeat_interleave(torch.arange(n_doc, device="cuda"), lens)
    return latent, lens, mix, n_mix, doc


def _pick(g, mix, n_mix, doc):
    """A random latent of each listed doc."""
    slot = (_rand(g, doc.shape[0]) * n_mix[doc]).long().clamp_(max=14)
    return mix[doc, slot]


def _index(case, seed):
    """An index's arrays on the GPU, and what queries are drawn from."""
    g = _gen(seed)
    C, b = case["n_centroid"], case["n_bit"]
    n_latent = min(20_000, C)
    latent, lens, mix, n_mix, doc = _corpus(g, case["n_doc"], n_latent, case.get("len_hi", 180))
    cen = latent[torch.arange(C, device="cuda") % n_latent]
    cen = _unit(cen + 0.06 / math.sqrt(DIM) * _randn(g, C, DIM))
    lat = _pick(g, mix, n_mix, doc)
    copies = (C - lat + n_latent - 1) // n_latent  # centroids beside each latent mean
    code = lat + n_latent * (_rand(g, doc.shape[0]) * copies).long()
    code = torch.minimum(code, torch.tensor(C - 1, device="cuda"))
    key = torch.unique(code * case["n_doc"] + doc)  # sorted by (centroid, doc)
    size = torch.bincount(key // case["n_doc"], minlength=C)
    off = torch.cumsum(size, 0) - size
    residual = torch.randint(0, 256, (doc.shape[0] * DIM * b // 8,), device="cuda", generator=g,
                             dtype=torch.uint8)
    arrays = dict(item_n_vec=lens.int(), centroid=cen.contiguous(), vq_code=code.int(),
                  ivf_off=off, ivf_size=size.int(), ivf_ids=(key % case["n_doc"]).int(),
                  weight=_weights(b), n_bit=b, residual=residual)
    return arrays, (g, latent, mix, n_mix)


def _queries(case, g, latent, mix, n_mix):
    n = case["n_query"]
    count = torch.randint(case["tok_lo"], case["tok_hi"] + 1, (n,), device="cuda", generator=g)
    doc = torch.randint(0, case["n_doc"], (n,), device="cuda", generator=g)
    lat = _pick(g, mix, n_mix, torch.repeat_interleave(doc, count))
    q = _unit(latent[lat] + 0.55 / math.sqrt(DIM) * _randn(g, lat.shape[0], DIM))
    off = np.zeros(n + 1, np.uint64)
    off[1:] = np.cumsum(count.cpu().numpy())
    return q.contiguous(), off


def _tokens(g, n_vec, latent):
    """Raw token vectors around latent means (every mean equally often)."""
    lat = torch.randint(0, latent.shape[0], (n_vec,), device="cuda", generator=g)
    return _unit(latent[lat] + 0.45 / math.sqrt(DIM) * _randn(g, n_vec, DIM)).contiguous()


def _inputs(case, seed):
    """The case's inputs, the same for `prepare` and `exact`."""
    kind = case["kind"]
    if kind == "search":
        arrays, rest = _index(case, seed)
        q, off = _queries(case, *rest)
        return dict(arrays=arrays, q=q, off=off)
    if kind == "decode":
        arrays, (g, *_) = _index(case, seed)
        ids = torch.randint(0, arrays["vq_code"].shape[0], (case["n_ids"],), device="cuda",
                            generator=g)
        return dict(arrays=arrays, ids=ids.cpu().numpy().astype(np.uint64))
    g = _gen(seed)
    if kind == "exhaustive":
        latent, lens, mix, n_mix, doc = _corpus(g, case["n_doc"], 2000, 180)
        lat = _pick(g, mix, n_mix, doc)
        tok = _unit(latent[lat] + 0.45 / math.sqrt(DIM) * _randn(g, lat.shape[0], DIM))
        q, off = _queries(dict(case, tok_lo=case["n_tok"], tok_hi=case["n_tok"]), g, latent, mix,
                          n_mix)
        return dict(q=q, off=off, tok=tok.contiguous(),
                    lens=lens.cpu().numpy().astype(np.uint32))
    latent = _unit(_randn(g, max(64, min(20_000, case["n_centroid"] // 3)), DIM))
    tok = _tokens(g, case["n_vec"], latent)
    if kind == "train":
        return dict(tok=tok)
    cen = latent[torch.arange(case["n_centroid"], device="cuda") % latent.shape[0]]
    cen = _unit(cen + 0.06 / math.sqrt(DIM) * _randn(g, case["n_centroid"], DIM)).contiguous()
    p = torch.arange(1, 1 << case["n_bit"], dtype=torch.float64) / (1 << case["n_bit"])
    cutoff = (torch.erfinv(2 * p - 1) * math.sqrt(2) * 0.45 / math.sqrt(DIM)).float().numpy()
    return dict(tok=tok, cen=cen, cutoff=cutoff)


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    if kind in ("search", "decode"):
        a = s.pop("arrays")
        s["index"] = Index.from_device_arrays(a["item_n_vec"], a["centroid"], a["vq_code"],
                                              a["ivf_off"], a["ivf_size"], a["ivf_ids"],
                                              a["weight"], a["n_bit"], a["residual"])
    if kind == "search":
        s["flags"] = _PREC[case["precision"]] | (SEM_BASIC if case["basic"] else 0)
        if case["graphs"]:
            s["index"].set_graphs(True)
        if case["tok_lo"] == case["tok_hi"]:
            s["off"] = None  # the uniform layout [n_query, n_tok, 128]
        if case["io"] == "host":
            q = s["q"].cpu().numpy()
            s["q"] = q.reshape(case["n_query"], -1, DIM) if s["off"] is None else q
        else:
            s["scores"] = torch.empty((case["n_query"], case["k"]), device="cuda")
            s["ids"] = torch.empty((case["n_query"], case["k"]), dtype=torch.int32, device="cuda")
    elif kind == "encode":
        s["code"] = torch.empty(case["n_vec"], dtype=torch.int32, device="cuda")
        s["residual"] = torch.empty(case["n_vec"] * DIM * case["n_bit"] // 8, dtype=torch.uint8,
                                    device="cuda")
    torch.cuda.synchronize()
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "search":
        if c["io"] == "host":
            return s["index"].search(s["q"], c["k"], c["nprobe"], c["probe_topk"],
                                     tok_off=s["off"], semantics=s["flags"])
        s["index"].search_device(s["q"].data_ptr(), s["off"], c["n_query"],
                                 c["tok_hi"] if s["off"] is None else 0, c["k"], c["nprobe"],
                                 c["probe_topk"], s["scores"].data_ptr(), s["ids"].data_ptr(),
                                 stream_ptr=torch.cuda.current_stream().cuda_stream,
                                 semantics=s["flags"])
        return s["scores"], s["ids"]
    if kind == "train":
        return build.train(s["tok"], c["n_centroid"], c["n_bit"], kmeans_iter=c["n_iter"])
    if kind == "encode":
        build.encode(s["tok"], s["cen"], s["cutoff"], c["n_bit"], s["code"], s["residual"],
                     assign_fn=build.assign_tc if c["assign"] == "tc" else build.assign)
        return s["code"], s["residual"]
    if kind == "decode":
        return s["index"].decompress(s["ids"])
    return exhaustive.exhaustive_topk(s["q"], s["off"], s["tok"], s["lens"], c["k"])


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind == "search":
        nq, C, b = (case["tok_lo"] + case["tok_hi"]) / 2, case["n_centroid"], case["n_bit"]
        q_tok = nq * case["n_query"]
        n_vec = 70.0 * case["n_doc"]
        short = min(case["probe_topk"], case["n_doc"]) * 70.0 * case["n_query"]
        # a list holds each doc of its centroid once: about half of its tokens are other docs'
        probed = min(q_tok * case["nprobe"], C) * (0.5 * n_vec / C)
        read = q_tok * 512 + C * 512 + 4 * probed + min(short, n_vec) * (4 + 16 * b)
        return {"bytes": int(read + 8 * case["n_query"] * case["k"]),
                "flops": int(2 * DIM * (q_tok * C + nq * short))}
    if kind == "train":
        n, C = case["n_vec"], case["n_centroid"]
        return {"bytes": int((case["n_iter"] + 2) * n * 512 + C * 512),
                "flops": int((case["n_iter"] + 1) * 2.0 * DIM * n * C)}
    if kind == "encode":
        n, C = case["n_vec"], case["n_centroid"]
        return {"bytes": int(n * (512 + 4 + 16 * case["n_bit"]) + C * 512),
                "flops": int(2.0 * DIM * n * C)}
    if kind == "decode":
        n = case["n_ids"]
        return {"bytes": int(n * (8 + 4 + 16 * case["n_bit"] + 512)), "flops": int(n * DIM)}
    tok = 70.0 * case["n_doc"]
    q_tok = case["n_query"] * case["n_tok"]
    return {"bytes": int(512 * (tok + q_tok) + 16 * case["n_query"] * case["k"]),
            "flops": int(2 * DIM * tok * q_tok)}


# ---------------------------------------------------------------- the same in 64 bits

def _decoded(a, tok):
    """Decoded vectors of the listed tokens, float64."""
    b = a["n_bit"]
    vpb = 8 // b
    byte = a["residual"].view(-1, DIM * b // 8)[tok].long().unsqueeze(-1)
    shift = torch.arange(vpb - 1, -1, -1, device="cuda") * b
    bucket = ((byte >> shift) & ((1 << b) - 1)).reshape(len(tok), DIM)
    return a["centroid"][a["vq_code"][tok].long()].double() + a["weight"].double()[bucket]


def _ranges(start, count):
    """start[0] .. start[0] + count[0] - 1, start[1] .., and the row of each."""
    row = torch.repeat_interleave(torch.arange(len(count), device="cuda"), count)
    first = torch.cumsum(count, 0) - count
    return start[row] + torch.arange(len(row), device="cuda") - first[row], row


def _exact_search(case, s):
    a, k = s["arrays"], case["k"]
    cen = a["centroid"].double()
    lens = a["item_n_vec"].long()
    first = torch.cumsum(lens, 0) - lens
    out = torch.full((case["n_query"], k), -math.inf, dtype=torch.float64, device="cuda")
    for i in range(case["n_query"]):
        q = s["q"][int(s["off"][i]):int(s["off"][i + 1])].double()
        probe_s, probe = torch.topk(q @ cen.T + 1.0, case["nprobe"], dim=1)
        at, row = _ranges(a["ivf_off"][probe.flatten()], a["ivf_size"].long()[probe.flatten()])
        doc, inv = torch.unique(a["ivf_ids"][at].long(), return_inverse=True)
        best = torch.full((len(doc) * len(q),), -math.inf, dtype=torch.float64, device="cuda")
        best.scatter_reduce_(0, inv * len(q) + row // case["nprobe"], probe_s.flatten()[row],
                             reduce="amax")
        best = torch.where(torch.isfinite(best), best, 0.0).view(len(doc), len(q)).sum(1)
        # (score descending, doc ascending)
        doc = doc[torch.sort(best, descending=True, stable=True).indices[:case["probe_topk"]]]
        tok, which = _ranges(first[doc], lens[doc])
        dot = q @ _decoded(a, tok).T
        m = torch.full((len(q), len(doc)), -math.inf, dtype=torch.float64, device="cuda")
        m.scatter_reduce_(1, which.expand(len(q), -1), dot, reduce="amax")
        if case["basic"]:  # docs shorter than the longest are padded with zero vectors
            m = torch.where(lens[doc] < lens.max(), m.clamp(min=0.0), m)
        top = torch.sort(m.sum(0), descending=True).values[:k]
        out[i, :len(top)] = top
    return out


def _exact_train(case, s):
    x = s["tok"].double()
    g = torch.Generator(device="cuda").manual_seed(123)
    cen = _unit(s["tok"][torch.randperm(len(x), device="cuda", generator=g)[:case["n_centroid"]]]
                .double())

    def assign():
        return torch.cat([(x[i:i + 65_536] @ cen.T).argmax(1) for i in range(0, len(x), 65_536)])
    for _ in range(case["n_iter"]):
        code = assign()
        total = torch.zeros_like(cen).index_add_(0, code, x)
        count = torch.bincount(code, minlength=len(cen))
        nz = count > 0
        cen[nz] = _unit(total[nz] / count[nz].unsqueeze(1))
    err = torch.sort((x - cen[assign()]).flatten()).values
    n, nb = err.numel(), 1 << case["n_bit"]
    cut = [float(err[int((i + 1) / nb * n)]) for i in range(nb - 1)]
    w = [float(err[int((i / nb + 0.5 / nb) * n)]) for i in range(nb)]
    return cen, np.asarray(cut), np.asarray(w)


def exact(case, seed):
    kind = case["kind"]
    if kind == "encode":
        return None  # codes and bytes
    if kind == "search":
        # about 2 ms and 4 GB/s of float64 work a query: left out where it adds up
        tok = case["n_query"] * (case["tok_lo"] + case["tok_hi"]) / 2
        if case["n_query"] > 600 or tok * case["n_centroid"] > 2.0e9:
            return None
        return _exact_search(case, _inputs(case, seed)), None
    s = _inputs(case, seed)
    if kind == "train":
        return _exact_train(case, s)
    if kind == "decode":
        return _decoded(s["arrays"], torch.from_numpy(s["ids"].astype(np.int64)).cuda())
    q, tok = s["q"].double(), s["tok"].double()
    lens = torch.from_numpy(s["lens"].astype(np.int64)).cuda()
    doc = torch.repeat_interleave(torch.arange(len(lens), device="cuda"), lens)
    per_q = []
    for i in range(case["n_query"]):
        dot = q[int(s["off"][i]):int(s["off"][i + 1])] @ tok.T
        m = torch.full((len(dot), len(lens)), -math.inf, dtype=torch.float64, device="cuda")
        m.scatter_reduce_(1, doc.expand(len(dot), -1), dot, reduce="amax")
        per_q.append(m.sum(0))
    return torch.sort(torch.stack(per_q), dim=1, descending=True).values[:, :case["k"]], None
