"""The work that users of this framework have it do, as measurable cases.

Each case goes through the package's public binding: read and database encoding, the two exact top-k searches, the
batching pipeline, the prototype descent and the reference's own identify descent.  Sequences are made on the GPU from
the seed alone: a taxonomy of 16S-like leaves (1,400-1,600 bp, branching ceil(n^(1/6)), the substitution rates of the
package's generator per rank) and reads sampled from its leaves with substitution errors and a few N.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.join(os.getcwd(), "bacterial-classification_gb300"))

import hdc_gb300 as H  # noqa: E402

MAX_BP = 1600
RANK_SUBST = (0.04, 0.03, 0.02, 0.015, 0.01, 0.005)
MIXED_SIGMA = 0.5  # reads of uneven length: log-normal, clipped to 100-1600 bp, 20 % of them with 6 % errors
EXACT_MACS = 4e12  # beyond this a 64-bit brute force takes too long


def listed():
    return [
        # one sample's first reads sent to a service: eight reads encoded to counts, the reference's own D and k
        dict(name="encode_few", kind="encode", n=8, bp=125, mixed=False, dim=10000, kmer=5, out="i16"),
        # a full batch of uneven reads on its way to the tensor-core search
        dict(name="encode_reads", kind="encode", n=38912, bp=250, mixed=True, dim=10240, kmer=10, out="bipolar_f16"),
        # building part of a reference database: noisy copies encoded, bundled to references, their norms
        dict(name="build_refs", kind="build", refs=2500, copies=8, dim=10240, kmer=10),
        # the drop-in's argmax for a handful of reads against a small database, the reference's own D and k
        dict(name="plain_few", kind="plain", nq=48, refs=2000, bp=125, dim=10000, kmer=5, k=1, mode="cos"),
        # the workload that the reference can run on a CPU: 10,000 reads against 2,000 leaves
        dict(name="plain_reads", kind="plain", nq=10000, refs=2000, bp=150, dim=8192, kmer=8, k=5, mode="norm"),
        # the drop-in search at the size of a real leaf database
        dict(name="plain_leaves", kind="plain", nq=9001, refs=50000, bp=150, dim=8192, kmer=8, k=5, mode="norm"),
        # an interactive request against the full bundled database: 33 reads, 200,000 references
        dict(name="tc_few", kind="tc", nq=33, refs=200000, copies=8, counts=False, bp=250, dim=10240, kmer=10, k=5,
             mode="norm"),
        # the headline batch: 38,912 reads against 200,000 bundled references
        dict(name="tc_batch", kind="tc", nq=38912, refs=200000, copies=8, counts=False, bp=250, dim=10240, kmer=10,
             k=5, mode="norm"),
        # count-valued reads on the tensor cores, as the drop-in scores them
        dict(name="tc_counts", kind="tc", nq=10000, refs=50000, copies=1, counts=True, bp=150, dim=8192, kmer=8, k=5,
             mode="norm"),
        # a stream of host batches of uneven reads through the graph pipeline, top-10
        dict(name="pipeline", kind="pipeline", nq=4000, refs=50000, copies=8, bp=250, dim=10240, kmer=10, k=10),
        # reads encoded to sign bits and taken down six ranks of bundled prototypes
        dict(name="descent", kind="descent", nq=20000, leaves=100000, bp=250, dim=16384, kmer=12, beam=5),
        # the reference's identify scoring: every node by its best window, all ranks
        dict(name="identify", kind="identify", nq=4096, leaves=2000, bp=150, dim=8192, kmer=8, beam=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["encode", "encode", "build", "plain", "plain", "plain", "tc", "tc", "tc", "pipeline", "descent",
                       "identify"])
    if kind == "encode":
        dim = rng.choice([200, 1000, 1024, 2048, 4096, 8192, 10000, 10240, 16384, rng.randint(200, 16384)])
        bp = rng.choice([100, 125, 150, 250, 400, 1500])
        n = _log(rng, 1, min(40000, 38912 * 283 * 10240 // (dim * bp)))
        return dict(kind=kind, n=n, bp=bp, mixed=bp == 250 and rng.random() < 0.7, dim=dim, kmer=rng.randint(3, 14),
                    out=rng.choice(["i16", "i32", "bipolar_f16", "f16", "sign_bits"]))
    if kind == "build":
        return dict(kind=kind, refs=_log(rng, 20, 2500), copies=rng.choice([4, 8, 9]) if rng.random() < 0.5 else 8,
                    dim=rng.choice([1024, 4096, 8192, 10000, 10240]), kmer=rng.choice([5, 8, 10, 12]))
    if kind == "plain":
        dim = rng.choice([1000, 1024, 2048, 4096, 8192, 10000, 10240, rng.randint(200, 10240)])
        nr = _log(rng, 50, 50000)
        nq = _log(rng, 1, min(20000, 9001 * 50000 * 8192 // (nr * dim)))
        return dict(kind=kind, nq=nq, refs=nr, bp=rng.choice([125, 150, 250]), dim=dim, kmer=rng.choice([5, 8, 10]),
                    k=rng.choice([1, 5, 5, 10, 32]), mode=rng.choice(["norm", "norm", "cos", "dot"]))
    if kind == "tc":
        counts = rng.random() < 0.3
        dim = 8 * rng.randint(32, 1280) if rng.random() < 0.4 else rng.choice([2048, 4096, 8192, 10000, 10240])
        nr = _log(rng, 500, 200000)
        nq = _log(rng, 1, min(20000 if counts else 40000, 38912 * 200000 * 10240 // (nr * dim)))
        return dict(kind=kind, nq=nq, refs=nr, copies=1 if counts else rng.choice([1, 8, 8]), counts=counts,
                    bp=rng.choice([150, 250]), dim=dim, kmer=rng.choice([8, 10]), k=rng.choice([1, 5, 5, 10, 16]),
                    mode=rng.choice(["norm", "norm", "cos", "dot"]))
    if kind == "pipeline":
        return dict(kind=kind, nq=_log(rng, 1, 8192), refs=_log(rng, 500, 50000), copies=rng.choice([1, 8]), bp=250,
                    dim=rng.choice([2048, 8192, 10000, 10240]), kmer=rng.choice([8, 10]), k=rng.choice([1, 5, 10]))
    if kind == "descent":
        dim = rng.choice([1024, 2048, 4096, 8192, 10240, 16384])
        return dict(kind=kind, nq=_log(rng, 50, 20000), leaves=_log(rng, 500, 100000), bp=rng.choice([150, 250]),
                    dim=dim, kmer=rng.choice([8, 10, 12]), beam=rng.choice([1, 3, 5, 8]))
    return dict(kind=kind, nq=_log(rng, 8, 4096), leaves=_log(rng, 100, 2000), bp=150,
                dim=rng.choice([1024, 2048, 4096, 8192]), kmer=rng.choice([5, 8]), beam=rng.choice([1, 3, 5]))


# ---------------------------------------------------------------- inputs
OUT = {"i16": (H.OUT_I16, torch.int16), "i32": (H.OUT_I32, torch.int32), "f16": (H.OUT_F16, torch.float16),
       "bipolar_f16": (H.OUT_BIPOLAR_F16, torch.float16), "sign_bits": (H.OUT_SIGN_BITS, torch.int32)}
MODE = {"norm": H.SCORE_NORM, "cos": H.SCORE_COS, "dot": H.SCORE_DOT}


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _mutate(g, x, rate):
    """Substitutions in base codes 0..3 (rate: a number, or one per row)."""
    hit = torch.rand(x.shape, device="cuda", generator=g) < rate
    other = torch.randint(1, 4, x.shape, dtype=torch.uint8, device="cuda", generator=g)
    return torch.where(hit, (x + other) & 3, x)


def _leaves(g, n):
    """Base codes [n][MAX_BP] of a taxonomy's leaves and their lengths."""
    b = 1
    while b ** 6 < n:
        b += 1
    x = torch.randint(0, 4, (1, MAX_BP), dtype=torch.uint8, device="cuda", generator=g)
    for r, rate in enumerate(RANK_SUBST, 1):
        count = (n + b ** (6 - r) - 1) // b ** (6 - r)
        x = _mutate(g, x[torch.arange(count, device="cuda") // b], rate)
    return x, torch.randint(1400, MAX_BP + 1, (n,), dtype=torch.int32, device="cuda", generator=g)


def _ascii(x):
    return torch.tensor([65, 67, 71, 84], dtype=torch.uint8, device="cuda")[x.int()]


def _reads(g, leaves, lens, n, bp, mixed):
    """Concatenated ASCII reads (bytes, offsets, lengths) sampled from the leaves, and the longest length."""
    src = torch.randint(0, len(leaves), (n,), device="cuda", generator=g)
    if mixed:
        ln = bp * torch.exp(MIXED_SIGMA * torch.randn(n, device="cuda", generator=g))
        ln = ln.clamp(100, MAX_BP).int()
        rate = torch.where(torch.rand(n, device="cuda", generator=g) < 0.2, 0.06, 0.01)[:, None]
    else:
        ln = torch.full((n,), bp, dtype=torch.int32, device="cuda")
        rate = 0.01
    ln = torch.minimum(ln, lens[src])
    first = (torch.rand(n, device="cuda", generator=g) * (lens[src] - ln + 1)).int()
    top = int(ln.max())
    at = torch.arange(top, device="cuda", dtype=torch.int32)
    x = leaves[src[:, None], (first[:, None] + at).clamp(max=MAX_BP - 1).long()]
    x = _ascii(_mutate(g, x, rate))
    x[torch.rand(x.shape, device="cuda", generator=g) < 5e-4] = ord("N")
    flat = torch.cat([x[at < ln[:, None]], torch.zeros(16, dtype=torch.uint8, device="cuda")])
    end = torch.cumsum(ln.long(), 0)
    return flat, end - ln, ln, top


def _encode_rows(ctx, x, lens, out, kind):
    """Rows of padded base codes encoded whole."""
    x = _ascii(x)
    off = torch.arange(len(x), device="cuda") * x.shape[1]
    ctx.encode_segments(x.reshape(-1), off, lens, out, kind, MAX_BP)
    return out


def _references(ctx, g, leaves, lens, copies):
    """int16 reference hypervectors: the leaves encoded, or bundles of noisy copies of each."""
    n = len(leaves)
    refs = torch.empty((n, ctx.dim), dtype=torch.int16, device="cuda")
    if copies == 1:
        return _encode_rows(ctx, leaves, lens, refs, H.OUT_I16)
    step = 20000
    for a in range(0, n, step):
        m = min(step, n - a)
        x = _mutate(g, leaves[a:a + m].repeat_interleave(copies, 0), 0.01)
        rows = torch.empty((m * copies, ctx.dim), dtype=torch.int16, device="cuda")
        _encode_rows(ctx, x, lens[a:a + m].repeat_interleave(copies), rows, H.OUT_I16)
        ptr, idx = _groups(m, copies)
        refs[a:a + m] = ctx.bundle(rows, ptr, idx)
        del x, rows
    return refs


def _groups(n, size):
    return (torch.arange(0, n * size + 1, size, dtype=torch.int64, device="cuda"),
            torch.arange(n * size, dtype=torch.int32, device="cuda"))


def _norms(ctx, rows):
    top = torch.zeros(1, dtype=torch.int32, device="cuda")
    n2 = ctx.norms(rows, top)
    return n2, int(top.item())


def _search_inputs(ctx, case, seed):
    """References and encoded reads of a search case: (refs, their largest value, reads, their norms and largest value)."""
    g = _generator(seed)
    leaves, lens = _leaves(g, case["refs"])
    flat, off, ln, top = _reads(g, leaves, lens, case["nq"], case["bp"], False)
    kind = "i16" if case["kind"] == "plain" else "f16" if case["counts"] else "bipolar_f16"
    q = torch.empty((case["nq"], case["dim"]), dtype=OUT[kind][1], device="cuda")
    ctx.encode_segments(flat, off, ln, q, OUT[kind][0], top)
    refs = _references(ctx, g, leaves, lens, case.get("copies", 1))
    qn, maxq = _norms(ctx, q)
    rn, maxr = _norms(ctx, refs)
    return refs, rn, maxr, q, qn, maxq


def prepare(case, seed):
    kind, dim, kmer = case["kind"], case["dim"], case["kmer"]
    s = dict(case)
    if kind == "encode":
        ctx = H.Context(dim, kmer, case["bp"], 10)
        g = _generator(seed)
        leaves, lens = _leaves(g, max(64, min(2000, case["n"])))
        s["bytes"], s["off"], s["len"], s["top"] = _reads(g, leaves, lens, case["n"], case["bp"], case["mixed"])
    elif kind == "build":
        ctx = H.Context(dim, kmer, 250, 10)
        g = _generator(seed)
        leaves, lens = _leaves(g, case["refs"])
        n = case["refs"] * case["copies"]
        x = _mutate(g, leaves.repeat_interleave(case["copies"], 0), 0.01)
        s["bytes"] = _ascii(x).reshape(-1)
        s["off"] = torch.arange(n, device="cuda") * MAX_BP
        s["len"] = lens.repeat_interleave(case["copies"])
        s["ptr"], s["idx"] = _groups(case["refs"], case["copies"])
    elif kind == "plain":
        ctx = H.Context(dim, kmer, case["bp"], 10)
        s["r"], s["rn"], s["maxr"], s["q"], s["qn"], s["maxq"] = _search_inputs(ctx, case, seed)
    elif kind == "tc":
        ctx = H.Context(dim, kmer, case["bp"], 10)
        refs, _, maxr, s["q"], s["qn"], s["maxq"] = _search_inputs(ctx, case, seed)
        s["db"] = ctx.refdb(refs, maxr, max_query_abs=s["maxq"])
    elif kind == "pipeline":
        ctx = H.Context(dim, kmer, 250, 10)
        g = _generator(seed)
        leaves, lens = _leaves(g, case["refs"])
        flat, off, ln, _ = _reads(g, leaves, lens, case["nq"], case["bp"], True)
        refs = _references(ctx, g, leaves, lens, case["copies"])
        s["db"] = ctx.refdb(refs, _norms(ctx, refs)[1], max_query_abs=1)
        s["seqs"] = H.Seqs(flat.cpu().numpy(), off.cpu().numpy(), ln.cpu().numpy())
        s["pipe"] = H.Pipeline(ctx, s["db"], case["nq"], flat.numel(), MAX_BP, case["k"])
    elif kind == "descent":
        ctx = H.Context(dim, kmer, case["bp"], 10)
        g = _generator(seed)
        leaves, lens = _leaves(g, case["leaves"])
        _, base, counts, ptr, idx = H.synth_tree_csr(case["leaves"])
        wide = int(base[5])
        s["p16"] = _encode_rows(ctx, leaves, lens, torch.empty((case["leaves"], dim), dtype=torch.int16, device="cuda"),
                                H.OUT_I16)
        s["p32"] = torch.empty((wide, dim), dtype=torch.int32, device="cuda")
        d_idx = torch.from_numpy(idx).cuda()
        for r in range(4, -1, -1):
            lo, hi = int(base[r]), int(base[r + 1])
            p = torch.from_numpy(ptr[lo:hi + 1].copy()).cuda()
            if r == 4:  # the parents of the leaves
                ctx.bundle(s["p16"], p, d_idx - wide, out=s["p32"][lo:hi])
            else:
                ctx.bundle(s["p32"], p, d_idx, out=s["p32"][lo:hi])
        s["pn"] = torch.cat([ctx.norms(s["p32"]), ctx.norms(s["p16"])])
        s["ptr"], s["idx"] = torch.from_numpy(ptr).cuda(), d_idx
        s["roots"] = torch.arange(counts[0], dtype=torch.int32, device="cuda")
        s["children"] = int(np.diff(ptr).max())
        s["bytes"], s["off"], s["len"], s["top"] = _reads(g, leaves, lens, case["nq"], case["bp"], case["bp"] == 250)
        s["qn"] = torch.full((case["nq"],), dim, dtype=torch.int64, device="cuda")
    else:  # identify: a leaf's rows are all its windows, an internal node's the first 20 of its first leaf
        ctx = H.Context(dim, kmer, 150, 10)
        g = _generator(seed)
        leaves, lens = _leaves(g, case["leaves"])
        b, base, counts, ptr, idx = H.synth_tree_csr(case["leaves"])
        host_len = lens.cpu().numpy()
        node = np.arange(int(base[-1]))
        rank = np.searchsorted(base, node, side="right") - 1
        leaf = (node - base[rank]) * b ** (5 - rank)
        windows = (host_len[leaf] - 150 + 9) // 10
        windows = np.where(rank < 5, np.minimum(windows, 20), windows)
        rows_ptr = np.concatenate([[0], np.cumsum(windows)])
        n_rows = int(rows_ptr[-1])
        off = np.repeat(leaf * MAX_BP, windows) + 10 * (np.arange(n_rows) - np.repeat(rows_ptr[:-1], windows))
        s["rows"] = torch.empty((n_rows, dim), dtype=torch.int16, device="cuda")
        ctx.encode_segments(_ascii(leaves).reshape(-1), torch.from_numpy(off.astype(np.int64)).cuda(),
                            torch.full((n_rows,), 150, dtype=torch.int32, device="cuda"), s["rows"], H.OUT_I16, 150)
        flat, roff, ln, top = _reads(g, leaves, lens, case["nq"], case["bp"], False)
        s["q"] = torch.empty((case["nq"], dim), dtype=torch.int16, device="cuda")
        ctx.encode_segments(flat, roff, ln, s["q"], H.OUT_I16, top)
        s["qn"], s["rn"] = ctx.norms(s["q"]), ctx.norms(s["rows"])
        s["node_rows"] = torch.from_numpy(rows_ptr.astype(np.int64)).cuda()
        s["ptr"], s["idx"] = torch.from_numpy(ptr).cuda(), torch.from_numpy(idx).cuda()
        s["roots"] = torch.arange(counts[0], dtype=torch.int32, device="cuda")
    s["ctx"] = ctx
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "encode":
        code, dtype = OUT[s["out"]]
        width = (s["dim"] + 31) // 32 if s["out"] == "sign_bits" else s["dim"]
        out = torch.empty((s["n"], width), dtype=dtype, device="cuda")
        kmers = torch.empty(s["n"], dtype=torch.int32, device="cuda")
        ctx.encode_segments(s["bytes"], s["off"], s["len"], out, code, s["top"], nkmers=kmers)
        return out, kmers
    if kind == "build":
        rows = torch.empty((s["refs"] * s["copies"], s["dim"]), dtype=torch.int32, device="cuda")
        ctx.encode_segments(s["bytes"], s["off"], s["len"], rows, H.OUT_I32, MAX_BP)
        refs = ctx.bundle(rows, s["ptr"], s["idx"])
        top = torch.zeros(1, dtype=torch.int32, device="cuda")
        return refs, ctx.norms(refs, top), top
    if kind == "plain":
        return ctx.search_plain(s["q"], s["qn"], s["maxq"], s["r"], s["rn"], s["maxr"], s["k"], MODE[s["mode"]])
    if kind == "tc":
        return ctx.search_tc(s["db"], s["q"], s["qn"], s["maxq"], s["k"], MODE[s["mode"]])
    if kind == "pipeline":
        return s["pipe"].run(s["seqs"])
    if kind == "descent":
        bits = torch.empty((s["nq"], s["dim"] // 32), dtype=torch.int32, device="cuda")
        ctx.encode_segments(s["bytes"], s["off"], s["len"], bits, H.OUT_SIGN_BITS, s["top"])
        return ctx.beam_search_split(bits, s["qn"], s["p32"], s["p16"], s["pn"], s["ptr"], s["idx"], s["roots"], 6,
                                     s["beam"], float("-inf"), max_children=s["children"])
    return ctx.identify(s["q"], s["qn"], s["rows"], s["rn"], s["node_rows"], s["ptr"], s["idx"], s["roots"], 6,
                        s["beam"], -2.0)


def _tree_pairs(leaves, beam):
    """Nodes that a descent scores per read, and the tree's nodes."""
    b, base, counts, _, _ = H.synth_tree_csr(leaves)
    return counts[0] + sum(min(counts[r], b * min(beam, counts[r - 1])) for r in range(1, 6)), int(base[-1]), int(base[5])


def work(case):
    kind, dim = case["kind"], case["dim"]
    mean = (case.get("bp", 0) * math.exp(MIXED_SIGMA ** 2 / 2)) if case.get("mixed") or kind == "pipeline" else \
        case.get("bp", 0)
    if kind == "encode":  # one addition per k-mer and dim
        size = dict(i16=2, i32=4, f16=2, bipolar_f16=2, sign_bits=0.125)[case["out"]]
        return {"bytes": case["n"] * (mean + 16 + dim * size), "flops": case["n"] * max(0, mean - case["kmer"] + 1) * dim}
    if kind == "build":
        n = case["refs"] * case["copies"]
        return {"bytes": n * 1500 + case["refs"] * (dim * 4 + 8), "flops": n * 1490 * dim}
    if kind in ("plain", "tc"):
        k = min(case["k"], case["refs"])
        return {"bytes": (case["nq"] + case["refs"]) * dim * 2 + case["nq"] * k * 24,
                "flops": 2 * case["nq"] * case["refs"] * dim}
    if kind == "pipeline":
        return {"bytes": case["nq"] * (mean + 16 + case["k"] * 8) + case["refs"] * dim * 2,
                "flops": 2 * case["nq"] * case["refs"] * dim + case["nq"] * mean * dim}
    pairs, nodes, wide = _tree_pairs(case["leaves"], case["beam"])
    if kind == "descent":
        return {"bytes": wide * dim * 4 + case["leaves"] * dim * 2 + case["nq"] * (mean + 48),
                "flops": 2 * case["nq"] * pairs * dim + case["nq"] * mean * dim}
    rows = (wide * 20 + case["leaves"] * 135) / nodes  # windows of a node, on average
    return {"bytes": (wide * 20 + case["leaves"] * 135 + case["nq"]) * dim * 2 + case["nq"] * 56,
            "flops": 2 * case["nq"] * pairs * rows * dim}


# ---------------------------------------------------------------- 64-bit results
def exact(case, seed):
    """The searches' scores and cosines by brute force in 64 bits (dots and norms are whole numbers below 2^53).
    Encodings are whole numbers or signs, which have to be equal; the descents and the largest searches take too long."""
    if case["kind"] not in ("plain", "tc") or case["nq"] * case["refs"] * case["dim"] > EXACT_MACS:
        return None
    ctx = H.Context(case["dim"], case["kmer"], case["bp"], 10)
    refs, _, _, q, _, _ = _search_inputs(ctx, case, seed)
    k = min(case["k"], case["refs"])
    few = min(k + 16, case["refs"])
    rn = torch.cat([x.double().square().sum(1) for x in refs.split(8192)]).sqrt()
    scores, cosines = [], []
    for a in range(0, len(q), 1024):
        x = q[a:a + 1024].double()
        dot = torch.cat([x @ y.double().T for y in refs.split(16384)], 1)
        den = x.square().sum(1).sqrt()[:, None] * rn[None]
        cos = torch.where(den > 0, dot / den, 0.0)
        if case["mode"] == "dot":
            score = dot
        else:
            score = torch.where(den > 0, 2 * (cos - 0.5) if case["mode"] == "norm" else cos, -1.0)
        at = torch.topk(score, few, 1).indices.sort(1).values
        near = score.gather(1, at).float()  # ranked as floats, ties to the lower index
        order = near.sort(dim=1, descending=True, stable=True).indices[:, :k]
        at = at.gather(1, order)
        scores.append(score.gather(1, at))
        cosines.append(cos.gather(1, at))
        del dot, den, cos, score
    return torch.cat(scores), None, torch.cat(cosines), None
