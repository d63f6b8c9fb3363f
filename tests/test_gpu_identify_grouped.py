"""The identify descent grouped by parent on the tensor cores (csrc/identify_grouped.cu) and its way back to the per-read
kernel, against the oracle: identical paths, float scores, depths and stop levels (exact dots, the same IEEE operations)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tree(g, branch, depth, rows_of, dim, vmax):
    """A tree of `branch` children a node and `depth` ranks, numbered rank by rank; rows_of(rank) rows a node."""
    counts = [branch ** (r + 1) for r in range(depth)]
    base = np.concatenate([[0], np.cumsum(counts)])
    n = int(base[-1])
    ptr, idx = np.zeros(n + 1, np.int64), []
    for node in range(n):
        rank = int(np.searchsorted(base, node, side="right")) - 1
        kids = [] if rank == depth - 1 else [int(base[rank + 1]) + (node - int(base[rank])) * branch + j for j in range(branch)]
        idx += kids
        ptr[node + 1] = ptr[node] + len(kids)
    per = [rows_of(int(np.searchsorted(base, node, side="right")) - 1, node) for node in range(n)]
    node_rows = np.concatenate([[0], np.cumsum(per)]).astype(np.int64)
    rows = g.integers(-vmax, vmax + 1, (int(node_rows[-1]), dim)).astype(np.int16)
    return rows, node_rows, ptr, np.array(idx, np.int32), list(range(branch))


def _run(hdc, orc, cuda, q, rows, node_rows, ptr, idx, roots, levels, beam, threshold, mode):
    import torch
    ctx = hdc.Context(q.shape[1], 8, 150, 10)
    t = lambda a: torch.from_numpy(a).to(cuda)
    tq, tr = t(q), t(rows)
    got = ctx.identify(tq, ctx.norms(tq), tr, ctx.norms(tr), t(node_rows), t(ptr), t(idx),
                       torch.tensor(roots, dtype=torch.int32, device=cuda), levels, beam, threshold, mode)
    torch.cuda.synchronize()
    assert ctx.status() == 0
    path, score, depth, stop = (x.cpu().numpy() for x in got)
    for i, (wp, ws, wstop) in enumerate(orc.identify(q, rows, node_rows, ptr, idx, roots, levels, beam, threshold, mode)):
        assert depth[i] == len(wp), i
        assert list(path[i, :len(wp)]) == wp, i
        assert np.array_equal(score[i, :len(wp)], np.array(ws, np.float32)), i
        assert stop[i] == wstop, i


# more entries than an item holds (128), more rows than one holds (192, and a candidate split between two), dims that
# are not a multiple of the 64-dim block, every score mode, a threshold that stops some reads
@pytest.mark.parametrize("dim,nq,branch,beam,threshold,mode,vmax,qmax", [
    (64, 1, 2, 1, -2.0, 0, 140, 140),
    (72, 300, 3, 5, -2.0, 1, 140, 140),
    (200, 129, 2, 8, -0.9, 0, 140, 140),
    (1032, 140, 3, 3, -1e9, 2, 140, 140),
    (128, 60, 2, 5, -2.0, 0, 600, 2048),     # beyond the conversion's short cut (|v| < 512), up to fp16's 2048
    (128, 60, 2, 5, -2.0, 0, 2100, 140),     # a value above 2048: the per-read kernel
    (4096, 40, 2, 5, -2.0, 0, 1500, 1500),   # |q| |r| above 2^24: the per-read kernel
])
def test_grouped_descent_matches_oracle(hdc, orc, cuda, dim, nq, branch, beam, threshold, mode, vmax, qmax):
    g = np.random.default_rng(dim + nq)
    rows_of = lambda rank, node: 0 if node == 3 else (5, 20, 130)[rank] + node % 3
    rows, node_rows, ptr, idx, roots = _tree(g, branch, 3, rows_of, dim, vmax)
    q = g.integers(-qmax, qmax + 1, (nq, dim)).astype(np.int16)
    rows[::17] = 0                                            # zero norms: -1
    rows[5] = rows[2]                                         # equal rows in one node
    a, b = int(node_rows[-2]), int(node_rows[-3])
    rows[a:a + 10] = rows[b:b + 10]                           # and in two: the lower node ranks first
    q[0] = np.clip(rows[a + 1], -qmax, qmax)
    if nq > 2:
        q[1] = 0
        q[2] = np.clip(rows[b + 3], -qmax, qmax)
    _run(hdc, orc, cuda, q, rows, node_rows, ptr, idx, roots, 3, beam, threshold, mode)


def test_more_candidates_than_the_workspace_takes_the_per_read_kernel(hdc, orc, cuda):
    """60 children a node and 300 reads: more candidates than a pass reserves (32 an entry)."""
    g = np.random.default_rng(5)
    rows, node_rows, ptr, idx, roots = _tree(g, 60, 2, lambda rank, node: 1, 64, 140)
    q = g.integers(-140, 141, (300, 64)).astype(np.int16)
    _run(hdc, orc, cuda, q, rows, node_rows, ptr, idx, roots[:4], 2, 1, -2.0, 0)


def test_identify_under_capture(hdc, cuda):
    """The call records into a CUDA graph (its workspace comes from the stream) and replays with new reads."""
    import torch
    g = np.random.default_rng(7)
    rows, node_rows, ptr, idx, roots = _tree(g, 3, 3, lambda rank, node: 10, 256, 140)
    t = lambda a: torch.from_numpy(a).to(cuda)
    ctx = hdc.Context(256, 8, 150, 10)
    qs = [t(g.integers(-140, 141, (50, 256)).astype(np.int16)) for _ in range(2)]
    tr, tree = t(rows), (t(node_rows), t(ptr), t(idx), torch.tensor(roots, dtype=torch.int32, device=cuda))
    rn = ctx.norms(tr)
    q, qn = qs[0].clone(), ctx.norms(qs[0])
    want = [ctx.identify(x, ctx.norms(x), tr, rn, *tree, 3, 5, -2.0) for x in qs]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = ctx.identify(q, qn, tr, rn, *tree, 3, 5, -2.0)
    for x, w in zip(qs, want):
        q.copy_(x)
        qn.copy_(ctx.norms(x))
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(got, w):
            assert torch.equal(a, b)


def test_workspaces_of_contexts_in_threads(hdc, cuda):
    """Contexts that come and go in three threads share a workspace pool: every call on its own stream, same results."""
    import threading
    import torch
    g = np.random.default_rng(11)
    rows, node_rows, ptr, idx, roots = _tree(g, 3, 3, lambda rank, node: 10, 256, 140)
    t = lambda a: torch.from_numpy(a).to(cuda)
    tr, tree = t(rows), (t(node_rows), t(ptr), t(idx), torch.tensor(roots, dtype=torch.int32, device=cuda))
    qs = [t(g.integers(-140, 141, (n, 256)).astype(np.int16)) for n in (3, 50, 400)]

    def call(q):
        ctx = hdc.Context(256, 8, 150, 10)
        out = ctx.identify(q, ctx.norms(q), tr, ctx.norms(tr), *tree, 3, 5, -2.0)
        torch.cuda.current_stream().synchronize()
        assert ctx.status() == 0
        return out
    want = [call(q) for q in qs]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for j in range(12):
                    n = (i + j) % 3
                    if not all(torch.equal(a, b) for a, b in zip(call(qs[n]), want[n])):
                        bad.append((i, j))
        except Exception as e:
            bad.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad
