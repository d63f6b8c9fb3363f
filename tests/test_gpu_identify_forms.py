"""How identify's descent runs (hdc_identify_last_form): grouped on the tensor cores as far down as a level fits there, one
CTA a read from the first level that does not, with the beams that the grouped levels kept.  Paths, float scores, depths
and stop levels equal the oracle's (exact dots, the same IEEE operations, so there is no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tree(branches, rows_of):
    """CSR of a tree with branches[r] children a node at rank r, numbered rank by rank, rows_of(rank, node) rows a node."""
    counts = np.cumprod(branches)
    base = np.concatenate([[0], np.cumsum(counts)])
    ptr, idx, per = [0], [], []
    for rank in range(len(branches)):
        for node in range(int(base[rank]), int(base[rank + 1])):
            if rank + 1 < len(branches):
                first = int(base[rank + 1]) + (node - int(base[rank])) * branches[rank + 1]
                idx += range(first, first + branches[rank + 1])
            ptr.append(len(idx))
            per.append(rows_of(rank, node))
    node_rows = np.concatenate([[0], np.cumsum(per)]).astype(np.int64)
    return node_rows, np.array(ptr, np.int64), np.array(idx or [0], np.int32), list(range(branches[0])), base


def _check(hdc, orc, cuda, ctx, q, rows, tree, levels, beam, threshold, mode, reads=None, sized=False):
    """Runs the descent (without the tree's sizes: small trees run grouped too) and compares the reads (all of them by
    default) with the oracle; returns the form."""
    import torch
    node_rows, ptr, idx, roots = tree[:4]
    t = lambda a: torch.from_numpy(a).to(cuda)
    tq, tr = t(q), t(rows)
    qn, rn = ctx.norms(tq), ctx.norms(tr)
    tables = [t(node_rows), t(ptr), t(idx), torch.tensor(roots, dtype=torch.int32, device=cuda)]
    if sized:
        got = ctx.identify(tq, qn, tr, rn, *tables, levels, beam, threshold, mode)
    else:
        i32 = dict(dtype=torch.int32, device=cuda)
        got = (torch.empty((len(q), levels), **i32), torch.empty((len(q), levels), dtype=torch.float32, device=cuda),
               torch.empty(len(q), **i32), torch.empty(len(q), **i32))
        p = hdc.ptr
        hdc.check(hdc.lib().hdc_identify(ctx.h, p(tq), p(qn), len(q), p(tr), p(rn), *(p(x) for x in tables), len(roots), levels,
                                         beam, threshold, mode, *(p(x) for x in got), hdc.stream_ptr()))
    path, score, depth, stop = (x.cpu().numpy() for x in got)
    at = np.arange(len(q)) if reads is None else np.asarray(reads, np.int64)
    want = orc.identify(q[at], rows, node_rows, ptr, idx, roots, levels, beam, threshold, mode)
    for i, (wp, ws, wstop) in zip(at, want):
        assert depth[i] == len(wp), i
        assert list(path[i, :len(wp)]) == wp, i
        assert np.array_equal(score[i, :len(wp)], np.array(ws, np.float32)), i
        assert stop[i] == wstop, i
    return ctx.identify_last_form()


def _inputs(seed, branches, dim, nq, rows_of=lambda rank, node: 4 + node % 3, vmax=140):
    g = np.random.default_rng(seed)
    tree = _tree(branches, rows_of)
    rows = g.integers(-vmax, vmax + 1, (int(tree[0][-1]), dim)).astype(np.int16)
    q = g.integers(-vmax, vmax + 1, (nq, dim)).astype(np.int16)
    near = g.integers(0, max(len(rows), 1), nq)
    if len(rows):
        q[::2] = np.clip(rows[near[::2]] // 2 + q[::2] // 2, -vmax, vmax)
    return g, tree, rows, q


# the level whose rows do not fit: values above 2,048, norms whose product passes 2^48; a threshold at which reads stop
# on every level (about one in ten: the best of 15 cosines of sigma 0.02; they keep their outputs), beams of one and several
@pytest.mark.parametrize("level", [0, 1, 2, None])
@pytest.mark.parametrize("what,beam,threshold,mode", [
    ("value", 5, -2.0, 0), ("value", 1, 0.02, 1), ("norm", 3, -0.96, 0), ("norm", 8, -1e9, 2),
])
def test_descent_goes_on_from_the_level_that_does_not_fit(hdc, orc, cuda, level, what, beam, threshold, mode):
    dim, nq = 2560, 170
    g, tree, rows, q = _inputs(level or 7, [3, 3, 4], dim, nq, vmax=100)  # |q|^2 |r|^2 near 2^46
    node_rows, base = tree[0], tree[4]
    if level is not None:
        # a row of each of the level's nodes
        for node in range(int(base[level]), int(base[level + 1])):
            r = int(node_rows[node])
            if what == "value":
                rows[r, 5] = 2049
            else:
                rows[r] = g.integers(1900, 2049, dim) * g.choice([-1, 1], dim)
    ctx = hdc.Context(dim, 8, 150, 10)
    form = _check(hdc, orc, cuda, ctx, q, rows, tree, 3, beam, threshold, mode)
    assert form == (0 if level is None else level + 1) and ctx.status() == 0


@pytest.mark.parametrize("branches,beam,form", [([2, 2, 300], 3, 3), ([2, 300], 1, 2), ([300], 1, 0), ([2, 2, 250], 3, 0)])
def test_levels_with_more_candidates_than_the_workspace(hdc, orc, cuda, branches, beam, form):
    """A pass of a few reads reserves 256 candidates an entry (and one a read and root)."""
    g, tree, rows, q = _inputs(3, branches, 64, 300, lambda rank, node: 1)
    ctx = hdc.Context(64, 8, 150, 10)
    assert _check(hdc, orc, cuda, ctx, q, rows, tree, len(branches), beam, -2.0, 0) == form
    assert ctx.status() == 0


def test_a_wait_that_runs_out_leaves_the_results_right(hdc, orc, cuda):
    """With its copies withheld the scoring kernel's waits give up within their limit, nothing in flight: the status says so,
    the per-read kernel does the descent, and the next call runs grouped again."""
    g, tree, rows, q = _inputs(9, [3, 3, 3], 256, 200)
    ctx = hdc.Context(256, 8, 150, 10)
    ctx.option(hdc.WAIT_LIMIT, 2000)
    ctx.option(hdc.TEST_WITHHOLD_LOADS, 1)
    assert _check(hdc, orc, cuda, ctx, q, rows, tree, 3, 5, -2.0, 0) == 1
    assert ctx.status() >= 100
    ctx.option(hdc.TEST_WITHHOLD_LOADS, 0)
    ctx.option(hdc.WAIT_LIMIT, 0)
    assert _check(hdc, orc, cuda, ctx, q, rows, tree, 3, 5, -2.0, 0) == 0
    assert ctx.status() == 0


# children counted by a thread (to 32) and by a warp, with none, a few or many rows each (several children a row chunk, and
# several chunks a child), at the roots and below; the last child empty
@pytest.mark.parametrize("branches", [[32], [33], [1000], [2, 33], [3, 200], [40, 5], [70, 40]])
def test_wide_parents(hdc, orc, cuda, branches):
    per = lambda rank, node: 0 if node % 5 == 4 else 500 if node % 31 == 7 else node % 4
    g, tree, rows, q = _inputs(len(branches) + branches[0], branches, 72, 200, per)
    ctx = hdc.Context(72, 8, 150, 10)
    reads = np.arange(0, 200, 1 if len(rows) < 3000 else 9)
    assert _check(hdc, orc, cuda, ctx, q, rows, tree, len(branches), 3, -2.0, 0, reads) == 0
    assert ctx.status() == 0


def test_a_flat_tree_of_many_roots(hdc, orc, cuda):
    """The time that an item's tables take does not grow with the number of roots: within short waits, 100,000 of them."""
    g, tree, rows, q = _inputs(1, [100000], 64, 160, lambda rank, node: 1)
    ctx = hdc.Context(64, 8, 150, 10)
    ctx.option(hdc.WAIT_LIMIT, 3000)  # 3 million cycles, 1.5 ms
    assert _check(hdc, orc, cuda, ctx, q, rows, tree, 1, 5, -2.0, 0, [0, 63, 159]) == 0
    assert ctx.status() == 0


@pytest.mark.parametrize("dim", [23960, 24216, 24224, 24576, 24584, 102400])
def test_reads_near_the_default_shared_memory(hdc, orc, cuda, dim):
    """A read beside the kernel's own shared memory, around the 48 KiB that a launch may take without asking, and the most."""
    g, tree, rows, q = _inputs(1, [3, 2], dim, 5, lambda rank, node: 2, 9)
    rows[0, 0] = 2049  # not for the tensor cores
    ctx = hdc.Context(dim, 8, 150, 10)
    assert _check(hdc, orc, cuda, ctx, q, rows, tree, 2, 3, -2.0, 0) == 1
    assert ctx.status() == 0


@pytest.mark.parametrize("roots,nq,reads,form", [
    (70000, 4000, [0, 2047, 2048, 3999], 0),  # two passes of 2,048 and 1,952 reads (a pass keeps 256 Mi reads times roots)
    (2097153, 160, [], -1),                   # more roots than that holds for 128 reads: one CTA a read
])
def test_passes_bounded_by_the_roots(hdc, orc, cuda, roots, nq, reads, form):
    dim = 64 if reads else 8
    g, tree, rows, q = _inputs(2, [roots], dim, nq, lambda rank, node: 1)
    ctx = hdc.Context(dim, 8, 150, 10)
    assert _check(hdc, orc, cuda, ctx, q, rows, tree, 1, 3, -2.0, 0, reads) == form
    assert ctx.status() == 0


# few nodes of few rows, and the same with many reads; a few reads with one beam row over many rows; wide trees; a leaf root
@pytest.mark.parametrize("branches,rows,dim,nq,beam,form", [
    ([2, 2, 2], 3, 8192, 8, 1, -1),
    ([2, 2, 2], 3, 1024, 152, 5, -1),
    ([2, 2, 2], 3, 1024, 3000, 5, 0),
    ([10], 1, 1024, 152, 5, -1),
    ([10], 1, 1024, 3000, 5, 0),
    ([1], 0, 64, 40, 1, -1),
    ([3, 3, 3, 3], 150, 1024, 17, 1, 0),
    ([3, 3, 3, 3, 3], 30, 1024, 17, 1, -1),
    ([4, 4, 4], 20, 1024, 200, 5, 0),
    ([5000], 1, 64, 20, 1, 0),
])
def test_the_sizes_of_a_tree_pick_the_form(hdc, orc, cuda, branches, rows, dim, nq, beam, form):
    g, tree, r, q = _inputs(4, branches, dim, nq, lambda rank, node: rows, 60)
    if not len(r):
        r = np.zeros((1, dim), np.int16)
    ctx = hdc.Context(dim, 8, 150, 10)
    args = (hdc, orc, cuda, ctx, q, r, tree, len(branches), beam, -2.0, 0, np.arange(0, nq, max(1, nq // 20)))
    assert _check(*args, sized=True) == form
    _check(*args)
    assert ctx.status() == 0
