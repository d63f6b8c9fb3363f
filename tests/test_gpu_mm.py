"""The single-accumulator tensor-core search (csrc/search_mm.cu) behind hdc_search_tc, at the edges of its
tiles, digits and segments: dots, scores, cosines and order equal to the oracle's bit for bit (whole-number dots
and the same IEEE operations, so there is no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(got, orc, q, r, k, mode):
    want = orc.topk(q.astype(np.int32), r.astype(np.int32), min(k, len(r)), mode)
    s, i, c, d = (x.cpu().numpy() for x in got)
    assert np.array_equal(i, want[1])
    assert np.array_equal(d, want[3])
    assert np.array_equal(s, want[0])
    assert np.array_equal(c, want[2])


def _values(g, n, dim, vmax, dtype=np.int16):
    v = g.integers(-vmax, vmax + 1, (n, dim)).astype(dtype)
    if n > 6:
        v[3] = v[1]          # a tie: the lower index first
        v[4] = 0             # zero norm
        v[5] = vmax          # extremes
        v[6, ::2] = -vmax
    return v


# digits: one to five of them, at the largest value that each holds; one and several segments (2048 x 18,724 does not
# fit 2^24); single CTAs (112 references a tile) and pairs (224)
@pytest.mark.parametrize("dim,nq,nr,k,mode,vmax", [
    (64, 3, 5, 5, 0, 4),
    (128, 128, 112, 1, 0, 36),
    (136, 129, 113, 8, 1, 292),
    (1000, 256, 224, 9, 0, 2340),
    (1024, 300, 225, 16, 2, 2341),
    (2048, 130, 1000, 5, 0, 18724),
    (512, 2000, 9000, 17, 0, 2340),
])
def test_tc_digits_vs_oracle(hdc, orc, cuda, dim, nq, nr, k, mode, vmax):
    import torch
    g = np.random.default_rng(dim + nr)
    r = _values(g, nr, dim, vmax)
    q = g.integers(-1, 2, (nq, dim)).astype(np.int8)  # zeros are allowed (max_abs_q = 1)
    q[0] = np.where(r[min(1, nr - 1)] >= 0, 1, -1)
    ctx = hdc.Context(dim, 10, 250, 10)
    db = ctx.refdb(torch.from_numpy(r).to(cuda), vmax)
    q16 = torch.from_numpy(q.astype(np.float16)).to(cuda)
    got = ctx.search_tc(db, q16, ctx.norms(q16), 1, k, mode)
    torch.cuda.synchronize()
    assert ctx.status() == 0 and ctx.tc_last_shape()[4] == 3
    _check(got, orc, q, r, k, mode)


@pytest.mark.parametrize("k", [5, 32])
def test_tc_families_of_relatives(hdc, orc, cuda, k):
    """Consecutive references near one centre: whole tiles beat a query's list at once, so the drain warps raise their
    threshold by bisection; equal scores within a tile and across tiles go to the lower index."""
    import torch
    g = np.random.default_rng(8)
    dim, nq, nr = 512, 300, 6000
    centres = g.integers(-900, 901, (10, dim))
    r = (centres[np.arange(nr) // 600] + g.integers(-30, 31, (nr, dim))).astype(np.int16)
    r[1000:1040] = r[1000]
    r[5000:5040] = r[1000]
    q = np.where(centres[g.integers(0, 10, nq)] + g.integers(-600, 601, (nq, dim)) >= 0, 1, -1).astype(np.int8)
    q[:20] = np.where(r[1000] >= 0, 1, -1)
    ctx = hdc.Context(dim, 10, 250, 10)
    db = ctx.refdb(torch.from_numpy(r).to(cuda), int(np.abs(r).max()))
    q16 = torch.from_numpy(q.astype(np.float16)).to(cuda)
    got = ctx.search_tc(db, q16, ctx.norms(q16), 1, k, 0)
    torch.cuda.synchronize()
    _check(got, orc, q, r, k, 0)


def test_tc_small_workspace_takes_the_limb_search(hdc, orc, cuda):
    """A workspace that held the limb search's lists is still accepted, with the same results."""
    import torch
    g = np.random.default_rng(12)
    dim, nq, nr, k = 1024, 500, 700, 5
    r = _values(g, nr, dim, 2340)
    q = np.where(g.random((nq, dim)) < 0.5, -1, 1).astype(np.int8)
    ctx = hdc.Context(dim, 10, 250, 10)
    db = ctx.refdb(torch.from_numpy(r).to(cuda), 2340)
    q16 = torch.from_numpy(q.astype(np.float16)).to(cuda)
    qn = ctx.norms(q16)
    p = hdc.ptr
    out = [torch.empty((nq, k), dtype=t, device=cuda) for t in (torch.float32, torch.int32, torch.float64, torch.int64)]
    small = torch.empty(min(152, (nr + 127) // 128) * nq * k * 16 + 152 * nq * 4, dtype=torch.uint8, device=cuda)
    need = hdc.lib().hdc_search_tc_workspace_bytes(ctx.h, db.h, nq, k)
    st = hdc.lib().hdc_search_tc(ctx.h, db.h, p(q16), p(qn), nq, 1, k, 0, *[p(o) for o in out], p(small),
                                 min(small.numel(), need - 1), hdc.stream_ptr())
    torch.cuda.synchronize()
    assert st == 0 and ctx.status() == 0 and ctx.tc_last_shape()[4] != 3
    _check(out, orc, q, r, k, 0)


@pytest.mark.parametrize("nq,counts", [(60, False), (600, False), (60, True), (600, True)])
def test_mm_bounded_wait_runs_out_and_context_recovers(hdc, orc, cuda, nq, counts):
    """With the operand loads withheld every wait of the search gives up within its limit (nothing is in flight); the
    status says so and the next search on the context is right."""
    import torch
    g = np.random.default_rng(3)
    dim, nr, k = 1024, 1500, 5
    qmax = 70 if counts else 1
    r = _values(g, nr, dim, 250)
    q = g.integers(-qmax, qmax + 1, (nq, dim)).astype(np.int16)
    ctx = hdc.Context(dim, 10, 250, 10)
    db = ctx.refdb(torch.from_numpy(r).to(cuda), 250, max_query_abs=qmax)
    q16 = torch.from_numpy(q.astype(np.float16)).to(cuda)
    qn = ctx.norms(q16)
    ctx.option(hdc.WAIT_LIMIT, 1000)
    ctx.option(hdc.TEST_WITHHOLD_LOADS, 1)
    ctx.search_tc(db, q16, qn, qmax, k)
    torch.cuda.synchronize()
    assert 101 <= ctx.status() <= 106
    ctx.option(hdc.TEST_WITHHOLD_LOADS, 0)
    ctx.option(hdc.WAIT_LIMIT, 0)
    got = ctx.search_tc(db, q16, qn, qmax, k)
    torch.cuda.synchronize()
    assert ctx.status() == 0
    _check(got, orc, q, r, k, 0)


def test_saved_database_searches_the_same(hdc, cuda, tmp_path):
    """The digits and the fp16 rows are rebuilt when a database file is loaded."""
    import torch
    g = np.random.default_rng(6)
    dim, nq, nr, k = 520, 200, 400, 5
    r = torch.from_numpy(_values(g, nr, dim, 250)).to(cuda)
    ctx = hdc.Context(dim, 10, 250, 10)
    for qmax in (1, 100):
        q = torch.from_numpy(g.integers(-qmax, qmax + 1, (nq, dim)).astype(np.float16)).to(cuda)
        db = ctx.refdb(r, 250, max_query_abs=qmax)
        db.save(tmp_path / "db", None)
        again, _ = hdc.RefDB.load(ctx, tmp_path / "db")
        a = ctx.search_tc(db, q, ctx.norms(q), qmax, k)
        b = ctx.search_tc(again, q, ctx.norms(q), qmax, k)
        torch.cuda.synchronize()
        assert ctx.tc_last_shape()[4] == (3 if qmax == 1 else 2)  # (packing,) dots, selection
        for x, y in zip(a, b):
            assert torch.equal(x, y)


@pytest.mark.parametrize("nr,k", [(300, 10), (100, 5)])
def test_tc_many_groups_of_few_tiles(hdc, cuda, nr, k):
    """Far more query tiles than SMs against one or two reference tiles: a drain warp may be a whole group of query tiles
    ahead of the other half's, and its candidates wait for their own group.  Equal to the limb search bit for bit."""
    import torch
    g = torch.Generator(device=cuda).manual_seed(nr)
    dim, nq = 256, 60001
    r = torch.randint(-200, 201, (nr, dim), dtype=torch.int16, device=cuda, generator=g)
    q = (torch.randint(0, 2, (nq, dim), device=cuda, generator=g) * 2 - 1).to(torch.float16)
    ctx = hdc.Context(dim, 10, 250, 10)
    db = ctx.refdb(r, 200)
    qn = torch.full((nq,), dim, dtype=torch.int64, device=cuda)
    a = ctx.search_tc(db, q, qn, 1, k)
    torch.cuda.synchronize()
    assert ctx.tc_last_shape()[4] == 3
    ctx.tc_option(hdc.TC_CLUSTER, 1)
    b = ctx.search_tc(db, q, qn, 1, k)
    torch.cuda.synchronize()
    assert ctx.status() == 0 and ctx.tc_last_shape()[0] == 1
    for x, y in zip(a, b):
        assert torch.equal(x, y)
