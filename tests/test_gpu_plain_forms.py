"""Which kernels hdc_search_plain takes (hdc_search_plain_last_form), at the borders of its rule, with the results equal
to the CUDA-core kernel's (whole-number dots and the same IEEE operations, so there is no tolerance)."""
import pytest

pytestmark = pytest.mark.gpu


def _rows(torch, cuda, seed, n, dim, top):
    g = torch.Generator(device=cuda).manual_seed(seed)
    v = torch.randint(-top, top + 1, (n, dim), dtype=torch.int16, device=cuda, generator=g)
    v[0, 0] = top
    return v


def _search(hdc, ctx, q, maxq, r, maxr, k, mode=0, work_bytes=None, offset=0):
    """hdc_search_plain with a workspace of work_bytes (default: all that it asks for) that starts `offset` bytes off."""
    import torch
    nq = q.shape[0]
    k = min(k, r.shape[0])
    out = [torch.empty((nq, k), dtype=t, device=q.device) for t in
           (torch.float32, torch.int32, torch.float64, torch.int64)]
    n = ctx.workspace_bytes(nq, r.shape[0], k) if work_bytes is None else work_bytes
    work = torch.empty(n + offset, dtype=torch.uint8, device=q.device)[offset:]
    qn, rn = ctx.norms(q), ctx.norms(r)
    p = hdc.ptr
    hdc.check(hdc.lib().hdc_search_plain(ctx.h, p(q), p(qn), nq, maxq, p(r), p(rn), r.shape[0], maxr, k, mode,
                                         *(p(x) for x in out), p(work), n, hdc.stream_ptr()))
    torch.cuda.synchronize()
    return out


CUDA, SPLIT, F16, DIGITS = 0, 1, 2, 3


# at most a tile an SM (12,288 references, 152 tiles of 64) and one more of each; a product whose K block does not fit;
# fp16's largest value and one above; five digits' largest and one above; small, unaligned and full workspaces
@pytest.mark.parametrize("dim,nq,nr,k,maxq,maxr,work,offset,form,kernels", [
    (64, 1, 1, 1, 3, 3, None, 0, SPLIT, 3),
    (1000, 48, 2000, 1, 121, 1490, None, 0, SPLIT, 3),
    (72, 3, 9728, 5, 60, 90, None, 0, SPLIT, 3),
    (72, 3, 9729, 5, 60, 90, None, 0, F16, 5),
    (72, 129, 4864, 5, 60, 90, None, 0, SPLIT, 3),
    (72, 129, 4865, 5, 60, 90, None, 0, F16, 5),
    (1024, 140, 300, 5, 2048, 128, None, 0, SPLIT, 3),
    (1024, 140, 300, 5, 2048, 129, None, 0, F16, 5),
    (256, 40, 300, 5, 511, 2048, None, 0, F16, 5),
    (256, 40, 300, 5, 2, 2049, None, 0, CUDA, 2),
    (256, 40, 300, 5, 1, 2048, None, 0, SPLIT, 3),
    (256, 40, 300, 5, 1, 2049, None, 0, DIGITS, 5),
    (256, 40, 300, 5, 1, 2340, None, 0, DIGITS, 5),
    (256, 40, 300, 5, 1, 18724, None, 0, DIGITS, 5),
    (256, 40, 300, 5, 1, 18725, None, 0, CUDA, 2),
    (256, 40, 300, 5, 60, 90, 1 << 16, 0, CUDA, 2),
    (256, 40, 300, 5, 60, 90, None, 16, CUDA, 2),
])
def test_plain_form_and_results(hdc, cuda, dim, nq, nr, k, maxq, maxr, work, offset, form, kernels):
    import torch
    ctx = hdc.Context(dim, 8, 150, 10)
    assert ctx.plain_last_form()[0] == -1
    q, r = _rows(torch, cuda, 1, nq, dim, maxq), _rows(torch, cuda, 2, nr, dim, maxr)
    got = _search(hdc, ctx, q, maxq, r, maxr, k, 0, work, offset)
    assert ctx.plain_last_form() == (form, kernels) and ctx.status() == 0
    want = _search(hdc, ctx, q, maxq, r, maxr, k, 0, None, 16)
    assert ctx.plain_last_form()[0] == CUDA
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dim,nq,nr,k,maxr,form", [
    (10240, 8, 100000, 5, 2340, DIGITS),   # four digits, more references than a chunk of either form holds
    (10240, 8, 100000, 5, 2341, DIGITS),   # five
    (10240, 8, 100000, 5, 2048, F16),
    (10240, 300, 70000, 32, 2340, DIGITS),
])
def test_the_workspace_asked_for_holds_every_form(hdc, cuda, dim, nq, nr, k, maxr, form):
    """hdc_search_workspace_bytes does not know the values; with all of it a search runs on the tensor cores."""
    import torch
    ctx = hdc.Context(dim, 8, 150, 10)
    r = torch.zeros((nr, dim), dtype=torch.int16, device=cuda)
    r[::7, ::3] = maxr
    q = torch.ones((nq, dim), dtype=torch.int16, device=cuda)
    _search(hdc, ctx, q, 1, r, maxr, k)
    assert ctx.plain_last_form()[0] == form and ctx.status() == 0


def _same_as_cuda_cores(hdc, ctx, got, q, maxq, r, maxr, k, rows):
    """The results of the given query rows against those of a search of these rows alone on CUDA cores."""
    import torch
    want = _search(hdc, ctx, q[rows].contiguous(), maxq, r, maxr, k, 0, None, 16)
    assert ctx.plain_last_form()[0] == CUDA
    for a, b in zip(got, want):
        assert torch.equal(a[rows], b)


def test_plain_digits_go_on_from_chunk_to_chunk(hdc, cuda):
    """+1/0/-1 queries against more references than one chunk of digits holds (1 GiB: 65,536 rows of 8,192 in four digits
    and 52,416 in five): answers on both sides of the border, ties across it to the lower index."""
    import torch
    dim, nq, nr, k = 8192, 140, 70000, 9
    q = _rows(torch, cuda, 3, nq, dim, 1)
    for maxr, border in ((2340, 65536 // 224 * 224), (2341, 52416)):
        r = _rows(torch, cuda, maxr, nr, dim, maxr)
        r[border - 3:border + 3] = q[:6] * 100
        r[border + 20] = r[border - 2]
        r[nr - 1] = r[5]
        ctx = hdc.Context(dim, 8, 150, 10)
        got = _search(hdc, ctx, q, 1, r, maxr, k)
        form, kernels = ctx.plain_last_form()
        assert form == DIGITS and kernels == 8 and ctx.status() == 0  # two chunks
        _same_as_cuda_cores(hdc, ctx, got, q, 1, r, maxr, k, torch.arange(nq, device=cuda))


@pytest.mark.parametrize("maxq,maxr,nr,kernels", [
    (60, 90, 300, 8),        # fp16 rows: two batches of queries, one chunk of references
    (60, 90, 33000, 16),     # and two chunks, converted again for the second batch
    (1, 2340, 400, 8),       # digits
])
def test_plain_query_batches(hdc, cuda, maxq, maxr, nr, kernels):
    """More converted queries than a batch holds (1 GiB: 32,768 rows of 16,384 in fp16, 131,072 in e2m1), with a short last
    batch of another plan: rows on both sides of the border and at the ends."""
    import torch
    dim, k = 16384, 7
    batch = 32768 if maxq > 1 else 131072
    nq = batch + 77
    ctx = hdc.Context(dim, 8, 150, 10)
    q, r = _rows(torch, cuda, 5, nq, dim, maxq), _rows(torch, cuda, 6, nr, dim, maxr)
    got = _search(hdc, ctx, q, maxq, r, maxr, k)
    form, n = ctx.plain_last_form()
    assert form == (DIGITS if maxq == 1 else F16) and n == kernels and ctx.status() == 0
    rows = torch.cat([torch.arange(a, b, device=cuda) for a, b in ((0, 40), (batch - 50, batch + 77))])
    _same_as_cuda_cores(hdc, ctx, got, q, maxq, r, maxr, k, rows)


def test_plain_without_room_for_the_full_workspace(hdc, cuda):
    """The binding goes on with the least workspace when the full one cannot be allocated, and a failed allocation
    through the library leaves nothing behind for the next launch."""
    import ctypes
    import torch
    ctx = hdc.Context(256, 8, 150, 10)
    q, r = _rows(torch, cuda, 7, 40, 256, 60), _rows(torch, cuda, 8, 500, 256, 90)
    qn, rn = ctx.norms(q), ctx.norms(r)
    want = ctx.search_plain(q, qn, 60, r, rn, 90, 5)
    assert ctx.plain_last_form()[0] == SPLIT
    p = ctypes.c_void_p()
    assert hdc.lib().hdc_device_alloc(1 << 50, ctypes.byref(p)) == 4 and not p.value
    assert torch.equal(ctx.norms(q), qn)
    ctx.workspace_bytes = lambda nq, nr, k: 1 << 50
    got = ctx.search_plain(q, qn, 60, r, rn, 90, 5)
    torch.cuda.synchronize()
    assert ctx.plain_last_form()[0] == CUDA
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    small = torch.empty(1 << 16, dtype=torch.uint8, device=cuda)
    ctx.search_plain(q, qn, 60, r, rn, 90, 5, work=small)
    assert ctx.plain_last_form()[0] == CUDA


@pytest.mark.parametrize("kind", ["plain", "tc"])
@pytest.mark.parametrize("at,value", [(0, 2), (39 * 256 + 255, -2), (7 * 256 + 31, 9), (20 * 256 + 64, -2048)])
def test_queries_beyond_their_declared_bound_are_reported(hdc, cuda, kind, at, value):
    """A search on digits declared for +1/0/-1 queries packs e2m1 codes: a larger value raises status 201."""
    import torch
    ctx = hdc.Context(256, 8, 150, 10)
    q, r = _rows(torch, cuda, 9, 40, 256, 1), _rows(torch, cuda, 10, 300, 256, 3000)

    def run():
        if kind == "plain":
            ctx.search_plain(q, ctx.norms(q), 1, r, ctx.norms(r), 3000, 5)
            assert ctx.plain_last_form()[0] == DIGITS
        else:
            h = q.half()
            ctx.search_tc(db, h, ctx.norms(h), 1, 5)
        torch.cuda.synchronize()
        return ctx.status()
    db = ctx.refdb(r, 3000) if kind == "tc" else None
    assert run() == 0
    q.view(-1)[at] = value
    assert run() == 201
    q.view(-1)[at] = 1
    assert run() == 0
