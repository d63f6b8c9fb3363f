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
    p = hdc.ptr
    hdc.check(hdc.lib().hdc_search_plain(ctx.h, p(q), p(ctx.norms(q)), nq, maxq, p(r), p(ctx.norms(r)), r.shape[0], maxr, k,
                                         mode, *(p(x) for x in out), p(work), n, hdc.stream_ptr()))
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
