"""The search forms that a tensor-core database keeps beside its limbs (digits, fp16 rows): built only where they leave
the caller a quarter of the device's memory, or not at all on request; the limbs serve then, with the same results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(torch, cuda, counts):
    g = torch.Generator(device=cuda).manual_seed(3)
    maxr = 2000 if counts else 2300  # two limbs either way
    refs = torch.randint(-maxr, maxr + 1, (20000, 1024), dtype=torch.int16, device=cuda, generator=g)
    top = 100 if counts else 1
    q = torch.randint(-top, top + 1, (200, 1024), device=cuda, generator=g).half()
    return refs, maxr, q, top


def _search(hdc, torch, ctx, db, q, top):
    out = ctx.search_tc(db, q, ctx.norms(q), top, 5)
    torch.cuda.synchronize()
    assert ctx.status() == 0
    # the kernels of the search: three with a form, two for each part of the limb search
    return [x.cpu().numpy() for x in out], ctx.tc_last_shape()[4]


def _used(torch):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, total = torch.cuda.mem_get_info()
    return total - free


@pytest.mark.parametrize("counts", [False, True])
def test_a_database_without_its_search_forms(hdc, cuda, counts):
    import torch
    ctx = hdc.Context(1024, 10, 250, 10)
    refs, maxr, q, top = _inputs(torch, cuda, counts)
    ctx.refdb(refs, maxr, max_query_abs=top).close()  # (the library's own first allocations)
    used = [_used(torch)]
    full = ctx.refdb(refs, maxr, max_query_abs=top)
    used.append(_used(torch))
    ctx.option(hdc.TC_FORMS, 0)
    bare = ctx.refdb(refs, maxr, max_query_abs=top)
    used.append(_used(torch))
    ctx.option(hdc.TC_FORMS, -1)
    want, n_full = _search(hdc, torch, ctx, full, q, top)
    got, n_bare = _search(hdc, torch, ctx, bare, q, top)
    assert n_full == 3 and n_bare != 3
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    form = 20000 * 1024 * 2  # fp16 rows, or four digits of half a byte
    assert abs(used[1] - used[0] - (used[2] - used[1]) - form) < 16 << 20
    with pytest.raises(hdc.HDCError):
        ctx.option(hdc.TC_FORMS, 1)


def test_forms_leave_the_caller_memory(hdc, cuda, tmp_path):
    import torch
    ctx = hdc.Context(1024, 10, 250, 10)
    refs, maxr, q, top = _inputs(torch, cuda, False)
    first = ctx.refdb(refs, maxr)
    want, n = _search(hdc, torch, ctx, first, q, top)
    assert n == 3
    path = str(tmp_path / "db")
    first.save(path)
    free, total = torch.cuda.mem_get_info()
    # room for 82 MB of limbs, not for half as much again of digits
    hold = torch.empty(free - total // 4 - (100 << 20), dtype=torch.uint8, device=cuda)
    for build in (lambda: ctx.refdb(refs, maxr), lambda: hdc.RefDB.load(ctx, path)[0]):
        db = build()
        got, n = _search(hdc, torch, ctx, db, q, top)
        assert n != 3
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
        db.close()
    del hold
    torch.cuda.empty_cache()
    assert _search(hdc, torch, ctx, ctx.refdb(refs, maxr), q, top)[1] == 3
