"""The single-accumulator tensor-core search (csrc/search_mm.cu) behind hdc_search_plain, at the edges of
its tiles, digits and segments: dots, scores, cosines and order equal to the oracle's bit for bit (whole-number dots
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


# single CTAs (64 references a tile) and pairs (256), ragged on every side; dims around the 64-dim K block, not
# multiples of 8; queries and references whose products force segments (the norms do not fit one) and that do not
@pytest.mark.parametrize("dim,nq,nr,k,mode,qmax,rmax", [
    (64, 1, 1, 1, 0, 3, 3),
    (63, 5, 64, 5, 0, 143, 250),
    (65, 128, 65, 8, 1, 143, 250),
    (1000, 129, 63, 9, 0, 143, 250),
    (200, 130, 129, 16, 2, 143, 250),
    (513, 257, 300, 17, 0, 143, 250),
    (1027, 40, 700, 32, 2, 143, 250),
    (2048, 3000, 5000, 5, 0, 60, 90),     # pairs, several lanes
    (2500, 300, 600, 5, 1, 2048, 125),    # a segment a K block
    (2500, 300, 600, 12, 2, 500, 500),    # a segment a K block, both large
    (1024, 140, 300, 5, 0, 2048, 128),    # the largest product that a K block's sums allow
    (1024, 140, 300, 5, 0, 2048, 129),    # one above: a segment two MMAs
    (1024, 140, 300, 5, 0, 2048, 256),    # the largest product of those
    (1100, 300, 700, 5, 1, 2048, 257),    # one above: a segment an MMA
    (1000, 40, 300, 9, 0, 1023, 1025),    # the largest product accepted
    (520, 7, 3000, 32, 0, 143, 250),      # a zero query: every score tied, more than are scored at once
    (72, 140, 9700, 5, 1, 143, 250),      # a tile an SM
    (70, 129, 20001, 12, 0, 143, 250),    # more tiles than SMs, ragged
    (4100, 2, 12288, 3, 2, 60, 60),       # the most references of a selection, one K block past whole splits
    (1030, 300, 600, 7, 2, 300, 300),     # several K blocks a segment by their norms, where the products allow two
    (1024, 140, 300, 5, 0, 1, 12000),     # +1/0/-1 queries on digits
    (300, 129, 225, 10, 2, 1, 18724),     # five digits at their largest
    (777, 17, 113, 20, 1, 1, 2341),       # five digits, the least that needs them
])
def test_plain_on_tensor_cores_vs_oracle(hdc, orc, cuda, dim, nq, nr, k, mode, qmax, rmax):
    import torch
    g = np.random.default_rng(dim + nq + nr)
    q, r = _values(g, nq, dim, qmax), _values(g, nr, dim, rmax)
    ctx = hdc.Context(dim, 8, 150, 10)
    tq, tr = torch.from_numpy(q).to(cuda), torch.from_numpy(r).to(cuda)
    got = ctx.search_plain(tq, ctx.norms(tq), qmax, tr, ctx.norms(tr), rmax, k, mode)
    torch.cuda.synchronize()
    assert ctx.status() == 0
    _check(got, orc, q, r, k, mode)


def test_plain_unaligned_rows(hdc, orc, cuda):
    """Rows that start 2 bytes off a 16-byte boundary take the element-wise loads of the conversion."""
    import torch
    g = np.random.default_rng(4)
    dim, nq, nr = 512, 70, 200
    q, r = _values(g, nq, dim, 143), _values(g, nr, dim, 250)
    ctx = hdc.Context(dim, 8, 150, 10)
    flat = [torch.zeros(x.size + 1, dtype=torch.int16, device=cuda) for x in (q, r)]
    for f, x in zip(flat, (q, r)):
        f[1:] = torch.from_numpy(x.ravel()).to(cuda)
    tq, tr = flat[0][1:].view(nq, dim), flat[1][1:].view(nr, dim)
    got = ctx.search_plain(tq, ctx.norms(tq), 143, tr, ctx.norms(tr), 250, 5, 0)
    torch.cuda.synchronize()
    _check(got, orc, q, r, 5, 0)


def _plain_raw(hdc, torch, ctx, q, qn, mq, r, rn, mr, k, mode, work_bytes):
    """hdc_search_plain with a workspace of exactly work_bytes."""
    nq = q.shape[0]
    out = (torch.empty((nq, k), dtype=torch.float32, device=q.device),
           torch.empty((nq, k), dtype=torch.int32, device=q.device),
           torch.empty((nq, k), dtype=torch.float64, device=q.device),
           torch.empty((nq, k), dtype=torch.int64, device=q.device))
    work = torch.empty(work_bytes, dtype=torch.uint8, device=q.device)
    p = hdc.ptr
    hdc.check(hdc.lib().hdc_search_plain(ctx.h, p(q), p(qn), nq, mq, p(r), p(rn), r.shape[0], mr, k, mode, p(out[0]),
                                         p(out[1]), p(out[2]), p(out[3]), p(work), work_bytes, hdc.stream_ptr()))
    return out


def test_plain_reference_chunks_equal_the_cuda_core_kernel(hdc, cuda):
    """More converted references than one chunk holds (1 GiB: 32,768 rows of 16,384): the lists go on from chunk to
    chunk; a workspace that is too small for the tensor cores takes the CUDA-core kernel, with the same results."""
    import torch
    dim, nq, nr, k = 16384, 300, 33000, 5
    g = torch.Generator(device=cuda).manual_seed(9)
    r = torch.randint(-100, 101, (nr, dim), dtype=torch.int16, device=cuda, generator=g)
    q = torch.randint(-60, 61, (nq, dim), dtype=torch.int16, device=cuda, generator=g)
    q[:50] = r[32740:32790].clamp(-60, 60)  # answers on both sides of the chunks' border
    r[32900] = r[100]
    ctx = hdc.Context(dim, 8, 150, 10)
    qn, rn = ctx.norms(q), ctx.norms(r)
    full = ctx.workspace_bytes(nq, nr, k)
    a = _plain_raw(hdc, torch, ctx, q, qn, 60, r, rn, 100, k, 0, full)
    b = _plain_raw(hdc, torch, ctx, q, qn, 60, r, rn, 100, k, 0, 64 << 20)
    torch.cuda.synchronize()
    assert full > 64 << 20 and ctx.status() == 0
    for x, y in zip(a, b):
        assert torch.equal(x, y)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("nq,nr", [(3, 64), (140, 20000)])
def test_plain_zero_norm_references_among_negative_scores(hdc, orc, cuda, nq, nr, mode):
    """A zero-norm reference scores -1 in every mode but DOT, below any negative cosine: many of them in a tile may not
    raise the threshold that the others are filtered by."""
    import torch
    g = np.random.default_rng(nr)
    dim = 72
    q = g.integers(1, 60, (nq, dim)).astype(np.int16)
    r = -g.integers(0, 60, (nr, dim)).astype(np.int16)
    r[g.random(nr) < 0.7] = 0
    r[nr // 2:, ::2] = 0
    ctx = hdc.Context(dim, 8, 150, 10)
    tq, tr = torch.from_numpy(q).to(cuda), torch.from_numpy(r).to(cuda)
    got = ctx.search_plain(tq, ctx.norms(tq), 60, tr, ctx.norms(tr), 60, 5, mode)
    torch.cuda.synchronize()
    assert ctx.status() == 0
    _check(got, orc, q, r, 5, mode)
