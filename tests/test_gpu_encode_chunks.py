"""The encoder at the edges of its 256-position chunks and 16-entry groups: every k-mer size, segment lengths around
them, k-mers lost to other bytes anywhere (whole runs of them too), every output kind; equal to the oracle's whole
numbers and their signs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 7, 8, 9, 10, 12, 13, 15, 16])
def test_encode_chunk_edges_vs_oracle(hdc, orc, cuda, k):
    import torch
    H = hdc
    g = np.random.default_rng(k)
    dim = 2120  # two slabs, the second one ragged
    seqs = []
    for n in (0, 1, 15, 16, 17, 31, 255, 256, 257, 271, 272, 273, 512, 700):  # k-mers
        for rate in (0.0, 0.02, 0.4):
            s = g.choice(list("ACGT"), size=n + k - 1 if n else max(0, k - 1))
            s[g.random(len(s)) < rate] = "N"
            seqs.append("".join(s))
    seqs.append("N" * 300 + "ACGTTGCAACGTTGCAGG" + "N" * 300)
    seqs.append("A" * 260)          # one k-mer over and over
    seqs.append("ACGT" * 80)        # its own reverse complement where k is even
    want, kmers = orc.encode(seqs, dim, k, "int32")
    ctx = H.Context(dim, k, 150, 10)
    buf, off, ln = H.pack_sequences(seqs)
    t = [torch.from_numpy(x.copy()).to(cuda) for x in (buf, off, ln)]
    sign = np.where(want >= 0, 1, -1)
    for kind, dtype, ref in ((H.OUT_I32, torch.int32, want), (H.OUT_I16, torch.int16, want.astype(np.int16)),
                             (H.OUT_F16, torch.float16, want), (H.OUT_BIPOLAR_I16, torch.int16, sign),
                             (H.OUT_BIPOLAR_F16, torch.float16, sign), (H.OUT_BIPOLAR_BF16, torch.bfloat16, sign),
                             (H.OUT_BIPOLAR_I8, torch.int8, sign)):
        out = torch.zeros((len(seqs), dim), dtype=dtype, device=cuda)
        nk = torch.zeros(len(seqs), dtype=torch.int32, device=cuda)
        ctx.encode_segments(*t, out, kind, int(ln.max()), nkmers=nk)
        torch.cuda.synchronize()
        assert np.array_equal(out.float().cpu().numpy(), ref.astype(np.float32)), kind
        assert np.array_equal(nk.cpu().numpy(), kmers)
    bits = torch.zeros((len(seqs), (dim + 31) // 32), dtype=torch.int32, device=cuda)
    ctx.encode_segments(*t, bits, H.OUT_SIGN_BITS, 5000)  # a longer hint: the widest counters
    torch.cuda.synchronize()
    w = bits.cpu().numpy().view(np.uint32)
    got = (w[:, :, None] >> np.arange(32, dtype=np.uint32)) & 1
    assert np.array_equal(got.reshape(len(seqs), -1)[:, :dim], (sign > 0).astype(np.uint32))
