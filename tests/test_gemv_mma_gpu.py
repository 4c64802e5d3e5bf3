"""The 16-bit tensor streaming projections (csrc/gemv_mma.cu) against the fp64 product of the dequantised weights."""
import pytest
import torch

from owl_engine_b200.formats import nvfp4 as NV
from owl_engine_b200.ops import kernels as K
from owl_engine_b200.ops import quant as Q

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _weight(fmt, n, k, gen):
    w = torch.randn(n, k, generator=gen) * 0.05
    if fmt == "nvfp4":
        q = NV.quantize(w)
        rs = torch.rand(n, generator=gen) + 0.5
        lin = Q.NvFp4Linear(q.codes.to(DEV), q.scales.to(DEV), q.global_scale, n, k, 128, "nvfp4", rs.to(DEV))
        return lin, NV.dequantize(q).double() * rs.double()[:, None]
    c = Q.quantize_w4(w, int(fmt[1:]))
    return Q.pack_skinny(c).to(DEV), c.dequant().double()


def _pack(w, x, flags):
    m, k = x.shape
    rows = (m + 7) // 8 * 8
    xp = torch.full((rows, 2 * k), 0xff, dtype=torch.uint8, device=DEV)          # NaN words in the rows that do not exist
    xs = torch.full((rows, k // w.group, 2), float("nan"), dtype=torch.float32, device=DEV)
    K.act_pack(x.to(DEV), xp, xs, m, k, w.group | K.ACT_FRAG | flags)
    return xp, xs


# tile edges: one row tile, a last row block of 1 to 7 tiles, fewer record columns than k slices, slices of unequal length, and
# matrices that take every k split (8 parts down to 1)
@pytest.mark.parametrize("fmt", ["g128", "g32", "nvfp4"])
@pytest.mark.parametrize("shape", [(16, 128), (144, 384), (256, 1152), (1040, 2176), (20480, 256), (40960, 128)])
@pytest.mark.parametrize("m", [1, 8, 9, 17, 32])
def test_mma_streaming_matches_dequantised_product(fmt, shape, m):
    n, k = shape
    gen = torch.Generator().manual_seed(n + k + m)
    w, deq = _weight(fmt, n, k, gen)
    # outlier channels and a range of magnitudes, as normalised activations have
    x = (torch.randn(m, k, generator=gen) * torch.exp2(torch.randint(-6, 5, (k,), generator=gen).float())).to(torch.bfloat16)
    xp, xs = _pack(w, x, K.ACT_NV if fmt == "nvfp4" else 0)
    want = x.double() @ deq.t()
    out = torch.zeros(m, n, dtype=torch.bfloat16, device=DEV)
    K.w4_mma(w, xp, xs, out, m)
    # bf16 result (2^-9, doubled) + fp32 sums of |products|, the zero points' part (16 steps of 0.05 / 2.5) among them
    size = x.double().abs() @ deq.abs().t() + (16 * 0.05 / 2.5 if fmt != "nvfp4" else 0.1) * x.double().abs().sum(1, keepdim=True)
    tol = want.abs() * 2.0 ** -8 + size * 2.0 ** -20
    assert ((out.double().cpu() - want).abs() <= tol).all()
    res = torch.randn(m, n, generator=gen).to(torch.bfloat16)
    out2 = torch.zeros(m, n, dtype=torch.bfloat16, device=DEV)
    K.w4_mma(w, xp, xs, out2, m, residual=res.to(DEV), epi=K.EPI_RESIDUAL)
    assert ((out2.double().cpu() - want - res.double()).abs() <= tol + (want + res.double()).abs() * 2.0 ** -8).all()
    # gate / up rows interleaved in eights
    out3 = torch.zeros(m, n // 2 + 8, dtype=torch.bfloat16, device=DEV)
    K.w4_mma(w, xp, xs, out3, m, epi=K.EPI_SILU_MUL)
    v = want.view(m, n // 16, 2, 8)
    act = (v[:, :, 0] * torch.sigmoid(v[:, :, 0]) * v[:, :, 1]).reshape(m, n // 2)
    got = out3.double().cpu()
    assert (got[:, n // 2:] == 0).all()
    assert (got[:, :n // 2] - act).norm() <= 5e-3 * act.norm() + 1e-6
    if m > 1:      # a row's bits do not depend on the rows beside it
        xp1, xs1 = _pack(w, x[m - 1:], K.ACT_NV if fmt == "nvfp4" else 0)
        one = torch.zeros(1, n, dtype=torch.bfloat16, device=DEV)
        K.w4_mma(w, xp1, xs1, one, 1)
        assert torch.equal(one[0], out[m - 1])


@pytest.mark.parametrize("fmt,m", [("g128", 1), ("g32", 5), ("g128", 20), ("nvfp4", 3)])
def test_eight_bit_activations(fmt, m):
    n, k = 512, 1024
    gen = torch.Generator().manual_seed(m)
    w, deq = _weight(fmt, n, k, gen)
    group = w.group
    x = torch.randn(m, k, generator=gen).to(torch.bfloat16)
    xp, xs = _pack(w, x, K.ACT_A8 | (K.ACT_NV if fmt == "nvfp4" else 0))
    out = torch.zeros(m, n, dtype=torch.bfloat16, device=DEV)
    K.w4_mma(w, xp, xs, out, m, a8=True)
    xg = x.float().view(m, k // group, group)
    sc = xg.abs().amax(-1, keepdim=True).clamp_min(1e-30) / 127.0
    x8 = (torch.round(xg / sc).clamp(-127, 127) * sc).view(m, k)
    want = x8.double() @ deq.t()
    assert (out.double().cpu() - want).norm() / want.norm() < 5e-3


@pytest.mark.parametrize("rows,m", [(16, 1), (96, 8), (32, 31)])
def test_dense_rows_beside_the_matrix(rows, m):
    n, k = 384, 1280
    gen = torch.Generator().manual_seed(rows)
    w, deq = _weight("g128", n, k, gen)
    x = torch.randn(m, k, generator=gen).to(torch.bfloat16)
    ab = (torch.randn(rows, k, generator=gen) * 0.02).to(torch.bfloat16)
    xp, xs = _pack(w, x, 0)
    out = torch.zeros(m, n, dtype=torch.bfloat16, device=DEV)
    abo = torch.zeros(m, rows, dtype=torch.bfloat16, device=DEV)
    K.w4_mma(w, xp, xs, out, m, ab_w=ab.to(DEV), ab_x=x.to(DEV), ab_out=abo)
    for got, want in ((out, x.double() @ deq.t()), (abo, x.double() @ ab.double().t())):
        assert (got.double().cpu() - want).norm() / want.norm() < 4e-3


@pytest.mark.parametrize("fmt", ["g128", "nvfp4"])
def test_extremes_of_the_activations(fmt):
    """Zero rows, rows of very small and very large values, NaN only where its row is."""
    n, k, m = 64, 512, 5
    gen = torch.Generator().manual_seed(3)
    w, deq = _weight(fmt, n, k, gen)
    x = torch.randn(m, k, generator=gen)
    x[0] = 0
    x[1] *= 2.0 ** -40
    x[2] *= 2.0 ** 55
    x[3, 7] = float("nan")
    x = x.to(torch.bfloat16)
    xp, xs = _pack(w, x, K.ACT_NV if fmt == "nvfp4" else 0)
    out = torch.zeros(m, n, dtype=torch.bfloat16, device=DEV)
    K.w4_mma(w, xp, xs, out, m)
    want = x.double() @ deq.t()
    assert (out[0] == 0).all() and out[3].isnan().all()
    for r in (1, 2, 4):
        assert (out[r].double().cpu() - want[r]).norm() / want[r].norm() < 4e-3


# k parts of two record columns at least: 3 and 4 columns in one and two parts, 7 in two, 8 in four
@pytest.mark.parametrize("fmt", ["g128", "g32", "nvfp4"])
@pytest.mark.parametrize("shape", [(144, 512), (144, 896), (16, 1024), (20480, 1024)])
@pytest.mark.parametrize("m", [1, 32])
def test_k_parts_of_narrow_matrices(fmt, shape, m):
    test_mma_streaming_matches_dequantised_product(fmt, shape, m)


def _same_pack(got, want, m, k, group):
    (xp, xs), (wp, ws) = got, want
    assert torch.equal(xp, wp)
    torch.testing.assert_close(xs, ws, rtol=2.0 ** -18, atol=0, equal_nan=True)          # the sums' order may differ


# what the kernels before a projection write for it, against the pack kernel on their plain outputs
@pytest.mark.parametrize("flags", [0, K.ACT_A8, K.ACT_NV, K.ACT_NV | K.ACT_A8])
@pytest.mark.parametrize("group", [128, 32])
@pytest.mark.parametrize("m", [1, 9])
def test_producers_write_the_fragments_of_their_outputs(flags, group, m):
    g = group | K.ACT_FRAG | flags
    gen = torch.Generator(device=DEV).manual_seed(m + group)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=gen).bfloat16()
    rows = (m + 7) // 8 * 8

    def buffers(k):
        return (torch.full((rows, 2 * k), 0x5a, dtype=torch.uint8, device=DEV),
                torch.full((rows, k // (128 if flags & K.ACT_NV else group), 2), 3.0, device=DEV))

    def packed(x):
        b = buffers(x.shape[1])
        K.act_pack(x, *b, m, x.shape[1], g)
        return b
    for k in (384, 5120, 8192, 8320):              # the row kernel up to 8192, half a warp of chunks at 384 and 8320
        h, w, y, b = rn(m, k), rn(k), torch.empty(m, k, dtype=torch.bfloat16, device=DEV), buffers(k)
        K.rmsnorm_pack(h, w, normed=y, xpack=b[0], xs=b[1], m=m, k=k, group=g)
        _same_pack(b, packed(y), m, k, group)
    # attention: two parts a head, three heads of 256
    hq, hd, splits = 3, 256, 2
    part_o, part_ml = torch.randn(m * hq * splits * hd, device=DEV, generator=gen), torch.rand(m * hq * splits * 2, device=DEV, generator=gen) + 0.5
    y, b = torch.empty(m, hq * hd, dtype=torch.bfloat16, device=DEV), buffers(hq * hd)
    K.attn_reduce(part_o, part_ml, splits, None, 0, m, hq, out=y)
    K.attn_reduce(part_o, part_ml, splits, None, 0, m, hq, xpack=b[0], xs=b[1], group=g)
    _same_pack(b, packed(y), m, hq * hd, group)
    # the recurrence: m rows of one sequence (at most 8) or m sequences
    nk, nv = 1, 3
    ld = (2 * nk + 2 * nv) * 128
    batch, t = (m, 1) if m > 8 else (1, m)
    args = (rn(m, ld), ld, rn(m, 2 * nv), 2 * nv, torch.randn((2 * nk + nv) * 128, 4, device=DEV, generator=gen), torch.zeros(nv, device=DEV),
            torch.ones(nv, device=DEV), torch.ones(128, device=DEV))
    conv, state = torch.zeros(batch, (2 * nk + nv) * 128, 3, device=DEV), torch.zeros(batch, nv, 128, 128, device=DEV)
    slots = torch.arange(batch, dtype=torch.int32, device=DEV)
    y, b = torch.empty(m, nv * 128, dtype=torch.bfloat16, device=DEV), buffers(nv * 128)
    K.gdn_decode(*args, conv, state, slots, out=y, xpack=b[0], xs=b[1], batch=batch, t=t, nk=nk, nv=nv, group=g)
    _same_pack(b, packed(y), m, nv * 128, group)
