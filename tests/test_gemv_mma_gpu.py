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
