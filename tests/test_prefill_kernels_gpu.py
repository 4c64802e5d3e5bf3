"""Prompt-sized forms of the prefill kernels against the forms that short inputs take."""
import gc
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch

from owl_engine_b200.models.hybrid import StatePool
from owl_engine_b200.models.spec import PRESETS
from owl_engine_b200.ops import gemm_tc, linear
from owl_engine_b200.ops import kernels as K
from owl_engine_b200.ops import quant as Q
from owl_engine_b200.ops import reference as R
from owl_engine_b200.utils.ledger import DeviceLedger

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("t", [512, 513, 519, 700])
@pytest.mark.parametrize("use_state", [False, True])
def test_conv_of_long_chunks_equals_short_chunks(t, use_state):
    """Eight rows per warp (from 512 rows) against one row per warp, fed the same rows in pieces with the history between them:
    the same products in the same order, so the same bits."""
    nk, nv, slot = 2, 4, 1
    gen = torch.Generator(device=DEV).manual_seed(t)
    cd = (2 * nk + nv) * 128
    x = torch.randn(t, cd + 64, device=DEV, generator=gen).bfloat16()
    w = torch.randn(cd, 4, device=DEV, generator=gen)
    hist = torch.randn(3, cd, 3, device=DEV, generator=gen)
    h1, h2 = hist.clone(), hist.clone()
    a, b = (torch.zeros(t, cd, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    K.gdn_conv_fwd(x, cd + 64, w, h1, slot, a, t, nk, nv, use_state)
    for r in range(0, t, 256):
        n = min(256, t - r)
        K.gdn_conv_fwd(x[r:], cd + 64, w, h2, slot, b[r:], n, nk, nv, use_state or r > 0)
    assert torch.equal(a, b) and torch.equal(h1, h2)


@pytest.mark.parametrize("t", [40, 128, 288, 289])
def test_prompt_kernels_that_start_early_wait_for_the_rows_before(t):
    """Up to 288 rows a kernel starts while the one before drains. Three layers back to back, which read and overwrite the same
    buffers, against the same launches with a synchronisation after each: the same bits."""
    nk, nv, slot = 2, 6, 1
    gen = torch.Generator(device=DEV).manual_seed(t)
    cd, vd = (2 * nk + nv) * 128, nv * 128
    wide = torch.randn(t, cd + vd, device=DEV, generator=gen).bfloat16()
    cw = torch.randn(cd, 4, device=DEV, generator=gen)
    ab = torch.randn(t, 2 * nv, device=DEV, generator=gen).bfloat16()
    a_log, dt, gamma = (torch.randn(n, device=DEV, generator=gen) for n in (nv, nv, 128))
    w = (torch.randn(cd + vd, vd, device=DEV, generator=gen) * vd ** -0.5).half()
    runs = []
    for sync in (True, False):
        hist, st = torch.zeros(2, cd, 3, device=DEV), torch.zeros(2, nv, 128, 128, device=DEV)
        conv, mix = torch.zeros(t, cd, dtype=torch.bfloat16, device=DEV), torch.zeros(t, vd, dtype=torch.float16, device=DEV)
        cur = wide.clone()
        torch.cuda.synchronize()
        for _ in range(3):
            for step in (lambda: K.gdn_conv_fwd(cur, cd + vd, cw, hist, slot, conv, t, nk, nv, True),
                         lambda: K.gdn_scan(conv, cur[:, cd:], cd + vd, ab, 2 * nv, a_log, dt, gamma, st, slot, mix, t, nk, nv, True),
                         lambda: gemm_tc.f16_gemm(mix, w, cur)):
                step()
                if sync:
                    torch.cuda.synchronize()
        runs.append((cur, hist, st, mix))
    assert torch.isfinite(runs[0][0].float()).all()
    assert all(torch.equal(a, b) for a, b in zip(*runs))


@pytest.mark.parametrize("t", [1, 128, 257, 2048, 9473])
def test_narrow_product_cut_along_k(t):
    """96 rows of k 5120 (the a / b projection of long prompts): from one row tile to more than half as many as there are SMs (not cut)."""
    n, k = 96, 5120
    gen = torch.Generator(device=DEV).manual_seed(t)
    x = torch.randn(t, k, device=DEV, generator=gen).half()
    w = (torch.randn(n, k, device=DEV, generator=gen) * 0.05).half()
    out = torch.zeros(t, n, dtype=torch.bfloat16, device=DEV)
    gemm_tc.f16_gemm(x, w, out, force_persist=True)
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    # one rounding to bf16 and fp32 sums (of at most 16 parts) of k / 16 MMA steps
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + size * (k / 16 + 16) * 2.0 ** -24).all()


@pytest.mark.parametrize("nv", [18, 36, 48, 75])
def test_chunked_scan_splits_its_columns(nv):
    """8, 4, 3 (of 5, 5 and 6 column tiles) and 2 parts: the sums of a column do not depend on the part it lies in, so three heads alone
    (8 parts) give the same bits. A ragged last chunk."""
    t, slot = 130, 1
    gen = torch.Generator(device=DEV).manual_seed(nv)
    nk = nv // 3
    q, k, v = (torch.randn(t, n, 128, device=DEV, generator=gen) for n in (nk, nk, nv))
    q, k = (x / x.norm(dim=2, keepdim=True) for x in (q, k))
    z, a, b = (torch.randn(t, n, device=DEV, generator=gen).bfloat16() for n in (nv * 128, nv, nv))
    a_log, dt, gamma = (torch.randn(n, device=DEV, generator=gen) for n in (nv, nv, 128))
    s0 = torch.randn(2, nv, 128, 128, device=DEV, generator=gen)

    def run(h0, n):
        kh = slice(h0 // 3, (h0 + n) // 3)
        qkv = torch.cat([x.reshape(t, -1) for x in (q[:, kh], k[:, kh], v[:, h0:h0 + n])], 1).bfloat16()
        st, out = s0[:, h0:h0 + n].clone(memory_format=torch.contiguous_format), torch.zeros(t, n * 128, dtype=torch.float16, device=DEV)
        ab = torch.cat([a[:, h0:h0 + n], b[:, h0:h0 + n]], 1).contiguous()
        K.gdn_scan(qkv, z[:, h0 * 128:(h0 + n) * 128].contiguous(), n * 128, ab, 2 * n, a_log[h0:h0 + n].contiguous(),
                   dt[h0:h0 + n].contiguous(), gamma, st, slot, out, t, n // 3, n, True, split="chunked")
        return out, st

    out, st = run(0, nv)
    for h0 in (0, nv - 3):
        o3, s3 = run(h0, 3)
        assert torch.isfinite(o3.float()).all()
        assert torch.equal(out[:, h0 * 128:(h0 + 3) * 128], o3) and torch.equal(st[:, h0:h0 + 3], s3)


@pytest.mark.parametrize("fmt", [0, 1, 2])
@pytest.mark.parametrize("ctx,pad,hkv", [(1, 64, 1), (63, 64, 2), (64, 128, 4), (65, 128, 1), (200, 320, 3)])
def test_gathered_keys_and_values(fmt, ctx, pad, hkv):
    """Tiles of 64 keys: whole, ragged and empty ones; every e4m3 and int8 value is exact in both outputs but for the scale's rounding."""
    gen = torch.Generator(device=DEV).manual_seed(ctx + fmt)
    pages = (ctx + 15) // 16
    bt = torch.randperm(pages + 3, device=DEV, generator=gen)[:pages].int()
    shape = (pages + 3, 16, hkv, 256)
    raw = [torch.randint(0, 256, shape, device=DEV, generator=gen, dtype=torch.uint8) for _ in range(2)]
    sc = [torch.rand(shape[:3], device=DEV, generator=gen) + 0.01 for _ in range(2)]
    if fmt == 0:
        pools = [r.masked_fill((r & 0x7f) == 0x7f, 0x7e) for r in raw]
        vals = [p.view(torch.float8_e4m3fn).float() for p in pools]
    elif fmt == 1:
        pools = raw
        vals = [p.view(torch.int8).float() * s[..., None] for p, s in zip(pools, sc)]
    else:
        pools = [torch.randn(shape, device=DEV, generator=gen).half() for _ in range(2)]
        vals = [p.float() for p in pools]
    k = torch.full((hkv, pad, 256), float("nan"), dtype=torch.bfloat16, device=DEV)
    vt = torch.full((hkv, 256, pad), float("nan"), dtype=torch.float16, device=DEV)
    K.call("owl_kv_gather", K.ptr(pools[0]), K.ptr(pools[1]), K.ptr(sc[0]), K.ptr(sc[1]), fmt, K.ptr(bt), ctx, pad, hkv, 256,
           K.ptr(k), K.ptr(vt), K.stream())
    flat = [v[bt.long()].reshape(-1, hkv, 256)[:ctx] for v in vals]
    assert torch.equal(k[:, :ctx], flat[0].bfloat16().permute(1, 0, 2)) and torch.equal(vt[..., :ctx], flat[1].half().permute(1, 2, 0))
    assert not k[:, ctx:].any() and not vt[..., ctx:].any()


@pytest.mark.parametrize("pool", ["fp8", "int8", "f16"])
@pytest.mark.parametrize("rows,hq,hkv,rot", [(128, 24, 4, 64), (131, 6, 2, 256), (200, 2, 1, 16)])
def test_qknorm_rope_of_many_rows_equals_few_rows(pool, rows, hq, hkv, rot):
    """A CTA per row (from 128 rows) against a CTA per (row, head): the same sums in the same order, so the same bits."""
    hd = 256
    gen = torch.Generator(device=DEV).manual_seed(rows)
    ld = 2 * hq * hd + 2 * hkv * hd
    wide = torch.randn(rows, ld, device=DEV, generator=gen).bfloat16()
    qw, kw = ((torch.randn(hd, device=DEV, generator=gen) * 0.1).bfloat16() for _ in range(2))
    pos3 = torch.randint(0, 200000, (3, rows), device=DEV, generator=gen, dtype=torch.int32)
    inv = R.rope_inv_freq(rot, 1e7).to(DEV)
    section = torch.tensor([j % 3 for j in range(rot // 2)], dtype=torch.uint8, device=DEV)
    slots = torch.randperm(16 * 16, device=DEV, generator=gen)[:rows].int()
    slots[3] = -1

    def run(step):
        dt = torch.float16 if pool == "f16" else torch.uint8
        kp, vp = (torch.zeros(16, 16, hkv, hd, dtype=dt, device=DEV) for _ in range(2))
        sc = (torch.zeros(16, 16, hkv, device=DEV), torch.zeros(16, 16, hkv, device=DEV)) if pool == "int8" else None
        q = torch.zeros(rows, hq, hd, dtype=torch.bfloat16, device=DEV)
        for r in range(0, rows, step):
            n = min(step, rows - r)
            x = wide[r:r + n]
            K.qknorm_rope_insert(x, ld, x[:, 2 * hq * hd:], ld, x[:, 2 * hq * hd + hkv * hd:], ld, qw, kw,
                                 pos3[:, r:r + n].contiguous(), inv, section, slots[r:r + n], q[r:], kp, vp, n, hq, hkv, hd, rot, scales=sc)
        f = (lambda p: p.float()) if pool == "f16" else (lambda p: p.view(torch.int8 if pool == "int8" else torch.float8_e4m3fn).float())
        return [q.float(), f(kp), f(vp)] + list(sc or ())
    for a, b in zip(run(rows), run(64)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("t", [256, 300])
@pytest.mark.parametrize("n,k", [(512, 128), (1072, 1024), (40960, 128)])
@pytest.mark.parametrize("fmt", ["f16", "bf16", "e4m3"])
def test_silu_epilogue(t, n, k, fmt):
    """Edges of the 256-column tile (1072 = 4 tiles + 48), the k-split form (few tiles, 16 k steps) and the unsplit one."""
    gen = torch.Generator(device=DEV).manual_seed(n + t)
    x, w = torch.randn(t, k, device=DEV, generator=gen), torch.randn(n, k, device=DEV, generator=gen) * 0.05
    out = torch.zeros(t, n // 2 + 8, dtype=torch.float16, device=DEV)
    gu = torch.zeros(t, n, dtype=torch.bfloat16, device=DEV)
    two = torch.zeros(t, n // 2, dtype=torch.float16, device=DEV)
    if fmt == "e4m3":
        xq, sx = gemm_tc.quant_e4m3_rows(x.half())
        wq, sw = gemm_tc.quant_e4m3_rows(w.half())
        gemm_tc.gemm_silu(xq, wq, out, sx, sw)
        gemm_tc.e4m3_gemm(xq, sx, wq, sw, gu)
    else:
        dt = torch.float16 if fmt == "f16" else torch.bfloat16
        x, w = x.to(dt), w.to(dt)
        gemm_tc.gemm_silu(x, w, out)
        gemm_tc.f16_gemm(x, w, gu, force_persist=True)
    K.silu_mul(gu, t, n // 2 // 128 * 128, out=two) if n % 256 == 0 else two.copy_(_silu_ref(gu))
    assert (out[:, n // 2:] == 0).all()
    if n % 256 == 0:
        assert torch.equal(out[:, :n // 2], two)          # the same sums, rounded to bf16 and activated the same way
    else:
        torch.testing.assert_close(out[:, :n // 2].float(), two.float(), rtol=2.0 ** -10, atol=2.0 ** -24)
    assert gemm_tc.gemm_status() == 0


def _silu_ref(gu):
    y = gu.float().view(gu.shape[0], -1, 2, 8)
    return (y[:, :, 0] * torch.sigmoid(y[:, :, 0]) * y[:, :, 1]).reshape(gu.shape[0], -1).half()


def test_gate_up_with_activation_matches_two_steps():
    gen = torch.Generator().manual_seed(1)
    c = Q.pack_skinny(Q.quantize_w4(torch.randn(1024, 512, generator=gen) * 0.05, 128)).to(DEV)
    for t in (32, 100, 256, 257):
        x = torch.randn(t, 512, generator=gen).half().to(DEV)
        out = torch.zeros(t, 512, dtype=torch.float16, device=DEV)
        done = linear.w4_gemm_silu(c, x, out, arm="tc")
        assert done == (t > linear.SKINNY_UPTO)
        if done:
            gu = linear.w4_gemm(c, x, torch.empty(t, 1024, dtype=torch.bfloat16, device=DEV), arm="tc")
            two = torch.empty_like(out)
            K.silu_mul(gu, t, 512, out=two)
            assert torch.equal(out, two)


# every token width of a stage (64, 128, 160, 256) at its edges; one row tile, a last row block of 1 to 7 tiles, slices of unequal
# length, and row counts that are cut along k (K from 1024 on)
@pytest.mark.parametrize("t", [1, 17, 64, 65, 137, 192, 241, 256])
@pytest.mark.parametrize("n,k", [(16, 128), (144, 384), (1040, 2176), (5120, 1024), (20480, 128)])
@pytest.mark.parametrize("group", [128, 32])
def test_rows_gemm_dequantises_once(t, n, k, group):
    gen = torch.Generator().manual_seed(n + k + t)
    c = Q.quantize_w4(torch.randn(n, k, generator=gen) * 0.05, group)
    if t == 65:
        c.zeros = c.zeros.half() + 0.3          # fractional zero points, as converted Q4_K blocks have
    w = Q.pack_skinny(c).to(DEV)
    x = torch.randn(t, k, generator=gen).half().to(DEV)
    dense = K.w4_dequant(w, torch.empty(n, k, dtype=torch.float16, device=DEV)).double()
    want = x.double() @ dense.t()
    out = torch.zeros(t, n + 8, dtype=torch.bfloat16, device=DEV)
    gemm_tc.w4_gemm_rows(w, x, out)
    # bf16 result + fp32 sums of products of the same fp16 weights
    size = x.double().abs() @ dense.abs().t()
    assert (out[:, n:] == 0).all()
    assert ((out[:, :n].double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -18).all()
    act = torch.zeros(t, n // 2 + 8, dtype=torch.float16, device=DEV)
    gemm_tc.w4_gemm_rows(w, x, act, silu=True)
    assert (act[:, n // 2:] == 0).all()
    torch.testing.assert_close(act[:, :n // 2].float(), _silu_ref(out[:, :n].contiguous()).float(), rtol=2.0 ** -9, atol=2.0 ** -20)
    assert K.all_status()["gemm_dense"] == 0


# the last and first token counts of every stage and accumulator layout; two units of an odd number of steps a CTA (one set starts the
# second unit), a lone step, parts cut along k (whose sums go through the scratch), one row tile; one to six chunks of tokens
@pytest.mark.parametrize("t", [128, 129, 160, 161, 257, 515, 1300])
@pytest.mark.parametrize("n,k", [(20480, 640), (19088, 384), (1040, 4736), (48, 128)])
def test_rows_gemm_walks_units_and_stages(t, n, k):
    gen = torch.Generator(device=DEV).manual_seed(n + k + t)
    w = Q.random_skinny(n, k, 32, DEV, 0.05, n + k)
    x = torch.randn(t, k, generator=gen, device=DEV).half()
    out = torch.zeros(t, n + 8, dtype=torch.bfloat16, device=DEV)
    gemm_tc.w4_gemm_rows(w, x, out)
    _check_against_dequant(w, x, out[:, :n])
    act = torch.zeros(t, n // 2 + 8, dtype=torch.float16, device=DEV)
    gemm_tc.w4_gemm_rows(w, x, act, silu=True)
    torch.testing.assert_close(act[:, :n // 2].float(), _silu_ref(out[:, :n].contiguous()).float(), rtol=2.0 ** -9, atol=2.0 ** -20)
    assert (out[:, n:] == 0).all() and (act[:, n // 2:] == 0).all() and K.all_status()["gemm_dense"] == 0


@pytest.mark.parametrize("vec", [4, 4096, 5000])
def test_copy_slot_moves_one_row_of_every_layer(vec):
    gen = torch.Generator(device=DEV).manual_seed(vec)
    conv, rec = torch.randn(3, 4, 12, device=DEV, generator=gen), torch.randn(3, 4, vec * 4, device=DEV, generator=gen)
    c2, r2 = conv.clone(), rec.clone()
    K.gdn_copy_slot(conv, rec, 1, 3)
    c2[:, 3], r2[:, 3] = c2[:, 1], r2[:, 1]
    assert torch.equal(conv, c2) and torch.equal(rec, r2)


def test_dequantising_ahead_gives_each_weight_in_turn():
    """More weights than buffers, of different sizes, over two chunks: every copy is the weight's own, and products made while the
    next one is dequantised equal those made one after the other."""
    gen = torch.Generator().manual_seed(4)
    ws = [Q.pack_skinny(Q.quantize_w4(torch.randn(n, k, generator=gen) * 0.05, 128)).to(DEV) for n, k in ((512, 256), (256, 1024), (1024, 128), (768, 512))]
    ahead = linear.DequantAhead(DEV)
    for _ in range(2):
        assert ahead.start(ws)
        for w in ws:
            x = torch.randn(300, w.k, generator=gen).half().to(DEV)
            out = linear.w4_gemm(w, x, torch.empty(300, w.n, dtype=torch.bfloat16, device=DEV), ahead=ahead)
            want = linear.w4_gemm(w, x, torch.empty(300, w.n, dtype=torch.bfloat16, device=DEV))
            assert torch.equal(out, want)


@pytest.mark.parametrize("t", [33, 128, 137, 256])
def test_dense_rows_cut_along_k(t):
    gen = torch.Generator(device=DEV).manual_seed(t)
    x, w = torch.randn(t, 1280, device=DEV, generator=gen).half(), (torch.randn(96, 1280, device=DEV, generator=gen) * 0.05).half()
    out = linear.dense_gemm(x, w, torch.zeros(t, 96, dtype=torch.bfloat16, device=DEV), split=True)
    want = x.double() @ w.double().t()
    # bf16 result + fp32 sums
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + (x.double().abs() @ w.double().abs().t()) * 2.0 ** -19).all()


def _big_zeros(n, k, layout):
    """Group-32 records with zero points outside 0..15, each in whole 16 x 128 records: whole numbers that fp16 sums of 1024 + z would
    round or overflow (a dead Q4_K sub-block has scale 1.2e-7 and its zero point clipped to 65504), negative ones, and fractional."""
    gen = torch.Generator().manual_seed(n + k)
    c = Q.quantize_w4(torch.randn(n, k, generator=gen) * 0.05, 32)
    z = c.zeros.half()
    for i, (zero, scale) in enumerate(((1024, 1e-3), (1025, 1e-3), (3001, 2e-4), (65504, 1.2e-7), (-3, 0.01), (-2040, 2e-4), (15.3, 0.01))):
        r, q = 16 * (i % (n // 16)), 4 * (i // (n // 16))
        z[r:r + 16, q:q + 4], c.scales[r:r + 16, q:q + 4] = zero, scale
    c.zeros = z
    return Q.pack_skinny(c, layout).to(DEV)


def _check_against_dequant(w, x, out):
    dense = K.w4_dequant(w, torch.empty(w.n, w.k, dtype=torch.float16, device=DEV)).double()
    assert dense.isfinite().all()
    want, size = x.double() @ dense.t(), x.double().abs() @ dense.abs().t()
    # bf16 result + fp32 sums of products of the same fp16 weights
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -18).all()


@pytest.mark.parametrize("t", [33, 137])
@pytest.mark.parametrize("n,k", [(112, 256), (32, 1024)])
def test_rows_gemm_with_large_zero_points(t, n, k):
    w = _big_zeros(n, k, "slice")
    x = torch.randn(t, k, generator=torch.Generator().manual_seed(t)).half().to(DEV)
    _check_against_dequant(w, x, gemm_tc.w4_gemm_rows(w, x, torch.zeros(t, n, dtype=torch.bfloat16, device=DEV)))


@pytest.mark.parametrize("layout", ["slice", "block"])
@pytest.mark.parametrize("t", [33, 127])
def test_tiled_gemm_with_large_zero_points(t, layout):
    n, k = 112, 256
    w = _big_zeros(n, k, layout)
    x = torch.randn(t, k, generator=torch.Generator().manual_seed(t)).half().to(DEV)
    _check_against_dequant(w, x, gemm_tc.w4a16_gemm(w, x, torch.zeros(t, n, dtype=torch.bfloat16, device=DEV)))


class _FullDevice(DeviceLedger):
    """A ledger without a budget on a device that has no memory left."""
    tries = 0

    def alloc(self, *a, **kw):
        self.tries += 1
        raise torch.cuda.OutOfMemoryError("out of memory")


def _int4(shapes, seed):
    gen = torch.Generator().manual_seed(seed)
    return [Q.pack_skinny(Q.quantize_w4(torch.randn(n, k, generator=gen) * 0.05, 128)).to(DEV) for n, k in shapes]


@pytest.mark.parametrize("full", [False, True])
def test_dequantising_ahead_is_refused_without_room(full, monkeypatch):
    """No room for the second buffer, in the declared budget or on the device: start() says so, and asks again only once there is
    more."""
    (w,) = _int4([(512, 256)], 9)
    linear._dense_scratch(512, 256, w.records.device, torch.float16)       # the first one is the scratch
    led = _FullDevice("cuda:0") if full else DeviceLedger("cuda:0", total_bytes=1000, enforce=True)
    monkeypatch.setattr(linear, "ledger_for", lambda dev: led)
    ahead = linear.DequantAhead(DEV)
    assert not ahead.start([w]) and not led.entries
    tries, refused = getattr(led, "tries", 0), led.refused
    assert not ahead.start([w]) and (getattr(led, "tries", 0), led.refused) == (tries, refused)
    if not full:
        led.total *= 1000
        monkeypatch.setattr(torch.cuda, "memory_allocated", lambda dev: 1 << 50)          # nothing would stay free
        assert not ahead.start([w])
        monkeypatch.undo()
        assert ahead.start([w])


def test_runners_of_a_device_share_the_buffer(monkeypatch):
    """One second buffer per device, held by one chunk at a time, given back with the last runner."""
    ws = _int4([(512, 256), (256, 512)], 10)
    led = DeviceLedger("cuda:0")
    monkeypatch.setattr(linear, "ledger_for", lambda dev: led)
    linear._dense_scratch(512, 256, ws[0].records.device, torch.float16)
    mine = lambda: [e for n, e in led.entries.items() if n.startswith("dequant ahead")]
    a, b = linear.DequantAhead(DEV), linear.DequantAhead(DEV)
    with ThreadPoolExecutor(1) as other:
        assert a.start(ws) and len(mine()) == 1
        assert not other.submit(b.start, ws).result()                     # a's chunk has the buffers
        x = torch.randn(300, 256, device=DEV).half()
        # the scratch is one of them: another thread's product in line must not write it
        got = other.submit(linear.w4_gemm, ws[0], x, torch.empty(300, 512, dtype=torch.bfloat16, device=DEV)).result()
        for w in ws:
            xw = torch.randn(300, w.k, device=DEV).half()
            out = linear.w4_gemm(w, xw, torch.empty(300, w.n, dtype=torch.bfloat16, device=DEV), ahead=a)
            assert torch.equal(out, gemm_tc.f16_gemm(xw, K.w4_dequant(w, torch.empty(w.n, w.k, dtype=torch.float16, device=DEV)), torch.empty_like(out)))
        assert torch.equal(got, linear.w4_gemm(ws[0], x, torch.empty_like(got)))
        assert other.submit(b.start, ws).result() and len(mine()) == 1    # a's chunk has ended
    del a, b
    gc.collect()
    assert not mine()


def test_unfinished_chunk_gives_its_buffers_up():
    """A chunk that ended in an exception leaves a dequantisation under way: the next user of the scratch waits for it, and the
    chunk's object dequantises in line until it starts again."""
    ws = _int4([(512, 256), (256, 512), (1024, 256)], 11)
    ahead = linear.DequantAhead(DEV)
    x = [torch.randn(300, w.k, device=DEV).half() for w in ws]
    empty = lambda w: torch.empty(300, w.n, dtype=torch.bfloat16, device=DEV)
    want = [linear.w4_gemm(w, xw, empty(w)) for w, xw in zip(ws, x)]
    assert ahead.start(ws)
    first = linear.w4_gemm(ws[0], x[0], empty(ws[0]), ahead=ahead)
    inline = linear.w4_gemm(ws[2], x[2], empty(ws[2]))
    rest = [linear.w4_gemm(w, xw, empty(w), ahead=ahead) for w, xw in zip(ws[1:], x[1:])]
    for got, w in zip([first, inline] + rest, [want[0], want[2], want[1], want[2]]):
        assert torch.equal(got, w)
    assert ahead.start(ws)
    for w, xw, y in zip(ws, x, want):
        assert torch.equal(linear.w4_gemm(w, xw, empty(w), ahead=ahead), y)


def test_second_buffer_makes_room_for_other_entries(monkeypatch):
    """An entry that does not fit the budget beside the second buffer gets its room, in the middle of a chunk."""
    ws = _int4([(512, 256), (256, 512), (1024, 128)], 12)
    led = DeviceLedger("cuda:0", total_bytes=512 * 256 * 2 + 1000, enforce=True)
    linear._dense_scratch(512, 256, ws[0].records.device, torch.float16)
    monkeypatch.setattr(linear, "ledger_for", lambda dev: led)
    ahead = linear.DequantAhead(DEV)
    assert ahead.start(ws)
    for i, w in enumerate(ws):
        x = torch.randn(300, w.k, device=DEV).half()
        out = linear.w4_gemm(w, x, torch.empty(300, w.n, dtype=torch.bfloat16, device=DEV), ahead=ahead)
        if i == 0:
            led.alloc("other", "workspace", (5000,), torch.uint8)
        assert torch.equal(out, gemm_tc.f16_gemm(x, K.w4_dequant(w, torch.empty(w.n, w.k, dtype=torch.float16, device=DEV)), torch.empty_like(out)))
    assert list(led.entries) == ["other"] and not ahead.start(ws)


# products that take longer than a dequantisation, and the other way round
@pytest.mark.parametrize("t,shapes", [(4096, ((2048, 1024), (1024, 2048), (2048, 512), (512, 1024), (1024, 1024))),
                                      (16, ((34816, 1280), (5120, 8704), (16384, 2560)))])
def test_dequantising_ahead_without_host_waits(t, shapes):
    """Two chunks with nothing between the projections that the host or the stream would wait for: results are looked at after the
    last launch only."""
    ws = _int4(shapes, t)
    gen = torch.Generator(device=DEV).manual_seed(t)
    x = [torch.randn(t, w.k, device=DEV, generator=gen).half() for w in ws]
    empty = lambda w: torch.empty(t, w.n, dtype=torch.bfloat16, device=DEV)
    dense = [K.w4_dequant(w, torch.empty(w.n, w.k, dtype=torch.float16, device=DEV)) for w in ws]
    want = [gemm_tc.f16_gemm(xw, d, empty(w)) for w, xw, d in zip(ws, x, dense)]
    out = [[empty(w).zero_() for w in ws] for _ in range(2)]
    ahead = linear.DequantAhead(DEV)
    assert ahead.start(ws)                                                # (allocates)
    for w, xw, y in zip(ws, x, out[0]):
        linear.w4_gemm(w, xw, y, ahead=ahead)
    torch.cuda.synchronize()
    out[0][0].zero_()
    for o in out:
        ahead.start(ws)
        for w, xw, y in zip(ws, x, o):
            linear.w4_gemm(w, xw, y, ahead=ahead)
    for o in out:
        for got, y in zip(o, want):
            assert torch.equal(got, y)


@pytest.mark.parametrize("t", [127, 128, 255, 256, 257])
def test_resident_copy_and_records_give_one_product(t):
    """Both sides of every limit of the resident arm, with the activation and without, against the 16-bit product of the same
    weights (bf16 results of fp32 sums)."""
    (w,) = _int4([(1024, 512)], t)
    x = torch.randn(t, 512, generator=torch.Generator().manual_seed(t)).half().to(DEV)
    dense = K.w4_dequant(w, torch.empty(1024, 512, dtype=torch.float16, device=DEV)).double()
    want, size = x.double() @ dense.t(), x.double().abs() @ dense.abs().t()
    out = linear.w4_gemm(w, x, torch.empty(t, 1024, dtype=torch.bfloat16, device=DEV), arm="tcr")
    assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -18).all()
    act = torch.empty(t, 512, dtype=torch.float16, device=DEV)
    if not linear.w4_gemm_silu(w, x, act, arm="tcr"):
        K.silu_mul(out, t, 512, out=act)
    torch.testing.assert_close(act.float(), _silu_ref(out).float(), rtol=2.0 ** -9, atol=2.0 ** -20)


def test_streams_share_the_scratch_of_cut_products():
    """Two threads, each on a stream of its own, with products that are cut along k (5120 x 1024, the a / b rows): the fp32 parts lie
    in one scratch."""
    (w, v), gen = _int4([(5120, 1024), (5120, 1024)], 21), torch.Generator(device=DEV).manual_seed(21)
    ab = (torch.randn(96, 1024, device=DEV, generator=gen) * 0.05).half()
    jobs = []
    for m, t in ((w, 64), (v, 137)):
        x = torch.randn(t, 1024, device=DEV, generator=gen).half()
        jobs.append((m, x, gemm_tc.w4_gemm_rows(m, x, torch.empty(t, 5120, dtype=torch.bfloat16, device=DEV)),
                     linear.dense_gemm(x, ab, torch.empty(t, 96, dtype=torch.bfloat16, device=DEV), split=True)))
    torch.cuda.synchronize()

    def work(m, x, want, want_ab):
        with torch.cuda.stream(torch.cuda.Stream()):
            y = [(torch.empty_like(want), torch.empty_like(want_ab)) for _ in range(40)]
            for a, b in y:
                gemm_tc.w4_gemm_rows(m, x, a)
                linear.dense_gemm(x, ab, b, split=True)
            return all(torch.equal(a, want) and torch.equal(b, want_ab) for a, b in y)
    with ThreadPoolExecutor(2) as ex:
        assert all(ex.map(lambda j: work(*j), jobs))


def test_copy_slot_indexes_like_a_tensor():
    pool = StatePool(PRESETS["test-hybrid"](), torch.device(DEV), 4, 5)
    pool.conv_state.normal_()
    pool.rec_state.normal_()
    a = [t.clone() for t in (pool.conv_state, pool.rec_state)]
    pool.copy_slot(-1, 0)
    for t, u in zip((pool.conv_state, pool.rec_state), a):
        u[:, 0] = u[:, -1]
        assert torch.equal(t, u)
    for src, dst in ((0, 5), (5, 0), (-6, 0)):
        with pytest.raises(IndexError):
            pool.copy_slot(src, dst)


@pytest.mark.parametrize("fmt", [0, 1, 2])
@pytest.mark.parametrize("pool_off,key_off", [(1, 0), (0, 1), (7, 3)])
def test_gather_of_pools_that_begin_anywhere(fmt, pool_off, key_off):
    """Pools and keys that are not 16-byte aligned (views into a larger allocation), in elements: what aligned ones give, and nothing
    beside the keys is written."""
    ctx, pad, hkv, pages = 83, 128, 2, 8
    gen = torch.Generator(device=DEV).manual_seed(fmt)
    bt = torch.randperm(pages, device=DEV, generator=gen)[:6].int()
    n = pages * 16 * hkv * 256
    flat = [torch.randn(n, device=DEV, generator=gen).half() if fmt == 2 else torch.randint(0, 0x7e, (n,), device=DEV, generator=gen, dtype=torch.uint8)
            for _ in range(2)]
    sc = [torch.rand(pages * 16 * hkv, device=DEV, generator=gen) + 0.01 for _ in range(2)]

    def gather(off_p, off_k):
        pools = [torch.cat([f[:off_p], f])[off_p:] for f in flat]
        k = torch.full((hkv * pad * 256 + 16,), 7.0, dtype=torch.bfloat16, device=DEV)
        vt = torch.zeros(hkv, 256, pad, dtype=torch.float16, device=DEV)
        K.call("owl_kv_gather", K.ptr(pools[0]), K.ptr(pools[1]), K.ptr(sc[0]), K.ptr(sc[1]), fmt, K.ptr(bt), ctx, pad, hkv, 256,
               K.ptr(k[off_k:]), K.ptr(vt), K.stream())
        assert (k[:off_k] == 7).all() and (k[off_k + hkv * pad * 256:] == 7).all()
        return k[off_k:][:hkv * pad * 256], vt
    for a, b in zip(gather(pool_off, key_off), gather(0, 0)):
        assert torch.equal(a, b)


def _one_hot_gates(k, group, cut):
    """A weight whose tiles give gate row r = scale_r * x[0] and up row = x[1], and rows of x for it: nearly every fp16 value of x[0] (some
    of them where the product is cut along k), with an up of 1.5 or one that takes silu(gate) * up out of fp16's range."""
    codes = torch.zeros(256, k, dtype=torch.uint8)
    codes[:, 0] = 1
    codes[7::16, 0] = 15                              # 15 * 65504: an infinite fp16 weight, so gates of -inf, +inf and (times 0) NaN
    up = torch.arange(256) % 16 >= 8
    codes[up, 0], codes[up, 1] = 0, 1
    scales = torch.ones(256, k // group)
    scales[~up] = torch.tensor([1.0, 2.0 ** -8, 2.0 ** -14, 96.0, 3000.0, 65504.0, 0.375, 65504.0]).repeat(16)[:, None]
    w = Q.pack_skinny(Q.W4Canonical(codes, scales.half(), torch.zeros(256, k // group).half(), group)).to(DEV)
    v = torch.arange(65535, dtype=torch.int32, device=DEV).to(torch.int16).view(torch.float16)
    if cut:
        edge = [0.0, -80.0, -79.5, -80.5, -88.0, -89.0, -104.0, -5000.0, 80.0, 90.0, float("inf"), -float("inf"), float("nan")]
        v = torch.cat([torch.tensor(edge, device=DEV).half(), v[7::391]])
    x = torch.zeros(v.numel(), k, dtype=torch.float16, device=DEV)
    x[:, 0] = v
    x[:, 1] = torch.where(torch.arange(v.numel(), device=DEV) % 3 == 0, 60000.0, 1.5).half()
    return w, x


# gates of -80 and below, subnormal results, infinities, NaN; one launch of 256 chunks of tokens, and k in parts
@pytest.mark.parametrize("k,cut", [(128, False), (8192, True)])
@pytest.mark.parametrize("group", [128, 32])
def test_activation_of_every_gate(k, cut, group):
    """The epilogue's silu, which divides without branches, against the two-step form's division on the same rounded products: equal but
    for the sign of a zero. And both against silu in 64 bits."""
    w, x = _one_hot_gates(k, group, cut)
    t = x.shape[0]
    gu, act = torch.zeros(t, 256, dtype=torch.bfloat16, device=DEV), torch.zeros(t, 128, dtype=torch.float16, device=DEV)
    gemm_tc.w4_gemm_rows(w, x, gu)
    gemm_tc.w4_gemm_rows(w, x, act, silu=True)
    two = torch.zeros_like(act)
    K.silu_mul(gu, t, 128, out=two)
    gu = gu.double().view(t, 16, 2, 8)
    g, u = gu[:, :, 0].reshape(t, 128), gu[:, :, 1].reshape(t, 128)
    assert torch.isinf(g).any() and torch.isnan(g).any() and ((g < -80) & (g > -90)).any() and (g < -1e8).any()
    assert (act == two).all()
    # fp32 exponential, quotient and product, then fp16
    want = (g / (1 + torch.exp(-g)) * u).clamp(-65504, 65504)
    assert ((act.double() - want).abs() <= want.abs() * 2.0 ** -10 + 2.0 ** -24)[torch.isfinite(g)].all()
    assert K.all_status()["gemm_dense"] == 0


@pytest.mark.parametrize("t", [40, 137, 256, 288, 289])
def test_mlp_chain_that_starts_early_equals_the_chain_with_host_waits(t):
    """Norm (residual added in place), gate / up with its activation, down twice in a row: the int4 GEMM reads weights before it waits,
    and its k parts (8 of the 512 x 8192 products) meet in the scratch that the next product writes. Four layers back to back against
    the same launches with a synchronisation after each: the same bits."""
    n, inter = 512, 8192
    gen = torch.Generator(device=DEV).manual_seed(t)
    gu, down, down2 = (Q.random_skinny(a, b, 32, DEV, b ** -0.5, i) for i, (a, b) in enumerate(((2 * inter, n), (n, inter), (n, inter))))
    gamma = 1 + 0.1 * torch.randn(n, device=DEV, generator=gen)
    h0 = torch.randn(t, n, device=DEV, generator=gen).bfloat16()
    runs = []
    for sync in (True, False):
        h, x = h0.clone(), torch.zeros(t, n, dtype=torch.float16, device=DEV)
        y, y2 = torch.zeros_like(h), torch.zeros_like(h)
        act = torch.zeros(t, inter, dtype=torch.float16, device=DEV)
        torch.cuda.synchronize()
        for i in range(4):
            for step in (lambda: K.rmsnorm_pack(h, gamma, delta=(y, y2)[i % 2], out_h=h, normed=x, m=t, k=n, group=32, eps=1e-6, pdl=True),
                         lambda: gemm_tc.w4_gemm_rows(gu, x, act, silu=True, pdl=True),
                         lambda: gemm_tc.w4_gemm_rows(down, act, y, pdl=True),
                         lambda: gemm_tc.w4_gemm_rows(down2, act, y2, pdl=True)):
                step()
                if sync:
                    torch.cuda.synchronize()
        runs.append((h, x, act, y, y2))
    assert torch.isfinite(runs[0][0].float()).all() and runs[0][3].float().std() > 0.01
    assert all(torch.equal(a, b) for a, b in zip(*runs))


# several chunks of tokens in groups of 128 (records of another length): two units of an odd number of steps a CTA; k in parts
@pytest.mark.parametrize("t", [257, 515])
@pytest.mark.parametrize("n,k", [(19088, 384), (1040, 4736)])
def test_rows_gemm_walks_units_in_groups_of_128(t, n, k):
    gen = torch.Generator(device=DEV).manual_seed(n + k + t)
    w = Q.random_skinny(n, k, 128, DEV, 0.05, n + k)
    x = torch.randn(t, k, generator=gen, device=DEV).half()
    out = torch.zeros(t, n + 8, dtype=torch.bfloat16, device=DEV)
    gemm_tc.w4_gemm_rows(w, x, out)
    _check_against_dequant(w, x, out[:, :n])
    assert (out[:, n:] == 0).all() and K.all_status()["gemm_dense"] == 0
