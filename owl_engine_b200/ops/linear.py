"""Prefill-shape linear layers over quantised weights.

``w4_gemm`` computes ``out[T, N] = x[T, K] @ dequant(w)^T`` for a ``W4Skinny`` weight with one of these arms:

* ``"tc"``        the product path, all steps our own sm_100a kernels. Slice-major weights: up to ``SKINNY_UPTO`` tokens the
                  decode-shape streaming kernel (``csrc/gemv_mma.cu``), above that the tcgen05 GEMM that reads the int4 records and
                  dequantises them into tensor memory, once per 256 tokens (``csrc/gemm_w4.cu``). Matrices under a million weights
                  above 256 tokens: dequantised into a dense fp16 matrix (``csrc/dequant.cu``) that the dense tcgen05 GEMM multiplies.
                  Block-layout weights and operands that are not 16-byte aligned: below ``DEQUANT_FROM`` tokens the tiled GEMM that
                  dequantises in the kernel once per 128 tokens (``csrc/gemm_tc.cu``), from there the dense form (beside the GEMM
                  before it where ``DequantAhead`` applies);
* ``"tc8"``       the W4A8 arm on tensor cores: like ``"tc"``, but from ``DEQUANT_FROM`` tokens the dequantised weight is
                  re-quantised per output row to e4m3 and the activations per token, and the product runs as
                  ``tcgen05.mma kind::f8f6f4`` at twice the 16-bit rate (the reference's W4A8 arm quantises
                  activations per token to int8 for IMMA, ``crates/kernels/cu/elems/quant_i8_act.cu:80-98``; int4
                  values times a group scale do not survive an integer MMA without a per-group epilogue, an
                  8-bit float product with per-row scales does);
* ``"tcr"`` / ``"tc8r"``  the same two arms with the dequantised (fp16) resp. re-quantised (e4m3) weight kept RESIDENT
                  on the weight object after its first use: 2 resp. 1 extra bytes per weight in HBM (48.7 / 24.3 GB for the
                  27B model on one GPU, which 180 GB leave room for) buy back the per-call dequantisation pass. The fp16
                  copies serve chunks above 256 tokens (``rows_pay``);
* ``"baseline"``  dequantise to a dense bf16 scratch matrix, then the library GEMM
                  (``torch.matmul`` = cuBLAS). This is the comparison arm, like the reference's
                  range-dequant -> cuBLAS arm (``crates/kernels/cu/gguf/gguf_smem.cu:415-552``).
"""
from __future__ import annotations

import threading
import weakref

import torch

from ..utils.ledger import BudgetError, ledger_for
from . import gemm_tc
from . import kernels as K

_scratch: dict = {}
DEQUANT_FROM = 128      # tokens per chunk from which the 8-bit arms re-quantise, and from which weights that gemm_w4.cu does not
                        # take are dequantised once (34816 x 5120: tiled form 116 us per 128 tokens, dense form 150 at 128,
                        # 204 at 137)
SILU_FROM = 256         # tokens from which the persistent GEMM, which has the silu(gate) * up epilogue, multiplies fp16 weights
SKINNY_UPTO = 32        # rows up to which the decode-shape weight-streaming kernel is used instead of a GEMM. Set against the tiled GEMM; the
                        # int4 GEMM has passed it since (17 / 32 rows with packing, streaming and GEMM, us: 16384 x 5120 27.7 / 33.0 and
                        # 16.0 / 16.2, 34816 x 5120 46.4 / 56.5 and 29.4 / 29.5, 5120 x 17408 45.2 / 52.3 and 27.7 / 29.0)


def _dense_scratch(n: int, k: int, device, dtype=torch.bfloat16) -> torch.Tensor:
    key = (str(device), dtype)
    shared = _ahead.get(str(torch.device(device))) if dtype == torch.float16 else None
    if shared is not None and not shared.leave_scratch():
        return torch.empty(n, k, dtype=dtype, device=device)
    buf = _scratch.get(key)
    if buf is None or buf.numel() < n * k:
        led = _ledger(device)
        led.release(f"dequant scratch {dtype}")
        _scratch.pop(key, None)
        buf = None
        buf = led.alloc(f"dequant scratch {dtype}", "workspace", (n * k,), dtype)
        _scratch[key] = buf
    return buf[:n * k].view(n, k)


def _ledger(device):
    return ledger_for(device)


def _fp8_scratch(tag: str, r: int, k: int, device):
    key = (tag, str(device))
    buf = _scratch.get(key)
    if buf is None or buf[0].numel() < r * k or buf[1].numel() < r:
        led = _ledger(device)
        led.release(f"e4m3 scratch {tag}")
        buf = (led.alloc(f"e4m3 scratch {tag}", "workspace", (r * k,), torch.uint8), torch.empty(r, dtype=torch.float32, device=device))
        _scratch[key] = buf
    return buf[0][:r * k].view(r, k), buf[1][:r]


# Weights x tokens of a chunk's projections, on average, from which they are dequantised one ahead: the hand-over between the two
# streams costs the host about 7 us a projection, which a pass that waits for the host pays in full. Prompts with / without, ms:
# 5 M weights a projection (0.8B) 400 tokens 6.2 / 6.0, 1000 6.5 / 6.7, 2048 8.2 / 8.6; 15 M 257 tokens 7.7 / 7.2, 700 8.6 / 9.0;
# 28 M 400 tokens 10.6 / 10.7; 54 M 257 tokens 12.4 / 13.3; 95 M (27B) 257 tokens 37.9 / 39.2, 2048 115.9 / 118.9.
AHEAD_FROM = 8e9


def ahead_pays(weights: list, t: int) -> bool:
    return sum(w.n * w.k for w in weights) * t >= AHEAD_FROM * len(weights)


class _AheadShared:
    """What the ``DequantAhead`` objects of a device share: the stream, and beside the dequantisation scratch one more buffer of
    its size (356 MB for the 27B model), a ledger entry that goes when the last of them does or when another entry needs the
    room. One chunk at a time holds both buffers; a second one that starts meanwhile is refused and dequantises in line."""

    NAME = "dequant ahead buffer"

    def __init__(self, device):
        self.device, self.side = device, torch.cuda.Stream(device=device)
        self.free, self.ready = torch.cuda.Event(), torch.cuda.Event()      # a wait takes the state an event has when it is called
        self.lock = threading.RLock()
        self.users = weakref.WeakSet()
        self.holder = self.last = None       # the object whose chunk has the buffers (weakly), and that chunk's stream
        self.extra = self.ledger = self.refused = None
        self.pending = False                 # a dequantisation has been launched that no stream but ``side`` waits for

    def reserve(self, need: int):
        """The second buffer, or None where it does not fit the device's budget or its memory (asked again only once the ledger
        has more room than it had then)."""
        led = _ledger(self.device)
        if self.extra is None or self.extra.numel() < need or self.ledger is not led:
            if self.refused is not None and self.refused[0] is led and need >= self.refused[1] and led.room() <= self.refused[2]:
                return None
            self.release()
            try:
                # allocations that no ledger makes cannot ask for it back: as much again has to stay free (by this process' own
                # count: asking the driver took up to 9 ms after a large release, in the first pass of a new engine)
                left = torch.cuda.get_device_properties(self.device).total_memory - torch.cuda.memory_allocated(self.device)
                if left < 4 * need + (2 << 30):
                    raise BudgetError(self.NAME)
                self.extra = led.alloc(self.NAME, "workspace", (need,), torch.float16)
            except (BudgetError, torch.cuda.OutOfMemoryError):
                self.refused = (led, need, led.room())
                return None
            self.ledger, self.refused = led, None
            led.on_pressure(self.give_back)
        return self.extra

    def give_back(self) -> None:
        """Another entry needs the room: a chunk under way dequantises its other weights in line."""
        with self.lock:
            h = self.holder() if self.holder is not None else None
            if h is not None:
                h.running = False
            self.release()

    def release(self) -> None:
        if self.extra is not None:
            self.ledger.release(self.NAME)
            self.extra = self.ledger = None

    def leave_scratch(self) -> bool:
        """The scratch is wanted for something else: a chunk of this thread that was not finished gives up its buffers, and the
        current stream waits for what may still be written. False while a chunk of another thread holds them."""
        with self.lock:
            h = self.holder() if self.holder is not None else None
            if h is not None and h.running:
                if h.thread != threading.get_ident():
                    return False
                h.running = False
            if self.pending:
                torch.cuda.current_stream(self.device).wait_event(self.ready)
                self.pending = False
        return True

    def user_gone(self) -> None:
        # (from a finaliser: a thread that holds the lock is a user itself, and waiting for it here could be waiting for oneself)
        if not list(self.users) and self.lock.acquire(blocking=False):
            try:
                self.release()
            finally:
                self.lock.release()


_ahead: dict = {}         # device -> _AheadShared
_ahead_lock = threading.Lock()


class DequantAhead:
    """Dequantises a chunk's weights one projection ahead, on a stream of its own: the dequantisation is bound by memory (44 us a
    projection of the 27B model, 11 of 112 ms at 2048 tokens), the GEMM beside it by the tensor cores. Two buffers alternate; a
    buffer is written again only after the GEMM that read it. One object per runner; every use of a buffer on either stream is
    ordered by events, and the allocator knows both streams. Once a chunk has lost its buffers ``take`` returns None."""

    def __init__(self, device):
        dev = torch.device(device)
        if dev.index is None:
            dev = torch.device(dev.type, torch.cuda.current_device())
        with _ahead_lock:
            if str(dev) not in _ahead:
                _ahead[str(dev)] = _AheadShared(dev)
        self.shared = sh = _ahead[str(dev)]
        self.running, self.thread, self.buf = False, 0, ()
        sh.users.add(self)
        weakref.finalize(self, sh.user_gone).atexit = False

    def start(self, weights: list) -> bool:
        """Begin a chunk that multiplies ``weights`` in this order on the current stream; False where there is no second buffer
        or another chunk holds it."""
        sh, need = self.shared, max(w.n * w.k for w in weights)
        with sh.lock:
            h = sh.holder() if sh.holder is not None else None
            if h is not None and h is not self and h.running and h.thread != threading.get_ident():
                return False
            if h is not None:
                h.running = False
            scratch = _dense_scratch(1, need, sh.device, torch.float16).view(-1)
            extra = sh.reserve(need)
            if extra is None:
                return False
            self.main = torch.cuda.current_stream(sh.device)
            if sh.last is not None and sh.last != self.main:
                self.main.wait_stream(sh.last)       # the last chunk's products, on another stream
            sh.last, sh.holder = self.main, weakref.ref(self)
            self.buf = (scratch, extra)
            for b in self.buf:
                b.record_stream(sh.side)
                b.record_stream(self.main)
            self.weights, self.i, self.running, self.thread = weights, -1, True, threading.get_ident()
            sh.free.record(self.main)
        self.kick()
        return True

    def kick(self) -> None:
        """Launch the next weight's dequantisation. Called after the GEMM beside which it is to run has been launched: the GEMM's
        CTAs take their place on the SMs first."""
        sh, j = self.shared, self.i + 1
        with sh.lock:
            if not self.running:
                return
            if j >= len(self.weights):
                self.running, self.buf = False, ()
                return
            w = self.weights[j]
            sh.side.wait_event(sh.free)
            K.w4_dequant(w, self.buf[j % 2][:w.n * w.k].view(w.n, w.k), on=sh.side.cuda_stream)
            sh.ready.record(sh.side)
            sh.pending = True

    def take(self, w) -> torch.Tensor | None:
        """The dense copy of the chunk's next weight, valid for the GEMM launched next on the chunk's stream."""
        sh = self.shared
        with sh.lock:
            self.i += 1
            assert self.weights[self.i] is w, "weights are taken in the order given to start()"
            if not self.running:
                self.buf = ()
                return None
            self.main.wait_event(sh.ready)
            sh.pending = False
            sh.free.record(self.main)            # the other buffer's GEMM has been launched before this point
            return self.buf[self.i % 2][:w.n * w.k].view(w.n, w.k)


def rows_pay(n: int, k: int, t: int, resident: bool) -> bool:
    """Whether ``t`` tokens times an [n, k] int4 weight read the records (``gemm_w4.cu``) rather than a dense copy.

    Up to 256 tokens always: the records are the faster operand even where a resident fp16 copy needs no dequantisation. us at 128 / 137
    / 255 / 256 tokens, records and copy: 16384 x 5120 20.4 / 22.6 / 34.5 / 34.3 and 46.7 / 47.0 / 49.6 / 44.4, 5120 x 6144 16.0 / 17.1
    / 23.3 / 23.3 and 48.0 / 46.5 / 47.3 / 30.3, 34816 x 5120 with the activation 39.5 / 43.7 / 71.3 / 70.9 and 72.6 / 128 / 137 / 92.7,
    5120 x 17408 40.4 / 30.4 / 43.9 / 44.2 and 156 / 123 / 121 / 57.8.

    Above, an arm with resident copies multiplies them: they are what it is asked for, and steps of 24 and more rows, whose graphs are
    captured, need them made before. It costs time below about 1400 tokens (257 / 512 / 1000 / 1400 / 2048, records and copy: 16384 x
    5120 40 / 65 / 129 / 186 / 255 and 71 / 77 / 147 / 194 / 278, 34816 x 5120 80 / 136 / 265 / 423 / 566 and 119 / 161 / 311 / 412 /
    571, 5120 x 17408 49 / 85 / 141 / 184 / 310 and 70 / 116 / 242 / 234 / 392). The other arms read the records from a million weights
    on (257 / 2048 tokens, copy made and multiplied, and records: 1024 x 1024 12.7 / 17.1 and 5.6 / 8.4, 1536 x 1024 17.5 / 15.3 and 5.7
    / 10.0, 1024 x 2048 14.2 / 20.4 and 7.8 / 11.2); smaller matrices, which only test models have, keep the copy made per call (1024 x
    512 12.1 / 15.9 and 4.6 / 6.9)."""
    return t <= gemm_tc.ROWS_UPTO or (not resident and n * k >= 1 << 20)


def _rows_ok(w, x: torch.Tensor, out: torch.Tensor, resident: bool) -> bool:
    """One launch reads the int4 records and dequantises each weight once per chunk of at most 256 tokens."""
    return w.layout == "slice" and x.dtype == torch.float16 and rows_pay(w.n, w.k, x.shape[0], resident) and x.stride(0) % 8 == 0 \
        and out.stride(0) % 8 == 0 and (x.data_ptr() | out.data_ptr()) % 16 == 0


def w4_gemm(w, x: torch.Tensor, out: torch.Tensor, arm: str = "tc", ahead: DequantAhead | None = None, pdl: bool = False) -> torch.Tensor:
    """out[T, N] = x[T, K] @ dequant(w)^T on one of the arms above. ``pdl``: kernels that read the weight's records may do so while the
    kernel before them on the stream still runs (for weights that nothing on it writes any more)."""
    dense = ahead.take(w) if ahead is not None else None
    if dense is not None:
        gemm_tc.f16_gemm(x, dense, out)
        ahead.kick()
        return out
    arm = "tc" if arm == "tc4" else arm                    # the 4-bit float product exists for NVFP4 weights only
    if arm == "baseline":
        dense = K.w4_dequant(w, _dense_scratch(w.n, w.k, x.device))
        torch.matmul(x, dense.t(), out=out)
        return out
    resident = arm in ("tcr", "tc8r")
    if arm in ("tc8", "tc8r") and x.shape[0] >= DEQUANT_FROM and w.k % 128 == 0:
        wq, sw = _e4m3_weight(w, x.device, resident)
        xq, sx = gemm_tc.quant_e4m3_rows(x, *_fp8_scratch("x", x.shape[0], w.k, x.device))
        return gemm_tc.e4m3_gemm(xq, sx, wq, sw, out)
    if arm in ("tc", "tc8", "tcr", "tc8r"):
        if x.shape[0] <= SKINNY_UPTO and w.layout == "slice":
            # a handful of rows (the tail chunk after the last block boundary): the weight-streaming kernel
            t, k = x.shape
            xb = x if x.dtype == torch.bfloat16 else x.to(torch.bfloat16)
            rows = (t + 7) // 8 * 8
            xp = torch.empty(rows * (2 * k + k // w.group * 8), dtype=torch.uint8, device=x.device)
            xs = xp[rows * 2 * k:]                               # (scale, sum) pairs behind the packed rows
            if out.stride(0) % 2 or out.data_ptr() % 4:          # the integer arm stores single values
                K.act_pack(xb, xp, xs, t, k, w.group)
                K.w4a16_skinny(w, xp, xs, out, t, ldo=out.stride(0))
                return out
            K.act_pack(xb, xp, xs, t, k, w.group | K.ACT_FRAG)
            K.w4_mma(w, xp, xs, out, t, ldo=out.stride(0))
            return out
        if _rows_ok(w, x, out, resident):
            return gemm_tc.w4_gemm_rows(w, x, out, pdl=pdl)
        if x.shape[0] >= DEQUANT_FROM:
            return gemm_tc.f16_gemm(x, w4_dense(w, x.dtype, x.device, resident=resident), out)
        return gemm_tc.w4a16_gemm(w, x, out)
    raise ValueError(f"unknown prefill GEMM arm {arm!r}")


def _e4m3_weight(w, device, resident: bool):
    """The weight as e4m3 rows with their scales: its resident copy (made on first use), or the shared scratch."""
    cached = getattr(w, "_owl_e4m3", None) if resident else None
    if cached is None:
        dense = K.w4_dequant(w, _dense_scratch(w.n, w.k, device, torch.float16))
        cached = gemm_tc.quant_e4m3_rows(dense) if resident else gemm_tc.quant_e4m3_rows(dense, *_fp8_scratch("w", w.n, w.k, device))
        if resident:
            _ledger(device).track("resident e4m3 weight copy", "resident copies", cached[0])
            w._owl_e4m3 = cached
    return cached


def w4_gemm_silu(w, x: torch.Tensor, out: torch.Tensor, arm: str = "tc", ahead: DequantAhead | None = None, pdl: bool = False) -> bool:
    """out[T, N/2] (fp16) = silu(gate) * up of the merged gate / up projection in one launch. False (and nothing done) where the
    arm or the shape has no such epilogue: the caller multiplies and activates in two steps. ``pdl``: as for ``w4_gemm``."""
    t = x.shape[0]
    if ahead is not None:
        if w.n < 512 or out.stride(0) % 8:
            return False
        dense = ahead.take(w)
        if dense is None:
            dense = w4_dense(w, x.dtype, x.device)
        gemm_tc.gemm_silu(x, dense, out)
        ahead.kick()
        return True
    if w.layout == "nvfp4" or x.dtype != torch.float16 or out.dtype != torch.float16 or out.stride(0) % 8:
        return False
    if arm in ("tc8", "tc8r") and t >= DEQUANT_FROM and w.k % 128 == 0:
        wq, sw = _e4m3_weight(w, x.device, arm == "tc8r")
        xq, sx = gemm_tc.quant_e4m3_rows(x, *_fp8_scratch("x", t, w.k, x.device))
        gemm_tc.gemm_silu(xq, wq, out, sx, sw)
        return True
    if arm in ("tc", "tc4", "tcr", "tc8", "tc8r") and t > SKINNY_UPTO and _rows_ok(w, x, out, arm in ("tcr", "tc8r")):
        gemm_tc.w4_gemm_rows(w, x, out, silu=True, pdl=pdl)
        return True
    if arm in ("tc", "tc4", "tcr", "tc8", "tc8r") and t >= SILU_FROM and w.n >= 512:
        gemm_tc.gemm_silu(x, w4_dense(w, x.dtype, x.device, resident=arm in ("tcr", "tc8r")), out)
        return True
    return False


def nvfp4_gemm(w, x: torch.Tensor, out: torch.Tensor, arm: str = "tc") -> torch.Tensor:
    """out[T, N] = x @ dequant(NVFP4 w)^T for a prefill chunk: the weight is dequantised once (bf16) and multiplied on the
    dense tcgen05 GEMM; ``"tc8"`` re-quantises rows to e4m3 and runs the 8-bit float product at twice the rate; ``"tc4"``
    (W4A4) quantises the chunk's activations to NVFP4 with one scale per token and multiplies codes by codes on the
    block-scaled tensor-core path (``ops/nvfp4_tc.py``), with no dense copy of the weight at all; a handful of rows take the
    streaming GEMV."""
    t = x.shape[0]
    if arm == "tc4":
        from . import nvfp4_tc

        if t >= nvfp4_tc.MIN_ROWS and w.k % 64 == 0:
            return nvfp4_tc.gemm(w, x, out)
    arm = {"tcr": "tc", "tc8r": "tc8", "tc4": "tc"}.get(arm, arm)       # no resident copies on this path
    if arm != "baseline" and t <= 8:
        K.nvfp4_linear_gemv(w, x if x.dtype == torch.bfloat16 else x.to(torch.bfloat16), out, t)
        return out
    dense = K.nvfp4_linear_dequant(w, _dense_scratch(w.n, w.k, x.device, torch.bfloat16))
    if arm == "baseline":
        torch.matmul(x.to(torch.bfloat16), dense.t(), out=out)
        return out
    if arm == "tc8" and t >= DEQUANT_FROM and w.k % 128 == 0:
        wq, sw = gemm_tc.quant_e4m3_rows(dense, *_fp8_scratch("w", w.n, w.k, x.device))
        xq, sx = gemm_tc.quant_e4m3_rows(x, *_fp8_scratch("x", t, w.k, x.device))
        return gemm_tc.e4m3_gemm(xq, sx, wq, sw, out)
    return gemm_tc.f16_gemm(x if x.dtype == torch.bfloat16 else x.to(torch.bfloat16), dense, out)


def w4_e4m3(w, device):
    """Resident per-row e4m3 copy of a W4 weight: (bytes [N, K], fp32 row scales [N]), created on first use."""
    cached = getattr(w, "_owl_e4m3", None)
    if cached is None:
        dense = K.w4_dequant(w, _dense_scratch(w.n, w.k, device, torch.float16))
        _ledger(device).check("resident e4m3 weight copy", w.n * w.k)
        cached = gemm_tc.quant_e4m3_rows(dense)
        _ledger(device).track("resident e4m3 weight copy", "resident copies", cached[0])
        w._owl_e4m3 = cached
    return cached


def w4_dense(w, dtype, device, resident: bool = False) -> torch.Tensor:
    """The weight dequantised into the shared dense scratch matrix (valid until the next call on this stream), or, with
    ``resident``, into a matrix of its own that stays attached to the weight."""
    if resident:
        d = getattr(w, "_owl_dense", None)
        if d is None or d.dtype != dtype:
            # 4x the int4 bytes: a named, budget-checked entry of the device ledger (a profile whose budget cannot hold
            # the copies is refused here, at the first chunk, instead of running the device out of memory later)
            d = K.w4_dequant(w, _ledger(device).alloc("resident dense weight copy", "resident copies", (w.n, w.k), dtype))
            w._owl_dense = d
        return d
    return K.w4_dequant(w, _dense_scratch(w.n, w.k, device, dtype))


def dense_gemm(x: torch.Tensor, w: torch.Tensor, out: torch.Tensor, arm: str = "tc", split: bool = False) -> torch.Tensor:
    """out[T, N] (bf16) = x @ w^T for a small dense bf16 weight (GDN a/b projections, draft heads). ``split``: cut k so that
    every SM has a part (the 96 rows of a / b are one or two tiles at a short prompt)."""
    if arm == "baseline":
        torch.matmul(x.to(w.dtype), w.t(), out=out)
        return out
    if x.dtype != w.dtype:
        # the converted copy lives on the weight tensor itself (a cache keyed by address would hand a stale copy to the
        # next tensor allocated at that address)
        cache = getattr(w, "_owl_cast", None)
        if cache is None or cache.dtype != x.dtype:
            cache = w.to(x.dtype)
            w._owl_cast = cache
        w = cache
    return gemm_tc.f16_gemm(x, w, out, force_persist=split)
