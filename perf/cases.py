"""What a user of the engine has it do, as cases that can be timed and compared: one step or one prompt through ``Engine`` or
``SpecRunner`` each, at the sizes of the shipped profiles (``configs/``), of ``bench.py`` and of the fixtures.

A case names the kind of pass (``decode``, ``spec``, ``prefill``, ``turn``), the model preset, the weight format (int4 groups of
128 or 32, NVFP4, int4 with 8-bit activations), the KV pool's format, the lm_head's and the rows and lengths. Every pass runs
the whole model, all layers, from the host's token ids to the logits.

Weights are random, with a residual stream as a trained network has it: it starts at the embedding's size and every layer adds
a small part to it (output projections drawn with std 0.02 / sqrt(2 layers), embedding rows with std 16). With equal scales
everywhere a random network of 64 layers is chaotic: two correct programs differ by 10 % in the logits. Caches of sequences that
are decoded or continued are filled with random values of the sizes a prompt leaves there.

Passes feed given token ids (``Engine.set_last_token``, as a host-side sampler does) instead of the model's own argmax: the
next pass then does not hang on which of two nearly equal logits is the larger. The logits come back whole; the sampled token
is their argmax and is not returned beside them.
"""
from __future__ import annotations

import math
from dataclasses import replace

import torch

from owl_engine_b200.engine.core import Engine, EngineConfig
from owl_engine_b200.engine.spec import SpecRunner
from owl_engine_b200.models import hybrid as H
from owl_engine_b200.models.spec import PRESETS
from owl_engine_b200.ops import quant as Q
from owl_engine_b200.utils.ledger import DeviceLedger, install

PAGE = 16
STEPS = 256          # decode passes until the sequences are taken back to the length they had at first


def listed():
    return [
        # the smallest call: one token of a 0.8B chat model with a short history, where launches and latency count
        dict(name="decode small model", kind="decode", model="qwen3.5-0.8b", weights="g128", kv="fp8", head="bf16", batch=1, ctx_lo=300, ctx_hi=300),
        # the headline: one stream of the 27B model behind a 2048-token prompt (bench.py)
        dict(name="decode 1", kind="decode", model="qwen3.8-27b", weights="g128", kv="fp8", head="int8", batch=1, ctx_lo=2048, ctx_hi=2048),
        # the same from an AWQ or GGUF Q4_K checkpoint (groups of 32) over the 16-bit pool
        dict(name="decode 1 group 32", kind="decode", model="qwen3.8-27b", weights="g32", kv="bf16", head="int8", batch=1, ctx_lo=1011, ctx_hi=1011),
        # a full step of the default profile: max_batch = 8 sessions of different lengths, bf16 head
        dict(name="decode 8", kind="decode", model="qwen3.8-27b", weights="g128", kv="fp8", head="bf16", batch=8, ctx_lo=400, ctx_hi=4000),
        # bench.py's 32 concurrent sessions with prompts of 1k to 8k tokens
        dict(name="decode 32", kind="decode", model="qwen3.8-27b", weights="g128", kv="fp8", head="int8", batch=32, ctx_lo=1024, ctx_hi=8192),
        # NVFP4 checkpoint, a few sessions over the int8 pool
        dict(name="decode 4 nvfp4", kind="decode", model="qwen3.8-27b", weights="nvfp4", kv="int8", head="int8", batch=4, ctx_lo=700, ctx_hi=3000),
        # a long agent session of the W4A8 profile between two tool calls, 128k tokens of history
        dict(name="decode 128k w4a8", kind="decode", model="qwen3.8-27b", weights="w4a8", kv="fp8", head="int8", batch=1, ctx_lo=131072, ctx_hi=131072),
        # one speculative round of 8 sessions, 3 drafts each, 2 of them accepted (verify, restore, fold), groups of 32
        dict(name="spec round 8x4", kind="spec", model="qwen3.8-27b", weights="g32", kv="fp8", head="int8", batch=8, depth=3, accept=2, ctx_lo=1024, ctx_hi=1536),
        # a short question: a prompt of 137 tokens
        dict(name="prefill 137", kind="prefill", model="qwen3.8-27b", weights="g32", kv="fp8", head="int8", tokens=137),
        # the headline's prompt: time to first token of 2048 tokens, default arm
        dict(name="prefill 2048", kind="prefill", model="qwen3.8-27b", weights="g128", kv="fp8", head="int8", tokens=2048),
        # a document of 8k tokens, four chunks: the largest pass
        dict(name="prefill 8192", kind="prefill", model="qwen3.8-27b", weights="g128", kv="fp8", head="int8", tokens=8192),
        # the next turn of a W4A8 agent session: 2k new tokens behind 32k cached ones (resident e4m3 copies of the weights)
        dict(name="turn 2k at 32k w4a8", kind="turn", model="qwen3.8-27b", weights="w4a8", kv="fp8", head="int8", tokens=2000, ctx=32768),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "spec", "prefill", "prefill", "turn"])
    # (a prompt's int8 codes are whole values that move by one wherever the keys differ in the third digit: the int8 pool is
    # drawn where a pass writes a few rows of it)
    pools = ["fp8", "fp8", "bf16"] + (["int8"] if kind in ("decode", "spec") else [])
    case = dict(kind=kind, model="qwen3.8-27b", weights=rng.choice(["g128", "g128", "g32"]), kv=rng.choice(pools),
                head=rng.choice(["int8", "int8", "bf16"]))
    if kind == "decode":
        case["model"] = rng.choice(["qwen3.8-27b", "qwen3.8-27b", "qwen3.8-27b", "qwen3.5-0.8b"])
        case["weights"] = rng.choice(["g128", "g128", "g32", "nvfp4", "w4a8"])
        case["batch"] = rng.choice([1, 1, 1, _log(rng, 2, 8), _log(rng, 8, 32)])
        case["ctx_hi"] = _log(rng, 150, 131072 if case["batch"] == 1 else 8192)
        case["ctx_lo"] = case["ctx_hi"] if case["batch"] == 1 else max(100, case["ctx_hi"] // rng.randint(1, 8))
    elif kind == "spec":
        case["depth"] = rng.randint(2, 7)
        case["batch"] = rng.randint(1, 32 // (case["depth"] + 1))
        case["accept"] = rng.randint(0, case["depth"])
        case["ctx_hi"] = _log(rng, 300, 8192)
        case["ctx_lo"] = max(100, case["ctx_hi"] // rng.randint(1, 4))
    elif kind == "prefill":
        case["weights"] = rng.choice(["g128", "g128", "g32", "w4a8"])
        case["tokens"] = _log(rng, 40, 8192)
    else:
        case["weights"] = rng.choice(["g128", "w4a8"])
        case["tokens"], case["ctx"] = _log(rng, 40, 2048), _log(rng, 1000, 65536)
    return case


BASE_LAYERS = 8      # layers drawn at random; the others hold the same records in another order (an equally random weight)


def _reordered(w, by):
    """The same weight with its records (NVFP4: its rows) moved on by ``by`` places, in memory of its own."""
    if isinstance(w, Q.NvFp4Linear):
        return replace(w, codes=w.codes.roll(by, 0), scales=w.scales.roll(by, 0))
    return replace(w, records=w.records.view(-1, w.rec_bytes).roll(by, 0).view(-1))


def _weights(case, seed):
    """Random device weights in the engine's layouts, scaled like a trained network's."""
    spec, dev = PRESETS[case["model"]](), torch.device("cuda:0")
    quant, group = ("nvfp4" if case["weights"] == "nvfp4" else "w4a16"), (32 if case["weights"] == "g32" else 128)
    w = H.random_weights(replace(spec, n_layers=BASE_LAYERS), dev, group=group, seed=seed, lm_head_int8=case["head"] == "int8", quant=quant)
    std = 0.02 / math.sqrt(2 * spec.n_layers)

    def small(old, s):
        if quant == "nvfp4":
            return Q.random_nvfp4(old.n, old.k, dev, std, s, group)
        return Q.random_skinny(old.n, old.k, group, dev, std, s, old.layout)
    for i, lw in enumerate(w.layers):
        s = seed * 1009 + 10 * i
        lw.down = small(lw.down, s)
        if lw.kind == "gdn":
            lw.out_proj = small(lw.out_proj, s + 1)
        else:
            lw.o_proj = small(lw.o_proj, s + 1)
    for i in range(BASE_LAYERS, spec.n_layers):
        base = w.layers[i % BASE_LAYERS]
        new = {nm: _reordered(getattr(base, nm), 37 * i) for nm in ("gate_up", "down", "qkvz", "out_proj", "qkv", "o_proj")
               if getattr(base, nm) is not None}
        if base.kind == "gdn":
            new.update(ab=replace(base.ab, records=base.ab.records.clone()), ab_dense=base.ab_dense.clone())
        w.layers.append(replace(base, **new))
    w.spec = spec
    # 8-bit activations round in steps of 6 %: a difference of a thousandth moves some of them to the next step, so the layers'
    # part is made smaller there, or two correct programs would drift apart over 64 layers
    w.embed.mul_(2400.0 if case["weights"] == "w4a8" else 800.0)
    return spec, w


def _fill(pool, gen):
    """Keys and values as a prompt leaves them (unit-size keys after their norm), and recurrent states."""
    dev = pool.device
    for p, std, scale in ((pool.k_pool, 1.0, pool.k_scale), (pool.v_pool, 1.5, pool.v_scale)):
        for i in range(p.shape[0]):
            x = torch.randn(p.shape[1:], device=dev, generator=gen)
            if scale is not None:
                p[i] = (x * 40.0).round_().clamp_(-127, 127).to(torch.int8).view(torch.uint8)
                scale[i] = std / 40.0 * (0.8 + 0.4 * torch.rand(scale.shape[1:], device=dev, generator=gen))
            elif p.dtype == torch.float16:
                p[i] = (x * std).bfloat16().half()
            else:
                p[i] = (x * std).to(torch.float8_e4m3fn).view(torch.uint8)
    for i in range(pool.rec_state.shape[0]):
        pool.rec_state[i].normal_(0.0, 0.01, generator=gen)
        pool.conv_state[i].normal_(0.0, 1.4, generator=gen)


def _lengths(case):
    """Cached tokens per sequence: from ``ctx_hi`` down to ``ctx_lo``."""
    b = case["batch"]
    return [case["ctx_hi"] - i * (case["ctx_hi"] - case["ctx_lo"]) // max(1, b - 1) for i in range(b)]


class _Drafts:
    """A draft source that proposes given tokens (the proposal is not the pass's subject: the target's verify is)."""

    def __init__(self, tokens):
        self.tokens = tokens

    def propose(self, engine, sid, depth):
        return self.tokens[sid][:depth]

    def observe(self, engine, sid, n_rows, emitted, row0=0):
        pass


def prepare(case, seed):
    """A booted engine: weights, pools, captured step graphs, and its sequences in the middle of their conversations."""
    rng = torch.Generator().manual_seed(seed)
    gen = torch.Generator(device="cuda:0").manual_seed(seed)
    spec, w = _weights(case, seed)
    kind, b = case["kind"], case.get("batch", 1)
    new = case.get("tokens", 0)
    if kind in ("decode", "spec"):
        lens = _lengths(case)
    else:
        lens = [case["ctx"]] if kind == "turn" else [0]
    room = [n + new + STEPS + 2 * PAGE for n in lens]
    spec_on = kind == "spec"
    cfg = EngineConfig(model=case["model"], group=w.group, quant="nvfp4" if case["weights"] == "nvfp4" else "w4a16",
                       act_bits=8 if case["weights"] == "w4a8" else 15, prefill_gemm="tc8r" if case["weights"] == "w4a8" else "tc",
                       lm_head_int8=case["head"] == "int8", kv_dtype=case["kv"], n_pages=sum(r // PAGE + 1 for r in room) + 32,
                       n_slots=b, n_snap_rows=2, max_seqs=b, max_seq=max(room), spec_rows=min(b, 8) if spec_on else 1, prefix_cache=False)
    eng = Engine(cfg, spec=spec, weights=w, device="cuda:0", ledger=install(DeviceLedger("cuda:0")))
    vocab = spec.vocab
    ids = lambda n: torch.randint(0, vocab, (n,), generator=rng).tolist()
    s = dict(case=case, eng=eng, at=0)
    if kind in ("prefill", "turn"):
        sid = eng.add_sequence(ids(160))              # an untimed first prompt: workspaces, resident copies
        eng.prefill(sid)
        eng.free_sequence(sid, publish=False)
        s["tokens"] = ids(new)
    if kind == "prefill":
        return s
    sids = []
    for n in lens:
        sid = eng.add_sequence(ids(n + 1))
        seq = eng.seqs[sid]
        eng._ensure_pages(seq, n + 1)
        seq.n_cached = n                              # n tokens cached, the last one not yet fed
        sids.append(sid)
    _fill(eng.pool, gen)
    s.update(sids=sids, lens=lens)
    if kind == "decode":
        hi = eng._ctx_bucket(max(lens) + 1)
        s["stream"] = torch.randint(0, vocab, (min(STEPS, hi - max(lens)), b), generator=rng).tolist()
        eng.runner.capture(b, 1, ctx_hint=hi)
    elif spec_on:
        rows = case["depth"] + 1
        s["anchors"] = ids(b)
        s["runner"] = SpecRunner(_Drafts({sid: ids(case["depth"]) for sid in sids}), depth=case["depth"], degrade_below=-1.0,
                                 force_accept=case["accept"])
        s["runner"].after_prefill(eng, sids[0])
        s["advance"] = case["accept"] + 1
        s["limit"] = max(1, min(STEPS, eng._ctx_bucket(max(lens) + rows) - max(lens) - rows) // s["advance"])
        run(s)                                        # captures the verify and fold graphs
    return s


def _rewind(s):
    for sid, n in zip(s["sids"], s["lens"]):
        seq = s["eng"].seqs[sid]
        del seq.tokens[n + 1:]
        seq.n_cached, seq.n_prompt = n, n + 1
    s["at"] = 0


def _pools(eng):
    p = eng.pool
    if p.k_scale is not None:
        kv = [p.k_pool.view(torch.int8), p.k_scale, p.v_pool.view(torch.int8), p.v_scale]
    elif p.k_pool.dtype == torch.float16:
        kv = [p.k_pool, p.v_pool]
    else:
        kv = [p.k_pool.view(torch.float8_e4m3fn), p.v_pool.view(torch.float8_e4m3fn)]
    return kv + [p.conv_state, p.rec_state]


def run(s):
    eng, kind = s["eng"], s["case"]["kind"]
    rows = 1
    if kind == "decode":
        if s["at"] == len(s["stream"]):
            _rewind(s)
        for sid, tok in zip(s["sids"], s["stream"][s["at"]]):
            eng.set_last_token(sid, tok)
        eng.decode_step(s["sids"])
        s["at"] += 1
        rows = len(s["sids"])
    elif kind == "spec":
        if s["at"] == s["limit"]:
            _rewind(s)
        for sid, tok in zip(s["sids"], s["anchors"]):
            eng.set_last_token(sid, tok)
        s["runner"].round_batch(eng, s["sids"])
        s["at"] += 1
        rows = len(s["sids"]) * (s["case"]["depth"] + 1)
        if len(s["sids"]) > eng.cfg.spec_rows:
            rows = (len(s["sids"]) % eng.cfg.spec_rows or eng.cfg.spec_rows) * (s["case"]["depth"] + 1)
    elif kind == "prefill":
        sid = eng.add_sequence(s["tokens"])
        eng.prefill(sid)
        eng.free_sequence(sid, publish=False)
    else:
        sid = s["sids"][0]
        eng.extend_sequence(sid, s["tokens"])
        _rewind(s)
    return [eng.runner.logits[:rows]] + _pools(eng)


def _linear(spec):
    """(rows, columns) of the projections of the GDN layers, of the attention layers, and of the MLP."""
    gdn = [(spec.conv_dim + spec.value_dim, spec.hidden), (spec.hidden, spec.value_dim)]
    full = [(2 * spec.hq * spec.hd + 2 * spec.hkv * spec.hd, spec.hidden), (spec.hidden, spec.hq * spec.hd)]
    mlp = [(2 * spec.inter, spec.hidden), (spec.hidden, spec.inter)]
    return spec.n_gdn * sum(n * k for n, k in gdn) + spec.n_full * sum(n * k for n, k in full) + spec.n_layers * sum(n * k for n, k in mlp)


def work(case):
    spec = PRESETS[case["model"]]()
    lin, head = _linear(spec), spec.vocab * spec.hidden
    ab = spec.n_gdn * 2 * spec.nv * spec.hidden
    per = {"g128": 0.5 + 4 / 128, "w4a8": 0.5 + 4 / 128, "g32": 0.5 + 4 / 32, "nvfp4": 0.5 + 1 / 16}[case["weights"]]
    nbytes = lin * per + ab * 2 + head * (1 if case["head"] == "int8" else 2)
    kvb = spec.kv_bytes_per_token(2 if case["kv"] == "bf16" else 1) + (spec.n_full * 2 * spec.hkv * 4 if case["kv"] == "int8" else 0)
    state = spec.gdn_state_bytes()
    kind, b = case["kind"], case.get("batch", 1)
    if kind in ("decode", "spec"):
        t = 1 + case.get("depth", 0)
        mean = case["ctx_hi"] if b == 1 else (case["ctx_hi"] + (b - 1) * (case["ctx_lo"] + case["ctx_hi"]) / 2) / b
        nbytes += b * (mean * kvb + 2 * state + t * spec.vocab * 2)
        flops = 2 * b * t * (lin + ab + head) + 4 * b * t * mean * spec.n_full * spec.hq * spec.hd
    else:
        t, ctx = case["tokens"], case.get("ctx", 0)
        nbytes += (ctx + t) * kvb + 2 * state
        pairs = t * ctx + t * (t + 1) / 2
        # the delta rule: per token and head, state times key, outer product, state times query
        flops = 2 * t * (lin + ab) + 2 * head + 4 * pairs * spec.n_full * spec.hq * spec.hd + 6 * t * spec.n_gdn * spec.nv * spec.kd * spec.vd
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # Measured by running every pass once more with its sums in another order or another form of the same precision: decode on the
    # integer arm against the half-precision one (logits 0.008 at 64 layers, states 0.004), prompts with the serial recurrence
    # instead of the chunked one, the warp-level attention instead of the fused one, or library GEMMs on bf16 operands (logits
    # 0.008 to 0.010, e4m3 keys and values 0.015 to 0.019, states 0.005 to 0.011). An int8 pool: the few rows a pass writes.
    return {"rel": 0.03, "differ": 0.01}
