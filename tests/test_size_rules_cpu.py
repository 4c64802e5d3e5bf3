"""Size rules of the prompt and step paths (no GPU: the rules look at sizes only)."""
import ctypes
from types import SimpleNamespace

import pytest

from owl_engine_b200.models.hybrid import HybridRunner
from owl_engine_b200.models.spec import PRESETS
from owl_engine_b200.ops import gemm_tc, linear
from owl_engine_b200.ops import kernels as K


def _projections(name):
    sp = PRESETS[name]()
    out = []
    for i in range(sp.n_layers):
        shapes = ((2 * sp.hq * sp.hd + 2 * sp.hkv * sp.hd, sp.hidden), (sp.hidden, sp.hq * sp.hd)) if sp.is_full(i) else \
            ((sp.conv_dim + sp.value_dim, sp.hidden), (sp.hidden, sp.value_dim))
        out += [SimpleNamespace(n=n, k=k) for n, k in shapes + ((2 * sp.inter, sp.hidden), (sp.hidden, sp.inter))]
    return out


@pytest.mark.parametrize("model,t,pays", [("qwen3.8-27b", 257, True), ("qwen3.8-27b", 2048, True), ("qwen3.5-0.8b", 300, False),
                                          ("qwen3.5-0.8b", 1000, False), ("qwen3.5-0.8b", 2048, True)])
def test_small_models_do_not_pay_for_dequantising_ahead(model, t, pays):
    assert linear.ahead_pays(_projections(model), t) == pays


# up to 256 tokens the records, whether there is a copy or not (us, records / resident copy: 16384 x 5120 128 tokens 20 / 47, 255 35 / 50, 256
# 34 / 44; 5120 x 17408 256 44 / 58; 34816 x 5120 128 40 / 73); above, the copy where one is kept, and where a matrix is small
@pytest.mark.parametrize("n,k,t,resident,rows", [(16384, 5120, 256, False, True), (16384, 5120, 257, False, True), (1024, 3584, 256, False, True),
                                                 (16384, 5120, 256, True, True), (5120, 17408, 256, True, True), (5120, 17408, 255, True, True),
                                                 (16384, 5120, 255, True, True), (34816, 5120, 128, True, True), (34816, 5120, 129, True, True),
                                                 (16384, 5120, 127, True, True), (5120, 17408, 33, True, True), (16384, 5120, 257, True, False),
                                                 (1024, 1024, 257, False, True), (1024, 1008, 257, False, False), (1024, 1008, 256, False, True)])
def test_operand_of_a_short_prompt(n, k, t, resident, rows):
    assert linear.rows_pay(n, k, t, resident) == rows


# one chunk of up to 256 tokens; two of a matrix that leaves SMs idle, is not cut along k and whose steps get shorter; longer prompts
@pytest.mark.parametrize("t,n,k,plan", [(128, 1024, 3584, (1, 1, 128)), (129, 1024, 3584, (1, 2, 80)), (256, 1024, 3584, (1, 2, 128)),
                                        (256, 9472, 1024, (1, 2, 128)), (256, 9488, 1024, (1, 1, 256)), (256, 16384, 5120, (1, 1, 256)),
                                        (137, 5120, 6144, (3, 1, 144)), (256, 5120, 17408, (3, 1, 256)), (2048, 5120, 17408, (1, 11, 192))])
def test_chunks_and_parts_of_an_int4_product(t, n, k, plan):
    out = (ctypes.c_int * 3)()
    f = K.fn("owl_w4_gemm_rows_plan")
    assert f(t, n, k, 148, gemm_tc.KS_SCRATCH_BYTES, out) == 0
    assert tuple(out) == plan


# (sequences, longest context, uniform rows) -> parts of a sequence's keys, 27B head geometry (4 kv heads)
@pytest.mark.parametrize("b,ctx,uniform,parts", [(1, 2048, False, 32), (8, 8192, False, 9), (15, 8192, False, 4), (16, 8192, False, 9),
                                                 (16, 2048, False, 4), (16, 2304, False, 9), (24, 2048, False, 6), (32, 1024, False, 4),
                                                 (32, 1008, False, 2), (32, 8192, True, 9), (32, 16, False, 1)])
def test_parts_of_the_keys(b, ctx, uniform, parts):
    r = SimpleNamespace(attn_splits=0, uniform_rows=uniform, max_splits=64, spec=PRESETS["qwen3.8-27b"]())
    assert HybridRunner._pick_splits(r, b, ctx) == parts


# projections through tensor memory: four blocks of 8 rows (three for a large NVFP4 model), never in a speculating engine
@pytest.mark.parametrize("layout,model,m,uniform,tm", [("slice", "qwen3.8-27b", 24, False, False), ("slice", "qwen3.8-27b", 25, False, True),
                                                       ("slice", "qwen3.8-27b", 32, True, False), ("slice", "qwen3.5-0.8b", 32, False, True),
                                                       ("nvfp4", "qwen3.8-27b", 16, False, False), ("nvfp4", "qwen3.8-27b", 17, False, True),
                                                       ("nvfp4", "qwen3.5-0.8b", 17, False, False), ("nvfp4", "qwen3.5-0.8b", 25, False, True)])
def test_projections_through_tensor_memory(layout, model, m, uniform, tm):
    assert HybridRunner._tm(SimpleNamespace(uniform_rows=uniform, w=SimpleNamespace(layout=layout), spec=PRESETS[model]()), m) == tm
