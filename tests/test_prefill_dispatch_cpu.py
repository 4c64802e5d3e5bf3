"""Size rules of the prompt path (no GPU: the rules look at sizes only)."""
from types import SimpleNamespace

import pytest

from owl_engine_b200.models.spec import PRESETS
from owl_engine_b200.ops import linear


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


@pytest.mark.parametrize("n,k,t,resident,rows", [(16384, 5120, 256, False, True), (16384, 5120, 257, False, False), (1024, 3584, 256, False, True),
                                                 (16384, 5120, 256, True, False), (5120, 17408, 256, True, False), (5120, 17408, 255, True, True),
                                                 (16384, 5120, 255, True, False), (34816, 5120, 128, True, False), (34816, 5120, 129, True, True),
                                                 (16384, 5120, 127, True, True), (5120, 17408, 33, True, True)])
def test_operand_of_a_short_prompt(n, k, t, resident, rows):
    assert linear.rows_pay(n, k, t, resident) == rows
