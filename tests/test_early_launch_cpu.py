"""Which prompt launches may start before the kernel in front of them is done (no GPU: the calls are recorded)."""
import re
from types import SimpleNamespace

import pytest
import torch

from owl_engine_b200.models.hybrid import HybridRunner
from owl_engine_b200.ops import gemm_tc, linear
from owl_engine_b200.ops import registry as R


@pytest.fixture
def calls(monkeypatch):
    made = []
    monkeypatch.setattr(gemm_tc, "ensure_scratch", lambda device: None)
    monkeypatch.setattr(gemm_tc, "_call", lambda device, name, *args: made.append((name, *args)))
    return made


def _operands(t=40, n=256, k=128):
    w = SimpleNamespace(layout="slice", n=n, k=k, group=128, records=torch.zeros(n // 16 * 1088, dtype=torch.uint8))
    return w, torch.zeros(t, k, dtype=torch.float16), torch.zeros(t, n, dtype=torch.bfloat16), torch.zeros(t, n // 2, dtype=torch.float16)


@pytest.mark.parametrize("given", [{}, {"pdl": False}, {"pdl": True}])
def test_records_are_read_early_only_where_the_caller_allows_it(calls, given):
    """The int4 GEMM reads its records before it waits for the kernel in front of it. That kernel may be the one that writes them, so
    an early launch is the caller's to ask for, as with the streaming projections."""
    w, x, out, act = _operands()
    gemm_tc.w4_gemm_rows(w, x, out, **given)
    linear.w4_gemm(w, x, out, **given)
    assert linear.w4_gemm_silu(w, x, act, **given)
    assert [c[0] for c in calls] == ["owl_w4_gemm_rows"] * 3
    assert all(c[-1] == int(given.get("pdl", False)) for c in calls)


@pytest.mark.parametrize("pdl", [False, True])
def test_runner_asks_for_early_launches_on_its_own_weights(calls, pdl):
    w, x, out, _ = _operands()
    HybridRunner._gemm(SimpleNamespace(prefill_gemm="tc", pdl=pdl), w, x, out)
    assert [c[-1] for c in calls] == [int(pdl)]


def test_both_sides_keep_one_limit_of_rows():
    text = (R.CSRC / "common.cuh").read_text()
    assert int(re.search(r"constexpr int DEP_ROWS = (\d+);", text).group(1)) == HybridRunner.PDL_UPTO
