"""The streaming projections through tensor memory (csrc/gemv_tm.cu): the tests of the warp-level form on this kernel, which takes the
same operands. Beside its tile edges: one and both sets of unpacking warps with work, one and two units a CTA, clusters of 1 to 8."""
import pytest
import torch

import test_gemv_mma_gpu as T
from owl_engine_b200.ops import kernels as K

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _through_tensor_memory(monkeypatch):
    monkeypatch.setattr(K, "w4_mma", K.w4_tm)
    monkeypatch.setattr(K, "ACT_FRAG", K.ACT_FRAG | K.ACT_TM)
    yield
    torch.cuda.synchronize()
    assert K.all_status()["stream_tc"] == 0


@pytest.mark.parametrize("fmt", ["g128", "g32", "nvfp4"])
@pytest.mark.parametrize("shape", [(16, 128), (144, 384), (256, 1152), (1040, 2176), (2080, 1280), (5120, 1152), (20480, 640), (40960, 128)])
@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32])
def test_streaming_matches_dequantised_product(fmt, shape, m):
    T.test_mma_streaming_matches_dequantised_product(fmt, shape, m)


@pytest.mark.parametrize("fmt,m", [("g128", 1), ("g32", 5), ("g128", 20), ("nvfp4", 3)])
def test_eight_bit_activations(fmt, m):
    T.test_eight_bit_activations(fmt, m)


@pytest.mark.parametrize("rows,m", [(16, 1), (96, 8), (32, 31)])
def test_dense_rows_beside_the_matrix(rows, m):
    T.test_dense_rows_beside_the_matrix(rows, m)


@pytest.mark.parametrize("fmt", ["g128", "nvfp4"])
def test_extremes_of_the_activations(fmt):
    T.test_extremes_of_the_activations(fmt)


@pytest.mark.parametrize("flags", [0, K.ACT_A8, K.ACT_NV])
@pytest.mark.parametrize("group", [128, 32])
@pytest.mark.parametrize("m", [1, 9])
def test_producers_write_the_blocks_of_their_outputs(flags, group, m):
    T.test_producers_write_the_fragments_of_their_outputs(flags, group, m)
