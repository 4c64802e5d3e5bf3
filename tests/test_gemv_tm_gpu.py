"""The streaming projections through tensor memory (csrc/gemv_tm.cu): the tests of the warp-level form on this kernel, which takes the
same operands. Beside its tile edges: one and both sets of unpacking warps with work, one and two units a CTA, clusters of 1 to 8."""
from dataclasses import replace

import pytest
import torch

import test_gemv_mma_gpu as T
from owl_engine_b200.ops import kernels as K
from owl_engine_b200.ops import quant as Q

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


def test_a_step_repeats_itself():
    """Weights from memory and not from L2 (eight equal copies in turn), each launch behind a norm that writes its activations: some
    ten thousand launches give one result. (The sums of the activations lie in a ring that copies refill behind eight reading warps; a
    slot given back before its last loads were through gave a wrong value to 4 tokens in one of about a thousand launches.)"""
    m, h, n, g = 32, 5120, 34816, 128 | K.ACT_FRAG
    gen = torch.Generator(device="cuda").manual_seed(1)
    w = Q.random_skinny(n, h, 128, "cuda", 0.02, 5)
    ws = [replace(w, records=w.records.clone()) for _ in range(8)]
    x, gamma = torch.randn(m, h, device="cuda", generator=gen).bfloat16(), torch.zeros(h, dtype=torch.bfloat16, device="cuda")      # 1 + gamma
    xp = torch.empty(32 * 2 * h, dtype=torch.uint8, device="cuda")
    xs = torch.empty(32 * h // 128 * 8, dtype=torch.uint8, device="cuda")
    out = torch.zeros(16, m, n, dtype=torch.bfloat16, device="cuda")

    def chain():
        for i in range(out.shape[0]):
            K.rmsnorm_pack(x, gamma, xpack=xp, xs=xs, m=m, k=h, group=g, eps=1e-6)
            K.w4_mma(ws[i % 8], xp, xs, out[i], m, ldo=n, pdl=True)
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        chain()
        st.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            chain()
        want = out[0].clone()
        wrong = torch.zeros((), dtype=torch.int64, device="cuda")
        for _ in range(640):
            graph.replay()
            wrong += (out != want).flatten(1).any(1).sum()
        st.synchronize()
    assert int(wrong) == 0
    dense = K.w4_dequant(w, torch.empty(n, h, dtype=torch.float16, device="cuda"))
    a = torch.nn.functional.rms_norm(x.float(), (h,), eps=1e-6).bfloat16().float()
    assert ((want.float() - a @ dense.float().t()).norm() / want.float().norm()) < 0.01
