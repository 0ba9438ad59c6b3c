"""-m gpu: the CTA-pair GEMM form at the edges of its token tiles - one box of 16 rows up to two of 128 and 32 a CTA, with and
without extension rows, one tile to several - and K that ends inside a 128-K stage."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from gpu_common import DEV, gpu_layer, oracle_layer, to_np  # noqa: E402
from helpers import assert_close_bf16  # noqa: E402
from vkernels_b200 import synthetic as syn  # noqa: E402
from vkernels_b200 import torch_ops as ops  # noqa: E402
from vkernels_b200.vllm_experts import B200FusedExperts  # noqa: E402


@pytest.mark.parametrize("H,I", [(64, 192), (320, 64), (192, 448)])
@pytest.mark.parametrize("counts", [(257, 1, 150), (320, 321), (289, 33, 256), (700, 16)])
@pytest.mark.parametrize("kw", [{}, {"activation": 1}, {"swiglu_limit": 0.25}])
def test_pair_tile_edges(H, I, counts, kw):
    cfg = syn.scaled(syn.CONFIGS["c0"], H=H, I=I, E=len(counts), top_k=1)
    T = sum(counts)
    w = syn.make_expert_weights(cfg, seed=5, device=DEV)
    A = syn.make_activations(cfg, T, seed=5, device=DEV)
    rng = np.random.default_rng(5)
    ids = torch.from_numpy(rng.permutation(np.repeat(np.arange(len(counts)), counts)).astype(np.int32)[:, None]).to(DEV)
    tw = torch.from_numpy((0.5 + rng.random((T, 1))).astype(np.float32)).to(DEV)
    b13 = torch.from_numpy(0.1 * rng.standard_normal((len(counts), 2 * I)).astype(np.float32)).to(DEV)
    b2 = torch.from_numpy(0.1 * rng.standard_normal((len(counts), H)).astype(np.float32)).to(DEV)
    got = to_np(gpu_layer(A, w, ids, tw, b13=b13, b2=b2, **kw))
    ref = oracle_layer(A, w, ids, tw, b13=to_np(b13), b2=to_np(b2), **kw)
    assert_close_bf16(got, ref, f"pair {H} {I} {counts} {kw}")


@pytest.mark.parametrize("H,I", [(64, 192), (320, 64)])
@pytest.mark.parametrize("counts", [(257, 1, 150), (289, 33, 256), (700, 16)])
def test_ordered_output_adds_the_down_bias_once(H, I, counts):
    """Above some 48 tokens an expert the bf16-output entry point runs the CTA-pair form, which leaves plain rows to the
    combine: biases as large as the result, so that one left out or added twice is off by the size of the result."""
    cfg = syn.scaled(syn.CONFIGS["c0"], H=H, I=I, E=len(counts), top_k=1)
    T = sum(counts)
    w = syn.make_expert_weights(cfg, seed=6, device=DEV)
    A = syn.make_activations(cfg, T, seed=6, device=DEV)
    rng = np.random.default_rng(6)
    ids = torch.from_numpy(rng.permutation(np.repeat(np.arange(len(counts)), counts)).astype(np.int32)[:, None]).to(DEV)
    tw = torch.from_numpy((0.5 + rng.random((T, 1))).astype(np.float32)).to(DEV)
    b13 = torch.from_numpy(0.1 * rng.standard_normal((len(counts), 2 * I)).astype(np.float32)).to(DEV)
    b2 = torch.from_numpy(rng.standard_normal((len(counts), H)).astype(np.float32)).to(DEV)
    sids, eids, _ = ops.moe_align_block_size(ids, len(counts), 16)
    act = torch.zeros((sids.numel(), I), dtype=torch.bfloat16, device=DEV)
    y = torch.full((T, H), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.fused_moe_mxfp4_bf16_into(y, act, A, w["w13"], w["w13_scale"], w["w2"], w["w2_scale"], tw.reshape(-1), sids, eids,
                                  top_k=1, b13=b13, b2=b2)
    torch.cuda.synchronize()
    ops.kernel_status()
    ref = oracle_layer(A, w, ids, tw, b13=to_np(b13), b2=to_np(b2))
    assert_close_bf16(to_np(y.float()), ref, f"ordered pair {H} {I} {counts}", got_is_bf16=True)


def test_experts_object_with_biases_on_a_prefill_batch():
    """The serving engine's call on a batch of 96 tokens an expert: the same path through ``apply``."""
    cfg = syn.scaled(syn.CONFIGS["c0"], H=256, I=128, E=8, top_k=2)
    T = 384
    w = syn.make_expert_weights(cfg, seed=7, device=DEV)
    A = syn.make_activations(cfg, T, seed=7, device=DEV)
    rng = np.random.default_rng(7)
    ids = torch.from_numpy(np.stack([rng.choice(cfg.E, 2, replace=False) for _ in range(T)]).astype(np.int32)).to(DEV)
    tw = torch.from_numpy((0.5 + rng.random((T, 2))).astype(np.float32)).to(DEV)
    b2 = torch.from_numpy(rng.standard_normal((cfg.E, cfg.H)).astype(np.float32)).to(DEV)
    experts = B200FusedExperts(w13_scale=w["w13_scale"], w2_scale=w["w2_scale"], w2_bias=b2, max_num_tokens=T)
    y = torch.empty((T, cfg.H), dtype=torch.bfloat16, device=DEV)
    experts.apply(y, A, w["w13"], w["w2"], tw, ids)
    torch.cuda.synchronize()
    ops.kernel_status()
    assert_close_bf16(to_np(y.float()), oracle_layer(A, w, ids, tw, b2=to_np(b2)), "apply, 96 tokens an expert", got_is_bf16=True)
