"""-m gpu: the CTA-pair GEMM form at the edges of its token tiles - one box of 16 rows up to two of 128 and 32 a CTA, with and
without extension rows, one tile to several - and K that ends inside a 128-K stage."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from gpu_common import DEV, gpu_layer, oracle_layer, to_np  # noqa: E402
from helpers import assert_close_bf16  # noqa: E402
from vkernels_b200 import synthetic as syn  # noqa: E402


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
