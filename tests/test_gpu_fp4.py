"""-m gpu: the small-tile fp4 GEMM form at the edges of its tiles - tokens per expert around 8, 16 and 32 (one MMA column
block of 8 or 16 tokens, two of 16, several tiles), K from a quarter of a stage to several, a ragged last feature tile - and
with everything its number format has no code for."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from gpu_common import DEV, gpu_layer, oracle_layer, to_np  # noqa: E402
from helpers import assert_close_bf16  # noqa: E402
from vkernels_b200 import synthetic as syn  # noqa: E402
from vkernels_b200 import torch_ops as ops  # noqa: E402


def _problem(H, I, counts, seed=3):
    """Expert e gets counts[e] tokens (top-1); weights, activations, ids, routing weights."""
    cfg = syn.scaled(syn.CONFIGS["c0"], H=H, I=I, E=len(counts), top_k=1)
    T = sum(counts)
    w = syn.make_expert_weights(cfg, seed=seed, device=DEV)
    A = syn.make_activations(cfg, T, seed=seed, device=DEV)
    rng = np.random.default_rng(seed)
    ids = rng.permutation(np.repeat(np.arange(len(counts)), counts)).astype(np.int32)[:, None]
    tw = (0.5 + rng.random((T, 1))).astype(np.float32)
    return w, A, torch.from_numpy(ids).to(DEV), torch.from_numpy(tw).to(DEV)


def _bf16_forms(w, A, ids, tw, **kw):
    """Outputs of the bf16-output form from the checkpoint layout and from prepacked weights."""
    E, I, H, T = w["w13"].shape[0], w["w13"].shape[1] // 2, A.shape[1], A.shape[0]
    sids, eids, _ = ops.moe_align_block_size(ids, E, 16)
    act = torch.zeros((sids.numel(), I), dtype=torch.bfloat16, device=DEV)
    y = [torch.full((T, H), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    args = (tw.reshape(-1).contiguous(), sids, eids)
    ops.fused_moe_mxfp4_bf16_into(y[0], act, A, w["w13"], w["w13_scale"], w["w2"], w["w2_scale"], *args, top_k=ids.shape[1], **kw)
    pk = ops.prepack_weights(w["w13"], w["w13_scale"], w["w2"], w["w2_scale"])
    if pk.usable:
        ops.fused_moe_mxfp4_bf16_prepacked_into(y[1], act, A, pk, *args, top_k=ids.shape[1], **kw)
    torch.cuda.synchronize()
    ops.kernel_status()
    return to_np(y[0].float()), to_np(y[1].float()) if pk.usable else None


@pytest.mark.parametrize("H,I", [(64, 64), (128, 320), (320, 192), (576, 2112)])
@pytest.mark.parametrize("counts", [(8,) * 2, (1, 0, 9, 3), (16, 7, 17), (31, 32, 33), (0, 70, 1)])
def test_tile_edges(H, I, counts):
    w, A, ids, tw = _problem(H, I, counts)
    w["w13_scale"][0, I + 3, -1] = 0xFF      # a zero group in an up row, one in a down row
    w["w2_scale"][-1, 7, 0] = 0xFF
    for kw in ({}, {"activation": 1}, {"swiglu_limit": 0.25}):
        ref = oracle_layer(A, w, ids, tw, **kw)
        got = to_np(gpu_layer(A, w, ids, tw, **kw))
        assert_close_bf16(got, ref, f"fp32 output {H} {I} {counts} {kw}")
        # The GEMMs are exact to fp32 rounding; what is left is the activation's rounding to bf16 falling the other way
        # for a few elements: at most one step of 2^-8 each.
        assert np.linalg.norm(got - ref) <= 2.0 ** -8 * np.linalg.norm(ref)
        if sum(counts) > 12:                 # (fewer slots take the flat kernels)
            for y in _bf16_forms(w, A, ids, tw, **kw):
                assert_close_bf16(y, ref, f"bf16 output {H} {I} {counts} {kw}", got_is_bf16=True)


@pytest.mark.parametrize("H,I", [(512, 4096), (4096, 192), (4800, 2112), (192, 7168)])
def test_several_items_a_cta(H, I):
    """Experts of one and two tiles and more items than CTAs: a CTA goes on to another tile, or to another feature tile of the
    same."""
    w, A, ids, tw = _problem(H, I, (40, 33, 3, 0, 20, 50))
    ref = oracle_layer(A, w, ids, tw)
    got = to_np(gpu_layer(A, w, ids, tw))
    assert np.linalg.norm(got - ref) <= 2.0 ** -8 * np.linalg.norm(ref)   # (the bound of test_tile_edges)
    for y in _bf16_forms(w, A, ids, tw):                                  # (and half a step of the bf16 result)
        assert np.linalg.norm(y - ref) <= (2.0 ** -8 + 2.0 ** -9) * np.linalg.norm(ref)


@pytest.mark.parametrize("M,k,E", [(4, 4, 1), (8, 4, 2), (8, 8, 3), (5, 3, 2)])
def test_an_expert_named_twice_by_a_token(M, k, E):
    """More rows in an expert than the batch has tokens: tiles of nine to sixteen rows, and several of them, in a batch of up
    to eight tokens."""
    H, I = 320, 192
    w, A, _, _ = _problem(H, I, (M,) + (0,) * (E - 1))
    rng = np.random.default_rng(M)
    ids = torch.from_numpy(rng.integers(0, E, (M, k)).astype(np.int32)).to(DEV)
    tw = torch.from_numpy((0.1 + rng.random((M, k))).astype(np.float32)).to(DEV)
    ref = oracle_layer(A, w, ids, tw)
    assert_close_bf16(to_np(gpu_layer(A, w, ids, tw)), ref, f"fp32 output {M} {k} {E}")
    for y in _bf16_forms(w, A, ids, tw):
        assert_close_bf16(y, ref, f"bf16 output {M} {k} {E}", got_is_bf16=True)


def test_real_rows_behind_padding():
    """A list whose blocks begin with padding: eight tokens, real rows in the last eight of sixteen."""
    H, I, M = 320, 192, 8
    w, A, ids, tw = _problem(H, I, (M,))
    sids = torch.cat([torch.full((8,), M), torch.arange(M)]).to(torch.int32).to(DEV)
    eids = torch.zeros(1, dtype=torch.int32, device=DEV)
    act = torch.zeros((16, I), dtype=torch.bfloat16, device=DEV)
    ref = oracle_layer(A, w, ids, tw)
    out = torch.zeros((M, H), dtype=torch.float32, device=DEV)
    ops.fused_moe_mxfp4_into(out, act, A, w["w13"], w["w13_scale"], w["w2"], w["w2_scale"], tw.reshape(-1), sids, eids, top_k=1)
    y = torch.empty((M, H), dtype=torch.bfloat16, device=DEV)
    pk = ops.prepack_weights(w["w13"], w["w13_scale"], w["w2"], w["w2_scale"])
    ops.fused_moe_mxfp4_bf16_prepacked_into(y, act, A, pk, tw.reshape(-1), sids, eids, top_k=1)
    torch.cuda.synchronize()
    ops.kernel_status()
    assert_close_bf16(to_np(out), ref, "checkpoint layout")
    assert_close_bf16(to_np(y.float()), ref, "prepacked", got_is_bf16=True)


@pytest.mark.parametrize("H,I", [(40064, 64), (40128, 64), (41792, 64), (64, 41792)])
def test_longest_reductions(H, I):
    """The scale bytes of an item next to three weight slots, and next to two."""
    counts = (9, 2, 5)
    w, A, ids, tw = _problem(H, I, counts)
    ref = oracle_layer(A, w, ids, tw)
    got = to_np(gpu_layer(A, w, ids, tw))
    assert np.linalg.norm(got - ref) <= 2.0 ** -8 * np.linalg.norm(ref)   # (the bound of test_tile_edges)


def _one_hot(rows, K, first=0):
    """[rows, K / 2] codes: row first + k holds a 1 (code 2) at k, everything else is zero."""
    codes = np.zeros((rows, K), np.uint8)
    codes[first + np.arange(K), np.arange(K)] = 2
    return codes[:, 0::2] | (codes[:, 1::2] << 4)


@pytest.mark.parametrize("lead", [(-133, -120), (-20, 20), (100, 121)])
def test_digit_planes_of_wide_range_rows(lead):
    """Both GEMMs made the identity (one-hot weights, a gate of 64 from its bias), so that what comes out is the token operand as
    its digit planes hold it: elements down to 2^-9 of the row's leading power of two exactly, smaller ones to half a unit of the
    integers, 2^-17 of it - in rows of subnormals, ordinary rows and rows up to the end of the bf16 range."""
    H = I = 256
    counts = (5, 20, 16)
    E, T = len(counts), sum(counts)
    w = {"w13": torch.from_numpy(np.stack([_one_hot(2 * I, H, I)] * E)).to(DEV), "w2": torch.from_numpy(np.stack([_one_hot(H, I)] * E)).to(DEV),
         "w13_scale": torch.full((E, 2 * I, H // 32), 127, dtype=torch.uint8, device=DEV),
         "w2_scale": torch.full((E, H, I // 32), 127, dtype=torch.uint8, device=DEV)}
    b13 = torch.zeros((E, 2 * I), device=DEV)
    b13[:, :I] = 64.0
    rng = np.random.default_rng(4)
    x = (1 + rng.integers(0, 128, (T, H)) / 128.0) * rng.choice([-1.0, 1.0], (T, H)) * 2.0 ** -rng.integers(0, 25, (T, H)).astype(np.float64)
    x[:, 7] = 1.5
    x *= 2.0 ** np.linspace(*lead, T).round()[:, None]
    A = torch.from_numpy(x).to(DEV).to(torch.bfloat16)
    ids = torch.from_numpy(rng.permutation(np.repeat(np.arange(E), counts)).astype(np.int32)[:, None]).to(DEV)
    tw = torch.ones((T, 1), device=DEV)

    def check(got, operand, gain, rounding, what, smallest=0.0):
        power = torch.exp2(torch.floor(torch.log2(operand.abs().amax(1, keepdim=True))))
        want = gain * operand
        exact = (operand.abs() >= power * 2.0 ** -9) & (want.abs() >= smallest)
        assert (operand != 0).any(1).all() and exact.any(1).all() and (lead[0] < -126 or not exact.all(1).any())
        assert torch.equal(got[exact], want[exact]), what
        # a bf16 result adds half a step of itself, or of the smallest subnormal
        bound = gain * power * 2.0 ** -17 + rounding * (2.0 ** -8 * want.abs() + 2.0 ** -134)
        assert ((got - want).abs() <= bound + torch.where(want.abs() < smallest, want.abs(), 0.0)).all(), what

    out, act, sids, _, _ = gpu_layer(A, w, ids, tw, b13=b13, return_parts=True)
    rows = torch.empty(T, dtype=torch.long, device=DEV)
    real = ((sids >= 0) & (sids < T)).nonzero().flatten()
    rows[sids[real].long()] = real
    act = act[rows].double()
    check(act, A.double(), 64.0, 1, "gate/up")
    check(out.double(), act, 1.0, 0, "down", smallest=2.0 ** -126)   # (red.global.add.f32 takes subnormals as zeros)
    sids, eids, _ = ops.moe_align_block_size(ids, E, 16)
    pk = ops.prepack_weights(w["w13"], w["w13_scale"], w["w2"], w["w2_scale"])
    act_p = torch.zeros((sids.numel(), I), dtype=torch.bfloat16, device=DEV)
    y = torch.empty((T, H), dtype=torch.bfloat16, device=DEV)
    ops.fused_moe_mxfp4_bf16_prepacked_into(y, act_p, A, pk, tw.reshape(-1), sids, eids, top_k=1, b13=b13)
    torch.cuda.synchronize()
    assert torch.equal(act_p[rows].double(), act)
    check(y.double(), act, 1.0, 1, "down, prepacked")


@pytest.mark.parametrize("code", [0x6, 0xE, 0x7])
@pytest.mark.parametrize("which", ["w13", "w2"])
def test_lone_nonfinite_codes(code, which):
    """One inf / NaN code (and one inside a zero group) in otherwise finite weights: the outputs that see it, and no
    others, are inf or NaN as in the CPU definition."""
    H, I, counts = 320, 192, (9, 17, 33)
    w, A, ids, tw = _problem(H, I, counts)
    A[3] = 0.0                                # inf * 0
    row, k = (I + 70, 257) if which == "w13" else (130, 100)
    w[which][1, row, k // 2] = (w[which][1, row, k // 2] & 0x0F) | (code << 4) if k & 1 else (w[which][1, row, k // 2] & 0xF0) | code
    w[which][2, 5, 0] = (w[which][2, 5, 0] & 0xF0) | code
    w[which + "_scale"][2, 5, 0] = 0xFF
    ref = oracle_layer(A, w, ids, tw)
    assert not np.isfinite(ref).all() and np.isfinite(ref).any()
    if which == "w13":   # an infinite activation enters the down GEMM as NaN in the fp4 form (VK_MOE_SMALL=bf16 keeps it inf)
        ref = np.where(np.isinf(ref), np.nan, ref)
    got = to_np(gpu_layer(A, w, ids, tw))
    assert_close_bf16(got, ref, f"{which} code {code}")
    y, packed = _bf16_forms(w, A, ids, tw)
    assert packed is None
    assert_close_bf16(y, ref, f"{which} code {code}, bf16 output", got_is_bf16=True)


def test_nonfinite_activations_poison_their_token_only():
    H, I, counts = 320, 192, (9, 17, 33)
    w, A, ids, tw = _problem(H, I, counts)
    A[2, 7] = float("nan")
    A[11, 300] = float("inf")
    got = to_np(gpu_layer(A, w, ids, tw))
    bad = np.zeros(A.shape[0], bool)
    bad[[2, 11]] = True
    assert np.isnan(got[bad]).all() and np.isfinite(got[~bad]).all()
