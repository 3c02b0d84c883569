"""Prefill-sized expert batches: intermediate sizes that put the up channels inside a weight tile, chunk sizes at their
steps, experts without rows, ids without an expert; many passes in flight at once; and the activation in the epilogue."""
import importlib

import numpy as np
import pytest
import torch

from oracle import fp8_oracle as O
from helpers import assert_parity, from_bf16, kernels, to_bf16_cuda
from test_gpu_moe import make_moe_case, upload_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,H,I", [
    ([256, 257, 0, 33], 272, 144),          # full chunks, one row over, no rows, a part of a chunk; up rows inside a tile
    ([31, 700, 1, 288], 512, 192),          # 64-row steps of the up channels
    ([513, 64, 512, 95], 144, 16),          # the narrowest intermediate size
    ([128, 129, 400, 0], 272, 128),         # up channels at a tile: rows as the MMA's M in both projections, an odd last tile in down
])
def test_prefill_experts_against_the_oracle(counts, H, I):
    moe = importlib.import_module("nano-vllm-moe_b200.executor.moe")
    E, T = len(counts), sum(counts)
    assert T >= 512
    c = make_moe_case(T + I, T, H, I, E, 1)
    ids = np.repeat(np.arange(E), counts)
    ids = np.random.default_rng(I).permutation(ids).astype(np.int64)[:, None]
    w = np.random.default_rng(H).uniform(0.2, 1.0, (T, 1)).astype(np.float32)
    cfg = moe.make_moe_parallel_config(tp_group=None, ep_group=None, global_num_experts=E, intermediate_size=I)
    kern = moe.MoEKernel(prepare_finalize=moe.NoEPPrepareFinalize(cfg), experts=moe.Fp8Experts(), parallel_config=cfg)
    ref = O.moe_experts_w8a8(c["x"], ids, w, c["w13_q"], c["w13_s"], c["in13"], c["w2_q"], c["w2_s"], c["in2"])
    wts = upload_weights(moe, c)
    x, wt = to_bf16_cuda(c["x"]), torch.from_numpy(w).cuda()
    y = from_bf16(kern(x, wt, torch.from_numpy(ids).cuda(), wts, model_dtype=torch.bfloat16))
    assert_parity(y, ref, f"prefill experts {counts} H={H} I={I}", ulps=3.0, min_cos=0.9999)
    # a token whose expert is not here gets nothing, the others the same bits
    ids[::7] = -1
    y2 = from_bf16(kern(x, wt, torch.from_numpy(ids).cuda(), wts, model_dtype=torch.bfloat16))
    assert (y2[::7] == 0).all()
    keep = np.ones(T, bool)
    keep[::7] = False
    np.testing.assert_array_equal(y2[keep], y[keep])
    assert kernels().read_status(torch.device("cuda", 0)) == 0


@pytest.mark.parametrize("T,H,E,I,k", [(1024, 512, 8, 384, 4), (700, 272, 5, 144, 4)])       # rows as M; channels as M
def test_passes_in_flight_give_the_bits_of_single_passes(T, H, E, I, k):
    """A serving loop never waits between blocks: every kernel of the chain starts under its predecessor, in the next pass too."""
    moe = importlib.import_module("nano-vllm-moe_b200.executor.moe")
    cfg = moe.make_moe_parallel_config(tp_group=None, ep_group=None, global_num_experts=E, intermediate_size=I)
    kern = moe.MoEKernel(prepare_finalize=moe.NoEPPrepareFinalize(cfg), experts=moe.Fp8Experts(), parallel_config=cfg)
    router = moe.SoftmaxTopKRouter(k, False)
    c = make_moe_case(T + I, T, H, I, E, k)
    wts = upload_weights(moe, c)
    gen = torch.Generator(device="cuda").manual_seed(T)
    inputs = [(torch.randn(T, H, generator=gen, device="cuda").bfloat16(), torch.randn(T, E, generator=gen, device="cuda").bfloat16())
              for _ in range(3)]

    def one_pass(x, logits):
        w, ids = router.select_experts(x, logits)
        return kern(x, w, ids, wts, model_dtype=torch.bfloat16)

    single = []
    for x, logits in inputs:
        single.append(one_pass(x, logits))
        torch.cuda.synchronize()
    last = [one_pass(*inputs[i % 3]) for i in range(300)][-6:]
    torch.cuda.synchronize()
    for i, y in enumerate(last):
        assert torch.equal(y, single[(294 + i) % 3])
    assert kernels().read_status(torch.device("cuda", 0)) == 0


@pytest.mark.parametrize("counts,H,I", [
    ([3, 0, 16, 17], 272, 144),             # 16-row chunks, gathered rows; up rows inside a tile
    ([30, 1, 33, 25], 144, 16),             # 32-row chunks, the narrowest intermediate size
    ([100, 64, 65, 1], 512, 192),           # 64
    ([200, 129], 256, 64),                  # 128
    ([4] * 130, 144, 48),                   # 16-row chunks of pre-quantised rows
])
def test_fused_activation_equals_the_separate_pass(counts, H, I):
    moe = importlib.import_module("nano-vllm-moe_b200.executor.moe")
    Kn = kernels()
    E, T = len(counts), sum(counts)
    c = make_moe_case(T + I, T, H, I, E, 1)
    ids = torch.from_numpy(np.random.default_rng(I).permutation(np.repeat(np.arange(E), counts)).astype(np.int64)[:, None]).cuda()
    w = torch.rand((T, 1), device="cuda") + 0.2
    cfg = moe.make_moe_parallel_config(tp_group=None, ep_group=None, global_num_experts=E, intermediate_size=I)
    kern = moe.MoEKernel(prepare_finalize=moe.NoEPPrepareFinalize(cfg), experts=moe.Fp8Experts(), parallel_config=cfg)
    wts, x = upload_weights(moe, c), to_bf16_cuda(c["x"])
    y = kern(x, w, ids, wts, model_dtype=torch.bfloat16)
    try:
        Kn.set_tuning("moe_fused", 0)
        assert torch.equal(y, kern(x, w, ids, wts, model_dtype=torch.bfloat16))
    finally:
        Kn.set_tuning("moe_fused", -1)
    assert Kn.read_status(torch.device("cuda", 0)) == 0


def test_silu_equals_the_division_for_every_bf16_value(pkg):
    """The epilogues refine an approximate reciprocal instead of dividing; no value may differ, also not in the sign of a zero."""
    L = pkg._lib
    g = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).cuda()
    fast, divided = torch.empty(65536, device="cuda"), torch.empty(65536, device="cuda")
    L.raise_for(L.load().fp8lin_debug_silu(g.data_ptr(), fast.data_ptr(), divided.data_ptr(), g.numel(),
                                           torch.cuda.current_stream().cuda_stream), "fp8lin_debug_silu")
    nan = divided.isnan()
    assert torch.equal(nan, fast.isnan())
    assert torch.equal(fast[~nan].view(torch.int32), divided[~nan].view(torch.int32))
    x = g.double()
    want = x / (1 + torch.exp(-x))
    ok = torch.isfinite(want) & (want.abs() > 1e-30)
    assert ((divided.double() - want).abs() <= 4e-7 * want.abs())[ok].all()              # 3 ulps: expf, the sum, the quotient
