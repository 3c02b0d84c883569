"""Expert batches on CTA pairs: the bits of the kernels that one CTA runs, at the edges of groups, MMA tiles, chunks and stretches."""
import importlib

import numpy as np
import pytest
import torch

from helpers import kernels, to_bf16_cuda
from test_gpu_moe import make_moe_case, upload_weights

pytestmark = pytest.mark.gpu


def block(E, I, T, H, seed):
    moe = importlib.import_module("nano-vllm-moe_b200.executor.moe")
    cfg = moe.make_moe_parallel_config(tp_group=None, ep_group=None, global_num_experts=E, intermediate_size=I)
    kern = moe.MoEKernel(prepare_finalize=moe.NoEPPrepareFinalize(cfg), experts=moe.Fp8Experts(), parallel_config=cfg)
    c = make_moe_case(seed, T, H, I, E, 1)
    return moe, kern, c


@pytest.mark.parametrize("counts,H,I,rows", [
    ([256, 257, 0, 33], 272, 144, 320),           # one MMA tile, two, a group and a row; up rows inside a weight tile
    ([320, 321, 31, 32, 1], 512, 192, 320),       # the longest chunk, two even ones; 64-row steps of the up channels
    ([700, 320], 256, 128, 320),                  # three work items for all pairs: cut between groups
    ([200, 500, 90], 144, 16, 32),                # one group per chunk, the narrowest intermediate size
    ([60] * 12 + [64, 65], 272, 272, 64),         # a lone last weight tile in down
    ([5, 17, 96, 40, 300] * 9, 144, 1040, 192),   # many work items, dealt out in turn
    ([290, 310, 320, 280] * 10, 128, 1024, 320),  # ... whose sums do not fit beside each other in tensor memory
])
def test_pairs_give_the_bits_of_one_cta(counts, H, I, rows):
    Kn = kernels()
    E, T = len(counts), sum(counts)
    _, kern, c = block(E, I, T, H, T + I)
    wts, x = upload_weights(importlib.import_module("nano-vllm-moe_b200.executor.moe"), c), to_bf16_cuda(c["x"])
    ids = torch.from_numpy(np.random.default_rng(I).permutation(np.repeat(np.arange(E), counts)).astype(np.int64)[:, None]).cuda()
    w = torch.rand((T, 1), device="cuda") + 0.2
    try:
        Kn.set_tuning("moe_pair", 0)
        want = kern(x, w, ids, wts, model_dtype=torch.bfloat16)
        Kn.set_tuning("moe_pair", rows)
        got = [kern(x, w, ids, wts, model_dtype=torch.bfloat16) for _ in range(3)]
    finally:
        Kn.set_tuning("moe_pair", -1)
    assert want.float().abs().max() > 0
    assert all(torch.equal(y, want) for y in got)
    assert Kn.read_status(torch.device("cuda", 0)) == 0


@pytest.mark.parametrize("pad,offset", [(0, 0), (2, 2), (1, 0), (0, 1)])       # the last two: no place for a 4-byte store
def test_output_rows_of_any_pitch_and_alignment(pkg, pad, offset):
    L, Kn = pkg._lib, kernels()
    lib = L.load()
    E, H, I, counts = 3, 256, 128, [300, 200, 100]
    T = sum(counts)
    moe, _, c = block(E, I, T, H, 11)
    wts, x = upload_weights(moe, c), to_bf16_cuda(c["x"])
    ids = torch.from_numpy(np.repeat(np.arange(E), counts).astype(np.int32)).cuda()
    w = torch.rand(T, device="cuda") + 0.2
    ws = torch.zeros(lib.fp8lin_moe_workspace_bytes(T, E, H, I), dtype=torch.uint8, device="cuda")

    def run(pad, offset):
        out = torch.full((offset + T * (H + pad),), 7.0, dtype=torch.bfloat16, device="cuda")
        rc = lib.fp8lin_moe_experts_w8a8(x.data_ptr(), H, 1, ids.data_ptr(), w.data_ptr(), T, wts.w13_packed.data_ptr(), wts.w13_scale.data_ptr(),
                                         wts.w13_input_scale.data_ptr(), wts.w2_packed.data_ptr(), wts.w2_scale.data_ptr(),
                                         wts.w2_input_scale.data_ptr(), E, H, I, out.data_ptr() + 2 * offset, H + pad, ws.data_ptr(), ws.numel(),
                                         torch.cuda.current_stream().cuda_stream)
        L.raise_for(rc, "fp8lin_moe_experts_w8a8")
        rows = out[offset:].view(T, H + pad)
        assert (out[:offset] == 7).all() and (rows[:, H:] == 7).all()
        return rows[:, :H].clone()

    try:
        Kn.set_tuning("moe_pair", 0)
        want = run(0, 0)
        Kn.set_tuning("moe_pair", 320)
        assert torch.equal(run(pad, offset), want)
    finally:
        Kn.set_tuning("moe_pair", -1)


@pytest.mark.parametrize("gate", [0.0, 30.0, 79.0, 81.0, 300.0, 1e30, float("inf"), float("nan")])
def test_gates_of_any_size_in_the_epilogue(gate):
    """Gates that overflow the exponential, zeros, infinities and NaN: the values of the separate activation pass."""
    Kn = kernels()
    E, H, I, counts = 3, 256, 144, [300, 290, 10]
    T = sum(counts)
    moe, kern, c = block(E, I, T, H, 5)
    wts, x = upload_weights(moe, c), to_bf16_cuda(c["x"])
    # the gates of expert 0's first channels, of either sign, grow by orders of magnitude; the others stay as they are
    wts.w13_scale[0, :16] *= gate
    wts.w13_scale[0, I:I + 8] *= gate                 # ... and half of their up values
    ids = torch.from_numpy(np.random.default_rng(3).permutation(np.repeat(np.arange(E), counts)).astype(np.int64)[:, None]).cuda()
    w = torch.rand((T, 1), device="cuda") + 0.2
    out = {}
    try:
        for name, knobs in {"pair": {"moe_pair": 320}, "one": {"moe_pair": 0}, "separate": {"moe_fused": 0}}.items():
            for k, v in knobs.items():
                Kn.set_tuning(k, v)
            out[name] = kern(x, w, ids, wts, model_dtype=torch.bfloat16)
            for k in knobs:
                Kn.set_tuning(k, -1)
    finally:
        Kn.set_tuning("moe_pair", -1)
        Kn.set_tuning("moe_fused", -1)
    for name in ("pair", "one"):
        assert torch.equal(out[name].isnan(), out["separate"].isnan()), name
        assert torch.equal(out[name].nan_to_num(0.0), out["separate"].nan_to_num(0.0)), name
    other = ids[:, 0] != 0
    assert torch.isfinite(out["pair"][other].float()).all()
    assert Kn.read_status(torch.device("cuda", 0)) == 0


@pytest.mark.parametrize("rows,x_div,E", [(512, 1, 3), (513, 5, 60), (1031, 4, 7), (70000, 3, 9), (2000, 600, 3000), (700, 2, 3071), (1500, 3, 1024), (9000, 1, 257), (300000, 300000, 3), (3000, 33, 5), (5000, 5000, 7), (20011, 1999, 40)])
def test_grouping_of_large_batches(pkg, rows, x_div, E):
    """Shares of whole tokens, a last one that is cut short, more than 128 times 512 rows, as many experts as there may be, one token with more
    slots than a rank inside a share can count: every routed row gets what it gets in a batch that one CTA groups."""
    L, Kn = pkg._lib, kernels()
    lib = L.load()
    H = I = 16
    gen = torch.Generator(device="cuda").manual_seed(rows)
    tokens = -(-rows // x_div)
    x = torch.randn(tokens, H, generator=gen, device="cuda").bfloat16()
    ids = torch.randint(-1, E + 1, (rows,), generator=gen, device="cuda", dtype=torch.int32)       # some of them no expert's here
    w = torch.rand(rows, generator=gen, device="cuda") + 0.2
    code = lambda *s: (torch.randn(*s, generator=gen, device="cuda") * 0.5).to(torch.float8_e4m3fn).view(torch.uint8)
    w13 = torch.cat([Kn.pack_weight_nk(code(2 * I, H)) for _ in range(min(E, 64))])
    w2 = torch.cat([Kn.pack_weight_nk(code(H, I)) for _ in range(min(E, 64))])
    if E > 64:                                                     # (the same 64 experts again and again)
        w13, w2 = (t.view(64, -1).repeat(-(-E // 64), 1)[:E].contiguous().view(-1) for t in (w13, w2))
    s13, s2 = torch.rand(E, 2 * I, generator=gen, device="cuda") + 0.5, torch.rand(E, H, generator=gen, device="cuda") + 0.5
    in13, in2 = torch.tensor(0.01, device="cuda"), torch.tensor(0.05, device="cuda")

    def run(x, x_div, ids, w):
        n = ids.numel()
        out = torch.zeros(n, H, dtype=torch.bfloat16, device="cuda")
        ws = torch.zeros(lib.fp8lin_moe_workspace_bytes(n, E, H, I), dtype=torch.uint8, device="cuda")
        L.raise_for(lib.fp8lin_moe_experts_w8a8(x.data_ptr(), H, x_div, ids.data_ptr(), w.data_ptr(), n, w13.data_ptr(), s13.data_ptr(), in13.data_ptr(), w2.data_ptr(),
                                                s2.data_ptr(), in2.data_ptr(), E, H, I, out.data_ptr(), H, ws.data_ptr(), ws.numel(),
                                                torch.cuda.current_stream().cuda_stream), "fp8lin_moe_experts_w8a8")
        torch.cuda.synchronize()
        return out

    got = run(x, x_div, ids, w)
    picked = torch.arange(rows, device="cuda")
    if rows > 4000:
        picked = torch.cat([picked[:511], picked[rows // 2:rows // 2 + 511], picked[-511:]])
    for part in picked.split(511):
        r = part.long()
        want = run(x[r // x_div].contiguous(), 1, ids[r].contiguous(), w[r].contiguous())
        assert torch.equal(got[r], want)
    assert (got[(ids < 0) | (ids >= E)] == 0).all() and got.float().abs().max() > 0
