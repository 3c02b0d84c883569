"""The W8A8 CTA-pair kernel with the rows as the MMA's N: token tiles, a smaller last tile, K slices in one pair and in a
cluster, ragged edges, the activation epilogue of the fused MLP, and the same bits as the kernels it stands in for."""
import numpy as np
import pytest
import torch

from oracle import fp8_oracle as O
from helpers import assert_parity, kernels, oracle_linear, run_linear, upload_case
from test_gpu_mlp import make_mlp_case, run_fused, upload_mlp

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _defaults():
    yield
    for knob in ("w8a8_pair", "w8a8_pair_tokens", "w8a8_pair_slices", "w8a8_pair_splits"):
        kernels().set_tuning(knob, -1)
    assert kernels().read_status(torch.device("cuda", 0)) == 0


# (M, K, N, tokens per tile, slices, slices of a cluster)
@pytest.mark.parametrize("m,k,n,tokens,slices,splits", [
    (1, 16, 8, 32, 1, 1), (33, 144, 264, 32, 1, 1), (96, 2064, 648, 96, 3, 3), (130, 1408, 520, 64, 2, 2), (224, 2048, 512, 224, 4, 4),
    (257, 640, 264, 256, 2, 1), (64, 4096, 4616, 64, 8, 1), (300, 2064, 1032, 128, 3, 1), (1031, 272, 520, 256, 1, 1), (513, 144, 4616, 128, 1, 1),
])
def test_pair_kernel_against_the_oracle(m, k, n, tokens, slices, splits):
    Kn = kernels()
    for knob, value in (("w8a8_pair", 1), ("w8a8_pair_tokens", tokens), ("w8a8_pair_slices", slices), ("w8a8_pair_splits", splits)):
        Kn.set_tuning(knob, value)
    assert Kn.kernel_name(1, m, k, n).startswith("umma_w8a8_pair_256x%d_s%d" % (tokens, slices))
    c = O.make_case(31 * m + k + n, m, k, n)
    d = upload_case(c)
    y = run_linear("fp8_w8a8_static", d)
    assert_parity(y, oracle_linear("fp8_w8a8_static", c), f"w8a8 pair {m}x{k}x{n} T={tokens} s={slices}")
    np.testing.assert_array_equal(y, run_linear("fp8_w8a8_static", d))
    assert_parity(run_linear("fp8_w8a8_static", d, bias=False), oracle_linear("fp8_w8a8_static", c, bias=False), f"no bias {m}x{k}x{n}")


@pytest.mark.parametrize("m,k,n", [(17, 2048, 1024), (64, 3584, 4608), (96, 2064, 1032), (200, 3584, 1160), (255, 448, 584), (1031, 704, 1928)])
def test_same_bits_as_the_kernels_it_stands_in_for(m, k, n):
    Kn = kernels()
    d = upload_case(O.make_case(m + k + n, m, k, n))
    Kn.set_tuning("w8a8_pair", 0)
    want = run_linear("fp8_w8a8_static", d)
    Kn.set_tuning("w8a8_pair", 1)
    np.testing.assert_array_equal(run_linear("fp8_w8a8_static", d), want)


@pytest.mark.parametrize("m,h,inter,tokens", [(17, 272, 128, 32), (64, 3584, 384, 32), (65, 2048, 384, 64), (300, 144, 256, 256), (515, 528, 640, 224)])
def test_mlp_epilogue_equals_the_other_kernels(m, h, inter, tokens):
    Kn = kernels()
    d = upload_mlp(*make_mlp_case(m + h, m, h, inter, 264), inter)
    Kn.set_tuning("w8a8_pair", 0)
    want = run_fused(d)
    Kn.set_tuning("w8a8_pair", 1)
    Kn.set_tuning("w8a8_pair_tokens", tokens)
    np.testing.assert_array_equal(run_fused(d), want)


@pytest.mark.parametrize("tokens", [32, 64])
@pytest.mark.parametrize("gate", [0.0, 30.0, 300.0, 1e4, 1e30, 3e38, float("inf"), float("nan")])
def test_mlp_epilogue_on_gates_of_any_size(gate, tokens):
    """Gates that overflow the exponential, zeros, infinities and NaN beside ordinary ones: the codes of the separate activation pass.  The
    rows lie orders of magnitude apart, so that those beside a row with a NaN stay finite."""
    Kn = kernels()
    m, h, inter = 64, 272, 256
    gu, down = make_mlp_case(23, m, h, inter, 264)
    gu["x"] = O.bf16_round((gu["x"] * 2.0 ** -(np.arange(m) % 8)[:, None]).astype(np.float32))
    gu["x"][5] = 0.0
    if np.isnan(gate):
        gu["x"][9::16, 3] = np.nan
    else:                                             # of the first channels, half of their up values with them
        gu["w_scale"][:16] *= np.float32(gate)
        gu["w_scale"][inter:inter + 8] *= np.float32(gate)
    d = upload_mlp(gu, down, inter)
    Kn.set_tuning("w8a8_pair", 0)
    want = run_fused(d)
    Kn.set_tuning("w8a8_pair", 1)
    Kn.set_tuning("w8a8_pair_tokens", tokens)
    got = run_fused(d)
    np.testing.assert_array_equal(got, want)          # (NaN equals NaN here)
    if np.isnan(gate):
        assert np.isnan(want[9::16]).all() and np.isfinite(np.delete(want, np.s_[9::16], 0)).all()
    elif np.isfinite(gate):
        assert np.isfinite(want[5]).all() and np.abs(want).max() > 0


@pytest.mark.parametrize("m,n,tokens", [(17, 72, 32), (47, 264, 32), (81, 584, 96), (160, 8, 160), (300, 648, 224)])
def test_results_stay_inside_the_output_matrix(m, n, tokens):
    """Boxes of 16 tokens and 64 channels, clipped at the last token and channel: rows of a wider, longer matrix keep what was there."""
    Kn = kernels()
    d = upload_case(O.make_case(m + n, m, 272, n))
    Kn.set_tuning("w8a8_pair", 0)
    want = Kn.launch_w8a8_gemm(d["x"], d["w_nk"], d["input_scale"], d["w_scale"], d["bias"])
    Kn.set_tuning("w8a8_pair", 1)
    Kn.set_tuning("w8a8_pair_tokens", tokens)
    around = torch.full((m + 40, n + 136), 7.0, dtype=torch.bfloat16, device="cuda")
    Kn.launch_w8a8_gemm(d["x"], d["w_nk"], d["input_scale"], d["w_scale"], d["bias"], out=around[:m, 64:64 + n])
    assert torch.equal(around[:m, 64:64 + n], want)
    around[:m, 64:64 + n] = 7.0
    assert (around == 7.0).all()
