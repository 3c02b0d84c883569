"""The W8A16 CTA-pair kernel (weights widened into tensor memory): token tiles, K slices, ragged edges, NaN codes."""
import numpy as np
import pytest
import torch

from oracle import fp8_oracle as O
from helpers import assert_parity, from_bf16, kernels, oracle_linear, run_linear, upload_case

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _defaults():
    yield
    for knob in ("w8a16_pair", "w8a16_pair_tokens", "w8a16_pair_splits"):
        kernels().set_tuning(knob, -1)


# (M, K, N, tokens per tile, slices); -1 = the planner's choice
@pytest.mark.parametrize("m,k,n,tokens,splits", [
    (65, 2048, 2048, -1, -1), (200, 3584, 1160, -1, -1), (255, 448, 584, -1, -1), (1031, 704, 1928, -1, -1),
    (1, 16, 8, 32, 1), (33, 144, 264, 32, 1), (96, 2064, 648, 96, 3), (130, 1408, 520, 64, 2), (224, 2048, 512, 224, 4), (257, 640, 264, 256, 2),
])
def test_pair_kernel_against_the_oracle(m, k, n, tokens, splits):
    Kn = kernels()
    Kn.set_tuning("w8a16_pair", 1)
    Kn.set_tuning("w8a16_pair_tokens", tokens)
    Kn.set_tuning("w8a16_pair_splits", splits)
    assert Kn.kernel_name(0, m, k, n).startswith("umma_w8a16_pair_256x")
    c = O.make_case(31 * m + k + n, m, k, n)
    d = upload_case(c)
    y = run_linear("fp8_w8a16", d)
    assert_parity(y, oracle_linear("fp8_w8a16", c), f"w8a16 pair {m}x{k}x{n} T={tokens} s={splits}")
    np.testing.assert_array_equal(y, run_linear("fp8_w8a16", d))
    assert_parity(run_linear("fp8_w8a16", d, bias=False), oracle_linear("fp8_w8a16", c, bias=False), f"no bias {m}x{k}x{n}")


def test_every_code_widens_exactly_and_nan_codes_stay_nan():
    """One-hot activations pick single weights: all 256 codes, the two NaN codes in a channel of their own."""
    Kn = kernels()
    Kn.set_tuning("w8a16_pair", 1)
    k, n = 128, 264
    codes = np.arange(n * k, dtype=np.int64).reshape(n, k) * 7 % 256
    codes[(codes & 0x7F) == 0x7F] = 0x33
    codes[5, 64] = 0x7F
    q = torch.from_numpy(codes.astype(np.uint8)).cuda()
    scale = torch.ones(n, device="cuda")
    y = from_bf16(Kn.launch_w8a16_gemm(torch.eye(k, dtype=torch.bfloat16, device="cuda"), Kn.pack_weight_nk(q), scale))
    want = q.view(torch.float8_e4m3fn).float().cpu().numpy().T
    finite = np.ones(n, bool)
    finite[5] = False
    np.testing.assert_array_equal(y[:, finite], want[:, finite])
    assert np.isnan(y[:, 5]).all()
