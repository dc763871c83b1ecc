"""The activation preparation of the tensor-core GEMM: one to eight tokens a CTA, 4 to 32 float4 a thread, two passes for the longest rows.

Tolerance: f16 roundings of both operands, NMSE about 2e-7 (bar of the GEMM: 1e-6).
"""
import numpy as np
import pytest

from oracle import sgref
from tests import util as U

pytestmark = pytest.mark.gpu


# eight, four, two tokens a CTA; one token with 4, 8, 16 and 32 float4 a thread (and just past each); two passes
@pytest.mark.parametrize("k", [96, 512, 544, 1024, 1056, 2048, 4096, 4128, 8192, 8224, 16384, 16416, 32768, 32800])
def test_row_lengths(sm100, stream, k):
    n, m = 24, 37
    wq = U.quantize(U.Q8_0, U.seeded_weights(k, n, k))
    x = U.seeded_acts(k, m, k)
    x[3] *= 1e6
    x[5] = 0.0
    x[7, k - 1] = 1e4   # the largest magnitude in the last element
    want = sgref.mul_mat(U.Q8_0, wq, k, x)
    got = U.device_mul_mat(sm100, stream, U.Q8_0, U.PACKED, wq, k, x)
    assert np.all(got[5] == 0.0)
    for t in [0, 3, 7, m - 1]:
        assert sgref.nmse(got[t], want[t]) <= 1e-6, t


# eight tokens a CTA (up to 64) and 32: one CTA's tokens, one more, one less; one block of K and several
@pytest.mark.parametrize("m", [33, 40, 41, 63, 64, 65, 96, 97, 128, 129, 160])
@pytest.mark.parametrize("k", [256, 1280])
def test_stage_images_of_q6_k_prompts(sm100, stream, k, m):
    """Both operands as two bf16 numbers: 16 bits each, NMSE (3e-5)^2 as for the split GEMM."""
    n = 32
    wq = U.quantize(U.Q6_K, U.seeded_weights(k, n, k))
    x = U.seeded_acts(m, m, k)
    want = sgref.mul_mat(U.Q6_K, wq, k, x)
    got = U.device_mul_mat(sm100, stream, U.Q6_K, U.PACKED, wq, k, x)
    for t in range(m):
        assert sgref.nmse(got[t], want[t]) <= 1e-9, t


# Row tiles of the GEMM: where it leaves few SMs, two, four and eight tokens a CTA, by the tokens; where it fills them (296) one; with 4 to 32 float4 a thread
@pytest.mark.parametrize("k", [1024, 2048, 4096, 8192, 8224])
@pytest.mark.parametrize("tiles,m", [(80, 37), (120, 100), (135, 64), (60, 250), (296, 45)])
def test_tokens_per_cta_beside_a_gemm(sm100, stream, tiles, m, k):
    """Every token on its own.  Rows repeat every 48, so that the oracle has few to multiply."""
    n = tiles * 128
    wq = U.quantize(U.Q4_0, U.seeded_weights(k, 48, k))
    x = U.seeded_acts(k + m, m, k)
    x *= np.float32(2.0) ** (np.arange(m, dtype=np.float32) % 7)[:, None]   # a factor taken from another token shows
    want = sgref.mul_mat(U.Q4_0, wq, k, x)
    got = U.device_mul_mat(sm100, stream, U.Q4_0, U.PACKED, np.ascontiguousarray(np.resize(wq, (n, wq.shape[1]))), k, x)
    assert np.array_equal(got, got[:, np.arange(n) % 48])
    for t in range(m):
        assert sgref.nmse(got[t, :48], want[t]) <= 1e-6, t


# more CTAs of the preparation than there are free SMs in the last wave of the GEMM before it: eight tokens each with 32 float4 a thread, one wave of the GEMM and two
@pytest.mark.parametrize("k", [544, 1024, 2048, 4128])
@pytest.mark.parametrize("tiles,m", [(32, 500), (96, 700)])
def test_crowded_preparation(sm100, stream, tiles, m, k):
    test_tokens_per_cta_beside_a_gemm(sm100, stream, tiles, m, k)
