"""The BF16 GEMM on both sides of the rule that takes a long K with few row
tiles to the TMA ring (more than 10 chunks of 64, at most 8 row tiles): a
last slot filled by half (an odd number of chunks), several row tiles and
column tiles.  Integer-valued inputs, whose products and sums (below 2^24)
are exact in FP32, so the results are the reference's to the bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(128, 64, 640), (128, 64, 704), (128, 128, 768), (256, 128, 832), (1024, 64, 704),
                                   (1152, 64, 704), (128, 64, 4736)])
def test_gemm_is_exact_on_integers(M, N, K):
    from tapsim_modified_b200 import _native as N_
    rng = np.random.default_rng(M + N + K)
    a = rng.integers(-15, 16, (M, K)).astype(np.float32)
    b = rng.integers(-15, 16, (N, K)).astype(np.float32)
    bits = [np.ascontiguousarray((x.view(np.uint32) >> 16).astype(np.uint16)) for x in (a, b)]
    c = np.full((M, N), np.nan, np.float32)
    N_.check(N_.lib().tg_gemm_bf16(N_.ptr(bits[0]), N_.ptr(bits[1]), N_.ptr(c), M, N, K))
    assert np.array_equal(c, (a.astype(np.float64) @ b.astype(np.float64).T).astype(np.float32))
