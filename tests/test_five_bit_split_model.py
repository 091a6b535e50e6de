"""Host model of the two-term operand split of the tcgen05 dequant-GEMM for int4 weights with f16 scales (tang_b200/csrc/qgemm_umma.cu):
    s_hi = scale rounded to five significant bits (half away from zero, on its f32 bits), s_lo = scale - s_hi,
    hi = fma(24 + q, s_hi, -24 s_hi), lo = fma(24 + q, s_lo, -24 s_lo), all in bf16.
The claim, for EVERY finite f16 scale and every q in -8..7: both parts of the scale, 24 times either, and both terms are bf16
numbers, so that no operation rounds and hi + lo = q * scale.  bf16 arithmetic is emulated in f64.  No GPU."""
import numpy as np

from test_hi_lo_split_model import rn_bf16


def test_both_terms_are_exact_for_every_f16_scale():
    bits = np.arange(1 << 16, dtype=np.uint16)
    scale = bits.view(np.float16).astype(np.float32)
    scale = scale[np.isfinite(scale)]
    s_hi = ((scale.view(np.uint32) + np.uint32(0x40000)) & np.uint32(0xFFF80000)).view(np.float32).astype(np.float64)
    s_lo = scale.astype(np.float64) - s_hi
    for s in (s_hi, s_lo):
        assert np.array_equal(rn_bf16(s), s)
        assert np.array_equal(rn_bf16(-24.0 * s), -24.0 * s)
    for q in range(-8, 8):
        hi, lo = rn_bf16((24.0 + q) * s_hi - 24.0 * s_hi), rn_bf16((24.0 + q) * s_lo - 24.0 * s_lo)
        assert np.array_equal(hi, q * s_hi) and np.array_equal(lo, q * s_lo)
        assert np.array_equal(hi + lo, q * scale.astype(np.float64)), q


def test_the_unpacked_integer_is_24_plus_q():
    """A nibble n = q + 8 in bits 3..6 of 0x4180 (bf16 16.0) is 16 + n."""
    n = np.arange(16, dtype=np.uint32)
    assert np.array_equal(((0x4180 | (n << 3)) << 16).astype(np.uint32).view(np.float32), 24.0 + (n.astype(np.float32) - 8.0))
