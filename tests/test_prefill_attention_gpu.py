"""The tcgen05 prefill attention (tang_b200/csrc/gqa_prefill_umma.cu, from 1024 rows per KV head and sequence on) against f64: edges of the query
tiles of 128 rows and key tiles of 128, every group size, and cache rows behind the last key that hold NaN."""
import numpy as np
import pytest

from util import bf16_round, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    import tang_b200

    d = tang_b200.QuantComputeDevice(0)
    yield d
    d.close()


@pytest.mark.parametrize("nh,nkv,q_len,starts", [(8, 8, 1024, [0]), (4, 2, 513, [0, 1]), (8, 2, 256, [0, 127, 128]), (8, 2, 257, [383]), (16, 2, 129, [0, 255]),
                                                 (8, 1, 383, [1]), (32, 8, 640, [0])])
@pytest.mark.parametrize("f32", [False, True])
def test_edges_of_query_and_key_tiles(dev, orc, nh, nkv, q_len, starts, f32):
    import tang_b200 as tb

    B, hd, behind = len(starts), 128, 70
    rng = np.random.default_rng(nh * q_len)
    max_seq = max(starts) + q_len + behind
    qb, qf = bf16_round(rng.standard_normal((B, q_len, nh * hd)).astype(np.float32))
    kb, kf = bf16_round(rng.standard_normal((B, max_seq, nkv * hd)).astype(np.float32))
    vb, vf = bf16_round(rng.standard_normal((B, max_seq, nkv * hd)).astype(np.float32))
    for b in range(B):
        kb[b, starts[b] + q_len:] = 0x7FC0            # never written rows may hold anything
        vb[b, starts[b] + q_len:] = 0x7FC0
    got = dev.gqa_prefill(dev.upload(qb, tb.BF16), dev.upload(kb, tb.BF16), dev.upload(vb, tb.BF16), np.array(starts, np.int32), B, q_len, nh, nkv, hd,
                          max_seq * nkv * hd, out_dtype=tb.F32 if f32 else tb.BF16).to_vec().reshape(B, q_len, nh * hd)
    dev.sync()
    if not f32:
        got = (got.astype(np.uint32) << 16).view(np.float32)
    assert np.isfinite(got).all()
    per = 128 // (nh // nkv)
    pick = sorted({0, 1, per - 1, per, 2 * per - 1, min(2 * per, q_len - 1), q_len // 2, q_len - 2, q_len - 1})
    for b in range(B):
        for i in pick:
            n = starts[b] + i + 1
            want = orc.attention_decode_f64(qf[b, i], kf[b, :n], vf[b, :n], n, nh, nkv, hd)
            # probabilities (and bf16 results) are rounded to 2^-9 of themselves: the bf16 bar of the interface
            assert rel_err(got[b, i], want, floor_frac=1.0) < 1e-2, (b, i)


def test_a_chunk_beyond_the_cache_is_reported(dev):
    import tang_b200 as tb

    nh, nkv, hd, q_len, max_seq = 8, 2, 128, 256, 300
    z = lambda *s: dev.upload(np.zeros(s, np.uint16), tb.BF16)
    dev.gqa_prefill(z(1, q_len, nh * hd), z(1, max_seq, nkv * hd), z(1, max_seq, nkv * hd), np.array([45], np.int32), 1, q_len, nh, nkv, hd, max_seq * nkv * hd)
    with pytest.raises(tb.TangqError):
        dev.sync()
    dev.sync()


@pytest.mark.parametrize("nh,nkv,q_len,start", [(8, 2, 320, 0), (8, 8, 1024, 3), (8, 1, 200, 100)])
@pytest.mark.parametrize("f32", [False, True])
def test_values_that_are_not_finite_reach_the_rows_that_see_them(dev, orc, nh, nkv, q_len, start, f32):
    """An infinity and a NaN in the values of two keys of the chunk: the positions before each do not see it, though they share tiles with it."""
    import tang_b200 as tb

    hd, per = 128, 256 // (nh // nkv)
    rng = np.random.default_rng(q_len)
    n = start + q_len
    qb, qf = bf16_round(rng.standard_normal((q_len, nh * hd)).astype(np.float32))
    kb, kf = bf16_round(rng.standard_normal((n, nkv * hd)).astype(np.float32))
    vb, vf = bf16_round(rng.standard_normal((n, nkv * hd)).astype(np.float32))
    at_inf, at_nan = start + per - 2, start + per + per // 2
    vb[at_inf, 5::hd], vf[at_inf, 5::hd] = 0x7F80, np.inf
    vb[at_nan, 9::hd], vf[at_nan, 9::hd] = 0x7FC0, np.nan
    got = dev.gqa_prefill(dev.upload(qb, tb.BF16), dev.upload(kb, tb.BF16), dev.upload(vb, tb.BF16), np.array([start], np.int32), 1, q_len, nh, nkv, hd,
                          n * nkv * hd, out_dtype=tb.F32 if f32 else tb.BF16).to_vec().reshape(q_len, nh, hd)
    dev.sync()
    if not f32:
        got = (got.astype(np.uint32) << 16).view(np.float32)
    pos = start + np.arange(q_len)
    sees = np.zeros((q_len, hd), bool)
    sees[pos >= at_inf, 5] = True
    sees[pos >= at_nan, 9] = True
    assert np.array_equal(~np.isfinite(got), np.broadcast_to(sees[:, None], got.shape))
    assert (got[pos >= at_inf, :, 5] == np.inf).all() and np.isnan(got[pos >= at_nan, :, 9]).all()
    vf[at_inf, 5::hd] = vf[at_nan, 9::hd] = 0
    for i in sorted({0, per - 3, per - 2, per - 1, per, at_nan - start - 1, at_nan - start, q_len - 1}):
        want = orc.attention_decode_f64(qf[i], kf[:start + i + 1], vf[:start + i + 1], start + i + 1, nh, nkv, hd).reshape(nh, hd)
        g = np.where(sees[i], want, got[i])
        assert rel_err(g, want, floor_frac=1.0) < 1e-2, i
