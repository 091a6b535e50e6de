"""GPU parity of the MLA decode attention against the oracle (parity unpinned: the reference has no
MLA).  The oracle's absorbed form mirrors the device's two bf16 rounding points; its naive form
(keys and values materialised per head) checks the absorption algebra itself."""
import numpy as np
import pytest

from util import bf16_round, rel_err

C_, R_, NOPE, VD = 512, 64, 128, 128


@pytest.fixture(scope="module")
def dev():
    import tang_b200

    d = tang_b200.QuantComputeDevice(0)
    yield d
    d.close()


def make(rng, H, B, max_seq):
    w_qk = rng.integers(-127, 128, (H * C_, NOPE), dtype=np.int8)
    s_qk = rng.uniform(0.001, 0.01, H * C_).astype(np.float32)
    w_uv = rng.integers(-127, 128, (H * VD, C_), dtype=np.int8)
    s_uv = rng.uniform(0.001, 0.01, H * VD).astype(np.float32)
    qn = bf16_round(rng.standard_normal((B, H, NOPE)).astype(np.float32))
    qr = bf16_round(rng.standard_normal((B, H, R_)).astype(np.float32))
    cache = bf16_round(rng.standard_normal((B, max_seq, C_ + R_)).astype(np.float32))
    return w_qk, s_qk, w_uv, s_uv, qn, qr, cache


@pytest.mark.gpu
@pytest.mark.parametrize("H,B,lens", [(16, 1, [200]), (32, 3, [1, 64, 333]), (128, 2, [4096, 1000]), (16, 4, [65, 128, 129, 700])])
def test_mla_decode_matches_oracle(dev, orc, H, B, lens):
    import tang_b200 as tb

    rng = np.random.default_rng(H + B)
    max_seq = max(lens) + 2
    w_qk, s_qk, w_uv, s_uv, qn, qr, cache = make(rng, H, B, max_seq)
    wq = dev.upload_qarrays(tb.I8_ROW, w_qk, s_qk, H * C_, NOPE)
    wu = dev.upload_qarrays(tb.I8_ROW, w_uv, s_uv, H * VD, C_)
    out = tb.mla_decode(dev, wq, wu, dev.upload(qn[0], tb.BF16), dev.upload(qr[0], tb.BF16), dev.upload(cache[0], tb.BF16),
                        np.array(lens, np.int32), B, H, NOPE, VD, max_seq * (C_ + R_), max(lens))
    dev.sync()
    got = out.to_vec().reshape(B, H * VD)
    dims = orc.MlaDims(H, C_, NOPE, R_, VD)
    for b in range(B):
        want = orc.mla_decode_f64(dims, qn[1][b].astype(np.float64), qr[1][b].astype(np.float64), cache[0][b], lens[b],
                                  w_qk, s_qk, w_uv, s_uv, absorbed=True)
        # q_lat and o_lat pass through bf16 on both sides: a one-ulp flip there moves the result by a
        # fraction of a percent of its rms, so the bar is relative to max(|ref|, rms)
        assert rel_err(got[b], want, floor_frac=1.0) < 2e-3, (b, lens[b])


def test_absorbed_equals_naive_in_the_oracle(orc):
    rng = np.random.default_rng(3)
    H, ctx = 4, 37
    w_qk, s_qk, w_uv, s_uv, qn, qr, cache = make(rng, H, 1, ctx)
    dims = orc.MlaDims(H, C_, NOPE, R_, VD)
    # small queries keep the softmax smooth, so the check is about the algebra and not about how a peaky
    # softmax amplifies the absorbed form's bf16 rounding of q_lat
    args = (dims, 0.05 * qn[1][0].astype(np.float64), 0.05 * qr[1][0].astype(np.float64), cache[0][0], ctx, w_qk, s_qk, w_uv, s_uv)
    a = orc.mla_decode_f64(*args, absorbed=True)
    n = orc.mla_decode_f64(*args, absorbed=False)
    assert rel_err(a, n, floor_frac=1.0) < 1e-2      # only the two bf16 roundings of the absorbed form apart


@pytest.mark.gpu
def test_head_shards_concatenate_to_the_full_result(dev, orc):
    """Tensor parallelism of MLA decode is by head with the latent cache replicated: running the two halves of
    the heads (their rows of W_UK / W_UV, their queries) separately gives the full output's halves bit for bit;
    only the row-parallel W_O that follows needs an all-reduce (tests/test_tp.py covers that pattern)."""
    import tang_b200 as tb

    rng = np.random.default_rng(77)
    H, B, lens = 32, 2, [300, 77]
    max_seq = max(lens) + 1
    w_qk, s_qk, w_uv, s_uv, qn, qr, cache = make(rng, H, B, max_seq)
    cbuf = dev.upload(cache[0], tb.BF16)

    def run(h0, h1):
        n = h1 - h0
        wq = dev.upload_qarrays(tb.I8_ROW, w_qk[h0 * C_:h1 * C_], s_qk[h0 * C_:h1 * C_], n * C_, NOPE)
        wu = dev.upload_qarrays(tb.I8_ROW, w_uv[h0 * VD:h1 * VD], s_uv[h0 * VD:h1 * VD], n * VD, C_)
        o = tb.mla_decode(dev, wq, wu, dev.upload(np.ascontiguousarray(qn[0][:, h0:h1]), tb.BF16),
                          dev.upload(np.ascontiguousarray(qr[0][:, h0:h1]), tb.BF16), cbuf, np.array(lens, np.int32), B, n, NOPE, VD,
                          max_seq * (C_ + R_), max(lens))
        dev.sync()
        return o.to_vec().reshape(B, n * VD)

    full = run(0, H)
    halves = np.concatenate([run(0, H // 2), run(H // 2, H)], axis=1)
    assert np.array_equal(full, halves)


@pytest.mark.gpu
@pytest.mark.parametrize("ctx,B", [(16384, 1), (32768, 1), (16384, 16)])
def test_mla_decode_long_contexts(dev, orc, ctx, B):
    """The benchmark's long contexts with all 128 heads; the oracle checks a seeded sample of the sequences."""
    import tang_b200 as tb

    H = 128
    rng = np.random.default_rng(ctx + B)
    max_seq = ctx
    w_qk = rng.integers(-127, 128, (H * C_, NOPE), dtype=np.int8)
    s_qk = rng.uniform(0.001, 0.01, H * C_).astype(np.float32)
    w_uv = rng.integers(-127, 128, (H * VD, C_), dtype=np.int8)
    s_uv = rng.uniform(0.001, 0.01, H * VD).astype(np.float32)
    qn = bf16_round(rng.standard_normal((B, H, NOPE)).astype(np.float32))
    qr = bf16_round(rng.standard_normal((B, H, R_)).astype(np.float32))
    lens = [ctx] + [int(v) for v in rng.integers(ctx // 2, ctx + 1, B - 1)]
    sample = [0] if B == 1 else [0, int(rng.integers(1, B))]
    cbuf = dev.alloc(B * max_seq * (C_ + R_), tb.BF16)
    kept = {}
    for b in range(B):                                         # sequence by sequence keeps the host arrays small
        cb = bf16_round(rng.standard_normal((max_seq, C_ + R_)).astype(np.float32))[0]
        dev._check(dev._L.tq_upload(dev._ctx, cbuf.ptr + b * max_seq * (C_ + R_) * 2, cb.ctypes.data, cb.nbytes))
        if b in sample:
            kept[b] = cb
    wq = dev.upload_qarrays(tb.I8_ROW, w_qk, s_qk, H * C_, NOPE)
    wu = dev.upload_qarrays(tb.I8_ROW, w_uv, s_uv, H * VD, C_)
    out = tb.mla_decode(dev, wq, wu, dev.upload(qn[0], tb.BF16), dev.upload(qr[0], tb.BF16), cbuf,
                        np.array(lens, np.int32), B, H, NOPE, VD, max_seq * (C_ + R_), max(lens))
    dev.sync()
    got = out.to_vec().reshape(B, H * VD)
    assert np.all(np.isfinite(got))
    dims = orc.MlaDims(H, C_, NOPE, R_, VD)
    for b in sample:
        want = orc.mla_decode_f64(dims, qn[1][b].astype(np.float64), qr[1][b].astype(np.float64), kept[b], lens[b],
                                  w_qk, s_qk, w_uv, s_uv, absorbed=True)
        assert rel_err(got[b], want, floor_frac=1.0) < 2e-3, (b, lens[b])


# ---- the MLA layer: q_a -> RMSNorm -> q_b -> RoPE -> absorbed attention -> W_UV -> row-parallel W_O ----------------
def _i8_matvec(w, s, x):
    """(w * s[:, None]) @ x in f64, a block of rows at a time (int8 weights, one f32 scale per row)."""
    out = np.empty(w.shape[0], np.float64)
    for r in range(0, w.shape[0], 2048):
        out[r:r + 2048] = (w[r:r + 2048].astype(np.float64) @ x) * s[r:r + 2048].astype(np.float64)
    return out


def _layer_weights(rng, d, H, q_lora):
    def mat(rows, cols):
        return rng.integers(-127, 128, (rows, cols), dtype=np.int8), rng.uniform(0.001, 0.01, rows).astype(np.float32)
    w = {"q_a": mat(q_lora, d), "q_b": mat(H * (NOPE + R_), q_lora), "w_qk": mat(H * C_, NOPE), "w_uv": mat(H * VD, C_),
         "w_o": mat(d, H * VD)}
    # a small gain keeps the queries (and with them the softmax) in a realistic range
    gain = bf16_round((0.03 * (1.0 + 0.1 * rng.standard_normal(q_lora))).astype(np.float32))
    return w, gain


def _layer_oracle(orc, w, gain, h, cache_b, length, H, heads, base, eps, max_pos):
    """Output of the heads in `heads` (a slice) for one sequence; the device's bf16 rounding points mirrored."""
    cq = _i8_matvec(*w["q_a"], h).astype(np.float32).astype(np.float64)
    xn = bf16_round(orc.rms_norm_f64(cq, gain[1].astype(np.float64), eps).astype(np.float32))[1].astype(np.float64)
    qh = NOPE + R_
    rows = slice(heads.start * qh, heads.stop * qh)
    q = bf16_round(_i8_matvec(w["q_b"][0][rows], w["q_b"][1][rows], xn).astype(np.float32))[1].reshape(-1, qh)
    nh = q.shape[0]
    cos, sin = orc.rope_tables_f32(R_, max_pos, base)
    pos = length - 1
    c, s = cos.reshape(max_pos, R_ // 2)[pos], sin.reshape(max_pos, R_ // 2)[pos]
    x0, x1 = q[:, NOPE::2], q[:, NOPE + 1::2]
    qr = np.empty((nh, R_), np.float32)
    qr[:, 0::2] = x0 * c - x1 * s
    qr[:, 1::2] = x0 * s + x1 * c
    qr = bf16_round(qr)[1]
    dims = orc.MlaDims(nh, C_, NOPE, R_, VD)
    hs = slice(heads.start * C_, heads.stop * C_)
    vs = slice(heads.start * VD, heads.stop * VD)
    o = orc.mla_decode_f64(dims, q[:, :NOPE].astype(np.float64), qr.astype(np.float64), cache_b, length, w["w_qk"][0][hs],
                           w["w_qk"][1][hs], w["w_uv"][0][vs], w["w_uv"][1][vs], absorbed=True)
    o = bf16_round(np.asarray(o, np.float32))[1].astype(np.float64)
    return _i8_matvec(np.ascontiguousarray(w["w_o"][0][:, vs]), w["w_o"][1], o)


def _make_layer(dev, tb, w, gain, d, H, heads, q_lora, max_batch, max_pos, base, eps):
    qh = NOPE + R_
    nh = heads.stop - heads.start
    up = lambda a, s, r, c: dev.upload_qarrays(tb.I8_ROW, np.ascontiguousarray(a), np.ascontiguousarray(s), r, c)
    cfg = tb.MlaConfig(d, nh, q_lora, C_, NOPE, R_, VD, max_batch, max_pos, eps)
    return tb.MlaLayer(
        dev, cfg, up(*w["q_a"], q_lora, d), dev.upload(gain[0], tb.BF16),
        up(w["q_b"][0][heads.start * qh:heads.stop * qh], w["q_b"][1][heads.start * qh:heads.stop * qh], nh * qh, q_lora),
        up(w["w_qk"][0][heads.start * C_:heads.stop * C_], w["w_qk"][1][heads.start * C_:heads.stop * C_], nh * C_, NOPE),
        up(w["w_uv"][0][heads.start * VD:heads.stop * VD], w["w_uv"][1][heads.start * VD:heads.stop * VD], nh * VD, C_),
        up(w["w_o"][0][:, heads.start * VD:heads.stop * VD], w["w_o"][1], d, nh * VD), rope_base=base)


@pytest.mark.gpu
@pytest.mark.parametrize("d,H,q_lora,B,lens", [(1024, 32, 512, 3, [5, 300, 64]), (7168, 128, 1536, 2, [700, 129]),
                                                (1024, 32, 512, 12, [40 + 17 * i for i in range(12)])])
def test_mla_layer_matches_oracle(dev, orc, d, H, q_lora, B, lens):
    """The whole layer at the DeepSeek-V3 widths (d_model 7168 is an assumption: the benchmark configuration names
    no hidden size), batches on both sides of the 8-row GEMV limit, and the heads split over two ranks' worth of
    weights whose outputs must add up to the unsharded result (the row-parallel W_O)."""
    import tang_b200 as tb

    rng = np.random.default_rng(d + H + B)
    base, eps, max_pos = 10000.0, 1e-6, max(lens) + 3
    max_seq = max(lens) + 2
    w, gain = _layer_weights(rng, d, H, q_lora)
    h = bf16_round(rng.standard_normal((B, d)).astype(np.float32))
    cache = bf16_round(rng.standard_normal((B, max_seq, C_ + R_)).astype(np.float32))
    hb, cb = dev.upload(h[0], tb.BF16), dev.upload(cache[0], tb.BF16)
    lb = dev.upload(np.array(lens, np.int32), tb.I32)
    full = _make_layer(dev, tb, w, gain, d, H, slice(0, H), q_lora, B, max_pos, base, eps)
    got = full.decode(hb, cb, lb, B, max_seq * (C_ + R_), max(lens))
    dev.sync()
    got = got.to_vec().reshape(B, d)
    for b in range(B if d < 7168 else 1):
        want = _layer_oracle(orc, w, gain, h[1][b].astype(np.float64), cache[0][b], lens[b], H, slice(0, H), base, eps, max_pos)
        # four bf16 hand-overs (c_q, q, q_lat, o_lat | o) on both sides: where the device's f32 sum and the oracle's
        # f64 sum land on different sides of a bf16 rounding boundary the result moves by a few 1e-3 of its rms
        # (observed: up to 3.6e-3); the bar is half of the 2e-2 allowed for bf16 outputs
        assert rel_err(got[b], want, floor_frac=1.0) < 1e-2, (b, lens[b])
    # two head shards, each with its rows of q_b / W_UK / W_UV and its columns of W_O: partial outputs add up
    parts = []
    for heads in (slice(0, H // 2), slice(H // 2, H)):
        layer = _make_layer(dev, tb, w, gain, d, H, heads, q_lora, B, max_pos, base, eps)
        o = layer.decode(hb, cb, lb, B, max_seq * (C_ + R_), max(lens))
        dev.sync()
        parts.append(o.to_vec().reshape(B, d).astype(np.float64))
        layer.destroy()
    # (a shard's projections have other shapes than the full layer's, so their f32 sums run in another order and a
    # bf16 hand-over can round the other way: a few 1e-3 of the rms on the rows where that happens)
    assert rel_err(parts[0] + parts[1], got, floor_frac=1.0) < 5e-3
    # graph capture: the layer allocates nothing while it runs
    out2 = dev.alloc(B * d, tb.F32)
    dev.begin_capture()
    full.decode(hb, cb, lb, B, max_seq * (C_ + R_), max(lens), out=out2)
    g = dev.end_capture()
    g.launch()
    dev.sync()
    assert np.array_equal(out2.to_vec().reshape(B, d), got.astype(np.float32))
    g.free()
    full.destroy()


# The attention core on the tensor cores (csrc/mla_umma.cu; 80 heads of one sequence and 16 heads: the mma.sync kernel): heads that fill the
# tile and that do not, one split and several, splits without positions, lengths around the 32-position tiles, flat and sharply peaked scores; what lies behind a sequence's
# end in the cache is NaN.  The queries are given, so the result may differ by its own rounding to bf16 (at most 2^-8 = 3.9e-3 of the
# value) and f32 sums only.
@pytest.mark.gpu
@pytest.mark.parametrize("H,B,lens,sharp", [(128, 80, [256, 255, 257, 33, 32, 31, 1, 0] * 10, 1.0), (64, 3, [9000, 31, 4097], 1.0),
                                            (144, 2, [8191, 5000], 6.0), (80, 1, [9473], 30.0), (16, 2, [9000, 77], 6.0)])
def test_attention_core(dev, H, B, lens, sharp):
    import ctypes as C

    import tang_b200 as tb
    import torch

    g = torch.Generator(device="cuda").manual_seed(H + B)
    rows = max(lens) + 3
    q = (torch.randn((B, H, C_ + R_), device="cuda", generator=g) * sharp).bfloat16()
    cache = torch.randn((B, rows, C_ + R_), device="cuda", generator=g).bfloat16()
    for b, n in enumerate(lens):
        cache[b, n:] = float("nan")
    out = torch.full((B, H, C_), float("nan"), device="cuda").bfloat16()
    lb = torch.tensor(lens, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    scale = 1.0 / np.sqrt(NOPE + R_)
    dev._check(dev._L.tq_mla_decode(dev._ctx, C.c_void_p(q.data_ptr()), C.c_void_p(cache.data_ptr()), C.c_void_p(lb.data_ptr()), B, H, C_, R_,
                                    rows * (C_ + R_), max(lens), scale, C.c_void_p(out.data_ptr())))
    dev.sync()
    for b, n in enumerate(lens):
        if n == 0:
            assert not out[b].any()
            continue
        kv = cache[b, :n].double()
        want = (q[b].double() @ kv.T * scale).softmax(-1) @ kv[:, :C_]
        assert rel_err(out[b].double().cpu().numpy(), want.cpu().numpy(), floor_frac=1.0) < 4.1e-3, (b, n)


def attend(dev, q, cache, starts, lens, stride, max_len, shift=0):
    """tq_mla_decode on torch tensors; `starts`: rows of `cache` at which the sequences begin; the result begins `shift` elements into
    its memory.  Returns the result and what it is in 64 bits."""
    import ctypes as C

    import torch

    B, H = q.shape[:2]
    out = torch.full((B * H * C_ + shift,), float("nan"), device="cuda").bfloat16()[shift:].view(B, H, C_)
    lb = torch.tensor(lens, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    scale = 1.0 / np.sqrt(NOPE + R_)
    dev._check(dev._L.tq_mla_decode(dev._ctx, C.c_void_p(q.data_ptr()), C.c_void_p(cache.data_ptr()), C.c_void_p(lb.data_ptr()), B, H, C_, R_,
                                    stride, max_len, scale, C.c_void_p(out.data_ptr())))
    dev.sync()
    want = torch.zeros((B, H, C_), device="cuda", dtype=torch.float64)
    for b, n in enumerate(lens):
        if n:
            kv = cache[starts[b]:starts[b] + n].double()
            want[b] = (q[b].double() @ kv.T * scale).softmax(-1) @ kv[:, :C_]
    return out, want


# Sequences that begin closer to one another than max_len rows: views of one cache that overlap, and a single sequence, whose stride says
# nothing.  Both sizes are the tcgen05 kernel's but for the stride.  The bar is test_attention_core's.
@pytest.mark.gpu
@pytest.mark.parametrize("B,n,step", [(40, 300, 100), (40, 300, 299), (1, 19000, 1), (1, 19000, 0)])
def test_attention_core_over_close_sequences(dev, B, n, step):
    import torch

    g = torch.Generator(device="cuda").manual_seed(B + step)
    q = torch.randn((B, 128, C_ + R_), device="cuda", generator=g).bfloat16()
    cache = torch.randn(((B - 1) * step + n, C_ + R_), device="cuda", generator=g).bfloat16()
    got, want = attend(dev, q, cache, [b * step for b in range(B)], [n - b % 7 for b in range(B)], step * (C_ + R_), n)
    assert rel_err(got.double().cpu().numpy(), want.cpu().numpy(), floor_frac=1.0) < 4.1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("B,short", [(1, 19969), (3, 9017), (40, 224), (40, 1)])
def test_attention_core_reads_no_row_behind_the_end(dev, B, short):
    """max_len and the stride leave room for more rows than the last sequence has, and its memory ends with it."""
    import torch

    n = 20001 if B == 1 else 9601 if B == 3 else 320
    g = torch.Generator(device="cuda").manual_seed(short)
    q = torch.randn((B, 128, C_ + R_), device="cuda", generator=g).bfloat16()
    cache = torch.randn(((B - 1) * n + short, C_ + R_), device="cuda", generator=g).bfloat16()
    got, want = attend(dev, q, cache, [b * n for b in range(B)], [n - b for b in range(B - 1)] + [short], n * (C_ + R_), n)
    assert rel_err(got.double().cpu().numpy(), want.cpu().numpy(), floor_frac=1.0) < 4.1e-3


def tcgen05_length(B, H, tiles=8):
    """The shortest max_len from which tq_mla_decode takes the tcgen05 kernel: `tiles` (eight at least) tiles of 32 positions for every CTA
    of one wave (csrc/mla.cu)."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return 32 * tiles * max(1, sms // (2 * B * ((H + 127) // 128)))


# Peaked scores that grow along the sequence, so that the reference of the exponentials moves, and the outputs are rescaled beside a
# pending product, in late tiles too; heads that leave rows of the last 128 empty; sequences with room between them.
@pytest.mark.gpu
@pytest.mark.parametrize("H,B,sharp", [(80, 4, 30.0), (64, 40, 30.0), (144, 3, 6.0), (128, 1, 30.0)])
def test_attention_core_with_growing_scores(dev, H, B, sharp):
    import torch

    g = torch.Generator(device="cuda").manual_seed(H + B)
    n = tcgen05_length(B, H, 11) + 5
    ramp = torch.linspace(0, 1, n, device="cuda")[:, None]
    u = torch.randn((C_ + R_,), device="cuda", generator=g)
    q = ((torch.randn((B, H, C_ + R_), device="cuda", generator=g) + u) * sharp / 24).bfloat16()
    cache = (torch.randn((B, n, C_ + R_), device="cuda", generator=g) * 0.3 + ramp * u).bfloat16()
    rows = torch.full((B, n + 37, C_ + R_), float("nan"), device="cuda", dtype=torch.bfloat16)
    rows[:, :n] = cache
    lens = [n - 33 * b for b in range(B)]
    got, want = attend(dev, q, rows.view(-1, C_ + R_), [b * (n + 37) for b in range(B)], lens, (n + 37) * (C_ + R_), n)
    assert rel_err(got.double().cpu().numpy(), want.cpu().numpy(), floor_frac=1.0) < 4.1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("H,B", [(128, 40), (64, 6)])
def test_attention_core_replayed_while_sequences_grow(dev, H, B):
    """One recorded call, the lengths raised between the replays: through full tiles, past them, and into splits that had no positions."""
    import ctypes as C

    import torch

    g = torch.Generator(device="cuda").manual_seed(H)
    n = tcgen05_length(B, H, 9)
    q = torch.randn((B, H, C_ + R_), device="cuda", generator=g).bfloat16()
    cache = torch.randn((B, n, C_ + R_), device="cuda", generator=g).bfloat16()
    out = torch.zeros((B, H, C_), device="cuda", dtype=torch.bfloat16)
    lens = torch.zeros((B,), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    call = lambda: dev._check(dev._L.tq_mla_decode(dev._ctx, C.c_void_p(q.data_ptr()), C.c_void_p(cache.data_ptr()), C.c_void_p(lens.data_ptr()), B, H, C_, R_,
                                                   n * (C_ + R_), n, 1.0 / np.sqrt(NOPE + R_), C.c_void_p(out.data_ptr())))
    call()                     # (sizes the workspace)
    dev.sync()
    dev.begin_capture()
    call()
    graph = dev.end_capture()
    for base in (1, 31, 32, 33, n // 2, n - B):
        lens.copy_(torch.arange(B, dtype=torch.int32, device="cuda") + base)
        torch.cuda.synchronize()
        graph.launch()
        dev.sync()
        for b in range(0, B, 5):
            kv = cache[b, :base + b].double()
            want = (q[b].double() @ kv.T / np.sqrt(NOPE + R_)).softmax(-1) @ kv[:, :C_]
            assert rel_err(out[b].double().cpu().numpy(), want.cpu().numpy(), floor_frac=1.0) < 4.1e-3, (base, b)
    graph.free()


@pytest.mark.gpu
@pytest.mark.parametrize("H,B,n", [(16, 2, 500), (128, 3, 9600)])
def test_merged_results_begin_anywhere(dev, H, B, n):
    """The merge of the splits of either kernel stores to a result at an odd multiple of two bytes."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(H)
    q = torch.randn((B, H, C_ + R_), device="cuda", generator=g).bfloat16()
    cache = torch.randn((B * n, C_ + R_), device="cuda", generator=g).bfloat16()
    for shift in (0, 1, 2):
        got, want = attend(dev, q, cache, [b * n for b in range(B)], [n] * B, n * (C_ + R_), n, shift)
        assert rel_err(got.double().cpu().numpy(), want.cpu().numpy(), floor_frac=1.0) < 4.1e-3, shift


@pytest.mark.gpu
@pytest.mark.parametrize("B,n", [(38, 32768), (40, 6000), (16, 16384)])
def test_attention_core_has_no_bias(dev, B, n):
    """Values of one sign: the tensor core truncates when it adds, about 6e-9 of the sum for a position, so a split takes 4096 positions at
    most: 2.6e-5 (all of 32768 in one had 2.1e-4).  The rounding of 512 x 128 results a sequence to bf16, 1.1e-3 each and the heads' not
    independent, leaves some 3e-6 in the mean."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(B)
    q = (torch.randn((B, 128, C_ + R_), device="cuda", generator=g) * 0.2).bfloat16()
    mean = torch.rand((B, 1, C_ + R_), device="cuda", generator=g) + 1
    cache = torch.empty((B, n, C_ + R_), device="cuda", dtype=torch.bfloat16)
    for b in range(B):
        cache[b] = (mean[b] + torch.rand((n, C_ + R_), device="cuda", generator=g)).bfloat16()
    got, want = attend(dev, q, cache.view(-1, C_ + R_), [b * n for b in range(B)], [n - 17 * b for b in range(B)], n * (C_ + R_), n)
    bias = (got.double() / want - 1).mean().item()
    assert abs(bias) < 3.5e-5, bias


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("H,B", [(16, 1), (80, 8), (75, 9), (128, 16), (33, 33), (128, 64)])
def test_per_head_products(dev, kind, H, B):
    """W_UK and W_UV as grouped products of a short K (csrc/qgemm_heads.cu), row counts around the eight-row column tiles, head counts
    whose row blocks do not fill the last CTA; exact products in f32 sums of at most 512 terms."""
    import ctypes as C

    import tang_b200 as tb
    import torch
    from util import make_weight

    rng = np.random.default_rng(kind * 100 + H + B)
    g = torch.Generator(device="cuda").manual_seed(H + B)
    for rows, cols in ((C_, NOPE), (VD, C_)):
        sc, pay = make_weight(rng, kind, H * rows, cols)
        w = dev.upload_qarrays(kind, pay, sc, H * rows, cols)
        deq = torch.from_numpy(dev.dequantize(w)[0]).cuda().double().view(H, rows, cols)
        x = torch.randn((B, H, cols), device="cuda", generator=g).bfloat16()
        rope = torch.zeros((B, H, R_), device="cuda").bfloat16()
        want = torch.einsum("bhc,hrc->bhr", x.double(), deq)
        if rows == C_:
            out = torch.empty((B, H, C_ + R_), device="cuda", dtype=torch.bfloat16)
            torch.cuda.synchronize()   # (`out` may be memory that the products above still use, on torch's stream)
            dev._check(dev._L.tq_mla_absorb_q(dev._ctx, C.c_void_p(w.handle), C.c_void_p(x.data_ptr()), C.c_void_p(rope.data_ptr()), B, H, cols,
                                              C.c_void_p(out.data_ptr())))
            dev.sync()
            assert rel_err(out[:, :, :C_].double().cpu().numpy(), want.cpu().numpy()) < 4.1e-3        # its own rounding to bf16: 2^-8
        else:
            out = torch.empty((B, H, VD), device="cuda")
            torch.cuda.synchronize()
            dev._check(dev._L.tq_mla_unabsorb(dev._ctx, C.c_void_p(w.handle), C.c_void_p(x.data_ptr()), B, H, VD, C.c_void_p(out.data_ptr()), tb.F32))
            dev.sync()
            assert rel_err(out.double().cpu().numpy(), want.cpu().numpy()) < 1e-3


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("H,B", [(16, 3), (128, 16)])
def test_per_head_products_have_no_bias(dev, kind, H, B):
    """W_UV's products as f32 results of positive terms: the tensor core truncates when it adds, so an accumulator that stayed there for all
    of K would be low by its number of steps; a 32-block's two steps lose less than 2^-23 of it each, f32 additions none on average."""
    import ctypes as C

    import tang_b200 as tb
    import torch

    rng = np.random.default_rng(kind + H)
    rows = H * VD
    sc = rng.uniform(0.5, 1.5, rows if kind == 3 else (rows, C_ // 32)).astype(np.float32)
    if kind < 2:
        lo, hi = (rng.integers(9, 16, (rows, C_ // 2), dtype=np.uint8) for _ in range(2))
        pay, sc = lo | (hi << 4), sc.astype(np.float16).view(np.uint16) if kind == 1 else sc
    else:
        pay = rng.integers(1, 128, (rows, C_), dtype=np.int8)
    w = dev.upload_qarrays(kind, pay, sc, rows, C_)
    deq = torch.from_numpy(dev.dequantize(w)[0]).cuda().double().view(H, VD, C_)
    x = torch.randn((B, H, C_), device="cuda", generator=torch.Generator(device="cuda").manual_seed(H)).abs().bfloat16()
    out = torch.empty((B, H, VD), device="cuda")
    torch.cuda.synchronize()
    dev._check(dev._L.tq_mla_unabsorb(dev._ctx, C.c_void_p(w.handle), C.c_void_p(x.data_ptr()), B, H, VD, C.c_void_p(out.data_ptr()), tb.F32))
    dev.sync()
    err = out.double() / torch.einsum("bhc,hrc->bhr", x.double(), deq) - 1
    # (rms: a result's own rounding 2.5e-8, three additions of tiles)
    assert abs(err.mean().item()) < 1.3e-7 and err.square().mean().sqrt().item() < 6e-8, (err.mean(), err.square().mean().sqrt())
