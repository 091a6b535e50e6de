"""GPU parity of the MoE FFN layer against the oracle composition (parity unpinned: the reference has
no MoE).  Expert selection must be bit-exact; outputs are f32-accumulated."""
import numpy as np
import pytest

from moe_util import HostMoe
from util import bf16_round, rel_err, rel_err_profile

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    import tang_b200

    d = tang_b200.QuantComputeDevice(0)
    yield d
    d.close()


def assert_moe_close(got, want, T):
    """The f32 bar, 1e-3 against max(|ref|, rms(ref)), with one stated exception.  The SwiGLU output is rounded to bf16
    on both sides (the oracle defines the layer that way); where that value lies within an f32-vs-f64 difference of a
    rounding tie, the two sides round it to neighbouring bf16 numbers, and ONE such flip of a large activation moves
    the whole output row of that token by up to 0.3 % of the rms (seen: one token of 130, 58 of 33 280 elements between
    1e-3 and 2.6e-3).  So: at most 0.5 % of the elements may exceed 1e-3, and none may exceed 1e-2 (half the bf16
    bar).  Small batches, which see few activations, must meet 1e-3 everywhere."""
    worst, frac = rel_err_profile(got, want, floor_frac=1.0)
    assert worst < (1e-3 if T < 24 else 1e-2), (T, worst)
    assert frac < 5e-3, (T, frac)


def check(dev, orc, host, T, seed):
    import tang_b200 as tb

    rng = np.random.default_rng(seed)
    hb, hf = bf16_round(rng.standard_normal((T, host.d)).astype(np.float32))
    want, idx_o, w_o, lg_o = host.oracle(orc, hf)
    hbuf = dev.upload(hb, tb.BF16)
    idx_d, w_d, lg_d = tb.moe_router(dev, hbuf, dev.upload(host.wg_bits, tb.BF16), T, host.d, host.E, host.k, host.renorm)
    assert np.array_equal(lg_d, lg_o)                 # f64, same order of additions: bit-identical logits
    assert np.array_equal(idx_d, idx_o)               # so the selection (and its order) is identical
    assert rel_err(w_d, w_o) < 1e-6
    layer = host.to_device(dev)
    out, idx, w = layer.forward(hbuf, T, want_routing=True)
    dev.sync()
    assert np.array_equal(idx.to_vec().reshape(T, host.k), idx_o)
    got = out.to_vec().reshape(T, host.d)
    assert_moe_close(got, want, T)
    layer.destroy()


@pytest.mark.parametrize("T", [1, 5, 70, 200])
def test_small_moe(dev, orc, T):
    host = HostMoe(np.random.default_rng(5), d=256, ffn=256, n_experts=8, top_k=2, n_shared=1)
    check(dev, orc, host, T, seed=T)


def test_router_ties_pick_lower_index(dev, orc):
    import tang_b200 as tb

    d, E, k = 128, 8, 3
    wg = np.zeros((E, d), np.float32)
    wg[[1, 4, 6], 0] = 1.0            # experts 1, 4, 6 tie exactly; the rest tie at zero
    wg[2, 0] = 2.0
    h = np.zeros((1, d), np.float32)
    h[0, 0] = 1.0
    idx, w, lg = tb.moe_router(dev, dev.upload(bf16_round(h)[0], tb.BF16), dev.upload(bf16_round(wg)[0], tb.BF16), 1, d, E, k)
    oi, ow, _ = orc.router_f64(h[0].astype(np.float64), wg.astype(np.float64), E, k)
    assert list(idx[0]) == [2, 1, 4] == list(oi)


def test_router_rows_that_round(dev, orc):
    """Rows whose additions DO round (tiny products beside large ones, cancellation, a huge term): the logits must still
    be the reference's sequential f64 sum bit for bit, which the kernel gets by joining runs of the row in order."""
    import tang_b200 as tb

    rng = np.random.default_rng(77)
    T, d, E, k = 12, 2048, 64, 6
    h = rng.standard_normal((T, d)).astype(np.float32)
    wg = (rng.standard_normal((E, d)) * 0.05).astype(np.float32)
    h[0, 5] = 3e-30
    h[1, [0, 1000, 2047]] = [1e-25, -2e-31, 7e-28]
    h[2, :] = 0.0
    h[2, [3, 900]] = [1e-20, 1.0]
    h[3, 100:140] *= 1e-22                      # a whole run of tiny terms
    h[4, [10, 11]] = [3e4, -3e4]                # cancellation: the sum returns to a finer last place
    wg[:, 10] = 1.0
    wg[:, 11] = 1.0
    h[5, 77] = 1e30                             # one huge term: everything after it rounds
    h[6, ::2] = 0.0
    wg[7, :] *= 1e-18
    wg[9, 1234] = 1e-33
    hb, hf = bf16_round(h)
    wb, wf = bf16_round(wg)
    idx, w, lg = tb.moe_router(dev, dev.upload(hb, tb.BF16), dev.upload(wb, tb.BF16), T, d, E, k)
    for t in range(T):
        oi, ow, ol = orc.router_f64(hf[t].astype(np.float64), wf.astype(np.float64), E, k)
        assert np.array_equal(lg[t], ol), t
        assert list(idx[t]) == list(oi), t


def test_renormalised_weights(dev, orc):
    host = HostMoe(np.random.default_rng(6), d=256, ffn=128, n_experts=16, top_k=4, n_shared=0, renorm=True)
    check(dev, orc, host, 9, seed=3)


@pytest.mark.parametrize("T", [1, 64])
def test_deepseek_v2_lite_shape(dev, orc, T):
    """d_model 2048, 64 routed + 2 shared experts of width 1408, top-6."""
    host = HostMoe(np.random.default_rng(7), d=2048, ffn=1408, n_experts=64, top_k=6, n_shared=2)
    check(dev, orc, host, T, seed=100 + T)


@pytest.mark.parametrize("T", [1, 7, 40, 130])
def test_dispatch_variant_on_one_rank_equals_the_oracle(dev, orc, T):
    """tq_moe_ffn_dispatch with a single rank: both exchanges are local copies, everything else is the same code
    the multi-rank path runs (places, buckets, scatter back, combine)."""
    import tang_b200 as tb

    host = HostMoe(np.random.default_rng(15), d=256, ffn=256, n_experts=8, top_k=2, n_shared=1)
    rng = np.random.default_rng(T)
    hb, hf = bf16_round(rng.standard_normal((T, host.d)).astype(np.float32))
    want, idx_o, _, _ = host.oracle(orc, hf)
    layer = host.to_device(dev)
    out, idx, _w = layer.forward_dispatch(dev.upload(hb, tb.BF16), T, want_routing=True)
    dev.sync()
    assert np.array_equal(idx.to_vec().reshape(T, host.k), idx_o)
    assert_moe_close(out.to_vec().reshape(T, host.d), want, T)
    layer.destroy()


@pytest.mark.parametrize("T", [256, 4096])
def test_deepseek_v2_lite_shape_large_batches(dev, orc, T):
    """The benchmark's larger token batches at the DeepSeek-V2-Lite shape: the router's selection is compared for EVERY
    token (bit-exact logits and choices), the layer output on a seeded sample of tokens (the oracle is a per-token
    loop)."""
    import tang_b200 as tb

    host = HostMoe(np.random.default_rng(7), d=2048, ffn=1408, n_experts=64, top_k=6, n_shared=2)
    rng = np.random.default_rng(500 + T)
    hb, hf = bf16_round(rng.standard_normal((T, host.d)).astype(np.float32))
    hbuf = dev.upload(hb, tb.BF16)
    idx_d, w_d, lg_d = tb.moe_router(dev, hbuf, dev.upload(host.wg_bits, tb.BF16), T, host.d, host.E, host.k, host.renorm)
    wg64 = host.wg.astype(np.float64)
    for t in range(T):
        idx_o, w_o, lg_o = orc.router_f64(hf[t].astype(np.float64), wg64, host.E, host.k, host.renorm)
        assert np.array_equal(lg_d[t], lg_o) and np.array_equal(idx_d[t], idx_o), t
    layer = host.to_device(dev)
    out, idx, w = layer.forward(hbuf, T, want_routing=True)
    dev.sync()
    assert np.array_equal(idx.to_vec().reshape(T, host.k), idx_d)
    got = out.to_vec().reshape(T, host.d)
    assert np.all(np.isfinite(got))
    sample = np.sort(rng.choice(T, 6, replace=False))
    want, _, _, _ = host.oracle(orc, hf[sample])
    assert_moe_close(got[sample], want, T)
    layer.destroy()


@pytest.mark.parametrize("renorm", [False, True])
def test_fused_gate_up_equals_the_separate_kernel(dev, renorm):
    """Many tokens: gate and up halves meet in the projection's epilogue (csrc/qgemm_umma.cu, swiglu 2), for the routed experts
    and, from 1024 tokens on, for the shared one.  The same tokens a few at a time take the other kernels: what differs is f32
    summation order and, through it, single bf16 roundings of the SwiGLU output (the layer's bar above)."""
    import tang_b200 as tb

    rng = np.random.default_rng(31 + renorm)
    moe = HostMoe(rng, 256, 384, 4, 2, 1, renorm)
    layer = moe.to_device(dev)
    T = 1061
    bits, _ = bf16_round(rng.standard_normal((T, 256)).astype(np.float32))
    whole = layer.forward(dev.upload(bits, tb.BF16), T).to_vec().reshape(T, 256)
    parts = np.concatenate([layer.forward(dev.upload(bits[t:t + 40], tb.BF16), min(40, T - t)).to_vec().reshape(-1, 256) for t in range(0, T, 40)])
    worst, share = rel_err_profile(whole, parts)
    assert worst < 1e-2 and share < 5e-3, (worst, share)
    layer.destroy()


@pytest.mark.parametrize("rows,cols", [(768 + 128, 256), (768, 384)])
@pytest.mark.parametrize("T", [40, 1061])
def test_shared_experts_of_another_size_are_refused(dev, rows, cols, T):
    """A shared gate/up projection with more rows or columns than the layer's: an error at every token count, whichever kernel would
    have run."""
    import tang_b200 as tb
    from util import make_weight

    rng = np.random.default_rng(rows + T)
    moe = HostMoe(rng, 256, 384, 4, 2, 0)
    up = lambda r, c: dev.upload_qarrays(1, *make_weight(rng, 1, r, c)[::-1], r, c)
    layer = tb.MoeLayer(dev, tb.MoeConfig(256, 384, 4, 2, 1, 0, 0, 1), dev.upload(moe.wg_bits, tb.BF16), up(4 * 768, 256), up(4 * 256, 384), [up(rows, cols)],
                        [up(256, 384)])
    x = dev.upload(bf16_round(rng.standard_normal((T, 256)).astype(np.float32))[0], tb.BF16)
    with pytest.raises(tb.TangqError):
        layer.forward(x, T)
    dev.sync()
    layer.destroy()


@pytest.mark.parametrize("d,f,T", [(256, 128, 1023), (256, 128, 1024), (512, 2048, 384), (512, 2048, 385), (256, 1408, 640), (256, 1408, 641), (256, 14336, 16), (256, 14336, 17)])
def test_shared_expert_on_both_sides_of_its_rule(dev, d, f, T):
    """Narrow and wide shared experts around the token counts where gate and up begin to meet in the projection's epilogue, against 64
    bits with the one rounding that the layer has, of the gated product to bf16.  A product within an f32 sum's error of a rounding tie
    (one in some thousand) may round the other way, 2^-8 of itself: about 1e-4 of the result's norm."""
    import tang_b200 as tb
    import torch

    rng = np.random.default_rng(f + T)
    moe = HostMoe(rng, d, f, 4, 2, 1)
    layer = moe.to_device(dev)
    bits, x = bf16_round(rng.standard_normal((T, d)).astype(np.float32))
    got = layer.forward(dev.upload(bits, tb.BF16), T).to_vec().reshape(T, d)
    layer.destroy()
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda().double()

    def weight(w):
        pay, sc = t(np.stack((w[1] & 15, w[1] >> 4), 2).reshape(w[2], -1).astype(np.int8) - 8), t(w[0].view(np.float16).astype(np.float32))
        return (pay.view(w[2], -1, 32) * sc[:, :, None]).view(w[2], -1)[:, :w[3]]

    def expert(e, h):
        g, u = h @ weight(e["gate"]).T, h @ weight(e["up"]).T
        return (g * torch.sigmoid(g) * u).bfloat16().double() @ weight(e["down"]).T

    h = t(x)
    top, idx = (h @ t(moe.wg).T).softmax(1).topk(2, 1)
    want = expert(moe.experts[4], h)
    for e in range(4):
        rows, c = (idx == e).nonzero(as_tuple=True)
        want[rows] += top[rows, c][:, None] * expert(moe.experts[e], h[rows])
    d_ = torch.from_numpy(got).cuda().double() - want
    assert (d_.norm() / want.norm()).item() < 5e-4, (d_.norm() / want.norm()).item()


@pytest.mark.parametrize("d", [8, 40, 264, 2048])
@pytest.mark.parametrize("T,E,k", [(1, 2, 2), (15, 8, 3), (16, 9, 1), (17, 64, 6), (33, 61, 16), (130, 256, 8)])
def test_router_blocks_of_tokens_and_experts(dev, orc, d, T, E, k):
    """Edges of the blocks of 16 tokens, 8 experts and 32 k; subnormals, infinities and NaN in some rows."""
    import tang_b200 as tb

    rng = np.random.default_rng(T * E + d)
    h = rng.standard_normal((T, d)).astype(np.float32)
    wg = (rng.standard_normal((E, d)) * 0.05).astype(np.float32)
    h[T // 2, d // 2] = 1e-39
    wg[E // 2, 0] = 2e-30
    if T > 16:
        h[3, 1] = np.inf
        h[16, d - 1] = np.nan
    hb, hf = bf16_round(h)
    wb, wf = bf16_round(wg)
    if T > 16:
        hb[16, d - 1] = 0x7FC0
        hf[16, d - 1] = np.nan
    idx, w, lg = tb.moe_router(dev, dev.upload(hb, tb.BF16), dev.upload(wb, tb.BF16), T, d, E, k)
    for t in range(T):
        oi, ow, ol = orc.router_f64(hf[t].astype(np.float64), wf.astype(np.float64), E, k)
        assert np.array_equal(lg[t], ol, equal_nan=True), t
        if not np.isnan(ol).any() and np.isfinite(ol).all():
            assert list(idx[t]) == list(oi), t
            assert np.abs(w[t] - ow).max() < 1e-6


@pytest.mark.parametrize("E,T", [(40, 300), (70, 600)])
def test_token_tiles_of_uneven_experts(dev, orc, E, T):
    """The grouped tcgen05 GEMM with groups beyond one warp's scan: a few experts get most of the tokens."""
    host = HostMoe(np.random.default_rng(E), d=256, ffn=128, n_experts=E, top_k=4, n_shared=0)
    scale = np.full((E, 1), 0.05)
    scale[1::E // 3] = 40.0
    host.wg_bits, host.wg = bf16_round((host.wg * scale).astype(np.float32))
    check(dev, orc, host, T, seed=E)


@pytest.mark.parametrize("T", [5, 40, 300])
def test_recorded_layer_replays(dev, T):
    """A layer recorded into a graph, shared experts on the context's side stream among it (40 and 300 tokens), against the same call outside:
    twice, with other activations in between, and beside a call that is not recorded."""
    import tang_b200 as tb

    rng = np.random.default_rng(T)
    layer = HostMoe(rng, 256, 384, 16, 4, 2).to_device(dev)
    xs = [dev.upload(bf16_round(rng.standard_normal((T, 256)).astype(np.float32))[0], tb.BF16) for _ in range(2)]
    want = [layer.forward(x, T).to_vec() for x in xs]
    x, out = dev.alloc(T * 256, tb.BF16), dev.alloc(T * 256, tb.F32)
    dev.upload_into(x, xs[0].to_vec())
    layer.forward(x, T, out=out)
    dev.sync()
    dev.begin_capture()
    layer.forward(x, T, out=out)
    graph = dev.end_capture()
    for i in (1, 0, 1):
        dev.upload_into(x, xs[i].to_vec())
        graph.launch()
        if i == 0:
            assert np.array_equal(layer.forward(xs[1], T).to_vec(), want[1])
        dev.sync()
        assert np.array_equal(out.to_vec(), want[i]), i
    graph.free()
    layer.destroy()


def _router_without_logits(dev, h, wg, T, d, E, k, renorm=0):
    """The form for callers that give no room for the logits."""
    import ctypes as C

    import tang_b200 as tb

    idx, w = dev.alloc(T * k, tb.I32), dev.alloc(T * k, tb.F32)
    dev._check(dev._L.tq_moe_router(dev._ctx, C.c_void_p(h.ptr), C.c_void_p(wg.ptr), T, d, E, k, renorm, C.c_void_p(idx.ptr), C.c_void_p(w.ptr), C.c_void_p(0)))
    dev.sync()
    return idx.to_vec().reshape(T, k), w.to_vec().reshape(T, k)


@pytest.mark.parametrize("T,d,E,k,renorm", [(1, 40, 2, 2, 0), (70, 2048, 64, 6, 1), (2049, 264, 61, 16, 0), (2100, 4104, 9, 1, 0)])
def test_router_without_logits_makes_the_same_choices(dev, T, d, E, k, renorm):
    """One and four tokens per CTA; rows that round, an infinity and a NaN among them."""
    import tang_b200 as tb

    rng = np.random.default_rng(T + d)
    h = rng.standard_normal((T, d)).astype(np.float32)
    h[T // 2, d // 2] = 1e-30
    bits = bf16_round(h)[0]
    if T > 1:
        bits[3, 1], bits[T - 1, d - 1] = 0x7F80, 0x7FC0
    hb, wb = dev.upload(bits, tb.BF16), dev.upload(bf16_round((rng.standard_normal((E, d)) * 0.05).astype(np.float32))[0], tb.BF16)
    want_i, want_w, _ = tb.moe_router(dev, hb, wb, T, d, E, k, bool(renorm))
    idx, w = _router_without_logits(dev, hb, wb, T, d, E, k, renorm)
    assert np.array_equal(idx, want_i) and np.array_equal(w, want_w, equal_nan=True)


def test_router_of_more_tokens_than_counters(dev):
    """More than 16 x 1024 tokens take the other router, with the logits written too."""
    import tang_b200 as tb

    T, d, E, k = 16400, 64, 5, 2
    rng = np.random.default_rng(4)
    bits = bf16_round(rng.standard_normal((T, d)).astype(np.float32))[0]
    wb = dev.upload(bf16_round((rng.standard_normal((E, d)) * 0.05).astype(np.float32))[0], tb.BF16)
    whole = tb.moe_router(dev, dev.upload(bits, tb.BF16), wb, T, d, E, k)
    parts = [tb.moe_router(dev, dev.upload(bits[t:t + 8200], tb.BF16), wb, 8200, d, E, k) for t in (0, 8200)]
    for a, b in zip(whole, zip(*parts)):
        assert np.array_equal(a, np.concatenate(b))


def test_plan_of_more_pairs_than_one_cta_takes(dev):
    """More than 32768 (token, choice) pairs: local ids, counts and slots in kernels of their own; the same tokens in two halves take one."""
    import tang_b200 as tb

    rng = np.random.default_rng(9)
    layer = HostMoe(rng, 128, 128, 8, 4, 1).to_device(dev)
    T = 8200
    bits, _ = bf16_round(rng.standard_normal((T, 128)).astype(np.float32))
    whole = layer.forward(dev.upload(bits, tb.BF16), T).to_vec().reshape(T, 128)
    parts = np.concatenate([layer.forward(dev.upload(bits[t:t + 4100], tb.BF16), 4100).to_vec().reshape(-1, 128) for t in (0, 4100)])
    worst, share = rel_err_profile(whole, parts)
    assert worst < 1e-2 and share < 5e-3, (worst, share)
    layer.destroy()
