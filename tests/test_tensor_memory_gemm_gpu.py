"""Edges of the tcgen05 dequant-GEMM (tang_b200/csrc/qgemm_umma.cu) against f64 products of the oracle's dequantised weights: token tiles of
one, two and four boxes, odd numbers of 128-k chunks, the split of K over clusters, rows of the result that are not 16-byte aligned.

f32 results with f16 scales or a row scale are exact products, so the error is that of the f32 sums: the tensor core truncates, at most
2^-23 of the sum of magnitudes per 16-k addition; K = 3200 in two accumulators has 200 additions, 2.4e-5 of the output's rms times the ratio
of the sum of magnitudes to it, which grows with the root of K, about 50: 1.2e-3 at worst, and a twentieth of that (additions of random sign to
partial sums that are smaller than the last) is what is asked for here.  f32 block scales keep 16 bits (2^-15 a product, 1e-4 after the sum)."""
import ctypes as C

import numpy as np
import pytest

from util import bf16_round, make_weight

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    import tang_b200

    d = tang_b200.QuantComputeDevice(0)
    yield d
    d.close()


def weights64(orc, kind, sc, pay, rows, cols):
    if kind == 3:
        return pay.astype(np.float64) * sc[:, None]
    q = (orc.unpack_q4(pay) if kind < 2 else pay).reshape(rows, cols // 32, 32).astype(np.float64)
    s = (sc.view(np.float16) if kind == 1 else sc).astype(np.float64)
    return (q * s[:, :, None]).reshape(rows, cols)


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("rows,cols", [(128, 128), (128, 640), (256, 3200), (1152, 1408), (2304, 1024), (6144, 1536)])
@pytest.mark.parametrize("m", [17, 32, 33, 64, 65, 127, 128, 129, 192, 193, 300])
def test_token_tiles_chunks_and_splits(dev, orc, kind, rows, cols, m):
    import tang_b200 as tb

    rng = np.random.default_rng(rows + cols + m + kind)
    sc, pay = make_weight(rng, kind, rows, cols)
    w = dev.upload_qarrays(kind, pay, sc, rows, cols)
    xbits, xf = bf16_round(rng.standard_normal((m, cols)).astype(np.float32))
    want = xf.astype(np.float64) @ weights64(orc, kind, sc, pay, rows, cols).T
    rms = np.sqrt(np.mean(want * want))
    y = dev.qlinear(dev.upload(xbits, tb.BF16), w, m, tb.F32).to_vec().reshape(m, rows)
    assert np.abs(y - want).max() < (1e-4 if kind in (0, 2) else 6e-5) * rms
    yb = (dev.qlinear(dev.upload(xbits, tb.BF16), w, m, tb.BF16).to_vec().reshape(m, rows).astype(np.uint32) << 16).view(np.float32)
    # the result rounded to bf16 (2^-9) and, but for row scales, every weight too (2^-9 each, of random sign: 2^-9 of the rms times six sigma)
    assert (np.abs(yb - want) < 2.0 ** -8 * np.abs(want) + 6 * 2.0 ** -9 * rms).all()


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("rows,cols,m,ld", [(512, 2048, 40, 515), (512, 2048, 40, 516), (128, 512, 20, 131), (14336, 256, 33, 14337)])
def test_result_rows_of_any_stride(dev, orc, dtype, rows, cols, m, ld):
    import tang_b200 as tb

    rng = np.random.default_rng(ld)
    sc, pay = make_weight(rng, 1, rows, cols)
    w = dev.upload_qarrays(1, pay, sc, rows, cols)
    x = dev.upload(bf16_round(rng.standard_normal((m, cols)).astype(np.float32))[0], tb.BF16)
    dt = tb.F32 if dtype == "f32" else tb.BF16
    dense = dev.qlinear(x, w, m, dt).to_vec().reshape(m, rows)
    fill = np.full(m * ld + 1, 7, np.float32 if dtype == "f32" else np.uint16)
    out = dev.upload(fill, dt)
    at = out.ptr + fill.itemsize              # one element in: no vector of four is aligned with ld 516 either
    dev._check(dev._L.tq_qlinear(dev._ctx, C.c_void_p(w.handle), C.c_void_p(x.ptr), x.dtype, 0, m, C.c_void_p(at), dt, ld, C.c_void_p(0)))
    got = out.to_vec()[1:].reshape(m, ld)
    dev.sync()
    assert np.array_equal(got[:, :rows], dense)
    assert (got[:, rows:] == 7).all() and out.to_vec()[0] == 7


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("rows,cols", [(256, 512), (14336, 1024)])
@pytest.mark.parametrize("m", [1, 4, 12, 17, 64, 300])
def test_product_right_behind_its_weight(dev, kind, rows, cols, m):
    """Both constructors that return before their kernels have run, and a product with the weight at once: the products copy their weights
    before they wait for the kernel in front.  Every product is of a weight of its own."""
    import tang_b200 as tb

    rng = np.random.default_rng(rows + m)
    sc, pay = make_weight(rng, kind, rows, cols)
    pay_d, sc_d = dev.upload(pay.view(np.uint8), tb.U8), dev.upload(np.ascontiguousarray(sc).view(np.uint8), tb.U8)
    x = dev.upload(bf16_round(rng.standard_normal((m, cols)).astype(np.float32))[0], tb.BF16)
    dev.sync()
    ws, ys = [], []
    for i in range(4):
        ws.append(dev.qweight_from_device(kind, pay_d.ptr, sc_d.ptr, rows, cols))
        if i & 1:
            ws.append(dev.interleave_gate_up(ws[-1], free_source=False))
        ys.append(dev.qlinear(x, ws[-1], m, tb.F32))
    dev.sync()
    plain, mixed = dev.qlinear(x, ws[0], m, tb.F32).to_vec(), dev.qlinear(x, ws[2], m, tb.F32).to_vec()
    for i, y in enumerate(ys):
        # (a row block's pieces may meet in another order: f32 roundings, 1e-5 of the rms; stale weights are off by all of it)
        assert np.abs(y.to_vec() - (mixed if i & 1 else plain)).max() < 1e-5 * np.sqrt(np.mean(plain.astype(np.float64) ** 2)), i


def sum_error(dev, kind, rows, cols, m):
    """Relative error (2-norm) of f32 results against f64, normal weights and activations."""
    import tang_b200 as tb
    import torch

    g = torch.Generator(device="cuda").manual_seed(rows + cols + m)
    w = torch.randn((rows, cols), device="cuda", generator=g) * cols ** -0.5
    if kind == 3:
        sc = w.abs().amax(1) / 127
        q = torch.round(w / sc[:, None]).clamp(-127, 127)
        pay, w64 = q.to(torch.int8), q.double() * sc.double()[:, None]
    else:
        b = w.view(rows, cols // 32, 32)
        sc = (b.abs().amax(2) / 7).half()
        q = torch.round(b / sc.float()[..., None]).clamp(-8, 7)
        u = (q + 8).to(torch.uint8)
        pay, w64 = u[..., 0::2] | (u[..., 1::2] << 4), (q.double() * sc.double()[..., None]).view(rows, cols)
    pay, sc = pay.contiguous(), sc.contiguous()
    x = torch.randn((m, cols), device="cuda", generator=g).bfloat16()
    torch.cuda.synchronize()
    wq = dev.qweight_from_device(kind, pay.data_ptr(), sc.data_ptr(), rows, cols)
    y = torch.empty((m, rows), device="cuda")
    dev._check(dev._L.tq_qlinear(dev._ctx, C.c_void_p(wq.handle), C.c_void_p(x.data_ptr()), tb.BF16, cols, m, C.c_void_p(y.data_ptr()), tb.F32, rows, C.c_void_p(0)))
    dev.sync()
    want = x.double() @ w64.T
    return ((y.double() - want).norm() / want.norm()).item()


# The tensor core truncates every addition of 16 k: 3.4e-9 of the result per addition that an accumulator sees with int8 rows, 1.2e-8 with the
# two terms of int4 weights (measured, 48 to 512 additions).  Outside it every f32 addition rounds, 2^-24 / sqrt(3) = 3.4e-8 rms of a partial sum:
# eight accumulators and eight splits are sixteen such additions, to sums of half the result's variance on average, 3.4e-8 * sqrt(8) = 1e-7.
def allowed(kind, additions):
    return (4e-9 if kind == 3 else 1.4e-8) * additions + 1e-7


@pytest.mark.parametrize("rows,cols", [(14336, 4096), (16384, 2048), (24576, 1536)])
@pytest.mark.parametrize("m", [129, 144, 160, 192, 193, 384])
def test_sums_of_two_token_tiles_per_cta(dev, rows, cols, m):
    """Two accumulators per tile where tensor memory holds them (up to 192 rows), one beyond."""
    assert sum_error(dev, 3, rows, cols, m) < allowed(3, cols // 16 // (2 if m <= 192 else 1))


@pytest.mark.parametrize("rows", [128, 2304])
@pytest.mark.parametrize("m", [65, 96, 128, 144, 400])
def test_sums_of_an_odd_chunk(dev, rows, m):
    """K = 128, one chunk for two issuers with an accumulator each: half of it for either (1.9e-7 with the chunk in one, 1.2e-7 so)."""
    assert sum_error(dev, 1, rows, 128, m) < 1.5e-7


@pytest.mark.parametrize("kind,rows,cols,m,chunks,accumulators", [
    (1, 6144, 4096, 64, 11, 4), (1, 6144, 4096, 33, 11, 4), (1, 6144, 4096, 96, 11, 2), (1, 2048, 8192, 48, 8, 4), (1, 1024, 14336, 40, 7, 4),
    (1, 512, 14336, 64, 7, 4), (3, 512, 14336, 20, 7, 8), (3, 1024, 14336, 100, 8, 2), (3, 5120, 7168, 129, 19, 2), (3, 6144, 4096, 192, 16, 2),
    (3, 7168, 16384, 160, 64, 2), (3, 3072, 7168, 300, 19, 2), (3, 4096, 14336, 320, 56, 2)])
def test_sums_are_cut_where_clusters_do_not_spread_k(dev, kind, rows, cols, m, chunks, accumulators):
    """As short as an even spread of K over the idle SMs gives: `chunks` of 128 k into that many accumulators."""
    assert sum_error(dev, kind, rows, cols, m) < allowed(kind, chunks * 8 * (1 if kind == 3 else 2) // accumulators)


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
@pytest.mark.parametrize("rows,cols", [(512, 7168), (640, 9216), (2304, 6272)])
@pytest.mark.parametrize("m", [17, 40, 70, 130, 200])
def test_cut_sums(dev, orc, kind, rows, cols, m):
    """Runs of four to twelve chunks, last runs of one chunk (without one for an issuer, or shared by both), splits that need no cut beside some that do."""
    import tang_b200 as tb

    rng = np.random.default_rng(rows + cols + m + kind)
    sc, pay = make_weight(rng, kind, rows, cols)
    w = dev.upload_qarrays(kind, pay, sc, rows, cols)
    xbits, xf = bf16_round(rng.standard_normal((m, cols)).astype(np.float32))
    want = xf.astype(np.float64) @ weights64(orc, kind, sc, pay, rows, cols).T
    rms = np.sqrt(np.mean(want * want))
    x = dev.upload(xbits, tb.BF16)
    got = [dev.qlinear(x, w, m, tb.F32).to_vec().reshape(m, rows) for _ in range(3)]
    assert np.abs(got[0] - want).max() < (1e-4 if kind in (0, 2) else 6e-5) * rms
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])


def test_two_threads_with_a_context_each(orc):
    """The shared-memory limit is the kernel's, not the context's: a thread's launches of large sizes and another's of small ones, with
    the query for clusters that a context's first narrow product makes, keep out of each other's way.  The router too."""
    import threading

    import tang_b200 as tb

    rng = np.random.default_rng(5)
    sc, pay = make_weight(rng, 1, 1024, 2048)
    sizes = [(1024, 2048, 17), (1024, 2048, 120)]
    routers = [(64, 512, 8), (64, 24576, 8)]
    xs = [bf16_round(rng.standard_normal((m, c)).astype(np.float32))[0] for _, c, m in sizes]
    hs = [bf16_round(rng.standard_normal((t, d)).astype(np.float32))[0] for t, d, _ in routers]
    wgs = [bf16_round((rng.standard_normal((e, d)) * 0.05).astype(np.float32))[0] for _, d, e in routers]
    out, errors = [[], []], []

    def work(i, times):
        try:
            for _ in range(times):
                dev = tb.QuantComputeDevice(0)                # (a new context asks for the clusters again)
                w = dev.upload_qarrays(1, pay, sc, 1024, 2048)
                x, h, wg = dev.upload(xs[i], tb.BF16), dev.upload(hs[i], tb.BF16), dev.upload(wgs[i], tb.BF16)
                for _ in range(20):
                    y = dev.qlinear(x, w, sizes[i][2], tb.F32)
                    r = tb.moe_router(dev, h, wg, routers[i][0], routers[i][1], routers[i][2], 2)
                dev.sync()
                out[i].append((y.to_vec(), r[2]))
                dev.close()
        except Exception as e:                                # noqa: BLE001
            errors.append(e)

    for i in (0, 1):
        work(i, 1)
    threads = [threading.Thread(target=work, args=(i, 5)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for o in out:
        for y, logits in o[1:]:
            assert np.array_equal(y, o[0][0]) and np.array_equal(logits, o[0][1])


def test_first_products_of_a_process_from_four_threads():
    """Each thread's first call asks for what the process looks up once; no thread may find the answer missing.  (A process of its own: here the
    question has been asked.)"""
    import subprocess
    import sys

    code = """
import threading, numpy as np, tang_b200 as tb
errors, gate = [], threading.Barrier(4)
def work():
    try:
        dev = tb.QuantComputeDevice(0)
        w = dev.upload_qarrays(1, np.zeros((128, 128), np.uint8), np.zeros((128, 8), np.uint16), 128, 256)
        x = dev.upload(np.zeros((64, 256), np.uint16), tb.BF16)
        dev.sync()
        gate.wait()
        dev.qlinear(x, w, 64, tb.F32)
        dev.sync()
    except Exception as e:
        errors.append(e)
        gate.abort()
ts = [threading.Thread(target=work) for _ in range(4)]
[t.start() for t in ts]; [t.join() for t in ts]
assert not errors, errors
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
