"""The tcgen05 form of differential attention (tang_b200/csrc/diff_attention_umma.cu: maps of 64, values of 128, many rows) against the plain numpy
implementation: edges of its tiles of 128 rows and 128 keys, windows and kept tokens, NaN in every cache row that no query may see."""
import ctypes as C

import numpy as np
import pytest

import test_diff_attention_gpu as D
from util import bf16_round

pytestmark = pytest.mark.gpu
dev = D.dev


class Aligned(D.Case):
    """As Case, with result rows that are 16-byte aligned."""

    def run(self, dev, dtype, poison=True, bits_of=0x7FC0):
        """bits_of: what stands for a NaN in bf16."""
        import tang_b200 as tb

        n_slots = len(self.seqs) + 2
        kc = np.full((n_slots, self.max_seq, self.G, 2, self.D), np.nan, np.float32)
        vc = np.full((n_slots, self.max_seq, self.G, self.V), np.nan, np.float32)
        row_pos, cache_row = [], []
        for b, (start, n) in enumerate(self.seqs):
            s = self.slots[b]
            kc[s, :start + n], vc[s, :start + n] = self.k[b], self.v[b]
            row_pos += range(start, start + n)
            cache_row += range(s * self.max_seq + start, s * self.max_seq + start + n)
        counts = [n for _, n in self.seqs]
        q = np.concatenate([x.reshape(x.shape[0], -1) for x in self.q])
        bits = lambda a: np.where(np.isnan(a), np.uint16(bits_of), bf16_round(np.nan_to_num(a))[0])
        up = (lambda a: dev.upload(bits(np.ascontiguousarray(a)), tb.BF16)) if dtype == tb.BF16 else dev.upload
        qb, kb, vb = up(q), up(kc), up(vc)
        i32 = lambda a: dev.upload(np.asarray(a, np.int32), tb.I32)
        cu, rp, cr = i32(np.cumsum([0] + counts)), i32(row_pos), i32(cache_row)
        R, ldo = len(row_pos), self.H * self.V + 8
        out = dev.alloc(R * ldo, dtype)
        dev.memset(out)
        cfg = D._Cfg(self.H, self.G, self.D, self.V, self.window, self.keep, self.scale, self.lam, 1 - self.diff, D.EPS)
        dev._check(dev._L.tq_diff_attention(dev._ctx, C.byref(cfg), dtype, C.c_void_p(qb.ptr), q.shape[1], C.c_void_p(kb.ptr), C.c_void_p(vb.ptr),
                                            n_slots * self.max_seq, C.c_void_p(cu.ptr), C.c_void_p(rp.ptr), C.c_void_p(cr.ptr), len(counts), R, max(counts),
                                            max(s + n for s, n in self.seqs), C.c_void_p(out.ptr), ldo))
        dev.sync()
        o = out.to_vec()
        o = (o if dtype == tb.F32 else (o.astype(np.uint32) << 16).view(np.float32)).reshape(R, ldo)
        assert np.all(o[:, self.H * self.V:] == 0)
        return np.split(o[:, :self.H * self.V].reshape(R, self.H, self.V), np.cumsum(counts)[:-1])


@pytest.mark.parametrize("H,G,window,keep,seqs", [
    (4, 1, 100, 3, [(0, 260), (0, 1), (0, 33)]), (4, 2, 128, 0, [(0, 513)]), (8, 1, 129, 130, [(300, 128), (0, 65)]), (2, 2, 1000, 0, [(0, 1025)]),
    (16, 4, 512, 4, [(0, 640), (100, 129)]), (4, 1, 1, 1, [(0, 257)]), (4, 1, 64, 300, [(250, 262)]), (16, 1, 40, 5, [(127, 66), (128, 64)])])
def test_tiles_windows_and_kept_tokens(dev, H, G, window, keep, seqs):
    rng = np.random.default_rng(H * 100 + window + keep)
    case = Aligned(rng, H, G, 64, 128, window, keep, seqs=seqs, max_seq=max(s + n for s, n in seqs) + 150)
    D.check(dev, case)


@pytest.mark.parametrize("window,keep", [(128, 70), (127, 128), (65, 4), (300, 0)])
def test_one_key_decides(dev, window, keep):
    """Keys just inside / outside the window, the last kept and the first dropped token, both sides of a tile of 128 keys."""
    rng = np.random.default_rng(window)
    pos = 383
    for n, j in enumerate(sorted({pos - window + 1, pos - window, 0, keep - 1, keep, 127, 128, 255, 256, pos, pos - 1} & set(range(pos + 1)))):
        case = Aligned(rng, 4, 1, 64, 128, window, keep, seqs=[(120, 264)], max_seq=384)
        D._stand_out(case, 0, pos - 120, j, 12.0, n % 4, n % 2)
        D.check(dev, case, rows=[pos - 120])


@pytest.mark.parametrize("grows", [0, 1])
@pytest.mark.parametrize("tiles", [2, 4, 5, 7])
def test_one_map_behind_the_other(dev, tiles, grows):
    """The row maxima of one map grow with every tile, so that its outputs are rescaled each time, and the other map's hardly do: the maps run apart
    by whole tiles, and the exchange of the second map's outputs has to wait for the first's last products."""
    rng = np.random.default_rng(tiles)
    case = Aligned(rng, 8, 1, 64, 128, 2000, 0, seqs=[(128 * (tiles - 1), 128), (128 * (tiles - 1) + 5, 123)], max_seq=128 * tiles)
    for b in range(2):
        u = case.q[b][0, 0, grows].copy()
        case.q[b][:, :, grows] = bf16_round(u * rng.uniform(0.8, 1.2, case.q[b].shape[:2] + (1,)).astype(np.float32))[1]
        n = case.k[b].shape[0]
        case.k[b][:, 0, grows] = bf16_round((u / np.dot(u, u) / case.scale * (np.arange(n) / 32)[:, None]).astype(np.float32))[1]
        case.k[b][:, 0, 1 - grows] = bf16_round(case.k[b][:, 0, 1 - grows] * 0.05)[1]
    D.check(dev, case, rows=[0, 1, 64, 122])


@pytest.mark.parametrize("window,keep,start", [(100, 3, 0), (64, 0, 200), (2000, 0, 0), (130, 140, 150)])
@pytest.mark.parametrize("bits", [0x7F80, 0x7FC0])
def test_values_that_are_not_finite_reach_the_rows_that_see_them(dev, window, keep, start, bits):
    """One key whose values hold an infinity or a NaN: the queries before it, and those behind its window, share tiles with it and do not see it."""
    import tang_b200 as tb

    rng = np.random.default_rng(window)
    case = Aligned(rng, 8, 1, 64, 128, window, keep, seqs=[(start, 260)], max_seq=start + 260)
    bad = start + 141
    case.v[0][bad, 0, 17] = np.nan
    got = case.run(dev, tb.BF16, bits_of=bits)[0]
    pos = start + np.arange(260)
    sees = (pos >= bad) & ((pos - bad < window) | (bad < keep))
    assert np.array_equal(np.isnan(got).any(axis=(1, 2)), sees)
    case.v[0][bad, 0, 17] = 0
    rows = [i for i in (0, 127, 128, 140, 141 + window, 200 + window, 259) if i < 260 and not sees[i]]
    want = case.want(0, rows)
    rms = np.sqrt(np.mean(want ** 2))
    assert np.abs(got[rows] - want).max() < 6e-3 * max(rms, np.abs(want).max())
