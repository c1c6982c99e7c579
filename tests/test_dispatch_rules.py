"""Rules by which the library picks a kernel (host arithmetic, no GPU)."""
import random

import pytest

from ceo_b200.ops import _lib

pytestmark = pytest.mark.skipif(not _lib.available(), reason="kernel library not built")


STORE, MORE, SWIGLU_BWD, ACCUMULATE, GENERAL = range(5)  # epilogues


def _pick(M, N, K, batch=1, fp8=0, epi=ACCUMULATE, sms=148):
    r = _lib.lib().ceo_gemm_pick(M, N, K, batch, fp8, epi, sms)
    assert r >= 4
    return r & 3, r >> 2


def _fills_badly(M, N, kb, batch, sms):
    """The 128 x 256 tiles leave so much of the last wave idle that two or three slices of at least
    16 k-blocks would fill 5 % more, after 5 % for every extra slice."""
    tiles, best, cut = -(-M // 128) * -(-N // 256) * batch, 0.0, False
    for s in range(1, 4):
        if s * 16 <= kb:
            waves = -(-tiles * s // sms)
            eff = tiles * s / (waves * sms) - 0.05 * (s - 1)
            if eff > best + (0.05 if s > 1 else 0.0):
                best, cut = eff, s > 1
    return cut


def test_only_products_that_fill_the_chip_badly_are_cut():
    # slices meet in arrival order: every other accumulation repeats bit for bit
    rng = random.Random(1)
    log = lambda lo, hi: int(2 ** rng.uniform(lo, hi))
    cut = 0
    for _ in range(20000):
        M, N, K, fp8 = log(3, 15), log(3, 15), log(6, 17), rng.randint(0, 1)
        batch, sms = rng.choice((1, 1, 1, 3, 40)), rng.choice((148, 148, 100, 1))
        kb = -(-K // (128 if fp8 else 64))
        kind, slices = _pick(M, N, K, batch, fp8, ACCUMULATE, sms)
        assert kind in (0, 1, 2) and (kind != 1 or sms >= 2)
        if slices > 1:
            assert _fills_badly(M, N, kb, batch, sms), (M, N, K, batch, fp8, sms)
            per = -(-kb // slices)
            assert slices <= 8 and per * (slices - 1) < kb  # no empty slice
            cut += 1
        assert _pick(M, N, K, batch, fp8, rng.choice((STORE, MORE, SWIGLU_BWD, GENERAL)), sms)[1] == 1
    assert cut > 1000
    assert _pick(1024, 1024, 1984)[1] == 1      # 31 k-blocks
    assert _pick(2048, 2048, 32768)[1] == 1     # 128 of 148 SMs
    assert _pick(1024, 1024, 16384)[1] > 1      # 32 of 148 SMs


def test_tiles_no_slower_than_the_wide_ones():
    # products with the microseconds of the 128 x 256 tile, of the pair and of the 128 x 128 tile: a
    # short K and many tiles (epilogues are all there is), a long K, a lone wave, whole products
    measured = [
        (7280, 11928, 40, 1, STORE, (57.1, 82.0, 76.7)), (1800, 4096, 136, 16, STORE, (76.6, 102.4, 106.6)),
        (4096, 1184, 104, 16, STORE, (56.1, 68.7, 74.9)), (15784, 6280, 304, 1, STORE, (81.8, 99.7, 98.0)),
        (13712, 14480, 168, 1, STORE, (124.4, 167.8, 169.9)), (368, 4096, 96, 5, STORE, (10.5, 15.4, 12.4)),
        (2472, 8616, 40, 1, MORE, (32.8, 37.1, 38.2)), (3184, 10520, 488, 1, STORE, (53.9, 46.1, 63.2)),
        (5760, 1552, 232, 1, MORE, (19.2, 20.8, 16.6)), (3176, 1472, 272, 1, SWIGLU_BWD, (23.1, 25.0, 20.5)),
        (32768, 6208, 2048, 1, STORE, (570.0, 535.0, 804.0)), (576, 2048, 5632, 1, STORE, (44.0, 38.0, 36.0))]
    for M, N, K, batch, epi, us in measured:
        kind, _ = _pick(M, N, K, batch, 0, epi)
        assert us[kind] <= 1.02 * us[0], (M, N, K, batch, epi, kind)


def test_spans_only_where_they_were_measured_faster():
    spans = lambda chains, n, d: _lib.lib().ceo_efla_fwd_segments(1, 64 * n, chains, d)
    # (chains, chunks, head size): plain faster by 2 % or more, spans faster by 2 % or more
    plain = [(32, 18, 128), (32, 64, 128), (32, 128, 128), (24, 24, 128), (20, 32, 128),
             (16, 18, 128), (16, 24, 128), (16, 32, 128), (12, 24, 128), (74, 32, 64), (64, 18, 64),
             (32, 18, 64), (40, 24, 64), (1, 12, 64), (148, 1024, 64)]
    spanned = [(16, 64, 128), (16, 128, 128), (8, 32, 128), (2, 64, 128), (24, 256, 128),
               (16, 1024, 64), (16, 24, 64), (1, 18, 64), (32, 64, 64), (4, 18, 64)]
    assert [s for s in plain if spans(*s) != 1] == []
    assert [s for s in spanned if spans(*s) < 3] == []
    for chains in (1, 7, 16, 33, 148, 1000):
        for n in (1, 5, 17, 18, 100, 1023):
            for d in (64, 128):
                g = spans(chains, n, d)
                assert g == 1 or (3 <= g <= n // 6 and (g - 1) * 2 * d // 64 * chains <= 296)
