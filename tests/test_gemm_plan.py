"""How a product's tiles are chosen (no GPU needed)."""
import ctypes
import random

import pytest

SMS = 148


def _plan(M, N, K, splits=1, a_mn=0, b_mn=0):
    from quantem_b200 import _lib

    bn, ctas, per = ctypes.c_int(0), ctypes.c_int64(0), ctypes.c_int(0)
    assert _lib.lib().ptycho_gemm_plan(M, N, K, splits, a_mn, b_mn, ctypes.byref(bn), ctypes.byref(ctas),
                                       ctypes.byref(per)) == 0
    return bn.value, ctas.value, per.value


def _rounds(M, N, bn):
    return -(-(-(-M // 128) * -(-N // bn)) // SMS)


@pytest.mark.parametrize("M,N,K", [(16384, 32, 9216), (16384, 64, 576), (17000, 32, 9216), (16384, 128, 9216),
                                   (18944, 32, 288), (14080, 32, 288)])
def test_one_round_stays_one_round(M, N, K):
    """Products whose widest tiles fit on the SMs at once are not cut into two rounds of narrower ones
    (128 CTAs of 32 columns take 58 us at 16384 x 32 x 9216, 256 CTAs of 16 columns 98)."""
    bn, ctas, per = _plan(M, N, K)
    assert bn == (32 if N <= 32 else 64 if N <= 64 else 128)
    assert ctas == -(-M // 128) * -(-N // bn) <= SMS and per == 1


@pytest.mark.parametrize("M,N", [(20000, 32), (65536, 32), (65536, 64), (262144, 16), (262144, 8), (20000, 50)])
def test_several_rounds_share_the_sms(M, N):
    """More CTAs than SMs at widths 32 and 64: two to an SM."""
    bn, ctas, per = _plan(M, N, 288)
    assert bn in (32, 64) and ctas > SMS and per == 2


@pytest.mark.parametrize("M,N", [(16, 1024), (4, 1024), (64, 512), (8, 16)])
def test_few_rows_take_narrow_tiles(M, N):
    assert _plan(M, N, 9216)[0] == 16


def test_no_other_width_is_cheaper():
    rng = random.Random(5)
    for _ in range(400):
        M, N = int(2 ** rng.uniform(0, 19)), int(2 ** rng.uniform(0, 11))
        rows = 128 if M >= 128 else (M + 7) // 8 * 8
        bn, ctas, _ = _plan(M, N, 512)
        assert ctas == -(-M // 128) * -(-N // bn)
        cost = _rounds(M, N, bn) * (rows + bn)
        for w in (16, 32, 64, 128):
            if w > max(32, 2 * N) or (w == 16 and _rounds(M, N, w) > 1) or (w == 128 and N <= 64) or (w == 64 and N <= 32):
                continue
            assert _rounds(M, N, w) * (rows + w) >= cost, (M, N, bn, w)


def test_plan_refuses_bad_arguments():
    from quantem_b200 import _lib

    for bad in ((0, 8, 8, 1, 0, 0), (8, 0, 8, 1, 0, 0), (8, 8, 0, 1, 0, 0), (8, 8, 8, 1, 1, 0)):
        assert _lib.lib().ptycho_gemm_plan(*bad, None, None, None) == 1
