"""Host replay of the integer arithmetic around the BF16 slices, checked on the CPU: the keys
by which magnitudes are compared and scales found (abs_key, key_exp in
dynemol_gb300/csrc/tc_ptx.cuh), a digit's BF16 bits (digit_bf16), and the tagged 128-bit partial
sums of oz_cheb_kernel (order_tag, store_partial, untag in ozaki.cu)."""
import math
import os
import random
import re
import struct

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dynemol_gb300", "csrc")
TC = re.sub(r"\s+", " ", open(os.path.join(CSRC, "tc_ptx.cuh")).read())
OZ = re.sub(r"\s+", " ", open(os.path.join(CSRC, "ozaki.cu")).read())


def test_replay_is_the_source():
    assert ("const unsigned k = ((unsigned)__double2hiint(x) & 0x7fffffffu) | (__double2loint(x) != 0 ? 1u : 0u); "
            "return k > 0x7ff00000u ? 0u : k;") in TC
    assert "return key ? (int)(key >> 20) - 1022 : 0;" in TC
    assert "__float_as_uint(__fsub_rn(__int_as_float(0x4b400000 + n), 12582912.0f)) >> 16" in TC
    assert "constexpr int kTagShift = 54;" in OZ
    assert "return (unsigned long long)(k % 1023 + 1);" in OZ
    assert "return I128{(long long)(w.y << (64 - kTagShift)) >> (64 - kTagShift), w.x};" in OZ
    assert "constexpr unsigned long long kMask = (1ull << kTagShift) - 1;" in OZ
    assert "((unsigned long long)A[u].hi & kMask) | (order_tag(k) << kTagShift)" in OZ


def words(x):
    b = struct.unpack("<Q", struct.pack("<d", x))[0]
    return b >> 32, b & 0xffffffff


def abs_key(x):
    hi, lo = words(x)
    k = (hi & 0x7fffffff) | (1 if lo else 0)
    return 0 if k > 0x7ff00000 else k


def key_exp(key):
    return (key >> 20) - 1022 if key else 0


SPECIAL = [0.0, -0.0, 1.0, -1.0, 0.5, math.nextafter(1.0, 0.0), math.nextafter(1.0, 2.0), math.nextafter(2.0, 0.0), 2.0,
           2.0 ** -1022, math.nextafter(2.0 ** -1022, 0.0), 5e-324, -5e-324, 2.0 ** -1030, 1.7976931348623157e308,
           -1.7976931348623157e308, 2.0 ** 1023]


def test_scale_of_an_element():
    rng = random.Random(1)
    values = SPECIAL + [math.ldexp(rng.uniform(-1, 1), rng.randint(-1070, 1024)) for _ in range(20000)]
    for x in values:
        e = key_exp(abs_key(x))
        if x == 0.0:
            assert abs_key(x) == 0 and e == 0
        else:
            assert abs_key(x) != 0
            # |x| < 2^e, and for normal x the smallest such power
            if e <= 1023:
                assert abs(x) < math.ldexp(1.0, e)
            if abs(x) >= 2.0 ** -1022:
                assert abs(x) >= math.ldexp(1.0, e - 1) and e == math.frexp(x)[1]
            else:
                assert e == -1022
    assert abs_key(math.nan) == 0 and abs_key(-math.nan) == 0  # as fmax: no element
    assert abs_key(math.inf) == 0x7ff00000 and key_exp(0x7ff00000) == 1025
    assert abs_key(math.inf) > abs_key(1.7976931348623157e308)


def test_the_largest_key_has_the_largest_scale():
    rng = random.Random(2)
    for _ in range(3000):
        xs = [math.ldexp(rng.uniform(-1, 1), rng.randint(-8, 8)) for _ in range(rng.randint(1, 40))]
        xs += rng.sample(SPECIAL, 2) + ([math.nan] if rng.random() < 0.2 else [])
        top = max((abs(x) for x in xs if not math.isnan(x)), default=0.0)
        assert key_exp(max(abs_key(x) for x in xs)) == key_exp(abs_key(top))


def test_digits_as_bf16():
    for n in range(-256, 257):
        magic = struct.unpack("<f", struct.pack("<I", (0x4b400000 + n) & 0xffffffff))[0]
        d = np.float32(magic) - np.float32(12582912.0)
        bits = struct.unpack("<I", struct.pack("<f", float(d)))[0]
        assert bits & 0xffff == 0  # exact in BF16
        assert struct.unpack("<f", struct.pack("<I", (bits >> 16) << 16))[0] == n


M64 = (1 << 64) - 1


def order_tag(k):
    return k % 1023 + 1


def pack(s, k):  # s: |s| < 2^116 as two's complement
    u = s & ((1 << 128) - 1)
    lo, hi = u & M64, u >> 64
    return lo, (hi & ((1 << 54) - 1)) | (order_tag(k) << 54)


def untag(w):
    lo, y = w
    hi = (y << 10) & M64
    hi = hi - (1 << 64) if hi >> 63 else hi
    return (hi >> 10 << 64) + lo


@pytest.mark.parametrize("k", [1, 2, 1021, 1022, 1023, 1024, 2045, 2046, 5000])
def test_tagged_partials(k):
    rng = random.Random(k)
    edge = 1 << 116
    for s in [0, 1, -1, edge - 1, -edge + 1, 1 << 64, -(1 << 64), (1 << 64) - 1, -(1 << 63)] + \
             [rng.randint(-edge, edge) >> rng.randint(0, 116) for _ in range(2000)]:
        w = pack(s, k)
        assert w[1] < 1 << 64 and w[1] >> 54 == order_tag(k)
        assert untag(w) == s


def test_tags_of_neighbouring_orders():
    """A slot holds the last order's word until this order's: never the tag that is waited for,
    nor the cleared memory's 0, at the wrap either."""
    for k in range(1, 5000):
        assert 1 <= order_tag(k) <= 1023
        assert order_tag(k) != order_tag(k - 1)
