"""The integer-pipe products and conversions of siminf_stream.h against the
hardware's, bit for bit, on the host (the same code runs on the device)."""
import ctypes as C

import numpy as np
import pytest


def exact_ops(oracle_lib, a, n):
    a = np.ascontiguousarray(a, dtype=np.float64)
    n = np.ascontiguousarray(n, dtype=np.int32)
    product, conv, trunc = np.empty(len(a)), np.empty(len(a)), np.empty(len(a), np.int32)
    f = oracle_lib.lib().oracle_exact_ops
    f.restype = None
    f.argtypes = [C.c_void_p] * 5 + [C.c_int64]
    f(a.ctypes.data, n.ctypes.data, product.ctypes.data, conv.ctypes.data, trunc.ctypes.data,
      len(a))
    return product, conv, trunc


EDGES_A = [0.0, -0.0, 1.0, -1.0, 0.16, 5e-324, 2.2250738585072014e-308, 1.7976931348623157e308,
           1e299, np.inf, -np.inf, np.nan, 2.0 ** 52 + 1, 2.0 ** 53 - 1, 1 + 2.0 ** -52]
EDGES_N = [0, 1, -1, 2, 3, 2 ** 31 - 1, -2 ** 31, 65535, 65536, 65537]


@pytest.mark.parametrize("kind", ["edges", "any", "rates", "ties"])
def test_exact_ops_match_the_hardware(oracle_lib, kind):
    rng = np.random.default_rng(5)
    k = 200000
    bits = rng.integers(0, 2 ** 64, k, dtype=np.uint64)
    n = (rng.integers(-2 ** 31, 2 ** 31, k) >> rng.integers(0, 31, k)).astype(np.int32)
    if kind == "edges":
        a, n = [x.reshape(-1) for x in np.meshgrid(EDGES_A, np.array(EDGES_N, dtype=np.int64))]
        n = n.astype(np.int32)
    elif kind == "any":
        a = bits.view(np.float64)
    elif kind == "rates":
        a = np.exp(rng.uniform(-12, 6, k))
    else:                                   # few mantissa bits: products halfway between doubles
        a = (bits & ~((np.uint64(1) << rng.integers(20, 53, k).astype(np.uint64)) - np.uint64(1)))
        a = ((a & np.uint64(0x800FFFFFFFFFFFFF)) | np.uint64(0x3FE0000000000000)).view(np.float64)
        a = a * (1 + 2.0 ** -rng.integers(20, 52, k))
    with np.errstate(all="ignore"):
        want = a * n.astype(np.float64)
    product, conv, trunc = exact_ops(oracle_lib, a, n)
    same = product.view(np.uint64) == want.view(np.uint64)
    assert np.all(same | (np.isnan(product) & np.isnan(want)))
    assert np.array_equal(conv, n.astype(np.float64))
    small = np.abs(a) < 2.0 ** 31
    assert np.array_equal(trunc[small], a[small].astype(np.int32))
