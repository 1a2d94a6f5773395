"""What a request is accounted for at admission: a budget holds as many FP32 requests as it did when a pair's rows,
CSR entries, tensors and slots took 92 bytes, which they still fit."""
import ctypes
import math

import pytest

from dmff_b200 import _lib as L


@pytest.mark.parametrize("n,rc,K,V,lpol", [(450, 8.0, (17, 17, 17), 4491.0, 1), (30000, 8.0, (68, 68, 68), 299401.0, 1),
                                           (3000, 6.0, (32, 30, 28), 29940.0, 0)])
def test_request_footprint(n, rc, K, V, lpol):
    half = n * n / V * 4.0 / 3.0 * math.pi * rc ** 3 / 2.0
    K3 = K[0] * K[1] * K[2]
    want = n * (920.0 if lpol else 600.0) + 92.0 * half + (20.0 if lpol else 16.0) * K3
    got = L.load().dmffb_request_footprint(n, rc, (ctypes.c_int32 * 3)(*K), V, lpol)
    assert abs(got - want) <= 1e-9 * want + 1
    # a half pair of an FP32 engine: rows, CSR, tensors with their headroom, slots
    assert 1.3 * (12 + 8 + 32) + 2 * 1.35 * 4 <= 92
