"""quotient() of the transport kernel's voxel step (the index by voxel sizes that
are no power of two): a * y refined twice with the correctly rounded reciprocal y
of b (CPU, float arithmetic with exact fused multiply-adds) equals the correctly
rounded a / b.
"""

import numpy as np
import pytest

F = np.float32


def _quotient(a, b):
    """quotient() of gg_transport.cu in numpy: products and sums of a fused
    multiply-add in 64-bit mantissas, rounded once to float."""
    L = np.longdouble
    y = (F(1.0) / b).astype(F)

    def fma(p, q, r):
        return (p.astype(L) * q.astype(L) + r.astype(L)).astype(F)

    q = (a * y).astype(F)
    q = fma(fma(-q, b, a), y, q)
    return fma(fma(-q, b, a), y, q)


@pytest.mark.parametrize("seed", [1, 2])
def test_quotient_is_the_correctly_rounded_division(seed):
    rng = np.random.default_rng(seed)
    n = 1_000_000
    # wider than the step's positions (5e-4 ... 2048 mm) and voxel sizes (8e-3 ... 2048 mm)
    a = np.exp(rng.uniform(np.log(5.9e-8), np.log(1e4), n)).astype(F)
    b = np.exp(rng.uniform(np.log(1e-25), np.log(1e25), n)).astype(F)
    assert np.array_equal(_quotient(a, b), a / b)
    # mantissas at the ends, where a rounding error would show first
    ends = np.array([0, 1, 2, 3, 0x3FFFFF, 0x400000, 0x400001, 0x7FFFFC, 0x7FFFFD, 0x7FFFFE, 0x7FFFFF], np.uint32)
    ma = np.concatenate([ends, rng.integers(0, 1 << 23, 3000).astype(np.uint32)])
    a = (ma | np.uint32(0x3F800000)).view(F)
    b = (np.concatenate([ends, rng.integers(0, 1 << 23, 500).astype(np.uint32)]) | np.uint32(0x3F800000)).view(F)
    a, b = [x.reshape(-1).copy() for x in np.meshgrid(a, b)]
    assert np.array_equal(_quotient(a, b), a / b)
    assert np.array_equal(_quotient(-a, b), -a / b)
    assert not _quotient(np.zeros(3, F), b[:3]).any()
