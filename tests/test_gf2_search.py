"""The GF(2) echelon panel at the edges of its pivot search (window of 128 positions by columns, rows
past it, columns without a pivot, single columns) and of the block updates.  Exact against the CPU
oracle."""
import numpy as np
import pytest

import oracle
from lela_b200 import gen


def _check(cuda, A, n):
    want, wr = oracle.echelon_gf2(A, n)
    got, gr = cuda.echelonize_gf2(A.copy(), n)
    assert gr == wr
    assert np.array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(1, 1), (31, 33), (32, 64), (33, 65), (64, 64), (63, 129), (127, 100), (128, 128),
                                 (129, 64), (130, 200), (300, 90), (700, 600), (1500, 1100)])
def test_shapes(cuda, m, n):
    _check(cuda, gen.dense_gf2(m + n, m, n), n)
    bits = gen.unpack_gf2(gen.dense_gf2(7, m, n), n).copy()
    g = np.random.default_rng(m * n)
    bits[:, g.random(n) < 0.3] = 0            # columns without a pivot
    bits[g.random(m) < 0.2] = 0               # zero rows
    bits[m // 2:] = bits[: m - m // 2]        # dependent rows
    _check(cuda, gen.pack_gf2(bits), n)


@pytest.mark.gpu
@pytest.mark.parametrize("zero", [100, 127, 128, 129, 200, 640])
def test_pivots_past_the_window(cuda, zero):
    g = np.random.default_rng(zero)
    m, n = 900, 700
    bits = gen.unpack_gf2(gen.dense_gf2(zero, m, n), n).copy()
    bits[:zero, :40] = 0                      # the first rows have none of the first pivots
    bits[zero:, 5:9] = 0
    bits[g.choice(m, 300, replace=False), 64:90] = 0
    _check(cuda, gen.pack_gf2(bits), n)


@pytest.mark.gpu
def test_bits_past_the_last_column(cuda):
    """Rows below the pivots keep the bits past column n of their last word while the panel's own block is
    updated: the form's columns are those of the clean matrix."""
    m, n = 800, 500
    A = gen.dense_gf2(3, m, n)
    want, wr = oracle.echelon_gf2(A, n)
    B = A.copy()
    B[:, -1] |= np.uint64(1) << np.uint64(60)
    got, gr = cuda.echelonize_gf2(B, n)
    mask = np.uint64((1 << (n & 63)) - 1)
    got[:, -1] &= mask
    assert gr == wr and np.array_equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n", [(1100, 577), (1400, 1153), (1100, 1090), (2000, 1600)])
@pytest.mark.parametrize("dependent", [0.0, 0.1, 0.6])
def test_block_solve(cuda, m, n, dependent):
    """Blocks of eight panels with words right of them: an even and an odd number of those, full
    blocks and blocks whose pivots end inside a word."""
    g = np.random.default_rng(m + n)
    bits = gen.unpack_gf2(gen.dense_gf2(m * n, m, n), n).copy()
    cols = np.flatnonzero(g.random(n) < dependent)
    bits[:, cols] = bits[:, g.permutation(n)[: len(cols)]]
    _check(cuda, gen.pack_gf2(bits), n)
