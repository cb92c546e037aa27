"""The digit products' accumulators: whole numbers that FP32 holds.

An accumulator of the FP64 Legendre contractions takes DG_KB chunks of 32
values of K before it is drained.  Levels 2 to 5 (digits i and j with i + j =
level) have to stay within 2^24 whatever the data's digits are, at most 256
in magnitude each: 256 times the sum of the table's digit magnitudes over a block
of K, computed here from the tables of the smallest, ordinary and largest
plans, with what the drain adds to a level before it is converted.
"""
import os
import re

import numpy as np
import pytest

from conftest import ROOT

SRC = os.path.join(ROOT, "dennou-ccm_gb300", "csrc", "legendre_dg.cu")
LIMIT = 2.0 ** 24


def block():
    text = open(SRC).read()
    return int(re.search(r"constexpr int DG_KB = (\d+)", text)[1]) * int(re.search(r"constexpr int DG_CHUNK = (\d+)", text)[1])


def pbar(N, m, mu):
    """Pbar_n^m(mu), n = m .. N, integral of the square 2, no sign factor."""
    P = np.zeros((N + 1 - m, len(mu)))
    k = np.arange(1, m + 1)
    P[0] = np.exp(0.5 * np.sum(np.log((2 * k + 1) / (2 * k))) + m * 0.5 * np.log1p(-mu ** 2))
    if m < N:
        P[1] = np.sqrt(2 * m + 3) * mu * P[0]
    for n in range(m + 2, N + 1):
        e, f = (np.sqrt((q * q - m * m) / (4.0 * q * q - 1)) for q in (n, n - 1))
        P[n - m] = (mu * P[n - m - 1] - f * P[n - m - 2]) / e
    return P


def digits(x, E):
    """The seven balanced 9-bit digits of x, |x| < 2^E (broadcast)."""
    q = np.rint(np.ldexp(x, 62 - E)).astype(np.int64)
    out = []
    for _ in range(6):
        d = (q + 256) % 512 - 256
        out.append(d)
        q = (q - d) >> 9
    return [q] + out[::-1]


def worst(table, K):
    """Largest sums over the blocks of K columns of the digit magnitudes: by
    the number of leading digits, 1 .. 5."""
    E = np.frexp(np.abs(table).max(axis=1))[1]
    d = np.abs(np.stack(digits(table, E[:, None])[:5])).cumsum(axis=0)
    return np.array([[d[j][:, k:k + K].sum(axis=1).max() for k in range(0, table.shape[1], K)] for j in range(5)]).max(axis=1)


@pytest.mark.parametrize("N,J,step", [(21, 32, 1), (85, 128, 1), (21, 2200, 1), (170, 256, 5), (300, 514, 13), (341, 512, 17),
                                      (511, 512, 29)])
def test_levels_stay_whole(N, J, step):
    mu, w = np.polynomial.legendre.leggauss(J)
    mu, w = mu[J // 2:], w[J // 2:]
    top = np.zeros(5)
    for m in sorted(set(range(0, min(N, 4) + 1)) | set(range(0, N + 1, step))):
        P = pbar(N, m, mu)
        for p in (0, 1):
            if m + p > N:
                continue
            # synthesis: rows of latitudes over the degrees of one parity (rows
            # that vanish to FP64 aside)
            rows = P[p::2].T
            rows = rows[np.abs(rows).max(axis=1) > 1e-290]
            if len(rows):
                top = np.maximum(top, worst(rows, block()))
            # analysis: rows of degrees over the latitudes, each latitude's
            # largest entry brought to [1/2, 1)
            t = 0.5 * w * P[p::2]
            scale = np.abs(t).max(axis=0)
            t = np.ldexp(t, -np.frexp(scale)[1])[:, scale > 1e-290]
            if t.shape[1]:
                top = np.maximum(top, worst(t, block()))
    level = 256.0 * top  # of levels 2 .. 6
    assert (level[:4] <= LIMIT).all(), level / LIMIT
    # converted with multiples of 512 of the level below, and 512 times what is
    # left of level 4
    assert level[1] + level[2] / 512 <= LIMIT
    assert level[3] + 256 * 512 + level[4] / 512 <= LIMIT
