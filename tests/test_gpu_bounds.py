"""The single-precision bounds that decide most draws, against the exact test."""
import numpy as np
import pytest

from b200sa import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_bounds_never_disagree_with_the_exact_test(seed):
    """Half of the samples lie within 2^-8 (relative) of the boundary: the
    band of 2^-10 holds 2^-10 / (2^-8 log2(e)) = 0.174 of those, 0.087 of all.
    Draws below 2^52 are left open: 0.01 of the Metropolis and Gibbs samples at
    the boundary.  Gibbs samples there with z below -6.2 (0.11) are at a draw of
    2^64 - 1 half of the time, inside the band too.  Path-integral samples beyond
    |x| = 12 (0.04) are at the ends of the draws.  One in 32 each has an extreme
    beta or draw, four in 32 an energy at the threshold, whose boundary is a draw
    below 2^52."""
    counts = np.zeros(9, dtype=np.int64)
    err = _lib.errbuf()
    n = 1 << 24
    _lib.check(_lib.load().b200sa_check_bounds(n, seed, 0, counts.ctypes.data, err, len(err)), err)
    for k, share in enumerate((0.087 + 0.005 + 4 / 32, 0.087 + 0.005 + 0.03 + 4 / 32, 0.087 + 0.02)):
        samples, decided, wrong = counts[3 * k:3 * k + 3]
        assert samples == n and wrong == 0
        assert decided > (1 - share - 0.02) * n
