"""Elements of the bispectrum that are not numbers, in the phase walk.

An element with an infinite real part is reported like one outside the array,
but only if a point is formed from it (calc_phase leaves a point that has its
phase alone, phasereco.h:81-84).  One with an infinite imaginary part and a
finite real part has the phasor (0, NaN): a point that is formed from it has a
consistency that is NaN and the phase zero, and so have the points formed from
that one.
"""
import numpy as np
import pytest

from oracle import bispec_desc

pytestmark = pytest.mark.gpu


def sparse(W, H, D, fraction, seed):
    """A bispectrum with zero elements, whose pairs are left out."""
    rng = np.random.default_rng(seed)
    size = bispec_desc(W, H, D)["base_size"]
    zero = rng.random(size) < fraction
    return np.where(zero, 0, np.exp(2j * np.pi * rng.random(size))).astype(np.complex64)


# pairs of (3, 0) or (4, 0) whose members get their phases after the point has
# its own (visits 31 and 57) and before its next visits (55 and 81); no other
# point is formed from these elements
@pytest.mark.parametrize("D,R,fraction,seed,element", [
    (8, 6, 0.5, 0, 2260), (8, 6, 0.5, 0, 3025), (8, 6, 0.7, 34, 836), (6, 6, 0.3, 13, 1884), (14, 7, 0.3, 8, 2204),
    (14, 7, 0.7, 23, 6016)])
def test_errors_of_a_point_that_has_its_phase(smip, oracle, D, R, fraction, seed, element):
    B = sparse(16, 16, D, fraction, seed)
    assert B[element] != 0
    bad = B.copy()
    bad[element] = complex(np.inf, 0)
    exp = smip.reconstruct_phases(B, 16, 16, D, R)
    for a, b in zip(oracle.reconstruct_phases(B, 16, 16, D, R), oracle.reconstruct_phases(bad, 16, 16, D, R)):
        assert np.array_equal(a, b)
    got = smip.reconstruct_phases(bad, 16, 16, D, R)
    for g, e in zip(got, exp):
        assert np.array_equal(g, e)


def test_errors_that_count(smip):
    B = sparse(16, 16, 8, 0.0, 1)
    B[smip.bispec_offsets(16, 16, 8, [[1, 0, 1, 0]])[0]] = complex(np.inf, 0)  # forms (2, 0), the spiral's first point
    with pytest.raises(smip.OutOfRange):
        smip.reconstruct_phases(B, 16, 16, 8, 6)


# recent pairs and older ones; a point near the origin and points of the last
# turns; a summing warp's plan row in one part and in several
@pytest.mark.parametrize("W,H,D,R,pair", [
    (32, 32, 8, 12, (9, 2, 2, -1)), (32, 32, 8, 12, (11, -3, -1, 4)), (32, 32, 8, 12, (2, 0, 1, 1)),
    (48, 40, 14, 18, (-17, 2, 1, 1)), (64, 64, 24, 20, (14, 5, 4, 3)), (96, 96, 40, 24, (10, -10, 10, 3))])
def test_infinite_imaginary_part(smip, oracle, W, H, D, R, pair):
    B = sparse(W, H, D, 0.0, W + D)
    off = smip.bispec_offsets(W, H, D, [pair])[0][0]
    B[off] = complex(0.5, np.inf)
    ph, fl, cs = oracle.reconstruct_phases(B, W, H, D, R)
    lost = np.isnan(cs)
    assert lost.any()
    got, gfl, gcs = smip.reconstruct_phases(B, W, H, D, R)
    assert np.array_equal(gfl, fl)
    assert np.array_equal(np.isnan(gcs), lost)
    assert np.array_equal(got[lost], ph[lost]) and np.all(got[lost] == 0)
