"""Phase recovery at the edges of the walk's cases, against the oracle on the
same packed bispectrum (reconstruct_phases, phasereco.h:33-123): one, two, four
and eight CTAs a job with one or several parts per visit, batches of every
length, radii inside and beyond the map, odd sizes, and a bispectrum with a
zero region, whose points get no phase and are visited again.

  flags ........ identical
  phases ....... max <= 1e-3 rad, RMS <= 1e-4 rad at the flagged points (the
                 bounds of the parity tests)
"""
import numpy as np
import pytest
from conftest import phase_err

from oracle import bispec_desc

pytestmark = pytest.mark.gpu


def bispectrum(oracle, W, H, D, seed):
    """Packed bispectrum of three frames of a blob field."""
    rng = np.random.default_rng(seed)
    yy, xx = np.mgrid[0:H, 0:W].astype(float)
    B = np.zeros(bispec_desc(W, H, D)["base_size"], np.complex128)
    for _ in range(3):
        img = 0.02 * rng.random((H, W))
        for _ in range(6):
            x0, y0, s = W * rng.uniform(0.4, 0.6), H * rng.uniform(0.4, 0.6), rng.uniform(0.5, 1.2)
            img += rng.uniform(0.3, 1.0) * np.exp(-((xx - x0) ** 2 + (yy - y0) ** 2) / (2 * s * s))
        oracle.accumulate(B, np.fft.fft2(1000.0 * img), D, fp64=True)
    return (B / 3).astype(np.complex64)


@pytest.mark.parametrize("W,H,D,R", [
    (16, 16, 2, 6), (17, 19, 8, 8), (48, 40, 20, 40), (64, 64, 26, 30), (64, 64, 28, 30), (72, 80, 38, 36),
    (96, 96, 40, 44), (99, 75, 46, 60), (128, 128, 56, 40), (130, 128, 64, 40), (40, 40, 14, 1), (33, 64, 30, 0)])
@pytest.mark.parametrize("holes", [False, True])
def test_walk_shapes(smip, oracle, W, H, D, R, holes):
    B = bispectrum(oracle, W, H, D, 7 * W + H + D)
    if holes:  # no closure phase beyond 0.6 of the u_x range
        d = D // 2 * 2
        B = B.reshape(W // 2 + 1, -1).copy()
        B[int(0.6 * len(B)):] = 0
        B = B.ravel()
        assert B.size == (W // 2 + 1) * (H // 2 * 2 + 1) * (d // 2 + 1) * (d + 1)
    try:
        ph, fl, cs = oracle.reconstruct_phases(B, W, H, D, R)
    except IndexError:
        with pytest.raises(smip.OutOfRange):
            smip.reconstruct_phases(B, W, H, D, R)
        return
    got, gfl, gcs = smip.reconstruct_phases(B, W, H, D, R)
    assert np.array_equal(gfl, fl)
    m = fl > 0
    e = phase_err(got, ph, m)
    assert e.max() <= 1e-3 and np.sqrt((e ** 2).mean()) <= 1e-4, (e.max(), np.sqrt((e ** 2).mean()))
    assert np.all(got[~m] == 0) and np.all(gcs[~m] == 0)
    assert np.abs(gcs[m] - cs[m]).max() <= 1e-3


# a summing warp's plan row: one batch (20 words), two, the longest row that is
# kept in shared memory (39 words) and the first that is not (43)
@pytest.mark.parametrize("W,H,D,R", [(80, 64, 24, 32), (64, 80, 32, 32), (80, 81, 34, 36), (81, 80, 36, 36)])
def test_walk_rows(smip, oracle, W, H, D, R):
    B = bispectrum(oracle, W, H, D, 5 * W + H + D)
    ph, fl, cs = oracle.reconstruct_phases(B, W, H, D, R)
    got, gfl, gcs = smip.reconstruct_phases(B, W, H, D, R)
    assert np.array_equal(gfl, fl)
    m = fl > 0
    e = phase_err(got, ph, m)
    assert e.max() <= 1e-3 and np.sqrt((e ** 2).mean()) <= 1e-4, (e.max(), np.sqrt((e ** 2).mean()))
    assert np.abs(gcs[m] - cs[m]).max() <= 1e-3
