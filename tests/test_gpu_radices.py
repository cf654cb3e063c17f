"""Every radix of the mixed-radix transforms through the whole pipeline, against
the FP64 oracle: 2 alone, 3, 4, 5, 7, 8 and larger primes in either direction,
odd numbers of rows and frames, the smallest sides, and each frame type.

  shifts, shift-and-add sum ............... bit-exact
  power spectrum .......................... max |dP| <= 1e-6 max P
  bispectrum (normalised) ................. rel-L2 <= 1e-5
"""
import numpy as np
import pytest
from conftest import rel_l2
from test_gpu_generic_sizes import speckle_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,D,n,dtype", [
    (56, 42, 8, 5, np.uint8),      # 7 8, 2 3 7
    (49, 30, 6, 4, np.uint16),     # 7 7, 2 3 5
    (52, 26, 6, 3, np.uint16),     # 13 4, 13 2
    (17, 34, 4, 4, np.uint8),      # primes
    (25, 27, 6, 7, np.float32),    # 5 5, 3 3 3
    (11, 9, 4, 3, np.uint8),
    (96, 31, 10, 9, np.float64),   # 3 8 4
    (1024, 36, 8, 2, np.uint16),   # 4 4 8 8
    (48, 640, 12, 18, np.uint16),  # long columns, more than one chunk of frames
    (6, 5, 2, 2, np.uint8)])
def test_radices(smip, oracle, W, H, D, n, dtype):
    base = np.uint8 if dtype == np.uint8 else np.uint16
    frames = speckle_frames(W, H, n, base, seed=W * 131 + H).astype(dtype)
    exp = oracle.run_stack(frames, D, 2.0, fp64=True, nthreads=8)
    with smip.Stack(W, H, D, batch_frames=17) as st:
        st.push_frames(frames)
        shifts, total, power, bispec = st.shifts(), st.sum(), st.power(), st.bispectrum()
    assert np.array_equal(shifts, exp["shifts"])
    assert np.array_equal(total, exp["sum"])
    p = np.real(exp["power"])
    assert np.abs(power - p).max() <= 1e-6 * p.max()
    assert rel_l2(bispec, exp["bispec"]) <= 1e-5
