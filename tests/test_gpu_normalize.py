"""The normalised bispectrum (bispectrum / nframes, smip-cli/main.cpp:307-312)
over the range of FP32, against the same arithmetic in FP64: within one unit
in the last place everywhere, and the same zeros, infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 1000, 2**20 + 7])
@pytest.mark.parametrize("shape", [(16, 16, 2), (17, 19, 2)])  # an even and an odd number of elements
def test_normalized_values(smip, n, shape):
    W, H, D = shape
    rng = np.random.default_rng(n)
    size = smip.bispec_base_size(W, H, D)
    mag = 10.0 ** rng.uniform(-44, 31, 2 * size) * rng.choice([-1, 1], 2 * size)
    mag[:8] = [0.0, -0.0, np.inf, -np.inf, np.nan, 1e-44, 3e31, -1e-24]
    b = mag.astype(np.float32)
    with smip.Stack(W, H, D) as st:
        st.set_bispectrum(b.view(np.complex64), n)
        got = st.bispectrum().view(np.float32)
    with np.errstate(all="ignore"):
        acc = (b.astype(np.float64) * n).astype(np.float32)  # what the accumulator resumes as
        exp = (acc.astype(np.float64) * (1.0 / n)).astype(np.float32)
    fine = np.isfinite(exp)
    assert np.array_equal(np.isnan(got), np.isnan(exp))
    assert np.array_equal(got[~fine & ~np.isnan(exp)], exp[~fine & ~np.isnan(exp)])
    assert np.array_equal(got[exp == 0], exp[exp == 0])
    assert np.all(np.abs(got[fine].astype(np.float64) - exp[fine]) <= np.spacing(np.abs(exp[fine])))
