"""A radius whose tables do not fit the device is refused, and the stack goes on
with the radii that do, the one it was prepared for among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_radius_beyond_the_memory(smip):
    rng = np.random.default_rng(8)
    size = smip.bispec_base_size(80, 80, 64)
    B = (1 + 0.1 * rng.standard_normal(size) + 0.1j * rng.standard_normal(size)).astype(np.complex64)
    with smip.Stack(80, 80, 64) as st:
        st.set_bispectrum(B)
        st.reconstruct_phases(20)
        with pytest.raises(smip.NoMemory):
            st.prepare_reco(2000)  # 15 million visits of 34 KB
        for radius in (20, 12):
            with smip.Stack(80, 80, 64) as fresh:
                fresh.set_bispectrum(B)
                exp = fresh.reconstruct_phases(radius)
            got = st.reconstruct_phases(radius)
            assert all(np.array_equal(g, e) for g, e in zip(got, exp))
