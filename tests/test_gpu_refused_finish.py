"""A refused reconstruction leaves nothing behind: no kernel is launched for it,
and the stack's next job reports only its own errors."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_refused_finish_launches_nothing(smip):
    rng = np.random.default_rng(3)
    frames = rng.integers(0, 4096, (4, 64, 64)).astype(np.uint16)
    b = np.ones(smip.bispec_base_size(64, 64, 16), np.complex64)
    b.real[:] = np.inf  # every phasor is out of range: a walk over it would record an error
    with smip.Stack(64, 64, 16) as st:
        st.prepare_reco(24)
        st.set_bispectrum(b)
        n = smip.kernel_launches()
        with pytest.raises(smip.BadFunctionCall):  # there is no power spectrum to form an image from
            st.finish(24)
        assert smip.kernel_launches() == n
        st.reset()
        st.push_frames(frames)
        st.sync()
        time.sleep(0.05)
        st.sync()
        assert st.nframes == 4
        n = smip.kernel_launches()
        with pytest.raises(smip.DomainError):  # no window without a radius
            st.finish(0.0)
        assert smip.kernel_launches() == n
        with smip.Stack(64, 64, 16) as fresh:
            fresh.push_frames(frames)
            exp = fresh.finish(24)
        for got, e in zip(st.finish(24), exp):
            assert np.array_equal(got, e)
