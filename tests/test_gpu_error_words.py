"""Every stack has an error word of its own, also where they fill more than one
page (64 words), and a word that is taken again holds no old error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_error_words(smip):
    good = np.ones(smip.bispec_base_size(16, 16, 4), np.complex64)
    bad = good.copy()
    bad.real[:] = np.inf
    for broken in (range(0, 70, 9), (69,), ()):  # the later rounds take the words of the first
        stacks = [smip.Stack(16, 16, 4, batch_frames=1) for _ in range(70)]
        for k, st in enumerate(stacks):
            st.set_bispectrum(bad if k in broken else good)
        for k, st in enumerate(stacks):
            if k in broken:
                with pytest.raises(smip.OutOfRange):
                    st.reconstruct_phases(5)
            else:
                st.reconstruct_phases(5)
        for st in stacks[::2] + stacks[1::2]:
            st.close()
