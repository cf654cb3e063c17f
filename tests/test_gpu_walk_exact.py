"""The phase walk to the bit and to the pair: the same results with one, two, four
and eight CTAs a job and from call to call, and at every point the number of
pairs that the reference forms it from (a pair lost, doubled or read too early
changes that number or the bits).

  consistency .. max <= 1e-4 (a mean over the pairs of errors of at most two
                 phases, each within 5e-5 of FP64)
"""
import numpy as np
import pytest
from test_gpu_walk import bispectrum

pytestmark = pytest.mark.gpu


def pair_counts(smip, W, H, D, R):
    """calc_phase's counts (phasereco.h:75-123) where no element of B is zero."""
    e = D // 2
    x0, y0 = -(W >> 1), -(H >> 1)
    flag = np.zeros((H + 2 * e, W + 2 * e), bool)  # centred, with a margin that holds no phase
    count = np.zeros((H, W), np.int32)
    for x, y in ((0, 0), (1, 0), (0, 1), (-1, 0), (0, -1)):
        flag[y - y0 + e, x - x0 + e] = True
        count[y, x] = -1
    box = slice(-y0, -y0 + 2 * e + 1), slice(-x0, -x0 + 2 * e + 1)  # the points v
    for x, y in smip.reco_visits(R):
        if not (x0 <= x < x0 + W and y0 <= y < y0 + H) or count[y, x] != 0:
            continue
        u = flag[y - y0:y - y0 + 2 * e + 1, x - x0:x - x0 + 2 * e + 1][::-1, ::-1]  # w - v
        n = int((u & flag[box]).sum())
        if n:
            count[y, x] = n
            flag[y - y0 + e, x - x0 + e] = True
    return count


@pytest.mark.parametrize("W,H,D,R", [
    (16, 16, 2, 6), (17, 19, 8, 8), (48, 40, 20, 40), (64, 64, 26, 30), (64, 64, 28, 30), (80, 81, 34, 36),
    (72, 80, 38, 36), (96, 96, 40, 44), (99, 75, 46, 60), (130, 128, 64, 40)])
def test_walk_exact(smip, oracle, W, H, D, R):
    B = bispectrum(oracle, W, H, D, 3 * W + H + D)
    B[B == 0] = 1  # every pair counts
    assert np.all(np.abs(B) > 1e-10)
    _, fl, cs = oracle.reconstruct_phases(B, W, H, D, R)
    counts = pair_counts(smip, W, H, D, R)
    with smip.Stack(W, H, D) as st:
        with pytest.raises(smip.BadFunctionCall):
            st.reco_counts()
        st.set_bispectrum(B)
        exp = st.reconstruct_phases(R)
        assert np.array_equal(exp[1], fl)
        assert np.abs(exp[2] - cs)[fl > 0].max() <= 1e-4
        for ctas in (0, 1, 2, 4, 8):
            st.set_walk_ctas(ctas)
            for _ in range(3):
                got = st.reconstruct_phases(R)
                assert all(np.array_equal(g, e) for g, e in zip(got, exp))
                assert np.array_equal(st.reco_counts(), counts)
        with pytest.raises(smip.InvalidArgument):
            st.set_walk_ctas(3)
