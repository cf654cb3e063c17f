"""The reference frame's sum of squares, which the peak search's bound holds: that
of integer frames is exact, that of floating ones within 2^-40 (a float pair per
block, whose terms are all positive).  It is the last number of the saved state
but the reference's spectrum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32, np.float64])
@pytest.mark.parametrize("W,H", [(16, 16), (512, 64), (48, 35), (3, 3), (1024, 31), (127, 130)])
def test_reference_norm(smip, tmp_path, dtype, W, H):
    rng = np.random.default_rng(W * H)
    if np.issubdtype(dtype, np.integer):
        ref = rng.integers(0, np.iinfo(dtype).max + 1, (H, W)).astype(dtype)
        exact = float(sum(int(v) ** 2 for v in ref.ravel()))
    else:
        ref = (rng.standard_normal((H, W)) * 10.0 ** rng.uniform(-3, 3, (H, W))).astype(dtype)
        exact = float((ref.astype(np.longdouble) ** 2).sum())
    path = str(tmp_path / "state")
    with smip.Stack(W, H, 2) as st:
        st.push_frames(np.stack([ref, ref]))
        st.save_state(path)
        half = (W // 2 + 1) * H
        at = 48 + 16 * st.base_size + 8 * half + 8 * W * H + 2 * 8 + ref.nbytes
    raw = open(path, "rb").read()
    assert len(raw) == at + 8 + 8 * half
    got = np.frombuffer(raw, np.float64, 1, at)[0]
    if np.issubdtype(dtype, np.integer):
        assert got == exact
    else:
        assert abs(got - exact) <= 2.0 ** -40 * exact
