"""The normalised bispectrum, (accumulator - compensation) / nframes, has the
bits of FP64 arithmetic rounded once, also where the quotient lies in the middle
of two floats or next to it, and the sign of a zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 7, 1000, 999983])
@pytest.mark.parametrize("off", [0, 1, -1])
def test_rounding(smip, tmp_path, n, off):
    W, H, D = 32, 17, 6
    rng = np.random.default_rng(n)
    size = 2 * smip.bispec_base_size(W, H, D)
    x = (2 * rng.integers(2**23, 2**24, size) + 1) * n + off  # 25 bits, odd, times n: an exact middle for off = 0
    b = x.astype(np.float32)
    c = (b.astype(np.int64) - x).astype(np.float32)
    assert np.array_equal(b.astype(np.float64) - c, x)
    scale = 2.0 ** rng.integers(-100, 60, size)
    b, c = (b * scale).astype(np.float32), (c * scale).astype(np.float32)
    b[:4], c[:4] = [0.0, -0.0, 0.0, -0.0], [0.0, 0.0, -0.0, -0.0]
    path = str(tmp_path / "state")
    with smip.Stack(W, H, D) as st:
        st.set_bispectrum(np.zeros(size // 2, np.complex64), n)
        st.save_state(path)
    raw = bytearray(open(path, "rb").read())
    raw[48:48 + 4 * size] = b.tobytes()  # the header, the accumulator, its compensation
    raw[48 + 4 * size:48 + 8 * size] = c.tobytes()
    open(path, "wb").write(raw)
    with smip.Stack(W, H, D) as st:
        st.load_state(path)
        got = st.bispectrum().view(np.float32)
    exp = ((b.astype(np.float64) - c) * (1.0 / n)).astype(np.float32)
    assert np.array_equal(got.view(np.uint32), exp.view(np.uint32))
