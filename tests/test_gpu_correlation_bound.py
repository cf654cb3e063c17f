"""The FP32 correlation's error against the bound that the peak search relies on
(k_xcorr.cu): positions within 8 2^-24 stages |ref| |frame| n of the FP32 peak are
scored exactly, so twice the error of any position has to stay below it.  The
largest sides, every radix, and images of one pixel, of noise and of a gradient.
The correlation in FP64 is numpy's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stages(L):
    """Stages that the bound counts for an axis of the mixed-radix path."""
    s, q = 0, 2
    while L > 1:
        while L % q == 0:
            s, L = s + q, L // q
        q += 1
    return s


@pytest.mark.parametrize("W,H", [(640, 480), (1000, 999), (1024, 1024), (768, 1024), (1023, 729), (997, 64), (875, 686),
                                 (64, 1009), (512, 512), (16, 512)])
@pytest.mark.parametrize("kind", ["noise", "centred", "point", "gradient"])
def test_correlation_error(smip, W, H, kind):
    rng = np.random.default_rng(W + H)
    ref = rng.integers(0, 4096, (H, W)).astype(float)
    if kind == "centred":
        ref -= 2048
    elif kind == "point":
        ref = np.zeros((H, W))
        ref[H // 3, W // 5] = 4095
    elif kind == "gradient":
        ref = np.floor(np.add.outer(np.arange(H), np.arange(W)) * 1.7)
    frame = np.roll(ref, (3, -7), (0, 1))
    if kind != "point":
        frame += rng.integers(0, 50, (H, W))
    c = smip.CrossCorrelation(ref)
    assert c(frame) == (-7, 3)
    n = W * H
    exact = np.fft.irfft2(np.conj(np.fft.rfft2(ref)) * np.fft.rfft2(frame), s=(H, W)) * n
    radix2 = all(v & (v - 1) == 0 and 16 <= v <= 512 for v in (W, H))
    count = np.log2(n) if radix2 else stages(W) + stages(H)
    bound = 8 * 2.0 ** -24 * count * np.linalg.norm(ref) * np.linalg.norm(frame) * n
    assert 2 * np.abs(c.get_correlation_array() - exact).max() <= bound
