"""The peak search's paths, against the oracle: a single candidate, several (a
periodic frame has equal peaks, the lowest index wins), more than the candidate
list holds, frames whose sums of squares leave the FP32 range, and the
allocation-free entry point with its frames a whole or a broken number of
pixels apart."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32, np.float64])
@pytest.mark.parametrize("W,H", [(64, 32), (48, 35)])
@pytest.mark.parametrize("kind", ["noise", "periodic", "constant", "zero"])
def test_stack_shifts(smip, oracle, dtype, W, H, kind):
    rng = np.random.default_rng(W + H)
    ref = rng.integers(0, 200, (H, W))
    if kind == "periodic":  # equal peaks every W / 4 columns
        ref = np.tile(ref[:, :W // 4], (1, 4))
    elif kind == "constant":  # every position is a peak
        ref = np.full((H, W), 7)
    elif kind == "zero":
        ref = np.zeros((H, W), int)
    frames = np.stack([np.roll(ref, s, (0, 1)) for s in ((0, 0), (2, -3), (-1, 5), (0, 0), (5, 1))]).astype(dtype)
    exp = oracle.run_stack(frames, 4, 2.0, fp64=True)["shifts"]
    for batch in (8, 2):  # the reference in the same batch, and kept from an earlier one
        with smip.Stack(W, H, 4, batch_frames=batch) as st:
            st.push_frames(frames)
            assert np.array_equal(st.shifts(), exp)


@pytest.mark.parametrize("scale", [1e-20, 1e-14, 1e16])
def test_norms_at_the_ends_of_the_range(smip, scale):
    rng = np.random.default_rng(5)
    ref = rng.random((32, 64))
    frames = np.stack([np.roll(ref, s, (0, 1)) for s in ((0, 0), (3, -4), (-2, 6))])
    with smip.Stack(64, 32, 4) as st:
        st.push_frames(frames)
        exp = st.shifts()
    assert exp.tolist() == [[0, 0], [-4, 3], [6, -2]]
    with smip.Stack(64, 32, 4) as st:
        st.push_frames(frames * scale)
        assert np.array_equal(st.shifts(), exp)


@pytest.mark.parametrize("W,H", [(16, 16), (64, 32), (256, 256)])
def test_noalloc_distances(smip, W, H):
    import torch

    rng = np.random.default_rng(W)
    ref = rng.integers(0, 3000, (H, W)).astype(np.float64)
    frame = np.roll(ref, (3, -2), (0, 1))
    exp = smip.CrossCorrelation(ref)(frame)
    n = W * H
    buf = torch.zeros(2 * n + 64, dtype=torch.float64, device="cuda")
    out = torch.zeros(2, dtype=torch.int32, device="cuda")
    for first, second in ((0, n), (n + 8, 3), (5, n + 20)):  # either order, any gap
        buf[first:first + n] = torch.from_numpy(ref.ravel())
        buf[second:second + n] = torch.from_numpy(frame.ravel())
        smip.xcorr_displacement_noalloc(buf[first:].data_ptr(), buf[second:].data_ptr(), W, H, out.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert tuple(out.tolist()) == exp
