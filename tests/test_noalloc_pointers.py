"""The allocation-free shift refuses pointers that its kernels could not load
through, on the host and before any device call (so these cases need no GPU)."""
import pytest


@pytest.mark.parametrize("ref,frame,shift", [(0x10004, 0x20000, 0x30000), (0x10000, 0x20004, 0x30000),
                                             (0x10001, 0x20001, 0x30000), (0x10000, 0x20000, 0x30002)])
def test_misaligned_pointers(smip, ref, frame, shift):
    with pytest.raises(smip.InvalidArgument, match="aligned"):
        smip.xcorr_displacement_noalloc(ref, frame, 64, 64, shift)


def test_refusals_keep_their_order(smip):
    with pytest.raises(smip.InvalidArgument, match="null"):
        smip.xcorr_displacement_noalloc(0, 0x20001, 64, 64, 0x30000)
    with pytest.raises(smip.Unsupported):
        smip.xcorr_displacement_noalloc(0x10001, 0x20000, 512, 64, 0x30000)
