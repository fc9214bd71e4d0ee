"""Which paths of a wave train the guiding network: as many as there are record slots, pass by pass and pixel by pixel,
each in a slot of its own."""
import numpy as np
import pytest

import mypbr_gb300 as mp


# slots for whole passes, for none, for part of one, for more than the wave has (those of an earlier, larger render)
@pytest.mark.parametrize("pixels,passes,slots", [(1, 1, 1), (7, 5, 35), (7, 5, 21), (7, 5, 24), (7, 5, 3), (7, 5, 0),
                                                 (7, 5, 100), (640, 9, 5000), (999, 3, 2073)])
def test_record_slots(pixels, passes, slots):
    out = np.zeros((pixels, passes), dtype=np.uint32)
    mp.check(mp.lib().mypbr_guide_test_record_slots(pixels, passes, slots, out.ctypes.data))
    has = out != 0xffffffff
    order = np.arange(passes)[None, :] * pixels + np.arange(pixels)[:, None]  # passes in turn
    assert np.array_equal(has, order < slots)
    assert len(np.unique(out[has])) == has.sum()
    assert not has.any() or out[has].max() < slots
