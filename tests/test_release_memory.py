"""Device memory that calls without a scene handle keep, given back on request."""
import numpy as np
import pytest
import torch

import mypbr_gb300 as mp


def test_release_without_a_gpu():
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    mp.release_memory()


@pytest.mark.gpu
def test_denoise_memory_is_given_back():
    h, w = 1000, 1000
    plane = np.ones((h, w, 3))

    def denoise():
        out = np.empty_like(plane)
        mp.denoise(plane, plane, plane, np.ones((h, w)), w, h, out)
        return out

    want = denoise()
    mp.release_memory()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert np.array_equal(denoise(), want)
    # 148 bytes a pixel are kept
    assert torch.cuda.mem_get_info()[0] <= free - 140 * h * w
    mp.release_memory()
    assert torch.cuda.mem_get_info()[0] >= free - (2 << 20)
    assert np.array_equal(denoise(), want)
