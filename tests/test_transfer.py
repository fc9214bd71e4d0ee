"""Frames between host memory and the GPU: the copies split over threads (from 2 MiB, in parts of whole pages and
chunks of 1 MiB) and the workspace that calls without a scene handle share."""
import threading

import numpy as np
import pytest

import mypbr_gb300 as mp


def _frame(pixels, seed=0):
    return np.random.default_rng(seed).lognormal(0.0, 1.0, (1, pixels, 3))


# with neither bloom nor vignette the linear output is the input: 24 bytes a pixel, around one chunk, the
# smallest split copy (2 MiB = 87,381.3 pixels), whole parts and ragged last parts
@pytest.mark.gpu
@pytest.mark.parametrize("pixels", [1, 43690, 43691, 87381, 87382, 349525, 349526, 700001, 2073600])
def test_a_frame_comes_back_as_it_went(pixels):
    frame = _frame(pixels)
    lin, rgb = mp.display(frame, mp.display_opts())
    assert np.array_equal(lin, frame)
    assert rgb.shape == frame.shape


@pytest.mark.gpu
def test_both_outputs_are_those_of_separate_calls():
    import ctypes
    frame = _frame(64 * 48).reshape(48, 64, 3)
    opts = mp.display_opts(exposure=0.3, tonemap="aces", bloom=0.2, vignette=0.4)
    lin, rgb = mp.display(frame, opts)
    dp, bp = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_uint8)
    only_lin, only_rgb = np.zeros_like(frame), np.zeros(frame.shape, np.uint8)
    ptr = frame.ctypes.data_as(dp)
    mp.check(mp.lib().mypbr_gpu_display(ptr, 64, 48, ctypes.byref(opts), only_lin.ctypes.data_as(dp), None, 0))
    mp.check(mp.lib().mypbr_gpu_display(ptr, 64, 48, ctypes.byref(opts), None, only_rgb.ctypes.data_as(bp), 0))
    assert np.array_equal(lin, only_lin) and np.array_equal(rgb, only_rgb)


@pytest.mark.gpu
def test_threads_share_the_workspace():
    """Two threads at once: one of them has the kept workspace, the other its own memory."""
    frames = [_frame(120000 + 4321 * k, k) for k in range(6)]
    bad = []

    def work(mine):
        for f in mine:
            lin, _ = mp.display(f, mp.display_opts())
            n = f.shape[1]
            ones = np.ones((1, n, 3))
            out = np.empty_like(f)
            mp.denoise(f, ones, ones, np.full((1, n), 1e-6), n, 1, out)
            if not np.array_equal(lin, f) or not np.isfinite(out).all():
                bad.append(n)

    threads = [threading.Thread(target=work, args=(frames[k::2],)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
