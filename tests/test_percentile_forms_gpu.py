"""The percentile's passes without 16-byte loads (a reticle) and with loads that start between the frame's pixels (off 16-byte
alignment): every count of pixels before and behind the aligned ones, more pixels than one step of the grid, and
the time that these forms take beside the plain one."""

import numpy as np
import pytest
import torch

from gpu_util import call, dev, empty, host, ptr, zeros

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu

LIMITS = ((0.5, 99.5), (0.0, 100.0), (37.0, 61.0))


def _percentiles(x, W, H, off, reticle):
    pad = np.concatenate([np.full(off, 1e30, np.float32), x.ravel(), np.full(5, -1e30, np.float32)])
    frame = dev(pad)
    out, work = zeros(8), empty(hv.lib().hv_percentile_workspace(W * H))
    got = []
    for lower, upper in LIMITS:
        call("hv_percentile", ptr(frame) + 4 * off, W, H, lower, upper, reticle, ptr(out), ptr(work), None)
        got.append(host(out, np.float32, (2,)).copy())
    return got


def _expected(v):
    s = np.sort(v.ravel())
    k = lambda p: min(int(np.float32(np.float32(p) / np.float32(100.0)) * np.float32(s.size)), s.size - 1)
    return [[max(s[k(p)], np.float32(1.0)) if s.size else np.float32(1.0) for p in pair] for pair in LIMITS]


@pytest.mark.parametrize("W,H", [(1, 1), (2, 1), (3, 1), (5, 1), (7, 3), (64, 64), (333, 101), (2049, 1301)])
@pytest.mark.parametrize("off", [0, 1, 2, 3])
def test_frames_off_alignment(cuda, W, H, off):
    x = np.random.default_rng(W + off).exponential(500.0, (H, W)).astype(np.float32)
    assert np.array_equal(_percentiles(x, W, H, off, 0.0), _expected(x))


@pytest.mark.parametrize("W,H", [(3, 3), (16, 17), (64, 64), (101, 333), (1000, 701), (1400, 1400)])
@pytest.mark.parametrize("reticle", [0.3, 0.8, 1.0, 2.0])
@pytest.mark.parametrize("off", [0, 1])
def test_reticle(cuda, W, H, reticle, off):
    x = np.random.default_rng(W).exponential(500.0, (H, W)).astype(np.float32)
    radius = int(np.float32(reticle) * np.float32(min(W, H)) / np.float32(2.0))
    y, c = np.mgrid[0:H, 0:W]
    inside = (c - W // 2) ** 2 + (y - H // 2) ** 2 <= radius * radius
    assert np.array_equal(_percentiles(x, W, H, off, reticle), _expected(x[inside] if radius else x))


def test_forms_take_no_longer_than_their_pixels(cuda):
    """Best of several times: off alignment as long as aligned, with a reticle at most 1.7 times as long (1.3 where a
    thread's loads go out together, 2.1 where each is waited for)."""
    W = H = 2048
    frame = torch.empty(W * H + 1, device="cuda").exponential_(1 / 500.0)
    out, work = zeros(8), empty(hv.lib().hv_percentile_workspace(W * H))

    def best(off, reticle):
        times = []
        for _ in range(12):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                call("hv_percentile", frame.data_ptr() + 4 * off, W, H, 0.5, 99.5, reticle, ptr(out), ptr(work),
                     torch.cuda.current_stream().cuda_stream)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[2:])

    plain = best(0, 0.0)
    assert best(1, 0.0) <= 1.3 * plain
    assert best(0, 1.0) <= 1.7 * plain
