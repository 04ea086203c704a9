"""The two-bin time view around its batches of frames, and the time it takes beside the views of one and three bins (its loads
are the same)."""

import numpy as np
import pytest
import torch

from gpu_util import call, dev, host, ptr, zeros

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [2, 3, 7, 8, 9, 10, 15, 16, 17, 25, 41])
@pytest.mark.parametrize("W,H,shift", [(64, 4, 1), (66, 6, 1), (34, 3, 0)])
def test_frame_batches(cuda, T, W, H, shift):
    rng = np.random.default_rng(T)
    ring = (rng.standard_normal((T, H, W)) + 1j * rng.standard_normal((T, H, W))).astype(np.complex64)
    w = np.exp(-2j * np.pi * np.outer([1, 2], np.arange(T)) / T).astype(np.complex64)
    out = zeros(H * W * 4)
    call("hv_time_view", ptr(dev(ring)), T, W, H, ptr(dev(w)), 2, hv.IMG_MODULUS, 1.0, shift, ptr(out), None, None)
    got = host(out, np.float32, (H, W)).astype(np.float64)
    r = ring.astype(np.complex128)
    ref = np.abs(np.tensordot(w.astype(np.complex128), r, axes=(1, 0))).mean(axis=0)
    # two fused multiply-adds per frame and component, then the modulus, the sum and the mean: 2 T + 6 roundings
    bound = (2 * T + 6) * 2.0 ** -24 * np.sqrt(2) * np.abs(r).sum(axis=0)
    if shift:
        ref, bound = (np.roll(a, (H // 2, W // 2), (0, 1)) for a in (ref, bound))
    assert np.all(np.abs(got - ref) <= bound)


def test_time_beside_other_bin_counts(cuda):
    """Best of several times: no more than 1.08 of the longer of the one- and the three-bin view (1.0 in batches of loads,
    1.12 one after another)."""
    W = H = 1024
    T = 128
    ring, out = zeros(T * W * H * 8), zeros(W * H * 4)
    part, w = zeros(hv.lib().hv_time_view_partials(W, H) * 8), zeros(4 * T * 8)

    def best(K):
        times = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(10):
                call("hv_time_view", ptr(ring), T, W, H, ptr(w), K, hv.IMG_MODULUS, 1.0, 0, ptr(out), ptr(part),
                     torch.cuda.current_stream().cuda_stream)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[2:])

    assert best(2) <= 1.08 * max(best(1), best(3))
