"""A sliding PCA pipe on a device whose free memory holds the pipe, but not the buffers that let its windows overlap: it is
created and gives the same holograms."""

import numpy as np
import pytest
import torch

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


def test_pipe_without_room_for_overlap(cuda):
    W = H = 512
    T, B, K, batches = 512, 256, 2, 4
    fd = hv.FrameDescriptor(W, H, 2, 0)
    s = hv.Settings.defaults().update(space_transformation=0, time_transformation=2, time_transformation_size=T,
                                      time_stride=B, batch_size=B, image_type=1, p_start=T - K, p_width=K - 1, renorm=1,
                                      contrast_enabled=1, output_buffer_size=batches, input_buffer_size=2 * B).validate(fd)
    rng = np.random.default_rng(5)
    t = np.arange(batches * B)[:, None, None]
    modes = sum((0.2 / (k + 1)) * np.sin(0.37 * (k + 1) * t + 6.0 * rng.random((1, H, W), np.float32)) for k in range(3))
    raw = np.clip((0.5 + modes + 0.02 * rng.standard_normal((batches * B, H, W), np.float32)) * 4095, 0, 4095)
    frames = torch.from_numpy(raw.astype(np.int16)).cuda()

    def run():
        with hv.Pipe(fd, s) as pipe:
            for b in range(batches):
                pipe.enqueue(frames[b * B:(b + 1) * B])
            return [o.copy() for o in pipe.pull_all()], pipe.ring()[0]

    want, want_ring = run()
    assert len(want) >= 2
    overlap = 2 * (T + 2 * B) * W * H + 4 * 16 * T * T
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    # half of the overlap's buffers are missing (cudaMalloc rounds a pipe's allocations up by a few MB in all)
    ballast = torch.empty(torch.cuda.mem_get_info()[0] - hv.Pipe.footprint(fd, s) + overlap // 2, dtype=torch.uint8,
                          device="cuda")
    try:
        got, got_ring = run()
    finally:
        del ballast
        torch.cuda.empty_cache()
    assert len(got) == len(want) and all(np.array_equal(a, b) for a, b in zip(got, want))
    assert np.array_equal(got_ring, want_ring)
