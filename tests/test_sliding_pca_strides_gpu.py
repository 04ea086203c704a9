"""Pipelined PCA windows of integer frames whose stride is larger than the batch (one batch per stride enters the ring, those
between are skipped): outputs equal those of the same frames sent as floats, whose windows run one after another."""

import numpy as np
import pytest

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,S", [(66, 3, 9), (72, 8, 16), (72, 8, 72), (100, 10, 200)])
@pytest.mark.parametrize("depth", [1, 2])
def test_strides_above_the_batch(cuda, T, B, S, depth):
    W, H, K = 40, 24, 3
    windows = 9
    n = -(-S * (T // B + windows) // B) * B
    top = 255 if depth == 1 else 65535
    rng = np.random.default_rng(T + S)
    t = np.arange(n)[:, None, None]
    img = sum((0.2 / (k + 1)) * np.sin(0.37 * (k + 1) * t + 6.0 * rng.random((1, H, W))) for k in range(5))
    raw = np.clip((0.5 + img + 0.02 * rng.standard_normal((n, H, W))) * top, 0, top).astype(np.uint8 if depth == 1 else np.uint16)

    def run(frames, depth):
        fd = hv.FrameDescriptor(W, H, depth, 0)
        s = hv.Settings.defaults().update(space_transformation=0, time_transformation=2, time_transformation_size=T,
                                          time_stride=S, batch_size=B, image_type=1, p_start=T - K, p_width=K - 1, renorm=1,
                                          contrast_enabled=1, output_buffer_size=n // B).validate(fd)
        with hv.Pipe(fd, s) as pipe:
            for i in range(0, n, B):
                pipe.enqueue(frames[i:i + B])
            return [o.copy() for o in pipe.pull_all()], pipe.float_frame().copy(), pipe.ring()

    want = run(raw.astype(np.float32) * (257.0 if depth == 1 else 1.0), 4)
    got = run(raw, depth)
    assert len(got[0]) == len(want[0]) >= 5
    assert all(np.array_equal(a, b) for a, b in zip(got[0], want[0]))
    assert np.array_equal(got[1], want[1])
    assert np.array_equal(got[2][0], want[2][0]) and got[2][1:] == want[2][1:]
