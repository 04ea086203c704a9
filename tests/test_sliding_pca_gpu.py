"""Sliding PCA windows of integer frames, whose views read a ring of 16-bit samples while later batches
are converted: outputs and ring storage equal those of the same frames sent as floats (whose windows run
one after another on the complex ring), bit for bit."""

import numpy as np
import pytest

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


def _run(raw, depth, big, T, B, K, batches, pull_each):
    H, W = raw.shape[1:]
    fd = hv.FrameDescriptor(W, H, depth, big)
    s = hv.Settings.defaults().update(space_transformation=0, time_transformation=2, time_transformation_size=T,
                                      time_stride=B, batch_size=B, image_type=1, p_start=T - K, p_width=K - 1, renorm=1,
                                      contrast_enabled=1, output_buffer_size=batches).validate(fd)
    with hv.Pipe(fd, s) as pipe:
        outs = []
        for b in range(batches):
            pipe.enqueue(raw[b * B:(b + 1) * B])
            while pull_each and pipe.output_count():
                outs.append(np.array(pipe.pull(), copy=True))
        outs += [np.array(o, copy=True) for o in pipe.pull_all()]
        return outs, pipe.float_frame().copy(), pipe.ring()


# T = 2 B (the smallest ratio), strides that are no multiple of 8 frames and wrap at other places in the
# window than in the sample ring, 8-bit batches off 16-byte alignment (B W H = 600), both byte orders
@pytest.mark.parametrize("T,B,W,H,depth,big,K", [(128, 64, 64, 64, 2, 0, 4), (66, 3, 20, 10, 1, 0, 1),
                                                 (70, 35, 24, 8, 2, 1, 2), (100, 7, 40, 24, 2, 0, 4),
                                                 (96, 32, 256, 192, 1, 0, 4)])
@pytest.mark.parametrize("cov_engine", [0, 1])
def test_sliding_windows_of_integers(cuda, T, B, W, H, depth, big, K, cov_engine):
    rng = np.random.default_rng(T + B)
    batches = -(-T // B) + 9
    top = 255 if depth == 1 else 65535
    n = batches * B
    # a few strong temporal modes, so that the kept components are well separated
    t = np.arange(n)[:, None, None]
    img = sum((0.2 / (k + 1)) * np.sin(0.37 * (k + 1) * t + 6.0 * rng.random((1, H, W))) for k in range(5))
    raw = np.clip((0.5 + img + 0.02 * rng.standard_normal((n, H, W))) * top, 0, top).astype(np.uint8 if depth == 1 else np.uint16)
    as_float = raw.astype(np.float32) * (257.0 if depth == 1 else 1.0)
    hv.lib().hv_pca_covariance_mode(cov_engine)
    try:
        ref = _run(as_float, 4, 0, T, B, K, batches, True)
        sent = raw.byteswap() if big else raw
        for pull_each in (True, False):  # False: windows in flight while their successors' batches are converted
            got = _run(sent, depth, big, T, B, K, batches, pull_each)
            assert len(got[0]) == len(ref[0]) >= 9
            for a, b in zip(got[0], ref[0]):
                assert np.array_equal(a, b)
            assert np.array_equal(got[1], ref[1])
            assert np.array_equal(got[2][0], ref[2][0]) and got[2][1:] == ref[2][1:]
    finally:
        hv.lib().hv_pca_covariance_mode(0)
