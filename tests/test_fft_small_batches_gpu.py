"""Column passes of few tiles (half as wide as the others): the same bits as the wide tiles, which the same
frames take in a larger batch; widths that leave a part of a tile, both sides of the rule's line."""

import numpy as np
import pytest

from gpu_util import call, dev, host, ptr, zeros

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [128, 192, 256, 384])
@pytest.mark.parametrize("W,frames", [(8, 1), (20, 3), (256, 4), (256, 5)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_few_column_tiles(cuda, N, W, frames, mode):
    rng = np.random.default_rng(N + W)
    many = -(-400 * 16 // W)  # at least 400 tiles
    x = (rng.standard_normal((frames, N, W)) + 1j * rng.standard_normal((frames, N, W))).astype(np.complex64)
    g = (rng.standard_normal((N, W)) + 1j * rng.standard_normal((N, W))).astype(np.complex64)
    gd = dev(g)
    outs = []
    for batch in (frames, many):
        xs = dev(np.resize(x, (batch, N, W)))
        out = zeros(batch * N * W * 8)
        call("hv_fft_cols", ptr(xs), ptr(out), W, N, batch, ptr(gd) if mode == 2 else None, mode, 0.5, 0, batch, None)
        outs.append(host(out, np.complex64, (batch, N, W))[:frames])
    assert np.array_equal(outs[0], outs[1])
    # against FP64: 2 log2(N) roundings of 2^-24 per transform on the norm (a butterfly and a twiddle per level)
    ref = np.fft.fft(x.astype(np.complex128), axis=1) if mode != 1 else np.fft.ifft(x.astype(np.complex128), axis=1) * N
    if mode == 2:
        ref = np.fft.ifft(ref * g, axis=1) * N
    err = np.linalg.norm(outs[0] - 0.5 * ref) / np.linalg.norm(0.5 * ref)
    assert err <= (2 if mode == 2 else 1) * 2 * np.ceil(np.log2(N)) * 2.0 ** -24 + 2.0 ** -22
