"""The view's renormalisation partials are FP64 sums: of values that differ by more than the 24 bits of a float they
keep what an FP64 addition tree keeps."""

import math

import numpy as np
import pytest

from gpu_util import call, dev, host, ptr, zeros

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


# one bright pixel per warp (32 or 64 pixels) among pixels 2^-small of it, with all bits of the mantissa in use
@pytest.mark.parametrize("small", [8, 30, 32, 33, 34, 40, 54, 60, 120])
@pytest.mark.parametrize("W,H", [(128, 4), (130, 6), (65, 3)])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -30, 2.0 ** 60])
def test_partials_of_uneven_values(cuda, small, W, H, scale):
    n = W * H
    x = np.full(n, (2.0 - 2.0 ** -23) * 2.0 ** -small)
    x[::32 if n % 2 else 64] = 1.0
    x = (x * scale).astype(np.float32).reshape(H, W)
    out = zeros(n * 4)
    parts = hv.lib().hv_time_view_partials(W, H)
    part = zeros(parts * 8)
    call("hv_time_view", ptr(dev(x.astype(np.complex64))), 1, W, H, ptr(dev(np.ones(1, np.complex64))), 1, hv.IMG_MODULUS,
         1.0, 0, ptr(out), ptr(part), None)
    view = host(out, np.float32, (n,)).astype(np.float64)
    got = host(part, np.float64, (parts,))
    for i in range(parts):
        run = view[i * 128:(i + 1) * 128]
        # five additions across a warp's lanes and one of a lane's two pixels, then one of two warps' sums, or five
        # and three of four: eight roundings at most
        assert abs(got[i] - math.fsum(run)) <= 8 * 2.0 ** -53 * np.abs(run).sum(), i
