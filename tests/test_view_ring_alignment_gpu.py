"""The time view of a complex64 ring that starts 8 bytes past a 16-byte boundary (a slice of a larger buffer):
the views and moments of up to 4 bins, whose kernel for aligned rings reads 16 bytes at a time."""

import numpy as np
import pytest
import torch

from gpu_util import call, dev, host, ptr, zeros

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 2, 3, 4])
@pytest.mark.parametrize("T", [5, 16, 33])
@pytest.mark.parametrize("W,H,shift", [(64, 4, 1), (34, 10, 1), (2, 1, 0)])
@pytest.mark.parametrize("moments", [False, True])
def test_ring_off_16_bytes(cuda, K, T, W, H, shift, moments):
    rng = np.random.default_rng(100 * K + T)
    ring = (rng.standard_normal((T, H, W)) + 1j * rng.standard_normal((T, H, W))).astype(np.complex64)
    w = np.exp(-2j * np.pi * np.outer(np.arange(K), np.arange(T)) / T).astype(np.complex64)
    bins = np.linspace(0.5, 1.5, K).astype(np.float32)
    shift = shift if W % 2 == 0 and H % 2 == 0 else 0
    flat = torch.zeros(2 * ring.size + 2, device="cuda")
    flat[2:] = dev(ring).flatten()
    base = ptr(flat) + 8
    assert base % 16 == 8
    wd, bd = dev(w), dev(bins)
    out, part = zeros(W * H * 4), zeros(hv.lib().hv_time_view_partials(W, H) * 8)
    if moments:
        call("hv_time_moments", base, T, W, H, ptr(wd), K, ptr(bd), shift, ptr(out), ptr(part), None)
    else:
        call("hv_time_view", base, T, W, H, ptr(wd), K, hv.IMG_MODULUS, 1.0, shift, ptr(out), ptr(part), None)
    got = host(out, np.float32, (H, W)).astype(np.float64)
    r = ring.astype(np.complex128)
    X = np.tensordot(w.astype(np.complex128), r, axes=(1, 0))
    # each component: two fused multiply-adds per frame, 2 T roundings of 2^-24 of sum |x|, so |X_k| is off by
    # e = 2 T 2^-24 sqrt(2) sum |x| (|w| = 1 to a rounding, in the 4 below); the modulus, the K additions and
    # the division round 4 + K times more
    s = np.sqrt(2) * np.abs(r).sum(axis=0)
    e = (2 * T + 4 + K) * 2.0 ** -24 * s
    if moments:
        ref = (np.abs(X) ** 2 * bins.astype(np.float64)[:, None, None]).sum(axis=0)
        bound = bins.astype(np.float64).sum() * ((2 * s + e) * e + (4 + K) * 2.0 ** -24 * s * s)
    else:
        ref, bound = np.abs(X).mean(axis=0), e
    if shift:
        ref, bound = (np.roll(a, (H // 2, W // 2), (0, 1)) for a in (ref, bound))
    assert np.all(np.abs(got - ref) <= bound)
    if not shift:
        view = host(out, np.float32, (W * H,)).astype(np.float64)
        for i, p in enumerate(host(part, np.float64, (-(-W * H // 128),))):
            assert abs(p - view[i * 128:(i + 1) * 128].sum()) <= 2.0 ** -45 * 128 * np.abs(view).max()
