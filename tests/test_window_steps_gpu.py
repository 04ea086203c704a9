"""The window steps at the edges of their vector paths, batches of loads and reductions: sizes that are
not multiples of the 4 pixels of a 16-byte access, buffers off 16-byte alignment, frame counts around
the batches of the one-bin view, sums of values of very different size, infinities and NaN."""

import numpy as np
import pytest

from gpu_util import call, dev, host, ptr, zeros

import holovibes_gb300 as hv

pytestmark = pytest.mark.gpu


def _offset(a, pixels):
    """A device copy of `a` that starts `pixels` elements into its buffer."""
    pad = np.concatenate([np.zeros(pixels, a.dtype), a.ravel()])
    return ptr(dev(pad)) + pixels * a.itemsize


@pytest.mark.parametrize("T", [1, 2, 3, 7, 8, 9, 15, 16, 17, 25, 32, 41])
@pytest.mark.parametrize("W,H,shift", [(64, 4, 1), (66, 6, 1), (33, 3, 0)])
def test_one_bin_view_frame_batches(cuda, T, W, H, shift):
    rng = np.random.default_rng(T)
    ring = (rng.standard_normal((T, H, W)) + 1j * rng.standard_normal((T, H, W))).astype(np.complex64)
    w = np.exp(-2j * np.pi * np.arange(T) / max(T, 2)).astype(np.complex64)
    out = zeros(H * W * 4)
    np_ = hv.lib().hv_time_view_partials(W, H)
    part = zeros(np_ * 8)
    call("hv_time_view", ptr(dev(ring)), T, W, H, ptr(dev(w)), 1, hv.IMG_MODULUS, 1.0, shift, ptr(out), ptr(part), None)
    got = host(out, np.float32, (H, W)).astype(np.float64)
    r = ring.astype(np.complex128)
    ref = np.abs(np.tensordot(w.astype(np.complex128), r, axes=(0, 0)))
    # two fused multiply-adds per frame and component, then the modulus: 2 T + 4 roundings of 2^-24
    bound = (2 * T + 4) * 2.0 ** -24 * np.sqrt(2) * np.abs(r).sum(axis=0)
    if shift:
        ref, bound = (np.roll(a, (H // 2, W // 2), (0, 1)) for a in (ref, bound))
    assert np.all(np.abs(got - ref) <= bound)


@pytest.mark.parametrize("img", [hv.IMG_MODULUS, hv.IMG_ARGUMENT])
@pytest.mark.parametrize("kind", ["plain", "wide", "tiny", "zero", "huge", "inf", "nan"])
@pytest.mark.parametrize("W,H", [(128, 4), (130, 6), (65, 3)])
def test_view_partials(cuda, img, kind, W, H):
    """The partials are the sums of the view's 128-pixel runs (view order, no quadrant swap)."""
    rng = np.random.default_rng(3)
    x = rng.standard_normal((H, W)) + 1j * rng.standard_normal((H, W))
    scale = {"plain": 1.0, "tiny": 1e-42, "zero": 0.0, "huge": 1e37}.get(kind, 1.0)
    if kind == "wide":
        x = x * 10.0 ** rng.uniform(-30, 10, (H, W))
    x = (x * scale).astype(np.complex64)
    if kind == "inf":
        x[H // 2, 5] = np.inf
    if kind == "nan":
        x[1, 7] = np.nan
    out = zeros(H * W * 4)
    n = hv.lib().hv_time_view_partials(W, H)
    part = zeros(n * 8)
    call("hv_time_view", ptr(dev(x)), 1, W, H, ptr(dev(np.ones(1, np.complex64))), 1, img, 1.0, 0, ptr(out), ptr(part),
         None)
    view = host(out, np.float32, (H * W,)).astype(np.float64)
    got = host(part, np.float64, (n,))
    for i in range(n):
        run = view[i * 128:(i + 1) * 128]
        want = run.sum()
        if not np.isfinite(want):
            assert np.array_equal(got[i], want, equal_nan=True)
            continue
        # each value keeps at least 54 bits below the largest, and a run is rounded a few times
        assert abs(got[i] - want) <= 2.0 ** -45 * np.abs(run).max(), (i, got[i], want)


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 1024, 4096, 4099, 152 * 4096 + 4])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("npart", [0, 1, 31, 1024, 8192 + 5])
def test_renormalize_partials(cuda, n, off, npart):
    rng = np.random.default_rng(n + npart)
    x = rng.exponential(3.0, n).astype(np.float32)
    buf = dev(np.concatenate([np.zeros(off, np.float32), x]))
    px = ptr(buf) + 4 * off
    work = zeros(hv.lib().hv_reduce_workspace(n))
    part = np.zeros(0)
    if npart:
        part = rng.exponential(1.0, npart)
        part *= x.astype(np.float64).sum() / part.sum()
    call("hv_renormalize", px, n, 5, ptr(dev(part)) if npart else None, npart, ptr(work), None)
    total = np.float32(part.sum() if npart else x.astype(np.float64).sum())
    want = (x * np.float32(32.0)) * (np.float32(n) / total)
    got = host(buf, np.float32, (off + n,))[off:]
    # the FP64 total may round to the neighbouring float: 1 ulp of the factor, 1/2 of each product
    assert np.all(np.abs(got - want) <= 3 * np.spacing(np.abs(want)))


@pytest.mark.parametrize("A,slot,start,count", [(1, 0, 0, 1), (3, 2, 0, 3), (8, 0, 1, 8), (9, 4, 5, 9), (20, 3, 17, 11)])
@pytest.mark.parametrize("n", [5, 64, 1000])
def test_accumulate_frames(cuda, A, slot, start, count, n):
    """The mean is taken in queue order in FP32, whatever the grouping of the loads."""
    rng = np.random.default_rng(A * n)
    ring = rng.exponential(2.0, (A, n)).astype(np.float32)
    frame = rng.exponential(2.0, n).astype(np.float32)
    rd, out = dev(ring), zeros(n * 4)
    call("hv_accumulate", ptr(dev(frame)), ptr(rd), A, slot, start, count, ptr(out), n, None)
    ring[slot] = frame
    s = np.zeros(n, np.float32)
    for i in range(count):
        s = s + ring[(start + i) % A]
    assert np.array_equal(host(out, np.float32, (n,)), s / np.float32(count))
    assert np.array_equal(host(rd, np.float32, (A, n)), ring)


@pytest.mark.parametrize("W,H", [(1, 1), (2, 2), (5, 1), (64, 64), (127, 33), (256, 64), (1000, 331), (1252, 1000)])
@pytest.mark.parametrize("kind", ["speckle", "equal", "signed", "tail"])
@pytest.mark.parametrize("off", [0, 1])
def test_percentile_passes(cuda, W, H, kind, off):
    rng = np.random.default_rng(W)
    n = W * H
    x = rng.exponential(500.0, n)
    if kind == "equal":
        x = np.full(n, 77.25)
    elif kind == "signed":
        x = rng.standard_normal(n) * 1e4
    elif kind == "tail":
        x = np.where(rng.random(n) < 0.02, 1e30, x)
    x = x.astype(np.float32)
    rng_out = zeros(8)
    work = zeros(hv.lib().hv_percentile_workspace(n))
    for lower, upper in ((0.5, 99.5), (0.0, 100.0), (50.0, 50.0)):
        call("hv_percentile", _offset(x, off), W, H, lower, upper, 0.0, ptr(rng_out), ptr(work), None)
        got = host(rng_out, np.float32, (2,))
        s = np.sort(x)
        for g, p in zip(got, (lower, upper)):
            k = min(int(np.float32(np.float32(p) / np.float32(100.0)) * np.float32(n)), n - 1)
            assert g == max(s[k], np.float32(1.0)), (p, k)


@pytest.mark.parametrize("n,off", [(1, 0), (7, 0), (8, 0), (8, 1), (1029, 0), (4096, 3)])
def test_contrast_and_log_maps(cuda, n, off):
    rng = np.random.default_rng(n)
    x = rng.uniform(-10.0, 300.0, n).astype(np.float32)
    r = np.array([20.0, 200.0], np.float32)
    out = zeros(n * 2)
    call("hv_contrast_to_ushort", _offset(x, off), ptr(dev(r)), 0, 1, ptr(out), n, None)
    f = np.float32(65535.0) / ((r[1] - r[0]) + np.float32(np.finfo(np.float32).eps))
    v = f * (x - r[0])
    assert np.array_equal(host(out, np.uint16, (n,)), np.clip(np.trunc(v.astype(np.float64)), 0, 65535).astype(np.uint16))
    y = np.abs(x) + np.float32(1e-3)
    yd = dev(y)
    call("hv_log10", ptr(yd), n, None)
    ref = np.log10(y.astype(np.float64))
    # log10f: 2 ulp of the result, or of 1 near log10(1) = 0
    assert np.all(np.abs(host(yd, np.float32, (n,)) - ref) <= 2.0 ** -22 * np.maximum(np.abs(ref), 0.1))


@pytest.mark.parametrize("W,H", [(16, 16), (48, 64), (512, 16), (768, 64)])
def test_unwrap_alignment(cuda, W, H):
    """Buffers off 16-byte alignment take the element-wise steps one value at a time: the same bits."""
    rng = np.random.default_rng(W)
    phase = rng.uniform(-np.pi, np.pi, (H, W)).astype(np.float32)
    n = W * H
    nw = hv.lib().hv_unwrap_workspace(W, H)
    got = []
    for off in (0, 1):
        out, work = zeros(n * 4 + 4), zeros(nw + 8)
        call("hv_unwrap_2d", _offset(phase, off), ptr(out) + 4 * off, W, H, ptr(work) + 8 * off, None)
        got.append(host(out, np.float32, (n + off,))[off:])
    assert np.all(np.isfinite(got[0]))
    assert np.array_equal(got[0], got[1])
