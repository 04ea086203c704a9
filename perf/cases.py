"""What a user of this framework has it do, as cases that can be timed and checked.

Two kinds of use, both through the public entry points of `holovibes_gb300`:

* a Pipe, the drop-in engine: raw camera frames in, uint16 holograms out ("pipe");
* the compute steps on caller-owned device buffers, for programs with a pipeline of their own: the
  spatial transform of a batch into the time ring ("spatial"), the time transform and view of a full
  ring ("view"), the PCA of a full ring ("pca"), the 2-D phase unwrap ("unwrap") and the window to
  hologram chain from a ring to uint16 ("hologram").

Sizes and settings are those of the benchmark's workloads, the serving mix and the tests: frames of
64 to 1024 pixels a side (and larger ones, not square ones), 8- and 16-bit and float pixels, time
windows of 4 to 512 frames, one bin to tens of bins.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import holovibes_gb300 as hv

PITCH_UM = 12.0  # camera pixel pitch of every case


# ------------------------------------------------------------------------------------ cases
def listed():
    return [
        # The drop-in engine on the plain angular-spectrum + STFT workload: a 12-bit camera, one bin, every batch a
        # whole window. Sixteen windows arrive on the device, sixteen holograms are read.
        dict(name="pipe_as_stft_512", kind="pipe", W=512, H=512, depth=2, space=2, time=1, T=16, S=16, B=16, p=1, pw=0,
             img=0, shift=1, renorm=0, acc=0, windows=16, host=False),
        # The benchmark's default workload: an 8-bit megapixel camera, Fresnel + PCA, 4 dominant components.
        dict(name="pipe_fresnel_pca_1024", kind="pipe", W=1024, H=1024, depth=1, space=1, time=2, T=32, S=32, B=32,
             p=28, pw=3, img=1, shift=0, renorm=1, acc=0, windows=8, host=False),
        # The large sliding window: PCA over the last 512 frames, a hologram every 64 frames.
        dict(name="pipe_pca_sliding_512", kind="pipe", W=512, H=512, depth=2, space=0, time=2, T=512, S=64, B=64,
             p=508, pw=3, img=0, shift=0, renorm=1, acc=0, windows=8, host=False),
        # The smallest stream of the serving mix, live: host frames in, host holograms out, a small sliding window.
        dict(name="pipe_live_256", kind="pipe", W=256, H=256, depth=1, space=2, time=1, T=16, S=4, B=4, p=1, pw=0,
             img=0, shift=1, renorm=1, acc=0, windows=4, host=True),
        # The spatial stage of the high-rate Doppler workload: a large batch of 768 x 768 angular spectra.
        dict(name="spatial_as_768", kind="spatial", W=768, H=768, depth=2, be=0, B=64, space=2, f2d=False),
        # A batch of the serving mix's frames that are not square, Fresnel.
        dict(name="spatial_fresnel_1024x768", kind="spatial", W=1024, H=768, depth=1, be=0, B=16, space=1, f2d=False),
        # The smallest call of the spatial stage: a few small frames, where launches and latency count.
        dict(name="spatial_as_256", kind="spatial", W=256, H=256, depth=2, be=0, B=4, space=2, f2d=False),
        # One STFT bin over the window of the 512 x 512 serving streams.
        dict(name="view_stft_512", kind="view", W=512, H=512, T=32, p=1, K=1, img=0, shift=1, tc=False),
        # The many-bin view of the high-rate Doppler workload: 33 bins of 256 frames, argument.
        dict(name="view_stft_768_33bins", kind="view", W=768, H=768, T=256, p=48, K=33, img=2, shift=1, tc=True),
        # One PCA window of the serving mix: covariance, eigensolve and the projected view.
        dict(name="pca_512_64", kind="pca", W=512, H=512, T=64, K=4, img=1),
        # The unwrapped-phase view of the high-rate Doppler workload.
        dict(name="unwrap_768", kind="unwrap", W=768, H=768),
        # From a short window to the hologram: view, renormalisation, image accumulation, log, autocontrast, uint16.
        dict(name="hologram_1024", kind="hologram", W=1024, H=1024, T=8, p=1, K=1, img=0, acc=8, log=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pipe", "pipe", "spatial", "spatial", "view", "view", "pca", "unwrap", "hologram"])
    sides = [64, 128, 192, 256, 384, 512, 768, 1024]  # transform lengths
    if kind == "pipe":
        W, H = rng.choice(sides[2:]), rng.choice(sides[2:])
        time = rng.choice([1, 1, 2])
        T = rng.choice([8, 16, 20, 32, 48, 64] if time == 1 else [16, 32, 64, 96, 128])
        B = rng.choice([d for d in range(4, T + 1) if T % d == 0])
        K = min(rng.randint(1, 5 if time == 2 else 12), T // 2)
        windows = max(1, min(12, (1 << 25) // (W * H * B)))
        return dict(kind="pipe", W=W, H=H, depth=rng.choice([1, 2]), space=rng.choice([1, 2, 2]), time=time, T=T, S=B,
                    B=B, p=T - K if time == 2 else 1, pw=K - 1, img=rng.choice([0, 1]), shift=rng.randint(0, 1),
                    renorm=rng.randint(0, 1), acc=rng.choice([0, 0, 3]), windows=windows, host=rng.random() < 0.2)
    if kind == "spatial":
        W, H = rng.choice(sides + [1536, 2048]), rng.choice(sides + [1536, 2048])
        top = max(1, min(64, (1 << 25) // (W * H)))
        depth = rng.choice([1, 2, 2, 4])
        return dict(kind="spatial", W=W, H=H, depth=depth, be=rng.randint(0, 1) if depth == 2 else 0,
                    B=_log_int(rng, 1, top), space=rng.choice([1, 2, 2]), f2d=rng.random() < 0.2)
    # the steps behind the ring take any frame size (the quadrant swap an even one)
    W, H = 2 * _log_int(rng, 32, 512), 2 * _log_int(rng, 32, 512)
    if kind == "view":
        T = _log_int(rng, 4, min(256, max(4, (1 << 26) // (W * H))))
        K = min(T - 1, _log_int(rng, 1, 40))
        return dict(kind="view", W=W, H=H, T=T, p=rng.randint(0, T - K), K=K, img=rng.choice([0, 1, 5, 6]),
                    shift=rng.randint(0, 1), tc=K >= 8)
    if kind == "pca":
        T = rng.choice([12, 16, 24, 32, 48, 64, 100, 128])
        return dict(kind="pca", W=W, H=H, T=T, K=rng.randint(1, 5), img=rng.choice([0, 1]))
    if kind == "unwrap":
        return dict(kind="unwrap", W=rng.choice(sides), H=rng.choice(sides))
    T = _log_int(rng, 4, 32)
    K = rng.randint(1, 4)
    return dict(kind="hologram", W=W, H=H, T=T, p=rng.randint(0, T - K), K=K, img=rng.choice([0, 1]),
                acc=rng.choice([1, 3, 8]), log=rng.random() < 0.5)


# ------------------------------------------------------------------------------------ inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn_c(g, *shape):
    return torch.complex(torch.randn(shape, generator=g, device="cuda"), torch.randn(shape, generator=g, device="cuda"))


def _speckle(g, W, H):
    """A random-phase object with smooth speckle amplitude of mean 1."""
    fy = torch.fft.fftfreq(H, device="cuda")[:, None]
    fx = torch.fft.fftfreq(W, device="cuda")[None, :]
    blur = torch.exp(-2.0 * (math.pi * 3.0) ** 2 * (fx * fx + fy * fy))
    a = torch.fft.ifft2(torch.fft.fft2(_randn_c(g, H, W)) * blur).abs()
    phase = 2.0 * math.pi * torch.rand((H, W), generator=g, device="cuda")
    return torch.polar(a / a.mean(), phase)


def _modes(g, n):
    """Frequencies (cycles per frame) and amplitudes of n temporal modes, eigenvalues decaying as 1 / m^2."""
    f = 0.03 + 0.44 * torch.rand((n,), generator=g, device="cuda")
    return f.tolist(), [1.0 / (m + 1) for m in range(n)]


def _frames(g, n, W, H, depth, modes=4):
    """n raw off-axis interferograms |R + O(t)|^2 with shot noise, as a camera of `depth` bytes per pixel gives them."""
    full = {1: 255, 2: 4095, 4: 4095}[depth]
    x = torch.arange(W, device="cuda", dtype=torch.float64)[None, :]
    ref = torch.polar(torch.ones((1, W), device="cuda", dtype=torch.float64), torch.remainder(2.3 * x, 2 * math.pi))
    ref = ref.to(torch.complex64).expand(H, W)
    freqs, amps = _modes(g, modes)
    fields = [0.3 * a * _speckle(g, W, H) for a in amps]
    out = torch.empty((n, H, W), device="cuda", dtype={1: torch.uint8, 2: torch.int16, 4: torch.float32}[depth])
    for t in range(n):
        u = ref + sum(o * complex(math.cos(2 * math.pi * f * t), math.sin(2 * math.pi * f * t))
                      for o, f in zip(fields, freqs))
        i = u.real.square() + u.imag.square()
        i = i * (0.4 * full / 1.13)
        i = (i + i.sqrt() * torch.randn((H, W), generator=g, device="cuda")).round().clamp(0, full)
        out[t] = i.to(out.dtype)
    return out


def _ring(g, T, W, H):
    """A full time ring: T propagated complex frames, a few temporal modes over noise (16-bit pixel scale)."""
    freqs, amps = _modes(g, 6)
    fields = [500.0 * a * _speckle(g, W, H) for a in amps]
    out = torch.empty((T, H, W), device="cuda", dtype=torch.complex64)
    for t in range(T):
        u = 20.0 * _randn_c(g, H, W)
        for o, f in zip(fields, freqs):
            u = u + o * complex(math.cos(2 * math.pi * f * t), math.sin(2 * math.pi * f * t))
        out[t] = u
    return out


def _bytes(n):
    return torch.zeros(max(int(n), 16), dtype=torch.uint8, device="cuda")


def _call(name, *args):
    hv.check(getattr(hv.lib(), name)(*args), name)


def _optics(space):
    return (785e-9, 0.45) if space == hv.SPACE_FRESNELTR else (852e-9, 0.30)


def _f2d_radii(W, H):
    m = min(W, H)
    return m // 16, m // 3, max(1, m // 32), max(1, m // 16)


# ------------------------------------------------------------------------------------ prepare
def prepare(case, seed):
    g = _generator(seed)
    s = dict(case)
    W, H = case["W"], case["H"]
    kind = case["kind"]
    if kind == "pipe":
        lam, z = _optics(case["space"])
        T, B, n = case["T"], case["B"], case["windows"]
        fd = hv.FrameDescriptor(W, H, case["depth"])
        st = hv.Settings.defaults().update(
            space_transformation=case["space"], time_transformation=case["time"], time_transformation_size=T,
            time_stride=case["S"], batch_size=B, lambda_=lam, z_distance=z, pixel_size=PITCH_UM,
            image_type=case["img"], p_start=case["p"], p_width=case["pw"], fft_shift=case["shift"],
            renorm=case["renorm"], accumulation=case["acc"], contrast_enabled=1, contrast_auto_refresh=1,
            contrast_lower=0.5, contrast_upper=99.5, output_buffer_size=32, input_buffer_size=4 * B).validate(fd)
        first = T - B  # frames that fill the ring up to the first hologram
        frames = _frames(g, first + n * B, W, H, case["depth"], modes=16 if T > 128 else 4)
        pipe = hv.Pipe(fd, st)
        if first:
            torch.cuda.synchronize()
            pipe.enqueue(frames[:first])
            pipe.sync()
        batches = [frames[first + i * B:first + (i + 1) * B].contiguous() for i in range(n)]
        if case["host"]:
            batches = [b.cpu().numpy() for b in batches]
            s["out"] = np.empty((n, H, W), dtype=np.uint16)
        else:
            s["out"] = torch.zeros((n, H, W), dtype=torch.int16, device="cuda")  # the bytes of uint16 pixels
        s.update(pipe=pipe, batches=batches)
    elif kind == "spatial":
        B, space = case["B"], case["space"]
        raw = _frames(g, B, W, H, case["depth"])
        if case["be"]:
            raw = raw.view(torch.uint8).reshape(B, H, W, 2).flip(-1).contiguous().view(torch.int16).reshape(B, H, W)
        lens = torch.zeros((H, W), dtype=torch.complex64, device="cuda")
        lam, z = _optics(space)
        _call("hv_fresnel_lens" if space == hv.SPACE_FRESNELTR else "hv_angular_spectrum_lens", lens.data_ptr(), W, H,
              lam, z, PITCH_UM, hv.LENS_FP64, None)
        s["mask"] = s["work2"] = None
        if case["f2d"]:
            if space == hv.SPACE_ANGULARSP:  # part of the transfer function
                _call("hv_filter2d_mask", lens.data_ptr(), W, H, *_f2d_radii(W, H), 1, None)
            else:
                s["mask"] = torch.zeros((H, W), dtype=torch.complex64, device="cuda")
                s["work2"] = torch.zeros((B, H, W), dtype=torch.complex64, device="cuda")
                _call("hv_filter2d_mask", s["mask"].data_ptr(), W, H, *_f2d_radii(W, H), 0, None)
        s.update(raw=raw, lens=lens, work=torch.zeros((B, H, W), dtype=torch.complex64, device="cuda"),
                 ring=torch.zeros((B, H, W), dtype=torch.complex64, device="cuda"))
    elif kind in ("view", "hologram"):
        T, K, img = case["T"], case["K"], case["img"]
        s["ring_c"] = _ring(g, T, W, H)
        s["weights"] = torch.zeros((K, T), dtype=torch.complex64, device="cuda")
        _call("hv_stft_weights", s["weights"].data_ptr(), T, case["p"], case["p"] + K - 1, None)
        s["view"] = torch.zeros((H, W), dtype=torch.float32, device="cuda")
        s["npart"] = hv.lib().hv_time_view_partials(W, H)
        s["partials"] = torch.zeros(s["npart"], dtype=torch.float64, device="cuda")
        if img >= hv.IMG_MOMENTS_0:
            s["bin_w"] = torch.zeros(K, dtype=torch.float32, device="cuda")
            _call("hv_moment_bin_weights", s["bin_w"].data_ptr(), T, case["p"], case["p"] + K - 1, img, 1000.0, None)
        elif case.get("tc"):
            s["tc_work"] = _bytes(hv.lib().hv_time_view_tc_workspace(K, T))
            _call("hv_time_view_tc_prepare", s["weights"].data_ptr(), K, T, s["tc_work"].data_ptr(), None)
        if kind == "hologram":
            A = case["acc"]
            s["reduce"] = _bytes(hv.lib().hv_reduce_workspace(W * H))
            s["pct"] = _bytes(hv.lib().hv_percentile_workspace(W * H))
            s["range"] = torch.zeros(2, dtype=torch.float32, device="cuda")
            # the accumulation queue, full: renormalised frames of the previous windows, the oldest in slot 0
            old = torch.rand((A, H, W), generator=g, device="cuda")
            s["acc_ring"] = old * 60.0 + 2.0
            s["image"] = torch.zeros((H, W), dtype=torch.float32, device="cuda")
            s["out"] = torch.zeros((H, W), dtype=torch.int16, device="cuda")  # the bytes of uint16 pixels
    elif kind == "pca":
        T, K = case["T"], case["K"]
        s["ring_c"] = _ring(g, T, W, H)
        s["cov"] = torch.zeros((T, T), dtype=torch.complex128, device="cuda")
        s["evecs"] = torch.zeros((T, T), dtype=torch.complex128, device="cuda")
        s["evals"] = torch.zeros(T, dtype=torch.float64, device="cuda")
        s["weights"] = torch.zeros((K, T), dtype=torch.complex64, device="cuda")
        s["cov_work"] = _bytes(hv.lib().hv_pca_cov_workspace(T, W * H))
        s["eig_work"] = _bytes(hv.lib().hv_pca_eigh_workspace(T))
        s["view"] = torch.zeros((H, W), dtype=torch.float32, device="cuda")
    elif kind == "unwrap":
        y = torch.arange(H, device="cuda", dtype=torch.float64)[:, None] / H
        x = torch.arange(W, device="cuda", dtype=torch.float64)[None, :] / W
        c = torch.rand(6, generator=g, device="cuda").tolist()
        ph = sum(a * torch.cos(2 * math.pi * (k * x + m * y) + 6 * b)
                 for a, b, k, m in ((4 + 4 * c[0], c[1], 1, 0), (4 + 4 * c[2], c[3], 0, 1), (2 + 2 * c[4], c[5], 2, 1)))
        ph = ph + 0.05 * torch.randn((H, W), generator=g, device="cuda")
        s["phase"] = torch.remainder(ph + math.pi, 2 * math.pi).sub(math.pi).to(torch.float32)
        s["out"] = torch.zeros((H, W), dtype=torch.float32, device="cuda")
        s["work"] = _bytes(hv.lib().hv_unwrap_workspace(W, H))
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------------------------ run
def run(s):
    return _RUN[s["kind"]](s)


def _run_pipe(s):
    pipe, out = s["pipe"], s["out"]
    for b in s["batches"]:
        pipe.enqueue(b)
    for i in range(len(s["batches"])):
        if s["host"]:
            out[i] = pipe.pull()
        else:
            pipe.pull_into(out[i].data_ptr(), hv.MEM_DEVICE)
    return out.view(np.int16) if s["host"] else out


def _run_spatial(s):
    B, W, H = s["B"], s["W"], s["H"]
    if s["mask"] is not None:
        _call("hv_spatial_transform_filter2d", s["raw"].data_ptr(), s["depth"], s["be"], W, H, B, s["space"],
              s["lens"].data_ptr(), s["mask"].data_ptr(), s["work"].data_ptr(), s["work2"].data_ptr(),
              s["ring"].data_ptr(), 0, B, None)
    else:
        _call("hv_spatial_transform", s["raw"].data_ptr(), s["depth"], s["be"], W, H, B, s["space"],
              s["lens"].data_ptr(), s["work"].data_ptr(), s["ring"].data_ptr(), 0, B, None)
    return s["ring"]


def _view(s, shift):
    ring, W, H, T, K = s["ring_c"].data_ptr(), s["W"], s["H"], s["T"], s["K"]
    if s["img"] >= hv.IMG_MOMENTS_0:
        _call("hv_time_moments", ring, T, W, H, s["weights"].data_ptr(), K, s["bin_w"].data_ptr(), shift,
              s["view"].data_ptr(), s["partials"].data_ptr(), None)
    elif s.get("tc"):
        _call("hv_time_view_tc_run", ring, T, W, H, K, s["img"], 1.0, shift, s["view"].data_ptr(),
              s["partials"].data_ptr(), s["tc_work"].data_ptr(), None)
    else:
        _call("hv_time_view", ring, T, W, H, s["weights"].data_ptr(), K, s["img"], 1.0, shift, s["view"].data_ptr(),
              s["partials"].data_ptr(), None)


def _run_view(s):
    _view(s, s["shift"])
    return s["view"]


def _run_hologram(s):
    W, H, A = s["W"], s["H"], s["acc"]
    n = W * H
    _view(s, 1)
    _call("hv_renormalize", s["view"].data_ptr(), n, 5, s["partials"].data_ptr(), s["npart"], s["reduce"].data_ptr(),
          None)
    image = s["view"]
    if A > 1:
        _call("hv_accumulate", image.data_ptr(), s["acc_ring"].data_ptr(), A, 0, 1, A, s["image"].data_ptr(), n, None)
        image = s["image"]
    if s["log"]:
        _call("hv_log10", image.data_ptr(), n, None)
    _call("hv_percentile", image.data_ptr(), W, H, 0.5, 99.5, 0.0, s["range"].data_ptr(), s["pct"].data_ptr(), None)
    _call("hv_contrast_to_ushort", image.data_ptr(), s["range"].data_ptr(), 0, 1, s["out"].data_ptr(), n, None)
    return {"image": image, "range": s["range"], "acc_ring": s["acc_ring"], "out": s["out"]}


def _run_pca(s):
    W, H, T, K = s["W"], s["H"], s["T"], s["K"]
    _call("hv_pca_covariance", s["ring_c"].data_ptr(), T, W * H, s["cov"].data_ptr(), s["cov_work"].data_ptr(), None)
    _call("hv_pca_eigh", s["cov"].data_ptr(), T, s["evals"].data_ptr(), s["evecs"].data_ptr(), T - K, T - 1,
          s["weights"].data_ptr(), s["eig_work"].data_ptr(), None)
    _call("hv_time_view", s["ring_c"].data_ptr(), T, W, H, s["weights"].data_ptr(), K, s["img"], 1.0, 1,
          s["view"].data_ptr(), None, None)
    return s["view"]


def _run_unwrap(s):
    _call("hv_unwrap_2d", s["phase"].data_ptr(), s["out"].data_ptr(), s["W"], s["H"], s["work"].data_ptr(), None)
    return s["out"]


_RUN = {"pipe": _run_pipe, "spatial": _run_spatial, "view": _run_view, "hologram": _run_hologram, "pca": _run_pca,
        "unwrap": _run_unwrap}


# ------------------------------------------------------------------------------------ work
def work(case):
    W, H, kind = case["W"], case["H"], case["kind"]
    n = W * H
    fft2 = 5.0 * n * math.log2(n)
    if kind == "spatial":
        B = case["B"]
        passes = (2 if case["space"] == hv.SPACE_ANGULARSP else 1) + (2 if case["f2d"] and case["space"] == 1 else 0)
        return {"bytes": B * n * (case["depth"] + 8) + 8 * n, "flops": B * (passes * fft2 + 6 * n)}
    if kind == "view":
        return {"bytes": 8 * n * case["T"] + 4 * n, "flops": 8.0 * n * case["T"] * case["K"]}
    if kind == "pca":
        T = case["T"]
        return {"bytes": 8 * n * T + 4 * n, "flops": 4.0 * n * T * T + 8.0 * n * T * case["K"]}
    if kind == "unwrap":
        return {"bytes": 8 * n, "flops": 6 * fft2}
    if kind == "hologram":
        # ring in; accumulation queue read and written in one slot; float image and uint16 hologram out
        return {"bytes": n * (8 * case["T"] + (4 * case["acc"] if case["acc"] > 1 else 0) + 4 + 2),
                "flops": 8.0 * n * case["T"] * case["K"]}
    # a pipe, per hologram: the new raw frames in, the rest of the window from the pipe's ring, uint16 out
    T, S, K = case["T"], case["S"], case["pw"] + 1
    keep = 8 if case["space"] else case["depth"]
    per = n * (S * case["depth"] + (T - S) * keep + 2)
    spatial = S * (fft2 * (2 if case["space"] == 2 else 1 if case["space"] == 1 else 0))
    # frames without a spatial transform stay real
    flops = spatial + (8.0 if case["space"] else 4.0) * n * T * K
    if case["time"] == hv.TIME_PCA:
        flops += (8.0 if case["space"] else 2.0) * n * T * S
    return {"bytes": case["windows"] * per, "flops": case["windows"] * flops}


# ------------------------------------------------------------------------------------ exact
def exact(case, seed):
    """What run() returns for these inputs in 64-bit arithmetic (uint16 holograms: no such value)."""
    kind = case["kind"]
    if kind == "pipe":
        return None
    s = prepare(case, seed)
    W, H = case["W"], case["H"]
    if kind == "spatial":
        return _exact_spatial(s)
    if kind == "unwrap":
        return _exact_unwrap(s["phase"].double(), W, H)
    if kind == "pca":
        T, K = case["T"], case["K"]
        c = torch.zeros((T, T), dtype=torch.complex128, device="cuda")
        flat = s["ring_c"].reshape(T, W * H)
        for part in flat.split(1 << 18, dim=1):
            x = part.to(torch.complex128)
            c += x.conj() @ x.T
        _, v = torch.linalg.eigh(c)
        return _exact_view(s["ring_c"], v[:, T - K:].T, case["img"], None, 1)
    T, K, p = case["T"], case["K"], case["p"]
    k = torch.arange(p, p + K, device="cuda", dtype=torch.float64)[:, None]
    t = torch.arange(T, device="cuda", dtype=torch.float64)[None, :]
    ang = -2.0 * math.pi * torch.remainder(k * t, T) / T
    w = torch.complex(torch.cos(ang), torch.sin(ang))
    if kind == "view":
        bins = _moment_weights(T, p, K, case["img"]) if case["img"] >= hv.IMG_MOMENTS_0 else None
        return _exact_view(s["ring_c"], w, case["img"], bins, case["shift"])
    v = _exact_view(s["ring_c"], w, case["img"], None, 1)
    v = v * 32.0 * (W * H) / v.sum()
    acc = s["acc_ring"].double()
    if case["acc"] > 1:
        acc[0] = v
        v = acc.mean(dim=0)
    if case["log"]:
        v = torch.log10(v)
    ordered = v.flatten().sort().values
    rank = [int(np.float32(np.float32(q) / np.float32(100.0)) * np.float32(W * H)) for q in (0.5, 99.5)]
    rng = torch.stack([ordered[min(r, W * H - 1)].clamp(min=1.0) for r in rank])
    return {"image": v, "range": rng, "acc_ring": acc, "out": None}


def _exact_view(ring, w, img, bins, shift):
    T, H, W = ring.shape
    out = torch.empty(H * W, dtype=torch.float64, device="cuda")
    flat = ring.reshape(T, H * W)
    for at in range(0, H * W, 1 << 17):
        x = w @ flat[:, at:at + (1 << 17)].to(torch.complex128)
        if bins is not None:
            v = (x.abs().square() * bins[:, None]).sum(dim=0)
        else:
            v = (x.angle() if img == hv.IMG_ARGUMENT else x.abs() if img == hv.IMG_MODULUS
                 else x.abs().square()).mean(dim=0)
        out[at:at + (1 << 17)] = v
    out = out.reshape(H, W)
    return torch.roll(out, (H // 2, W // 2), (0, 1)) if shift else out


def _moment_weights(T, p, K, img):
    """f_k^n of the bins, f_k the signed frequency in units of 1000 / T, the Nyquist bin of an even window twice for
    n = 0, 2 and not at all for n = 1."""
    n = img - hv.IMG_MOMENTS_0
    step = float(np.float32(1000.0) / np.float32(T))
    w = []
    for k in range(p, p + K):
        nyquist = T % 2 == 0 and k == T // 2
        f = step * (k if k < (T + 1) // 2 else k - T)
        w.append((0.0 if n == 1 else 2.0) * f ** n if nyquist else f ** n)
    return torch.tensor(w, dtype=torch.float64, device="cuda")


def _exact_spatial(s):
    W, H, space = s["W"], s["H"], s["space"]
    lam, z = (float(np.float32(v)) for v in _optics(space))
    pitch = float(np.float32(PITCH_UM)) * 1e-6
    f64 = dict(dtype=torch.float64, device="cuda")
    if space == hv.SPACE_FRESNELTR:
        m = max(W, H)
        x = (torch.arange(W, **f64) + (m - W) // 2 - m // 2)[None, :] * pitch
        y = (torch.arange(H, **f64) + (m - H) // 2 - m // 2)[:, None] * pitch
        ph = math.pi / (lam * z) * (x * x + y * y)
    else:
        u = (torch.fft.fftfreq(W, **f64) / pitch)[None, :]
        v = (torch.fft.fftfreq(H, **f64) / pitch)[:, None]
        ph = 2 * math.pi * z / lam * torch.sqrt((1.0 - lam * lam * (u * u + v * v)).clamp(min=0.0))
    ph = torch.remainder(ph, 2 * math.pi)
    lens = torch.complex(torch.cos(ph), torch.sin(ph))
    mask = None
    if s["f2d"]:
        n1, n2, sl, sh = _f2d_radii(W, H)
        r = torch.hypot((torch.fft.fftfreq(W, **f64) * W)[None, :], (torch.fft.fftfreq(H, **f64) * H)[:, None])

        def disc(radius, smooth):
            edge = torch.cos((r - radius) / smooth * (math.pi / 2))
            return torch.where(r < radius, torch.ones_like(r), torch.where(r < radius + smooth, edge,
                                                                           torch.zeros_like(r)))
        mask = disc(n2, sh) * (1.0 - disc(n1, sl))
    raw = s["raw"]
    if s["be"]:
        B = s["B"]
        raw = raw.view(torch.uint8).reshape(B, H, W, 2).flip(-1).contiguous().view(torch.int16).reshape(B, H, W)
    out = torch.empty((s["B"], H, W), dtype=torch.complex128, device="cuda")
    for b in range(s["B"]):
        x = raw[b].double() * (257.0 if s["depth"] == 1 else 1.0)
        x = x.to(torch.complex128)
        if space == hv.SPACE_FRESNELTR:
            if mask is not None:
                x = torch.fft.ifft2(torch.fft.fft2(x) * mask) * (W * H)
            out[b] = torch.fft.fft2(x * lens)
        else:
            out[b] = torch.fft.ifft2(torch.fft.fft2(x) * (lens if mask is None else lens * mask))
    return out


def _exact_unwrap(p, W, H):
    """The Fourier unwrap of the flat frame taken as W rows of H samples, rescaled to [0, 65535]."""
    e = torch.arange(W * H, device="cuda")
    fx = ((e % W + W // 2) % W - W // 2).double().reshape(W, H)
    fy = ((e // W + H // 2) % H - H // 2).double().reshape(W, H)
    z = torch.polar(torch.ones_like(p), p).reshape(W, H)
    spectrum = torch.fft.fft2(z)
    acc = torch.zeros_like(spectrum)
    norm = fx * fx + fy * fy
    norm[norm == 0] = 1.0  # both numerators are 0 there
    for f in (fx, fy):
        grad = torch.fft.ifft2(spectrum * f) * (2j * math.pi) * torch.conj(1j * z)
        acc += torch.fft.fft2(grad) * (f / norm)
    v = torch.fft.ifft2(acc).imag / (-2 * math.pi)
    lo, hi = v.min(), v.max()
    return ((v - lo) / (hi - lo) * 65535.0).reshape(H, W)
