// Rendering stage on the float view frame: 2-D phase unwrap, renormalisation, fftshift,
// image accumulation, log10, percentile autocontrast and the contrast map to uint16.
//
// Reference behaviour (Holovibes):
//   unwrap_2d      Backend/cuda_sources/tools_unwrap.cu:79-95,269-369, tools.cu:50-68
//   rescale        Backend/cuda_sources/tools_conversion.cu:315-335
//   renorm         Backend/cuda_sources/tools_compute.cu:99-123, Backend/sources/compute/postprocessing.cc:135-155
//   fftshift       Backend/cuda_sources/shift_corners.cu:8-70
//   accumulation   Backend/cuda_sources/tools_conversion.cu:418-458, Backend/sources/compute/image_accumulation.cc:136-157
//   percentile     Backend/cuda_sources/percentile.cu:15-43,75-94,139-222, Backend/sources/api/contrast_api.cc:137-146
//   contrast       Backend/cuda_sources/contrast_correction.cu:5-17
//   float->ushort  Backend/cuda_sources/tools_conversion.cu:350-387
//
// GB300 design: the percentile is an exact three-pass radix select on order-preserving float keys
// (11/11/10 bits) instead of a full thrust sort, and the selected range never leaves the device:
// the contrast kernel reads it from device memory, so no host round trip or stream sync happens.
#include <float.h>
#include <math.h>

#include <initializer_list>
#include <mutex>
#include <string>

#include "hv_common.cuh"
#include "hv_internal.h"

namespace hv {

constexpr int EW_THREADS = 256;

static int ew_grid(size_t n)
{
    size_t g = (n + EW_THREADS - 1) / EW_THREADS;
    const size_t cap = 152 * 32;
    return static_cast<int>(g < cap ? (g > 0 ? g : 1) : cap);
}

// V consecutive floats (V = 4: one 16-byte access).
template <int V>
__device__ __forceinline__ void load_v(const float* p, float (&v)[V])
{
    if constexpr (V == 4)
    {
        const float4 f = *reinterpret_cast<const float4*>(p);
        v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
    }
    else
        v[0] = *p;
}
template <int V>
__device__ __forceinline__ void store_v(float* p, const float (&v)[V])
{
    if constexpr (V == 4)
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else
        *p = v[0];
}

// 16-byte accesses: every buffer aligned, a multiple of 4 pixels (and, with the quadrant swap, rows
// whose halves are a multiple of 4).
static bool vec4_ok(size_t n, std::initializer_list<const void*> buffers)
{
    uintptr_t bits = n % 4 ? 1 : 0;
    for (const void* p : buffers)
        bits |= reinterpret_cast<uintptr_t>(p) & 15;
    return bits == 0;
}

// ====================================================================================== unwrap

// The element-wise steps run on V consecutive elements per thread (V = 4: 16-byte accesses). Between
// the eight FFT passes of one frame they are bound by latency; 32-bit index divisions, and one
// atomic pair per CTA for the extremes (one per warp held k_unwrap_last at 26 us for 768 x 768).

// V consecutive complex values (V = 1 or 4).
template <int V>
__device__ __forceinline__ void load_c(const float2* p, float2 (&v)[V])
{
    if constexpr (V == 4)
    {
        const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
        v[0] = make_float2(a.x, a.y), v[1] = make_float2(a.z, a.w);
        v[2] = make_float2(b.x, b.y), v[3] = make_float2(b.z, b.w);
    }
    else
        v[0] = *p;
}
template <int V>
__device__ __forceinline__ void store_c(float2* p, const float2 (&v)[V])
{
    if constexpr (V == 4)
    {
        reinterpret_cast<float4*>(p)[0] = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
        reinterpret_cast<float4*>(p)[1] = make_float4(v[2].x, v[2].y, v[3].x, v[3].y);
    }
    else
        *p = v[0];
}

// z = exp(i*phase) (kernel_init_unwrap_2d); the extremes' keys start empty
template <int V>
__global__ void k_unwrap_init(const float* in, float2* z, unsigned int n, unsigned int* minmax)
{
    wait_prior_kernels();
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        minmax[0] = 0xffffffffu;
        minmax[1] = 0u;
    }
    const unsigned int e = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (e >= n)
        return;
    float v[V];
    load_v<V>(in + e, v);
    float2 o[V];
#pragma unroll
    for (int k = 0; k < V; ++k)
    {
        float s, c;
        sincosf(v[k], &s, &c);
        o[k] = make_float2(c, s);
    }
    store_c<V>(z + e, o);
}

// Frequency index of flat element e after circ_shift(-W/2, -H/2) of the fx / fy grids:
// sfx[y][x] = ((x + W/2) % W) - W/2, sfy[y][x] = ((y + H/2) % H) - H/2.
__device__ __forceinline__ void shifted_freqs(unsigned int e, int W, int H, float& fx, float& fy)
{
    const int y = static_cast<int>(e / static_cast<unsigned int>(W));
    const int x = static_cast<int>(e - static_cast<unsigned int>(y) * static_cast<unsigned int>(W));
    fx = static_cast<float>((x + (W >> 1)) % W - (W >> 1));
    fy = static_cast<float>((y + (H >> 1)) % H - (H >> 1));
}

// gx = Z * sfx, gy = Z * sfy (kernel_multiply_complexes_by_floats_)
template <int V>
__global__ void k_unwrap_grad_freq(const float2* Z, float2* gx, float2* gy, int W, int H)
{
    wait_prior_kernels();
    const unsigned int n = static_cast<unsigned int>(W) * H, e = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (e >= n)
        return;
    float2 v[V], ox[V], oy[V];
    load_c<V>(Z + e, v);
#pragma unroll
    for (int k = 0; k < V; ++k)
    {
        float fx, fy;
        shifted_freqs(e + k, W, H, fx, fy);
        ox[k] = cscale(v[k], fx);
        oy[k] = cscale(v[k], fy);
    }
    store_c<V>(gx + e, ox);
    store_c<V>(gy + e, oy);
}

// g *= (i * 2pi) then g *= conj(i z) (kernel_multiply_complexes_by_single_complex, eq_unwrap_2d)
template <int V>
__global__ void k_unwrap_eq(float2* gx, float2* gy, const float2* z, unsigned int n, float two_pi)
{
    wait_prior_kernels();
    const float2 i2pi = make_float2(0.f, two_pi);
    const unsigned int e = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (e >= n)
        return;
    float2 vz[V], vx[V], vy[V];
    load_c<V>(z + e, vz);
    load_c<V>(gx + e, vx);
    load_c<V>(gy + e, vy);
#pragma unroll
    for (int k = 0; k < V; ++k)
    {
        const float2 zc = cconj(cmul(vz[k], make_float2(0.f, 1.f)));
        vx[k] = cmul(cmul(vx[k], i2pi), zc);
        vy[k] = cmul(cmul(vy[k], i2pi), zc);
    }
    store_c<V>(gx + e, vx);
    store_c<V>(gy + e, vy);
}

// acc = gx * sfx/(sfx^2+sfy^2) + gy * sfy/(...) (kernel_norm_ratio + kernel_add_complex_frames)
template <int V>
__global__ void k_unwrap_ratio(const float2* gx, const float2* gy, float2* acc, int W, int H)
{
    wait_prior_kernels();
    const unsigned int n = static_cast<unsigned int>(W) * H, e = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (e >= n)
        return;
    float2 vx[V], vy[V], r[V];
    load_c<V>(gx + e, vx);
    load_c<V>(gy + e, vy);
#pragma unroll
    for (int k = 0; k < V; ++k)
    {
        float fx, fy;
        shifted_freqs(e + k, W, H, fx, fy);
        const float norm = fx * fx + fy * fy;
        r[k] = make_float2(0.f, 0.f);
        if (norm != 0.f)
        {
            const float cx = fx / norm, cy = fy / norm;
            r[k] = cadd(cscale(vx[k], cx), cscale(vy[k], cy));
        }
    }
    store_c<V>(acc + e, r);
}

// order-preserving keys of floats
__device__ __forceinline__ unsigned int float_key(float f)
{
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned int k)
{
    const unsigned int u = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    return __uint_as_float(u);
}

// out = Im(acc) / -2pi (kernel_unwrap2d_last_step) and the frame's extremes
template <int V>
__global__ void __launch_bounds__(EW_THREADS) k_unwrap_last(const float2* acc, float* out, unsigned int n,
                                                            float two_pi, unsigned int* minmax)
{
    wait_prior_kernels();
    __shared__ unsigned int lo[EW_THREADS / 32], hi[EW_THREADS / 32];
    unsigned int kmin = 0xffffffffu, kmax = 0u;
    const unsigned int e = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (e < n)
    {
        float2 a[V];
        float v[V];
        load_c<V>(acc + e, a);
#pragma unroll
        for (int k = 0; k < V; ++k)
        {
            v[k] = a[k].y / -two_pi;
            const unsigned int key = float_key(v[k]);
            kmin = min(kmin, key);
            kmax = max(kmax, key);
        }
        store_v<V>(out + e, v);
    }
    kmin = __reduce_min_sync(0xffffffffu, kmin);
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    if ((threadIdx.x & 31) == 0)
    {
        lo[threadIdx.x >> 5] = kmin;
        hi[threadIdx.x >> 5] = kmax;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
#pragma unroll
        for (int w = 1; w < EW_THREADS / 32; ++w)
        {
            kmin = min(kmin, lo[w]);
            kmax = max(kmax, hi[w]);
        }
        atomicMin(minmax, kmin);
        atomicMax(minmax + 1, kmax);
    }
}

// rescale_float_unwrap2d: (in + |min|)/(|min| + max)*65535 if min < 0 else (in - min)/(max - min)*65535
template <int V>
__global__ void k_unwrap_rescale(float* io, unsigned int n, const unsigned int* minmax)
{
    wait_prior_kernels();
    const float mn = key_float(minmax[0]), mx = key_float(minmax[1]);
    const unsigned int e = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (e >= n)
        return;
    float v[V];
    load_v<V>(io + e, v);
#pragma unroll
    for (int k = 0; k < V; ++k)
    {
        // a constant frame maps to 0 (the reference divides 0 by 0 there)
        if (mx == mn)
            v[k] = 0.0f;
        else if (mn < 0.f)
            v[k] = __fdiv_rn(__fadd_rn(v[k], fabsf(mn)), __fadd_rn(fabsf(mn), mx)) * 65535.0f;
        else
            v[k] = __fdiv_rn(__fsub_rn(v[k], mn), __fsub_rn(mx, mn)) * 65535.0f;
    }
    store_v<V>(io + e, v);
}

size_t unwrap_workspace(int W, int H)
{
    const size_t n = static_cast<size_t>(W) * H;
    return 4 * n * sizeof(float2) + 256;
}

template <int V>
static hv_status unwrap_steps(const float* in, float* out, int W, int H, void* work, cudaStream_t st)
{
    const unsigned int n = static_cast<unsigned int>(W) * H;
    // The reference plans its unwrap FFT with plan(width, height) (icompute.hh:140): the
    // row-major buffer is transformed as `width` rows of `height` samples.
    const int n0 = W, n1 = H;
    float2* z = static_cast<float2*>(work);
    float2* g = z + n;  // gx, gy contiguous (batch of 2)
    float2* gx = g;
    float2* gy = g + n;
    float2* Z = g + 2 * static_cast<size_t>(n);
    unsigned int* minmax = reinterpret_cast<unsigned int*>(Z + n);
    const float two_pi = 6.28318530717959f;  // M_2PI of common.cuh:29
    const int grid = static_cast<int>((n / V + EW_THREADS - 1) / EW_THREADS);
    hv_status s;
    HV_LAUNCH(k_unwrap_init<V>, grid, EW_THREADS, 0, st, in, z, n, minmax);
    if ((s = fft2d(z, Z, n0, n1, 1, 0, 1.0f, st)) != HV_OK)
        return s;
    HV_LAUNCH(k_unwrap_grad_freq<V>, grid, EW_THREADS, 0, st, Z, gx, gy, W, H);
    if ((s = fft2d(g, g, n0, n1, 2, 1, 1.0f, st)) != HV_OK)
        return s;
    HV_LAUNCH(k_unwrap_eq<V>, grid, EW_THREADS, 0, st, gx, gy, z, n, two_pi);
    if ((s = fft2d(g, g, n0, n1, 2, 0, 1.0f, st)) != HV_OK)
        return s;
    HV_LAUNCH(k_unwrap_ratio<V>, grid, EW_THREADS, 0, st, gx, gy, Z, W, H);
    if ((s = fft2d(Z, Z, n0, n1, 1, 1, 1.0f, st)) != HV_OK)
        return s;
    HV_LAUNCH(k_unwrap_last<V>, grid, EW_THREADS, 0, st, Z, out, n, two_pi, minmax);
    HV_LAUNCH(k_unwrap_rescale<V>, grid, EW_THREADS, 0, st, out, n, minmax);
    count_launch(6);
    return HV_OK;
}

hv_status unwrap_2d(const float* in, float* out, int W, int H, void* work, cudaStream_t st)
{
    if (!fft_size_supported(W) || !fft_size_supported(H))
    {
        set_last_error_msg("unwrap_2d: frame size not supported by the shared-memory FFT");
        return HV_ERR_UNSUPPORTED;
    }
    // transform lengths are multiples of 16, so only the buffers' alignment decides
    return vec4_ok(static_cast<size_t>(W) * H, {in, out, work}) ? unwrap_steps<4>(in, out, W, H, work, st)
                                                                : unwrap_steps<1>(in, out, W, H, work, st);
}

// ---------------------------------------------------------------------- unwrap without allocation
// Some callers cannot allocate device memory at all: a frame-grabber or acquisition callback that
// runs on a driver thread with a real-time budget, or a host application whose memory policy
// forbids cudaMalloc once streaming has started. hv_unwrap_2d_noalloc serves them: its scratch
// (four complex frames and the min/max keys, the same layout hv_unwrap_2d takes from `work`) is
// this file-scope device array, sized for frames of at most HV_UNWRAP_NOALLOC_MAX_PIXELS pixels.
// Every GPU that loads the library keeps the array (8 MiB) until the process exits. With CUDA's
// lazy module loading the driver creates the array (and this module's other device data) when
// one of the module's kernels first runs on a device, so the first call on each device is the
// one that may allocate inside the driver: make it before streaming starts.

constexpr size_t kUnwrapNoallocMaxPixels = HV_UNWRAP_NOALLOC_MAX_PIXELS;
static __device__ __align__(256) float2 g_unwrap_scratch[4 * kUnwrapNoallocMaxPixels + 32];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mu;
void* g_scratch_ptr[kMaxDevices] = {};
}  // namespace

hv_status unwrap_2d_noalloc(const float* in, float* out, int W, int H, cudaStream_t st)
{
    if (W <= 0 || H <= 0)
    {
        set_last_error_msg("hv_unwrap_2d_noalloc: width and height must be positive");
        return HV_INVALID_VALUE;
    }
    const size_t n = static_cast<size_t>(W) * H;
    if (n > kUnwrapNoallocMaxPixels)
    {
        set_last_error_msg(("hv_unwrap_2d_noalloc: the frame's " + std::to_string(n) +
                            " pixels exceed the 262144-pixel static scratch").c_str());
        return HV_INVALID_VALUE;
    }
    int dev = 0;
    HV_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices)
    {
        set_last_error_msg(("hv_unwrap_2d_noalloc: device index " + std::to_string(dev) +
                            " beyond the 64 devices this entry point serves").c_str());
        return HV_INVALID_VALUE;
    }
    void* ptr = nullptr;
    {
        // set-up on the first call on each device (with that device current): the host-side name
        // of the array is not a device address, so fetch the address once and keep it
        std::lock_guard<std::mutex> g(g_scratch_mu);
        if (!g_scratch_ptr[dev])
        {
            void* p = nullptr;
            HV_CUDA_TRY(cudaGetSymbolAddress(&p, g_unwrap_scratch));
            g_scratch_ptr[dev] = p;
        }
        ptr = g_scratch_ptr[dev];
    }
    // every buffer of the scratch is fully written before it is read, and the min/max keys are
    // re-initialised by unwrap_2d itself, so the previous call's contents never leak into this one
    return unwrap_2d(in, out, W, H, ptr, st);
}

// ====================================================================================== renorm

size_t reduce_workspace(size_t n)
{
    return static_cast<size_t>(ew_grid(n)) * sizeof(double) + 64;
}

__global__ void k_partial_sums(const float* in, size_t n, double* partials, const CycleCtl* ctl)
{
    wait_prior_kernels();
    if (!ctl_render(ctl))
        return;
    __shared__ double red[EW_THREADS / 32];
    double s = 0.0;
    for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < n;
         e += static_cast<size_t>(gridDim.x) * blockDim.x)
        s += in[e];
    for (int o = 16; o > 0; o >>= 1)
        s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double t = 0.0;
        for (int i = 0; i < EW_THREADS / 32; ++i)
            t += red[i];
        partials[blockIdx.x] = t;
    }
}

hv_status renorm_sum(const float* frame, size_t n, int renorm_constant, const double* partials, int npartials,
                     void* work, cudaStream_t st, RenormSum* sum, const CycleCtl* ctl)
{
    if (!partials)
    {
        double* p = static_cast<double*>(work);
        const int grid = ew_grid(n);
        HV_LAUNCH(k_partial_sums, grid, EW_THREADS, 0, st, frame, n, p, ctl);
        count_launch();
        partials = p;
        npartials = grid;
    }
    *sum = RenormSum{partials, npartials, n, renorm_constant};
    return HV_OK;
}

// The renormalisation factors x' = (x * f[0]) * f[1], f[0] = 2^c and f[1] = (float)N / (float)sum of
// the partial sums, for every thread of a CTA of RN_THREADS. FP64 additions run at a few per clock
// and SM here, so the tree adds each pair once (47 warp additions; every lane of a shuffle tree adds
// in 160). The order of the additions is fixed: thread i sums entries i, i + 1024, ..., then each
// warp's 32 sums as a tree, then the warps in order.
constexpr int RN_THREADS = 1024;

__device__ __forceinline__ void renorm_factors(const RenormSum& r, float& f0, float& f1)
{
    __shared__ double a[RN_THREADS], b[RN_THREADS / 2];
    __shared__ float f[2];
    const int tid = threadIdx.x;
    double s = 0.0;
    int i = tid;
    for (; i + 7 * RN_THREADS < r.np; i += 8 * RN_THREADS)
    {
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            v[k] = r.partials[i + k * RN_THREADS];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            s += v[k];
    }
    for (; i < r.np; i += RN_THREADS)
        s += r.partials[i];
    a[tid] = s;
    __syncthreads();
    if (tid < RN_THREADS / 2)  // lanes l and l + 16 of warp w
        b[tid] = a[(tid >> 4) * 32 + (tid & 15)] + a[(tid >> 4) * 32 + (tid & 15) + 16];
    __syncthreads();
    if (tid < RN_THREADS / 4)  // eight lanes per warp's tree
    {
        double t = b[(tid >> 3) * 16 + (tid & 7)] + b[(tid >> 3) * 16 + (tid & 7) + 8];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
            t += __shfl_down_sync(0xffffffffu, t, o, 8);
        if ((tid & 7) == 0)
            a[tid >> 3] = t;
    }
    __syncthreads();
    if (tid == 0)
    {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < RN_THREADS / 32; ++w)
            t += a[w];
        f[0] = static_cast<float>(1 << r.c);
        // a zero-sum frame (all zero) stays zero instead of the reference's N / 0 = inf, 0 * inf = NaN
        f[1] = t != 0.0 ? __fdiv_rn(static_cast<float>(r.n), static_cast<float>(t)) : 0.0f;
    }
    __syncthreads();
    f0 = f[0];
    f1 = f[1];
}

// Fused: renormalise (sum.partials null: not), optional quadrant swap (out of place), optional
// accumulation into an A-frame ring (write slot, mean of `count` frames from `start`), optional
// log10. V pixels per thread and step. Bound by latency (a few MB from L2): the factors without a
// launch of their own and 16-byte accesses take the renormalisation of 1024 x 1024 from 8.8 + 10.2 to
// 9.8 us, log10 from 5.3 to 4.0 us and the contrast map below from 6.1 to 3.8 us (serialised launch
// times, cold caches); the mean of 8 frames, whose loads go out together, stays at 10.4 us (its 38 MB
// come from DRAM there).
template <int V>
__global__ void __launch_bounds__(RN_THREADS) k_renorm_shift_acc(const float* in, float* out, int W, int H,
                                                                 RenormSum sum, int shift, float* acc, int A, int slot,
                                                                 int start, int count, int log_enabled, float prescale,
                                                                 const CycleCtl* ctl)
{
    wait_prior_kernels();
    if (!ctl_render(ctl))
        return;
    if (ctl)
    {
        slot = ctl->acc_slot;
        start = ctl->acc_start;
        count = ctl->acc_count;
    }
    const size_t n = static_cast<size_t>(W) * H;
    float m0 = 1.f, m1 = 1.f;
    if (sum.partials)
        renorm_factors(sum, m0, m1);
    for (size_t e = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) * V; e < n;
         e += static_cast<size_t>(gridDim.x) * blockDim.x * V)
    {
        size_t src = e;
        if (shift)  // V = 4: W a multiple of 8, so the four pixels stay together
        {
            const int x = static_cast<int>(e % W), y = static_cast<int>(e / W);
            src = static_cast<size_t>((y + H / 2) % H) * W + (x + W / 2) % W;
        }
        float v[V];
        load_v<V>(in + src, v);
#pragma unroll
        for (int k = 0; k < V; ++k)
        {
            if (prescale != 1.0f)
                v[k] = v[k] * prescale;
            if (sum.partials)
                v[k] = (v[k] * m0) * m1;
        }
        if (acc)
        {
            store_v<V>(acc + static_cast<size_t>(slot) * n + e, v);
            float s[V];
#pragma unroll
            for (int k = 0; k < V; ++k)
                s[k] = 0.f;
            constexpr int D = 8;  // frames whose loads are issued together
            int pos = start;
            for (int i = 0; i < count; i += D)
            {
                float q[D][V];
                int at = pos;
#pragma unroll
                for (int d = 0; d < D; ++d)
                {
                    if (i + d < count && at != slot)
                        load_v<V>(acc + static_cast<size_t>(at) * n + e, q[d]);
                    if (++at == A)
                        at = 0;
                }
#pragma unroll
                for (int d = 0; d < D; ++d)
                {
                    if (i + d < count)
                    {
#pragma unroll
                        for (int k = 0; k < V; ++k)
                            s[k] += pos == slot ? v[k] : q[d][k];
                    }
                    if (++pos == A)
                        pos = 0;
                }
            }
#pragma unroll
            for (int k = 0; k < V; ++k)
                v[k] = s[k] / static_cast<float>(count);
        }
        if (log_enabled)
        {
#pragma unroll
            for (int k = 0; k < V; ++k)
                v[k] = log10f(v[k]);
        }
        store_v<V>(out + e, v);
    }
}

static hv_status launch_renorm_shift_acc(const float* in, float* out, int W, int H, const RenormSum& sum, int shift,
                                         float* acc, int A, int slot, int start, int count, int log_enabled,
                                         float prescale, const CycleCtl* ctl, cudaStream_t st)
{
    const size_t n = static_cast<size_t>(W) * H;
    const bool v4 = vec4_ok(n, {in, out, acc}) && (!shift || W % 8 == 0);
    // with the factors: CTAs of 1024 threads, one per SM (each sums the partials: the SM's FP64 rate
    // bounds that, so a second CTA would double it). Without 16-byte accesses large frames wait for their loads: two
    // per SM from where each thread still has 8 pixels (2048 x 2048 46.8 -> 44.1 us, 4096 x 3000 94.4 -> 83.4, but
    // 512 x 512 10.0 -> 10.6; with 16-byte accesses 40.5 -> 44.7 and 75.6 -> 79.4)
    const int block = sum.partials ? RN_THREADS : EW_THREADS;
    const size_t per = static_cast<size_t>(block) * (v4 ? 4 : 1);
    const size_t want = (n + per - 1) / per, cap = !sum.partials ? 152 * 32 : !v4 && n >= 2 * 152 * RN_THREADS * size_t(8) ? 2 * 152 : 152;
    const int grid = static_cast<int>(want < cap ? (want > 0 ? want : 1) : cap);
    if (v4)
        HV_LAUNCH(k_renorm_shift_acc<4>, grid, block, 0, st, in, out, W, H, sum, shift, acc, A, slot, start, count,
                  log_enabled, prescale, ctl);
    else
        HV_LAUNCH(k_renorm_shift_acc<1>, grid, block, 0, st, in, out, W, H, sum, shift, acc, A, slot, start, count,
                  log_enabled, prescale, ctl);
    count_launch();
    return HV_OK;
}

hv_status renorm_shift_accumulate(const float* in, float* out, int W, int H, const RenormSum* sum, int shift,
                                  float* acc_ring, int A, int slot, int start, int count, int log_enabled,
                                  cudaStream_t st, float prescale, const CycleCtl* ctl)
{
    if (shift && ((W & 1) || (H & 1)))
    {
        set_last_error_msg("fftshift needs even width and height");
        return HV_INVALID_VALUE;
    }
    if (shift && in == out)
    {
        set_last_error_msg("renorm_shift_accumulate: shift must be out of place");
        return HV_INVALID_VALUE;
    }
    return launch_renorm_shift_acc(in, out, W, H, sum ? *sum : RenormSum{}, shift, acc_ring, A, slot, start, count,
                                   log_enabled, prescale, ctl, st);
}

// In-place quadrant swap: thread owns pixel (x, y) of the top half and swaps it with its partner.
__global__ void k_shift_corners(float* f, int W, int H)
{
    wait_prior_kernels();
    const size_t half = static_cast<size_t>(W) * (H / 2);
    for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < half;
         e += static_cast<size_t>(gridDim.x) * blockDim.x)
    {
        const int x = static_cast<int>(e % W), y = static_cast<int>(e / W);
        const int nx = x < W / 2 ? x + W / 2 : x - W / 2;
        const size_t a = static_cast<size_t>(y) * W + x;
        const size_t b = static_cast<size_t>(y + H / 2) * W + nx;
        const float t = f[b];
        f[b] = f[a];
        f[a] = t;
    }
}

hv_status shift_corners(float* frame, int W, int H, cudaStream_t st)
{
    if ((W & 1) || (H & 1))
    {
        set_last_error_msg("shift_corners needs even width and height");
        return HV_INVALID_VALUE;
    }
    HV_LAUNCH(k_shift_corners, ew_grid(static_cast<size_t>(W) * H / 2), EW_THREADS, 0, st, frame, W, H);
    count_launch();
    return HV_OK;
}

hv_status accumulate(const float* frame, float* acc_ring, int A, int slot, int start, int count, float* out, size_t n,
                     cudaStream_t st)
{
    if (A <= 0 || slot < 0 || slot >= A || start < 0 || start >= A || count <= 0 || count > A)
        return HV_INVALID_VALUE;
    // 1-row frame of n pixels: no shift, no renorm
    return launch_renorm_shift_acc(frame, out, static_cast<int>(n), 1, RenormSum{}, 0, acc_ring, A, slot, start, count, 0,
                                   1.0f, nullptr, st);
}

template <int V>
__global__ void k_log10(float* f, size_t n)
{
    wait_prior_kernels();
    for (size_t e = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) * V; e < n;
         e += static_cast<size_t>(gridDim.x) * blockDim.x * V)
    {
        float v[V];
        load_v<V>(f + e, v);
#pragma unroll
        for (int k = 0; k < V; ++k)
            v[k] = log10f(v[k]);
        store_v<V>(f + e, v);
    }
}

hv_status log10_map(float* frame, size_t n, cudaStream_t st)
{
    if (vec4_ok(n, {frame}))
        HV_LAUNCH(k_log10<4>, ew_grid(n / 4), EW_THREADS, 0, st, frame, n);
    else
        HV_LAUNCH(k_log10<1>, ew_grid(n), EW_THREADS, 0, st, frame, n);
    count_launch();
    return HV_OK;
}

// ====================================================================================== percentile
// Exact k-th smallest selection for two ranks at once. Pass d (d = 0, 1, 2) histograms the
// digit d of the order-preserving key of the elements whose higher digits match the prefix
// selected so far for that rank; the CTA that finishes the pass last then picks the digit holding
// the rank. Digits: bits [31:21] (2048 bins), [20:10] (2048 bins), [9:0] (1024 bins).
// Bound by latency and by shared-memory atomics on few addresses (a frame's values share a handful
// of first digits): 16 pixels per thread are loaded together, equal digits of a warp are counted by
// one atomic, and the scan rides on the pass. 1024 x 1024: 3 x (9.0 + 5.1) us as separate histogram and
// scan launches, 3 x 10.4 us here (serialised launch times, cold caches). With a reticle or a pitch, 4 pixels per
// thread are loaded together and their positions take 32-bit divisions: 2048 x 2048 with a reticle of the whole height
// 67 us as separate launches, 97 one pixel after another on the grid of the 16-byte loads, 59.6 here.

constexpr int PCT_BINS = 2048;
constexpr int PCT_SCALAR = 4;  // pixels that a thread of the passes without 16-byte loads asks for together

struct PctState
{
    unsigned int prefix[2];  // selected high bits per rank
    unsigned int rank[2];    // remaining rank inside the prefix
    unsigned int count;      // number of candidate elements (frame or reticle disc)
    unsigned int done[3];    // CTAs that finished each pass
};

__device__ __forceinline__ int digit_shift(int d) { return d == 0 ? 21 : (d == 1 ? 10 : 0); }
__device__ __forceinline__ unsigned int digit_mask(int d) { return d == 2 ? 1023u : 2047u; }
__device__ __forceinline__ unsigned int high_mask(int d) { return d == 0 ? 0u : (d == 1 ? 0xffe00000u : 0xfffffc00u); }

// Where pixel e of the frame lies in memory, and whether it counts (inside the reticle's disc); 32-bit divisions
// where the index allows.
__device__ __forceinline__ size_t pct_pixel(size_t e, int W, int H, int pitch, unsigned int r2, int use_reticle, bool& on)
{
    int x, y;
    if (e >> 32)
    {
        y = static_cast<int>(e / W);
        x = static_cast<int>(e % W);
    }
    else
    {
        const unsigned int q = static_cast<unsigned int>(e) / static_cast<unsigned int>(W);
        y = static_cast<int>(q);
        x = static_cast<int>(static_cast<unsigned int>(e) - q * static_cast<unsigned int>(W));
    }
    if (use_reticle)
    {
        const int dx = x - W / 2, dy = y - H / 2;
        on = on && static_cast<unsigned int>(dx * dx + dy * dy) <= r2;
    }
    return static_cast<size_t>(y) * pitch + x;
}

// Digit of rank r (0 or 1) after pass d from the histogram hh, by a CTA of EW_THREADS (PCT_BINS / 8).
__device__ void pct_select(const unsigned int* hh, PctState* st, int r, int d, float pct, float* range)
{
    constexpr int PER = PCT_BINS / EW_THREADS;
    __shared__ unsigned int warp_tot[EW_THREADS / 32];
    const int nb = (d == 2) ? 1024 : PCT_BINS;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned int c[PER], v = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i)
    {
        const int bin = threadIdx.x * PER + i;
        c[i] = bin < nb ? __ldcg(hh + bin) : 0u;
        v += c[i];
    }
    unsigned int incl = v;
    for (int o = 1; o < 32; o <<= 1)
    {
        const unsigned int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o)
            incl += t;
    }
    __syncthreads();  // warp_tot of the previous rank is read
    if (lane == 31)
        warp_tot[w] = incl;
    __syncthreads();
    unsigned int before = incl - v, total = 0;
#pragma unroll
    for (int i = 0; i < EW_THREADS / 32; ++i)
    {
        before += i < w ? warp_tot[i] : 0u;
        total += warp_tot[i];
    }
    unsigned int rank, candidates;
    if (d == 0)
    {
        // total candidates and the percentile index, float32 as percentile.cu:85, clamped
        candidates = total;
        rank = static_cast<unsigned int>(__fmul_rn(__fdiv_rn(pct, 100.0f), static_cast<float>(total)));
        if (total == 0)
            rank = 0;
        else if (rank >= total)
            rank = total - 1;
    }
    else
    {
        candidates = __ldcg(&st->count);
        rank = __ldcg(&st->rank[r]);
    }
    __syncthreads();  // every thread has the state that one of them replaces
    // first bin whose inclusive count exceeds rank (the last bin when none does)
    const bool mine = rank >= before && rank < before + v;
    const bool last = rank >= total && threadIdx.x == (nb - 1) / PER;
    if (mine || last)
    {
        int bin = threadIdx.x * PER;
        unsigned int below = before;
        if (mine)
        {
            int i = 0;
#pragma unroll
            for (int k = 0; k < PER; ++k)
                if (k == i && rank >= below + c[k])
                {
                    below += c[k];
                    ++i;
                }
            bin += i;
        }
        else
        {
            bin = nb - 1;
            below = total - c[(nb - 1) % PER];
        }
        const unsigned int prefix = (d == 0 ? 0u : st->prefix[r]) | (static_cast<unsigned int>(bin) << digit_shift(d));
        if (d == 0)
            st->count = candidates;
        st->rank[r] = rank - below;
        st->prefix[r] = prefix;
        if (d == 2)
        {
            const float val = candidates ? key_float(prefix) : 0.f;
            // ContrastApi::update_contrast clamps both ends to >= 1
            range[r] = val > 1.0f ? val : 1.0f;
        }
    }
}

// VEC: rows without gaps and no reticle, so the order of the pixels does not matter: 16-byte loads. With EDGES they start
// at the first 16-byte boundary, and the pixels before and behind them are one warp's (a kernel of its own: in the
// aligned one this cost 0.1 of 25.4 us for 1024 x 1024).
template <bool VEC, bool EDGES>
__global__ void __launch_bounds__(EW_THREADS) k_pct_pass(const float* __restrict__ f, int W, int H, int pitch,
                                                         unsigned int r2, int use_reticle, PctState* st, int d,
                                                         unsigned int* hist, float lower, float upper, float* range,
                                                         const CycleCtl* ctl)
{
    wait_prior_kernels();
    if (ctl && !(ctl->render && ctl->pct_enable))
        return;
    __shared__ unsigned int sh[2][PCT_BINS];
    __shared__ bool s_last;
    const int nh = d == 0 ? 1 : 2;
    for (int i = threadIdx.x; i < nh * PCT_BINS; i += EW_THREADS)
        (&sh[0][0])[i] = 0u;
    const size_t n = static_cast<size_t>(W) * H;
    const int sft = digit_shift(d);
    const unsigned int dm = digit_mask(d), hm = high_mask(d);
    const unsigned int pre0 = (d == 0) ? 0u : st->prefix[0];
    const unsigned int pre1 = (d == 0) ? 0u : st->prefix[1];
    __syncthreads();
    // one atomic per distinct digit among the warp's lanes that count one
    auto count = [&](unsigned int* h, unsigned int dig, bool on) {
        const unsigned int active = __ballot_sync(0xffffffffu, on);
        if (!active)
            return;
        if (on)
        {
            const unsigned int same = __match_any_sync(active, dig);
            if ((threadIdx.x & 31) == __ffs(same) - 1)
                atomicAdd(&h[dig], static_cast<unsigned int>(__popc(same)));
        }
    };
    auto take = [&](float x, bool on) {
        const unsigned int k = float_key(x), dig = (k >> sft) & dm;
        if (d == 0)
            count(sh[0], dig, on);
        else
        {
            if (on && (k & hm) == pre0)
                atomicAdd(&sh[0][dig], 1u);
            if (on && (k & hm) == pre1)
                atomicAdd(&sh[1][dig], 1u);
        }
    };
    if constexpr (VEC)
    {
        constexpr int Q = 4;
        const size_t head = EDGES ? min(n, ((16 - (reinterpret_cast<uintptr_t>(f) & 15)) & 15) / sizeof(float)) : 0;
        const size_t n4 = (n - head) / 4, step = static_cast<size_t>(gridDim.x) * EW_THREADS;
        const float4* f4 = reinterpret_cast<const float4*>(f + head);
        if (EDGES && blockIdx.x == 0 && threadIdx.x < 32)
        {
            const bool on = threadIdx.x < n - 4 * n4;
            take(on ? f[threadIdx.x < head ? threadIdx.x : 4 * n4 + threadIdx.x] : 0.f, on);
        }
        // uniform trip count: every lane of a warp takes part in the votes
        const size_t first = blockIdx.x * static_cast<size_t>(EW_THREADS) + threadIdx.x;
        for (size_t base = 0; base < n4; base += Q * step)
        {
            float4 v[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q)
            {
                const size_t e = base + first + q * step;
                v[q] = e < n4 ? f4[e] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int q = 0; q < Q; ++q)
            {
                const bool on = base + first + q * step < n4;
                take(v[q].x, on);
                take(v[q].y, on);
                take(v[q].z, on);
                take(v[q].w, on);
            }
        }
    }
    else
    {
        constexpr int Q = PCT_SCALAR;
        const size_t step = static_cast<size_t>(gridDim.x) * EW_THREADS;
        for (size_t base = blockIdx.x * static_cast<size_t>(EW_THREADS); base < n; base += Q * step)
        {
            float v[Q];
            bool on[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q)
            {
                const size_t e = base + threadIdx.x + q * step;
                on[q] = e < n;
                const size_t a = pct_pixel(e, W, H, pitch, r2, use_reticle, on[q]);
                v[q] = on[q] ? f[a] : 0.f;
            }
#pragma unroll
            for (int q = 0; q < Q; ++q)
                take(v[q], on[q]);
        }
    }
    __syncthreads();
    for (int h = 0; h < nh; ++h)
        for (int i = threadIdx.x; i < PCT_BINS; i += EW_THREADS)
            if (sh[h][i])
                atomicAdd(&hist[h * PCT_BINS + i], sh[h][i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        s_last = atomicAdd(&st->done[d], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    pct_select(hist, st, 0, d, lower, range);
    pct_select(hist + (d == 0 ? 0 : PCT_BINS), st, 1, d, upper, range);
}

size_t percentile_workspace(size_t n)
{
    (void)n;
    return 2 * PCT_BINS * sizeof(unsigned int) * 3 + sizeof(PctState) + 256;
}

hv_status percentile(const float* frame, int W, int H, float lower, float upper, float reticle_scale, float* range,
                     void* work, cudaStream_t st, const CycleCtl* ctl)
{
    return percentile_pitched(frame, W, H, W, lower, upper, reticle_scale, range, work, st, ctl);
}

// The W x H sub-image of rows `pitch` floats apart (the YZ cut's columns between the offsets,
// compute_percentile_yz_view's cudaMemcpy2DAsync, percentile.cu:230-250).
hv_status percentile_pitched(const float* frame, int W, int H, int pitch, float lower, float upper,
                             float reticle_scale, float* range, void* work, cudaStream_t st, const CycleCtl* ctl)
{
    const size_t n = static_cast<size_t>(W) * H;
    if (n == 0 || pitch < W)
        return HV_INVALID_VALUE;
    unsigned int* hist = static_cast<unsigned int*>(work);  // 3 passes x 2 ranks x PCT_BINS
    PctState* state = reinterpret_cast<PctState*>(hist + 3 * 2 * PCT_BINS);
    static_assert(sizeof(PctState) <= sizeof(unsigned int) * 8, "the state fits behind the histograms");
    HV_LAUNCH_ZERO(hist, 3 * 2 * PCT_BINS * sizeof(unsigned int) + sizeof(PctState), st);
    int use_reticle = 0;
    unsigned int r2 = 0;
    if (reticle_scale > 0.f)
    {
        // radius = (uint)(scale * min(W, H) / 2) (percentile.cu:113, 163)
        const unsigned int radius = static_cast<unsigned int>(reticle_scale * static_cast<float>(W < H ? W : H) / 2.0f);
        if (radius > 0)
        {
            use_reticle = 1;
            r2 = radius * radius;
        }
    }
    const bool vec = pitch == W && !use_reticle;
    // 16 pixels per thread (VEC) or PCT_SCALAR, up to four CTAs per SM: with two, large frames wait for the votes and
    // shared-memory atomics of a few warps (4096 x 3000: 98.8 -> 88.8 us, with a reticle 180.7 -> 131.3), with six or eight
    // the histograms of the CTAs cost more than they bring (98.6 to 109.9 us)
    const size_t per = static_cast<size_t>(vec ? 16 : PCT_SCALAR) * EW_THREADS, cap = 152 * 4;
    const size_t want = (n + per - 1) / per;
    const int grid = static_cast<int>(want < cap ? want : cap);
    auto kern = !vec ? k_pct_pass<false, false> : vec4_ok(n, {frame}) ? k_pct_pass<true, false> : k_pct_pass<true, true>;
    for (int d = 0; d < 3; ++d)
        HV_LAUNCH(kern, grid, EW_THREADS, 0, st, frame, W, H, pitch, r2, use_reticle, state, d, hist + d * 2 * PCT_BINS, lower,
                  upper, range, ctl);
    count_launch(3);
    return HV_OK;
}

// ====================================================================================== contrast + ushort

__device__ __forceinline__ uint16_t to_ushort(float x)
{
    if (x <= 0.0f)
        return 0;
    const unsigned int u = static_cast<unsigned int>(x);
    if (u > 65535u)
        return 65535;
    return static_cast<uint16_t>(u);
}

template <int V>
__global__ void k_contrast_ushort(const float* __restrict__ in, const float* __restrict__ range, int invert, int apply,
                                  uint16_t* __restrict__ out, size_t n, const CycleCtl* ctl)
{
    wait_prior_kernels();
    if (!ctl_render(ctl))
        return;
    if (ctl)
        out += static_cast<size_t>(ctl->out_slot) * n;
    float mn = 0.f, factor = 1.f;
    if (apply)
    {
        float lo = range[0], hi = range[1];
        if (invert)
        {
            const float t = lo;
            lo = hi;
            hi = t;
        }
        mn = lo;
        factor = __fdiv_rn(65535.0f, __fadd_rn(__fsub_rn(hi, lo), FLT_EPSILON));
    }
    for (size_t e = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) * V; e < n;
         e += static_cast<size_t>(gridDim.x) * blockDim.x * V)
    {
        float v[V];
        load_v<V>(in + e, v);
        uint16_t u[V];
#pragma unroll
        for (int k = 0; k < V; ++k)
            u[k] = to_ushort(apply ? __fmul_rn(factor, __fsub_rn(v[k], mn)) : v[k]);
        if constexpr (V == 4)
            *reinterpret_cast<ushort4*>(out + e) = make_ushort4(u[0], u[1], u[2], u[3]);
        else
            out[e] = u[0];
    }
}

// ====================================================================================== filter2D view

// The filter2D view frame (Pipe::insert_filter2d_view, pipe.cc:526-546): the stored spectrum
// (spectrum x multiplier, FFT layout: apply_mask by the mask or by the masked transfer function)
// quadrant-swapped (shift_corners) and taken to its modulus (complex_to_modulus with one bin).
__global__ void k_f2d_view(const float2* __restrict__ spec, const float2* __restrict__ mult, int W, int H,
                           float* __restrict__ out)
{
    wait_prior_kernels();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= W)
        return;
    const size_t src = static_cast<size_t>((y + H / 2) % H) * W + (x + W / 2) % W;
    const float2 a = spec[src], m = mult[src];
    const float re = a.x * m.x - a.y * m.y, im = a.x * m.y + a.y * m.x;
    out[static_cast<size_t>(y) * W + x] = hypotf(re, im);
}

hv_status filter2d_view_frame(const float2* spec, const float2* mult, int W, int H, float* out, cudaStream_t st)
{
    if ((W & 1) || (H & 1))
        return HV_INVALID_VALUE;
    dim3 block(128), grid((W + 127) / 128, H);
    HV_LAUNCH(k_f2d_view, grid, block, 0, st, spec, mult, W, H, out);
    count_launch();
    return HV_OK;
}

// Contrast (apply_contrast_correction when `apply`) then float_to_ushort_normalized
// (tools_conversion.cu:389-393): trunc(x * 65535) saturated to [0, 65535] (NaN -> 0), the
// filter2D view's conversion.
__global__ void k_contrast_ushort_normalized(const float* __restrict__ in, const float* __restrict__ range, int invert,
                                             int apply, uint16_t* __restrict__ out, size_t n)
{
    wait_prior_kernels();
    float mn = 0.f, factor = 1.f;
    if (apply)
    {
        float lo = range[0], hi = range[1];
        if (invert)
        {
            const float t = lo;
            lo = hi;
            hi = t;
        }
        mn = lo;
        factor = __fdiv_rn(65535.0f, __fadd_rn(__fsub_rn(hi, lo), FLT_EPSILON));
    }
    for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < n;
         e += static_cast<size_t>(gridDim.x) * blockDim.x)
    {
        float v = in[e];
        if (apply)
            v = __fmul_rn(factor, __fsub_rn(v, mn));
        const float w = __fmul_rn(v, 65535.0f);
        out[e] = w >= 65535.0f ? static_cast<uint16_t>(65535) : (w > 0.0f ? static_cast<uint16_t>(w) : static_cast<uint16_t>(0));
    }
}

hv_status contrast_to_ushort_normalized(const float* frame, const float* range, int invert, int apply, uint16_t* out,
                                        size_t n, cudaStream_t st)
{
    HV_LAUNCH(k_contrast_ushort_normalized, ew_grid(n), EW_THREADS, 0, st, frame, range, invert, apply, out, n);
    count_launch();
    return HV_OK;
}

hv_status contrast_to_ushort(const float* frame, const float* range, int invert, int apply, uint16_t* out, size_t n,
                             cudaStream_t st, const CycleCtl* ctl)
{
    // (an output slot is n pixels of 2 bytes: a multiple of 8 bytes when n is one of 4)
    if (vec4_ok(n, {frame}) && (reinterpret_cast<uintptr_t>(out) & 7) == 0)
        HV_LAUNCH(k_contrast_ushort<4>, ew_grid(n / 4), EW_THREADS, 0, st, frame, range, invert, apply, out, n, ctl);
    else
        HV_LAUNCH(k_contrast_ushort<1>, ew_grid(n), EW_THREADS, 0, st, frame, range, invert, apply, out, n, ctl);
    count_launch();
    return HV_OK;
}

}  // namespace hv
