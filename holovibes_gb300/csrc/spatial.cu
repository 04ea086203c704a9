// Spatial stage: lenses, fused convert + 2-D FFT passes, Fresnel / angular-spectrum propagation.
//
// Reference behaviour (Holovibes):
//   convert        Backend/cuda_sources/tools_conversion.cu:107-171
//   Fresnel lens   Backend/cuda_sources/masks.cu:7-29, fresnel_transform.cu:14-63
//   AS lens        Backend/cuda_sources/masks.cu:31-59, angular_spectrum.cu:14-31, fourier_transform.cc:121-137
//   Fresnel        Backend/cuda_sources/fresnel_transform.cu:65-83   (x*L then forward FFT2, no 1/N)
//   angular spec.  Backend/cuda_sources/angular_spectrum.cu:33-63     (FFT2, *G, inverse FFT2, /(H*W))
//   ring enqueue   Backend/sources/data_struct/queue.cc:332-380
//   filter2D       Backend/cuda_sources/filter2D.cu:28-115, fourier_transform.cc:30-72,121-137
//                  (circular band-pass mask, shifted to FFT layout; x <- IFFT2(FFT2(x) M)
//                  unnormalised before Fresnel / no propagation, folded into G for AS)
//
// GB300 design: no cuFFT. A batch of B frames goes through two or three shared-memory passes:
//   row pass   : raw u8/u16/f32 -> complex (+ Fresnel lens) -> forward row FFT
//   column pass: forward column FFT (+ transfer function G, inverse column FFT for AS)
//   row pass   : inverse row FFT * 1/(H*W) (AS only)
// and the last pass writes straight into the time-ring slots, so the reference's separate
// mask, divide and ring-copy passes disappear. Passes of 512, 768 and 1024 points use the warp
// engine (fft_warp.cuh: 32 samples per thread, one transpose; the passes are persistent and
// fed by bulk copies), every other length the shared-memory Stockham tile engine
// (fft_smem.cuh).
#include <math.h>

#include <atomic>
#include <mutex>
#include <type_traits>
#include <vector>

#include "fft_smem.cuh"
#include "fft_warp.cuh"
#include "tc_common.cuh"
#include "hv_internal.h"

namespace hv {

// ====================================================================================== lenses

__global__ void k_fresnel_lens(float2* out, int W, int H, double lam, double z, double pixel_size_um, int mode)
{
    wait_prior_kernels();
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W || y >= H)
        return;
    const int S = W > H ? W : H;
    // centre crop of the S x S lens (fresnel_transform.cu:37-62)
    const int si = (H > W) ? x + (S - W) / 2 : x;
    const int sj = (W > H) ? y + (S - H) / 2 : y;
    float2 v;
    if (mode == HV_LENS_REF32)
    {
        const float lam32 = static_cast<float>(lam), z32 = static_cast<float>(z);
        const float c = static_cast<float>(M_PI / static_cast<double>(__fmul_rn(lam32, z32)));
        const float dx = __fmul_rn(static_cast<float>(pixel_size_um), 1.0e-6f);
        const float xf = __fmul_rn(__fsub_rn(static_cast<float>(si), static_cast<float>(S >> 1)), dx);
        const float yf = __fmul_rn(__fsub_rn(static_cast<float>(sj), static_cast<float>(S >> 1)), dx);
        // x * x + y * y contracted into one fused multiply-add, as the reference's build compiles it
        const float cs = __fmul_rn(c, __fmaf_rn(xf, xf, __fmul_rn(yf, yf)));
        v = make_float2(cosf(cs), sinf(cs));
    }
    else
    {
        const double dx = pixel_size_um * 1e-6;
        const double xd = (si - (S >> 1)) * dx;
        const double yd = (sj - (S >> 1)) * dx;
        double ph = M_PI / (lam * z) * (xd * xd + yd * yd);
        ph = fmod(ph, 2.0 * M_PI);
        double s, c;
        sincos(ph, &s, &c);
        v = make_float2(static_cast<float>(c), static_cast<float>(s));
    }
    out[static_cast<size_t>(y) * W + x] = v;
}

__global__ void k_spectral_lens(float2* out, int W, int H, double lam, double z, double pixel_size_um, int mode)
{
    wait_prior_kernels();
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= W || y >= H)
        return;
    float2 v;
    if (mode == HV_LENS_REF32)
    {
        const float lam32 = static_cast<float>(lam), z32 = static_cast<float>(z);
        const float step = __fmul_rn(static_cast<float>(pixel_size_um), 1e-6f);
        const float u_step = __fdiv_rn(1.0f, __fmul_rn(static_cast<float>(W), step));
        const float v_step = __fdiv_rn(1.0f, __fmul_rn(static_cast<float>(H), step));
        const float u = __fmul_rn(static_cast<float>(x - (W >> 1)), u_step);
        const float vv = __fmul_rn(static_cast<float>(y - (H >> 1)), v_step);
        // the reference's build contracts u * u + v * v and 1 - (lam^2 * s) into fused multiply-adds
        // (matched bit for bit against its lens on the benchmark sizes)
        const float s2 = __fmaf_rn(u, u, __fmul_rn(vv, vv));
        float tmp = __fmaf_rn(-__fmul_rn(lam32, lam32), s2, 1.0f);
        if (tmp < 0.0f)
            tmp = 0.0f;
        const double ph_d = __dmul_rn(__ddiv_rn(__dmul_rn(2.0 * M_PI, static_cast<double>(z32)), static_cast<double>(lam32)),
                                      static_cast<double>(__fsqrt_rn(tmp)));
        const float ph = static_cast<float>(ph_d);
        v = make_float2(cosf(ph), sinf(ph));
    }
    else
    {
        const double step = pixel_size_um * 1e-6;
        const double u = (x - (W >> 1)) / (W * step);
        const double vv = (y - (H >> 1)) / (H * step);
        double tmp = 1.0 - lam * lam * (u * u + vv * vv);
        if (tmp < 0.0)
            tmp = 0.0;
        double ph = 2.0 * M_PI * z / lam * sqrt(tmp);
        ph = fmod(ph, 2.0 * M_PI);
        double s, c;
        sincos(ph, &s, &c);
        v = make_float2(static_cast<float>(c), static_cast<float>(s));
    }
    // quadrant swap into FFT layout (shift_corners on the lens, fourier_transform.cc:134)
    const int xs = (x + W / 2) % W;
    const int ys = (y + H / 2) % H;
    out[static_cast<size_t>(ys) * W + xs] = v;
}

// ====================================================================================== FFT passes

struct RowPass
{
    const void* in;        // batch of frames, row-major rows x N
    int in_kind;           // InKind
    size_t in_frame;       // elements between input frames
    float2* out;
    FrameMap out_map;      // output frame slots
    const float2* premul;  // rows x N multiplier applied before the transform (or null)
    int rows;              // rows per frame
    int inverse;           // 1: conj in / conj out (unnormalised inverse)
    float scale;
    const float2* tw;      // per-stage twiddle tables of the N-point plan (device)
    int tw_count;
    int stream_out;        // 1: output written with an evict-first hint (ring slots)
    const CycleCtl* ctl = nullptr;  // served cycle: gate (active) and, with raw_from_ctl, the input offset
    int raw_from_ctl = 0;           // 1: `in` is the input ring base, the batch is at ctl->raw_offset
    int reserve_sms = 0;            // persistent passes leave this many SMs to kernels of other streams
};

// Copies the plan's twiddle tables next to the tile in shared memory (read conflict-free:
// consecutive threads read consecutive entries in row tiles, one broadcast entry in column tiles).
__device__ __forceinline__ const float2* stage_twiddles(float2* dst, const float2* __restrict__ src, int count,
                                                        int nthreads)
{
    for (int e = threadIdx.x; e < count; e += nthreads)
        dst[e] = __ldg(src + e);
    __syncthreads();
    return dst;
}

template <int N, int F>
__global__ void __launch_bounds__(fft::Tile<N, F, false>::NT) k_fft_rows(RowPass p)
{
    wait_prior_kernels();
    using Tl = fft::Tile<N, F, false>;
    extern __shared__ float2 smem[];
    if (!ctl_active(p.ctl))
        return;
    const void* p_in = p.raw_from_ctl ? static_cast<const void*>(static_cast<const uint8_t*>(p.in) + p.ctl->raw_offset)
                                      : p.in;
    float2* sm = smem;
    const float2* tw = stage_twiddles(smem + F * N, p.tw, p.tw_count, Tl::NT);

    const int b = blockIdx.y;
    const int row0 = blockIdx.x * F;
    const size_t in_base = static_cast<size_t>(b) * p.in_frame;
    const int rows = p.rows;
    const bool inv = p.inverse != 0;
    constexpr int E = Tl::E, R0 = Tl::R0, Q0 = E / R0, M0 = N / R0;

    // First-stage inputs: every load of the thread is issued before any is used (the input kind
    // and the lens multiply are uniform branches outside the element loops).
    float2 x[E];
    size_t rb[Q0];  // element (q, j) sits at rb[q] + j * M0
    bool ok[Q0];
#pragma unroll
    for (int q = 0; q < Q0; ++q)
    {
        int f, i;
        Tl::template index<R0>(static_cast<int>(threadIdx.x) + q * Tl::NT, f, i);
        const int y = row0 + f;
        ok[q] = y < rows;
        rb[q] = static_cast<size_t>(ok[q] ? y : 0) * N + i;
    }
#define HV_EIDX(e) (rb[(e) / R0] + ((e) % R0) * M0)
    switch (p.in_kind)
    {
    case IN_U8:
    {
        const uint8_t* in = static_cast<const uint8_t*>(p_in) + in_base;
        uint8_t v[E];
#pragma unroll
        for (int e = 0; e < E; ++e)
            v[e] = __ldcs(in + HV_EIDX(e));
#pragma unroll
        for (int e = 0; e < E; ++e)
            x[e] = make_float2(static_cast<float>(v[e]) * 257.0f, 0.f);
        break;
    }
    case IN_U16:
    case IN_U16_BE:
    {
        const uint16_t* in = static_cast<const uint16_t*>(p_in) + in_base;
        uint16_t v[E];
#pragma unroll
        for (int e = 0; e < E; ++e)
            v[e] = __ldcs(in + HV_EIDX(e));
        const bool swap = p.in_kind == IN_U16_BE;
#pragma unroll
        for (int e = 0; e < E; ++e)
        {
            const uint16_t u = swap ? static_cast<uint16_t>((v[e] << 8) | (v[e] >> 8)) : v[e];
            x[e] = make_float2(static_cast<float>(u), 0.f);
        }
        break;
    }
    case IN_F32:
    {
        const float* in = static_cast<const float*>(p_in) + in_base;
#pragma unroll
        for (int e = 0; e < E; ++e)
            x[e] = make_float2(__ldcs(in + HV_EIDX(e)), 0.f);
        break;
    }
    default:
    {
        const float2* in = static_cast<const float2*>(p_in) + in_base;
#pragma unroll
        for (int e = 0; e < E; ++e)
            x[e] = __ldg(in + HV_EIDX(e));
        break;
    }
    }
    if (p.premul)
    {
        float2 L[E];
#pragma unroll
        for (int e = 0; e < E; ++e)
            L[e] = __ldg(p.premul + HV_EIDX(e));
#pragma unroll
        for (int e = 0; e < E; ++e)
            x[e] = cmul(x[e], L[e]);
    }
#undef HV_EIDX
#pragma unroll
    for (int q = 0; q < Q0; ++q)
#pragma unroll
        for (int j = 0; j < R0; ++j)
        {
            float2& v = x[q * R0 + j];
            if (!ok[q])
                v = make_float2(0.f, 0.f);
            else if (inv)
                v = cconj(v);
        }

    float2* out = p.out + p.out_map.offset(b);
    const float sc = p.scale;
    const bool stream_out = p.stream_out != 0;
    auto dst = [&](int f, int n, float2 v) {
        const int y = row0 + f;
        if (y >= rows)
            return;
        if (inv)
            v = cconj(v);
        float2* o = out + static_cast<size_t>(y) * N + n;
        if (stream_out)
            __stcs(o, cscale(v, sc));
        else
            *o = cscale(v, sc);
    };
    Tl::run_regs(x, sm, tw, dst);
}

struct ColPass
{
    const float2* in;
    size_t in_frame;
    float2* out;
    FrameMap out_map;
    const float2* postmul;  // rows x width multiplier applied between forward and inverse (AS), or null
    int width;              // row length (number of columns)
    int mode;               // 0 forward, 1 inverse, 2 forward * postmul then inverse
    float scale;
    const float2* tw;       // per-stage twiddle tables of the N-point plan (device)
    int tw_count;
    int stream_out;         // 1: output written with an evict-first hint (ring slots)
    const CycleCtl* ctl = nullptr;  // served cycle: gate (active)
    int reserve_sms = 0;            // persistent passes leave this many SMs to kernels of other streams
};

template <int N, int F>
__global__ void __launch_bounds__(fft::Tile<N, F, true>::NT) k_fft_cols(ColPass p)
{
    wait_prior_kernels();
    using Tl = fft::Tile<N, F, true>;
    extern __shared__ float2 smem[];
    if (!ctl_active(p.ctl))
        return;
    float2* sm = smem;
    const float2* tw = stage_twiddles(smem + F * N, p.tw, p.tw_count, Tl::NT);

    const int b = blockIdx.y;
    const int c0 = blockIdx.x * F;
    const int W = p.width;
    const float2* in = p.in + static_cast<size_t>(b) * p.in_frame;
    float2* out = p.out + p.out_map.offset(b);
    const float sc = p.scale;
    if (p.mode == 2)
    {
        auto src = [&](int f, int n) -> float2 {
            const int c = c0 + f;
            return (c < W) ? in[static_cast<size_t>(n) * W + c] : make_float2(0.f, 0.f);
        };
        const float2* G = p.postmul;
        // forward result * G, conjugated for the inverse transform, parked in shared memory
        auto mid = [&](int f, int n, float2 v) {
            const int c = c0 + f;
            const float2 g = (c < W) ? __ldg(G + static_cast<size_t>(n) * W + c) : make_float2(0.f, 0.f);
            sm[Tl::addr(f, n)] = cconj(cmul(v, g));
        };
        Tl::run(sm, tw, src, mid);
        __syncthreads();
        auto src2 = [&](int f, int n) -> float2 { return sm[Tl::addr(f, n)]; };
        auto dst2 = [&](int f, int n, float2 v) {
            const int c = c0 + f;
            if (c < W)
                out[static_cast<size_t>(n) * W + c] = cscale(cconj(v), sc);
        };
        Tl::run(sm, tw, src2, dst2);
    }
    else
    {
        const bool inv = p.mode == 1;
        auto src = [&](int f, int n) -> float2 {
            const int c = c0 + f;
            if (c >= W)
                return make_float2(0.f, 0.f);
            const float2 v = in[static_cast<size_t>(n) * W + c];
            return inv ? cconj(v) : v;
        };
        const bool stream_out = p.stream_out != 0;
        auto dst = [&](int f, int n, float2 v) {
            const int c = c0 + f;
            if (c >= W)
                return;
            if (inv)
                v = cconj(v);
            float2* o = out + static_cast<size_t>(n) * W + c;
            if (stream_out)
                __stcs(o, cscale(v, sc));
            else
                *o = cscale(v, sc);
        };
        Tl::run(sm, tw, src, dst);
    }
}

// ------------------------------------------------------------------ warp engine (N = 512, 768, 1024)
// Persistent passes of two 256-thread CTAs per SM, fed by bulk copies into the buffer that the
// transpose has just left: a row warp (or a column CTA) asks for its next tile as soon as the
// transposed samples are in registers, so the copy runs beside the second half of the transform
// and the stores. The waits are bounded; one that gives up sets g_fft_wait_error, lets the copy
// already issued land and ends the warp (or the CTA).
//
// Rows: 32 / NG rows per warp (2 for N = 512), lane (r, g) = (lane / NG, lane % NG); the transpose
// in the warp's own [row][n2][k1] block, k1 rows padded by one entry (conflict-free both ways), no
// CTA barrier inside the loop. N = 768 runs DFT24 first: 32 lanes load 24 samples each, lanes
// 0..23 run the DFT32 and store.
// Columns: 256 / NG adjacent columns per CTA (8, or 16 for N = 512), thread (c, g) = (t % C, t / C)
// holds samples g + NG i of column c; the transpose goes through a [k1][n2][c] block
// (conflict-free: k1 rows padded to 264 entries when C = 8).
//
// What bounds them: issue slots and latency at 16 warps per SM (64 data registers per thread), and
// DRAM for large batches of complex input. Measured (us; one CTA per row block or column tile,
// its own loads and scalar arithmetic -> here): rows of 16-bit frames, 64 x 768 x 768 102.7 -> 74.4,
// 32 x 1024 x 1024 78.1 -> 63.1, times a lens 89.2 -> 71.1; columns forward, 768 141.7 -> 103.8, 1024
// 93.1 -> 89.0 (0.89 of the measured copy bandwidth); columns * G inverse, 768 207.6 -> 168.2, 1024
// 169.3 -> 138.1. The kernels are specialised on the input encoding and the multiplier, or on the
// column mode: run-time branches on them spilled and cost a quarter of the instructions (rows of
// 64 x 768 x 768: 69.8 M against 52.4 M with the packed arithmetic).
__device__ int g_fft_wait_error = 0;

constexpr int W32_WARPS = 8;
constexpr int W32_THREADS = 256;

template <int N>
struct W32Geom
{
    static constexpr int NG = N == 768 ? 32 : N / 32;   // threads per transform
    static constexpr int NS = N / NG;                   // samples a thread loads (32; 24 for 768)
    static constexpr int K1 = N == 768 ? 24 : NG;       // stage-A outputs per n2
    static constexpr int RPW = 32 / NG;                 // rows per warp
    static constexpr int ROW_PAD = K1 + 1;
    static constexpr int ROW_BUF = RPW * 32 * ROW_PAD;  // float2 per warp; holds RPW rows of input too
    static constexpr int COLS = W32_THREADS / NG;       // columns per CTA
    static constexpr int COL_PAD = 32 * COLS + (COLS == 8 ? 8 : 0);
    static constexpr int COL_BUF = (N == 768 ? 32 : NG) * COL_PAD;  // float2 per CTA; holds a tile too
    static constexpr int tw_count()
    {
        if constexpr (N == 768)
            return fftw::W768::TW_COUNT;
        else
            return fftw::Warp<N>::TW_COUNT;
    }
    static constexpr int TW = tw_count();
    static_assert(ROW_BUF >= RPW * N && COL_BUF >= COLS * N, "the transpose buffers hold the input tiles");
    static_assert(TW % 2 == 0 && ROW_BUF % 2 == 0 && COL_BUF % 2 == 0, "16-byte aligned buffers");
    // the column tile sits on a 128-byte boundary (tensor copies)
    static constexpr size_t ROW_SMEM =
        (TW + static_cast<size_t>(W32_WARPS) * ROW_BUF) * sizeof(float2) + W32_WARPS * sizeof(uint64_t);
    static constexpr size_t COL_SMEM =
        128 + (TW + static_cast<size_t>(COL_BUF)) * sizeof(float2) + 2 * sizeof(uint64_t);
};

// Converted sample j of a row in shared memory at `row` + STRIDE j.
template <int KIND>
__device__ __forceinline__ float2 staged_sample(const void* row, int at, bool swap)
{
    if constexpr (KIND == IN_U8)
        return make_float2(static_cast<float>(static_cast<const uint8_t*>(row)[at]) * 257.0f, 0.f);
    else if constexpr (KIND == IN_U16)
    {
        uint16_t u = static_cast<const uint16_t*>(row)[at];
        if (swap)
            u = static_cast<uint16_t>((u << 8) | (u >> 8));
        return make_float2(static_cast<float>(u), 0.f);
    }
    else if constexpr (KIND == IN_F32)
        return make_float2(static_cast<const float*>(row)[at], 0.f);
    else
        return static_cast<const float2*>(row)[at];
}

// Row pass: units of RPW rows, `per_frame` per frame; with a premultiplier the frames of one row
// block are adjacent (the multiplier rows stay in L1), else the rows of one frame. KIND: the input
// encoding (IN_U16 for both byte orders). The input rows of the next unit land in the warp's
// transpose block by one bulk copy; without `bulk` (input off 16-byte alignment, engine mode 2)
// the lanes copy them there, several loads at a time (one after another: 32 x 1024 x 1024 8-bit rows 161 us, so 78,
// 8-bit Fresnel windows of 1024 x 1024, T = 32, off alignment 351 and 270 us). Loading them into registers instead
// is faster still without bulk copies (58 us), but made the passes with them 1 to 2 % slower, as a branch and as
// kernels of their own.
template <int N, int KIND, bool PREMUL>
__global__ void __launch_bounds__(W32_THREADS, 2) k_fft_rows_warp(RowPass p, int per_frame, int nframes, int bulk)
{
    wait_prior_kernels();
    using Gm = W32Geom<N>;
    constexpr int NG = Gm::NG, NS = Gm::NS;
    constexpr int ESIZE = KIND == IN_U8 ? 1 : KIND == IN_U16 ? 2 : KIND == IN_F32 ? 4 : 8;
    extern __shared__ __align__(16) float2 smem[];
    if (!ctl_active(p.ctl))
        return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float2* buf = smem + Gm::TW + warp * Gm::ROW_BUF;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + Gm::TW + W32_WARPS * Gm::ROW_BUF) + warp;
    const uint8_t* p_in = static_cast<const uint8_t*>(p.in) + (p.raw_from_ctl ? p.ctl->raw_offset : 0);
    const int units = per_frame * nframes;
    const bool inv = p.inverse != 0, swap = p.in_kind == IN_U16_BE;
    // unit u: rows y0 .. of frame f
    auto locate = [&](int u, int& f, int& y0) {
        if (PREMUL)
        {
            const int rb = u / nframes;
            f = u - rb * nframes;
            y0 = rb * Gm::RPW;
        }
        else
        {
            f = u / per_frame;
            y0 = (u - f * per_frame) * Gm::RPW;
        }
    };
    auto source = [&](int f, int y0) {
        return p_in + (static_cast<size_t>(f) * p.in_frame + static_cast<size_t>(y0) * N) * ESIZE;
    };
    auto issue = [&](int u) {
        int f, y0;
        locate(u, f, y0);
        const uint32_t bytes = static_cast<uint32_t>(min(Gm::RPW, p.rows - y0)) * N * ESIZE;
        tc::mbar_arrive_expect_tx(bar, bytes);
        tc::bulk_g2s(buf, source(f, y0), bytes, bar);
    };
    const int u0 = blockIdx.x * W32_WARPS + warp, du = gridDim.x * W32_WARPS;
    if (lane == 0)
    {
        tc::mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tc::fence_async_smem();
        if (bulk && u0 < units)
            issue(u0);
    }
    const float2* tw = stage_twiddles(smem, p.tw, Gm::TW, W32_THREADS);  // ends with a CTA barrier

    const int r = lane / NG, g = lane % NG;
    const float2 scale = make_float2(p.scale, inv ? -p.scale : p.scale);
    uint32_t phase = 0;
    for (int u = u0; u < units; u += du)
    {
        int f, y0;
        locate(u, f, y0);
        const int y = y0 + r;
        // lanes of a row past the frame's last row compute on other rows' samples and store nothing
        const bool row_ok = y < p.rows;
        float2 x[32];
        if constexpr (PREMUL)
        {
            const float2* L = p.premul + static_cast<size_t>(row_ok ? y : y0) * N + g;
#pragma unroll
            for (int j = 0; j < NS; ++j)
                x[j] = __ldg(L + NG * j);
        }
        if (bulk)
        {
            const bool landed = tc::mbar_wait(bar, phase);
            if (!__all_sync(0xffffffffu, landed))
            {
                tc::mbar_wait(bar, phase);  // the copy lands before the shared memory is released
                if (lane == 0)
                    atomicExch(&g_fft_wait_error, 1);
                return;
            }
            phase ^= 1;
        }
        else
        {
            using E = std::conditional_t<ESIZE == 1, uint8_t,
                                         std::conditional_t<ESIZE == 2, uint16_t, std::conditional_t<ESIZE == 4, float, float2>>>;
            // loads that a lane issues together; whole rows are a multiple of 32 D samples
            constexpr int D = N == 768 && KIND == IN_C64 ? 12 : 8;
            static_assert(N % (32 * D) == 0, "rows divide into batches");
            const E* src = reinterpret_cast<const E*>(source(f, y0)) + lane;
            E* dst = reinterpret_cast<E*>(buf) + lane;
            const int n = min(Gm::RPW, p.rows - y0) * N;
            for (int i = 0; i < n; i += 32 * D)
            {
                E v[D];
#pragma unroll
                for (int d = 0; d < D; ++d)
                    v[d] = src[i + 32 * d];
#pragma unroll
                for (int d = 0; d < D; ++d)
                    dst[i + 32 * d] = v[d];
            }
            __syncwarp();
        }
        {
            const int at = (row_ok ? r : 0) * N + g;
#pragma unroll
            for (int j = 0; j < NS; ++j)
            {
                const float2 v = staged_sample<KIND>(buf, at + NG * j, swap);
                if constexpr (PREMUL && KIND == IN_C64)
                    x[j] = cmul_fma(v, x[j]);
                else if constexpr (PREMUL)
                    x[j] = make_float2(v.x * x[j].x, v.x * x[j].y);
                else
                    x[j] = v;
            }
            if (inv)
            {
#pragma unroll
                for (int j = 0; j < NS; ++j)
                    x[j] = cconj(x[j]);
            }
        }
        __syncwarp();  // the block is rewritten by the transpose

        float2* tb = buf + r * 32 * Gm::ROW_PAD;
        if constexpr (N == 768)
        {
            fftw::W768::stage_a24(x, tw, lane);
#pragma unroll
            for (int k1 = 0; k1 < 24; ++k1)
                tb[lane * Gm::ROW_PAD + k1] = x[k1];
        }
        else
        {
            using Wp = fftw::Warp<N>;
            Wp::stage_a(x, tw, g);
            // transpose: z[n2][k1] at tb[n2 * ROW_PAD + k1]; thread g then reads z[n2][g] for every n2
#pragma unroll
            for (int e = 0; e < 32; ++e)
                tb[Wp::n2_of(e, g) * Gm::ROW_PAD + Wp::k1_of(e)] = x[e];
        }
        __syncwarp();
        const int k1 = g < Gm::K1 ? g : 0;
#pragma unroll
        for (int n2 = 0; n2 < 32; ++n2)
            x[n2] = tb[n2 * Gm::ROW_PAD + k1];
        tc::fence_async_smem();
        __syncwarp();  // the block is rewritten by the next unit's input
        if (bulk && lane == 0 && u + du < units)
            issue(u + du);
        fftw::dft32(x);

        if (!row_ok || g >= Gm::K1)
            continue;
        float2* o = p.out + p.out_map.offset(f) + static_cast<size_t>(y) * N + g;
        if (p.stream_out)
        {
#pragma unroll
            for (int k2 = 0; k2 < 32; ++k2)
                __stcs(o + Gm::K1 * k2, fft::pmul(x[k2], scale));
        }
        else
        {
#pragma unroll
            for (int k2 = 0; k2 < 32; ++k2)
                o[Gm::K1 * k2] = fft::pmul(x[k2], scale);
        }
    }
}

// Column pass. One tile = COLS adjacent columns of one frame; the CTA walks tiles blockIdx.x,
// + gridDim.x, ... MODE: 0 forward, 1 inverse, 2 forward * G then inverse (the AS middle pass).
// BULK: the tile (and, for MODE 2, the transfer function's tile) lands in the transpose block by tensor
// copies of 256 rows each; else (alignment, engine mode 2) the threads load their samples (32 x 1024 x 1024: forward
// 117 us, 336 through the block; with G 169 and 565).
// (The outputs of the forward and inverse modes are addressed from their base: with a running pointer, or with the
// base computed before the wait, the pass alone takes the same time or less, and the Fresnel + PCA windows of 1024 x 1024,
// where it runs beside three render lanes, 1 to 2 % more.)
template <int N, int MODE, bool BULK>
__global__ void __launch_bounds__(W32_THREADS, 2) k_fft_cols_warp(const __grid_constant__ CUtensorMap in_map,
                                                                  const __grid_constant__ CUtensorMap g_map, ColPass p,
                                                                  int tiles_x, int ntiles)
{
    wait_prior_kernels();
    using Gm = W32Geom<N>;
    constexpr int NG = Gm::NG, NS = Gm::NS, K1 = Gm::K1, C = Gm::COLS;
    extern __shared__ unsigned char smem_raw[];
    if (!ctl_active(p.ctl))
        return;
    float2* S = reinterpret_cast<float2*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    float2* tw = S + Gm::COL_BUF;
    uint64_t* bar = reinterpret_cast<uint64_t*>(tw + Gm::TW);
    __shared__ int s_abort;
    volatile int* abort = &s_abort;
    const int tid = threadIdx.x;
    // one tile of `map` (columns tx C .., rows fb N ..) into S
    auto issue = [&](const CUtensorMap* map, int fb, int tx) {
        tc::mbar_arrive_expect_tx(bar, C * N * sizeof(float2));
#pragma unroll
        for (int q = 0; q < N / 256; ++q)
            tc::tma_load_2d(S + q * 256 * C, map, tx * C * 2, fb * N + q * 256, bar);
    };
    if (tid == 0)
    {
        s_abort = 0;
        tc::mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tc::fence_async_smem();
        if (BULK && static_cast<int>(blockIdx.x) < ntiles)
            issue(&in_map, blockIdx.x / tiles_x, blockIdx.x % tiles_x);
    }
    stage_twiddles(tw, p.tw, Gm::TW, W32_THREADS);  // ends with a CTA barrier

    const int c = tid % C, g = tid / C;
    const size_t W = static_cast<size_t>(p.width);
    const float2 scale = make_float2(p.scale, MODE != 0 ? -p.scale : p.scale);
    const bool active_b = g < K1;  // N = 768: a quarter of the threads idle in one stage
    uint32_t phase = 0;
    // the tile asked for last is in S: every thread waits for the copies, and the CTA agrees on the
    // outcome so that all of it leaves together
    auto landed = [&]() -> bool {
        if constexpr (!BULK)
            return true;
        const bool ok = tc::mbar_wait(bar, phase, abort);
        phase ^= 1;
        return __syncthreads_and(ok);
    };
    // every thread has read what it needs from S: ask for the tile of the next use
    auto refill = [&](const CUtensorMap* map, int fb, int tx, bool any) {
        if constexpr (BULK)
            tc::fence_async_smem();
        __syncthreads();
        if (BULK && any && tid == 0)
            issue(map, fb, tx);
    };
    bool gave_up = false;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x)
    {
        const int fb = t / tiles_x, tx = t - fb * tiles_x;
        const int tn = t + static_cast<int>(gridDim.x);
        const bool in_range = tx * C + c < p.width;
        if (!landed())
        {
            gave_up = true;
            break;
        }
        float2 x[32];
        if constexpr (BULK)
        {
#pragma unroll
            for (int j = 0; j < NS; ++j)
                x[j] = S[(g + NG * j) * C + c];
            __syncthreads();
        }
        else
        {
            // (a column past the frame repeats the last one; it is not stored)
            const float2* src = p.in + static_cast<size_t>(fb) * p.in_frame + static_cast<size_t>(g) * W + min(tx * C + c, p.width - 1);
            const size_t step = static_cast<size_t>(NG) * W;
#pragma unroll
            for (int j = 0; j < NS; ++j, src += step)
                x[j] = *src;
        }
        if constexpr (MODE == 1)
        {
#pragma unroll
            for (int j = 0; j < NS; ++j)
                x[j] = cconj(x[j]);
        }
        // forward: stage A, transpose ([k1][n2][c]), stage B; element k2 of thread g < K1 is X[g + K1 k2]
        if constexpr (N == 768)
        {
            fftw::W768::stage_a24(x, tw, g);
#pragma unroll
            for (int k1 = 0; k1 < 24; ++k1)
                S[k1 * Gm::COL_PAD + g * C + c] = x[k1];
        }
        else
        {
            using Wp = fftw::Warp<N>;
            Wp::stage_a(x, tw, g);
#pragma unroll
            for (int e = 0; e < 32; ++e)
                S[Wp::k1_of(e) * Gm::COL_PAD + Wp::n2_of(e, g) * C + c] = x[e];
        }
        __syncthreads();
        if (active_b)
        {
#pragma unroll
            for (int n2 = 0; n2 < 32; ++n2)
                x[n2] = S[g * Gm::COL_PAD + n2 * C + c];
        }
        float2* o = p.out + p.out_map.offset(fb) + static_cast<size_t>(g) * W + (tx * C + c);
        if constexpr (MODE != 2)
        {
            refill(&in_map, tn / tiles_x, tn % tiles_x, tn < ntiles);
            if (!active_b)
                continue;
            fftw::dft32(x);
            if (!in_range)
                continue;
            const size_t step = static_cast<size_t>(K1) * W;
            if (p.stream_out)
            {
#pragma unroll
                for (int k2 = 0; k2 < 32; ++k2)
                    __stcs(o + k2 * step, fft::pmul(x[k2], scale));
            }
            else
            {
#pragma unroll
                for (int k2 = 0; k2 < 32; ++k2, o += step)
                    *o = fft::pmul(x[k2], scale);
            }
        }
        else
        {
            // * G, conjugate, inverse transform: stage B's output has stage A's input shape (for
            // N = 768 that of the DFT32-first order)
            refill(&g_map, 0, tx, true);
            if (active_b)
                fftw::dft32(x);
            if (!landed())
            {
                gave_up = true;
                break;
            }
            if (active_b)
            {
                const float2* gm = p.postmul + static_cast<size_t>(g) * W + min(tx * C + c, p.width - 1);
                const size_t step = static_cast<size_t>(K1) * W;
#pragma unroll
                for (int k2 = 0; k2 < 32; ++k2, gm += step)
                    x[k2] = cconj(cmul_fma(x[k2], BULK ? S[(g + K1 * k2) * C + c] : __ldg(gm)));
            }
            if constexpr (BULK)
                __syncthreads();
            if constexpr (N == 768)
            {
                if (active_b)
                {
                    fftw::W768::stage_a32(x, tw, g);
#pragma unroll
                    for (int k1 = 0; k1 < 32; ++k1)
                        S[k1 * Gm::COL_PAD + g * C + c] = x[k1];
                }
            }
            else
            {
                using Wp = fftw::Warp<N>;
                Wp::stage_a(x, tw, g);
#pragma unroll
                for (int e = 0; e < 32; ++e)
                    S[Wp::k1_of(e) * Gm::COL_PAD + Wp::n2_of(e, g) * C + c] = x[e];
            }
            __syncthreads();
#pragma unroll
            for (int n2 = 0; n2 < NS; ++n2)
                x[n2] = S[g * Gm::COL_PAD + n2 * C + c];
            refill(&in_map, tn / tiles_x, tn % tiles_x, tn < ntiles);
            if constexpr (N == 768)
                fftw::dft24(x);
            else
                fftw::dft32(x);
            if (!in_range)
                continue;
            const size_t step = static_cast<size_t>(NG) * W;
#pragma unroll
            for (int k2 = 0; k2 < NS; ++k2, o += step)
                *o = fft::pmul(x[k2], scale);
        }
    }
    if (BULK && gave_up && tid == 0)
    {
        // the copy still in flight lands before the CTA's shared memory is released
        tc::mbar_wait(bar, phase ^ 1);
        atomicExch(&g_fft_wait_error, 1);
    }
}

// Raw -> complex into ring slots (space transformation NONE), 8 pixels of one frame per thread
// (frames of a multiple of 8 pixels, 16-byte aligned rows of the raw batch); with `planes`, the
// real rows of the ring's split-BF16 planes of those slots as well (planes[p][slot][px]: the
// covariance operands of a ring with zero imaginary parts), so the frame is read once. Registers for six CTAs per
// SM: with the 32 that the compiler takes for eight the same pass is slower (64 16-bit frames of 512 x 512 49.4 -> 45.0 us, float
// 55.6 -> 50.9, 16 8-bit frames of 2048 x 2048 210.5 -> 200.5).
__global__ void __launch_bounds__(256, 6) k_convert8(const void* in, int kind, size_t frame_px, int batch, float2* ring, FrameMap map,
                           const CycleCtl* ctl, uint16_t* planes)
{
    wait_prior_kernels();
    if (!ctl_active(ctl))
        return;
    if (ctl)
        in = static_cast<const uint8_t*>(in) + ctl->raw_offset;
    const size_t groups = frame_px / 8;
    const size_t total = groups * batch;
    const size_t plane = static_cast<size_t>(map.nslots) * frame_px;
    for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < total;
         e += static_cast<size_t>(gridDim.x) * blockDim.x)
    {
        const int b = static_cast<int>(e / groups);
        const size_t px = (e - static_cast<size_t>(b) * groups) * 8;
        const size_t src = static_cast<size_t>(b) * frame_px + px;
        float v[8];
        if (kind == IN_U8)
        {
            const uint2 w = *reinterpret_cast<const uint2*>(static_cast<const uint8_t*>(in) + src);
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                v[i] = static_cast<float>((w.x >> (8 * i)) & 0xffu) * 257.0f;
                v[4 + i] = static_cast<float>((w.y >> (8 * i)) & 0xffu) * 257.0f;
            }
        }
        else if (kind == IN_U16 || kind == IN_U16_BE)
        {
            const uint4 w = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(in) + src);
            const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                uint32_t x = ww[i];
                if (kind == IN_U16_BE)
                    x = ((x & 0x00ff00ffu) << 8) | ((x >> 8) & 0x00ff00ffu);
                v[2 * i] = static_cast<float>(x & 0xffffu);
                v[2 * i + 1] = static_cast<float>(x >> 16);
            }
        }
        else
        {
            const float4* f = reinterpret_cast<const float4*>(static_cast<const float*>(in) + src);
            const float4 a = f[0], c = f[1];
            v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = c.x, v[5] = c.y, v[6] = c.z, v[7] = c.w;
        }
        const size_t off = map.offset(b);
        float4* o = reinterpret_cast<float4*>(ring + off + px);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            __stcs(o + i, make_float4(v[2 * i], 0.f, v[2 * i + 1], 0.f));
        if (planes)
        {
            uint4 hi, lo;
            tc::split2(v[0], v[1], hi.x, lo.x);
            tc::split2(v[2], v[3], hi.y, lo.y);
            tc::split2(v[4], v[5], hi.z, lo.z);
            tc::split2(v[6], v[7], hi.w, lo.w);
            const size_t slot_px = off / map.frame_stride * frame_px + px;
            *reinterpret_cast<uint4*>(planes + slot_px) = hi;
            *reinterpret_cast<uint4*>(planes + plane + slot_px) = lo;
        }
    }
}

// Raw 8/16-bit frames (no spatial transform) -> the real split planes of ring slots slot0 .. (mod T)
// and, as 16-bit integers, frames sample0 .. (mod cap) of the sample ring: what the pipelined PCA
// windows' covariance and views read. 8 pixels per thread; without VEC (a batch off 16-byte
// alignment) the pixels are loaded one by one. DRAM-bound: 64 16-bit frames of 512 x 512 (33.6 MB read,
// 100.7 MB written).
template <int KIND, bool VEC>
__global__ void k_convert_window(const void* __restrict__ in, int swap, size_t frame_px, int batch, int slot0, int T,
                                 uint16_t* __restrict__ planes, int sample0, int cap, uint16_t* __restrict__ samples)
{
    wait_prior_kernels();
    const size_t groups = frame_px / 8;
    const size_t total = groups * batch;
    const size_t plane = static_cast<size_t>(T) * frame_px;
    for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < total;
         e += static_cast<size_t>(gridDim.x) * blockDim.x)
    {
        const int b = static_cast<int>(e / groups);
        const size_t px = (e - static_cast<size_t>(b) * groups) * 8;
        const size_t src = static_cast<size_t>(b) * frame_px + px;
        uint32_t x[4];  // pixel pairs
        if constexpr (KIND == IN_U8)
        {
            const uint8_t* p = static_cast<const uint8_t*>(in) + src;
            uint32_t w[2];
            if constexpr (VEC)
            {
                const uint2 v = *reinterpret_cast<const uint2*>(p);
                w[0] = v.x, w[1] = v.y;
            }
            else
            {
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    w[i] = p[4 * i] | (p[4 * i + 1] << 8) | (p[4 * i + 2] << 16) | (static_cast<uint32_t>(p[4 * i + 3]) << 24);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                const uint32_t h = w[i / 2] >> (16 * (i % 2));
                x[i] = ((h & 0xffu) | ((h & 0xff00u) << 8)) * 257u;
            }
        }
        else
        {
            const uint16_t* p = static_cast<const uint16_t*>(in) + src;
            if constexpr (VEC)
            {
                const uint4 v = *reinterpret_cast<const uint4*>(p);
                x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
            }
            else
            {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    x[i] = p[2 * i] | (static_cast<uint32_t>(p[2 * i + 1]) << 16);
            }
            if (swap)
            {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    x[i] = ((x[i] & 0x00ff00ffu) << 8) | ((x[i] >> 8) & 0x00ff00ffu);
            }
        }
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            tc::split2(static_cast<float>(x[i] & 0xffffu), static_cast<float>(x[i] >> 16), hi[i], lo[i]);
        uint16_t* o = planes + static_cast<size_t>((slot0 + b) % T) * frame_px + px;
        *reinterpret_cast<uint4*>(o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(o + plane) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        *reinterpret_cast<uint4*>(samples + static_cast<size_t>((sample0 + b) % cap) * frame_px + px) =
            make_uint4(x[0], x[1], x[2], x[3]);
    }
}

// Ring slots slot0 .. slot0 + n - 1 (mod T) from their real split planes: x = hi + lo, exact for
// integer pixels below 2^16 (hi keeps the top 8 significant bits, lo the rest), imaginary part 0.
__global__ void k_ring_from_planes(const uint16_t* __restrict__ planes, int T, size_t frame_px, int slot0, int n,
                                   float2* __restrict__ ring)
{
    wait_prior_kernels();
    const size_t groups = frame_px / 8;
    const size_t total = groups * n;
    const size_t plane = static_cast<size_t>(T) * frame_px;
    for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < total;
         e += static_cast<size_t>(gridDim.x) * blockDim.x)
    {
        const int f = static_cast<int>(e / groups);
        const size_t px = (e - static_cast<size_t>(f) * groups) * 8;
        const size_t at = static_cast<size_t>((slot0 + f) % T) * frame_px + px;
        const uint4 hi = *reinterpret_cast<const uint4*>(planes + at);
        const uint4 lo = *reinterpret_cast<const uint4*>(planes + plane + at);
        const uint32_t h[4] = {hi.x, hi.y, hi.z, hi.w}, l[4] = {lo.x, lo.y, lo.z, lo.w};
        float4* o = reinterpret_cast<float4*>(ring + at);
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            // bf16 = the top half of an FP32 word
            const float a = __uint_as_float(h[i] << 16) + __uint_as_float(l[i] << 16);
            const float b = __uint_as_float(h[i] & 0xffff0000u) + __uint_as_float(l[i] & 0xffff0000u);
            __stcs(o + i, make_float4(a, 0.f, b, 0.f));
        }
    }
}

// Raw -> complex into ring slots (space transformation NONE).
__global__ void k_convert(const void* in, int kind, size_t frame_px, int batch, float2* ring, FrameMap map,
                          const CycleCtl* ctl)
{
    wait_prior_kernels();
    if (!ctl_active(ctl))
        return;
    if (ctl)
        in = static_cast<const uint8_t*>(in) + ctl->raw_offset;
    const size_t total = frame_px * batch;
    for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < total;
         e += static_cast<size_t>(gridDim.x) * blockDim.x)
    {
        const int b = static_cast<int>(e / frame_px);
        const size_t px = e - static_cast<size_t>(b) * frame_px;
        ring[map.offset(b) + px] = load_pixel(in, e, kind);
    }
}

// ====================================================================================== twiddles
// All plans' per-stage twiddle tables live in one static device array, filled from the host (FP64
// cos/sin rounded to FP32) by a synchronous copy the first time a size is used on a device: no
// device allocation, so the allocation-free entry points can use the FFT too. That first use on a
// device must not happen inside a stream capture.

#define HV_FFT_SIZES(X)                                                                                                \
    X(16) X(32) X(64) X(128) X(256) X(512) X(1024) X(2048) X(4096) X(48) X(96) X(192) X(384) X(768) X(1536)

constexpr int kTwiddleCapacity = 32768;
static __device__ float2 g_fft_twiddles[kTwiddleCapacity];

namespace {

constexpr int kMaxTwDevices = 64;
std::mutex g_tw_mu;
const float2* g_tw_base[kMaxTwDevices] = {};
int g_tw_offset[8192];  // offset of size N's tables in g_fft_twiddles
int g_tw_w32_offset[2] = {};  // offsets of the warp engine's tables (N = 512, 1024)
int g_tw_w768_offset = 0;    // offset of the warp engine's N = 768 tables
bool g_tw_layout_ready = false;
std::vector<float2> g_tw_host;

void tw_layout()
{
    if (g_tw_layout_ready)
        return;
    int off = 0;
#define HV_TW(N)                                                                                                       \
    {                                                                                                                  \
        g_tw_offset[N] = off;                                                                                          \
        const int cnt = fft::twiddle_count(typename fft::Plan<N>::List{});                                             \
        g_tw_host.resize(off + cnt + 1);                                                                               \
        fft::twiddle_fill(typename fft::Plan<N>::List{}, g_tw_host.data() + off);                                      \
        off += cnt;                                                                                                    \
    }
    HV_FFT_SIZES(HV_TW)
#undef HV_TW
    g_tw_w32_offset[1] = off;
    g_tw_host.resize(off + fftw::Warp<1024>::TW_COUNT + 1);
    fftw::Warp<1024>::twiddle_fill(g_tw_host.data() + off);
    off += fftw::Warp<1024>::TW_COUNT;
    g_tw_w32_offset[0] = off;
    g_tw_host.resize(off + fftw::Warp<512>::TW_COUNT + 1);
    fftw::Warp<512>::twiddle_fill(g_tw_host.data() + off);
    off += fftw::Warp<512>::TW_COUNT;
    g_tw_w768_offset = off;
    g_tw_host.resize(off + fftw::W768::TW_COUNT + 1);
    fftw::W768::twiddle_fill(g_tw_host.data() + off);
    off += fftw::W768::TW_COUNT;
    g_tw_layout_ready = true;
}

// Base of the twiddle array on the current device (uploaded on first use), or null.
const float2* twiddle_base()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxTwDevices)
        return nullptr;
    std::lock_guard<std::mutex> g(g_tw_mu);
    if (!g_tw_base[dev])
    {
        tw_layout();
        if (g_tw_host.size() > static_cast<size_t>(kTwiddleCapacity))
            return nullptr;
        if (cudaMemcpyToSymbol(g_fft_twiddles, g_tw_host.data(), g_tw_host.size() * sizeof(float2)) != cudaSuccess)
            return nullptr;
        void* base = nullptr;
        if (cudaGetSymbolAddress(&base, g_fft_twiddles) != cudaSuccess)
            return nullptr;
        g_tw_base[dev] = static_cast<const float2*>(base);
    }
    return g_tw_base[dev];
}

template <int N>
const float2* twiddles()
{
    const float2* base = twiddle_base();
    return base ? base + g_tw_offset[N] : nullptr;
}

// the warp engine's tables (N = 512, 768, 1024)
template <int N>
const float2* twiddles_warp()
{
    const float2* base = twiddle_base();
    return base ? base + (N == 768 ? g_tw_w768_offset : g_tw_w32_offset[N == 1024 ? 1 : 0]) : nullptr;
}

}  // namespace

// ====================================================================================== dispatch

namespace {

// Rows per CTA for the row pass (about 256 threads) and columns per CTA for the column pass.
template <int N>
constexpr int row_lanes()
{
    constexpr int per_row = N / fft::Plan<N>::E;
    return per_row >= 256 ? 1 : 256 / per_row;
}
template <int N>
constexpr int col_lanes()
{
    constexpr int E = fft::Plan<N>::E;
    // at most 512 threads and 128 KB of tile per CTA
    int f = 16;
    while (f > 1 && (f * N / E > 512 || f * N * 8 > 128 * 1024))
        f /= 2;
    return f;
}

std::atomic<int> g_fft_engine{0};  // 0 automatic (warp engine for 512-, 768- and 1024-point transforms), 1 tile engine only

std::atomic<int> g_fft_bulk{1};  // 1: the warp engine's passes are fed by bulk copies where they apply

int device_sms()
{
    static const int sms = [] {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return 0;
        return n;
    }();
    return sms;
}

constexpr size_t kL2Bytes = size_t(128) << 20;

// CTAs of a persistent pass: two per SM, less the SMs left to other streams, at most one per tile.
int warp_grid(int tiles, int reserve_sms)
{
    const int sms = device_sms();
    const int use = 2 * (sms - reserve_sms > 0 ? sms - reserve_sms : 1);
    return tiles < use ? tiles : use;
}

template <int N>
hv_status launch_rows_warp(const RowPass& p, int nframes, cudaStream_t st)
{
    using Gm = W32Geom<N>;
    RowPass q = p;
    if ((q.tw = twiddles_warp<N>()) == nullptr)
        return HV_ERR_CUDA;
    q.tw_count = Gm::TW;
    const int per_frame = (p.rows + Gm::RPW - 1) / Gm::RPW;
    const int units = per_frame * nframes;
    int grid = warp_grid((units + W32_WARPS - 1) / W32_WARPS, p.reserve_sms);
    // Complex input (the inverse rows of the angular spectrum) whose input and output exceed L2 is
    // bound by DRAM: two units per warp instead of a persistent grid read and write it faster
    // (inverse rows of 64 frames of 768 x 768: 110.4 -> 94.7 us, 32 of 1024 x 1024: 95.2 -> 85.0 us),
    // and below that size slower (12 frames of 768 x 768: 22.9 -> 24.5 us).
    if (p.in_kind == IN_C64 && p.reserve_sms == 0 && 16 * p.in_frame * static_cast<size_t>(nframes) > kL2Bytes)
        grid = (units + 2 * W32_WARPS - 1) / (2 * W32_WARPS);
    // bulk copies start on 16 bytes (rows of every input kind are a multiple of 16 bytes long)
    const bool bulk = g_fft_bulk.load() && (reinterpret_cast<uintptr_t>(p.in) & 15) == 0 &&
                      (p.in_frame * static_cast<size_t>(in_kind_bytes(p.in_kind))) % 16 == 0;
    void (*kern)(RowPass, int, int, int) = nullptr;
    const bool pre = p.premul != nullptr;
    switch (p.in_kind)
    {
    case IN_U8: kern = pre ? k_fft_rows_warp<N, IN_U8, true> : k_fft_rows_warp<N, IN_U8, false>; break;
    case IN_U16:
    case IN_U16_BE: kern = pre ? k_fft_rows_warp<N, IN_U16, true> : k_fft_rows_warp<N, IN_U16, false>; break;
    case IN_F32: kern = pre ? k_fft_rows_warp<N, IN_F32, true> : k_fft_rows_warp<N, IN_F32, false>; break;
    default: kern = pre ? k_fft_rows_warp<N, IN_C64, true> : k_fft_rows_warp<N, IN_C64, false>; break;
    }
    HV_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Gm::ROW_SMEM)));
    HV_LAUNCH(kern, grid, W32_THREADS, Gm::ROW_SMEM, st, q, per_frame, nframes, bulk ? 1 : 0);
    count_launch();
    return HV_OK;
}

template <int N>
hv_status launch_cols_warp(const ColPass& p, int nframes, cudaStream_t st)
{
    using Gm = W32Geom<N>;
    ColPass q = p;
    if ((q.tw = twiddles_warp<N>()) == nullptr)
        return HV_ERR_CUDA;
    q.tw_count = Gm::TW;
    const int tiles_x = (p.width + Gm::COLS - 1) / Gm::COLS;
    const int ntiles = tiles_x * nframes;
    const int grid = warp_grid(ntiles, p.reserve_sms);
    // tensor copies: 16-byte aligned base and row pitch, contiguous frames
    const uint64_t pitch = static_cast<uint64_t>(p.width) * sizeof(float2);
    CUtensorMap in_map{}, g_map{};
    bool bulk = g_fft_bulk.load() && p.in_frame == static_cast<size_t>(p.width) * N && pitch % 16 == 0 &&
                (reinterpret_cast<uintptr_t>(p.in) & 15) == 0 &&
                tc::encode_tmap_2d_f32(&in_map, p.in, static_cast<uint64_t>(p.width) * 2,
                                       static_cast<uint64_t>(nframes) * N, pitch, Gm::COLS * 2, 256);
    if (bulk && p.mode == 2)
        bulk = (reinterpret_cast<uintptr_t>(p.postmul) & 15) == 0 &&
               tc::encode_tmap_2d_f32(&g_map, p.postmul, static_cast<uint64_t>(p.width) * 2, N, pitch, Gm::COLS * 2, 256);
    auto kern = p.mode == 2   ? (bulk ? k_fft_cols_warp<N, 2, true> : k_fft_cols_warp<N, 2, false>)
                : p.mode == 1 ? (bulk ? k_fft_cols_warp<N, 1, true> : k_fft_cols_warp<N, 1, false>)
                              : (bulk ? k_fft_cols_warp<N, 0, true> : k_fft_cols_warp<N, 0, false>);
    HV_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(Gm::COL_SMEM)));
    HV_LAUNCH(kern, grid, W32_THREADS, Gm::COL_SMEM, st, in_map, g_map, q, tiles_x, ntiles);
    count_launch();
    return HV_OK;
}

template <int N>
hv_status launch_rows(const RowPass& p, int nframes, cudaStream_t st)
{
    if constexpr (N == 512 || N == 768 || N == 1024)
        if (g_fft_engine.load() == 0)
            return launch_rows_warp<N>(p, nframes, st);
    constexpr int F = row_lanes<N>();
    using Tl = fft::Tile<N, F, false>;
    const int tw_count = fft::twiddle_count(typename fft::Plan<N>::List{});
    const size_t smem = (static_cast<size_t>(F) * N + tw_count) * sizeof(float2);
    if (smem > 48 * 1024)
        HV_CUDA_TRY(cudaFuncSetAttribute(k_fft_rows<N, F>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem)));
    RowPass q = p;
    if ((q.tw = twiddles<N>()) == nullptr)
        return HV_ERR_CUDA;
    q.tw_count = tw_count;
    dim3 grid((p.rows + F - 1) / F, nframes);
    HV_LAUNCH((k_fft_rows<N, F>), grid, Tl::NT, smem, st, q);
    count_launch();
    return HV_OK;
}

template <int N, int F>
hv_status launch_cols_tiles(const ColPass& p, int nframes, cudaStream_t st)
{
    using Tl = fft::Tile<N, F, true>;
    const int tw_count = fft::twiddle_count(typename fft::Plan<N>::List{});
    const size_t smem = (static_cast<size_t>(F) * N + tw_count) * sizeof(float2);
    if (smem > 48 * 1024)
        HV_CUDA_TRY(cudaFuncSetAttribute(k_fft_cols<N, F>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem)));
    ColPass q = p;
    if ((q.tw = twiddles<N>()) == nullptr)
        return HV_ERR_CUDA;
    q.tw_count = tw_count;
    dim3 grid((p.width + F - 1) / F, nframes);
    HV_LAUNCH((k_fft_cols<N, F>), grid, Tl::NT, smem, st, q);
    count_launch();
    return HV_OK;
}

template <int N>
hv_status launch_cols(const ColPass& p, int nframes, cudaStream_t st)
{
    if constexpr (N == 512 || N == 768 || N == 1024)
        if (g_fft_engine.load() == 0)
            return launch_cols_warp<N>(p, nframes, st);
    constexpr int F = col_lanes<N>();
    // While half as wide tiles still find an SM each, they are the faster ones (AS middle pass, 1 to 4 frames of
    // 256 x 256 4.8 -> 3.7 us, 384 x 384 7.3 -> 6.2, 192 x 192 5.6 -> 5.3); beyond that both sizes take the same time
    // (256: 8 frames 4.9 and 5.0 us) and more frames fill the wide ones better. Tiles of a quarter gained nothing more.
    // Shorter lengths stay with the wide tiles: a launch's 3.2 to 3.4 us either way for 16 to 64 points (1, 4 and 16 frames),
    // 4.9 and 4.8 us for 96.
    if constexpr (F == 16 && (N == 128 || N == 192 || N == 256 || N == 384))
        if (static_cast<long long>((p.width + F - 1) / F) * nframes * 2 <= device_sms())
            return launch_cols_tiles<N, F / 2>(p, nframes, st);
    return launch_cols_tiles<N, F>(p, nframes, st);
}

}  // namespace

void set_fft_engine(int mode)
{
    g_fft_engine = mode == 2 ? 0 : mode;
    g_fft_bulk = mode == 2 ? 0 : 1;
}

hv_status fft_status()
{
    int err = 0;
    HV_CUDA_TRY(cudaMemcpyFromSymbol(&err, g_fft_wait_error, sizeof(int)));
    return err ? HV_ERR_TIMEOUT : HV_OK;
}

bool fft_size_supported(int n)
{
    switch (n)
    {
#define HV_CASE(N)                                                                                                     \
    case N: return true;
        HV_FFT_SIZES(HV_CASE)
#undef HV_CASE
    default: return false;
    }
}

hv_status fft_rows(const RowPass& p, int N, int nframes, cudaStream_t st)
{
    switch (N)
    {
#define HV_CASE(NN)                                                                                                    \
    case NN: return launch_rows<NN>(p, nframes, st);
        HV_FFT_SIZES(HV_CASE)
#undef HV_CASE
    default: set_last_error_msg("unsupported FFT length"); return HV_ERR_UNSUPPORTED;
    }
}

hv_status fft_cols(const ColPass& p, int N, int nframes, cudaStream_t st)
{
    switch (N)
    {
#define HV_CASE(NN)                                                                                                    \
    case NN: return launch_cols<NN>(p, nframes, st);
        HV_FFT_SIZES(HV_CASE)
#undef HV_CASE
    default: set_last_error_msg("unsupported FFT length"); return HV_ERR_UNSUPPORTED;
    }
}

hv_status make_fresnel_lens(float2* lens, int W, int H, float lam, float z, float ps, int mode, cudaStream_t st)
{
    dim3 block(128), grid((W + 127) / 128, H);
    HV_LAUNCH(k_fresnel_lens, grid, block, 0, st, lens, W, H, lam, z, ps, mode);
    count_launch();
    return HV_OK;
}

hv_status make_spectral_lens(float2* lens, int W, int H, float lam, float z, float ps, int mode, cudaStream_t st)
{
    dim3 block(128), grid((W + 127) / 128, H);
    HV_LAUNCH(k_spectral_lens, grid, block, 0, st, lens, W, H, lam, z, ps, mode);
    count_launch();
    return HV_OK;
}

// ====================================================================================== filter2D

// Band-pass mask of kernel_update_filter2d_circles_mask (filter2D.cu:52-88) in the reference's
// float arithmetic: r = hypotf(x - W/2, y - H/2), A = 1 inside radius n2 with a cosine roll-off of
// width sh, B the same for n1 / sl, mask = A (1 - B); written quadrant-swapped (FFT layout, the
// shift_corners of update_filter2d_circles_mask) as complex (multiply = 0) or multiplied into an
// FFT-layout complex array in place (multiply = 1: the AS transfer function, fourier_transform.cc:134-137).
__global__ void k_filter2d_mask(float2* dst, int W, int H, int n1, int n2, int sl, int sh, int multiply)
{
    wait_prior_kernels();
    const int X = blockIdx.x * blockDim.x + threadIdx.x, Y = blockIdx.y;
    if (X >= W || Y >= H)
        return;
    const int x = (X + W / 2) % W, y = (Y + H / 2) % H;  // source of the quadrant swap (even W, H)
    const float rx = static_cast<float>(x) - static_cast<float>(W / 2);
    const float ry = static_cast<float>(y) - static_cast<float>(H / 2);
    const float len = hypotf(rx, ry);
    float a = 0.0f, b = 0.0f;
    if (len < static_cast<float>(n2))
        a = 1.0f;
    else if (len < static_cast<float>(n2 + sh))
        a = cosf(static_cast<float>(static_cast<double>(__fdiv_rn(len - static_cast<float>(n2), static_cast<float>(sh))) *
                                    1.57079632679489661923));
    if (len < static_cast<float>(n1))
        b = 1.0f;
    else if (len < static_cast<float>(n1 + sl))
        b = cosf(static_cast<float>(static_cast<double>(__fdiv_rn(len - static_cast<float>(n1), static_cast<float>(sl))) *
                                    1.57079632679489661923));
    const float m = a * (1.0f - b);
    float2* o = dst + static_cast<size_t>(Y) * W + X;
    if (multiply)
    {
        const float2 v = *o;
        *o = make_float2(v.x * m, v.y * m);
    }
    else
        *o = make_float2(m, 0.0f);
}

hv_status filter2d_mask(float2* dst, int W, int H, int n1, int n2, int smooth_low, int smooth_high, int multiply,
                        cudaStream_t st)
{
    if (!dst || W <= 0 || H <= 0 || (W & 1) || (H & 1) || n1 < 0 || n2 <= n1 || smooth_low < 0 || smooth_high < 0)
        return HV_INVALID_VALUE;
    dim3 block(128), grid((W + 127) / 128, H);
    HV_LAUNCH(k_filter2d_mask, grid, block, 0, st, dst, W, H, n1, n2, smooth_low, smooth_high, multiply);
    count_launch();
    return HV_OK;
}

int raw_kind(int raw_bytes, int big_endian)
{
    switch (raw_bytes)
    {
    case 1: return IN_U8;
    case 2: return big_endian ? IN_U16_BE : IN_U16;
    case 4: return IN_F32;
    case 8: return IN_C64;
    default: return -1;
    }
}

static std::atomic<int> g_spatial_sub_mb{0};
void set_spatial_sub_batch_mb(int mb) { g_spatial_sub_mb = mb < 0 ? 0 : mb; }

hv_status spatial_transform(const void* raw, int kind, int W, int H, int batch, int space, const float2* lens,
                            float2* work, float2* ring, int slot0, int nslots, cudaStream_t st, const CycleCtl* ctl,
                            const float2* f2d_mask, float2* work2, uint16_t* real_planes, int reserve_sms)
{
    // With a cycle control block, `raw` is the input ring base (the batch sits at ctl->raw_offset)
    // and the ring slot of frame 0 is slot0 + ctl->ring_begin; every pass is gated by ctl->active.
    const int* begin_dev = ctl ? &ctl->ring_begin : nullptr;
    const size_t HW = static_cast<size_t>(W) * H;
    const FrameMap ring_map{HW, slot0, nslots, begin_dev};
    const FrameMap work_map{HW, 0, batch > 0 ? batch : 1};
    if (batch <= 0)
        return HV_OK;
    // filter2D before Fresnel or without propagation (fourier_transform.cc:55-58, filter2D.cu:28-46);
    // for AS the mask is part of the transfer function and nothing changes here
    const bool f2d = f2d_mask && space != HV_SPACE_ANGULARSP;
    if (f2d && (!work || (space == HV_SPACE_FRESNELTR && !work2)))
        return HV_INVALID_VALUE;
    if (space == HV_SPACE_NONE && !f2d)
    {
        const int block = 256;
        // 8-pixel groups: 8-byte (8-bit), 16-byte (16-bit) and 32-byte (float) aligned loads when the
        // batch starts on 16 bytes and frames hold a multiple of 8 pixels
        if (HW % 8 == 0 && kind != IN_C64 && (reinterpret_cast<uintptr_t>(raw) & 15) == 0 &&
            (reinterpret_cast<uintptr_t>(ring) & 15) == 0)
        {
            const size_t total = HW / 8 * batch;
            const int grid = static_cast<int>((total + block - 1) / block < 152 * 8 ? (total + block - 1) / block : 152 * 8);
            HV_LAUNCH(k_convert8, grid, block, 0, st, raw, kind, HW, batch, ring, ring_map, ctl, real_planes);
            count_launch();
            return HV_OK;
        }
        if (real_planes)
        {
            set_last_error_msg("converting into the split planes needs frames of a multiple of 8 pixels");
            return HV_ERR_UNSUPPORTED;
        }
        const size_t total = HW * batch;
        const int grid = static_cast<int>((total + block - 1) / block < 152 * 16 ? (total + block - 1) / block : 152 * 16);
        HV_LAUNCH(k_convert, grid, block, 0, st, raw, kind, HW, batch, ring, ring_map, ctl);
        count_launch();
        return HV_OK;
    }
    if (!fft_size_supported(W) || !fft_size_supported(H))
    {
        set_last_error_msg("frame width/height not supported by the shared-memory FFT");
        return HV_ERR_UNSUPPORTED;
    }
    // One launch per pass over the whole batch when g_spatial_sub_mb is 0; otherwise sub-batches
    // whose complex intermediate (sb frames) fits in that many MB of L2 between the passes. Raw
    // input is read and ring slots are written with streaming hints.
    const size_t frame_c64 = HW * sizeof(float2);
    const int sub_mb = g_spatial_sub_mb.load();
    int sb = sub_mb > 0 ? static_cast<int>((static_cast<size_t>(sub_mb) << 20) / frame_c64) : batch;
    if (sb < 1)
        sb = 1;
    if (sb > batch)
        sb = batch;
    const size_t raw_frame_bytes = HW * static_cast<size_t>(in_kind_bytes(kind));
    for (int b0 = 0; b0 < batch; b0 += sb)
    {
        const int nb = (batch - b0) < sb ? (batch - b0) : sb;
        const void* raw_b = static_cast<const uint8_t*>(raw) + static_cast<size_t>(b0) * raw_frame_bytes;
        const FrameMap ring_b{HW, (slot0 + b0) % nslots, nslots, begin_dev};
        const FrameMap work_b{HW, 0, nb};
        hv_status s;
        if (f2d)
        {
            // forward rows -> work; columns: forward, *M, inverse (in place); then the unnormalised
            // inverse rows: -> ring slots (no propagation) or -> work2, *L and forward rows -> work,
            // forward columns -> ring slots (Fresnel)
            RowPass r{raw_b, kind, HW, work, work_b, nullptr, H, 0, 1.0f};
            r.ctl = ctl;
            r.raw_from_ctl = ctl ? 1 : 0;
            if ((s = fft_rows(r, W, nb, st)) != HV_OK)
                return s;
            ColPass c{work, HW, work, work_b, f2d_mask, W, 2, 1.0f};
            c.ctl = ctl;
            if ((s = fft_cols(c, H, nb, st)) != HV_OK)
                return s;
            if (space == HV_SPACE_NONE)
            {
                RowPass r2{work, IN_C64, HW, ring, ring_b, nullptr, H, 1, 1.0f};
                r2.stream_out = 1;
                r2.ctl = ctl;
                if ((s = fft_rows(r2, W, nb, st)) != HV_OK)
                    return s;
                continue;
            }
            RowPass r2{work, IN_C64, HW, work2, work_b, nullptr, H, 1, 1.0f};
            r2.ctl = ctl;
            if ((s = fft_rows(r2, W, nb, st)) != HV_OK)
                return s;
            RowPass r3{work2, IN_C64, HW, work, work_b, lens, H, 0, 1.0f};
            r3.ctl = ctl;
            if ((s = fft_rows(r3, W, nb, st)) != HV_OK)
                return s;
            ColPass c2{work, HW, ring, ring_b, nullptr, W, 0, 1.0f};
            c2.stream_out = 1;
            c2.ctl = ctl;
            if ((s = fft_cols(c2, H, nb, st)) != HV_OK)
                return s;
            continue;
        }
        if (space == HV_SPACE_FRESNELTR)
        {
            // x*L, forward rows -> work; forward columns -> ring slots
            RowPass r{raw_b, kind, HW, work, work_b, lens, H, 0, 1.0f};
            r.ctl = ctl;
            r.raw_from_ctl = ctl ? 1 : 0;
            r.reserve_sms = reserve_sms;
            if ((s = fft_rows(r, W, nb, st)) != HV_OK)
                return s;
            ColPass c{work, HW, ring, ring_b, nullptr, W, 0, 1.0f};
            c.stream_out = 1;
            c.ctl = ctl;
            c.reserve_sms = reserve_sms;
            if ((s = fft_cols(c, H, nb, st)) != HV_OK)
                return s;
        }
        else if (space == HV_SPACE_ANGULARSP)
        {
            // forward rows -> work; columns: forward, *G, inverse (in place); inverse rows /(H*W) -> ring
            RowPass r{raw_b, kind, HW, work, work_b, nullptr, H, 0, 1.0f};
            r.ctl = ctl;
            r.raw_from_ctl = ctl ? 1 : 0;
            r.reserve_sms = reserve_sms;
            if ((s = fft_rows(r, W, nb, st)) != HV_OK)
                return s;
            ColPass c{work, HW, work, work_b, lens, W, 2, 1.0f};
            c.ctl = ctl;
            if ((s = fft_cols(c, H, nb, st)) != HV_OK)
                return s;
            RowPass r2{work, IN_C64, HW, ring, ring_b, nullptr, H, 1, 1.0f / static_cast<float>(HW)};
            r2.stream_out = 1;
            r2.ctl = ctl;
            if ((s = fft_rows(r2, W, nb, st)) != HV_OK)
                return s;
        }
        else
        {
            set_last_error_msg("unknown space transformation");
            return HV_INVALID_VALUE;
        }
    }
    return HV_OK;
}

hv_status convert_window(const void* raw, int kind, size_t HW, int batch, int slot0, int T, uint16_t* planes,
                         int sample0, int cap, uint16_t* samples, cudaStream_t st)
{
    if (HW % 8 != 0 || (kind != IN_U8 && kind != IN_U16 && kind != IN_U16_BE) || batch <= 0)
        return HV_ERR_UNSUPPORTED;
    const size_t total = HW / 8 * batch;
    const int block = 256;
    // three quarters of the SMs' thread slots: the pipelined windows' eigensolve kernels (another
    // stream) find room beside this pass
    const int cap_ctas = device_sms() * 6;
    const int grid = static_cast<int>((total + block - 1) / block < static_cast<size_t>(cap_ctas) ? (total + block - 1) / block : cap_ctas);
    const bool vec = (reinterpret_cast<uintptr_t>(raw) & 15) == 0;
    auto kern = kind == IN_U8 ? (vec ? k_convert_window<IN_U8, true> : k_convert_window<IN_U8, false>)
                              : (vec ? k_convert_window<IN_U16, true> : k_convert_window<IN_U16, false>);
    HV_LAUNCH_BESIDE(kern, grid, block, 0, st, raw, kind == IN_U16_BE ? 1 : 0, HW, batch, slot0, T, planes, sample0, cap, samples);
    count_launch();
    return HV_OK;
}

hv_status ring_from_planes(const uint16_t* planes, int T, size_t HW, int slot0, int n, float2* ring, cudaStream_t st)
{
    if (HW % 8 != 0 || n <= 0)
        return n <= 0 ? HV_OK : HV_ERR_UNSUPPORTED;
    const size_t total = HW / 8 * n;
    const int block = 256;
    const int cap = device_sms() * 6;  // as convert_window: room for the eigensolve stream's kernels
    const int grid = static_cast<int>((total + block - 1) / block < static_cast<size_t>(cap) ? (total + block - 1) / block : cap);
    HV_LAUNCH(k_ring_from_planes, grid, block, 0, st, planes, T, HW, slot0, n, ring);
    count_launch();
    return HV_OK;
}

hv_status fft_rows_pass(const void* in, int kind, float2* out, int W, int H, int batch, const float2* premul,
                        int inverse, float scale, int slot0, int nslots, cudaStream_t st)
{
    const size_t HW = static_cast<size_t>(W) * H;
    RowPass r{in, kind, HW, out, FrameMap{HW, slot0, nslots}, premul, H, inverse, scale};
    return fft_rows(r, W, batch, st);
}

hv_status fft_cols_pass(const float2* in, float2* out, int W, int H, int batch, const float2* postmul, int mode,
                        float scale, int slot0, int nslots, cudaStream_t st)
{
    const size_t HW = static_cast<size_t>(W) * H;
    ColPass c{in, HW, out, FrameMap{HW, slot0, nslots}, postmul, W, mode, scale};
    return fft_cols(c, H, batch, st);
}

hv_status fft2d(const float2* in, float2* out, int n0, int n1, int batch, int inverse, float scale, cudaStream_t st)
{
    if (!fft_size_supported(n0) || !fft_size_supported(n1))
    {
        set_last_error_msg("FFT length not supported");
        return HV_ERR_UNSUPPORTED;
    }
    const size_t HW = static_cast<size_t>(n0) * n1;
    const FrameMap map{HW, 0, batch};
    RowPass r{in, IN_C64, HW, out, map, nullptr, n0, inverse, 1.0f};
    hv_status s = fft_rows(r, n1, batch, st);
    if (s != HV_OK)
        return s;
    ColPass c{out, HW, out, map, nullptr, n1, inverse ? 1 : 0, scale};
    return fft_cols(c, n0, batch, st);
}

}  // namespace hv
