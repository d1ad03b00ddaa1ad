// Projection pre-processing on arrival (minirecast preprocess.py), block layout
// [rows, k, cols] (ASTRA) in and out, FP32.
//
//   rotate_projections preprocess.py:31-56: out(r,c) = bilinear(in, rs, cs), zero
//       outside, rs = cos t * rr + sin t * cc + (R-1)/2, cs = -sin t * rr + cos t * cc + (C-1)/2
//   gaussian_blur      preprocess.py:8-28: per axis, edge padding by pad = ceil(3 sigma),
//       circular convolution of length N = n + 2 pad with g = irfft(exp(-2 (pi f sigma)^2)),
//       crop. The caller passes g[0..K] (g is even; |m| > K contributes < 1e-20).
#include <type_traits>

#include "mr_common.cuh"

namespace mr {

// Where an output samples its view, and with what weights, is the same in every view: a thread
// forms both once for RT_VIEWS views and has the taps of all of them in flight, where a thread of
// one output waited for its four loads alone (486 x 384, 0.3 degrees: 600 views 483 -> 227 us,
// 64 views 57 -> 32 us, 8 views 12 -> 10 us; 1944 x 1536: 64 views 816 -> 352 us, 8 views 106 ->
// 46, 2 views 29 -> 25; the same outputs). One view has nothing to share and keeps a kernel of its
// own (1944 x 1536: 18.3 us, 23.2 with the other). A read and a write of the 600 views take 137
// us; what is left is latency and issue (63 %) of the four loads an output.
constexpr int RT_VIEWS = 8;
template <int VIEWS>
__global__ void __launch_bounds__(128) rotate_kernel(const float* __restrict__ in, float* __restrict__ out, int R,
                                                     int A, int C, float ct, float st) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y;
    const int a0 = blockIdx.z * VIEWS;
    if (c >= C) return;
    const float rr = (float)r - 0.5f * (float)(R - 1);
    const float cc = (float)c - 0.5f * (float)(C - 1);
    const float rs = fmaf(ct, rr, st * cc) + 0.5f * (float)(R - 1);
    const float cs = fmaf(-st, rr, ct * cc) + 0.5f * (float)(C - 1);
    const float r0f = floorf(rs), c0f = floorf(cs);
    const float fr = rs - r0f, fc = cs - c0f;
    const int r0 = (int)r0f, c0 = (int)c0f;
    const long long srow = (long long)A * C;
    float w[4];
    bool ok[4];
    const float* p[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int ri = r0 + (t >> 1), ci = c0 + (t & 1);
        w[t] = (t >> 1 ? fr : 1.f - fr) * (t & 1 ? fc : 1.f - fc);
        ok[t] = (unsigned)ri < (unsigned)R && (unsigned)ci < (unsigned)C;
        p[t] = in + (ok[t] ? ri * srow + (long long)a0 * C + ci : 0);
    }
    float* o = out + r * srow + (long long)a0 * C + c;
    auto views = [&](int a, auto n) {               // views a0 + a .. a0 + a + n - 1
        constexpr int V = decltype(n)::value;
        float x[V][4];
#pragma unroll
        for (int v = 0; v < V; ++v)
#pragma unroll
            for (int t = 0; t < 4; ++t) x[v][t] = ok[t] ? __ldg(p[t] + (long long)(a + v) * C) : 0.f;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            float acc = 0.f;
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (ok[t]) acc = fmaf(w[t], x[v][t], acc);
            o[(long long)(a + v) * C] = acc;
        }
    };
    const int n = min(VIEWS, A - a0);
    if (n == VIEWS) views(0, std::integral_constant<int, VIEWS>{});
    else
        for (int a = 0; a < n; ++a) views(a, std::integral_constant<int, 1>{});
}

// One axis of the edge-padded circular Gaussian: along rows (axis 0) or cols (axis 2).
__global__ void gauss_axis_kernel(const float* __restrict__ in, float* __restrict__ out, int R, int A,
                                  int C, int axis, int pad, const float* __restrict__ g, int K) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y;
    const int a = blockIdx.z;
    if (c >= C) return;
    const long long srow = (long long)A * C;
    const int n = axis == 0 ? R : C;
    const int i = axis == 0 ? r : c;
    const int Np = n + 2 * pad;
    const float* base = axis == 0 ? in + (long long)a * C + c : in + r * srow + (long long)a * C;
    const long long step = axis == 0 ? srow : 1;
    float acc = 0.f;
    for (int m = -K; m <= K; ++m) {
        int t = i + pad - m;                 // index into the padded signal, circular
        t %= Np;
        if (t < 0) t += Np;
        int src = t - pad;                   // edge padding
        src = src < 0 ? 0 : (src >= n ? n - 1 : src);
        acc = fmaf(__ldg(g + (m < 0 ? -m : m)), __ldg(base + src * step), acc);
    }
    out[r * srow + (long long)a * C + c] = acc;
}

// The same axis convolution organised for the SM. For small sigma the taps reach about half
// the padded length (the spectrum is cut at Nyquist), so a direct loop costs ~n/2 taps per
// output. A block takes L lines (rows along axis 2, columns along axis 0) and TO outputs of
// each: it stages the stretch of the edge-padded, periodically extended line those outputs
// read into shared memory once, then every thread computes 16 consecutive outputs of two
// neighbouring lines, 8 taps at a time. Both lines share every instruction (packed f32x2
// multiply-adds), and the 23 staged positions that a block of 8 taps reaches stay in
// registers from one block to the next, 8 new ones a block: 128 packed multiply-adds on 12
// shared-memory loads. The taps are padded in front with zeros to a multiple of 8 (m from
// K - 8 nb + 1); those add 0 * x to a zero sum, exactly, so each output is the same FMA chain
// over m = -K .. K as in gauss_axis_kernel and the results are identical.
// Bound by the FMA pipe (64 views of 486 x 384, sigma 1, 390 and 492 taps an output: rows 328 ->
// 222 us, columns 465 -> 278 us, 60 % of its rate, of them about 60 and 90 us staging and
// stores). Before, a thread computed 8 outputs of one line and loaded its 15 positions anew for
// every block of taps; without the unrolling by 3 the window's moves cost 10 %.
constexpr int GS_THREADS = 256;
constexpr int GS_TAPS = 8;                      // taps per block
constexpr int GS_RUN = 16;                      // consecutive outputs per thread

template <int L, int LP>
__global__ void __launch_bounds__(GS_THREADS, 2)
gauss_lines_kernel(const float* __restrict__ in, float* __restrict__ out, int R, int A, int C, int axis,
                   int pad, const float* __restrict__ g, int K, int TO) {
    static_assert(L % 2 == 0 && LP % 2 == 0, "lines in pairs");
    extern __shared__ __align__(16) float gsm[];
    const int nb = (2 * K + GS_TAPS) / GS_TAPS;                 // blocks of 8 taps
    const int m0 = K - GS_TAPS * nb + 1;                       // first (zero-padded) tap
    const int T = TO + GS_TAPS * nb;            // staged positions per line
    float2* taps = reinterpret_cast<float2*>(gsm);              // [8 nb]: tap m0 + i, twice
    float* ext = gsm + 2 * GS_TAPS * nb;        // [T][LP]
    const long long srow = (long long)A * C;
    const int n = axis == 0 ? R : C;
    const int Np = n + 2 * pad;
    const long long n_lines = axis == 0 ? (long long)A * C : (long long)R * A;
    const long long line0 = (long long)blockIdx.x * L;
    const int i0 = blockIdx.y * TO;
    const long long step = axis == 0 ? srow : 1;
    auto line_base = [&](long long line) -> long long {
        if (axis == 0) return line;                                     // a * C + c
        const long long r = line / A, a = line - r * A;
        return r * srow + a * C;
    };
    for (int i = threadIdx.x; i < GS_TAPS * nb; i += blockDim.x) {
        const int m = m0 + i;
        const float v = m < -K ? 0.f : __ldg(g + (m < 0 ? -m : m));
        taps[i] = make_float2(v, v);
    }
    // staged position t holds padded position i0 + pad - K + t; output o at tap m reads t = o + K - m.
    // The line position behind it (circular, edge padding) is the same for every line: a table,
    // then asynchronous copies that need only an address each.
    const int nl = (int)min((long long)L, n_lines - line0);
    int* from = reinterpret_cast<int*>(ext + T * LP);           // [T]
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
        int u = i0 + pad - K + t;                                       // padded position
        u %= Np;
        if (u < 0) u += Np;                                             // circular
        from[t] = min(max(u - pad, 0), n - 1);                          // edge padding
    }
    __syncthreads();
    const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(ext));
    auto copy = [&](int t, int l, const float* src) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to + (t * LP + l) * 4), "l"(src) : "memory");
    };
    if (axis == 0) {                                                    // lanes along neighbouring columns
        const int l = threadIdx.x % L;
        if (l < nl) {
            const float* line = in + line0 + l;
#pragma unroll 4
            for (int t = threadIdx.x / L; t < T; t += blockDim.x / L) copy(t, l, line + from[t] * step);
        }
    } else {                                                            // lanes along one row
        const int lane = threadIdx.x & 31;
        for (int l = threadIdx.x >> 5; l < nl; l += blockDim.x >> 5) {
            const float* line = in + line_base(line0 + l);
#pragma unroll 4
            for (int t = lane; t < T; t += 32) copy(t, l, line + from[t]);
        }
    }
    if (nl & 1)                                                         // a pair's missing line
        for (int t = threadIdx.x; t < T; t += blockDim.x) ext[t * LP + nl] = 0.f;
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int groups = (TO + GS_RUN - 1) / GS_RUN;
    for (int task = threadIdx.x; task < L / 2 * groups; task += blockDim.x) {
        const int l = 2 * (task % (L / 2)), q = task / (L / 2);         // lines l, l + 1
        const int o0 = q * GS_RUN;                                      // first output (block-local)
        if (l >= nl || i0 + o0 >= n) continue;
        float2 acc[GS_RUN];
#pragma unroll
        for (int j = 0; j < GS_RUN; ++j) acc[j] = make_float2(0.f, 0.f);
        // taps m0 + 8 b + u (u < 8) of output o0 + j read position first + 8 (nb - 1 - b) + 7 + j - u;
        // w holds the block's positions .. + 0 .. 22
        const float2* p = reinterpret_cast<const float2*>(ext + (o0 + K - m0 - (GS_TAPS - 1)) * LP + l);
        float2 w[GS_RUN + GS_TAPS - 1];
#pragma unroll
        for (int k = GS_TAPS; k < GS_RUN + GS_TAPS - 1; ++k) w[k] = p[k * (LP / 2)];
#pragma unroll 3                                // the window's three parts change names, not registers
        for (int b = 0; b < nb; ++b) {
#pragma unroll
            for (int k = 0; k < GS_TAPS; ++k) w[k] = p[k * (LP / 2)];
#pragma unroll
            for (int u = 0; u < GS_TAPS; ++u) {
                const float2 gm = taps[GS_TAPS * b + u];
#pragma unroll
                for (int j = 0; j < GS_RUN; ++j) acc[j] = __ffma2_rn(gm, w[j - u + GS_TAPS - 1], acc[j]);
            }
#pragma unroll
            for (int k = GS_RUN + GS_TAPS - 2; k >= GS_TAPS; --k) w[k] = w[k - GS_TAPS];
            p -= GS_TAPS * (LP / 2);
        }
        const long long lb0 = line_base(line0 + l), lb1 = line_base(min(line0 + l + 1, n_lines - 1));
#pragma unroll
        for (int j = 0; j < GS_RUN; ++j) {
            const int i = i0 + o0 + j;
            if (i >= n || o0 + j >= TO) continue;
            out[lb0 + (long long)i * step] = acc[j].x;
            if (l + 1 < nl) out[lb1 + (long long)i * step] = acc[j].y;
        }
    }
}

template <int LP>
static size_t gauss_lines_smem(int K, int TO) {
    const int nb = (2 * K + GS_TAPS) / GS_TAPS;
    return ((size_t)(TO + GS_TAPS * nb) * (LP + 1) + 2 * (size_t)GS_TAPS * nb) * sizeof(float);
}

// Most outputs of 4 lines that gauss_lines_smem<4> leaves room for (a multiple of GS_RUN; may be
// negative).
static int gauss_few_outputs(int K, size_t limit) {
    const long long span = GS_TAPS * (long long)((2 * (long long)K + GS_TAPS) / GS_TAPS);
    const long long room = ((long long)(limit / sizeof(float)) - 2 * span) / 5 - span;
    return (int)(room / GS_RUN * GS_RUN);
}

template <int L, int LP>
static int launch_gauss_lines(const float* in, float* out, int R, int A, int C, int axis, int pad, const float* taps,
                              int K, int TO, cudaStream_t st) {
    const int n = axis == 0 ? R : C;
    const long long n_lines = axis == 0 ? (long long)A * C : (long long)R * A;
    const size_t smem = gauss_lines_smem<LP>(K, TO);
    MR_CUDA_TRY(cudaFuncSetAttribute(gauss_lines_kernel<L, LP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
    // no more threads than tasks (rounded to warps), but four warps for the staging
    const int tasks = L / 2 * ((TO + GS_RUN - 1) / GS_RUN);
    const int threads = tasks < 128 ? 128 : (tasks < GS_THREADS ? (tasks + 31) / 32 * 32 : GS_THREADS);
    const dim3 grid((unsigned)((n_lines + L - 1) / L), (unsigned)((n + TO - 1) / TO));
    gauss_lines_kernel<L, LP><<<grid, threads, smem, st>>>(in, out, R, A, C, axis, pad, taps, K, TO);
    return MR_OK;
}

}  // namespace mr

extern "C" int mr_rotate_f32(const float* in, float* out, int32_t rows, int32_t k, int32_t cols,
                             double degrees, void* stream) {
    if (!in || !out || rows <= 0 || cols <= 0 || k < 0 || in == out) return MR_ERR_INVALID;
    if (k == 0) return MR_OK;
    const double t = degrees * 3.14159265358979323846 / 180.0;
    const dim3 block(128);
    const int views = k == 1 ? 1 : mr::RT_VIEWS;
    const dim3 grid((cols + 127) / 128, rows, (k + views - 1) / views);
    if (k > 65535 || rows > 65535) return MR_ERR_INVALID;
    (views == 1 ? mr::rotate_kernel<1> : mr::rotate_kernel<mr::RT_VIEWS>)<<<grid, block, 0, static_cast<cudaStream_t>(stream)>>>(
        in, out, rows, k, cols, (float)cos(t), (float)sin(t));
    MR_CUDA_TRY(cudaGetLastError());
    return MR_OK;
}

extern "C" int mr_gaussian_axis_f32(const float* in, float* out, int32_t rows, int32_t k,
                                    int32_t cols, int32_t axis, int32_t pad, const float* taps,
                                    int32_t n_taps, void* stream) {
    if (!in || !out || !taps || rows <= 0 || cols <= 0 || k < 0 || in == out) return MR_ERR_INVALID;
    if ((axis != 0 && axis != 2) || pad < 0 || n_taps < 1) return MR_ERR_INVALID;
    if (k == 0) return MR_OK;
    if (k > 65535 || rows > 65535) return MR_ERR_INVALID;
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int K = n_taps - 1;
    const int n = axis == 0 ? rows : cols;
    constexpr size_t kSmemMax = 200 * 1024;
    // whole lines per block (16 lines: every input staged about twice, the periodic
    // extension) where they fit, else 8 lines x 512 outputs, else 4 lines and as many outputs as
    // fit (more than 1750 taps a side: axes of 3500 to 7000 pixels; one view of 3600 x 3504, both
    // axes, 6.0 ms, 115.9 by the loop without staging, which longer axes are left to)
    const int few = mr::gauss_few_outputs(K, kSmemMax);
    const int whole = (n + mr::GS_RUN - 1) / mr::GS_RUN * mr::GS_RUN;
    if (K <= n + 2 * pad && mr::gauss_lines_smem<18>(K, whole) <= kSmemMax) {
        const int rc = mr::launch_gauss_lines<16, 18>(in, out, rows, k, cols, axis, pad, taps, K, whole, st);
        if (rc != MR_OK) return rc;
    } else if (K <= n + 2 * pad && mr::gauss_lines_smem<10>(K, 512) <= kSmemMax) {
        const int rc = mr::launch_gauss_lines<8, 10>(in, out, rows, k, cols, axis, pad, taps, K, 512, st);
        if (rc != MR_OK) return rc;
    } else if (K <= n + 2 * pad && few >= 256) {
        const int rc = mr::launch_gauss_lines<4, 4>(in, out, rows, k, cols, axis, pad, taps, K, few < whole ? few : whole, st);
        if (rc != MR_OK) return rc;
    } else {
        const dim3 block(128);
        const dim3 grid((cols + 127) / 128, rows, k);
        mr::gauss_axis_kernel<<<grid, block, 0, st>>>(in, out, rows, k, cols, axis, pad, taps, K);
    }
    MR_CUDA_TRY(cudaGetLastError());
    return MR_OK;
}
