// Volume consumers on the device: the Otsu threshold of minirecast model.py:18-29,
//   v = vol[vol != 0]; lo, hi = np.percentile(v, [0.1, 99.95])
//   hist, edges = np.histogram(np.clip(v, lo, hi), bins=bins, range=(lo, hi))
// reduced to three streaming passes over the volume (any number of voxels, FP32):
//   mr_volume_stats      count of non-zero voxels and NaNs, min / max order key
//   mr_volume_select     exact order statistics of the non-zero voxels (radix select on
//                        order-preserving keys, 11-bit digits below the bits that the
//                        smallest and largest key share: at most 3 passes)
//   mr_volume_histogram  numpy's uniform-bin histogram of the FP64-clipped values
// and, for the two percentiles of the clip, one pass in the place of stats and select:
//   mr_volume_tails      brackets both percentiles by a sample, then counts the voxels and
//                        collects those outside the brackets (a few per mille; those equal to
//                        a bracket, which may be any number, are only counted)
//   mr_volume_tail_select  exact order statistics among the collected ones
// The percentile interpolation and the Otsu arithmetic over the bins stay on the host,
// in FP64 as the reference computes them.
//
// Every pass reads the voxels as float4 where aligned. The select passes combine the
// increments of neighbouring lanes that fall in the same bin into one shared-memory atomic;
// the histogram leaves that to the hardware, which adds equal addresses of a warp together.
#include <cooperative_groups.h>
#include <cstddef>

#include "mr_common.cuh"

namespace cg = cooperative_groups;

namespace mr {

constexpr int VOL_THREADS = 256;
constexpr int VOL_MAX_RANKS = 4;
constexpr int VOL_MAX_BINS = 2048;
constexpr int VOL_RADIX = 11;                   // digit bits of one select pass
constexpr int VOL_DIGITS = 1 << VOL_RADIX;
constexpr uint32_t VOL_NONE = 0xffffffffu;
constexpr unsigned FULL = 0xffffffffu;

constexpr int TAIL_CAP = 1 << 22;               // voxels kept of each tail
constexpr int TAIL_SAMPLE = 16384;

// Device workspace of the entry points (the first part zeroed by mr_volume_stats, the tails'
// counts by mr_volume_tails).
struct VolState {
    unsigned long long nonzero;             // voxels != 0 (NaNs included, as vol != 0 keeps them)
    unsigned long long nan;                 // NaN voxels
    unsigned int kmin, kmax;                // order keys of the smallest / largest non-NaN value != 0
    unsigned int prefix[VOL_MAX_RANKS];     // key bits found so far, per requested rank
    unsigned long long rank[VOL_MAX_RANKS]; // rank left inside the current prefix
    unsigned long long hist[VOL_MAX_RANKS][VOL_DIGITS];
    unsigned long long t_nonzero, t_nan, t_count[2];    // mr_volume_tails: voxels != 0, NaNs, size of each tail
    unsigned long long t_beyond[2];         // those that are not equal to the edge
    float t_edge[2];                        // tail 0: x <= t_edge[0]; tail 1: x >= t_edge[1]
    __align__(16) float tail[2][TAIL_CAP];  // the voxels beyond the edges
};

// Order-preserving map of a float onto an unsigned key (negatives reversed below positives).
__device__ __forceinline__ uint32_t order_key(float x) {
    const uint32_t b = __float_as_uint(x);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// hist[b] += 1 for every lane whose b != VOL_NONE; a run of equal b in consecutive lanes
// is one atomic of the run length. All 32 lanes of the warp call it.
__device__ __forceinline__ void warp_run_add(unsigned int* hist, uint32_t b, int lane) {
    const uint32_t prev = __shfl_up_sync(FULL, b, 1);
    const bool head = lane == 0 || prev != b;
    const uint32_t heads = __ballot_sync(FULL, head);
    if (head && b != VOL_NONE) {
        const uint32_t above = lane == 31 ? 0u : (heads & (0xffffffffu << (lane + 1)));
        const int next = above ? __ffs(above) - 1 : 32;
        atomicAdd(hist + b, (unsigned)(next - lane));
    }
}

// Visits every voxel once: aligned float4 body in warp-uniform steps of 4 loads per lane
// (fn receives 4 values per load slot and a validity flag, called by all lanes), then the
// unaligned head and the tail (fewer than 4 + 3 voxels) by warp 0 of block 0.
template <typename Fn>
__device__ __forceinline__ void for_each_voxel(const float* __restrict__ v, long long n, Fn&& fn) {
    const int lane = threadIdx.x & 31;
    long long head = (long long)((((uint32_t)(uintptr_t)v) & 15u) ? (16u - (((uint32_t)(uintptr_t)v) & 15u)) >> 2 : 0u);
    if (head > n) head = n;
    const float4* __restrict__ v4 = reinterpret_cast<const float4*>(v + head);
    const long long n4 = (n - head) >> 2;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    const long long gw = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    constexpr int U = 4;
    for (long long base = gw * 32 * U; base < n4; base += warps * 32 * U) {
        float4 q[U];
        bool ok[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long long i = base + u * 32 + lane;
            ok[u] = i < n4;
            q[u] = ok[u] ? __ldg(v4 + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            fn(q[u].x, ok[u]);
            fn(q[u].y, ok[u]);
            fn(q[u].z, ok[u]);
            fn(q[u].w, ok[u]);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        const long long t0 = head + (n4 << 2);             // tail: [t0, n), fewer than 4
        const long long i = lane < head ? lane : t0 + (lane - 4);
        const bool ok = lane < head || (lane >= 4 && lane < 8 && i < n);
        fn(ok ? v[i] : 0.f, ok);
    }
}

__global__ void __launch_bounds__(VOL_THREADS)
vol_stats_kernel(const float* __restrict__ v, long long n, VolState* st) {
    unsigned long long nz = 0, nan = 0;
    uint32_t kmin = 0xffffffffu, kmax = 0u;
    for_each_voxel(v, n, [&](float x, bool ok) {
        if (!ok) return;
        nz += (x != 0.f);
        nan += (x != x);
        if (x != 0.f && x == x) {
            const uint32_t k = order_key(x);
            kmin = min(kmin, k);
            kmax = max(kmax, k);
        }
    });
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        nz += __shfl_xor_sync(FULL, nz, o);
        nan += __shfl_xor_sync(FULL, nan, o);
        kmin = min(kmin, __shfl_xor_sync(FULL, kmin, o));
        kmax = max(kmax, __shfl_xor_sync(FULL, kmax, o));
    }
    if ((threadIdx.x & 31) == 0) {
        if (nz) atomicAdd(&st->nonzero, nz);
        if (nan) atomicAdd(&st->nan, nan);
        if (kmin <= kmax) {
            atomicMin(&st->kmin, kmin);
            atomicMax(&st->kmax, kmax);
        }
    }
}

// One radix digit for every requested rank: voxels whose key matches the rank's prefix
// above the digit count into that rank's 2^width bins. shared = 1: all ranks still share
// their prefix, so one histogram serves them all. After the first pass a prefix covers a
// small part of the voxels, so a warp whose voxels match no prefix moves on after one vote.
__global__ void __launch_bounds__(VOL_THREADS)
vol_select_pass_kernel(const float* __restrict__ v, long long n, VolState* st, int n_ranks, int shared,
                       int shift, int width, uint32_t mask_hi) {
    __shared__ unsigned int h[VOL_MAX_RANKS][VOL_DIGITS];
    const int n_hist = shared ? 1 : n_ranks;
    for (int i = threadIdx.x; i < n_hist * VOL_DIGITS; i += blockDim.x) (&h[0][0])[i] = 0u;
    uint32_t pre[VOL_MAX_RANKS];
#pragma unroll
    for (int j = 0; j < VOL_MAX_RANKS; ++j) pre[j] = st->prefix[j] & mask_hi;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint32_t dmask = (1u << width) - 1u;
    for_each_voxel(v, n, [&](float x, bool ok) {
        const bool live = ok && x != 0.f && x == x;
        const uint32_t k = order_key(x);
        const uint32_t hi = k & mask_hi;
        bool m[VOL_MAX_RANKS];
        bool any = false;
#pragma unroll
        for (int j = 0; j < VOL_MAX_RANKS; ++j) {
            m[j] = live && j < n_hist && hi == pre[j];
            any |= m[j];
        }
        if (!__any_sync(FULL, any)) return;                 // warp-uniform
        const uint32_t d = (k >> shift) & dmask;
#pragma unroll
        for (int j = 0; j < VOL_MAX_RANKS; ++j) {
            if (j < n_hist && __any_sync(FULL, m[j]))       // warp-uniform
                warp_run_add(h[j], m[j] ? d : VOL_NONE, lane);
        }
    });
    __syncthreads();
    for (int i = threadIdx.x; i < n_hist * VOL_DIGITS; i += blockDim.x) {
        const unsigned int c = (&h[0][0])[i];
        if (c) atomicAdd(&st->hist[i / VOL_DIGITS][i % VOL_DIGITS], (unsigned long long)c);
    }
}

// Picks each rank's digit from its histogram (exclusive prefix sums over the bins), narrows
// the rank, clears the histograms. One block of 256 threads, 8 bins per thread.
__global__ void __launch_bounds__(256) vol_select_pick_kernel(VolState* st, int n_ranks, int shared, int shift) {
    constexpr int PER = VOL_DIGITS / 256;
    __shared__ unsigned long long warp_tot[8];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int j = 0; j < n_ranks; ++j) {
        const unsigned long long* hj = st->hist[shared ? 0 : j] + t * PER;
        unsigned long long c = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) c += hj[i];
        unsigned long long incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        unsigned long long off = 0;
        for (int w = 0; w < warp; ++w) off += warp_tot[w];
        incl += off;
        unsigned long long excl = incl - c;
        const unsigned long long r = st->rank[j];
        __syncthreads();                    // every thread has read rank[j] and warp_tot
        if (c > 0 && excl <= r && r < incl) {
            int b = 0;
            for (; b < PER - 1 && excl + hj[b] <= r; ++b) excl += hj[b];
            st->prefix[j] |= (uint32_t)(t * PER + b) << shift;
            st->rank[j] = r - excl;
        }
        __syncthreads();
    }
    for (int i = t; i < VOL_MAX_RANKS * VOL_DIGITS; i += 256) (&st->hist[0][0])[i] = 0ull;
}

struct RankList {
    long long r[VOL_MAX_RANKS];
};

__global__ void vol_select_init_kernel(VolState* st, RankList ranks, int n_ranks, uint32_t prefix) {
    const int j = threadIdx.x;
    if (j < VOL_MAX_RANKS) {
        st->prefix[j] = prefix;
        st->rank[j] = j < n_ranks ? (unsigned long long)ranks.r[j] : 0ull;
    }
    for (int i = threadIdx.x; i < VOL_MAX_RANKS * VOL_DIGITS; i += blockDim.x) (&st->hist[0][0])[i] = 0ull;
}

__global__ void vol_select_out_kernel(const VolState* st, int n_ranks, float* out) {
    const int j = threadIdx.x;
    if (j < n_ranks) out[j] = key_value(st->prefix[j]);
}

// np.histogram(np.clip(v, lo, hi), bins, range) over the non-zero voxels, in FP32: a float
// x lies in bin k (edges[k] <= x < edges[k+1], FP64 edges = numpy's linspace, passed in)
// exactly when lb[k] <= x < lb[k+1], lb[i] = edges[i] rounded up to a float (the smallest
// float >= the edge); the top edge counts in the last bin. The clip is exact the same way:
// x < lo exactly when x < lo rounded up, x > hi exactly when x > hi rounded down, and those
// voxels take the bin of lo / hi. numpy's own rule (index from ((x - first) / (last -
// first)) * bins, corrected by one step against the same edges) lands in the same bin.
//
// The bin is the integer part of (x - first) * bins / (last - first) unless that lies within
// `band` of an integer, where the voxel is compared with the edges themselves; band covers the
// rounding of the product and of the edges (4 roundings of at most bins, and three of the
// largest edge's in units of a bin, each taken twice), and is 1 where a bin is not many
// roundings wide. 134 M voxels of noise and bodies, 512 bins: 322 -> 136 us; the run-merged
// increments that were here before cost more than the conflicts they avoid (a constant volume:
// 340 -> 250 us).
__global__ void __launch_bounds__(VOL_THREADS)
vol_histogram_kernel(const float* __restrict__ v, long long n, const double* __restrict__ edges, int bins,
                     double lo, double hi, unsigned long long* __restrict__ hist) {
    __shared__ unsigned int h[VOL_MAX_BINS + 1];            // [bins]: zeros, NaNs, lanes past the end
    __shared__ float lb[VOL_MAX_BINS + 1];
    __shared__ int s_bin_lo, s_bin_hi;
    if (threadIdx.x == 0) s_bin_lo = s_bin_hi = 0;
    __syncthreads();
    // the bins of the clip bounds themselves: how many inner edges lie at or below them (a search
    // by one thread took 100 us at 2048 bins where both lie in the middle, a volume of one value)
    int below_lo = 0, below_hi = 0;
    for (int i = threadIdx.x; i <= bins; i += blockDim.x) {
        const double e = edges[i];
        h[i] = 0u;
        lb[i] = __double2float_ru(e);
        below_lo += i > 0 && i < bins && e <= lo;
        below_hi += i > 0 && i < bins && e <= hi;
    }
    below_lo = __reduce_add_sync(FULL, below_lo);
    below_hi = __reduce_add_sync(FULL, below_hi);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&s_bin_lo, below_lo);
        atomicAdd(&s_bin_hi, below_hi);
    }
    __syncthreads();
    const float lo_up = __double2float_ru(lo), hi_dn = __double2float_rd(hi);
    const float first = lb[0], last = lb[bins], scale = (float)bins / (last - first);
    const int bin_lo = s_bin_lo, bin_hi = s_bin_hi;
    auto exact = [&](float x) {
        if (x < lo_up) return bin_lo;
        if (x > hi_dn) return bin_hi;
        const float f = (x - first) * scale;
        int k = f >= (float)bins ? bins - 1 : (f > 0.f ? (int)f : 0);
        while (k > 0 && x < lb[k]) --k;
        while (k < bins - 1 && x >= lb[k + 1]) ++k;
        return k;
    };
    float band = (float)bins * 4.8e-7f + scale * fmaxf(fabsf(first), fabsf(last)) * 7.2e-7f;
    if (!(band < 0.25f)) band = 1.f;
    for_each_voxel(v, n, [&](float x, bool ok) {
        // voxels past a clip bound land on an outer edge (or an inner one, lo == hi): exact
        const float f = (fminf(fmaxf(x, lo_up), hi_dn) - first) * scale;
        int k = (int)f;
        const float part = f - (float)k;
        const bool count = ok && fabsf(x) > 0.f;            // not zero, not NaN
        if (!(part > band && part < 1.f - band) && count) k = exact(x);
        atomicAdd(h + (count ? k : bins), 1u);
    });
    __syncthreads();
    for (int i = threadIdx.x; i < bins; i += blockDim.x)
        if (h[i]) atomicAdd(&hist[i], (unsigned long long)h[i]);
}

// ------------------------------------------------------------------ tails
// The clip range needs order statistics at 0.1 % and 99.95 %. A sample says where they lie: the
// voxels up to the sample's value 6 standard deviations above the lower rank, and from the
// value as far below the upper one, hold them all but surely (the host checks the counts and
// otherwise takes the radix select over the volume). One pass then counts the non-zero voxels
// and collects both tails, a few per mille, for an exact selection: one read of the volume
// instead of four. 134 M voxels: 30 us sample, 106 us pass (82 us at the copy rate), 34 us
// selection, against 124 us stats and 728 us of select passes. A sample of 32768 made the
// tails 0.6 times as large and took 45 us itself.
// Voxels equal to a bracket are counted and not collected: where one value is frequent (clipped,
// masked or whole-numbered volumes) they may be most of the volume (512^3, the whole threshold, by
// the select passes / by tails that hold them / by these: one value 0.71 / 6.05 / 0.71 ms, two
// values 2.06 / 4.68 / 0.75 ms, half the voxels clipped 1.87 / 3.61 / 0.70 ms).
constexpr int TAIL_THREADS = 1024;
constexpr int TAIL_OWN = TAIL_SAMPLE / TAIL_THREADS;

// One count more, by the lanes that call it together: as one where their digits are all the same
// (the leading digits of any volume, all four of a volume of one value, which otherwise took 70 us
// longer).
__device__ __forceinline__ void sample_add(unsigned int* bin, uint32_t digit) {
    const unsigned active = __activemask();
    int same;
    __match_all_sync(active, digit, &same);
    if (!same) atomicAdd(bin, 1u);
    else if ((int)(threadIdx.x & 31) == __ffs(active) - 1) atomicAdd(bin, (unsigned)__popc(active));
}

// One block; each thread holds 16 sampled keys, and both ranks are found by four rounds of
// 8-bit digits.
__global__ void __launch_bounds__(TAIL_THREADS)
vol_tail_sample_kernel(const float* __restrict__ v, long long n, double q_lo, double q_hi, VolState* st) {
    __shared__ unsigned int hist[2][256];
    __shared__ unsigned int s_count, s_prefix[2], s_rank[2];
    const int tid = threadIdx.x;
    const long long m = n < TAIL_SAMPLE ? n : TAIL_SAMPLE;
    const double stride = (double)n / (double)m;
    uint32_t key[TAIL_OWN];
    unsigned int own = 0;
#pragma unroll
    for (int u = 0; u < TAIL_OWN; ++u) {
        const int i = u * TAIL_THREADS + tid;
        // a scattered position of the i-th share: a fixed step would follow the volume's rows
        uint32_t s = (uint32_t)i * 2654435761u;
        s ^= s >> 15;
        s *= 2246822519u;
        s ^= s >> 13;
        long long at = (long long)(((double)i + (double)s * 2.3283064365386963e-10) * stride);
        at = min(at, n - 1);
        const float x = i < m ? v[at] : 0.f;
        const bool live = fabsf(x) > 0.f;
        key[u] = live ? order_key(x) : VOL_NONE;            // VOL_NONE: the key of a NaN, never live
        own += live;
    }
    if (tid == 0) s_count = 0u;
    __syncthreads();
    own = __reduce_add_sync(FULL, own);
    if ((tid & 31) == 0) atomicAdd(&s_count, own);
    __syncthreads();
    const unsigned int live = s_count;
    if (live < 64u) {                                       // nearly all zero: collect everything
        if (tid == 0) {
            st->t_edge[0] = __uint_as_float(0x7f800000u);
            st->t_edge[1] = __uint_as_float(0xff800000u);
        }
        return;
    }
    if (tid < 2) {
        const double q = tid == 0 ? q_lo : q_hi, at = q * (live - 1.0);
        const double margin = 6.0 * sqrt(live * q * (1.0 - q)) + 4.0;
        const double r = tid == 0 ? at + margin : at - margin;
        s_rank[tid] = (unsigned int)fmin(fmax(r, 0.0), live - 1.0);
        s_prefix[tid] = 0u;
    }
    for (int shift = 24; shift >= 0; shift -= 8) {
        if (tid < 512) (&hist[0][0])[tid] = 0u;
        __syncthreads();
        const uint32_t above = shift == 24 ? 0u : 0xffffffffu << (shift + 8);
        const uint32_t p0 = s_prefix[0], p1 = s_prefix[1];
#pragma unroll
        for (int u = 0; u < TAIL_OWN; ++u) {
            if (key[u] == VOL_NONE) continue;
            const uint32_t d = (key[u] >> shift) & 255u;
            if ((key[u] & above) == p0) sample_add(&hist[0][d], d);
            if (p1 != p0 && (key[u] & above) == p1) sample_add(&hist[1][d], d);
        }
        __syncthreads();
        if (tid < 64) {                                     // a warp per rank, 8 bins a lane
            const int t = tid >> 5, lane = tid & 31;
            const unsigned int* ht = hist[p1 != p0 ? t : 0];
            unsigned int c = 0;
#pragma unroll
            for (int b = 0; b < 8; ++b) c += ht[8 * lane + b];
            unsigned int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int y = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += y;
            }
            const unsigned int r = s_rank[t];
            unsigned int excl = incl - c;
            __syncwarp();
            if (c > 0 && excl <= r && r < incl) {
                int b = 0;
                for (; b < 7 && excl + ht[8 * lane + b] <= r; ++b) excl += ht[8 * lane + b];
                s_prefix[t] |= (uint32_t)(8 * lane + b) << shift;
                s_rank[t] = r - excl;
            }
        }
        __syncthreads();
    }
    if (tid < 2) st->t_edge[tid] = key_value(s_prefix[tid]);
}

constexpr int TAIL_LIST = 2048;                  // voxels of each tail a block collects before it hands them on

__global__ void __launch_bounds__(VOL_THREADS) vol_tail_kernel(const float* __restrict__ v, long long n, VolState* st) {
    __shared__ float list[2][TAIL_LIST];
    __shared__ unsigned int s_n[2], s_sum[4];               // s_sum: as t_nonzero, t_nan, t_count
    __shared__ unsigned long long first[2];
    const float low = st->t_edge[0], high = st->t_edge[1];
    if (threadIdx.x < 2) s_n[threadIdx.x] = 0u;
    if (threadIdx.x < 4) s_sum[threadIdx.x] = 0u;
    __syncthreads();
    unsigned int nz = 0, nan = 0, size[2] = {0u, 0u};       // < 2^32: a block sees fewer than 2^32 voxels
    auto put = [&](int t, float x) {
        const unsigned int at = atomicAdd(&s_n[t], 1u);
        if (at < TAIL_LIST) {
            list[t][at] = x;
        } else {                                            // the block's list is full: straight to the tail
            const unsigned long long o = atomicAdd(&st->t_beyond[t], 1ull);
            if (o < TAIL_CAP) st->tail[t][o] = x;
        }
    };
    for_each_voxel(v, n, [&](float x, bool ok) {
        const bool some = ok && x != 0.f;
        nz += some;
        if (some && !(x > low && x < high)) {               // a tail's voxel, or NaN
            nan += x != x;
            if (x <= low) {
                ++size[0];
                if (x < low) put(0, x);
            }
            if (x >= high) {
                ++size[1];
                if (x > high) put(1, x);
            }
        }
    });
    const unsigned int sum[4] = {__reduce_add_sync(FULL, nz), __reduce_add_sync(FULL, nan),
                                 __reduce_add_sync(FULL, size[0]), __reduce_add_sync(FULL, size[1])};
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (sum[i]) atomicAdd(&s_sum[i], sum[i]);
    }
    __syncthreads();
    if (threadIdx.x < 4 && s_sum[threadIdx.x])              // one of each a block: they all meet at one address
        atomicAdd(&st->t_nonzero + threadIdx.x, (unsigned long long)s_sum[threadIdx.x]);
    for (int t = 0; t < 2; ++t) {
        const unsigned int k = min(s_n[t], (unsigned int)TAIL_LIST);
        if (threadIdx.x == 0 && k) first[t] = atomicAdd(&st->t_beyond[t], (unsigned long long)k);
        __syncthreads();
        for (unsigned int i = threadIdx.x; i < k; i += VOL_THREADS)
            if (first[t] + i < TAIL_CAP) st->tail[t][first[t] + i] = list[t][i];
    }
}

// Exact order statistics of the tails, of which a run of voxels equals the edge: a cluster of 8 CTAs per rank, three rounds
// of 11, 11 and 10 bit digits, the digit histograms added through distributed shared memory.
constexpr int TSEL_CLUSTER = 8;
struct TailRanks {
    long long rank[VOL_MAX_RANKS];              // within its tail
    int tail[VOL_MAX_RANKS];
};
__global__ void __launch_bounds__(TAIL_THREADS)
vol_tail_select_kernel(const VolState* __restrict__ st, TailRanks tr, float* __restrict__ out) {
    __shared__ unsigned int hist[VOL_DIGITS], sum[VOL_DIGITS];
    __shared__ unsigned int warp_tot[TAIL_THREADS / 32];
    __shared__ uint32_t s_prefix;
    __shared__ unsigned long long s_rank;
    cg::cluster_group cluster = cg::this_cluster();
    const int crank = (int)cluster.block_rank(), j = blockIdx.x / TSEL_CLUSTER;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = tr.tail[j];
    const float* __restrict__ x = st->tail[t];
    const long long n = (long long)st->t_beyond[t], equal = (long long)st->t_count[t] - n;
    // the edge's own run: the lower tail's last voxels, the upper one's first
    const long long rank = t == 0 ? tr.rank[j] : tr.rank[j] - equal;
    if (t == 0 ? rank >= n : rank < 0) {                    // the same for the whole cluster
        if (crank == 0 && tid == 0) out[j] = st->t_edge[t];
        return;
    }
    const long long per = ((n + TSEL_CLUSTER - 1) / TSEL_CLUSTER + 3) / 4 * 4;
    const long long b = min(n, per * crank), e = min(n, b + per);
    if (tid == 0) {
        s_prefix = 0u;
        s_rank = (unsigned long long)rank;
    }
    for (int shift = 21; shift >= 0; shift = shift == 21 ? 10 : (shift == 10 ? 0 : -1)) {
        const int width = shift == 0 ? 10 : 11;
        const uint32_t above = shift == 21 ? 0u : 0xffffffffu << (shift + width);
        for (int i = tid; i < VOL_DIGITS; i += TAIL_THREADS) hist[i] = 0u;
        __syncthreads();
        const uint32_t prefix = s_prefix, dmask = (1u << width) - 1u;
        for (long long i = b + tid; i < e; i += TAIL_THREADS) {
            const uint32_t k = order_key(x[i]);
            if ((k & above) == prefix) atomicAdd(&hist[(k >> shift) & dmask], 1u);
        }
        cluster.sync();
        for (int i = tid; i < VOL_DIGITS; i += TAIL_THREADS) {
            unsigned int t = 0;
            for (int r = 0; r < TSEL_CLUSTER; ++r) t += cluster.map_shared_rank(hist, r)[i];
            sum[i] = t;
        }
        cluster.sync();                                     // the histograms may be cleared again
        // every CTA picks the digit (2 bins a thread)
        const unsigned int c0 = sum[2 * tid], c = c0 + sum[2 * tid + 1];
        unsigned int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        for (int w = 0; w < warp; ++w) incl += warp_tot[w];
        const unsigned long long r = s_rank, excl = incl - c;
        __syncthreads();
        if (c > 0 && excl <= r && r < incl) {
            const bool second = r >= excl + c0;
            s_prefix = prefix | (uint32_t)(2 * tid + second) << shift;
            s_rank = r - excl - (second ? c0 : 0u);
        }
        __syncthreads();
    }
    if (crank == 0 && tid == 0) out[j] = key_value(s_prefix);
}

static int vol_grid(int* blocks) {
    int dev = 0, sms = 0;
    MR_CUDA_TRY(cudaGetDevice(&dev));
    MR_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    *blocks = 8 * (sms > 0 ? sms : 1);
    return MR_OK;
}

}  // namespace mr

extern "C" int64_t mr_volume_workspace_bytes(void) { return (int64_t)sizeof(mr::VolState); }

extern "C" int mr_volume_stats(const float* vol, int64_t n, void* ws, uint64_t* stats_host, void* stream) {
    if (!ws || n < 0 || (n > 0 && !vol)) return MR_ERR_INVALID;
    if (((uintptr_t)vol & 3u) || ((uintptr_t)ws & 7u)) return MR_ERR_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    mr::VolState* s = static_cast<mr::VolState*>(ws);
    MR_CUDA_TRY(cudaMemsetAsync(s, 0, offsetof(mr::VolState, t_nonzero), st));
    MR_CUDA_TRY(cudaMemsetAsync(&s->kmin, 0xff, sizeof(unsigned int), st));
    int blocks = 0;
    const int rc = mr::vol_grid(&blocks);
    if (rc != MR_OK) return rc;
    if (n > 0) mr::vol_stats_kernel<<<blocks, mr::VOL_THREADS, 0, st>>>(vol, (long long)n, s);
    MR_CUDA_TRY(cudaGetLastError());
    if (stats_host) {
        // nonzero, nan, (kmin | kmax << 32): 24 bytes of the workspace head
        MR_CUDA_TRY(cudaMemcpyAsync(stats_host, s, 3 * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
        MR_CUDA_TRY(cudaStreamSynchronize(st));
    }
    return MR_OK;
}

extern "C" int mr_volume_select(const float* vol, int64_t n, const int64_t* ranks, int32_t n_ranks,
                                uint32_t kmin, uint32_t kmax, void* ws, float* values_dev, void* stream) {
    if (!ws || !ranks || !values_dev || n <= 0 || !vol) return MR_ERR_INVALID;
    if (n_ranks < 1 || n_ranks > mr::VOL_MAX_RANKS || kmin > kmax) return MR_ERR_INVALID;
    mr::RankList rl = {};
    for (int j = 0; j < n_ranks; ++j) {
        if (ranks[j] < 0 || ranks[j] >= n) return MR_ERR_INVALID;
        rl.r[j] = (long long)ranks[j];
    }
    if (((uintptr_t)vol & 3u) || ((uintptr_t)ws & 7u)) return MR_ERR_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    mr::VolState* s = static_cast<mr::VolState*>(ws);
    int blocks = 0;
    const int rc = mr::vol_grid(&blocks);
    if (rc != MR_OK) return rc;
    // bits [0, L) vary between the smallest and largest key; the bits above are known
    const int L = (kmin == kmax) ? 0 : 32 - __builtin_clz(kmin ^ kmax);
    const uint32_t known = L >= 32 ? 0u : ~((1u << L) - 1u);
    mr::vol_select_init_kernel<<<1, 256, 0, st>>>(s, rl, n_ranks, kmin & known);
    for (int top = L, pass = 0; top > 0; top -= mr::VOL_RADIX, ++pass) {
        const int shift = top > mr::VOL_RADIX ? top - mr::VOL_RADIX : 0;
        const int width = top - shift;
        const uint32_t mask_hi = top >= 32 ? 0u : ~((1u << top) - 1u);
        const int shared = pass == 0 ? 1 : 0;
        mr::vol_select_pass_kernel<<<blocks, mr::VOL_THREADS, 0, st>>>(vol, (long long)n, s, n_ranks, shared,
                                                                      shift, width, mask_hi);
        mr::vol_select_pick_kernel<<<1, 256, 0, st>>>(s, n_ranks, shared, shift);
    }
    mr::vol_select_out_kernel<<<1, 32, 0, st>>>(s, n_ranks, values_dev);
    MR_CUDA_TRY(cudaGetLastError());
    return MR_OK;
}

extern "C" int mr_volume_tails(const float* vol, int64_t n, double q_lo, double q_hi, void* ws, uint64_t* stats_host,
                               void* stream) {
    if (!ws || !stats_host || n < 0 || (n > 0 && !vol)) return MR_ERR_INVALID;
    if (!(q_lo >= 0.0 && q_lo <= q_hi && q_hi <= 1.0)) return MR_ERR_INVALID;
    if (((uintptr_t)vol & 3u) || ((uintptr_t)ws & 15u)) return MR_ERR_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    mr::VolState* s = static_cast<mr::VolState*>(ws);
    int blocks = 0;
    const int rc = mr::vol_grid(&blocks);
    if (rc != MR_OK) return rc;
    MR_CUDA_TRY(cudaMemsetAsync(&s->t_nonzero, 0, 6 * sizeof(uint64_t), st));
    if (n > 0) {
        mr::vol_tail_sample_kernel<<<1, mr::TAIL_THREADS, 0, st>>>(vol, (long long)n, q_lo, q_hi, s);
        mr::vol_tail_kernel<<<blocks, mr::VOL_THREADS, 0, st>>>(vol, (long long)n, s);
    }
    MR_CUDA_TRY(cudaGetLastError());
    MR_CUDA_TRY(cudaMemcpyAsync(stats_host, &s->t_nonzero, 4 * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    MR_CUDA_TRY(cudaStreamSynchronize(st));
    return MR_OK;
}

// beyond: how many voxels lie beyond each edge, at most the tails' places; null: the tails of
// stats_host, edges included, have to be no larger than those.
static int tail_select(const int64_t* ranks, int32_t n_ranks, const uint64_t* stats_host, const uint64_t* beyond,
                       void* ws, float* values_dev, void* stream) {
    const uint64_t live = stats_host[0] - stats_host[1];
    mr::TailRanks tr = {};
    for (int j = 0; j < n_ranks; ++j) {
        if (ranks[j] < 0 || (uint64_t)ranks[j] >= live) return MR_ERR_INVALID;
        const uint64_t r = (uint64_t)ranks[j];
        const uint64_t* kept = beyond ? beyond : stats_host + 2;
        if (kept[0] <= mr::TAIL_CAP && r < stats_host[2]) {
            tr.tail[j] = 0;
            tr.rank[j] = (long long)r;
        } else if (kept[1] <= mr::TAIL_CAP && r >= live - stats_host[3]) {
            tr.tail[j] = 1;
            tr.rank[j] = (long long)(r - (live - stats_host[3]));
        } else {
            return MR_ERR_UNSUPPORTED;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n_ranks * mr::TSEL_CLUSTER));
    cfg.blockDim = dim3(mr::TAIL_THREADS);
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = mr::TSEL_CLUSTER;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MR_CUDA_TRY(cudaLaunchKernelEx(&cfg, mr::vol_tail_select_kernel, (const mr::VolState*)ws, tr, values_dev));
    MR_CUDA_TRY(cudaGetLastError());
    return MR_OK;
}

static bool tail_args(const int64_t* ranks, int32_t n_ranks, const uint64_t* stats_host, void* ws, float* values_dev) {
    return ranks && stats_host && ws && values_dev && n_ranks >= 1 && n_ranks <= mr::VOL_MAX_RANKS &&
           !((uintptr_t)ws & 15u);
}

extern "C" int mr_volume_tail_select(const int64_t* ranks, int32_t n_ranks, const uint64_t* stats_host, void* ws,
                                     float* values_dev, void* stream) {
    if (!tail_args(ranks, n_ranks, stats_host, ws, values_dev)) return MR_ERR_INVALID;
    return tail_select(ranks, n_ranks, stats_host, nullptr, ws, values_dev, stream);
}

extern "C" int mr_volume_tail_select_equal(const int64_t* ranks, int32_t n_ranks, const uint64_t* stats_host, void* ws,
                                           float* values_dev, void* stream) {
    if (!tail_args(ranks, n_ranks, stats_host, ws, values_dev)) return MR_ERR_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint64_t beyond[2];
    MR_CUDA_TRY(cudaMemcpyAsync(beyond, static_cast<mr::VolState*>(ws)->t_beyond, sizeof(beyond), cudaMemcpyDeviceToHost, st));
    MR_CUDA_TRY(cudaStreamSynchronize(st));
    return tail_select(ranks, n_ranks, stats_host, beyond, ws, values_dev, stream);
}

extern "C" int mr_volume_histogram(const float* vol, int64_t n, const double* edges_dev, int32_t bins,
                                   double lo, double hi, uint64_t* hist_dev, void* stream) {
    if (!edges_dev || !hist_dev || n < 0 || (n > 0 && !vol)) return MR_ERR_INVALID;
    if (bins < 1 || bins > mr::VOL_MAX_BINS || !(lo <= hi)) return MR_ERR_INVALID;
    if (((uintptr_t)vol & 3u) || ((uintptr_t)edges_dev & 7u) || ((uintptr_t)hist_dev & 7u)) return MR_ERR_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // numpy widens an empty range by 0.5 on each side; the edges passed in already are
    double first = lo, last = hi;
    if (first == last) { first -= 0.5; last += 0.5; }
    const double scale = (double)bins / (last - first);
    if (!(scale > 0.0) || scale != scale || scale > 1.7976931348623157e308) return MR_ERR_INVALID;
    MR_CUDA_TRY(cudaMemsetAsync(hist_dev, 0, sizeof(uint64_t) * (size_t)bins, st));
    int blocks = 0;
    const int rc = mr::vol_grid(&blocks);
    if (rc != MR_OK) return rc;
    if (n > 0)
        mr::vol_histogram_kernel<<<blocks, mr::VOL_THREADS, 0, st>>>(
            vol, (long long)n, edges_dev, bins, lo, hi, reinterpret_cast<unsigned long long*>(hist_dev));
    MR_CUDA_TRY(cudaGetLastError());
    return MR_OK;
}
