// TMA-staged voxel-driven back-projection for regular grids (slices, windows, volumes).
//
// Same result as bp.cu (minirecast recon.py:156-219 semantics), different data path:
//   * per (tile, view) the CTA projects the tile's 4 corners (a planar tile maps to the
//     convex hull of its corners' projections) and derives the detector footprint;
//   * one thread issues cp.async.bulk.tensor 3D box loads (W cols x 8 rows, single CTA,
//     no multicast) of that footprint into a shared-memory stage; loads outside the
//     detector are zero-filled by the TMA unit, which is exactly the reference's
//     "bilinear taps outside [0,R)x[0,C) contribute 0";
//   * a warp-specialised ring of stages: one producer warp computes footprints and issues
//     the TMA loads, eight (four in the slim form) consumer warps back-project; full/empty
//     mbarriers (bounded waits) are the only synchronisation inside the view loop;
//   * the consumer loop is predicate-free: floor via a round-down FMA against a magic
//     constant (FMA pipe only), one unsigned clamp for memory safety, four LDS, lerps;
//   * footprints that miss the detector entirely are skipped (exactly zero), and the
//     rare footprints larger than a stage fall back to predicated global loads.
// Each warp covers 16 (j) x 2 (i) sample patches, which keep its taps on distinct banks for most
// plane orientations.
#include <cooperative_groups.h>
#include <cmath>

#include "bp_stage.cuh"

namespace cg = cooperative_groups;

namespace mr {

constexpr int ST_TI = 32, ST_TJ = 32;        // tile (samples) - same tiling as bp.cu
// Consumer warps of a 32 x 32 tile, and one producer warp. SLIM: half the warps with twice the
// samples each, which share a view's records and waits and run interleaved, and two stages, so
// that five CTAs fit an SM (four of FP32); for launches of many staged tiles (slim_pays).
// Three 512^2 slices, 600 views, BF16: 508 -> 462 us; one 1024^2 slice 990 -> 876 us; ten 601^2
// slices of 160 full-resolution views, FP32: 0.94 to 1.09 times, by how many of their footprints
// are staged. Three stages and four CTAs an SM:
// 459, 819 and 1290 us; a ring of footprint-sized pieces in the place of fixed stages: 518 and
// 910 us (its bookkeeping is in the producer's path, which the consumers wait for).
template <bool SLIM> struct Shape {
    static constexpr int CONSUMERS = SLIM ? 4 : 8;
    static constexpr int THREADS = 32 * (CONSUMERS + 1);
    static constexpr int PPT = 32 / CONSUMERS;    // samples per consumer thread (rows i, i+2, ..)
    static constexpr int CTAS = SLIM ? 5 : 3;     // an SM's, for the register bound
};
constexpr int ST_DI = 2;                      // row step between a thread's samples
constexpr int ST_CLUSTER = 4;                 // CTAs per tile, each a quarter of the views

template <typename T> struct StageGeom;
// Row widths (elements) are 16-byte multiples whose word pitch shifts successive rows
// across banks (88 bf16 = 44 words, 84 f32 = 84 words). MAXB boxes of 8 rows per stage:
// FP32 stages hold 64 rows, so three CTAs fit an SM (80-row FP32 stages allowed two, and
// the three-slice launch ran 18 % slower); taller footprints use the global-load path.
// W2 / W3: the same stage as fewer, wider boxes, for footprints that are wide and flat - a tile
// of an axial slice at a few pixels a sample covers 100 to 250 columns and two or three rows
// (25 axial slices of 192^2, 600 views of 486 x 384, FP32: 1739 us with the global-load path
// for them, 1003 us with these). A variant of the kernel, as the branch costs launches without
// such footprints 8 % (three 512^2 slices 508 -> 549 us).
template <> struct StageGeom<__nv_bfloat16> {
    static constexpr int W = 88, ALIGN = 8, STAGES = 4, MAXB = 10, W2 = 176, MAXB2 = 5, W3 = 248, MAXB3 = 3;
};
template <> struct StageGeom<__half> : StageGeom<__nv_bfloat16> {};
template <> struct StageGeom<float> {
    static constexpr int W = 84, ALIGN = 4, STAGES = 3, MAXB = 8, W2 = 168, MAXB2 = 4, W3 = 252, MAXB3 = 2;
};
enum : int { MODE_WIDE2 = 3, MODE_WIDE3 = 4 };       // beside MODE_STAGED / MODE_GLOBAL / MODE_SKIP


// What the consumer warps read per (tile, view): the local affine maps of the projective
// numerators u, v and denominator w, (value at the tile origin, d/di, d/dj), in stage-local
// coordinates, packed into three 16-byte words:
//   a = (u0, u_i, u_j, v0), b = (v_i, v_j, w0, w_i), c = (w_j, qscale, max tap offset, mode)
struct __align__(16) ViewRec {
    float4 a, b, c;
};
// The producer's copy adds the TMA box origin and count.
struct __align__(16) ViewMeta {
    ViewRec rec;
    int x0, r0, nbox, mode;
};

__device__ __forceinline__ bool in_box_fp64_t(const mr_grid& g, int i, int j) {
    const double aj = __dmul_rn((double)j - g.mask_half, g.mask_delta);
    const double ai = __dmul_rn((double)i - g.mask_half, g.mask_delta);
    bool ok = true;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const double p = __dadd_rn(__dadd_rn(g.mask_c[e], __dmul_rn(aj, g.mask_ej[e])),
                                   __dmul_rn(ai, g.mask_ei[e]));
        ok = ok && (fabs(p) <= g.box[e]);
    }
    return ok;
}

// Where one tile lies in a view, and how its footprint is read: the affine maps of column and
// row numerator and depth, (value at the tile origin, d/di, d/dj), and the boxes.
struct Footprint {
    float3 au, av, aw;
    int x0, r0, nbox, mode;
};
template <int KIND, bool WIDE, typename T>
__host__ __device__ __forceinline__ Footprint footprint(const mr_view& V, const mr_grid& g, float ox, float oy,
                                                        float oz, int di_max, int dj_max, int R, int C) {
    constexpr int W = StageGeom<T>::W;
    float pu[4], pv[4];
    view_map(V, g, R, C, pu, pv);
    auto aff = [&](const float* m) {
        return make_float3(mul_add(m[0], ox, mul_add(m[1], oy, mul_add(m[2], oz, m[3]))),
                           mul_add(m[0], g.step_i[0], mul_add(m[1], g.step_i[1], m[2] * g.step_i[2])),
                           mul_add(m[0], g.step_j[0], mul_add(m[1], g.step_j[1], m[2] * g.step_j[2])));
    };
    float3 au = aff(pu), av = aff(pv), aw = aff(V.pw);
    if (KIND == MR_CONE && V.qscale != 1.f) {
        // col = nu/nw and row = nv/nw are scale free, 1/nw^2 picks up qscale
        const float k = rsqrtf(V.qscale);
        au = make_float3(au.x * k, au.y * k, au.z * k);
        av = make_float3(av.x * k, av.y * k, av.z * k);
        aw = make_float3(aw.x * k, aw.y * k, aw.z * k);
    }
    float cmin = 3e38f, cmax = -3e38f, rmin = 3e38f, rmax = -3e38f;
    bool behind = false;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float di = (c & 1) ? (float)di_max : 0.f;
        const float dj = (c & 2) ? (float)dj_max : 0.f;
        const float w = mul_add(di, aw.y, mul_add(dj, aw.z, aw.x));
        float cc = mul_add(di, au.y, mul_add(dj, au.z, au.x));
        float rr = mul_add(di, av.y, mul_add(dj, av.z, av.x));
        if (KIND == MR_CONE) {
            behind |= !(w > 1e-3f);
            const float inv = 1.f / w;
            cc *= inv;
            rr *= inv;
        }
        cmin = fminf(cmin, cc); cmax = fmaxf(cmax, cc);
        rmin = fminf(rmin, rr); rmax = fmaxf(rmax, rr);
    }
    int mode = MODE_GLOBAL, x0 = 0, r0 = 0, nbox = 0;
    if (!behind && cmax == cmax && rmax == rmax && cmin == cmin && rmin == rmin) {
        if (cmax < -2.f || cmin > (float)C + 1.f || rmax < -2.f || rmin > (float)R + 1.f) {
            mode = MODE_SKIP;
        } else if (cmax - cmin < (float)(W - StageGeom<T>::ALIGN - 4) &&
                   rmax - rmin < (float)(ST_BOX_H * StageGeom<T>::MAXB - 4)) {
            x0 = ((int)floorf(cmin) - 1) & ~(StageGeom<T>::ALIGN - 1);
            r0 = (int)floorf(rmin) - 1;
            const int rows = (int)floorf(rmax) + 3 - r0;
            nbox = (rows + ST_BOX_H - 1) / ST_BOX_H;
            if ((int)floorf(cmax) + 3 - x0 <= W && nbox <= StageGeom<T>::MAXB) mode = MODE_STAGED;
        }
        if (WIDE && mode == MODE_GLOBAL && cmax - cmin < 256.f && rmax - rmin < 64.f) {
            x0 = ((int)floorf(cmin) - 1) & ~(StageGeom<T>::ALIGN - 1);
            r0 = (int)floorf(rmin) - 1;
            const int wide = (int)floorf(cmax) + 3 - x0;
            nbox = ((int)floorf(rmax) + 3 - r0 + ST_BOX_H - 1) / ST_BOX_H;
            if (wide <= StageGeom<T>::W2 && nbox <= StageGeom<T>::MAXB2) mode = MODE_WIDE2;
            else if (wide <= StageGeom<T>::W3 && nbox <= StageGeom<T>::MAXB3) mode = MODE_WIDE3;
        }
    }
    return Footprint{au, av, aw, x0, r0, nbox, mode};
}

// Per-view footprint + local affine coefficients of one tile (computed by one lane of
// the producer warp).
template <int KIND, bool WIDE, typename T>
__device__ __forceinline__ ViewMeta view_meta(const mr_view& V, const mr_grid& g, float ox, float oy,
                                              float oz, int di_max, int dj_max, int R, int C) {
    constexpr int W = StageGeom<T>::W;
    const Footprint f = footprint<KIND, WIDE, T>(V, g, ox, oy, oz, di_max, dj_max, R, C);
    const float3 au = f.au, av = f.av, aw = f.aw;
    const int x0 = f.x0, r0 = f.r0, nbox = f.nbox, mode = f.mode;
    ViewMeta m;
    float3 cu = au, cv = av;
    if (mode == MODE_STAGED) {
        const float fx0 = (float)x0, fr0 = (float)r0;
        cu = make_float3(fmaf(-fx0, aw.x, au.x), fmaf(-fx0, aw.y, au.y), fmaf(-fx0, aw.z, au.z));
        cv = make_float3(fmaf(-fr0, aw.x, av.x), fmaf(-fr0, aw.y, av.y), fmaf(-fr0, aw.z, av.z));
    }
    // largest byte offset of a tap pair's left tap inside the staged boxes
    constexpr int ESZ = (int)sizeof(T);
    const int wcols = mode == MODE_WIDE2 ? StageGeom<T>::W2 : (mode == MODE_WIDE3 ? StageGeom<T>::W3 : W);
    const bool boxes = mode != MODE_GLOBAL && mode != MODE_SKIP;
    const uint32_t maxoff = boxes ? (uint32_t)(nbox * wcols * ST_BOX_H * ESZ - (wcols + 1) * ESZ - ESZ) : 0u;
    m.rec.a = make_float4(cu.x, cu.y, cu.z, cv.x);
    m.rec.b = make_float4(cv.y, cv.z, aw.x, aw.y);
    m.rec.c = make_float4(aw.z, V.qscale, __uint_as_float(maxoff), __int_as_float(mode));
    m.x0 = x0; m.r0 = r0; m.nbox = nbox; m.mode = mode;
    return m;
}

// Warp-specialised: the first warps consume (eight of 4 samples a thread or, SLIM, four of 8: one
// 32 x 32 tile), the last one produces. Stage s carries the TMA data and its ViewMeta; full[s] (1 arrival + TMA bytes)
// and empty[s] (one arrival per consumer warp) hand it back and forth. No CTA-wide barrier
// in the view loop, so consumer warps may run up to S views apart.
// A thread-block cluster of ST_CLUSTER CTAs shares one tile: CTA rank r back-projects the
// r-th quarter of the views and rank 0 sums the partials from the others' shared memory
// (DSMEM) in rank order - deterministic, no atomics, no scratch - and writes the tile.
// Three CTAs fit an SM (shared memory; SLIM: five, four of FP32); the launch bound says so, or
// ptxas aims at four and spills the FP32 variant to fit its registers. SLIM spills 4 bytes.
template <int KIND, bool WIDE, bool SLIM, typename T>
__global__ void __launch_bounds__(Shape<SLIM>::THREADS, Shape<SLIM>::CTAS)
bp_staged_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap tmap2,
                 const __grid_constant__ CUtensorMap tmap3, const T* __restrict__ ring, int R, int C,
                 int pitch, long long slot_stride, int n_slots, const mr_view* __restrict__ views,
                 const mr_grid* __restrict__ grids, const mr_tile* __restrict__ tiles,
                 float* __restrict__ out, int* status, const int64_t* __restrict__ n_tiles_dev,
                 unsigned int* __restrict__ counter, long long tile_cap) {
    constexpr int W = StageGeom<T>::W;
    constexpr int ST_CONSUMERS = Shape<SLIM>::CONSUMERS, ST_PPT = Shape<SLIM>::PPT;
    constexpr int S = SLIM ? 2 : StageGeom<T>::STAGES;
    constexpr int ESZ = (int)sizeof(T);
    constexpr int STAGE_BYTES = W * ST_BOX_H * StageGeom<T>::MAXB * ESZ;
    constexpr int BOX_BYTES = W * ST_BOX_H * ESZ;
    // every TMA destination (stage start + b * BOX_BYTES) must be 128-byte aligned
    static_assert(BOX_BYTES % 128 == 0 && STAGE_BYTES % 128 == 0, "TMA box / stage not 128-byte aligned");
    constexpr int W2 = StageGeom<T>::W2, W3 = StageGeom<T>::W3;
    constexpr int BOX2_BYTES = W2 * ST_BOX_H * ESZ, BOX3_BYTES = W3 * ST_BOX_H * ESZ;
    static_assert(BOX2_BYTES % 128 == 0 && BOX3_BYTES % 128 == 0 && W2 <= 256 && W3 <= 256, "wide TMA boxes");
    static_assert(BOX2_BYTES * StageGeom<T>::MAXB2 <= STAGE_BYTES && BOX3_BYTES * StageGeom<T>::MAXB3 <= STAGE_BYTES,
                  "wide boxes fit the stage");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    // TMA destinations must be 128-byte aligned: round the dynamic buffer up (the host
    // allocates 128 spare bytes), whatever static shared memory precedes it.
    unsigned char* stages = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
    ViewRec* meta_ring = reinterpret_cast<ViewRec*>(stages + S * STAGE_BYTES);     // S
    ViewMeta* meta_new = reinterpret_cast<ViewMeta*>(meta_ring + S);                // 32
    uint64_t* full = reinterpret_cast<uint64_t*>(meta_new + 32);                    // S
    uint64_t* empty = full + S;                                                      // S
    float4* partial = reinterpret_cast<float4*>(empty + S);                          // cluster sum: 1024 floats
    __shared__ mr_grid s_g;
    // wide modes keep detector coordinates (the arithmetic of the global path, bit for bit): the
    // offset that the magic-constant bits of (r0, x0) have
    __shared__ uint32_t origin_ring[S];

    cg::cluster_group cluster = cg::this_cluster();
    const int crank = (int)cluster.block_rank();
    const int csize = (int)cluster.num_blocks();
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const bool producer = warp == ST_CONSUMERS;
    __shared__ unsigned int s_next;
    if (tid < S) {
        mbar_init(&full[tid], 1);
        mbar_init(&empty[tid], ST_CONSUMERS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    uint32_t used = 0;              // views this CTA has put through the stage ring so far

    // One tile per cluster (counter == nullptr), or persistent: clusters pull tile indices
    // from the device work counter until it passes *n_tiles_dev.
    for (int iter = 0;; ++iter) {
        long long tile_idx;
        if (counter) {
            // rank 0 pushes the tile index into every CTA's own shared memory before the
            // barrier; after it each CTA reads only its local copy, so no CTA touches a
            // peer's shared memory once the cluster may start exiting (the final break)
            if (crank == 0 && tid == 0) {
                const unsigned int nx = atomicAdd(counter, 1u);
                for (int r = 0; r < csize; ++r) *cluster.map_shared_rank(&s_next, r) = nx;
            }
            cluster.sync();
            tile_idx = (long long)s_next;
            // the device count is clamped to the capacity of the tile buffer
            if (tile_idx >= min((long long)*n_tiles_dev, tile_cap)) break;
        } else {
            if (iter > 0) break;
            tile_idx = (long long)(blockIdx.x / csize);
        }
        const mr_tile t = tiles[tile_idx];
        __syncthreads();                    // previous tile's readers of s_g are done
        if (tid < (int)(sizeof(mr_grid) / 4))
            reinterpret_cast<int*>(&s_g)[tid] = reinterpret_cast<const int*>(grids + t.grid)[tid];
        __syncthreads();
        const mr_grid& g = s_g;
        // this CTA's share of the views: [v_begin, v_end)
        int first, count;                   // the grid's slots [first, first + count)
        grid_view_range(g.view_begin, g.n_views, n_slots, &first, &count);
        const int v_begin = first + (int)(((long long)count * crank) / csize);
        const int v_end = first + (int)(((long long)count * (crank + 1)) / csize);
        const int nv = v_end - v_begin;

        const float ox = g.origin[0] + t.i0 * g.step_i[0] + t.j0 * g.step_j[0] + t.k * g.step_k[0];
        const float oy = g.origin[1] + t.i0 * g.step_i[1] + t.j0 * g.step_j[1] + t.k * g.step_k[1];
        const float oz = g.origin[2] + t.i0 * g.step_i[2] + t.j0 * g.step_j[2] + t.k * g.step_k[2];
        // warp w covers columns 16 (w & 1) .. + 15 and 8 (SLIM: 16) rows from those of w >> 1; its
        // p-th sample step is a 16 x 2 patch (rows ty + 2p). The patch shape keeps the 32
        // lanes' bilinear taps on distinct shared-memory banks for most plane orientations
        // (1.10 wavefronts per 16-bit tap load on the bench slices, 1.35 for 8 x 4 patches)
        // and makes each half-warp's output a 64-byte row segment.
        const int tx = ((warp & 1) << 4) | (lane & 15);
        const int ty = (warp >> 1) * (2 * ST_PPT) + (lane >> 4);
        bool inside[ST_PPT];
        bool any = false;
#pragma unroll
        for (int p = 0; p < ST_PPT; ++p) {
            const int i = t.i0 + ty + ST_DI * p, j = t.j0 + tx;
            bool ok = !producer && i < g.n_i && j < g.n_j;
            if (ok && (g.flags & MR_GRID_MASK_BOX)) ok = in_box_fp64_t(g, i, j);
            inside[p] = ok;
            any |= ok;
        }
        const bool tile_live = __syncthreads_or(any) != 0;
        // warp-uniform: a 16 x 2 sample patch wholly outside the box is not computed. SLIM: only
        // if all of the warp's are (a branch per pair keeps the pairs from running interleaved)
        bool wlive[ST_PPT], wany = false;
#pragma unroll
        for (int p = 0; p < ST_PPT; ++p) {
            wlive[p] = __any_sync(0xffffffffu, inside[p]);
            wany |= wlive[p];
        }

        if (producer && tile_live) {
            const int di_max = min(ST_TI, g.n_i - t.i0) - 1;
            const int dj_max = min(ST_TJ, g.n_j - t.j0) - 1;
            for (int vb = 0; vb < nv; vb += 32) {
                const int cnt = min(32, nv - vb);
                __syncwarp();
                if (lane < cnt)
                    meta_new[lane] = view_meta<KIND, WIDE, T>(views[v_begin + vb + lane], g, ox, oy, oz, di_max,
                                                        dj_max, R, C);
                __syncwarp();
                // lane 0 frees and arms the stage, then lane b issues the copy of box b: the
                // boxes of a view go out in one warp instruction instead of one after another
                for (int l = 0; l < cnt; ++l) {
                    const uint32_t ua = used + (uint32_t)(vb + l);          // absolute stage use
                    const int s = (int)(ua % S);
                    const uint32_t u = ua / S;
                    const int mode = meta_new[l].mode, nbox = meta_new[l].nbox;
                    if (lane == 0) {
                        if (u > 0) mbar_wait(&empty[s], (u - 1) & 1u, status);
                        meta_ring[s] = meta_new[l].rec;
                        if (mode == MODE_STAGED) {
                            mbar_arrive_tx(&full[s], (uint32_t)(nbox * BOX_BYTES));
                        } else if (WIDE && (mode == MODE_WIDE2 || mode == MODE_WIDE3)) {
                            const bool w2 = mode == MODE_WIDE2;
                            origin_ring[s] = (uint32_t)(MAGIC_BITS + meta_new[l].r0) * (uint32_t)((w2 ? W2 : W3) * ESZ) +
                                             (uint32_t)(MAGIC_BITS + meta_new[l].x0) * (uint32_t)ESZ;
                            mbar_arrive_tx(&full[s], (uint32_t)(nbox * (w2 ? BOX2_BYTES : BOX3_BYTES)));
                        } else {
                            mbar_arrive(&full[s]);
                        }
                    }
                    __syncwarp();                   // the stage is free and armed for every lane
                    if (mode == MODE_STAGED) {
                        if (lane < nbox)
                            tma_load_3d(stages + s * STAGE_BYTES + lane * BOX_BYTES, &tmap, meta_new[l].x0,
                                        meta_new[l].r0 + lane * ST_BOX_H, v_begin + vb + l, &full[s]);
                    } else if (WIDE && mode == MODE_WIDE2 && lane < nbox) {
                        tma_load_3d(stages + s * STAGE_BYTES + lane * BOX2_BYTES, &tmap2, meta_new[l].x0,
                                    meta_new[l].r0 + lane * ST_BOX_H, v_begin + vb + l, &full[s]);
                    } else if (WIDE && mode == MODE_WIDE3 && lane < nbox) {
                        tma_load_3d(stages + s * STAGE_BYTES + lane * BOX3_BYTES, &tmap3, meta_new[l].x0,
                                    meta_new[l].r0 + lane * ST_BOX_H, v_begin + vb + l, &full[s]);
                    }
                }
            }
        }

        // sample p sits in pair p / 2, lane p % 2 (pairs of rows i and i + ST_DI)
        float2 acc2[ST_PPT / 2];
        float2 fi2[ST_PPT / 2];
#pragma unroll
        for (int h = 0; h < ST_PPT / 2; ++h) {
            acc2[h] = make_float2(0.f, 0.f);
            fi2[h] = make_float2((float)(ty + 2 * ST_DI * h), (float)(ty + 2 * ST_DI * h + ST_DI));
        }
        if (!producer && tile_live) {
            const float fj = (float)tx;
            int s = (int)(used % S);                    // stage of view 0 of this tile
            uint32_t phase = (used / S) & 1u;           // and the parity of its fill
            for (int v = 0; v < nv; ++v) {
                mbar_wait(&full[s], phase, status);
                const ViewRec m = meta_ring[s];
                const int mode = __float_as_int(m.c.w);
                const float bu = fmaf(fj, m.a.z, m.a.x);
                const float bv = fmaf(fj, m.b.y, m.a.w);
                const float bw = fmaf(fj, m.c.x, m.b.z);
                if (mode == MODE_STAGED && (!SLIM || wany)) {
                    const uint32_t base = smem_u32(stages + s * STAGE_BYTES);
                    const uint32_t maxoff = __float_as_uint(m.c.z);
                    // byte offset = (bits_r - MAGIC_BITS) * W*ESZ + (bits_c - MAGIC_BITS) * ESZ
                    const uint32_t kofs = (uint32_t)MAGIC_BITS * (uint32_t)(W * ESZ + ESZ);
                    // Two samples (rows i and i + 2) per packed f32x2 instruction: every
                    // component is the scalar FMA / add / multiply it replaces, so the result
                    // is the same bit for bit; only the issue slots halve.
                    const float2 cuy = make_float2(m.a.y, m.a.y), cvy = make_float2(m.b.x, m.b.x);
                    const float2 cwy = make_float2(m.b.w, m.b.w);
                    const float2 bu2 = make_float2(bu, bu), bv2 = make_float2(bv, bv), bw2 = make_float2(bw, bw);
#pragma unroll
                    for (int h = 0; h < ST_PPT / 2; ++h) {
                        if (!SLIM && !(wlive[2 * h] | wlive[2 * h + 1])) continue;
                        const float2 nu = __ffma2_rn(fi2[h], cuy, bu2);
                        const float2 nv2 = __ffma2_rn(fi2[h], cvy, bv2);
                        float2 r = make_float2(1.f, 1.f), yc, yr, fc, fr;
                        if (KIND == MR_CONE) {
                            const float2 w = __ffma2_rn(fi2[h], cwy, bw2);
                            r = make_float2(rcp_approx(w.x), rcp_approx(w.y));
                            yc = __ffma2_rd(nu, r, kMagic2);
                            yr = __ffma2_rd(nv2, r, kMagic2);
                            // MAGIC - y is exact; fma(y, -1, MAGIC) is that subtraction
                            fc = __ffma2_rn(nu, r, __ffma2_rn(yc, kNeg2, kMagic2));
                            fr = __ffma2_rn(nv2, r, __ffma2_rn(yr, kNeg2, kMagic2));
                        } else {
                            yc = __fadd2_rd(nu, kMagic2);
                            yr = __fadd2_rd(nv2, kMagic2);
                            fc = __fadd2_rn(nu, __ffma2_rn(yc, kNeg2, kMagic2));
                            fr = __fadd2_rn(nv2, __ffma2_rn(yr, kNeg2, kMagic2));
                        }
                        uint32_t a[2];
                        a[0] = base + min((uint32_t)__float_as_int(yr.x) * (uint32_t)(W * ESZ) +
                                              (uint32_t)__float_as_int(yc.x) * (uint32_t)ESZ - kofs, maxoff);
                        a[1] = base + min((uint32_t)__float_as_int(yr.y) * (uint32_t)(W * ESZ) +
                                              (uint32_t)__float_as_int(yc.y) * (uint32_t)ESZ - kofs, maxoff);
                        float2 q00, q10, d0, d1;
                        if constexpr (sizeof(T) == 2) {
                            // the right taps stay 16-bit: one mixed-precision subtraction each
                            // (16-bit values widen exactly, so it is the FP32 difference)
                            q00 = make_float2(lds_elem<T>(a[0]), lds_elem<T>(a[1]));
                            q10 = make_float2(lds_elem<T>(a[0] + W * ESZ), lds_elem<T>(a[1] + W * ESZ));
                            d0 = make_float2(sub16_f32<T>(lds_u16(a[0] + ESZ), q00.x),
                                             sub16_f32<T>(lds_u16(a[1] + ESZ), q00.y));
                            d1 = make_float2(sub16_f32<T>(lds_u16(a[0] + W * ESZ + ESZ), q10.x),
                                             sub16_f32<T>(lds_u16(a[1] + W * ESZ + ESZ), q10.y));
                        } else {
                            q00 = make_float2(lds_elem<T>(a[0]), lds_elem<T>(a[1]));
                            q10 = make_float2(lds_elem<T>(a[0] + W * ESZ), lds_elem<T>(a[1] + W * ESZ));
                            const float2 q01 = make_float2(lds_elem<T>(a[0] + ESZ), lds_elem<T>(a[1] + ESZ));
                            const float2 q11 = make_float2(lds_elem<T>(a[0] + W * ESZ + ESZ),
                                                           lds_elem<T>(a[1] + W * ESZ + ESZ));
                            d0 = __ffma2_rn(q00, kNeg2, q01);          // q01 - q00
                            d1 = __ffma2_rn(q10, kNeg2, q11);          // q11 - q10
                        }
                        const float2 ta = __ffma2_rn(fc, d0, q00);
                        const float2 tb = __ffma2_rn(fc, d1, q10);
                        const float2 val = __ffma2_rn(fr, __ffma2_rn(ta, kNeg2, tb), ta);
                        const float2 wgt = KIND == MR_CONE ? __fmul2_rn(r, r) : make_float2(m.c.y, m.c.y);
                        acc2[h] = __ffma2_rn(wgt, val, acc2[h]);
                    }
                } else if (WIDE && (mode == MODE_WIDE2 || mode == MODE_WIDE3)) {
                    // the global path's arithmetic on taps from a wide box
                    const uint32_t base = smem_u32(stages + s * STAGE_BYTES);
                    const uint32_t maxoff = __float_as_uint(m.c.z), kofs = origin_ring[s];
                    const uint32_t pitch_b = mode == MODE_WIDE2 ? W2 * ESZ : W3 * ESZ;
#pragma unroll
                    for (int h = 0; h < ST_PPT / 2; ++h) {
                        if (!(wlive[2 * h] | wlive[2 * h + 1])) continue;
                        float2 col = __ffma2_rn(fi2[h], make_float2(m.a.y, m.a.y), make_float2(bu, bu));
                        float2 row = __ffma2_rn(fi2[h], make_float2(m.b.x, m.b.x), make_float2(bv, bv));
                        float2 r = make_float2(1.f, 1.f);
                        if (KIND == MR_CONE) {
                            const float2 w = __ffma2_rn(fi2[h], make_float2(m.b.w, m.b.w), make_float2(bw, bw));
                            r = make_float2(rcp_approx(w.x), rcp_approx(w.y));
                            col = __fmul2_rn(col, r);
                            row = __fmul2_rn(row, r);
                        }
                        const float2 yc = __fadd2_rd(col, kMagic2), yr = __fadd2_rd(row, kMagic2);
                        const float2 fc = __ffma2_rn(__fadd2_rn(yc, make_float2(-MAGIC, -MAGIC)), kNeg2, col);
                        const float2 fr = __ffma2_rn(__fadd2_rn(yr, make_float2(-MAGIC, -MAGIC)), kNeg2, row);
                        const uint32_t a0 = base + min((uint32_t)__float_as_int(yr.x) * pitch_b +
                                                           (uint32_t)__float_as_int(yc.x) * (uint32_t)ESZ - kofs, maxoff);
                        const uint32_t a1 = base + min((uint32_t)__float_as_int(yr.y) * pitch_b +
                                                           (uint32_t)__float_as_int(yc.y) * (uint32_t)ESZ - kofs, maxoff);
                        const float2 q00 = make_float2(lds_elem<T>(a0), lds_elem<T>(a1));
                        const float2 q01 = make_float2(lds_elem<T>(a0 + ESZ), lds_elem<T>(a1 + ESZ));
                        const float2 q10 = make_float2(lds_elem<T>(a0 + pitch_b), lds_elem<T>(a1 + pitch_b));
                        const float2 q11 = make_float2(lds_elem<T>(a0 + pitch_b + ESZ), lds_elem<T>(a1 + pitch_b + ESZ));
                        const float2 ta = __ffma2_rn(fc, __ffma2_rn(q00, kNeg2, q01), q00);
                        const float2 tb = __ffma2_rn(fc, __ffma2_rn(q10, kNeg2, q11), q10);
                        const float2 val = __ffma2_rn(fr, __ffma2_rn(ta, kNeg2, tb), ta);
                        const float2 wgt = KIND == MR_CONE ? __fmul2_rn(r, r) : make_float2(m.c.y, m.c.y);
                        acc2[h] = __ffma2_rn(wgt, val, acc2[h]);
                    }
                } else if (mode == MODE_GLOBAL) {
                    const T* q = ring + (long long)(v_begin + v) * slot_stride;
#pragma unroll
                    for (int p = 0; p < ST_PPT; ++p) {
                        if (!wlive[p]) continue;
                        const float fi = (float)(ty + ST_DI * p);
                        const float nu = fmaf(fi, m.a.y, bu);
                        const float nvv = fmaf(fi, m.b.x, bv);
                        float& ap = (p & 1) ? acc2[p >> 1].y : acc2[p >> 1].x;
                        if (KIND == MR_CONE) {
                            const float r = rcp_approx(fmaf(fi, m.b.w, bw));
                            ap = fmaf(r * r, bilerp_global(q, R, C, pitch, nvv * r, nu * r), ap);
                        } else {
                            ap = fmaf(m.c.y, bilerp_global(q, R, C, pitch, nvv, nu), ap);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[s]);      // this warp is done with stage s
                if (++s == S) {
                    s = 0;
                    phase ^= 1u;
                }
            }
        }
        if (tile_live) used += (uint32_t)nv;

        // ---- cluster reduction of the view-quarter partial sums (rank order), rank 0 writes
        float acc[ST_PPT];
#pragma unroll
        for (int p = 0; p < ST_PPT; ++p) acc[p] = (p & 1) ? acc2[p >> 1].y : acc2[p >> 1].x;
        if (csize > 1) {
            if (!producer) {
#pragma unroll
                for (int q = 0; q < ST_PPT / 4; ++q)
                    partial[q * (32 * ST_CONSUMERS) + tid] =
                        make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
            }
            cluster.sync();
            if (crank == 0 && !producer) {
                for (int r = 1; r < csize; ++r) {
#pragma unroll
                    for (int q = 0; q < ST_PPT / 4; ++q) {
                        const float4 o = cluster.map_shared_rank(partial, r)[q * (32 * ST_CONSUMERS) + tid];
                        acc[4 * q] += o.x; acc[4 * q + 1] += o.y; acc[4 * q + 2] += o.z; acc[4 * q + 3] += o.w;
                    }
                }
            }
        }
        if (crank == 0 && !producer) {
#pragma unroll
            for (int p = 0; p < ST_PPT; ++p) {
                const int i = t.i0 + ty + ST_DI * p, j = t.j0 + tx;
                if (i < g.n_i && j < g.n_j) {
                    const long long o = g.out_offset + (long long)i * g.out_stride_i +
                                        (long long)j * g.out_stride_j + (long long)t.k * g.out_stride_k;
                    const float val = inside[p] ? acc[p] * g.scale : 0.f;
                    out[o] = g.accumulate ? out[o] + val : val;
                }
            }
        }
        if (csize > 1) cluster.sync();      // keep every partial alive until rank 0 has read it
    }
}

// ---------------------------------------------------------------- host side
template <int KIND, bool WIDE, bool SLIM, typename T>
static int launch_staged(const mr_ring* ring, const mr_view* views, const mr_grid* grids,
                         const mr_tile* tiles, int64_t n_tiles, float* out, int* status, cudaStream_t st,
                         const int64_t* n_tiles_dev = nullptr, unsigned int* counter = nullptr) {
    CUtensorMap map;
    int rc = make_ring_map<T>(ring, StageGeom<T>::W, &map);
    CUtensorMap map2 = map, map3 = map;           // read by WIDE alone
    if (WIDE && rc == MR_OK) rc = make_ring_map<T>(ring, StageGeom<T>::W2, &map2);
    if (WIDE && rc == MR_OK) rc = make_ring_map<T>(ring, StageGeom<T>::W3, &map3);
    if (rc != MR_OK) return rc;
    constexpr int S = SLIM ? 2 : StageGeom<T>::STAGES;
    const size_t smem = (size_t)S * StageGeom<T>::W * ST_BOX_H * StageGeom<T>::MAXB * sizeof(T) +
                        S * sizeof(ViewRec) + 32 * sizeof(ViewMeta) + 2 * S * sizeof(uint64_t) +
                        ST_TI * ST_TJ * sizeof(float) + 128;
    auto kern = bp_staged_kernel<KIND, WIDE, SLIM, T>;
    MR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(Shape<SLIM>::THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ST_CLUSTER;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (counter) {
        // persistent: as many clusters as fit at once, pulling tiles from the counter
        int clusters = 0;
        cfg.gridDim = dim3(ST_CLUSTER);
        MR_CUDA_TRY(cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg));
        if (clusters < 1) clusters = 1;
        if ((int64_t)clusters > n_tiles) clusters = (int)(n_tiles > 0 ? n_tiles : 1);
        MR_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(unsigned int), st));
        cfg.gridDim = dim3((unsigned)(clusters * ST_CLUSTER));
        MR_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, map, map2, map3, static_cast<const T*>(ring->data), ring->rows, ring->cols,
                                       ring->col_pitch, (long long)ring->slot_stride, (int)ring->n_slots, views,
                                       grids, tiles, out, status, n_tiles_dev, counter, (long long)n_tiles));
    } else {
        const int64_t max_chunk = 2147483647LL / ST_CLUSTER;
        for (int64_t t0 = 0; t0 < n_tiles; t0 += max_chunk) {
            const int64_t n = (n_tiles - t0) < max_chunk ? (n_tiles - t0) : max_chunk;
            cfg.gridDim = dim3((unsigned)(n * ST_CLUSTER));
            MR_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, map, map2, map3, static_cast<const T*>(ring->data), ring->rows,
                                           ring->cols, ring->col_pitch, (long long)ring->slot_stride,
                                           (int)ring->n_slots, views, grids, tiles + t0, out, status,
                                           (const int64_t*)nullptr, (unsigned int*)nullptr, (long long)n));
        }
    }
    MR_CUDA_TRY(cudaGetLastError());
    return MR_OK;
}

template <bool WIDE, bool SLIM, typename... Args>
static int dispatch_staged(const mr_ring* ring, Args... args) {
    const bool cone = ring->kind == MR_CONE;
    switch (ring->dtype) {
        case MR_F32:
            return cone ? launch_staged<MR_CONE, WIDE, SLIM, float>(ring, args...)
                        : launch_staged<MR_PARALLEL, WIDE, SLIM, float>(ring, args...);
        case MR_BF16:
            return cone ? launch_staged<MR_CONE, WIDE, SLIM, __nv_bfloat16>(ring, args...)
                        : launch_staged<MR_PARALLEL, WIDE, SLIM, __nv_bfloat16>(ring, args...);
        default:
            return cone ? launch_staged<MR_CONE, WIDE, SLIM, __half>(ring, args...)
                        : launch_staged<MR_PARALLEL, WIDE, SLIM, __half>(ring, args...);
    }
}

// Whether a launch of n busy tiles whose footprints are staged is faster with SLIM: its CTAs take
// 1.47 (FP32: 1.24) times as long, but 175 (142) clusters run at once where 104 of the full form do
// (cudaOccupancyMaxActiveClusters, 148 SMs: fewer than the CTAs an SM would give, as a cluster
// stays inside a GPC). A launch of x waves costs between x and the next whole number of them; half
// way between is taken. Of 3076 random lists of slices (1 to 25 slices of 64 to 1024 samples a
// side, 40 to 600 views, six detectors) it takes 889, none of them slower: 0.70 to 1.0 times the
// full form's time, 0.86 in the median. By the CTAs an SM alone (111, 148 and 185 clusters), and
// with tiles counted that lie outside the box or read global memory, 730 of 2024 were slower,
// up to 2.0 times.
static bool slim_pays(int64_t n, bool fp32) {
    auto cost = [&](int clusters, double time) {
        const double x = (double)n / clusters;
        return 0.5 * (x + ceil(x)) * time;
    };
    return cost(fp32 ? 142 : 175, fp32 ? 1.24 : 1.47) < cost(104, 1.0);
}

// Tiles of a regular grid that may hold a sample inside the box (all of them without a mask):
// those whose centre lies no further outside than the tile reaches.
template <typename F>
static int64_t for_busy_tiles(const mr_grid& g, F each) {
    const bool mask = (g.flags & MR_GRID_MASK_BOX) != 0;
    const double half = 0.5 * (ST_TI - 1) * fabs(g.mask_delta);
    double reach[3];
    for (int e = 0; e < 3; ++e) reach[e] = g.box[e] + half * (fabs(g.mask_ej[e]) + fabs(g.mask_ei[e])) * (1 + 1e-9);
    int64_t n = 0;
    for (int32_t k = 0; k < g.n_k; ++k)
        for (int32_t i0 = 0; i0 < g.n_i; i0 += ST_TI)
            for (int32_t j0 = 0; j0 < g.n_j; j0 += ST_TJ) {
                const double ai = (i0 + 0.5 * (ST_TI - 1) - g.mask_half) * g.mask_delta;
                const double aj = (j0 + 0.5 * (ST_TJ - 1) - g.mask_half) * g.mask_delta;
                bool in = true;
                for (int e = 0; mask && e < 3; ++e)
                    in = in && fabs(g.mask_c[e] + aj * g.mask_ej[e] + ai * g.mask_ei[e]) <= reach[e];
                if (in) each(n++, i0, j0, k);
            }
    return n;
}

constexpr int TRAIT_PAIRS = 64;                   // (tile, view) pairs looked at

// How the footprints of TRAIT_PAIRS busy tiles, spread over the grid, are read, each in a view of
// its own: count[0] from a stage (or not at all), count[1] from a wide box. The views run round
// the orbit 27 times while the tiles run once through the grid.
template <int KIND, typename T>
static void pair_modes(const mr_view* views, int n_views, const mr_grid& g, int R, int C, int64_t busy, int* count) {
    int64_t pair = 0;
    for_busy_tiles(g, [&](int64_t at, int32_t i0, int32_t j0, int32_t k) {
        for (; pair < TRAIT_PAIRS && pair * busy / TRAIT_PAIRS == at; ++pair) {
            const mr_view& V = views[pair * 27 % TRAIT_PAIRS * n_views / TRAIT_PAIRS];
            const float x = g.origin[0] + i0 * g.step_i[0] + j0 * g.step_j[0] + k * g.step_k[0];
            const float y = g.origin[1] + i0 * g.step_i[1] + j0 * g.step_j[1] + k * g.step_k[1];
            const float z = g.origin[2] + i0 * g.step_i[2] + j0 * g.step_j[2] + k * g.step_k[2];
            const int di = g.n_i - i0 < ST_TI ? g.n_i - i0 - 1 : ST_TI - 1;
            const int dj = g.n_j - j0 < ST_TJ ? g.n_j - j0 - 1 : ST_TJ - 1;
            const int mode = footprint<KIND, true, T>(V, g, x, y, z, di, dj, R, C).mode;
            count[0] += mode == MODE_STAGED || mode == MODE_SKIP;
            count[1] += mode == MODE_WIDE2 || mode == MODE_WIDE3;
        }
    });
}

}  // namespace mr

extern "C" int mr_staged_traits(const mr_view* views, int32_t n_views, int32_t kind, int32_t rows, int32_t cols,
                                int32_t dtype, const mr_grid* grid, double* traits) {
    if (!views || n_views < 1 || !grid || !traits || rows < 1 || cols < 1) return MR_ERR_INVALID;
    if (grid->n_i < 0 || grid->n_j < 0 || grid->n_k < 0 || (grid->flags & MR_GRID_POINTS)) return MR_ERR_INVALID;
    if (kind != MR_CONE && kind != MR_PARALLEL) return MR_ERR_INVALID;
    if (dtype != MR_F32 && dtype != MR_BF16 && dtype != MR_F16) return MR_ERR_INVALID;
    const int64_t busy = mr::for_busy_tiles(*grid, [](int64_t, int32_t, int32_t, int32_t) {});
    int count[2] = {0, 0};
    auto modes = dtype == MR_F32 ? (kind == MR_CONE ? mr::pair_modes<MR_CONE, float> : mr::pair_modes<MR_PARALLEL, float>)
                                 : (kind == MR_CONE ? mr::pair_modes<MR_CONE, __half> : mr::pair_modes<MR_PARALLEL, __half>);
    if (busy > 0) modes(views, n_views, *grid, rows, cols, busy, count);    // both 16-bit types have the same stages
    traits[0] = (double)busy;
    traits[1] = busy > 0 ? (double)count[0] / mr::TRAIT_PAIRS : 1.0;
    traits[2] = (double)count[1] / mr::TRAIT_PAIRS;
    return MR_OK;
}

extern "C" int mr_staged_slim_pays(int64_t busy_tiles, int32_t dtype) {
    return mr::slim_pays(busy_tiles, dtype == MR_F32) ? 1 : 0;
}

template <bool WIDE, bool SLIM>
static int backproject_staged(const mr_ring* ring, const mr_view* views, const mr_grid* grids, const mr_tile* tiles,
                              int64_t n_tiles, float* out, int32_t* status, void* stream) {
    int rc = mr::check_staged_ring(ring);
    if (rc != MR_OK) return rc;
    if (!views || !grids || !out || n_tiles < 0 || (n_tiles > 0 && !tiles)) return MR_ERR_INVALID;
    if (n_tiles == 0) return MR_OK;
    return mr::dispatch_staged<WIDE, SLIM>(ring, views, grids, tiles, n_tiles, out, status,
                                           static_cast<cudaStream_t>(stream), (const int64_t*)nullptr,
                                           (unsigned int*)nullptr);
}

extern "C" int mr_backproject_staged(const mr_ring* ring, const mr_view* views, const mr_grid* grids,
                                     const mr_tile* tiles, int64_t n_tiles, float* out, int32_t* status,
                                     void* stream) {
    return backproject_staged<false, false>(ring, views, grids, tiles, n_tiles, out, status, stream);
}

extern "C" int mr_backproject_staged_slim(const mr_ring* ring, const mr_view* views, const mr_grid* grids,
                                          const mr_tile* tiles, int64_t n_tiles, float* out, int32_t* status,
                                          void* stream) {
    return backproject_staged<false, true>(ring, views, grids, tiles, n_tiles, out, status, stream);
}

extern "C" int mr_backproject_staged_wide(const mr_ring* ring, const mr_view* views, const mr_grid* grids,
                                          const mr_tile* tiles, int64_t n_tiles, float* out, int32_t* status,
                                          void* stream) {
    return backproject_staged<true, false>(ring, views, grids, tiles, n_tiles, out, status, stream);
}

extern "C" int mr_backproject_persistent(const mr_ring* ring, const mr_view* views, const mr_grid* grids,
                                         const mr_tile* tiles, const int64_t* n_tiles_dev, int64_t max_tiles,
                                         uint32_t* counter_dev, float* out, int32_t* status, void* stream) {
    int rc = mr::check_staged_ring(ring);
    if (rc != MR_OK) return rc;
    if (!views || !grids || !tiles || !n_tiles_dev || !counter_dev || !out || max_tiles < 1) return MR_ERR_INVALID;
    // the 32-bit work counter must not wrap while the last clusters overshoot the count
    if (max_tiles > (int64_t(1) << 31)) return MR_ERR_INVALID;
    if ((reinterpret_cast<uintptr_t>(counter_dev) & 3) != 0) return MR_ERR_INVALID;
    return mr::dispatch_staged<false, false>(ring, views, grids, tiles, max_tiles, out, status, static_cast<cudaStream_t>(stream),
                               n_tiles_dev, reinterpret_cast<unsigned int*>(counter_dev));
}

// ---------------------------------------------------------------- no-allocation variant
// The persistent launch needs one 32-bit work counter in device memory. Callers that
// cannot allocate device memory get it from this file-scope array instead; every GPU that
// loads the library holds it until the process exits, and every call shares it.
static __device__ __align__(256) unsigned int g_noalloc_scratch[MR_NOALLOC_SCRATCH_BYTES / 4];

namespace {
constexpr int kNoallocMaxDevices = 64;
std::mutex g_noalloc_mutex;
unsigned int* g_noalloc_addr[kNoallocMaxDevices] = {};

// Device address of g_noalloc_scratch on the current device, looked up once per device.
// In host code the array's name is only a host-side stand-in, never a device address.
int noalloc_counter(cudaStream_t stream, unsigned int** counter) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return MR_ERR_CUDA;
    if (dev >= kNoallocMaxDevices) return MR_ERR_UNSUPPORTED;
    if (stream) {
        int sdev = -1;
        if (cudaStreamGetDevice(stream, &sdev) != cudaSuccess) return MR_ERR_CUDA;
        if (sdev != dev) return MR_ERR_INVALID;      // the stream's device must be current
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_addr[dev]) {
        // the symbol lookup may load device code, which a capture in progress forbids
        if (stream) {
            cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
            if (cudaStreamIsCapturing(stream, &cs) != cudaSuccess) {
                cudaGetLastError();
                return MR_ERR_CUDA;
            }
            if (cs != cudaStreamCaptureStatusNone) return MR_ERR_CAPTURE;
        }
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
            cudaGetLastError();
            return MR_ERR_CUDA;
        }
        g_noalloc_addr[dev] = static_cast<unsigned int*>(p);
    }
    *counter = g_noalloc_addr[dev];
    return MR_OK;
}
}  // namespace

extern "C" int mr_backproject_persistent_noalloc(const mr_ring* ring, const mr_view* views,
                                                 const mr_grid* grids, const mr_tile* tiles,
                                                 const int64_t* n_tiles_dev, int64_t max_tiles, float* out,
                                                 int32_t* status, void* stream) {
    int rc = mr::check_staged_ring(ring);
    if (rc != MR_OK) return rc;
    if (!views || !grids || !tiles || !n_tiles_dev || !out || max_tiles < 1) return MR_ERR_INVALID;
    if (max_tiles > MR_NOALLOC_MAX_TILES) return MR_ERR_SCRATCH_LIMIT;
    unsigned int* counter = nullptr;
    rc = noalloc_counter(static_cast<cudaStream_t>(stream), &counter);
    if (rc != MR_OK) return rc;
    // the shared launch path zeroes the counter on `stream` before the kernel
    return mr::dispatch_staged<false, false>(ring, views, grids, tiles, max_tiles, out, status, static_cast<cudaStream_t>(stream),
                               n_tiles_dev, counter);
}
