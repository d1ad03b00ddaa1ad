// Back-projection of a regular volume grid (minirecast recon.py:442-470, the sum of
// recon.py:156-219 over every voxel), in blocks of 16 x 16 x 16 voxels.
//
// The staged kernel (bp_tma.cu) treats a volume as a stack of 32 x 32 planes: every voxel
// forms its own divide, column and row, and every plane stages its own footprint. Here a
// block's footprint is staged once per view for 4096 voxels, and a thread owns a whole
// column of the block along j (16 voxels). On the usual orbit the detector's rows run
// along j, so that the depth and the detector column do not change along j: one
// reciprocal, one column and one horizontal weight serve the 16 voxels, whose rows are
// r0 + z dr. What is left per voxel is the row (floor and fraction), four shared-memory
// taps and three lerps. Whether a view is of this kind is seen from its map (the
// coefficients of column and depth along j are zero), view by view; the others take the
// full projection per voxel, and footprints wider than a stage read global memory.
//
// Measured (600 views of 486 x 384, against the staged kernel's tiles): 256 x 256 x 203
// voxels, BF16 ring, 16.9 -> 5.9 ms (1360 G updates/s); FP32 ring, whose tile footprints
// there did not fit a stage, 52.5 -> 6.2 ms; 400 x 400 x 317 voxels 57.3 -> 22.4 ms; views
// that are not aligned with j, 16.9 -> 8.1 ms. What bounds it: four shared-memory loads a
// sample (8 samples a clock and SM at most, 2270 G/s) beside 13 issue slots. Three CTAs an SM
// leave 72 registers (the cone variants spill 48 to 52 bytes); two CTAs with all the registers
// they want measured 6.5 ms.
#include <cooperative_groups.h>

#include "bp_stage.cuh"

namespace cg = cooperative_groups;

namespace mr {

constexpr int VB = 16;                            // block edge (voxels)
constexpr int VB_CONSUMERS = 8;                   // consumer warps: one thread per (i, k) column
constexpr int VB_THREADS = 32 * (VB_CONSUMERS + 1);
constexpr int VB_PAD = VB + 1;                    // partial sums: padded column of 16

// Row pitches as in the staged kernel (bp_tma.cu); a 16-voxel block is half as tall, so a
// stage holds MAXB boxes of 8 rows, 64 of either type, and CTAS = three CTAs fit an SM.
// COARSE: stages for blocks of voxels several detector pixels wide, whose footprints the plain
// ones (76 x 60 pixels) do not hold: 124 columns by 124 rows, by 92 of an FP32 ring. Two of them,
// so that three CTAs fit an SM (two of FP32). 600 views of 486 x 384, BF16, plain / coarse: 64 x
// 64 x 51 voxels (7.6 pixels) 1.11 / 0.99 ms, 96 x 96 x 76 1.97 / 0.66, 128 x 128 x 102 (3.8
// pixels) 2.86 / 1.11, 144 x 144 x 114 2.03 / 1.50; FP32 96 x 96 x 76 1.96 / 1.00, 128 x 128 x
// 102 3.24 / 1.40 ms. 96 rows of BF16: 96 x 96 x 76 0.88 ms; 168 columns by 96 rows: 0.90 ms there,
// 1.07 ms at 128 x 128 x 102; three stages, two CTAs: 0.84 and 1.15 ms.
template <typename T, bool COARSE> struct BlockGeom {
    static constexpr int W = 88, ALIGN = 8, STAGES = 4, MAXB = 8, CTAS = 3;
};
template <> struct BlockGeom<float, false> { static constexpr int W = 84, ALIGN = 4, STAGES = 3, MAXB = 8, CTAS = 3; };
template <typename T> struct BlockGeom<T, true> {
    static constexpr int W = 136, ALIGN = 8, STAGES = 2, MAXB = 16, CTAS = 3;
};
template <> struct BlockGeom<float, true> { static constexpr int W = 132, ALIGN = 4, STAGES = 2, MAXB = 12, CTAS = 2; };

enum : int { VB_COLUMN = 3 };                     // beside MODE_STAGED / MODE_GLOBAL / MODE_SKIP

// Affine maps of column numerator, row numerator and depth over the block: (value at voxel
// (0, 0, 0), d/di, d/dk, d/dj), from detector pixel `at` = (column, row), which is the
// stage's first one where the footprint is staged; m = (qscale, rows staged - 1, -, mode).
struct __align__(16) BlockRec {
    float4 u, v, w, m;
    int2 at;
};
struct __align__(16) BlockMeta {
    BlockRec rec;
    int x0, r0, nbox, mode;
};

template <int KIND, typename T, bool COARSE>
__device__ __forceinline__ BlockMeta block_meta(const mr_view& V, const mr_grid& g, int i0, int j0, int k0, int R,
                                                int C) {
    using Geom = BlockGeom<T, COARSE>;
    constexpr int W = Geom::W, ALIGN = Geom::ALIGN, MAXB = Geom::MAXB;
    float pu[4], pv[4];
    view_map(V, g, R, C, pu, pv);
    // the value at the block's origin in FP64: its FP32 rounding (half an ulp of a detector
    // coordinate) would move all 4096 voxels of the block together
    double o[3];
#pragma unroll
    for (int e = 0; e < 3; ++e)
        o[e] = (double)g.origin[e] + (double)i0 * g.step_i[e] + (double)j0 * g.step_j[e] + (double)k0 * g.step_k[e];
    double base[3];
    int at = 0;
    auto aff = [&](const float* m) {
        const double b = (double)m[0] * o[0] + (double)m[1] * o[1] + (double)m[2] * o[2] + (double)m[3];
        base[at++] = b;
        return make_float4((float)b,
                           fmaf(m[0], g.step_i[0], fmaf(m[1], g.step_i[1], m[2] * g.step_i[2])),
                           fmaf(m[0], g.step_k[0], fmaf(m[1], g.step_k[1], m[2] * g.step_k[2])),
                           fmaf(m[0], g.step_j[0], fmaf(m[1], g.step_j[1], m[2] * g.step_j[2])));
    };
    float4 au = aff(pu), av = aff(pv), aw = aff(V.pw);
    if (KIND == MR_CONE && V.qscale != 1.f) {
        // col = nu/nw and row = nv/nw are scale free, 1/nw^2 picks up qscale
        const float k = rsqrtf(V.qscale);
        au = make_float4(au.x * k, au.y * k, au.z * k, au.w * k);
        av = make_float4(av.x * k, av.y * k, av.z * k, av.w * k);
        aw = make_float4(aw.x * k, aw.y * k, aw.z * k, aw.w * k);
        for (double& b : base) b *= k;
    }
    // footprint of the whole block (its voxels past the grid's end included: they are
    // summed like the others and not written)
    float cmin = 3e38f, cmax = -3e38f, rmin = 3e38f, rmax = -3e38f;
    bool behind = false;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const float di = (c & 1) ? (float)(VB - 1) : 0.f;
        const float dk = (c & 2) ? (float)(VB - 1) : 0.f;
        const float dj = (c & 4) ? (float)(VB - 1) : 0.f;
        const float w = fmaf(di, aw.y, fmaf(dk, aw.z, fmaf(dj, aw.w, aw.x)));
        float cc = fmaf(di, au.y, fmaf(dk, au.z, fmaf(dj, au.w, au.x)));
        float rr = fmaf(di, av.y, fmaf(dk, av.z, fmaf(dj, av.w, av.x)));
        if (KIND == MR_CONE) {
            behind |= !(w > 1e-3f);
            const float inv = 1.f / w;
            cc *= inv;
            rr *= inv;
        }
        cmin = fminf(cmin, cc); cmax = fmaxf(cmax, cc);
        rmin = fminf(rmin, rr); rmax = fmaxf(rmax, rr);
    }
    BlockMeta m;
    int mode = MODE_GLOBAL, x0 = 0, r0 = 0, nbox = 0;
    if (!behind && cmax == cmax && rmax == rmax && cmin == cmin && rmin == rmin) {
        if (cmax < -2.f || cmin > (float)C + 1.f || rmax < -2.f || rmin > (float)R + 1.f) {
            mode = MODE_SKIP;
        } else if (cmax - cmin < (float)(W - ALIGN - 4) && rmax - rmin < (float)(ST_BOX_H * MAXB - 4)) {
            x0 = ((int)floorf(cmin) - 1) & ~(ALIGN - 1);
            r0 = (int)floorf(rmin) - 1;
            const int rows = (int)floorf(rmax) + 3 - r0;
            nbox = (rows + ST_BOX_H - 1) / ST_BOX_H;
            if ((int)floorf(cmax) + 3 - x0 <= W && nbox <= MAXB)
                mode = (au.w == 0.f && aw.w == 0.f) ? VB_COLUMN : MODE_STAGED;
        } else if (cmax - cmin < (float)(C + 2) && rmax - rmin < (float)(R + 2)) {
            // too wide to stage, on or near the detector: coordinates still count from a
            // pixel nearby, which keeps their rounding that of the footprint's size
            x0 = (int)floorf(cmin);
            r0 = (int)floorf(rmin);
        }
    }
    if (mode != MODE_SKIP) {
        const float fx0 = (float)x0, fr0 = (float)r0;
        au = make_float4((float)(base[0] - x0 * base[2]), fmaf(-fx0, aw.y, au.y), fmaf(-fx0, aw.z, au.z),
                         fmaf(-fx0, aw.w, au.w));
        av = make_float4((float)(base[1] - r0 * base[2]), fmaf(-fr0, aw.y, av.y), fmaf(-fr0, aw.z, av.z),
                         fmaf(-fr0, aw.w, av.w));
    }
    m.rec.u = au;
    m.rec.v = av;
    m.rec.w = aw;
    m.rec.m = make_float4(V.qscale, (float)(nbox * ST_BOX_H - 1), 0.f, __int_as_float(mode));
    m.rec.at = make_int2(x0, r0);
    m.x0 = x0; m.r0 = r0; m.nbox = nbox; m.mode = mode;
    return m;
}

// One pair of voxels: taps at shared-memory addresses a0, a1 (top left), weights fc, fr.
template <typename T, int PITCH>
__device__ __forceinline__ float2 lerp_pair(uint32_t a0, uint32_t a1, float2 fc, float2 fr) {
    constexpr int ESZ = (int)sizeof(T);
    float2 q00, q10, d0, d1;
    q00 = make_float2(lds_elem<T>(a0), lds_elem<T>(a1));
    q10 = make_float2(lds_elem<T>(a0 + PITCH), lds_elem<T>(a1 + PITCH));
    if constexpr (sizeof(T) == 2) {
        d0 = make_float2(sub16_f32<T>(lds_u16(a0 + ESZ), q00.x), sub16_f32<T>(lds_u16(a1 + ESZ), q00.y));
        d1 = make_float2(sub16_f32<T>(lds_u16(a0 + PITCH + ESZ), q10.x),
                         sub16_f32<T>(lds_u16(a1 + PITCH + ESZ), q10.y));
    } else {
        d0 = __ffma2_rn(q00, kNeg2, make_float2(lds_elem<T>(a0 + ESZ), lds_elem<T>(a1 + ESZ)));
        d1 = __ffma2_rn(q10, kNeg2, make_float2(lds_elem<T>(a0 + PITCH + ESZ), lds_elem<T>(a1 + PITCH + ESZ)));
    }
    const float2 ta = __ffma2_rn(fc, d0, q00);
    const float2 tb = __ffma2_rn(fc, d1, q10);
    return __ffma2_rn(fr, __ffma2_rn(ta, kNeg2, tb), ta);
}

// Warp roles and the stage ring are those of bp_staged_kernel: warp 8 computes footprints
// and issues the box loads, warps 0..7 sum; full / empty mbarriers with bounded waits. A
// cluster of four or two CTAs (view_shares) splits the views of a block and adds the partial sums in rank
// order through distributed shared memory, each rank finishing its share of the columns.
template <int KIND, typename T, bool COARSE>
__global__ void __launch_bounds__(VB_THREADS, BlockGeom<T, COARSE>::CTAS)
bp_volume_kernel(const __grid_constant__ CUtensorMap tmap, const T* __restrict__ ring, int R, int C, int pitch,
                 long long slot_stride, int n_slots, const mr_view* __restrict__ views,
                 const __grid_constant__ mr_grid g, int blocks_i, int blocks_k, int blocks_j,
                 float* __restrict__ out, int* status) {
    using Geom = BlockGeom<T, COARSE>;
    constexpr int W = Geom::W;
    constexpr int S = Geom::STAGES;
    constexpr int ESZ = (int)sizeof(T);
    constexpr int PITCH = W * ESZ;
    constexpr int BOX_BYTES = PITCH * ST_BOX_H;
    constexpr int STAGE_BYTES = BOX_BYTES * Geom::MAXB;
    static_assert(BOX_BYTES % 128 == 0 && STAGE_BYTES % 128 == 0, "TMA box / stage not 128-byte aligned");
    static_assert(S * STAGE_BYTES >= VB_CONSUMERS * 32 * VB_PAD * 4, "partial sums reuse the stages");

    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* stages = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~static_cast<uintptr_t>(127));
    BlockRec* rec_ring = reinterpret_cast<BlockRec*>(stages + S * STAGE_BYTES);      // S
    BlockMeta* meta_new = reinterpret_cast<BlockMeta*>(rec_ring + S);                // 32
    uint64_t* full = reinterpret_cast<uint64_t*>(meta_new + 32);                     // S
    uint64_t* empty = full + S;                                                      // S

    cg::cluster_group cluster = cg::this_cluster();
    const int crank = (int)cluster.block_rank();
    const int csize = (int)cluster.num_blocks();
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const bool producer = warp == VB_CONSUMERS;
    if (tid < S) {
        mbar_init(&full[tid], 1);
        mbar_init(&empty[tid], VB_CONSUMERS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();

    // blocks in planes of equal j, last plane first: the blocks in flight together project
    // onto one band of detector rows, so their footprints are read from L2
    const unsigned int block = blockIdx.x / csize;
    const int i0 = (int)(block % blocks_i) * VB;
    const int k0 = (int)((block / blocks_i) % blocks_k) * VB;
    const int j0 = (blocks_j - 1 - (int)(block / ((unsigned)blocks_i * blocks_k))) * VB;
    int first, count;
    grid_view_range(g.view_begin, g.n_views, n_slots, &first, &count);
    const int v_begin = first + (int)(((long long)count * crank) / csize);
    const int nv = first + (int)(((long long)count * (crank + 1)) / csize) - v_begin;

    float2 acc[VB / 2];
#pragma unroll
    for (int h = 0; h < VB / 2; ++h) acc[h] = make_float2(0.f, 0.f);

    if (producer) {
        for (int vb = 0; vb < nv; vb += 32) {
            const int cnt = min(32, nv - vb);
            __syncwarp();
            if (lane < cnt) meta_new[lane] = block_meta<KIND, T, COARSE>(views[v_begin + vb + lane], g, i0, j0, k0, R, C);
            __syncwarp();
            for (int l = 0; l < cnt; ++l) {
                const uint32_t ua = (uint32_t)(vb + l);
                const int s = (int)(ua % S);
                const uint32_t u = ua / S;
                const int mode = meta_new[l].mode, nbox = meta_new[l].nbox;
                const bool boxes = mode == VB_COLUMN || mode == MODE_STAGED;
                if (lane == 0) {
                    if (u > 0) mbar_wait(&empty[s], (u - 1) & 1u, status);
                    rec_ring[s] = meta_new[l].rec;
                    if (boxes) mbar_arrive_tx(&full[s], (uint32_t)(nbox * BOX_BYTES));
                    else mbar_arrive(&full[s]);
                }
                __syncwarp();                   // the stage is free and armed for every lane
                if (boxes && lane < nbox)
                    tma_load_3d(stages + s * STAGE_BYTES + lane * BOX_BYTES, &tmap, meta_new[l].x0,
                                meta_new[l].r0 + lane * ST_BOX_H, v_begin + vb + l, &full[s]);
            }
        }
    } else {
        const float fi = (float)(tid & (VB - 1)), fk = (float)(tid / VB);     // a warp: 16 i x 2 k
        int s = 0;
        uint32_t phase = 0;
        for (int v = 0; v < nv; ++v) {
            mbar_wait(&full[s], phase, status);
            const BlockRec& rec = rec_ring[s];
            const float4 cu = rec.u, cv = rec.v, cw = rec.w, cm = rec.m;
            const int mode = __float_as_int(cm.w);
            const float nu = fmaf(fi, cu.y, fmaf(fk, cu.z, cu.x));
            const float nr = fmaf(fi, cv.y, fmaf(fk, cv.z, cv.x));
            const float nw = fmaf(fi, cw.y, fmaf(fk, cw.z, cw.x));
            const uint32_t base = smem_u32(stages + s * STAGE_BYTES);
            if (mode == VB_COLUMN) {
                const float r = KIND == MR_CONE ? rcp_approx(nw) : 1.f;
                const float yc = KIND == MR_CONE ? __fmaf_rd(nu, r, MAGIC) : __fadd_rd(nu, MAGIC);
                const float fc = KIND == MR_CONE ? fmaf(nu, r, MAGIC - yc) : nu + (MAGIC - yc);
                float ra = KIND == MR_CONE ? nr * r : nr, rs = KIND == MR_CONE ? cv.w * r : cv.w;
                const float re = fmaf((float)(VB - 1), rs, ra);
                int c0 = __float_as_int(yc) - MAGIC_BITS;
                // rows are linear along j, so the two ends bound every tap (memory safety only:
                // the footprint covers the block with a margin of a pixel)
                const bool ok = fminf(ra, re) >= 0.f && fmaxf(ra, re) < cm.y && (unsigned)c0 < (unsigned)(W - 1);
                if (!ok) ra = rs = 0.f, c0 = 0;
                const float wgt = KIND == MR_CONE ? r * r : cm.x;
                const float2 fc2 = make_float2(fc, fc), ra2 = make_float2(ra, ra), rs2 = make_float2(rs, rs);
                const float2 wgt2 = make_float2(wgt, wgt);
                const uint32_t col = base + (uint32_t)c0 * ESZ - (uint32_t)MAGIC_BITS * (uint32_t)PITCH;
#pragma unroll
                for (int h = 0; h < VB / 2; ++h) {
                    const float2 row = __ffma2_rn(make_float2((float)(2 * h), (float)(2 * h + 1)), rs2, ra2);
                    const float2 yr = __fadd2_rd(row, kMagic2);
                    const float2 fr = __fadd2_rn(row, __ffma2_rn(yr, kNeg2, kMagic2));
                    const uint32_t a0 = (uint32_t)__float_as_int(yr.x) * (uint32_t)PITCH + col;
                    const uint32_t a1 = (uint32_t)__float_as_int(yr.y) * (uint32_t)PITCH + col;
                    acc[h] = __ffma2_rn(wgt2, lerp_pair<T, PITCH>(a0, a1, fc2, fr), acc[h]);
                }
            } else if (mode == MODE_STAGED) {
                const uint32_t last = ((uint32_t)cm.y - 1u) * PITCH + (W - 2) * ESZ;
                const uint32_t kofs = (uint32_t)MAGIC_BITS * (uint32_t)(PITCH + ESZ);
#pragma unroll
                for (int h = 0; h < VB / 2; ++h) {
                    const float2 z = make_float2((float)(2 * h), (float)(2 * h + 1));
                    const float2 u2 = __ffma2_rn(z, make_float2(cu.w, cu.w), make_float2(nu, nu));
                    const float2 v2 = __ffma2_rn(z, make_float2(cv.w, cv.w), make_float2(nr, nr));
                    float2 r = make_float2(1.f, 1.f), yc, yr, fc, fr;
                    if (KIND == MR_CONE) {
                        const float2 w2 = __ffma2_rn(z, make_float2(cw.w, cw.w), make_float2(nw, nw));
                        r = make_float2(rcp_approx(w2.x), rcp_approx(w2.y));
                        yc = __ffma2_rd(u2, r, kMagic2);
                        yr = __ffma2_rd(v2, r, kMagic2);
                        fc = __ffma2_rn(u2, r, __ffma2_rn(yc, kNeg2, kMagic2));
                        fr = __ffma2_rn(v2, r, __ffma2_rn(yr, kNeg2, kMagic2));
                    } else {
                        yc = __fadd2_rd(u2, kMagic2);
                        yr = __fadd2_rd(v2, kMagic2);
                        fc = __fadd2_rn(u2, __ffma2_rn(yc, kNeg2, kMagic2));
                        fr = __fadd2_rn(v2, __ffma2_rn(yr, kNeg2, kMagic2));
                    }
                    const uint32_t a0 = base + min((uint32_t)__float_as_int(yr.x) * (uint32_t)PITCH +
                                                       (uint32_t)__float_as_int(yc.x) * (uint32_t)ESZ - kofs, last);
                    const uint32_t a1 = base + min((uint32_t)__float_as_int(yr.y) * (uint32_t)PITCH +
                                                       (uint32_t)__float_as_int(yc.y) * (uint32_t)ESZ - kofs, last);
                    const float2 wgt = KIND == MR_CONE ? __fmul2_rn(r, r) : make_float2(cm.x, cm.x);
                    acc[h] = __ffma2_rn(wgt, lerp_pair<T, PITCH>(a0, a1, fc, fr), acc[h]);
                }
            } else if (mode == MODE_GLOBAL) {
                const T* q = ring + (long long)(v_begin + v) * slot_stride;
                const int2 at = rec.at;
#pragma unroll
                for (int z = 0; z < VB; ++z) {
                    const float u = fmaf((float)z, cu.w, nu), vr = fmaf((float)z, cv.w, nr);
                    float& a = (z & 1) ? acc[z >> 1].y : acc[z >> 1].x;
                    if (KIND == MR_CONE) {
                        const float r = rcp_approx(fmaf((float)z, cw.w, nw));
                        a = fmaf(r * r, bilerp_global(q, R, C, pitch, vr * r, u * r, at.y, at.x), a);
                    } else {
                        a = fmaf(cm.x, bilerp_global(q, R, C, pitch, vr, u, at.y, at.x), a);
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

    // every stage has been filled and read: the partial sums take their place
    __syncthreads();
    float* partial = reinterpret_cast<float*>(stages);                  // [column][VB_PAD]
    if (!producer) {
#pragma unroll
        for (int h = 0; h < VB / 2; ++h) {
            partial[tid * VB_PAD + 2 * h] = acc[h].x;
            partial[tid * VB_PAD + 2 * h + 1] = acc[h].y;
        }
    }
    cluster.sync();
    const int cols = VB * VB / csize;                                   // columns this rank finishes
    for (int e = tid; e < cols * VB; e += VB_THREADS) {
        const int column = crank * cols + e / VB, z = e % VB;           // neighbours along j: one row of out
        float sum = cluster.map_shared_rank(partial, 0)[column * VB_PAD + z];
        for (int rk = 1; rk < csize; ++rk) sum += cluster.map_shared_rank(partial, rk)[column * VB_PAD + z];
        const int i = i0 + column % VB, k = k0 + column / VB, j = j0 + z;
        if (i < g.n_i && j < g.n_j && k < g.n_k) {
            const long long o = g.out_offset + (long long)i * g.out_stride_i + (long long)j * g.out_stride_j +
                                (long long)k * g.out_stride_k;
            const float val = sum * g.scale;
            out[o] = g.accumulate ? out[o] + val : val;
        }
    }
    cluster.sync();                             // partial sums stay alive until every rank has read them
}

// CTAs per block, each a share of the views: four where two would leave SMs idle (below two and
// a half blocks an SM), else two, which end and wait for one another half as often (600 views of
// 486 x 384, BF16, four / two: 100 blocks 1.06 / 2.01 ms, 294 blocks 2.54 / 3.06, 384 blocks
// 3.09 / 2.88, 800 blocks 1.70 / 1.64, 3328 blocks 6.19 / 5.88 ms).
static unsigned view_shares(long long blocks) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        sms = 148;
    return 2 * blocks >= 5LL * sms ? 2u : 4u;
}

template <int KIND, bool COARSE, typename T>
static int launch_volume(const mr_ring* ring, const mr_view* views, const mr_grid& g, float* out, int* status,
                         cudaStream_t st) {
    const long long bi = (g.n_i + VB - 1) / VB, bj = (g.n_j + VB - 1) / VB, bk = (g.n_k + VB - 1) / VB;
    if (bi * bj > 2147483647LL / 4 || bi * bj * bk > 2147483647LL / 4) return MR_ERR_UNSUPPORTED;
    const unsigned cluster = view_shares(bi * bj * bk);
    using Geom = BlockGeom<T, COARSE>;
    CUtensorMap map;
    int rc = make_ring_map<T>(ring, Geom::W, &map);
    if (rc != MR_OK) return rc;
    constexpr int S = Geom::STAGES;
    const size_t smem = (size_t)S * Geom::W * ST_BOX_H * Geom::MAXB * sizeof(T) + S * sizeof(BlockRec) +
                        32 * sizeof(BlockMeta) + 2 * S * sizeof(uint64_t) + 128;
    auto kern = bp_volume_kernel<KIND, T, COARSE>;
    MR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(bi * bj * bk) * cluster);
    cfg.blockDim = dim3(VB_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MR_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, map, static_cast<const T*>(ring->data), ring->rows, ring->cols,
                                   ring->col_pitch, (long long)ring->slot_stride, (int)ring->n_slots, views, g,
                                   (int)bi, (int)bk, (int)bj, out, status));
    MR_CUDA_TRY(cudaGetLastError());
    return MR_OK;
}

template <bool COARSE>
static int dispatch_volume(const mr_ring* ring, const mr_view* views, const mr_grid* grid, float* out, int32_t* status,
                           void* stream) {
    int rc = check_staged_ring(ring);
    if (rc != MR_OK) return rc;
    if (!views || !grid || !out || grid->n_i < 0 || grid->n_j < 0 || grid->n_k < 0) return MR_ERR_INVALID;
    if (grid->flags & (MR_GRID_POINTS | MR_GRID_MASK_BOX)) return MR_ERR_INVALID;
    if (grid->n_i == 0 || grid->n_j == 0 || grid->n_k == 0) return MR_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool cone = ring->kind == MR_CONE;
    switch (ring->dtype) {
        case MR_F32:
            return cone ? launch_volume<MR_CONE, COARSE, float>(ring, views, *grid, out, status, st)
                        : launch_volume<MR_PARALLEL, COARSE, float>(ring, views, *grid, out, status, st);
        case MR_BF16:
            return cone ? launch_volume<MR_CONE, COARSE, __nv_bfloat16>(ring, views, *grid, out, status, st)
                        : launch_volume<MR_PARALLEL, COARSE, __nv_bfloat16>(ring, views, *grid, out, status, st);
        default:
            return cone ? launch_volume<MR_CONE, COARSE, __half>(ring, views, *grid, out, status, st)
                        : launch_volume<MR_PARALLEL, COARSE, __half>(ring, views, *grid, out, status, st);
    }
}

}  // namespace mr

extern "C" int mr_backproject_volume(const mr_ring* ring, const mr_view* views, const mr_grid* grid, float* out,
                                     int32_t* status, void* stream) {
    return mr::dispatch_volume<false>(ring, views, grid, out, status, stream);
}

extern "C" int mr_backproject_volume_coarse(const mr_ring* ring, const mr_view* views, const mr_grid* grid, float* out,
                                            int32_t* status, void* stream) {
    return mr::dispatch_volume<true>(ring, views, grid, out, status, stream);
}
