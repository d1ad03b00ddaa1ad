// Derivatives of the back-projection f = B(q; shift, tilt) for the differentiable
// back-projector (no counterpart in minirecast; the forward operator is recon.py:156-219).
//
//   mr_project_adjoint : grad_q = B^T g - the matched forward projector: every sample's
//                        upstream gradient g[p] is scattered to the same four bilinear taps,
//                        with the same weights, that the forward kernel gathers from (the
//                        exact transpose, taps outside the detector dropped as in forward).
//   mr_backproject_matched : the forward B q with exactly the coordinate arithmetic of
//                        the two kernels below (its transpose is mr_project_adjoint to
//                        the last rounding of the sums);
//   mr_bp_grad_geom    : d<g, f>/d shift and d<g, f>/d tilt per grid, from the analytic
//                        derivative of the bilinear interpolant:
//                          dv/dcol = (1-fr)(q01-q00) + fr (q11-q10)
//                          dv/drow = (1-fc)(q10-q00) + fc (q11-q01)
//                        with dcol/dshift = 1, drow/dshift = uv, dcol/dtilt = row - shift uv - cr,
//                        drow/dtilt = -(col - shift - cc); the distance weight depends on neither.
// Geometry is recomputed from the per-view maps (nothing from the forward pass is stored).
//
// A tile's views may be split over a thread-block cluster of up to 8 CTAs (few tiles: the
// calibration's slices are a few dozen tiles): each CTA takes a contiguous share of the
// views; forward partial sums are reduced through distributed shared memory in rank order
// (deterministic, no scratch), geometry partials go through the FP64 atomics that already
// combine the tiles, and adjoint taps are scattered atomically either way.
#include <cooperative_groups.h>

#include "mr_common.cuh"

namespace cg = cooperative_groups;

namespace mr {

constexpr int GR_THREADS = 256;
constexpr int GR_PPT = 4;
constexpr int GR_STEP = GR_THREADS / 32;       // lines between a thread's samples
constexpr int GR_VCH = 128;
constexpr int GR_TILE = 32;                    // tile edge (samples), as planned by mr_plan_tiles

enum : int { ALONG_J = 0, ALONG_I = 1, PATCHES = 2 };      // a warp's 32 samples
enum : int { GRAD_ADJOINT = 0, GRAD_GEOM = 1, GRAD_FORWARD = 2 };

// One coordinate of a grid's sample. The roundings are written out: left to the compiler they
// depend on the code around, and all three kernels use the same coordinates.
__device__ __forceinline__ float grid_point(const mr_grid& g, int e, int i, int j, int k) {
    return fmaf((float)k, g.step_k[e], fmaf((float)j, g.step_j[e], fmaf((float)i, g.step_i[e], g.origin[e])));
}

// Where the footprint of a whole 32 x 32 tile lies in a view: wholly on the detector with a
// margin of half a pixel (no tap of any lane needs a check), wholly off it (nothing to add),
// or neither. The tile's four corners bound it: it is planar, and in front of the source.
enum : int { FOOT_EDGE = 0, FOOT_INSIDE = 1, FOOT_OFF = 2 };

template <int KIND>
__device__ __forceinline__ int tile_footprint(const float* pu, const float* pv, const float* pw, const mr_grid& g,
                                              const mr_tile& t, int R, int C) {
    float cmin = 3e38f, cmax = -3e38f, rmin = 3e38f, rmax = -3e38f;
    bool front = true;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float i = (float)(t.i0 + ((c & 1) ? GR_TILE - 1 : 0)), j = (float)(t.j0 + ((c & 2) ? GR_TILE - 1 : 0));
        float p[3];
#pragma unroll
        for (int e = 0; e < 3; ++e) p[e] = g.origin[e] + i * g.step_i[e] + j * g.step_j[e] + t.k * g.step_k[e];
        float col = fmaf(pu[0], p[0], fmaf(pu[1], p[1], fmaf(pu[2], p[2], pu[3])));
        float row = fmaf(pv[0], p[0], fmaf(pv[1], p[1], fmaf(pv[2], p[2], pv[3])));
        if (KIND == MR_CONE) {
            const float w = fmaf(pw[0], p[0], fmaf(pw[1], p[1], fmaf(pw[2], p[2], pw[3])));
            front = front && w > 1e-3f;
            col /= w;
            row /= w;
        }
        cmin = fminf(cmin, col); cmax = fmaxf(cmax, col);
        rmin = fminf(rmin, row); rmax = fmaxf(rmax, row);
        front = front && col == col && row == row;
    }
    if (!front) return FOOT_EDGE;
    if (cmax < -2.f || rmax < -2.f || cmin > (float)C + 1.f || rmin > (float)R + 1.f) return FOOT_OFF;
    return cmin > 0.5f && rmin > 0.5f && cmax < (float)C - 1.5f && rmax < (float)R - 1.5f ? FOOT_INSIDE : FOOT_EDGE;
}

// Four CTAs an SM for the forward kernel (64 registers, up to 88 bytes spilled), three for the others:
// by 68 grids, forward with three 1.06 times, geometry with four 1.10 times the time.
template <int KIND, int MODE, typename T>
__global__ void __launch_bounds__(GR_THREADS, MODE == GRAD_FORWARD ? 4 : 3)
bp_grad_kernel(const T* __restrict__ ring, float* __restrict__ gring, int R, int C, int pitch,
               long long slot_stride, int n_slots, const mr_view* __restrict__ views,
               const mr_grid* __restrict__ grids,
               const mr_tile* __restrict__ tiles, const float* __restrict__ gout, double* __restrict__ dgeom) {
    __shared__ float4 s_u[GR_VCH], s_v[GR_VCH], s_w[GR_VCH];
    __shared__ float s_q[GR_VCH], s_uv[GR_VCH];
    __shared__ int s_foot[GR_VCH];
    __shared__ mr_grid s_g;
    __shared__ double s_red[2][GR_THREADS / 32];
    __shared__ float4 s_part[GR_THREADS];
    cg::cluster_group cluster = cg::this_cluster();
    const int crank = (int)cluster.block_rank();
    const int csize = (int)cluster.num_blocks();
    const mr_tile t = tiles[blockIdx.x / csize];
    const int tid = threadIdx.x;
    if (tid < (int)(sizeof(mr_grid) / 4))
        reinterpret_cast<int*>(&s_g)[tid] = reinterpret_cast<const int*>(grids + t.grid)[tid];
    __syncthreads();
    const mr_grid& g = s_g;
    const bool pts = (g.flags & MR_GRID_POINTS) != 0;
    const int warp = tid >> 5, lane = tid & 31;
    int first, nv;                      // slots [first, first + nv)
    grid_view_range(g.view_begin, g.n_views, n_slots, &first, &nv);
    // Where a warp's 32 samples lie. On a line, eight lines apart, along the grid direction that
    // moves less along the detector's rows (j on a slice, i on a volume, whose j is the rotation
    // axis): its taps then lie on one or two detector rows, and a warp-wide gather or reduction
    // touches few lines of memory. Where neither direction moves along them (axial slices) and a
    // sample is wider than 2.5 pixels, in patches of 8 x 4: a line of samples would cover more
    // memory. Patches / lines along j / this rule:
    //   512^2 slice, 600 views of 486 x 384, whole calls (the kernels alone by this rule: 364 to
    //   403, 510 and 336 to 350 us): forward 505 / 459 / 459 us, adjoint 830 / 705 / 705, geometry
    //   497 / 459 / 459
    //   160 x 160 x 127 voxels, 180 views of 300 x 200: forward 1.77 / 3.04 / 1.20 ms, adjoint
    //   4.32 / 8.47 / 2.47 ms, geometry 1.74 / 3.06 / 1.59 ms
    //   axial 96^2 slice (5 pixels a sample), 300 views of 486 x 384: adjoint 51 / 77 / 51 us
    int lanes = ALONG_J;
    if (!pts && nv > 0) {
        const mr_view& V = views[first];
        float p[3], row = V.pv[3], col = V.pu[3], vi = 0.f, vj = 0.f, ui = 0.f, uj = 0.f, wi = 0.f, wj = 0.f;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
            p[e] = grid_point(g, e, t.i0, t.j0, t.k);
            row = fmaf(V.pv[e], p[e], row);
            col = fmaf(V.pu[e], p[e], col);
            ui = fmaf(V.pu[e], g.step_i[e], ui);
            uj = fmaf(V.pu[e], g.step_j[e], uj);
            vi = fmaf(V.pv[e], g.step_i[e], vi);
            vj = fmaf(V.pv[e], g.step_j[e], vj);
            wi = fmaf(V.pw[e], g.step_i[e], wi);
            wj = fmaf(V.pw[e], g.step_j[e], wj);
        }
        if (KIND == MR_CONE) {          // d(row) = (d(numerator) - row d(depth)) / depth, and so the column
            const float w = fmaf(V.pw[0], p[0], fmaf(V.pw[1], p[1], fmaf(V.pw[2], p[2], V.pw[3])));
            vi = (vi - row / w * wi) / w;
            vj = (vj - row / w * wj) / w;
            ui = (ui - col / w * wi) / w;
            uj = (uj - col / w * wj) / w;
        }
        if (fabsf(vi) < 0.7f * fabsf(vj)) lanes = ALONG_I;
        if (fmaxf(fabsf(vi), fabsf(vj)) < 0.5f && ui * ui + uj * uj > 6.25f) lanes = PATCHES;
    }
    const int tx = lanes == ALONG_J ? lane : lanes == ALONG_I ? warp : ((warp & 3) << 3) | (lane & 7);
    const int ty = lanes == ALONG_J ? warp : lanes == ALONG_I ? lane : ((warp >> 2) << 4) | (lane >> 3);
    const int dj = lanes == ALONG_I ? GR_STEP : 0, di = lanes == ALONG_J ? GR_STEP : lanes == ALONG_I ? 0 : 4;

    float px[GR_PPT], py[GR_PPT], pz[GR_PPT], gp[GR_PPT], acc[GR_PPT];
    long long oidx[GR_PPT];
    bool live[GR_PPT];
#pragma unroll
    for (int p = 0; p < GR_PPT; ++p) {
        int i, j;
        long long o;
        bool ok;
        if (pts) {
            i = 0;
            j = t.j0 + tid + GR_THREADS * p;
            ok = j < g.n_j;
            o = g.out_offset + (long long)j * g.out_stride_j;
        } else {
            i = t.i0 + ty + di * p;
            j = t.j0 + tx + dj * p;
            ok = i < g.n_i && j < g.n_j;
            o = g.out_offset + (long long)i * g.out_stride_i + (long long)j * g.out_stride_j +
                (long long)t.k * g.out_stride_k;
        }
        bool inside = ok;
        if (ok && !pts && (g.flags & MR_GRID_MASK_BOX)) {
            const double aj = __dmul_rn((double)j - g.mask_half, g.mask_delta);
            const double ai = __dmul_rn((double)i - g.mask_half, g.mask_delta);
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                const double q = __dadd_rn(__dadd_rn(g.mask_c[e], __dmul_rn(aj, g.mask_ej[e])),
                                           __dmul_rn(ai, g.mask_ei[e]));
                inside = inside && (fabs(q) <= g.box[e]);
            }
        }
        live[p] = inside;
        oidx[p] = o;
        acc[p] = 0.f;
        gp[p] = (MODE != GRAD_FORWARD && inside) ? gout[o] * g.scale : 0.f;
        if (pts) {
            const int jj = ok ? j : 0;
            px[p] = g.points[3 * jj];
            py[p] = g.points[3 * jj + 1];
            pz[p] = g.points[3 * jj + 2];
        } else {
            px[p] = grid_point(g, 0, i, j, t.k);
            py[p] = grid_point(g, 1, i, j, t.k);
            pz[p] = grid_point(g, 2, i, j, t.k);
        }
    }
    // a warp none of whose samples counts has nothing to do in the view loop
    bool own = false;
#pragma unroll
    for (int p = 0; p < GR_PPT; ++p) own |= MODE == GRAD_FORWARD ? live[p] : gp[p] != 0.f;
    const bool busy = __any_sync(0xffffffffu, own);
    const float shift = g.cor_shift;
    const float cc = 0.5f * (float)(C - 1), cr = 0.5f * (float)(R - 1);
    float ds = 0.f, dt = 0.f;
    {                                   // this CTA's share of them
        const int b = first + (int)(((long long)nv * crank) / csize);
        const int e = first + (int)(((long long)nv * (crank + 1)) / csize);
        first = b;
        nv = e - b;
    }
    for (int v0 = 0; v0 < nv; v0 += GR_VCH) {
        const int nch = min(GR_VCH, nv - v0);
        __syncthreads();
        if (tid < nch) {
            const mr_view V = views[first + v0 + tid];
            float pu[4], pv[4];
            view_map(V, g, R, C, pu, pv);
            s_u[tid] = make_float4(pu[0], pu[1], pu[2], pu[3]);
            s_v[tid] = make_float4(pv[0], pv[1], pv[2], pv[3]);
            s_w[tid] = make_float4(V.pw[0], V.pw[1], V.pw[2], V.pw[3]);
            s_q[tid] = V.qscale;
            s_uv[tid] = V.uv;
            s_foot[tid] = pts ? FOOT_EDGE : tile_footprint<KIND>(pu, pv, V.pw, g, t, R, C);
        }
        __syncthreads();
        for (int vv = 0; vv < nch; ++vv) {
            const int foot = s_foot[vv];
            if (foot == FOOT_OFF || !busy) continue;
            const float4 cu = s_u[vv], cv = s_v[vv], cw = s_w[vv];
            const float qs = s_q[vv], uv = s_uv[vv];
            const long long slot = (long long)(first + v0 + vv) * slot_stride;
            if (foot == FOOT_INSIDE) {
                // The arithmetic of the general path below without its checks, the taps of all
                // four samples in flight together: with a branch between the samples each one
                // waited for its own loads.
                float col[GR_PPT], row[GR_PPT], w[GR_PPT], fr[GR_PPT], fc[GR_PPT];
                float q00[GR_PPT], q01[GR_PPT], q10[GR_PPT], q11[GR_PPT];
                int off[GR_PPT];
#pragma unroll
                for (int p = 0; p < GR_PPT; ++p) {
                    col[p] = fmaf(cu.x, px[p], fmaf(cu.y, py[p], fmaf(cu.z, pz[p], cu.w)));
                    row[p] = fmaf(cv.x, px[p], fmaf(cv.y, py[p], fmaf(cv.z, pz[p], cv.w)));
                    w[p] = qs;
                    if (KIND == MR_CONE) {
                        const float r = rcp_approx(fmaf(cw.x, px[p], fmaf(cw.y, py[p], fmaf(cw.z, pz[p], cw.w))));
                        col[p] *= r;
                        row[p] *= r;
                        w[p] *= r * r;
                    }
                    const float r0f = floorf(row[p]), c0f = floorf(col[p]);
                    fr[p] = row[p] - r0f;
                    fc[p] = col[p] - c0f;
                    off[p] = (int)r0f * pitch + (int)c0f;
                }
                if (MODE != GRAD_ADJOINT) {
                    const T* __restrict__ q = ring + slot;
#pragma unroll
                    for (int p = 0; p < GR_PPT; ++p) {
                        const T* a = q + off[p];
                        q00[p] = ld_elem(a);
                        q01[p] = ld_elem(a + 1);
                        q10[p] = ld_elem(a + pitch);
                        q11[p] = ld_elem(a + pitch + 1);
                    }
                }
#pragma unroll
                for (int p = 0; p < GR_PPT; ++p) {
                    if (MODE == GRAD_FORWARD) {             // samples that are not live are not written
                        const float a = fmaf(fc[p], q01[p] - q00[p], q00[p]);
                        const float b = fmaf(fc[p], q11[p] - q10[p], q10[p]);
                        acc[p] = fmaf(w[p], fmaf(fr[p], b - a, a), acc[p]);
                    } else if (MODE == GRAD_ADJOINT) {
                        if (gp[p] != 0.f) {
                            float* o = gring + slot + off[p];
                            const float a = w[p] * gp[p];
                            atomicAdd(o, a * (1.f - fr[p]) * (1.f - fc[p]));
                            atomicAdd(o + 1, a * (1.f - fr[p]) * fc[p]);
                            atomicAdd(o + pitch, a * fr[p] * (1.f - fc[p]));
                            atomicAdd(o + pitch + 1, a * fr[p] * fc[p]);
                        }
                    } else if (gp[p] != 0.f) {
                        const float dcol = fmaf(fr[p], q11[p] - q10[p], (1.f - fr[p]) * (q01[p] - q00[p]));
                        const float drow = fmaf(fc[p], q11[p] - q01[p], (1.f - fc[p]) * (q10[p] - q00[p]));
                        const float a = w[p] * gp[p];
                        ds = fmaf(a, fmaf(drow, uv, dcol), ds);
                        dt = fmaf(a, dcol * (row[p] - shift * uv - cr) - drow * (col[p] - shift - cc), dt);
                    }
                }
                continue;
            }
#pragma unroll
            for (int p = 0; p < GR_PPT; ++p) {
                if (MODE == GRAD_FORWARD ? !live[p] : gp[p] == 0.f) continue;
                float col = fmaf(cu.x, px[p], fmaf(cu.y, py[p], fmaf(cu.z, pz[p], cu.w)));
                float row = fmaf(cv.x, px[p], fmaf(cv.y, py[p], fmaf(cv.z, pz[p], cv.w)));
                float w = qs;
                if (KIND == MR_CONE) {
                    const float r = rcp_approx(fmaf(cw.x, px[p], fmaf(cw.y, py[p], fmaf(cw.z, pz[p], cw.w))));
                    col *= r;
                    row *= r;
                    w *= r * r;
                }
                const float rowc = fminf(fmaxf(row, -2.f), (float)R + 1.f);
                const float colc = fminf(fmaxf(col, -2.f), (float)C + 1.f);
                const float r0f = floorf(rowc), c0f = floorf(colc);
                const float fr = rowc - r0f, fc = colc - c0f;
                const int r0 = (int)r0f, c0 = (int)c0f;
                const bool ri0 = (unsigned)r0 < (unsigned)R, ri1 = (unsigned)(r0 + 1) < (unsigned)R;
                const bool ci0 = (unsigned)c0 < (unsigned)C, ci1 = (unsigned)(c0 + 1) < (unsigned)C;
                const long long base = slot + (long long)r0 * pitch + c0;
                if (MODE == GRAD_FORWARD) {
                    const float q00 = (ri0 && ci0) ? ld_elem(ring + base) : 0.f;
                    const float q01 = (ri0 && ci1) ? ld_elem(ring + base + 1) : 0.f;
                    const float q10 = (ri1 && ci0) ? ld_elem(ring + base + pitch) : 0.f;
                    const float q11 = (ri1 && ci1) ? ld_elem(ring + base + pitch + 1) : 0.f;
                    const float a = fmaf(fc, q01 - q00, q00);
                    const float b = fmaf(fc, q11 - q10, q10);
                    acc[p] = fmaf(w, fmaf(fr, b - a, a), acc[p]);
                } else if (MODE == GRAD_ADJOINT) {
                    const float a = w * gp[p];
                    if (ri0 && ci0) atomicAdd(gring + base, a * (1.f - fr) * (1.f - fc));
                    if (ri0 && ci1) atomicAdd(gring + base + 1, a * (1.f - fr) * fc);
                    if (ri1 && ci0) atomicAdd(gring + base + pitch, a * fr * (1.f - fc));
                    if (ri1 && ci1) atomicAdd(gring + base + pitch + 1, a * fr * fc);
                } else {
                    const float q00 = (ri0 && ci0) ? ld_elem(ring + base) : 0.f;
                    const float q01 = (ri0 && ci1) ? ld_elem(ring + base + 1) : 0.f;
                    const float q10 = (ri1 && ci0) ? ld_elem(ring + base + pitch) : 0.f;
                    const float q11 = (ri1 && ci1) ? ld_elem(ring + base + pitch + 1) : 0.f;
                    // the clamped coordinate has zero slope outside [-2, C+1] x [-2, R+1]
                    const bool live_c = col == colc, live_r = row == rowc;
                    const float dcol = live_c ? fmaf(fr, q11 - q10, (1.f - fr) * (q01 - q00)) : 0.f;
                    const float drow = live_r ? fmaf(fc, q11 - q01, (1.f - fc) * (q10 - q00)) : 0.f;
                    const float a = w * gp[p];
                    ds = fmaf(a, fmaf(drow, uv, dcol), ds);
                    dt = fmaf(a, dcol * (row - shift * uv - cr) - drow * (col - shift - cc), dt);
                }
            }
        }
    }
    if (MODE == GRAD_FORWARD && csize > 1) {
        s_part[tid] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        cluster.sync();
        if (crank == 0) {
            for (int r = 1; r < csize; ++r) {
                const float4 o = cluster.map_shared_rank(s_part, r)[tid];
                acc[0] += o.x; acc[1] += o.y; acc[2] += o.z; acc[3] += o.w;
            }
        }
    }
    if (MODE == GRAD_FORWARD && crank == 0) {
#pragma unroll
        for (int p = 0; p < GR_PPT; ++p) {
            const bool ok = pts ? (t.j0 + tid + GR_THREADS * p < g.n_j)
                                : (t.i0 + ty + di * p < g.n_i && t.j0 + tx + dj * p < g.n_j);
            if (ok) {
                const float val = live[p] ? acc[p] * g.scale : 0.f;
                gring[oidx[p]] = g.accumulate ? gring[oidx[p]] + val : val;
            }
        }
    }
    if (MODE == GRAD_GEOM) {
        double a = ds, b = dt;
        for (int o = 16; o; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if (lane == 0) { s_red[0][warp] = a; s_red[1][warp] = b; }
        __syncthreads();
        if (tid == 0) {
            double sa = 0.0, sb = 0.0;
            for (int w = 0; w < GR_THREADS / 32; ++w) { sa += s_red[0][w]; sb += s_red[1][w]; }
            atomicAdd(dgeom + 2 * t.grid, sa);
            atomicAdd(dgeom + 2 * t.grid + 1, sb);
        }
    }
    if (MODE == GRAD_FORWARD && csize > 1) cluster.sync();   // partials stay alive until read
}

template <int KIND, int MODE, typename T>
static int launch_grad(const mr_ring* ring, float* gring, const mr_view* views, const mr_grid* grids,
                       const mr_tile* tiles, int64_t n_tiles, const float* gout, double* dgeom, cudaStream_t st) {
    // CTAs per tile: enough for eight an SM, at most 8 (portable cluster). Tiles differ in how
    // many of their samples count, so short CTAs even out (256 tiles: 8 CTAs each 551, 4 each
    // 698 us for the geometry gradient); more than that cost more than they even out (864 tiles
    // of a 96 x 96 x 76 volume, 180 views: 376 us forward with one, 405 with two, 468 with four)
    int dev = 0, sms = 148;
    MR_CUDA_TRY(cudaGetDevice(&dev));
    MR_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int cl = 1;
    while (cl < 8 && n_tiles * cl < 8LL * sms) cl *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(GR_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cl;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int64_t max_chunk = 2147483647LL / cl;
    for (int64_t t0 = 0; t0 < n_tiles; t0 += max_chunk) {
        const int64_t n = (n_tiles - t0) < max_chunk ? (n_tiles - t0) : max_chunk;
        cfg.gridDim = dim3((unsigned)(n * cl));
        MR_CUDA_TRY(cudaLaunchKernelEx(&cfg, bp_grad_kernel<KIND, MODE, T>, static_cast<const T*>(ring->data), gring,
                                       ring->rows, ring->cols, ring->col_pitch, (long long)ring->slot_stride,
                                       (int)ring->n_slots, views, grids, tiles + t0, gout, dgeom));
    }
    MR_CUDA_TRY(cudaGetLastError());
    return MR_OK;
}

static int check_ring(const mr_ring* ring) {
    if (!ring || !ring->data) return MR_ERR_INVALID;
    if (ring->rows <= 0 || ring->cols <= 0 || ring->col_pitch < ring->cols) return MR_ERR_INVALID;
    if (ring->slot_stride < (int64_t)ring->rows * ring->col_pitch) return MR_ERR_INVALID;
    if (ring->kind != MR_CONE && ring->kind != MR_PARALLEL) return MR_ERR_INVALID;
    return MR_OK;
}

}  // namespace mr

extern "C" int mr_project_adjoint(const mr_ring* grad_ring, const mr_view* views, const mr_grid* grids,
                                  const mr_tile* tiles, int64_t n_tiles, const float* grad_out, void* stream) {
    int rc = mr::check_ring(grad_ring);
    if (rc != MR_OK) return rc;
    if (grad_ring->dtype != MR_F32 || !views || !grids || !grad_out || n_tiles < 0) return MR_ERR_INVALID;
    if (n_tiles > 0 && !tiles) return MR_ERR_INVALID;
    if (n_tiles == 0) return MR_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    float* g = static_cast<float*>(grad_ring->data);
    return grad_ring->kind == MR_CONE
               ? mr::launch_grad<MR_CONE, mr::GRAD_ADJOINT, float>(grad_ring, g, views, grids, tiles, n_tiles,
                                                                  grad_out, nullptr, st)
               : mr::launch_grad<MR_PARALLEL, mr::GRAD_ADJOINT, float>(grad_ring, g, views, grids, tiles,
                                                                      n_tiles, grad_out, nullptr, st);
}

extern "C" int mr_backproject_matched(const mr_ring* ring, const mr_view* views, const mr_grid* grids,
                                      const mr_tile* tiles, int64_t n_tiles, float* out, void* stream) {
    int rc = mr::check_ring(ring);
    if (rc != MR_OK) return rc;
    if (!views || !grids || !out || n_tiles < 0 || (n_tiles > 0 && !tiles)) return MR_ERR_INVALID;
    if (n_tiles == 0) return MR_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool cone = ring->kind == MR_CONE;
    switch (ring->dtype) {
        case MR_F32:
            return cone ? mr::launch_grad<MR_CONE, mr::GRAD_FORWARD, float>(ring, out, views, grids, tiles, n_tiles,
                                                                           nullptr, nullptr, st)
                        : mr::launch_grad<MR_PARALLEL, mr::GRAD_FORWARD, float>(ring, out, views, grids, tiles,
                                                                               n_tiles, nullptr, nullptr, st);
        case MR_BF16:
            return cone ? mr::launch_grad<MR_CONE, mr::GRAD_FORWARD, __nv_bfloat16>(ring, out, views, grids, tiles,
                                                                                   n_tiles, nullptr, nullptr, st)
                        : mr::launch_grad<MR_PARALLEL, mr::GRAD_FORWARD, __nv_bfloat16>(ring, out, views, grids,
                                                                                       tiles, n_tiles, nullptr,
                                                                                       nullptr, st);
        case MR_F16:
            return cone ? mr::launch_grad<MR_CONE, mr::GRAD_FORWARD, __half>(ring, out, views, grids, tiles, n_tiles,
                                                                            nullptr, nullptr, st)
                        : mr::launch_grad<MR_PARALLEL, mr::GRAD_FORWARD, __half>(ring, out, views, grids, tiles,
                                                                                n_tiles, nullptr, nullptr, st);
        default:
            return MR_ERR_INVALID;
    }
}

extern "C" int mr_bp_grad_geom(const mr_ring* ring, const mr_view* views, const mr_grid* grids,
                               const mr_tile* tiles, int64_t n_tiles, const float* grad_out,
                               double* dgeom, void* stream) {
    int rc = mr::check_ring(ring);
    if (rc != MR_OK) return rc;
    if (!views || !grids || !grad_out || !dgeom || n_tiles < 0) return MR_ERR_INVALID;
    if (n_tiles > 0 && !tiles) return MR_ERR_INVALID;
    if (n_tiles == 0) return MR_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool cone = ring->kind == MR_CONE;
    switch (ring->dtype) {
        case MR_F32:
            return cone ? mr::launch_grad<MR_CONE, mr::GRAD_GEOM, float>(ring, nullptr, views, grids, tiles,
                                                                        n_tiles, grad_out, dgeom, st)
                        : mr::launch_grad<MR_PARALLEL, mr::GRAD_GEOM, float>(ring, nullptr, views, grids, tiles,
                                                                            n_tiles, grad_out, dgeom, st);
        case MR_BF16:
            return cone ? mr::launch_grad<MR_CONE, mr::GRAD_GEOM, __nv_bfloat16>(ring, nullptr, views, grids,
                                                                                tiles, n_tiles, grad_out, dgeom, st)
                        : mr::launch_grad<MR_PARALLEL, mr::GRAD_GEOM, __nv_bfloat16>(ring, nullptr, views, grids,
                                                                                    tiles, n_tiles, grad_out, dgeom,
                                                                                    st);
        case MR_F16:
            return cone ? mr::launch_grad<MR_CONE, mr::GRAD_GEOM, __half>(ring, nullptr, views, grids, tiles,
                                                                         n_tiles, grad_out, dgeom, st)
                        : mr::launch_grad<MR_PARALLEL, mr::GRAD_GEOM, __half>(ring, nullptr, views, grids, tiles,
                                                                             n_tiles, grad_out, dgeom, st);
        default:
            return MR_ERR_INVALID;
    }
}
