// Iso-surface of a reconstructed volume by marching cubes: the contour step of minirecast
// model.py:40-69 (extract_surface), which the reference hands to VTK's flying edges (or
// scikit-image). Two passes over the cells of a float32 volume [nx][ny][nz] (z fastest):
//   mr_mc_count  triangles per block of up to 256 cells of one z row (the host scans these
//                into offsets)
//   mr_mc_emit   each cell's triangles at its block's offset + its rank inside the block:
//                per vertex the grid edge it lies on (for sharing vertices between cells)
//                and its position, interpolated in FP32 along the edge
// and an indexed mesh with shared vertices directly (what model.marching_cubes returns):
//   mr_mesh_plan the volume, read once, becomes one inside bit per grid point; crossed edges
//                and triangles are counted from the bits alone
//   mr_mesh_emit vertices in grid-edge order, then the faces of the cells, each vertex
//                number looked up as a rank among the crossed edges
// The case table is built here from the cube's geometry (the rule is described at
// build_table) and kept in constant memory, uploaded once per device; mr_mc_table hands it
// to the host so that a binding (and the tests) can check it.
#include <cmath>
#include <mutex>

#include "mr_common.cuh"

namespace mr {

constexpr int MC_THREADS = 256;
constexpr int MC_MAX_TRI = 5;

__constant__ __align__(16) int8_t c_mc_tri[256][16];          // 3 edges per triangle, -1 padding; [15] = count
__constant__ int8_t c_mc_edge[12][2];           // corners of each edge (second = first + 2^axis)

// Corners c = dx + 2 dy + 4 dz; edges 0-3 along axis 0 (from the corners with dx = 0),
// 4-7 along axis 1, 8-11 along axis 2. Per inside/outside pattern (inside: value > iso),
// every cube face is walked counter-clockwise as seen from outside; each edge where the
// walk leaves the inside corners is joined to the edge where that run of inside corners
// began, and on a face whose two inside corners are diagonal (ambiguous) each inside
// corner is cut off alone. The rule depends on the face alone, so neighbouring cells cut
// a shared face alike and the surface closes. The joined segments form loops; each loop,
// reversed, is fanned into triangles whose normals point from inside to outside, from the
// first vertex whose diagonals stay off the cube faces (a diagonal on a face would touch
// the neighbouring cell's surface along it).
static void build_table(int8_t tri[256][16], int8_t edge[12][2]) {
    int ec[12][2], ne = 0;
    for (int a = 0; a < 3; ++a)
        for (int c0 = 0; c0 < 8; ++c0)
            if (!((c0 >> a) & 1)) { ec[ne][0] = c0; ec[ne][1] = c0 | (1 << a); ++ne; }
    auto edge_of = [&](int p, int q) {
        for (int e = 0; e < 12; ++e)
            if ((ec[e][0] == p && ec[e][1] == q) || (ec[e][0] == q && ec[e][1] == p)) return e;
        return -1;
    };
    int faces[6][4];
    for (int a = 0, f = 0; a < 3; ++a)
        for (int side = 0; side < 2; ++side, ++f) {
            int cs[4], n = 0;
            for (int c = 0; c < 8; ++c)
                if (((c >> a) & 1) == side) cs[n++] = c;
            double nrm[3] = {0, 0, 0}, u[3] = {0, 0, 0}, v[3];
            nrm[a] = side ? 1.0 : -1.0;
            u[(a + 1) % 3] = 1.0;
            v[0] = nrm[1] * u[2] - nrm[2] * u[1];
            v[1] = nrm[2] * u[0] - nrm[0] * u[2];
            v[2] = nrm[0] * u[1] - nrm[1] * u[0];
            double ang[4];
            for (int i = 0; i < 4; ++i) {
                double p[3] = {(double)(cs[i] & 1) - 0.5, (double)((cs[i] >> 1) & 1) - 0.5,
                               (double)((cs[i] >> 2) & 1) - 0.5};
                p[a] = 0.0;
                ang[i] = std::atan2(p[0] * v[0] + p[1] * v[1] + p[2] * v[2], p[0] * u[0] + p[1] * u[1] + p[2] * u[2]);
            }
            for (int i = 0; i < 4; ++i)                         // sort by angle
                for (int j = i + 1; j < 4; ++j)
                    if (ang[j] < ang[i]) {
                        std::swap(ang[i], ang[j]);
                        std::swap(cs[i], cs[j]);
                    }
            for (int i = 0; i < 4; ++i) faces[f][i] = cs[i];
        }
    int eface[12] = {0};                                        // faces holding each edge (bits)
    for (int e = 0; e < 12; ++e)
        for (int f = 0; f < 6; ++f) {
            int hits = 0;
            for (int i = 0; i < 4; ++i) hits += (faces[f][i] == ec[e][0]) + (faces[f][i] == ec[e][1]);
            if (hits == 2) eface[e] |= 1 << f;
        }
    for (int m = 0; m < 256; ++m) {
        int nxt[12];
        for (int e = 0; e < 12; ++e) nxt[e] = -1;
        for (int f = 0; f < 6; ++f) {
            const int* cs = faces[f];
            int in[4];
            for (int i = 0; i < 4; ++i) in[i] = (m >> cs[i]) & 1;
            const bool amb = in[0] + in[1] + in[2] + in[3] == 2 && in[0] == in[2];
            for (int i = 0; i < 4; ++i) {
                if (!(in[i] && !in[(i + 1) % 4])) continue;
                int j = i;
                if (!amb)
                    while (in[(j + 3) % 4]) j = (j + 3) % 4;
                nxt[edge_of(cs[i], cs[(i + 1) % 4])] = edge_of(cs[(j + 3) % 4], cs[j]);
            }
        }
        int out[3 * MC_MAX_TRI], nt = 0;
        bool seen[12] = {false};
        for (int e0 = 0; e0 < 12; ++e0) {
            if (nxt[e0] < 0 || seen[e0]) continue;
            int loop[12], n = 0, e = e0;
            do {
                loop[n++] = e;
                seen[e] = true;
                e = nxt[e];
            } while (e != e0);
            for (int i = 0; i < n / 2; ++i) std::swap(loop[i], loop[n - 1 - i]);
            // fan apex: the first vertex none of whose diagonals lies on a cube face
            int r = 0;
            for (; r < n; ++r) {
                bool on_face = false;
                for (int i = 2; i < n - 1; ++i)
                    if (eface[loop[r]] & eface[loop[(r + i) % n]]) on_face = true;
                if (!on_face) break;
            }
            if (r == n) r = 0;
            for (int i = 1; i + 1 < n && nt < MC_MAX_TRI; ++i) {
                out[3 * nt] = loop[r];
                out[3 * nt + 1] = loop[(r + i) % n];
                out[3 * nt + 2] = loop[(r + i + 1) % n];
                ++nt;
            }
        }
        for (int i = 0; i < 16; ++i) tri[m][i] = -1;
        for (int i = 0; i < 3 * nt; ++i) tri[m][i] = (int8_t)out[i];
        tri[m][15] = (int8_t)nt;
    }
    for (int e = 0; e < 12; ++e) {
        edge[e][0] = (int8_t)ec[e][0];
        edge[e][1] = (int8_t)ec[e][1];
    }
}

static std::once_flag g_table_once;
static int8_t g_tri[256][16], g_edge[12][2];
static std::mutex g_upload_mutex;
static bool g_uploaded[64];

static int ensure_table() {
    std::call_once(g_table_once, [] { build_table(g_tri, g_edge); });
    int dev = 0;
    MR_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return MR_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_upload_mutex);
    if (!g_uploaded[dev]) {
        MR_CUDA_TRY(cudaMemcpyToSymbol(c_mc_tri, g_tri, sizeof(g_tri)));
        MR_CUDA_TRY(cudaMemcpyToSymbol(c_mc_edge, g_edge, sizeof(g_edge)));
        g_uploaded[dev] = true;
    }
    return MR_OK;
}

struct McArgs {
    const float* vol;
    int nx, ny, nz;
    int kchunks;                                // blocks of 256 cells along z per (i, j) row
    long long cells;
    float iso;
    float ox, oy, oz, h;
};

// Cell (i, j, k) of this thread: blocks run over rows of cells along z (blockIdx.x: 256-cell
// chunk of the row, blockIdx.y: j, blockIdx.z: i), so block order is cell memory order.
// Returns the case of the cell, or -1 past the row's end.
__device__ __forceinline__ int cell_case(const McArgs& g, int& i, int& j, int& k, float val[8]) {
    i = blockIdx.z;
    j = blockIdx.y;
    k = blockIdx.x * MC_THREADS + threadIdx.x;
    if (k >= g.nz - 1) return -1;
    const float* p = g.vol + ((long long)i * g.ny + j) * g.nz + k;
    const long long sx = (long long)g.ny * g.nz, sy = g.nz;
    int m = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        val[c] = __ldg(p + (c & 1) * sx + ((c >> 1) & 1) * sy + ((c >> 2) & 1));
        m |= (val[c] > g.iso ? 1 : 0) << c;
    }
    return m;
}

__device__ __forceinline__ long long block_id(const McArgs& g) {
    return ((long long)blockIdx.z * gridDim.y + blockIdx.y) * g.kchunks + blockIdx.x;
}

__global__ void __launch_bounds__(MC_THREADS) mc_count_kernel(McArgs g, int* __restrict__ block_counts) {
    __shared__ int warp_sum[MC_THREADS / 32];
    int i, j, k;
    float val[8];
    const int m = cell_case(g, i, j, k, val);
    int cnt = m >= 0 ? c_mc_tri[m][15] : 0;
#pragma unroll
    for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int w = 0; w < MC_THREADS / 32; ++w) s += warp_sum[w];
        block_counts[block_id(g)] = s;
    }
}

__global__ void __launch_bounds__(MC_THREADS)
mc_emit_kernel(McArgs g, const long long* __restrict__ block_offsets, long long n_tri,
               long long* __restrict__ tri_edges, float* __restrict__ tri_pos) {
    __shared__ int warp_sum[MC_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int i, j, k;
    float val[8];
    const int m = cell_case(g, i, j, k, val);
    const int cnt = m >= 0 ? c_mc_tri[m][15] : 0;
    // exclusive rank of this cell's triangles inside the block
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += warp_sum[w];
    const long long first = block_offsets[block_id(g)] + before + incl - cnt;
    for (int t = 0; t < cnt; ++t) {
        const long long o = first + t;
        if (o >= n_tri) break;                          // never write past the caller's buffers
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int e = c_mc_tri[m][3 * t + q];
            const int a = c_mc_edge[e][0], b = c_mc_edge[e][1];
            const int axis = (b - a) == 1 ? 0 : ((b - a) == 2 ? 1 : 2);
            const int ia = i + (a & 1), ja = j + ((a >> 1) & 1), ka = k + ((a >> 2) & 1);
            // FP32, each operation rounded on its own: t = (iso - va) / (vb - va)
            const float s = __fdiv_rn(__fsub_rn(g.iso, val[a]), __fsub_rn(val[b], val[a]));
            float cx = (float)ia, cy = (float)ja, cz = (float)ka;
            if (axis == 0) cx = __fadd_rn(cx, s);
            else if (axis == 1) cy = __fadd_rn(cy, s);
            else cz = __fadd_rn(cz, s);
            const long long vtx = 3 * o + q;
            tri_edges[vtx] = (((long long)ia * g.ny + ja) * g.nz + ka) * 3 + axis;
            tri_pos[3 * vtx + 0] = __fadd_rn(g.ox, __fmul_rn(g.h, cx));
            tri_pos[3 * vtx + 1] = __fadd_rn(g.oy, __fmul_rn(g.h, cy));
            tri_pos[3 * vtx + 2] = __fadd_rn(g.oz, __fmul_rn(g.h, cz));
        }
    }
}

static int fill_args(McArgs& g, const float* vol, int32_t nx, int32_t ny, int32_t nz, float iso) {
    if (!vol || nx < 2 || ny < 2 || nz < 2 || !(iso == iso)) return MR_ERR_INVALID;
    if (((uintptr_t)vol & 3u)) return MR_ERR_INVALID;
    if (nx - 1 > 65535 || ny - 1 > 65535) return MR_ERR_UNSUPPORTED;     // grid y / z limits
    g.vol = vol;
    g.nx = nx;
    g.ny = ny;
    g.nz = nz;
    g.kchunks = (nz - 1 + MC_THREADS - 1) / MC_THREADS;
    g.cells = (long long)(nx - 1) * (ny - 1) * (nz - 1);
    g.iso = iso;
    return MR_OK;
}

static dim3 mc_grid(const McArgs& g) { return dim3((unsigned)g.kchunks, (unsigned)(g.ny - 1), (unsigned)(g.nx - 1)); }

// ------------------------------------------------------------------ indexed mesh
// The grid's rows along z are cut into words of 32 points. A word's crossed edges are bit
// operations on its inside bits and its neighbours' (x: next row in i, y: next row in j,
// z: the bits shifted by one), so everything after the first pass works on 1/32 of the
// volume's size plus the surface itself: no vertex is emitted twice, and no sort is needed
// to find the copies, because the vertices are numbered in grid-edge order by prefix sums.
// The words with crossings or cut cells are listed, and the last pass takes a warp for four of them, so
// it does not matter how the surface lies in the volume (a CTA per 256 consecutive words
// took 62 us for the faces alone: most have none, some 256 words full).
// 320 x 320 x 301 voxels, 0.5 M triangles: 0.156 ms for the whole call (0.981 ms with the
// cell passes above, whose vertex copies were merged by a sort); first pass 33 us for 123 MB,
// emit 52 us, the passes over the words 43 us, the rest the host's read of the totals.
constexpr int MS_PER = 4;                         // words per thread of the passes over all words
constexpr int MS_WORDS = MC_THREADS * MS_PER;     // words per block of those passes
constexpr int MS_UNROLL = 16;                     // words a warp of the first pass loads at once
constexpr int MS_TAKE = 4;                        // listed words per warp of the last pass

struct MeshShape {
    long long words, blocks;                      // nx * ny rows of wpr words; MS_WORDS words a block
    int nx, ny, nz, wpr;
};
struct MeshSum {
    long long tri, vert, listed;
};
struct __align__(16) MeshItem {
    long long word, tri;                          // a listed word and its first triangle
};
// Workspace, in this order (the parts of 16-byte elements first)
struct MeshWs {
    MeshSum* totals;                              // padded to 32 bytes
    uint4* cross;                                 // [words] crossed x, y, z edges; first vertex (listed words)
    MeshItem* items;                              // [words] listed words, in memory order
    MeshSum* offsets;                             // [blocks] counts, then exclusive prefix sums
    uint32_t* bits;                               // [words] inside bits
    uchar2* count;                                // [words] triangles (at most 160), vertices (96)
};

static MeshShape mesh_shape(int nx, int ny, int nz) {
    MeshShape m;
    m.nx = nx; m.ny = ny; m.nz = nz;
    m.wpr = (nz + 31) / 32;
    m.words = (long long)nx * ny * m.wpr;
    m.blocks = (m.words + MS_WORDS - 1) / MS_WORDS;
    return m;
}
static MeshWs mesh_ws(void* ws, const MeshShape& m, long long* bytes = nullptr) {
    MeshWs w;
    char* p = static_cast<char*>(ws);
    long long o = 32;
    w.totals = reinterpret_cast<MeshSum*>(p);
    w.cross = reinterpret_cast<uint4*>(p + o), o += 16 * m.words;
    w.items = reinterpret_cast<MeshItem*>(p + o), o += 16 * m.words;
    w.offsets = reinterpret_cast<MeshSum*>(p + o), o += (long long)sizeof(MeshSum) * m.blocks;
    w.bits = reinterpret_cast<uint32_t*>(p + o), o += 4 * m.words;
    w.count = reinterpret_cast<uchar2*>(p + o), o += 2 * m.words;
    if (bytes) *bytes = o;
    return w;
}

// Row and word within the row of word w (a 32-bit division wherever the index fits).
__device__ __forceinline__ long long word_row(const MeshShape& m, long long w, int* seg) {
    const long long row = (unsigned long long)w >> 32 ? w / m.wpr : (long long)((uint32_t)w / (uint32_t)m.wpr);
    *seg = (int)(w - row * m.wpr);
    return row;
}

// Inside bits: a warp takes 16 consecutive words, 16 loads a lane in flight. Bound by the
// one read of the volume.
__global__ void __launch_bounds__(MC_THREADS) mesh_bits_kernel(const float* __restrict__ vol, MeshShape m, float iso,
                                                               uint32_t* __restrict__ bits) {
    const int lane = threadIdx.x & 31;
    const long long w0 = ((long long)blockIdx.x * (MC_THREADS / 32) + (threadIdx.x >> 5)) * MS_UNROLL;
    if (w0 >= m.words) return;
    int seg;
    const long long row = word_row(m, w0, &seg);
    const int words = (int)min((long long)MS_UNROLL, m.words - w0);
    const float* p = vol + row * m.nz + seg * 32 + lane;
    const int wrap = m.nz - 32 * (m.wpr - 1);     // from a row's last word to the next row
    int left = m.nz - seg * 32;                   // points of the row from this word on
    float v[MS_UNROLL];
    bool ok[MS_UNROLL];
#pragma unroll
    for (int u = 0; u < MS_UNROLL; ++u) {
        ok[u] = lane < left && u < words;
        v[u] = ok[u] ? __ldg(p) : 0.f;
        p += left > 32 ? 32 : wrap;
        left = left > 32 ? left - 32 : m.nz;
    }
    uint32_t mine = 0;
#pragma unroll
    for (int u = 0; u < MS_UNROLL; ++u) {
        const uint32_t b = __ballot_sync(0xffffffffu, ok[u] && v[u] > iso);
        if (lane == u) mine = b;
    }
    if (lane < MS_UNROLL && w0 + lane < m.words) bits[w0 + lane] = mine;
}

// The words around the cells of word w: m[c] the bits of corner row (dx, dy) = (c & 1, c >> 1),
// s[c] the same rows one point further along z.
struct WordBits {
    uint32_t m[4], s[4];
};
// What follows from them: the crossed edges along x, y, z from the word's points, and the
// cells that the surface cuts.
struct WordCuts {
    uint32_t cx, cy, cz, cells;
};
__device__ __forceinline__ WordCuts word_cuts(const WordBits& b, const MeshShape& m, int i, int j, int seg) {
    const bool x = i + 1 < m.nx, y = j + 1 < m.ny;
    const int left = m.nz - 32 * seg;             // points of the row from this word on
    const uint32_t points = left >= 32 ? 0xffffffffu : (1u << left) - 1u;
    const uint32_t steps = left > 32 ? 0xffffffffu : points >> 1;           // points with a successor
    WordCuts c;
    c.cx = x ? (b.m[0] ^ b.m[1]) & points : 0u;
    c.cy = y ? (b.m[0] ^ b.m[2]) & points : 0u;
    c.cz = (b.m[0] ^ b.s[0]) & steps;
    uint32_t any = 0, all = 0xffffffffu;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        any |= b.m[r] | b.s[r];
        all &= b.m[r] & b.s[r];
    }
    c.cells = x && y ? any & ~all & steps : 0u;
    return c;
}
__device__ __forceinline__ WordBits load_bits(const uint32_t* __restrict__ bits, const MeshShape& m, long long w, int i,
                                              int j, int seg) {
    WordBits b;
    const bool x = i + 1 < m.nx, y = j + 1 < m.ny, more = seg + 1 < m.wpr;
    const long long dx = (long long)m.ny * m.wpr, dy = m.wpr;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const bool ok = ((c & 1) == 0 || x) && ((c >> 1) == 0 || y);
        const uint32_t* p = bits + w + (c & 1) * dx + (c >> 1) * dy;
        b.m[c] = ok ? __ldg(p) : 0u;
        b.s[c] = (b.m[c] >> 1) | ((ok && more ? __ldg(p + 1) : 0u) << 31);
    }
    return b;
}
__device__ __forceinline__ int word_case(const WordBits& b, int k) {
    int r = 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) r |= (int)((b.m[c] >> k) & 1u) << c | (int)((b.s[c] >> k) & 1u) << (c + 4);
    return r;
}
__device__ __forceinline__ int warp_inclusive(int v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// Triangles, vertices and whether listed, per word and per block.
__global__ void __launch_bounds__(MC_THREADS) mesh_count_kernel(MeshShape m, MeshWs ws) {
    __shared__ int sum[3][MC_THREADS / 32];
    __shared__ uint8_t count[256];
    count[threadIdx.x] = (uint8_t)c_mc_tri[threadIdx.x][15];
    __syncthreads();
    const long long w0 = (long long)blockIdx.x * MS_WORDS + threadIdx.x;
    WordBits b[MS_PER];
    WordCuts c[MS_PER];
#pragma unroll
    for (int u = 0; u < MS_PER; ++u) {
        const long long w = w0 + u * MC_THREADS;
        c[u] = WordCuts{0, 0, 0, 0};
        if (w >= m.words) continue;
        int seg;
        const uint32_t row = (uint32_t)word_row(m, w, &seg);    // nx, ny <= 65536: rows fit 32 bits
        const int i = (int)(row / (uint32_t)m.ny), j = (int)(row - (uint32_t)i * (uint32_t)m.ny);
        b[u] = load_bits(ws.bits, m, w, i, j, seg);
        c[u] = word_cuts(b[u], m, i, j, seg);
    }
    int tri = 0, vert = 0, listed = 0;
#pragma unroll
    for (int u = 0; u < MS_PER; ++u) {
        const long long w = w0 + u * MC_THREADS;
        const int v = __popc(c[u].cx) + __popc(c[u].cy) + __popc(c[u].cz);
        int t = 0;
        for (uint32_t left = c[u].cells; left; left &= left - 1) t += count[word_case(b[u], __ffs(left) - 1)];
        if (w < m.words) ws.count[w] = make_uchar2((unsigned char)t, (unsigned char)v);
        tri += t;
        vert += v;
        listed += (t | v) != 0;                   // a cell may be cut on its other rows' edges alone
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    tri = __reduce_add_sync(0xffffffffu, tri);
    vert = __reduce_add_sync(0xffffffffu, vert);
    listed = __reduce_add_sync(0xffffffffu, listed);
    if (lane == 0) { sum[0][warp] = tri; sum[1][warp] = vert; sum[2][warp] = listed; }
    __syncthreads();
    if (threadIdx.x == 0) {
        MeshSum s = {0, 0, 0};
        for (int w = 0; w < MC_THREADS / 32; ++w) { s.tri += sum[0][w]; s.vert += sum[1][w]; s.listed += sum[2][w]; }
        ws.offsets[blockIdx.x] = s;
    }
}

// Exclusive prefix sums of the block counts and their totals: one block, a count a thread and
// round (8 rounds for a 640^3 volume).
__global__ void __launch_bounds__(1024) mesh_scan_kernel(MeshWs ws, long long n) {
    __shared__ MeshSum warp_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    MeshSum carry = {0, 0, 0};
    for (long long at = threadIdx.x; at - threadIdx.x < n; at += 1024) {
        const MeshSum v = at < n ? ws.offsets[at] : MeshSum{0, 0, 0};
        MeshSum incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, incl.tri, o), p = __shfl_up_sync(0xffffffffu, incl.vert, o),
                            l = __shfl_up_sync(0xffffffffu, incl.listed, o);
            if (lane >= o) { incl.tri += t; incl.vert += p; incl.listed += l; }
        }
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        MeshSum before = carry;
        for (int w = 0; w < 32; ++w) {
            const MeshSum t = warp_sum[w];
            if (w < warp) { before.tri += t.tri; before.vert += t.vert; before.listed += t.listed; }
            carry.tri += t.tri; carry.vert += t.vert; carry.listed += t.listed;
        }
        if (at < n)
            ws.offsets[at] = MeshSum{before.tri + incl.tri - v.tri, before.vert + incl.vert - v.vert,
                                     before.listed + incl.listed - v.listed};
        __syncthreads();
    }
    if (threadIdx.x == 0) *ws.totals = carry;
}

// The list of words with crossings or cut cells, each with its first triangle and first vertex.
__global__ void __launch_bounds__(MC_THREADS) mesh_list_kernel(MeshShape m, MeshWs ws) {
    __shared__ int3 warp_sum[MS_PER][MC_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long w0 = (long long)blockIdx.x * MS_WORDS + threadIdx.x;
    int3 own[MS_PER], incl[MS_PER];
#pragma unroll
    for (int u = 0; u < MS_PER; ++u) {
        const long long w = w0 + u * MC_THREADS;
        const uchar2 c = w < m.words ? ws.count[w] : make_uchar2(0, 0);
        own[u] = make_int3(c.x, c.y, (c.x | c.y) != 0);
    }
#pragma unroll
    for (int u = 0; u < MS_PER; ++u) {
        incl[u] = make_int3(warp_inclusive(own[u].x, lane), warp_inclusive(own[u].y, lane),
                            warp_inclusive(own[u].z, lane));
        if (lane == 31) warp_sum[u][warp] = incl[u];
    }
    __syncthreads();
    const MeshSum base = ws.offsets[blockIdx.x];
    int3 before = make_int3(0, 0, 0);
#pragma unroll
    for (int u = 0; u < MS_PER; ++u) {
        for (int x = 0; x < MC_THREADS / 32; ++x) {
            const int3 t = warp_sum[u][x];
            if (x == warp && own[u].z) {
                const long long w = w0 + u * MC_THREADS;
                int seg;
                const uint32_t row = (uint32_t)word_row(m, w, &seg);
                const int i = (int)(row / (uint32_t)m.ny), j = (int)(row - (uint32_t)i * (uint32_t)m.ny);
                const WordCuts c = word_cuts(load_bits(ws.bits, m, w, i, j, seg), m, i, j, seg);
                const long long v = base.vert + before.y + incl[u].y - own[u].y;
                ws.cross[w] = make_uint4(c.cx, c.cy, c.cz, (uint32_t)v);
                ws.items[base.listed + before.z + incl[u].z - own[u].z] =
                    MeshItem{w, base.tri + before.x + incl[u].x - own[u].x};
            }
            before.x += t.x;
            before.y += t.y;
            before.z += t.z;
        }
    }
}

struct MeshGeom {
    float iso, ox, oy, oz, h;
};

// The mesh: a warp takes four listed words. Lane 8 q + p first fetches part p (row p & 3,
// successor along z p >> 2) of what word q's cells reach, all four words at once; then, word
// by word, a lane is a point (its vertices) and a cell (its faces). A vertex number is the
// first one of its point's word plus the crossed edges below the point (all axes) plus those
// of the point itself along earlier axes. The case table is read from shared memory: the
// lanes' cases differ, which constant memory would serialise.
__global__ void __launch_bounds__(MC_THREADS)
mesh_emit_kernel(const float* __restrict__ vol, MeshShape m, MeshWs ws, MeshGeom g, long long n_tri, long long n_vert,
                 float* __restrict__ points, long long* __restrict__ faces) {
    __shared__ __align__(16) int8_t table[256][16];
    __shared__ uint4 reach[MC_THREADS / 32][32];
    __shared__ uint32_t rows[MC_THREADS / 32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    *reinterpret_cast<int4*>(table[threadIdx.x]) = *reinterpret_cast<const int4*>(c_mc_tri[threadIdx.x]);
    const long long listed = ws.totals->listed;
    const long long e0 = ((long long)blockIdx.x * (MC_THREADS / 32) + warp) * MS_TAKE;
    MeshItem item = {0, 0};
    int wi = 0, wj = 0, seg = 0;
    uint4 cr = make_uint4(0, 0, 0, 0);
    uint32_t bits = 0;
    if (e0 + (lane >> 3) < listed) {
        item = ws.items[e0 + (lane >> 3)];
        const uint32_t row = (uint32_t)word_row(m, item.word, &seg);
        wi = (int)(row / (uint32_t)m.ny);
        wj = (int)(row - (uint32_t)wi * (uint32_t)m.ny);
        const int dx = lane & 1, dy = (lane >> 1) & 1, dz = (lane >> 2) & 1;
        if (wi + dx < m.nx && wj + dy < m.ny && seg + dz < m.wpr) {
            const long long at = item.word + dx * (long long)m.ny * m.wpr + dy * m.wpr + dz;
            cr = __ldg(ws.cross + at);                    // unset where nothing crosses: not used then
            bits = __ldg(ws.bits + at);
        }
    }
    reach[warp][lane] = cr;
    rows[warp][lane] = bits;
    __syncthreads();
    const uint32_t below = (1u << lane) - 1u;
    // the values at both ends of every crossed edge, all four words' loads in flight together
    float va[MS_TAKE], vb[MS_TAKE][3];
#pragma unroll
    for (int q = 0; q < MS_TAKE; ++q) {
        const uint4 own = reach[warp][8 * q];             // 0 past the list's end
        const long long row = (long long)__shfl_sync(0xffffffffu, wi, 8 * q) * m.ny + __shfl_sync(0xffffffffu, wj, 8 * q);
        const float* p = vol + row * m.nz + 32 * __shfl_sync(0xffffffffu, seg, 8 * q) + lane;
        if (((own.x | own.y | own.z) >> lane) & 1u) va[q] = __ldg(p);
        if ((own.x >> lane) & 1u) vb[q][0] = __ldg(p + (long long)m.ny * m.nz);
        if ((own.y >> lane) & 1u) vb[q][1] = __ldg(p + m.nz);
        if ((own.z >> lane) & 1u) vb[q][2] = __ldg(p + 1);
    }
#pragma unroll
    for (int q = 0; q < MS_TAKE; ++q) {
        if (e0 + q >= listed) break;
        const int i = __shfl_sync(0xffffffffu, wi, 8 * q), j = __shfl_sync(0xffffffffu, wj, 8 * q);
        const int sg = __shfl_sync(0xffffffffu, seg, 8 * q);
        WordBits b;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            b.m[c] = rows[warp][8 * q + c];
            b.s[c] = (b.m[c] >> 1) | (rows[warp][8 * q + 4 + c] << 31);
        }
        const uint4 own = reach[warp][8 * q];
        const uint32_t wc[3] = {own.x, own.y, own.z};
        long long o = (long long)own.w + __popc(own.x & below) + __popc(own.y & below) + __popc(own.z & below);
#pragma unroll
        for (int axis = 0; axis < 3; ++axis) {
            if (!((wc[axis] >> lane) & 1u)) continue;
            if (o >= n_vert) break;                       // never write past the caller's buffer
            // FP32, each operation rounded on its own: t = (iso - va) / (vb - va)
            const float s = __fdiv_rn(__fsub_rn(g.iso, va[q]), __fsub_rn(vb[q][axis], va[q]));
            float c[3] = {(float)i, (float)j, (float)(32 * sg + lane)};
            c[axis] = __fadd_rn(c[axis], s);
            points[3 * o + 0] = __fadd_rn(g.ox, __fmul_rn(g.h, c[0]));
            points[3 * o + 1] = __fadd_rn(g.oy, __fmul_rn(g.h, c[1]));
            points[3 * o + 2] = __fadd_rn(g.oz, __fmul_rn(g.h, c[2]));
            ++o;
        }
        const uint32_t cells = word_cuts(b, m, i, j, sg).cells;
        const int8_t* row = table[(cells >> lane) & 1u ? word_case(b, lane) : 0];
        const int cnt = row[15];                          // 0 for an uncut cell
        long long f = __shfl_sync(0xffffffffu, item.tri, 8 * q) + warp_inclusive(cnt, lane) - cnt;
        for (int t = 0; t < cnt; ++t, ++f) {
            if (f >= n_tri) break;                        // never write past the caller's buffer
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                // edge number -> axis and lower corner (4 edges an axis, corners ascending)
                const int ed = row[3 * t + x];
                const int a = (int)(0x321054106420ull >> (4 * ed)) & 7, axis = ed >> 2;
                const int at = lane + (a >> 2), bit = at & 31;
                const uint4 r = reach[warp][8 * q + (a & 3) + 4 * (at >> 5)];
                const uint32_t low = (1u << bit) - 1u;
                uint32_t v = r.w + __popc(r.x & low) + __popc(r.y & low) + __popc(r.z & low);
                if (axis > 0) v += (r.x >> bit) & 1u;
                if (axis > 1) v += (r.y >> bit) & 1u;
                faces[3 * f + x] = (long long)v;
            }
        }
    }
}

static int mesh_args(const float* vol, int32_t nx, int32_t ny, int32_t nz, float iso, const void* ws, MeshShape* m) {
    McArgs g{};
    const int rc = fill_args(g, vol, nx, ny, nz, iso);
    if (rc != MR_OK) return rc;
    if (!ws || ((uintptr_t)ws & 15u)) return MR_ERR_INVALID;
    *m = mesh_shape(nx, ny, nz);
    return m->blocks > 2147483647LL ? MR_ERR_UNSUPPORTED : MR_OK;
}

}  // namespace mr

extern "C" int64_t mr_mc_blocks(int32_t nx, int32_t ny, int32_t nz) {
    if (nx < 2 || ny < 2 || nz < 2) return 0;
    return (int64_t)(nx - 1) * (ny - 1) * ((nz - 1 + mr::MC_THREADS - 1) / mr::MC_THREADS);
}

extern "C" int mr_mc_table(int8_t* table_host) {
    if (!table_host) return MR_ERR_INVALID;
    std::call_once(mr::g_table_once, [] { mr::build_table(mr::g_tri, mr::g_edge); });
    for (int m = 0; m < 256; ++m)
        for (int i = 0; i < 16; ++i) table_host[16 * m + i] = mr::g_tri[m][i];
    return MR_OK;
}

extern "C" int mr_mc_count(const float* vol, int32_t nx, int32_t ny, int32_t nz, float iso, int32_t* block_counts,
                           void* stream) {
    mr::McArgs g{};
    int rc = mr::fill_args(g, vol, nx, ny, nz, iso);
    if (rc != MR_OK) return rc;
    if (!block_counts) return MR_ERR_INVALID;
    rc = mr::ensure_table();
    if (rc != MR_OK) return rc;
    mr::mc_count_kernel<<<mr::mc_grid(g), mr::MC_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(g, block_counts);
    MR_CUDA_TRY(cudaGetLastError());
    return MR_OK;
}

extern "C" int mr_mc_emit(const float* vol, int32_t nx, int32_t ny, int32_t nz, float iso, const double* origin,
                          double spacing, const int64_t* block_offsets, int64_t n_tri, int64_t* tri_edges,
                          float* tri_pos, void* stream) {
    mr::McArgs g{};
    int rc = mr::fill_args(g, vol, nx, ny, nz, iso);
    if (rc != MR_OK) return rc;
    if (!origin || !block_offsets || n_tri < 0 || (n_tri > 0 && (!tri_edges || !tri_pos))) return MR_ERR_INVALID;
    rc = mr::ensure_table();
    if (rc != MR_OK) return rc;
    if (n_tri == 0) return MR_OK;
    g.ox = (float)origin[0];
    g.oy = (float)origin[1];
    g.oz = (float)origin[2];
    g.h = (float)spacing;
    mr::mc_emit_kernel<<<mr::mc_grid(g), mr::MC_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
        g, reinterpret_cast<const long long*>(block_offsets), (long long)n_tri,
        reinterpret_cast<long long*>(tri_edges), tri_pos);
    MR_CUDA_TRY(cudaGetLastError());
    return MR_OK;
}

extern "C" int64_t mr_mesh_workspace_bytes(int32_t nx, int32_t ny, int32_t nz) {
    if (nx < 2 || ny < 2 || nz < 2) return 0;
    long long bytes = 0;
    mr::mesh_ws(nullptr, mr::mesh_shape(nx, ny, nz), &bytes);
    return bytes;
}

extern "C" int mr_mesh_plan(const float* vol, int32_t nx, int32_t ny, int32_t nz, float iso, void* ws,
                            int64_t* totals_host, void* stream) {
    mr::MeshShape m;
    int rc = mr::mesh_args(vol, nx, ny, nz, iso, ws, &m);
    if (rc != MR_OK) return rc;
    if (!totals_host) return MR_ERR_INVALID;
    rc = mr::ensure_table();
    if (rc != MR_OK) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const mr::MeshWs w = mr::mesh_ws(ws, m);
    constexpr int per = mr::MC_THREADS / 32 * mr::MS_UNROLL;            // words per block of the first pass
    mr::mesh_bits_kernel<<<(unsigned)((m.words + per - 1) / per), mr::MC_THREADS, 0, st>>>(vol, m, iso, w.bits);
    mr::mesh_count_kernel<<<(unsigned)m.blocks, mr::MC_THREADS, 0, st>>>(m, w);
    mr::mesh_scan_kernel<<<1, 1024, 0, st>>>(w, m.blocks);
    mr::mesh_list_kernel<<<(unsigned)m.blocks, mr::MC_THREADS, 0, st>>>(m, w);
    MR_CUDA_TRY(cudaGetLastError());
    MR_CUDA_TRY(cudaMemcpyAsync(totals_host, w.totals, 3 * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    MR_CUDA_TRY(cudaStreamSynchronize(st));
    return totals_host[1] > 0xffffffffLL ? MR_ERR_UNSUPPORTED : MR_OK;
}

extern "C" int mr_mesh_emit(const float* vol, int32_t nx, int32_t ny, int32_t nz, float iso, const double* origin,
                            double spacing, void* ws, const int64_t* totals_host, float* points, int64_t* faces,
                            void* stream) {
    mr::MeshShape m;
    int rc = mr::mesh_args(vol, nx, ny, nz, iso, ws, &m);
    if (rc != MR_OK) return rc;
    if (!origin || !totals_host) return MR_ERR_INVALID;
    const int64_t n_tri = totals_host[0], n_vert = totals_host[1], listed = totals_host[2];
    if (n_tri < 0 || n_vert < 0 || listed < 0 || listed > m.words) return MR_ERR_INVALID;
    if ((n_vert > 0 && !points) || (n_tri > 0 && !faces)) return MR_ERR_INVALID;
    if (listed == 0) return MR_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const mr::MeshWs w = mr::mesh_ws(ws, m);
    const mr::MeshGeom g = {iso, (float)origin[0], (float)origin[1], (float)origin[2], (float)spacing};
    constexpr int per = mr::MC_THREADS / 32 * mr::MS_TAKE;              // listed words per block
    mr::mesh_emit_kernel<<<(unsigned)((listed + per - 1) / per), mr::MC_THREADS, 0, st>>>(
        vol, m, w, g, (long long)n_tri, (long long)n_vert, points, reinterpret_cast<long long*>(faces));
    MR_CUDA_TRY(cudaGetLastError());
    return MR_OK;
}
