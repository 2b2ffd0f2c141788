// GPU marching cubes for block-wise mesh extraction.
//
// Reference path: projects/neuralangelo/utils/mesh.py
//   marching_cubes (:119-133)           -> PyMCubes on the CPU, then V * intv + xyz[0,0,0]
//   filter_points_outside_bounding_sphere (:136-148)
// Here one block volume [nx, ny, nz] (float32, x-major, already negated as
// scripts/extract_mesh.py:85 does) goes through classify -> exclusive scan -> emit
// on the device:
//   1. crossing edges (grid edge (i,j,k,axis) whose end values straddle iso) whose vertex
//      passes the unit-sphere filter (|v| < 1); the vertex in double: t = (iso - v0) /
//      (v1 - v0), index-space position, * intv + origin;
//   2. triangles of every cube whose vertices are all kept, from the case table;
//   3. sums per block of points, scanned: vertices are numbered in global edge order
//      ((i*ny + j)*nz + k)*3 + axis, faces in x-major cube order;
//   4. vertices and faces.
// The case table follows the canonical triangulation stated in oracle/mc.c
// (face walks with positive corners separated on ambiguous faces, loops fanned
// from their smallest edge id); it is generated on the host at first use.
#include <mutex>

#include "common.cuh"

namespace gbsdf {

// ---------------------------------------------------------------------------
// case table (host generation)

struct McTable {
    int8_t tri[256][16][3];   // edge ids, -1 padded
    int8_t count[256];
};

static int mc_edge_of_pair(int ca, int cb) {
    const int d = ca ^ cb;
    const int axis = d == 1 ? 0 : (d == 2 ? 1 : 2);
    const int lo = ca & cb;
    // the two remaining axes, ascending, give the bits of the edge's rank
    int others[2], m = 0;
    for (int ax = 0; ax < 3; ++ax)
        if (ax != axis) others[m++] = ax;
    const int r = ((lo >> others[0]) & 1) | (((lo >> others[1]) & 1) << 1);
    return axis * 4 + r;
}

static void mc_build_table(McTable& t) {
    // counter-clockwise corner cycle of every face as seen from outside the cube
    int cycles[6][4];
    for (int f = 0; f < 6; ++f) {
        const int n = f >> 1, side = f & 1, u = (n + 1) % 3, w = (n + 2) % 3;
        static const int uv[4][2] = {{0, 0}, {1, 0}, {1, 1}, {0, 1}};
        for (int k = 0; k < 4; ++k) {
            const int q = side ? k : (4 - k) & 3;
            cycles[f][k] = (side << n) | (uv[q][0] << u) | (uv[q][1] << w);
        }
    }
    for (int cfg = 0; cfg < 256; ++cfg) {
        int succ[12];
        for (int e = 0; e < 12; ++e) succ[e] = -1;
        for (int f = 0; f < 6; ++f) {
            const int* cy = cycles[f];
            bool pos[4];
            for (int k = 0; k < 4; ++k) pos[k] = (cfg >> cy[k]) & 1;
            for (int k = 0; k < 4; ++k) {
                if (!pos[k] || pos[(k + 1) & 3]) continue;       // not an exit
                int j = k;
                while (pos[j]) j = (j + 3) & 3;                   // walk back over the positive run
                succ[mc_edge_of_pair(cy[k], cy[(k + 1) & 3])] = mc_edge_of_pair(cy[j], cy[(j + 1) & 3]);
            }
        }
        bool seen[12] = {false};
        int nt = 0;
        for (int e = 0; e < 12; ++e) {
            if (succ[e] < 0 || seen[e]) continue;
            int loop[12], m = 0;
            for (int x = e; !seen[x]; x = succ[x]) {
                seen[x] = true;
                loop[m++] = x;
            }
            for (int i = 1; i + 1 < m; ++i) {
                t.tri[cfg][nt][0] = (int8_t)loop[0];
                t.tri[cfg][nt][1] = (int8_t)loop[i + 1];
                t.tri[cfg][nt][2] = (int8_t)loop[i];
                ++nt;
            }
        }
        t.count[cfg] = (int8_t)nt;
        for (int k = nt; k < 16; ++k) t.tri[cfg][k][0] = t.tri[cfg][k][1] = t.tri[cfg][k][2] = -1;
    }
}

static const McTable& mc_table() {
    static McTable t;
    static std::once_flag once;
    std::call_once(once, [] { mc_build_table(t); });
    return t;
}

__constant__ int8_t c_tri[256][16][3];
__constant__ int8_t c_count[256];

static int upload_table_once() {
    // constant memory is per device: upload on every device the first time it is used
    static bool done[64] = {false};
    static std::mutex mu;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    if (dev >= 0 && dev < 64 && done[dev]) return GBSDF_OK;
    const McTable& t = mc_table();
    if (cudaMemcpyToSymbol(c_tri, t.tri, sizeof(t.tri)) != cudaSuccess ||
        cudaMemcpyToSymbol(c_count, t.count, sizeof(t.count)) != cudaSuccess) {
        set_error("uploading the marching-cubes table failed: %s", cudaGetErrorString(cudaGetLastError()));
        return GBSDF_ERR_CUDA;
    }
    if (dev >= 0 && dev < 64) done[dev] = true;
    return GBSDF_OK;
}

__device__ __forceinline__ void edge_lo_corner(int e, int& a, int& dx, int& dy, int& dz) {
    a = e >> 2;
    const int r = e & 3;
    // the two other axes ascending take the bits of r
    if (a == 0) { dx = 0; dy = r & 1; dz = r >> 1; }
    else if (a == 1) { dx = r & 1; dy = 0; dz = r >> 1; }
    else { dx = r & 1; dy = r >> 1; dz = 0; }
}

// ---------------------------------------------------------------------------
// marching-cubes kernels

struct McDims {
    int nx, ny, nz;
};

__device__ __forceinline__ int64_t vol_index(const McDims& d, int i, int j, int k) {
    return ((int64_t)i * d.ny + j) * d.nz + k;
}

// A thread block takes 512 consecutive lattice points, a thread four of them: one division by the
// lattice's extents, one place in the block's scan and 32-bit accesses of the byte arrays for four
// points.  With a point per thread the four kernels of a 129^3 block took 97 us, most of it for points
// away from the surface; this way 35.
constexpr int MC_PER = 4, MC_T = 128, MC_POINTS = MC_T * MC_PER;

// A point owns its three edges (towards +x, +y, +z) and the cube at its +x +y +z side, so that point
// order is edge order and cube order at once.
struct McPoint {
    int i, j, k;
};
__device__ __forceinline__ McPoint mc_point(const McDims& d, uint32_t p) {
    McPoint q;
    const uint32_t ij = p / (uint32_t)d.nz;
    q.k = (int)(p - ij * (uint32_t)d.nz);
    q.i = (int)(ij / (uint32_t)d.ny);
    q.j = (int)(ij - (uint32_t)q.i * (uint32_t)d.ny);
    return q;
}
__device__ __forceinline__ void mc_next(const McDims& d, McPoint& q) {
    if (++q.k == d.nz) {
        q.k = 0;
        if (++q.j == d.ny) {
            q.j = 0;
            ++q.i;
        }
    }
}
// iso rounded down to float: a float lies above it exactly when it lies above iso (the chip has
// little double arithmetic, and this comparison runs for every point)
__device__ __forceinline__ float mc_iso(double iso) { return __double2float_rd(iso); }

// the vertex on the edge along axis a: t = (iso - v0) / (v1 - v0) in double, index space * intv + origin
struct McGeometry {
    double iso, intv, org[3];
};
__device__ __forceinline__ void mc_vertex(const McGeometry& g, const McPoint& q, int a, float f0, float f1, double* x) {
    const double v0 = f0, v1 = f1;
    const double t = __ddiv_rn(__dsub_rn(g.iso, v0), __dsub_rn(v1, v0));
    const double idx[3] = {(double)q.i, (double)q.j, (double)q.k};
#pragma unroll
    for (int c = 0; c < 3; ++c)
        x[c] = __dadd_rn(__dmul_rn(c == a ? __dadd_rn(idx[c], t) : idx[c], g.intv), g.org[c]);
}

// unit-sphere filter (mesh.py:136-148): |v| < 1 in double.  Both ends of the edge inside a
// slightly smaller sphere decide it without the double arithmetic (a vertex of finite values lies
// between them), which the chip has little of.
__device__ __forceinline__ bool mc_keeps(const McGeometry& g, const McPoint& q, int a, float f0, float f1) {
    if (isfinite(f0) && isfinite(f1)) {
        const float intv = (float)g.intv;
        float r0 = 0.0f, r1 = 0.0f;
        const int idx[3] = {q.i, q.j, q.k};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float x0 = (float)idx[c] * intv + (float)g.org[c], x1 = (float)(idx[c] + (c == a)) * intv + (float)g.org[c];
            r0 = fmaf(x0, x0, r0);
            r1 = fmaf(x1, x1, r1);
        }
        // (float coordinates below 1 built from at most 2^28 steps: off by less than 1e-3 unless origin
        // and steps nearly cancel, which the bound on the origin rules out)
        if (r0 < 0.99f && r1 < 0.99f && fabs(g.org[0]) < 1e3 && fabs(g.org[1]) < 1e3 && fabs(g.org[2]) < 1e3) return true;
    }
    double x[3];
    mc_vertex(g, q, a, f0, f1, x);
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(x[0], x[0]), __dmul_rn(x[1], x[1])), __dmul_rn(x[2], x[2]))) < 1.0;
}

// sum over the block; every thread's `before` is the sum over earlier threads
__device__ __forceinline__ uint32_t mc_block_scan(uint32_t v, uint32_t* warp_s, uint32_t& before) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_s[warp] = x;
    __syncthreads();
    uint32_t total = 0;
    before = x - v;
#pragma unroll
    for (int w = 0; w < MC_T / 32; ++w) {
        before += w < warp ? warp_s[w] : 0u;
        total += warp_s[w];
    }
    return total;
}

// 1: the kept crossing edges of every point (bits 0-2 of code), whether its cube has triangles
// (bit 3) and which (cfg); kept vertices per block
__global__ void __launch_bounds__(MC_T) k_mc_classify(const float* __restrict__ vol, McDims d, McGeometry g, uint32_t np,
                                                      uint8_t* __restrict__ code, uint8_t* __restrict__ cfg,
                                                      uint2* __restrict__ sums) {
    __shared__ uint32_t total;
    const uint32_t p = (blockIdx.x * (uint32_t)MC_T + threadIdx.x) * MC_PER;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    uint32_t codes = 0;
    if (p < np) {
        const uint32_t sx = (uint32_t)d.ny * (uint32_t)d.nz, sy = (uint32_t)d.nz;
        const float iso = mc_iso(g.iso);
        // signs of the points and of their +x, +y and +x +y neighbours, and one further along z
        // (np is at most 2^28 and the steps below np: no index wraps)
        auto signs = [&](uint32_t at) {
            uint32_t m = 0;
#pragma unroll
            for (int u = 0; u <= MC_PER; ++u)
                if (at + u < np) m |= (uint32_t)(vol[at + u] > iso) << u;
            return m;
        };
        const uint32_t s0 = signs(p), s1 = signs(p + sx), s2 = signs(p + sy), s3 = signs(p + sx + sy);
        const McPoint q0 = mc_point(d, p);
        McPoint q = q0;
        uint32_t cross = 0, cfgs = 0;                 // crossing edges: bit 4u + axis
#pragma unroll
        for (int u = 0; u < MC_PER; ++u, mc_next(d, q)) {
            if (p + u >= np) break;
            const bool hx = q.i + 1 < d.nx, hy = q.j + 1 < d.ny, hz = q.k + 1 < d.nz;
            // corner c: +1 along axis a where bit a is set
            const uint32_t c = ((s0 >> u) & 1u) | ((s1 >> u) & 1u) << 1 | ((s2 >> u) & 1u) << 2 | ((s3 >> u) & 1u) << 3 |
                               ((s0 >> (u + 1)) & 1u) << 4 | ((s1 >> (u + 1)) & 1u) << 5 | ((s2 >> (u + 1)) & 1u) << 6 |
                               ((s3 >> (u + 1)) & 1u) << 7;
            if (hx && hy && hz && c != 0 && c != 255) {
                codes |= 8u << (8 * u);
                cfgs |= c << (8 * u);
            }
            const uint32_t diff = (c & 1u) ? ~c : c;  // bits 1, 2, 4: the +x, +y, +z neighbour's sign differs
            cross |= ((hx ? (diff >> 1) & 1u : 0u) | (hy ? (diff >> 1) & 2u : 0u) | (hz ? (diff >> 2) & 4u : 0u)) << (4 * u);
        }
        if (cfgs) *reinterpret_cast<uint32_t*>(cfg + p) = cfgs;
        for (; cross; cross &= cross - 1) {           // few: the edges through the surface
            const int b = __ffs(cross) - 1, u = b >> 2, a = b & 3;
            McPoint e = q0;
            for (int i = 0; i < u; ++i) mc_next(d, e);
            if (mc_keeps(g, e, a, vol[p + u], vol[p + u + (a == 0 ? sx : a == 1 ? sy : 1u)])) codes |= 1u << (8 * u + a);
        }
        *reinterpret_cast<uint32_t*>(code + p) = codes;
    }
    if (codes & 0x07070707u) atomicAdd(&total, (uint32_t)__popc(codes & 0x07070707u));
    __syncthreads();
    if (threadIdx.x == 0) sums[blockIdx.x].x = total;
}

// Steps 2, 4 and 5 first list the block's items (few: the surface passes through), then take one
// per thread: spread over the points, a warp would run the table walk or the double division for a
// lane or two.

// 2: kept triangles of every cube (tri[p], a bit each, in table order) and per block
__global__ void __launch_bounds__(MC_T) k_mc_count_faces(McDims d, uint32_t np, const uint8_t* __restrict__ code,
                                                         const uint8_t* __restrict__ cfg, uint8_t* __restrict__ tri,
                                                         uint2* __restrict__ sums) {
    __shared__ uint32_t warp_s[MC_T / 32];
    __shared__ uint16_t list[MC_POINTS];
    __shared__ uint32_t faces;
    const uint32_t p0 = blockIdx.x * (uint32_t)MC_POINTS, p = p0 + threadIdx.x * MC_PER;
    const uint32_t active = p < np ? *reinterpret_cast<const uint32_t*>(code + p) & 0x08080808u : 0u;
    if (p < np) *reinterpret_cast<uint32_t*>(tri + p) = 0;
    if (threadIdx.x == 0) faces = 0;
    uint32_t at;
    const uint32_t n = mc_block_scan(__popc(active), warp_s, at);
    for (uint32_t left = active; left; left &= left - 1) list[at++] = (uint16_t)(threadIdx.x * MC_PER + (__ffs(left) >> 3));
    __syncthreads();
    for (uint32_t r = threadIdx.x; r < n; r += MC_T) {
        const uint32_t pt = p0 + list[r];
        const McPoint q = mc_point(d, pt);
        const int c = cfg[pt];
        // the kept vertices of the cube's twelve edges
        uint32_t edges = 0;
#pragma unroll
        for (int e = 0; e < 12; ++e) {
            int a, dx, dy, dz;
            edge_lo_corner(e, a, dx, dy, dz);
            edges |= ((uint32_t)(code[vol_index(d, q.i + dx, q.j + dy, q.k + dz)] >> a) & 1u) << e;
        }
        uint32_t kept = 0;
        const int nt = c_count[c];
        for (int t = 0; t < nt; ++t) {
            const uint32_t need = 1u << c_tri[c][t][0] | 1u << c_tri[c][t][1] | 1u << c_tri[c][t][2];
            if ((edges & need) == need) kept |= 1u << t;
        }
        tri[pt] = (uint8_t)kept;
        if (kept) atomicAdd(&faces, (uint32_t)__popc(kept));
    }
    __syncthreads();
    if (threadIdx.x == 0) sums[blockIdx.x].y = faces;
}

// 3: exclusive sums over the blocks (one thread block, eight entries per thread and round)
constexpr int MC_SCAN_T = 1024, MC_SCAN_PER = 8;
__global__ void __launch_bounds__(MC_SCAN_T) k_mc_scan_blocks(uint2* __restrict__ sums, uint32_t nb,
                                                              int64_t* __restrict__ counts) {
    __shared__ uint2 warp_s[MC_SCAN_T / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint2 carry = make_uint2(0, 0);
    for (uint32_t base = 0; base < nb; base += MC_SCAN_T * MC_SCAN_PER) {
        const uint32_t at = base + threadIdx.x * MC_SCAN_PER;
        uint2 v[MC_SCAN_PER], sum = make_uint2(0, 0);
#pragma unroll
        for (int i = 0; i < MC_SCAN_PER; ++i) {
            v[i] = at + i < nb ? sums[at + i] : make_uint2(0, 0);
            sum.x += v[i].x;
            sum.y += v[i].y;
        }
        uint2 x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t yx = __shfl_up_sync(0xffffffffu, x.x, o), yy = __shfl_up_sync(0xffffffffu, x.y, o);
            if (lane >= o) {
                x.x += yx;
                x.y += yy;
            }
        }
        if (lane == 31) warp_s[warp] = x;
        __syncthreads();
        uint2 before = carry;
        for (int w = 0; w < MC_SCAN_T / 32; ++w) {
            const uint2 t = warp_s[w];
            if (w < warp) {
                before.x += t.x;
                before.y += t.y;
            }
            carry.x += t.x;
            carry.y += t.y;
        }
        before.x += x.x - sum.x;
        before.y += x.y - sum.y;
#pragma unroll
        for (int i = 0; i < MC_SCAN_PER; ++i) {
            if (at + i < nb) sums[at + i] = before;
            before.x += v[i].x;
            before.y += v[i].y;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        counts[0] = carry.x;
        counts[1] = carry.y;
    }
}

// 4: kept vertices, and the number of each point's first one
__global__ void __launch_bounds__(MC_T) k_mc_vertices(const float* __restrict__ vol, McDims d, McGeometry g, uint32_t np,
                                                      const uint8_t* __restrict__ code, const uint2* __restrict__ sums,
                                                      uint32_t* __restrict__ first, double* __restrict__ V) {
    __shared__ uint32_t warp_s[MC_T / 32];
    __shared__ uint16_t list[3 * MC_POINTS];
    const uint32_t p0 = blockIdx.x * (uint32_t)MC_POINTS, p = p0 + threadIdx.x * MC_PER;
    const uint32_t bits = p < np ? *reinterpret_cast<const uint32_t*>(code + p) & 0x07070707u : 0u, v0 = sums[blockIdx.x].x;
    uint32_t at;
    const uint32_t n = mc_block_scan(__popc(bits), warp_s, at);
    if (bits) {
        uint32_t f[MC_PER];
#pragma unroll
        for (int u = 0; u < MC_PER; ++u) f[u] = v0 + at + __popc(bits & ((1u << (8 * u)) - 1u));
        *reinterpret_cast<uint4*>(first + p) = make_uint4(f[0], f[1], f[2], f[3]);
        for (uint32_t left = bits; left; left &= left - 1) {
            const uint32_t b = __ffs(left) - 1;
            list[at++] = (uint16_t)((threadIdx.x * MC_PER + (b >> 3)) * 3 + (b & 7u));
        }
    }
    __syncthreads();
    for (uint32_t r = threadIdx.x; r < n; r += MC_T) {
        const uint32_t lp = list[r] / 3u, a = list[r] - 3u * lp, pt = p0 + lp;
        const McPoint q = mc_point(d, pt);
        const int64_t step = a == 0 ? (int64_t)d.ny * d.nz : a == 1 ? d.nz : 1;
        double x[3];
        mc_vertex(g, q, (int)a, vol[pt], vol[pt + step], x);
#pragma unroll
        for (int c = 0; c < 3; ++c) V[3 * ((int64_t)v0 + r) + c] = x[c];
    }
}

// 5: kept faces
__global__ void __launch_bounds__(MC_T) k_mc_faces(McDims d, uint32_t np, const uint8_t* __restrict__ code,
                                                   const uint8_t* __restrict__ cfg, const uint8_t* __restrict__ tri,
                                                   const uint2* __restrict__ sums, const uint32_t* __restrict__ first,
                                                   int64_t* __restrict__ F) {
    __shared__ uint32_t warp_s[MC_T / 32];
    __shared__ uint16_t list[5 * MC_POINTS];
    const uint32_t p0 = blockIdx.x * (uint32_t)MC_POINTS, p = p0 + threadIdx.x * MC_PER;
    const uint32_t kept = p < np ? *reinterpret_cast<const uint32_t*>(tri + p) : 0u;
    const int64_t o0 = sums[blockIdx.x].y;
    uint32_t at;
    const uint32_t n = mc_block_scan(__popc(kept), warp_s, at);
    for (uint32_t left = kept; left; left &= left - 1) list[at++] = (uint16_t)(threadIdx.x * 8 * MC_PER + __ffs(left) - 1);
    __syncthreads();
    for (uint32_t r = threadIdx.x; r < n; r += MC_T) {
        const uint32_t pt = p0 + (list[r] >> 3), t = list[r] & 7u;
        const McPoint q = mc_point(d, pt);
        const int8_t* tr = c_tri[cfg[pt]][t];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            int a, dx, dy, dz;
            edge_lo_corner(tr[c], a, dx, dy, dz);
            const int64_t m = vol_index(d, q.i + dx, q.j + dy, q.k + dz);
            F[3 * (o0 + r) + c] = (int64_t)first[m] + __popc(code[m] & ((1u << a) - 1u));
        }
    }
}

struct McWorkspace {
    uint8_t* code;     // [points] kept edges, cube with triangles
    uint8_t* cfg;      // [points] corner signs of a cube with triangles
    uint8_t* tri;      // [points] kept triangles of the cube
    uint32_t* first;   // [points] number of the point's first kept vertex
    uint2* sums;       // [blocks] kept vertices and faces, then those of earlier blocks
};

static size_t align256(size_t b) { return (b + 255) / 256 * 256; }

static size_t mc_layout(int nx, int ny, int nz, uint8_t* base, McWorkspace* w) {
    const size_t np = (size_t)nx * ny * nz, nb = (np + MC_POINTS - 1) / MC_POINTS;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        uint8_t* p = base ? base + off : nullptr;
        off += align256(bytes);
        return p;
    };
    McWorkspace t;
    t.code = take(np);
    t.cfg = take(np);
    t.tri = take(np);
    t.first = (uint32_t*)take(4 * np);
    t.sums = (uint2*)take(8 * nb);
    if (w) *w = t;
    return off;
}

// worst-case output sizes of one block: one vertex per grid edge, five triangles per cube
static int64_t mc_vcap(int nx, int ny, int nz) { return (int64_t)nx * ny * nz * 3; }
static int64_t mc_fcap(int nx, int ny, int nz) { return 5 * (int64_t)(nx - 1) * (ny - 1) * (nz - 1); }

// One pass over the volume classifies every point, two passes over one byte per point emit.
// Counting per edge and per cube into int64 arrays, scanning those and the worst-case vertex and
// face lists (30 launches) took 621 us for a 129^3 block, the scans alone 321; this takes 41.
static int mc_run(const float* vol, int nx, int ny, int nz, double iso, const double* origin, double intv,
                  const McWorkspace& w, double* V, int64_t* F, int64_t* counts, cudaStream_t s) {
    const McDims d{nx, ny, nz};
    const McGeometry g{iso, intv, {origin[0], origin[1], origin[2]}};
    // at most 2^28 points (checked by the entry points): vertices and faces below 2^32
    const uint32_t np = (uint32_t)((int64_t)nx * ny * nz), nb = (np + MC_POINTS - 1) / MC_POINTS;
    k_mc_classify<<<nb, MC_T, 0, s>>>(vol, d, g, np, w.code, w.cfg, w.sums);
    k_mc_count_faces<<<nb, MC_T, 0, s>>>(d, np, w.code, w.cfg, w.tri, w.sums);
    k_mc_scan_blocks<<<1, MC_SCAN_T, 0, s>>>(w.sums, nb, counts);
    k_mc_vertices<<<nb, MC_T, 0, s>>>(vol, d, g, np, w.code, w.sums, w.first, V);
    k_mc_faces<<<nb, MC_T, 0, s>>>(d, np, w.code, w.cfg, w.tri, w.sums, w.first, F);
    return launch_status("marching_cubes");
}

}  // namespace gbsdf

using namespace gbsdf;

extern "C" int gbsdf_mc_table(int32_t* tri, int32_t* count) {
    clear_error();
    GBSDF_CHECK_ARG(tri && count, "NULL pointer");
    const McTable& t = mc_table();
    for (int c = 0; c < 256; ++c) {
        count[c] = t.count[c];
        for (int k = 0; k < 16; ++k)
            for (int q = 0; q < 3; ++q) tri[(c * 16 + k) * 3 + q] = t.tri[c][k][q];
    }
    return GBSDF_OK;
}

extern "C" size_t gbsdf_mc_workspace_size(int nx, int ny, int nz) {
    if (nx < 2 || ny < 2 || nz < 2) return 0;
    return mc_layout(nx, ny, nz, nullptr, nullptr);
}

extern "C" int gbsdf_mc_block(const float* vol, int nx, int ny, int nz, double iso, const double* origin, double intv,
                              void* workspace, size_t ws_bytes, double* V, int64_t V_cap, int64_t* F, int64_t F_cap,
                              int64_t* counts, void* stream) {
    clear_error();
    GBSDF_CHECK_ARG(vol && origin && V && F && counts, "NULL pointer");
    GBSDF_CHECK_ARG(nx >= 2 && ny >= 2 && nz >= 2, "block must have at least 2 points per axis");
    GBSDF_CHECK_ARG((int64_t)nx * ny * nz <= (int64_t)1 << 28, "block too large");
    GBSDF_CHECK_ARG(V_cap >= mc_vcap(nx, ny, nz) && F_cap >= mc_fcap(nx, ny, nz),
                    "output capacity below the worst case (3 nx ny nz vertices, 5 (nx-1)(ny-1)(nz-1) faces)");
    const size_t need = gbsdf_mc_workspace_size(nx, ny, nz);
    GBSDF_CHECK_ARG(workspace && ws_bytes >= need, "workspace of %zu bytes needed", need);
    GBSDF_CHECK_ARG(aligned(workspace, 256), "workspace must be 256-byte aligned");
    if (int st = upload_table_once()) return st;
    McWorkspace w;
    mc_layout(nx, ny, nz, (uint8_t*)workspace, &w);
    return mc_run(vol, nx, ny, nz, iso, origin, intv, w, V, F, counts, as_stream(stream));
}

// ---------------------------------------------------------------------------
// Marching cubes without any device allocation.
//
// Some callers cannot allocate device memory: a host application that owns the
// whole device budget and forbids allocations after start-up (a renderer or an
// engine plugin with a fixed pool), or a caller in a latency-critical loop where
// cudaMalloc / cudaFree could synchronise the device.  For them this variant
// keeps its scratch in a file-scope __device__ array of fixed size, enough for
// blocks of up to 33 x 33 x 33 lattice points (32^3 cubes).  The array exists on
// every device that loads this library, for the life of the process
// (247 KiB).  Host code may not take the array's name as a device address, so
// the device address is looked up with cudaGetSymbolAddress once per device, on
// the first call made with that device current; make that first call before any
// stream capture.  Every call reuses the same array: two calls whose kernels
// overlap on the GPU (different streams, or several host threads) race, so
// serialise them.  Every scratch element is written before it is read in a
// call, so nothing carries over from the previous call.

constexpr int kNoAllocMaxPoints = 33;
constexpr size_t kNoAllocScratchBytes = 252928;   // gbsdf_mc_workspace_size(33, 33, 33)

static __device__ __align__(256) uint8_t g_mc_scratch[kNoAllocScratchBytes];

static int noalloc_scratch(void** out) {
    static void* addr[64] = {nullptr};
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        set_error("no current CUDA device");
        return GBSDF_ERR_CUDA;
    }
    std::lock_guard<std::mutex> lk(mu);
    if (!addr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_mc_scratch);
        if (e != cudaSuccess || p == nullptr) {
            set_error("cudaGetSymbolAddress of the marching-cubes scratch failed: %s", cudaGetErrorString(e));
            return GBSDF_ERR_CUDA;
        }
        addr[dev] = p;
    }
    *out = addr[dev];
    return GBSDF_OK;
}

extern "C" int gbsdf_mc_block_noalloc(const float* vol, int nx, int ny, int nz, double iso, const double* origin,
                                      double intv, double* V, int64_t V_cap, int64_t* F, int64_t F_cap,
                                      int64_t* counts, void* stream) {
    clear_error();
    GBSDF_CHECK_ARG(vol && origin && V && F && counts, "NULL pointer");
    GBSDF_CHECK_ARG(nx >= 2 && ny >= 2 && nz >= 2, "block must have at least 2 points per axis");
    GBSDF_CHECK_ARG(nx <= kNoAllocMaxPoints && ny <= kNoAllocMaxPoints && nz <= kNoAllocMaxPoints,
                    "block %d x %d x %d exceeds the allocation-free limit of %d points per axis "
                    "(use gbsdf_mc_block with a caller workspace for larger blocks)",
                    nx, ny, nz, kNoAllocMaxPoints);
    GBSDF_CHECK_ARG(V_cap >= mc_vcap(nx, ny, nz) && F_cap >= mc_fcap(nx, ny, nz),
                    "output capacity below the worst case (3 nx ny nz vertices, 5 (nx-1)(ny-1)(nz-1) faces)");
    if (gbsdf_mc_workspace_size(nx, ny, nz) > kNoAllocScratchBytes) {
        set_error("internal: scratch layout larger than the static array");
        return GBSDF_ERR_UNSUPPORTED;
    }
    if (int st = upload_table_once()) return st;
    void* scratch = nullptr;
    if (int st = noalloc_scratch(&scratch)) return st;
    McWorkspace w;
    mc_layout(nx, ny, nz, (uint8_t*)scratch, &w);
    return mc_run(vol, nx, ny, nz, iso, origin, intv, w, V, F, counts, as_stream(stream));
}
