// Fused neural-SDF field kernels (hash grid + SDF layer 0 + head + numerical
// gradient taps) on tcgen05, forward and backward.
//
// Reference path: NeuralSDF.forward / sdf / compute_gradients (6 taps)
// (projects/neuralangelo/utils/modules.py:68-95, 131-156), MLPforNeuralSDF
// layer 0 + SDF head (utils/mlp.py:55-69), the outside overwrite
// (projects/neuralangelo/model.py:163) and the input of NeuralRGB
// (modules.py:209-220: x, SH(view dir), normalize(gradient), feature, appearance).
//
// Tile = 18 samples x 7 evaluations (centre + 6 taps) = 126 rows (+2 dead rows)
// of a 128-row tcgen05 tile.  Row r holds evaluation e = r / 18 of sample r % 18:
// e = 0 centre, 1 +x, 2 -x, 3 +y, 4 -y, 5 +z, 6 -z.  With 4 taps (the tetrahedral
// stencil, modules.py:157-175) a tile is 25 samples x 5 evaluations = 125 rows.  The hash-grid features of
// the active levels are gathered into rows of global memory (x0ext: fp16 hi,
// position/bias tail, fp16 lo) by a kernel of its own and loaded from there by TMA;
// layer 0's weights are resident; softplus and the SDF head run in fp32 in the
// epilogue, so SDF values and the tap differences keep fp32 accuracy.
#include "dense.cuh"
#include "tma.cuh"

namespace gbsdf {

// Evaluations of one sample (the centre, then the taps) and samples per 128-row tile:
// 6 taps (modules.py:132-156): 18 samples x 7 = 126 rows; 4 taps (modules.py:157-175):
// 25 samples x 5 = 125 rows.
template <int TAPS>
struct TapTile {
    static_assert(TAPS == 6 || TAPS == 4, "4 or 6 taps");
    static constexpr int EVALS = TAPS + 1;
    static constexpr int SPT = TAPS == 6 ? 18 : 25;
    static constexpr int ROWS = SPT * EVALS;
    // the backward's double-buffered d f per evaluation row (+4 floats of slack), rounded up to
    // 4 floats so the d_h0c rows after it stay 16-byte aligned (cp.async and float4 accesses)
    static constexpr int DF_FLOATS = (2 * ROWS + 4 + 3) / 4 * 4;
};
constexpr int FWD_SDF_FLOATS = 128;   // forward's per-evaluation SDF values (<= 126) + padding
constexpr int FIELD_THREADS = 256;
constexpr int HID = 256;         // SDF hidden width (base.yaml:41)

typedef gbsdf_field_args FieldParams;   // layout and field meanings: include/gbsdf.h

// ray of sample s (32-bit division: the launchers keep the sample count below 2^32)
__device__ __forceinline__ int ray_of(const FieldParams& p, int64_t s) {
    return p.S > 0 ? (int)((uint32_t)s / (uint32_t)p.S) : p.sample_ray[s];
}

// float32 centre point c + d t (camera.py:314-320: one multiply, one add)
__device__ __forceinline__ void sample_point_of_ray(const FieldParams& p, int64_t s, int r, float* x) {
    const float t = p.dists[s];
#pragma unroll
    for (int i = 0; i < 3; ++i) x[i] = __fadd_rn(p.center[3 * r + i], __fmul_rn(p.ray_unit[3 * r + i], t));
}
__device__ __forceinline__ void sample_point(const FieldParams& p, int64_t s, float* x) {
    sample_point_of_ray(p, s, ray_of(p, s), x);
}

// evaluation position: the reference adds a float32 tap vector to the point.
// 6 taps: e = 1..6 -> +x, -x, +y, -y, +z, -z by eps (modules.py:135-143).
// 4 taps: e = 1..4 -> k1 (1,-1,-1), k2 (-1,-1,1), k3 (-1,1,-1), k4 (1,1,1) times the
// displacement eps / sqrt(3), which the caller passes as `eps` (modules.py:158-166).
template <int TAPS>
__device__ __forceinline__ void eval_point(const float* c, int e, float eps, float* x) {
    x[0] = c[0]; x[1] = c[1]; x[2] = c[2];
    if (e == 0) return;
    if constexpr (TAPS == 6) {
        const int d = (e - 1) >> 1;
        x[d] = (e & 1) ? __fadd_rn(x[d], eps) : __fsub_rn(x[d], eps);
    } else {
        const bool px = e == 1 || e == 4, py = e == 3 || e == 4, pz = e == 2 || e == 4;
        x[0] = px ? __fadd_rn(x[0], eps) : __fsub_rn(x[0], eps);
        x[1] = py ? __fadd_rn(x[1], eps) : __fsub_rn(x[1], eps);
        x[2] = pz ? __fadd_rn(x[2], eps) : __fsub_rn(x[2], eps);
    }
}

template <int F>
__device__ __forceinline__ void write_half_row(uint8_t* dst, const float* v) {
    if constexpr (F == 8) {
        store_half8(reinterpret_cast<__half*>(dst), v);
    } else if constexpr (F == 4) {
        __half2 h[2] = {__floats2half2_rn(v[0], v[1]), __floats2half2_rn(v[2], v[3])};
        *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(h);
    } else {
#pragma unroll
        for (int f = 0; f < F; ++f) reinterpret_cast<__half*>(dst)[f] = __float2half_rn(v[f]);
    }
}

// The features go in as an fp16 pair (hi + lo, ~2^-22 relative): the +eps and
// -eps taps of a sample differ by tiny amounts, and independent fp16 rounding
// of their features would dominate the pre-activation differences that the
// table gradient is made of.
template <int F>
__device__ __forceinline__ void write_tile_features(uint8_t* a_s, uint8_t* a2_s, int row, int l, int K0,
                                                    const float* v) {
    const uint32_t off = umma::kmajor_offset(row, l * F, K0);
    float lo[F];
#pragma unroll
    for (int f = 0; f < F; ++f) lo[f] = v[f] - __half2float(__float2half_rn(v[f]));
    write_half_row<F>(a_s + off, v);
    write_half_row<F>(a2_s + off, lo);
}

// Deterministic mode: each contribution as a 64-bit fixed-point integer with DET_FRAC_BITS
// fraction bits, added with integer atomics.  Integer addition is associative, so the sums
// do not depend on the order the atomics land in: two runs give bit-identical results.
constexpr int DET_FRAC_BITS = 48;
template <int F>
__device__ __forceinline__ void scatter_add_fixed(unsigned long long* dst, const float* v) {
#pragma unroll
    for (int f = 0; f < F; ++f)
        if (v[f] != 0.0f) atomicAdd(dst + f, (unsigned long long)__float2ll_rn(v[f] * 0x1p48f));
}

__global__ void k_fixed_to_table(int64_t n, const unsigned long long* __restrict__ fix, float* __restrict__ d_table) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long q = (long long)fix[i];
    if (q != 0) d_table[i] += (float)((double)q * 0x1p-48);
}

template <int F>
__device__ __forceinline__ void scatter_add(float* dst, const float* v) {
    if constexpr (F == 4) {
        atomicAdd(reinterpret_cast<float4*>(dst), make_float4(v[0], v[1], v[2], v[3]));
    } else {
#pragma unroll
        for (int f = 0; f < F; ++f) atomicAdd(dst + f, v[f]);
    }
}

// ---------------------------------------------------------------------------
// hash-grid gather and table-gradient scatter as their own kernels: one thread
// per (sample, level) keeps thousands of independent loads and atomics in flight,
// which the tensor-core kernels (one CTA of eight warps per SM) cannot.

// one table row of F fp16 features
template <int F>
struct TableRow {
    uint32_t u[F / 2];
    __device__ __forceinline__ void load(const __half* row) {
        if constexpr (F == 8) {
            const uint4 q = __ldg(reinterpret_cast<const uint4*>(row));
            u[0] = q.x; u[1] = q.y; u[2] = q.z; u[3] = q.w;
        } else if constexpr (F == 4) {
            const uint2 q = __ldg(reinterpret_cast<const uint2*>(row));
            u[0] = q.x; u[1] = q.y;
        } else {
            u[0] = __ldg(reinterpret_cast<const uint32_t*>(row));
        }
    }
    // v += w * row, each feature one fmaf
    __device__ __forceinline__ void fma(float w, uint64_t* v) const {
        const uint64_t ww = pack_f32x2(w, w);
#pragma unroll
        for (int i = 0; i < F / 2; ++i) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u[i]));
            v[i] = fma_f32x2(ww, pack_f32x2(f.x, f.y), v[i]);
        }
    }
};

// The level table in shared memory: lanes of a warp sit on different levels, and a
// lane-dependent index into the kernel parameters is serialised per level.
__device__ __forceinline__ void stage_levels(const gbsdf_grid& g, LevelDesc* lv_s, int active) {
    for (int l = threadIdx.x; l < active; l += blockDim.x) lv_s[l] = level_desc(g, l);
}

// grid cell and fraction of a point on one level
struct GridCell {
    uint32_t b[3];
    float f[3];
};
__device__ __forceinline__ GridCell grid_cell(float scale, const float* x) {
    GridCell g;
#pragma unroll
    for (int k = 0; k < 3; ++k) grid_pos(scale, to_unit(x[k]), g.b[k], g.f[k]);
    return g;
}

// The (lane, evaluation) pairs of a warp named in each lane's `mask` (bit e), packed into
// list (lane << 3 | e); returns their number.  EVALS <= 8.
template <int EVALS>
__device__ __forceinline__ int warp_pack_evals(uint32_t mask, uint8_t* list, int lane) {
    const int n = __popc(mask);
    int at = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += v;
    }
    const int total = __shfl_sync(0xffffffffu, at, 31);
    at -= n;
#pragma unroll
    for (int e = 1; e < EVALS; ++e)
        if (mask & (1u << e)) list[at++] = (uint8_t)(lane << 3 | e);
    __syncwarp();
    return total;
}

// x0ext row t*126 + r (r = e*18 + sl) of every tile: the features of level l in
// columns [l F, l F + F) as fp16 hi and, at K0 + 16 + l F, the fp16 residual lo; then the
// 16-column tail after the hi features and the zeroed padding columns.  Rows of samples
// past the end are zeros.
//
// One thread per (sample, level), levels fastest, so that a warp's stores of one evaluation
// cover whole rows.  The taps lie a fraction of a cell from the centre (a quarter at the
// finest active level, less below it), so most evaluations interpolate the centre's own
// eight corners: they are loaded once, kept in registers as fp16, and every evaluation
// in the centre's cell costs arithmetic only.  The evaluations in another cell (about one in
// nine) are packed across the warp and taken one per lane, so they cost one or two dense
// passes instead of a divergent one per tap.  Values and order of the products are those of
// an evaluation that loads its own corners.
// One thread per (evaluation, level), each loading its own eight corners, was bound by L1
// (73 %): 2.60 ms for 2.1 M samples x 8 levels, 20.7 ms for 6.3 M samples x 16 levels; this
// takes 1.34 and 8.1 ms (the rows it writes: 0.63 and 3.5 ms at the copy rate).  Latency
// bounds it: the corners kept as float32 (120 registers, two blocks per SM) took 2.07 ms, the
// tap loop unrolled 1.37 ms at two blocks and 1.73 at three, five blocks (spills) 1.75 ms.
constexpr int GATHER_THREADS = 256;
template <int F, int TAPS>
__global__ void __launch_bounds__(GATHER_THREADS, 4) k_field_gather(FieldParams p, int64_t ntiles) {
    constexpr int EVALS = TapTile<TAPS>::EVALS, SPT = TapTile<TAPS>::SPT;
    __shared__ LevelDesc lv_s[GBSDF_MAX_LEVELS];
    __shared__ uint8_t list_s[GATHER_THREADS / 32][32 * TAPS];
    const int A = p.active, K0 = p.K0, KX = 2 * K0 + 16;
    stage_levels(p.grid, lv_s, A);
    __syncthreads();
    // 32-bit index arithmetic: the launcher checks rows * A < 2^32
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t slots = (uint32_t)(ntiles * SPT);      // sample slots, tile-major
    const bool in = i < slots * (uint32_t)A;              // (whole warps go on: they pack their crossings together)
    const uint32_t se = in ? i / (uint32_t)A : 0u;
    const int l = in ? (int)(i - se * (uint32_t)A) : 0;
    const uint32_t t = se / SPT;
    const uint32_t row0 = t * (SPT * EVALS) + (se - t * SPT);   // evaluation e's row: row0 + e * SPT
    const bool live = in && (int64_t)se < p.Ns;
    const int lane = threadIdx.x & 31;
    __half* const x0 = (__half*)p.x0ext;
    const __half* const table = (const __half*)p.table;

    auto emit = [&](uint32_t row, int lev, const uint64_t* v) {
        __half* dst = x0 + (int64_t)row * KX + lev * F;          // 64-bit: rows * KX can exceed 2^32
        float hi[F], lo[F];
#pragma unroll
        for (int k = 0; k < F / 2; ++k) unpack_f32x2(v[k], hi[2 * k], hi[2 * k + 1]);
#pragma unroll
        for (int f = 0; f < F; ++f) lo[f] = hi[f] - __half2float(__float2half_rn(hi[f]));
        write_half_row<F>(reinterpret_cast<uint8_t*>(dst), hi);
        write_half_row<F>(reinterpret_cast<uint8_t*>(dst + K0 + 16), lo);
    };

    float c[3] = {0.f, 0.f, 0.f};
    uint32_t mask = 0;                                    // evaluations outside the centre's cell
    if (live) {
        sample_point(p, se, c);
        const LevelDesc d = lv_s[l];
        const GridCell g0 = grid_cell(d.scale, c);
        TableRow<F> home[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            home[k].load(table + (d.offset + grid_index(d, g0.b[0] + (k & 1), g0.b[1] + ((k >> 1) & 1),
                                                             g0.b[2] + ((k >> 2) & 1))) * F);
#pragma unroll 1
        for (int e = 0; e < EVALS; ++e) {
            float x[3];
            eval_point<TAPS>(c, e, p.eps, x);
            const GridCell g = grid_cell(d.scale, x);
            if (g.b[0] == g0.b[0] && g.b[1] == g0.b[1] && g.b[2] == g0.b[2]) {
                uint64_t v[F / 2];
#pragma unroll
                for (int k = 0; k < F / 2; ++k) v[k] = 0ull;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float w = corner_weight(k, g.f[0], g.f[1], g.f[2]);
                    home[k].fma(w, v);
                }
                emit(row0 + e * SPT, l, v);
            } else {
                mask |= 1u << e;
            }
        }
    } else if (in) {
        const uint64_t v[F / 2] = {};
        for (int e = 0; e < EVALS; ++e) emit(row0 + e * SPT, l, v);
    }
    // tail (multiplied by w0b's position and bias columns in the forward MMA): x hi, 1, x lo, 1,
    // x hi, zeros -- w0x x + b0 as fp16 hi/lo products; lane l of a sample takes evaluations l, l + A, ..
    for (int e = l; in && e < EVALS; e += A) {
        __half* dst = x0 + (int64_t)(row0 + e * SPT) * KX;
        float tail[16] = {0.f};
        if (live) {
            float x[3];
            eval_point<TAPS>(c, e, p.eps, x);
            tail[0] = x[0]; tail[1] = x[1]; tail[2] = x[2]; tail[3] = 1.0f;
#pragma unroll
            for (int k = 0; k < 3; ++k) tail[4 + k] = x[k] - __half2float(__float2half_rn(x[k]));
            tail[7] = 1.0f;
            tail[8] = x[0]; tail[9] = x[1]; tail[10] = x[2];
        }
        store_half8(dst + K0, tail);
        store_half8(dst + K0 + 8, tail + 8);
        for (int c0 = A * F; c0 < K0; ++c0) {
            dst[c0] = __float2half_rn(0.0f);
            dst[K0 + 16 + c0] = __float2half_rn(0.0f);
        }
    }
    uint8_t* list = list_s[threadIdx.x >> 5];
    const int total = warp_pack_evals<EVALS>(mask, list, lane);
    for (int k0 = 0; k0 < total; k0 += 32) {
        const bool on = k0 + lane < total;
        const int ent = on ? list[k0 + lane] : 0, own = ent >> 3, e = ent & 7;
        const float oc[3] = {__shfl_sync(0xffffffffu, c[0], own), __shfl_sync(0xffffffffu, c[1], own),
                             __shfl_sync(0xffffffffu, c[2], own)};
        const int ol = __shfl_sync(0xffffffffu, l, own);
        const uint32_t orow = __shfl_sync(0xffffffffu, row0, own);
        if (!on) continue;
        float x[3];
        eval_point<TAPS>(oc, e, p.eps, x);
        const LevelDesc d = lv_s[ol];
        const GridCell g = grid_cell(d.scale, x);
        uint64_t v[F / 2];
        TableRow<F> r[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            r[k].load(table + (d.offset + grid_index(d, g.b[0] + (k & 1), g.b[1] + ((k >> 1) & 1),
                                                             g.b[2] + ((k >> 2) & 1))) * F);
#pragma unroll
        for (int f = 0; f < F / 2; ++f) v[f] = 0ull;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float w = corner_weight(k, g.f[0], g.f[1], g.f[2]);
            r[k].fma(w, v);
        }
        emit(orow + e * SPT, ol, v);
    }
}

// Table gradient of one level over NS consecutive samples and their evaluations.  The thread owns
// the eight corners of the centre's cell: an evaluation in that cell adds to all eight, one in a
// neighbouring cell to the corners the two cells share (its weight at a shared corner is a
// product of one factor per axis, zero for the corners it does not reach).  While the next sample's
// centre stays in the cell, as it mostly does at coarse levels, the sums go on in registers; then
// each owned corner leaves as one vector atomic.  The corners of neighbouring cells that the
// centre's cell does not have (typically four per evaluation, of about one evaluation in nine) go
// out directly, the evaluations packed across the warp so that they cost a few dense passes.
// Eight features are two lanes' work, four each: the accumulators fit the registers in one pass,
// and the pair's atomics cover whole 32-byte rows.
// 2.1 M samples x 8 levels: 3.05 ms merging consecutive evaluations of equal cells, 2.28 ms with the
// corners owned over one sample (four per pass, all features in one lane, neighbouring samples
// merged by shuffles), 2.09 ms so; 0.24 M samples x 16 levels: 0.99, 0.72 and 0.50 ms (there the half
// sectors of 16-byte atomics counted).  Evaluations not unrolled 2.38 ms, two blocks per SM 2.55.
constexpr int SCATTER_THREADS = 256;

// d_enc of one evaluation and level
template <int F>
__device__ __forceinline__ void load_d_enc(const float* dv, float* g) {
    if constexpr (F % 4 == 0) {
#pragma unroll
        for (int f = 0; f < F; f += 4) {
            const float4 q4 = __ldg(reinterpret_cast<const float4*>(dv + f));
            g[f] = q4.x; g[f + 1] = q4.y; g[f + 2] = q4.z; g[f + 3] = q4.w;
        }
    } else {
#pragma unroll
        for (int f = 0; f < F; ++f) g[f] = __ldg(dv + f);
    }
}
template <int F>
__device__ __forceinline__ bool any_nonfinite(const float* g) {
    bool bad = false;
#pragma unroll
    for (int f = 0; f < F; ++f) bad |= !isfinite(g[f]);
    return bad;
}

template <int F, int TAPS, bool DET, int NS>
__global__ void __launch_bounds__(SCATTER_THREADS, 3) k_field_scatter(FieldParams p) {
    constexpr int EVALS = TapTile<TAPS>::EVALS, SPT = TapTile<TAPS>::SPT;
    constexpr int FS = F < 4 ? F : 4, PARTS = F / FS;     // features per lane, lanes per (samples, level)
    __shared__ LevelDesc lv_s[GBSDF_MAX_LEVELS];
    __shared__ uint16_t list_s[SCATTER_THREADS / 32][32 / PARTS * NS * TAPS];
    const int A = p.active, K0 = p.K0;
    stage_levels(p.grid, lv_s, A);
    __syncthreads();
    // 32-bit index arithmetic: the launcher checks Ns * active * 8 < 2^32
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const int part = (int)(i % PARTS), lane = threadIdx.x & 31;
    const uint32_t item = i / PARTS, group = item / (uint32_t)A;
    const int l = (int)(item - group * (uint32_t)A);
    const uint32_t s0 = group * NS;
    const uint32_t n = s0 < (uint32_t)p.Ns ? min((uint32_t)p.Ns - s0, (uint32_t)NS) : 0u;   // (whole warps go on)
    const float gscale = p.d_table_scale_dev ? *p.d_table_scale_dev : (p.d_table_scale != 0.0f ? p.d_table_scale : 1.0f);
    auto add = [&](uint64_t entry, const float* v) {
        if constexpr (DET) scatter_add_fixed<FS>(p.d_table_fix + entry * F + part * FS, v);
        else scatter_add<FS>(p.d_table + entry * F + part * FS, v);
    };
    // (first row of sample s; evaluation e's is e * SPT rows on)
    auto row_of = [](uint32_t s) {
        const uint32_t t = s / SPT;
        return t * (SPT * EVALS) + (s - t * SPT);
    };
    bool nonfinite = false;
    uint32_t mask[NS];                                    // per sample: evaluations outside the centre's cell
    const LevelDesc d = lv_s[n > 0 ? l : 0];
    uint32_t home[3] = {0, 0, 0};
    float acc[8][FS];
    auto flush = [&]() {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            add(d.offset + grid_index(d, home[0] + (c & 1), home[1] + ((c >> 1) & 1), home[2] + ((c >> 2) & 1)), acc[c]);
#pragma unroll
            for (int f = 0; f < FS; ++f) acc[c][f] = 0.0f;
        }
    };
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int f = 0; f < FS; ++f) acc[c][f] = 0.0f;
#pragma unroll 1
    for (uint32_t k = 0; k < n; ++k) {
        float c[3];
        sample_point(p, s0 + k, c);
        const GridCell g0 = grid_cell(d.scale, c);
        if (k > 0 && (g0.b[0] != home[0] || g0.b[1] != home[1] || g0.b[2] != home[2])) flush();
#pragma unroll
        for (int x = 0; x < 3; ++x) home[x] = g0.b[x];
        const float* dv = p.d_enc + (int64_t)row_of(s0 + k) * K0 + l * F + part * FS;
        uint32_t m = 0;
#pragma unroll
        for (int e = 0; e < EVALS; ++e) {
            float x[3], g[FS];
            load_d_enc<FS>(dv + (int64_t)e * SPT * K0, g);
            eval_point<TAPS>(c, e, p.eps, x);
            const GridCell gc = grid_cell(d.scale, x);
            // per axis: the weight of the owned corners at 0 and 1
            float w0[3], w1[3];
            bool other = false;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const int db = (int)(gc.b[a] - home[a]);
                const float one_f = __fsub_rn(1.0f, gc.f[a]);
                w0[a] = db == 0 ? one_f : (db == -1 ? gc.f[a] : 0.0f);
                w1[a] = db == 0 ? gc.f[a] : (db == 1 ? one_f : 0.0f);
                other |= db != 0;
            }
            const bool bad = any_nonfinite<FS>(g);
            nonfinite |= bad;
            if (other) m |= 1u << e;
            // (a non-finite gradient of another cell would reach every owned corner as 0 * inf:
            // that evaluation goes out corner by corner below)
            if (other && bad) continue;
#pragma unroll
            for (int f = 0; f < FS; ++f) g[f] *= gscale;
#pragma unroll
            for (int corner = 0; corner < 8; ++corner) {
                const float wx = (corner & 1) ? w1[0] : w0[0], wy = (corner & 2) ? w1[1] : w0[1];
                const float wz = (corner & 4) ? w1[2] : w0[2];
                const float w = __fmul_rn(__fmul_rn(wx, wy), wz);
#pragma unroll
                for (int f = 0; f < FS; ++f) acc[corner][f] = fmaf(w, g[f], acc[corner][f]);
            }
        }
#pragma unroll
        for (int j = 0; j < NS; ++j)
            if ((uint32_t)j == k) mask[j] = m;
    }
    if (n > 0) flush();
    if (nonfinite && p.found_inf) *p.found_inf = 1.0f;     // any writer stores the same value
    // the corners that the centre's cell does not have: (lane, sample, evaluation) entries of the first lane of
    // each pair, taken by the pairs in turn
    uint16_t* list = list_s[threadIdx.x >> 5];
    int mine = 0;
#pragma unroll
    for (int j = 0; j < NS; ++j) {
        if ((uint32_t)j >= n || part > 0) mask[j] = 0;
        mine += __popc(mask[j]);
    }
    int at = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += v;
    }
    const int total = __shfl_sync(0xffffffffu, at, 31);
    at -= mine;
#pragma unroll
    for (int j = 0; j < NS; ++j)
        for (uint32_t left = mask[j]; left; left &= left - 1)
            list[at++] = (uint16_t)(lane << 8 | j << 4 | (__ffs(left) - 1));
    __syncwarp();
    for (int k0 = 0; k0 < total; k0 += 32 / PARTS) {
        const int k = k0 + lane / PARTS;
        const bool on = k < total;
        const uint32_t ent = on ? list[k] : 0u;
        const int own = (int)(ent >> 8), e = (int)(ent & 15u);
        const uint32_t s = __shfl_sync(0xffffffffu, s0, own) + ((ent >> 4) & 15u);
        const int ol = __shfl_sync(0xffffffffu, l, own);
        if (!on) continue;
        float c[3], x[3], g[FS];
        sample_point(p, s, c);
        load_d_enc<FS>(p.d_enc + (int64_t)(row_of(s) + e * SPT) * K0 + ol * F + part * FS, g);
        eval_point<TAPS>(c, e, p.eps, x);
        const LevelDesc od = lv_s[ol];
        const GridCell centre = grid_cell(od.scale, c), gc = grid_cell(od.scale, x);
        const bool bad = any_nonfinite<FS>(g);
        uint32_t db[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) db[a] = gc.b[a] - centre.b[a];
#pragma unroll
        for (int corner = 0; corner < 8; ++corner) {
            const uint32_t bx = corner & 1, by = (corner >> 1) & 1, bz = (corner >> 2) & 1;
            // owned: the corner's coordinate relative to the centre's cell is 0 or 1 on every axis
            if (!bad && db[0] + bx <= 1u && db[1] + by <= 1u && db[2] + bz <= 1u) continue;
            const float w = corner_weight(corner, gc.f[0], gc.f[1], gc.f[2]) * gscale;
            float v[FS];
#pragma unroll
            for (int f = 0; f < FS; ++f) v[f] = w * g[f];
            add(od.offset + grid_index(od, gc.b[0] + bx, gc.b[1] + by, gc.b[2] + bz), v);
        }
    }
}

// ---------------------------------------------------------------------------
// forward

// Two CTAs per SM: one CTA's epilogue overlaps the other's staging, MMAs and
// per-sample phase.  The pre-activation comes out of the MMA complete: the A
// tile is x0ext's [features hi | tail] columns and B = w0b = [W0e | position and
// bias columns], so the epilogue reads W0x x + b0 + W0e f from TMEM and adds
// nothing; the fp16 residual of the features is a second MMA over the W0e prefix.
constexpr int FWD_CTAS_PER_SM = 2;
// One sample's per-ray inputs of the forward's per-sample phase, prefetched into a ring of
// four tiles in shared memory (see k_field_fwd)
struct FwdSample {
    int r;                       // ray; -1 past the last sample
    int out;                     // the ray's `outside` flag
    int appi;                    // appearance-code row
    float c[3];                  // sample point c + d t
    float dv[3];                 // ray direction
};
constexpr int FWD_RING = 4;
constexpr int FWD_APP_RING = 2;  // appearance codes: this tile's and the next one's

// shared memory of one group: feature tiles, partial sums, SDF values, barriers, prefetch rings
// (1024-byte multiples, as the swizzled feature tiles need)
//
// The feature tiles: 64-column boxes of 128 rows in the 128-byte swizzle, ceil(K0 / 64) of the
// hi columns (from column 0) and of the lo columns (from K0 + 16), and the 16 tail columns as two
// 16-byte chunks of 128 rows without a swizzle.  A box row is a 128-byte line; the core-matrix
// layout, loaded as 16-byte rows, moved 8 times as many of them and bounded the kernel: 12.7 ms
// for 6.3 M samples at K0 = 128 against 9.8, 2.80 ms for 2.1 M at K0 = 64 against 2.38.
constexpr int FWD_BOX_BYTES = TILE_M * 128;
__host__ __device__ constexpr int fwd_tile_bytes(int K0) { return 2 * ((K0 + 63) / 64) * FWD_BOX_BYTES + TILE_M * 32; }
// (appearance rows an odd number of floats apart: one bank each)
__host__ __device__ constexpr int fwd_app_ld(int app_dim) { return app_dim > 0 ? app_dim | 1 : 0; }
template <int TAPS>
__host__ __device__ constexpr int fwd_group_bytes(int K0, int app_dim) {
    return (fwd_tile_bytes(K0) + (2 * TILE_M + FWD_SDF_FLOATS) * 4 + 24 +
            FWD_RING * TapTile<TAPS>::SPT * (int)sizeof(FwdSample) +
            FWD_APP_RING * TapTile<TAPS>::SPT * fwd_app_ld(app_dim) * 4 + 1023) / 1024 * 1024;
}

// GROUPS: independent groups of eight warps in a CTA, each on tiles of its own with its own
// feature buffers, accumulator and barriers, sharing the resident weights.  Where the shared
// memory holds two CTAs per SM (K0 <= 80) one group per CTA is the same thing; above that one
// CTA of two groups keeps two tiles in flight per SM where one CTA of one group left every
// phase exposed.  K0 = 128 (16 levels x 8 features): 6.3 M samples 15.4 ms with one group, 12.7
// with two; 0.24 M samples 0.50 and 0.40 ms (both before the swizzled feature tiles).
template <int F, int TAPS, int GROUPS>
__global__ void __launch_bounds__(FIELD_THREADS * GROUPS, GROUPS == 1 ? FWD_CTAS_PER_SM : 1)
    k_field_fwd(FieldParams p, const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_tail) {
    constexpr int EVALS = TapTile<TAPS>::EVALS, SPT = TapTile<TAPS>::SPT;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int K0 = p.K0;
    const int KB = K0 + 16;                                     // features hi + tail
    const int nbox = (K0 + 63) / 64;                            // 64-column boxes of the hi (and of the lo) features
    const int grp = GROUPS == 1 ? 0 : (int)(threadIdx.x / FIELD_THREADS);
    const int app_cols = p.xc ? p.app_dim : 0, app_ld = fwd_app_ld(app_cols), group_bytes = fwd_group_bytes<TAPS>(K0, app_cols);
    uint8_t* w_s = smem;                                        // [256 x KB]  w0b
    float* wh_s = reinterpret_cast<float*>(w_s + HID * KB * 2); // [256]
    uint8_t* a_s = reinterpret_cast<uint8_t*>(wh_s + HID) + grp * group_bytes;   // [boxes]  features hi
    uint8_t* a2_s = a_s + nbox * FWD_BOX_BYTES;                 // [boxes]  features lo
    uint8_t* at_s = a2_s + nbox * FWD_BOX_BYTES;                // [2 chunks][128 x 16 bytes]  tail
    float* part_s = reinterpret_cast<float*>(at_s + TILE_M * 32);   // [2][128] partial head sums
    float* sdf_s = part_s + 2 * TILE_M;                         // [7][18]
    // the mbarrier 8-byte aligned whatever the tile's row count: 128 floats past sdf_s
    // (125 or 126 evaluation rows + padding)
    uint64_t* mbar = reinterpret_cast<uint64_t*>(sdf_s + FWD_SDF_FLOATS);
    uint64_t* mbar_a = mbar + 1;                                // the A tile's TMA loads
    uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 2);    // (group 0's)
    FwdSample* ring = reinterpret_cast<FwdSample*>(mbar + 3);   // [FWD_RING][SPT]
    float* app_s = reinterpret_cast<float*>(ring + FWD_RING * SPT);   // [FWD_APP_RING][SPT][app_ld]

    // thread and warp within the group; the group's barrier
    const int tid = threadIdx.x % FIELD_THREADS, warp = tid >> 5, lane = tid & 31;
    auto group_sync = [&]() { named_barrier_sync(1 + grp, FIELD_THREADS); };
    stage_rows_kmajor(w_s, (const __half*)p.w0b, 0, HID, KB, KB, threadIdx.x, FIELD_THREADS * GROUPS, HID);
    for (int i = threadIdx.x; i < HID; i += FIELD_THREADS * GROUPS) wh_s[i] = p.whead[i];
    if (tid == 0) {
        umma::mbar_init(mbar, 1);
        umma::mbar_init(mbar_a, 1);
        umma::fence_mbar_init();
    }
    if (threadIdx.x < 32) {
        umma::tmem_alloc(tslot, HID * GROUPS);
        umma::tmem_relinquish();
    }
    cp_async_wait_all();
    umma::fence_proxy_async_smem();
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem0 = *reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(tslot) - grp * group_bytes);
    const uint32_t tmem = tmem0 + (uint32_t)(grp * HID);
    const uint32_t idesc = umma::idesc_f16(TILE_M, HID);
    const uint32_t a_addr = umma::smem_u32(a_s), w_addr = umma::smem_u32(w_s), a2_addr = umma::smem_u32(a2_s);
    const uint32_t at_addr = umma::smem_u32(at_s);
    const float bhead = p.bhead[0];
    const int64_t ntiles = (p.Ns + SPT - 1) / SPT;
    const int q = warp & 3, half = warp >> 2;
    const int row = q * 32 + lane;
    const int e_row = row / SPT, sl_row = row % SPT;
    uint32_t phase = 0;

    // features of a tile, gathered by k_field_gather into x0ext, loaded by TMA (thread 0; rows past
    // the end arrive as zeros, columns past a part are not used); the next tile's load overlaps
    // this tile's epilogue (A is free once its MMAs completed)
    // (a timed-out tile ends the loop at its top, before its load_a: no load is left in flight)
    auto load_a = [&](int64_t tt) {
        umma::mbar_arrive_expect_tx(mbar_a, (uint32_t)fwd_tile_bytes(K0));
        const int row0 = (int)(tt * (SPT * EVALS));
        for (int j = 0; j < nbox; ++j) {
            umma::tma_load_2d(a2_s + j * FWD_BOX_BYTES, &tm_x, KB + 64 * j, row0, mbar_a);
            umma::tma_load_2d(a_s + j * FWD_BOX_BYTES, &tm_x, 64 * j, row0, mbar_a);
        }
        umma::tma_load_3d(at_s, &tm_tail, 0, row0, 0, mbar_a);
    };
    auto issue = [&](uint32_t phase_a) {           // the k-th call waits for the k-th load: phase k & 1
        if (tid == 0) {
            if (!umma::mbar_wait(mbar_a, phase_a)) flag_timeout(p.err, 1);   // the A tile's TMA loads
            umma::fence_after_sync();
            // smallest terms first: the tensor core's FP32 accumulation drops low
            // bits of addends much smaller than the running sum, so the fp16
            // residuals go in before the hi features and the large position/bias tail
            const uint32_t sbo = (uint32_t)KB * 16u;
            for (int i = 0; i < 2; ++i) {
                const uint32_t base = i == 0 ? a2_addr : a_addr;
                for (int ks = 0; ks < K0 / 16; ++ks)
                    umma::mma_f16(tmem, umma::make_desc_sw128(base + (ks >> 2) * FWD_BOX_BYTES + (ks & 3) * 32u),
                                  umma::make_desc(w_addr + ks * 256u, 128u, sbo), idesc, (i > 0 || ks > 0) ? 1u : 0u);
            }
            umma::mma_f16(tmem, umma::make_desc(at_addr, TILE_M * 16u, 128u),
                          umma::make_desc(w_addr + (K0 / 16) * 256u, 128u, sbo), idesc, 1u);
            umma::mma_commit(mbar);
        }
    };
    // The per-sample phase reads per-ray inputs (flags, direction, centre, appearance code)
    // behind one or two dependent global loads.  They are prefetched into a ring of FWD_RING
    // tiles by the threads that have no sample of their own in that phase, one load level per
    // tile: the ray index three tiles ahead, the per-ray values two tiles ahead, the appearance
    // row one tile ahead; each level lands before the next reads it (a CTA barrier apart).
    const bool want_xc = p.xc != nullptr;
    const bool want_app = want_xc && p.app_table && p.app_dim > 0;
    auto slot = [&](int k) { return ring + (k & (FWD_RING - 1)) * SPT; };
    auto app_of = [&](int k, int js) { return app_s + ((k & (FWD_APP_RING - 1)) * SPT + js) * app_ld; };
    auto tile_of = [&](int k) { return (int64_t)blockIdx.x * GROUPS + grp + (int64_t)k * gridDim.x * GROUPS; };
    auto pre_ray = [&](int k, int js) {
        const int64_t tk = tile_of(k), ss = tk * SPT + js;
        slot(k)[js].r = (tk < ntiles && ss < p.Ns) ? ray_of(p, ss) : -1;
    };
    auto pre_vals = [&](int k, int js) {
        FwdSample& e = slot(k)[js];
        const int r = e.r;
        if (r < 0) return;
        e.out = p.outside && p.outside[r];
        if (want_xc) {
            const int64_t ss = tile_of(k) * SPT + js;
            sample_point_of_ray(p, ss, r, e.c);
#pragma unroll
            for (int i = 0; i < 3; ++i) e.dv[i] = p.ray_unit[3 * r + i];
        }
        if (want_app) e.appi = p.app_idx[r];
    };
    auto pre_app = [&](int k, int js) {
        const FwdSample& e = slot(k)[js];
        if (e.r < 0 || !want_app) return;
        float* dst = app_of(k, js);
        const float* a = p.app_table + (int64_t)e.appi * p.app_dim;
        for (int i0 = 0; i0 < p.app_dim; i0 += 8) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = i0 + j < p.app_dim ? a[i0 + j] : 0.0f;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (i0 + j < p.app_dim) dst[i0 + j] = v[j];
        }
    };
    constexpr int LD0 = (SPT * 6 + 31) / 32 * 32;    // first loader thread
    static_assert(LD0 + 3 * SPT <= FIELD_THREADS, "the forward's prefetch loaders fit the CTA");
    if (tid < SPT) {
        pre_ray(0, tid);
        pre_ray(1, tid);
        pre_ray(2, tid);
    }
    group_sync();
    if (tid < SPT) {
        pre_vals(0, tid);
        pre_vals(1, tid);
    }
    group_sync();
    if (tid < SPT) pre_app(0, tid);
    int64_t t = tile_of(0);
    const int64_t t_step = (int64_t)gridDim.x * GROUPS;
    if (t < ntiles && tid == 0) load_a(t);
    group_sync();
    if (t < ntiles) issue(0u);
    for (int it = 0; t < ntiles; t += t_step, ++it) {
        const int64_t s0 = t * SPT;
        const bool ok = named_barrier_and(1 + grp, FIELD_THREADS, umma::mbar_wait(mbar, phase));
        phase ^= 1u;
        if (!ok) {
            flag_timeout(p.err, 1);
            break;
        }
        umma::fence_after_sync();
        const int64_t tn = t + t_step;
        if (tn < ntiles && tid == 0) load_a(tn);
        // epilogue: h = softplus(pre) ; partial head dot ; centre rows keep h in h0c
        const int64_t s = s0 + sl_row;
        const bool keep = row < SPT * EVALS && s < p.Ns && e_row == 0;
        uint64_t part01 = 0ull, part23 = 0ull;          // partial sums of columns j % 4 = 0, 1 and 2, 3
        const SoftplusK spk = softplus_k(p.beta);
#pragma unroll 1
        for (int c0 = half * 128; c0 < half * 128 + 128; c0 += 32) {
            float v[32];
            umma::tmem_ld32(umma::taddr(tmem, q * 32, c0), v);
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                const uint64_t h0 = softplus_fast_h2(pack_f32x2(v[j], v[j + 1]), spk);
                const uint64_t h1 = softplus_fast_h2(pack_f32x2(v[j + 2], v[j + 3]), spk);
                unpack_f32x2(h0, v[j], v[j + 1]);
                unpack_f32x2(h1, v[j + 2], v[j + 3]);
                const ulonglong2 wh = *reinterpret_cast<const ulonglong2*>(wh_s + c0 + j);
                part01 = fma_f32x2(wh.x, h0, part01);
                part23 = fma_f32x2(wh.y, h1, part23);
            }
            if (keep) {
                const int64_t off = s * (int64_t)(p.ld_h0c > 0 ? p.ld_h0c : HID) + c0;
                __half* dst = (__half*)p.h0c + off;
#pragma unroll
                for (int j = 0; j < 32; j += 8) store_half8(dst + j, v + j);
                if (p.h0c_lo) {
                    __half* lo = (__half*)p.h0c_lo + off;
#pragma unroll
                    for (int j = 0; j < 32; j += 8) store_half8_lo(lo + j, v + j);
                }
            }
        }
        part_s[half * TILE_M + row] = sum_f32x2(part01) + sum_f32x2(part23);
        umma::fence_before_sync();
        group_sync();
        // the accumulator has been read: the next tile's MMAs run under the per-sample phase (behind it,
        // 2.39 ms for 2.1 M samples where this takes 2.32)
        if (tn < ntiles) issue((uint32_t)(it + 1) & 1u);
        if (tid < SPT * EVALS) {
            sdf_s[tid] = part_s[tid] + part_s[TILE_M + tid] + bhead;
        }
        group_sync();
        // per-sample: gradient, Hessian diagonal, outside overwrite, colour-input columns;
        // six threads per sample, each storing one 8-column chunk of the colour-input tail
        // (the first of them also the SDF, gradient and Hessian)
        if (tid >= LD0 && tid < LD0 + 3 * SPT) {
            const int li = tid - LD0, st = li / SPT, js = li - st * SPT;
            if (st == 0) pre_ray(it + 3, js);
            else if (st == 1) pre_vals(it + 2, js);
            else pre_app(it + 1, js);
        }
        if (tid < SPT * 6) {
            const int js = tid / 6, kc8 = tid - 6 * js;
            const int64_t ss = s0 + js;
            const FwdSample& e = slot(it)[js];
            if (ss < p.Ns) {
                const int r = e.r;
                const bool out = e.out != 0;
                const float fc = out ? p.outside_val : sdf_s[js];
                float g[3], hh[3];
                if constexpr (TAPS == 6) {
                    // g_d = (f+ - f-) / (2 eps); H_dd = (f+ + f- - 2 f) / eps^2 (modules.py:144-155)
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const float fp = sdf_s[(1 + 2 * d) * SPT + js], fm = sdf_s[(2 + 2 * d) * SPT + js];
                        g[d] = __fdiv_rn(__fsub_rn(fp, fm), p.two_eps);
                        hh[d] = __fdiv_rn(__fsub_rn(__fadd_rn(fp, fm), __fmul_rn(2.0f, fc)), p.eps2);
                    }
                } else {
                    // g = (k1 f1 + k2 f2 + k3 f3 + k4 f4) / (4 e); H_xx = ((f1 + f2 + f3 + f4) / 2 - 2 f) / e^2,
                    // every diagonal entry H_xx / 3 (modules.py:167-174); two_eps = 4 e, eps2 = e^2
                    const float f1 = sdf_s[SPT + js], f2 = sdf_s[2 * SPT + js];
                    const float f3 = sdf_s[3 * SPT + js], f4 = sdf_s[4 * SPT + js];
                    const float sx = __fadd_rn(__fsub_rn(__fsub_rn(f1, f2), f3), f4);
                    const float sy = __fadd_rn(__fadd_rn(__fsub_rn(-f1, f2), f3), f4);
                    const float sz = __fadd_rn(__fsub_rn(__fadd_rn(-f1, f2), f3), f4);
                    g[0] = __fdiv_rn(sx, p.two_eps);
                    g[1] = __fdiv_rn(sy, p.two_eps);
                    g[2] = __fdiv_rn(sz, p.two_eps);
                    const float sum = __fadd_rn(__fadd_rn(__fadd_rn(f1, f2), f3), f4);
                    const float hxx = __fdiv_rn(__fsub_rn(__fmul_rn(sum, 0.5f), __fmul_rn(2.0f, fc)), p.eps2);
                    hh[0] = hh[1] = hh[2] = __fdiv_rn(hxx, 3.0f);
                }
                if (kc8 == 0) {
                    p.sdf[ss] = fc;
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        p.grad[3 * ss + d] = g[d];
                        p.hess[3 * ss + d] = hh[d];
                    }
                }
                if (p.xc && 8 * kc8 < p.ldxc - HID) {
                    // NeuralRGB input tail (modules.py:209-213): x, SH(d), normalize(g), app
                    const float* c = e.c;
                    const float dx = e.dv[0], dy = e.dv[1], dz = e.dv[2];
                    const float xx = dx * dx, yy = dy * dy, zz = dz * dz;
                    float col[22];
                    col[0] = c[0]; col[1] = c[1]; col[2] = c[2];
                    // real spherical-harmonic basis, degree <= 3 (spherical_harmonics.py:47-84)
                    col[3] = 0.28209479177387814f;
                    col[4] = -0.4886025119029199f * dy;
                    col[5] = 0.4886025119029199f * dz;
                    col[6] = -0.4886025119029199f * dx;
                    col[7] = 1.0925484305920792f * dx * dy;
                    col[8] = -1.0925484305920792f * dy * dz;
                    col[9] = 0.31539156525252005f * (2.0f * zz - xx - yy);
                    col[10] = -1.0925484305920792f * dx * dz;
                    col[11] = 0.5462742152960396f * (xx - yy);
                    col[12] = -0.5900435899266435f * dy * (3.0f * xx - yy);
                    col[13] = 2.890611442640554f * dx * dy * dz;
                    col[14] = -0.4570457994644658f * dy * (4.0f * zz - xx - yy);
                    col[15] = 0.3731763325901154f * dz * (2.0f * zz - 3.0f * xx - 3.0f * yy);
                    col[16] = -0.4570457994644658f * dx * (4.0f * zz - xx - yy);
                    col[17] = 1.445305721320277f * dz * (xx - yy);
                    col[18] = -0.5900435899266435f * dx * (xx - 3.0f * yy);
                    const float nrm = fmaxf(sqrtf(g[0] * g[0] + g[1] * g[1] + g[2] * g[2]), 1e-12f);
                    col[19] = g[0] / nrm; col[20] = g[1] / nrm; col[21] = g[2] / nrm;
                    // this thread's 8 columns k = 8 kc8 + i: the 22 computed ones picked with
                    // compile-time indices (col[] stays in registers), the appearance code read
                    // straight from the table, and the last (padding) column a constant 1: the
                    // colour layer-0 weight gradient dZ^T xc then carries the bias gradient there
                    const float* a = want_app ? app_of(it, js) : nullptr;
                    (void)r;
                    __half* dst = (__half*)p.xc + ss * (int64_t)p.ldxc + HID;
                    const int ncol = p.ldxc - HID;
                    float o8[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int k = 8 * kc8 + i;
                        float val = 0.0f;
#pragma unroll
                        for (int cc = 0; cc < 22; ++cc)
                            if (cc == k) val = col[cc];
                        if (a && k >= 22 && k - 22 < p.app_dim) val = a[k - 22];
                        if (k == ncol - 1) val = 1.0f;
                        o8[i] = val;
                    }
                    store_half8(dst + 8 * kc8, o8);
                    if (p.xc_lo) store_half8_lo((__half*)p.xc_lo + ss * (int64_t)p.ldxc + HID + 8 * kc8, o8);
                }
            }
        }
        group_sync();
    }
    umma::fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) umma::tmem_dealloc(tmem0, HID * GROUPS);
}

// ---------------------------------------------------------------------------
// backward

// One 128-row tile (18 samples x 7 evaluations) per iteration:
//   MMA1 recomputes the pre-activations (A = x0ext's features hi | tail, B = w0b;
//        plus the features lo against the W0e prefix), exactly as the forward;
//   the epilogue forms d_pre = (d f w_head + [centre] d_h0c) softplus'(pre) and the
//        head-weight gradient, writes d_pre as an fp16 hi + lo pair into TMEM (the A
//        operand of MMA2) and its hi half to shared memory: the A operand of the in-kernel
//        layer-0 weight gradient (DW below), or staging for the global d_pre0 rows;
//   MMA2 d_enc = d_pre W0e (A from TMEM, B = the W0e part of MMA1's w0b tile read
//        MN-major) goes to global for k_field_scatter.
// The +eps and -eps taps of a sample carry large, nearly cancelling d_pre, so a
// single fp16 rounding of d_pre would dominate the table-gradient error: hence the pair.
// TMEM without DW (512 columns, one CTA per SM): [0, 256) MMA1's accumulator, reused
// for MMA2's [128 x K0] result; [256, 384) d_pre hi, [384, 512) d_pre lo.
// d_pre0 (without DW) and d_enc leave through a 4 KB staging buffer per warp and TMA stores
// (one thread per row would touch 32 cache lines per store instruction); a tile has
// 126 rows, so the last lane quadrant stores a 30-row box.
constexpr size_t BWD_SMEM_FLOOR = 120 * 1024;   // > half an SM's shared memory: one CTA per SM
constexpr int BWD_EPI_WARPS = 16;                // 4 lane quadrants x 4 parts of the hidden units
constexpr int BWD_EPI_THREADS = BWD_EPI_WARPS * 32;
// and a warp that loads, issues the MMAs and runs the prologue: as an epilogue warp's extra work those
// held the other fifteen up.  With it and the halves below 6.49 ms for 2.1 M samples at K0 = 64, 6.99
// with one epilogue warp issuing everything after the whole epilogue (17 warps leave 96 registers
// a thread, which the epilogue just fits).
constexpr int BWD_THREADS = BWD_EPI_THREADS + 32;
constexpr int BWD_STAGE_BYTES = 4096;            // per warp: 32 rows x 128 bytes
constexpr int DH0_LD = HID + 4;                  // d_h0c rows in shared memory, padded against bank conflicts

// DW (K0 <= 64, the caller passes d_w0): the layer-0 weight gradient dW0 = d_pre^T [x hi |
// tail] + d_pre^T x lo is accumulated here instead of through d_pre0 and a separate GEMM.
//   * d_pre's hi/lo pair is written over MMA1's accumulator in place (chunk c: hi in
//     columns [16c, 16c + 8), lo in [16c + 8, 16c + 16)), which frees TMEM for MMA2's
//     result at 256 and two dW0 accumulators (hidden halves, K0 + 16 columns each) after it.
//   * The dW0 MMAs read both operands MN-major: A = the d_pre hi rows of the staging
//     buffers (128-byte swizzle atoms of 64 hidden units x 8 rows), B = the tile's x0ext rows.
//   * The feature tile is double-buffered: the next tile's load may not overwrite what
//     dW0 reads.
//   * Hidden units 0-127 come first: the lo part of MMA2 and the hi dW0 MMAs of them run under the
//     epilogue of units 128-255, then their lo rows replace the hi rows in the staging area, so that
//     the tile's second phase is MMA2's rest, the other half's hi dW0 and this half's lo dW0.  Every
//     accumulator takes its products in one order: MMA2 lo then hi, dW0 hi x hi, hi x lo, lo x hi.
//   * d_enc leaves through the rows of units 0-127, whose MMAs are done by then, while the lo dW0 MMAs of
//     units 128-255 read theirs.
//   * The lo feature rows are K0 + 16 columns wide, the last 16 zero, so that the lo dW0
//     MMAs have the hi MMAs' shape (MMAs into one accumulator are ordered when their
//     shapes agree).
//   * MMA1 of the next tile is issued as soon as MMA2 has completed and the warps have read d_pre's lo
//     half (D1 is free then), under the d_enc epilogue.
//   * Each CTA adds its dW0 into d_w0 with atomics at the end.
template <int F, bool DW, int TAPS>
__global__ void __launch_bounds__(BWD_THREADS, 1) k_field_bwd(FieldParams p,
                                                             const __grid_constant__ CUtensorMap tm_pre32,
                                                             const __grid_constant__ CUtensorMap tm_pre30,
                                                             const __grid_constant__ CUtensorMap tm_enc32,
                                                             const __grid_constant__ CUtensorMap tm_enc30,
                                                             const __grid_constant__ CUtensorMap tm_plo32,
                                                             const __grid_constant__ CUtensorMap tm_plo30,
                                                             const __grid_constant__ CUtensorMap tm_xhi,
                                                             const __grid_constant__ CUtensorMap tm_xlo) {
    constexpr int EVALS = TapTile<TAPS>::EVALS, SPT = TapTile<TAPS>::SPT, TILE_ROWS = TapTile<TAPS>::ROWS;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int K0 = p.K0;
    const int KB = K0 + 16;                                     // features hi + tail
    uint8_t* stage_s = smem;                                    // [16][4 KB] TMA store staging, dW0's A operand
    uint8_t* w_s = stage_s + BWD_EPI_WARPS * BWD_STAGE_BYTES;   // [256 x KB]  w0b: B of MMA1
    uint8_t* a_s0 = w_s + HID * KB * 2;                         // [128 x KB]  features hi | tail
    const int KL = DW ? KB : K0;                                // lo row width (DW: zero-padded)
    uint8_t* a3_s0 = a_s0 + TILE_M * KB * 2;                    // [128 x KL]  features lo
    uint8_t* a_s1 = DW ? a3_s0 + TILE_M * KL * 2 : a_s0;        // the second buffer (DW)
    uint8_t* a3_s1 = DW ? a_s1 + TILE_M * KB * 2 : a3_s0;
    float* wh_s = reinterpret_cast<float*>(a3_s1 + TILE_M * KL * 2);   // [256] head weights
    float* dwh_s = wh_s + HID;                                  // [256] d_whead accumulator
    float* df_s = dwh_s + HID;                                  // [2][7][18] d f per evaluation, double-buffered
    float* dh0_s = df_s + TapTile<TAPS>::DF_FLOATS;              // [SPT][DH0_LD] d_h0c of the tile's samples
    uint64_t* mbar = reinterpret_cast<uint64_t*>(dh0_s + SPT * DH0_LD);
    uint64_t* mbar_a = mbar + 1;                                // the A tile's TMA loads
    // DW: hidden units 0-127 written (every epilogue warp); their hi dW0 MMAs done; the lo rows of
    // units 128-255 written (every epilogue warp)
    uint64_t *mbar_half = mbar + 2, *mbar_dw = mbar + 3, *mbar_lo = mbar + 4;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 5);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    stage_rows_kmajor(w_s, (const __half*)p.w0b, 0, HID, KB, KB, tid, BWD_THREADS, HID);
    for (int i = tid; i < HID; i += BWD_THREADS) {
        wh_s[i] = p.whead[i];
        dwh_s[i] = 0.0f;
    }
    if (DW) {
        // the zero columns [K0, K0 + 16) of both lo tiles: 16 row groups x 256 bytes each
        for (int i = tid; i < 2 * (TILE_M / 8) * 16; i += BWD_THREADS) {
            uint8_t* base = (i >> 8) ? a3_s1 : a3_s0;
            *reinterpret_cast<uint4*>(base + ((i >> 4) & 15) * (KL * 16) + K0 * 16 + (i & 15) * 16) =
                make_uint4(0, 0, 0, 0);
        }
    }
    if (tid == 0) {
        umma::mbar_init(mbar, 1);
        umma::mbar_init(mbar_a, 1);
        umma::mbar_init(mbar_half, BWD_EPI_WARPS);
        umma::mbar_init(mbar_dw, 1);
        umma::mbar_init(mbar_lo, BWD_EPI_WARPS);
        umma::fence_mbar_init();
    }
    if (warp == 0) {
        umma::tmem_alloc(tslot, 512);
        umma::tmem_relinquish();
    }
    cp_async_wait_all();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tslot;
    // d_pre hi/lo of hidden units [16c, 16c + 16): separate TMEM regions, or in place (DW)
    auto t_hi = [&](int c) { return DW ? tmem + 16u * c : tmem + HID + 8u * c; };
    auto t_lo = [&](int c) { return DW ? tmem + 16u * c + 8u : tmem + HID + HID / 2 + 8u * c; };
    const uint32_t t_enc = DW ? tmem + HID : tmem;              // MMA2's result
    const uint32_t t_dw = tmem + HID + K0;                      // DW: dW0 of hidden half h at + h KB
    const uint32_t idesc1 = umma::idesc_f16(TILE_M, HID);
    const uint32_t idesc2 = umma::idesc_f16_bmn(TILE_M, K0);
    const uint32_t w_addr = umma::smem_u32(w_s);
    // MMA2's and dW0's descriptors are built once per tile: a K = 16 step only moves the start
    // address (bits 0-13, in 16-byte units, below 2^14 for any shared-memory address), so each
    // MMA adds a multiple of a per-tile step
    auto desc_step = [](uint32_t bytes) { return (uint64_t)(bytes >> 4); };
    // feature buffer b (0, or 1 with DW): selects, not arrays, which would go to local memory
    auto a_buf = [&](int b) { return b ? a_s1 : a_s0; };
    auto a3_buf = [&](int b) { return b ? a3_s1 : a3_s0; };
    auto a_addr = [&](int b) { return umma::smem_u32(a_buf(b)); };
    auto a3_addr = [&](int b) { return umma::smem_u32(a3_buf(b)); };
    bool dw_first = true;                                       // the CTA's first dW0 MMA initialises
    const int64_t ntiles = (p.Ns + SPT - 1) / SPT;
    const bool epi = warp < BWD_EPI_WARPS;                      // an epilogue warp
    const int q = warp & 3, part = warp >> 2;                   // its lane quadrant and part of the hidden units
    // its i-th chunk of 16 hidden units: a quarter of them in a row, or (DW) an eighth of units 0-127,
    // then of 128-255
    auto chunk = [&](int i) { return DW ? (i >> 1) * 8 + part * 2 + (i & 1) : part * 4 + i; };
    const int row = q * 32 + lane;
    const int e_row = row / SPT, sl_row = row % SPT;
    uint32_t phase = 0;
    float dbh = 0.0f;
    bool ok = true;

    // the prologue, on the issuing warp (lane = sample of the tile): per-sample output gradients -> d f
    // of each evaluation (modules.py:144-156) into df_s[buf], for the next tile under this one's epilogue
    static_assert(TapTile<TAPS>::SPT <= 32, "the prologue's samples fit one warp");
    auto prologue = [&](int64_t tt, int buf) {
        if (!epi && lane < SPT) {
            const int64_t s = tt * SPT + lane;
            float* dfb = df_s + buf * (EVALS * SPT);
            float df[EVALS];
#pragma unroll
            for (int e = 0; e < EVALS; ++e) df[e] = 0.0f;
            if (s < p.Ns) {
                const int r = ray_of(p, s);
                float dg[3], dh[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    dg[d] = p.d_grad[3 * s + d];
                    dh[d] = p.d_hess[3 * s + d];
                }
                const float g0 = p.grad[3 * s], g1 = p.grad[3 * s + 1], g2 = p.grad[3 * s + 2];
                // normals = g / max(|g|, 1e-12) feed the colour MLP (model.py:167)
                const float* dn = p.d_xc + s * (int64_t)p.ld_dxc + p.normal_col;
                const float n0 = dn[0], n1 = dn[1], n2 = dn[2], dsdf = p.d_sdf[s];
                const bool out = p.outside && p.outside[r];
                const float len = sqrtf(g0 * g0 + g1 * g1 + g2 * g2);
                if (len > 1e-12f) {
                    const float inv = 1.0f / len;
                    const float u0 = g0 * inv, u1 = g1 * inv, u2 = g2 * inv;
                    const float dot = u0 * n0 + u1 * n1 + u2 * n2;
                    dg[0] += (n0 - u0 * dot) * inv;
                    dg[1] += (n1 - u1 * dot) * inv;
                    dg[2] += (n2 - u2 * dot) * inv;
                } else {
                    dg[0] += n0 * 1e12f; dg[1] += n1 * 1e12f; dg[2] += n2 * 1e12f;
                }
                float hsum = 0.0f;
                if constexpr (TAPS == 6) {
#pragma unroll
                    for (int d = 0; d < 3; ++d) {
                        const float a = dg[d] / p.two_eps, b = dh[d] / p.eps2;
                        df[1 + 2 * d] = a + b;
                        df[2 + 2 * d] = -a + b;
                        hsum += b;
                    }
                } else {
                    // d H_xx = (dH_x + dH_y + dH_z) / 3; tap i: k_i . dg / (4 e) + d H_xx / (2 e^2)
                    const float dhxx = (dh[0] + dh[1] + dh[2]) / 3.0f;
                    const float b = 0.5f * dhxx / p.eps2;
                    const float ax = dg[0] / p.two_eps, ay = dg[1] / p.two_eps, az = dg[2] / p.two_eps;
                    df[1] = ax - ay - az + b;
                    df[2] = -ax - ay + az + b;
                    df[3] = -ax + ay - az + b;
                    df[4] = ax + ay + az + b;
                    hsum = dhxx / p.eps2;
                }
                // the centre feeds alpha and the Hessian only where it was not overwritten
                df[0] = out ? 0.0f : (dsdf - 2.0f * hsum);
            }
#pragma unroll
            for (int e = 0; e < EVALS; ++e) {
                dfb[e * SPT + lane] = df[e];
                dbh += df[e];
            }
        }
    };
    // encoder features of a tile, streamed back from the forward's x0ext rows (rows
    // 126-127 of a tile read the next tile's first rows or zeros; their MMA results
    // are never used) by TMA: one thread, one box per 8-row group and part, straight into
    // the core-matrix layout (rows past the end, and the lo part's zero columns, arrive
    // as zeros); 512 threads' cp.async copies of the same bytes cost them ~2k clocks a tile
    const bool loader = tid == BWD_EPI_THREADS;
    bool a_pending = false;                         // (the loader, which issues and waits for these loads)
    auto load_a = [&](int64_t tt, int buf) {
        a_pending = true;
        umma::mbar_arrive_expect_tx(mbar_a, (uint32_t)(TILE_M * (KB + KL) * 2));
        const int row0 = (int)(tt * (SPT * EVALS));
#pragma unroll 1
        for (int g = 0; g < TILE_M / 8; ++g) {
            umma::tma_load_3d(a_buf(buf) + g * KB * 16, &tm_xhi, 0, row0 + 8 * g, 0, mbar_a);
            umma::tma_load_3d(a3_buf(buf) + g * KL * 16, &tm_xlo, 0, row0 + 8 * g, 0, mbar_a);
        }
    };
    uint32_t phase_a = 0;
    auto stage_dh0 = [&](int64_t tt) {             // one cp.async group
        for (int c = tid; c < SPT * (HID / 4); c += BWD_THREADS) {
            const int js = c / (HID / 4), k4 = c - js * (HID / 4);
            const int64_t ss = tt * SPT + js;
            float* dst = dh0_s + js * DH0_LD + 4 * k4;
            if (ss < p.Ns) cp_async16(dst, p.d_h0c + ss * HID + 4 * k4);
            else *reinterpret_cast<float4*>(dst) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        cp_async_commit();
    };
    auto issue1 = [&](int buf) {                   // the issuing warp converged
        if (!epi) {
            if (umma::elect_one()) {
                if (!umma::mbar_wait(mbar_a, phase_a)) flag_timeout(p.err, 1);   // the A tile's TMA loads
                a_pending = false;
                umma::fence_after_sync();
                issue_tile_mma_strided(tmem, a3_addr(buf), KL, w_addr, KB, K0, idesc1);   // residuals first
                issue_tile_mma(tmem, a_addr(buf), w_addr, KB, idesc1, true);
                umma::mma_commit(mbar);
            }
            __syncwarp();
            phase_a ^= 1u;
        }
    };
    int64_t t = blockIdx.x;
    if (t < ntiles) {
        prologue(t, 0);
        if (loader) load_a(t, 0);
        stage_dh0(t);
        cp_async_wait_all();
        umma::fence_proxy_async_smem();
    }
    __syncthreads();
    if (t < ntiles) issue1(0);
    int it = 0;
    // MMA completions: one thread polls the mbarrier and the CTA barrier hands on its result.  A wait that
    // ran out in one warp alone (ok differs) ends the loop for all at the next barrier.
    for (; t < ntiles; t += gridDim.x, ++it) {
        const int64_t s0 = t * SPT;
        cp_async_wait_group<0>();                    // this tile's d_h0c rows
        if (DW && lane == 0) umma::bulk_wait_read0();   // the previous tile's d_enc store has read its rows
        ok = __syncthreads_and(ok && (loader ? umma::mbar_wait(mbar, phase) : true));   // one poller
        phase ^= 1u;
        if (!ok) {
            flag_timeout(p.err, 1);
            break;
        }
        const int64_t tn = t + gridDim.x;
        const int cb = DW ? (it & 1) : 0, nb = DW ? ((it + 1) & 1) : 0;   // this tile's / the next tile's A
        const uint32_t par = (uint32_t)it & 1u;      // this tile's parity of the barriers that complete once per tile
        umma::fence_after_sync();
        // the next tile's A tile, under the d_pre epilogue: MMA1 of tile t has completed, and with DW
        // it goes to the other buffer, whose last readers (the previous tile's lo dW0 MMAs) completed
        // before MMA1(t).  (Issued after MMA2 instead, its writes slowed the shared-memory-bound dW0
        // MMAs.)
        if (tn < ntiles && loader) load_a(tn, nb);
        if (tn < ntiles) prologue(tn, (it + 1) & 1);
        uint8_t* stg = stage_s + warp * BWD_STAGE_BYTES;
        // d_pre's rows in the staging area: 64 hidden units, 128 rows of 128 bytes, per 16 KB; 128-byte
        // swizzle: 16-byte unit u of row r sits at u ^ (r & 7)
        auto stage16 = [&](int c, uint4 u0, uint4 u1) {
            uint8_t* r = stage_s + (c >> 2) * (4 * BWD_STAGE_BYTES) + row * 128;
            const int u = (c & 3) * 2;
            *reinterpret_cast<uint4*>(r + ((u ^ (lane & 7)) * 16)) = u0;
            *reinterpret_cast<uint4*>(r + (((u + 1) ^ (lane & 7)) * 16)) = u1;
        };
        // d_pre's lo half of chunk c, read back from TMEM, into those rows
        auto stage_lo = [&](int c) {
            float f[8];
            umma::tmem_ld8(umma::taddr(t_lo(c), q * 32, 0), f);
            stage16(c, make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3])),
                    make_uint4(__float_as_uint(f[4]), __float_as_uint(f[5]), __float_as_uint(f[6]), __float_as_uint(f[7])));
        };
        // descriptors of this tile's MMA2 and dW0 (warp-uniform values; the elected lane adds constant
        // multiples of row_step per MMA)
        const uint64_t row_step = desc_step(2u * KB * 16u);   // 16 rows (dW0's B) / 16 hidden units (MMA2's B)
        const uint64_t d_stage = umma::make_desc_sw128_mn(umma::smem_u32(stage_s), 16384u, 1024u);
        const uint32_t id_dw = umma::idesc_f16_mn(TILE_M, KB);
        const uint64_t d_w = umma::make_desc(w_addr, (uint32_t)KB * 16u, 128u);
        const uint64_t bx = umma::make_desc(a_addr(cb), KB * 16u, 128u);
        const uint64_t bx3 = umma::make_desc(a3_addr(cb), KB * 16u, 128u);
        // d_enc = d_pre * W0e, 32 steps: A = d_pre [128 x 256] in TMEM, lo chunks first (smaller addends),
        // then hi; B = W0e read MN-major from MMA1's w0b tile: the core matrix of hidden rows 8g..8g+7 and
        // feature columns 8c..8c+7 sits at g * KB * 16 + c * 128 bytes
        auto mma2 = [&](int i) {
            const int ks = i & (HID / 16 - 1);
            umma::mma_f16_ta(t_enc, i < HID / 16 ? t_lo(ks) : t_hi(ks), d_w + ks * row_step, idesc2, i > 0 ? 1u : 0u);
        };
        // dW0[h], 24 steps: += d_pre hi^T [x hi | tail], then d_pre hi^T [x lo | 0], then (the lo rows
        // staged) d_pre lo^T [x hi | tail].  A (hidden half h = staging blocks 2h, 2h + 1): atoms of 64
        // units x 8 rows, next 64 units 16 KB on, next 8 rows 1 KB on; B (the tile's rows, MN-major):
        // next 8 rows KB*16 bytes on, next 8 features 128 bytes on.
        auto mma_dw = [&](int h, int i) {
            const int k8 = i & (TILE_M / 16 - 1);
            umma::mma_f16(t_dw + (uint32_t)(h * KB), d_stage + desc_step(h * 32768 + k8 * 2048),
                          (i >= TILE_M / 16 && i < 2 * (TILE_M / 16) ? bx3 : bx) + k8 * row_step, id_dw,
                          (dw_first && i == 0) ? 0u : 1u);
        };
        if (DW && !epi) {
            // units 0-127, under the epilogue of the others: the lo part of MMA2 and the hi dW0 MMAs
            ok = __any_sync(0xffffffffu, lane == 0 && umma::mbar_wait(mbar_half, par)) != 0;
            if (ok && umma::elect_one()) {
                umma::fence_after_sync();
#pragma unroll
                for (int i = 0; i < 2 * (TILE_M / 16); ++i) {
                    if (i < HID / 32) mma2(i);
                    mma_dw(0, i);
                }
                umma::mma_commit(mbar_dw);
            }
            __syncwarp();
        }
        // (2) d_pre = (d f * w_head + [centre] d_h0c) * softplus'(pre) -> TMEM (hi, lo) and d_pre0
        const CUtensorMap* tm_pre = q == 3 ? &tm_pre30 : &tm_pre32;
        const CUtensorMap* tm_enc = q == 3 ? &tm_enc30 : &tm_enc32;
        const int y0 = (int)(t * TILE_ROWS) + q * 32;
        if (!DW && lane == 0) umma::bulk_wait_read0();  // the previous tile's d_enc store has read the buffer
        __syncwarp();
        if (epi) {
            // dead rows (past Ns, and rows 126-127) get d f = 0 and no d_h0c: their
            // pre-activations are finite, so their d_pre and head terms come out 0
            const int64_t s = s0 + sl_row;
            const bool live = row < SPT * EVALS && s < p.Ns;
            const float df = live ? df_s[(it & 1) * (EVALS * SPT) + row] : 0.0f;
            const bool centre = live && e_row == 0;
            const SoftplusK spk = softplus_k(p.beta);
            const uint64_t df2 = pack_f32x2(df, df);
            // the next chunk's TMEM load is in flight while this chunk is processed
            uint32_t rn[16];
            umma::tmem_ld16_nowait(umma::taddr(tmem, q * 32, 16 * chunk(0)), rn);
            umma::tmem_ld_wait16(rn);
#pragma unroll 1
            for (int i = 0; i < 4; ++i) {
                const int c = chunk(i), c0 = 16 * c;
                uint64_t v2[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v2[j] = pack_f32x2(__uint_as_float(rn[2 * j]), __uint_as_float(rn[2 * j + 1]));
                const bool more = i < 3;
                if (more) umma::tmem_ld16_nowait(umma::taddr(tmem, q * 32, 16 * chunk(i + 1)), rn);
                uint64_t dh0[8];
                if (centre) {
                    const ulonglong2* src = reinterpret_cast<const ulonglong2*>(dh0_s + sl_row * DH0_LD + c0);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const ulonglong2 f = src[j];
                        dh0[2 * j] = f.x;
                        dh0[2 * j + 1] = f.y;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) dh0[j] = 0ull;
                }
                float hc[16];   // d f * h per column: d w_head = sum over rows
                uint32_t hi[8], lo[8];
                // pairs of columns: the packed products and sums round as the single ones do and take half
                // the issue slots (7.12 -> 6.99 ms for 2.1 M samples)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    uint64_t h, sg;
                    softplus_fast2(v2[j], spk, h, sg);
                    const uint64_t wh = *reinterpret_cast<const uint64_t*>(wh_s + c0 + 2 * j);
                    const uint64_t d2 = mul_f32x2(fma_f32x2(df2, wh, dh0[j]), sg);
                    unpack_f32x2(mul_f32x2(df2, h), hc[2 * j], hc[2 * j + 1]);
                    float a, b;
                    unpack_f32x2(d2, a, b);
                    const __half2 h2 = __floats2half2_rn(a, b);
                    const float2 back = __half22float2(h2);
                    unpack_f32x2(sub_f32x2(d2, pack_f32x2(back.x, back.y)), a, b);
                    const __half2 l2 = __floats2half2_rn(a, b);
                    hi[j] = *reinterpret_cast<const uint32_t*>(&h2);
                    lo[j] = *reinterpret_cast<const uint32_t*>(&l2);
                }
                {
                    const float colsum = warp_column_sum16(hc, lane);
                    if (lane < 16 && colsum != 0.0f) atomicAdd(&dwh_s[c0 + lane], colsum);
                }
                if (more) umma::tmem_ld_wait16(rn);
                umma::tmem_st8(umma::taddr(t_hi(c), q * 32, 0), hi);
                umma::tmem_st8(umma::taddr(t_lo(c), q * 32, 0), lo);
                // d_pre0 (hi) into the staging rows; dead samples store zeros (their x0ext
                // rows are zero too)
                stage16(c, make_uint4(hi[0], hi[1], hi[2], hi[3]), make_uint4(hi[4], hi[5], hi[6], hi[7]));
                if (DW && i == 1) {                  // units 0-127 are complete
                    umma::tmem_wait_st();
                    umma::fence_proxy_async_smem();
                    umma::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) umma::mbar_arrive(mbar_half);
                }
            }
            if constexpr (DW) {
                // the lo rows of units 0-127 over their hi rows, which dW0 has read by now
                umma::tmem_wait_st();
                ok = __any_sync(0xffffffffu, lane == 0 && umma::mbar_wait(mbar_dw, par)) != 0;
#pragma unroll
                for (int i = 0; i < 2; ++i) stage_lo(chunk(i));
            }
        }
        umma::fence_proxy_async_smem();
        __syncwarp();
        if (!DW && epi && lane == 0) {
            umma::tma_store_2d(tm_pre, part * 64, y0, stg);
            umma::bulk_commit();
        }
        umma::tmem_wait_st();
        if (!DW && epi && p.d_pre0_lo) {
            // d_pre's lo half to d_pre0_lo through the same staging rows, read back from TMEM
            // once the hi store has read them (the layer-0 weight gradient needs the pair)
            if (lane == 0) umma::bulk_wait_read0();
            __syncwarp();
#pragma unroll 1
            for (int i = 0; i < 4; ++i) stage_lo(chunk(i));
            umma::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                umma::tma_store_2d(q == 3 ? &tm_plo30 : &tm_plo32, part * 64, y0, stg);
                umma::bulk_commit();
            }
        }
        umma::fence_before_sync();
        ok = __syncthreads_and(ok);
        if (!ok) {
            flag_timeout(p.err, 1);
            break;
        }
        // (3) what is left of MMA2 and of dW0, but for the lo rows of units 128-255
        if (!epi) {
            if (umma::elect_one()) {
                umma::fence_after_sync();
#pragma unroll
                for (int i = DW ? HID / 32 : 0; i < 2 * (HID / 16); ++i) {
                    mma2(i);
                    if (DW && i - HID / 32 < 2 * (TILE_M / 16)) mma_dw(1, i - HID / 32);
                    if (DW && i >= 2 * (HID / 16) - TILE_M / 16) mma_dw(0, i - 2 * (HID / 16) + 3 * (TILE_M / 16));
                }
                umma::mma_commit(mbar);
            }
            __syncwarp();                            // the issuing lane rejoins its warp before the barrier
        }
        if constexpr (DW) dw_first = false;
        if (tn < ntiles) {
            // the next tile's d_h0c rows, issued while every thread waits for MMA2 (copies landing
            // under the d_pre epilogue stretch it)
            stage_dh0(tn);                           // every warp has read this tile's d_h0c rows
        }
        ok = __syncthreads_and(loader ? umma::mbar_wait(mbar, phase) : true);   // one poller
        phase ^= 1u;
        if (!ok) {
            flag_timeout(p.err, 1);
            break;
        }
        umma::fence_after_sync();
        if constexpr (DW) {
            // dW0[1] += d_pre lo^T [x hi | tail]: its hi MMAs have completed with MMA2, so the staging
            // rows take d_pre's lo half, read back from TMEM before the next tile's MMA1
            // overwrites it.  The +eps / -eps taps carry large, nearly cancelling d_pre, and a
            // single fp16 rounding of d_pre in dW0 would leave ~1e-3 of it behind.
            if (epi) {
#pragma unroll
                for (int i = 2; i < 4; ++i) stage_lo(chunk(i));
                umma::fence_proxy_async_smem();
                umma::fence_before_sync();
                __syncwarp();
                if (lane == 0) umma::mbar_arrive(mbar_lo);
            } else {
                ok = __any_sync(0xffffffffu, lane == 0 && umma::mbar_wait(mbar_lo, par)) != 0;
                if (ok && umma::elect_one()) {
                    umma::fence_after_sync();
#pragma unroll
                    for (int i = 2 * (TILE_M / 16); i < 3 * (TILE_M / 16); ++i) mma_dw(1, i);
                    if (tn >= ntiles) umma::mma_commit(mbar);      // else MMA1's commit covers them
                }
                __syncwarp();
                // D1 is free: MMA2 has read d_pre, the warps its lo half
                if (ok && tn < ntiles) issue1(nb);
            }
        }
        // (4) d_enc rows to global for k_field_scatter: 16-column chunks dealt in turn
        // to the four warps of a lane quadrant (K0 <= 128: at most two per warp, one
        // 2 KB half of the staging buffer each; 64-byte swizzle: unit j of row r at j ^ ((r >> 1) & 3))
        // With DW (one chunk) they go through the rows of units 0-127, 2 KB per warp: dW0's MMAs have
        // read those, and are about to read the others.
        if (!DW && lane == 0) umma::bulk_wait_read0();   // the d_pre0 store has read the buffer
        __syncwarp();
        for (int c0 = part * 16, i = 0; epi && c0 < K0; c0 += 64, ++i) {
            float v[16];
            umma::tmem_ld16(umma::taddr(t_enc, q * 32, c0), v);
            uint8_t* eb = DW ? stage_s + warp * 2048 : stg + i * 2048;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float4*>(eb + lane * 64 + ((j ^ ((lane >> 1) & 3)) * 16)) =
                    make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            umma::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                umma::tma_store_2d(tm_enc, c0, y0, eb);
                umma::bulk_commit();
            }
        }
        umma::fence_before_sync();
        if constexpr (!DW) {
            __syncthreads();                         // the TMEM accumulator of tile t read; tile tn's A tile and d f in place
            if (tn < ntiles) issue1(nb);
        }                                            // (DW: the next tile's first barrier says so)
    }
    if (DW && blockIdx.x < ntiles) {                 // the last tile's lo dW0 MMAs
        const bool done = ok && (loader ? umma::mbar_wait(mbar, phase) : true);
        if (!done) flag_timeout(p.err, 1);
        ok = __syncthreads_and(done);
        umma::fence_after_sync();
    }
    cp_async_wait_all();
    if (loader && a_pending && !umma::mbar_wait(mbar_a, phase_a)) flag_timeout(p.err, 1);   // a load left in flight
    if (lane == 0) umma::bulk_wait0();               // this warp's TMA stores have completed
    umma::fence_before_sync();
    __syncthreads();
    if constexpr (DW) {
        // the CTA's dW0 (complete: the last tile's lo MMAs were waited for): warps with part 2h, 2h + 1
        // read hidden half h, one half of its KB columns each
        if (!dw_first && ok && epi) {
            umma::fence_after_sync();
            const int h = part >> 1, half_cols = KB / 2, cbeg = (part & 1) * half_cols;
            float* dst = p.d_w0 + (int64_t)(h * 128 + q * 32 + lane) * KB;
            // four columns per atomic (rows are multiples of 64 bytes): one element each, every lane in a
            // row of its own, cost as much as a tile: 32.7 us against 19.4 for 114 one-tile CTAs (K0 = 32)
            const bool vec = (reinterpret_cast<uintptr_t>(p.d_w0) & 15) == 0;
            for (int c = cbeg; c < cbeg + half_cols; c += 8) {
                float v[8];
                umma::tmem_ld8(umma::taddr(t_dw + (uint32_t)(h * KB), q * 32, c), v);
                if (vec) {
                    atomicAdd(reinterpret_cast<float4*>(dst + c), make_float4(v[0], v[1], v[2], v[3]));
                    atomicAdd(reinterpret_cast<float4*>(dst + c + 4), make_float4(v[4], v[5], v[6], v[7]));
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (v[j] != 0.0f) atomicAdd(dst + c + j, v[j]);
                }
            }
        }
        umma::fence_before_sync();
        __syncthreads();
    }
    for (int i = tid; i < HID; i += BWD_THREADS)
        if (dwh_s[i] != 0.0f) atomicAdd(&p.d_whead[i], dwh_s[i]);
    dbh = warp_sum(dbh);
    if (lane == 0 && dbh != 0.0f) atomicAdd(p.d_bhead, dbh);
    if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------
// SDF-only evaluation at arbitrary points or on a lattice block (forward only):
// NeuralSDF.sdf (modules.py:73-74) for mesh extraction (mesh.py:33-35, with the
// sign flip of scripts/extract_mesh.py:85) and for the sampler's no-grad
// evaluations (model.py:238, 245).  Tile = 128 points, one evaluation each.

struct SdfPointsArgs {
    int64_t M;
    const float* pts;          // [M, 3] or NULL for lattice mode
    const float* ax;           // lattice axes: x [nx], y [ny], z [nz]
    const float* ay;
    const float* az;
    int nx, ny, nz;
    float sign;                // +1, or -1 for the mesh's negated field
    float* out;                // [M], or rows of `inner` values `ld` apart (inner > 0)
    int inner, ld;
};

// Warp-specialised, one persistent CTA per SM, two tiles in flight:
//   warps 0-15   gather: warp w fills rows 32 (w & 3) .. of every fourth level starting at
//                w >> 2, one lane per row, so the lanes of a warp share their level's constants
//                and neighbouring points of a lattice row share corners; a buffer is full when
//                all sixteen have arrived on full[b];
//   warp 24      issues the tile's MMAs (A: the features' fp16 residuals, then hi; B: W0e) into
//                one of two TMEM accumulators; their completion (done[b]) frees the
//                feature buffer and starts the epilogue;
//   warps 16-23  the epilogue: the position columns, bias, softplus and the head in fp32, one
//                half of the hidden units per warp; tempty[b] hands the accumulator back.
// Gather, MMAs and epilogue of one tile used to follow one another in eight warps, so the
// table's latency stood in every tile.  2.1 M lattice points x 16 levels: 3.79 ms
// in that form, 1.16 ms in this one; 5.5 M scattered points of a view (four calls) 12.1 and 4.4 ms.
constexpr int SP_GATHER_WARPS = 16;
constexpr int SP_EPI_WARPS = 8;
constexpr int SP_TPB = (SP_GATHER_WARPS + SP_EPI_WARPS + 1) * 32;
constexpr int SP_XRING = 4;      // points kept for the epilogue: two tiles ahead of the one it may still read

static size_t sdf_points_smem(int K0) {
    return (size_t)HID * K0 * 2 + 4 * (size_t)TILE_M * K0 * 2 + HID * 20 + 2 * 2 * TILE_M * 4 +
           SP_XRING * TILE_M * 12 + 6 * 8 + 16;
}

template <int F>
__global__ void __launch_bounds__(SP_TPB, 1) k_sdf_points(FieldParams p, SdfPointsArgs q) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int K0 = p.K0, A = p.active;
    const uint32_t a_bytes = (uint32_t)TILE_M * K0 * 2;
    uint8_t* w_s = smem;                                        // [256 x K0]  W0e
    uint8_t* a_s = w_s + HID * K0 * 2;                          // [2 buffers][lo, hi][128 x K0]  features
    float4* wx_s = reinterpret_cast<float4*>(a_s + 4 * a_bytes);   // [256] position columns, bias
    float* wh_s = reinterpret_cast<float*>(wx_s + HID);         // [256] head
    float* part_s = wh_s + HID;                                 // [2][2][128] partial head sums
    float* x_s = part_s + 4 * TILE_M;                           // [SP_XRING][3][128] points
    uint64_t* full = reinterpret_cast<uint64_t*>(x_s + SP_XRING * 3 * TILE_M);   // [2]
    uint64_t* done = full + 2;                                  // [2]
    uint64_t* tempty = done + 2;                                // [2]
    uint32_t* tslot = reinterpret_cast<uint32_t*>(tempty + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (A * F < K0)                                             // the padding columns stay zero
        for (uint32_t i = tid; i < 4 * a_bytes / 16; i += SP_TPB)
            reinterpret_cast<uint4*>(a_s)[i] = make_uint4(0, 0, 0, 0);
    umma::fence_proxy_async_smem();
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            umma::mbar_init(&full[b], SP_GATHER_WARPS);
            umma::mbar_init(&done[b], 2);
            umma::mbar_init(&tempty[b], SP_EPI_WARPS);
        }
        umma::fence_mbar_init();
    }
    if (warp == SP_GATHER_WARPS + SP_EPI_WARPS) {
        umma::tmem_alloc(tslot, 2 * HID);
        umma::tmem_relinquish();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tslot;
    const int64_t ntiles = (q.M + TILE_M - 1) / TILE_M;

    if (warp < SP_GATHER_WARPS) {
        // ---------------- gather ----------------
        const int row = (warp & 3) * 32 + lane;
        const __half* const table = (const __half*)p.table;
        const bool small = q.M <= (int64_t)0xffffffffll;        // 32-bit lattice index arithmetic
        int it = 0;
        for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
            const int b = it & 1;
            if (it >= 2 && !umma::mbar_wait(&done[b], (uint32_t)((it >> 1) - 1) & 1u)) {
                if (lane == 0) flag_timeout(p.err, 1);
                break;
            }
            const int64_t m = t * TILE_M + row;
            const bool live = m < q.M;
            float x[3] = {0.f, 0.f, 0.f};
            if (live) {
                if (q.pts) {
                    x[0] = q.pts[3 * m]; x[1] = q.pts[3 * m + 1]; x[2] = q.pts[3 * m + 2];
                } else if (small) {
                    const uint32_t m32 = (uint32_t)m, jk = m32 / (uint32_t)q.nz, i = jk / (uint32_t)q.ny;
                    x[0] = q.ax[i]; x[1] = q.ay[jk - i * (uint32_t)q.ny]; x[2] = q.az[m32 - jk * (uint32_t)q.nz];
                } else {
                    const int64_t jk = m / q.nz, i = jk / q.ny;
                    x[0] = q.ax[i]; x[1] = q.ay[jk - i * q.ny]; x[2] = q.az[m - jk * q.nz];
                }
            }
            if (warp < 4) {
                float* xr = x_s + (it & (SP_XRING - 1)) * 3 * TILE_M + row;
                xr[0] = x[0]; xr[TILE_M] = x[1]; xr[2 * TILE_M] = x[2];
            }
            uint8_t* lo_s = a_s + (size_t)(2 * b) * a_bytes;
            uint8_t* hi_s = lo_s + a_bytes;
#pragma unroll 1
            for (int l = warp >> 2; l < A; l += SP_GATHER_WARPS / 4) {
                uint64_t acc[F / 2];
#pragma unroll
                for (int f = 0; f < F / 2; ++f) acc[f] = 0ull;
                if (live) {
                    const LevelDesc d = level_desc(p.grid, l);
                    const GridCell g = grid_cell(d.scale, x);
                    TableRow<F> r[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        r[k].load(table + (d.offset + grid_index(d, g.b[0] + (k & 1), g.b[1] + ((k >> 1) & 1),
                                                                 g.b[2] + ((k >> 2) & 1))) * F);
#pragma unroll
                    for (int k = 0; k < 8; ++k) r[k].fma(corner_weight(k, g.f[0], g.f[1], g.f[2]), acc);
                }
                float v[F];
#pragma unroll
                for (int f = 0; f < F / 2; ++f) unpack_f32x2(acc[f], v[2 * f], v[2 * f + 1]);
                write_tile_features<F>(hi_s, lo_s, row, l, K0, v);
            }
            umma::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&full[b]);
        }
    } else if (warp == SP_GATHER_WARPS + SP_EPI_WARPS) {
        // ---------------- MMA issue ----------------
        named_barrier_sync(1, (SP_EPI_WARPS + 1) * 32);          // the weights are staged
        if (umma::elect_one()) {
            const uint32_t idesc = umma::idesc_f16(TILE_M, HID);
            const uint32_t w_addr = umma::smem_u32(w_s), a_addr = umma::smem_u32(a_s);
            int it = 0;
            for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
                const int b = it & 1;
                const uint32_t use = (uint32_t)(it >> 1);
                if (!umma::mbar_wait(&full[b], use & 1u) || (use > 0 && !umma::mbar_wait(&tempty[b], (use - 1) & 1u))) {
                    flag_timeout(p.err, 1);
                    break;
                }
                umma::fence_after_sync();
                const uint32_t d_tmem = tmem + (uint32_t)(b * HID), lo = a_addr + 2u * b * a_bytes;
                issue_tile_mma(d_tmem, lo, w_addr, K0, idesc);                  // residuals first
                issue_tile_mma(d_tmem, lo + a_bytes, w_addr, K0, idesc, true);
                umma::mma_commit(&done[b]);
                umma::mbar_arrive(&done[b]);         // hands the points' shared-memory writes on, too
            }
        }
        __syncwarp();
    } else {
        // ---------------- epilogue ----------------
        const int et = tid - SP_GATHER_WARPS * 32;
        stage_rows_kmajor(w_s, (const __half*)p.w0e, 0, HID, K0, K0, et, SP_EPI_WARPS * 32, HID);
        for (int i = et; i < HID; i += SP_EPI_WARPS * 32) {
            wx_s[i] = make_float4(p.w0x[3 * i], p.w0x[3 * i + 1], p.w0x[3 * i + 2], p.b0[i]);
            wh_s[i] = p.whead[i];
        }
        cp_async_wait_all();
        umma::fence_proxy_async_smem();
        named_barrier_sync(1, (SP_EPI_WARPS + 1) * 32);
        const float bhead = p.bhead[0];
        const SoftplusK spk = softplus_k(p.beta);
        const int qd = warp & 3, half = (warp - SP_GATHER_WARPS) >> 2;
        const int row = qd * 32 + lane;
        int it = 0;
        for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
            const int b = it & 1;
            // (all eight warps leave together: they share the barriers below)
            if (!named_barrier_and(2, SP_EPI_WARPS * 32, umma::mbar_wait(&done[b], (uint32_t)(it >> 1) & 1u))) {
                if (lane == 0) flag_timeout(p.err, 1);
                break;
            }
            umma::fence_after_sync();
            const float* xr = x_s + (it & (SP_XRING - 1)) * 3 * TILE_M + row;
            const float x[3] = {xr[0], xr[TILE_M], xr[2 * TILE_M]};
            float part4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
            for (int c0 = half * 128; c0 < half * 128 + 128; c0 += 32) {
                float v[32];
                umma::tmem_ld32(umma::taddr(tmem, qd * 32, b * HID + c0), v);
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    const float4 w = wx_s[c0 + j];
                    const float z = v[j] + w.x * x[0] + w.y * x[1] + w.z * x[2] + w.w;
                    part4[j & 3] = fmaf(wh_s[c0 + j], softplus_fast_h(z, spk), part4[j & 3]);
                }
            }
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&tempty[b]);
            float* ps = part_s + b * 2 * TILE_M;
            ps[half * TILE_M + row] = (part4[0] + part4[1]) + (part4[2] + part4[3]);
            named_barrier_sync(2, SP_EPI_WARPS * 32);
            const int64_t m = t * TILE_M + et;
            if (et < TILE_M && m < q.M) {
                const int64_t row = q.inner > 0 ? m / q.inner : 0;
                q.out[row * q.ld + m - row * q.inner] = q.sign * (ps[et] + ps[TILE_M + et] + bhead);
            }
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    if (warp == SP_GATHER_WARPS + SP_EPI_WARPS) umma::tmem_dealloc(tmem, 2 * HID);
}

static int num_sms() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

template <int TAPS>
static size_t fwd_smem(int K0, int app_dim, int groups) {
    return (size_t)HID * (K0 + 16) * 2 + HID * 4 + (size_t)groups * fwd_group_bytes<TAPS>(K0, app_dim);
}
template <int TAPS>
static size_t bwd_smem(int K0, bool dw) {
    const size_t KB = (size_t)K0 + 16;
    const size_t need = (size_t)BWD_EPI_WARPS * BWD_STAGE_BYTES + (size_t)HID * KB * 2 +
                        (size_t)TILE_M * (KB + (dw ? KB : K0)) * 2 * (dw ? 2 : 1) +
                        (2 * HID + TapTile<TAPS>::DF_FLOATS + TapTile<TAPS>::SPT * DH0_LD) * 4 + 48;
    return need > BWD_SMEM_FLOOR ? need : BWD_SMEM_FLOOR;
}

// The field's four kernels, in step order.  `which`: bit 0 the hash-grid gather,
// bit 1 the MLP forward, bit 2 the MLP backward, bit 3 the table-gradient scatter.
enum FieldKernels : int { FK_GATHER = 1, FK_MLP_FWD = 2, FK_MLP_BWD = 4, FK_SCATTER = 8 };

// TMA maps of the x0ext rows as the field MLP's A tiles (8-row groups in the core-matrix layout):
// features hi | tail (K0 + 16 columns), and features lo into a tile lo_cols wide (K0, or K0 + 16
// whose last two chunks lie past the tensor and arrive as zeros)
static int x0ext_maps(const FieldParams& p, int64_t rows, int lo_cols, CUtensorMap* hi, CUtensorMap* lo) {
    const int KX = 2 * p.K0 + 16;
    if (rows <= 0) rows = 1;                          // (no tile is loaded)
    if (int st = tensor_map_kmajor_groups(hi, p.x0ext, rows, (p.K0 + 16) / 8, KX, (p.K0 + 16) / 8, "x0ext hi"))
        return st;
    return tensor_map_kmajor_groups(lo, (const __half*)p.x0ext + p.K0 + 16, rows, p.K0 / 8, KX, lo_cols / 8,
                                    "x0ext lo");
}

template <int F, int TAPS, bool DET>
static void launch_scatter(int ns, unsigned blocks, const FieldParams& p, cudaStream_t s) {
    if (ns == 4) k_field_scatter<F, TAPS, DET, 4><<<blocks, SCATTER_THREADS, 0, s>>>(p);
    else if (ns == 2) k_field_scatter<F, TAPS, DET, 2><<<blocks, SCATTER_THREADS, 0, s>>>(p);
    else k_field_scatter<F, TAPS, DET, 1><<<blocks, SCATTER_THREADS, 0, s>>>(p);
}

template <int F, int TAPS>
static int launch_field(const FieldParams& p, int which, cudaStream_t s) {
    constexpr int EVALS = TapTile<TAPS>::EVALS, SPT = TapTile<TAPS>::SPT, TILE_ROWS = TapTile<TAPS>::ROWS;
    constexpr int LAST_BOX = TILE_ROWS - 96;          // rows of a tile's last 32-row lane quadrant
    const int64_t ntiles = (p.Ns + SPT - 1) / SPT;
    // largest thread index: gather ntiles * rows per tile * active, scatter Ns * active * 8
    const int64_t gather_items = ntiles * (SPT * EVALS) * (int64_t)p.active;
    const int64_t scatter_items = p.Ns * (int64_t)p.active * 8;
    if ((gather_items > scatter_items ? gather_items : scatter_items) >= ((int64_t)1 << 32)) {
        set_error("%lld samples x %d levels exceed the 32-bit index range of one launch", (long long)p.Ns,
                  p.active);
        return GBSDF_ERR_UNSUPPORTED;
    }
    if (which & FK_GATHER) {
        const int64_t items = ntiles * SPT * p.active;
        k_field_gather<F, TAPS><<<(unsigned)((items + GATHER_THREADS - 1) / GATHER_THREADS), GATHER_THREADS, 0, s>>>(
            p, ntiles);
        if (int st = launch_status("field gather")) return st;
    }
    if (which & FK_MLP_FWD) {
        constexpr size_t limit = 227 * 1024, per_sm = 228 * 1024, reserved = 1024;   // per CTA, per SM, per CTA resident
        const int app_cols = p.xc ? p.app_dim : 0;
        const size_t one = fwd_smem<TAPS>(p.K0, app_cols, 1);
        if (one > limit) {
            set_error("field forward needs %zu B of shared memory", one);
            return GBSDF_ERR_UNSUPPORTED;
        }
        // Two tiles in flight per SM: two CTAs where they fit, else (K0 > 80) one CTA of two groups
        // where that fits (with 4 taps' larger rings not K0 = 128 and more than 17 appearance columns).
        // p.fwd_ctas (a tuning choice): 1 keeps one tile in flight (0 = 2)
        const bool two = p.fwd_ctas != 1;
        const int groups = two && FWD_CTAS_PER_SM * (one + reserved) > per_sm && fwd_smem<TAPS>(p.K0, app_cols, 2) <= limit ? 2 : 1;
        const size_t smem = fwd_smem<TAPS>(p.K0, app_cols, groups);
        int64_t grid = num_sms() * (two && groups == 1 ? FWD_CTAS_PER_SM : 1);
        const int64_t need = (ntiles + groups - 1) / groups;
        if (grid > need) grid = need;
        const int KX = 2 * p.K0 + 16;
        CUtensorMap tm_x, tm_tail;
        if (int st = tensor_map_2d(&tm_x, false, p.x0ext, ntiles * TILE_ROWS, KX, KX, 64, TILE_M,
                                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, "x0ext"))
            return st;
        if (int st = tensor_map_kmajor_groups(&tm_tail, (const __half*)p.x0ext + p.K0, ntiles * TILE_ROWS, 2, KX, 2,
                                              "x0ext tail", TILE_M))
            return st;
        if (groups == 2) {
            allow_max_smem(k_field_fwd<F, TAPS, 2>);
            k_field_fwd<F, TAPS, 2><<<(unsigned)grid, 2 * FIELD_THREADS, smem, s>>>(p, tm_x, tm_tail);
        } else {
            allow_max_smem(k_field_fwd<F, TAPS, 1>);
            k_field_fwd<F, TAPS, 1><<<(unsigned)grid, FIELD_THREADS, smem, s>>>(p, tm_x, tm_tail);
        }
        if (int st = launch_status("field forward")) return st;
    }
    if (which & FK_MLP_BWD) {
        const bool dw = p.d_w0 != nullptr;
        const size_t smem = bwd_smem<TAPS>(p.K0, dw);
        if (smem > 227 * 1024) {
            set_error("field backward needs %zu B of shared memory", smem);
            return GBSDF_ERR_UNSUPPORTED;
        }
        // d_pre0 [rows, 256] fp16 (without d_w0) and d_enc [rows, K0] fp32 as TMA store targets
        // (rows = tiles x 126 or 125); with d_w0 the d_pre0 maps are never used and describe
        // d_enc's memory.  The '30' maps are the last lane quadrant's LAST_BOX-row boxes.
        const int64_t rows = ntiles * TILE_ROWS;
        if (rows >= ((int64_t)1 << 31)) {
            set_error("%lld backward rows exceed the TMA coordinate range", (long long)rows);
            return GBSDF_ERR_UNSUPPORTED;
        }
        CUtensorMap tm_pre32, tm_pre30, tm_enc32, tm_enc30, tm_plo32, tm_plo30;
        const CUtensorMapL2promotion l2n = CU_TENSOR_MAP_L2_PROMOTION_NONE;
        if (!dw) {
            if (int st = tensor_map_2d(&tm_pre32, false, p.d_pre0, rows, HID, HID, 64, 32,
                                       CU_TENSOR_MAP_SWIZZLE_128B, l2n, "d_pre0"))
                return st;
            if (int st = tensor_map_2d(&tm_pre30, false, p.d_pre0, rows, HID, HID, 64, LAST_BOX,
                                       CU_TENSOR_MAP_SWIZZLE_128B, l2n, "d_pre0"))
                return st;
        }
        if (int st = tensor_map_2d(&tm_enc32, true, p.d_enc, rows, p.K0, p.K0, 16, 32, CU_TENSOR_MAP_SWIZZLE_64B, l2n,
                                   "d_enc"))
            return st;
        if (int st = tensor_map_2d(&tm_enc30, true, p.d_enc, rows, p.K0, p.K0, 16, LAST_BOX, CU_TENSOR_MAP_SWIZZLE_64B, l2n,
                                   "d_enc"))
            return st;
        if (dw) tm_pre32 = tm_pre30 = tm_enc32;
        if (!dw && p.d_pre0_lo) {
            if (int st = tensor_map_2d(&tm_plo32, false, p.d_pre0_lo, rows, HID, HID, 64, 32,
                                       CU_TENSOR_MAP_SWIZZLE_128B, l2n, "d_pre0_lo"))
                return st;
            if (int st = tensor_map_2d(&tm_plo30, false, p.d_pre0_lo, rows, HID, HID, 64, LAST_BOX,
                                       CU_TENSOR_MAP_SWIZZLE_128B, l2n, "d_pre0_lo"))
                return st;
        } else {
            tm_plo32 = tm_plo30 = tm_pre32;              // unused
        }
        CUtensorMap tm_xhi, tm_xlo;
        if (int st = x0ext_maps(p, rows, dw ? p.K0 + 16 : p.K0, &tm_xhi, &tm_xlo)) return st;
        int64_t grid = num_sms();
        if (grid > ntiles) grid = ntiles;
        if (dw) {
            allow_max_smem(k_field_bwd<F, true, TAPS>);
            k_field_bwd<F, true, TAPS><<<(unsigned)grid, BWD_THREADS, smem, s>>>(p, tm_pre32, tm_pre30, tm_enc32, tm_enc30,
                                                                             tm_plo32, tm_plo30, tm_xhi, tm_xlo);
        } else {
            allow_max_smem(k_field_bwd<F, false, TAPS>);
            k_field_bwd<F, false, TAPS><<<(unsigned)grid, BWD_THREADS, smem, s>>>(p, tm_pre32, tm_pre30, tm_enc32, tm_enc30,
                                                                              tm_plo32, tm_plo30, tm_xhi, tm_xlo);
        }
        if (int st = launch_status("field backward")) return st;
    }
    if (which & FK_SCATTER) {
        constexpr int PARTS = F < 4 ? 1 : F / 4;
        // Samples per thread: four where that leaves two blocks' threads for every slot of the chip, fewer
        // for small batches (2048 samples x 8 levels: 6.3 us with one, 20.1 with four; 2.1 M x 8: 2.53 ms
        // with one, 2.31 with two, 2.09 with four, 2.21 with eight).
        // p.scatter_cpt (a tuning choice): 2, 4 or 8 for one, two or four samples per thread
        const int64_t slots = (int64_t)num_sms() * 3 * SCATTER_THREADS, lanes = p.Ns * p.active * PARTS;
        int ns = lanes >= 8 * slots ? 4 : lanes >= 4 * slots ? 2 : 1;
        if (p.scatter_cpt) ns = p.scatter_cpt / 2;
        const int64_t threads = (p.Ns + ns - 1) / ns * p.active * PARTS;
        const unsigned blocks = (unsigned)((threads + SCATTER_THREADS - 1) / SCATTER_THREADS);
        if (p.d_table_fix) {
            // deterministic mode: integer accumulation into the caller's buffer, then into d_table
            const int64_t n = (int64_t)p.grid.offset[p.grid.n_levels] * F;
            if (cudaMemsetAsync(p.d_table_fix, 0, (size_t)n * 8, s) != cudaSuccess) {
                set_error("clearing d_table_fix failed");
                return GBSDF_ERR_CUDA;
            }
            launch_scatter<F, TAPS, true>(ns, blocks, p, s);
            if (int st = launch_status("field scatter (deterministic)")) return st;
            k_fixed_to_table<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, p.d_table_fix, p.d_table);
        } else {
            launch_scatter<F, TAPS, false>(ns, blocks, p, s);
        }
        if (int st = launch_status("field scatter")) return st;
    }
    return GBSDF_OK;
}

static int check_field_weights(const FieldParams& p) {
    GBSDF_CHECK_ARG(p.active >= 1 && p.active <= p.grid.n_levels, "active levels %d", p.active);
    const int F = p.grid.n_features;
    GBSDF_CHECK_ARG(F == 2 || F == 4 || F == 8, "n_features %d unsupported by the fused field", F);
    GBSDF_CHECK_ARG(p.K0 % 16 == 0 && p.K0 >= p.active * F && p.K0 <= 128, "K0 %d", p.K0);
    GBSDF_CHECK_ARG(p.table && p.w0e && p.w0x && p.b0 && p.whead && p.bhead, "NULL weight pointer");
    GBSDF_CHECK_ARG(aligned(p.table, 16) && aligned(p.w0e, 16), "table / w0e alignment");
    return GBSDF_OK;
}

static int check_field(const FieldParams& p) {
    GBSDF_CHECK_ARG(p.Ns >= 0, "Ns < 0");
    GBSDF_CHECK_ARG(p.taps == 0 || p.taps == 4 || p.taps == 6, "taps %d (4 or 6; 0 means 6)", p.taps);
    GBSDF_CHECK_ARG(p.scatter_cpt == 0 || p.scatter_cpt == 2 || p.scatter_cpt == 4 || p.scatter_cpt == 8,
                    "scatter_cpt %d (2, 4 or 8; 0 = by size)", p.scatter_cpt);
    GBSDF_CHECK_ARG(p.fwd_ctas >= 0 && p.fwd_ctas <= 2, "fwd_ctas %d (1 or 2; 0 = 2)", p.fwd_ctas);
    if (int st = check_field_weights(p)) return st;
    GBSDF_CHECK_ARG(p.S > 0 || p.sample_ray, "need S > 0 or sample_ray");
    GBSDF_CHECK_ARG(p.center && p.ray_unit && p.dists, "NULL ray pointer");
    return GBSDF_OK;
}

}  // namespace gbsdf

using namespace gbsdf;

extern "C" size_t gbsdf_field_args_size(void) { return sizeof(gbsdf_field_args); }

template <int TAPS>
static int field_dispatch_taps(const FieldParams& p, int which, void* stream) {
    switch (p.grid.n_features) {
        case 2: return launch_field<2, TAPS>(p, which, as_stream(stream));
        case 4: return launch_field<4, TAPS>(p, which, as_stream(stream));
        default: return launch_field<8, TAPS>(p, which, as_stream(stream));
    }
}
static int field_dispatch(const FieldParams& p, int which, void* stream) {
    return p.taps == 4 ? field_dispatch_taps<4>(p, which, stream) : field_dispatch_taps<6>(p, which, stream);
}

static int check_fwd(const FieldParams& p, int which) {
    if (int st = check_field(p)) return st;
    GBSDF_CHECK_ARG(p.x0ext && aligned(p.x0ext, 16), "x0ext missing or misaligned (16 bytes: its rows are loaded by TMA)");
    if (which & FK_MLP_FWD) {
        GBSDF_CHECK_ARG(p.sdf && p.grad && p.hess && p.h0c, "NULL output");
        GBSDF_CHECK_ARG(p.w0b && aligned(p.w0b, 16), "w0b (fp16 [256, K0 + 16]) missing or misaligned");
        GBSDF_CHECK_ARG(p.ld_h0c == 0 || (p.ld_h0c >= HID && p.ld_h0c % 8 == 0), "ld_h0c %d", p.ld_h0c);
        GBSDF_CHECK_ARG(!p.xc || (p.ldxc % 16 == 0 && p.ldxc - HID >= 23 + p.app_dim && p.ldxc - HID <= 48),
                        "xc leading dimension %d (needs 256 + 23 + app_dim <= ldxc <= 304, multiple of 16)", p.ldxc);
        GBSDF_CHECK_ARG(!p.xc || p.app_dim == 0 || (p.app_table && p.app_idx), "appearance table / index missing");
        GBSDF_CHECK_ARG(!p.h0c_lo || aligned(p.h0c_lo, 16), "h0c_lo misaligned");
        GBSDF_CHECK_ARG(!p.xc_lo || (p.xc && aligned(p.xc_lo, 16)), "xc_lo needs xc and 16-byte alignment");
    }
    return GBSDF_OK;
}

static int check_bwd(const FieldParams& p, int which) {
    if (int st = check_field(p)) return st;
    GBSDF_CHECK_ARG(p.d_enc && aligned(p.d_enc, 16), "d_enc missing or misaligned");
    if (which & FK_MLP_BWD) {
        GBSDF_CHECK_ARG(p.w0b && aligned(p.w0b, 16), "w0b (fp16 [256, K0 + 16]) missing or misaligned");
        GBSDF_CHECK_ARG(p.grad && p.d_sdf && p.d_grad && p.d_hess && p.d_xc && p.d_h0c && p.x0ext && p.d_whead &&
                            p.d_bhead,
                        "NULL pointer");
        GBSDF_CHECK_ARG(p.d_w0 || (p.d_pre0 && aligned(p.d_pre0, 16)), "d_pre0 missing or misaligned (no d_w0)");
        GBSDF_CHECK_ARG(!p.d_w0 || p.K0 <= 64, "d_w0 needs K0 <= 64 (K0 %d): pass d_pre0 instead", p.K0);
        GBSDF_CHECK_ARG(aligned(p.d_h0c, 16), "d_h0c alignment");
        GBSDF_CHECK_ARG(!p.d_pre0_lo || aligned(p.d_pre0_lo, 16), "d_pre0_lo alignment");
        GBSDF_CHECK_ARG(aligned(p.x0ext, 16), "x0ext misaligned (16 bytes: its rows are loaded by TMA)");
    }
    if (which & FK_SCATTER) {
        GBSDF_CHECK_ARG(p.d_table && aligned(p.d_table, 16), "d_table missing or misaligned");
        GBSDF_CHECK_ARG(!p.d_table_fix || aligned(p.d_table_fix, 16), "d_table_fix misaligned");
    }
    return GBSDF_OK;
}

static int field_call(const gbsdf_field_args* params, int which, void* stream) {
    clear_error();
    GBSDF_CHECK_ARG(params != nullptr, "params NULL");
    const FieldParams& p = *params;
    const bool fwd = (which & (FK_GATHER | FK_MLP_FWD)) != 0;
    if (int st = fwd ? check_fwd(p, which) : check_bwd(p, which)) return st;
    if (p.Ns == 0) return GBSDF_OK;
    return field_dispatch(p, which, stream);
}

extern "C" int gbsdf_field_fwd(const gbsdf_field_args* params, void* stream) {
    return field_call(params, FK_GATHER | FK_MLP_FWD, stream);
}
extern "C" int gbsdf_field_bwd(const gbsdf_field_args* params, void* stream) {
    return field_call(params, FK_MLP_BWD | FK_SCATTER, stream);
}
extern "C" int gbsdf_field_encode(const gbsdf_field_args* params, void* stream) {
    return field_call(params, FK_GATHER, stream);
}
extern "C" int gbsdf_field_mlp_fwd(const gbsdf_field_args* params, void* stream) {
    return field_call(params, FK_MLP_FWD, stream);
}
extern "C" int gbsdf_field_mlp_bwd(const gbsdf_field_args* params, void* stream) {
    return field_call(params, FK_MLP_BWD, stream);
}
extern "C" int gbsdf_field_scatter(const gbsdf_field_args* params, void* stream) {
    return field_call(params, FK_SCATTER, stream);
}

extern "C" int gbsdf_field_workspace_size(int64_t Ns, int32_t K0, int32_t taps, int32_t deterministic,
                                          const gbsdf_grid* grid, gbsdf_field_workspace* out) {
    clear_error();
    GBSDF_CHECK_ARG(out != nullptr && Ns >= 0, "bad arguments");
    GBSDF_CHECK_ARG(K0 % 16 == 0 && K0 >= 16 && K0 <= 128, "K0 %d", K0);
    GBSDF_CHECK_ARG(taps == 0 || taps == 4 || taps == 6, "taps %d", taps);
    GBSDF_CHECK_ARG(!deterministic || grid != nullptr, "the deterministic scatter's size needs the grid");
    const int spt = taps == 4 ? TapTile<4>::SPT : TapTile<6>::SPT;
    const int rows_per_tile = taps == 4 ? TapTile<4>::ROWS : TapTile<6>::ROWS;
    const int64_t rows = (Ns + spt - 1) / spt * rows_per_tile;
    out->rows = rows;
    out->x0ext_bytes = (size_t)rows * (2 * K0 + 16) * 2;
    out->d_enc_bytes = (size_t)rows * K0 * 4;
    out->d_w0_bytes = K0 <= 64 ? (size_t)HID * (K0 + 16) * 4 : 0;
    out->d_pre0_bytes = K0 > 64 ? (size_t)rows * HID * 2 : 0;
    out->d_table_fix_bytes = deterministic ? (size_t)grid->offset[grid->n_levels] * grid->n_features * 8 : 0;
    return GBSDF_OK;
}

int gbsdf::sdf_points_run(const gbsdf_field_args* params, int64_t M, const float* pts, const float* ax, const float* ay,
                          const float* az, int nx, int ny, int nz, float sign, float* out, int inner, int ld,
                          cudaStream_t s) {
    GBSDF_CHECK_ARG(params != nullptr && out != nullptr, "NULL pointer");
    const FieldParams& p = *params;
    if (int st = check_field_weights(p)) return st;
    GBSDF_CHECK_ARG(M >= 0, "M < 0");
    if (M == 0) return GBSDF_OK;
    SdfPointsArgs q;
    q.M = M; q.pts = pts; q.ax = ax; q.ay = ay; q.az = az; q.nx = nx; q.ny = ny; q.nz = nz; q.sign = sign; q.out = out;
    q.inner = inner; q.ld = ld;
    if (!pts) {
        GBSDF_CHECK_ARG(ax && ay && az && nx > 0 && ny > 0 && nz > 0 && (int64_t)nx * ny * nz == M,
                        "lattice mode needs axes with nx*ny*nz == M");
    }
    const size_t smem = sdf_points_smem(p.K0);
    GBSDF_CHECK_ARG(smem <= 227 * 1024, "K0 too large");
    const int64_t ntiles = (M + TILE_M - 1) / TILE_M;
    int64_t grid = num_sms();
    if (grid > ntiles) grid = ntiles;
    switch (p.grid.n_features) {
        case 2:
            allow_max_smem(k_sdf_points<2>);
            k_sdf_points<2><<<(unsigned)grid, SP_TPB, smem, s>>>(p, q);
            break;
        case 4:
            allow_max_smem(k_sdf_points<4>);
            k_sdf_points<4><<<(unsigned)grid, SP_TPB, smem, s>>>(p, q);
            break;
        default:
            allow_max_smem(k_sdf_points<8>);
            k_sdf_points<8><<<(unsigned)grid, SP_TPB, smem, s>>>(p, q);
            break;
    }
    return launch_status("sdf_points");
}

extern "C" int gbsdf_sdf_points(const gbsdf_field_args* params, int64_t M, const float* pts, const float* ax,
                                const float* ay, const float* az, int nx, int ny, int nz, float sign, float* out,
                                void* stream) {
    clear_error();
    return sdf_points_run(params, M, pts, ax, ay, az, nx, ny, nz, sign, out, 0, 0, as_stream(stream));
}
