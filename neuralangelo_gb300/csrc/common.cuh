// Shared device helpers for the gbsdf kernels (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "../../include/gbsdf.h"

namespace gbsdf {

// ---------------------------------------------------------------------------
// error reporting (thread-local message, defined in capi.cu)
void set_error(const char* fmt, ...);
void clear_error();

#define GBSDF_CHECK_ARG(cond, ...)            \
    do {                                      \
        if (!(cond)) {                        \
            ::gbsdf::set_error(__VA_ARGS__);  \
            return GBSDF_ERR_ARG;             \
        }                                     \
    } while (0)

int launch_status(const char* what);   // checks cudaGetLastError after a launch

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// gbsdf_sdf_points with the values in rows of `inner`, `ld` floats apart (inner 0: contiguous); field.cu
int sdf_points_run(const gbsdf_field_args* params, int64_t M, const float* pts, const float* ax, const float* ay,
                   const float* az, int nx, int ny, int nz, float sign, float* out, int inner, int ld, cudaStream_t s);

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// Lets kernel k take up to the device's opt-in maximum of dynamic shared memory per
// block.  Always the same ceiling, never the current launch's size: a per-launch value
// would leave the attribute at the last launch's size, below what an earlier launch of
// the same kernel recorded in a CUDA graph asks for when that node is launched on its
// own (as a profiler does with graph nodes).
template <typename Kernel>
inline void allow_max_smem(Kernel k) {
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
}

// ---------------------------------------------------------------------------
// hash-grid level arithmetic, shared by every kernel that evaluates the field.
// Follows tiny-cuda-nn's HashGrid (the encoder behind modules.py:42-50):
// position p = fma(scale, x, 0.5); corner = floor(p); frac = p - corner; the
// corner index is dense (x + y*res + z*res^2) or the XOR prime hash, modulo the
// level size.  The per-level scale arrives precomputed in gbsdf_grid.scale.

struct LevelDesc {
    float scale;
    uint32_t res;
    uint32_t size;
    uint32_t hashed;
    uint64_t offset;
};

__device__ __forceinline__ LevelDesc level_desc(const gbsdf_grid& g, int l) {
    LevelDesc d;
    d.scale = g.scale[l];
    d.res = g.resolution[l];
    d.size = g.size[l];
    d.hashed = g.hashed[l];
    d.offset = g.offset[l];
    return d;
}

__device__ __forceinline__ void grid_pos(float scale, float x, uint32_t& base, float& frac) {
    const float p = __fmaf_rn(scale, x, 0.5f);
    const float f = floorf(p);
    base = (uint32_t)(int)f;
    frac = __fsub_rn(p, f);
}

// Same result as idx % size without a division in the common cases: a hashed
// level's size is the power of two 2^log2_hashmap_size (it is hashed exactly when
// res^3 exceeds that), and a dense index of an in-range corner is already below
// the level size (size >= res^3).
__device__ __forceinline__ uint32_t grid_index(const LevelDesc& d, uint32_t cx, uint32_t cy, uint32_t cz) {
    if (d.hashed) {
        const uint32_t idx = (cx * 1u) ^ (cy * 2654435761u) ^ (cz * 805459861u);
        return (d.size & (d.size - 1u)) == 0u ? (idx & (d.size - 1u)) : idx % d.size;
    }
    const uint32_t idx = cx + cy * d.res + cz * (d.res * d.res);
    return idx < d.size ? idx : idx % d.size;
}

// Corner c (0..7) selects +1 in dimension d when bit d of c is set.
__device__ __forceinline__ float corner_weight(int c, float fx, float fy, float fz) {
    const float wx = (c & 1) ? fx : __fsub_rn(1.0f, fx);
    const float wy = (c & 2) ? fy : __fsub_rn(1.0f, fy);
    const float wz = (c & 4) ? fz : __fsub_rn(1.0f, fz);
    return __fmul_rn(__fmul_rn(wx, wy), wz);
}

// Normalisation of a world point into the grid's unit cube, as NeuralSDF.encode
// does it (modules.py:82-83): (p - vmin) / (vmax - vmin) with range [-2, 2].
__device__ __forceinline__ float to_unit(float p) { return __fmul_rn(__fadd_rn(p, 2.0f), 0.25f); }

// ---------------------------------------------------------------------------
// numerics shared with the reference's activations

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }

// MUFU approximations with subnormals flushed to zero (PTX ex2/lg2/rcp .approx.ftz):
// the fused FP16 path's activations never need subnormal precision, and the flushing
// forms take no range fix-ups around the MUFU op.
__device__ __forceinline__ float ex2_ftz(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_ftz(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_ftz(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Fast-path softplus(beta) and its derivative for the fused FP16 kernels, from one
// exponential by change of base (e^x = 2^(x log2 e), ln y = log2(y) ln 2):
// t = beta z log2(e), e = 2^t, softplus = log2(1 + e) ln(2) / beta, d/dz = e / (1 + e).
// Above torch's threshold (beta z > 20) softplus is z; t is capped at 64 so that e
// stays finite there (and d/dz rounds to 1).  Checked against torch's softplus (CUDA's
// expf / log1pf) to 1e-5 relative, with a ~2e-8 absolute floor where 1 + e is near 1.
struct SoftplusK {
    float c1;      // beta log2(e)
    float c2;      // ln(2) / beta
    float tthr;    // 20 log2(e): the threshold in units of t
};
__device__ __forceinline__ SoftplusK softplus_k(float beta) {
    SoftplusK k;
    k.c1 = beta * 1.4426950408889634f;
    k.c2 = 0.6931471805599453f / beta;
    k.tthr = 20.0f * 1.4426950408889634f;
    return k;
}
__device__ __forceinline__ float softplus_fast_h(float z, const SoftplusK& k) {
    const float t = fminf(z * k.c1, 64.0f);
    const float hl = lg2_ftz(1.0f + ex2_ftz(t)) * k.c2;
    return t > k.tthr ? z : hl;
}

// Two float32 values in one register pair.  The packed operations round each as the single one does and
// take half the issue slots.
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t sub_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float sum_f32x2(uint64_t v) {
    float a, b;
    unpack_f32x2(v, a, b);
    return a + b;
}

// softplus and its derivative, or softplus alone, of a pair; softplus as softplus_fast_h, value by value
__device__ __forceinline__ void softplus_fast2(uint64_t z, const SoftplusK& k, uint64_t& h, uint64_t& dh) {
    float z0, z1, t0, t1, o0, o1, h0, h1;
    unpack_f32x2(z, z0, z1);
    unpack_f32x2(mul_f32x2(z, pack_f32x2(k.c1, k.c1)), t0, t1);
    t0 = fminf(t0, 64.0f);
    t1 = fminf(t1, 64.0f);
    const uint64_t e = pack_f32x2(ex2_ftz(t0), ex2_ftz(t1)), one_e = add_f32x2(pack_f32x2(1.0f, 1.0f), e);
    unpack_f32x2(one_e, o0, o1);
    dh = mul_f32x2(e, pack_f32x2(rcp_ftz(o0), rcp_ftz(o1)));
    unpack_f32x2(mul_f32x2(pack_f32x2(lg2_ftz(o0), lg2_ftz(o1)), pack_f32x2(k.c2, k.c2)), h0, h1);
    h = pack_f32x2(t0 > k.tthr ? z0 : h0, t1 > k.tthr ? z1 : h1);
}
__device__ __forceinline__ uint64_t softplus_fast_h2(uint64_t z, const SoftplusK& k) {
    float z0, z1, t0, t1, o0, o1, h0, h1;
    unpack_f32x2(z, z0, z1);
    unpack_f32x2(mul_f32x2(z, pack_f32x2(k.c1, k.c1)), t0, t1);
    t0 = fminf(t0, 64.0f);
    t1 = fminf(t1, 64.0f);
    unpack_f32x2(add_f32x2(pack_f32x2(1.0f, 1.0f), pack_f32x2(ex2_ftz(t0), ex2_ftz(t1))), o0, o1);
    unpack_f32x2(mul_f32x2(pack_f32x2(lg2_ftz(o0), lg2_ftz(o1)), pack_f32x2(k.c2, k.c2)), h0, h1);
    return pack_f32x2(t0 > k.tthr ? z0 : h0, t1 > k.tthr ? z1 : h1);
}

// Column sums of a 32 x 16 block held one row per lane (v[j] = element (lane, j)):
// four halving exchanges leave lane L with column L % 16 summed over the 16 lanes
// that share L's bit 4; one more exchange adds the other half.  Lanes L and L + 16
// both return the sum of column L % 16 (15 + 1 shuffles).
__device__ __forceinline__ float warp_column_sum16(float* v, int lane) {
#pragma unroll
    for (int h = 8; h >= 1; h >>= 1) {
        const bool upper = (lane & h) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float send = upper ? v[i] : v[i + h];
            const float keep = upper ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}

// Adds v into row `entry` (8 floats, 16-byte aligned) of table for every lane with `on`; the whole
// warp calls.  Neighbouring lanes trade halves first, so that each of the two vector atomics
// covers whole 32-byte rows of every other lane: with one row per lane in both, each touched 32 half
// sectors, twice the requests at L1 and L2.
__device__ __forceinline__ void scatter_add_rows8(float* table, uint64_t entry, bool on, const float* v, int lane) {
    const bool odd = lane & 1;
    float a[4], b[4];                       // this lane's half of the even and of the odd lane's row
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float got = __shfl_xor_sync(0xffffffffu, odd ? v[k] : v[4 + k], 1);
        a[k] = odd ? got : v[k];
        b[k] = odd ? v[4 + k] : got;
    }
    const uint64_t other = __shfl_xor_sync(0xffffffffu, (unsigned long long)entry, 1);
    const unsigned both = __ballot_sync(0xffffffffu, on);
    float* half = table + (odd ? 4 : 0);
    if ((both >> (lane & ~1)) & 1u)
        atomicAdd(reinterpret_cast<float4*>(half + (odd ? other : entry) * 8), make_float4(a[0], a[1], a[2], a[3]));
    if ((both >> (lane | 1)) & 1u)
        atomicAdd(reinterpret_cast<float4*>(half + (odd ? entry : other) * 8), make_float4(b[0], b[1], b[2], b[3]));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace gbsdf
