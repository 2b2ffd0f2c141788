// A chain of dense layers on tcgen05, each layer's output fed to the next one on chip:
//     y_l = epi_l([y_{l-1} | in_l] W_l^T + b_l),     y as an fp16 hi + lo pair between layers.
// The forward of the SDF feature layer and the colour MLP (projects/neuralangelo/utils/mlp.py:55-69,
// projects/neuralangelo/utils/modules.py:199-220 via projects/nerf/utils/nerf_util.py:158-196) and
// of the background NeRF's feature MLP and colour layer (modules.py:268-284): every layer's hi half
// that the backward reads goes to global memory, the pair itself stays in tensor memory.
//
// One persistent CTA per SM takes 128 rows through all layers.  TMEM is two regions of 256
// columns: layer g accumulates in region g & 1 while it reads its A operand, the pair of the layer
// before, from the other; the epilogue writes the pair over the accumulator in place (16 units: hi
// in 8 columns, lo in the next 8), which makes that region the next layer's A.
//   warps 0-15   epilogue: four warps per TMEM lane quadrant; output columns 0-127 while the MMAs of
//                columns 128-255 run, then those; outputs leave afterwards, under the next layer's
//                MMAs (through 2 KB per warp, as 64-byte row pieces);
//   warp 16      MMAs: per half of 128 output columns all lo products before the hi products (small
//                addends keep their bits in FP32), in column order, as k_dense issues them; the lo
//                products of the columns whose pair is ready go out for both halves while the
//                epilogue converts the rest;
//   warp 17      weights in 16 KB units (128 rows x 64 columns, 128-byte swizzle): a half's four in one
//                slot, two slots: a half's slot is free for the next layer while the other half
//                runs, which covers the L2 latency (the first layer's slots hold two chunks of both
//                halves instead); units of appended columns in a slot of their own, once per pass;
//   warp 18      inputs from global memory (the first layer's, and columns appended at later
//                layers, those once per half): chunks [128 x 64] of the lo, then the hi half, in a
//                ring of three, the next tile's requested into L2 a tile ahead.
// One barrier wait per 64 KB and straight runs of MMAs from warp-uniform descriptors: with a wait and a
// descriptor per 16 KB unit, computed by a lone lane, the MMA warp's own instructions took longer
// than its MMAs (4.1 ms where this takes 2.7).
// Layer by layer through k_dense, each layer read and wrote both halves: 2 KB per row and layer of
// 256 against 0.5 KB written here.  2.1 M rows, feature layer and four colour layers: 4.50 ms
// there, 2.67 ms here; 6.3 M object and 1.6 M background rows of a view (no outputs kept but the
// last): 19.3 and 10.1 ms.
// Bound: the weights' way from L2.  Every tile streams all layers' weights (670 KB for those five)
// and the SMs draw about 26 bytes a clock each when all of them do; the MMAs alone would take
// half as long.
// Every wait is bounded; a timed-out wait sets *err and the roles leave their loops.
#include <type_traits>

#include "dense.cuh"
#include "tma.cuh"

namespace gbsdf {
namespace {

constexpr int MC_EPI_WARPS = 16;
constexpr int MC_THREADS = (MC_EPI_WARPS + 3) * 32;
constexpr int MC_KCH = 64;                              // columns per chunk
constexpr uint32_t MC_NW = 2, MC_NT = 1, MC_NA = 3;      // slots: weights, appended weight units, input chunks
constexpr uint32_t MC_UNIT = 128 * 128, MC_W_BYTES = 4 * MC_UNIT, MC_A_BYTES = TILE_M * 128;
constexpr int MC_MAX_FIRST = 256, MC_MAX_TAIL = 128;    // input columns of the first and of a later layer
constexpr uint32_t MC_STAGE = 2048;                     // per epilogue warp: 32 rows x 32 columns
struct ChainLayer {
    int k_chain, k_in, n, epi;       // columns from the layer before, from global memory; width; activation
    int ld_out;
    __half *out, *out_lo;            // where the hi / lo halves go, or NULL
    const float* bias;
};
constexpr size_t MC_SMEM = MC_NW * (size_t)MC_W_BYTES + MC_NT * (size_t)MC_UNIT + MC_NA * (size_t)MC_A_BYTES +
                           MC_EPI_WARPS * MC_STAGE + 2 * 256 * 4 + (2 * (MC_NW + MC_NT + MC_NA) + 4) * 8 + 16 + GBSDF_MLP_MAX_LAYERS * sizeof(ChainLayer);
static_assert(MC_SMEM <= 227 * 1024, "one CTA's shared memory");

struct ChainParams {
    ChainLayer layer[GBSDF_MLP_MAX_LAYERS];
    int n_layers;
    int64_t M;
    float beta;
    int* err;
};
struct ChainMaps {
    CUtensorMap w[GBSDF_MLP_MAX_LAYERS], in[GBSDF_MLP_MAX_LAYERS], in_lo[GBSDF_MLP_MAX_LAYERS];
};

__device__ __forceinline__ int chain_chunks(int k) { return (k + MC_KCH - 1) / MC_KCH; }

__global__ void __launch_bounds__(MC_THREADS, 1) k_mlp_chain(const __grid_constant__ ChainMaps maps,
                                                             const __grid_constant__ ChainParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* w_s = smem;                                              // [MC_NW][4 units][128 x 64]
    uint8_t* t_s = w_s + MC_NW * MC_W_BYTES;                          // [MC_NT][128 x 64]
    uint8_t* a_s = t_s + MC_NT * MC_UNIT;                             // [MC_NA][128 x 64]
    uint8_t* stage_s = a_s + MC_NA * MC_A_BYTES;                      // [16][32 x 32]
    float* bias_s = reinterpret_cast<float*>(stage_s + MC_EPI_WARPS * MC_STAGE);   // [2][256]
    uint64_t* wfull = reinterpret_cast<uint64_t*>(bias_s + 2 * 256);
    uint64_t* wempty = wfull + MC_NW;
    uint64_t* tfull = wempty + MC_NW;
    uint64_t* tempty = tfull + MC_NT;
    uint64_t* afull = tempty + MC_NT;
    uint64_t* aempty = afull + MC_NA;
    uint64_t* dfull = aempty + MC_NA;                                 // [2] accumulator columns 0-127 / 128-255 complete
    uint64_t* half_done = dfull + 2;                                  // [2] columns 0-127 / 128-255 read, and the next A
    uint32_t* tslot = reinterpret_cast<uint32_t*>(half_done + 2);
    // the layer table in shared memory: the roles index it per layer, and the parameters' constant bank
    // is larger than the constant cache
    ChainLayer* layer_s = reinterpret_cast<ChainLayer*>(tslot + 4);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid >= 64 && tid < 64 + p.n_layers) layer_s[tid - 64] = p.layer[tid - 64];
    if (tid == 0) {
        for (uint64_t* bar = wfull; bar < dfull; ++bar) umma::mbar_init(bar, 1);
        umma::mbar_init(&dfull[0], 1);
        umma::mbar_init(&dfull[1], 1);
        umma::mbar_init(&half_done[0], MC_EPI_WARPS);
        umma::mbar_init(&half_done[1], MC_EPI_WARPS);
        umma::fence_mbar_init();
    }
    if (warp == MC_EPI_WARPS) {
        umma::tmem_alloc(tslot, 512);
        umma::tmem_relinquish();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = *tslot;
    const int64_t ntiles = (p.M + TILE_M - 1) / TILE_M;
    const int L = p.n_layers;

    if (warp == MC_EPI_WARPS + 1) {
        // ---------------- weights ----------------
        if (lane == 0) {
            uint32_t n = 0, nt = 0;
            bool ok = true;
            for (int64_t t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
                for (int l = 0; l < L && ok; ++l) {
                    const ChainLayer y = layer_s[l];
                    const int halves = y.n >> 7, main = chain_chunks(y.k_chain), nin = chain_chunks(y.k_in);
                    const int slots = l == 0 ? (nin + 1) / 2 : halves;
                    for (int j = 0; j < slots && ok; ++j, ++n) {
                        const uint32_t slot = n % MC_NW, use = n / MC_NW;
                        if (use > 0) ok = umma::mbar_wait(&wempty[slot], (use - 1) & 1u);
                        if (!ok) break;
                        // first layer: chunks 2j and 2j + 1 of every half; later: half j
                        const int units = l == 0 ? min(nin - 2 * j, 2) * halves : main;
                        umma::mbar_arrive_expect_tx(&wfull[slot], (uint32_t)units * MC_UNIT);
                        for (int u = 0; u < units; ++u) {
                            const int c = l == 0 ? 2 * j + u / halves : u, h = l == 0 ? u % halves : j;
                            umma::tma_load_2d(w_s + slot * MC_W_BYTES + u * MC_UNIT, &maps.w[l], c * MC_KCH, h * 128,
                                              &wfull[slot]);
                        }
                    }
                    if (l == 0) continue;
                    for (int i = 0; i < 2 * nin * halves && ok; ++i, ++nt) {          // half, pass, chunk
                        const uint32_t ts = nt % MC_NT, tu = nt / MC_NT;
                        if (tu > 0) ok = umma::mbar_wait(&tempty[ts], (tu - 1) & 1u);
                        if (!ok) break;
                        umma::mbar_arrive_expect_tx(&tfull[ts], MC_UNIT);
                        umma::tma_load_2d(t_s + ts * MC_UNIT, &maps.w[l], (main + i % nin) * MC_KCH, i / (2 * nin) * 128,
                                          &tfull[ts]);
                    }
                }
            if (!ok) flag_timeout(p.err, 1);
        }
        __syncwarp();
    } else if (warp == MC_EPI_WARPS + 2) {
        // ---------------- inputs ----------------
        if (lane == 0) {
            uint32_t n = 0;
            bool ok = true;
            for (int64_t t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
                for (int l = 0; l < L && ok; ++l) {
                    const ChainLayer y = layer_s[l];
                    const int nc = chain_chunks(y.k_in), reps = l == 0 ? 1 : y.n >> 7;
                    for (int i = 0; i < 2 * nc * reps; ++i, ++n) {
                        const uint32_t slot = n % MC_NA, use = n / MC_NA;
                        if (use > 0 && !umma::mbar_wait(&aempty[slot], (use - 1) & 1u)) {
                            ok = false;
                            break;
                        }
                        umma::mbar_arrive_expect_tx(&afull[slot], MC_A_BYTES);
                        umma::tma_load_2d(a_s + slot * MC_A_BYTES, i % (2 * nc) < nc ? &maps.in_lo[l] : &maps.in[l],
                                          (i % nc) * MC_KCH, (int)(t * TILE_M), &afull[slot]);
                    }
                    // the next tile's into L2
                    if (l == 0 && t + gridDim.x < ntiles)
                        for (int i = 0; i < 2 * nc; ++i)
                            umma::tma_prefetch_2d(i < nc ? &maps.in_lo[0] : &maps.in[0], (i % nc) * MC_KCH,
                                                  (int)((t + gridDim.x) * TILE_M));
                }
            if (!ok) flag_timeout(p.err, 1);
        }
        __syncwarp();
    } else if (warp == MC_EPI_WARPS) {
        // ---------------- MMA issue ----------------
        // The whole warp walks the layers and waits; one elected lane issues.  Slots, addresses and
        // descriptors are warp-uniform that way.
        const bool leader = umma::elect_one();
        const uint64_t w_desc = umma::make_desc_sw128(umma::smem_u32(w_s)), t_desc = umma::make_desc_sw128(umma::smem_u32(t_s));
        const uint64_t a_desc = umma::make_desc_sw128(umma::smem_u32(a_s));
        const uint32_t idesc = umma::idesc_f16(TILE_M, 128);
        // (one lane polls: 32 lanes' polls of one barrier are served one after another, some 300 clocks a wait)
        auto wait = [&](uint64_t* bar, uint32_t phase) {
            return __any_sync(0xffffffffu, lane == 0 && umma::mbar_wait(bar, phase & 1u)) != 0;
        };
        // NCH chunks of the pair (at: its hi or lo columns) against consecutive units of a weight slot
        auto mma_pair = [&](auto nch, uint32_t dst, uint32_t at, uint64_t bd, uint32_t acc) {
            if (leader) {
#pragma unroll
                for (int i = 0; i < 4 * decltype(nch)::value; ++i)
                    umma::mma_f16_ta(dst, at + 16u * i, bd + (uint64_t)((i >> 2) * (MC_UNIT >> 4) + 2 * (i & 3)), idesc,
                                     i > 0 ? 1u : acc);
            }
        };
        // one chunk of inputs (up to four K = 16 steps)
        auto mma_in = [&](uint32_t dst, uint64_t ad, uint64_t bd, int steps, uint32_t acc) {
            if (leader) {
                umma::mma_f16(dst, ad, bd, idesc, acc);
                if (steps > 1) umma::mma_f16(dst, ad + 2, bd + 2, idesc, 1u);
                if (steps > 2) umma::mma_f16(dst, ad + 4, bd + 4, idesc, 1u);
                if (steps > 3) umma::mma_f16(dst, ad + 6, bd + 6, idesc, 1u);
            }
        };
        constexpr std::integral_constant<int, 2> two{};
        constexpr std::integral_constant<int, 4> four{};
        uint32_t g = 0, nw = 0, nt = 0, na = 0;                  // layers, weight halves, appended units, input chunks so far
        uint32_t nh0 = 0, nh1 = 0, nd0 = 0, nd1 = 0;             // phases of half_done and dfull so far
        bool ok = true;
        for (int64_t t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
            for (int l = 0; l < L && ok; ++l, ++g) {
                const ChainLayer y = layer_s[l];
                const int k_in = y.k_in, nin = chain_chunks(k_in), halves = y.n >> 7;
                const bool wide = y.k_chain == 256;
                const uint32_t d = tmem + (g & 1u) * 256u, a = tmem + ((g + 1u) & 1u) * 256u;
                // this layer's accumulator is the region that the layer before has been reading
                if (nd0 > 0) ok = wait(&dfull[0], nd0 - 1);
                if (nd1 > 0 && ok) ok = wait(&dfull[1], nd1 - 1);
                if (ok && l == 0) {
                    // every chunk of the inputs against both halves, lo pass, then hi pass
                    for (int i = 0; i < 2 * nin && ok; ++i, ++na) {
                        const uint32_t as = na % MC_NA;
                        const int c = i < nin ? i : i - nin, steps = min(k_in - c * MC_KCH, MC_KCH) / 16;
                        const uint32_t ws = (nw + (uint32_t)(c >> 1)) % MC_NW;
                        if (i < nin && (c & 1) == 0) ok = wait(&wfull[ws], (nw + (uint32_t)(c >> 1)) / MC_NW);
                        if (ok) ok = wait(&afull[as], na / MC_NA);
                        if (!ok) break;
                        umma::fence_after_sync();
                        for (int h = 0; h < halves; ++h)
                            mma_in(d + 128u * h, a_desc + as * (MC_A_BYTES >> 4),
                                   w_desc + ws * (MC_W_BYTES >> 4) + (uint32_t)((c & 1) * halves + h) * (MC_UNIT >> 4), steps,
                                   i > 0 ? 1u : 0u);
                        if (leader) {
                            umma::mma_commit(&aempty[as]);
                            if (i >= nin && ((c & 1) == 1 || c + 1 == nin)) umma::mma_commit(&wempty[ws]);
                        }
                        __syncwarp();
                    }
                    // a tile's first layer depends on nothing of the epilogue's: hold its completion back until
                    // every warp has seen the last layer's (their phase must not run two ahead)
                    if (ok && g > 0) {
                        ok = wait(&half_done[0], nh0++);
                        if (ok && layer_s[L - 1].n == 256) ok = wait(&half_done[1], nh1++);
                    }
                    if (!ok) break;
                    for (int h = 0; h < halves; ++h)
                        if (leader) umma::mma_commit(&dfull[h]);
                } else if (ok) {
                    // lo products of the first 128 columns for both halves, while the epilogue converts the others
                    ok = wait(&half_done[0], nh0++);
                    for (int h = 0; h < halves && ok; ++h) {
                        const uint32_t ws = (nw + h) % MC_NW;
                        ok = wait(&wfull[ws], (nw + h) / MC_NW);
                        if (!ok) break;
                        umma::fence_after_sync();
                        mma_pair(two, d + 128u * h, a + 8u, w_desc + ws * (MC_W_BYTES >> 4), 0u);
                        __syncwarp();
                    }
                    if (ok && wide) {
                        ok = wait(&half_done[1], nh1++);
                        umma::fence_after_sync();
                    }
                    for (int h = 0; h < halves && ok; ++h) {
                        const uint32_t ws = (nw + h) % MC_NW, dst = d + 128u * h;
                        const uint64_t bd = w_desc + ws * (MC_W_BYTES >> 4);
                        if (wide) mma_pair(two, dst, a + 128u + 8u, bd + 2 * (MC_UNIT >> 4), 1u);
                        for (int pass = 0; pass < 2 && ok; ++pass) {
                            if (pass == 1) {
                                if (wide) mma_pair(four, dst, a, bd, 1u);
                                else mma_pair(two, dst, a, bd, 1u);
                            }
                            for (int c = 0; c < nin && ok; ++c, ++na, ++nt) {    // the appended columns
                                const uint32_t as = na % MC_NA, ts = nt % MC_NT;
                                ok = wait(&afull[as], na / MC_NA);
                                if (ok) ok = wait(&tfull[ts], nt / MC_NT);
                                if (!ok) break;
                                umma::fence_after_sync();
                                mma_in(dst, a_desc + as * (MC_A_BYTES >> 4), t_desc + ts * (MC_UNIT >> 4),
                                       min(k_in - c * MC_KCH, MC_KCH) / 16, 1u);
                                if (leader) {
                                    umma::mma_commit(&aempty[as]);
                                    umma::mma_commit(&tempty[ts]);
                                }
                                __syncwarp();
                            }
                        }
                        if (!ok) break;
                        if (leader) {
                            umma::mma_commit(&wempty[ws]);
                            umma::mma_commit(&dfull[h]);
                        }
                        __syncwarp();
                    }
                }
                if (!ok) break;
                __syncwarp();
                ++nd0;
                if (halves == 2) ++nd1;
                nw += (uint32_t)(l == 0 ? (nin + 1) / 2 : halves);
            }
        if (!ok && leader) flag_timeout(p.err, 1);
        __syncwarp();
    } else {
        // ---------------- epilogue ----------------
        const SoftplusK spk = softplus_k(p.beta);
        const int q = warp & 3, part = warp >> 2;
        uint8_t* stg = stage_s + warp * MC_STAGE;
        uint32_t g = 0, nd0 = 0, nd1 = 0;                        // layers and dfull phases so far
        bool ok = true;
        for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
            const int64_t row0 = t * TILE_M + q * 32;
            // 32 columns (16 packed registers) of this warp's 32 rows, turned over in shared memory so that
            // four lanes write 64 contiguous bytes of a row; 16-byte unit u of row r sits at u ^ (r >> 1 & 3)
            auto store32 = [&](__half* dst, int ld, int col, const uint32_t* r) {
                __syncwarp();                                  // the previous block has been read
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    *reinterpret_cast<uint4*>(stg + lane * 64 + ((u ^ ((lane >> 1) & 3)) * 16)) =
                        make_uint4(r[4 * u], r[4 * u + 1], r[4 * u + 2], r[4 * u + 3]);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int rr = 8 * i + (lane >> 2), u = lane & 3;
                    const uint4 w = *reinterpret_cast<const uint4*>(stg + rr * 64 + ((u ^ ((rr >> 1) & 3)) * 16));
                    if (row0 + rr < p.M) *reinterpret_cast<uint4*>(dst + (row0 + rr) * ld + col + 8 * u) = w;
                }
            };
            for (int l = 0; l < L && ok; ++l, ++g) {
                const ChainLayer y = layer_s[l];
                const int halves = y.n >> 7;
                const bool last = l + 1 == L;
                // this warp's biases (the four warps of a part write the same values; the buffer's last
                // readers are two layers back, and a tile starts behind a barrier)
                float* bs = bias_s + (g & 1u) * 256u + part * 32;
                for (int h = 0; h < halves; ++h) bs[h * 128 + lane] = y.bias ? __ldg(y.bias + h * 128 + part * 32 + lane) : 0.0f;
                __syncwarp();
                uint32_t hi[2][16];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (h >= halves) break;
                    {
                        const uint32_t phase = (h == 0 ? nd0++ : nd1++) & 1u;
                        ok = __any_sync(0xffffffffu, lane == 0 && umma::mbar_wait(&dfull[h], phase)) != 0;
                    }
                    if (!ok) break;
                    umma::fence_after_sync();
                    const uint32_t c0 = (uint32_t)(h * 128 + part * 32), ta = umma::taddr(tmem, q * 32, (g & 1u) * 256u + c0);
                    float v[32];
                    umma::tmem_ld32(ta, v);
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 b = *reinterpret_cast<const float4*>(bs + h * 128 + j);
                        v[j] += b.x; v[j + 1] += b.y; v[j + 2] += b.z; v[j + 3] += b.w;
                    }
                    if (y.epi == 2) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = softplus_fast_h(v[j], spk);
                    } else if (y.epi == 1) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.0f);
                    }
                    uint32_t lo[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const __half2 h2 = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
                        const float2 b = __half22float2(h2);
                        const __half2 l2 = __floats2half2_rn(v[2 * i] - b.x, v[2 * i + 1] - b.y);
                        hi[h][i] = *reinterpret_cast<const uint32_t*>(&h2);
                        lo[i] = *reinterpret_cast<const uint32_t*>(&l2);
                    }
                    if (!last) {
                        umma::tmem_st8(ta, hi[h]);
                        umma::tmem_st8(ta + 8, lo);
                        umma::tmem_st8(ta + 16, hi[h] + 8);
                        umma::tmem_st8(ta + 24, lo + 8);
                        umma::tmem_wait_st();
                    }
                    umma::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) umma::mbar_arrive(&half_done[h]);
                    if (y.out_lo) store32(y.out_lo, y.ld_out, (int)c0, lo);
                }
                if (!ok) {
                    if (lane == 0) flag_timeout(p.err, 1);
                    break;
                }
                if (y.out) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (h >= halves) break;
                        store32(y.out, y.ld_out, h * 128 + part * 32, hi[h]);
                    }
                }
            }
            umma::fence_before_sync();
            ok = named_barrier_and(1, MC_EPI_WARPS * 32, ok);
            if (!ok) break;
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (warp == MC_EPI_WARPS) umma::tmem_dealloc(tmem, 512);
}

}  // namespace
}  // namespace gbsdf

using namespace gbsdf;

extern "C" size_t gbsdf_mlp_layer_size(void) { return sizeof(gbsdf_mlp_layer); }

extern "C" int gbsdf_mlp_chain(int64_t M, int32_t n, const gbsdf_mlp_layer* layers, float beta, int* err, void* stream) {
    clear_error();
    GBSDF_CHECK_ARG(M >= 0 && M < ((int64_t)1 << 31), "M=%lld", (long long)M);
    // (one layer alone would leave nothing between a tile's epilogue and the MMAs two tiles on)
    GBSDF_CHECK_ARG(n >= 2 && n <= GBSDF_MLP_MAX_LAYERS && layers, "%d layers (2 to %d)", n, GBSDF_MLP_MAX_LAYERS);
    ChainParams p{};
    ChainMaps maps{};
    p.n_layers = n;
    p.M = M;
    p.beta = beta;
    p.err = err;
    for (int l = 0; l < n; ++l) {
        const gbsdf_mlp_layer& y = layers[l];
        const int k_chain = l > 0 ? layers[l - 1].N : 0, K = k_chain + y.K_in;
        GBSDF_CHECK_ARG(y.N == 128 || y.N == 256, "layer %d: width %d (128 or 256)", l, y.N);
        GBSDF_CHECK_ARG(y.K_in >= 0 && y.K_in % 16 == 0 && K > 0, "layer %d: %d input columns", l, y.K_in);
        GBSDF_CHECK_ARG(y.epi >= 0 && y.epi <= 2, "layer %d: activation %d", l, y.epi);
        GBSDF_CHECK_ARG(y.W && aligned(y.W, 16), "layer %d: W missing or misaligned", l);
        GBSDF_CHECK_ARG(y.K_in == 0 || (y.in_hi && y.in_lo && aligned(y.in_hi, 16) && aligned(y.in_lo, 16) &&
                                        y.ld_in >= y.K_in && y.ld_in % 8 == 0),
                        "layer %d: input", l);
        GBSDF_CHECK_ARG((!y.out_hi || aligned(y.out_hi, 16)) && (!y.out_lo || aligned(y.out_lo, 16)) &&
                            ((!y.out_hi && !y.out_lo) || (y.ld_out >= y.N && y.ld_out % 8 == 0)),
                        "layer %d: output", l);
        GBSDF_CHECK_ARG(y.K_in <= (l == 0 ? MC_MAX_FIRST : MC_MAX_TAIL), "layer %d: %d input columns (at most %d)", l, y.K_in,
                        l == 0 ? MC_MAX_FIRST : MC_MAX_TAIL);
        p.layer[l] = ChainLayer{k_chain, y.K_in, y.N, y.epi, y.ld_out, (__half*)y.out_hi, (__half*)y.out_lo, y.bias};
    }
    if (M == 0) return GBSDF_OK;
    const CUtensorMapL2promotion l2 = CU_TENSOR_MAP_L2_PROMOTION_L2_256B;
    for (int l = 0; l < n; ++l) {
        const gbsdf_mlp_layer& y = layers[l];
        const int K = p.layer[l].k_chain + y.K_in;
        if (int st = tensor_map_2d(&maps.w[l], false, y.W, y.N, K, K, MC_KCH, 128,
                                   CU_TENSOR_MAP_SWIZZLE_128B, l2, "W"))
            return st;
        if (y.K_in > 0) {
            if (int st = tensor_map_2d(&maps.in[l], false, y.in_hi, M, y.K_in, y.ld_in, MC_KCH, TILE_M,
                                       CU_TENSOR_MAP_SWIZZLE_128B, l2, "input"))
                return st;
            if (int st = tensor_map_2d(&maps.in_lo[l], false, y.in_lo, M, y.K_in, y.ld_in, MC_KCH, TILE_M,
                                       CU_TENSOR_MAP_SWIZZLE_128B, l2, "input lo"))
                return st;
        }
    }
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int64_t grid = (M + TILE_M - 1) / TILE_M;
    if (grid > sms) grid = sms > 0 ? sms : 1;
    allow_max_smem(k_mlp_chain);
    k_mlp_chain<<<(unsigned)grid, MC_THREADS, MC_SMEM, as_stream(stream)>>>(maps, p);
    return launch_status("mlp_chain");
}
