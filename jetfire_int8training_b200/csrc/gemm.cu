// Per-block (32x32) quantised INT8 GEMMs for sm_100a: forward Y = X W^T, input gradient dX = dY W and weight gradient
// dW = dY^T X, all from one persistent, warp-specialised kernel (gemm_kernel.cuh).
//
// Algorithm (fixed by the reference and its oracle): for every 32-wide K block p, in ascending order,
//     I_p = A_blk x B_blk^T  (exact int32),      acc = fma(sa[i,p] * sb[j,p], float(I_p), acc)   (fp32)
// followed by a per-32x32-block re-quantisation (or a dense fp16/fp32 store) of acc.
//
// Mapping to the hardware
//   * CTA tile 128 x 64, two CTAs per SM, persistent over a static list of (tile, K-split) work items.
//   * producer: one 128-byte-swizzled box per operand per stage = four K blocks; a 4-stage mbarrier ring (96 KB).
//   * issuer: tcgen05.mma kind::i8 has K = 32 = one quantisation block, so every K block is ONE 128x64x32 MMA with accumulation disabled.
//   * consumers: tcgen05.ld (a thread = one row of one quantisation block), int32 -> fp32, scale FMA into 32 fp32 registers.  This
//     CUDA-core work, not the tensor core, bounds the kernel.
//   * operands are consumed in place in either orientation: K-major (row-major [rows, K]) or MN-major (row-major
//     [K, rows]) through the UMMA descriptor major bits, so no transposed copy of W, dY or X is ever materialised.
//   * epilogue: a 32x32 block = 32 lanes x 32 thread-local values; absmax is a local max + one redux.sync.
// Every mbarrier wait is bounded by a clock budget; on expiry the CTA raises an error flag (read with jf_igemm_error_flag),
// leaves its loops, waits (bounded) for its copies and MMAs in flight and frees its tensor memory.
#include <cuda.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "jf_common.cuh"
#include "ptx_sm100.cuh"

namespace jf {

constexpr int BM = 128, BN = 64;                // CTA tile; two CTAs share an SM
constexpr int KB_PER_STAGE = 4;                 // 32-wide K blocks per pipeline stage (128 bytes of K)
constexpr int STAGES = 4;
constexpr int A_BYTES = BM * 128, B_BYTES = BN * 128, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int CONSUMER_WARPS = 8;
constexpr int GEMM_THREADS = (CONSUMER_WARPS + 2) * 32;
constexpr int TMEM_COLS = 4 * BN;               // four accumulators
constexpr size_t GEMM_SMEM = STAGES * STAGE_BYTES + 1024 /*alignment slack*/ + 128 /*barriers*/;
constexpr long long DRAIN_BUDGET_CLOCKS = 20000000LL;   // ~10 ms: abort-path wait for copies / MMAs already in flight
constexpr uint32_t WAIT_BUDGET_CLOCKS = 4000000000u;    // ~2 s at 2 GHz (32-bit clock)

enum GemmMode : int {
    MODE_INT8 = 0,      // int8 payload + fp16 scales
    MODE_DEQ16 = 1,     // fp16(q) * scale
    MODE_F16 = 2,       // dense fp16(acc)
    MODE_F32 = 3,       // dense fp32 acc (also used for split-K partials)
    MODE_INT32 = 4      // plain int32 accumulation (diagnostic)
};

struct GemmParams {
    int64_t M, N, K;
    int64_t tiles_m, tiles_n;
    int64_t nkb;            // K / 32
    int64_t splits;         // number of K ranges
    int64_t kb_per_split;   // K blocks per range (last may be shorter)
    const __half* sa; int64_t sa_sm, sa_sk;   // sa(i,p) = sa[i*sa_sm + p*sa_sk]
    const __half* sb; int64_t sb_sn, sb_sk;   // sb(j,p) = sb[j*sb_sn + p*sb_sk]
    int mode;
    int8_t* out8; __half* out_scale; __half* out16; float* out32; int32_t* out_i32;
    int stochastic; const float* noise; uint64_t offset; PhiloxKeys keys;
};
struct GemmPair {                       // the parameters of PairWalk
    GemmParams g[2];                    // dX, dW
    uint32_t long_one, rounds, short_from, level, short_items;
};

__device__ int g_gemm_error = 0;   // 0 = ok; otherwise the code of the first wait that expired

// Abort path: wait for a barrier phase that operations already in flight will complete, without touching the abort state.
__device__ __forceinline__ void drain_wait(uint64_t* bar, uint32_t parity) {
    const long long t0 = clock64();
    while (!ptx::mbar_try_wait_hint(bar, parity, 2000u))
        if (clock64() - t0 > DRAIN_BUDGET_CLOCKS) break;
}

// ---------------------------------------------------------------------------------------------------------
// Consumer arithmetic.  acc is kept as packed pairs of fp32 so the scale FMA can use the two-wide fma.rn.f32x2.
// int32 -> fp32 (cvt.rn.f32.s32) is exact: |I| <= 32*127^2 < 2^22.  (Building the float with an integer multiply-add of 0x4B400000 on the
// FMA pipe and a subtraction of 1.5*2^23 for 1/8, 1/4 or 1/2 of the values, to relieve the ALU pipe, measured 1-15 % slower.)
// CONV_INT32 adds the raw integers instead: the plain int32 GEMM behind jf_igemm_int32.
// ---------------------------------------------------------------------------------------------------------
constexpr int NO_SR = -1;     // beside the values of Noise
enum ConvMode : int { CONV_I2F = 0, CONV_INT32 = 1 };

// acc2[j] (16 packed pairs) += s * float(r[2j], r[2j+1]) for the 32 int32 values in r
template <int CONV>
__device__ __forceinline__ void scale_accumulate(uint64_t (&acc2)[16], const uint32_t (&r)[32], float s) {
    if (CONV == CONV_INT32) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const uint32_t lo = (uint32_t)acc2[j] + r[2 * j], hi = (uint32_t)(acc2[j] >> 32) + r[2 * j + 1];
            acc2[j] = ((uint64_t)hi << 32) | lo;
        }
        return;
    }
    const uint64_t s2 = f2_pack(s, s);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const uint64_t v = f2_pack(__int2float_rn((int)r[2 * j]), __int2float_rn((int)r[2 * j + 1]));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc2[j]) : "l"(s2), "l"(v));
    }
}

// Re-quantise / convert one 32x32 block held as 32 lanes x 16 packed pairs and store it.  Two values per instruction throughout.
enum StoreKind : int { STORE_DENSE = 1, STORE_QUANTISED = 2 };
template <int KINDS>
__device__ __forceinline__ void store_block(const GemmParams& p, const uint64_t (&acc2)[16], int64_t row, int64_t col, int64_t rowblk,
                                            int64_t colblk, int64_t split, int lane) {
    if ((KINDS & STORE_DENSE) && p.mode == MODE_INT32) {
        int4* dst = reinterpret_cast<int4*>(p.out_i32 + row * p.N + col);
#pragma unroll
        for (int k = 0; k < 8; ++k) dst[k] = make_int4((int)acc2[2 * k], (int)(acc2[2 * k] >> 32), (int)acc2[2 * k + 1], (int)(acc2[2 * k + 1] >> 32));
    } else if ((KINDS & STORE_DENSE) && p.mode == MODE_F32) {
        float4* dst = reinterpret_cast<float4*>(p.out32 + (split * p.M + row) * p.N + col);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            float4 v;
            f2_unpack(acc2[2 * k], v.x, v.y);
            f2_unpack(acc2[2 * k + 1], v.z, v.w);
            dst[k] = v;
        }
    } else if ((KINDS & STORE_DENSE) && p.mode == MODE_F16) {
        int4* dst = reinterpret_cast<int4*>(p.out16 + row * p.N + col);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            __half2 h[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float lo, hi;
                f2_unpack(acc2[4 * k + u], lo, hi);
                h[u] = __floats2half2_rn(lo, hi);
            }
            dst[k] = *reinterpret_cast<int4*>(h);
        }
    } else if (KINDS & STORE_QUANTISED) {
        float m = 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            float lo, hi;
            f2_unpack(acc2[j], lo, hi);
            m = fmaxf(m, fmaxf(fabsf(lo), fabsf(hi)));
        }
        const float amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
        const __half sc16 = __float2half_rn(__fdiv_rn(amax, 127.0f));
        const Divisor d = make_divisor(amax);
        const bool zero = (amax == 0.f);
        const uint64_t c127 = f2_pack(127.0f, 127.0f), inv2 = f2_pack(d.inv, d.inv), negb2 = f2_pack(-d.b, -d.b);
        const uint64_t magic2 = f2_pack(12582912.0f, 12582912.0f), nmagic2 = f2_pack(-12582912.0f, -12582912.0f);
        const float scf = __half2float(sc16);
        const uint64_t scf2 = f2_pack(scf, scf);
        // One decision per warp each: the exact-quotient fast path is valid for the whole block (same divisor in every lane), and
        // only stochastic rounding can leave [-127, 127], so only it needs the clamp.
        const bool fast = __all_sync(0xffffffffu, d.fast || zero);
        auto quantise_all = [&](auto fast_c, auto sr_c, auto deq_c) {
            constexpr bool FAST = decltype(fast_c)::value, SRND = decltype(sr_c)::value != NO_SR, DEQ = decltype(deq_c)::value;
            uint32_t words[8];
#pragma unroll
            for (int k8 = 0; k8 < 4; ++k8) {      // 8 elements = one Philox call
                uint64_t nz2[4] = {0ull, 0ull, 0ull, 0ull};
                if (SRND) {
                    if (decltype(sr_c)::value == NOISE_GIVEN) {
                        const float4 n0 = __ldg(reinterpret_cast<const float4*>(p.noise + row * p.N + col + 8 * k8));
                        const float4 n1 = __ldg(reinterpret_cast<const float4*>(p.noise + row * p.N + col + 8 * k8 + 4));
                        nz2[0] = f2_pack(n0.x, n0.y); nz2[1] = f2_pack(n0.z, n0.w); nz2[2] = f2_pack(n1.x, n1.y); nz2[3] = f2_pack(n1.z, n1.w);
                    } else {
                        philox_noise8x2<decltype(sr_c)::value == NOISE_PHILOX_WIDE>((uint64_t)(row * p.N + col + 8 * k8), p.keys, p.offset, nz2);
                    }
                }
                uint32_t bits[8], h16[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint64_t a127 = f2_mul(c127, acc2[4 * k8 + u]);
                    uint64_t v2;
                    if (FAST) {
                        v2 = f2_div_fast(a127, inv2, negb2);
                    } else {
                        float lo, hi;
                        f2_unpack(a127, lo, hi);
                        v2 = f2_pack(__fdiv_rn(lo, d.b), __fdiv_rn(hi, d.b));
                    }
                    if (SRND) {
                        float lo, hi;
                        f2_unpack(f2_add(v2, nz2[u]), lo, hi);
                        v2 = f2_pack(fminf(fmaxf(lo, -127.f), 127.f), fminf(fmaxf(hi, -127.f), 127.f));
                    }
                    v2 = f2_add(v2, magic2);                   // round to nearest even; the low byte is the payload
                    float lo, hi;
                    if (DEQ) {
                        f2_unpack(f2_mul(f2_add(v2, nmagic2), scf2), lo, hi);      // payload x scale, exact in fp32
                        const __half2 h = __floats2half2_rn(lo, hi);
                        h16[u] = zero ? 0u : *reinterpret_cast<const uint32_t*>(&h);
                    } else {
                        f2_unpack(v2, lo, hi);
                        bits[2 * u] = __float_as_uint(lo); bits[2 * u + 1] = __float_as_uint(hi);
                    }
                }
                if (DEQ) {
                    reinterpret_cast<uint4*>(p.out16 + row * p.N + col)[k8] = make_uint4(h16[0], h16[1], h16[2], h16[3]);
                } else {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        words[2 * k8 + h] = zero ? 0u : __byte_perm(__byte_perm(bits[4 * h], bits[4 * h + 1], 0x0040),
                                                                    __byte_perm(bits[4 * h + 2], bits[4 * h + 3], 0x0040), 0x5410);
                }
            }
            if (!DEQ) {
                int4* dst = reinterpret_cast<int4*>(p.out8 + row * p.N + col);
                dst[0] = make_int4(words[0], words[1], words[2], words[3]);
                dst[1] = make_int4(words[4], words[5], words[6], words[7]);
                if (lane == 0) p.out_scale[rowblk * (p.N / QB) + colblk] = sc16;
            }
        };
        using T_ = std::true_type; using F_ = std::false_type;
        auto rounding = [&](auto fast_c, auto sr_c) {
            if (p.mode == MODE_INT8) quantise_all(fast_c, sr_c, F_{}); else quantise_all(fast_c, sr_c, T_{});
        };
        if (!p.stochastic) {
            using N_ = std::integral_constant<int, NO_SR>;
            if (fast) rounding(T_{}, N_{}); else rounding(F_{}, N_{});
        } else if (p.noise) {
            using G_ = std::integral_constant<int, NOISE_GIVEN>;
            if (fast) rounding(T_{}, G_{}); else rounding(F_{}, G_{});
        } else if (fast && p.M < PHILOX_WIDE_ELEMENTS / p.N) {
            rounding(T_{}, std::integral_constant<int, NOISE_PHILOX>{});
        } else {
            using W_ = std::integral_constant<int, NOISE_PHILOX_WIDE>;
            if (fast) rounding(T_{}, W_{}); else rounding(F_{}, W_{});
        }
    }
}

#include "gemm_kernel.cuh"

// out[i] = ((p0[i] + p1[i]) + p2[i]) + ...   then converted to the output type
template <typename OutT>
__global__ void splitk_reduce_kernel(const float* partials, int64_t splits, int64_t count, OutT* __restrict__ out) {
    const int64_t i = ((int64_t)(blockIdx.x + grid_dependency()) * blockDim.x + threadIdx.x) * 4;
    if (i >= count) return;
    float4 a = *reinterpret_cast<const float4*>(partials + i);
    for (int64_t k = 1; k < splits; ++k) {
        const float4 b = *reinterpret_cast<const float4*>(partials + k * count + i);
        a.x = __fadd_rn(a.x, b.x); a.y = __fadd_rn(a.y, b.y); a.z = __fadd_rn(a.z, b.z); a.w = __fadd_rn(a.w, b.w);
    }
    if constexpr (sizeof(OutT) == 4) {
        *reinterpret_cast<float4*>(out + i) = a;
    } else {
        __half2 h[2] = {__floats2half2_rn(a.x, a.y), __floats2half2_rn(a.z, a.w)};
        *reinterpret_cast<uint2*>(out + i) = *reinterpret_cast<uint2*>(h);
    }
}

// ------------------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    });
    return fn;
}

// 2-D uint8 tensor [outer, inner], box box_inner x box_outer, swizzle of the box's width (64 or 128 bytes), zero fill outside.
static int make_map(CUtensorMap* map, const void* base, int64_t inner, int64_t outer, int box_inner, int box_outer) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return JF_ERR_UNSUPPORTED;
    const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
    const cuuint64_t strides[1] = {(cuuint64_t)inner};
    const cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, box_inner == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        g_last_cuda_error = (int)r;
        return JF_ERR_LAUNCH;
    }
    return JF_OK;
}

struct DeviceInfo {
    int sm_count = 0;
    int cc_major = 0;
    bool attr_set[32] = {};
};
static DeviceInfo g_dev[64];
static std::mutex g_dev_mutex;

static int device_info(DeviceInfo** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return JF_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_dev_mutex);
    DeviceInfo& d = g_dev[dev];
    if (d.sm_count == 0) {
        cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev);
        cudaDeviceGetAttribute(&d.cc_major, cudaDevAttrComputeCapabilityMajor, dev);
    }
    *out = &d;
    return d.cc_major == 10 ? JF_OK : JF_ERR_UNSUPPORTED;
}

#include "gemm_launch.inc"

// Number of K ranges of a weight-gradient GEMM.  It fixes the order in which dW is summed, hence its bits, and stochastic rounding turns a
// last-bit difference in the weights into percents of the next step's gradients: the plan therefore stays the one of 128 x 128 tiles, one
// per SM, although the CTAs are 128 x 64.  (A plan that counts rounds of CTA slots gives [768 x 2304], K = 12288 two ranges: 76 us, not 92.)
static int plan_splits(int64_t M, int64_t N, int64_t K, int split_k, int sm_count, int64_t* per_out) {
    const int64_t nkb = K / QB;
    int64_t s = split_k;
    if (s <= 0) {
        s = sm_count / (((M + 127) / 128) * ((N + 127) / 128));
        const int64_t cap = nkb / 16;   // keep at least 16 K blocks per range
        if (s > cap) s = cap;
        if (s < 1) s = 1;
    }
    if (s > nkb) s = nkb;
    const int64_t per = (nkb + s - 1) / s;
    if (per_out) *per_out = per;
    return (int)((nkb + per - 1) / per);
}

}  // namespace jf

using namespace jf;

static inline int check_gemm_dims(int64_t M, int64_t N, int64_t K) {
    if (!mult32(M) || !mult32(N) || !mult32(K)) return JF_ERR_SHAPE;
    if (M > (1LL << 30) || N > (1LL << 30) || K > (1LL << 30)) return JF_ERR_SHAPE;
    return JF_OK;
}

// What the entry points of the two gradients check and fill in.
static int dgrad_params(GemmParams& p, const int8_t* g, const int8_t* w, const void* sg, int64_t sg_stride_m, int64_t sg_stride_k,
                        const void* sw, int64_t sw_stride_k, int64_t sw_stride_n, int64_t M, int64_t N, int64_t K, int out_mode, int8_t* dx8,
                        void* sdx, void* dx16, int stochastic, const float* noise, uint64_t seed, uint64_t offset) {
    if (!g || !w || !sg || !sw) return JF_ERR_NULL;
    if (int e = check_gemm_dims(M, N, K)) return e;
    if (!aligned16(g) || !aligned16(w) || (noise && !aligned16(noise))) return JF_ERR_ALIGN;
    p.M = M; p.N = N; p.K = K; p.splits = 1; p.kb_per_split = K / QB;
    p.sa = (const __half*)sg; p.sa_sm = sg_stride_m; p.sa_sk = sg_stride_k;
    p.sb = (const __half*)sw; p.sb_sn = sw_stride_n; p.sb_sk = sw_stride_k;
    p.stochastic = stochastic; p.noise = noise; p.keys = make_philox_keys(seed, offset); p.offset = offset;
    if (out_mode == JF_OUT_INT8) {
        if (!dx8 || !sdx) return JF_ERR_NULL;
        if (!aligned16(dx8)) return JF_ERR_ALIGN;
        p.mode = MODE_INT8; p.out8 = dx8; p.out_scale = (__half*)sdx;
    } else if (out_mode == JF_OUT_DEQUANT_F16) {
        if (!dx16) return JF_ERR_NULL;
        if (!aligned16(dx16)) return JF_ERR_ALIGN;
        p.mode = MODE_DEQ16; p.out16 = (__half*)dx16;
    } else {
        return JF_ERR_ARG;
    }
    return JF_OK;
}
static int wgrad_params(GemmParams& p, const int8_t* g, const int8_t* x, const void* sg, int64_t sg_stride_k, int64_t sg_stride_m,
                        const void* sx, int64_t sx_stride_k, int64_t sx_stride_n, int64_t M, int64_t N, int64_t K, int out_dtype, void* dw,
                        int split_k, float* scratch) {
    if (!g || !x || !sg || !sx || !dw) return JF_ERR_NULL;
    if (int e = check_gemm_dims(M, N, K)) return e;
    if (!aligned16(g) || !aligned16(x) || !aligned16(dw)) return JF_ERR_ALIGN;
    if (out_dtype != JF_F16 && out_dtype != JF_F32) return JF_ERR_DTYPE;
    DeviceInfo* di = nullptr;
    if (int e = device_info(&di)) return e;
    p.M = M; p.N = N; p.K = K;
    p.splits = plan_splits(M, N, K, split_k, di->sm_count, &p.kb_per_split);
    p.sa = (const __half*)sg; p.sa_sm = sg_stride_m; p.sa_sk = sg_stride_k;
    p.sb = (const __half*)sx; p.sb_sn = sx_stride_n; p.sb_sk = sx_stride_k;
    if (p.splits == 1) {
        if (out_dtype == JF_F16) { p.mode = MODE_F16; p.out16 = (__half*)dw; }
        else { p.mode = MODE_F32; p.out32 = (float*)dw; }
        return JF_OK;
    }
    if (!scratch) return JF_ERR_NULL;
    if (!aligned16(scratch)) return JF_ERR_ALIGN;
    p.mode = MODE_F32; p.out32 = scratch;
    return JF_OK;
}
static int reduce_splits(const GemmParams& p, const float* scratch, int out_dtype, void* dw, cudaStream_t st) {
    if (p.splits == 1) return JF_OK;
    const int64_t count = p.M * p.N;
    const unsigned grid = (unsigned)((count / 4 + 255) / 256);
    if (out_dtype == JF_F16) jf::launch(splitk_reduce_kernel<__half>, grid, 256, 0, st, scratch, p.splits, count, (__half*)dw);
    else jf::launch(splitk_reduce_kernel<float>, grid, 256, 0, st, scratch, p.splits, count, (float*)dw);
    return check_launch();
}

extern "C" {

int jf_igemm_forward(const int8_t* x, const int8_t* w, const void* sx, int64_t sx_stride_m, int64_t sx_stride_k, const void* sw,
                     int64_t sw_stride_n, int64_t sw_stride_k, int64_t M, int64_t N, int64_t K, int out_mode, int8_t* y8, void* sy,
                     void* y16, void* op16, int64_t op16_bytes, void* stream) {
    if (!x || !w || !sx || !sw) return JF_ERR_NULL;
    if (int e = check_gemm_dims(M, N, K)) return e;
    if (!aligned16(x) || !aligned16(w)) return JF_ERR_ALIGN;
    GemmParams p{};
    p.M = M; p.N = N; p.K = K; p.splits = 1; p.kb_per_split = K / QB;
    p.sa = (const __half*)sx; p.sa_sm = sx_stride_m; p.sa_sk = sx_stride_k;
    p.sb = (const __half*)sw; p.sb_sn = sw_stride_n; p.sb_sk = sw_stride_k;
    if (out_mode == JF_OUT_INT8) {
        if (!y8 || !sy) return JF_ERR_NULL;
        if (!aligned16(y8)) return JF_ERR_ALIGN;
        p.mode = MODE_INT8; p.out8 = y8; p.out_scale = (__half*)sy;
    } else if (out_mode == JF_OUT_DEQUANT_F16) {
        if (!y16) return JF_ERR_NULL;
        if (!aligned16(y16)) return JF_ERR_ALIGN;
        p.mode = MODE_DEQ16; p.out16 = (__half*)y16;
    } else {
        return JF_ERR_ARG;
    }
    (void)op16; (void)op16_bytes;
    return launch_fwd(x, w, p, (cudaStream_t)stream);
}

/* Bytes of operand scratch worth passing to a GEMM with these dimensions: none, the kernel reads the int8 operands in place
 * (the `op16` arguments of the GEMM entry points are accepted and not used). */
int64_t jf_igemm_op16_bytes(int64_t, int64_t, int64_t) { return 0; }

int jf_igemm_dgrad(const int8_t* g, const int8_t* w, const void* sg, int64_t sg_stride_m, int64_t sg_stride_k, const void* sw,
                   int64_t sw_stride_k, int64_t sw_stride_n, int64_t M, int64_t N, int64_t K, int out_mode, int8_t* dx8, void* sdx,
                   void* dx16, int stochastic, const float* noise, uint64_t seed, uint64_t offset, void* op16, int64_t op16_bytes,
                   void* stream) {
    GemmParams p{};
    if (int e = dgrad_params(p, g, w, sg, sg_stride_m, sg_stride_k, sw, sw_stride_k, sw_stride_n, M, N, K, out_mode, dx8, sdx, dx16,
                             stochastic, noise, seed, offset)) return e;
    (void)op16; (void)op16_bytes;
    return launch_dgrad_layout(g, w, p, (cudaStream_t)stream);
}

int jf_igemm_wgrad_plan(int64_t M, int64_t N, int64_t K, int split_k) {
    if (check_gemm_dims(M, N, K)) return JF_ERR_SHAPE;
    int sm = 148;
    DeviceInfo* di = nullptr;
    if (device_info(&di) == JF_OK) sm = di->sm_count;
    return plan_splits(M, N, K, split_k, sm, nullptr);
}

int jf_igemm_wgrad(const int8_t* g, int g_transposed, const int8_t* x, const void* sg, int64_t sg_stride_k, int64_t sg_stride_m,
                   const void* sx, int64_t sx_stride_k, int64_t sx_stride_n, int64_t M, int64_t N, int64_t K, int out_dtype, void* dw,
                   int split_k, float* scratch, void* op16, int64_t op16_bytes, void* stream) {
    GemmParams p{};
    if (int e = wgrad_params(p, g, x, sg, sg_stride_k, sg_stride_m, sx, sx_stride_k, sx_stride_n, M, N, K, out_dtype, dw, split_k, scratch)) return e;
    cudaStream_t st = (cudaStream_t)stream;
    (void)op16; (void)op16_bytes;
    if (int e = g_transposed ? launch_dgrad_layout(g, x, p, st) : launch_wgrad_layout(g, x, p, st)) return e;
    return reduce_splits(p, scratch, out_dtype, dw, st);
}

int jf_igemm_backward(const int8_t* g, const int8_t* w, const int8_t* x, const void* sg, int64_t sg_stride_m, int64_t sg_stride_n,
                      const void* sw, int64_t sw_stride_n, int64_t sw_stride_k, const void* sx, int64_t sx_stride_m, int64_t sx_stride_k,
                      int64_t tokens, int64_t cout, int64_t cin, int out_mode, int8_t* dx8, void* sdx, void* dx16, int stochastic,
                      const float* noise, uint64_t seed, uint64_t offset, int dw_dtype, void* dw, int split_k, float* scratch, void* stream) {
    GemmParams d{}, q{};
    if (int e = dgrad_params(d, g, w, sg, sg_stride_m, sg_stride_n, sw, sw_stride_n, sw_stride_k, tokens, cin, cout, out_mode, dx8, sdx, dx16,
                             stochastic, noise, seed, offset)) return e;
    if (int e = wgrad_params(q, g, x, sg, sg_stride_m, sg_stride_n, sx, sx_stride_m, sx_stride_k, cout, cin, tokens, dw_dtype, dw, split_k,
                             scratch)) return e;
    cudaStream_t st = (cudaStream_t)stream;
    if (int e = launch_pair(g, w, x, d, q, st)) return e;
    return reduce_splits(q, scratch, dw_dtype, dw, st);
}

int jf_igemm_backward_launches(int64_t tokens, int64_t cout, int64_t cin, int split_k) {
    if (check_gemm_dims(tokens, cout, cin)) return JF_ERR_SHAPE;
    int sm = 148;
    DeviceInfo* di = nullptr;
    if (device_info(&di) == JF_OK) sm = di->sm_count;
    GemmPair pair{};
    GemmParams &d = pair.g[0], &w = pair.g[1];
    d.M = tokens; d.N = cin; d.K = cout; d.splits = 1; d.kb_per_split = cout / QB;
    w.M = cout; w.N = cin; w.K = tokens; w.splits = plan_splits(cout, cin, tokens, split_k, sm, &w.kb_per_split);
    count_tiles(d);
    count_tiles(w);
    int64_t grid;
    return (plan_pair(pair, 2 * (int64_t)sm, &grid) ? 1 : 2) + (w.splits > 1 ? 1 : 0);
}

int jf_igemm_int32(const int8_t* a, const int8_t* b, int64_t M, int64_t N, int64_t K, int32_t* c, void* stream) {
    if (!a || !b || !c) return JF_ERR_NULL;
    if (int e = check_gemm_dims(M, N, K)) return e;
    if (!aligned16(a) || !aligned16(b) || !aligned16(c)) return JF_ERR_ALIGN;
    GemmParams p{};
    p.M = M; p.N = N; p.K = K; p.splits = 1; p.kb_per_split = K / QB;
    p.mode = MODE_INT32; p.out_i32 = c;
    return launch_int32(a, b, p, (cudaStream_t)stream);
}

/* Reads (and clears) the device-side error flag raised when a bounded wait inside the GEMM kernel expired.
 * Synchronises the device.  0 = no error. */
int jf_igemm_error_flag(void) {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_gemm_error, sizeof(int)) != cudaSuccess) return JF_ERR_LAUNCH;
    if (v != 0) cudaMemcpyToSymbol(g_gemm_error, &zero, sizeof(int));
    return v;
}

}  // extern "C"
