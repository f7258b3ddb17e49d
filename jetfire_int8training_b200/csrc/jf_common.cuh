// Shared device helpers for the Jetfire INT8 kernels (sm_100a).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/jetfire_b200.h"

namespace jf {

constexpr int QB = 32;  // quantisation block edge

// ---------------------------------------------------------------------------------------------------------
// host-side status plumbing
// ---------------------------------------------------------------------------------------------------------
extern thread_local int g_last_cuda_error;

inline int check_launch() {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        return JF_ERR_LAUNCH;
    }
    return JF_OK;
}
// Every operator kernel is launched while its predecessor in the stream still runs (programmatic dependent launch) and begins with
// grid_dependency(): it waits until that kernel has completed and its writes are visible, and then lets the next one be launched.  Wait
// first, then release: at most two neighbouring kernels overlap, and nothing is read or written before everything earlier is done.  What
// it saves is the launch latency and ramp of each call.  A predecessor that does not release early -- a framework's kernel, a copy -- is
// simply waited for, and so is this kernel by such a successor.
// The result is 0, but the compiler does not know that: added to the block index it makes every address depend on the wait, so that no
// read-only load (__ldg, const __restrict__), which a memory clobber does not hold back, can be scheduled ahead of it.
__device__ __forceinline__ uint32_t grid_dependency() {
    uint32_t zero;
    asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, 0;" : "=r"(zero)::"memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    return zero;
}
// (errors are left for check_launch())
template <class... P, class... A>
inline void launch(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool mult32(int64_t v) { return v > 0 && (v % 32) == 0; }

// ---------------------------------------------------------------------------------------------------------
// Philox4x32-10 (Random123) and the stochastic-rounding noise
// ---------------------------------------------------------------------------------------------------------
// Noise mapping.  One Philox call (four 32-bit words) serves the 8 consecutive elements of group g = e / 8; element e uses the
// 16-bit half (e & 1) of word (e >> 1) & 3:  noise = h * 2^-16 - 0.5, a multiple of 2^-16 in [-0.5, 0.5) like the reference's
// uniform_(-0.5, 0.5).  Built without an int->float conversion: the half is placed in the low mantissa bits of 2^23, and one
// FMA rescales it: (2^23 + h) * 2^-16 - 128.5 = h * 2^-16 - 0.5, exact in fp32 (noise2 below).

// What a call of Philox4x32-10 needs besides the group number: the ten round keys of the seed (key schedule: k + r * (0x9E3779B9,
// 0xBB67AE85)), computed on the host and passed with the kernel parameters (constant-bank operands of the rounds' XORs), and the parts
// of the first three rounds that do not depend on the low half of the group number.  With the counter (g_lo, 0, offset_lo, offset_hi)
//   round 1: one product of g_lo; the product of offset_lo is a constant of the launch,
//   round 2: x is such a constant too, so its product is, and round 3 sees one of its halves:
// 18 multiplications instead of 20 per call of 8 elements.  Group numbers of 2^32 and more (2^35 elements) take all rounds.
struct PhiloxKeys {
    uint32_t k[20];
    uint32_t z1, x2, z2, z3;    // XOR constants: z of round 1, x and z of round 2, z of round 3
};
inline PhiloxKeys make_philox_keys(uint64_t seed, uint64_t offset) {
    PhiloxKeys ks;
    uint32_t kx = (uint32_t)seed, ky = (uint32_t)(seed >> 32);
    for (int r = 0; r < 10; ++r) {
        ks.k[2 * r] = kx;
        ks.k[2 * r + 1] = ky;
        kx += 0x9E3779B9u;
        ky += 0xBB67AE85u;
    }
    const uint64_t p1 = 0xCD9E8D57ull * (uint32_t)offset;                       // round 1, product of z = offset_lo
    const uint32_t x = (uint32_t)(p1 >> 32) ^ ks.k[0];                          // round 1: x' = hi ^ y (= 0) ^ key
    const uint64_t p0 = 0xD2511F53ull * x;                                      // round 2, product of x
    ks.z1 = (uint32_t)(offset >> 32) ^ ks.k[1];
    ks.x2 = (uint32_t)p1 ^ ks.k[2];
    ks.z2 = (uint32_t)(p0 >> 32) ^ ks.k[3];
    ks.z3 = (uint32_t)p0 ^ ks.k[5];
    return ks;
}
// (64-bit products: one wide multiply-add instruction yields both halves)
__device__ __forceinline__ uint4 philox_rounds(uint4 c, const PhiloxKeys& ks, int first) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        if (r < first) continue;
        const uint64_t p0 = (uint64_t)0xD2511F53u * c.x, p1 = (uint64_t)0xCD9E8D57u * c.z;
        c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ ks.k[2 * r], (uint32_t)p1, (uint32_t)(p0 >> 32) ^ c.w ^ ks.k[2 * r + 1], (uint32_t)p0);
    }
    return c;
}
// WIDE: group numbers may need more than 32 bits.  A template parameter, chosen once per launch: a test inside would end the basic block,
// and the scheduler could not interleave the serial chains of several calls (quantize + SR of [12288 x 2304]: 29.4 us with the test).
template <bool WIDE>
__device__ __forceinline__ uint4 philox_group(uint64_t g, const PhiloxKeys& ks, uint64_t offset) {
    if (WIDE) return philox_rounds(make_uint4((uint32_t)g, (uint32_t)(g >> 32), (uint32_t)offset, (uint32_t)(offset >> 32)), ks, 0);
    const uint64_t a = (uint64_t)0xD2511F53u * (uint32_t)g;                     // round 1
    const uint64_t b = (uint64_t)0xCD9E8D57u * ((uint32_t)(a >> 32) ^ ks.z1);   // round 2
    const uint32_t x = (uint32_t)(b >> 32) ^ ks.x2, z = (uint32_t)a ^ ks.z2;
    const uint64_t p0 = (uint64_t)0xD2511F53u * x, p1 = (uint64_t)0xCD9E8D57u * z;   // round 3: y = lo of b, w = constant
    return philox_rounds(make_uint4((uint32_t)(p1 >> 32) ^ (uint32_t)b ^ ks.k[4], (uint32_t)p1, (uint32_t)(p0 >> 32) ^ ks.z3, (uint32_t)p0), ks, 3);
}

// ---------------------------------------------------------------------------------------------------------
// Exact IEEE division by a value shared across many elements.
// With y = RN(1/b) (correctly rounded reciprocal), q0 = RN(a*y), r = a - b*q0 (exact in one FMA) and
// q = RN(q0 + r*y) is the correctly rounded quotient RN(a/b) (Markstein's correction step), provided nothing
// under/overflows.  The fast path is taken only for b in [2^-60, 2^60]; otherwise div.rn is used.
// ---------------------------------------------------------------------------------------------------------
struct Divisor {
    float b;     // divisor
    float inv;   // RN(1/b)
    bool fast;   // fast path is valid
};
__device__ __forceinline__ Divisor make_divisor(float b) {
    Divisor d;
    d.b = b;
    d.inv = __frcp_rn(b);
    const float ab = fabsf(b);
    d.fast = (ab >= 8.673617379884035e-19f) && (ab <= 1.152921504606847e18f);
    return d;
}
// use: q0 = a * d.inv;  q = fma(fma(-d.b, q0, a), d.inv, q0)   (d.fast)      or      q = a / d.b   (otherwise)

// Two fp32 values in one 64-bit register and the two-wide IEEE operations on them (each half is rounded exactly like the scalar
// mul.rn / add.rn / fma.rn; subnormals are kept): one issue slot for two elements in the kernels that are bound by instruction issue.
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// the exact quotients a / d.b of two values (d.fast)
__device__ __forceinline__ uint64_t f2_div_fast(uint64_t a2, uint64_t inv2, uint64_t negb2) {
    const uint64_t q0 = f2_mul(a2, inv2);
    return f2_fma(f2_fma(negb2, q0, a2), inv2, q0);
}

// fp16 product of an int8 payload value and its fp16 scale, as the reference's "int8 * fp16" does
// (the int8 is converted to fp16 exactly, the product is rounded to fp16 once).  q*s is exact in fp32.
__device__ __forceinline__ __half deq16(int q, float s_as_float) { return __float2half_rn(__fmul_rn((float)q, s_as_float)); }

__device__ __forceinline__ int sbyte(uint32_t w, int i) { return (int)(int8_t)(w >> (8 * i)); }

// Exact int8 -> fp32 without the conversion unit: byte k of w (two's complement), with its sign bit flipped, goes into the low
// mantissa byte of 2^23; (2^23 + u) - (2^23 + 128) = q exactly.  `wx` must be w ^ 0x80808080.
__device__ __forceinline__ float byte_to_float(uint32_t wx, int k) {
    const uint32_t sel = k == 0 ? 0x7440u : k == 1 ? 0x7441u : k == 2 ? 0x7442u : 0x7443u;   // {byte k, 0x00, 0x00, 0x4B}
    return __fadd_rn(__uint_as_float(__byte_perm(wx, 0x4B000000u, sel)), -8388736.0f);
}

// The noise of the two elements of one generator word: both halves are placed over the exponent of 2^23 and rescaled by one two-wide FMA.
__device__ __forceinline__ uint64_t noise2(uint32_t w) {
    return f2_fma(f2_pack(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7410)), __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7432))),
                  f2_pack(1.52587890625e-05f, 1.52587890625e-05f), f2_pack(-128.5f, -128.5f));
}
// Noise for the 8 consecutive elements starting at linear index e (e % 8 == 0), as four packed pairs.
template <bool WIDE>
__device__ __forceinline__ void philox_noise8x2(uint64_t e, const PhiloxKeys& keys, uint64_t offset, uint64_t (&out)[4]) {
    const uint4 w = philox_group<WIDE>(e >> 3, keys, offset);
    out[0] = noise2(w.x); out[1] = noise2(w.y); out[2] = noise2(w.z); out[3] = noise2(w.w);
}
// Where the noise of a launch comes from
enum Noise : int { NOISE_GIVEN = 0, NOISE_PHILOX = 1, NOISE_PHILOX_WIDE = 2 };
constexpr int64_t PHILOX_WIDE_ELEMENTS = int64_t(1) << 35;      // 8 elements per group number
// v + sign(v) * noise for two values, i.e. sign(v) * (|v| + noise): rounding is symmetric, so the sign moves to the noise
__device__ __forceinline__ uint64_t f2_add_noise(uint64_t v2, uint64_t nz2) { return f2_add(v2, nz2 ^ (v2 & 0x8000000080000000ull)); }

// dtype-generic 16-element row chunk loads -> fp32
template <typename T>
struct Load16;
template <>
struct Load16<float> {
    static __device__ __forceinline__ void load(const float* p, float v[16]) {
        const float4* p4 = reinterpret_cast<const float4*>(p);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 t = __ldg(p4 + i);
            v[4 * i + 0] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
        }
    }
};
template <>
struct Load16<__half> {
    static __device__ __forceinline__ void load(const __half* p, float v[16]) {
        const uint4* p4 = reinterpret_cast<const uint4*>(p);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint4 t = __ldg(p4 + i);
            const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __half2 h = *reinterpret_cast<const __half2*>(&w[j]);
                const float2 f = __half22float2(h);
                v[8 * i + 2 * j] = f.x; v[8 * i + 2 * j + 1] = f.y;
            }
        }
    }
};
template <>
struct Load16<__nv_bfloat16> {
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, float v[16]) {
        const uint4* p4 = reinterpret_cast<const uint4*>(p);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint4 t = __ldg(p4 + i);
            const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[8 * i + 2 * j] = __uint_as_float(w[j] << 16);
                v[8 * i + 2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u);
            }
        }
    }
};

}  // namespace jf
