// The persistent per-block INT8 GEMM kernel (included by gemm.cu inside namespace jf, after the helpers it uses).
//
// What bounds it.  Every 128 x 128 x 32 block product (64 clocks on the tensor core) leaves tensor memory as 16384 int32 values that the
// CUDA cores owe a conversion and a scale FMA each: 512 warp conversions on the ALU pipe (2 clocks each: 256 SM clocks) and 256
// fma.rn.f32x2 on the FMA pipe (144 clocks).  The kernel needs ~440 SM clocks per block product (ALU pipe 69 % busy, issue slots 65 %).
//
// Two CTAs share an SM.  One CTA of 16 consumer warps per SM moves in step: all its warps leave the same barrier, load the same
// accumulator and then queue for the same pipe, and nothing computes during an epilogue.  Two independent CTAs of 128 x 64 tiles with
// eight consumer warps each fill one another's gaps: 12288 x 3072 x 768 forward 131 -> 111 us (520 TOPS), both gradients of 7392 x 1600 x 1600 227 -> 158 us.
// Their operand traffic (12 KB per block product and SM; TMA delivers 56 B per clock and SM from L2) stays below the arithmetic.
// Copying the operands to fp16 first (kind::f16 delivers floats, no conversion) is no way around it: at 16 KB per block product the
// loads alone take 290 clocks, and the copies cost as much as they save at the layer shapes; at 8192^3 that kernel drew 1725 MHz from the
// power cap against 1920 MHz here and the two took the same time (1.55-1.60 ms).
//
// Warp roles (10 warps): 8 consumers, 1 TMA producer, 1 MMA issuer, each of the latter two with one elected lane (elect.sync: with
// `lane == 0` instead, every tcgen05.mma and commit costs its thread ~100 clocks more).
//
// Hand-over.  Tensor memory (256 columns per CTA) holds four 64-column accumulators in two PAIRS; K blocks 0, 1 of a stage go to pair 0,
// K blocks 2, 3 to pair 1, one tcgen05.commit each.  One barrier wait and one arrival per warp serve two K blocks: the number of
// instructions around the arithmetic is what the consumers' time depends on.  A short last stage passes its second pair on empty, so
// that every tile starts at pair 0 and the consumers' loop has no branch and no register that names a slot.
//
// Consumers.  Warp w owns TMEM lanes 32*(w%4).. (rows) and columns 32*(w/4).. of every accumulator: a thread is one row of one 32x32
// quantisation block (32 fp32 accumulators).  The scale products sa*sb of 32 K blocks sit one per lane and are broadcast by shuffle.
//
// Abort path.  Every wait is bounded; when one expires the CTA's flag is raised, the producer and the issuer leave their loops, the
// consumers run through theirs without waiting.  Before the CTA frees its tensor memory the producer waits (bounded) for the bulk copies
// it has in flight and the issuer commits its outstanding MMAs to a scratch barrier and waits (bounded) for it.
#pragma once

// Tiles are numbered in groups of RASTER_GM tile rows, M-fastest inside a group, so that the CTAs in flight together share A and B
// panels that stay in L2.  (32-bit arithmetic: the launcher refuses problems with 2^31 tiles or more.)
constexpr int RASTER_GM = 16;
__device__ __forceinline__ void tile_coords(uint32_t tile, uint32_t tiles_m, uint32_t tiles_n, int& tm, int& tn) {
    const uint32_t group_size = RASTER_GM * tiles_n;
    const uint32_t group = tile / group_size, in_group = tile % group_size;
    const uint32_t first_m = group * RASTER_GM;
    const uint32_t gm = min((uint32_t)RASTER_GM, tiles_m - first_m);
    tm = (int)(first_m + in_group % gm);
    tn = (int)(in_group / gm);
}

// Wait for a barrier phase in as few instructions as the ready case allows (one try_wait and one branch).  A wait that outlasts the
// clock budget, or that meets a raised abort flag, ends; the caller goes on (its results are void, every loop is finite).
// OFF / ABORT_OFF: byte offsets of the barrier and of the abort flag from `base`.
template <int OFF, int ABORT_OFF>
__device__ __forceinline__ void tight_wait(uint32_t base, uint32_t parity) {
    asm volatile(
        "{\n\t.reg .pred P, Q;\n\t.reg .u32 t0, t1, f;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P, [%0+%2], %1;\n\t"
        "@P bra DONE;\n\t"
        "mov.u32 t0, %%clock;\n\t"
        "LOOP:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P, [%0+%2], %1;\n\t"
        "@P bra DONE;\n\t"
        "ld.volatile.shared.u32 f, [%0+%3];\n\t"
        "mov.u32 t1, %%clock;\n\t"
        "sub.u32 t1, t1, t0;\n\t"
        "setp.gt.u32 Q, t1, %4;\n\t"
        "@Q st.volatile.shared.u32 [%0+%3], 4;\n\t"
        "setp.ne.or.u32 Q, f, 0, Q;\n\t"
        "@!Q bra LOOP;\n\t"
        "DONE:\n\t}" ::"r"(base), "r"(parity), "n"(OFF), "n"(ABORT_OFF), "n"(WAIT_BUDGET_CLOCKS) : "memory");
}
// lane 0 arrives on the barrier at base + OFF
template <int OFF>
__device__ __forceinline__ void arrive_lane0(uint32_t base, int lane) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0+%2];\n\t}" ::"r"(base), "r"(lane), "n"(OFF) : "memory");
}
// The producer's and the issuer's wait: every try lets the hardware park the thread for up to 2 us.  False when it expired.
__device__ __forceinline__ bool lean_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {
    if (__builtin_expect(ptx::mbar_try_wait_hint(bar, parity, 2000u), 1)) return true;
    const uint32_t t0 = (uint32_t)clock();
    while (!ptx::mbar_try_wait_hint(bar, parity, 2000u)) {
        if (__builtin_expect(*abort_flag != 0, 0)) return false;
        if (__builtin_expect((uint32_t)clock() - t0 > WAIT_BUDGET_CLOCKS, 0)) {
            *abort_flag = code;
            return false;
        }
    }
    return true;
}

struct Item {        // tile and K range of a work item
    uint32_t tile, split;
    int kb0, kb1;
    __device__ __forceinline__ Item(const GemmParams& p, uint32_t item) {
        const uint32_t num_tiles = (uint32_t)(p.tiles_m * p.tiles_n);
        tile = item % num_tiles;
        split = item / num_tiles;
        kb0 = (int)split * (int)p.kb_per_split;
        kb1 = min((int)p.nkb, kb0 + (int)p.kb_per_split);
    }
};
// The work items (tile, K range) of one CTA, in order.  SingleWalk: one GEMM, every gridDim.x-th item.
template <bool A_MN>
struct SingleWalk {
    using Params = GemmParams;
    const Params& p;
    uint32_t item;
    const uint32_t num_items;
    __device__ __forceinline__ SingleWalk(const Params& p_, uint32_t cta)
        : p(p_), item(cta), num_items((uint32_t)(p_.tiles_m * p_.tiles_n) * (uint32_t)p_.splits) {}
    __device__ __forceinline__ bool valid() const { return item < num_items; }
    __device__ __forceinline__ void next() { item += gridDim.x; }
    __device__ __forceinline__ const GemmParams& gemm() const { return p; }
    static __device__ __forceinline__ bool second() { return false; }
    static __device__ __forceinline__ bool a_mn() { return A_MN; }
    __device__ __forceinline__ void store(const uint64_t (&acc)[16], int64_t row, int64_t col, int64_t rowblk, int64_t colblk, int64_t split, int lane) const {
        store_block<STORE_DENSE | STORE_QUANTISED>(p, acc, row, col, rowblk, colblk, split, lane);
    }
};
// PairWalk: both gradients of a linear layer in one launch, the one with the longer K loop per item ("long") before the other.  Run one
// after the other, each ends with CTA slots idle in its last round (dY 12288 x 2304, W 2304 x 768: 216 weight-gradient tiles of 384 K
// blocks on 296 slots).  Here a CTA takes its long items round-robin; the CTAs that get one less than the others take `level` short items
// in its place; the rest of the short items goes round-robin, first to those CTAs.  Fixed lists, no counter: a tile costs the same
// wherever it runs.  Both gradients in us, two launches -> one: 12288 x 2304 x 768 169 -> 151, 7392 x 1600 x 1600 152 -> 136.
// The epilogue names dX's and dW's parameters statically: with a run-time index the Philox round keys are loads, no longer operands.
struct PairWalk {
    using Params = GemmPair;
    const Params& p;
    const uint32_t cta;
    uint32_t seq = 0, item = 0, which = 0;      // which: 0 dX, 1 dW
    bool ok = false;
    __device__ __forceinline__ PairWalk(const Params& p_, uint32_t cta_) : p(p_), cta(cta_) { locate(); }
    __device__ __forceinline__ void locate() {
        const uint32_t ctas = gridDim.x, short_from = p.short_from;             // CTAs from short_from on have one long item less
        const uint32_t longs = p.rounds + (cta < short_from ? 1u : 0u);
        if (seq < longs) {
            which = p.long_one;
            item = cta + seq * ctas;
            ok = true;
            return;
        }
        which = p.long_one ^ 1u;
        const uint32_t q = seq - longs, level = cta >= short_from ? p.level : 0u;
        if (q < level) item = cta - short_from + (ctas - short_from) * q;
        else item = (ctas - short_from) * p.level + (cta >= short_from ? cta - short_from : cta + ctas - short_from) + ctas * (q - level);
        ok = item < p.short_items;
    }
    __device__ __forceinline__ bool valid() const { return ok; }
    __device__ __forceinline__ void next() { ++seq; locate(); }
    __device__ __forceinline__ const GemmParams& gemm() const { return p.g[which]; }
    __device__ __forceinline__ bool second() const { return which != 0u; }
    __device__ __forceinline__ bool a_mn() const { return which != 0u; }
    __device__ __forceinline__ void store(const uint64_t (&acc)[16], int64_t row, int64_t col, int64_t rowblk, int64_t colblk, int64_t split, int lane) const {
        if (which == 0u) store_block<STORE_QUANTISED>(p.g[0], acc, row, col, rowblk, colblk, split, lane);
        else store_block<STORE_DENSE>(p.g[1], acc, row, col, rowblk, colblk, split, lane);
    }
};

// map_b1: dW's B operand (PairWalk; both gradients have the same A operand)
template <class Walk, bool B_MN, int CONV>
__global__ void __launch_bounds__(GEMM_THREADS, 2)
gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_b1,
            const __grid_constant__ typename Walk::Params params) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    // barriers: pair_full[2] at 0, pair_empty[2] at 16, abort flag at 32, tmem slot at 36, drain at 40, full[STAGES] at 48,
    // empty[STAGES] after them
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
    uint64_t* pair_full = bars;
    uint64_t* pair_empty = bars + 2;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 4);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4) + 1;
    uint64_t* drain_bar = bars + 5;
    uint64_t* full_bar = bars + 6;
    uint64_t* empty_bar = full_bar + STAGES;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { ptx::mbar_init(&full_bar[s], 1); ptx::mbar_init(&empty_bar[s], 1); }
        for (int g = 0; g < 2; ++g) { ptx::mbar_init(&pair_full[g], 1); ptx::mbar_init(&pair_empty[g], CONSUMER_WARPS); }
        ptx::mbar_init(drain_bar, 1);
        *abort_flag = 0;
        ptx::fence_barrier_init();
    }
    if (warp == CONSUMER_WARPS + 1) {
        ptx::tmem_alloc(tmem_slot, TMEM_COLS);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t block_x = blockIdx.x + grid_dependency();      // barriers and tensor memory are set up while the previous kernel ends

    if (warp == CONSUMER_WARPS) {
        // ------------------------------------------------------------------ producer
        if (ptx::elect_one()) {
            uint32_t it = 0, s = 0, ph = 0;
            bool ok = true;
            for (Walk w(params, block_x); w.valid() && ok; w.next()) {
                const GemmParams& p = w.gemm();
                const Item i(p, w.item);
                int tm, tn;
                tile_coords(i.tile, (uint32_t)p.tiles_m, (uint32_t)p.tiles_n, tm, tn);
                const bool a_mn = w.a_mn();
                const CUtensorMap* mb = w.second() ? &map_b1 : &map_b;
                const int row = tm * BM, col = tn * BN;
                for (int kb = i.kb0; kb < i.kb1; kb += KB_PER_STAGE) {
                    if (!(ok = lean_wait(&empty_bar[s], ph ^ 1u, abort_flag, 1))) break;
                    ptx::mbar_arrive_expect_tx(&full_bar[s], STAGE_BYTES);
                    uint8_t* a = smem + s * STAGE_BYTES;
                    const int k = kb * QB;
                    ptx::tma_load_2d(a, &map_a, &full_bar[s], a_mn ? row : k, a_mn ? k : row);
                    ptx::tma_load_2d(a + A_BYTES, mb, &full_bar[s], B_MN ? col : k, B_MN ? k : col);
                    ++it;
                    if (++s == STAGES) { s = 0; ph ^= 1u; }
                }
            }
            if (*abort_flag)
                for (uint32_t j = it > STAGES ? it - STAGES : 0u; j < it; ++j) drain_wait(&full_bar[j % STAGES], (j / STAGES) & 1u);
        }
    } else if (warp == CONSUMER_WARPS + 1) {
        // ------------------------------------------------------------------ MMA issuer
        uint32_t s = 0, ph = 0, par = 1;
        bool ok = true;
        const uint64_t db_base = B_MN ? ptx::make_smem_desc_sw64(ptx::smem_u32(smem + A_BYTES), 128 * 64, 512)
                                      : ptx::make_smem_desc_sw128(ptx::smem_u32(smem + A_BYTES), 16, 1024);
        for (Walk w(params, block_x); w.valid() && ok; w.next()) {
            const Item i(w.gemm(), w.item);
            const bool a_mn = w.a_mn();
            const uint32_t idesc = a_mn ? ptx::make_idesc_i8(BM, BN, true, B_MN) : ptx::make_idesc_i8(BM, BN, false, B_MN);
            const uint64_t da_base = ptx::make_smem_desc_sw128(ptx::smem_u32(smem), a_mn ? 128 * 128 : 16, 1024);
            const uint32_t a_step = a_mn ? 256 : 2;         // descriptor units (16 bytes) from one K block to the next
            for (int kb = i.kb0; kb < i.kb1 && ok; kb += KB_PER_STAGE) {
                if (!(ok = __all_sync(0xffffffffu, lean_wait(&full_bar[s], ph, abort_flag, 2)))) break;
                ptx::tc_fence_after();
                const uint64_t da = da_base + (uint64_t)(s * (STAGE_BYTES / 16)), db = db_base + (uint64_t)(s * (STAGE_BYTES / 16));
                const int nblk = min(KB_PER_STAGE, i.kb1 - kb);
#pragma unroll
                for (int pp = 0; pp < 2; ++pp) {
                    if (!(ok = __all_sync(0xffffffffu, lean_wait(&pair_empty[pp], par, abort_flag, 3)))) break;
                    ptx::tc_fence_after();
                    if (ptx::elect_one()) {
#pragma unroll
                        for (int j = 2 * pp; j < 2 * pp + 2; ++j)
                            if (j < nblk)
                                ptx::umma_i8(tmem_base + j * BN, da + (uint64_t)(j * a_step),
                                             db + (uint64_t)(B_MN ? j * 128 : j * 2), idesc, 0u);
                        ptx::umma_commit(&pair_full[pp]);       // a pair without a K block is passed on empty: every tile starts at pair 0
                        if (pp == 1) ptx::umma_commit(&empty_bar[s]);
                    }
                    __syncwarp();
                }
                par ^= 1u;
                if (++s == STAGES) { s = 0; ph ^= 1u; }
            }
        }
        if (*abort_flag && ptx::elect_one()) {
            ptx::umma_commit(drain_bar);
            drain_wait(drain_bar, 0u);
        }
    } else {
        // ------------------------------------------------------------------ consumers
        const int quad = warp & 3, cg = warp >> 2;
        const uint32_t base = ptx::smem_u32(bars);
        const uint32_t t0 = tmem_base + ((uint32_t)(quad * 32) << 16) + cg * 32;
        uint32_t par = 0;
        for (Walk w(params, block_x); w.valid(); w.next()) {
            const GemmParams& p = w.gemm();
            const Item item(p, w.item);
            int tm, tn;
            tile_coords(item.tile, (uint32_t)p.tiles_m, (uint32_t)p.tiles_n, tm, tn);
            const int kb0 = item.kb0, n = item.kb1 - kb0;
            const int rowblk = tm * (BM / QB) + quad, colblk = tn * (BN / QB) + cg;
            const bool blk_ok = rowblk < (int)(p.M / QB) && colblk < (int)(p.N / QB);   // warp-uniform

            uint64_t acc[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[j] = 0ull;
            // lane l holds the scale product of K block 32 i + l
            const __half* sa_ptr = p.sa + (int64_t)rowblk * p.sa_sm + (int64_t)(kb0 + lane) * p.sa_sk;
            const __half* sb_ptr = p.sb + (int64_t)colblk * p.sb_sn + (int64_t)(kb0 + lane) * p.sb_sk;
            unsigned short ha = 0, hb = 0;
            auto fetch_scales = [&](int t) {
                if (CONV != CONV_INT32 && t + lane < n && blk_ok) {
                    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(ha) : "l"(sa_ptr + (int64_t)t * p.sa_sk));
                    asm volatile("ld.global.nc.u16 %0, [%1];" : "=h"(hb) : "l"(sb_ptr + (int64_t)t * p.sb_sk));
                }
            };
            fetch_scales(0);
            float sc = 0.f;
            auto pair = [&](auto pp_c, int k, int left) {          // `left` K blocks remain (the pair holds min(2, left) of them)
                constexpr int PP = decltype(pp_c)::value;
                const float s0 = __shfl_sync(0xffffffffu, sc, k), s1 = __shfl_sync(0xffffffffu, sc, k + 1);
                tight_wait<8 * PP, 32>(base, par);
                __syncwarp();
                ptx::tc_fence_after();
                uint32_t r[32];
                if (left > 1) {
                    ptx::tmem_ld_wait_32x32b_x32(t0 + 128 * PP, r);
                    scale_accumulate<CONV>(acc, r, s0);
                    ptx::tmem_ld_wait_32x32b_x32(t0 + 128 * PP + 64, r);
                    ptx::tc_fence_before();
                    arrive_lane0<16 + 8 * PP>(base, lane);
                    scale_accumulate<CONV>(acc, r, s1);
                } else {
                    if (left == 1) {
                        ptx::tmem_ld_wait_32x32b_x32(t0 + 128 * PP, r);
                        scale_accumulate<CONV>(acc, r, s0);
                    }
                    ptx::tc_fence_before();
                    arrive_lane0<16 + 8 * PP>(base, lane);
                }
            };
            using I0 = std::integral_constant<int, 0>; using I1 = std::integral_constant<int, 1>;
// eight K blocks (both pairs twice) without a branch
            auto full_pair = [&](auto pp_c, float s0, float s1) {
                constexpr int PP = decltype(pp_c)::value;
                tight_wait<8 * PP, 32>(base, par);
                __syncwarp();
                ptx::tc_fence_after();
                uint32_t r[32];
                ptx::tmem_ld_wait_32x32b_x32(t0 + 128 * PP, r);
                scale_accumulate<CONV>(acc, r, s0);
                ptx::tmem_ld_wait_32x32b_x32(t0 + 128 * PP + 64, r);
                ptx::tc_fence_before();
                arrive_lane0<16 + 8 * PP>(base, lane);
                scale_accumulate<CONV>(acc, r, s1);
            };
            int t = 0;
#pragma unroll 1
            for (; t + 8 <= n; t += 8) {
                const int k = t & 31;
                if (k == 0) {
                    sc = __fmul_rn(__half2float(__ushort_as_half(ha)), __half2float(__ushort_as_half(hb)));
                    fetch_scales(t + 32);
                }
                const float sk = __shfl_sync(0xffffffffu, sc, k + (lane & 7));     // lane l: K block k + l % 8
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    full_pair(I0{}, __shfl_sync(0xffffffffu, sk, 4 * q), __shfl_sync(0xffffffffu, sk, 4 * q + 1));
                    full_pair(I1{}, __shfl_sync(0xffffffffu, sk, 4 * q + 2), __shfl_sync(0xffffffffu, sk, 4 * q + 3));
                    par ^= 1u;
                }
            }
#pragma unroll 1
            for (; t < n; t += 4) {
                const int k = t & 31;
                if (k == 0) {
                    sc = __fmul_rn(__half2float(__ushort_as_half(ha)), __half2float(__ushort_as_half(hb)));
                    fetch_scales(t + 32);
                }
                pair(I0{}, k, n - t);
                pair(I1{}, k + 2, n - t - 2);
                par ^= 1u;
            }
            if (!blk_ok) continue;
            w.store(acc, (int64_t)rowblk * QB + lane, (int64_t)colblk * QB, rowblk, colblk, item.split, lane);
        }
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) atomicCAS(&g_gemm_error, 0, *abort_flag);
    if (warp == CONSUMER_WARPS + 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

