// Q8_0 x Q8 product on the 5th-generation tensor cores (tcgen05, sm_100a).
//
// Stands in for the INT8-MMA kernels of the reference (mmq_q8_0_vmed_kernel / mmq_q8_0_v8_kernel,
// src/mmq_q8.cu:1795-2248, mma.sync.m16n8k32.s8) with the same arithmetic per output: the exact int32
// dot of every 32-block, acc = fma(d_w*d_x, float(dot), acc) over the blocks of a K segment in
// ascending order, one partial sum per segment (bit-identical to the CUDA-core kernel of this library).
//
// Shape of the kernel ("swap-AB"): the 128 weight rows of a CTA are the MMA's M dimension, the
// activation rows are its N dimension (16..128), and one tcgen05.mma.kind::i8 (K = 32 bytes) covers
// exactly one Q8_0 block.  Every block therefore gets its OWN accumulator columns in tensor memory
// (never accumulated across blocks), and the epilogue warps drain them and apply the per-block scales
// in order.  The weight record of a stage (quants already in the swizzled operand order + scales)
// arrives as one 17 KB bulk copy, the activation tile and its scales by tensor-map TMA (128-byte
// swizzle), all through one mbarrier pipeline; the kernel is an HBM streaming kernel until the
// activation-row count reaches the hundreds.
//
// Warp roles: warp 0 = TMA producer, warp 1 = MMA issuer (owns the TMEM allocation), warps 2.. = epilogue
// (TMEM lane quarter = warp % 4; 4, 8, 12 or 16 warps by tile).  Every wait is bounded: when a wait runs out
// the CTA raises the context's error flag, lets its copies land, frees its TMEM and returns.
#include "qb_internal.h"
#include "tc_common.cuh"

#include <mutex>
#include <type_traits>

namespace {
using namespace qbtc;

// 16 lanes x 32, 16 or 8 columns: register 4j+i of lane t is row t/4 + 8*(i/2), column 8j + 2*(t%4) + i%2
__device__ __forceinline__ void tmem_ld_16x256b(uint32_t taddr, int32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_16x256b(uint32_t taddr, int32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_16x256b(uint32_t taddr, int32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_dep2(int32_t (&r)[8], int32_t (&s)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(s[0]), "+r"(s[1]), "+r"(s[2]),
                   "+r"(s[3]), "+r"(s[4]), "+r"(s[5]), "+r"(s[6]), "+r"(s[7]));
}
__device__ __forceinline__ void tmem_wait_dep2(int32_t (&r)[4], int32_t (&s)[4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(s[0]), "+r"(s[1]), "+r"(s[2]), "+r"(s[3]));
}
__device__ __forceinline__ void tmem_wait_dep2(int32_t (&r)[16], int32_t (&s)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(s[0]), "+r"(s[1]), "+r"(s[2]),
                   "+r"(s[3]), "+r"(s[4]), "+r"(s[5]), "+r"(s[6]), "+r"(s[7]), "+r"(s[8]), "+r"(s[9]), "+r"(s[10]), "+r"(s[11]),
                   "+r"(s[12]), "+r"(s[13]), "+r"(s[14]), "+r"(s[15]));
}

// MT = activation rows per tile (MMA N).  NLD = accumulator columns the epilogue reads (<= MT).
// A pipeline stage holds one weight record (17 KB, one bulk copy, already the swizzled operand image
// plus its scales), the activation tile (MT x 128 B, tensor-map TMA with the 128-byte swizzle) and
// the activation scales.  TMEM: every stage (MT <= 64) or half stage (MT > 64) has its own slot.
template <int MT, int NLD>
struct TcCfg {
    static constexpr int KPS = MT > 64 ? 2 : 4;              // 32-blocks per TMEM slot
    static constexpr int SPS = 4 / KPS;                        // slots per pipeline stage
    // Small tiles run two CTAs per SM (two independent producer/MMA/epilogue chains per SM: the per-stage
    // handshake chain of one CTA, not the memory system, limits a single chain to ~33 GB/s), so each CTA
    // takes half the tensor memory and half the shared memory.
    static constexpr int CTAS_PER_SM = MT == 16 ? 2 : 1;
    // Second launch bound.  Left unspecified, the compiler keeps several variants at 64 registers with spills inside
    // the drain loop (it assumes more resident CTAs than the shared memory allows); told the real residency it uses
    // 90-168 registers, with 106 bytes of spill stores left in the 16-column one and none in the others.  The 32-column
    // variant measured faster with the default (64 registers, 4 bytes of spill stores), so it keeps it (0).
    static constexpr int MIN_CTAS = MT == 32 ? 0 : CTAS_PER_SM;
    static constexpr int NSLOT = 512 / CTAS_PER_SM / (KPS * MT);
    static constexpr int TMEM_COLS = 512 / CTAS_PER_SM;
    static constexpr int B_OFF = (int)QB_REC_BYTES;            // 17 * 1024: the activation tile stays 1024-aligned
    static constexpr int B_BYTES = MT * 128;
    static constexpr int XD_OFF = B_OFF + B_BYTES;
    static constexpr int XD_BYTES = 4 * MT * 4;
    static constexpr int TX_BYTES = (int)QB_REC_BYTES + B_BYTES + XD_BYTES;
    static constexpr int STAGE = (XD_OFF + XD_BYTES + 1023) / 1024 * 1024;
    static constexpr int BAR_BYTES = 1024;
    // fused SwiGLU (small tiles only): the up half of a tile's rows hands its sums to the gate half, two buffers
    static constexpr int EX_BYTES = MT == 16 ? 2 * NLD * 64 * 4 : 0;
    static constexpr int NST_FIT = (232448 / CTAS_PER_SM - BAR_BYTES - EX_BYTES - 2048) / STAGE;
    static constexpr int NST = NST_FIT > 8 ? 8 : NST_FIT;
    static constexpr int TOTAL = STAGE * NST + BAR_BYTES + EX_BYTES + 1024;   // + slack to align the base to 1024
    static constexpr int CH = NLD < 16 ? NLD : 16;               // columns per tcgen05.ld
    // The producer and issuer threads are elected (steps of 1 to 4 requests take 1 to 4 percent less than with lane 0), except in the
    // form for 5 to 8 rows, where lane 0 is the faster one (steps of 5 to 8 requests of eight 27B layers: 0.5 to 1.2 percent less).
    static constexpr bool ELECT = NLD != 8;
    // Epilogue warps: four for tiles of 16 rows (one per TMEM lane quarter), twelve at 48 rows, sixteen at 64 and eight at the others
    // (three / four / two per quarter, each taking a slice of the activation columns).
    static constexpr int EPI_WARPS = MT == 64 ? 16 : MT == 48 ? 12 : MT >= 32 ? 8 : 4;
    static constexpr int THREADS = 64 + 32 * EPI_WARPS;
    static constexpr int NC = NLD / (EPI_WARPS / 4);             // accumulator columns per epilogue thread
};

// Persistent kernel: CTA b works on units b, b + gridDim.x, ...; a unit is (activation tile, K segment,
// 128-row weight tile).  The TMA / MMA / TMEM pipeline keeps running across unit boundaries.
template <int MT, int NLD>
__global__ void __launch_bounds__((TcCfg<MT, NLD>::THREADS), (TcCfg<MT, NLD>::MIN_CTAS))
gemm_tc_kernel(const uint8_t *__restrict__ rec, const __grid_constant__ CUtensorMap map_xq,
               const __grid_constant__ CUtensorMap map_xd, uint32_t K, uint32_t N, uint32_t M, float *__restrict__ part,
               uint32_t S, uint32_t tiles, uint32_t units, int *err_flag, unsigned long long *tl,
               const __grid_constant__ QbGemmPush push, const QbGemmSwiglu swz) {
    using C = TcCfg<MT, NLD>;
    constexpr uint32_t NST = C::NST, NSLOT = C::NSLOT;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align1024(smem_raw);
    uint8_t *bar_mem = smem + (size_t)C::STAGE * NST;
    // barrier layout: full[NST], empty[NST], tmem_full[NSLOT], tmem_empty[NSLOT]
    const uint32_t bar_full = smem_u32(bar_mem), bar_empty = bar_full + 8 * NST;
    const uint32_t bar_tfull = bar_empty + 8 * NST, bar_tempty = bar_tfull + 8 * NSLOT;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar_mem + 8 * (2 * NST + 2 * NSLOT));
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    const uint32_t bar_ex = smem_u32(bar_mem + 512);                  // two "up half stored" barriers (fused SwiGLU)
    float *ex = reinterpret_cast<float *>(bar_mem + C::BAR_BYTES);    // [2][NLD][64]

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nchunks = K / 128;
    constexpr uint32_t tmem_cols = C::TMEM_COLS;

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < NST; ++i) {
            mbar_init(bar_full + 8 * i, 1);
            mbar_init(bar_empty + 8 * i, 1 + C::EPI_WARPS);   // MMA commit + one lane of every epilogue warp
        }
        for (uint32_t i = 0; i < NSLOT; ++i) {
            mbar_init(bar_tfull + 8 * i, 1);
            mbar_init(bar_tempty + 8 * i, C::EPI_WARPS);
        }
        mbar_init(bar_ex, 2);
        mbar_init(bar_ex + 8, 2);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the consumer of the partials may be scheduled already

    // unit -> (m tile, segment, row tile); consecutive units of a CTA differ in the row tile
    auto decode = [&](uint32_t u, uint32_t &tile, uint32_t &seg, uint32_t &m0, uint32_t &c_begin, uint32_t &n_it) {
        const uint32_t per_m = tiles * S;
        m0 = (u / per_m) * MT;
        const uint32_t rem = u % per_m;
        seg = rem / tiles;
        tile = rem % tiles;
        c_begin = tc_seg_begin(seg, S, nchunks);
        n_it = tc_seg_begin(seg + 1, S, nchunks) - c_begin;
    };

    if (warp == 0) {
        if (C::ELECT ? elect_one() : lane == 0) {
            // Stage cursor over this CTA's units.  The launch is programmatically serialised behind the kernel
            // that produces the activations: the weight records of the first NST stages (which depend on nothing)
            // are requested at once, then the CTA waits for the preceding grid and only then requests activations.
            struct Cursor { uint32_t u, it, n_it, tile, m0, c_begin; bool valid; };
            auto start = [&](uint32_t u) {
                Cursor c; c.u = u; c.it = 0; c.valid = u < units; c.n_it = 0; c.tile = c.m0 = c.c_begin = 0;
                if (c.valid) { uint32_t seg; decode(u, c.tile, seg, c.m0, c.c_begin, c.n_it); }
                return c;
            };
            auto next = [&](Cursor &c) {
                if (++c.it >= c.n_it) c = start(c.u + gridDim.x);
            };
            auto load_w = [&](const Cursor &c, uint32_t st) {
                const uint32_t base = smem_u32(smem + (size_t)st * C::STAGE), full = bar_full + 8 * st;
                mbar_expect_tx(full, C::TX_BYTES);
                bulk_load(base, rec + ((size_t)c.tile * nchunks + c.c_begin + c.it) * QB_REC_BYTES, QB_REC_BYTES, full);
            };
            auto load_x = [&](const Cursor &c, uint32_t st) {
                const uint32_t base = smem_u32(smem + (size_t)st * C::STAGE), full = bar_full + 8 * st;
                const int k0 = (int)((c.c_begin + c.it) * 128);
                tma_load_2d(base + C::B_OFF, &map_xq, k0, (int)c.m0, full);
                tma_load_2d(base + C::XD_OFF, &map_xd, (int)c.m0, k0 / 32, full);
            };
            if (tl) tl[blockIdx.x * 4 + 0] = qb_globaltimer();
            Cursor head = start(blockIdx.x), c = head;
            uint32_t npre = 0;
            for (; npre < NST && c.valid; ++npre, next(c)) load_w(c, npre);
            asm volatile("griddepcontrol.wait;" ::: "memory");
            if (tl) tl[blockIdx.x * 4 + 1] = qb_globaltimer();
            c = head;
            for (uint32_t g = 0; g < npre; ++g, next(c)) load_x(c, g);
            for (uint32_t git = npre; c.valid; ++git, next(c)) {
                const uint32_t st = git % NST, ph = (git / NST) & 1;
                if (!mbar_wait(bar_empty + 8 * st, ph ^ 1, abort_flag)) break;
                load_w(c, st);
                load_x(c, st);
            }
        }
    } else if (warp == 1) {
        if (C::ELECT ? elect_one() : lane == 0) {
            // instruction descriptor: D = s32, A = B = signed 8-bit, both K-major, N = MT, M = 128
            constexpr uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(MT >> 3) << 17) | ((128u >> 4) << 24);
            uint32_t git = 0, j = 0;
            bool ok = true;
            for (uint32_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
                uint32_t tile, seg, m0, c_begin, n_it;
                decode(u, tile, seg, m0, c_begin, n_it);
                for (uint32_t it = 0; it < n_it && ok; ++it, ++git) {
                    const uint32_t st = git % NST, ph = (git / NST) & 1;
                    if (!mbar_wait(bar_full + 8 * st, ph, abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + (size_t)st * C::STAGE), b_addr = a_addr + C::B_OFF;
                    for (int sp = 0; sp < C::SPS; ++sp, ++j) {
                        const uint32_t slot = j % NSLOT, sph = (j / NSLOT) & 1;
                        if (!mbar_wait(bar_tempty + 8 * slot, sph ^ 1, abort_flag)) { ok = false; break; }
                        tc_fence_after();
#pragma unroll
                        for (int kl = 0; kl < C::KPS; ++kl) {
                            const int kb = sp * C::KPS + kl;
                            tc_mma_i8(tmem_base + slot * (C::KPS * MT) + kl * MT, smem_desc_sw128(a_addr + kb * 32),
                                      smem_desc_sw128(b_addr + kb * 32), idesc);
                        }
                        tc_commit(bar_tfull + 8 * slot);
                    }
                    if (ok) tc_commit(bar_empty + 8 * st);
                }
            }
        }
    } else {
        const uint32_t quarter = warp & 3;                     // TMEM lanes [32*quarter, +32)
        const uint32_t r = quarter * 32 + lane;                // weight row inside the tile
        uint32_t git = 0, j = 0;
        bool ok = true;
        for (uint32_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
            uint32_t tile, seg, m0, c_begin, n_it;
            decode(u, tile, seg, m0, c_begin, n_it);
            float acc[C::NC];
#pragma unroll
            for (int i = 0; i < C::NC; ++i) acc[i] = 0.0f;
            if constexpr (NLD <= 16) {
                // Small activation tiles (the HBM-bound regime): the scales of a stage are copied to registers
                // as soon as the stage has landed and the stage is released at once, one stage ahead of the
                // TMEM work, so the producer never waits for the accumulator drain.
                float dw_n[4], dx_n[4][NLD];
                auto fetch_scales = [&](uint32_t g) -> bool {
                    const uint32_t st = g % NST, ph = (g / NST) & 1;
                    if (!__all_sync(0xffffffffu, mbar_wait(bar_full + 8 * st, ph, abort_flag))) return false;
                    const uint8_t *stage = smem + (size_t)st * C::STAGE;
                    const __half *wd = reinterpret_cast<const __half *>(stage + QB_REC_Q_BYTES);
                    const float *xd = reinterpret_cast<const float *>(stage + C::XD_OFF);
#pragma unroll
                    for (int kb = 0; kb < 4; ++kb) {
                        dw_n[kb] = __half2float(wd[kb * 128 + r]);
#pragma unroll
                        for (int i = 0; i < NLD; ++i) dx_n[kb][i] = xd[kb * MT + i];
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_empty + 8 * st);
                    return true;
                };
                if (n_it > 0 && !fetch_scales(git)) ok = false;
                for (uint32_t it = 0; it < n_it && ok; ++it, ++git, ++j) {
                    float sc[4][NLD];
#pragma unroll
                    for (int kb = 0; kb < 4; ++kb)
#pragma unroll
                        for (int i = 0; i < NLD; ++i) sc[kb][i] = __fmul_rn(dw_n[kb], dx_n[kb][i]);
                    if (it + 1 < n_it && !fetch_scales(git + 1)) { ok = false; break; }
                    const uint32_t slot = j % NSLOT, sph = (j / NSLOT) & 1;      // one slot per stage here
                    if (!__all_sync(0xffffffffu, mbar_wait(bar_tfull + 8 * slot, sph, abort_flag))) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t taddr = tmem_base + ((quarter * 32u) << 16) + slot * (4 * MT);
                    int32_t v[4][NLD];
#pragma unroll
                    for (int kb = 0; kb < 4; ++kb) tmem_ld<NLD>(taddr + kb * MT, v[kb]);
                    tmem_ld_wait();
#pragma unroll
                    for (int kb = 0; kb < 4; ++kb)
#pragma unroll
                        for (int i = 0; i < NLD; ++i) acc[i] = __fmaf_rn(sc[kb][i], (float)v[kb][i], acc[i]);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_tempty + 8 * slot);
                }
            } else if constexpr (MT <= 64) {
                // Middling activation tiles: this warp drains columns [c_base, c_base + NC) of its lane quarter.  The
                // TMEM loads are software-pipelined: the next 16 columns are in flight while the current 16 are
                // rescaled.
                constexpr int NC = C::NC, NCH = NC / 16;                // 16-column chunks per 32-block
                const uint32_t c_base = ((warp - 2) >> 2) * NC;
                f32x2 acc2[NC / 2];                                     // column pairs, packed arithmetic
#pragma unroll
                for (int i = 0; i < NC / 2; ++i) acc2[i] = pack2(0.0f, 0.0f);
                for (uint32_t it = 0; it < n_it && ok; ++it, ++git) {
                    // The stage's own barrier is not waited for: the MMAs whose completion the slot barrier reports were
                    // issued after the stage had landed, and a wait that has nothing to wait for still costs this warp a
                    // barrier round trip per stage (the drain is a chain of such latencies).
                    const uint32_t st = git % NST;
                    const uint8_t *stage = smem + (size_t)st * C::STAGE;
                    const __half *wd = reinterpret_cast<const __half *>(stage + QB_REC_Q_BYTES);
                    const float *xd = reinterpret_cast<const float *>(stage + C::XD_OFF) + c_base;
                    for (int sp = 0; sp < C::SPS; ++sp, ++j) {
                        const uint32_t slot = j % NSLOT, sph = (j / NSLOT) & 1;
                        // warp-uniform results: the TMEM loads below are .aligned
                        if (!__all_sync(0xffffffffu, mbar_wait(bar_tfull + 8 * slot, sph, abort_flag))) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t tbase = tmem_base + ((quarter * 32u) << 16) + slot * (C::KPS * MT) + c_base;
                        int32_t v[2][16];
                        tmem_ld<16>(tbase, v[0]);
#pragma unroll
                        for (int q = 0; q < C::KPS * NCH; ++q) {
                            const int kl = q / NCH, c0 = (q % NCH) * 16, kb = sp * C::KPS + kl;
                            tmem_ld_wait16(v[q & 1]);
                            if (q + 1 < C::KPS * NCH) tmem_ld<16>(tbase + ((q + 1) / NCH) * MT + ((q + 1) % NCH) * 16, v[(q + 1) & 1]);
                            const float dw = __half2float(wd[kb * 128 + r]);
                            const f32x2 dw2 = pack2(dw, dw);
                            // four scales per shared-memory load, read as the two packed pairs the arithmetic takes (no repacking)
                            const ulonglong2 *xd4 = reinterpret_cast<const ulonglong2 *>(xd + kb * MT + c0);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const ulonglong2 x4 = xd4[i];
                                acc2[c0 / 2 + 2 * i] = fma2(mul2(dw2, x4.x), pack2((float)v[q & 1][4 * i], (float)v[q & 1][4 * i + 1]), acc2[c0 / 2 + 2 * i]);
                                acc2[c0 / 2 + 2 * i + 1] = fma2(mul2(dw2, x4.y), pack2((float)v[q & 1][4 * i + 2], (float)v[q & 1][4 * i + 3]), acc2[c0 / 2 + 2 * i + 1]);
                            }
                        }
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_tempty + 8 * slot);
                    }
                    if (ok) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_empty + 8 * st);
                    }
                }
#pragma unroll
                for (int i = 0; i < NC / 2; ++i) unpack2(acc2[i], acc[2 * i], acc[2 * i + 1]);
            } else {
                // Tiles of 80 to 128 rows.  The 16x256b loads give a thread four rows x every fourth pair of columns, so it reads NC / 4 activation scales
                // per block and not NC: a scale that every lane reads costs its full width in shared-memory wavefronts (13 M of them in a
                // 17408 x 5120 x 128 product with the 32x32b loads, which give one row x all columns).  Eight warps of half the columns; with 16 warps
                // of 32 a tile of 128 takes 1.15 times as long, at 64 rows and below there is no gain.  A slot is one straight line of code: the
                // compiler then starts the next chunk's loads before it rescales the one at hand, which branches that skip the columns beyond the
                // last row prevent (34816 x 5120 with 128 rows 125 us, with such branches 163).
                // A warp tests the next slot's barrier before it rescales the last columns of the one at hand, and a stage's slots are unrolled (34816 x 5120,
                // 70 / 96 / 128 rows: 100 / 117 / 127 us without, 93 / 102 / 121 with).  Not at 112 rows: there it gives tall weights 1 to 2 percent
                // (34816 x 5120 with 331 rows 316.4 / 312.3) and costs short K segments 2 to 6 (4096 x 4096 in eight of 512, 331 rows: 52.3 / 54.3;
                // 12288 x 2048 in three, 224 rows: 46.1 / 48.1).
                constexpr int NC = C::NC;
                constexpr bool AHEAD = MT != 112;
                bool ready = false;
                const uint32_t r0 = quarter * 32 + (lane >> 2), cw = ((warp - 2) >> 2) * NC, c0 = cw + 2 * (lane & 3);
                f32x2 a2[NC / 8][4];                                    // [column pair][row]
#pragma unroll
                for (int i = 0; i < NC / 8; ++i)
#pragma unroll
                    for (int p = 0; p < 4; ++p) a2[i][p] = pack2(0.0f, 0.0f);
                for (uint32_t it = 0; it < n_it && ok; ++it, ++git) {
                    const uint32_t st = git % NST;                      // (landed: the slot barrier implies it)
                    const uint8_t *stage = smem + (size_t)st * C::STAGE;
                    const __half *wd = reinterpret_cast<const __half *>(stage + QB_REC_Q_BYTES) + r0;
                    const float *xd = reinterpret_cast<const float *>(stage + C::XD_OFF) + c0;
#pragma unroll(AHEAD ? C::SPS : 1)
                    for (int sp = 0; sp < C::SPS; ++sp, ++j) {
                        const uint32_t slot = AHEAD && NSLOT == C::SPS ? (uint32_t)sp : j % NSLOT, sph = (j / NSLOT) & 1;
                        if constexpr (AHEAD) {
                            // (a lane's own test may have come too early; the outcome is the warp's.  No way out on a failed wait, which would break the straight
                            // line: to the end of the stage the warp reads tensor memory that is allocated and shared memory that is its own, the
                            // abort flag lets every other wait fail at once, and nothing is stored once ok is false.)
                            const bool full = ready || mbar_wait(bar_tfull + 8 * slot, sph, abort_flag);
                            ok = __all_sync(0xffffffffu, full) && ok;
                        } else if (!__all_sync(0xffffffffu, mbar_wait(bar_tfull + 8 * slot, sph, abort_flag))) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t t = tmem_base + ((quarter * 32u) << 16) + slot * (C::KPS * MT) + cw;
#pragma unroll
                        for (int kl = 0; kl < C::KPS; ++kl) {
                            const int kb = sp * C::KPS + kl;
                            f32x2 dw[4];
#pragma unroll
                            for (int p = 0; p < 4; ++p) { const float f = __half2float(wd[kb * 128 + 8 * p]); dw[p] = pack2(f, f); }
                            // 4, 2 or 1 groups of 8 columns from group h on
                            auto chunk = [&](auto groups, int h) {
                                constexpr int G = decltype(groups)::value;
                                int32_t va[4 * G], vb[4 * G];
                                tmem_ld_16x256b(t + kl * MT + h * 8, va);
                                tmem_ld_16x256b(t + (16u << 16) + kl * MT + h * 8, vb);
                                f32x2 x[G];
#pragma unroll
                                for (int q = 0; q < G; ++q) x[q] = *reinterpret_cast<const f32x2 *>(xd + kb * MT + (h + q) * 8);
                                tmem_wait_dep2(va, vb);
                                if (h + G == NC / 8 && kl == C::KPS - 1) {        // the whole slot is in registers
                                    tc_fence_before();
                                    __syncwarp();
                                    if (lane == 0) mbar_arrive(bar_tempty + 8 * slot);
                                    if constexpr (AHEAD)
                                        ready = (sp + 1 < C::SPS || it + 1 < n_it) && mbar_test(bar_tfull + 8 * ((j + 1) % NSLOT), ((j + 1) / NSLOT) & 1);
                                }
#pragma unroll
                                for (int q = 0; q < G; ++q) {
                                    f32x2 (&a)[4] = a2[h + q];
                                    a[0] = fma2(mul2(dw[0], x[q]), pack2((float)va[4 * q], (float)va[4 * q + 1]), a[0]);
                                    a[1] = fma2(mul2(dw[1], x[q]), pack2((float)va[4 * q + 2], (float)va[4 * q + 3]), a[1]);
                                    a[2] = fma2(mul2(dw[2], x[q]), pack2((float)vb[4 * q], (float)vb[4 * q + 1]), a[2]);
                                    a[3] = fma2(mul2(dw[3], x[q]), pack2((float)vb[4 * q + 2], (float)vb[4 * q + 3]), a[3]);
                                }
                            };
#pragma unroll
                            for (int h = 0; h + 4 <= NC / 8; h += 4) chunk(std::integral_constant<int, 4>(), h);
                            if constexpr (NC / 8 % 4 >= 2) chunk(std::integral_constant<int, 2>(), NC / 32 * 4);
                            if constexpr (NC / 8 % 2 == 1) chunk(std::integral_constant<int, 1>(), NC / 8 - 1);
                        }
                    }
                    if (ok) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_empty + 8 * st);
                    }
                }
                if (ok) {
#pragma unroll
                    for (int i = 0; i < NC / 4; ++i) {
                        const uint32_t m = m0 + c0 + 8 * (i / 2) + (i & 1);
                        if (m >= M) continue;
#pragma unroll
                        for (int p = 0; p < 4; ++p) {
                            const uint32_t row = tile * 128 + r0 + 8 * p;
                            if (row >= N) continue;
                            float lo, hi;
                            unpack2(a2[i / 2][p], lo, hi);
                            const float val = (i & 1) ? hi : lo;
                            const size_t o = ((size_t)seg * M + m) * N + row;
                            if (push.n == 0) part[o] = val;
                            else for (uint32_t d = 0; d < push.n; ++d) push.dst[d][o] = val;
                        }
                    }
                }
                continue;
            }
            if constexpr (MT == 16) {
                if (swz.q != nullptr) {
                    // fused SwiGLU: rows 64..127 of the tile are the up rows of the hidden indices whose gate rows are
                    // rows 0..63: the up warps hand their sums over, the gate warps finish (a warp = one 32-block)
                    const uint32_t n_unit = (u - blockIdx.x) / gridDim.x, buf = n_unit & 1, exph = (n_unit >> 1) & 1;
                    float *exb = ex + buf * (NLD * 64);
                    if (quarter >= 2) {
                        if (ok) {
#pragma unroll
                            for (int i = 0; i < NLD; ++i) exb[i * 64 + (r - 64)] = acc[i];
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_ex + 8 * buf);          // arrives also when aborting: nobody waits in vain
                    } else {
                        if (!__all_sync(0xffffffffu, mbar_wait(bar_ex + 8 * buf, exph, abort_flag))) ok = false;
                        if (ok) {
                            const uint32_t hidx = tile * 64 + r;               // hidden index of this thread's gate row
#pragma unroll
                            for (int i = 0; i < NLD; ++i) {
                                const uint32_t m = m0 + i;
                                if (m < M)                                       // warp-uniform
                                    quant_block_store(qb_swiglu(acc[i], exb[i * 64 + r]), (int)lane, swz.q + (size_t)m * swz.q_pitch + (hidx & ~31u),
                                                      swz.d + (size_t)(hidx >> 5) * swz.d_ld + m);
                            }
                        }
                    }
                    continue;
                }
            }
            const uint32_t row = tile * 128 + r;
            if (ok && row < N) {
#pragma unroll
                for (int i = 0; i < C::NC; ++i) {
                    const uint32_t m = m0 + (C::EPI_WARPS > 4 ? ((warp - 2) >> 2) * C::NC : 0u) + i;
                    if (m < M) {
                        const size_t o = ((size_t)seg * M + m) * N + row;
                        if (push.n == 0) part[o] = acc[i];
                        else for (uint32_t p = 0; p < push.n; ++p) push.dst[p][o] = acc[i];
                    }
                }
            }
        }
        if (push.n) __threadfence_system();     // this thread's partial sums are visible to every GPU before the CTA signals
    }
    tc_fence_before();
    __syncthreads();
    if (push.n && threadIdx.x == 0) {
        __threadfence_system();
        for (uint32_t p = 0; p < push.n; ++p) atomicAdd_system(push.counter[p], 1u);
    }
    if (tl && threadIdx.x == 0) {
        tl[blockIdx.x * 4 + 2] = qb_globaltimer();
        uint32_t smid;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
        tl[blockIdx.x * 4 + 3] = smid;
    }
    if (*abort_flag) {
        if (threadIdx.x == 0) atomicExch(err_flag, 1000 + (int)(blockIdx.x % 1000));
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);      // let this CTA's copies in flight land
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}

// Tensor maps of the activation buffers, cached per (device, buffer, shape): the engine reuses a handful of buffers,
// the op-level entry points may see many, so the cache is emptied when it grows large.  One lock for both maps.
struct MapKey {
    int dev; const void *p; uint32_t a, b, c;
    bool operator<(const MapKey &o) const { return std::tie(dev, p, a, b, c) < std::tie(o.dev, o.p, o.a, o.b, o.c); }
};
std::map<MapKey, CUtensorMap> g_xq_maps, g_xd_maps;
std::mutex g_map_lock;
constexpr size_t MAP_CACHE_MAX = 4096;

template <int MT, int NLD>
int launch_tc(qb_ctx *ctx, const qb_weight *w, const int8_t *q, const float *d, uint32_t M, float *part, uint32_t S,
              const QbGemmPush *push, uint32_t *grid_out, const QbGemmSwiglu *swiglu) {
    using C = TcCfg<MT, NLD>;
    // the attribute belongs to the current device: set on every launch (a process may drive several GPUs)
    QB_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<MT, NLD>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::TOTAL));
    const uint32_t K = w->cols, ld = qb_act_ld(M);
    MapKey kq{ctx->device, q, M, K, (uint32_t)MT}, kd{ctx->device, d, M, K, (uint32_t)MT};
    CUtensorMap map_q, map_d;
    {
        std::lock_guard<std::mutex> lock(g_map_lock);
        if (g_xq_maps.size() > MAP_CACHE_MAX) g_xq_maps.clear();
        if (g_xd_maps.size() > MAP_CACHE_MAX) g_xd_maps.clear();
        auto iq = g_xq_maps.find(kq);
        if (iq == g_xq_maps.end()) {
            CUtensorMap mq;
            QB_TRY(qb_make_tmap_2d(&mq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, q, K, M, K, 128, MT, CU_TENSOR_MAP_SWIZZLE_128B));
            iq = g_xq_maps.emplace(kq, mq).first;
        }
        auto id = g_xd_maps.find(kd);
        if (id == g_xd_maps.end()) {
            CUtensorMap md;
            QB_TRY(qb_make_tmap_2d(&md, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, d, ld, K / 32, (uint64_t)ld * 4, MT, 4, CU_TENSOR_MAP_SWIZZLE_NONE));
            id = g_xd_maps.emplace(kd, md).first;
        }
        map_q = iq->second; map_d = id->second;
    }
    const uint32_t tiles = w->rows_pad / 128;
    const uint32_t units = tiles * S * ((M + MT - 1) / MT);
    const uint32_t grid = std::min<uint32_t>(units, (uint32_t)ctx->sm_count * C::CTAS_PER_SM);
    const size_t smem_bytes = C::TOTAL;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(C::THREADS);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attrs[1];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // may start while the previous kernel drains
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = 1;
    QB_CUDA(cudaLaunchKernelEx(&cfg, gemm_tc_kernel<MT, NLD>, (const uint8_t *)w->rec, map_q, map_d, K, w->rows, M, part, S,
                               tiles, units, ctx->err_flag_dev, qb_timeline_slot(ctx, grid, (double)w->rows_pad * K / 32.0 * 34.0 + (double)M * K * 1.125 + (double)S * M * w->rows * 4.0), push ? *push : QbGemmPush(),
                               swiglu ? *swiglu : QbGemmSwiglu()));
    if (grid_out) *grid_out = grid;
    QB_LAUNCHED(ctx, "gemm_tc_kernel");
    return QB_OK;
}

}  // namespace

bool qb_gemm_tc_supported(const qb_weight *w, uint32_t M) {
    return w->rec != nullptr && M >= 1 && w->cols % 128 == 0;
}

int qb_launch_gemm_tc(qb_ctx *ctx, const qb_weight *w, const int8_t *q, const float *d, uint32_t M, float *part, uint32_t S,
                      const QbGemmPush *push, uint32_t *grid_out, const QbGemmSwiglu *swiglu, const QbGemmWork &work) {
    QB_REQUIRE(!swiglu || (M <= 16 && S == 1 && w->rows % 128 == 0 && w->cols / 128 > 8 && swiglu->q && swiglu->d),
               "gemm: the fused SwiGLU needs M <= 16, one K segment, whole 128-row tiles and K > 1024");
    QB_REQUIRE(M > 0 && S > 0 && S <= w->cols / 128, "gemm: bad M=%u or ksplit=%u", M, S);
    QB_REQUIRE(((uintptr_t)q & 15) == 0 && ((uintptr_t)d & 15) == 0, "gemm: activation buffers must be 16-byte aligned");
    if (M <= 4) return launch_tc<16, 4>(ctx, w, q, d, M, part, S, push, grid_out, swiglu);
    if (M <= 8) return launch_tc<16, 8>(ctx, w, q, d, M, part, S, push, grid_out, swiglu);
    if (M <= 16) return launch_tc<16, 16>(ctx, w, q, d, M, part, S, push, grid_out, swiglu);
    if (M <= 32) return launch_tc<32, 32>(ctx, w, q, d, M, part, S, push, grid_out, swiglu);
    if (M <= 48) return launch_tc<48, 48>(ctx, w, q, d, M, part, S, push, grid_out, swiglu);
    if (M <= 64) return launch_tc<64, 64>(ctx, w, q, d, M, part, S, push, grid_out, swiglu);
    if (!push && work.bytes >= (size_t)M * w->cols * 2 && ((uintptr_t)work.p & 15) == 0 && qb_gemm_f16_wins(w, M, S, (uint32_t)ctx->sm_count))
        return qb_launch_gemm_f16(ctx, w, q, d, M, work.p, part, S, grid_out);
    // From 65 rows on the tile is as wide as the rows divide evenly over as few tiles as 128 columns allow, in steps of 16 (331 rows: three tiles of
    // 112): every column of a tile costs drain time, whether it holds a row or not.  34816 x 5120 from a cold L2, tiles of 128 / as wide as needed,
    // neither with the next slot tested ahead: 65 rows 123 / 100 us, 100 rows 125 / 115, 160 rows 232 / 187, 331 rows 343 / 313 (now 90, 114, 169, 316).
    // For the same reason 48 columns between 32 and 64 (48 rows 70 / 65.5 us).
    const uint32_t m_tiles = (M + 127) / 128, width = ((M + m_tiles - 1) / m_tiles + 15) / 16 * 16;
    if (width == 80) return launch_tc<80, 80>(ctx, w, q, d, M, part, S, push, grid_out, swiglu);
    if (width == 96) return launch_tc<96, 96>(ctx, w, q, d, M, part, S, push, grid_out, swiglu);
    if (width == 112) return launch_tc<112, 112>(ctx, w, q, d, M, part, S, push, grid_out, swiglu);
    return launch_tc<128, 128>(ctx, w, q, d, M, part, S, push, grid_out, swiglu);
}
