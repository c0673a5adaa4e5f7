// Q8_0 x Q8 product for many activation rows: the tensor cores deliver every 32-block's dot as fp32 (tcgen05 kind::f16, sm_100a).
//
// Same arithmetic per output as the int8 form (q8_gemm_tc.cu), bit for bit: quants are whole numbers up to 128, so fp16 holds them, their
// products and the 32-term sums (below 2^20) exactly, and acc = fma(d_w*d_x, dot, acc) runs over the blocks of a K segment in ascending
// order.  Stands in for the INT8-MMA kernels of the reference (mmq_q8_0_vmed_kernel / mmq_q8_0_v8_kernel, src/mmq_q8.cu:1795-2248).
//
// What bounds it: one multiplication (d_w*d_x) and one fma per (row, column, block) on the fp32 pipe, 128 a clock and SM: 512 cycles per
// 128 x 256 x 32 block, which takes about 1080.  In the int8 form the conversion of every dot to fp32 takes a third of the issue slots and half
// of another pipe's rate beside that (1160 cycles).  34816 x 5120 from a cold L2, 512 / 2048 rows: 431 / 1564 us in int8 form, 400 / 1455 here with
// the widening launch.
//
// Shape: 128 weight rows (MMA M) x 256 activation rows (MMA N) per CTA.  Twelve warps: warp 0 requests copies, warp 1 issues the MMAs,
// warps 2-3 widen a stage's int8 weights to fp16 in shared memory, warps 4-11 drain, each 32 rows x 128 columns of a block (224 registers by
// setmaxnreg: short of them the compiler copies registers around).  A stage is 64 k (two blocks): fp16 weights in a ring of their own,
// activations (widened once per launch into a workspace by act_widen_kernel) and both scales in another.  Tensor memory holds two blocks, the
// even and the odd one of a stage.  A stage's two blocks are straight lines of code with constant addresses (in a loop over blocks 4 percent
// more at 2048 rows), and a drain warp tests the next block's barrier before it rescales the last columns of the one at hand (without, in that loop, 3 more).
// Every wait is bounded; when one runs out the CTA raises the context's error flag, lets its copies land, frees its tensor memory and returns.
#include "qb_internal.h"
#include "tc_common.cuh"

#include <cuda_fp16.h>
#include <mutex>

namespace {
using namespace qbtc;

constexpr uint32_t MIN_CHUNKS = 4;                                      // of 128 columns in a K segment
constexpr uint32_t MT = 256, NSLOT = 2, NRAW = 2, NA = 3, NB = 4;         // activation rows of a tile; tensor-memory slots; rings: int8 weights, fp16 weights, rest
constexpr uint32_t CONV_WARPS = 2, EPI_WARPS = 8, NC = MT / 2, THREADS = 384;
constexpr uint32_t A_BYTES = 128 * 128, B_BYTES = MT * 128, XD_BYTES = 2 * MT * 4, WS_BYTES = 512;
constexpr uint32_t RAW_OFF = 0, A_OFF = NRAW * QB_REC_Q_BYTES, B_OFF = A_OFF + NA * A_BYTES, XD_OFF = B_OFF + NB * B_BYTES, WS_OFF = XD_OFF + NB * XD_BYTES;
constexpr uint32_t BAR_OFF = WS_OFF + NB * WS_BYTES, SMEM = BAR_OFF + 1024 + 1024;       // barriers, slack to align the base to 1024

// registers 4q .. 4q+3 of lane t: rows t/4 and t/4 + 8 (2 columns each), columns 8q + 2*(t%4) + {0, 1}
__device__ __forceinline__ void tmem_ld_16x256b_x4(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}
// tcgen05.wait::ld naming the registers of the loads it waits for: what consumes them is ordered after it by a data dependency.
__device__ __forceinline__ void tmem_wait_dep(uint32_t (&r)[16], uint32_t (&s)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(s[0]), "+r"(s[1]), "+r"(s[2]),
                   "+r"(s[3]), "+r"(s[4]), "+r"(s[5]), "+r"(s[6]), "+r"(s[7]), "+r"(s[8]), "+r"(s[9]), "+r"(s[10]), "+r"(s[11]),
                   "+r"(s[12]), "+r"(s[13]), "+r"(s[14]), "+r"(s[15]));
}
__device__ __forceinline__ f32x2 pair(const uint32_t (&v)[16], int i) { return pack2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])); }

// Four int8 to fp16, exactly: u = q + 128 is placed into the low bits of 1024.0, then 1152 is taken off.
__device__ __forceinline__ void widen4(uint32_t q, uint32_t &lo, uint32_t &hi) {
    const uint32_t u = q ^ 0x80808080u;
    const __half2 off = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));        // 1152
    uint32_t a = __byte_perm(u, 0x64646464u, 0x4140), b = __byte_perm(u, 0x64646464u, 0x4342);
    __half2 x = __hsub2(*reinterpret_cast<__half2 *>(&a), off), y = __hsub2(*reinterpret_cast<__half2 *>(&b), off);
    lo = *reinterpret_cast<uint32_t *>(&x);
    hi = *reinterpret_cast<uint32_t *>(&y);
}
__device__ __forceinline__ void widen16(const uint4 q, uint4 &a, uint4 &b) {
    widen4(q.x, a.x, a.y);
    widen4(q.y, a.z, a.w);
    widen4(q.z, b.x, b.y);
    widen4(q.w, b.z, b.w);
}

__global__ void __launch_bounds__(256) act_widen_kernel(const int8_t *__restrict__ q, __half *__restrict__ out, uint64_t pieces) {
    QB_PDL_ENTER();
    const uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= pieces) return;
    uint4 a, b;
    widen16(reinterpret_cast<const uint4 *>(q)[i], a, b);
    reinterpret_cast<uint4 *>(out)[2 * i] = a;
    reinterpret_cast<uint4 *>(out)[2 * i + 1] = b;
}

// Persistent: CTA b works on units b, b + gridDim.x, ...; a unit is (activation tile, K segment, 128-row weight tile).
__global__ void __launch_bounds__(THREADS, 1)
gemm_f16_kernel(const uint8_t *__restrict__ rec, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_xd, uint32_t K,
                uint32_t N, uint32_t M, float *__restrict__ part, uint32_t S, uint32_t tiles, uint32_t units, int *err_flag, unsigned long long *tl) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align1024(smem_raw);
    uint8_t *bar_mem = smem + BAR_OFF;
    const uint32_t base = smem_u32(smem), bars = smem_u32(bar_mem);
    const uint32_t raw_full = bars, raw_empty = raw_full + 8 * NRAW, a_full = raw_empty + 8 * NRAW, a_empty = a_full + 8 * NA;
    const uint32_t b_full = a_empty + 8 * NA, b_empty = b_full + 8 * NB, t_full = b_empty + 8 * NB, t_empty = t_full + 8 * NSLOT;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar_mem + 512);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(bar_mem + 516);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nchunks = K / 128;

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < NRAW; ++i) { mbar_init(raw_full + 8 * i, 1); mbar_init(raw_empty + 8 * i, CONV_WARPS); }
        for (uint32_t i = 0; i < NA; ++i) { mbar_init(a_full + 8 * i, CONV_WARPS); mbar_init(a_empty + 8 * i, 1); }
        for (uint32_t i = 0; i < NB; ++i) { mbar_init(b_full + 8 * i, 1); mbar_init(b_empty + 8 * i, 1 + EPI_WARPS); }   // MMA commit + every drain warp
        for (uint32_t i = 0; i < NSLOT; ++i) { mbar_init(t_full + 8 * i, 1); mbar_init(t_empty + 8 * i, EPI_WARPS); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    auto decode = [&](uint32_t u, uint32_t &tile, uint32_t &seg, uint32_t &m0, uint32_t &c_begin, uint32_t &n_it) {
        const uint32_t per_m = tiles * S, rem = u % per_m;
        m0 = (u / per_m) * MT;
        seg = rem / tiles;
        tile = rem % tiles;
        c_begin = tc_seg_begin(seg, S, nchunks);
        n_it = tc_seg_begin(seg + 1, S, nchunks) - c_begin;
    };

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == 0) {
            if (elect_one()) {
                if (tl) tl[blockIdx.x * 4 + 0] = qb_globaltimer();
                uint32_t g = 0, c = 0;                                  // stages of 64 k and chunks of 128 k so far
                bool ok = true, first = true;
                for (uint32_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
                    uint32_t tile, seg, m0, c_begin, n_it;
                    decode(u, tile, seg, m0, c_begin, n_it);
                    for (uint32_t it = 0; it < n_it && ok; ++it, ++c) {
                        const uint8_t *src = rec + ((size_t)tile * nchunks + c_begin + it) * QB_REC_BYTES;
                        const uint32_t rs = c % NRAW, rp = (c / NRAW) & 1;
                        if (!mbar_wait(raw_empty + 8 * rs, rp ^ 1, abort_flag)) { ok = false; break; }
                        mbar_expect_tx(raw_full + 8 * rs, QB_REC_Q_BYTES);
                        bulk_load(base + RAW_OFF + rs * QB_REC_Q_BYTES, src, QB_REC_Q_BYTES, raw_full + 8 * rs);
                        if (first) {                                    // the activations come from the preceding kernels
                            asm volatile("griddepcontrol.wait;" ::: "memory");
                            if (tl) tl[blockIdx.x * 4 + 1] = qb_globaltimer();
                            first = false;
                        }
                        for (uint32_t h = 0; h < 2; ++h, ++g) {
                            const uint32_t st = g % NB, ph = (g / NB) & 1, bar = b_full + 8 * st;
                            if (!mbar_wait(b_empty + 8 * st, ph ^ 1, abort_flag)) { ok = false; break; }
                            const int k0 = (int)((c_begin + it) * 128 + h * 64);
                            mbar_expect_tx(bar, B_BYTES + XD_BYTES + WS_BYTES);
                            tma_load_2d(base + B_OFF + st * B_BYTES, &map_x, k0, (int)m0, bar);
                            tma_load_2d(base + XD_OFF + st * XD_BYTES, &map_xd, (int)m0, k0 / 32, bar);
                            bulk_load(base + WS_OFF + st * WS_BYTES, src + QB_REC_Q_BYTES + h * WS_BYTES, WS_BYTES, bar);
                        }
                    }
                }
            }
        } else if (warp == 1) {
            if (elect_one()) {
                // instruction descriptor: D fp32, A = B = fp16, both K-major, N = MT, M = 128
                constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(MT >> 3) << 17) | ((128u >> 4) << 24);
                uint32_t g = 0;
                bool ok = true;
                for (uint32_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
                    uint32_t tile, seg, m0, c_begin, n_it;
                    decode(u, tile, seg, m0, c_begin, n_it);
                    for (uint32_t it = 0; it < 2 * n_it && ok; ++it, ++g) {
                        const uint32_t as = g % NA, ap = (g / NA) & 1, st = g % NB, ph = (g / NB) & 1;
                        if (!mbar_wait(b_full + 8 * st, ph, abort_flag) || !mbar_wait(a_full + 8 * as, ap, abort_flag)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t a_addr = base + A_OFF + as * A_BYTES, b_addr = base + B_OFF + st * B_BYTES;
#pragma unroll
                        for (int kb = 0; kb < 2; ++kb) {
                            if (!mbar_wait(t_empty + 8 * kb, (g & 1) ^ 1, abort_flag)) { ok = false; break; }
                            tc_fence_after();
#pragma unroll
                            for (int ks = 0; ks < 2; ++ks)
                                tc_mma_f16(tmem_base + kb * MT, smem_desc_sw128(a_addr + (kb * 2 + ks) * 32), smem_desc_sw128(b_addr + (kb * 2 + ks) * 32),
                                           idesc, (uint32_t)ks);
                            tc_commit(t_full + 8 * kb);
                        }
                        if (!ok) break;
                        tc_commit(a_empty + 8 * as);
                        tc_commit(b_empty + 8 * st);
                    }
                }
            }
        } else {
            // int8 -> fp16: a thread takes 16 weights of a row (a 16-byte piece of the swizzled record) and writes the two pieces of the
            // swizzled fp16 tile; the eight lanes of a shared-memory phase are eight rows, so neither side has bank conflicts
            const uint32_t r8 = lane & 7, pp = lane >> 3, half = warp - 2;
            uint32_t g = 0, c = 0;
            bool ok = true;
            for (uint32_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
                uint32_t tile, seg, m0, c_begin, n_it;
                decode(u, tile, seg, m0, c_begin, n_it);
                for (uint32_t it = 0; it < n_it && ok; ++it, ++c) {
                    const uint32_t rs = c % NRAW, rp = (c / NRAW) & 1;
                    if (!__all_sync(0xffffffffu, mbar_wait(raw_full + 8 * rs, rp, abort_flag))) { ok = false; break; }
                    for (uint32_t h = 0; h < 2; ++h, ++g) {
                        const uint32_t as = g % NA, ap = (g / NA) & 1;
                        if (!__all_sync(0xffffffffu, mbar_wait(a_empty + 8 * as, ap ^ 1, abort_flag))) { ok = false; break; }
                        const uint8_t *src = smem + RAW_OFF + rs * QB_REC_Q_BYTES + (half * 64 + r8) * 128 + (((h * 4 + pp) ^ r8) << 4);
                        uint8_t *dst = smem + A_OFF + as * A_BYTES + (half * 64 + r8) * 128;
                        const uint32_t d0 = (2 * pp ^ r8) << 4, d1 = ((2 * pp + 1) ^ r8) << 4;
#pragma unroll 4
                        for (int i = 0; i < 8; ++i) {
                            uint4 a, b;
                            widen16(*reinterpret_cast<const uint4 *>(src + i * 1024), a, b);
                            *reinterpret_cast<uint4 *>(dst + i * 1024 + d0) = a;
                            *reinterpret_cast<uint4 *>(dst + i * 1024 + d1) = b;
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");    // the MMA reads through the async proxy
                        __syncwarp();
                        if (lane == 0) mbar_arrive(a_full + 8 * as);
                    }
                    if (ok && lane == 0) mbar_arrive(raw_empty + 8 * rs);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        const uint32_t quarter = warp & 3, r0 = quarter * 32 + (lane >> 2), cw = ((warp - 4) >> 2) * NC, c0 = cw + 2 * (lane & 3);
        uint32_t g = 0;                                                 // stages so far
        bool ok = true, ready = false;
        for (uint32_t u = blockIdx.x; u < units && ok; u += gridDim.x) {
            uint32_t tile, seg, m0, c_begin, n_it;
            decode(u, tile, seg, m0, c_begin, n_it);
            f32x2 acc[NC / 8][4];                                       // [column pair][row]
#pragma unroll
            for (uint32_t i = 0; i < NC / 8; ++i)
#pragma unroll
                for (int p = 0; p < 4; ++p) acc[i][p] = pack2(0.0f, 0.0f);
            for (const uint32_t end = g + 2 * n_it; g < end; ++g) {
                const uint32_t st = g % NB;
#pragma unroll
                for (uint32_t kb = 0; kb < 2; ++kb) {
                    // (no way out of the loop on a failed wait: what follows then reads allocated memory, and the CTA's other waits fail at once)
                    if (!ready) ok = mbar_wait(t_full + 8 * kb, g & 1, abort_flag) && ok;
                    __syncwarp();
                    tc_fence_after();
                    // (the stage has landed: the slot barrier implies it)
                    const __half *wd = reinterpret_cast<const __half *>(smem + WS_OFF + st * WS_BYTES) + kb * 128 + r0;
                    const float *xd = reinterpret_cast<const float *>(smem + XD_OFF + st * XD_BYTES) + kb * MT + c0;
                    const uint32_t t = tmem_base + ((quarter * 32u) << 16) + kb * MT + cw;
                    f32x2 dw[4];
#pragma unroll
                    for (int p = 0; p < 4; ++p) { const float f = __half2float(wd[8 * p]); dw[p] = pack2(f, f); }
#pragma unroll
                    for (uint32_t h = 0; h < NC / 32; ++h) {
                        uint32_t va[16], vb[16];
                        tmem_ld_16x256b_x4(t + h * 32, va);
                        tmem_ld_16x256b_x4(t + (16u << 16) + h * 32, vb);
                        f32x2 x[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) x[q] = *reinterpret_cast<const f32x2 *>(xd + h * 32 + 8 * q);
                        tmem_wait_dep(va, vb);
                        if (h == NC / 32 - 1) {                         // the warp's part of the block is in registers
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) {
                                mbar_arrive(t_empty + 8 * kb);
                                if (kb) mbar_arrive(b_empty + 8 * st);
                            }
                            ready = (kb == 0 || g + 1 < end) && mbar_test(t_full + 8 * (kb ^ 1), (g + kb) & 1);
                        }
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            f32x2 (&a)[4] = acc[h * 4 + q];
                            a[0] = fma2(mul2(dw[0], x[q]), pair(va, 2 * q), a[0]);
                            a[1] = fma2(mul2(dw[1], x[q]), pair(va, 2 * q + 1), a[1]);
                            a[2] = fma2(mul2(dw[2], x[q]), pair(vb, 2 * q), a[2]);
                            a[3] = fma2(mul2(dw[3], x[q]), pair(vb, 2 * q + 1), a[3]);
                        }
                    }
                }
            }
            ok = __all_sync(0xffffffffu, ok);                           // (the outcome is the warp's)
            if (ok) {
                // one pointer that walks over the columns (with an index computed for each of them 2 percent more)
                const uint32_t row = tile * 128 + r0;
                float *o = part + ((size_t)seg * M + m0 + c0) * N + row;
#pragma unroll
                for (uint32_t i = 0; i < NC / 8; ++i) {
                    float v[4][2];
#pragma unroll
                    for (int p = 0; p < 4; ++p) unpack2(acc[i][p], v[p][0], v[p][1]);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        if (m0 + c0 + 8 * i + e < M) {
#pragma unroll
                            for (int p = 0; p < 4; ++p) if (row + 8 * p < N) o[8 * p] = v[p][e];
                        }
                        o += e ? 7 * (size_t)N : N;
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
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
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    }
}

// Tensor maps cached per (device, buffer, shape); emptied when the cache grows large.
struct MapKey {
    int dev; const void *p; uint32_t a, b;
    bool operator<(const MapKey &o) const { return std::tie(dev, p, a, b) < std::tie(o.dev, o.p, o.a, o.b); }
};
std::map<MapKey, CUtensorMap> g_x_maps, g_xd_maps;
std::mutex g_map_lock;
constexpr size_t MAP_CACHE_MAX = 4096;

}  // namespace

// Waves of units over the SMs times a unit's time, in us for 5120 columns: 100 of this form, its share of the widening launch included; of the int8 form
// 33 and 0.17 for each of its tile's rows (fitted to 34816 x 5120: 97 to 104 and 52 to 56).  What counts is their ratio: this form wins
// where it needs 1 / 1.83 of the waves that tiles of 128 rows need, 1 / 1.92 of those of 112.  Over nine weights of the 27B shape and of widths
// 2048 and 4096 at 16 row counts from 256 to 2048 the choice is within 2 percent of the faster form in 142 cases of 144 and within 3.3 in all.
// 34816 x 5120, int8 / this form: 256 rows 224 / 208 us, 330 rows 316 / 398, 512 rows 431 / 400, 640
// rows 533 / 591, 1000 rows 794 / 783, 2048 rows 1564 / 1455.
// Segments of fewer than four records keep the int8 form, which is one launch and fills its pipeline sooner.
bool qb_gemm_f16_wins(const qb_weight *w, uint32_t M, uint32_t S, uint32_t sms) {
    if (M < 256 || w->cols / 128 / S < MIN_CHUNKS) return false;
    const uint32_t tiles = w->rows_pad / 128 * S, m128 = (M + 127) / 128, width = ((M + m128 - 1) / m128 + 15) / 16 * 16;
    const uint32_t here = (tiles * ((M + MT - 1) / MT) + sms - 1) / sms, int8 = (tiles * m128 + sms - 1) / sms;
    return 100.0 * here < (33.0 + 0.17 * width) * int8;
}

int qb_launch_gemm_f16(qb_ctx *ctx, const qb_weight *w, const int8_t *q, const float *d, uint32_t M, void *work, float *part, uint32_t S,
                       uint32_t *grid_out) {
    const uint32_t K = w->cols, ld = qb_act_ld(M);
    const uint64_t pieces = (uint64_t)M * K / 16;
    QB_CUDA(qb_launch_pdl(ctx->stream, act_widen_kernel, dim3((uint32_t)((pieces + 255) / 256)), dim3(256), (size_t)0, q, (__half *)work, pieces));
    QB_LAUNCHED(ctx, "act_widen_kernel");
    QB_CUDA(cudaFuncSetAttribute(gemm_f16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    const MapKey kx{ctx->device, work, M, K}, kd{ctx->device, d, M, K};
    CUtensorMap map_x, map_d;
    {
        std::lock_guard<std::mutex> lock(g_map_lock);
        if (g_x_maps.size() > MAP_CACHE_MAX) g_x_maps.clear();
        if (g_xd_maps.size() > MAP_CACHE_MAX) g_xd_maps.clear();
        auto ix = g_x_maps.find(kx);
        if (ix == g_x_maps.end()) {
            CUtensorMap m;
            QB_TRY(qb_make_tmap_2d(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, work, K, M, (uint64_t)K * 2, 64, MT, CU_TENSOR_MAP_SWIZZLE_128B));
            ix = g_x_maps.emplace(kx, m).first;
        }
        auto id = g_xd_maps.find(kd);
        if (id == g_xd_maps.end()) {
            CUtensorMap m;
            QB_TRY(qb_make_tmap_2d(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, d, ld, K / 32, (uint64_t)ld * 4, MT, 2, CU_TENSOR_MAP_SWIZZLE_NONE));
            id = g_xd_maps.emplace(kd, m).first;
        }
        map_x = ix->second; map_d = id->second;
    }
    const uint32_t tiles = w->rows_pad / 128, units = tiles * S * ((M + MT - 1) / MT), grid = std::min<uint32_t>(units, (uint32_t)ctx->sm_count);
    const double bytes = (double)w->rows_pad * K / 32.0 * 34.0 + (double)M * K * 1.125 + (double)S * M * w->rows * 4.0;
    QB_CUDA(qb_launch_pdl(ctx->stream, gemm_f16_kernel, dim3(grid), dim3(THREADS), (size_t)SMEM, (const uint8_t *)w->rec, map_x, map_d, K, w->rows, M, part, S,
                          tiles, units, ctx->err_flag_dev, qb_timeline_slot(ctx, grid, bytes)));
    if (grid_out) *grid_out = grid;
    QB_LAUNCHED(ctx, "gemm_f16_kernel");
    return QB_OK;
}
