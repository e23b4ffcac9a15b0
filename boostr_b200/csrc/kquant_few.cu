// Quantized matmul of the K-quants for 9 ... 63 activation rows with the bits of boostr's CPU path
// (src/quant/cpu/kernels/quant_matmul.rs:107-135): activations quantised to Q8_K (quantize_act_q8k.rs:26-98), per 256-block
// (d * d8) * isum - (dmin * d8) * summs with exact integer sums (fused_q4k_q8k_dot.rs:111-172, fused_q5k_q8k_dot.rs:27-122,
// fused_q6k_q8k_dot.rs:27-154 under src/quant/cpu/kernels/simd; Q6_K has no min term), blocks added in K order.
//
// The PRODUCT of a code and its sub-block's scale goes into the operand, so a 256-block is one K = 256 integer product and one
// sum per (weight row, activation row, block) is scaled, not one per sub-block.  The products need two bytes:
//   * Q4_K, Q5_K: the 6-bit scale is cut, sc = sl + 8 sh; nibble * sl and nibble * sh (at most 105) are signed bytes, four of
//     them out of ONE 32-bit multiply, and the sum is S_lo + 8 S_hi.  Q5_K's fifth bit f adds 16 f sc = 8 (2 f sc): a third
//     plane of bytes (at most 126) into S_hi;
//   * Q6_K: (q - 32) * sc in 16-bit lanes, two of them out of one multiply-add, as signed bytes lo + 256 hi; the sum is
//     S_lo + 256 S_hi.
// The min term is a product of the mins with the activation's sums of 16 codes, both exact in f16, their f32 sums below 2^24
// exact too.
//
// Tile: 128 weight rows (the lanes of tensor memory) x mt = 16, 32 or 48 activation rows.  The decoded operand goes straight
// into TENSOR MEMORY (tcgen05.st; the MMA takes its A operand from there): no swizzled shared-memory stores, no proxy fence,
// and shared memory is left to the packed blocks in flight.  A stage is HALF a block (128 codes); four sets of four decode
// warps take the halves in turn.
// Work: whole tiles dealt round-robin, or, where a matrix has few tiles, a thread-block cluster of 2, 4 or 8 CTAs per tile, which
// takes that many blocks of K at a time, one per CTA.  Each CTA adds up some of the tile's weight rows: the terms of a round come
// to it from all CTAs by st.async into shared memory and are added in K order while the next round is drained, so the results
// have the CPU's bits at every K.  (Shares of K added as sums, which have other bits, are up to 15 % faster at K = 14336: 4096 x 14336 at 37
// rows Q4_K 25.7 against 27.1 us.  Up to K = 4096 the exchange by rounds is the faster one too: 4096 x 4096 at 37 rows Q4_K 14.8 -> 11.1 us.)
// What bounds it: instructions.  At 37 rows a block costs some 5500 (Q4_K), 6700 (Q5_K) or 7200 (Q6_K) warp instructions, in a cluster 1600 more; issue
// slots 59 ... 63 % busy, the ALU pipe 36 / 44 / 59 %; the MMAs themselves take 10 ... 20 cycles each with the A operand in tensor memory (34 ... 38 from
// shared memory).  One MMA-issuing warp spent 90 cycles on each and set the pace (2.0 us a Q4_K block instead of 0.9 at 16 rows), hence two.
// Measured, us (graph replays; the kernels that took these rows before -> here): 14336 x 4096 at 24 / 40 / 63 rows Q4_K 21.2 / 25.5 / 41.2 -> 18.7 / 21.2 / 34.5,
// Q5_K 26.9 / 28.9 / 50.1 -> 22.8 / 24.9 / 42.0, Q6_K 40.8 / 59.7 / 80.6 -> 26.0 / 27.2 / 46.6; 4096 x 14336 at 40 rows 49.2, 56.6, 60.4 -> 27.3, 29.7, 33.0; 4096 x
// 4096 at 40 rows 21.1, 25.8, 26.9 -> 10.9, 11.9, 12.8; SwiGLU 2 x 14336 x 4096 at 40 rows 53.8, 60.6, 120 -> 41.8, 51.4, 51.4, 2 x 14336 x 1024 Q4_K 20.7 -> 17.2,
// Q5_K 22.9 -> 20.3 (with the lanes of gate alone gating 20.3 and 24.1); Q6_K 128256 x 4096 at 37 rows 378 -> 158.
// Every wait is bounded; on a timeout the CTA is marked dead, records a status and frees its tensor memory.
#include <cuda.h>

#include <cstdio>

#include "../../include/b200q.h"
#include "common.cuh"
#include "tcgen05_i8.cuh"
#include "tmap.cuh"

namespace b200q {

bool smallm_i8_preferred(int fmt, size_t M, size_t K, size_t N, int sm_count);
size_t kq_i8_workspace_bytes(size_t M, size_t K);
size_t gemv_workspace_bytes(int fmt, size_t M, size_t K, size_t N, bool swiglu, int sm_count);
cudaError_t launch_kq_prep(const void* act, int act_dtype, size_t M, size_t K, void* ws, bool early, int sm_count, cudaStream_t st);
void kq_image(void* ws, size_t M, size_t K, uint8_t** codes, __half** sums, float** d8);

namespace {

__host__ __device__ constexpr uint32_t kf_pitch(int fmt) { return fmt == FMT_Q6_K ? 240 : (uint32_t)fmt_block_bytes(fmt); }
__host__ __device__ constexpr uint32_t kf_half_cols(int fmt) { return fmt == FMT_Q5_K ? 96 : 64; }  // tensor-memory columns of an operand half
__host__ __device__ constexpr bool kf_min(int fmt) { return fmt != FMT_Q6_K; }
__host__ __device__ constexpr uint32_t kf_raw(int fmt) { return 128 * kf_pitch(fmt); }

struct KfParams {
    const uint8_t *w, *w_up;  // w_up: SwiGLU (w is gate)
    void* out;
    const float* d8;  // [nblk][M]
    uint32_t M, N, nblk, row_bytes;
    uint32_t mt, nct, nunits;  // activation rows of a tile; column tiles; row tiles x column tiles
    uint32_t cs, cs_log;       // CTAs per tile: a cluster of 2^cs_log, each of which takes every cs-th block of K
    uint32_t ns, nr, nb;       // ring depths: operand halves in tensor memory, packed blocks (even), activation blocks
    uint32_t off_rec, off_raw, off_x;  // of shared memory
    uint32_t idesc_i, idesc_h;
    int out_dtype;
    bool raw_tma, swiglu;
    unsigned int* status;
};

constexpr int KF_DEC = 16, KF_DRAIN = 8, KF_COPY = 2;
constexpr int KF_W_DRAIN = KF_DEC, KF_W_COPY = KF_DEC + KF_DRAIN, KF_W_ACT = KF_W_COPY + KF_COPY, KF_W_MMA = KF_W_ACT + 1;
constexpr int KF_THREADS = (KF_W_MMA + 1) * 32;
constexpr uint32_t KF_NQ = 4, KF_REC = 1024;  // 128 x (d | dmin), then the activation rows' d8
constexpr uint32_t KF_MT_MAX = 48;
constexpr int KF_FULL = 0, KF_SET_EMPTY = 32, KF_RAW_FULL = 64, KF_RAW_EMPTY = 160, KF_B_FULL = 256, KF_B_EMPTY = 288, KF_ACC_FULL = 320,
              KF_ACC_EMPTY = 336, KF_REC_FULL = 352, KF_REC_EMPTY = 384, KF_MEET = 416, KF_TMEM = 424, KF_DEAD = 428, KF_READY = 432, KF_FREE = 448, KF_STAGES = 1024;
constexpr uint32_t KF_NR_MAX = 12;
__host__ __device__ constexpr uint32_t kf_btile(uint32_t mt) { return (mt * 288 + 1023) / 1024 * 1024; }

__device__ __forceinline__ uint64_t kf_desc_sw32(uint32_t lo) {  // rows of 32 bytes, 32-byte swizzle, 8-row groups 256 bytes apart
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"((256u >> 4) | (1u << 14) | (6u << 29)));
    return d;
}
// A operand in tensor memory: 128 lanes x 32 bytes (eight columns)
__device__ __forceinline__ void mma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, 0, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc)
        : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t kf_byte(uint32_t x, uint32_t i) { return __byte_perm(x, 0u, 0x4440u | i); }
// byte i with its sign (__byte_perm uses three bits of a selector, prmt.b32 the fourth for the sign)
__device__ __forceinline__ uint32_t kf_sbyte(uint32_t x, uint32_t i) {
    uint32_t r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(x), "r"(0x8880u | (i * 0x1111u)));
    return r;
}
__device__ __forceinline__ void kf_store(void* out, int dt, size_t idx, float v) {
    if (dt == DT_F32) static_cast<float*>(out)[idx] = v;
    else if (dt == DT_BF16) static_cast<__nv_bfloat16*>(out)[idx] = __float2bfloat16_rn(v);
    else static_cast<__half*>(out)[idx] = __float2half_rn(v);
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// A store to a CTA of the cluster that counts its bytes at a barrier there: nothing waits for it on this side, while stores
// released by an arrival (st.shared::cluster, mbarrier.arrive.release.cluster) cost 2 us a round.
__device__ __forceinline__ void st_async4(uint32_t addr, float a, float b, float c, float d, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "f"(a), "f"(b), "f"(c),
                 "f"(d), "r"(bar)
                 : "memory");
}
// Arrival at a barrier of a CTA of the cluster.  What it has to keep behind it are this warp's loads from its own shared memory, so the
// release at the CTA's scope (the default) does: one at the cluster's scope also waits for the stores on their way to other CTAs (0.6 us a
// round, 4096 x 14336 at 63 rows 43 -> 60 us; 50 where one idle warp does it for the others).
__device__ __forceinline__ void mbar_arrive_remote(uint32_t addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __noinline__ void kf_linger() {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
}
// i8_wait for a barrier that other CTAs of the cluster complete
__device__ __forceinline__ bool kf_try_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __noinline__ bool kf_wait_cluster(uint32_t bar, uint32_t parity, volatile uint32_t* dead) {
    const uint64_t t0 = global_timer_ns();
#pragma unroll 1
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 64; ++i)
            if (kf_try_cluster(bar, parity)) return true;
        if (*dead || global_timer_ns() - t0 > 2000000000ull) return false;
    }
}
// silu(g) u as in swiglu_gate_kernel
__device__ __forceinline__ float kf_gate(float g, float u) { return g / (1.0f + expf(-g)) * u; }

// Sixteen lanes a row copy the 16-byte chunks that hold the Q6_K blocks at blk, blk + row_bytes, ... (64 rows, `in` of which exist);
// each lands at byte (its address & 15) of its slot.  Only the tensor's last chunk can reach past its end; it is clipped there.
__device__ __forceinline__ void kf_copy_q6(uint32_t dst, const uint8_t* blk, uint32_t row_bytes, uint32_t lane, uint32_t in, const uint8_t* wend) {
    const uint32_t c = lane & 15;
    if (c >= 14) return;
    dst += (lane >> 4) * 240 + 16 * c;
    const uint8_t* src = blk + (size_t)(lane >> 4) * row_bytes;
#pragma unroll 8
    for (uint32_t q = lane >> 4; q < 64; q += 2) {
        const uint8_t* s = reinterpret_cast<const uint8_t*>((reinterpret_cast<uintptr_t>(src) & ~(uintptr_t)15) + 16 * c);
        if (q < in && s < wend)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(s), "r"((uint32_t)min((long long)16, (long long)(wend - s))) : "memory");
        src += 2 * (size_t)row_bytes;
        dst += 480;
    }
}

template <int FMT, bool CLUSTER>
__global__ void __launch_bounds__(KF_THREADS, 1) kq_few_kernel(const __grid_constant__ CUtensorMap tmap_act, const __grid_constant__ CUtensorMap tmap_sum,
                                                               const __grid_constant__ CUtensorMap tmap_w0, const __grid_constant__ CUtensorMap tmap_w1,
                                                               const KfParams p) {
    constexpr bool MIN = kf_min(FMT), Q6 = FMT == FMT_Q6_K;
    constexpr uint32_t BB = fmt_block_bytes(FMT), PITCH = kf_pitch(FMT), RAW = kf_raw(FMT), HI_SHIFT = Q6 ? 8 : 3, HALF = kf_half_cols(FMT);
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // the launch reserves 1 KB of slack
    const uint32_t sbase = smem_u32(smem);
    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    volatile uint32_t* dead = reinterpret_cast<volatile uint32_t*>(smem + KF_DEAD);
    // tensor memory: two accumulators (lo | hi (| mins), mt columns each), ns operand halves (lo 32 | hi 32 (| fifth bits 32)), two tiles of mins
    const uint32_t acc_cols = (MIN ? 3 : 2) * p.mt, a_col0 = 2 * acc_cols, m_col0 = a_col0 + HALF * p.ns;
    // Blocks of this CTA: all of the units blockIdx.x, + gridDim.x, ..., or of one unit the blocks rank, + cs, ...
    const uint32_t cs = CLUSTER ? p.cs : 1, cs_log = CLUSTER ? p.cs_log : 0, rank = CLUSTER ? cluster_rank() : 0;
    const uint32_t stride = gridDim.x >> cs_log, unit0 = blockIdx.x >> cs_log, nb = (p.nblk - rank + cs - 1) >> cs_log;
    const uint32_t units = (p.nunits - unit0 + stride - 1) / stride, total = units * nb;
    const uint32_t rows = p.swiglu ? 64 : 128;  // weight rows of a row tile (SwiGLU: as many of gate and of up)
    const uint32_t in = min(p.mt, p.M - unit0 % p.nct * p.mt);  // activation rows of a cluster's tile
    // round i of a cluster is one block per CTA: how many there are, and the bytes of their terms that one CTA gets
    auto round_blocks = [&](uint32_t i) { return i << cs_log < p.nblk ? min(cs, p.nblk - (i << cs_log)) : 0u; };
    auto round_bytes = [&](uint32_t i) { return round_blocks(i) * (((in + 7) & ~7u) >> cs_log) * 512; };
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < 4; ++s) {
            mbar_init(sbase + KF_FULL + 8 * s, 4);       // the four warps of the set that wrote the half
            mbar_init(sbase + KF_SET_EMPTY + 8 * s, 1);  // commit: the half that this set writes next is free
            mbar_init(sbase + KF_B_FULL + 8 * s, 1);
            mbar_init(sbase + KF_B_EMPTY + 8 * s, 1);
        }
        for (uint32_t s = 0; s < p.nr; ++s) {
            mbar_init(sbase + KF_RAW_FULL + 8 * s, p.raw_tma ? 1 : KF_COPY * 32);
            mbar_init(sbase + KF_RAW_EMPTY + 8 * s, 8);  // the two sets that take its halves
        }
        for (uint32_t s = 0; s < 2; ++s) {
            mbar_init(sbase + KF_ACC_FULL + 8 * s, 1);
            mbar_init(sbase + KF_ACC_EMPTY + 8 * s, KF_DRAIN);
        }
        for (uint32_t s = 0; s < KF_NQ; ++s) {
            mbar_init(sbase + KF_REC_FULL + 8 * s, 4 + 32);  // four decode warps + the lanes that copy d8
            mbar_init(sbase + KF_REC_EMPTY + 8 * s, KF_DRAIN);
        }
        mbar_init(sbase + KF_MEET, KF_DRAIN);
        if constexpr (CLUSTER)
            for (uint32_t s = 0; s < 2; ++s) {
                mbar_init(sbase + KF_READY + 8 * s, 1);              // the bytes of a round's terms
                mbar_init(sbase + KF_FREE + 8 * s, KF_DRAIN << p.cs_log);  // the drain warps of the whole cluster
            }
        *dead = 0;
        mbar_fence_init();
        if constexpr (CLUSTER)
            for (uint32_t s = 0; s < 2; ++s)
                if (round_bytes(s)) mbar_expect_tx(sbase + KF_READY + 8 * s, round_bytes(s));
    }
    if (warp == KF_W_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + KF_TMEM), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_before();
    __syncthreads();
    tc_after();
    // (through a shuffle: the operands of the MMAs stay in uniform registers)
    const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *reinterpret_cast<volatile uint32_t*>(smem + KF_TMEM), 0);
    // A wait of a whole warp: all lanes leave together; on a timeout the CTA is marked dead and every role ends.
    auto wait = [&](uint32_t off, uint32_t parity, unsigned int code) {
        const bool ok = __all_sync(0xFFFFFFFFu, i8_wait(sbase + off, parity, dead));
        if (!ok && lane == 0) i8_fail(dead, p.status, code);
        return ok;
    };
    if constexpr (CLUSTER) cluster_arrive();  // this CTA's barriers exist

    // Two warps issue the MMAs, one for the even and one for the odd blocks, where the second copying warp has nothing to copy and
    // every operand half has a slot of its own (a slot then belongs to one of them).
    const uint32_t nm = p.raw_tma && p.ns == 4 ? 2 : 1;
    const bool second = warp == KF_W_COPY + 1 && nm == 2;

    if (warp >= KF_W_COPY && warp < KF_W_ACT && !second) {
        // ------------------------------------------------------------ packed blocks (do not depend on the kernel that is still running)
        const uint32_t half = (uint32_t)(warp - KF_W_COPY);
        const uint32_t mine = p.raw_tma && half ? 0 : total;  // by TMA one warp brings all
        uint32_t unit = unit0, b = rank, rs = 0, par = 1;
        for (uint32_t i = 0; i < mine; ++i) {
            if (!wait(KF_RAW_EMPTY + 8 * rs, par, STATUS_TIMEOUT_EMPTY)) break;
            const uint32_t n0 = unit / p.nct * rows;
            const uint32_t dst = sbase + p.off_raw + rs * RAW, bar = sbase + KF_RAW_FULL + 8 * rs;
            if (p.raw_tma) {
                if (lane == 0) {
                    mbar_expect_tx(bar, RAW);
                    const int x = (int)((b * BB & ~15u) / 2);
                    tma2d(dst, &tmap_w0, x, (int)n0, bar);
                    if (p.swiglu) tma2d(dst + RAW / 2, &tmap_w1, x, (int)n0, bar);  // boxes of 64 rows
                }
            } else if constexpr (Q6) {
                const uint8_t* w = p.swiglu && half ? p.w_up : p.w;
                const uint32_t r0 = p.swiglu ? n0 : n0 + 64 * half;
                kf_copy_q6(dst + half * (RAW / 2), w + (size_t)r0 * p.row_bytes + (size_t)b * BB, p.row_bytes, lane, r0 < p.N ? p.N - r0 : 0,
                           w + (size_t)p.N * p.row_bytes);
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
            }
            b += cs;
            if (b >= p.nblk) {
                b = rank;
                unit += stride;
            }
            if (++rs == p.nr) {
                rs = 0;
                par ^= 1;
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == KF_W_ACT) {
        // ------------------------------------------------------------ activation codes, sums and scales (previous kernel's output)
        grid_dep_wait();
        grid_dep_launch();  // not before: the next product of a batch may be one that reads its weights in order
        uint32_t unit = unit0, b = rank, bs = 0, par = 1;
        const uint32_t btile = kf_btile(p.mt);
        for (uint32_t i = 0; i < total; ++i) {
            const uint32_t q = i % KF_NQ, m0 = unit % p.nct * p.mt, dst = sbase + KF_STAGES + bs * btile, bar = sbase + KF_B_FULL + 8 * bs;
            if (!wait(KF_B_EMPTY + 8 * bs, par, STATUS_TIMEOUT_EMPTY)) break;
            if (lane == 0) {
                mbar_expect_tx(bar, (MIN ? 288 : 256) * p.mt);
                tma2d(dst, &tmap_act, (int)(b * 256), (int)m0, bar);
                tma2d(dst + 128 * p.mt, &tmap_act, (int)(b * 256 + 128), (int)m0, bar);
                if constexpr (MIN) tma2d(dst + 256 * p.mt, &tmap_sum, (int)(b * 16), (int)m0, bar);
            }
            __syncwarp();
            if (!wait(KF_REC_EMPTY + 8 * q, ((i / KF_NQ) & 1) ^ 1, STATUS_TIMEOUT_EMPTY)) break;
            const uint32_t rec = sbase + p.off_rec + q * KF_REC + 512;
            const float* src = p.d8 + (size_t)b * p.M + m0;
            for (uint32_t m = lane; m < p.mt; m += 32)  // rows past M are zero-filled
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(rec + 4 * m), "l"(m0 + m < p.M ? src + m : p.d8), "r"(m0 + m < p.M ? 4u : 0u) : "memory");
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(sbase + KF_REC_FULL + 8 * q) : "memory");
            b += cs;
            if (b >= p.nblk) {
                b = rank;
                unit += stride;
            }
            if (++bs == p.nb) {
                bs = 0;
                par ^= 1;
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (*dead) kf_linger();  // TMA copies in flight land within microseconds: the CTA's shared memory stays until then
    } else if (warp == KF_W_MMA || second) {
        // ------------------------------------------------------------ MMA issue
        const uint32_t btile = kf_btile(p.mt);
        uint32_t st = second ? 2 : 0, st_par = 0, bs = second ? 1 : 0, b_par = 0;
        bool ok = true;
        for (uint32_t i = second ? 1 : 0; i < total && ok; i += nm) {
            const uint32_t buf = i & 1, d = tmem + buf * acc_cols, bt = sbase + KF_STAGES + bs * btile;
            if (!wait(KF_ACC_EMPTY + 8 * buf, ((i >> 1) & 1) ^ 1, STATUS_TIMEOUT_EMPTY)) break;
            if (!wait(KF_B_FULL + 8 * bs, b_par, STATUS_TIMEOUT_FULL)) break;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                if (!wait(KF_FULL + 8 * st, st_par, STATUS_TIMEOUT_FULL)) {
                    ok = false;
                    break;
                }
                tc_after();
                const uint32_t a = tmem + a_col0 + HALF * st, b_lo = desc_lo(bt + h * 128 * p.mt);
                if (elect_one_lane()) {
                    if constexpr (MIN)
                        if (h == 0) mma_f16_ts(d + 2 * p.mt, tmem + m_col0 + 8 * buf, kf_desc_sw32(desc_lo(bt + 256 * p.mt)), p.idesc_h);
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k) {
                        mma_i8_ts(d, a + 8 * k, desc_sw128(b_lo + 2 * k), p.idesc_i, h + k > 0);
                        mma_i8_ts(d + p.mt, a + 32 + 8 * k, desc_sw128(b_lo + 2 * k), p.idesc_i, h + k > 0);
                        if constexpr (FMT == FMT_Q5_K) mma_i8_ts(d + p.mt, a + 64 + 8 * k, desc_sw128(b_lo + 2 * k), p.idesc_i, true);
                    }
                    tc_commit_to(sbase + KF_SET_EMPTY + 8 * ((2 * i + h + p.ns) & 3));
                    if (h == 1) {
                        tc_commit_to(sbase + KF_B_EMPTY + 8 * bs);
                        tc_commit_to(sbase + KF_ACC_FULL + 8 * buf);
                    }
                }
                __syncwarp();
                if (++st == p.ns) {
                    st = 0;
                    st_par ^= 1;
                }
            }
            if (nm == 2) {  // over the other warp's block
                st = second ? 2 : 0;
                if (!second) st_par ^= 1;
            }
            bs += nm;
            if (bs >= p.nb) {
                bs -= p.nb;
                b_par ^= 1;
            }
        }
    } else if (warp < KF_DEC) {
        // ------------------------------------------------------------ decode: one thread per weight row, the sets take the half blocks in turn
        const uint32_t r = threadIdx.x & 127, set = (uint32_t)warp >> 2, h = set & 1;
        const uint32_t lanes = tmem + (((uint32_t)warp & 3) << 21);
        uint32_t b = rank + cs * ((set >> 1) % nb), st = set % p.ns, rs = set >> 1, rpar = 0;
        const uint32_t b_step = cs * (2 % nb), b_end = rank + cs * nb, st_step = 4 % p.ns;
        for (uint32_t i = set >> 1; i < total; i += 2) {
            const uint32_t q = i % KF_NQ, x = 2 * i + h;
            if (!wait(KF_RAW_FULL + 8 * rs, rpar, STATUS_TIMEOUT_FULL)) break;
            const uint32_t col = a_col0 + HALF * st;
            uint32_t dm = 0;
            // all columns of this half may be overwritten: the MMAs that read them have completed, and the stores stay behind that
            auto take = [&]() { return x < p.ns || wait(KF_SET_EMPTY + 8 * set, ((x - p.ns) >> 2) & 1, STATUS_TIMEOUT_EMPTY); };
            auto release = [&]() {
                __syncwarp();
                if (lane == 0) mbar_arrive(sbase + KF_RAW_EMPTY + 8 * rs);
            };
            if constexpr (Q6) {
                // 128 bytes low nibbles, 64 bytes bit pairs, 16 scales, f16 d; element 128 h + 32 g + l: nibble g >> 1 of byte
                // 64 h + 32 (g & 1) + l, bits 2 g of byte 32 h + l, scale 8 h + 2 g + (l >> 4)
                const uint32_t at = (r * p.row_bytes + b * BB) & 15u, sh = 8 * (at & 2u);  // (64 rows are a multiple of 16 bytes)
                const uint32_t* raw = reinterpret_cast<const uint32_t*>(smem + p.off_raw + rs * RAW + r * PITCH + (at & 12u));
                uint32_t hw[9], sw[3];
#pragma unroll
                for (int k = 0; k < 9; ++k) hw[k] = raw[32 + 8 * h + k];
#pragma unroll
                for (int k = 0; k < 3; ++k) sw[k] = raw[48 + 2 * h + k];
                dm = (raw[52] >> sh) & 0xFFFFu;
#pragma unroll
                for (int k = 0; k < 8; ++k) hw[k] = __funnelshift_r(hw[k], hw[k + 1], sh);
#pragma unroll
                for (int k = 0; k < 2; ++k) sw[k] = __funnelshift_r(sw[k], sw[k + 1], sh);
                if (!take()) break;
                tc_after();
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                    uint32_t lw[9];
#pragma unroll
                    for (int k = 0; k < 9; ++k) lw[k] = raw[16 * h + 8 * part + k];
#pragma unroll
                    for (int k = 0; k < 8; ++k) lw[k] = __funnelshift_r(lw[k], lw[k + 1], sh);
                    if (part == 1) release();
#pragma unroll
                    for (int gg = 0; gg < 2; ++gg) {
                        const int g = part + 2 * gg;
                        uint32_t lo[8], hi[8];
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const uint32_t sc = kf_sbyte(sw[g >> 1], 2 * (g & 1) + (k >> 2));
                            const uint32_t bias = 0x80808080u - sc * 0x200020u;  // 2^15 + 128 - 32 sc in both lanes
                            const uint32_t pair = g == 0 ? hw[k] << 4 : g == 1 ? hw[k] << 2 : g == 2 ? hw[k] : hw[k] >> 2;
                            const uint32_t u = ((gg ? lw[k] >> 4 : lw[k]) & 0x0F0F0F0Fu) | (pair & 0x30303030u);
                            const uint32_t pe = (u & 0x00FF00FFu) * sc + bias, po = __byte_perm(u, 0u, 0x4341) * sc + bias;
                            lo[k] = __byte_perm(pe, po, 0x6240) ^ 0x80808080u;
                            hi[k] = __byte_perm(pe, po, 0x7351) ^ 0x80808080u;
                        }
                        tmem_st8(lanes + col + 8 * g, lo);
                        tmem_st8(lanes + col + 32 + 8 * g, hi);
                    }
                }
            } else {
                // Q4_K: d, dmin, 12 bytes scales and mins, 128 bytes nibbles; Q5_K: 32 bytes fifth bits before the nibbles.  Bytes 32 j of low
                // nibbles are sub-block 2 j, of high nibbles 2 j + 1; bit e of word j of the fifth bits is element e of sub-block j.
                const uint4* raw = reinterpret_cast<const uint4*>(smem + p.off_raw + rs * RAW + r * PITCH);
                const uint4 hd = raw[0];
                uint4 hb = make_uint4(0, 0, 0, 0);
                if constexpr (FMT == FMT_Q5_K) hb = raw[1 + h];
                dm = hd.x;
                const uint32_t scw = h ? (hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u) : hd.y & 0x3F3F3F3Fu;
                const uint32_t slw = scw & 0x07070707u, shw = (scw >> 3) & 0x07070707u;
                if (!take()) break;
                tc_after();
#pragma unroll
                for (int part = 0; part < 2; ++part) {  // 32 bytes of nibbles: sub-blocks 4 h + 2 part and the next
                    uint32_t cw[8];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const uint4 v = raw[(FMT == FMT_Q5_K ? 3 : 1) + 4 * h + 2 * part + k];
                        cw[4 * k] = v.x; cw[4 * k + 1] = v.y; cw[4 * k + 2] = v.z; cw[4 * k + 3] = v.w;
                    }
                    if (part == 1) release();
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint32_t sl = kf_byte(slw, 2 * part + j), sh = kf_byte(shw, 2 * part + j);
                        uint32_t lo[8], hi[8];
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const uint32_t c = (j ? cw[k] >> 4 : cw[k]) & 0x0F0F0F0Fu;
                            lo[k] = c * sl;
                            hi[k] = c * sh;
                        }
                        tmem_st8(lanes + col + 8 * (2 * part + j), lo);
                        tmem_st8(lanes + col + 32 + 8 * (2 * part + j), hi);
                        if constexpr (FMT == FMT_Q5_K) {
                            const uint32_t bits = part ? (j ? hb.w : hb.z) : (j ? hb.y : hb.x), even = bits & 0x0F0F0F0Fu, odd = (bits >> 4) & 0x0F0F0F0Fu;
                            const uint32_t sc2 = 2 * kf_byte(scw, 2 * part + j);
                            uint32_t f[8];  // four bits of a nibble to four bytes
#pragma unroll
                            for (int k = 0; k < 8; ++k) f[k] = ((kf_byte(k & 1 ? odd : even, k >> 1) * 0x00204081u) & 0x01010101u) * sc2;
                            tmem_st8(lanes + col + 64 + 8 * (2 * part + j), f);
                        }
                    }
                }
                if (h == 0) {
                    // sixteen f16 mins (each covers two sums of 16): 1024 + m is 0x6400 | m
                    const uint32_t m0 = hd.z & 0x3F3F3F3Fu, m1 = ((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u);
                    uint32_t mn[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t two = __byte_perm(j < 4 ? m0 : m1, 0x64646464u, 0x4040 | (j & 3) | ((j & 3) << 8));
                        const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&two), __float2half2_rn(1024.f));
                        mn[j] = *reinterpret_cast<const uint32_t*>(&v);
                    }
                    tmem_st8(lanes + m_col0 + 8 * (i & 1), mn);
                }
            }
            tmem_st_wait();
            tc_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(sbase + KF_FULL + 8 * st);
            if (h == 0) {
                if (!wait(KF_REC_EMPTY + 8 * q, ((i / KF_NQ) & 1) ^ 1, STATUS_TIMEOUT_EMPTY)) break;
                reinterpret_cast<uint32_t*>(smem + p.off_rec + q * KF_REC)[r] = dm;
                __syncwarp();
                if (lane == 0) mbar_arrive(sbase + KF_REC_FULL + 8 * q);
            }
            b += b_step;
            if (b >= b_end) b -= cs * nb;
            st += st_step;
            if (st >= p.ns) st -= p.ns;
            rs += 2;
            if (rs >= p.nr) {
                rs -= p.nr;
                rpar ^= 1;
            }
        }
    } else {
        // ------------------------------------------------------------ drain: integer sums -> scaled f32 terms, in K order
        const uint32_t quarter = warp & 3, cg = (uint32_t)(warp - KF_W_DRAIN) >> 2, r = quarter * 32 + lane;
        const uint32_t t_base = tmem + ((quarter * 32) << 16);
        constexpr int CHUNKS = KF_MT_MAX / 16;
        float sum[CHUNKS][8];  // activation rows 8 (cg + 2 c) + j; in a cluster the units of `from`
        float* xch = reinterpret_cast<float*>(smem + p.off_x);
        grid_dep_wait();  // the output may still be in use by the previous kernel
        // Cluster: in a round every CTA drains one block.  The weight rows of the tile are shared out; their CTA gets the round's terms from
        // all, [buffer][CTA][activation rows / 4][weight row][4], and adds them in the CTAs' order, which is K order, while the next round
        // is drained.  A buffer is written again once all CTAs have added what was in theirs.
        const uint32_t dt = threadIdx.x - KF_W_DRAIN * 32, rounds = CLUSTER ? (p.nblk + cs - 1) >> cs_log : total;
        const uint32_t own = rows >> cs_log, own_log = (p.swiglu ? 6 : 7) - cs_log, lines = 128 >> cs_log;  // its weight rows; with those of up
        const uint32_t line = (r & (own - 1)) + (r >= rows ? own : 0), owner = CLUSTER ? (r & (rows - 1)) >> own_log : 0;
        const uint32_t to = CLUSTER ? mapa(sbase + p.off_x + (rank * (p.mt / 4) * lines + line) * 16, owner) : 0;
        const uint32_t to_bar = CLUSTER ? mapa(sbase + KF_READY, owner) : 0;
        // what this thread adds: units (4 activation rows of a weight row) dt, dt + 256, dt + 512; SwiGLU: dt, dt + 256 of gate (0, 1) and of up (2, 3)
        auto unit_of = [&](int q) { return dt + 256 * (p.swiglu ? q & 1 : q); };
        uint32_t from[4] = {};  // addresses of the units (0: none) in the first buffer
        if constexpr (CLUSTER)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if ((unit_of(q) >> own_log) * 4 < in && (q < 3 || p.swiglu))
                    from[q] = sbase + p.off_x + ((unit_of(q) >> own_log) * lines + (unit_of(q) & (own - 1)) + (p.swiglu && q >= 2 ? own : 0)) * 16;
        constexpr uint32_t ZERO = 0x80000000u;  // -0.0: x + -0.0 is x
        auto wait_cluster = [&](uint32_t off, uint32_t parity, unsigned int code) {
            const bool ok = __all_sync(0xFFFFFFFFu, kf_try_cluster(sbase + off, parity) || kf_wait_cluster(sbase + off, parity, dead));
            if (!ok && lane == 0) i8_fail(dead, p.status, code);
            return ok;
        };
        auto collect = [&](uint32_t i) {
            if (!wait_cluster(KF_READY + 8 * (i & 1), (i >> 1) & 1, STATUS_TIMEOUT_FULL)) return false;
            if (dt == 0 && round_bytes(i + 2)) mbar_expect_tx(sbase + KF_READY + 8 * (i & 1), round_bytes(i + 2));
            const uint32_t cnt = round_blocks(i), step = p.mt * lines * 4;
#pragma unroll
            for (int q = 0; q < 4; q += 2) {
                if (!from[q]) continue;
                uint32_t a = (i & 1) * p.mt * 512;
#pragma unroll 1
                for (uint32_t c = 0; c < cnt; c += 2, a += 2 * step) {  // two units of two blocks are on their way together
                    uint4 v[2][2];
#pragma unroll
                    for (int k = 0; k < 2; ++k)
#pragma unroll
                        for (int u = 0; u < 2; ++u) v[k][u] = from[q + u] && c + k < cnt ? sld128(from[q + u] + a + k * step) : make_uint4(ZERO, ZERO, ZERO, ZERO);
#pragma unroll
                    for (int k = 0; k < 2; ++k)
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            float* s = &sum[q >> 1][u * 4];
                            s[0] = __fadd_rn(s[0], __uint_as_float(v[k][u].x));
                            s[1] = __fadd_rn(s[1], __uint_as_float(v[k][u].y));
                            s[2] = __fadd_rn(s[2], __uint_as_float(v[k][u].z));
                            s[3] = __fadd_rn(s[3], __uint_as_float(v[k][u].w));
                        }
                }
            }
            __syncwarp();
            if ((uint32_t)lane < cs) mbar_arrive_remote(mapa(sbase + KF_FREE + 8 * (i & 1), lane));
            return true;
        };
        if constexpr (CLUSTER) cluster_wait();  // the barriers of all CTAs exist
        uint32_t unit = unit0, b = 0, tiles = 0;
        bool ok = true;
        for (uint32_t i = 0; i < total; ++i) {
            const uint32_t q = i % KF_NQ, buf = i & 1, m0 = unit % p.nct * p.mt;
            if (!wait(KF_REC_FULL + 8 * q, (i / KF_NQ) & 1, STATUS_TIMEOUT_FULL)) {
                ok = false;
                break;
            }
            const uint8_t* rec = smem + p.off_rec + q * KF_REC;
            const uint32_t dm = reinterpret_cast<const uint32_t*>(rec)[r];
            const float d = f16bits_to_f32(dm & 0xFFFF), dmin = f16bits_to_f32(dm >> 16);
            if (CLUSTER ? i == 0 : b == 0)
#pragma unroll
                for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
                    for (int j = 0; j < 8; ++j) sum[c][j] = 0.f;
            if (CLUSTER && i >= 2 && !wait_cluster(KF_FREE + 8 * buf, ((i >> 1) & 1) ^ 1, STATUS_TIMEOUT_EMPTY)) {
                ok = false;
                break;
            }
            if (!wait(KF_ACC_FULL + 8 * buf, (i >> 1) & 1, STATUS_TIMEOUT_MMA)) {
                ok = false;
                break;
            }
            tc_after();
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
                const uint32_t col = 8 * (cg + 2 * c);
                if (col < p.mt && m0 + col < p.M) {  // warp-uniform
                    uint32_t v[8], vh[8], u[8];
                    const uint32_t tc = t_base + buf * acc_cols + col;
                    tmem_ld8_async(tc, v);
                    tmem_ld8_async(tc + p.mt, vh);
                    if constexpr (MIN) tmem_ld8_async(tc + 2 * p.mt, u);
                    const float4* d8 = reinterpret_cast<const float4*>(rec + 512 + 4 * col);
                    const float4 e0 = d8[0], e1 = d8[1];
                    const float e[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
                    tmem_ld_wait();
                    float t[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        t[j] = __fmul_rn(__fmul_rn(d, e[j]), (float)(int)(v[j] + (vh[j] << HI_SHIFT)));
                        if constexpr (MIN) t[j] = __fsub_rn(t[j], __fmul_rn(__fmul_rn(dmin, e[j]), __uint_as_float(u[j])));
                    }
                    if constexpr (CLUSTER) {
                        const uint32_t dst = to + (buf * p.mt * 128 + col * lines) * 4, bar = to_bar + 8 * buf;
                        st_async4(dst, t[0], t[1], t[2], t[3], bar);
                        st_async4(dst + lines * 16, t[4], t[5], t[6], t[7], bar);
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; ++j) sum[c][j] = __fadd_rn(sum[c][j], t[j]);
                    }
                }
            }
            tc_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(sbase + KF_ACC_EMPTY + 8 * buf);
                mbar_arrive(sbase + KF_REC_EMPTY + 8 * q);
            }
            if constexpr (CLUSTER) {
                if (i > 0 && !collect(i - 1)) {
                    ok = false;
                    break;
                }
                continue;
            }
            if (++b < nb) continue;
            b = 0;
            const uint32_t n = unit / p.nct * rows + r;
            unit += stride;
            if (p.swiglu) {
                // A lane of gate and its lane of up swap half of their sums, so that both gate and store half of the row's results; two
                // buffers, so one meeting a tile is enough.
                const bool up = r >= 64;  // warp-uniform
                float* swap = xch + (tiles & 1) * p.mt * 64 + (r & 63);
#pragma unroll
                for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (8 * (cg + 2 * c) < p.mt) swap[(8 * (cg + 2 * c) + j + (up ? 0 : 4)) * 64] = up ? sum[c][j] : sum[c][j + 4];
                __syncwarp();
                if (lane == 0) mbar_arrive(sbase + KF_MEET);
                if (!wait(KF_MEET, tiles & 1, STATUS_TIMEOUT_EMPTY)) break;
                ++tiles;
#pragma unroll
                for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t mr = 8 * (cg + 2 * c) + j + (up ? 4 : 0);
                        if (mr < p.mt && m0 + mr < p.M && n - (up ? 64 : 0) < p.N) {
                            const float other = swap[mr * 64], own_sum = up ? sum[c][j + 4] : sum[c][j];
                            kf_store(p.out, p.out_dtype, (size_t)(m0 + mr) * p.N + n - (up ? 64 : 0), up ? kf_gate(other, own_sum) : kf_gate(own_sum, other));
                        }
                    }
            } else if (n < p.N) {
#pragma unroll
                for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t m = 8 * (cg + 2 * c) + j;
                        if (m < p.mt && m0 + m < p.M) kf_store(p.out, p.out_dtype, (size_t)(m0 + m) * p.N + n, sum[c][j]);
                    }
            }
        }
        // the rounds that are left: the last one, and the one before where this CTA had no block in the last
        if (CLUSTER)
            for (uint32_t i = total - 1; ok && i < rounds; ++i) ok = collect(i);
        if (CLUSTER && ok) {
            const uint32_t n0 = unit0 / p.nct * rows + (rank << own_log), m0 = unit0 % p.nct * p.mt;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const uint32_t n = n0 + (unit_of(q) & (own - 1)), m = (unit_of(q) >> own_log) * 4;
                if (n < p.N && from[q] && (q < 2 || !p.swiglu))
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float v = sum[q >> 1][(q & 1) * 4 + j];
                        if (q < 2 && p.swiglu) v = kf_gate(v, sum[1][(q & 1) * 4 + j]);
                        if (m + j < in) kf_store(p.out, p.out_dtype, (size_t)(m0 + m + j) * p.N + n, v);
                    }
            }
        }
    }
    __syncwarp();
    if constexpr (CLUSTER) {  // nobody's shared memory goes before all have done with it
        if (warp < KF_W_DRAIN || warp >= KF_W_COPY) cluster_wait();  // (the drain warps have waited for the barriers to exist)
        cluster_arrive();
        cluster_wait();
    }
    tc_before();
    __syncthreads();
    if (warp == KF_W_MMA) {
        tc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
        // Terms of other CTAs may be on their way to a CTA that gave up: its shared memory stays until they have landed.
        if (CLUSTER && *dead) kf_linger();
    }
}

struct KfPlan {
    uint32_t mt = 0, cs = 1;
    double us = 0;  // expected time behind the first block
};
constexpr uint32_t KF_SMEM = 232448;
uint32_t kf_x_bytes(const KfPlan& pl, bool swiglu) { return pl.cs > 1 ? 2 * pl.mt * 512 : swiglu ? pl.mt * 512 : 0u; }
// Operand halves in tensor memory: at most one ahead of every set (KF_SET_EMPTY); activation blocks in shared memory.
uint32_t kf_stages(int fmt, uint32_t mt) {
    const uint32_t n = (512 - 2 * (kf_min(fmt) ? 3 : 2) * mt - 16) / kf_half_cols(fmt);
    return n > 4 ? 4 : n;
}
uint32_t kf_acts(int fmt, uint32_t mt) { return kf_stages(fmt, mt) == 4 || mt <= 32 ? 4 : 3; }
// packed blocks that fit beside the rest (even: a slot belongs to the sets of one block parity)
uint32_t kf_ring(int fmt, const KfPlan& pl, bool swiglu) {
    const uint32_t fixed = 2048 + kf_acts(fmt, pl.mt) * kf_btile(pl.mt) + KF_NQ * KF_REC + kf_x_bytes(pl, swiglu);
    const uint32_t nr = (KF_SMEM - fixed) / kf_raw(fmt) & ~1u;
    return nr > KF_NR_MAX ? KF_NR_MAX : nr;
}

template <int FMT, bool CLUSTER>
cudaError_t kf_attr() {
    static PerDeviceOnce attrs;
    return attrs.run([] { return cudaFuncSetAttribute(kq_few_kernel<FMT, CLUSTER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)KF_SMEM); });
}
// Tiles of `cs` CTAs that can run at the same time.
uint32_t kf_clusters(uint32_t cs) {
    static std::atomic<int> cached[64][4];
    const int k = cs == 2 ? 1 : cs == 4 ? 2 : 3;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int n = cached[dev][k].load(std::memory_order_relaxed);
    if (n) return (uint32_t)(n - 1);
    n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(KF_THREADS);
    cfg.dynamicSmemBytes = KF_SMEM;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (kf_attr<FMT_Q4_K, true>() != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, kq_few_kernel<FMT_Q4_K, true>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cached[dev][k].store(n + 1, std::memory_order_relaxed);
    return (uint32_t)n;
}

// Tile and cluster of least time, in us: blocks of K one after the other x the time of one (a line in mt, measured at 14336 x
// 4096: 16 / 32 / 48 rows Q4_K 0.86 / 0.99 / 1.14, Q5_K 1.02 / 1.18 / 1.32, Q6_K 1.31 / 1.37 / 1.45, or 1.97 where
// its rows are no multiple of 16 bytes: 13825 x 5120).  In a cluster the exchange of a block's terms takes 0.15 + 0.0075 a row more, and 0.7 once
// (fitted to 512 ... 9216 weight rows, K = 1024 ... 14336).
KfPlan kf_plan(int fmt, size_t M, size_t K, size_t row_tiles, bool swiglu, int sm_count, bool estimate = false) {
    KfPlan best;
    const uint32_t nblk = (uint32_t)(K / 256);
    const double c0 = fmt == FMT_Q4_K ? 0.72 : fmt == FMT_Q5_K ? 0.87 : nblk % 8 ? 1.9 : 1.24, c1 = fmt == FMT_Q4_K ? 0.0088 : fmt == FMT_Q5_K ? 0.0094 : 0.0044;
    for (uint32_t mt = 16; mt <= KF_MT_MAX; mt += 16) {
        const size_t units = row_tiles * ((M + mt - 1) / mt);
        for (uint32_t cs = 1; cs <= 8 && cs <= nblk; cs *= 2) {
            KfPlan c;
            c.mt = mt;
            c.cs = cs;
            if (cs > 1 && (units * cs > (size_t)sm_count || (!estimate && units > kf_clusters(cs)))) continue;
            const size_t blocks = cs > 1 ? (nblk + cs - 1) / cs : (units + sm_count - 1) / sm_count * nblk;
            c.us = (double)blocks * (c0 + c1 * mt + (cs > 1 ? 0.15 + 0.0075 * mt : 0.0)) + (cs > 1 ? 0.7 : 0.0);
            if (!best.mt || c.us < best.us) best = c;
        }
        if (mt >= M) break;
    }
    return best;
}

bool kf_encode(CUtensorMap* map, CUtensorMapDataType type, size_t elem, const void* base, size_t inner, size_t rows, uint32_t box_inner, uint32_t box_rows,
               CUtensorMapSwizzle sw) {
    const cuuint32_t estr[2] = {1, 1}, box[2] = {box_inner, box_rows};
    const cuuint64_t gdim[2] = {inner, rows}, gstride[1] = {inner * elem};
    return encode_tiled()(map, type, 2, const_cast<void*>(base), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int FMT, bool CLUSTER>
cudaError_t kf_launch(const CUtensorMap& am, const CUtensorMap& sm, const CUtensorMap* wm, const KfParams& p, uint32_t grid, size_t smem, cudaStream_t st) {
    cudaError_t e = kf_attr<FMT, CLUSTER>();
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(KF_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = p.cs;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = CLUSTER ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, kq_few_kernel<FMT, CLUSTER>, am, sm, wm[0], wm[1], p);
    note_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

// From 17 rows on one pass here beats passes of 16 rows by mma.sync (gemv.cu), except where K is long and the matrix has so few tiles that
// clusters of 8 leave SMs idle, which the other kernel's chunks of K occupy (5 us a pass, and 0.12 ... 0.15 more for every tile of 128 rows
// and chunk past the tenth): Q6_K at 17 rows 64 x 28672 13.4 us there, 24.3 here, 512 x 14336 13.9 and 15.2, 1024 x 14336 18.8 and 16.3; at 48 rows 512 x 14336
// 20.4 and 15.4.  At 9 ... 16 rows the two are
// even on most shapes (14336 x 4096 at 16 rows: Q6_K 24.2 there, 25.0 here) and this kernel wins where the other's fixed shares of K (chunks of 16
// blocks; 5 + 0.13 ... 0.155 us a tile of 128 rows and chunk) are badly filled: 13825 x 5120 at 13 rows Q4_K 30.6 -> 21.1, Q5_K 34.9 -> 24.4; 14336 x
// 2048 Q5_K 20.1 -> 12.4, Q6_K 20.1 -> 14.3; SwiGLU 2 x 5632 x 2048 17.8 -> 12.4, 20.7 -> 14.0, 19.5 -> 14.9.  Up to 8 rows mma.sync is 1.1 ... 1.9 times as fast.
bool kq_few_supported(int fmt, size_t M, size_t K, size_t N, bool swiglu, int sm_count) {
    if ((fmt != FMT_Q4_K && fmt != FMT_Q5_K && fmt != FMT_Q6_K) || M < 9 || M >= 64 || K < 256 || K % 256 != 0 || K > 65536 || N < 1 ||
        !tma_available())
        return false;
    const size_t nblk = K / 256, row_tiles = swiglu ? (N + 63) / 64 : (N + 127) / 128, tiles = (N + 127) / 128 * (swiglu ? 2 : 1), chunks = tiles * ((nblk + 15) / 16);
    if (M >= 17) {
        if (swiglu || 8 * tiles > (size_t)sm_count) return true;
        const double pass = fmt == FMT_Q4_K ? 4.6 : fmt == FMT_Q5_K ? 5.0 : 5.2, more = fmt == FMT_Q4_K ? 0.12 : fmt == FMT_Q5_K ? 0.14 : 0.15;
        const double there = 2.5 + (double)((M + 15) / 16) * (pass + (chunks > 10 ? more * (double)(chunks - 10) : 0.0));
        // (a call without scratch of its own must not come to need more than there is: its partial sums grow with K, M and N)
        return 4.2 + kf_plan(fmt, M, K, row_tiles, false, sm_count, true).us < 1.05 * there ||
               gemv_workspace_bytes(fmt, M, K, N, false, sm_count) > B200Q_STATIC_SCRATCH_BYTES;
    }
    if (smallm_i8_preferred(fmt, M, K, N, sm_count)) return false;
    const double there = 5.0 + (double)chunks * (fmt == FMT_Q4_K ? 0.128 : fmt == FMT_Q5_K ? 0.155 : 0.13);
    // (the estimate spares shapes that stay with the other kernel the question how many clusters fit, which loads this one)
    return 4.0 + kf_plan(fmt, M, K, row_tiles, swiglu, sm_count, true).us < 0.95 * there && 4.0 + kf_plan(fmt, M, K, row_tiles, swiglu, sm_count).us < 0.95 * there;
}
int kq_few_tile_rows(int fmt, size_t M, size_t K, size_t N, int sm_count) { return (int)kf_plan(fmt, M, K, (N + 127) / 128, false, sm_count).mt; }

// w_up: SwiGLU of the products with w (gate) and w_up; else null.
cudaError_t launch_kq_few(int fmt, const void* act, int act_dtype, const void* w, const void* w_up, void* out, int out_dtype, size_t M, size_t K,
                          size_t N, void* ws, size_t ws_bytes, int sm_count, cudaStream_t st, unsigned int* status, bool* ws_too_small, char* err,
                          size_t err_len, bool acts_prepared) {
    *ws_too_small = false;
    if (!ws || ws_bytes < kq_i8_workspace_bytes(M, K) || (reinterpret_cast<uintptr_t>(ws) & 15)) {
        *ws_too_small = true;
        return cudaSuccess;
    }
    const uint32_t nblk = (uint32_t)(K / 256);
    uint8_t* codes;
    __half* sums;
    float* d8;
    kq_image(ws, M, K, &codes, &sums, &d8);
    if (!acts_prepared) {
        const cudaError_t e = launch_kq_prep(act, act_dtype, M, K, ws, true, sm_count, st);
        if (e != cudaSuccess) return e;
    }
    KfParams p{};
    const bool swiglu = w_up != nullptr;
    const uint32_t rows = swiglu ? 64 : 128, rt = (uint32_t)((N + rows - 1) / rows);
    const KfPlan pl = kf_plan(fmt, M, K, rt, swiglu, sm_count);
    p.w = static_cast<const uint8_t*>(w);
    p.w_up = static_cast<const uint8_t*>(w_up);
    p.out = out;
    p.N = (uint32_t)N;
    p.d8 = d8;
    p.M = (uint32_t)M;
    p.nblk = nblk;
    p.row_bytes = nblk * (uint32_t)fmt_block_bytes(fmt);
    p.mt = pl.mt;
    p.nct = (uint32_t)((M + pl.mt - 1) / pl.mt);
    p.nunits = rt * p.nct;
    p.cs = pl.cs;
    p.cs_log = pl.cs == 8 ? 3 : pl.cs == 4 ? 2 : pl.cs == 2 ? 1 : 0;
    p.ns = kf_stages(fmt, pl.mt);
    p.nb = kf_acts(fmt, pl.mt);
    p.nr = kf_ring(fmt, pl, swiglu);
    p.off_rec = KF_STAGES + p.nb * kf_btile(pl.mt);
    p.off_raw = p.off_rec + KF_NQ * KF_REC;
    p.off_x = p.off_raw + p.nr * kf_raw(fmt);
    const uint32_t shape = ((p.mt >> 3) << 17) | ((128u >> 4) << 24);  // K-major, N = mt, M = 128
    p.idesc_i = (2u << 4) | (1u << 7) | (1u << 10) | shape;            // int32 <- s8 x s8
    p.idesc_h = (1u << 4) | shape;                                     // f32 <- f16 x f16
    p.out_dtype = out_dtype;
    p.raw_tma = p.row_bytes % 16 == 0;
    p.swiglu = swiglu;
    p.status = status;
    CUtensorMap am, sm, wm[2];
    bool ok = kf_encode(&am, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, codes, K, M, 128, p.mt, CU_TENSOR_MAP_SWIZZLE_128B) &&
              kf_encode(&sm, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, sums, (size_t)nblk * 16, M, 16, p.mt, CU_TENSOR_MAP_SWIZZLE_32B);
    for (int i = 0; i < 2 && ok; ++i) {
        if (p.raw_tma && (i == 0 || swiglu))
            ok = kf_encode(&wm[i], CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, i ? w_up : w, p.row_bytes / 2, N, kf_pitch(fmt) / 2, rows, CU_TENSOR_MAP_SWIZZLE_NONE);
        else
            wm[i] = am;
    }
    if (!ok) {
        snprintf(err, err_len, "cuTensorMapEncodeTiled failed (activation image %p, M=%zu K=%zu)", (void*)codes, M, K);
        return cudaErrorInvalidValue;
    }
    const uint32_t grid = pl.cs > 1 ? p.nunits * pl.cs : p.nunits < (uint32_t)sm_count ? p.nunits : (uint32_t)sm_count;
    const size_t smem = 1024 + p.off_x + kf_x_bytes(pl, swiglu);
    if (pl.cs > 1)
        return fmt == FMT_Q4_K   ? kf_launch<FMT_Q4_K, true>(am, sm, wm, p, grid, smem, st)
               : fmt == FMT_Q5_K ? kf_launch<FMT_Q5_K, true>(am, sm, wm, p, grid, smem, st)
                                 : kf_launch<FMT_Q6_K, true>(am, sm, wm, p, grid, smem, st);
    return fmt == FMT_Q4_K   ? kf_launch<FMT_Q4_K, false>(am, sm, wm, p, grid, smem, st)
           : fmt == FMT_Q5_K ? kf_launch<FMT_Q5_K, false>(am, sm, wm, p, grid, smem, st)
                             : kf_launch<FMT_Q6_K, false>(am, sm, wm, p, grid, smem, st);
}

}  // namespace b200q
