// Quantized matmul of the K-quant formats with the bits of boostr's CPU path
// (src/quant/cpu/kernels/quant_matmul.rs:107-135) on the integer tensor cores: Q2_K and Q3_K for every number of activation
// rows (Q4_K, Q5_K and Q6_K with few rows: kquant_few.cu, which reads the same image).  Each activation row is quantised to Q8_K
// (src/quant/cpu/kernels/simd/quantize_act_q8k.rs:26-98), a 256-block contributes
// (d * d8) * isum - (dmin * d8) * summs with exact integer sums (src/quant/cpu/kernels/simd/fused_q2k_q8k_dot.rs:152-214,
// fused_q3k_q8k_dot.rs:33-205 in the form x86-64 runs; Q3_K has no min term) and the blocks are added in K order without FMA contraction.
//
// What both kernels build on: the PRODUCT of a code and its sub-block's scale goes into the operand, so a whole 256-block is
// one K = 256 integer product and only one sum per (row, activation row, block) has to be scaled.  For Q2_K (0..3 times
// 0..15) and Q3_K (-(-4..3) times -32..31 lies in [-128, 124]; the sign is given back by the f32 factor) it fits a signed
// byte.  The min term is another integer product, of the mins with the activation's sums of 16 codes, which travel as two
// bytes, sum = lo + 16 hi.
//
//   * kq_act_prep_kernel: codes [M][K], min operand [M][K / 256][lo 16 | hi 16], scales d8 [K / 256][M]: 292 bytes per run; below
//     64 rows the sums of 16 also as f16, for kquant_few.cu;
//   * kq_tc_kernel<FMT>: tcgen05.mma.kind::i8, tiles of 128 weight rows x up to 128 activation rows;
//   * kq_small_kernel<FMT, NT>: mma.sync, slabs of 16 weight rows x 8 NT activation rows, Q2_K / Q3_K with few rows.
#include <cuda.h>

#include <cstdio>
#include <type_traits>

#include "common.cuh"
#include "tcgen05_i8.cuh"
#include "tmap.cuh"

namespace b200q {

bool kq_few_supported(int fmt, size_t M, size_t K, size_t N, bool swiglu, int sm_count);
int kq_few_tile_rows(int fmt, size_t M, size_t K, size_t N, int sm_count);

namespace {

constexpr uint32_t RUN_BYTES = 292;  // of scratch per (activation row, 256-block): 256 codes, 32 bytes of sums, f32 d8

// Packed blocks start 4-byte (Q2_K) or 2-byte (Q3_K) aligned in a row and are brought as the 16-byte chunks that hold them:
// CHUNKS at most, PITCH bytes from row to row in shared memory.  (Copies of 4 bytes - cp.async - ran at about one lane per
// cycle and took 2-4 us per 128 rows, more than everything else.)  Any such pitch puts one word of 32 rows into eight banks:
// 112 and 144 use all of these.
__host__ __device__ constexpr uint32_t kq_chunks(int fmt) { return fmt == FMT_Q2_K ? 6 : 8; }
__host__ __device__ constexpr uint32_t kq_pitch(int fmt) { return fmt == FMT_Q2_K ? 112 : 144; }

// One warp per (activation row, 256-block): Q8_K codes (d = amax / 127, id = 127 / amax, round half to even), the sums of
// 16 codes as lo + 16 hi with lo in [-8, 7] (a sum is at most 2048 in size, so hi fits a signed byte), the scale.
template <typename InT>
__global__ void __launch_bounds__(256) kq_act_prep_kernel(const InT* __restrict__ act, uint8_t* __restrict__ codes, uint8_t* __restrict__ mins,
                                                          float* __restrict__ d8, __half* __restrict__ sums, size_t M, uint32_t nblk, bool early) {
    const int lane = threadIdx.x & 31;
    // The product reads its packed weights as soon as it is started.  Q2_K and Q3_K weights may have been written by whatever ran
    // before this kernel; those of the other formats are complete before a call of so few rows (include/b200q.h), and their
    // product starts beside that kernel's tail: 2 us of 25 ... 36 a call.
    if (early) grid_dep_launch();
    grid_dep_wait();  // the activations may be the previous kernel's output; the image may still be read by it
    if (!early) grid_dep_launch();
    const size_t nruns = M * nblk;
    for (size_t run = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5); run < nruns; run += (size_t)gridDim.x * 8) {
        float v[8];
        const size_t base = run * 256 + 8 * lane;
        if constexpr (sizeof(InT) == 4) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(act + base)), b = __ldg(reinterpret_cast<const float4*>(act + base) + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
            const uint4 r = __ldg(reinterpret_cast<const uint4*>(act + base));
            v[0] = __uint_as_float(r.x << 16); v[1] = __uint_as_float(r.x & 0xFFFF0000u);
            v[2] = __uint_as_float(r.y << 16); v[3] = __uint_as_float(r.y & 0xFFFF0000u);
            v[4] = __uint_as_float(r.z << 16); v[5] = __uint_as_float(r.z & 0xFFFF0000u);
            v[6] = __uint_as_float(r.w << 16); v[7] = __uint_as_float(r.w & 0xFFFF0000u);
        }
        float amax = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
        const float id = amax != 0.f ? __fdiv_rn(127.0f, amax) : 0.f;
        int c[8], s = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            c[i] = max(-128, min(127, __float2int_rn(__fmul_rn(v[i], id))));  // round half to even, as the AVX2 quantiser
            s += c[i];
        }
        uint32_t w0 = 0, w1 = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            w0 |= (uint32_t)(c[i] & 0xFF) << (8 * i);
            w1 |= (uint32_t)(c[4 + i] & 0xFF) << (8 * i);
        }
        *reinterpret_cast<uint2*>(codes + base) = make_uint2(w0, w1);
        s += __shfl_xor_sync(0xFFFFFFFFu, s, 1);  // 16 codes = two lanes
        if ((lane & 1) == 0) {
            const int hi = (s + 8) >> 4;
            mins[run * 32 + (lane >> 1)] = (uint8_t)(s - 16 * hi);
            mins[run * 32 + 16 + (lane >> 1)] = (uint8_t)hi;
            if (sums) sums[run * 16 + (lane >> 1)] = __int2half_rn(s);  // at most 2048 in size: exact
        }
        const size_t m = run / nblk, b = run % nblk;
        if (lane == 0) d8[b * M + m] = __fdiv_rn(amax, 127.0f);
    }
}

// ------------------------------------------------------------------------------------------ scaled codes of a block
// Q2_K (src/quant/cpu/kernels/dequant_k_quants/q2k_q3k.rs:13-58): 16 bytes scale | min << 4, 64 code bytes, f16 d, f16 dmin;
// element 128 n + 32 g + 16 h + l takes bits 2g..2g+1 of code byte 32 n + 16 h + l and the scale of sub-block 8 n + 2 g + h.
// Four codes (bytes 0..3) times one scale below 16 cannot carry into the next byte.
template <int G>
__device__ __forceinline__ uint32_t q2k_scaled(uint32_t w, uint32_t sc) {
    return ((w >> (2 * G)) & 0x03030303u) * sc;
}
// Q3_K (q2k_q3k.rs:64-144): 32 bytes of high bits, 64 code bytes as Q2_K, 12 bytes of 6-bit scales (plus 32), f16 d; the high
// bit 4 n + g of byte 16 h + l, clear, subtracts 4.  With c = 0..7 and the stored scale u = s + 32, the byte wanted is
// -s (c - 4) = c (32 - u) + 4 u - 128; c (32 - u) + 4 u lies in 0..252, so the four bytes of a word come out of ONE
// multiply-add exactly and the 128 is a sign-bit flip.  `hw`: high bits shifted right by 4 n.
template <int G>
__device__ __forceinline__ uint32_t q3k_scaled(uint32_t w, uint32_t hw, uint32_t neg_s, uint32_t u4) {
    const uint32_t high = (G < 2 ? hw << (2 - G) : hw >> (G - 2)) & 0x04040404u;
    const uint32_t c = ((w >> (2 * G)) & 0x03030303u) | high;
    return (c * neg_s + u4) ^ 0x80808080u;
}
__device__ __forceinline__ uint32_t byte_of(uint32_t x, uint32_t i) { return __byte_perm(x, 0u, 0x4440u | i); }

__device__ __forceinline__ void store_as(void* out, int dt, size_t idx, float v) {
    if (dt == DT_F32) static_cast<float*>(out)[idx] = v;
    else if (dt == DT_BF16) static_cast<__nv_bfloat16*>(out)[idx] = __float2bfloat16_rn(v);
    else static_cast<__half*>(out)[idx] = __float2half_rn(v);
}

// Eight lanes a row copy the 16-byte chunks of the blocks at blk, blk + row_bytes, ... (ROWS of them, `in` of which exist) to
// dst, one PITCH apart; each lands at byte (its address & 15) of its slot.  Rows that do not exist are left as they are:
// their sums are never stored.  `inner`: all exist and none is the tensor's last row, whose last chunk may reach past the
// end and is clipped there.
template <int FMT, uint32_t ROWS>
__device__ __forceinline__ void copy_rows(uint32_t dst, const uint8_t* blk, uint32_t row_bytes, uint32_t lane, bool inner, uint32_t in, const uint8_t* wend) {
    const uint32_t c = lane & 7, r0 = lane >> 3;
    if (c >= kq_chunks(FMT)) return;
    const uint8_t* src = blk + (size_t)r0 * row_bytes;
    dst += r0 * kq_pitch(FMT) + 16 * c;
    auto chunk = [&](const uint8_t* q) { return reinterpret_cast<const uint8_t*>((reinterpret_cast<uintptr_t>(q) & ~(uintptr_t)15) + 16 * c); };
    if (inner) {
#pragma unroll
        for (uint32_t q = 0; q < ROWS; q += 4) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + q * kq_pitch(FMT)), "l"(chunk(src)) : "memory");
            src += 4 * (size_t)row_bytes;
        }
        return;
    }
#pragma unroll 1
    for (uint32_t q = r0; q < ROWS && q < in; q += 4) {
        const uint8_t* s = chunk(src);
        if (s < wend)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(s), "r"(min(16u, (uint32_t)(wend - s))) : "memory");
        src += 4 * (size_t)row_bytes;
        dst += 4 * kq_pitch(FMT);
    }
}

// =================================================================================================== tensor-core kernel
// One CTA per SM, persistent over (128 weight rows, mt activation rows) tiles, all of K each (the sums grow in K order, so
// no tile is cut).  Per 256-block: the 128 packed blocks come by TMA (by cp.async from two warps where rows are not 16-byte aligned),
// two sets of four decode warps, taking the blocks in turn, write the scaled codes as 128-byte-swizzled K-major operand tiles,
// the activation codes come by TMA, one thread issues 8 MMAs
// (+ 2 for the mins) into one of two accumulators, and sixteen drain warps (thread = weight
// row x every fourth group of 8 activation rows) scale the sums and add them to their registers.
// What bounds it: with 128 activation rows a tile the issue slots (Q2_K 72 %, Q3_K 67 % busy; ALU pipe 41 / 55 %, tensor pipe
// 20 / 18 %): decode, and 8 (Q2_K) or 5 (Q3_K) instructions a sum of drain; with few the latency of a block's chain through
// the barriers, the proxy fence and two decode sets, 0.8 us a block.  Measured: 512 rows x 14336 x 4096 Q2_K 99 us, Q3_K 93 us (a layer of such
// products 0.42 ms; 69 ms with a kernel that took eight rows at a time).  Tried and not kept: packed f32x2
// arithmetic in the drain, which suits one format and not the other (Q2_K 107, Q3_K 87 us) and needs an operand hidden from
// the assembler, which else makes one rounding of mul.rn.f32x2 and add.rn.f32x2; and halves of a block as stages
// (4096 x 14336 at 64 rows 49 -> 58 us).
struct KqTcParams {
    const uint8_t* w;
    void* out;
    const float* d8;  // [nblk][M]
    uint32_t M, N, nblk;
    uint32_t mt;              // activation rows of a tile: a multiple of 16, at most 128
    uint32_t nct, nunits;     // column tiles; row tiles x column tiles
    uint32_t row_bytes;
    bool raw_tma;             // rows start 16-byte aligned: packed blocks come by TMA
    uint32_t idesc;
    int out_dtype;
    unsigned int* status;
};

constexpr int KT_DEC = 8, KT_DRAIN = 16, KT_COPY = 2;
constexpr int KT_W_COPY = KT_DEC + KT_DRAIN, KT_W_ACT = KT_W_COPY + KT_COPY, KT_W_MMA = KT_W_ACT + 1;
constexpr int KT_THREADS = (KT_W_MMA + 1) * 32;
constexpr uint32_t KT_NS = 2, KT_NQ = 4;
constexpr uint32_t KT_NR = 4;
constexpr uint32_t KT_ATOM = 128 * 128;
constexpr uint32_t KT_REC = 512 + 512;  // the rows' d | dmin, the activation rows' d8
// Every ring has an even depth: the decode sets take the blocks in turn, so a slot belongs to one set, which sees every
// phase of the slot's barriers (a parity wait cannot tell phase k from k - 2).
constexpr int KO_FULL = 0, KO_EMPTY = 32, KO_RAW_FULL = 64, KO_RAW_EMPTY = 96, KO_ACC_FULL = 128, KO_ACC_EMPTY = 144, KO_REC_FULL = 160,
              KO_REC_EMPTY = 192, KO_TMEM = 224, KO_DEAD = 228, KO_RECS = 1024, KO_STAGES = KO_RECS + KT_NQ * KT_REC;
// a stage: two operand tiles of scaled codes | tile of mins | two tiles of activation codes | sums of 16
constexpr uint32_t KT_MT_MAX = 128;
__host__ __device__ constexpr uint32_t kt_stage(int fmt) {
    return (2 * KT_ATOM + (fmt == FMT_Q3_K ? 0 : 128 * 64) + KT_MT_MAX * (256 + (fmt == FMT_Q3_K ? 0 : 32)) + 1023) / 1024 * 1024;
}
__host__ __device__ constexpr uint32_t kt_raw(int fmt) { return 128 * kq_pitch(fmt); }
__host__ __device__ constexpr size_t kt_smem(int fmt) { return 1024 + KO_STAGES + KT_NS * kt_stage(fmt) + KT_NR * kt_raw(fmt); }
static_assert(KO_STAGES % 1024 == 0 && kt_smem(FMT_Q2_K) <= 232448 && kt_smem(FMT_Q3_K) <= 232448, "shared memory");

// rows of 64 bytes with 64-byte swizzle (8-row groups 512 bytes apart) and of 32 bytes with 32-byte swizzle
__device__ __forceinline__ uint64_t desc_sw64(uint32_t lo) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"((512u >> 4) | (1u << 14) | (4u << 29)));
    return d;
}
__device__ __forceinline__ uint64_t desc_sw32(uint32_t lo) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"((256u >> 4) | (1u << 14) | (6u << 29)));
    return d;
}

template <int FMT>
__global__ void __launch_bounds__(KT_THREADS, 1) kq_tc_kernel(const __grid_constant__ CUtensorMap tmap_act, const __grid_constant__ CUtensorMap tmap_min,
                                                              const __grid_constant__ CUtensorMap tmap_w, const KqTcParams p) {
    constexpr bool MIN = FMT != FMT_Q3_K;
    constexpr uint32_t BB = fmt_block_bytes(FMT), PITCH = kq_pitch(FMT), RAW = kt_raw(FMT), STAGE = kt_stage(FMT), NR = KT_NR;
    constexpr uint32_t MT_MAX = KT_MT_MAX, B_TILE = MT_MAX * 128, CHUNKS = (MT_MAX / 8 + 3) / 4;  // groups of 8 activation rows of a drain warp
    constexpr uint32_t OFF_AM = 2 * KT_ATOM, OFF_B = OFF_AM + (MIN ? 128 * 64 : 0), OFF_BM = OFF_B + 2 * B_TILE;
    // an accumulator: sums (| mins)
    constexpr uint32_t COL = 128, ACC_COLS = MIN ? 256 : 128, TMEM_COLS = 2 * ACC_COLS;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // the launch reserves 1 KB of slack
    const uint32_t sbase = smem_u32(smem), st_base = sbase + KO_STAGES;
    constexpr uint32_t OFF_RAW = KO_STAGES + KT_NS * STAGE;
    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    volatile uint32_t* dead = reinterpret_cast<volatile uint32_t*>(smem + KO_DEAD);
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < KT_NS; ++s) {
            mbar_init(sbase + KO_FULL + 8 * s, 5);   // four decode warps + the activation copies (with their byte count)
            mbar_init(sbase + KO_EMPTY + 8 * s, 1);  // the commit behind the block's MMAs
        }
        for (uint32_t s = 0; s < NR; ++s) {
            mbar_init(sbase + KO_RAW_FULL + 8 * s, p.raw_tma ? 1 : KT_COPY * 32);  // the TMA copy, or every copying thread
            mbar_init(sbase + KO_RAW_EMPTY + 8 * s, 4);
        }
        for (uint32_t s = 0; s < 2; ++s) {
            mbar_init(sbase + KO_ACC_FULL + 8 * s, 1);
            mbar_init(sbase + KO_ACC_EMPTY + 8 * s, KT_DRAIN);
        }
        for (uint32_t s = 0; s < KT_NQ; ++s) {
            mbar_init(sbase + KO_REC_FULL + 8 * s, 4 + 32);  // four decode warps + the lanes that copy d8
            mbar_init(sbase + KO_REC_EMPTY + 8 * s, KT_DRAIN);
        }
        *dead = 0;
        mbar_fence_init();
    }
    if (warp == KT_W_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + KO_TMEM), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + KO_TMEM);
    grid_dep_launch();
    // A wait of a whole warp: all lanes leave together; on a timeout the CTA is marked dead and every role ends.
    auto wait = [&](uint32_t off, uint32_t parity, unsigned int code) {
        const bool ok = __all_sync(0xFFFFFFFFu, i8_wait(sbase + off, parity, dead));
        if (!ok && lane == 0) i8_fail(dead, p.status, code);
        return ok;
    };
    // blocks of this CTA: its units (blockIdx.x, + gridDim.x, ...) one after the other, nblk blocks each
    const uint32_t units = (p.nunits - blockIdx.x + gridDim.x - 1) / gridDim.x, total = units * p.nblk;

    if (warp >= KT_W_COPY && warp < KT_W_ACT) {
        // ------------------------------------------------------------ packed blocks (do not depend on the kernel that is still running)
        const uint32_t r0 = (uint32_t)(warp - KT_W_COPY) * (128 / KT_COPY);
        const uint8_t* wend = p.w + (size_t)p.N * p.row_bytes;
        uint32_t unit = blockIdx.x, b = 0, n0 = unit / p.nct * 128 + r0;
        // By TMA one warp brings the packed blocks and the other has no part in the ring: a warp that waited on RAW_EMPTY without
        // being counted in RAW_FULL could miss a phase, and at the end of the work would wait for one that never comes.
        const uint32_t mine = p.raw_tma && warp != KT_W_COPY ? 0 : total;
        for (uint32_t i = 0; i < mine; ++i) {
            const uint32_t rs = i % NR;
            if (!wait(KO_RAW_EMPTY + 8 * rs, ((i / NR) & 1) ^ 1, STATUS_TIMEOUT_EMPTY)) break;
            if (p.raw_tma) {  // one copy a block: rows past N and bytes past the row's end are zero-filled
                if (lane == 0) {
                    mbar_expect_tx(sbase + KO_RAW_FULL + 8 * rs, RAW);
                    tma2d(sbase + OFF_RAW + rs * RAW, &tmap_w, (int)((b * BB & ~15u) / 2), (int)n0, sbase + KO_RAW_FULL + 8 * rs);
                    // The block that this slot takes next goes to L2: what is in flight into shared memory does not cover the
                    // latency of DRAM.
                    if (i + NR < total) {
                        const uint32_t ab = b + NR, at_b = ab < p.nblk ? ab : ab % p.nblk, at_n = ab < p.nblk ? n0 : (unit + ab / p.nblk * gridDim.x) / p.nct * 128;
                        asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(&tmap_w), "r"((int)((at_b * BB & ~15u) / 2)), "r"((int)at_n)
                                     : "memory");
                    }
                }
            } else {
                copy_rows<FMT, 128 / KT_COPY>(sbase + OFF_RAW + rs * RAW + r0 * PITCH, p.w + (size_t)n0 * p.row_bytes + (size_t)b * BB, p.row_bytes, lane,
                                              n0 + 128 / KT_COPY < p.N, n0 < p.N ? p.N - n0 : 0u, wend);
            }
            if (!p.raw_tma)  // arrives once this thread's copies have landed
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(sbase + KO_RAW_FULL + 8 * rs) : "memory");
            if (++b == p.nblk) {
                b = 0;
                unit += gridDim.x;
                n0 = unit / p.nct * 128 + r0;
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == KT_W_ACT) {
        // ------------------------------------------------------------ activation codes, sums and scales (previous kernel's output)
        grid_dep_wait();
        uint32_t unit = blockIdx.x, b = 0, m0 = unit % p.nct * p.mt;
        for (uint32_t i = 0; i < total; ++i) {
            const uint32_t s = i % KT_NS, q = i % KT_NQ;
            const uint32_t st = st_base + s * STAGE;
            if (!wait(KO_EMPTY + 8 * s, ((i / KT_NS) & 1) ^ 1, STATUS_TIMEOUT_EMPTY)) break;
            if (lane == 0) {
                const uint32_t bar = sbase + KO_FULL + 8 * s;
                mbar_expect_tx(bar, 256 * p.mt + (MIN ? 32 * p.mt : 0));
                tma2d(st + OFF_B, &tmap_act, (int)(b * 256), (int)m0, bar);
                tma2d(st + OFF_B + B_TILE, &tmap_act, (int)(b * 256 + 128), (int)m0, bar);
                if constexpr (MIN) tma2d(st + OFF_BM, &tmap_min, (int)(b * 32), (int)m0, bar);
            }
            __syncwarp();
            if (!wait(KO_REC_EMPTY + 8 * q, ((i / KT_NQ) & 1) ^ 1, STATUS_TIMEOUT_EMPTY)) break;
            const uint32_t dst = sbase + KO_RECS + q * KT_REC + 512;
            const float* src = p.d8 + (size_t)b * p.M + m0;
            for (uint32_t m = lane; m < p.mt; m += 32)  // rows past M are zero-filled
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * m), "l"(m0 + m < p.M ? src + m : p.d8), "r"(m0 + m < p.M ? 4u : 0u) : "memory");
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(sbase + KO_REC_FULL + 8 * q) : "memory");
            if (++b == p.nblk) {
                b = 0;
                unit += gridDim.x;
                m0 = unit % p.nct * p.mt;
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (*dead) {  // TMA copies in flight land within microseconds: the CTA's shared memory stays until then
            const uint64_t t0 = global_timer_ns();
            while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
        }
    } else if (warp == KT_W_MMA) {
        // ------------------------------------------------------------ MMA issue
        for (uint32_t i = 0; i < total; ++i) {
            const uint32_t s = i % KT_NS, buf = i & 1;
            const uint32_t st = st_base + s * STAGE, a_lo = desc_lo(st), b_lo = desc_lo(st + OFF_B), d = tmem + buf * ACC_COLS;
            if (!wait(KO_ACC_EMPTY + 8 * buf, ((i >> 1) & 1) ^ 1, STATUS_TIMEOUT_EMPTY)) break;
            if (!wait(KO_FULL + 8 * s, (i / KT_NS) & 1, STATUS_TIMEOUT_FULL)) break;
            tc_after();
            if (elect_one_lane()) {
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k)
                    tc_mma_i8(d, desc_sw128(a_lo + (k >> 2) * (KT_ATOM >> 4) + 2 * (k & 3)), desc_sw128(b_lo + (k >> 2) * (B_TILE >> 4) + 2 * (k & 3)), p.idesc, k > 0);
                if constexpr (MIN) {
                    // sum of 16 = lo + 16 hi in one accumulator, [m | 8 m] . [lo | hi] + [0 | 8 m] . [lo | hi]
                    const uint32_t am = desc_lo(st + OFF_AM), bm = desc_lo(st + OFF_BM);
                    tc_mma_i8(d + COL, desc_sw64(am), desc_sw32(bm), p.idesc, false);
                    tc_mma_i8(d + COL, desc_sw64(am + 2), desc_sw32(bm), p.idesc, true);
                }
                tc_commit_to(sbase + KO_EMPTY + 8 * s);       // the stage may be overwritten once these MMAs have read it
                tc_commit_to(sbase + KO_ACC_FULL + 8 * buf);  // and the sums are complete
            }
            __syncwarp();
        }
    } else if (warp < KT_DEC) {
        // ------------------------------------------------------------ decode: one thread per weight row, the sets take blocks in turn
        const uint32_t r = threadIdx.x & 127, set = (uint32_t)warp >> 2, x7 = r & 7;
        uint32_t b = set % p.nblk;  // block of K
        for (uint32_t i = set; i < total; i += 2, b += 2, b -= b >= p.nblk ? p.nblk : 0, b -= b >= p.nblk ? p.nblk : 0) {
            const uint32_t rs = i % NR, s = i % KT_NS, q = i % KT_NQ;
            if (!wait(KO_RAW_FULL + 8 * rs, (i / NR) & 1, STATUS_TIMEOUT_FULL)) break;
            const uint32_t at = (r * p.row_bytes + b * BB) & 15u;  // where the row's block sits in its slot (128 rows are a multiple of 16 bytes)
            const uint32_t* raw = reinterpret_cast<const uint32_t*>(smem + OFF_RAW + rs * RAW + r * PITCH + (at & 12u));
            uint32_t* rec = reinterpret_cast<uint32_t*>(smem + KO_RECS + q * KT_REC) + r;
            uint8_t* a0 = smem + KO_STAGES + s * STAGE + (r >> 3) * 1024 + x7 * 128;
            auto put = [&](uint32_t plane, uint32_t c, uint4 v) { *reinterpret_cast<uint4*>(a0 + plane * KT_ATOM + ((c ^ x7) << 4)) = v; };
            uint32_t dm = 0;
            bool lost = false;
#pragma unroll
            for (uint32_t n = 0; n < 2; ++n) {  // the halves of the block: operand tiles n (and 2 + n)
                // All words of the half leave shared memory before the first store into the operand: nothing waits on a load in the
                // middle of the arithmetic.
                uint32_t cw[8], hw[8], sw[4];  // d (| dmin); codes; high bits; scales
                if constexpr (FMT == FMT_Q2_K) {
                    dm = raw[20];
#pragma unroll
                    for (int k = 0; k < 4; ++k) sw[k] = raw[k];
#pragma unroll
                    for (int k = 0; k < 8; ++k) cw[k] = raw[4 + 8 * n + k];
                } else {
                    const uint32_t sh = 8 * (at & 2u);
                    uint32_t u[9], v[9], x[4];
#pragma unroll
                    for (int k = 0; k < 9; ++k) {
                        u[k] = raw[k];
                        v[k] = raw[8 + 8 * n + k];
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) x[k] = raw[24 + k];
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        hw[k] = __funnelshift_r(u[k], u[k + 1], sh) >> (4 * n);
                        cw[k] = __funnelshift_r(v[k], v[k + 1], sh);
                    }
#pragma unroll
                    for (int k = 0; k < 3; ++k) sw[k] = __funnelshift_r(x[k], x[k + 1], sh);
                    dm = (x[3] >> sh) & 0xFFFFu;
                }
                if (n == 1) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(sbase + KO_RAW_EMPTY + 8 * rs);
                } else if (!wait(KO_EMPTY + 8 * s, ((i / KT_NS) & 1) ^ 1, STATUS_TIMEOUT_EMPTY)) {
                    lost = true;
                    break;
                }
                if (MIN && n == 0) {  // the tile of mins, 64 bytes a row
                    const uint4 mn = make_uint4((sw[0] >> 4) & 0x0F0F0F0Fu, (sw[1] >> 4) & 0x0F0F0F0Fu, (sw[2] >> 4) & 0x0F0F0F0Fu, (sw[3] >> 4) & 0x0F0F0F0Fu);
                    const uint4 m8 = make_uint4(mn.x << 3, mn.y << 3, mn.z << 3, mn.w << 3);
                    uint4* am = reinterpret_cast<uint4*>(smem + KO_STAGES + s * STAGE + OFF_AM + r * 64);
                    const uint32_t x3 = (r >> 1) & 3;
                    am[0 ^ x3] = mn;
                    am[1 ^ x3] = m8;
                    am[2 ^ x3] = make_uint4(0, 0, 0, 0);
                    am[3 ^ x3] = m8;
                }
                {
                    uint32_t scw[2];  // the half's eight scales
                    if constexpr (FMT == FMT_Q2_K) {
                        scw[0] = (n ? sw[2] : sw[0]) & 0x0F0F0F0Fu;
                        scw[1] = (n ? sw[3] : sw[1]) & 0x0F0F0F0Fu;
                    } else {
                        scw[0] = ((sw[0] >> (4 * n)) & 0x0F0F0F0Fu) | ((n ? sw[2] : sw[2] << 4) & 0x30303030u);
                        scw[1] = ((sw[1] >> (4 * n)) & 0x0F0F0F0Fu) | ((n ? sw[2] >> 2 : sw[2] << 2) & 0x30303030u);
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        auto one = [&](auto gc) {  // sub-block 8 n + 2 g + h = 16-byte chunk 2 g + h of the tile
                            constexpr int G = decltype(gc)::value;
                            const uint32_t sc = byte_of(scw[G >> 1], 2 * (G & 1) + h);
                            uint32_t v[4];
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                if constexpr (FMT == FMT_Q2_K) v[k] = q2k_scaled<G>(cw[4 * h + k], sc);
                                else v[k] = q3k_scaled<G>(cw[4 * h + k], hw[4 * h + k], 32u - sc, sc * 0x04040404u);
                            }
                            put(n, 2 * G + h, make_uint4(v[0], v[1], v[2], v[3]));
                        };
                        one(std::integral_constant<int, 0>{});
                        one(std::integral_constant<int, 1>{});
                        one(std::integral_constant<int, 2>{});
                        one(std::integral_constant<int, 3>{});
                    }
                }
            }
            if (lost) break;
            proxy_fence();  // the operand bytes are read by the tensor core (async proxy)
            __syncwarp();
            if (lane == 0) mbar_arrive(sbase + KO_FULL + 8 * s);
            if (!wait(KO_REC_EMPTY + 8 * q, ((i / KT_NQ) & 1) ^ 1, STATUS_TIMEOUT_EMPTY)) break;
            *rec = dm;
            __syncwarp();
            if (lane == 0) mbar_arrive(sbase + KO_REC_FULL + 8 * q);
        }
    } else {
        // ------------------------------------------------------------ drain: integer sums -> scaled f32 terms, in K order
        const uint32_t quarter = warp & 3, cg = (uint32_t)(warp - KT_DEC) >> 2, r = quarter * 32 + lane;
        const uint32_t t_base = tmem + ((quarter * 32) << 16);
        float sum[CHUNKS][8];  // activation rows 8 (cg + 4 c) + j
        grid_dep_wait();  // the output may still be in use by the previous kernel
        uint32_t unit = blockIdx.x, b = 0;
        for (uint32_t i = 0; i < total; ++i) {
            const uint32_t q = i % KT_NQ, buf = i & 1;
            if (!wait(KO_REC_FULL + 8 * q, (i / KT_NQ) & 1, STATUS_TIMEOUT_FULL)) break;
            const uint8_t* rec = smem + KO_RECS + q * KT_REC;
            const uint32_t dm = reinterpret_cast<const uint32_t*>(rec)[r];
            const float df = f16bits_to_f32(dm & 0xFFFF);
            const float d = MIN ? df : -df, dmin = MIN ? f16bits_to_f32(dm >> 16) : 0.f;
            if (b == 0)
#pragma unroll
                for (int c = 0; c < (int)CHUNKS; ++c)
#pragma unroll
                    for (int j = 0; j < 8; ++j) sum[c][j] = 0.f;
            if (!wait(KO_ACC_FULL + 8 * buf, (i >> 1) & 1, STATUS_TIMEOUT_MMA)) break;
            tc_after();
#pragma unroll
            for (int c = 0; c < (int)CHUNKS; ++c) {
                const uint32_t col = 8 * (cg + 4 * c);
                if (col < p.mt) {  // warp-uniform
                    uint32_t v[8], u[8];
                    const uint32_t tc = t_base + buf * ACC_COLS + col;
                    tmem_ld8_async(tc, v);
                    if constexpr (MIN) tmem_ld8_async(tc + COL, u);
                    const float4* d8 = reinterpret_cast<const float4*>(rec + 512 + 4 * col);
                    const float4 e0 = d8[0], e1 = d8[1];
                    const float e[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float t = __fmul_rn(__fmul_rn(d, e[j]), (float)(int)v[j]);
                        if constexpr (MIN) t = __fsub_rn(t, __fmul_rn(__fmul_rn(dmin, e[j]), (float)(int)u[j]));
                        sum[c][j] = __fadd_rn(sum[c][j], t);
                    }
                }
            }
            tc_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(sbase + KO_ACC_EMPTY + 8 * buf);
                mbar_arrive(sbase + KO_REC_EMPTY + 8 * q);
            }
            if (++b < p.nblk) continue;
            b = 0;
            const uint32_t n = unit / p.nct * 128 + r, m0 = unit % p.nct * p.mt;
            unit += gridDim.x;
            if (n < p.N)
#pragma unroll
                for (int c = 0; c < (int)CHUNKS; ++c)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint32_t m = 8 * (cg + 4 * c) + j;
                        if (m < p.mt && m0 + m < p.M)
                            store_as(p.out, p.out_dtype, (size_t)(m0 + m) * p.N + n, sum[c][j]);
                    }
        }
    }
    tc_before();
    __syncthreads();
    if (warp == KT_W_MMA) {
        tc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// ================================================================================================== few activation rows
// CTA = 16 warps and a contiguous range of 16-row slabs; an item is one (slab, 256-block), the items of the CTA in order are
// dealt to its warps in turn.  A warp brings its items through a private ring (cp.async, no barrier), multiplies the 16
// rows with 8 NT activation rows (8 mma.sync per 8 activation rows; one more for the mins), scales the sums and leaves the
// 16 x 8 NT terms in a table.  Once per R items the CTA meets and a few warps (in turn) add the terms of every slab in K
// order.  Inside a block the operand's K order is free: lane t of a quad takes the 16 code bytes 16 t .. of its row, whose
// four bit pairs belong to four sub-blocks, and the same elements of the activation row (16-byte loads of the code image).
// What bounds it: shared-memory and integer instructions (issue slots 41 ... 44 % busy, ALU pipe 32 ... 46 %; a lane's words of a
// row lie in eight banks, 4 cycles a load).  4 rows x 14336 x 4096: Q2_K 13.1 us (1.47 TB/s), Q3_K 16.2 us (1.56 TB/s); with
// copies of 4 bytes Q3_K 24.8 us.
struct KqSmallParams {
    const uint8_t *w, *codes, *mins;
    const float* d8;
    void* out;
    uint32_t M, N, nblk, row_bytes;
    uint32_t m_first;  // activation row of the grid's first group
    int out_dtype;
};
constexpr int KS_WARPS = 16;
__host__ __device__ constexpr uint32_t ks_depth(int fmt, int nt) { return fmt == FMT_Q2_K ? (nt == 4 ? 5 : 6) : (nt == 4 ? 3 : 5); }  // ring slots of a warp
__host__ __device__ constexpr uint32_t ks_slot(int fmt) { return 16 * kq_pitch(fmt); }  // bytes of an item
__host__ __device__ constexpr uint32_t ks_round(int nt) { return nt == 1 ? 32 : 16; }    // items between two meetings
constexpr uint32_t KS_COL = 20;  // floats from one activation row's 16 terms to the next: 8 lanes x 4 quads hit 32 banks
__host__ __device__ constexpr uint32_t ks_table(int nt) { return ks_round(nt) * 8 * nt * KS_COL * 4; }
__host__ __device__ constexpr size_t ks_smem(int fmt, int nt) { return KS_WARPS * ks_depth(fmt, nt) * ks_slot(fmt) + 2 * ks_table(nt) + 128 * nt * 4; }
static_assert(ks_smem(FMT_Q2_K, 1) <= 232448 && ks_smem(FMT_Q3_K, 4) <= 232448 && ks_smem(FMT_Q2_K, 4) <= 232448, "shared memory");

// The operand words of one row of an item: v[g][k] = scaled codes of bit pair g, word k of the lane's 16 code bytes.
__device__ __forceinline__ void q2k_row(const uint32_t* raw, uint32_t t, uint32_t (&v)[4][4]) {
    const uint32_t n = t >> 1, h8 = 8 * (t & 1);
    const uint32_t s0 = (raw[2 * n] >> h8) & 0x000F000Fu, s1 = (raw[2 * n + 1] >> h8) & 0x000F000Fu;
    const uint32_t sc[4] = {s0 & 0xFFu, s0 >> 16, s1 & 0xFFu, s1 >> 16};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t w = raw[4 + 4 * t + k];
        v[0][k] = q2k_scaled<0>(w, sc[0]);
        v[1][k] = q2k_scaled<1>(w, sc[1]);
        v[2][k] = q2k_scaled<2>(w, sc[2]);
        v[3][k] = q2k_scaled<3>(w, sc[3]);
    }
}
__device__ __forceinline__ void q3k_row(const uint32_t* raw, uint32_t sh, uint32_t t, uint32_t (&v)[4][4]) {
    const uint32_t n = t >> 1, h = t & 1;
    auto word = [&](uint32_t k) { return __funnelshift_r(raw[k], raw[k + 1], sh); };
    const uint32_t l0 = word(24) >> (4 * n), l1 = word(25) >> (4 * n), hh = word(26);
    const uint32_t sa = (l0 & 0x0F0F0F0Fu) | ((n ? hh : hh << 4) & 0x30303030u), sb = (l1 & 0x0F0F0F0Fu) | ((n ? hh >> 2 : hh << 2) & 0x30303030u);
    const uint32_t u[4] = {byte_of(sa, h), byte_of(sa, 2 + h), byte_of(sb, h), byte_of(sb, 2 + h)};
    uint32_t ns[4], u4[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        ns[g] = 32u - u[g];
        u4[g] = u[g] * 0x04040404u;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t w = word(8 + 4 * t + k), hw = word(4 * h + k) >> (4 * n);
        v[0][k] = q3k_scaled<0>(w, hw, ns[0], u4[0]);
        v[1][k] = q3k_scaled<1>(w, hw, ns[1], u4[1]);
        v[2][k] = q3k_scaled<2>(w, hw, ns[2], u4[2]);
        v[3][k] = q3k_scaled<3>(w, hw, ns[3], u4[3]);
    }
}

template <int FMT, int NT>
__global__ void __launch_bounds__(KS_WARPS * 32, 1) kq_small_kernel(const KqSmallParams p) {
    constexpr bool MIN = FMT == FMT_Q2_K;
    constexpr uint32_t BB = fmt_block_bytes(FMT), PITCH = kq_pitch(FMT), DEPTH = ks_depth(FMT, NT), SLOT = ks_slot(FMT), R = ks_round(NT);
    constexpr uint32_t ITEM = 8 * NT * KS_COL;  // floats of an item's terms
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint32_t ring = smem_u32(smem) + warp * DEPTH * SLOT;
    float* table = reinterpret_cast<float*>(smem + KS_WARPS * DEPTH * SLOT);
    float* run = table + 2 * R * ITEM;  // running sums of the slab that the last round left unfinished
    const uint32_t m_base = p.m_first + blockIdx.y * 8 * NT, nslab = (p.N + 15) / 16;
    const uint32_t s_lo = (uint32_t)((uint64_t)nslab * blockIdx.x / gridDim.x), s_hi = (uint32_t)((uint64_t)nslab * (blockIdx.x + 1) / gridDim.x);
    const uint32_t total = (s_hi - s_lo) * p.nblk;
    const uint8_t* wend = p.w + (size_t)p.N * p.row_bytes;
    grid_dep_launch();

    const uint32_t step_s = KS_WARPS / p.nblk, step_b = KS_WARPS % p.nblk;  // KS_WARPS items further, in slabs and blocks
    uint32_t fx = warp, fb = warp % p.nblk, fn = (s_lo + warp / p.nblk) * 16, fslot = 0;  // next item to fetch: its block, first row and ring slot
    auto fetch = [&]() {
        if (fx < total)
            copy_rows<FMT, 16>(ring + fslot * SLOT, p.w + (size_t)fn * p.row_bytes + (size_t)fb * BB, p.row_bytes, lane, fn + 16 < p.N, p.N - fn, wend);
        asm volatile("cp.async.commit_group;" ::: "memory");
        fx += KS_WARPS;
        fn += 16 * step_s;
        fb += step_b;
        if (fb >= p.nblk) {
            fb -= p.nblk;
            fn += 16;
        }
        if (++fslot == DEPTH) fslot = 0;
    };
#pragma unroll 1
    for (uint32_t k = 0; k + 1 < DEPTH; ++k) fetch();
    if (threadIdx.x < 128 * NT) run[threadIdx.x] = 0.f;
    grid_dep_wait();

    uint4 bf[NT][4];       // the activation codes of the lane's elements: bit pair g of the code bytes
    uint32_t bm[NT][2];
    float d8[NT][2];
    uint32_t have = 0xFFFFFFFFu, slot = 0, xb = warp % p.nblk;  // xb: block of the warp's next item
    for (uint32_t x0 = 0, rd = 0; x0 < total; x0 += R, ++rd) {
        float* tab = table + (rd & 1) * R * ITEM;
#pragma unroll 1
        for (uint32_t x = x0 + warp; x < min(x0 + R, total); x += KS_WARPS) {
            fetch();
            const uint32_t b = xb;
            xb += step_b;
            if (xb >= p.nblk) xb -= p.nblk;
            if (b != have) {  // stays the same where 16 is a multiple of nblk or nblk is 16
                have = b;
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const uint32_t m = m_base + 8 * nt + g;
                    const bool in = m < p.M;
                    const uint4* src = reinterpret_cast<const uint4*>(p.codes + ((size_t)(in ? m : 0) * p.nblk + b) * 256 + 128 * (t >> 1) + 16 * (t & 1));
#pragma unroll
                    for (int k = 0; k < 4; ++k) bf[nt][k] = in ? __ldg(src + 2 * k) : make_uint4(0, 0, 0, 0);
                    if constexpr (MIN) {
                        const uint32_t* ms = reinterpret_cast<const uint32_t*>(p.mins + ((size_t)(in ? m : 0) * p.nblk + b) * 32);
                        bm[nt][0] = in ? __ldg(ms + t) : 0u;
                        bm[nt][1] = in ? __ldg(ms + 4 + t) : 0u;
                    }
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint32_t mc = m_base + 8 * nt + 2 * t + j;
                        d8[nt][j] = mc < p.M ? __ldg(p.d8 + (size_t)b * p.M + mc) : 0.f;
                    }
                }
            }
            asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
            __syncwarp();
            const uint32_t at = (g * p.row_bytes + b * BB) & 15u;  // where the row's block sits in its slot (eight rows are a multiple of 16 bytes)
            const uint32_t* ra = reinterpret_cast<const uint32_t*>(smem + (warp * DEPTH + slot) * SLOT + g * PITCH + (at & 12u));
            const uint32_t* rb = ra + 8 * PITCH / 4;
            uint32_t va[4][4], vb[4][4], dma, dmb;
            if constexpr (MIN) {
                q2k_row(ra, t, va);
                q2k_row(rb, t, vb);
                dma = ra[20];
                dmb = rb[20];
            } else {
                const uint32_t sh = 8 * (at & 2u);
                q3k_row(ra, sh, t, va);
                q3k_row(rb, sh, t, vb);
                dma = (ra[27] >> sh) & 0xFFFFu;
                dmb = (rb[27] >> sh) & 0xFFFFu;
            }
            const float da = f16bits_to_f32(dma & 0xFFFF), db = f16bits_to_f32(dmb & 0xFFFF);
            float* to = tab + (x - x0) * ITEM;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                int acc[4] = {0, 0, 0, 0};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    mma_s8s8_k32(acc, va[k][0], vb[k][0], va[k][1], vb[k][1], bf[nt][k].x, bf[nt][k].y, acc);
                    mma_s8s8_k32(acc, va[k][2], vb[k][2], va[k][3], vb[k][3], bf[nt][k].z, bf[nt][k].w, acc);
                }
                float tm[4];
                if constexpr (MIN) {
                    const uint32_t ma = (ra[t] >> 4) & 0x0F0F0F0Fu, mb = (rb[t] >> 4) & 0x0F0F0F0Fu;
                    int ms[4] = {0, 0, 0, 0};
                    mma_u8s8_k32(ms, ma, mb, ma << 4, mb << 4, bm[nt][0], bm[nt][1], ms);
                    const float na = f16bits_to_f32(dma >> 16), nb = f16bits_to_f32(dmb >> 16);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float d = j < 2 ? da : db, dn = j < 2 ? na : nb, s = d8[nt][j & 1];
                        tm[j] = __fsub_rn(__fmul_rn(__fmul_rn(d, s), (float)acc[j]), __fmul_rn(__fmul_rn(dn, s), (float)ms[j]));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) tm[j] = __fmul_rn(__fmul_rn(j < 2 ? -da : -db, d8[nt][j & 1]), (float)acc[j]);
                }
                float* tn = to + (8 * nt + 2 * t) * KS_COL + g;
                tn[0] = tm[0];
                tn[KS_COL] = tm[1];
                tn[8] = tm[2];
                tn[KS_COL + 8] = tm[3];
            }
            __syncwarp();  // the slot is refilled by the next fetch
            if (++slot == DEPTH) slot = 0;
        }
        __syncthreads();  // the table of this round is complete; the other one is free again
        // 128 NT sums (activation row, weight row) by 4 NT warps, another group each round
        const uint32_t pos = (threadIdx.x + KS_WARPS * 32 - (rd * 128 * NT) % (KS_WARPS * 32)) % (KS_WARPS * 32);
        if (pos < 128 * NT) {
            const uint32_t m = m_base + (pos >> 4), row = pos & 15, cnt = min(R, total - x0);
            const float* tp = tab + (pos >> 4) * KS_COL + row;
            float s = run[pos];
            uint32_t b = x0 % p.nblk, n = (s_lo + x0 / p.nblk) * 16 + row;
#pragma unroll 8
            for (uint32_t x = 0; x < cnt; ++x) {
                s = __fadd_rn(s, tp[x * ITEM]);
                if (++b == p.nblk) {
                    if (m < p.M && n < p.N) store_as(p.out, p.out_dtype, (size_t)m * p.N + n, s);
                    s = 0.f;
                    b = 0;
                    n += 16;
                }
            }
            run[pos] = s;
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

struct KqScratch {
    uint8_t *codes, *mins;
    float* d8;
    __half* sums;  // the sums of 16 codes as f16, where kquant_few.cu may read the image too
};
bool kq_has_sums(size_t M, size_t K) { return M < 64 && K <= 65536; }
size_t kq_sums_at(size_t M, size_t K) { return (M * (K / 256) * RUN_BYTES + 15) & ~(size_t)15; }
KqScratch kq_scratch(void* ws, size_t M, size_t K) {
    uint8_t* b = static_cast<uint8_t*>(ws);
    return {b, b + M * K, reinterpret_cast<float*>(b + M * K + M * (K / 256) * 32), kq_has_sums(M, K) ? reinterpret_cast<__half*>(b + kq_sums_at(M, K)) : nullptr};
}

// Time of the two kernels per block of K in SM cycles, fitted to graph replays (Q2_K / Q3_K, 1024 ... 14336 weight rows): a round of
// tensor-core tiles takes 1300 and 7 a row of the tile; a 16-row slab of the other kernel 90 (Q2_K) or
// 130 (Q3_K) and 20 per 8 activation rows.  Up to 8 rows the latter always wins (Q3_K 4096 x 4096 at 4 rows 7 us; one round
// of tiles is 17 us).
struct KqPlan {
    uint32_t mt = 0;  // activation rows of a tensor-core tile; 0: the kernel for few activation rows
    size_t cost = 0;
};
KqPlan kq_tc_plan(int fmt, size_t M, size_t N, int sm_count) {
    KqPlan best;
    const size_t rt = (N + 127) / 128, fixed = 1300, per_row = 7;
    for (uint32_t mt = 16; mt <= KT_MT_MAX; mt += 16) {
        const size_t units = rt * ((M + mt - 1) / mt), cost = (units + sm_count - 1) / sm_count * (fixed + per_row * mt);
        if (!best.mt || cost <= best.cost) best = {mt, cost};
        if (mt >= M) break;
    }
    return best;
}
KqPlan kq_plan(int fmt, size_t M, size_t K, size_t N, int sm_count) {
    const KqPlan tc = kq_tc_plan(fmt, M, N, sm_count);
    const size_t slabs = (N + 15) / 16, nt = M <= 8 ? 1 : M <= 16 ? 2 : 4, groups = (M + 8 * nt - 1) / (8 * nt);
    const size_t small = (slabs + sm_count - 1) / sm_count * groups * (fmt == FMT_Q2_K ? 90 + 20 * nt : 130 + 20 * nt);
    const size_t units = (N + 127) / 128 * ((M + 15) / 16);
    if (M <= 8 || small <= tc.cost || units > (1u << 30) / (K / 256) || !tma_available()) return {0, small};
    return tc;
}

template <int FMT>
cudaError_t launch_tc(const KqTcParams& p, const CUtensorMap& amap, const CUtensorMap& mmap, const CUtensorMap& wmap, int sm_count, cudaStream_t st) {
    static PerDeviceOnce attrs;
    cudaError_t e = attrs.run([] { return cudaFuncSetAttribute(kq_tc_kernel<FMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kt_smem(FMT)); });
    if (e != cudaSuccess) return e;
    return launch_pdl(kq_tc_kernel<FMT>, dim3(p.nunits < (uint32_t)sm_count ? p.nunits : (uint32_t)sm_count), dim3(KT_THREADS), kt_smem(FMT), st, amap, mmap, wmap, p);
}
template <int FMT, int NT>
cudaError_t launch_small(const KqSmallParams& p, int sm_count, cudaStream_t st) {
    static PerDeviceOnce attrs;
    cudaError_t e = attrs.run([] { return cudaFuncSetAttribute(kq_small_kernel<FMT, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ks_smem(FMT, NT)); });
    if (e != cudaSuccess) return e;
    const uint32_t slabs = (p.N + 15) / 16, groups = (p.M + 8 * NT - 1) / (8 * NT);
    // at most 65535 groups of activation rows in a grid: the rest in further launches
    for (uint32_t g0 = 0; g0 < groups && e == cudaSuccess; g0 += 65535) {
        KqSmallParams q = p;
        q.m_first = g0 * 8 * NT;
        const uint32_t n = groups - g0 < 65535 ? groups - g0 : 65535;
        e = launch_pdl(kq_small_kernel<FMT, NT>, dim3(slabs < (uint32_t)sm_count ? slabs : (uint32_t)sm_count, n), dim3(KS_WARPS * 32), ks_smem(FMT, NT), st, q);
    }
    return e;
}

bool encode(CUtensorMap* map, CUtensorMapDataType type, size_t elem, void* base, size_t inner, size_t rows, uint32_t box_inner, uint32_t box_rows,
            CUtensorMapSwizzle sw) {
    const cuuint32_t estr[2] = {1, 1}, box[2] = {box_inner, box_rows};
    const cuuint64_t gdim[2] = {inner, rows}, gstride[1] = {inner * elem};
    return encode_tiled()(map, type, 2, base, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// Q2_K and Q3_K: every shape.
bool kq_i8_supported(int fmt, size_t M, size_t K, size_t N) {
    return (fmt == FMT_Q2_K || fmt == FMT_Q3_K) && M >= 1 && N >= 1 && K >= 256 && K % 256 == 0;
}

size_t kq_i8_workspace_bytes(size_t M, size_t K) {
    const size_t image = M * (K / 256) * RUN_BYTES;
    return ((kq_has_sums(M, K) ? kq_sums_at(M, K) + M * (K / 256) * 32 : image) + 255) & ~(size_t)255;
}

// Writes the image of the activations that all K-quant products of up to 63 rows (and those of Q2_K and Q3_K) read; early: the
// product may start before this kernel's wait (kq_act_prep_kernel).
cudaError_t launch_kq_prep(const void* act, int act_dtype, size_t M, size_t K, void* ws, bool early, int sm_count, cudaStream_t st) {
    const KqScratch s = kq_scratch(ws, M, K);
    const uint32_t nblk = (uint32_t)(K / 256);
    size_t grid = (M * nblk + 7) / 8;
    if (grid > (size_t)sm_count * 8) grid = (size_t)sm_count * 8;
    const cudaError_t e = act_dtype == DT_F32 ? launch_pdl(kq_act_prep_kernel<float>, dim3((unsigned)grid), dim3(256), 0, st, static_cast<const float*>(act), s.codes,
                                                           s.mins, s.d8, s.sums, M, nblk, early)
                                              : launch_pdl(kq_act_prep_kernel<__nv_bfloat16>, dim3((unsigned)grid), dim3(256), 0, st,
                                                           static_cast<const __nv_bfloat16*>(act), s.codes, s.mins, s.d8, s.sums, M, nblk, early);
    note_launch();
    return e;
}
void kq_image(void* ws, size_t M, size_t K, uint8_t** codes, __half** sums, float** d8) {
    const KqScratch s = kq_scratch(ws, M, K);
    *codes = s.codes;
    *sums = s.sums;
    *d8 = s.d8;
}

// acts_prepared: a previous call with the same activations and scratch left the image there (both formats read the same).
cudaError_t launch_kq_i8(int fmt, const void* act, int act_dtype, const void* w, void* out, int out_dtype, size_t M, size_t K, size_t N, void* ws,
                             size_t ws_bytes, int sm_count, cudaStream_t st, unsigned int* status, bool* ws_too_small, char* err, size_t err_len,
                             bool acts_prepared) {
    *ws_too_small = false;
    const size_t need = kq_i8_workspace_bytes(M, K);
    if (!ws || ws_bytes < need || (reinterpret_cast<uintptr_t>(ws) & 15)) {
        *ws_too_small = true;
        return cudaSuccess;
    }
    if (fmt != FMT_Q2_K && fmt != FMT_Q3_K) return cudaErrorInvalidValue;
    const KqScratch s = kq_scratch(ws, M, K);
    const uint32_t nblk = (uint32_t)(K / 256);
    cudaError_t e;
    if (!acts_prepared) {
        e = launch_kq_prep(act, act_dtype, M, K, ws, false, sm_count, st);
        if (e != cudaSuccess) return e;
    }
    const KqPlan plan = kq_plan(fmt, M, K, N, sm_count);
    if (plan.mt) {
        KqTcParams p{};
        p.w = static_cast<const uint8_t*>(w);
        p.out = out;
        p.d8 = s.d8;
        p.M = (uint32_t)M; p.N = (uint32_t)N; p.nblk = nblk;
        p.mt = plan.mt;
        p.nct = (uint32_t)((M + plan.mt - 1) / plan.mt);
        p.nunits = (uint32_t)((N + 127) / 128) * p.nct;
        p.row_bytes = nblk * (uint32_t)fmt_block_bytes(fmt);
        p.idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((p.mt >> 3) << 17) | ((128u >> 4) << 24);  // int32 <- s8 x s8, K-major, N = mt, M = 128
        p.out_dtype = out_dtype;
        p.status = status;
        p.raw_tma = p.row_bytes % 16 == 0;
        CUtensorMap amap, mmap, wmap{};
        if (!encode(&amap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, s.codes, K, M, 128, plan.mt, CU_TENSOR_MAP_SWIZZLE_128B) ||
            !encode(&mmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, s.mins, (size_t)nblk * 32, M, 32, plan.mt, CU_TENSOR_MAP_SWIZZLE_32B) ||
            (p.raw_tma && !encode(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(w), p.row_bytes / 2, N, kq_pitch(fmt) / 2, 128,
                                  CU_TENSOR_MAP_SWIZZLE_NONE))) {
            snprintf(err, err_len, "cuTensorMapEncodeTiled failed (activation image %p, weight %p, M=%zu K=%zu N=%zu)", (void*)s.codes, w, M, K, N);
            return cudaErrorInvalidValue;
        }
        e = fmt == FMT_Q2_K   ? launch_tc<FMT_Q2_K>(p, amap, mmap, wmap, sm_count, st)
                              : launch_tc<FMT_Q3_K>(p, amap, mmap, wmap, sm_count, st);
    } else {
        KqSmallParams p{};
        p.w = static_cast<const uint8_t*>(w);
        p.codes = s.codes; p.mins = s.mins; p.d8 = s.d8;
        p.out = out;
        p.M = (uint32_t)M; p.N = (uint32_t)N; p.nblk = nblk;
        p.row_bytes = nblk * (uint32_t)fmt_block_bytes(fmt);
        p.out_dtype = out_dtype;
        const int nt = M <= 8 ? 1 : M <= 16 ? 2 : 4;
        if (fmt == FMT_Q2_K)
            e = nt == 1 ? launch_small<FMT_Q2_K, 1>(p, sm_count, st) : nt == 2 ? launch_small<FMT_Q2_K, 2>(p, sm_count, st) : launch_small<FMT_Q2_K, 4>(p, sm_count, st);
        else
            e = nt == 1 ? launch_small<FMT_Q3_K, 1>(p, sm_count, st) : nt == 2 ? launch_small<FMT_Q3_K, 2>(p, sm_count, st) : launch_small<FMT_Q3_K, 4>(p, sm_count, st);
    }
    note_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace b200q

// Activation rows of the tensor-core tile that a product takes (0: the kernel for few rows, -1: another path).  Not part of
// the C ABI: the tests hold their shapes to the tiles that they are meant for.
extern "C" __attribute__((visibility("default"))) int b200q_kq_tile_rows(int fmt, size_t M, size_t K, size_t N, int sm_count) {
    if (b200q::kq_few_supported(fmt, M, K, N, false, sm_count)) return b200q::kq_few_tile_rows(fmt, M, K, N, sm_count);
    if (!b200q::kq_i8_supported(fmt, M, K, N)) return -1;
    return (int)b200q::kq_plan(fmt, M, K, N, sm_count).mt;
}
