// Small-M quantized matmul (8 <= M <= 16) for Q4_K on the 5th-generation tensor cores' INTEGER path:
//   out[M,N] = act[M,K] x W[N,K]^T  with boostr's CPU arithmetic (activations quantised to Q8_K,
//   src/quant/cpu/kernels/simd/quantize_act_q8k.rs:26-98; per 256-block (d*d8)*sumi - (dmin*d8)*sumi_mins with exact
//   integer sums, src/quant/cpu/kernels/simd/fused_q4k_q8k_dot.rs:111-172).
//
// The mma.sync kernel (gemv.cu) spends ~540 warp instructions per (16 weight rows x 256 K x 16 activation rows), is bound
// by instruction issue.  Here ONE tcgen05.mma.kind::i8 (128 weight rows x 16 activation rows x 32 K) computes the integer dot
// products of a whole 32-wide sub-block for 128 rows, and the per-sub-block scales are applied by the warps that drain the accumulator:
//   * tile = 128 weight rows (the MMA's M = the 128 lanes of tensor memory); the activations are the B operand,
//     MP = 16 rows (MMA N); every 32-wide sub-block j of a 256-block gets its OWN accumulator columns
//     [MP j, MP j + MP), so no scale has to enter the tensor core; tensor memory holds two such accumulators;
//   * packed weight blocks arrive by TMA as tiles of 128 rows x 144 bytes (conflict-free 16-byte reads, one thread
//     per row); two sets of four decode warps, taking the blocks in turn, split the nibbles into bytes and write them
//     as the K-major, 128-byte-swizzled A operand in shared memory (two tiles of 128 rows x 128 codes per block), and
//     leave the row's 6-bit scales, mins, d and dmin in a small ring of records for the drain;
//   * the activations are quantised once per call (i8_act_prep_kernel) into an int8 image [M][K] that TMA brings in
//     as the B operand; the Q8_K scales and the 32-wide block sums the min term needs travel beside the records;
//   * one thread issues the 8 MMAs of a block; two teams of eight drain warps, one per accumulator (a thread owns a
//     weight row and half of the activation rows), read the 8 x MP integer sums from tensor memory, form
//     sumi = sum_j sc_j dot_j and sumi_mins = sum_j m_j bsum_j in integers and the block's f32 term; the running f32
//     sums pass from team to team through shared memory, so the blocks are still added in K order;
//   * work = whole tiles, dealt to the CTAs as equal contiguous ranges: the result has the CPU's bits.
// What bounds it: the drain is ~200 instructions per (weight row, 8 activation rows, block), about 2600 warp
// instructions per (128 rows x 256 K x 16 activation rows) for the whole CTA against ~4300 in the mma.sync kernel.
// Every mbarrier wait is bounded; on a timeout the CTA records a status code and still frees its tensor memory.
#include <cuda.h>

#include <cstdio>

#include "common.cuh"
#include "tcgen05_i8.cuh"
#include "tmap.cuh"

namespace b200q {

struct I8Params {
    void* out;
    const uint8_t* aux;     // [nblk][AUX_BYTES]: per block the eight int16 sums of 32 codes of every activation row, then the rows' Q8_K scales
    uint32_t M, N;
    uint32_t nblk;          // K / 256
    uint32_t tbase, trem;   // tiles / grid and tiles % grid: CTA c takes tiles [c tbase + min(c, trem), ...)
    uint32_t ns;          // ring depth of operand stages (one 256-block each)
    uint32_t nr;          // ring depth of packed-weight tiles
    uint32_t nsc;         // ring depth of the scale records
    uint32_t idesc;
    int out_dtype;
    unsigned int* status;
};

namespace {


constexpr int DEC_WARPS = 8, DRAIN_WARPS = 16;  // decode: two sets of four warps; drain: two teams of eight warps
constexpr int I8_THREADS = (DEC_WARPS + DRAIN_WARPS + 3) * 32;  // decode | drain | packed-weight TMA | activation TMA | MMA issue, TMEM
constexpr int W_RAW = DEC_WARPS + DRAIN_WARPS, W_ACT = W_RAW + 1, W_MMA = W_RAW + 2;
constexpr uint32_t RAW_PITCH = 144, RAW_TILE = 128 * RAW_PITCH;  // 18432 = 18 x 1024
constexpr uint32_t A_ATOM = 128 * 128;                            // 128 rows x 128 codes
constexpr uint32_t SC_WORDS = 5;                                  // d|dmin, 8 scales, 8 mins
constexpr uint32_t SC_REC = 128 * SC_WORDS * 4;                  // the 128 row records of a block
constexpr uint32_t I8_MP = 16;                                    // activation rows of the MMA
constexpr uint32_t AUX_BYTES = I8_MP * 20;                        // per block: MP x 8 int16 block sums | MP x f32 d8
constexpr uint32_t SC_SLOT = SC_REC + AUX_BYTES;
// barriers (8 bytes each) at the start of dynamic shared memory
constexpr int OFF_FULL = 0, OFF_EMPTY = 64, OFF_RAW_FULL = 128, OFF_RAW_EMPTY = 192, OFF_ACC_FULL = 256, OFF_ACC_EMPTY = 272,
              OFF_SC_FULL = 320, OFF_TMEM = 448, OFF_DEAD = 452, OFF_XFER = 480, OFF_SC = 1024;

// First tile of CTA c: the first trem CTAs take one more than the others
__device__ __forceinline__ uint32_t i8_tile_begin(const I8Params& p, uint32_t c) { return c * p.tbase + min(c, p.trem); }

__global__ void __launch_bounds__(I8_THREADS, 1) smallm_i8_q4k_kernel(const __grid_constant__ CUtensorMap tmap_act,
                                                                      const __grid_constant__ CUtensorMap tmap_w, const I8Params p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // the launch reserves 1 KB of slack
    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar_full = sbase + OFF_FULL, bar_empty = sbase + OFF_EMPTY, bar_raw_full = sbase + OFF_RAW_FULL,
                   bar_raw_empty = sbase + OFF_RAW_EMPTY, bar_acc_full = sbase + OFF_ACC_FULL, bar_acc_empty = sbase + OFF_ACC_EMPTY,
                   bar_sc_full = sbase + OFF_SC_FULL;
    volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(smem + OFF_TMEM);
    volatile uint32_t* dead = reinterpret_cast<volatile uint32_t*>(smem + OFF_DEAD);
    constexpr uint32_t MP = I8_MP, NACC = 2, ACC_COLS = 8 * MP, TMEM_COLS = NACC * ACC_COLS;  // 256
    constexpr uint32_t B_ATOM = MP * 128, STAGE = 2 * A_ATOM + 2 * B_ATOM;
    // shared memory: barriers | scale records | exchange buffer of the drain teams | packed tiles | operand stages (A atom
    // 0, A atom 1, B atom 0, B atom 1)
    const uint32_t sc_off = OFF_SC, x_off = sc_off + p.nsc * SC_SLOT, raw_off = (x_off + 128 * MP * 4 + 1023u) & ~1023u,
                   st_off = raw_off + p.nr * RAW_TILE;

    constexpr int MH = MP / 2;  // activation rows of a drain warp: a team is 2 groups of 4 warps
    const uint32_t team_warps = 4 * min(2u, (p.M + MH - 1) / MH);  // warps of a team whose activation rows exist
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < p.ns; ++s) {
            mbar_init(bar_full + 8 * s, 5);   // the four decode warps of a set + the activation copy (with its byte count)
            mbar_init(bar_empty + 8 * s, 1);  // the commit behind the block's MMAs
        }
        for (uint32_t s = 0; s < p.nr; ++s) {
            mbar_init(bar_raw_full + 8 * s, 1);
            mbar_init(bar_raw_empty + 8 * s, 4);
        }
        for (uint32_t s = 0; s < NACC; ++s) {
            mbar_init(bar_acc_full + 8 * s, 1);
            mbar_init(bar_acc_empty + 8 * s, team_warps);  // the team that drains this accumulator
            mbar_init(sbase + OFF_XFER + 8 * s, team_warps);  // the team's running sums are in the exchange buffer
        }
        for (uint32_t s = 0; s < p.nsc; ++s) mbar_init(bar_sc_full + 8 * s, 5);  // four decode warps write the records, one copy brings the activation side
        *dead = 0;
        mbar_fence_init();
    }
    if (warp == W_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + OFF_TMEM), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = *tmem_holder;
    grid_dep_launch();
    const uint32_t t_begin = i8_tile_begin(p, blockIdx.x), t_end = i8_tile_begin(p, blockIdx.x + 1);

    if (warp == W_RAW) {
        // ------------------------------------------------------------ packed weight tiles (do not depend on the previous kernel)
        if (lane == 0) {
            uint32_t s = 0, par = 0;
            for (uint32_t tile = t_begin; tile < t_end && !*dead; ++tile) {
                for (uint32_t j = 0; j < p.nblk; ++j) {
                    if (!i8_wait(bar_raw_empty + 8 * s, par ^ 1, dead)) {
                        i8_fail(dead, p.status, STATUS_TIMEOUT_EMPTY);
                        break;
                    }
                    mbar_expect_tx(bar_raw_full + 8 * s, RAW_TILE);
                    tma2d(sbase + raw_off + s * RAW_TILE, &tmap_w, (int)(j * RAW_PITCH), (int)(tile * 128), bar_raw_full + 8 * s);
                    if (++s == p.nr) { s = 0; par ^= 1; }
                }
            }
        }
    } else if (warp == W_ACT) {
        // ------------------------------------------------------------ activation codes (written by the previous kernel)
        if (lane == 0) {
            grid_dep_wait();
            uint32_t s = 0, par = 0, i = 0;
            for (uint32_t tile = t_begin; tile < t_end && !*dead; ++tile) {
                for (uint32_t j = 0; j < p.nblk; ++j, ++i) {
                    if (!i8_wait(bar_empty + 8 * s, par ^ 1, dead)) {
                        i8_fail(dead, p.status, STATUS_TIMEOUT_EMPTY);
                        break;
                    }
                    const uint32_t b0 = sbase + st_off + s * STAGE + 2 * A_ATOM;
                    mbar_expect_tx(bar_full + 8 * s, 2 * B_ATOM);
                    tma2d(b0, &tmap_act, (int)(j * 256), 0, bar_full + 8 * s);
                    tma2d(b0 + B_ATOM, &tmap_act, (int)(j * 256 + 128), 0, bar_full + 8 * s);
                    // block sums and scales of the activation rows, next to the row records (same life time)
                    const uint32_t q = i % p.nsc;
                    mbar_expect_tx(bar_sc_full + 8 * q, AUX_BYTES);
                    bulk_g2s(sbase + sc_off + q * SC_SLOT + SC_REC, p.aux + (size_t)j * AUX_BYTES, AUX_BYTES, bar_sc_full + 8 * q);
                    if (++s == p.ns) { s = 0; par ^= 1; }
                }
            }
        }
    } else if (warp == W_MMA) {
        // ------------------------------------------------------------ MMA issue: 8 sub-blocks, 8 column groups
        uint32_t s = 0, par = 0, i = 0;
        bool ok = true;
        for (uint32_t tile = t_begin; ok && tile < t_end; ++tile) {
            for (uint32_t j = 0; j < p.nblk; ++j, ++i) {
                const uint32_t buf = i % NACC, use = i / NACC;
                if (!i8_wait(bar_full + 8 * s, par, dead)) {
                    if (lane == 0) i8_fail(dead, p.status, STATUS_TIMEOUT_FULL);
                    ok = false;
                    break;
                }
                if (use > 0 && !i8_wait(bar_acc_empty + 8 * buf, (use - 1) & 1, dead)) {
                    if (lane == 0) i8_fail(dead, p.status, STATUS_TIMEOUT_EMPTY);
                    ok = false;
                    break;
                }
                tc_after();
                if (elect_one_lane()) {
                    const uint32_t a_lo = desc_lo(sbase + st_off + s * STAGE), b_lo = desc_lo(sbase + st_off + s * STAGE + 2 * A_ATOM);
                    const uint32_t d0 = tmem + buf * ACC_COLS;
#pragma unroll
                    for (uint32_t sb = 0; sb < 8; ++sb)
                        tc_mma_i8(d0 + MP * sb, desc_sw128(a_lo + (sb >> 2) * (A_ATOM >> 4) + 2 * (sb & 3)),
                                  desc_sw128(b_lo + (sb >> 2) * (B_ATOM >> 4) + 2 * (sb & 3)), p.idesc);
                    tc_commit_to(bar_empty + 8 * s);         // the stage may be overwritten once these MMAs have read it
                    tc_commit_to(bar_acc_full + 8 * buf);    // and the sums are complete
                }
                __syncwarp();
                if (++s == p.ns) { s = 0; par ^= 1; }
            }
        }
    } else if (warp < DEC_WARPS) {
        // ------------------------------------------------------------ decode: nibbles -> int8 A operand, one thread per row
        // the sets of four warps take the CTA's blocks in turn, so DEC_WARPS / 4 blocks are in work at a time
        const uint32_t r = threadIdx.x & 127, set = threadIdx.x >> 7;
        const uint32_t row_sw = (r >> 3) * 1024 + (r & 7) * 128, x7 = r & 7;
        bool ok = true;
        uint32_t i = 0;
        for (uint32_t tile = t_begin; tile < t_end; ++tile) {
            const bool row_ok = tile * 128 + r < p.N;
            for (uint32_t j = 0; j < p.nblk; ++j, ++i) {
                if (i % (DEC_WARPS / 4) != set) continue;
                const uint32_t rs = i % p.nr, rpar = (i / p.nr) & 1, s = i % p.ns, par = (i / p.ns) & 1;
                if (ok && !i8_wait(bar_raw_full + 8 * rs, rpar, dead)) {
                    i8_fail(dead, p.status, STATUS_TIMEOUT_FULL);
                    ok = false;
                }
                const uint4* src = reinterpret_cast<const uint4*>(smem + raw_off + rs * RAW_TILE + r * RAW_PITCH);
                uint4 h = make_uint4(0, 0, 0, 0), q[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) q[k] = make_uint4(0, 0, 0, 0);
                if (ok && row_ok) {
                    h = src[0];
#pragma unroll
                    for (int k = 0; k < 8; ++k) q[k] = src[1 + k];
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_raw_empty + 8 * rs);
                if (ok && !i8_wait(bar_empty + 8 * s, par ^ 1, dead)) {
                    i8_fail(dead, p.status, STATUS_TIMEOUT_EMPTY);
                    ok = false;
                }
                // 16 nibble bytes q[k] = bytes 16k .. 16k+15 of qs: low nibbles -> sub-block 2 (k / 2), codes 16 (k & 1) ..;
                // high nibbles -> sub-block 2 (k / 2) + 1.  Sub-block sb sits at bytes 32 sb .. of the 256-byte operand
                // row: 16-byte chunk c = 2 sb + (k & 1) -> tile (c / 8), chunk (c % 8) ^ (row % 8) of the swizzled row.
                uint8_t* a0 = smem + st_off + s * STAGE + row_sw;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t c_lo = 4 * (k >> 1) + (k & 1), c_hi = c_lo + 2;
                    const uint4 lo = make_uint4(q[k].x & 0x0F0F0F0Fu, q[k].y & 0x0F0F0F0Fu, q[k].z & 0x0F0F0F0Fu, q[k].w & 0x0F0F0F0Fu);
                    const uint4 hi = make_uint4((q[k].x >> 4) & 0x0F0F0F0Fu, (q[k].y >> 4) & 0x0F0F0F0Fu, (q[k].z >> 4) & 0x0F0F0F0Fu,
                                                (q[k].w >> 4) & 0x0F0F0F0Fu);
                    *reinterpret_cast<uint4*>(a0 + (c_lo >> 3) * A_ATOM + (((c_lo & 7) ^ x7) << 4)) = lo;
                    *reinterpret_cast<uint4*>(a0 + (c_hi >> 3) * A_ATOM + (((c_hi & 7) ^ x7) << 4)) = hi;
                }
                // the row's record for the drain: d | dmin, the 6-bit scales and mins as bytes (unpack_q4k_q5k_scales,
                // src/quant/cpu/kernels/dequant_k_quants/q4k_q5k.rs:108-122)
                uint32_t* rec = reinterpret_cast<uint32_t*>(smem + sc_off + (i % p.nsc) * SC_SLOT) + r * SC_WORDS;
                rec[0] = h.x;
                rec[1] = h.y & 0x3F3F3F3Fu;
                rec[2] = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
                rec[3] = h.z & 0x3F3F3F3Fu;
                rec[4] = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
                proxy_fence();  // the operand bytes are read by the tensor core (async proxy)
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(bar_full + 8 * s);
                    mbar_arrive(bar_sc_full + 8 * (i % p.nsc));
                }
            }
        }
    } else {
        // ------------------------------------------------------------ drain: integer sums -> scaled f32 terms
        // Two teams of eight warps take the CTA's blocks in turn (team = block index & 1 = accumulator), so the latencies
        // of two blocks overlap.  In a team, a thread owns one weight row (two warps per quarter of the rows) and MH of
        // the activation rows; warps whose rows do not exist have nothing to do.  The f32 sums still grow block by block,
        // in K order: the running sums of a tile pass from team to team through a buffer in shared memory.
        const uint32_t dw = (uint32_t)warp - DEC_WARPS, team = dw >> 3, quarter = dw & 3, r = quarter * 32 + lane, m_lo = ((dw >> 2) & 1) * MH;
        const bool rows_exist = m_lo < p.M;
        const uint32_t lane_addr = (quarter * 32) << 16;
        const uint32_t nblocks = (t_end - t_begin) * p.nblk, bar_x = sbase + OFF_XFER;
        float* xch = reinterpret_cast<float*>(smem + x_off) + m_lo * 128 + r;                   // [activation row][weight row]
        grid_dep_wait();  // the output may still be in use by the previous kernel
        bool ok = true;
        auto store_out = [&](uint32_t n, uint32_t m, float v) {
            const size_t idx = (size_t)m * p.N + n;
            if (p.out_dtype == DT_F32) static_cast<float*>(p.out)[idx] = v;
            else if (p.out_dtype == DT_BF16) static_cast<__nv_bfloat16*>(p.out)[idx] = __float2bfloat16_rn(v);
            else static_cast<__half*>(p.out)[idx] = __float2half_rn(v);
        };
        for (uint32_t i = team; i < nblocks && ok && rows_exist; i += 2) {
            const uint32_t buf = team, use = i >> 1, q = i % p.nsc, tile = t_begin + i / p.nblk, blk = i % p.nblk;
            if (!i8_wait(bar_sc_full + 8 * q, (i / p.nsc) & 1, dead)) {
                i8_fail(dead, p.status, STATUS_TIMEOUT_FULL);
                ok = false;
                break;
            }
            const uint8_t* slot = smem + sc_off + q * SC_SLOT;
            const uint32_t* rec = reinterpret_cast<const uint32_t*>(slot) + r * SC_WORDS;
            const uint32_t hd = rec[0], s0 = rec[1], s1 = rec[2], m0 = rec[3], m1 = rec[4];
            const uint4* bsum = reinterpret_cast<const uint4*>(slot + SC_REC) + m_lo;
            const float* d8s = reinterpret_cast<const float*>(slot + SC_REC + MP * 16) + m_lo;
            const int sc[8] = {ubyte<0>(s0), ubyte<1>(s0), ubyte<2>(s0), ubyte<3>(s0), ubyte<0>(s1), ubyte<1>(s1), ubyte<2>(s1), ubyte<3>(s1)};
            if (!i8_wait(bar_acc_full + 8 * buf, use & 1, dead)) {
                i8_fail(dead, p.status, STATUS_TIMEOUT_MMA);
                ok = false;
                break;
            }
            tc_after();
            const uint32_t t0 = tmem + lane_addr + buf * ACC_COLS + m_lo;
            constexpr int GB = 2;  // sub-blocks whose loads are in flight together
            int sumi[MH];
#pragma unroll
            for (int m = 0; m < MH; ++m) sumi[m] = 0;
#pragma unroll
            for (int g = 0; g < 8 / GB; ++g) {
                uint32_t v[GB][MH];
#pragma unroll
                for (int k = 0; k < GB; ++k) tmem_ld8_async(t0 + MP * (GB * g + k), v[k]);
                tmem_ld_wait();
#pragma unroll
                for (int k = 0; k < GB; ++k)
#pragma unroll
                    for (int m = 0; m < MH; ++m) sumi[m] += sc[GB * g + k] * (int)v[k][m];
            }
            tc_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_acc_empty + 8 * buf);  // the MMA warp may reuse the columns
            // the block's terms: (d d8) sumi - (dmin d8) sum_j m_j bsum_j
            const float d = f16bits_to_f32(hd & 0xFFFF), dmin = f16bits_to_f32(hd >> 16);
            float term[MH];
#pragma unroll
            for (int m = 0; m < MH; ++m) {
                const uint4 bs = bsum[m];
                const float d8 = d8s[m];
                const int summ = __dp2a_lo((int)bs.x, (int)m0, __dp2a_hi((int)bs.y, (int)m0, __dp2a_lo((int)bs.z, (int)m1, __dp2a_hi((int)bs.w, (int)m1, 0))));
                term[m] = __fsub_rn(__fmul_rn(__fmul_rn(d, d8), (float)sumi[m]), __fmul_rn(__fmul_rn(dmin, d8), (float)summ));
            }
            // the running sums after the previous block (the other team's); every block waits for its predecessor, so the
            // teams never drift apart by more than one block
            if (i > 0 && !i8_wait(bar_x + 8 * (team ^ 1), ((i - 1) >> 1) & 1, dead)) {
                i8_fail(dead, p.status, STATUS_TIMEOUT_EMPTY);
                ok = false;
                break;
            }
            if (blk > 0)
#pragma unroll
                for (int m = 0; m < MH; ++m) term[m] = __fadd_rn(xch[m * 128], term[m]);
            const bool last_of_tile = blk + 1 == p.nblk;
            if (!last_of_tile)
#pragma unroll
                for (int m = 0; m < MH; ++m) xch[m * 128] = term[m];
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_x + 8 * team);
            if (!last_of_tile) continue;
            const uint32_t n = tile * 128 + r;
            if (n < p.N)
#pragma unroll
                for (int m = 0; m < MH; ++m)
                    if (m_lo + m < p.M) store_out(n, m_lo + m, term[m]);
        }
    }
    tc_before();
    __syncthreads();
    if (warp == W_MMA) {
        tc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// One warp per (activation row, 256-block): Q8_K codes (quantize_act_q8k.rs:26-98: d = amax / 127, id = 127 / amax,
// round half to even) into the int8 image [M][K]; the eight sums of 32 codes and the scale go to the block's record in
// `aux` (AUX_BYTES).
template <typename InT>
__global__ void __launch_bounds__(256) i8_act_prep_kernel(const InT* __restrict__ act, uint8_t* __restrict__ codes, uint8_t* __restrict__ aux,
                                                          uint32_t M, uint32_t nblk) {
    const int lane = threadIdx.x & 31;
    grid_dep_launch();
    grid_dep_wait();  // the activations may be the previous kernel's output; the image may still be read by it
    const uint32_t run = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (run >= M * nblk) return;
    const uint32_t m = run / nblk, b = run % nblk;
    float v[8];
    const size_t base = (size_t)run * 256 + 8 * lane;  // row m, block b of [M][K]
    if constexpr (sizeof(InT) == 4) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(act + base)), y = __ldg(reinterpret_cast<const float4*>(act + base) + 1);
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
    } else {
        const uint4 rr = __ldg(reinterpret_cast<const uint4*>(act + base));
        v[0] = __uint_as_float(rr.x << 16); v[1] = __uint_as_float(rr.x & 0xFFFF0000u);
        v[2] = __uint_as_float(rr.y << 16); v[3] = __uint_as_float(rr.y & 0xFFFF0000u);
        v[4] = __uint_as_float(rr.z << 16); v[5] = __uint_as_float(rr.z & 0xFFFF0000u);
        v[6] = __uint_as_float(rr.w << 16); v[7] = __uint_as_float(rr.w & 0xFFFF0000u);
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
        c[i] = max(-128, min(127, __float2int_rn(__fmul_rn(v[i], id))));
        s += c[i];
    }
    uint32_t w0 = 0, w1 = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        w0 |= (uint32_t)(c[i] & 0xFF) << (8 * i);
        w1 |= (uint32_t)(c[4 + i] & 0xFF) << (8 * i);
    }
    *reinterpret_cast<uint2*>(codes + base) = make_uint2(w0, w1);
    s += __shfl_xor_sync(0xFFFFFFFFu, s, 1);  // 32 codes = four lanes
    s += __shfl_xor_sync(0xFFFFFFFFu, s, 2);
    uint8_t* ab = aux + (size_t)b * AUX_BYTES;
    if ((lane & 3) == 0) reinterpret_cast<short*>(ab)[m * 8 + (lane >> 2)] = (short)s;
    if (lane == 0) reinterpret_cast<float*>(ab + I8_MP * 16)[m] = __fdiv_rn(amax, 127.0f);
}

// ---------------------------------------------------------------------------------------------------------------------
// Q8_0, 17..32 activation rows (f32 activations on boostr's CPU path: dequantised row . f32 dot,
// src/quant/cpu/kernels/quant_matmul.rs:193-209).  The weight codes are int8 already; every activation is two int8
// PIECES, x = amax/127 (a1 + a2/254) with amax over its 256-run (~3e-5 of the run's amax), stacked as 2 x 32 rows of the
// B operand.  One MMA per 32-block (128 weight rows x 64 x 32) leaves the block's integer sums of both pieces in its own
// columns; the drain converts them, weighs the pieces, multiplies by the block's d and adds in f32.  Same pipeline as
// above with these differences: an accumulator holds the four blocks of half a 256-run (one 128-byte operand tile, 256
// columns), so a stage feeds both accumulators and each is reused every block; all sixteen drain warps work on every
// accumulator (four groups of four warps, 8 activation rows each) and keep their sums in registers for the whole tile;
// whole tiles are dealt round-robin.
struct Q8Params {
    const uint8_t* w;
    void* out;
    const float* scale;   // [nblk256][32] amax / 127 of (256-run, activation row)
    uint32_t M, N, K;
    uint32_t nblk;        // K / 256
    uint32_t ntiles;      // ceil(N / 128)
    uint32_t ns, nr, nsc;
    uint32_t idesc;
    int out_dtype;
    unsigned int* status;
};
constexpr uint32_t Q8_RAW_PITCH = 272, Q8_RAW_TILE = 128 * Q8_RAW_PITCH;  // 34816 = 34 x 1024
constexpr uint32_t Q8_REC_WORDS = 4;                                       // the eight f16 d of a row's 256-run
constexpr uint32_t Q8_REC = 128 * Q8_REC_WORDS * 4;
constexpr uint32_t Q8_SLOT = Q8_REC + 32 * 4;                              // + the activation rows' scales of the run
constexpr float Q8_STEP = 254.0f;

__global__ void __launch_bounds__(I8_THREADS, 1) smallm_i8_q8_0_kernel(const __grid_constant__ CUtensorMap tmap_act,
                                                                       const __grid_constant__ CUtensorMap tmap_w, const Q8Params p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar_full = sbase + OFF_FULL, bar_empty = sbase + OFF_EMPTY, bar_raw_full = sbase + OFF_RAW_FULL,
                   bar_raw_empty = sbase + OFF_RAW_EMPTY, bar_acc_full = sbase + OFF_ACC_FULL, bar_acc_empty = sbase + OFF_ACC_EMPTY,
                   bar_sc_full = sbase + OFF_SC_FULL;
    volatile uint32_t* tmem_holder = reinterpret_cast<volatile uint32_t*>(smem + OFF_TMEM);
    volatile uint32_t* dead = reinterpret_cast<volatile uint32_t*>(smem + OFF_DEAD);
    constexpr uint32_t MP = 32, P = 2;                   // activation rows of the MMA, pieces per activation
    constexpr uint32_t NB = P * MP;                      // MMA N: the pieces' rows
    constexpr uint32_t ACC_COLS = 4 * NB;                // four 32-blocks
    constexpr uint32_t TMEM_COLS = 2 * ACC_COLS;         // 512
    constexpr uint32_t B_ATOM = NB * 128, STAGE = 2 * A_ATOM + 2 * B_ATOM;
    constexpr int MH = 8;                                // activation rows of a drain thread
    const uint32_t sc_off = OFF_SC, raw_off = (sc_off + p.nsc * Q8_SLOT + 1023u) & ~1023u, st_off = raw_off + p.nr * Q8_RAW_TILE;
    // drain warps whose activation rows exist, per accumulator
    const uint32_t groups = min((uint32_t)MP / MH, (p.M + MH - 1) / MH), acc_warps = 4 * groups;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < p.ns; ++s) {
            mbar_init(bar_full + 8 * s, 5);   // the four decode warps of a set + the activation copy
            mbar_init(bar_empty + 8 * s, 1);  // the commit behind the stage's second group of MMAs
        }
        for (uint32_t s = 0; s < p.nr; ++s) {
            mbar_init(bar_raw_full + 8 * s, 1);
            mbar_init(bar_raw_empty + 8 * s, 4);
        }
        for (uint32_t s = 0; s < 2; ++s) {
            mbar_init(bar_acc_full + 8 * s, 1);
            mbar_init(bar_acc_empty + 8 * s, acc_warps);
        }
        for (uint32_t s = 0; s < p.nsc; ++s) mbar_init(bar_sc_full + 8 * s, 5);
        *dead = 0;
        mbar_fence_init();
    }
    if (warp == W_MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + OFF_TMEM), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = *tmem_holder;
    grid_dep_launch();
    // the CTA's tiles: blockIdx.x, blockIdx.x + gridDim.x, ...; block i of the CTA = block i % nblk of its (i / nblk)-th tile
    const uint32_t my_tiles = p.ntiles > blockIdx.x ? (p.ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
    const uint32_t nblocks = my_tiles * p.nblk;

    if (warp == W_RAW) {
        if (lane == 0) {
            for (uint32_t i = 0; i < nblocks && !*dead; ++i) {
                const uint32_t s = i % p.nr, par = (i / p.nr) & 1, tile = blockIdx.x + (i / p.nblk) * gridDim.x, blk = i % p.nblk;
                if (!i8_wait(bar_raw_empty + 8 * s, par ^ 1, dead)) {
                    i8_fail(dead, p.status, STATUS_TIMEOUT_EMPTY);
                    break;
                }
                mbar_expect_tx(bar_raw_full + 8 * s, Q8_RAW_TILE);
                tma2d(sbase + raw_off + s * Q8_RAW_TILE, &tmap_w, (int)(blk * 136), (int)(tile * 128), bar_raw_full + 8 * s);  // x in 16-bit units
            }
        }
    } else if (warp == W_ACT) {
        if (lane == 0) {
            grid_dep_wait();
            for (uint32_t i = 0; i < nblocks && !*dead; ++i) {
                const uint32_t s = i % p.ns, par = (i / p.ns) & 1, blk = i % p.nblk, q = i % p.nsc;
                if (!i8_wait(bar_empty + 8 * s, par ^ 1, dead)) {
                    i8_fail(dead, p.status, STATUS_TIMEOUT_EMPTY);
                    break;
                }
                const uint32_t b0 = sbase + st_off + s * STAGE + 2 * A_ATOM;
                mbar_expect_tx(bar_full + 8 * s, 2 * B_ATOM);
                tma2d(b0, &tmap_act, (int)(blk * 256), 0, bar_full + 8 * s);
                tma2d(b0 + B_ATOM, &tmap_act, (int)(blk * 256 + 128), 0, bar_full + 8 * s);
                mbar_expect_tx(bar_sc_full + 8 * q, MP * 4);
                bulk_g2s(sbase + sc_off + q * Q8_SLOT + Q8_REC, p.scale + (size_t)blk * MP, MP * 4, bar_sc_full + 8 * q);
            }
        }
    } else if (warp == W_MMA) {
        // ------------------------------------------------------------ MMA issue: per stage two accumulators of four blocks
        bool ok = true;
        for (uint32_t i = 0; ok && i < nblocks; ++i) {
            const uint32_t s = i % p.ns, par = (i / p.ns) & 1;
            if (!i8_wait(bar_full + 8 * s, par, dead)) {
                if (lane == 0) i8_fail(dead, p.status, STATUS_TIMEOUT_FULL);
                break;
            }
            for (uint32_t h = 0; h < 2; ++h) {  // accumulator h = half-run h of the block: use number i of this accumulator
                if (i > 0 && !i8_wait(bar_acc_empty + 8 * h, (i - 1) & 1, dead)) {
                    if (lane == 0) i8_fail(dead, p.status, STATUS_TIMEOUT_EMPTY);
                    ok = false;
                    break;
                }
                tc_after();
                if (elect_one_lane()) {
                    const uint32_t a_lo = desc_lo(sbase + st_off + s * STAGE + h * A_ATOM), b_lo = desc_lo(sbase + st_off + s * STAGE + 2 * A_ATOM + h * B_ATOM);
#pragma unroll
                    for (uint32_t b = 0; b < 4; ++b) tc_mma_i8(tmem + h * ACC_COLS + NB * b, desc_sw128(a_lo + 2 * b), desc_sw128(b_lo + 2 * b), p.idesc);
                    if (h == 1) tc_commit_to(bar_empty + 8 * s);
                    tc_commit_to(bar_acc_full + 8 * h);
                }
                __syncwarp();
            }
        }
    } else if (warp < DEC_WARPS) {
        // ------------------------------------------------------------ decode: copy the codes into the A operand, one thread per row
        // Raw row of a 256-run: eight blocks of 34 bytes (f16 d | 32 x i8) = 68 words.  The codes of block b start at byte
        // 34 b + 2: on a word boundary for odd b, two bytes past one for even b (a word = two neighbours and a byte permute).
        const uint32_t r = threadIdx.x & 127, set = threadIdx.x >> 7;
        const uint32_t row_sw = (r >> 3) * 1024 + (r & 7) * 128, x7 = r & 7;
        bool ok = true;
        for (uint32_t i = set; i < nblocks; i += DEC_WARPS / 4) {
            const uint32_t rs = i % p.nr, rpar = (i / p.nr) & 1, s = i % p.ns, par = (i / p.ns) & 1;
            const bool row_ok = (blockIdx.x + (i / p.nblk) * gridDim.x) * 128 + r < p.N;
            if (ok && !i8_wait(bar_raw_full + 8 * rs, rpar, dead)) {
                i8_fail(dead, p.status, STATUS_TIMEOUT_FULL);
                ok = false;
            }
            if (ok && !i8_wait(bar_empty + 8 * s, par ^ 1, dead)) {
                i8_fail(dead, p.status, STATUS_TIMEOUT_EMPTY);
                ok = false;
            }
            const uint4* src = reinterpret_cast<const uint4*>(smem + raw_off + rs * Q8_RAW_TILE + r * Q8_RAW_PITCH);
            uint8_t* a0 = smem + st_off + s * STAGE + row_sw;
            uint32_t dd[8];
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                constexpr int K0[8] = {0, 9, 17, 26, 34, 43, 51, 60};  // first word that holds codes of block b
                const int q0 = (K0[b] - (b & 1)) / 4, off = K0[b] - 4 * q0;  // three 16-byte loads from word 4 q0 cover d and the codes
                uint32_t a[12];
                if (ok && row_ok) {
                    const uint4 u0 = src[q0], u1 = src[q0 + 1], u2 = src[q0 + 2];
                    a[0] = u0.x; a[1] = u0.y; a[2] = u0.z; a[3] = u0.w; a[4] = u1.x; a[5] = u1.y; a[6] = u1.z; a[7] = u1.w;
                    a[8] = u2.x; a[9] = u2.y; a[10] = u2.z; a[11] = u2.w;
                } else {
#pragma unroll
                    for (int k = 0; k < 12; ++k) a[k] = 0;
                }
                uint32_t o[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) o[j] = (b & 1) ? a[off + j] : __byte_perm(a[off + j], a[off + j + 1], 0x5432);
                dd[b] = (b & 1) ? a[off - 1] >> 16 : a[off] & 0xFFFFu;
                // block b = bytes 32 b .. of the 256-byte operand row: 16-byte chunks 2 b, 2 b + 1 -> tile b / 4
                uint8_t* at = a0 + (b >> 2) * A_ATOM;
                *reinterpret_cast<uint4*>(at + ((((2 * b) & 7) ^ x7) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
                *reinterpret_cast<uint4*>(at + ((((2 * b + 1) & 7) ^ x7) << 4)) = make_uint4(o[4], o[5], o[6], o[7]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_raw_empty + 8 * rs);
            uint32_t* rec = reinterpret_cast<uint32_t*>(smem + sc_off + (i % p.nsc) * Q8_SLOT) + r * Q8_REC_WORDS;
#pragma unroll
            for (int k = 0; k < 4; ++k) rec[k] = dd[2 * k] | (dd[2 * k + 1] << 16);
            proxy_fence();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(bar_full + 8 * s);
                mbar_arrive(bar_sc_full + 8 * (i % p.nsc));
            }
        }
    } else {
        // ------------------------------------------------------------ drain: four groups of four warps, 8 activation rows each
        const uint32_t dw = (uint32_t)warp - DEC_WARPS, quarter = dw & 3, r = quarter * 32 + lane, m_lo = (dw >> 2) * MH;
        const bool rows_exist = m_lo < p.M;
        const uint32_t lane_addr = (quarter * 32) << 16;
        grid_dep_wait();
        bool ok = true;
        float acc[MH];
#pragma unroll
        for (int m = 0; m < MH; ++m) acc[m] = 0.f;
        constexpr float C1 = 1.0f / Q8_STEP;
        for (uint32_t i = 0; i < nblocks && ok && rows_exist; ++i) {
            const uint32_t q = i % p.nsc, blk = i % p.nblk, tl = i / p.nblk;
            if (!i8_wait(bar_sc_full + 8 * q, (i / p.nsc) & 1, dead)) {
                i8_fail(dead, p.status, STATUS_TIMEOUT_FULL);
                ok = false;
                break;
            }
            const uint8_t* slot = smem + sc_off + q * Q8_SLOT;
            const uint32_t* rec = reinterpret_cast<const uint32_t*>(slot) + r * Q8_REC_WORDS;
            const float* scl = reinterpret_cast<const float*>(slot + Q8_REC) + m_lo;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {  // the two half-runs of the block
                const uint32_t d01 = rec[2 * h], d23 = rec[2 * h + 1];
                const float db[4] = {f16bits_to_f32(d01 & 0xFFFF), f16bits_to_f32(d01 >> 16), f16bits_to_f32(d23 & 0xFFFF), f16bits_to_f32(d23 >> 16)};
                if (!i8_wait(bar_acc_full + 8 * h, i & 1, dead)) {
                    i8_fail(dead, p.status, STATUS_TIMEOUT_MMA);
                    ok = false;
                    break;
                }
                tc_after();
                float sacc[MH];
#pragma unroll
                for (int m = 0; m < MH; ++m) sacc[m] = 0.f;
                const uint32_t t0 = tmem + lane_addr + h * ACC_COLS + m_lo;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    uint32_t v[P][MH];
#pragma unroll
                    for (int pc = 0; pc < (int)P; ++pc) tmem_ld8_async(t0 + NB * b + MP * pc, v[pc]);
                    tmem_ld_wait();
                    // the two pieces meet as integers, 254 a1 + a2 (|.| < 2^28), so a block costs one conversion and one FMA
#pragma unroll
                    for (int m = 0; m < MH; ++m) sacc[m] = fmaf(db[b], (float)(254 * (int)v[0][m] + (int)v[1][m]), sacc[m]);
                }
                tc_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_acc_empty + 8 * h);
#pragma unroll
                for (int m = 0; m < MH; ++m) acc[m] = fmaf(sacc[m], scl[m] * C1, acc[m]);
            }
            if (!ok || blk + 1 != p.nblk) continue;
            // ---- the tile is complete
            const uint32_t n = (blockIdx.x + tl * gridDim.x) * 128 + r;
            if (n < p.N)
#pragma unroll
                for (int m = 0; m < MH; ++m) {
                    if (m_lo + m < p.M) {
                        const size_t idx = (size_t)(m_lo + m) * p.N + n;
                        if (p.out_dtype == DT_F32) static_cast<float*>(p.out)[idx] = acc[m];
                        else if (p.out_dtype == DT_BF16) static_cast<__nv_bfloat16*>(p.out)[idx] = __float2bfloat16_rn(acc[m]);
                        else static_cast<__half*>(p.out)[idx] = __float2half_rn(acc[m]);
                    }
                }
#pragma unroll
            for (int m = 0; m < MH; ++m) acc[m] = 0.f;
        }
    }
    tc_before();
    __syncthreads();
    if (warp == W_MMA) {
        tc_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// One warp per (activation row, 256-run): the run's amax / 127 into scale[run][row] and every value as P int8 pieces,
// x = amax/127 (a1 + a2/254 + a3/254^2), piece pc of row m into row pc MP + m of the image [P MP][K]; rows that do not
// exist are written as zeros (the B operand reads all MP rows of a piece).
template <typename InT, int P>
__global__ void __launch_bounds__(256) q8_act_prep_kernel(const InT* __restrict__ act, uint8_t* __restrict__ img, float* __restrict__ scale,
                                                          uint32_t M, uint32_t K, uint32_t MP) {
    const int lane = threadIdx.x & 31;
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t nblk = K / 256, run = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (run >= MP * nblk) return;
    const uint32_t m = run / nblk, b = run % nblk;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.f;
    if (m < M) {
        const size_t base = (size_t)m * K + (size_t)b * 256 + 8 * lane;
        if constexpr (sizeof(InT) == 4) {
            const float4 x = __ldg(reinterpret_cast<const float4*>(act + base)), y = __ldg(reinterpret_cast<const float4*>(act + base) + 1);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
        } else {
            const uint4 rr = __ldg(reinterpret_cast<const uint4*>(act + base));
            v[0] = __uint_as_float(rr.x << 16); v[1] = __uint_as_float(rr.x & 0xFFFF0000u);
            v[2] = __uint_as_float(rr.y << 16); v[3] = __uint_as_float(rr.y & 0xFFFF0000u);
            v[4] = __uint_as_float(rr.z << 16); v[5] = __uint_as_float(rr.z & 0xFFFF0000u);
            v[6] = __uint_as_float(rr.w << 16); v[7] = __uint_as_float(rr.w & 0xFFFF0000u);
        }
    }
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
    const float id = amax != 0.f ? __fdiv_rn(127.0f, amax) : 0.f;
    uint32_t w[P][2];
#pragma unroll
    for (int pc = 0; pc < P; ++pc) w[pc][0] = w[pc][1] = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float rr = __fmul_rn(v[i], id);  // |rr| <= 127 (+ one rounding)
#pragma unroll
        for (int pc = 0; pc < P; ++pc) {
            const int c = max(-127, min(127, (int)rintf(rr)));
            w[pc][i >> 2] |= (uint32_t)(c & 0xFF) << (8 * (i & 3));
            rr = __fmul_rn(__fsub_rn(rr, (float)c), Q8_STEP);  // remainder in [-0.5, 0.5] -> [-127, 127]
        }
    }
#pragma unroll
    for (int pc = 0; pc < P; ++pc)
        *reinterpret_cast<uint2*>(img + ((size_t)(pc * MP + m) * K + (size_t)b * 256 + 8 * lane)) = make_uint2(w[pc][0], w[pc][1]);
    if (lane == 0) scale[(size_t)b * MP + m] = m < M ? __fdiv_rn(amax, 127.0f) : 0.f;
}

struct I8Layout {
    uint32_t nblk, ntiles, grid;
    size_t aux_off, total;
};
I8Layout i8_layout(size_t M, size_t K, size_t N, int sm_count) {
    I8Layout l{};
    l.nblk = (uint32_t)(K / 256);
    l.ntiles = (uint32_t)((N + 127) / 128);
    l.grid = l.ntiles < (uint32_t)sm_count ? l.ntiles : (uint32_t)sm_count;
    l.aux_off = (M * K + 255) & ~(size_t)255;
    l.total = l.aux_off + (((size_t)l.nblk * AUX_BYTES + 255) & ~(size_t)255);
    return l;
}

struct Q8Layout {
    uint32_t MP, P, nblk, ntiles, grid;
    size_t img_bytes, scale_off, total;
};
Q8Layout q8_layout(size_t M, size_t K, size_t N, int sm_count) {
    Q8Layout l{};
    (void)M;
    l.MP = 32u;  // 17..32 rows
    l.P = 2u;
    l.nblk = (uint32_t)(K / 256);
    l.ntiles = (uint32_t)((N + 127) / 128);
    l.grid = l.ntiles < (uint32_t)sm_count ? l.ntiles : (uint32_t)sm_count;
    l.img_bytes = ((size_t)l.P * l.MP * K + 255) & ~(size_t)255;
    l.scale_off = l.img_bytes;
    l.total = l.scale_off + (((size_t)l.nblk * l.MP * 4 + 255) & ~(size_t)255);
    return l;
}

cudaError_t launch_q8_kernel(const CUtensorMap& amap, const CUtensorMap& wmap, const Q8Params& p, uint32_t grid, size_t smem, cudaStream_t st) {
    static PerDeviceOnce attrs;
    cudaError_t e = attrs.run([] { return cudaFuncSetAttribute(smallm_i8_q8_0_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448); });
    if (e != cudaSuccess) return e;
    return launch_pdl(smallm_i8_q8_0_kernel, dim3(grid), dim3(I8_THREADS), smem, st, amap, wmap, p);
}

cudaError_t launch_smallm_q8_0(const void* act, int act_dtype, const void* w, void* out, int out_dtype, size_t M, size_t K, size_t N, void* ws,
                               size_t ws_bytes, int sm_count, cudaStream_t st, unsigned int* status, bool* ws_too_small, char* err,
                               size_t err_len, bool acts_prepared) {
    *ws_too_small = false;
    const Q8Layout l = q8_layout(M, K, N, sm_count);
    if (!ws || ws_bytes < l.total || (reinterpret_cast<uintptr_t>(ws) & 15)) { *ws_too_small = true; return cudaSuccess; }
    uint8_t* base = static_cast<uint8_t*>(ws);
    float* scale = reinterpret_cast<float*>(base + l.scale_off);
    if (!acts_prepared) {
        const dim3 pg((l.MP * l.nblk + 7) / 8);
        cudaError_t e;
        if (act_dtype == DT_F32)
            e = launch_pdl(q8_act_prep_kernel<float, 2>, pg, dim3(256), 0, st, static_cast<const float*>(act), base, scale, (uint32_t)M, (uint32_t)K, l.MP);
        else
            e = launch_pdl(q8_act_prep_kernel<__nv_bfloat16, 2>, pg, dim3(256), 0, st, static_cast<const __nv_bfloat16*>(act), base, scale, (uint32_t)M,
                           (uint32_t)K, l.MP);
        note_launch();
        if (e != cudaSuccess) return e;
    }
    EncodeTiledFn enc = encode_tiled();
    if (!enc) {
        snprintf(err, err_len, "cuTensorMapEncodeTiled is not available from this driver");
        return cudaErrorNotSupported;
    }
    Q8Params p{};
    p.w = static_cast<const uint8_t*>(w);
    p.out = out;
    p.scale = scale;
    p.M = (uint32_t)M; p.N = (uint32_t)N; p.K = (uint32_t)K;
    p.nblk = l.nblk; p.ntiles = l.ntiles;
    const uint32_t NB = l.P * l.MP;
    p.idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((NB >> 3) << 17) | ((128u >> 4) << 24);  // int32 <- s8 x s8, K-major, N = P MP, M = 128
    p.out_dtype = out_dtype;
    p.status = status;
    const uint32_t stage = 2 * A_ATOM + 2 * NB * 128;
    p.ns = 2;
    p.nsc = p.ns + 2 + 2;
    const uint32_t fixed = 1024 + ((p.nsc * Q8_SLOT + 1023u) & ~1023u) + p.ns * stage;
    p.nr = ((232448u - 1024u - 1024u - fixed) / Q8_RAW_TILE) & ~1u;  // even: see launch_smallm_i8
    if (p.nr > 4) p.nr = 4;
    const size_t smem = 1024 + fixed + (size_t)p.nr * Q8_RAW_TILE;

    const cuuint32_t estr[2] = {1, 1};
    CUtensorMap amap, wmap;
    {
        const cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)NB};
        const cuuint64_t gstride[1] = {(cuuint64_t)K};
        const cuuint32_t box[2] = {128u, NB};
        CUresult cr = enc(&amap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, base, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cr != CUDA_SUCCESS) {
            snprintf(err, err_len, "cuTensorMapEncodeTiled failed with code %d (activation image %p, K=%zu, rows %u)", (int)cr, (void*)base, K, NB);
            return cudaErrorInvalidValue;
        }
    }
    {
        // packed rows as 16-bit units (a box dimension holds at most 256 elements): 136 units = the 272 bytes of a 256-run
        const uint32_t row_bytes = l.nblk * 272;
        const cuuint64_t gdim[2] = {(cuuint64_t)(row_bytes / 2), (cuuint64_t)N};
        const cuuint64_t gstride[1] = {(cuuint64_t)row_bytes};
        const cuuint32_t box[2] = {136u, 128u};
        CUresult cr = enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(w), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cr != CUDA_SUCCESS) {
            snprintf(err, err_len, "cuTensorMapEncodeTiled failed with code %d (weight pointer %p, row bytes %u, N=%zu)", (int)cr, w, row_bytes, N);
            return cudaErrorInvalidValue;
        }
    }
    cudaError_t e = launch_q8_kernel(amap, wmap, p, l.grid, smem, st);
    note_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

// Shapes the integer tensor-core kernels take.  Q4_K: 8 <= M <= 16, whole 256-blocks (rows are multiples of 16 bytes:
// 144-byte blocks), (tile, block) pairs within 32 bits.  Q8_0: 17 <= M <= 32 (up to 16 rows the mma.sync kernel is as fast), K a multiple
// of 256 (rows of whole 272-byte runs).  Both deal whole tiles only.
bool smallm_i8_supported(int fmt, size_t M, size_t K, size_t N) {
    if (K % 256 != 0 || K < 256 || N < 1 || (N + 127) / 128 * (K / 256) >= (1u << 30)) return false;
    return (fmt == FMT_Q8_0 && M > 16 && M <= 32) || (fmt == FMT_Q4_K && M >= 8 && M <= 16 && K / 256 <= 64);
}
size_t smallm_i8_workspace_bytes(int fmt, size_t M, size_t K, size_t N, int sm_count) {
    return fmt == FMT_Q8_0 ? q8_layout(M, K, N, sm_count).total : i8_layout(M, K, N, sm_count).total;
}
// Where they beat the mma.sync kernel (measured).  Q4_K: matrices with enough 128-row tiles for whole tiles on every SM: the longest CTA
// has at most eight blocks more than an even share would give it.  Q8_0: one pass over the weights instead of two,
// matrices with enough tiles to occupy half of the SMs.
bool smallm_i8_preferred(int fmt, size_t M, size_t K, size_t N, int sm_count) {
    if (!smallm_i8_supported(fmt, M, K, N)) return false;
    const size_t tiles = (N + 127) / 128, sms = (size_t)sm_count, nblk = K / 256;
    if (fmt == FMT_Q8_0) return tiles >= sms / 2;
    return (tiles + sms - 1) / sms * nblk <= (tiles * nblk + sms - 1) / sms + 8 && tiles >= sms * 3 / 4;
}

// acts_prepared: a previous call with the same activations and scratch left the image there (gate, then up).
cudaError_t launch_smallm_i8(int fmt, const void* act, int act_dtype, const void* w, void* out, int out_dtype, size_t M, size_t K,
                             size_t N, void* ws, size_t ws_bytes, int sm_count, cudaStream_t st, unsigned int* status,
                             bool* ws_too_small, char* err, size_t err_len, bool acts_prepared) {
    if (fmt == FMT_Q8_0)
        return launch_smallm_q8_0(act, act_dtype, w, out, out_dtype, M, K, N, ws, ws_bytes, sm_count, st, status, ws_too_small, err, err_len, acts_prepared);
    *ws_too_small = false;
    const I8Layout l = i8_layout(M, K, N, sm_count);
    if (!ws || ws_bytes < l.total || (reinterpret_cast<uintptr_t>(ws) & 15)) { *ws_too_small = true; return cudaSuccess; }
    uint8_t* base = static_cast<uint8_t*>(ws);
    uint8_t* codes = base;
    uint8_t* aux = base + l.aux_off;
    if (!acts_prepared) {
        const uint32_t runs = (uint32_t)M * l.nblk;
        const dim3 pg((runs + 7) / 8);
        cudaError_t e = act_dtype == DT_F32
                            ? launch_pdl(i8_act_prep_kernel<float>, pg, dim3(256), 0, st, static_cast<const float*>(act), codes, aux, (uint32_t)M, l.nblk)
                            : launch_pdl(i8_act_prep_kernel<__nv_bfloat16>, pg, dim3(256), 0, st, static_cast<const __nv_bfloat16*>(act), codes, aux,
                                         (uint32_t)M, l.nblk);
        note_launch();
        if (e != cudaSuccess) return e;
    }
    EncodeTiledFn enc = encode_tiled();
    if (!enc) {
        snprintf(err, err_len, "cuTensorMapEncodeTiled is not available from this driver");
        return cudaErrorNotSupported;
    }
    I8Params p{};
    p.out = out;
    p.aux = aux;
    p.M = (uint32_t)M; p.N = (uint32_t)N;
    p.nblk = l.nblk;
    p.tbase = l.ntiles / l.grid; p.trem = l.ntiles % l.grid;
    // int32 accumulator, signed 8-bit x signed 8-bit, both K-major, N = MP, M = 128
    p.idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((I8_MP >> 3) << 17) | ((128u >> 4) << 24);
    p.out_dtype = out_dtype;
    p.status = status;
    const uint32_t stage = 2 * A_ATOM + 2 * I8_MP * 128;
    p.ns = 3;
    p.nsc = p.ns + 2 + 2;
    const uint32_t fixed = 1024 + ((p.nsc * SC_SLOT + 128 * I8_MP * 4 + 1023u) & ~1023u) + p.ns * stage;
    // The ring of packed tiles must have an EVEN depth: block i lives in slot i % nr and is read by decode set i & 1, so with
    // an even depth a slot always belongs to one set and that set sees every phase of the slot's barrier.  With an odd depth
    // the sets would alternate on a slot, a set would wait for phase k having last seen phase k - 2, and a parity wait cannot
    // tell those apart when the fill in between is late (fills may complete out of order).
    p.nr = ((232448u - 1024u - 1024u - fixed) / RAW_TILE) & ~1u;
    if (p.nr > 6) p.nr = 6;
    const size_t smem = 1024 + fixed + (size_t)p.nr * RAW_TILE;

    const cuuint32_t estr[2] = {1, 1};
    CUtensorMap amap, wmap;
    {
        const cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)M};
        const cuuint64_t gstride[1] = {(cuuint64_t)K};
        const cuuint32_t box[2] = {128u, I8_MP};
        CUresult cr = enc(&amap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, codes, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cr != CUDA_SUCCESS) {
            snprintf(err, err_len, "cuTensorMapEncodeTiled failed with code %d (activation image %p, K=%zu, M=%zu)", (int)cr, (void*)codes, K, M);
            return cudaErrorInvalidValue;
        }
    }
    {
        const uint32_t row_bytes = l.nblk * 144;
        const cuuint64_t gdim[2] = {(cuuint64_t)row_bytes, (cuuint64_t)N};
        const cuuint64_t gstride[1] = {(cuuint64_t)row_bytes};
        const cuuint32_t box[2] = {RAW_PITCH, 128u};
        CUresult cr = enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(w), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cr != CUDA_SUCCESS) {
            snprintf(err, err_len, "cuTensorMapEncodeTiled failed with code %d (weight pointer %p, row bytes %u, N=%zu)", (int)cr, w, row_bytes, N);
            return cudaErrorInvalidValue;
        }
    }
    static PerDeviceOnce attrs;
    cudaError_t e = attrs.run([] { return cudaFuncSetAttribute(smallm_i8_q4k_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448); });
    if (e != cudaSuccess) return e;
    e = launch_pdl(smallm_i8_q4k_kernel, dim3(l.grid), dim3(I8_THREADS), smem, st, amap, wmap, p);
    note_launch();
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

}  // namespace b200q
