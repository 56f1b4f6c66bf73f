// Batched rows on the 5th-generation tensor cores (tcgen05.mma, accumulators and A operand in TMEM) for Q4_K weights: prompts,
// and decode steps of many sequences.
//
// The reference's arithmetic for one 256-element super-block (native/src/q4k_matmul.c:143-251) is
//     y += d_x * ( d_w * S1 - dmin_w * S2 ),   S1 = sum_sb sc[sb] * <codes_sb, xq_sb>,   S2 = sum_sb mn[sb] * sum(xq_sb)
// with 4-bit codes, 6-bit sc / mn and int8 activation codes xq. Both sums are products of small integers, exact in f16 x f16 -> f32
// as long as their sums stay below 2^24: the A operand carries code*sc (<= 945 < 2048, exact in f16), the
// B operand the activation codes, and one super-block is 16 MMAs of K = 16 accumulated in TMEM. S2 is one
// more K = 16 MMA of (mn[sb] twice) x (sums of 16 codes, <= 2032). |S1| can reach 945 * 127 * 256 = 1.83 * 2^24: tiles of 32 and 64 rows
// accumulate its halves (128 products, below 2^24) apart and add them once, which gives the integer sum rounded to fp32 as the
// mma.sync kernel has it; tiles of 128 rows have no TMEM left for that and may lose last places of sums beyond 2^24 (all codes and
// scales near their largest and activations of one sign: error 9.1e-8 of the result instead of 5.9e-8; normal data is not affected).
// The CUDA cores only unpack nibbles into
// the A operand (one LOP3 + one HFMA2 per two elements, using the 0x6400|n trick: f16(1024+n)*s - 1024*s
// is n*s exactly under the fused rounding) and apply the three fp32 block scales once per super-block.
//
// CTA = 128 weight rows (TMEM lanes) x N activation rows (TMEM columns; N = 32, 64 or 128 by the batch). Warps:
//   producers   a thread owns a weight row and unpacks 64-element groups of a super-block into the row's TMEM lane
//               (tcgen05.st): sets of four warps, one set per group (N <= 64) or per two groups (N = 128, whose epilogue needs the
//               registers). Half a super-block, two groups, is one stage: the MMAs of one half run while the other is written.
//   epilogue    eight warps fold a finished super-block out of TMEM (tcgen05.ld), N / 2 fp32 accumulators per thread;
//   one warp    issues the MMAs and commits; two accumulators, so the MMAs of super-block i+1 overlap the fold of i;
//   two warps   post the copies: packed weight tiles (128 rows x 128 B, a tensor map), activation tiles (bulk).
// Few tiles leave SMs idle, so a cluster of CTAs may share a tile by parts of the contraction; their sums meet in shared memory
// and are added in the order of the parts, whoever finishes first.
// The activation side is prepared once per call by act_f16_tiles_kernel in the order of the operand (K-major, 128-byte swizzle).
// Every mbarrier wait is bounded; a wait that runs out raises the device flag, and the CTA still reaches
// the common exit where TMEM is freed.
//
// What bounds it: the chain of barrier waits between the roles (a wait on a phase that is already complete takes 60 to 120 cycles),
// so a super-block takes few of them and large stages.
#include "common.cuh"
#include "actquant.cuh"
#include "tma.cuh"
#include "f32x2.cuh"
#include "matvec_fused.cuh"
#include "tensor_map.cuh"

#include <cuda_fp16.h>
#include <algorithm>
#include <atomic>

namespace sk {

namespace {

constexpr int TC_M = 128;                       // weight rows of a tile
constexpr int TC_W_BYTES = TC_M * 128, TC_S2A_BYTES = TC_M * 32;      // codes and mins of a super-block
constexpr int TC_EPI_WARPS = 8;

template <int N>
struct TcShape {
    static constexpr int SETS = N == 128 ? 2 : 4, PROD_WARPS = 4 * SETS, THREADS = (PROD_WARPS + TC_EPI_WARPS + 3) * 32;
    static constexpr int WS = N == 128 ? 3 : N == 64 ? 5 : 6, BS = N == 128 ? 2 : N == 64 ? 3 : 4;      // super-blocks of weights, of activations in flight
    static constexpr int B_BYTES = N * 512, S2B_BYTES = N * 32, SLOT = B_BYTES + S2B_BYTES;
    static constexpr int OFF_B = WS * TC_W_BYTES, OFF_S2A = OFF_B + BS * SLOT, OFF_DX = OFF_S2A + 4 * TC_S2A_BYTES, OFF_DD = OFF_DX + 4 * N * 4;
    static constexpr int OFF_BAR = OFF_DD + 4 * TC_M * 4, BARS = 2 * WS + 2 * BS + 4 + 4 + 4;
    static constexpr int SMEM = OFF_BAR + BARS * 8 + 16 + 1024;             // the dynamic area is aligned to 1024 by hand
    // TMEM columns: two sets of S1 accumulators, one for each half of a super-block where there is room, one or two of S2, four A groups of 32
    static constexpr int S1_ACC = N == 128 ? 1 : 2, S2_SETS = N == 128 ? 1 : 2;
    static constexpr int COL_S2 = 2 * S1_ACC * N, COL_A = COL_S2 + S2_SETS * N;
    static_assert(COL_A + 128 <= 512, "TMEM");
    static constexpr uint32_t IDESC = (1u << 4) | ((uint32_t) (N >> 3) << 17) | ((uint32_t) (TC_M >> 4) << 24);   // f16 x f16 -> f32, K-major both
};

// K-major operand in the 128-byte swizzle: rows of 128 B (64 f16), groups of 8 rows 1024 B apart; a K = 16 step
// moves the start address by 32 B inside the swizzle atom.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
    return (uint64_t) ((saddr & 0x3ffffu) >> 4) | (1ull << 16) | ((uint64_t) (1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// K-major operand without swizzle: 8 rows x 16 B core matrices, lbo = next 8 k-elements, sbo = next 8 rows.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    return (uint64_t) ((saddr & 0x3ffffu) >> 4) | ((uint64_t) (lbo_bytes >> 4) << 16) | ((uint64_t) (sbo_bytes >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
// A operand in TMEM: lane = row, a 32-bit column holds two consecutive k
__device__ __forceinline__ void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t ta, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n\t"
        "tcgen05.wait::st.sync.aligned;"
        ::"r"(ta), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
          "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]),
          "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(skd::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ uint4 ld_nc_v4(const void* p) {      // volatile: stays where it is written, ahead of the waits
    uint4 r;
    asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive1(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(skd::smem_u32(bar)) : "memory");
}
// TMEM loads of eight columns each and the wait for them in ONE asm statement: the destination registers are only defined
// for the compiler once the wait has been issued, so no use of them can be scheduled ahead of it.
__device__ __forceinline__ void tmem_ld8(uint32_t ta, uint32_t tb, float (&u)[8], float (&v)[8]) {
    uint32_t r[8], q[8];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7])
        : "r"(ta), "r"(tb)
        : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) { u[i] = __uint_as_float(r[i]); v[i] = __uint_as_float(q[i]); }
}
// the same of three places, four columns each
__device__ __forceinline__ void tmem_ld3(uint32_t ta, uint32_t tb, uint32_t tc, float (&u)[4], float (&v)[4], float (&w)[4]) {
    uint32_t r[12];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%12];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4,%5,%6,%7}, [%13];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8,%9,%10,%11}, [%14];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11])
        : "r"(ta), "r"(tb), "r"(tc)
        : "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) { u[i] = __uint_as_float(r[i]); v[i] = __uint_as_float(r[4 + i]); w[i] = __uint_as_float(r[8 + i]); }
}
// ---- activation side: int8 codes -> f16 in core-matrix order, sums of 16 codes, transposed block scales (tile = N = 1 << nlog rows) ----
//   xh  [m_pad/N][cols/64][N/8][8 rows][8][8]  f16: the N x 64 k pieces of a super-block are contiguous, rows of 128 B
//                                               whose 16-byte chunks are XOR-swizzled with the row (128B swizzle);
//                                               inside every group of four k the order is (0,2,1,3), matching the
//                                               order in which the weight nibbles leave a 32-bit word
//   hs  [m_pad/N][bpr][N/8][2][8 rows][8]      f16 sums of 16 consecutive codes: 32 N bytes per (tile, super-block)
//   dxt [bpr][m_pad]                            fp32 block scales
__global__ void __launch_bounds__(256)
act_f16_tiles_kernel(ActQ8K act, int m, int m_pad, int cols, int nlog, __half* __restrict__ xh, __half* __restrict__ hs, float* __restrict__ dxt) {
    skd::pdl_launch_dependents();
    skd::pdl_wait();
    const int per_row = cols >> 4;
    const int64_t idx = (int64_t) blockIdx.x * 256 + threadIdx.x;
    if (idx >= (int64_t) m_pad * per_row) return;
    const int n = (int) (idx / per_row), seg = (int) (idx % per_row);        // 16 codes: elements 16*seg ..
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (n < m) raw = *reinterpret_cast<const uint4*>(act.q + (size_t) n * cols + (size_t) seg * 16);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    int sum = 0;
    __half out[16];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int b0 = (int8_t) (w[j] & 0xff), b1 = (int8_t) ((w[j] >> 8) & 0xff), b2 = (int8_t) ((w[j] >> 16) & 0xff), b3 = (int8_t) (w[j] >> 24);
        sum += b0 + b1 + b2 + b3;
        out[4 * j] = __int2half_rn(b0); out[4 * j + 1] = __int2half_rn(b2); out[4 * j + 2] = __int2half_rn(b1); out[4 * j + 3] = __int2half_rn(b3);
    }
    const int groups = 1 << (nlog - 3), tile = n >> nlog, ng = (n >> 3) & (groups - 1), r = n & 7;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int kcg = seg * 2 + c, it = kcg >> 3, kc = kcg & 7;            // 8-element chunk: 64-k piece it, chunk kc of the piece
        *reinterpret_cast<uint4*>(xh + (((((size_t) tile * (cols >> 6) + it) * groups + ng) * 8 + r) * 8 + (kc ^ r)) * 8) = *reinterpret_cast<const uint4*>(out + 8 * c);
    }
    const int kb = seg >> 4, j = seg & 15;
    hs[(((((size_t) tile * (cols >> 8) + kb) * groups + ng) * 2 + (j >> 3)) * 8 + r) * 8 + (j & 7)] = __int2half_rn(sum);
    if (j == 0) dxt[(size_t) kb * m_pad + n] = n < m ? act.d[(size_t) n * (cols >> 8) + kb] : 0.0f;
}

template <int N>
__global__ void __launch_bounds__(TcShape<N>::THREADS, 1)
q4k_gemm_tc_kernel(const __grid_constant__ CUtensorMap map_qs, const uint8_t* __restrict__ hdr, int rows, int bpr, int parts,
                   const __half* xh, const __half* hs, const float* dxt, int m, int m_pad,
                   float* y, const float* resid, int* __restrict__ timeout_flag) {
    typedef TcShape<N> S;
    extern __shared__ uint8_t raw[];
    uint8_t* smem = raw + ((1024 - (skd::smem_u32(raw) & 1023)) & 1023);
    uint64_t* w_full = (uint64_t*) (smem + S::OFF_BAR);      // weight tile landed (bytes)
    uint64_t* w_empty = w_full + S::WS;                      // read by all producer warps
    uint64_t* b_full = w_empty + S::WS;                      // activation tile and its sums landed (bytes)
    uint64_t* b_empty = b_full + S::BS;                      // read by the MMAs
    uint64_t* a_full = b_empty + S::BS;                      // half a super-block of A written, the second half with the mins
    uint64_t* a_empty = a_full + 2;                          // read by the MMAs
    uint64_t* s2_full = a_empty + 2;                         // scales of a super-block for the epilogue: (d, dmin) of the rows, block scales of the columns
    uint64_t* acc_full = s2_full + 4;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = (uint32_t*) (acc_empty + 2);
    uint32_t* gave_up = tmem_slot + 1;                       // a wait of the fold ran out: this part's sums are not whole

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int MMA_WARP = S::PROD_WARPS + TC_EPI_WARPS;
    const int part = blockIdx.x % parts, row0 = blockIdx.x / parts * TC_M, tile_n = blockIdx.y, col0 = tile_n * N;
    const int kb0 = (int) ((int64_t) bpr * part / parts), nk = (int) ((int64_t) bpr * (part + 1) / parts) - kb0;      // this CTA's super-blocks
    skd::pdl_launch_dependents();

    if (warp == MMA_WARP) {
        if (lane == 0) {
            for (int i = 0; i < S::WS; ++i) { skd::mbar_init(w_full + i, 1); skd::mbar_init(w_empty + i, S::PROD_WARPS); }
            for (int i = 0; i < S::BS; ++i) { skd::mbar_init(b_full + i, 1); skd::mbar_init(b_empty + i, 1); }
            for (int i = 0; i < 2; ++i) { skd::mbar_init(a_full + i, 8); skd::mbar_init(a_empty + i, 1); skd::mbar_init(acc_full + i, 1); skd::mbar_init(acc_empty + i, TC_EPI_WARPS); }
            for (int i = 0; i < 4; ++i) skd::mbar_init(s2_full + i, 8);
            skd::mbar_fence_init();
            *gave_up = 0;
        }
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(skd::smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == MMA_WARP) {
        // ------------------------------------------------ MMA issuer ------------------------------------------------
        const uint64_t d_b = smem_desc_sw128(skd::smem_u32(smem + S::OFF_B));
        int s = 0, round = 0;
        for (int i = 0; i < nk; ++i) {
            const int set = i & 1;
            if (i >= 2 && !skd::mbar_wait_warp(acc_empty + set, ((i >> 1) - 1) & 1, timeout_flag)) break;
            if (!skd::mbar_wait_warp(b_full + s, round & 1, timeout_flag)) break;
            bool ok = true;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (!(ok = skd::mbar_wait_warp(a_full + h, i & 1, timeout_flag))) break;
                // the one S2 accumulator: super-block i - 1 has been folded
                if (S::S2_SETS == 1 && h == 1 && i >= 1 && !(ok = skd::mbar_wait_warp(acc_empty + (set ^ 1), ((i - 1) >> 1) & 1, timeout_flag))) break;
                tc_fence_after();
                if (skd::elect_one()) {
                    // descriptors move in 16-byte units: a 64-k piece is 128 N bytes, a K = 16 step 32 bytes
                    const uint64_t db = d_b + (uint64_t) ((s * S::SLOT + h * (S::B_BYTES / 2)) >> 4);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        umma_f16_ta(tmem + (set * S::S1_ACC + (S::S1_ACC == 2 ? h : 0)) * N, tmem + S::COL_A + h * 64 + j * 8, db + (uint64_t) (((j >> 2) * (S::B_BYTES / 4) + (j & 3) * 32) >> 4),
                                    S::IDESC, (S::S1_ACC == 2 ? j : h | j) != 0 ? 1u : 0u);
                    umma_commit(a_empty + h);
                    if (h == 1) {
                        const uint32_t a2 = skd::smem_u32(smem + S::OFF_S2A + (i & 3) * TC_S2A_BYTES), b2 = skd::smem_u32(smem + S::OFF_B + s * S::SLOT + S::B_BYTES);
                        umma_f16(tmem + S::COL_S2 + (S::S2_SETS == 2 ? set * N : 0), smem_desc(a2, 128, 256), smem_desc(b2, 128, 256), S::IDESC, 0u);
                        umma_commit(b_empty + s);
                        umma_commit(acc_full + set);
                    }
                }
                __syncwarp();
            }
            if (!ok) break;
            if (++s == S::BS) { s = 0; ++round; }
        }
    } else if (warp == MMA_WARP + 1) {
        // ---------------------------------------- copies of weight tiles ----------------------------------------
        bool ok = true;
        for (int i = 0; i < nk; ++i) {
            const int s = i % S::WS;
            if (i >= S::WS && !(ok = skd::mbar_wait_warp(w_empty + s, (i / S::WS - 1) & 1, timeout_flag))) break;
            if (skd::elect_one()) {
                skd::mbar_expect_tx(w_full + s, TC_W_BYTES);
                skd::tma_load_2d(smem + s * TC_W_BYTES, &map_qs, (kb0 + i) * 128, row0, w_full + s);
            }
            __syncwarp();
        }
        if (!ok)                                       // give copies in flight time to land before the CTA leaves
            for (int i = 0; i < 64; ++i) __nanosleep(1000);
    } else if (warp == MMA_WARP + 2) {
        // ---------------------------------------- copies of activation tiles ----------------------------------------
        skd::pdl_wait();                               // the activation side is the predecessor's output
        bool ok = true;
        int s = 0, round = 0;
        for (int i = 0; i < nk; ++i) {
            if (round > 0 && !(ok = skd::mbar_wait_warp(b_empty + s, (round - 1) & 1, timeout_flag))) break;
            if (skd::elect_one()) {
                const size_t blk = (size_t) tile_n * bpr + kb0 + i;
                skd::mbar_expect_tx(b_full + s, S::SLOT);
                skd::bulk_g2s(smem + S::OFF_B + s * S::SLOT, xh + blk * (S::B_BYTES / 2), S::B_BYTES, b_full + s);
                skd::bulk_g2s(smem + S::OFF_B + s * S::SLOT + S::B_BYTES, hs + blk * (S::S2B_BYTES / 2), S::S2B_BYTES, b_full + s);
            }
            __syncwarp();
            if (++s == S::BS) { s = 0; ++round; }
        }
        if (!ok)
            for (int i = 0; i < 64; ++i) __nanosleep(1000);
    } else if (warp < S::PROD_WARPS) {
        // ------------------------------------------- producers of the A operand -------------------------------------------
        constexpr int PER = 4 / S::SETS;                // groups a set unpacks: its number, and two further where it takes two
        const int r = tid & 127, my = warp >> 2;        // weight row of the tile = TMEM lane (warp % 4 is its 32-lane quarter); set
        const bool writes_mins = my == S::SETS - 1;     // the set whose last group is the super-block's last; set 0 writes the columns' block scales
        const uint32_t a_lane = tmem + ((uint32_t) ((warp & 3) * 32) << 16) + S::COL_A;
        // headers straight from global memory, two super-blocks ahead (a tensor copy of 16-byte rows is no faster)
        const uint8_t* hrow = hdr + ((size_t) min(row0 + r, rows - 1) * bpr + kb0) * 16;
        uint4 hd1 = ld_nc_v4(hrow), hd2 = ld_nc_v4(hrow + (nk > 1 ? 16 : 0));
        float dx = 0.0f;
        for (int i = 0; i < nk; ++i) {
            const int s = i % S::WS;
            const uint4 hd = hd1;
            hd1 = hd2;
            if (i + 2 < nk) hd2 = ld_nc_v4(hrow + (size_t) (i + 2) * 16);
            if (!skd::mbar_wait_warp(w_full + s, (i / S::WS) & 1, timeout_flag)) break;
            const uint8_t* wrow = smem + s * TC_W_BYTES + r * 128;
            uint4 q[PER][2];
#pragma unroll
            for (int e = 0; e < PER; ++e)
#pragma unroll
                for (int c = 0; c < 2; ++c) q[e][c] = skd::lds128(wrow + (((2 * (my + 2 * e) + c) ^ (r & 7)) << 4));
            uint32_t sc_lo, sc_hi, mn_lo, mn_hi;
            skd::k4_unpack(hd.y, hd.z, hd.w, sc_lo, sc_hi, mn_lo, mn_hi);
            bool ok = true;
#pragma unroll
            for (int e = 0; e < PER; ++e) {
                const int st = my + 2 * e, h = st >> 1;          // k 0..31 of the group = low nibbles x sc[2 st], k 32..63 = high nibbles x sc[2 st + 1]
                // high nibbles stay in place (f16 1024 + 16 n) and take scale / 16, so only the odd bytes need a shift
                const uint32_t scw = (h ? sc_hi : sc_lo) >> (16 * (st & 1));
                const __half2 ml = __half2half2(__int2half_rn((int) (scw & 0xff))), mh = __half2half2(__hmul(__int2half_rn((int) ((scw >> 8) & 0xff)), __float2half_rn(0.0625f)));
                const __half2 nl = __hmul2(ml, __float2half2_rn(-1024.0f)), nh = __hmul2(mh, __float2half2_rn(-1024.0f));
                const uint32_t wv[8] = {q[e][0].x, q[e][0].y, q[e][0].z, q[e][0].w, q[e][1].x, q[e][1].y, q[e][1].z, q[e][1].w};
                uint32_t out[32];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t w = wv[k], w8 = w >> 8;
                    const uint32_t x02 = (w & 0x000f000fu) | 0x64006400u, x13 = (w8 & 0x000f000fu) | 0x64006400u;
                    const uint32_t y02 = (w & 0x00f000f0u) | 0x64006400u, y13 = (w8 & 0x00f000f0u) | 0x64006400u;
                    __half2 v;
                    v = __hfma2(*reinterpret_cast<const __half2*>(&x02), ml, nl); out[2 * k] = *reinterpret_cast<uint32_t*>(&v);
                    v = __hfma2(*reinterpret_cast<const __half2*>(&x13), ml, nl); out[2 * k + 1] = *reinterpret_cast<uint32_t*>(&v);
                    v = __hfma2(*reinterpret_cast<const __half2*>(&y02), mh, nh); out[16 + 2 * k] = *reinterpret_cast<uint32_t*>(&v);
                    v = __hfma2(*reinterpret_cast<const __half2*>(&y13), mh, nh); out[16 + 2 * k + 1] = *reinterpret_cast<uint32_t*>(&v);
                }
                if (i >= 1 && !(ok = skd::mbar_wait_warp(a_empty + h, (i - 1) & 1, timeout_flag))) break;
                tc_fence_after();
                tmem_st32(a_lane + st * 32, out);
                // Scales and mins go to one of four slots. The slot's last use was super-block i - 4, folded before the MMAs of i - 2 were
                // issued, and the wait above has seen MMAs of i - 1 complete.
                if (writes_mins && e == PER - 1) {
                    uint8_t* s2 = smem + S::OFF_S2A + (i & 3) * TC_S2A_BYTES + (r >> 3) * 256 + (r & 7) * 16;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {       // mins, each twice, against the sums of 16 codes
                        const uint32_t mnw = c ? mn_hi : mn_lo;
                        uint32_t mm[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const __half2 vv = __half2half2(__int2half_rn((int) ((mnw >> (8 * j)) & 0xff)));
                            mm[j] = *reinterpret_cast<const uint32_t*>(&vv);
                        }
                        *reinterpret_cast<uint4*>(s2 + c * 128) = make_uint4(mm[0], mm[1], mm[2], mm[3]);
                    }
                    *reinterpret_cast<uint32_t*>(smem + S::OFF_DD + ((i & 3) * TC_M + r) * 4) = hd.x;
                    fence_async_smem();
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive1(a_full + h);
                    // The weight slot goes back only now that what was read from it lies in TMEM. Given back right behind the reads, the next
                    // tile could overtake them: at 32 and 64 rows of 11008 x 4096 up to 15 of 100 queued calls had a warp's 32 rows of a
                    // group from the super-block WS further on.
                    if (e == PER - 1) mbar_arrive1(w_empty + s);
                    if (writes_mins && e == PER - 1) mbar_arrive1(s2_full + (i & 3));
                }
            }
            if (!ok) break;
            if (my == 0) {
                if (i == 0) { skd::pdl_wait(); if (r < N) dx = __ldcg(dxt + (size_t) kb0 * m_pad + col0 + r); }
                if (r < N) *reinterpret_cast<float*>(smem + S::OFF_DX + ((i & 3) * N + r) * 4) = dx;
                if (r < N && i + 1 < nk) dx = __ldcg(dxt + (size_t) (kb0 + i + 1) * m_pad + col0 + r);
                __syncwarp();
                if (lane == 0) mbar_arrive1(s2_full + (i & 3));
            }
        }
    } else {
        // ------------------------------- epilogue: fold every super-block out of TMEM -------------------------------
        const int r = tid & 127, ch = (warp - S::PROD_WARPS) >> 2;      // TMEM lane = weight row; which half of the columns
        constexpr int NC = N / 2, LD = S::S1_ACC == 2 ? 4 : 8;          // columns a load: what the registers take (eight are no faster at N = 32)
        uint64_t yacc[NC / 2];
#pragma unroll
        for (int c = 0; c < NC / 2; ++c) yacc[c] = 0;
        bool ok = true;
        for (int i = 0; i < nk; ++i) {
            const int set = i & 1;
            // the second long complete; observed for what it guards
            if (!(ok = skd::mbar_wait_warp(acc_full + set, (i >> 1) & 1, timeout_flag) && skd::mbar_wait_warp(s2_full + (i & 3), (i >> 2) & 1, timeout_flag))) { *gave_up = 1; break; }
            tc_fence_after();
            const uint32_t dd = *reinterpret_cast<const uint32_t*>(smem + S::OFF_DD + ((i & 3) * TC_M + r) * 4);
            const float dw = __half2float(__ushort_as_half((unsigned short) (dd & 0xffff))), dminw = __half2float(__ushort_as_half((unsigned short) (dd >> 16)));
            const uint64_t dw2 = skd::pk2(dw, dw), nd2 = skd::pk2(-dminw, -dminw);
            const float* dx = (const float*) (smem + S::OFF_DX) + (i & 3) * N + ch * NC;
            const uint32_t t0 = tmem + ((uint32_t) ((warp & 3) * 32) << 16) + ch * NC, t2 = t0 + S::COL_S2 + (S::S2_SETS == 2 ? set * N : 0);
#pragma unroll
            for (int c = 0; c < NC; c += LD) {
                float s1[LD], s2[LD], s1b[LD];
                if constexpr (S::S1_ACC == 2) tmem_ld3(t0 + 2 * set * N + c, t0 + (2 * set + 1) * N + c, t2 + c, s1, s1b, s2);
                else tmem_ld8(t0 + set * N + c, t2 + c, s1, s2);
                if (c + LD == NC) {                    // all accumulators have been read
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive1(acc_empty + set);
                }
#pragma unroll
                for (int j = 0; j < LD; j += 2) {
                    const float2 x2 = *reinterpret_cast<const float2*>(dx + c + j);
                    uint64_t sum = skd::pk2(s1[j], s1[j + 1]);
                    if (S::S1_ACC == 2) sum = skd::add2(sum, skd::pk2(s1b[j], s1b[j + 1]));
                    uint64_t& y2 = yacc[(c + j) / 2];
                    y2 = skd::fma2(skd::pk2(x2.x, x2.y), skd::fma2(dw2, sum, skd::mul2(nd2, skd::pk2(s2[j], s2[j + 1]))), y2);
                }
            }
        }
        if (parts > 1) {
            // this part's sums into shared memory, [column][row], where the activation tiles were (all MMAs have read them)
            float* mine = (float*) (smem + S::OFF_B) + (ch * NC) * TC_M + r;
#pragma unroll
            for (int c = 0; c < NC / 2; ++c) {
                const float2 v = skd::up2(yacc[c]);
                mine[(2 * c) * TC_M] = v.x; mine[(2 * c + 1) * TC_M] = v.y;
            }
        } else {
            skd::pdl_wait();                           // y and resid may still be in use by kernels launched before this one
            if (ok && row0 + r < rows) {
#pragma unroll
                for (int c = 0; c < NC / 2; ++c) {
                    const float2 v = skd::up2(yacc[c]);
                    const int col = col0 + ch * NC + 2 * c;
                    const size_t o = (size_t) col * rows + row0 + r;
                    if (col < m) y[o] = resid ? resid[o] + v.x : v.x;
                    if (col + 1 < m) y[o + rows] = resid ? resid[o + rows] + v.y : v.y;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
    if (parts > 1) {
        __syncwarp();
        skd::cluster_sync_all();                            // every part's sums are in place
        skd::pdl_wait();
        const uint32_t base = skd::smem_u32(smem + S::OFF_B);
        // one flag a lane: read in turn they cost 0.4 us a call of four parts
        const bool whole = !__any_sync(0xffffffffu, lane < parts && skd::ld_cluster(skd::smem_u32(gave_up), lane) != 0.0f);
        const int per = (N * TC_M / 4 + parts - 1) / parts * 4, e0 = part * per, e1 = min(N * TC_M, e0 + per);
        for (int e = e0 + tid; e < e1; e += S::THREADS) {
            const int row = row0 + (e & (TC_M - 1)), col = col0 + e / TC_M;
            if (!whole || row >= rows || col >= m) continue;
            float v = 0.0f;
            for (int p = 0; p < parts; ++p) v += skd::ld_cluster(base + e * 4, p);
            const size_t o = (size_t) col * rows + row;
            y[o] = resid ? resid[o] + v : v;           // resid may be y itself: read and written by this thread only
        }
        __syncwarp();
        skd::cluster_sync_all();                            // nobody leaves while its sums are still read
    }
}

// Clusters of `parts` CTAs the current device holds at once (they lie within a GPC, so 148 SMs hold 33 of four), found once per device; two
// threads that both find it missing find the same.
template <int N>
int tc_clusters(int parts) {
    static std::atomic<int> known[64][9];
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
    if (dev < 0 || dev >= 64) return std::max(1, sm_count() / parts);
    int n = known[dev][parts].load(std::memory_order_relaxed);
    if (n == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned) parts); cfg.blockDim = dim3(TcShape<N>::THREADS); cfg.dynamicSmemBytes = TcShape<N>::SMEM;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned) parts; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.attrs = at; cfg.numAttrs = 1;
        if (ensure_dynamic_smem((const void*) q4k_gemm_tc_kernel<N>, TcShape<N>::SMEM) != SKAINET_CUDA_OK ||
            cudaOccupancyMaxActiveClusters(&n, q4k_gemm_tc_kernel<N>, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = std::max(1, sm_count() / parts); }
        known[dev][parts].store(n, std::memory_order_relaxed);
    }
    return n;
}

// Microseconds fitted to calls of 1 K x 1 K to 22 K x 4 K weights: what precedes the kernel, a super-block, a round of CTAs (prologue, first
// loads, store), the exchange of a cluster.
constexpr float TC_BEFORE = 6.0f, TC_ROUND = 3.5f;
template <int N> constexpr float tc_unit() { return N == 128 ? 1.7f : N == 64 ? 1.28f : 1.1f; }
template <int N> constexpr float tc_exchange() { return N == 128 ? 3.5f : N == 64 ? 2.0f : 1.0f; }

// Parts of the contraction that share a tile: the number whose rounds of CTAs cost least (512 rows of 11008 x 4096: three rounds of whole
// tiles 100 us, five of halves 112). *cost is the whole call.
template <int N>
int tc_parts(int64_t tiles, int bpr, float* cost) {
    int best = 1;
    *cost = 1e30f;
    for (int p = 1; p <= 8 && p <= bpr; ++p) {
        const int64_t slots = p == 1 ? sm_count() : tc_clusters<N>(p), rounds = (tiles + slots - 1) / slots;
        const float c = TC_BEFORE + (float) rounds * (tc_unit<N>() * (float) ((bpr + p - 1) / p) + TC_ROUND + (p > 1 ? tc_exchange<N>() : 0.0f));
        if (c < *cost) { *cost = c; best = p; }
    }
    return best;
}

// What the mma.sync tile kernel takes for fewer than TC_ALWAYS_ROWS rows, fitted alike: its throughput, or its chain over the super-blocks.
float mma_cost(const Weight& w, int m) {
    const int mp = m <= 16 ? 16 : (m + 31) / 32 * 32;
    const int64_t ctas = (int64_t) ((w.rows + 63) / 64);
    const float rate = 2.0f * (float) mp * (float) w.rows * (float) w.cols / 210e6f;
    const float chain = (float) w.bpr * (m <= 16 ? 0.55f : m <= 32 ? 0.75f * (float) std::min<int64_t>(2, (ctas + sm_count() - 1) / sm_count()) : 1.2f);
    return 3.5f + std::max(rate, chain);
}

// Parts of a tile for m rows where this kernel is expected to cost less than the mma.sync one; 0 where it is not.
template <int N>
int tc_plan_n(const Weight& w, int m) {
    const float other = m < TC_ALWAYS_ROWS ? mma_cost(w, m) : 1e30f;
    if (other <= TC_BEFORE + TC_ROUND + tc_unit<N>()) return 0;              // below any call of this kernel
    float cost;
    const int parts = tc_parts<N>((int64_t) ((w.rows + TC_M - 1) / TC_M) * ((m + N - 1) / N), w.bpr, &cost);
    return cost > other ? 0 : parts;
}

// 1 = not taken: scratch that cannot be had (or would have to grow while the stream is being captured), or a weight no tensor map describes
template <int N>
int32_t launch_tc_n(const Weight& w, ActQ8K a, int m, float* y, const float* resid, int parts, cudaStream_t s) {
    typedef TcShape<N> S;
    const int m_pad = (m + N - 1) / N * N, m_tiles = (w.rows + TC_M - 1) / TC_M, n_tiles = m_pad / N;
    CUtensorMap mq;
    if (tensor_map_bytes(&mq, w.qs, w.rows, (int64_t) w.bpr * 128, TC_M) != SKAINET_CUDA_OK) return 1;
    SK_TRY(ensure_dynamic_smem((const void*) q4k_gemm_tc_kernel<N>, S::SMEM));
    const size_t xh_bytes = (size_t) m_pad * w.cols * 2, hs_bytes = (size_t) m_pad * (w.cols / 16) * 2;
    const size_t need = gemm_tc_scratch_bytes(m, w.cols);
    // the operand tiles live in the calling stream's own scratch (calls on different streams do not share them)
    if (scratch_capacity(s, SCRATCH_GEMM) < need) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) { cudaGetLastError(); return 1; }
    }
    void* base = nullptr;
    const int32_t st = scratch_get(s, SCRATCH_GEMM, need, &base);
    if (st == SKAINET_CUDA_ERR_OOM) return 1;
    if (st != SKAINET_CUDA_OK) return st;
    auto up = [](size_t v) { return (v + 255) & ~(size_t) 255; };
    __half* xh = (__half*) base;
    __half* hs = (__half*) ((uint8_t*) base + up(xh_bytes));
    float* dxt = (float*) ((uint8_t*) base + up(xh_bytes) + up(hs_bytes));
    const int64_t n16 = (int64_t) m_pad * (w.cols / 16);
    SK_CUDA(launch_pdl(act_f16_tiles_kernel, dim3((unsigned) ((n16 + 255) / 256)), dim3(256), 0, s, a, m, m_pad, w.cols, N == 128 ? 7 : N == 64 ? 6 : 5, xh, hs, dxt));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) (m_tiles * parts), (unsigned) n_tiles); cfg.blockDim = dim3(S::THREADS); cfg.dynamicSmemBytes = S::SMEM; cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned) parts; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    SK_CUDA(cudaLaunchKernelEx(&cfg, q4k_gemm_tc_kernel<N>, mq, (const uint8_t*) w.hdr, w.rows, w.bpr, parts, (const __half*) xh, (const __half*) hs, (const float*) dxt, m, m_pad, y, resid,
                               device_timeout_flag()));
    return SKAINET_CUDA_OK;
}

}  // namespace

// What launch_gemm_tc needs of SCRATCH_GEMM for m rows of cols inputs.
size_t gemm_tc_scratch_bytes(int m, int cols) {
    const size_t m_pad = (size_t) (m + 127) / 128 * 128;
    return m_pad * cols * 2 + m_pad * (cols / 16) * 2 + m_pad * (cols / 256) * 4 + 3 * 256;
}

// The tile (32, 64 or 128 activation rows) and the parts that share one for m rows; 0 where the mma.sync tile kernel is the quicker.
int gemm_tc_plan(const Weight& w, int m, int* parts) {
    *parts = 0;
    if (w.enc != SKAINET_ENC_Q4_K || m < TC_MIN_ROWS || w.bpr < 1) return 0;
    const int tile = m <= 32 ? 32 : m <= 64 ? 64 : 128;
    *parts = tile == 32 ? tc_plan_n<32>(w, m) : tile == 64 ? tc_plan_n<64>(w, m) : tc_plan_n<128>(w, m);
    return *parts ? tile : 0;
}

// y[m][w.rows] (= resid +) for quantized activation rows through tiles of 32, 64 or 128, `parts` CTAs a tile
int32_t launch_gemm_tc_tiles(const Weight& w, ActQ8K a, int m, float* y, const float* resid, int tile, int parts, cudaStream_t s) {
    return tile == 32 ? launch_tc_n<32>(w, a, m, y, resid, parts, s) : tile == 64 ? launch_tc_n<64>(w, a, m, y, resid, parts, s) : launch_tc_n<128>(w, a, m, y, resid, parts, s);
}

// The same where it is the quicker. Returns 1 when not taken (the caller falls back to the mma.sync tile kernel).
int32_t launch_gemm_tc(const Weight& w, ActQ8K a, int m, float* y, const float* resid, cudaStream_t s) {
    int parts;
    const int tile = gemm_tc_plan(w, m, &parts);
    return tile ? launch_gemm_tc_tiles(w, a, m, y, resid, tile, parts, s) : 1;
}

}  // namespace sk
