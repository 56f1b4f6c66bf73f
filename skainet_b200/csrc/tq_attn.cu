// Decode attention over a TurboQuant store without a residual stage (kvstore.cu), straight from the packed blocks: split-K as
// attn_decode_mma_kernel (attention.cu), each warp decoding its 16-key tiles into shared memory just before it multiplies them.
// The decoded rows, rounded to binary16, equal those of tq_decode_kernel bit for bit: same products, same butterflies in the same
// order, same rounding.
//
// Two lanes decode a row (head_dim / 2 elements each, so all Walsh-Hadamard stages but the last stay inside a lane, and run as
// packed fp32 pairs); a tile's 16 rows are one pass of the warp. The blocks are a quarter of the binary16 rows or less, so what
// bounds the kernel is the instructions of the transform (some 900 per lane and tile), not the bytes: 8 heads x 128 over 4096
// positions (4 bits) read 6 MB. There a call takes 13.2 us, merge included; decoding the window to HBM first and attending the
// copy, as stores with a residual stage still do, took five launches and 38.9 us.
#include "common.cuh"
#include "turboquant.cuh"
#include "attn_frag.cuh"
#include "tma.cuh"
#include "f32x2.cuh"

#include <algorithm>

namespace sk {

namespace {

constexpr int TA_WARPS = 8;

// Half a row's block as it lies in the store: EL elements
template <int EL>
struct Packed {
    uint32_t w[EL / 4];            // as many words as eight bits per code take
    float scale[EL / 32];
    uint32_t sign[EL / 32];
};

template <int EL>
__device__ __forceinline__ void load_packed(Packed<EL>& p, const TqPlane& pl, int64_t half_row, bool live) {
    const uint8_t* codes = pl.codes + half_row * (EL / 8) * pl.bits;
    if (EL == 64) {                // 16, 24, 32 or 64 bytes on an 8-byte boundary
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            uint2 v = make_uint2(0, 0);
            if (live && i < pl.bits) v = __ldg(reinterpret_cast<const uint2*>(codes) + i);
            p.w[2 * i] = v.x; p.w[(2 * i + 1) % (EL / 4)] = v.y;
        }
    } else {                       // 8, 12, 16 or 32 bytes on a 4-byte boundary
#pragma unroll
        for (int i = 0; i < 8; ++i) p.w[i] = live && i < pl.bits ? __ldg(reinterpret_cast<const uint32_t*>(codes) + i) : 0u;
    }
#pragma unroll
    for (int g = 0; g < EL / 32; ++g) {
        p.scale[g] = live ? __ldg(pl.scales + half_row * (EL / 32) + g) : 0.0f;
        p.sign[g] = live ? __ldg(pl.signs + half_row * (EL / 32) + g) : 0u;
    }
}

// codes -> fp32 (exact) times the group's scale; v[i] holds elements 2 i, 2 i + 1
template <int EL, int BITS>
__device__ __forceinline__ void scaled_codes(const Packed<EL>& p, uint64_t (&v)[EL / 2]) {
    constexpr float BIAS = 8388608.0f + (float) (1 << (BITS - 1));       // 2^23 + u has u in its low mantissa bits
    const uint64_t nb = skd::pk2(-BIAS, -BIAS);
#pragma unroll
    for (int i = 0; i < EL / 2; ++i) {
        uint32_t u[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int bit = (2 * i + k) * BITS, word = bit >> 5, off = bit & 31;
            if (BITS == 8) u[k] = __byte_perm(p.w[word] ^ 0x80808080u, 0x4b000000u, 0x7440 + (off >> 3));
            else {
                const uint32_t x = off + BITS <= 32 ? p.w[word] >> off : __funnelshift_r(p.w[word], p.w[(word + 1) % (EL / 4)], off);
                u[k] = (x & ((1u << BITS) - 1)) | 0x4b000000u;
            }
        }
        const uint64_t sc = skd::pk2(p.scale[i / 16], p.scale[i / 16]);
        v[i] = skd::mul2(skd::add2(skd::pk2(__uint_as_float(u[0]), __uint_as_float(u[1])), nb), sc);
    }
}

// Half a row decoded to binary16 at dst (EL elements, 16-byte chunks in order); the other half is with lane ^ 1.
template <int EL>
__device__ __forceinline__ void decode_half_row(const Packed<EL>& p, int bits, int half, uint8_t* dst) {
    uint64_t v[EL / 2];
    switch (bits) {
        case 2: scaled_codes<EL, 2>(p, v); break;
        case 3: scaled_codes<EL, 3>(p, v); break;
        case 4: scaled_codes<EL, 4>(p, v); break;
        default: scaled_codes<EL, 8>(p, v); break;
    }
    const uint64_t minus = skd::pk2(-1.0f, -1.0f);
#pragma unroll
    for (int i = 0; i < EL / 2; ++i) { const float2 a = skd::up2(v[i]); v[i] = skd::pk2(__fadd_rn(a.x, a.y), __fsub_rn(a.x, a.y)); }
#pragma unroll
    for (int h = 1; h < EL / 2; h <<= 1) {
#pragma unroll
        for (int i = 0; i < EL / 2; ++i) {
            if ((i & h) == 0) {
                const uint64_t a = v[i], b = v[i + h];
                v[i] = skd::add2(a, b); v[i + h] = skd::fma2(b, minus, a);
            }
        }
    }
    const float s = half ? -1.0f : 1.0f, nf = __fdiv_rn(1.0f, __fsqrt_rn((float) (2 * EL)));
    const uint64_t s2 = skd::pk2(s, s), norm = skd::pk2(nf, nf);
    uint32_t z[EL / 32];                               // signs of the even elements in the low half, of the odd ones in the high half
#pragma unroll
    for (int g = 0; g < EL / 32; ++g) {
        uint32_t e = p.sign[g] & 0x55555555u, o = (p.sign[g] >> 1) & 0x55555555u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            constexpr uint32_t m[4] = {0x33333333u, 0x0f0f0f0fu, 0x00ff00ffu, 0x0000ffffu};
            e = (e | (e >> (1 << k))) & m[k]; o = (o | (o >> (1 << k))) & m[k];
        }
        z[g] = e | (o << 16);
    }
    uint32_t out[EL / 2];
#pragma unroll
    for (int i = 0; i < EL / 2; ++i) {
        const float2 a = skd::up2(v[i]);
        const uint64_t o = skd::pk2(__shfl_xor_sync(0xffffffffu, a.x, 1), __shfl_xor_sync(0xffffffffu, a.y, 1));
        const float2 r = skd::up2(skd::mul2(skd::fma2(v[i], s2, o), norm));       // the lower half takes the sums, the upper the differences
        const __half2 h = __floats2half2_rn(r.x, r.y);
        out[i] = *reinterpret_cast<const uint32_t*>(&h) ^ ((z[i / 16] << (15 - i % 16)) & 0x80008000u);
    }
#pragma unroll
    for (int c = 0; c < EL / 8; ++c) *reinterpret_cast<uint4*>(dst + 16 * c) = make_uint4(out[4 * c], out[4 * c + 1], out[4 * c + 2], out[4 * c + 3]);
}

// A decoded row in shared memory: its halves HO apart, rows STRIDE apart, so that the writes of two lanes per row and the
// fragment reads (rows 2 t of the values; the keys' rows g meet two ways at worst) spread over the banks.
template <int D>
struct Row {
    static constexpr int HO = D == 128 ? 192 : 64, STRIDE = D == 128 ? 336 : 144;
    static __device__ __forceinline__ int chunk(int c) { return c < D / 16 ? 16 * c : HO + 16 * (c - D / 16); }
};

// grid (key splits, cache heads)
template <int D>
__global__ void __launch_bounds__(TA_WARPS * 32)
tq_attn_decode_kernel(const float* q, TqPlane kp, TqPlane vp, int64_t row0, int kv_heads, int G, int len, float scale, int chunk, int splits,
                      float* __restrict__ part, float* __restrict__ out_direct) {
    constexpr int EL = D / 2, S4 = D / 32, KS = D / 16, U = D / 64, NT = D / 8;
    __shared__ float sm_m[TA_WARPS][8], sm_l[TA_WARPS][8], sm_c[TA_WARPS][8];
    __shared__ uint4 sm_q[KS][32];
    __shared__ __align__(16) uint8_t sm_rows[TA_WARPS * 16 * Row<D>::STRIDE];        // tiles; after the loop the warps' accumulators
    static_assert(sizeof(float) * 8 * (D + 4) <= 16 * Row<D>::STRIDE, "a warp's accumulators take the place of its tile");
    skd::pdl_launch_dependents();
    skd::pdl_wait();
    const int split = blockIdx.x, kvh = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int begin = split * chunk, stop = min(len, begin + chunk);
    uint8_t* tile = sm_rows + warp * 16 * Row<D>::STRIDE;

    const int row = lane >> 1, half = lane & 1;
    auto load = [&](Packed<EL>& p, const TqPlane& pl, int k0) {
        const int key = k0 + row;
        load_packed<EL>(p, pl, ((row0 + min(key, len - 1)) * kv_heads + kvh) * 2 + half, key < stop);
    };
    constexpr int STEP = TA_WARPS * 16;
    int k0 = begin + warp * 16;
    Packed<EL> pk, pv;
    load(pk, kp, k0);
    load(pv, vp, k0);

    // q of head g as A fragments, per k-step {hi(k 2t..), lo(k 2t..), hi(k 2t+8..), lo(k 2t+8..)} (k-step 2s+j: floats 4j.. of chunk t+4s)
    for (int ks = warp; ks < KS; ks += TA_WARPS) {
        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
        if (g < G) f = skd::ld_dep((const float4*) (q + (int64_t) (kvh * G + g) * D + (t + 4 * (ks >> 1)) * 8 + 4 * (ks & 1)));
        uint4 a;
        split_pack(f.x, f.y, a.x, a.y);
        split_pack(f.z, f.w, a.z, a.w);
        sm_q[ks][lane] = a;
    }
    __syncthreads();

    float m = MASKED, l = 0.0f;
    float o[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) { o[i][0] = 0.f; o[i][1] = 0.f; o[i][2] = 0.f; o[i][3] = 0.f; }

    for (; k0 < stop; k0 += STEP) {
        decode_half_row<EL>(pk, kp.bits, half, tile + row * Row<D>::STRIDE + half * Row<D>::HO);
        if (k0 + STEP < stop) load(pk, kp, k0 + STEP);
        __syncwarp();
        // ---- scores of head g for keys k0 + {2t, 2t+1, 8+2t, 8+2t+1}
        float sc[4];
        {
            float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int s = 0; s < S4; ++s) {
                const uint4 qa = sm_q[2 * s][lane], qb = sm_q[2 * s + 1][lane];
                const uint32_t a0[4] = {qa.x, qa.y, qa.z, qa.w}, a1[4] = {qb.x, qb.y, qb.z, qb.w};
#pragma unroll
                for (int nt = 0; nt < 2; ++nt) {
                    const uint4 kr = *reinterpret_cast<const uint4*>(tile + (8 * nt + g) * Row<D>::STRIDE + Row<D>::chunk(t + 4 * s));
                    mma_f16(c[nt], a0, kr.x, kr.y);
                    mma_f16(c[nt], a1, kr.z, kr.w);
                }
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const int key = k0 + 8 * nt + 2 * t;
                sc[2 * nt] = key < stop ? (c[nt][0] + c[nt][2]) * scale : MASKED;
                sc[2 * nt + 1] = key + 1 < stop ? (c[nt][1] + c[nt][3]) * scale : MASKED;
            }
        }
        float mx = fmaxf(fmaxf(sc[0], sc[1]), fmaxf(sc[2], sc[3]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float mnew = fmaxf(m, mx);
        const float corr = fast_exp(m - mnew);
        const bool rescale = m != mnew && l != 0.0f;
        m = mnew;
        float p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = sc[i] > 0.5f * MASKED ? fast_exp(sc[i] - mnew) : 0.0f;
        l = l * corr + (p[0] + p[1]) + (p[2] + p[3]);
        if (__any_sync(0xffffffffu, rescale)) {
#pragma unroll
            for (int i = 0; i < NT; ++i) { o[i][0] *= corr; o[i][1] *= corr; o[i][2] *= corr; o[i][3] *= corr; }
        }
        uint32_t pa[4];
        split_pack(p[0], p[1], pa[0], pa[1]);
        split_pack(p[2], p[3], pa[2], pa[3]);
        __syncwarp();                                  // the keys of the tile have been read
        decode_half_row<EL>(pv, vp.bits, half, tile + row * Row<D>::STRIDE + half * Row<D>::HO);
        if (k0 + STEP < stop) load(pv, vp, k0 + STEP);
        __syncwarp();
        // ---- out[head g][dims] += P . V ; tile (u, i): column n <-> dim 8*(n + 8u) + i
#pragma unroll
        for (int u = 0; u < U; ++u) {
            uint32_t vr[4][4];
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const uint4 x = *reinterpret_cast<const uint4*>(tile + (2 * t + (kk & 1) + 8 * (kk >> 1)) * Row<D>::STRIDE + Row<D>::chunk(g + 8 * u));
                vr[kk][0] = x.x; vr[kk][1] = x.y; vr[kk][2] = x.z; vr[kk][3] = x.w;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                mma_f16(o[u * 8 + 2 * r], pa, __byte_perm(vr[0][r], vr[1][r], 0x5410), __byte_perm(vr[2][r], vr[3][r], 0x5410));
                mma_f16(o[u * 8 + 2 * r + 1], pa, __byte_perm(vr[0][r], vr[1][r], 0x7632), __byte_perm(vr[2][r], vr[3][r], 0x7632));
            }
        }
        __syncwarp();
    }
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    // ---- merge the warps (fixed order), one partial record per (head, split)
    if (t == 0) { sm_m[warp][g] = m; sm_l[warp][g] = l; }
    float* acc = reinterpret_cast<float*>(tile);       // [8][D + 4]
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            acc[g * (D + 4) + 8 * (2 * t + 8 * u) + i] = o[u * 8 + i][0] + o[u * 8 + i][2];
            acc[g * (D + 4) + 8 * (2 * t + 1 + 8 * u) + i] = o[u * 8 + i][1] + o[u * 8 + i][3];
        }
    __syncthreads();
    if (threadIdx.x < 8 * TA_WARPS) {
        const int w = threadIdx.x >> 3, hg = threadIdx.x & 7;
        float mxx = MASKED;
#pragma unroll
        for (int w2 = 0; w2 < TA_WARPS; ++w2) mxx = fmaxf(mxx, sm_m[w2][hg]);
        sm_c[w][hg] = sm_m[w][hg] > 0.5f * MASKED ? fast_exp(sm_m[w][hg] - mxx) : 0.0f;
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < G * D; idx += TA_WARPS * 32) {
        const int hg = idx / D, dd = idx % D;
        float at = 0.0f, lt = 0.0f, mxx = MASKED;
#pragma unroll
        for (int w = 0; w < TA_WARPS; ++w) {
            at += sm_c[w][hg] * reinterpret_cast<const float*>(sm_rows + w * 16 * Row<D>::STRIDE)[hg * (D + 4) + dd];
            lt += sm_c[w][hg] * sm_l[w][hg];
            mxx = fmaxf(mxx, sm_m[w][hg]);
        }
        if (out_direct) { out_direct[(int64_t) (kvh * G + hg) * D + dd] = lt > 0.0f ? at / lt : 0.0f; continue; }
        float* rec = part + ((int64_t) (kvh * G + hg) * splits + split) * (D + 2);
        rec[2 + dd] = at;
        if (dd == 0) { rec[0] = mxx; rec[1] = lt; }
    }
}

template <int D>
int32_t launch_d(const float* q, const TqPlane& kp, const TqPlane& vp, int64_t row0, int kv_heads, int G, int len, float scale, float* out, void* scratch, cudaStream_t s) {
    const int splits = decode_splits(1, kv_heads, len);
    const int chunk = ((len + splits - 1) / splits + 31) & ~31;
    float* part = (float*) scratch;
    SK_CUDA(launch_pdl(tq_attn_decode_kernel<D>, dim3(splits, kv_heads), dim3(TA_WARPS * 32), 0, s, q, kp, vp, row0, kv_heads, G, len, scale, chunk, splits, part,
                       splits == 1 ? out : (float*) nullptr));
    return splits == 1 ? SKAINET_CUDA_OK : launch_attn_merge(part, out, kv_heads * G, D, splits, s);
}

}  // namespace

// The route for stores without a residual stage, head_dim 64 or 128 and groups of 1, 2, 4 or 8 query heads: 1 = not taken.
int32_t launch_tq_attn_decode(const float* q, const TqPlane& kp, const TqPlane& vp, int layer, int start_pos, int len, int kv_heads, int q_heads, int head_dim,
                              int max_seq, float scale, float* out, void* scratch, cudaStream_t s) {
    const int G = q_heads / kv_heads;
    if (kp.rbits || vp.rbits || !kp.signs || !vp.signs || (G != 1 && G != 2 && G != 4 && G != 8) || (head_dim != 64 && head_dim != 128)) return 1;
    const int64_t row0 = (int64_t) layer * max_seq + start_pos;
    return head_dim == 128 ? launch_d<128>(q, kp, vp, row0, kv_heads, G, len, scale, out, scratch, s) : launch_d<64>(q, kp, vp, row0, kv_heads, G, len, scale, out, scratch, s);
}

}  // namespace sk
