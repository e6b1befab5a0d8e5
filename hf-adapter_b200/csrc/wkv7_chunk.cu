// Chunked (WY / DPLR) WKV-7 prefill scan, the intra-chunk contractions on tensor cores.
//
// One CTA per (sequence, head), two CTAs an SM.  The sequence is cut into chunks of 16 tokens (the result does not depend on
// it, so the caller's chunk size is only validated).  With a~ = -kk, b~ = kk*a, the state S0 [value i x key n] before the chunk, R_t
// the product of the decays of the chunk's tokens behind t, R_-1 that of all sixteen:
//
//   S0d = S0 R_-1   aE = a~_t / R_{t-1}   rP = r_t / R_t   kD = k_s R_s   bD = b~_s R_s        (16 x 64, tf32 operands)
//   A_ak = tril_strict(aE kD^T)   A_ab = tril_strict(aE bD^T)   A_qk = tril(rP kD^T)   A_qb = tril(rP bD^T)
//   U^T = (S0d aE^T + V^T A_ak^T) T^T,   T = (I - A_ab)^-1
//   Y^T = S0d rP^T + V^T A_qk^T + U^T A_qb^T
//   S'  = S0d + V^T kD + U^T bD
//
// (Scaled to the chunk's end, so that the keys which enter the state and those which the tokens behind them read are rounded alike:
// a rounded key is then a slightly other key in the same recurrence, and the delta rule takes part of the difference back.  Scaled to
// its start the states came out 2..4 % further from 64 bits; 16 tokens, 4 sequences x 40 heads, relative error of y / state 4.18e-4 /
// 1.617e-4 so, 4.147e-4 / 1.581e-4 now, and 4.146e-4 / 1.595e-4 with the former tiles of 64 tokens.)
//
// What bounds it: the shared-memory pipe on an SM with two heads (99 % of its active cycles in the fullest SM, 85 % on average; tensor
// pipe 52 / 45 %, issue slots 57 / 49 %, HBM 27 %) and the serial chain S0 -> U -> S' of a head, which is kept in
// registers.  Four STATE warps own 16 value rows each; the rows of the state never meet, so these warps never wait for one another,
// and a warp's state is an mma accumulator that becomes the next product's A operand where it is: the two columns a lane holds of an
// accumulator tile are read as k positions tq and tq + 4 of the A fragment, and the B operands are read in the same permuted order
// (physical column 16 p + 4 tq + 2 e + f is column 2 tq + f of tile 2 p + e, so a lane's share of two tiles is one 16-byte
// piece).  Everything that does not depend on the state is made ahead by four PREP warps, one chunk
// each in turn, into a ring of six slots: decay products, scaled operands, the four 16 x 16 products, the inverse.  mma.sync
// and not tcgen05: these products are 16 rows high, and through tensor memory every link of the chain costs a store, a
// fence, an issue, a commit and a load, about 700 cycles (a tile of 64 tokens with five such links took 16.9 k cycles with one CTA
// an SM).  8 sequences x 4096 tokens x 32 heads, in a row: 1150 -> 434 us (0.38 of the HBM floor of 165 us; 420..436 by box), raw decays 1209 -> 454.
//
// Products that contain decay-scaled factors (range e^9.7 over 16 tokens with the model's decays) run on operands rounded to tf32;
// products of bounded quantities (A_* against V and U, the keys decayed to the chunk's end) run in fp16; T is inverted in fp32.
// U = rhs T^T takes both operands as tf32 pairs (hi + lo, three products: 21 bits, where a substitution in fp32 has 24; rhs itself
// has the 11 of its operands).  U enters the state as an fp16 pair: the state is rounded to tf32 as an operand four times as
// often as with 64-token tiles, and with U in one fp16 its error against 64 bits came out up to 2 % larger than theirs.  Relative
// errors now, over 16..4096 tokens, three forms of decay, slow and fast: y 4.05e-4..4.71e-4, states 1.19e-4..3.07e-4; with the former tiles
// 4.06e-4..5.29e-4 and 1.23e-4..4.07e-4.
#include <type_traits>

#include "umma.cuh"

namespace rwkv7 {
namespace ck {
constexpr int C = 16, N = 64;       // tokens per chunk, head size
constexpr int SLOTS = 6;            // chunks in the ring
constexpr int STATE_WARPS = 4, PREP_WARPS = 4, THREADS = 32 * (STATE_WARPS + PREP_WARPS);
// byte offsets in a slot
constexpr int O_AE = 0;                 // aE [16][64] tf32, 16-byte pieces of odd rows swapped in groups of four
constexpr int O_RP = O_AE + 4096;       // rP, same layout
constexpr int O_KD = O_RP + 4096;       // kD [16][64] fp16 in permuted columns, 16-byte pieces xored by row & 7
constexpr int O_BD = O_KD + 2048;       // bD, same layout
constexpr int O_V = O_BD + 2048;        // v [16][64] fp16, pieces xored by row & 7
constexpr int O_T = O_V + 2048;         // T [16][TS] fp32 (before that A_ab transposed)
constexpr int TS = 24;                  // row stride of T: the lanes' 8-byte reads of four rows meet no bank twice
constexpr int O_M = O_T + 16 * TS * 4;  // A_ak, A_qk, A_qb as B fragments: [matrix][lane][4] pairs of fp16
constexpr int O_GL = O_M + 3 * 512;     // product of all decays of the chunk [64] fp32
constexpr int SLOT_BYTES = O_GL + 256;
constexpr int O_KD32 = O_KD;            // kD [16][64] fp32 while the four products are formed; then kD and bD in fp16
constexpr int O_BD32 = O_V;             // bD, likewise; then v, T and the A_* fragments
static_assert(O_BD32 + 4096 <= O_GL, "bD fits before the decays");
constexpr int YS = 48;                  // row stride (bytes) of a state warp's 16 x 16 output tile: conflict-free
constexpr int O_Y = SLOTS * SLOT_BYTES;
constexpr int O_BAR = O_Y + STATE_WARPS * 16 * YS;
constexpr int SMEM_BYTES = O_BAR + 2 * SLOTS * 8 + 16;
static_assert(2 * (SMEM_BYTES + 1024) <= 228 * 1024, "two CTAs an SM");
static_assert(SLOT_BYTES % 128 == 0 && O_BAR % 8 == 0, "alignment of the slots and barriers");
}  // namespace ck

struct ChunkArgs {
    const __half *r, *k, *v, *kk, *a;
    const void* w;
    const float* state_in;
    float* state_out;
    __half* y;
    int T, H;
    unsigned int* error;
};

// Round to tf32 (nearest, ties away) with one integer add: the tensor core ignores the 13 low mantissa bits, so adding
// half an ulp of tf32 to the bit pattern is all the rounding needs (cvt.rna.tf32 runs on the quarter-rate conversion pipe).
__device__ __forceinline__ uint32_t tf32_bits(float x) { return __float_as_uint(x) + 0x1000u; }
// x = hi + lo to 22 bits, both usable as tf32 operands
__device__ __forceinline__ void tf32_pair(float x, uint32_t& hi, uint32_t& lo) {
    hi = tf32_bits(x) & 0xffffe000u;
    lo = tf32_bits(x - __uint_as_float(hi));
}
__device__ __forceinline__ float fast_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&d)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void stmatrix4_trans(uint32_t addr, const uint32_t (&d)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};"
                 ::"r"(addr), "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]) : "memory");
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// W_MODE 0: decay in fp16, 1: decay in fp32, 2: raw w in fp16 (decay = e^(-0.606531 sigmoid w))
template <int W_MODE>
__global__ void __launch_bounds__(ck::THREADS, 2) wkv7_chunk_kernel(const ChunkArgs p) {
    using namespace ck;
    using WPair = typename std::conditional<W_MODE == 1, float2, __half2>::type;
    extern __shared__ __align__(128) unsigned char sm[];
    uint64_t* full = reinterpret_cast<uint64_t*>(sm + O_BAR);  // [SLOTS] the chunk is in the slot
    uint64_t* empty = full + SLOTS;                            // [SLOTS] the four state warps have read it
    volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + SLOTS);
    const AbortCtx actx{abort_flag, p.error};

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tq = lane & 3;  // row / column group of a lane in an mma fragment
    const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H;
    const size_t stride = (size_t)p.H * N;                      // elements between consecutive tokens
    const size_t base = ((size_t)b * p.T * p.H + h) * N;        // element offset of token 0
    const int nchunks = p.T / C;
    if (tid == 0) {
        for (int s = 0; s < SLOTS; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], STATE_WARPS);
        }
        *abort_flag = 0;
        mbar_fence_init();
    }
    __syncthreads();

    if (warp >= STATE_WARPS) {
        // ------------------------------------------------------------------------------------------------ PREP
        // lane = channels 2 lane, 2 lane + 1 of all 16 tokens
        const int pw = warp - STATE_WARPS;
        const uint32_t f_even = (lane >> 1) * 16 + (lane & 1) * 8;         // fp32 row, even token
        const uint32_t f_odd = ((lane >> 1) ^ 4) * 16 + (lane & 1) * 8;    // odd token
        const uint32_t h_piece = (lane >> 3) * 2 + (lane & 1), h_in = ((lane >> 1) & 3) * 4;  // fp16 row: piece and byte of the permuted pair
        for (int c = pw; c < nchunks; c += PREP_WARPS) {
            const int slot = c % SLOTS;
            unsigned char* sl = sm + slot * SLOT_BYTES;
            const size_t row0 = base + (size_t)c * C * stride;
            const size_t off = row0 + 2 * lane;
            if (c + PREP_WARPS < nchunks) {  // the warp's next chunk on its way to L2: lane = token, half of its operands
                const size_t o = row0 + (size_t)(PREP_WARPS * C + (lane >> 1)) * stride;
                if (lane & 1) {
                    prefetch_l2(p.kk + o);
                    prefetch_l2(p.a + o);
                    prefetch_l2(reinterpret_cast<const char*>(p.w) + o * (W_MODE == 1 ? 4 : 2));
                    if (W_MODE == 1) prefetch_l2(reinterpret_cast<const char*>(p.w) + o * 4 + 128);
                } else {
                    prefetch_l2(p.r + o);
                    prefetch_l2(p.k + o);
                    prefetch_l2(p.v + o);
                }
            }
            // from the last token to the first: R = product of the decays behind a token, inv = 1 / R
            float2 R = make_float2(1.f, 1.f), lr = make_float2(0.f, 0.f);
#pragma unroll
            for (int tb = 1; tb >= 0; --tb) {
                __half2 r2[8], k2[8], kk2[8], a2[8];
                WPair w2[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const size_t o = off + (size_t)(tb * 8 + j) * stride;
                    w2[j] = *reinterpret_cast<const WPair*>(reinterpret_cast<const char*>(p.w) + o * (W_MODE == 1 ? 4 : 2));
                    kk2[j] = *reinterpret_cast<const __half2*>(p.kk + o);
                    a2[j] = *reinterpret_cast<const __half2*>(p.a + o);
                    k2[j] = *reinterpret_cast<const __half2*>(p.k + o);
                    r2[j] = *reinterpret_cast<const __half2*>(p.r + o);
                }
                float2 inv = make_float2(fast_rcp(R.x), fast_rcp(R.y));
                if (tb == 1 && c >= SLOTS && !mbar_wait(&empty[slot], (c / SLOTS - 1) & 1, actx, kErrWaitEmpty)) goto out;
#pragma unroll
                for (int j = 7; j >= 0; --j) {
                    float2 w;
                    if constexpr (W_MODE == 1) w = w2[j];
                    else w = __half22float2(w2[j]);
                    const float2 kk = __half22float2(kk2[j]), a = __half22float2(a2[j]), k = __half22float2(k2[j]), r = __half22float2(r2[j]);
                    const uint32_t o = (tb * 8 + j) * 256 + ((j & 1) ? f_odd : f_even);
                    *reinterpret_cast<float2*>(sl + O_KD32 + o) = make_float2(k.x * R.x, k.y * R.y);
                    *reinterpret_cast<float2*>(sl + O_BD32 + o) = make_float2(kk.x * a.x * R.x, kk.y * a.y * R.y);
                    *reinterpret_cast<uint2*>(sl + O_RP + o) = make_uint2(tf32_bits(r.x * inv.x), tf32_bits(r.y * inv.y));
                    if constexpr (W_MODE == 2) {
                        // logarithms are summed, and what the state itself is multiplied by, chunk after chunk, is rounded to nearest: an
                        // approximate exponential a token, multiplied up, took 6.1e-5 off a state that 8192 tokens hardly decay
                        // (raw w of -6), this 1.2e-6, and the former tiles 1.9e-6
                        lr.x -= 0.606531f * fast_rcp(1.f + __expf(-w.x));
                        lr.y -= 0.606531f * fast_rcp(1.f + __expf(-w.y));
                        R = tb == 0 && j == 0 ? make_float2(1.f + expm1f(lr.x), 1.f + expm1f(lr.y)) : make_float2(__expf(lr.x), __expf(lr.y));
                    } else {
                        R.x *= w.x;
                        R.y *= w.y;
                    }
                    inv = make_float2(fast_rcp(R.x), fast_rcp(R.y));
                    *reinterpret_cast<uint2*>(sl + O_AE + o) = make_uint2(tf32_bits(-kk.x * inv.x), tf32_bits(-kk.y * inv.y));
                }
            }
            *reinterpret_cast<float2*>(sl + O_GL + lane * 8) = R;
            uint4 vv[4];  // v of the chunk: 128 pieces of 16 bytes
#pragma unroll
            for (int i = 0; i < 4; ++i)
                vv[i] = *reinterpret_cast<const uint4*>(p.v + row0 + (size_t)(i * 4 + (lane >> 3)) * stride + (lane & 7) * 8);
            __syncwarp();
            // the four products: rows t of aE (0) and rP (1) against kD (n-tiles 0, 1) and bD (2, 3)
            float acc[2][4][4];
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[m][q][e] = 0.f;
#pragma unroll
            for (int pp = 0; pp < 4; ++pp) {
                const uint32_t o = g * 256 + tq * 16 + ((pp ^ (g & 1)) * 64);  // row g; row g + 8 has the same parity
                uint4 A[2][2], B[4];
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    A[0][hf] = *reinterpret_cast<const uint4*>(sl + O_AE + hf * 2048 + o);
                    A[1][hf] = *reinterpret_cast<const uint4*>(sl + O_RP + hf * 2048 + o);
                    B[hf] = *reinterpret_cast<const uint4*>(sl + O_KD32 + hf * 2048 + o);
                    B[2 + hf] = *reinterpret_cast<const uint4*>(sl + O_BD32 + hf * 2048 + o);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    B[q].x += 0x1000u; B[q].y += 0x1000u; B[q].z += 0x1000u; B[q].w += 0x1000u;  // round to tf32
                }
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int q = 0; q < 4; ++q) mma_tf32(acc[m][q], A[m][0].x, A[m][1].x, A[m][0].y, A[m][1].y, B[q].x, B[q].y);
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int q = 0; q < 4; ++q) mma_tf32(acc[m][q], A[m][0].z, A[m][1].z, A[m][0].w, A[m][1].w, B[q].z, B[q].w);
            }
            // kD and bD in fp16
            uint32_t kd[16], bd[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                const uint32_t o = t * 256 + ((t & 1) ? f_odd : f_even);
                const float2 k2 = *reinterpret_cast<const float2*>(sl + O_KD32 + o), b2 = *reinterpret_cast<const float2*>(sl + O_BD32 + o);
                kd[t] = pack_half2(k2.x, k2.y);
                bd[t] = pack_half2(b2.x, b2.y);
            }
            __syncwarp();  // kD and bD are read: their room is free
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                const uint32_t o = t * 128 + ((h_piece ^ (t & 7)) << 4) + h_in;
                *reinterpret_cast<uint32_t*>(sl + O_KD + o) = kd[t];
                *reinterpret_cast<uint32_t*>(sl + O_BD + o) = bd[t];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = i * 4 + (lane >> 3);
                *reinterpret_cast<uint4*>(sl + O_V + t * 128 + (((lane & 7) ^ (t & 7)) << 4)) = vv[i];
            }
            // masks; tile q of a product holds (t = g, s = 8 q + 2 tq, + 1) in [0], [1] and t = g + 8 in [2], [3], which is what
            // the B fragment of its transpose wants in the same lane
            auto masked = [&](const float (&lo)[4], const float (&hi)[4], int diag, float (&o)[8]) {  // keeps s < t + diag
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int t = g + (e >> 1) * 8, s = 2 * tq + (e & 1);
                    o[e] = s < t + diag ? lo[e] : 0.f;
                    o[4 + e] = s + 8 < t + diag ? hi[e] : 0.f;
                }
            };
            auto store_frag = [&](int which, const float (&o)[8]) {
                *reinterpret_cast<uint4*>(sl + O_M + which * 512 + lane * 16) =
                    make_uint4(pack_half2(o[0], o[1]), pack_half2(o[4], o[5]), pack_half2(o[2], o[3]), pack_half2(o[6], o[7]));
            };
            float mk[8];
            masked(acc[0][0], acc[0][1], 0, mk);
            store_frag(0, mk);
            masked(acc[1][0], acc[1][1], 1, mk);
            store_frag(1, mk);
            masked(acc[1][2], acc[1][3], 1, mk);
            store_frag(2, mk);
            masked(acc[0][2], acc[0][3], 0, mk);
            float* Tm = reinterpret_cast<float*>(sl + O_T);
#pragma unroll
            for (int e = 0; e < 4; ++e) {  // A_ab transposed: row s, column t
                Tm[(2 * tq + (e & 1)) * TS + g + (e >> 1) * 8] = mk[e];
                Tm[(8 + 2 * tq + (e & 1)) * TS + g + (e >> 1) * 8] = mk[4 + e];
            }
            __syncwarp();
            // T = (I - A_ab)^-1 by forward substitution, lane = column (both halves of the warp do the same)
            float x[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) x[t] = t == (lane & 15) ? 1.f : 0.f;
#pragma unroll
            for (int s = 0; s < 15; ++s) {
#pragma unroll
                for (int t4 = (s + 1) / 4; t4 < 4; ++t4) {
                    const float4 l4 = *reinterpret_cast<const float4*>(Tm + s * TS + t4 * 4);
                    const float l[4] = {l4.x, l4.y, l4.z, l4.w};
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (t4 * 4 + e > s) x[t4 * 4 + e] = fmaf(l[e], x[s], x[t4 * 4 + e]);
                }
            }
            __syncwarp();
            if (lane < 16) {
#pragma unroll
                for (int t = 0; t < 16; ++t) Tm[t * TS + lane] = x[t];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[slot]);
        }
    } else {
        // ------------------------------------------------------------------------------------------------ STATE
        // rows 16 warp + g (+ 8); S[j] is accumulator tile j: [0], [1] = row g, [2], [3] = row g + 8
        float S[8][4];
        const size_t srow = ((size_t)bh * N + warp * 16 + g) * N + tq * 4;
#pragma unroll
        for (int pp = 0; pp < 4; ++pp)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const float4 t4 = *reinterpret_cast<const float4*>(p.state_in + srow + hf * 8 * N + pp * 16);
                S[2 * pp][2 * hf] = t4.x; S[2 * pp][2 * hf + 1] = t4.y;
                S[2 * pp + 1][2 * hf] = t4.z; S[2 * pp + 1][2 * hf + 1] = t4.w;
            }
        const int l7 = lane & 7, mi = lane >> 3;                              // ldmatrix / stmatrix: row and matrix this lane addresses
        const uint32_t v_at = (l7 + (mi >> 1) * 8) * 128 + (((2 * warp + (mi & 1)) ^ l7) << 4);
        const uint32_t d_row = (l7 + (mi & 1) * 8) * 128;
        unsigned char* ystage = sm + O_Y + warp * 16 * YS;
        const uint32_t y_st = smem_u32(ystage + (l7 + (mi >> 1) * 8) * YS + (mi & 1) * 16);
        const uint32_t y_ld = (lane >> 1) * YS + (lane & 1) * 16;
        __half* yp = p.y + base + (size_t)(lane >> 1) * stride + warp * 16 + (lane & 1) * 8;
        const uint32_t f_at = g * 256 + tq * 16;
        for (int c = 0; c < nchunks; ++c) {
            const int slot = c % SLOTS;
            const unsigned char* sl = sm + slot * SLOT_BYTES;
            const uint32_t sl_u32 = smem_u32(sl);
            if (!mbar_wait(&full[slot], (c / SLOTS) & 1, actx, kErrWaitFull)) goto out;
            __syncwarp();
            uint32_t va[4];
            ldmatrix4_trans(va, sl_u32 + O_V + v_at);
            const uint4 mak = *reinterpret_cast<const uint4*>(sl + O_M + lane * 16);
            const uint4 mqk = *reinterpret_cast<const uint4*>(sl + O_M + 512 + lane * 16);
            float au[2][2][4], ar[2][4];  // [tokens 0..7, 8..15][tiles of even, odd index]: S0d aE^T + V^T A_ak^T, S0d rP^T + V^T A_qk^T
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) au[nt][0][e] = au[nt][1][e] = ar[nt][e] = 0.f;
            mma_f16(au[0][0], va, mak.x, mak.y);
            mma_f16(au[1][0], va, mak.z, mak.w);
            mma_f16(ar[0], va, mqk.x, mqk.y);
            mma_f16(ar[1], va, mqk.z, mqk.w);
#pragma unroll
            for (int pp = 0; pp < 4; ++pp) {
                const uint32_t o = f_at + ((pp ^ (g & 1)) * 64);
                const uint4 a0 = *reinterpret_cast<const uint4*>(sl + O_AE + o), a1 = *reinterpret_cast<const uint4*>(sl + O_AE + 2048 + o);
                const uint4 r0 = *reinterpret_cast<const uint4*>(sl + O_RP + o), r1 = *reinterpret_cast<const uint4*>(sl + O_RP + 2048 + o);
                const float4 gl = *reinterpret_cast<const float4*>(sl + O_GL + pp * 64 + tq * 16);
                uint32_t kd[4];
                ldmatrix4_trans(kd, sl_u32 + O_KD + d_row + (((2 * pp + (mi >> 1)) ^ l7) << 4));
                float(&s0)[4] = S[2 * pp];
                float(&s1)[4] = S[2 * pp + 1];
                s0[0] *= gl.x; s0[1] *= gl.y; s0[2] *= gl.x; s0[3] *= gl.y;
                s1[0] *= gl.z; s1[1] *= gl.w; s1[2] *= gl.z; s1[3] *= gl.w;
                const uint32_t e0 = tf32_bits(s0[0]), e1 = tf32_bits(s0[2]), e2 = tf32_bits(s0[1]), e3 = tf32_bits(s0[3]);
                const uint32_t o0 = tf32_bits(s1[0]), o1 = tf32_bits(s1[2]), o2 = tf32_bits(s1[1]), o3 = tf32_bits(s1[3]);
                mma_tf32(au[0][0], e0, e1, e2, e3, a0.x, a0.y);
                mma_tf32(au[1][0], e0, e1, e2, e3, a1.x, a1.y);
                mma_tf32(au[0][1], o0, o1, o2, o3, a0.z, a0.w);
                mma_tf32(au[1][1], o0, o1, o2, o3, a1.z, a1.w);
                mma_tf32(ar[0], e0, e1, e2, e3, r0.x, r0.y);
                mma_tf32(ar[1], e0, e1, e2, e3, r1.x, r1.y);
                mma_tf32(ar[0], o0, o1, o2, o3, r0.z, r0.w);
                mma_tf32(ar[1], o0, o1, o2, o3, r1.z, r1.w);
                mma_f16(s0, va, kd[0], kd[1]);
                mma_f16(s1, va, kd[2], kd[3]);
            }
            // U^T = rhs T^T: the two halves of T's lower triangle that are not zero, operands as hi + lo
            uint32_t ua[4], ul[4];  // fp16 and what it leaves
            {
                const float* Tm = reinterpret_cast<const float*>(sl + O_T) + g * TS + 2 * tq;
                const float2 t00 = *reinterpret_cast<const float2*>(Tm), t10 = *reinterpret_cast<const float2*>(Tm + 8 * TS),
                             t11 = *reinterpret_cast<const float2*>(Tm + 8 * TS + 8);
                uint32_t th[6], tl[6];
                tf32_pair(t00.x, th[0], tl[0]); tf32_pair(t00.y, th[1], tl[1]);
                tf32_pair(t10.x, th[2], tl[2]); tf32_pair(t10.y, th[3], tl[3]);
                tf32_pair(t11.x, th[4], tl[4]); tf32_pair(t11.y, th[5], tl[5]);
                uint32_t rh[2][4], rl[2][4];
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) tf32_pair(au[nt][0][e] + au[nt][1][e], rh[nt][e], rl[nt][e]);
                float u0[4], u1[4], c0[4], c1[4];  // products of the high parts, and the corrections
#pragma unroll
                for (int e = 0; e < 4; ++e) u0[e] = u1[e] = c0[e] = c1[e] = 0.f;
                mma_tf32(u1, rh[0][0], rh[0][2], rh[0][1], rh[0][3], th[2], th[3]);
                mma_tf32(c1, rl[0][0], rl[0][2], rl[0][1], rl[0][3], th[2], th[3]);
                mma_tf32(u0, rh[0][0], rh[0][2], rh[0][1], rh[0][3], th[0], th[1]);
                mma_tf32(c0, rl[0][0], rl[0][2], rl[0][1], rl[0][3], th[0], th[1]);
                mma_tf32(u1, rh[1][0], rh[1][2], rh[1][1], rh[1][3], th[4], th[5]);
                mma_tf32(c1, rh[0][0], rh[0][2], rh[0][1], rh[0][3], tl[2], tl[3]);
                mma_tf32(c0, rh[0][0], rh[0][2], rh[0][1], rh[0][3], tl[0], tl[1]);
                mma_tf32(c1, rl[1][0], rl[1][2], rl[1][1], rl[1][3], th[4], th[5]);
                mma_tf32(c1, rh[1][0], rh[1][2], rh[1][1], rh[1][3], tl[4], tl[5]);
                auto pair = [](float x, float y, uint32_t& hi, uint32_t& lo) {
                    const __half2 h = __floats2half2_rn(x, y);
                    const float2 f = __half22float2(h);
                    hi = *reinterpret_cast<const uint32_t*>(&h);
                    lo = pack_half2(x - f.x, y - f.y);
                };
                pair(u0[0] + c0[0], u0[1] + c0[1], ua[0], ul[0]);
                pair(u0[2] + c0[2], u0[3] + c0[3], ua[1], ul[1]);
                pair(u1[0] + c1[0], u1[1] + c1[1], ua[2], ul[2]);
                pair(u1[2] + c1[2], u1[3] + c1[3], ua[3], ul[3]);
            }
#pragma unroll
            for (int pp = 0; pp < 4; ++pp) {
                uint32_t bd[4];
                ldmatrix4_trans(bd, sl_u32 + O_BD + d_row + (((2 * pp + (mi >> 1)) ^ l7) << 4));
                mma_f16(S[2 * pp], ua, bd[0], bd[1]);
                mma_f16(S[2 * pp + 1], ua, bd[2], bd[3]);
                mma_f16(S[2 * pp], ul, bd[0], bd[1]);
                mma_f16(S[2 * pp + 1], ul, bd[2], bd[3]);
            }
            const uint4 mqb = *reinterpret_cast<const uint4*>(sl + O_M + 1024 + lane * 16);
            mma_f16(ar[0], ua, mqb.x, mqb.y);
            mma_f16(ar[1], ua, mqb.z, mqb.w);
            __syncwarp();  // the slot is read; the previous chunk's output tile as well
            if (lane == 0) mbar_arrive(&empty[slot]);
            const uint32_t yt[4] = {pack_half2(ar[0][0], ar[0][1]), pack_half2(ar[0][2], ar[0][3]),
                                    pack_half2(ar[1][0], ar[1][1]), pack_half2(ar[1][2], ar[1][3])};
            stmatrix4_trans(y_st, yt);  // Y^T fragments as rows of 16 values per token
            __syncwarp();
            *reinterpret_cast<uint4*>(yp + (size_t)c * C * stride) = *reinterpret_cast<const uint4*>(ystage + y_ld);
        }
#pragma unroll
        for (int pp = 0; pp < 4; ++pp)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf)
                *reinterpret_cast<float4*>(p.state_out + srow + hf * 8 * N + pp * 16) =
                    make_float4(S[2 * pp][2 * hf], S[2 * pp][2 * hf + 1], S[2 * pp + 1][2 * hf], S[2 * pp + 1][2 * hf + 1]);
    }
out:;
}

template <int W_MODE>
static int launch_chunk(const ChunkArgs& p, int ctas, cudaStream_t st) {
    const cudaError_t e = cudaFuncSetAttribute(wkv7_chunk_kernel<W_MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, ck::SMEM_BYTES);
    RWKV7_REQUIRE(e == cudaSuccess, RWKV7_ERR_CUDA, "wkv7_chunk_scan: %s", cudaGetErrorString(e));
    wkv7_chunk_kernel<W_MODE><<<ctas, ck::THREADS, ck::SMEM_BYTES, st>>>(p);
    return check_launch("wkv7_chunk_kernel");
}

}  // namespace rwkv7

using namespace rwkv7;

extern "C" int rwkv7_wkv7_chunk_scan(const void* r, const void* w, const void* k, const void* v, const void* kk, const void* a,
                                     const float* state_in, float* state_out, void* y, int B, int T, int H, int N, int chunk,
                                     int dtype, int w_mode, void* stream) {
    RWKV7_REQUIRE(N == 64, RWKV7_ERR_UNSUPPORTED, "wkv7_chunk_scan: head size must be 64, got %d", N);
    RWKV7_REQUIRE(dtype == RWKV7_F16, RWKV7_ERR_UNSUPPORTED, "wkv7_chunk_scan: fp16 activations only");
    RWKV7_REQUIRE(chunk == 16 || chunk == 32 || chunk == 64, RWKV7_ERR_UNSUPPORTED, "wkv7_chunk_scan: chunk must be 16, 32 or 64");
    RWKV7_REQUIRE(B > 0 && H > 0 && T > 0 && T % chunk == 0, RWKV7_ERR_INVALID,
                  "wkv7_chunk_scan: B, H, T must be positive and T a multiple of chunk (B=%d T=%d H=%d chunk=%d)", B, T, H, chunk);
    RWKV7_REQUIRE(w_mode >= 0 && w_mode <= 2, RWKV7_ERR_INVALID, "wkv7_chunk_scan: w_mode must be 0, 1 or 2");
    RWKV7_REQUIRE(r && w && k && v && kk && a && state_in && state_out && y, RWKV7_ERR_INVALID, "wkv7_chunk_scan: null pointer");
    const void* ptrs[] = {r, w, k, v, kk, a, state_in, state_out, y};
    for (const void* q : ptrs) RWKV7_REQUIRE(aligned(q, 16), RWKV7_ERR_ALIGN, "wkv7_chunk_scan: pointers must be 16-byte aligned");
    ChunkArgs p{reinterpret_cast<const __half*>(r), reinterpret_cast<const __half*>(k), reinterpret_cast<const __half*>(v),
                reinterpret_cast<const __half*>(kk), reinterpret_cast<const __half*>(a), w, state_in, state_out,
                reinterpret_cast<__half*>(y), T, H, kernel_error_word()};
    RWKV7_REQUIRE(p.error != nullptr, RWKV7_ERR_CUDA, "wkv7_chunk_scan: cannot resolve the device error word");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return w_mode == 0 ? launch_chunk<0>(p, B * H, st) : w_mode == 1 ? launch_chunk<1>(p, B * H, st) : launch_chunk<2>(p, B * H, st);
}
