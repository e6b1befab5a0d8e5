// Projections of a decode step over a few rows (1..8): several independent problems in ONE launch,
//
//   out_p[M, N_p] = epilogue_p( x_p[M, K_p] . W_p[N_p, K_p]^T )      p = 0..n_problems-1
//
// with W dense fp16 / bf16 ([N, K] rows), int4 group-wise or int8 per channel (the tiled copies of w4g_umma.cu).  A layer
// needs five such launches beside its recurrence: r / k / v with the LoRA "down" products, the LoRA "up" products, o, and
// the two of the FFN.
//
// Bound: HBM (the weights, once).  At these row counts the tcgen05 kernels pay for 64 activation rows whatever M is (a
// [128 x 128] block holds the tensor pipe 512 cycles = 4.2 TB/s over the chip) and a library GEMM adds a launch per
// epilogue, so here the weights go HBM -> registers -> mma.sync m16n8k16 with M as the narrow n side:
//   * every lane loads 16 bytes of one channel; the k order inside a unit is permuted so that those bytes ARE its
//     fragments of the A operand (x is read in the same order), no shared memory and no shuffle in between;
//   * a warp works on 32 channels, two units of K ahead; the warps of a CTA (eight, or four), and the CTAs of a cluster where
//     one CTA per channel tile would leave SMs idle, split K, and their sums are added in fixed order;
//   * the first units of weights are requested before the grid-dependency wait, under the preceding kernel's tail.
#include "umma.cuh"

namespace rwkv7 {

bool take_tiled_fresh(const void* tiled);  // w4g_umma.cu: the tiled copy was written by a kernel that may still run

namespace rg {
constexpr int kMaxProblems = 8;
constexpr int kMaxRows = 8;
constexpr int kWarps = 8, kThreads = kWarps * 32;  // of a CTA at most
constexpr int kSlots = 16;  // partial sums per CTA: warps x cluster size
constexpr int TM = 2, kTile = TM * 16;  // channels of a warp: with one 16-channel tile the reads of x weigh double (4096 -> 16384
                                        // int4, 8 rows: 24.6 us against 17.5)
// Tiled formats (w4g_umma.cu): blocks of [128 channels x 128 k], eight pieces of 16 channels each: [4 or 8 chunks of k][channel][16 bytes],
// for int4 then eight bytes for channels c and c + 8: their scales, their zeros.  Read by warps of 16 channels such pieces run at 5.9 TB/s; from
// blocks of [chunk][128 channels][16 bytes], where a warp's part of a block is 256 bytes here and there, at 3.6 (cp.async of nothing but
// weights).  In this kernel, which also converts, 4096 -> 16384 took 15.2 us, 14.8 with pieces, 14.4 with the scales of two channels in one load.
constexpr int kW4Block = 8704, kW8Block = 16384, kW4Piece = 1088, kW8Piece = 2048, kW4Scales = 1024, kChunk = 256;
enum Fmt { kDense = 0, kInt4 = 1, kInt8 = 2 };

struct Problem {
    const void *x, *W, *scale, *residual;
    void* out;
    int K, N, fmt, epi;
    int cta0;  // first CTA (of rank 0) of the problem
};
struct Args {
    Problem p[kMaxProblems];
    int n, M;
    int early;   // the weights may be read before the grid-dependency wait
    int wk;      // warps of a CTA that split K (1, 2, 4, 8); the others take further channels
    int splits;  // CTAs of a cluster, which split K further
};

template <typename T> __device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1);
template <> __device__ __forceinline__ void mma<__half>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <> __device__ __forceinline__ void mma<__nv_bfloat16>(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint4 ldg_stream(const void* p) {  // weights: read once, not kept in L1
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t orv) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(mask), "r"(orv));
    return d;
}
__device__ __forceinline__ uint32_t h2_sub_mul(uint32_t t, uint32_t z, uint32_t s) {
    uint32_t d;
    asm("{\n\t.reg .b32 u;\n\tsub.f16x2 u, %1, %2;\n\tmul.f16x2 %0, u, %3;\n\t}" : "=r"(d) : "r"(t), "r"(z), "r"(s));
    return d;
}
__device__ __forceinline__ uint32_t h2_fma_mul(uint32_t t, uint32_t m, uint32_t z, uint32_t s) {
    uint32_t d;
    asm("{\n\t.reg .b32 u;\n\tfma.rn.f16x2 u, %1, %2, %3;\n\tmul.f16x2 %0, u, %4;\n\t}" : "=r"(d) : "r"(t), "r"(m), "r"(z), "r"(s));
    return d;
}
// eight nibbles of one channel -> four fp16 pairs (k0 k1) (k2 k3) (k4 k5) (k6 k7) of the materialised weight: exact
// (q - zero), one rounding for the scale; the same steps as the tcgen05 kernel, so the two agree bit for bit in W
__device__ __forceinline__ void int4_word(uint32_t w, uint32_t z, uint32_t s, uint32_t (&o)[4]) {
    const uint32_t zlo = z * 0x00010001u + 0x64006400u, zhi = z * 0x00100010u + 0xD400D400u, w2 = w >> 8;
    o[0] = h2_sub_mul(and_or(w, 0x000F000Fu, 0x64006400u), zlo, s);
    o[1] = h2_fma_mul(and_or(w, 0x00F000F0u, 0x64006400u), 0x2C002C00u, zhi, s);
    o[2] = h2_sub_mul(and_or(w2, 0x000F000Fu, 0x64006400u), zlo, s);
    o[3] = h2_fma_mul(and_or(w2, 0x00F000F0u, 0x64006400u), 0x2C002C00u, zhi, s);
}
// four offset-binary bytes -> (k0 k1) (k2 k3), exact; the channel scale multiplies the fp32 sum
__device__ __forceinline__ void int8_word(uint32_t w, uint32_t& a, uint32_t& b) {
    asm("prmt.b32 %0, %1, %2, 0x4140;" : "=r"(a) : "r"(w), "r"(0x64646464u));
    asm("prmt.b32 %0, %1, %2, 0x4342;" : "=r"(b) : "r"(w), "r"(0x64646464u));
    asm("sub.f16x2 %0, %0, %1;" : "+r"(a) : "r"(0x64806480u));
    asm("sub.f16x2 %0, %0, %1;" : "+r"(b) : "r"(0x64806480u));
}

// ---- one unit of K: per lane W16 16-byte pieces of each of its channels, X16 of its x row ------------------------------
template <int FMT> struct Unit;
template <> struct Unit<kDense> { static constexpr int K = 64, W16 = 2, X16 = 2; };
template <> struct Unit<kInt4> { static constexpr int K = 128, W16 = 1, X16 = 4; };
template <> struct Unit<kInt8> { static constexpr int K = 128, W16 = 2, X16 = 4; };

template <int FMT> struct Regs {
    uint4 w[TM][2][Unit<FMT>::W16];  // [16-channel tile][channel gid / gid + 8][piece]
    uint2 sz[FMT == kInt4 ? TM : 1];  // scales of the lane's two channels of a tile, their zeros
    uint4 x[Unit<FMT>::X16];
};

// x row gid, unit u: the k of a lane's pieces follow the order its weight bytes have
template <int FMT>
__device__ __forceinline__ void load_x(uint4 (&x)[Unit<FMT>::X16], const uint4* row, bool live, int K, int u, int tig) {
#pragma unroll
    for (int q = 0; q < Unit<FMT>::X16; ++q) {
        int k;  // first of the eight k of piece q
        if constexpr (FMT == kDense) k = u * 64 + q * 32 + tig * 8;
        else if constexpr (FMT == kInt4) k = u * 128 + tig * 32 + q * 8;
        else k = u * 128 + (tig + (q >> 1) * 4) * 16 + (q & 1) * 8;
        x[q] = (live && (FMT != kDense || k < K)) ? row[k >> 3] : make_uint4(0, 0, 0, 0);
    }
}

// two accumulators per tile: consecutive MMAs do not wait for one another
template <typename T, int FMT>
__device__ __forceinline__ void unit_mma(float (&acc)[TM][2][4], const Regs<FMT>& r) {
#pragma unroll
    for (int q = 0; q < Unit<FMT>::X16; ++q)  // eight k per lane: two MMAs
#pragma unroll
        for (int t = 0; t < TM; ++t) {
            uint32_t a[2][4];  // [channel half][k pair]
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                if constexpr (FMT == kDense) {
                    const uint4 v = r.w[t][hh][q];
                    a[hh][0] = v.x; a[hh][1] = v.y; a[hh][2] = v.z; a[hh][3] = v.w;
                } else if constexpr (FMT == kInt4) {
                    const uint4 v = r.w[t][hh][0];
                    int4_word(q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w, (r.sz[t].y >> (hh * 8)) & 255u, __byte_perm(r.sz[t].x, 0, hh ? 0x3232 : 0x1010), a[hh]);
                } else {
                    const uint4 v = r.w[t][hh][q >> 1];
                    int8_word(q & 1 ? v.z : v.x, a[hh][0], a[hh][1]);
                    int8_word(q & 1 ? v.w : v.y, a[hh][2], a[hh][3]);
                }
            }
            mma<T>(acc[t][0], a[0][0], a[1][0], a[0][1], a[1][1], r.x[q].x, r.x[q].y);
            mma<T>(acc[t][1], a[0][2], a[1][2], a[0][3], a[1][3], r.x[q].z, r.x[q].w);
        }
}

// units [u0, u1) of the 32 channels from n0.  HALVES: the sums of those before `mid` go to slot 2 x warp
template <typename T, int FMT, bool HALVES>
__device__ __forceinline__ void stream(float (&sum)[TM][4], const Problem& p, const Args& args, int n0, int u0, int mid, int u1, float (*slots)[kMaxRows * (kTile + 1)]) {
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int K = p.K;
    const uint4* xrow = reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(p.x) + (size_t)gid * K);
    const bool live = gid < args.M;
    // one pointer per lane, one addition per unit; a 32-channel tile never leaves its 128-channel block
    const char* wp;
    const size_t row8 = (size_t)K * 16;  // dense: bytes between channels n and n + 8
    if constexpr (FMT == kDense) wp = reinterpret_cast<const char*>(p.W) + ((size_t)(n0 + gid) * K + (size_t)u0 * 64 + tig * 8) * 2;
    else wp = reinterpret_cast<const char*>(p.W) + ((size_t)(n0 >> 7) * (K >> 7) + u0) * (FMT == kInt4 ? kW4Block : kW8Block) +
              ((n0 >> 4) & 7) * (FMT == kInt4 ? kW4Piece : kW8Piece) + gid * 16 + tig * kChunk;
    const int soff = kW4Scales - gid * 8 - tig * kChunk;
    const int rows8 = (p.N - n0 - gid + 7) >> 3;  // dense: channels n0 + gid + 8 i that exist
    auto load_w = [&](Regs<FMT>& r, int u) {
#pragma unroll
        for (int t = 0; t < TM; ++t)
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const int i = t * 2 + hh;
                if constexpr (FMT == kDense) {
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        r.w[t][hh][q] = (i < rows8 && u * 64 + q * 32 + tig * 8 < K) ? ldg_stream(wp + i * row8 + q * 64) : make_uint4(0, 0, 0, 0);
                } else {
                    const char* q = wp + t * (FMT == kInt4 ? kW4Piece : kW8Piece);
                    r.w[t][hh][0] = ldg_stream(q + hh * 128);
                    if constexpr (FMT == kInt8) r.w[t][hh][1] = ldg_stream(q + hh * 128 + 4 * kChunk);
                    else if (hh == 0) r.sz[t] = *reinterpret_cast<const uint2*>(q + soff);
                }
            }
        wp += FMT == kDense ? 128 : FMT == kInt4 ? kW4Block : kW8Block;
    };
    float acc[TM][2][4];
#pragma unroll
    for (int t = 0; t < TM; ++t)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[t][e >> 2][e & 3] = 0.f;
    auto leave_first = [&] {
        float* first = slots[(threadIdx.x >> 5) * 2];  // (nothing but the lane's place is kept for this through the loop)
#pragma unroll
        for (int t = 0; t < TM; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                first[(tig * 2 + (e & 1)) * (kTile + 1) + t * 16 + (e >> 1) * 8 + gid] = acc[t][0][e] + acc[t][1][e];
                acc[t][0][e] = acc[t][1][e] = 0.f;
            }
    };
    Regs<FMT> r[2];
    if (!args.early) grid_dependency_wait();
    if (u0 < u1) load_w(r[0], u0);
    if (u0 + 1 < u1) load_w(r[1], u0 + 1);
    if (args.early) grid_dependency_wait();
    if (threadIdx.x == 0) grid_launch_dependents();
    if (u0 < u1) load_x<FMT>(r[0].x, xrow, live, K, u0, tig);
    if (u0 + 1 < u1) load_x<FMT>(r[1].x, xrow, live, K, u0 + 1, tig);
    for (int u = u0; u < u1; u += 2) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            if (u + b < u1) {
                if (HALVES && u + b == mid) leave_first();
                unit_mma<T, FMT>(acc, r[b]);
                if (u + b + 2 < u1) {
                    load_w(r[b], u + b + 2);
                    load_x<FMT>(r[b].x, xrow, live, K, u + b + 2, tig);
                }
            }
        }
    }
    if (HALVES && mid >= u1) leave_first();  // (a part of one unit or none)
#pragma unroll
    for (int t = 0; t < TM; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[t][e] = acc[t][0][e] + acc[t][1][e];
}

template <typename T, bool HALVES>
__global__ void __launch_bounds__(HALVES ? kThreads / 2 : kThreads, HALVES ? 4 : 2) rows_gemv_kernel(const __grid_constant__ Args args) {
    __shared__ float slots[kSlots][kMaxRows * (kTile + 1)];  // partial sums [row][channel], padded
    constexpr int threads = HALVES ? kThreads / 2 : kThreads;
    const int S = HALVES ? 1 : args.splits, wk = HALVES ? kWarps / 2 : args.wk, groups = (threads >> 5) / wk;  // `groups` channel tiles per CTA, wk warps each
    const int rank = blockIdx.x % S, cta = blockIdx.x / S;
    int pi = 0;
    while (pi + 1 < args.n && cta >= args.p[pi + 1].cta0) ++pi;
    const Problem& p = args.p[pi];
    const int warp = threadIdx.x >> 5, t = warp / wk, n0 = ((cta - p.cta0) * groups + t) * kTile;
    if (S > 1) cluster_arrive_relaxed();  // every CTA of the cluster has started before partial sums are pushed
    float sum[TM][4];
    const int units = n0 >= p.N ? 0 : p.fmt == kDense ? (p.K + 63) >> 6 : p.K >> 7;
    const int part = rank * wk + warp % wk, parts = S * wk;
    const int u0 = (int)((long long)units * part / parts), u1 = (int)((long long)units * (part + 1) / parts);
    // as many partial sums as eight warps would leave, and the same bits: with one chain of MMAs twice as long the sums were a little
    // further from the exact ones (4096 -> 16384 int4, one row: 0.37 % of the results not the correctly rounded ones, 0.26 % so).  In a kernel
    // of its own: the branch in the loop cost the others 2 %.
    constexpr int H = HALVES ? 1 : 0;
    const int mid = HALVES ? (int)((long long)units * (2 * part + 1) / (2 * parts)) : 0, nslots = parts << H;
    if (p.fmt == kDense) stream<T, kDense, HALVES>(sum, p, args, n0, u0, mid, u1, slots);
    else if (p.fmt == kInt4) stream<__half, kInt4, HALVES>(sum, p, args, n0, u0, mid, u1, slots);
    else stream<__half, kInt8, HALVES>(sum, p, args, n0, u0, mid, u1, slots);

    // rank 0 of the cluster receives every partial sum and adds them in fixed order
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    float* mine = slots[t * nslots + (part << H) + H];
    const uint32_t dst = S > 1 ? mapa_shared(smem_u32(mine), 0) : 0;
    if (S > 1) cluster_wait();
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int o = (tig * 2 + (e & 1)) * (kTile + 1) + i * 16 + (e >> 1) * 8 + gid;
            if (S > 1) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + (uint32_t)o * 4), "f"(sum[i][e]) : "memory");
            else mine[o] = sum[i][e];
        }
    if (S > 1) {
        cluster_arrive_release();
        cluster_wait();
        if (rank != 0) return;
    } else {
        __syncthreads();
    }
    const int channels = groups * kTile, nbase = (cta - p.cta0) * channels;
    for (int i = threadIdx.x; i < channels * args.M; i += threads) {
        const int c = i % channels, m = i / channels, n = nbase + c;
        if (n >= p.N) continue;
        const int o = m * (kTile + 1) + c % kTile, s0 = c / kTile * nslots;
        float v = 0.f;
        for (int r = 0; r < nslots; ++r) v += slots[s0 + r][o];
        if (p.fmt == kInt8) v *= to_f<T>(reinterpret_cast<const T*>(p.scale)[n]);
        v = round_to<T>(v);
        const size_t oo = (size_t)m * p.N + n;
        switch (p.epi) {
            case RWKV7_EPI_RELU2: v = fmaxf(v, 0.f); v *= v; break;
            case RWKV7_EPI_ADD: v += to_f<T>(reinterpret_cast<const T*>(p.residual)[oo]); break;
            case RWKV7_EPI_TANH: v = tanhf(v); break;
            case RWKV7_EPI_SIGMOID: v = sigmoidf_(v); break;
            default: break;
        }
        reinterpret_cast<T*>(p.out)[oo] = from_f<T>(v);
    }
}
}  // namespace rg
}  // namespace rwkv7

using namespace rwkv7;

extern "C" int rwkv7_rows_gemv(int n_problems, const void* const* x, const void* const* W, const void* const* scale,
                               const void* const* residual, void* const* out, const int* K, const int* N, const int* fmt,
                               const int* epilogue, int M, int dtype, int static_weights, void* stream) {
    using namespace rg;
    RWKV7_REQUIRE(n_problems >= 1 && n_problems <= kMaxProblems, RWKV7_ERR_INVALID, "rows_gemv: 1..%d problems", kMaxProblems);
    RWKV7_REQUIRE(M >= 1 && M <= kMaxRows, RWKV7_ERR_UNSUPPORTED, "rows_gemv: M must be in 1..%d (got %d)", kMaxRows, M);
    RWKV7_REQUIRE(dtype == RWKV7_F16 || dtype == RWKV7_BF16, RWKV7_ERR_UNSUPPORTED, "rows_gemv: fp16 / bf16 only");
    RWKV7_REQUIRE(x && W && out && K && N && fmt && epilogue, RWKV7_ERR_INVALID, "rows_gemv: null argument array");
    Args a{};
    a.n = n_problems;
    a.M = M;
    a.early = static_weights != 0;
    bool fresh = false;
    int max_units = 1;
    for (int i = 0; i < n_problems; ++i) {
        Problem& p = a.p[i];
        RWKV7_REQUIRE(x[i] && W[i] && out[i], RWKV7_ERR_INVALID, "rows_gemv: null pointer in problem %d", i);
        RWKV7_REQUIRE(fmt[i] >= kDense && fmt[i] <= kInt8, RWKV7_ERR_INVALID, "rows_gemv: bad weight format %d", fmt[i]);
        RWKV7_REQUIRE(N[i] > 0 && K[i] > 0 && K[i] % (fmt[i] == kDense ? 8 : 128) == 0, RWKV7_ERR_UNSUPPORTED,
                      "rows_gemv: K must be a positive multiple of %d (problem %d: K=%d N=%d)", fmt[i] == kDense ? 8 : 128, i, K[i], N[i]);
        RWKV7_REQUIRE(fmt[i] == kDense || dtype == RWKV7_F16, RWKV7_ERR_UNSUPPORTED, "rows_gemv: quantised weights take fp16 activations");
        RWKV7_REQUIRE(epilogue[i] >= 0 && epilogue[i] <= RWKV7_EPI_SIGMOID, RWKV7_ERR_INVALID, "rows_gemv: bad epilogue code %d", epilogue[i]);
        p.x = x[i]; p.W = W[i]; p.out = out[i]; p.K = K[i]; p.N = N[i]; p.fmt = fmt[i]; p.epi = epilogue[i];
        p.scale = scale ? scale[i] : nullptr;
        p.residual = residual ? residual[i] : nullptr;
        RWKV7_REQUIRE(fmt[i] != kInt8 || p.scale, RWKV7_ERR_INVALID, "rows_gemv: int8 weights need their channel scales");
        RWKV7_REQUIRE(epilogue[i] != RWKV7_EPI_ADD || p.residual, RWKV7_ERR_INVALID, "rows_gemv: the add epilogue needs a residual");
        RWKV7_REQUIRE(aligned(x[i], 16) && aligned(W[i], 16), RWKV7_ERR_ALIGN, "rows_gemv: x and W must be 16-byte aligned");
        if (fmt[i] != kDense) fresh |= take_tiled_fresh(W[i]);
        const int units = (K[i] + (fmt[i] == kDense ? 63 : 127)) / (fmt[i] == kDense ? 64 : 128);
        max_units = units > max_units ? units : max_units;
    }
    a.wk = max_units >= 8 ? 8 : max_units >= 4 ? 4 : max_units >= 2 ? 2 : 1;
    // Two CTAs of eight warps fit an SM, or four of four, which take twice as long over their tile: those where the eight-warp CTAs
    // would start a second wave that is nearly empty.  us, 8 -> 4 warps, 1 / 8 rows: int4 2048 -> 9600 7.4 / 8.6 -> 6.9 / 8.3, 4096 -> 16384 14.7 / 17.2 ->
    // 12.9 / 14.9, 4096 -> 18944 15.2 / 17.6 -> 13.3 / 15.2, 4096 -> 32768 26.5 / 30.2 -> 23.8 / 28.1; int8 2560 -> 10240 11.0 -> 9.1; dense 2560 -> 10240 14.1 /
    // 15.0 -> 12.4 / 13.0, 2560 -> 14336 15.4 / 16.1 -> 13.7 / 14.5.  With as many waves either way but one: dense 4096 -> 20480 33.8 / 35.1 -> 38.5 / 39.9.
    const auto deal = [&](int warps) {
        const int per = warps / a.wk * kTile;
        int ctas = 0;
        for (int i = 0; i < n_problems; ++i) {
            a.p[i].cta0 = ctas;
            ctas += (N[i] + per - 1) / per;
        }
        return ctas;
    };
    int warps = kWarps, ctas = deal(warps);
    bool halves = false;  // a warp has the K of two of eight, and leaves the partial sums of either
    if (a.wk == kWarps && ctas > 2 * kSMs && 2 * ((ctas + 4 * kSMs - 1) / (4 * kSMs)) <= (ctas + 2 * kSMs - 1) / (2 * kSMs)) {
        warps = a.wk = kWarps / 2;
        halves = true;
        ctas = deal(warps);
    }
    // Up to one CTA an SM and at least two units a warp: pairs of CTAs halve K.  1 row, fp16 / int4 / int8, one CTA against two:
    // 2560 x 2560 5.7 / 4.0 / 4.3 -> 4.6 / 3.9 / 4.2 us, 10240 -> 2560 19.9 / 13.1 / 13.4 -> 13.1 / 8.9 / 9.7, 16384 -> 4096
    // 34.7 / 20.6 / 21.6 -> 25.0 / 14.2 / 16.0; beyond one CTA an SM pairs only add their exchange (4096 -> 16384 int4
    // 15.0 -> 19.9), and so do fours (16384 -> 4096 int4 18.5).
    a.splits = ctas <= kSMs && max_units >= 16 ? 2 : 1;
    auto kern = dtype == RWKV7_F16 ? (halves ? rows_gemv_kernel<__half, true> : rows_gemv_kernel<__half, false>)
                                   : (halves ? rows_gemv_kernel<__nv_bfloat16, true> : rows_gemv_kernel<__nv_bfloat16, false>);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas * a.splits);
    cfg.blockDim = dim3(warps * 32);
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = a.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (!fresh && programmatic_launch_ok(cfg.stream)) ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a);
    RWKV7_REQUIRE(e == cudaSuccess, RWKV7_ERR_CUDA, "rows_gemv launch: %s", cudaGetErrorString(e));
    return RWKV7_OK;
}
