// WKV-7 sequential scan over T tokens: one CTA per (sequence, head), the 64x64 fp32 state lives in registers for the
// whole sequence as a tile of R rows x C columns per thread, token vectors are staged through shared memory in blocks
// of kTS tokens with cp.async double buffering and converted to fp32 once per block.  HBM traffic is the algorithmic
// minimum (each token vector read once, y written once, state read/written once).
//
// Bound: 5 * 64 * 64 multiply-adds per token and head in fp32 (1 S.kk, 1 decay, 2 rank-one terms, 1 S.r), issued as
// packed pairs; 160 cycles of an SM's FMA pipe per token and head, measured 308 (64 sequences x 512 tokens x 64 heads,
// fp16, output prepared: 2.21 ms, 6.04 ms with one row half per thread, unpacked, and the conversion in the chain).  Few
// CTAs are bound by the latency of a token's chain instead: 120 CTAs x 777 tokens 242 us (772 us).  Operands come from
// shared memory as 16-byte reads that the lanes of a row group share.  Counted in the source, not profiled: the 2 x 32 tile
// makes 40 of them a thread and token, and at four cycles a warp the two warps of a head hold the shared-memory pipe 320
// cycles, which is about what a token takes at full grids.
#include "common.cuh"

namespace rwkv7 {

constexpr int kSN = 64;
constexpr int kTS = 8;     // tokens per shared-memory block
constexpr int kSMs = 148;  // B200

struct ScanArgs {
    const void *r, *w, *k, *v, *kk, *a;
    const void* state_in;  // fp32, or fp16 when state_f16
    void* state_out;
    void* y;
    const void *g, *r_k, *gn_w, *gn_b;
    float eps;
    int T, H;
    int w_mode;  // 0: decay in T, 1: decay fp32, 2: raw w in T
    // the reference's FP16-state sequence lane (rwkv7_hf/native_wkv_fp16.py:335-452)
    int state_f16;       // the state is stored in fp16 (loaded to fp32 registers, rounded back once at the end)
    int ab_mode;         // `kk` holds -kk and `a` holds kk*a (the lane's neg_kk / kka operands)
    const void* w0;      // w_mode 2: per-channel bias [H*64] added to raw w before the decay (may be NULL)
    const int* elapsed;  // w_mode 2: per-sequence step counters [B]; token t uses the dither phase elapsed + channel + t
    int params_vec;      // r_k, gn_w and gn_b all start on 16 bytes; else (views into a flat buffer) they are read by element
};

// zero-mean pseudo-random offset of the reference's FP16-state kernels (rwkv7_hf/native_wkv_fp16.py:118-121)
__device__ __forceinline__ float scan_rotator1(int x) {
    const uint32_t bits = 2654435769u * static_cast<uint32_t>(x);
    return 4.547473508864641e-13f * static_cast<float>(static_cast<int32_t>(bits));
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// ---- packed pairs of fp32 (one instruction, two lanes of arithmetic, each rounded on its own)
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Raw staging buffer for one block of tokens: six vectors (r,k,v,kk,a in T; w in T or fp32).
template <typename T>
struct alignas(16) RawStage {
    T r[kTS][kSN], k[kTS][kSN], v[kTS][kSN], kk[kTS][kSN], a[kTS][kSN];
    float w[kTS][kSN];  // sized for the fp32 case; the T case uses a prefix of it
};

// fp32 operands of one block of tokens, as the token loop reads them (nb = -kk a)
struct alignas(16) Operands {
    float kk[kTS][kSN], w[kTS][kSN], k[kTS][kSN], nb[kTS][kSN], r[kTS][kSN], v[kTS][kSN];
    float y[kTS][kSN];
};

// Sum R row values over the G lanes that share a row group, halving the rows a lane keeps while there is more than one
// (R - 1 shuffles instead of R log2 G).  On return the lane owns row `row` of the group's R; `first` marks the one lane
// that owns it when there are more lanes than rows.
template <int R, int G>
__device__ __forceinline__ float scatter_sum(float (&v)[R], int cg, int& row, bool& first) {
    row = 0;
    first = true;
    if constexpr (G == 1) {
        return v[0];
    } else if constexpr (R == 1) {
        float t = v[0];
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        first = (cg & (G - 1)) == 0;
        return t;
    } else {
        constexpr int HALF = G / 2, RH = R / 2;
        const bool up = (cg & HALF) != 0;
        float keep[RH];
#pragma unroll
        for (int i = 0; i < RH; ++i) {
            const float mine = up ? v[RH + i] : v[i], send = up ? v[i] : v[RH + i];
            keep[i] = mine + __shfl_xor_sync(0xffffffffu, send, HALF);
        }
        int sub;
        const float t = scatter_sum<RH, HALF>(keep, cg, sub, first);
        row = (up ? RH : 0) + sub;
        return t;
    }
}

// One block of `nt` tokens on the register tile S (R rows x C columns per thread; pairs along the columns).
// Column j*4G + 4 cg + q belongs to lane cg of the row group: a 16-byte read by the G lanes covers 16 G contiguous bytes.
template <int R, int C>
__device__ __forceinline__ void scan_block(f2 (&S)[R][C / 2], Operands& op, int nt, int row0, int cg) {
    constexpr int G = kSN / C;
    auto load = [&](f2 (&x)[C / 2], const float* src) {
#pragma unroll
        for (int j = 0; j < C / 4; ++j) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(src + j * 4 * G + cg * 4);
            x[2 * j] = t.x;
            x[2 * j + 1] = t.y;
        }
    };
    auto dot = [&](float (&out)[R], const f2 (&x)[C / 2]) {  // four partial sums per row
#pragma unroll
        for (int i = 0; i < R; ++i) {
            f2 acc0 = mul2(S[i][0], x[0]), acc1 = mul2(S[i][1], x[1]);
#pragma unroll
            for (int j = 2; j < C / 2; j += 2) {
                acc0 = fma2(S[i][j], x[j], acc0);
                acc1 = fma2(S[i][j + 1], x[j + 1], acc1);
            }
            float a, b, c, d;
            unpack2(acc0, a, b);
            unpack2(acc1, c, d);
            out[i] = (a + b) + (c + d);
        }
    };
    float y[R];  // the output of token tt - 1, summed over the lanes while token tt's sum is on its way too
    f2 x[C / 2];
    load(x, op.kk[0]);
#pragma unroll 1
    for (int tt = 0; tt < nt; ++tt) {
        float sa[R];
        dot(sa, x);
        load(x, op.w[tt]);
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < C / 2; ++j) S[i][j] = mul2(S[i][j], x[j]);
        load(x, op.k[tt]);
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < R; ++i) sa[i] += __shfl_xor_sync(0xffffffffu, sa[i], o);
        if (tt > 0) {
            int row;
            bool first;
            const float ysum = scatter_sum<R, G>(y, cg, row, first);
            if (first) op.y[tt - 1][row0 + row] = ysum;
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float vi = op.v[tt][row0 + i];
            const f2 v2 = pack2(vi, vi);
#pragma unroll
            for (int j = 0; j < C / 2; ++j) S[i][j] = fma2(v2, x[j], S[i][j]);
        }
        load(x, op.nb[tt]);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const f2 s2 = pack2(sa[i], sa[i]);
#pragma unroll
            for (int j = 0; j < C / 2; ++j) S[i][j] = fma2(s2, x[j], S[i][j]);
        }
        load(x, op.r[tt]);
        dot(y, x);
        if (tt + 1 < nt) load(x, op.kk[tt + 1]);
    }
    {
        int row;
        bool first;
        const float ysum = scatter_sum<R, G>(y, cg, row, first);
        if (first) op.y[nt - 1][row0 + row] = ysum;
    }
}

// A CTA owns one (sequence, head).  (64 / R) * (64 / C) threads run the token loop; 64 threads load and convert a block of
// tokens, 64 write one out.  SPEC: these are four further warps that prepare block s+1 and write block s-1 while block s
// runs (for grids that leave an SM with one or two CTAs, where both would otherwise sit in the serial chain); without
// it the 64 threads of the token loop do all three in turn and the other CTAs of the SM fill the gaps.
template <typename T, bool PREP, int R, int C, bool SPEC>
__global__ void __launch_bounds__(kSN / R * (kSN / C) + (SPEC ? 128 : 0)) wkv7_scan_kernel(const ScanArgs p) {
    constexpr int G = kSN / C;
    constexpr int NT = kSN / R * G;  // threads of the token loop
    static_assert(SPEC || NT == 64, "the helpers are 64 threads");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RawStage<T>* raw = reinterpret_cast<RawStage<T>*>(smem_raw);  // [2]
    Operands* ops = reinterpret_cast<Operands*>(smem_raw + 2 * sizeof(RawStage<T>));  // [SPEC ? 3 : 1]

    const int bh = blockIdx.x;
    const int b = bh / p.H, h = bh % p.H;
    const int tid = threadIdx.x;
    const int T_ = p.T;
    const size_t tok_stride = (size_t)p.H * kSN;              // elements between consecutive tokens
    const size_t base = ((size_t)b * T_ * p.H + h) * kSN;     // element offset of token 0
    const int phase0 = p.elapsed ? p.elapsed[b] + h * kSN : 0;
    const int nstages = (T_ + kTS - 1) / kTS;
    const int ht = SPEC ? (tid - NT) & 63 : tid;  // index among the 64 loading or the 64 writing threads

    // ---- in and out--------------------------------------------------------------------------------------------------
    auto loader_sync = [] { asm volatile("barrier.sync 1, 64;" ::: "memory"); };
    auto issue_stage = [&](int s) {
        constexpr int CH = kSN * (int)sizeof(T) / 16;  // 16-byte chunks per token vector
        RawStage<T>& rs = raw[s & 1];
        const int t0 = s * kTS, nt = min(kTS, T_ - t0);
        const T* srcs[5] = {reinterpret_cast<const T*>(p.r), reinterpret_cast<const T*>(p.k), reinterpret_cast<const T*>(p.v),
                            reinterpret_cast<const T*>(p.kk), reinterpret_cast<const T*>(p.a)};
        T(*dsts[5])[kSN] = {rs.r, rs.k, rs.v, rs.kk, rs.a};
#pragma unroll
        for (int q = 0; q < 5; ++q)
            for (int idx = ht; idx < nt * CH; idx += 64) {
                const int tt = idx / CH, ch = idx % CH;
                cp_async16(reinterpret_cast<char*>(dsts[q][tt]) + ch * 16,
                           reinterpret_cast<const char*>(srcs[q] + base + (size_t)(t0 + tt) * tok_stride) + ch * 16);
            }
        const int wsz = (p.w_mode == 1) ? 4 : (int)sizeof(T), chw = kSN * wsz / 16;
        for (int idx = ht; idx < nt * chw; idx += 64) {
            const int tt = idx / chw, ch = idx % chw;
            cp_async16(reinterpret_cast<char*>(rs.w[tt]) + ch * 16,
                       reinterpret_cast<const char*>(p.w) + (base + (size_t)(t0 + tt) * tok_stride) * wsz + ch * 16);
        }
        cp_async_commit();
    };

    // thread = two channels x half of the block's tokens
    auto convert = [&](int s, Operands& op) {
        RawStage<T>& rs = raw[s & 1];
        const int t0 = s * kTS, nt = min(kTS, T_ - t0);
        const int c = (ht & 31) * 2;
        auto two = [](const T* q) {
            if constexpr (sizeof(T) == 4) return *reinterpret_cast<const float2*>(q);
            else return make_float2(to_f<T>(q[0]), to_f<T>(q[1]));
        };
#pragma unroll
        for (int u = 0; u < kTS / 2; ++u) {
            const int tt = (ht >> 5) * (kTS / 2) + u;
            if (tt >= nt) continue;
            float2 w;
            if (p.w_mode == 1) w = *reinterpret_cast<const float2*>(&rs.w[tt][c]);
            else {
                w = two(reinterpret_cast<const T*>(rs.w[tt]) + c);
                if (p.w_mode == 2) {
                    float e[2] = {w.x, w.y};
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        if (p.w0) e[i] += to_f<T>(reinterpret_cast<const T*>(p.w0)[h * kSN + c + i]);
                        e[i] = decay_from_raw(e[i]);
                        // (decay - 1 + rotator) rounded to fp16, as the reference's kernel forms its decay operand
                        if (p.elapsed) e[i] = 1.0f + __half2float(__float2half_rn(e[i] - 1.0f + scan_rotator1(phase0 + c + i + t0 + tt)));
                    }
                    w = make_float2(e[0], e[1]);
                }
            }
            const float2 kk = two(&rs.kk[tt][c]), a = two(&rs.a[tt][c]);
            *reinterpret_cast<float2*>(&op.w[tt][c]) = w;
            *reinterpret_cast<float2*>(&op.kk[tt][c]) = p.ab_mode ? make_float2(-kk.x, -kk.y) : kk;
            *reinterpret_cast<float2*>(&op.nb[tt][c]) = p.ab_mode ? make_float2(-a.x, -a.y) : make_float2(-(kk.x * a.x), -(kk.y * a.y));
            *reinterpret_cast<float2*>(&op.r[tt][c]) = two(&rs.r[tt][c]);
            *reinterpret_cast<float2*>(&op.k[tt][c]) = two(&rs.k[tt][c]);
            *reinterpret_cast<float2*>(&op.v[tt][c]) = two(&rs.v[tt][c]);
        }
    };

    // eight lanes per token, eight channels per lane
    auto flush = [&](int s, Operands& op) {
        const int t0 = s * kTS, nt = min(kTS, T_ - t0);
        const int l8 = ht & 7, c = l8 * 8;
        auto load_param = [&](const void* param, float (&o)[8]) {
            const T* q = reinterpret_cast<const T*>(param) + h * kSN + c;
            if (p.params_vec) {
                load8(q, o);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = to_f<T>(q[i]);
            }
        };
        for (int tt = ht >> 3; tt < kTS; tt += 8) {
            const bool live = tt < nt;  // the shuffles below run in all lanes
            const size_t o = base + (size_t)(t0 + (live ? tt : 0)) * tok_stride + c;
            float y[8];
            load8<float>(&op.y[live ? tt : 0][c], y);
            if constexpr (PREP) {
                float r[8], k[8], v[8], rk[8], gw[8], gb[8], g[8];
                load8<float>(&op.r[live ? tt : 0][c], r);
                load8<float>(&op.k[live ? tt : 0][c], k);
                load8<float>(&op.v[live ? tt : 0][c], v);
                load8(reinterpret_cast<const T*>(p.g) + o, g);
                load_param(p.r_k, rk);
                load_param(p.gn_w, gw);
                load_param(p.gn_b, gb);
                float sum = 0.f, corr = 0.f, var = 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) { sum += y[i]; corr += r[i] * k[i] * rk[i]; }
                const float mean = group_sum<8>(sum) * (1.0f / kSN);
                corr = group_sum<8>(corr);
#pragma unroll
                for (int i = 0; i < 8; ++i) { y[i] -= mean; var += y[i] * y[i]; }
                const float rstd = rsqrtf(group_sum<8>(var) * (1.0f / kSN) + p.eps);
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] = (y[i] * rstd * gw[i] + gb[i] + corr * v[i]) * g[i];
            }
            if (live) store8(reinterpret_cast<T*>(p.y) + o, y);
        }
    };

    // ---- the state tile ----------------------------------------------------------------------------------------------
    const int cg = tid % G, row0 = tid / G * R;
    const size_t soff = ((size_t)bh * kSN + row0) * kSN + cg * 4;
    f2 S[R][C / 2];
    if (!SPEC || tid < NT) {
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < C / 4; ++j) {
                const size_t o = soff + (size_t)i * kSN + j * 4 * G;
                float x[4];
                if (p.state_f16) load4(reinterpret_cast<const __half*>(p.state_in) + o, x);
                else load4(reinterpret_cast<const float*>(p.state_in) + o, x);
                S[i][2 * j] = pack2(x[0], x[1]);
                S[i][2 * j + 1] = pack2(x[2], x[3]);
            }
    }
    auto run_block = [&](int s, Operands& op) { scan_block<R, C>(S, op, min(kTS, T_ - s * kTS), row0, cg); };

    if constexpr (SPEC) {
        const bool loader = tid >= NT && tid < NT + 64, writer = tid >= NT + 64;
        if (loader) {
            issue_stage(0);
            if (nstages > 1) issue_stage(1);
        }
        for (int s = -1; s <= nstages; ++s) {  // block s+1 in, block s through the recurrence, block s-1 out
            if (loader) {
                if (s + 1 < nstages) {
                    if (s + 2 < nstages) cp_async_wait<1>(); else cp_async_wait<0>();
                    loader_sync();  // raw block s+1 visible to both loader warps
                    convert(s + 1, ops[(s + 1) % 3]);
                    loader_sync();  // ... and read by both
                    if (s + 3 < nstages) issue_stage(s + 3);
                }
            } else if (writer) {
                if (s >= 1) flush(s - 1, ops[(s - 1) % 3]);
            } else if (s >= 0 && s < nstages) {
                run_block(s, ops[s % 3]);
            }
            __syncthreads();
        }
    } else {
        issue_stage(0);
        for (int s = 0; s < nstages; ++s) {
            if (s + 1 < nstages) {
                issue_stage(s + 1);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncthreads();  // raw block visible; the previous block's flush has read the operands
            convert(s, ops[0]);
            __syncthreads();
            run_block(s, ops[0]);
            __syncthreads();
            flush(s, ops[0]);
        }
    }

    if (!SPEC || tid < NT) {
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < C / 4; ++j) {
                const size_t o = soff + (size_t)i * kSN + j * 4 * G;
                float x[4];
                unpack2(S[i][2 * j], x[0], x[1]);
                unpack2(S[i][2 * j + 1], x[2], x[3]);
                if (p.state_f16) store4(reinterpret_cast<__half*>(p.state_out) + o, x);
                else store4(reinterpret_cast<float*>(p.state_out) + o, x);
            }
    }
}

template <typename T, bool PREP, int R, int C, bool SPEC>
static int launch_scan(const ScanArgs& p, int B, cudaStream_t st) {
    constexpr size_t smem = 2 * sizeof(RawStage<T>) + (SPEC ? 3 : 1) * sizeof(Operands);
    auto kern = wkv7_scan_kernel<T, PREP, R, C, SPEC>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    RWKV7_REQUIRE(e == cudaSuccess, RWKV7_ERR_CUDA, "wkv7_scan: %s", cudaGetErrorString(e));
    kern<<<B * p.H, kSN / R * (kSN / C) + (SPEC ? 128 : 0), smem, st>>>(p);
    return check_launch("wkv7_scan_kernel");
}

template <typename T, bool PREP>
static int dispatch_scan(const ScanArgs& p, int B, cudaStream_t st) {
    // Chosen by how many CTAs an SM gets.  Up to one: the serial chain of a token is all there is, so the rows are spread
    // over four warps (160 multiply-adds a thread and token, 80 packed, where the 2 x 32 tile has 320) and loads /
    // conversion / output run on warps of their own: 242 us for 120 CTAs x 777 tokens against 391 without.  Up to two: the
    // tile with the fewer operand reads, still with the extra warps (335 us against 401 for 240 CTAs x 777).  More: the CTAs
    // of an SM hide each other's loads and the extra warps only take registers (2211 us against 3159 for 4096 CTAs x 512).
    // The three forms in this order, us for 512 tokens, fp16, output prepared: 148 CTAs 158 / 199 / 247, 149 235 / 215 / 250,
    // 296 235 / 215 / 263, 297 379 / 409 / 370, 448 464 / 426 / 377, 600 602 / 635 / 512, 896 824 / 846 / 697, 2048 1606 / 1486 / 1164.
    const int ctas = B * p.H;
    if (ctas <= kSMs) return launch_scan<T, PREP, 1, 32, true>(p, B, st);
    if (ctas <= 2 * kSMs) return launch_scan<T, PREP, 4, 16, true>(p, B, st);
    return launch_scan<T, PREP, 2, 32, false>(p, B, st);
}

}  // namespace rwkv7

using namespace rwkv7;

static int scan_impl(const void* r, const void* w, const void* k, const void* v, const void* kk, const void* a,
                     const void* state_in, void* state_out, void* y, const void* g, const void* r_k, const void* gn_w,
                     const void* gn_b, float eps, int B, int T, int H, int N, int dtype, int w_mode, int state_f16,
                     int ab_mode, const void* w0, const int* elapsed, void* stream) {
    RWKV7_REQUIRE(N == kSN, RWKV7_ERR_UNSUPPORTED, "wkv7_scan: head size must be 64, got %d", N);
    RWKV7_REQUIRE(B > 0 && H > 0 && T >= 0, RWKV7_ERR_INVALID, "wkv7_scan: bad sizes B=%d T=%d H=%d", B, T, H);
    RWKV7_REQUIRE(w_mode >= 0 && w_mode <= 2, RWKV7_ERR_INVALID, "wkv7_scan: w_mode must be 0, 1 or 2");
    RWKV7_REQUIRE(state_in && state_out, RWKV7_ERR_INVALID, "wkv7_scan: null state pointer");
    const bool prep = g || r_k || gn_w || gn_b;
    if (prep) RWKV7_REQUIRE(g && r_k && gn_w && gn_b, RWKV7_ERR_INVALID, "wkv7_scan: g, r_k, gn_w, gn_b go together");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (T == 0) {  // empty sequence: the state passes through
        if (state_out != state_in) {
            cudaError_t e = cudaMemcpyAsync(state_out, state_in, (size_t)B * H * N * N * (state_f16 ? 2 : 4),
                                            cudaMemcpyDeviceToDevice, st);
            RWKV7_REQUIRE(e == cudaSuccess, RWKV7_ERR_CUDA, "wkv7_scan: %s", cudaGetErrorString(e));
        }
        return RWKV7_OK;
    }
    RWKV7_REQUIRE(r && w && k && v && kk && a && y, RWKV7_ERR_INVALID, "wkv7_scan: null tensor pointer");
    const void* ptrs[] = {r, w, k, v, kk, a, state_in, state_out, y, g};
    for (const void* q : ptrs) RWKV7_REQUIRE(aligned(q, 16), RWKV7_ERR_ALIGN, "wkv7_scan: pointers must be 16-byte aligned");
    RWKV7_REQUIRE((!w0 && !elapsed) || w_mode == 2, RWKV7_ERR_INVALID, "wkv7_scan: w0 / elapsed apply to raw w (w_mode 2)");
    ScanArgs p{r, w, k, v, kk, a, state_in, state_out, y, g, r_k, gn_w, gn_b, eps, T, H, w_mode, state_f16 != 0, ab_mode != 0, w0, elapsed,
               aligned(r_k, 16) && aligned(gn_w, 16) && aligned(gn_b, 16)};
    RWKV7_DISPATCH_DTYPE(dtype, TT, {
        return prep ? dispatch_scan<TT, true>(p, B, st) : dispatch_scan<TT, false>(p, B, st);
    });
    return RWKV7_OK;
}

extern "C" int rwkv7_wkv7_scan(const void* r, const void* w, const void* k, const void* v, const void* kk,
                               const void* a, const float* state_in, float* state_out, void* y, const void* g,
                               const void* r_k, const void* gn_w, const void* gn_b, float eps, int B, int T, int H,
                               int N, int dtype, int w_mode, void* stream) {
    return scan_impl(r, w, k, v, kk, a, state_in, state_out, y, g, r_k, gn_w, gn_b, eps, B, T, H, N, dtype, w_mode, 0, 0,
                     nullptr, nullptr, stream);
}

extern "C" int rwkv7_wkv7_scan_f16state(const void* r, const void* w, const void* k, const void* v, const void* kk,
                                        const void* a, const void* state_in, void* state_out, void* y, const void* g,
                                        const void* r_k, const void* gn_w, const void* gn_b, float eps, int B, int T,
                                        int H, int N, int dtype, int w_mode, int ab_mode, const void* w0,
                                        const int* elapsed, void* stream) {
    return scan_impl(r, w, k, v, kk, a, state_in, state_out, y, g, r_k, gn_w, gn_b, eps, B, T, H, N, dtype, w_mode, 1,
                     ab_mode, w0, elapsed, stream);
}
