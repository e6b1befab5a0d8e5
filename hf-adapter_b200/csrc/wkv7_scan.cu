// WKV-7 sequential scan over T tokens: one CTA per (sequence, head), the 64x64 fp32 state lives in registers for the
// whole sequence as a tile of R rows x C columns per thread, token vectors are staged through shared memory in blocks
// of kTS tokens with cp.async double buffering and converted to fp32 once per block.  HBM traffic is the algorithmic
// minimum (each token vector read once, y written once, state read/written once).
//
// Bound: 5 * 64 * 64 multiply-adds per token and head in fp32 (1 S.kk, 1 decay, 2 rank-one terms, 1 S.r), issued as
// packed pairs; 160 cycles of an SM's FMA pipe per token and head, measured 308 (64 sequences x 512 tokens x 64 heads,
// fp16, output prepared: 2.21 ms, 6.04 ms with one row half per thread, unpacked, and the conversion in the chain).  Few
// CTAs are bound by the chain of a token instead and have a kernel of their own.  Operands come from
// shared memory as 16-byte reads that the lanes of a row group share: 40 a thread and token with the 2 x 32 tile.
#include "common.cuh"

namespace rwkv7 {

constexpr int kSN = 64;
constexpr int kTS = 8;     // tokens per shared-memory block

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

// Sum R row values over the R lanes that share a row group, halving the rows a lane keeps (R - 1 shuffles instead of
// R log2 R).  On return the lane owns row `row` of the group's.
template <int R>
__device__ __forceinline__ float scatter_sum(float (&v)[R], int cg, int& row) {
    row = 0;
    if constexpr (R == 1) {
        return v[0];
    } else {
        constexpr int RH = R / 2;
        const bool up = (cg & RH) != 0;
        float keep[RH];
#pragma unroll
        for (int i = 0; i < RH; ++i) {
            const float mine = up ? v[RH + i] : v[i], send = up ? v[i] : v[RH + i];
            keep[i] = mine + __shfl_xor_sync(0xffffffffu, send, RH);
        }
        int sub;
        const float t = scatter_sum<RH>(keep, cg, sub);
        row = (up ? RH : 0) + sub;
        return t;
    }
}

// One block of `nt` tokens on the register tile S (R rows x C columns per thread; pairs along the columns).
// Column j*4G + 4 cg + q belongs to lane cg of the row group: a 16-byte read by the G lanes covers 16 G contiguous bytes.
template <int R, int C>
__device__ __forceinline__ void scan_block(f2 (&S)[R][C / 2], Operands& op, int nt, int row0, int cg) {
    constexpr int G = kSN / C;
    static_assert(R == G, "as many rows as lanes: each ends up with one row's sum");
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
            const float ysum = scatter_sum<R>(y, cg, row);
            op.y[tt - 1][row0 + row] = ysum;
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
        const float ysum = scatter_sum<R>(y, cg, row);
        op.y[nt - 1][row0 + row] = ysum;
    }
}

// ---- grids that leave an SM with one or two CTAs: the serial chain of a token is all there is -----------------------------
// Operands of one token in registers: the columns of a lane (4 cg .. + 3 and 32 + 4 cg .. + 3) and the values of its four rows.
constexpr int kFewRows = 4, kFewLanes = 8;  // rows a thread has eight columns of, lanes that share them
struct TokenRegs {
    f2 kk[4], w[4], k[4], nb[4], r[4];
    float v[kFewRows];
};
__device__ __forceinline__ void load_token(TokenRegs& o, const Operands& op, int t, int row0, int cg) {
    auto load = [&](f2 (&x)[4], const float* src) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(src + j * 32 + cg * 4);
            x[2 * j] = q.x;
            x[2 * j + 1] = q.y;
        }
    };
    load(o.kk, op.kk[t]);
    load(o.w, op.w[t]);
    load(o.k, op.k[t]);
    load(o.nb, op.nb[t]);
    load(o.r, op.r[t]);
    load4<float>(&op.v[t][row0], o.v);
}

template <typename T> struct alignas(2 * sizeof(T)) Pair { T x, y; };
template <typename T> __device__ __forceinline__ float2 to_f2(const Pair<T>& q) { return make_float2(to_f<T>(q.x), to_f<T>(q.y)); }

// A CTA owns one (sequence, head).  Warps 0..3 run the recurrence: 8 lanes share four rows, a lane has 8 columns of each.  Warps
// 4, 5 read a block of tokens ahead (in registers while the block before it runs) and convert it, warps 6, 7 write out the block that
// is done.  In the token loop everything that does not wait for S.kk of this token sits in its shadow: the operands of the next
// token, the decay and the v k^T term, the output sums of the token before.  With three BLOCKS of operands in shared memory (one ahead,
// one behind the one that runs) a block's first token has no such shadow; with five (two and two) it has, at two more barriers a call.
// What bounds it: the instructions of four warps, one a scheduler (about 190 a token and warp at 2.2 cycles; two tokens a step, with
// half the chain and as many instructions, took as long), and the shared-memory pipe, which hands a warp its 16-byte operand pieces
// at four cycles each whoever shares them: two rows a thread on twice the warps are 30 % slower.  A partial sum is one chain of
// four packed steps and one add (two chains and three adds: 5 % slower).  120 CTAs x 512 tokens 127.3 -> 116.0 us with three blocks (227 ns a
// token), with five 2 us less.
template <typename T, bool PREP, int CTAS, int BLOCKS>
__global__ void __launch_bounds__(256, CTAS) wkv7_scan_few_kernel(const ScanArgs p) {
    constexpr int R = kFewRows, G = kFewLanes, NT = kSN / R * G, LAG = BLOCKS / 2;
    constexpr bool ACROSS = BLOCKS == 5;  // a token's shadow reaches across the blocks
    static_assert(BLOCKS == 3 || (BLOCKS == 5 && CTAS == 1), "LAG blocks on either side; five with one CTA an SM");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Operands* ops = reinterpret_cast<Operands*>(smem_raw);  // [BLOCKS]
    const int bh = blockIdx.x, b = bh / p.H, h = bh % p.H;
    const int tid = threadIdx.x;
    const int T_ = p.T;
    const size_t tok_stride = (size_t)p.H * kSN;
    const size_t base = ((size_t)b * T_ * p.H + h) * kSN;
    const int nblocks = (T_ + kTS - 1) / kTS;

    if (tid < NT) {
        const int cg = tid % G, row0 = tid / G * R;
        const size_t soff = ((size_t)bh * kSN + row0) * kSN + cg * 4;
        f2 S[R][4];
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const size_t o = soff + (size_t)i * kSN + j * 32;
                float x[4];
                if (p.state_f16) load4(reinterpret_cast<const __half*>(p.state_in) + o, x);
                else load4(reinterpret_cast<const float*>(p.state_in) + o, x);
                S[i][2 * j] = pack2(x[0], x[1]);
                S[i][2 * j + 1] = pack2(x[2], x[3]);
            }
        float y[R] = {};
        auto dot = [&](float (&out)[R], const f2 (&x)[4]) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const f2 q = fma2(S[i][3], x[3], fma2(S[i][2], x[2], fma2(S[i][1], x[1], mul2(S[i][0], x[0]))));
                float lo, hi;
                unpack2(q, lo, hi);
                out[i] = lo + hi;
            }
        };
        // Sums over the eight lanes of a row group in three steps, with work that does not wait for them in between: S.kk of this
        // token goes to all lanes; the output of the token before is halved to one row a lane on the way (which rows go up is
        // decided by the bits of the lane), and one of the lanes that end up with a row stores it.
        const bool hi4 = (cg & 4) != 0, hi2 = (cg & 2) != 0;
        const int yrow = row0 + (hi4 ? 2 : 0) + (hi2 ? 1 : 0);
        const bool ystore = (cg & 1) == 0;
        auto xchg = [](float v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); };
        auto decay_rows = [&](int i0, const TokenRegs& o) {
#pragma unroll
            for (int i = i0; i < i0 + R / 2; ++i) {
                const f2 v2 = pack2(o.v[i], o.v[i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) S[i][j] = fma2(v2, o.k[j], mul2(S[i][j], o.w[j]));
            }
        };
        float ya[R / 2], yb[R / 2], y1 = 0.f, y1q = 0.f;  // the output sum on its way
        auto y_step4 = [&] {
#pragma unroll
            for (int i = 0; i < R / 2; ++i) {
                ya[i] = hi4 ? y[R / 2 + i] : y[i];
                yb[i] = xchg(hi4 ? y[i] : y[R / 2 + i], 4);
            }
        };
        auto y_step2 = [&] {
#pragma unroll
            for (int i = 0; i < R / 2; ++i) ya[i] += yb[i];
            y1 = hi2 ? ya[1] : ya[0];
            y1q = xchg(hi2 ? ya[0] : ya[1], 2);
        };
        auto y_step1 = [&] {
            y1 += y1q;
            y1q = xchg(y1, 1);
        };
        auto token = [&](bool prev, float* yprev, const TokenRegs& o) {  // `yprev`: where the output of the token before goes
            float sa[R], q[R];
            dot(sa, o.kk);
#pragma unroll
            for (int i = 0; i < R; ++i) q[i] = xchg(sa[i], 4);
            if (prev) y_step4();
            decay_rows(0, o);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                sa[i] += q[i];
                q[i] = xchg(sa[i], 2);
            }
            if (prev) y_step2();
            decay_rows(R / 2, o);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                sa[i] += q[i];
                q[i] = xchg(sa[i], 1);
            }
            if (prev) y_step1();
#pragma unroll
            for (int i = 0; i < R; ++i) {
                sa[i] += q[i];
                const f2 s2 = pack2(sa[i], sa[i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) S[i][j] = fma2(s2, o.nb[j], S[i][j]);
            }
            if (prev && ystore) yprev[yrow] = y1 + y1q;
            dot(y, o.r);
        };
        auto last_output = [&](float* ylast) {
            y_step4();
            y_step2();
            y_step1();
            if (ystore) ylast[yrow] = y1 + y1q;
        };
        TokenRegs o[CTAS == 1 ? 2 : 1];
        for (int it = -LAG; it < nblocks + LAG; ++it) {
            if (it >= 0 && it < nblocks) {
                Operands& op = ops[it % BLOCKS];
                const Operands& next = ops[(it + 1) % BLOCKS];  // ACROSS: there since the last barrier; past the end: nobody's
                // before a block's first token comes the last one of the block before; before the first of all: overwritten by the next token
                float* y0 = ACROSS && it > 0 ? ops[(it - 1) % BLOCKS].y[kTS - 1] : op.y[0];
                const int nt = min(kTS, T_ - it * kTS);
                if (ACROSS && it == 0) load_token(o[0], op, 0, row0, cg);
                if (nt == kTS) {
                    if (!ACROSS) load_token(o[0], op, 0, row0, cg);
#pragma unroll
                    for (int t = 0; t < kTS; ++t) {
                        float* yprev = t > 0 ? op.y[t - 1] : y0;
                        if constexpr (CTAS == 1) {  // the next token's operands a token ahead
                            const Operands& from = t + 1 < kTS ? op : next;
                            if (ACROSS || t + 1 < kTS) load_token(o[(t + 1) & 1], from, (t + 1) % kTS, row0, cg);
                            token(ACROSS || t > 0, yprev, o[t & 1]);
                        } else {  // two CTAs an SM: no registers for that, and less need
                            token(t > 0, yprev, o[0]);
                            if (t + 1 < kTS) load_token(o[0], op, t + 1, row0, cg);
                        }
                    }
                } else {
#pragma unroll 1
                    for (int t = 0; t < nt; ++t) {
                        load_token(o[0], op, t, row0, cg);
                        token(ACROSS || t > 0, t > 0 ? op.y[t - 1] : y0, o[0]);
                    }
                }
                if (!ACROSS) last_output(op.y[nt - 1]);
            } else if (ACROSS && it == nblocks) {
                last_output(ops[(it - 1) % BLOCKS].y[T_ - 1 - (it - 1) * kTS]);
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const size_t o = soff + (size_t)i * kSN + j * 32;
                float x[4];
                unpack2(S[i][2 * j], x[0], x[1]);
                unpack2(S[i][2 * j + 1], x[2], x[3]);
                if (p.state_f16) store4(reinterpret_cast<__half*>(p.state_out) + o, x);
                else store4(reinterpret_cast<float*>(p.state_out) + o, x);
            }
    } else if (tid < NT + 64) {
        // two channels of four tokens a thread
        const int ht = tid - NT, c = (ht & 31) * 2, tt0 = (ht >> 5) * 4;
        const int wsz = p.w_mode == 1 ? 4 : (int)sizeof(T);
        const int phase0 = p.elapsed ? p.elapsed[b] + h * kSN : 0;
        float w0[2] = {0.f, 0.f};
        if (p.w0) {
#pragma unroll
            for (int i = 0; i < 2; ++i) w0[i] = to_f<T>(reinterpret_cast<const T*>(p.w0)[h * kSN + c + i]);
        }
        Pair<T> r[4], k[4], v[4], kk[4], a[4], wt[4];
        float2 wf[4];
        auto fetch = [&](int s) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int t = min(s * kTS + tt0 + u, T_ - 1);  // past the end: a token that exists, whose operands nobody uses
                const size_t o = base + (size_t)t * tok_stride + c;
                auto get = [&](const void* q) { return *reinterpret_cast<const Pair<T>*>(reinterpret_cast<const T*>(q) + o); };
                r[u] = get(p.r); k[u] = get(p.k); v[u] = get(p.v); kk[u] = get(p.kk); a[u] = get(p.a);
                if (p.w_mode == 1) wf[u] = *reinterpret_cast<const float2*>(reinterpret_cast<const float*>(p.w) + o);
                else wt[u] = get(p.w);
            }
        };
        // rows of a later block on their way to L2: eight threads a token, one operand each
        auto announce = [&](int s) {
            const int t = s * kTS + (ht >> 3), q = ht & 7;
            if (t >= T_ || q > 5) return;
            const void* src = q == 0 ? p.r : q == 1 ? p.k : q == 2 ? p.v : q == 3 ? p.kk : q == 4 ? p.a : p.w;
            const int size = q == 5 ? wsz : (int)sizeof(T);
            const char* row = reinterpret_cast<const char*>(src) + (base + (size_t)t * tok_stride) * size;
            prefetch_l2(row);
            if (size == 4) prefetch_l2(row + 128);
        };
        fetch(0);
        announce(1);
        announce(2);
        for (int it = -LAG; it < nblocks + LAG; ++it) {
            const int s = it + LAG;
            if (s < nblocks) {
                Operands& op = ops[s % BLOCKS];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int tt = tt0 + u;
                    float2 w;
                    if (p.w_mode == 1) w = wf[u];
                    else {
                        w = to_f2(wt[u]);
                        if (p.w_mode == 2) {
                            float e[2] = {w.x, w.y};
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                if (p.w0) e[i] += w0[i];
                                e[i] = decay_from_raw(e[i]);
                                // (decay - 1 + rotator) rounded to fp16, as the reference's kernel forms its decay operand
                                if (p.elapsed) e[i] = 1.0f + __half2float(__float2half_rn(e[i] - 1.0f + scan_rotator1(phase0 + c + i + s * kTS + tt)));
                            }
                            w = make_float2(e[0], e[1]);
                        }
                    }
                    const float2 kkf = to_f2(kk[u]), af = to_f2(a[u]);
                    *reinterpret_cast<float2*>(&op.w[tt][c]) = w;
                    *reinterpret_cast<float2*>(&op.kk[tt][c]) = p.ab_mode ? make_float2(-kkf.x, -kkf.y) : kkf;
                    *reinterpret_cast<float2*>(&op.nb[tt][c]) = p.ab_mode ? make_float2(-af.x, -af.y) : make_float2(-(kkf.x * af.x), -(kkf.y * af.y));
                    *reinterpret_cast<float2*>(&op.r[tt][c]) = to_f2(r[u]);
                    *reinterpret_cast<float2*>(&op.k[tt][c]) = to_f2(k[u]);
                    *reinterpret_cast<float2*>(&op.v[tt][c]) = to_f2(v[u]);
                }
                if (s + 1 < nblocks) fetch(s + 1);
                announce(s + 3);
            }
            __syncthreads();
        }
    } else {
        // eight lanes a token, eight channels a lane
        const int ht = tid & 63, tt = ht >> 3, c = (ht & 7) * 8;
        float rk[8], gw[8], gb[8];
        Vec8<T> g{};
        if constexpr (PREP) {
            auto load_param = [&](const void* param, float (&o)[8]) {
                const T* q = reinterpret_cast<const T*>(param) + h * kSN + c;
                if (p.params_vec) {
                    load8(q, o);
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) o[i] = to_f<T>(q[i]);
                }
            };
            load_param(p.r_k, rk);
            load_param(p.gn_w, gw);
            load_param(p.gn_b, gb);
        }
        for (int it = -LAG; it < nblocks + LAG; ++it) {
            const int s = it - LAG;
            if (s >= 0) {
                const Operands& op = ops[s % BLOCKS];
                const int t = s * kTS + tt;
                const bool live = t < T_;  // the shuffles below run in all lanes
                float y[8];
                load8<float>(&op.y[live ? tt : 0][c], y);
                if constexpr (PREP) {
                    float r[8], k[8], v[8];
                    load8<float>(&op.r[live ? tt : 0][c], r);
                    load8<float>(&op.k[live ? tt : 0][c], k);
                    load8<float>(&op.v[live ? tt : 0][c], v);
                    float sum = 0.f, corr = 0.f, var = 0.f;
#pragma unroll
                    for (int i = 0; i < 8; ++i) { sum += y[i]; corr += r[i] * k[i] * rk[i]; }
                    const float mean = group_sum<8>(sum) * (1.0f / kSN);
                    corr = group_sum<8>(corr);
#pragma unroll
                    for (int i = 0; i < 8; ++i) { y[i] -= mean; var += y[i] * y[i]; }
                    const float rstd = rsqrtf(group_sum<8>(var) * (1.0f / kSN) + p.eps);
#pragma unroll
                    for (int i = 0; i < 8; ++i) y[i] = (y[i] * rstd * gw[i] + gb[i] + corr * v[i]) * to_f<T>(g.v[i]);
                }
                if (live) store8(reinterpret_cast<T*>(p.y) + base + (size_t)t * tok_stride + c, y);
            }
            if constexpr (PREP) {  // the gate of the block that is written next
                const int t = (s + 1) * kTS + tt;
                if (s >= -1 && t < T_) {
                    const T* q = reinterpret_cast<const T*>(p.g) + base + (size_t)t * tok_stride + c;
                    reinterpret_cast<uint4*>(&g)[0] = reinterpret_cast<const uint4*>(q)[0];
                    if constexpr (sizeof(T) == 4) reinterpret_cast<uint4*>(&g)[1] = reinterpret_cast<const uint4*>(q)[1];
                }
            }
            __syncthreads();
        }
    }
}

// ---- more CTAs an SM: they hide each other's loads, and 64 threads load, convert, run and write a block in turn ------------
template <typename T, bool PREP, int R, int C>
__global__ void __launch_bounds__(kSN / R * (kSN / C)) wkv7_scan_kernel(const ScanArgs p) {
    constexpr int G = kSN / C;
    constexpr int NT = kSN / R * G;  // threads of the token loop
    static_assert(NT == 64, "64 threads load and write");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RawStage<T>* raw = reinterpret_cast<RawStage<T>*>(smem_raw);  // [2]
    Operands& op = *reinterpret_cast<Operands*>(smem_raw + 2 * sizeof(RawStage<T>));

    const int bh = blockIdx.x;
    const int b = bh / p.H, h = bh % p.H;
    const int tid = threadIdx.x;
    const int T_ = p.T;
    const size_t tok_stride = (size_t)p.H * kSN;              // elements between consecutive tokens
    const size_t base = ((size_t)b * T_ * p.H + h) * kSN;     // element offset of token 0
    const int phase0 = p.elapsed ? p.elapsed[b] + h * kSN : 0;
    const int nstages = (T_ + kTS - 1) / kTS;

    // ---- in and out--------------------------------------------------------------------------------------------------
    auto issue_stage = [&](int s) {
        constexpr int CH = kSN * (int)sizeof(T) / 16;  // 16-byte chunks per token vector
        RawStage<T>& rs = raw[s & 1];
        const int t0 = s * kTS, nt = min(kTS, T_ - t0);
        const T* srcs[5] = {reinterpret_cast<const T*>(p.r), reinterpret_cast<const T*>(p.k), reinterpret_cast<const T*>(p.v),
                            reinterpret_cast<const T*>(p.kk), reinterpret_cast<const T*>(p.a)};
        T(*dsts[5])[kSN] = {rs.r, rs.k, rs.v, rs.kk, rs.a};
#pragma unroll
        for (int q = 0; q < 5; ++q)
            for (int idx = tid; idx < nt * CH; idx += 64) {
                const int tt = idx / CH, ch = idx % CH;
                cp_async16(reinterpret_cast<char*>(dsts[q][tt]) + ch * 16,
                           reinterpret_cast<const char*>(srcs[q] + base + (size_t)(t0 + tt) * tok_stride) + ch * 16);
            }
        const int wsz = (p.w_mode == 1) ? 4 : (int)sizeof(T), chw = kSN * wsz / 16;
        for (int idx = tid; idx < nt * chw; idx += 64) {
            const int tt = idx / chw, ch = idx % chw;
            cp_async16(reinterpret_cast<char*>(rs.w[tt]) + ch * 16,
                       reinterpret_cast<const char*>(p.w) + (base + (size_t)(t0 + tt) * tok_stride) * wsz + ch * 16);
        }
        cp_async_commit();
    };

    // thread = two channels x half of the block's tokens
    auto convert = [&](int s) {
        RawStage<T>& rs = raw[s & 1];
        const int t0 = s * kTS, nt = min(kTS, T_ - t0);
        const int c = (tid & 31) * 2;
        auto two = [](const T* q) {
            if constexpr (sizeof(T) == 4) return *reinterpret_cast<const float2*>(q);
            else return make_float2(to_f<T>(q[0]), to_f<T>(q[1]));
        };
#pragma unroll
        for (int u = 0; u < kTS / 2; ++u) {
            const int tt = (tid >> 5) * (kTS / 2) + u;
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
    auto flush = [&](int s) {
        const int t0 = s * kTS, nt = min(kTS, T_ - t0);
        const int l8 = tid & 7, c = l8 * 8;
        auto load_param = [&](const void* param, float (&o)[8]) {
            const T* q = reinterpret_cast<const T*>(param) + h * kSN + c;
            if (p.params_vec) {
                load8(q, o);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = to_f<T>(q[i]);
            }
        };
        for (int tt = tid >> 3; tt < kTS; tt += 8) {
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
    issue_stage(0);
    for (int s = 0; s < nstages; ++s) {
        if (s + 1 < nstages) {
            issue_stage(s + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();  // raw block visible; the previous block's flush has read the operands
        convert(s);
        __syncthreads();
        scan_block<R, C>(S, op, min(kTS, T_ - s * kTS), row0, cg);
        __syncthreads();
        flush(s);
    }

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

template <typename T, bool PREP>
static int dispatch_scan(const ScanArgs& p, int B, cudaStream_t st) {
    // Chosen by how many CTAs an SM gets.  Up to one, and up to two (with fewer registers a thread): the form with loads, output
    // and recurrence on warps of their own.  More: the CTAs of an SM hide each other's loads and the extra warps only take
    // registers.  us for 512 tokens, fp16, output prepared, by CTAs, before -> three blocks: 12 126 -> 115, 148 129 -> 117, 149 193 -> 185,
    // 296 194 -> 185; for 16 tokens 7.2 -> 7.0, 7.7 -> 7.5, 9.4 -> 9.2, 9.8 -> 9.6.  320: 405, where the form for fewer takes two waves (438).
    const int ctas = B * p.H;
    const bool few = ctas <= 2 * kSMs;
    // Five blocks instead of three with the output prepared and one CTA an SM, from where their two barriers are paid for.  us, three -> five, 12 / 120 CTAs,
    // fp16: 16 tokens 6.6 / 7.3 -> 7.3 / 7.9, 128 31.4 / 32.1 -> 31.7 / 32.7, 192 45.1 / 46.0 -> 45.0 / 46.2, 224 52.0 / 53.0 -> 51.7 / 52.9, 256 59.0 / 60.1 -> 58.4 / 59.8, 512 114.0 /
    // 116.0 -> 111.7 / 114.7, 777 171.6 / 176.5 -> 167.4 / 173.3; fp32: 192 46.1 / 47.0 -> 45.8 / 46.7, 777 176.9 / 180.7 -> 172.8 / 176.4.  Without it, or at two CTAs an SM,
    // five take 0..2 % longer at every length.
    const bool across = PREP && ctas <= kSMs && p.T > 192;
    void (*kern)(const ScanArgs) = !few           ? wkv7_scan_kernel<T, PREP, 2, 32>
                                   : ctas > kSMs  ? wkv7_scan_few_kernel<T, PREP, 2, 3>
                                   : across       ? wkv7_scan_few_kernel<T, PREP, 1, PREP ? 5 : 3>
                                                  : wkv7_scan_few_kernel<T, PREP, 1, 3>;
    const int threads = few ? 256 : 64;
    const size_t smem = few ? (across ? 5 : 3) * sizeof(Operands) : 2 * sizeof(RawStage<T>) + sizeof(Operands);
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    RWKV7_REQUIRE(e == cudaSuccess, RWKV7_ERR_CUDA, "wkv7_scan: %s", cudaGetErrorString(e));
    kern<<<ctas, threads, smem, st>>>(p);
    return check_launch(few ? "wkv7_scan_few_kernel" : "wkv7_scan_kernel");
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
