// WKV-7 single-token recurrence for decode: one CTA per (sequence, head).
//
// The 64x64 fp32 state tile is streamed HBM -> registers -> HBM exactly once
// (16 KiB in, 16 KiB out); everything else the decode layer does around the
// recurrence (decay, kk normalisation, k adjustment, v interpolation, a/w LoRA
// biases, GroupNorm, bonus term, output gate) is folded into the same pass so
// no intermediate vector touches HBM.  The kernel is HBM-bound: algorithmic
// traffic is 2*64*64*4 + ~7*64*sizeof(T) bytes per (sequence, head).
//
// The state may also be stored in fp16 (the reference's opt-in FP16-state lanes: the Triton output-prepare kernels
// load it to fp32 and round the result back, rwkv7_hf/fused_recurrent_update.py:655-699; the native_wkv_fp16
// extension additionally dithers the decay, rwkv7_hf/native_wkv_fp16.py:118-128): the arithmetic stays fp32, the
// traffic halves.
//
// Thread map (128 threads): lane16 = tid & 15 owns columns 4*lane16..+3 (key
// index j), rowgroup = tid >> 4 owns rows rowgroup + 8*it (value index i), so a
// warp instruction touches two full 256-byte state rows = 512 contiguous bytes.
//
// What it costs beside the state is instructions, of which a head has few warps to hide them: the vectors of the head are
// made once, by one warp each (when all eight row groups made them for themselves that was two thirds of the kernel), and the
// sums over the columns of a thread's eight rows run together (sum_rows).  us a launch, before -> now: 64 rows of 64 heads, fp32
// state 27.7 -> 22.9 (6.0 TB/s of the bytes above), 256 rows 100 -> 82 (6.7: above the rate of a copy, because up to an L2 of written state
// drains under the kernels behind; at 64 rows DRAM sees 80 of the 138 MB within the kernel); 64 rows of 40 heads, fp16 state 18.3 -> 13; one row of 12 heads 5.9 -> 4.0.
#include "common.cuh"

namespace rwkv7 {

constexpr int kN = 64;
constexpr int kStepThreads = 128;

enum StepMode { kUpdate = 0, kPrepare = 1, kRaw = 2 };

struct StepArgs {
    const void *r, *w, *k, *v, *kk, *a;
    const void* state_in;  // fp32 or fp16 [B,H,64,64]
    void* state_out;
    void* out;
    const void *g, *r_k, *gn_w, *gn_b;
    const void *k_k, *k_a;
    const void *w_bias, *a_bias, *v_first, *v_gate, *v_gate_bias;
    void* v_out;
    int a_is_raw, v_gate_is_raw;
    int H;
    float eps;
    int prefetch_state;  // load the state tile before the grid-dependency wait (state_prefetch argument of the raw entry point)
    int idle_slot;       // state pool: the row of padding rows, which are not computed (-1: none)
    const int* slots;    // state pool: row b of the batch lives in pool row slots[b] (state, v_first / v_out, elapsed); NULL = row b
    const int* elapsed;  // fp16 state, raw mode: per-sequence step counters [B] that phase the decay dither (NULL = no dither)
};

// Deterministic zero-mean rotator of the reference's FP16-state kernel (rwkv7_hf/native_wkv_fp16.py:118-121): the
// decay of a half-precision state is often smaller than half an ulp of the entry it multiplies, which would freeze it
// under round-to-nearest; a pseudo-random offset of up to +-2^-10 on (decay - 1), different for every channel and
// step, makes the rounding unbiased on average.
__device__ __forceinline__ float rotator1(int x) {
    const uint32_t bits = 2654435769u * static_cast<uint32_t>(x);
    return 4.547473508864641e-13f * static_cast<float>(static_cast<int32_t>(bits));
}

// Two elements in storage type: requested together, converted where they are used, so that the operands of a step cost one
// trip to memory and not one per branch (zeros when `ok` is false).
template <typename T> struct alignas(sizeof(T) * 2) Raw2 { T v[2]; };
template <typename T>
__device__ __forceinline__ Raw2<T> ld_raw2(const void* base, size_t off, bool ok = true) {
    Raw2<T> r{};
    if (ok) r = *reinterpret_cast<const Raw2<T>*>(reinterpret_cast<const T*>(base) + off);
    return r;
}
template <typename T>
__device__ __forceinline__ float2 cvt2(const Raw2<T>& r) { return make_float2(to_f<T>(r.v[0]), to_f<T>(r.v[1])); }
template <typename T>
__device__ __forceinline__ void st2(void* base, size_t off, float x, float y) {
    Raw2<T> r;
    r.v[0] = from_f<T>(x);
    r.v[1] = from_f<T>(y);
    *reinterpret_cast<Raw2<T>*>(reinterpret_cast<T*>(base) + off) = r;
}

template <typename TS> struct StateIO;
template <> struct StateIO<float> {
    typedef float4 Raw;  // four columns as they are stored
    static __device__ __forceinline__ Raw load(const void* base, size_t off) {
        return *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + off);  // plain load: may alias state_out
    }
    static __device__ __forceinline__ float4 value(const Raw& r) { return r; }
    // streaming store: the new state is not read again before the next token, so it should not linger in L2 and
    // be written back under the kernels that follow (measured: -8 % time)
    static __device__ __forceinline__ void store(void* base, size_t off, const float4& s) {
        __stcs(reinterpret_cast<float4*>(reinterpret_cast<float*>(base) + off), s);
    }
};
template <> struct StateIO<__half> {
    typedef uint2 Raw;
    static __device__ __forceinline__ Raw load(const void* base, size_t off) {
        return *reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(base) + off);
    }
    static __device__ __forceinline__ float4 value(const Raw& u) {
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
    static __device__ __forceinline__ void store(void* base, size_t off, const float4& s) {
        const __half2 a = __floats2half2_rn(s.x, s.y), b = __floats2half2_rn(s.z, s.w);
        uint2 u;
        u.x = *reinterpret_cast<const uint32_t*>(&a);
        u.y = *reinterpret_cast<const uint32_t*>(&b);
        __stcs(reinterpret_cast<uint2*>(reinterpret_cast<__half*>(base) + off), u);
    }
};

// Sums over the 16 lanes of a row group, of eight rows at once: each exchange halves the rows that a lane goes on with, so eight sums
// cost eight shuffles and not 32.  Lane l16 ends with the sum of row (l16 & 7) (lanes l16 and l16 ^ 8 alike).
__device__ __forceinline__ float sum_rows(const float (&v)[8], int l16) {
    float a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // rows 2 i and 2 i + 1: the lane keeps the one of its bit 0
        const float keep = l16 & 1 ? v[2 * i + 1] : v[2 * i], give = l16 & 1 ? v[2 * i] : v[2 * i + 1];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float keep = l16 & 2 ? a[2 * i + 1] : a[2 * i], give = l16 & 2 ? a[2 * i] : a[2 * i + 1];
        b[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
    }
    const float keep = l16 & 4 ? b[1] : b[0], give = l16 & 4 ? b[0] : b[1];
    const float c = keep + __shfl_xor_sync(0xffffffffu, give, 4);
    return c + __shfl_xor_sync(0xffffffffu, c, 8);
}

template <typename T, typename TW, int MODE, typename TS, bool POOL = false>
__global__ void __launch_bounds__(kStepThreads, 8) wkv7_step_kernel(const StepArgs p) {  // 64 registers: 8 CTAs per SM (measured: 7 -> 8 CTAs is -9 % time)
    const int bh = blockIdx.x;
    const int h = bh % p.H;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int l16 = tid & 15;
    const int rg = tid >> 4;
    const size_t vbase = (size_t)bh * kN;
    // with a state pool the recurrent rows of sequence b sit at pool row slots[b]; the step's operands stay batch-ordered
    // (a template parameter, not a run-time test: the dense kernel keeps its exact instruction stream and registers)
    const int srow = POOL ? __ldg(p.slots + bh / p.H) : bh / p.H;
    const size_t sbh = POOL ? (size_t)srow * p.H + h : (size_t)bh;
    const size_t vsbase = sbh * kN;
    const int hbase = h * kN;
    const int c0 = l16 * 4, c2 = lane * 2;

    __shared__ __align__(16) float s_w[kN], s_k[kN], s_kk[kN], s_kka[kN], s_r[kN], s_v[kN], s_y[kN];
    __shared__ float s_corr;

    // Launched programmatically: resident under the tail of the preceding kernel.  By default everything waits for it.
    if (!p.prefetch_state) grid_dependency_wait();
    if (POOL && srow == p.idle_slot) {  // a padding row of a fixed-size batch: nobody's state, nobody reads the output
        if (p.prefetch_state) grid_dependency_wait();
        if (tid == 0) grid_launch_dependents();
        if (tid < 32) st2<T>(p.out, vbase + c2, 0.f, 0.f);
        return;
    }
    // ---- state tile: issue all 8 row loads first (memory-level parallelism)
    const size_t sbase = sbh * kN * kN;
    typename StateIO<TS>::Raw S[8];
#pragma unroll
    for (int it = 0; it < 8; ++it) S[it] = StateIO<TS>::load(p.state_in, sbase + (size_t)(it * 8 + rg) * kN + c0);

    if constexpr (MODE == kRaw) {
        // the parameters of the head are read after the wait like everything else, but are on their way to L2 by then
        if (tid < 8) {
            const void* par[8] = {p.k_k, p.k_a, p.r_k, p.gn_w, p.gn_b, p.w_bias, p.a_bias, p.v_gate_bias};
            const void* q = par[0];
#pragma unroll
            for (int i = 1; i < 8; ++i)
                if (tid == i) q = par[i];
            if (q != nullptr) prefetch_l2(reinterpret_cast<const T*>(q) + hbase);
        }
    }
    // With the state-prefetch option the loads above are already in flight while the preceding kernel (the r/k/v
    // projection of a decode step) finishes: the caller promises that kernel does not write the state, and every
    // kernel of this library releases its successor only after its own wait, so whatever wrote the state earlier has
    // completed.  Everything below reads the preceding kernel's output.
    if (p.prefetch_state) grid_dependency_wait();
    if (tid == 0) grid_launch_dependents();  // the output projection sets up and streams weights under this grid's tail

    // ---- the vectors of the head, two channels a lane, one warp each; shared.  (Formed by every row group for itself they were
    // two thirds of the kernel's instructions.)
    float2 r{};
    if constexpr (MODE != kUpdate) r = cvt2(ld_raw2<T>(p.r, vbase + c2));
    auto put = [&](float* s, float x, float y) { *reinterpret_cast<float2*>(s + c2) = make_float2(x, y); };
    Raw2<T> q_gw{}, q_gb{}, q_g{};
    // The plain update has nothing to make of them: every lane takes its four columns from the operands.  (Through shared memory a
    // grid of more than eight CTAs an SM took longer than before: 22 rows of 64 heads 8.7 -> 9.5 us, so 8.3; 48 rows into a new state 13.6 -> 15.1, so 12.8.)
    float4 w4, k4, kk4, kka4, r4;
    if constexpr (MODE == kUpdate) {
        auto vec4 = [&](auto tag, const void* base) {
            float x[4];
            load4(reinterpret_cast<const decltype(tag)*>(base) + vbase + c0, x);
            return make_float4(x[0], x[1], x[2], x[3]);
        };
        if (tid < kN) s_v[tid] = to_f<T>(reinterpret_cast<const T*>(p.v)[vbase + tid]);
        kk4 = vec4(T{}, p.kk);
        w4 = vec4(TW{}, p.w);
        k4 = vec4(T{}, p.k);
        const float4 a4 = vec4(T{}, p.a);
        r4 = vec4(T{}, p.r);
        kka4 = make_float4(kk4.x * a4.x, kk4.y * a4.y, kk4.z * a4.z, kk4.w * a4.w);
    } else if (warp == 0) {
        float2 w;
        if constexpr (MODE == kRaw) {
            const Raw2<T> q_w = ld_raw2<T>(p.w, vbase + c2), q_wb = ld_raw2<T>(p.w_bias, hbase + c2, p.w_bias != nullptr);
            w = cvt2(q_w);
            if (p.w_bias) {
                const float2 wb = cvt2(q_wb);
                w = make_float2(round_to<T>(w.x + wb.x), round_to<T>(w.y + wb.y));
            }
            w = make_float2(decay_from_raw(w.x), decay_from_raw(w.y));
            if constexpr (sizeof(TS) == 2) {
                if (p.elapsed != nullptr) {  // (decay - 1 + rotator) rounded to fp16, as the reference's FP16-state kernel forms it
                    const int phase = p.elapsed[srow] + hbase + c2;
                    w.x = 1.0f + __half2float(__float2half_rn(w.x - 1.0f + rotator1(phase)));
                    w.y = 1.0f + __half2float(__float2half_rn(w.y - 1.0f + rotator1(phase + 1)));
                }
            }
        } else {
            w = cvt2(ld_raw2<TW>(p.w, vbase + c2));
        }
        put(s_w, w.x, w.y);
        put(s_r, r.x, r.y);
    } else if (warp == 1) {
        const Raw2<T> q_a = ld_raw2<T>(p.a, vbase + c2), q_k = ld_raw2<T>(p.k, vbase + c2);
        float2 k, kk, a;
        if constexpr (MODE == kRaw) {
            const bool has_ab = p.a_is_raw && p.a_bias != nullptr;
            const Raw2<T> q_ks = ld_raw2<T>(p.k_k, hbase + c2), q_ka = ld_raw2<T>(p.k_a, hbase + c2), q_ab = ld_raw2<T>(p.a_bias, hbase + c2, has_ab);
            a = cvt2(q_a);
            k = cvt2(q_k);
            if (p.a_is_raw) {
                const float2 ab = cvt2(q_ab);
                a.x = round_to<T>(sigmoidf_(round_to<T>(a.x + ab.x)));
                a.y = round_to<T>(sigmoidf_(round_to<T>(a.y + ab.y)));
            }
            const float2 ks = cvt2(q_ks), ka = cvt2(q_ka);
            kk = make_float2(k.x * ks.x, k.y * ks.y);
            const float inv = 1.0f / fmaxf(sqrtf(group_sum<32>(kk.x * kk.x + kk.y * kk.y)), 1e-12f);
            kk.x *= inv;
            kk.y *= inv;
            k.x *= 1.0f + (a.x - 1.0f) * ka.x;
            k.y *= 1.0f + (a.y - 1.0f) * ka.y;
        } else {
            a = cvt2(q_a);
            k = cvt2(q_k);
            kk = cvt2(ld_raw2<T>(p.kk, vbase + c2));
        }
        put(s_k, k.x, k.y);
        put(s_kk, kk.x, kk.y);
        put(s_kka, kk.x * a.x, kk.y * a.y);
        const float2 rk = cvt2(ld_raw2<T>(p.r_k, hbase + c2));
        const float corr = group_sum<32>(r.x * k.x * rk.x + r.y * k.y * rk.y);
        if (lane == 0) s_corr = corr;
    } else if (warp == 2) {
        // ---- row-indexed value vector (with the optional v_first interpolation); this warp also makes the output
        const bool interp = MODE == kRaw && p.v_first != nullptr && p.v_gate != nullptr;
        const Raw2<T> q_v = ld_raw2<T>(p.v, vbase + c2);
        q_gw = ld_raw2<T>(p.gn_w, hbase + c2);
        q_gb = ld_raw2<T>(p.gn_b, hbase + c2);
        q_g = ld_raw2<T>(p.g, vbase + c2);
        float2 v = cvt2(q_v);
        if constexpr (MODE == kRaw) {
            if (interp) {
                const Raw2<T> q_gate = ld_raw2<T>(p.v_gate, vbase + c2), q_vf = ld_raw2<T>(p.v_first, vsbase + c2),
                              q_vb = ld_raw2<T>(p.v_gate_bias, hbase + c2, p.v_gate_bias != nullptr);
                float2 gate = cvt2(q_gate);
                const float2 vf = cvt2(q_vf), vb = cvt2(q_vb);
                if (p.v_gate_is_raw) {
                    gate.x = round_to<T>(sigmoidf_(round_to<T>(gate.x + vb.x)));
                    gate.y = round_to<T>(sigmoidf_(round_to<T>(gate.y + vb.y)));
                }
                v.x = round_to<T>(v.x + (vf.x - v.x) * gate.x);
                v.y = round_to<T>(v.y + (vf.y - v.y) * gate.y);
            }
            if (p.v_out) st2<T>(p.v_out, vsbase + c2, v.x, v.y);
        }
        put(s_v, v.x, v.y);
    }
    __syncthreads();

    // ---- the recurrence: eight rows a thread, sums over the columns of all of them together
    {
        auto four = [&](const float* s) { return *reinterpret_cast<const float4*>(s + c0); };
        float sa[8], y[8];
        const float4 kk = MODE == kUpdate ? kk4 : four(s_kk);
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            const float4 s = StateIO<TS>::value(S[it]);
            sa[it] = s.x * kk.x + s.y * kk.y + s.z * kk.z + s.w * kk.w;
        }
        const float mine = sum_rows(sa, l16);
        float4 w = w4, k = k4, kka = kka4;
        if constexpr (MODE != kUpdate) {
            w = four(s_w);
            k = four(s_k);
            kka = four(s_kka);
            r4 = four(s_r);
        }
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            const int i = it * 8 + rg;
            float4 s = StateIO<TS>::value(S[it]);
            const float vi = s_v[i], a = __shfl_sync(0xffffffffu, mine, it, 16);
            s.x = s.x * w.x + vi * k.x - a * kka.x;
            s.y = s.y * w.y + vi * k.y - a * kka.y;
            s.z = s.z * w.z + vi * k.z - a * kka.z;
            s.w = s.w * w.w + vi * k.w - a * kka.w;
            StateIO<TS>::store(p.state_out, sbase + (size_t)i * kN + c0, s);
            if constexpr (sizeof(TS) == 2) {  // the output is formed from the state as stored
                s.x = round_to<__half>(s.x); s.y = round_to<__half>(s.y); s.z = round_to<__half>(s.z); s.w = round_to<__half>(s.w);
            }
            y[it] = s.x * r4.x + s.y * r4.y + s.z * r4.z + s.w * r4.w;
        }
        const float row = sum_rows(y, l16);
        if (l16 < 8) s_y[l16 * 8 + rg] = row;
    }
    __syncthreads();

    if (warp == 2) {
        const float2 y = *reinterpret_cast<const float2*>(s_y + c2);
        if constexpr (MODE == kUpdate) {
            st2<T>(p.out, vbase + c2, y.x, y.y);
        } else {
            const float mean = group_sum<32>(y.x + y.y) * (1.0f / kN);
            const float dx = y.x - mean, dy = y.y - mean;
            const float rstd = rsqrtf(group_sum<32>(dx * dx + dy * dy) * (1.0f / kN) + p.eps), corr = s_corr;
            const float2 gw = cvt2(q_gw), gb = cvt2(q_gb), gate = cvt2(q_g), v = *reinterpret_cast<const float2*>(s_v + c2);
            st2<T>(p.out, vbase + c2, (dx * rstd * gw.x + gb.x + corr * v.x) * gate.x, (dy * rstd * gw.y + gb.y + corr * v.y) * gate.y);
        }
    }
}

template <typename T, typename TW, int MODE, typename TS = float, bool POOL = false>
static int launch_step(StepArgs p, int B, cudaStream_t st) {
    launch_programmatic(wkv7_step_kernel<T, TW, MODE, TS, POOL>, dim3(B * p.H), dim3(kStepThreads), 0, st, p);
    return check_launch("wkv7_step_kernel");
}

__global__ void advance_elapsed_kernel(int* elapsed, int B) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < B) elapsed[b] += 1;
}

static int check_step_common(const StepArgs& p, int B, int H, int N) {
    RWKV7_REQUIRE(N == kN, RWKV7_ERR_UNSUPPORTED, "wkv7: head size must be 64, got %d", N);
    RWKV7_REQUIRE(B > 0 && H > 0, RWKV7_ERR_INVALID, "wkv7: B and H must be positive (B=%d H=%d)", B, H);
    RWKV7_REQUIRE(p.r && p.w && p.k && p.v && p.a && p.state_in && p.state_out && p.out, RWKV7_ERR_INVALID,
                  "wkv7: null tensor pointer");
    const void* ptrs[] = {p.r, p.w, p.k, p.v, p.a, p.kk, p.state_in, p.state_out, p.out, p.g, p.r_k, p.gn_w,
                          p.gn_b, p.k_k, p.k_a, p.w_bias, p.a_bias, p.v_first, p.v_gate, p.v_gate_bias, p.v_out};
    for (const void* q : ptrs) RWKV7_REQUIRE(aligned(q, 16), RWKV7_ERR_ALIGN, "wkv7: pointers must be 16-byte aligned");
    return RWKV7_OK;
}

}  // namespace rwkv7

using namespace rwkv7;

extern "C" int rwkv7_wkv7_update(const void* r, const void* w, const void* k, const void* v, const void* kk,
                                 const void* a, const float* state_in, float* state_out, void* y, int B, int H,
                                 int N, int dtype, int w_is_f32, void* stream) {
    StepArgs p{};
    p.r = r; p.w = w; p.k = k; p.v = v; p.kk = kk; p.a = a;
    p.state_in = state_in; p.state_out = state_out; p.out = y; p.H = H;
    RWKV7_REQUIRE(kk != nullptr, RWKV7_ERR_INVALID, "wkv7_update: kk is null");
    if (int e = check_step_common(p, B, H, N)) return e;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RWKV7_DISPATCH_DTYPE(dtype, T, {
        if (w_is_f32) return launch_step<T, float, kUpdate>(p, B, st);
        return launch_step<T, T, kUpdate>(p, B, st);
    });
    return RWKV7_OK;
}

extern "C" int rwkv7_wkv7_output_prepare(const void* r, const void* w, const void* k, const void* v, const void* kk,
                                         const void* a, const float* state_in, float* state_out, const void* g,
                                         const void* r_k, const void* gn_w, const void* gn_b, void* out, int B,
                                         int H, int N, float eps, int dtype, int w_is_f32, void* stream) {
    StepArgs p{};
    p.r = r; p.w = w; p.k = k; p.v = v; p.kk = kk; p.a = a;
    p.state_in = state_in; p.state_out = state_out; p.out = out; p.H = H;
    p.g = g; p.r_k = r_k; p.gn_w = gn_w; p.gn_b = gn_b; p.eps = eps;
    RWKV7_REQUIRE(kk && g && r_k && gn_w && gn_b, RWKV7_ERR_INVALID, "wkv7_output_prepare: null tensor pointer");
    if (int e = check_step_common(p, B, H, N)) return e;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RWKV7_DISPATCH_DTYPE(dtype, T, {
        if (w_is_f32) return launch_step<T, float, kPrepare>(p, B, st);
        return launch_step<T, T, kPrepare>(p, B, st);
    });
    return RWKV7_OK;
}

extern "C" int rwkv7_wkv7_output_prepare_raw(const void* r, const void* w_raw, const void* k_raw, const void* v,
                                             const void* a, const float* state_in, float* state_out, const void* g,
                                             const void* k_k, const void* k_a, const void* r_k, const void* gn_w,
                                             const void* gn_b, void* out, const void* w_bias, const void* a_bias,
                                             int a_is_raw, const void* v_first, const void* v_gate,
                                             const void* v_gate_bias, int v_gate_is_raw, void* v_out, int state_prefetch,
                                             int B, int H, int N, float eps, int dtype, void* stream) {
    StepArgs p{};
    p.r = r; p.w = w_raw; p.k = k_raw; p.v = v; p.a = a;
    p.state_in = state_in; p.state_out = state_out; p.out = out; p.H = H;
    p.g = g; p.r_k = r_k; p.gn_w = gn_w; p.gn_b = gn_b; p.eps = eps;
    p.k_k = k_k; p.k_a = k_a;
    p.w_bias = w_bias; p.a_bias = a_bias; p.a_is_raw = a_is_raw;
    p.v_first = v_first; p.v_gate = v_gate; p.v_gate_bias = v_gate_bias; p.v_gate_is_raw = v_gate_is_raw;
    p.v_out = v_out;
    p.prefetch_state = state_prefetch != 0;
    RWKV7_REQUIRE(g && r_k && gn_w && gn_b && k_k && k_a, RWKV7_ERR_INVALID,
                  "wkv7_output_prepare_raw: null tensor pointer");
    RWKV7_REQUIRE((v_first == nullptr) == (v_gate == nullptr), RWKV7_ERR_INVALID,
                  "wkv7_output_prepare_raw: v_first and v_gate must be given together");
    if (int e = check_step_common(p, B, H, N)) return e;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RWKV7_DISPATCH_DTYPE(dtype, T, { return launch_step<T, T, kRaw>(p, B, st); });
    return RWKV7_OK;
}

// ---------------------------------------------------------------- state pool
extern "C" int rwkv7_wkv7_output_prepare_raw_pool_idle(const void* r, const void* w_raw, const void* k_raw, const void* v,
                                                  const void* a, float* state_pool, const int32_t* slot_ids, const void* g,
                                                  const void* k_k, const void* k_a, const void* r_k, const void* gn_w,
                                                  const void* gn_b, void* out, const void* w_bias, const void* a_bias,
                                                  int a_is_raw, const void* v_first_pool, const void* v_gate,
                                                  const void* v_gate_bias, int v_gate_is_raw, void* v_out_pool,
                                                  int state_prefetch, int idle_slot, int B, int H, int N, float eps, int dtype,
                                                  void* stream) {
    StepArgs p{};
    p.r = r; p.w = w_raw; p.k = k_raw; p.v = v; p.a = a;
    p.state_in = state_pool; p.state_out = state_pool; p.out = out; p.H = H;
    p.g = g; p.r_k = r_k; p.gn_w = gn_w; p.gn_b = gn_b; p.eps = eps;
    p.k_k = k_k; p.k_a = k_a;
    p.w_bias = w_bias; p.a_bias = a_bias; p.a_is_raw = a_is_raw;
    p.v_first = v_first_pool; p.v_gate = v_gate; p.v_gate_bias = v_gate_bias; p.v_gate_is_raw = v_gate_is_raw;
    p.v_out = v_out_pool;
    p.prefetch_state = state_prefetch != 0;
    p.slots = slot_ids;
    p.idle_slot = idle_slot;
    RWKV7_REQUIRE(slot_ids && g && r_k && gn_w && gn_b && k_k && k_a, RWKV7_ERR_INVALID,
                  "wkv7_output_prepare_raw_pool: null tensor pointer");
    RWKV7_REQUIRE((v_first_pool == nullptr) == (v_gate == nullptr), RWKV7_ERR_INVALID,
                  "wkv7_output_prepare_raw_pool: v_first_pool and v_gate must be given together");
    if (int e = check_step_common(p, B, H, N)) return e;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RWKV7_DISPATCH_DTYPE(dtype, T, { return launch_step<T, T, kRaw, float, true>(p, B, st); });
    return RWKV7_OK;
}

extern "C" int rwkv7_wkv7_output_prepare_raw_pool(const void* r, const void* w_raw, const void* k_raw, const void* v, const void* a, float* state_pool,
                                                  const int32_t* slot_ids, const void* g, const void* k_k, const void* k_a, const void* r_k,
                                                  const void* gn_w, const void* gn_b, void* out, const void* w_bias, const void* a_bias, int a_is_raw,
                                                  const void* v_first_pool, const void* v_gate, const void* v_gate_bias, int v_gate_is_raw,
                                                  void* v_out_pool, int state_prefetch, int B, int H, int N, float eps, int dtype, void* stream) {
    return rwkv7_wkv7_output_prepare_raw_pool_idle(r, w_raw, k_raw, v, a, state_pool, slot_ids, g, k_k, k_a, r_k, gn_w, gn_b, out, w_bias, a_bias, a_is_raw,
                                                   v_first_pool, v_gate, v_gate_bias, v_gate_is_raw, v_out_pool, state_prefetch, -1, B, H, N, eps, dtype,
                                                   stream);
}

// ---------------------------------------------------------------- fp16 recurrent state
extern "C" int rwkv7_wkv7_output_prepare_f16state(const void* r, const void* w, const void* k, const void* v, const void* kk,
                                                  const void* a, const void* state_in, void* state_out, const void* g,
                                                  const void* r_k, const void* gn_w, const void* gn_b, void* out, int B,
                                                  int H, int N, float eps, int dtype, int w_is_f32, void* stream) {
    StepArgs p{};
    p.r = r; p.w = w; p.k = k; p.v = v; p.kk = kk; p.a = a;
    p.state_in = state_in; p.state_out = state_out; p.out = out; p.H = H;
    p.g = g; p.r_k = r_k; p.gn_w = gn_w; p.gn_b = gn_b; p.eps = eps;
    RWKV7_REQUIRE(kk && g && r_k && gn_w && gn_b, RWKV7_ERR_INVALID, "wkv7_output_prepare_f16state: null tensor pointer");
    if (int e = check_step_common(p, B, H, N)) return e;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RWKV7_DISPATCH_DTYPE(dtype, T, {
        if (w_is_f32) return launch_step<T, float, kPrepare, __half>(p, B, st);
        return launch_step<T, T, kPrepare, __half>(p, B, st);
    });
    return RWKV7_OK;
}

extern "C" int rwkv7_wkv7_output_prepare_raw_f16state(const void* r, const void* w_raw, const void* k_raw, const void* v,
                                                      const void* a, const void* state_in, void* state_out, const void* g,
                                                      const void* k_k, const void* k_a, const void* r_k, const void* gn_w,
                                                      const void* gn_b, void* out, const void* w_bias, const void* a_bias,
                                                      int a_is_raw, const void* v_first, const void* v_gate,
                                                      const void* v_gate_bias, int v_gate_is_raw, void* v_out,
                                                      int* elapsed, int advance_elapsed, int state_prefetch, int B, int H,
                                                      int N, float eps, int dtype, void* stream) {
    StepArgs p{};
    p.r = r; p.w = w_raw; p.k = k_raw; p.v = v; p.a = a;
    p.state_in = state_in; p.state_out = state_out; p.out = out; p.H = H;
    p.g = g; p.r_k = r_k; p.gn_w = gn_w; p.gn_b = gn_b; p.eps = eps;
    p.k_k = k_k; p.k_a = k_a;
    p.w_bias = w_bias; p.a_bias = a_bias; p.a_is_raw = a_is_raw;
    p.v_first = v_first; p.v_gate = v_gate; p.v_gate_bias = v_gate_bias; p.v_gate_is_raw = v_gate_is_raw;
    p.v_out = v_out;
    p.prefetch_state = state_prefetch != 0;
    p.elapsed = elapsed;
    RWKV7_REQUIRE(g && r_k && gn_w && gn_b && k_k && k_a, RWKV7_ERR_INVALID,
                  "wkv7_output_prepare_raw_f16state: null tensor pointer");
    RWKV7_REQUIRE((v_first == nullptr) == (v_gate == nullptr), RWKV7_ERR_INVALID,
                  "wkv7_output_prepare_raw_f16state: v_first and v_gate must be given together");
    RWKV7_REQUIRE(!advance_elapsed || elapsed, RWKV7_ERR_INVALID, "wkv7_output_prepare_raw_f16state: advance_elapsed needs elapsed");
    if (int e = check_step_common(p, B, H, N)) return e;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RWKV7_DISPATCH_DTYPE(dtype, T, {
        if (int e = launch_step<T, T, kRaw, __half>(p, B, st)) return e;
        if (advance_elapsed) {  // after the step, in stream order: no CTA of the step can see the new count
            advance_elapsed_kernel<<<(B + 127) / 128, 128, 0, st>>>(elapsed, B);
            return check_launch("advance_elapsed_kernel");
        }
        return RWKV7_OK;
    });
    return RWKV7_OK;
}
