// Small fused element/row kernels around the recurrence: the rank-R LoRA linears with
// their activations, prefill state preparation, and attention-output preparation.
#include "common.cuh"

namespace rwkv7 {

// ---------------------------------------------------------------- dense_small
// out[rows,Nout] = act_out(act_in(x) . W^T + bias).  One warp per (row-block, output);
// the K loop is split across the 32 lanes with 128-bit loads.  ROWS rows share each
// weight load.  Used for the rank-R LoRA projections, where either K or Nout is small.
__device__ __forceinline__ float apply_act(float v, int act) {
    if (act == 1) return tanhf(v);
    if (act == 2) return sigmoidf_(v);
    return v;
}

struct DenseArgs {
    const void *x, *W, *bias;
    void* out;
    int rows, K, Nout, act_in, act_out;
};

template <typename T, int ROWS>
__global__ void __launch_bounds__(256) dense_small_kernel(const DenseArgs p) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = blockIdx.x * 8 + warp;
    const int r0 = blockIdx.y * ROWS;
    if (n >= p.Nout) return;
    const T* W = reinterpret_cast<const T*>(p.W) + (size_t)n * p.K;
    const T* x = reinterpret_cast<const T*>(p.x);
    float acc[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) acc[r] = 0.f;
    for (int k0 = lane * 8; k0 < p.K; k0 += 256) {
        float w[8];
        load8(W + k0, w);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            if (r0 + r < p.rows) {
                float xv[8];
                load8(x + (size_t)(r0 + r) * p.K + k0, xv);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    float t = xv[e];
                    if (p.act_in) t = round_to<T>(apply_act(t, p.act_in));
                    acc[r] = fmaf(t, w[e], acc[r]);
                }
            }
        }
    }
    const float bias = p.bias ? to_f<T>(reinterpret_cast<const T*>(p.bias)[n]) : 0.f;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const float s = group_sum<32>(acc[r]);
        if (lane == 0 && r0 + r < p.rows) {
            float o = s + bias;
            if (p.act_out) o = apply_act(round_to<T>(o), p.act_out);
            reinterpret_cast<T*>(p.out)[(size_t)(r0 + r) * p.Nout + n] = from_f<T>(o);
        }
    }
}

// ---------------------------------------------------------------- prefill_state_prep
struct PrepArgs {
    const void *w_raw, *k_raw, *v_raw, *a, *k_k, *k_a, *v_first, *v_gate;
    float* w_out;
    void *k_out, *v_out, *kk_out, *a_out;
    int H, a_is_raw, v_gate_is_raw, log_decay;
    long long total_heads;  // rows * H
};

// V consecutive columns in storage type, 8 or 16 bytes: requested together and converted where they are used
template <typename T, int V> struct alignas(V * sizeof(T)) Piece { T v[V]; };
template <typename T, int V>
__device__ __forceinline__ Piece<T, V> get_piece(const void* base, size_t off, bool ok = true) {
    Piece<T, V> r{};
    if (ok) r = *reinterpret_cast<const Piece<T, V>*>(reinterpret_cast<const T*>(base) + off);
    return r;
}
template <typename T, int V>
__device__ __forceinline__ void put_piece(void* base, size_t off, const float (&o)[V]) {
    Piece<T, V> r;
#pragma unroll
    for (int c = 0; c < V; ++c) r.v[c] = from_f<T>(o[c]);
    *reinterpret_cast<Piece<T, V>*>(reinterpret_cast<T*>(base) + off) = r;
}

// 64 / V lanes per (row, head), V columns per lane.  Bound: HBM.  32768 rows of 4096 fp16 with raw gates, no decay (five tensors read,
// three written, 2.1 GB): 565 us with four columns a lane and the v gate requested behind the head's norm, 416 now; the gate
// written as well 438, where a pass of its own took 114.  V: 16 bytes of columns a lane, or 8 where the heads are too few to fill the SMs.
template <typename T, int V>
__global__ void __launch_bounds__(256) state_prep_kernel(const PrepArgs p) {
    constexpr int LANES = 64 / V;
    const long long gidx = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
    const int l = threadIdx.x % LANES;
    const bool active = gidx < p.total_heads;
    const long long g = active ? gidx : p.total_heads - 1;  // keep the shuffle groups converged
    const int h = (int)(g % p.H);
    const size_t off = (size_t)g * 64 + l * V;
    const int hoff = h * 64 + l * V;
    const bool interp = p.v_first && p.v_gate;
    const Piece<T, V> q_k = get_piece<T, V>(p.k_raw, off), q_a = get_piece<T, V>(p.a, off), q_v = get_piece<T, V>(p.v_raw, off),
                      q_vf = get_piece<T, V>(p.v_first, off, interp), q_vg = get_piece<T, V>(p.v_gate, off, interp),
                      q_w = get_piece<T, V>(p.w_raw, off, p.w_raw != nullptr),  // absent: k / v / kk only (the scan takes raw w)
                      q_ks = get_piece<T, V>(p.k_k, hoff), q_ka = get_piece<T, V>(p.k_a, hoff);
    float a[V], kk[V], ko[V], n2 = 0.f;
#pragma unroll
    for (int c = 0; c < V; ++c) {
        a[c] = to_f<T>(q_a.v[c]);
        if (p.a_is_raw) a[c] = sigmoidf_(a[c]);
        const float k = to_f<T>(q_k.v[c]);
        kk[c] = k * to_f<T>(q_ks.v[c]);
        ko[c] = k * (1.0f + (a[c] - 1.0f) * to_f<T>(q_ka.v[c]));
        n2 += kk[c] * kk[c];
    }
    n2 = group_sum<LANES>(n2);
    const float inv = 1.0f / fmaxf(sqrtf(n2), 1e-12f);
    float v[V];
#pragma unroll
    for (int c = 0; c < V; ++c) {
        kk[c] *= inv;
        v[c] = to_f<T>(q_v.v[c]);
        if (interp) {
            float vg = to_f<T>(q_vg.v[c]);
            if (p.v_gate_is_raw) vg = sigmoidf_(vg);
            v[c] = v[c] + (to_f<T>(q_vf.v[c]) - v[c]) * vg;
        }
    }
    if (!active) return;
    if (p.w_out) {  // two exponentials and a division an element that the tensor-core scan's caller does not want
#pragma unroll
        for (int c = 0; c < V; c += 4) {
            float wo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float lw = -0.606531f * sigmoidf_(to_f<T>(q_w.v[c + e]));
                wo[e] = p.log_decay ? lw : expf(lw);
            }
            *reinterpret_cast<float4*>(p.w_out + off + c) = make_float4(wo[0], wo[1], wo[2], wo[3]);
        }
    }
    put_piece<T, V>(p.k_out, off, ko);
    put_piece<T, V>(p.v_out, off, v);
    put_piece<T, V>(p.kk_out, off, kk);
    if (p.a_out) put_piece<T, V>(p.a_out, off, a);
}

// ---------------------------------------------------------------- attn_output_prepare
struct OutPrepArgs {
    const void *rec, *r, *k, *v, *g, *r_k, *gn_w, *gn_b;
    void* out;
    int H;
    float eps;
    long long total_heads;
};

template <typename T>
__global__ void __launch_bounds__(256) output_prepare_kernel(const OutPrepArgs p) {
    const long long gidx = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const int l16 = threadIdx.x & 15;
    const bool active = gidx < p.total_heads;
    const long long g = active ? gidx : p.total_heads - 1;
    const int h = (int)(g % p.H);
    const size_t off = (size_t)g * 64 + l16 * 4;
    const int hoff = h * 64 + l16 * 4;
    float y[4], r[4], k[4], v[4], gt[4], rk[4], gw[4], gb[4];
    load4(reinterpret_cast<const T*>(p.rec) + off, y);
    load4(reinterpret_cast<const T*>(p.r) + off, r);
    load4(reinterpret_cast<const T*>(p.k) + off, k);
    load4(reinterpret_cast<const T*>(p.v) + off, v);
    load4(reinterpret_cast<const T*>(p.g) + off, gt);
    load4(reinterpret_cast<const T*>(p.r_k) + hoff, rk);
    load4(reinterpret_cast<const T*>(p.gn_w) + hoff, gw);
    load4(reinterpret_cast<const T*>(p.gn_b) + hoff, gb);
    const float mean = group_sum<16>(y[0] + y[1] + y[2] + y[3]) * (1.0f / 64);
    float q = 0.f, corr = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        y[c] -= mean;
        q += y[c] * y[c];
        corr += r[c] * k[c] * rk[c];
    }
    const float rstd = rsqrtf(group_sum<16>(q) * (1.0f / 64) + p.eps);
    corr = group_sum<16>(corr);
    float o[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) o[c] = (y[c] * rstd * gw[c] + gb[c] + corr * v[c]) * gt[c];
    if (active) store4(reinterpret_cast<T*>(p.out) + off, o);
}

}  // namespace rwkv7

using namespace rwkv7;

extern "C" int rwkv7_dense_small(const void* x, const void* W, const void* bias, void* out, int rows, int K, int Nout,
                                 int act_in, int act_out, int dtype, void* stream) {
    RWKV7_REQUIRE(rows > 0 && K > 0 && Nout > 0, RWKV7_ERR_INVALID, "dense_small: sizes must be positive");
    RWKV7_REQUIRE(K % 8 == 0, RWKV7_ERR_UNSUPPORTED, "dense_small: K must be a multiple of 8 (got %d)", K);
    RWKV7_REQUIRE(x && W && out, RWKV7_ERR_INVALID, "dense_small: null pointer");
    RWKV7_REQUIRE(act_in >= 0 && act_in <= 2 && act_out >= 0 && act_out <= 2, RWKV7_ERR_INVALID, "dense_small: bad activation code");
    RWKV7_REQUIRE(aligned(x, 16) && aligned(W, 16), RWKV7_ERR_ALIGN, "dense_small: x and W must be 16-byte aligned");
    DenseArgs p{x, W, bias, out, rows, K, Nout, act_in, act_out};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    constexpr int ROWS = 8;
    dim3 grid((Nout + 7) / 8, (rows + ROWS - 1) / ROWS);
    RWKV7_DISPATCH_DTYPE(dtype, T, {
        dense_small_kernel<T, ROWS><<<grid, 256, 0, st>>>(p);
        return check_launch("dense_small_kernel");
    });
    return RWKV7_OK;
}

extern "C" int rwkv7_prefill_state_prep_gate(const void* w_raw, const void* k_raw, const void* v_raw, const void* a,
                                             const void* k_k, const void* k_a, const void* v_first, const void* v_gate,
                                             float* w_out, void* k_out, void* v_out, void* kk_out, void* a_out, int rows, int H, int N,
                                             int a_is_raw, int v_gate_is_raw, int log_decay, int dtype, void* stream) {
    RWKV7_REQUIRE(N == 64, RWKV7_ERR_UNSUPPORTED, "prefill_state_prep: head size must be 64, got %d", N);
    RWKV7_REQUIRE(rows > 0 && H > 0, RWKV7_ERR_INVALID, "prefill_state_prep: sizes must be positive");
    RWKV7_REQUIRE(k_raw && v_raw && a && k_k && k_a && k_out && v_out && kk_out, RWKV7_ERR_INVALID,
                  "prefill_state_prep: null pointer");
    RWKV7_REQUIRE((w_raw == nullptr) == (w_out == nullptr), RWKV7_ERR_INVALID,
                  "prefill_state_prep: w_raw and w_out must be given together (both NULL = no decay output)");
    RWKV7_REQUIRE((v_first == nullptr) == (v_gate == nullptr), RWKV7_ERR_INVALID,
                  "prefill_state_prep: v_first and v_gate must be given together");
    const void* ptrs[] = {w_raw, k_raw, v_raw, a, k_k, k_a, v_first, v_gate, w_out, k_out, v_out, kk_out, a_out};
    for (const void* q : ptrs) RWKV7_REQUIRE(aligned(q, 16), RWKV7_ERR_ALIGN, "prefill_state_prep: unaligned pointer");
    PrepArgs p{w_raw, k_raw, v_raw, a, k_k, k_a, v_first, v_gate, w_out, k_out, v_out, kk_out, a_out,
               H, a_is_raw, v_gate_is_raw, log_decay, (long long)rows * H};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // us with 8 / 4 columns a lane, fp16, decay written: 16 x 40 heads 4.8 / 3.8, 150 x 64 5.9 / 5.4, 800 x 12 5.9 / 5.3, 1024 x 12 6.4 / 6.4, 450 x 40 6.9 / 7.3,
    // 1024 x 64 19.5 / 20.3
    const bool wide = dtype != RWKV7_F32 && p.total_heads >= 12288;
    const long long threads = p.total_heads * (wide ? 8 : 16);
    const int grid = (int)((threads + 255) / 256);
    RWKV7_DISPATCH_DTYPE(dtype, T, {
        if (wide) state_prep_kernel<T, sizeof(T) == 2 ? 8 : 4><<<grid, 256, 0, st>>>(p);
        else state_prep_kernel<T, 4><<<grid, 256, 0, st>>>(p);
        return check_launch("state_prep_kernel");
    });
    return RWKV7_OK;
}

extern "C" int rwkv7_prefill_state_prep(const void* w_raw, const void* k_raw, const void* v_raw, const void* a,
                                        const void* k_k, const void* k_a, const void* v_first, const void* v_gate,
                                        float* w_out, void* k_out, void* v_out, void* kk_out, int rows, int H, int N,
                                        int a_is_raw, int v_gate_is_raw, int log_decay, int dtype, void* stream) {
    return rwkv7_prefill_state_prep_gate(w_raw, k_raw, v_raw, a, k_k, k_a, v_first, v_gate, w_out, k_out, v_out, kk_out, nullptr,
                                         rows, H, N, a_is_raw, v_gate_is_raw, log_decay, dtype, stream);
}

// y = max(x, 0)^2 elementwise (in place allowed), 8 elements per thread
template <typename T>
__global__ void __launch_bounds__(256) relu2_kernel(const T* __restrict__ x, T* __restrict__ y, long long nvec) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
        float v[8];
        load8(x + i * 8, v);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float r = fmaxf(round_to<T>(v[e]), 0.f);
            v[e] = r * r;
        }
        store8(y + i * 8, v);
    }
}

extern "C" int rwkv7_relu2(const void* x, void* y, long long n, int dtype, void* stream) {
    RWKV7_REQUIRE(n > 0 && n % 8 == 0, RWKV7_ERR_UNSUPPORTED, "relu2: element count must be a positive multiple of 8");
    RWKV7_REQUIRE(x && y, RWKV7_ERR_INVALID, "relu2: null pointer");
    RWKV7_REQUIRE(aligned(x, 16) && aligned(y, 16), RWKV7_ERR_ALIGN, "relu2: unaligned pointer");
    const long long nvec = n / 8;
    const int grid = (int)((nvec + 255) / 256 < (long long)kSMs * 32 ? (nvec + 255) / 256 : (long long)kSMs * 32);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RWKV7_DISPATCH_DTYPE(dtype, T, {
        relu2_kernel<T><<<grid, 256, 0, st>>>(reinterpret_cast<const T*>(x), reinterpret_cast<T*>(y), nvec);
        return check_launch("relu2_kernel");
    });
    return RWKV7_OK;
}

extern "C" int rwkv7_attn_output_prepare(const void* recurrent, const void* r, const void* k, const void* v,
                                         const void* g, const void* r_k, const void* gn_w, const void* gn_b, void* out,
                                         int rows, int H, int N, float eps, int dtype, void* stream) {
    RWKV7_REQUIRE(N == 64, RWKV7_ERR_UNSUPPORTED, "attn_output_prepare: head size must be 64, got %d", N);
    RWKV7_REQUIRE(rows > 0 && H > 0, RWKV7_ERR_INVALID, "attn_output_prepare: sizes must be positive");
    RWKV7_REQUIRE(recurrent && r && k && v && g && r_k && gn_w && gn_b && out, RWKV7_ERR_INVALID,
                  "attn_output_prepare: null pointer");
    const void* ptrs[] = {recurrent, r, k, v, g, r_k, gn_w, gn_b, out};
    for (const void* q : ptrs) RWKV7_REQUIRE(aligned(q, 16), RWKV7_ERR_ALIGN, "attn_output_prepare: unaligned pointer");
    OutPrepArgs p{recurrent, r, k, v, g, r_k, gn_w, gn_b, out, H, eps, (long long)rows * H};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const long long threads = p.total_heads * 16;
    const int grid = (int)((threads + 255) / 256);
    RWKV7_DISPATCH_DTYPE(dtype, T, {
        output_prepare_kernel<T><<<grid, 256, 0, st>>>(p);
        return check_launch("output_prepare_kernel");
    });
    return RWKV7_OK;
}
