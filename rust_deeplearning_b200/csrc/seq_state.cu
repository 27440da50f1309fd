// Row kernels that look one or a few tokens back along a sequence and keep what they need of earlier steps per slot.
//
// norm_shift:  n_t = x_t / sqrt(mean(x_t^2) + eps) * w;   m_t = n_t + (n_(t-1) - n_t) * shift   (n_(-1) = 0)
//              the norm and the mix in float; the slot keeps n of the sequence's last token.
// short_conv:  y_t[c] = act(b[c] + sum_j w[c][j] x_(t-(K-1-j))[c])  (inputs before the sequence's start are zero)
//              the sum in float in the order of the taps; the slot keeps the last K - 1 inputs.
//
// Both are cut-invariant by construction: a value that comes from the slot was formed by the same operations in
// the same order as the value a longer step would have read from its own rows.  Only the block that owns a
// sequence's first row of the step touches the slot (it reads the old state, then writes the new one, element by
// element in the thread that read it), so a step's blocks need no order among themselves; with a convolution the
// first rows of a sequence, which all read the slot, are that block's too.
#include "api.h"
#include "common.cuh"
#include "launch.cuh"
#include "row_vec.cuh"

namespace {

__device__ __forceinline__ float silu_exact(float z) { return z / (1.0f + expf(-z)); }

// sum of squares of a float row, every thread gets it
__device__ __forceinline__ float row_square_sum(const float* __restrict__ x, int width, float* scratch) {
    float ss = 0.f;
    for (int i = threadIdx.x; i < width; i += blockDim.x) ss = fmaf(x[i], x[i], ss);
    return block_sum(ss, scratch);
}

template <typename T>
__global__ void __launch_bounds__(256) norm_shift_kernel(const float* __restrict__ x, const void* __restrict__ w, int w_dtype, float eps,
                                                         const void* __restrict__ shift, int shift_dtype, float* __restrict__ state,
                                                         const int* __restrict__ tok_seq, const int* __restrict__ tok_pos,
                                                         const int* __restrict__ seq_start, const int* __restrict__ slots,
                                                         T* __restrict__ normed, T* __restrict__ mixed, int width) {
    __shared__ float scratch[33];
    rdl_grid_wait();
    rdl_grid_launch_dependents();
    const int t = blockIdx.x;
    const float* xr = x + (long long)t * width;
    const float inv = 1.0f / sqrtf(row_square_sum(xr, width, scratch) / (float)width + eps);
    const int p = tok_pos[t];
    if (p < 0) {   // a padding row of a fixed-size batch: finite values, no slot
        for (int i = threadIdx.x; i < width; i += blockDim.x) {
            const T v = from_float<T>(xr[i] * inv * rdl_load(w, i, w_dtype));
            normed[(long long)t * width + i] = v;
            mixed[(long long)t * width + i] = v;
        }
        return;
    }
    const int seq = tok_seq[t], row0 = seq_start[seq];
    const bool first = t == row0;
    float inv_prev = 0.f;
    const float* xp = xr - width;
    if (!first) inv_prev = 1.0f / sqrtf(row_square_sum(xp, width, scratch) / (float)width + eps);
    float* st = state + (long long)slots[seq] * width;
    const int last = seq_start[seq + 1] - 1;
    float inv_last = inv;
    const float* xl = x + (long long)last * width;
    if (first && last != t) inv_last = 1.0f / sqrtf(row_square_sum(xl, width, scratch) / (float)width + eps);
    for (int i = threadIdx.x; i < width; i += blockDim.x) {
        const float wi = rdl_load(w, i, w_dtype);
        const float n = xr[i] * inv * wi;
        float prev;
        if (!first) prev = xp[i] * inv_prev * wi;
        else prev = p == 0 ? 0.f : st[i];
        normed[(long long)t * width + i] = from_float<T>(n);
        mixed[(long long)t * width + i] = from_float<T>(n + (prev - n) * rdl_load(shift, i, shift_dtype));
        if (first) st[i] = xl[i] * inv_last * wi;
    }
}

// A thread's values of a row, all asked for before one is used: no branch and no conversion between the loads (a place beyond
// the row reads its last value, which nothing uses).
template <int NIT, typename S>
__device__ __forceinline__ void row_load(const S* __restrict__ p, int width, float (&f)[NIT]) {
    S raw[NIT];
#pragma unroll
    for (int it = 0; it < NIT; ++it) raw[it] = p[min((int)(threadIdx.x + it * blockDim.x), width - 1)];
#pragma unroll
    for (int it = 0; it < NIT; ++it) f[it] = to_float(raw[it]);
}
template <int NIT>
__device__ __forceinline__ void row_load(const void* p, int dtype, int width, float (&f)[NIT]) {
    if (dtype == RDL_BF16) row_load<NIT>((const __nv_bfloat16*)p, width, f);
    else row_load<NIT>((const float*)p, width, f);
}

// The same with a row in registers: thread i holds values i, i + threads, ... (NIT of them at most).  The kernel is bound by
// latency: a row's sum, the sum of the one other row its block may need (the row before it, or for a sequence's first row
// the sequence's last) and the element-wise pass each went to memory in turn, element after element.  Here the
// constants are asked for before the wait, the rows, the batch description and the slot's state in three trips, and both
// sums meet in one exchange.  Every sum takes the order of the kernel above (a thread's values from the first on, the warp's
// lanes, the warps as the lanes of one), so both give the same bits, whichever block does it.  Groups of four values a
// thread load wider and sum in another order; they are no faster where it counts.
// Width 2,048, bfloat16: 3,399 rows 30.7 us in the kernel above, 22.5 in groups of four, 21.5 here; four prompts of 200 to
// 1,500 rows and 16 single-token steps of a model of four such layers 10.76, 9.45 and 9.49 ms.
template <typename T, int NIT>
__global__ void __launch_bounds__(256) norm_shift_row_kernel(const float* __restrict__ x, const void* __restrict__ w, int w_dtype, float eps,
                                                             const void* __restrict__ shift, int shift_dtype, float* __restrict__ state,
                                                             const int* __restrict__ tok_seq, const int* __restrict__ tok_pos,
                                                             const int* __restrict__ seq_start, const int* __restrict__ slots,
                                                             T* __restrict__ normed, T* __restrict__ mixed, int width) {
    __shared__ float2 sums[8];
    const int t = blockIdx.x, tid = threadIdx.x, n_thr = blockDim.x;
    float wv[NIT], sh[NIT], own[NIT], other[NIT], old[NIT];
    row_load<NIT>(w, w_dtype, width, wv);
    row_load<NIT>(shift, shift_dtype, width, sh);
    rdl_grid_wait();
    rdl_grid_launch_dependents();
    const int p = tok_pos[t], seq = tok_seq[t];
    const float* xr = x + (long long)t * width;
    row_load<NIT>(xr, width, own);
    bool first = false, more = false;      // the sequence's first row of the step; it has further rows
    float* st = nullptr;
    if (p >= 0) {                          // (a padding row of a fixed-size batch has finite values and no slot)
        const int row0 = seq_start[seq], row_end = seq_start[seq + 1];
        st = state + (long long)slots[seq] * width;
        first = t == row0;
        more = first && row_end - 1 != t;
        const float* xo = first ? x + (long long)(row_end - 1) * width : xr - width;
        if (!first || more) row_load<NIT>(xo, width, other);
        if (first && p > 0) row_load<NIT>(st, width, old);
    }
    const bool has_other = p >= 0 && (!first || more);
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
        if (tid + it * n_thr < width) {
            s0 = fmaf(own[it], own[it], s0);
            if (has_other) s1 = fmaf(other[it], other[it], s1);
        }
    }
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    if ((tid & 31) == 0) sums[tid >> 5] = make_float2(s0, s1);
    __syncthreads();
    const bool a_warps = (tid & 31) < n_thr >> 5;
    s0 = warp_sum(a_warps ? sums[tid & 31].x : 0.f);
    s1 = warp_sum(a_warps ? sums[tid & 31].y : 0.f);
    const float inv = 1.0f / sqrtf(s0 / (float)width + eps), inv_other = 1.0f / sqrtf(s1 / (float)width + eps);
#pragma unroll
    for (int it = 0; it < NIT; ++it) {
        const int e = tid + it * n_thr;
        if (e >= width) continue;
        const float n = own[it] * inv * wv[it];
        const float o = has_other ? other[it] * inv_other * wv[it] : n;      // the row before, or the sequence's last
        const float prev = first ? (p == 0 ? 0.f : old[it]) : o;
        normed[(long long)t * width + e] = from_float<T>(n);
        mixed[(long long)t * width + e] = from_float<T>(p < 0 ? n : n + (prev - n) * sh[it]);
        if (first) st[e] = o;
    }
}

constexpr int CONV_MAX_TAPS = 8;

// One row's outputs for the block's channels.  r: the row's index within its sequence's rows of this step.
template <typename T>
__device__ __forceinline__ void conv_row(const T* __restrict__ in, long long in_stride, int row0, int r, int past, int c, int channels,
                                         int taps, const float (&wt)[CONV_MAX_TAPS], float bias, int silu, const float (&old)[CONV_MAX_TAPS],
                                         T* __restrict__ out) {
    float acc = bias;
    for (int j = 0; j < taps; ++j) {
        const int src = r - (taps - 1 - j);
        float v;
        if (src >= 0) v = to_float(in[(long long)(row0 + src) * in_stride + c]);
        else v = past + src < 0 ? 0.f : old[taps - 1 + src];
        acc = fmaf(wt[j], v, acc);
    }
    out[(long long)(row0 + r) * channels + c] = from_float<T>(silu ? silu_exact(acc) : acc);
}

template <typename T>
__global__ void __launch_bounds__(128) short_conv_kernel(const T* __restrict__ in, long long in_stride, int channels, int taps,
                                                         const void* __restrict__ w, int w_dtype, const void* __restrict__ b, int silu,
                                                         float* __restrict__ state, const int* __restrict__ tok_seq,
                                                         const int* __restrict__ tok_pos, const int* __restrict__ seq_start,
                                                         const int* __restrict__ slots, T* __restrict__ out) {
    rdl_grid_wait();
    rdl_grid_launch_dependents();
    const int t = blockIdx.x, c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= channels) return;
    const int p = tok_pos[t];
    if (p < 0) { out[(long long)t * channels + c] = from_float<T>(0.f); return; }
    const int seq = tok_seq[t], row0 = seq_start[seq], r = t - row0;
    if (r > 0 && r < taps - 1) return;          // the block of the sequence's first row forms these rows
    float wt[CONV_MAX_TAPS], old[CONV_MAX_TAPS];
    for (int j = 0; j < taps; ++j) wt[j] = rdl_load(w, (long long)c * taps + j, w_dtype);
    const float bias = b ? rdl_load(b, c, w_dtype) : 0.f;
    for (int j = 0; j < CONV_MAX_TAPS; ++j) old[j] = 0.f;
    if (r > 0) {                                 // every input lies in the step's own rows
        conv_row<T>(in, in_stride, row0, r, p - r, c, channels, taps, wt, bias, silu, old, out);
        return;
    }
    const int n = seq_start[seq + 1] - row0, keep = taps - 1;
    float* st = state + (long long)slots[seq] * keep * channels;
    if (p > 0)
        for (int j = 0; j < keep; ++j) old[j] = st[(long long)j * channels + c];
    for (int rr = 0; rr < min(n, max(keep, 1)); ++rr) conv_row<T>(in, in_stride, row0, rr, p, c, channels, taps, wt, bias, silu, old, out);
    for (int j = 0; j < keep; ++j) {
        const int src = n - keep + j;
        float v;
        if (src >= 0) v = to_float(in[(long long)(row0 + src) * in_stride + c]);
        else v = p + src < 0 ? 0.f : old[keep + src];
        st[(long long)j * channels + c] = v;
    }
}

// Four taps over many rows (a prompt): a thread takes 16 bytes of channels and four rows, whose seven inputs it loads once; the
// kernel above loads two bytes at a time and every input four times.  Every output goes through the same operations.
// Four prompts (3,400 rows) with two such layers and 16 single-token steps: 9.70 -> 9.51 ms; the rule at the launch has more.
constexpr int CONV_RUN = 4;
template <typename T>
__global__ void __launch_bounds__(128) short_conv4_rows_kernel(const T* __restrict__ in, long long in_stride, int n_rows, int channels,
                                                               const T* __restrict__ w, const void* __restrict__ b, int b_dtype, int silu,
                                                               float* __restrict__ state, const int* __restrict__ tok_seq,
                                                               const int* __restrict__ tok_pos, const int* __restrict__ seq_start,
                                                               const int* __restrict__ slots, T* __restrict__ out) {
    constexpr int N = 16 / (int)sizeof(T), TAPS = 4, KEEP = TAPS - 1;
    rdl_grid_wait();
    rdl_grid_launch_dependents();
    const int t0 = blockIdx.x * CONV_RUN, c0 = (blockIdx.y * blockDim.x + threadIdx.x) * N;
    if (c0 >= channels) return;
    auto load = [&](const T* p, float (&f)[N]) {
#pragma unroll
        for (int i = 0; i < N; i += 4) {
            float g[4];
            rn_load4(p + i, g);
            f[i] = g[0]; f[i + 1] = g[1]; f[i + 2] = g[2]; f[i + 3] = g[3];
        }
    };
    auto store = [&](int t, const float (&f)[N]) {
#pragma unroll
        for (int i = 0; i < N; i += 4) {
            const float g[4] = {f[i], f[i + 1], f[i + 2], f[i + 3]};
            rn_store4(out + (long long)t * channels + c0 + i, g);
        }
    };
    float x[CONV_RUN + KEEP][N], wt[TAPS][N], bias[N];
#pragma unroll
    for (int i = 0; i < CONV_RUN + KEEP; ++i) {            // rows t0 - 3 .. t0 + 3; which of them are a row's own inputs shows below
        const int t = t0 + i - KEEP;
        if (t >= 0 && t < n_rows) load(in + (long long)t * in_stride + c0, x[i]);
    }
#pragma unroll
    for (int j = 0; j < TAPS; ++j) {                       // the weights lie channel by channel
        float f[N];
        load(w + (long long)c0 * TAPS + j * N, f);
#pragma unroll
        for (int i = 0; i < N; ++i) wt[(j * N + i) % TAPS][(j * N + i) / TAPS] = f[i];
    }
#pragma unroll
    for (int i = 0; i < N; ++i) bias[i] = b ? rdl_load(b, c0 + i, b_dtype) : 0.f;
#pragma unroll
    for (int u = 0; u < CONV_RUN; ++u) {
        const int t = t0 + u;
        if (t >= n_rows) break;
        const int p = tok_pos[t];
        float acc[N];
#pragma unroll
        for (int i = 0; i < N; ++i) acc[i] = p < 0 ? 0.f : bias[i];
        if (p < 0) { store(t, acc); continue; }
        const int seq = tok_seq[t], row0 = seq_start[seq], r = t - row0;
        if (r >= KEEP) {
#pragma unroll
            for (int j = 0; j < TAPS; ++j)
#pragma unroll
                for (int i = 0; i < N; ++i) acc[i] = fmaf(wt[j][i], x[u + j][i], acc[i]);
            if (silu) {
#pragma unroll
                for (int i = 0; i < N; ++i) acc[i] = silu_exact(acc[i]);
            }
            store(t, acc);
        } else if (r == 0) {
            // a sequence's first rows, which read the slot, and the slot's new rows: channel by channel as above
            const int n = seq_start[seq + 1] - row0;
            float* st = state + (long long)slots[seq] * KEEP * channels;
            for (int i = 0; i < N; ++i) {
                const int c = c0 + i;
                float old[CONV_MAX_TAPS], wc[CONV_MAX_TAPS];
                for (int j = 0; j < TAPS; ++j) wc[j] = to_float(w[(long long)c * TAPS + j]);
                for (int j = 0; j < KEEP; ++j) old[j] = p > 0 ? st[(long long)j * channels + c] : 0.f;
                const float bc = b ? rdl_load(b, c, b_dtype) : 0.f;
                for (int rr = 0; rr < min(n, KEEP); ++rr) conv_row<T>(in, in_stride, row0, rr, p, c, channels, TAPS, wc, bc, silu, old, out);
                for (int j = 0; j < KEEP; ++j) {
                    const int src = n - KEEP + j;
                    float v;
                    if (src >= 0) v = to_float(in[(long long)(row0 + src) * in_stride + c]);
                    else v = p + src < 0 ? 0.f : old[KEEP + src];
                    st[(long long)j * channels + c] = v;
                }
            }
        }
    }
}

template <typename T>
__global__ void gated_residual_kernel(float* __restrict__ res, const T* __restrict__ gates, long long gates_stride,
                                      const void* __restrict__ bias_a, const void* __restrict__ bias_b, int bias_dtype,
                                      const T* __restrict__ a, const T* __restrict__ b1, const T* __restrict__ b2, int width, long long total) {
    rdl_grid_wait();
    rdl_grid_launch_dependents();
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x) {
        const long long t = idx / width;
        const int i = (int)(idx - t * width);
        const float ga = to_float(gates[t * gates_stride + i]) + rdl_load(bias_a, i, bias_dtype);
        float sum = to_float(a[idx]) / (1.0f + expf(-ga));
        if (b1) {
            const float gb = to_float(gates[t * gates_stride + width + i]) + rdl_load(bias_b, i, bias_dtype);
            float f = to_float(b1[idx]);
            if (b2) f += to_float(b2[idx]);
            sum += f / (1.0f + expf(-gb));
        }
        res[idx] += sum;
    }
}

// the same sum for bfloat16 rows whose width is a multiple of 8: eight elements a thread, 16-byte accesses, one division
// by the width a thread instead of a 64-bit one an element; every element goes through the same operations as above
__global__ void __launch_bounds__(256) gated_residual_vec_kernel(float* __restrict__ res, const __nv_bfloat16* __restrict__ gates, long long gates_stride,
                                                                 const void* __restrict__ bias_a, const void* __restrict__ bias_b, int bias_dtype,
                                                                 const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b1,
                                                                 const __nv_bfloat16* __restrict__ b2, int width, int groups) {
    rdl_grid_wait();
    rdl_grid_launch_dependents();
    const int per_row = width >> 3;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < groups; v += gridDim.x * blockDim.x) {
        const int t = v / per_row, i = (v - t * per_row) << 3;
        const long long idx = (long long)t * width + i;
        const uint4 ga4 = *reinterpret_cast<const uint4*>(gates + t * gates_stride + i);
        const uint4 a4 = *reinterpret_cast<const uint4*>(a + idx);
        uint4 gb4 = make_uint4(0, 0, 0, 0), b14 = gb4, b24 = gb4;
        if (b1) {
            gb4 = *reinterpret_cast<const uint4*>(gates + t * gates_stride + width + i);
            b14 = *reinterpret_cast<const uint4*>(b1 + idx);
            if (b2) b24 = *reinterpret_cast<const uint4*>(b2 + idx);
        }
        float4 r0 = *reinterpret_cast<const float4*>(res + idx), r1 = *reinterpret_cast<const float4*>(res + idx + 4);
        const __nv_bfloat16* gav = reinterpret_cast<const __nv_bfloat16*>(&ga4);
        const __nv_bfloat16* gbv = reinterpret_cast<const __nv_bfloat16*>(&gb4);
        const __nv_bfloat16* av = reinterpret_cast<const __nv_bfloat16*>(&a4);
        const __nv_bfloat16* b1v = reinterpret_cast<const __nv_bfloat16*>(&b14);
        const __nv_bfloat16* b2v = reinterpret_cast<const __nv_bfloat16*>(&b24);
        float o[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float ga = __bfloat162float(gav[e]) + rdl_load(bias_a, i + e, bias_dtype);
            float sum = __bfloat162float(av[e]) / (1.0f + expf(-ga));
            if (b1) {
                const float gb = __bfloat162float(gbv[e]) + rdl_load(bias_b, i + e, bias_dtype);
                float f = __bfloat162float(b1v[e]);
                if (b2) f += __bfloat162float(b2v[e]);
                sum += f / (1.0f + expf(-gb));
            }
            o[e] += sum;
        }
        *reinterpret_cast<float4*>(res + idx) = make_float4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<float4*>(res + idx + 4) = make_float4(o[4], o[5], o[6], o[7]);
    }
}

template <typename T>
__global__ void activation_kernel(T* __restrict__ x, long long total, int act) {
    rdl_grid_wait();
    rdl_grid_launch_dependents();
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += (long long)gridDim.x * blockDim.x) {
        const float v = to_float(x[idx]);
        float o;
        switch (act) {
            case RDL_UNARY_RELU2: { const float r = fmaxf(v, 0.f); o = r * r; break; }
            case RDL_UNARY_SILU: o = silu_exact(v); break;
            default: o = v;
        }
        x[idx] = from_float<T>(o);
    }
}

}  // namespace

extern "C" int rdl_norm_shift(const float* x, const void* w, int w_dtype, float eps, const void* shift, int shift_dtype, float* state,
                              const int* tok_seq, const int* tok_pos, const int* seq_start, const int* slots, void* normed, void* mixed,
                              int out_dtype, int n_rows, int width, void* stream) {
    RDL_REQUIRE(rdl_valid_dtype(out_dtype) && rdl_valid_dtype(w_dtype) && rdl_valid_dtype(shift_dtype), "norm_shift: bad dtype");
    RDL_REQUIRE(x && w && shift && state && tok_seq && tok_pos && seq_start && slots && normed && mixed && width > 0 && n_rows >= 0,
                "norm_shift: bad arguments");
    if (n_rows == 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 grid(n_rows), block(width <= 512 ? 64 : (width <= 2048 ? 128 : 256));
    if (width <= 8192) {                     // a thread's share of a row fits its registers
        cudaError_t e;
#define NORM_SHIFT_LAUNCH(T, N)                                                                                                          \
    rdl_launch(norm_shift_row_kernel<T, N>, grid, block, 0, st, x, w, w_dtype, eps, shift, shift_dtype, state, tok_seq, tok_pos, seq_start, \
               slots, (T*)normed, (T*)mixed, width)
#define NORM_SHIFT_BY_DEPTH(T) (width <= 512 ? NORM_SHIFT_LAUNCH(T, 8) : width <= 4096 ? NORM_SHIFT_LAUNCH(T, 16) : NORM_SHIFT_LAUNCH(T, 32))
        if (out_dtype == RDL_BF16) e = NORM_SHIFT_BY_DEPTH(__nv_bfloat16);
        else e = NORM_SHIFT_BY_DEPTH(float);
#undef NORM_SHIFT_BY_DEPTH
#undef NORM_SHIFT_LAUNCH
        RDL_CHECK_EX(e, "norm_shift");
        return 0;
    }
    if (out_dtype == RDL_BF16)
        RDL_CHECK_EX(rdl_launch(norm_shift_kernel<__nv_bfloat16>, grid, block, 0, st, x, w, w_dtype, eps, shift, shift_dtype, state, tok_seq, tok_pos,
                                seq_start, slots, (__nv_bfloat16*)normed, (__nv_bfloat16*)mixed, width), "norm_shift");
    else
        RDL_CHECK_EX(rdl_launch(norm_shift_kernel<float>, grid, block, 0, st, x, w, w_dtype, eps, shift, shift_dtype, state, tok_seq, tok_pos,
                                seq_start, slots, (float*)normed, (float*)mixed, width), "norm_shift");
    return 0;
}

extern "C" int rdl_short_conv(const void* in, long long in_stride, int dtype, int channels, int taps, const void* w, int w_dtype,
                              const void* bias, int silu, float* state, const int* tok_seq, const int* tok_pos, const int* seq_start,
                              const int* slots, void* out, int n_rows, int n_seqs, void* stream) {
    RDL_REQUIRE(rdl_valid_dtype(dtype) && rdl_valid_dtype(w_dtype), "short_conv: bad dtype");
    RDL_REQUIRE(in && w && tok_seq && tok_pos && seq_start && slots && out && channels > 0 && in_stride >= channels && n_rows >= 0,
                "short_conv: bad arguments");
    RDL_REQUIRE(taps >= 1 && taps <= CONV_MAX_TAPS, "short_conv: %d taps, the kernel takes 1 to %d", taps, CONV_MAX_TAPS);
    RDL_REQUIRE(state || taps == 1, "short_conv: more than one tap needs the slots' state");
    if (n_rows == 0) return 0;
    RDL_REQUIRE((channels + 127) / 128 <= 65535, "short_conv: too many channels for one grid");
    const dim3 grid(n_rows, (channels + 127) / 128), block(128);
    cudaStream_t st = (cudaStream_t)stream;
    const int piece = dtype == RDL_BF16 ? 8 : 4;
    // Runs of four rows where there are many and most are not a sequence's first ones, which one thread takes for eight channels one
    // after the other.  Microseconds, a thread a channel / runs of four, rows in sequences of L:
    //   2,304 channels   512 rows    L 1 20 / 40    L 4 14 / 18    L 8 15 / 16    L 32 16 / 13    one 15 / 11       256 rows, one 10 / 11
    //                    4,096 rows  L 1 150 / 216  L 4 82 / 79    L 8 82 / 55    L 32 84 / 38    one 82 / 30
    //   6,144 channels   512 rows    L 1 46 / 77    L 4 30 / 31    L 8 31 / 24    L 32 32 / 19    one 32 / 16
    if (n_rows >= 512 && n_rows >= 8LL * n_seqs && taps == 4 && w_dtype == dtype && channels % piece == 0 && in_stride % piece == 0 && aligned16(in) && aligned16(w) && aligned16(out)) {
        const dim3 runs((n_rows + CONV_RUN - 1) / CONV_RUN, (channels / piece + 127) / 128);
        if (dtype == RDL_BF16)
            RDL_CHECK_EX(rdl_launch(short_conv4_rows_kernel<__nv_bfloat16>, runs, block, 0, st, (const __nv_bfloat16*)in, in_stride, n_rows, channels,
                                    (const __nv_bfloat16*)w, bias, w_dtype, silu, state, tok_seq, tok_pos, seq_start, slots, (__nv_bfloat16*)out), "short_conv");
        else
            RDL_CHECK_EX(rdl_launch(short_conv4_rows_kernel<float>, runs, block, 0, st, (const float*)in, in_stride, n_rows, channels, (const float*)w, bias,
                                    w_dtype, silu, state, tok_seq, tok_pos, seq_start, slots, (float*)out), "short_conv");
        return 0;
    }
    if (dtype == RDL_BF16)
        RDL_CHECK_EX(rdl_launch(short_conv_kernel<__nv_bfloat16>, grid, block, 0, st, (const __nv_bfloat16*)in, in_stride, channels, taps, w, w_dtype,
                                bias, silu, state, tok_seq, tok_pos, seq_start, slots, (__nv_bfloat16*)out), "short_conv");
    else
        RDL_CHECK_EX(rdl_launch(short_conv_kernel<float>, grid, block, 0, st, (const float*)in, in_stride, channels, taps, w, w_dtype, bias, silu,
                                state, tok_seq, tok_pos, seq_start, slots, (float*)out), "short_conv");
    return 0;
}

extern "C" int rdl_gated_residual_add(float* res, const void* gates, long long gates_stride, const void* bias_a, const void* bias_b,
                                      int bias_dtype, const void* a, const void* b1, const void* b2, int dtype, int n_rows, int width,
                                      void* stream) {
    RDL_REQUIRE(rdl_valid_dtype(dtype) && rdl_valid_dtype(bias_dtype), "gated_residual_add: bad dtype");
    RDL_REQUIRE(res && gates && bias_a && a && width > 0 && n_rows >= 0 && (!b1 || bias_b) && (b1 || !b2), "gated_residual_add: bad arguments");
    RDL_REQUIRE(gates_stride >= (b1 ? 2LL : 1LL) * width, "gated_residual_add: the gates' rows are narrower than the branches");
    if (n_rows == 0) return 0;
    const long long total = (long long)n_rows * width;
    const dim3 grid((unsigned)min((total + 255) / 256, 65535LL * 16)), block(256);
    cudaStream_t st = (cudaStream_t)stream;
    const bool aligned = (((uintptr_t)res | (uintptr_t)gates | (uintptr_t)a | (uintptr_t)b1 | (uintptr_t)b2) & 15) == 0;
    if (dtype == RDL_BF16 && width % 8 == 0 && gates_stride % 8 == 0 && aligned && total / 8 < (1LL << 31)) {
        const int groups = (int)(total / 8);
        RDL_CHECK_EX(rdl_launch(gated_residual_vec_kernel, dim3((unsigned)min((groups + 255) / 256, 148 * 16)), block, 0, st, res, (const __nv_bfloat16*)gates,
                                gates_stride, bias_a, bias_b, bias_dtype, (const __nv_bfloat16*)a, (const __nv_bfloat16*)b1, (const __nv_bfloat16*)b2, width, groups),
                     "gated_residual_add");
    } else if (dtype == RDL_BF16)
        RDL_CHECK_EX(rdl_launch(gated_residual_kernel<__nv_bfloat16>, grid, block, 0, st, res, (const __nv_bfloat16*)gates, gates_stride, bias_a, bias_b,
                                bias_dtype, (const __nv_bfloat16*)a, (const __nv_bfloat16*)b1, (const __nv_bfloat16*)b2, width, total),
                     "gated_residual_add");
    else
        RDL_CHECK_EX(rdl_launch(gated_residual_kernel<float>, grid, block, 0, st, res, (const float*)gates, gates_stride, bias_a, bias_b, bias_dtype,
                                (const float*)a, (const float*)b1, (const float*)b2, width, total), "gated_residual_add");
    return 0;
}

extern "C" int rdl_activation_inplace(void* x, int dtype, long long total, int act, void* stream) {
    RDL_REQUIRE(rdl_valid_dtype(dtype) && x && total >= 0, "activation_inplace: bad arguments");
    RDL_REQUIRE(act == RDL_UNARY_RELU2 || act == RDL_UNARY_SILU, "activation_inplace: unknown activation %d", act);
    if (total == 0) return 0;
    const dim3 grid((unsigned)min((total + 255) / 256, 65535LL * 16)), block(256);
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == RDL_BF16) RDL_CHECK_EX(rdl_launch(activation_kernel<__nv_bfloat16>, grid, block, 0, st, (__nv_bfloat16*)x, total, act), "activation_inplace");
    else RDL_CHECK_EX(rdl_launch(activation_kernel<float>, grid, block, 0, st, (float*)x, total, act), "activation_inplace");
    return 0;
}
