// Plain attention over new tokens and a paged cache: float arithmetic throughout, a fixed order of
// operations that depends only on absolute positions.  It is the attention of the 32-bit path (prefill
// and decode alike) and the reference the fast kernels are tested against.  Two kernels: one warp per
// (query token, head), any type and head size; and, for float rows that 16-byte loads can take, one block per
// (query token, head) whose eight warps share the keys (attention_f32_kernel below).
//
// For query position p of a sequence and query head h (kv head g = h / (n_heads / n_kv_heads),
// reference: rustml/core/main/src/core/tensor/ops.rs:980-987):
//   s_j = (q_h . k_g,j) * score_scale                    attention.rs:413-416
//   s_j = cap * tanh(s_j / cap)            if cap > 0    attention.rs:419-423
//   keys kept: j <= p and (window == 0 or p - j < window)  ops.rs:905-922, :932-952
//   (with chunk: j / chunk == p / chunk as well; with rel_bias: s_j += rel_bias[h][min(p - j, rel_len - 1)]; the reference has neither)
//   a = softmax_j(s)                                      ops.rs:598-608
//   (with sinks: the denominator also holds exp(sinks[h]); the reference has none)
//   (with sigmoid_bias: a_j = sigmoid(s_j + sigmoid_bias[h]) for the keys kept, not normalised; the reference has none)
//   o_h = sum_j a_j v_g,j                                 attention.rs:442-446
// (paths within rustml/; attention.rs = nn/main/src/core/attention.rs).  The window holds for
// single-token steps too, which the reference's cached path skips (attention.rs:429).
//
// Keys at positions below seq_cached[s] are read from the cache, later ones from the step's
// own packed key/value rows.
#include "api.h"
#include "common.cuh"
#include "launch.cuh"

#define PLAIN_MAX_CHUNKS 32  // head_dim <= 1024 in the wide form (the rows of a latent cache are wider than ordinary heads); 16 otherwise

template <typename T, int CHUNKS>
__global__ void attention_plain_kernel(AttentionArgs a) {
    const int warps_per_block = blockDim.x >> 5;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * warps_per_block + warp;
    if (item >= (long long)a.n_tokens * a.n_heads) return;
    const int t = (int)(item / a.n_heads), h = (int)(item % a.n_heads);
    const int hd = a.head_dim;
    const int g = h / (a.n_heads / a.n_kv_heads);
    const int seq = a.tok_seq[t], p = a.tok_pos[t];
    if (p < 0) return;  // a padding row of a fixed-size batch
    const int cached = a.seq_cached[seq];
    const int new_row0 = a.seq_start[seq] - a.seq_past[seq];  // packed row of position j is new_row0 + j
    const int* table = a.tables ? a.tables + (long long)seq * a.table_width : nullptr;
    const T* q = (const T*)a.q + (long long)t * a.q_stride + (long long)h * hd;
    const int lo = rdl_first_key(p, a.window, a.chunk);
    const float* rel = a.rel_bias ? a.rel_bias + (long long)h * a.rel_len : nullptr;

    float acc[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) acc[c] = 0.f;
    float m = -INFINITY, l = 0.f;
    const bool sig = a.sigmoid_bias != nullptr;
    const float sig_bias = sig ? a.sigmoid_bias[h] : 0.f;

    for (int jb = (lo / 32) * 32; jb <= p; jb += 32) {
        const int j = jb + lane;
        const bool valid = j >= lo && j <= p;
        const T* kp = nullptr;
        const T* vp = nullptr;
        float s = -INFINITY;
        int sw = -1;   // place of the row in its cache page (rows there are stored swizzled); -1: a packed new row
        if (valid) {
            if (j < cached) {
                const long long off = rdl_cache_offset(table, j, a.page_size, a.ring_pages, a.n_kv_heads, g, hd);
                kp = (const T*)a.k_cache + off;
                vp = (const T*)a.v_cache + off;
                sw = j % a.page_size;
            } else {
                const long long off = (long long)(new_row0 + j) * a.kv_stride + (long long)g * hd;
                kp = (const T*)a.k_new + off;
                vp = (const T*)a.v_new + off;
            }
            float d = 0.f;
            for (int i = 0; i < hd; ++i) d = fmaf(to_float(q[i]), to_float(kp[sw < 0 ? i : rdl_cache_col<T>(sw, i, hd)]), d);
            d *= a.score_scale;
            if (a.softcap > 0.f) d = a.softcap * tanhf(d / a.softcap);
            if (rel) d += rel[min(p - j, a.rel_len - 1)];
            s = d;
        }
        float pj;
        if (sig) {
            pj = valid ? 1.0f / (1.0f + expf(-(s + sig_bias))) : 0.f;
        } else {
            const float m_new = fmaxf(m, warp_max(s));
            const float corr = expf(m - m_new);   // exp(-inf) = 0 on the first block
            pj = valid ? expf(s - m_new) : 0.f;
            l = l * corr + warp_sum(pj);
            m = m_new;
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) acc[c] *= corr;
        }
        const unsigned long long vaddr = (unsigned long long)vp;
        for (int jj = 0; jj < 32; ++jj) {
            const int jk = jb + jj;
            if (jk < lo || jk > p) continue;  // uniform over the warp
            const float pw = __shfl_sync(0xffffffffu, pj, jj);
            const unsigned lo32 = __shfl_sync(0xffffffffu, (unsigned)(vaddr & 0xffffffffull), jj);
            const unsigned hi32 = __shfl_sync(0xffffffffu, (unsigned)(vaddr >> 32), jj);
            const int vsw = __shfl_sync(0xffffffffu, sw, jj);
            const T* vrow = (const T*)(((unsigned long long)hi32 << 32) | lo32);
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
                const int d = c * 32 + lane;
                if (d < hd) acc[c] = fmaf(pw, to_float(vrow[vsw < 0 ? d : rdl_cache_col<T>(vsw, d, hd)]), acc[c]);
            }
        }
    }
    T* o = (T*)a.out + (long long)t * a.out_stride + (long long)h * hd;
    // a sink is a logit without key or value: it joins the denominator once, neither scaled nor capped
    if (a.sinks) {
        const float sink = a.sinks[h];
        const float m_all = fmaxf(m, sink);
        const float corr = expf(m - m_all);
        l = l * corr + expf(sink - m_all);
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) acc[c] *= corr;
    }
    const float inv = sig ? 1.0f : 1.0f / l;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
        const int d = c * 32 + lane;
        if (d < hd) o[d] = from_float<T>(acc[c] * inv);
    }
}

// ---------------------------------------------------------------------------------------------
// The same for float rows whose head size is a multiple of four (up to 512): a block of eight warps per (query token, head).
//
// What bounds it is the latency of reading a few dozen to a few hundred keys; the one-warp kernel reads a key's row four bytes at a
// time in one lane, a chain of head_dim fused multiply-adds behind each load (164 us a layer for 45 queries or 2 single
// tokens over 40 keys of 256).  Here the warps take the groups of four absolute positions in turn, so that a short context
// is short for every warp.  Eight lanes share a key (16-byte loads, four keys at a time, sums by exchanges among the eight), the
// values are read by whole warps, and the warps' sums meet in shared memory in warp order.  The order of operations depends on
// positions and head size alone, not on the step, so logits stay bit-equal however a request is cut.
// What keeps it fast behind long contexts is the number of loads in flight: where all 32 of a warp's positions are visible the
// loops have fixed lengths, elsewhere what is left over does not come one by one, and the registers leave room for four blocks a
// multiprocessor (heads of up to 64; three up to 128).  A test of every position's address between the loads instead kept the
// next load behind the test.  One token, microseconds with 32 neighbouring positions a warp / with that test / now:
//     heads of 256:  40 keys 10.2 / 6.6 / 5.5    250 11.0 / 15.9 / 11.8    500 19.0 / 29.0 / 18.1    1,000 35.6 / 54.8 / 32.7    8,000 310 / 476 / 280
//     heads of 128:  40 keys 10.7 / 6.4 / 4.8    250 11.0 / 15.5 /  8.6    500 19.5 / 28.4 / 13.8    1,000 36.4 / 54.3 / 25.0    8,000 290 / 445 / 190
// and a prompt of 1,500 tokens 1,399 / 1,823 / 1,245 (8 heads of 256), 407 / 424 / 368 (6 of 32).  Contexts of 210 to 255 keys
// of 256 are what neighbouring positions still do better (by 3 to 8 %: there the last places come in fewer trips).
// ---------------------------------------------------------------------------------------------
constexpr int PF_WARPS = 8;

// NC: 32-value slices of a head (head_dim <= 32 NC).  Wider heads are left to the compiler (bounds of one block: 0.6 of the speed).
template <int NC>
__global__ void __launch_bounds__(PF_WARPS * 32, NC <= 2 ? 4 : NC == 4 ? 3 : 0) attention_f32_kernel(AttentionArgs a) {
    constexpr int VC = (NC + 3) / 4;                       // 128-value slices of a head
    __shared__ float4 part[PF_WARPS][VC][32];
    __shared__ float part_m[PF_WARPS], part_l[PF_WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane & 7;
    const int t = blockIdx.x, h = blockIdx.y;
    const int hd = a.head_dim, chunks = hd / 4;            // 16-byte chunks of a row
    const int g = h / (a.n_heads / a.n_kv_heads);
    rdl_grid_wait();
    rdl_grid_launch_dependents();
    const int seq = a.tok_seq[t], p = a.tok_pos[t];
    if (p < 0) return;  // a padding row of a fixed-size batch
    const int cached = a.seq_cached[seq];
    const int new_row0 = a.seq_start[seq] - a.seq_past[seq];  // packed row of position j is new_row0 + j
    const int* table = a.tables ? a.tables + (long long)seq * a.table_width : nullptr;
    const int lo = rdl_first_key(p, a.window, a.chunk);
    const float* rel = a.rel_bias ? a.rel_bias + (long long)h * a.rel_len : nullptr;
    const bool sig = a.sigmoid_bias != nullptr;
    const float sig_bias = sig ? a.sigmoid_bias[h] : 0.f;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);

    // slice c of a lane: chunk 8 c + sub of the query
    float4 q[NC];
    const float4* q4 = reinterpret_cast<const float4*>((const float*)a.q + (long long)t * a.q_stride + (long long)h * hd);
#pragma unroll
    for (int c = 0; c < NC; ++c) q[c] = 8 * c + sub < chunks ? q4[8 * c + sub] : zero4;
    float4 acc[VC];
#pragma unroll
    for (int c = 0; c < VC; ++c) acc[c] = zero4;
    float m = -INFINITY, l = 0.f;

    // Superblock sb: 256 positions; this warp's 32 of them are the groups of four positions 4 (8 g + warp) .. + 3, g = 0..7, lane
    // 4 g + i holding number i of group g.
    for (int sb = lo / (32 * PF_WARPS); sb * 32 * PF_WARPS <= p; ++sb) {
        const int j_warp = sb * 32 * PF_WARPS + 4 * warp;
        if (j_warp > p) break;                              // no position of this warp's is left
        // lane: where its key lies (a row of the cache, stored swizzled, or a packed new row)
        const int j = j_warp + 4 * PF_WARPS * (lane >> 2) + (lane & 3);
        const bool valid = j >= lo && j <= p;
        unsigned long long k_at = 0, v_at = 0;
        int sw = -1;                                        // place of the row in its cache page; -1: a packed new row
        if (valid) {
            if (j < cached) {
                const long long off = rdl_cache_offset(table, j, a.page_size, a.ring_pages, a.n_kv_heads, g, hd);
                k_at = (unsigned long long)((const float*)a.k_cache + off);
                v_at = (unsigned long long)((const float*)a.v_cache + off);
                sw = j % a.page_size;
            } else {
                const long long off = (long long)(new_row0 + j) * a.kv_stride + (long long)g * hd;
                k_at = (unsigned long long)((const float*)a.k_new + off);
                v_at = (unsigned long long)((const float*)a.v_new + off);
            }
        }
        // the groups with a visible position, and its places: neighbours, since positions rise with the lane
        const unsigned seen = __ballot_sync(0xffffffffu, valid);
        const bool whole = seen == 0xffffffffu;
        const int first = seen ? __ffs(seen) - 1 : 32, last = seen ? 31 - __clz(seen) : -1;
        // scores: a group of four keys a pass, eight lanes a key
        float s = 0.f;
        auto score = [&](int pass) {
            const int key = pass * 4 + (lane >> 3);
            const float4* k4 = reinterpret_cast<const float4*>(__shfl_sync(0xffffffffu, k_at, key));
            const int ksw = __shfl_sync(0xffffffffu, sw, key);
            float4 kv[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int i = 8 * c + sub;
                kv[c] = k4 && i < chunks ? k4[ksw < 0 ? i : rdl_swizzled_chunk(ksw, i, chunks)] : zero4;
            }
            float d = 0.f;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                d = fmaf(q[c].x, kv[c].x, d);
                d = fmaf(q[c].y, kv[c].y, d);
                d = fmaf(q[c].z, kv[c].z, d);
                d = fmaf(q[c].w, kv[c].w, d);
            }
            d += __shfl_xor_sync(0xffffffffu, d, 1);
            d += __shfl_xor_sync(0xffffffffu, d, 2);
            d += __shfl_xor_sync(0xffffffffu, d, 4);
            const float mine = __shfl_sync(0xffffffffu, d, (lane & 3) * 8);      // key pass * 4 + (lane & 3)
            if ((lane >> 2) == pass) s = mine;
        };
        if (whole) {
#pragma unroll 2
            for (int pass = 0; pass < 8; ++pass) score(pass);
        } else {
#pragma unroll 2
            for (int pass = first >> 2; pass <= last >> 2; ++pass) score(pass);
        }
        s *= a.score_scale;
        if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
        if (rel && valid) s += rel[min(p - j, a.rel_len - 1)];
        float pj;
        if (sig) {
            pj = valid ? 1.0f / (1.0f + expf(-(s + sig_bias))) : 0.f;
        } else {
            const float m_new = fmaxf(m, warp_max(valid ? s : -INFINITY));
            const float corr = m == m_new ? 1.f : expf(m - m_new);                // exp(-inf) = 0 on the first block
            pj = !valid || s == -INFINITY ? 0.f : expf(s - m_new);
            l = l * corr + warp_sum(pj);
            m = m_new;
#pragma unroll
            for (int c = 0; c < VC; ++c) { acc[c].x *= corr; acc[c].y *= corr; acc[c].z *= corr; acc[c].w *= corr; }
        }
        // values: the visible places in turn, whole warps
        auto add = [](float4& sum, float w, const float4& v) {
            sum.x = fmaf(w, v.x, sum.x);
            sum.y = fmaf(w, v.y, sum.y);
            sum.z = fmaf(w, v.z, sum.z);
            sum.w = fmaf(w, v.w, sum.w);
        };
        auto value = [&](int key) {
            const float pw = __shfl_sync(0xffffffffu, pj, key);
            const float4* v4 = reinterpret_cast<const float4*>(__shfl_sync(0xffffffffu, v_at, key));
            const int vsw = __shfl_sync(0xffffffffu, sw, key);
#pragma unroll
            for (int c = 0; c < VC; ++c) {
                const int i = 32 * c + lane;
                const float4 v = i < chunks ? v4[vsw < 0 ? i : rdl_swizzled_chunk(vsw, i, chunks)] : zero4;
                add(acc[c], pw, v);
            }
        };
        if (whole) {
#pragma unroll 8
            for (int key = 0; key < 32; ++key) value(key);
        } else if constexpr (VC == 1) {
            // eight loads at a time to the end: what is left over does not come one by one (places beyond the last add 0 * 0)
#pragma unroll 1
            for (int key0 = first; key0 <= last; key0 += 8) {
                float4 v[8];
                float pw[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int key = key0 + u;
                    const bool there = key <= last;
                    const float w = __shfl_sync(0xffffffffu, pj, key);
                    const float4* v4 = reinterpret_cast<const float4*>(__shfl_sync(0xffffffffu, v_at, key));
                    const int vsw = __shfl_sync(0xffffffffu, sw, key);
                    v[u] = there && lane < chunks ? v4[vsw < 0 ? lane : rdl_swizzled_chunk(vsw, lane, chunks)] : zero4;
                    pw[u] = there ? w : 0.f;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) add(acc[0], pw[u], v[u]);
            }
        } else {
            int key = first;
#pragma unroll 2
            for (; key + 3 <= last; key += 4) {
#pragma unroll
                for (int u = 0; u < 4; ++u) value(key + u);
            }
            for (; key <= last; ++key) value(key);
        }
    }
#pragma unroll
    for (int c = 0; c < VC; ++c) part[warp][c][lane] = acc[c];
    if (lane == 0) { part_m[warp] = m; part_l[warp] = l; }
    __syncthreads();
    // the warps' sums, in warp order; the sink joins the denominator once, neither scaled nor capped
    float m_all = a.sinks ? a.sinks[h] : -INFINITY;
#pragma unroll
    for (int w = 0; w < PF_WARPS; ++w) m_all = fmaxf(m_all, part_m[w]);
    float f[PF_WARPS], l_all = 0.f;
#pragma unroll
    for (int w = 0; w < PF_WARPS; ++w) {
        f[w] = sig ? 1.f : (part_m[w] == m_all ? 1.f : expf(part_m[w] - m_all));
        l_all += part_l[w] * f[w];
    }
    if (a.sinks) l_all += expf(a.sinks[h] - m_all);
    const float inv = sig ? 1.0f : 1.0f / l_all;
    float* o = (float*)a.out + (long long)t * a.out_stride + (long long)h * hd;
    for (int i = threadIdx.x; i < hd; i += PF_WARPS * 32) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < PF_WARPS; ++w) v = fmaf(reinterpret_cast<const float*>(part[w])[i], f[w], v);
        o[i] = v * inv;
    }
}

template <int NC>
static cudaError_t launch_attention_f32(const AttentionArgs& a, cudaStream_t st) {
    return rdl_launch(attention_f32_kernel<NC>, dim3(a.n_tokens, a.n_heads), dim3(PF_WARPS * 32), 0, st, a);
}

int rdl_check_attention_args(const AttentionArgs* a, const char* who) {
    RDL_REQUIRE(rdl_valid_dtype(a->dtype), "%s: bad dtype %d", who, a->dtype);
    RDL_REQUIRE(a->n_tokens >= 0 && a->n_seqs >= 0, "%s: bad token or sequence count", who);
    RDL_REQUIRE(a->n_heads > 0 && a->n_kv_heads > 0 && a->n_heads % a->n_kv_heads == 0,
                "%s: %d heads cannot share %d key/value heads", who, a->n_heads, a->n_kv_heads);
    RDL_REQUIRE(a->head_dim > 0, "%s: bad head_dim %d", who, a->head_dim);
    RDL_REQUIRE(a->window >= 0 && a->chunk >= 0 && a->softcap >= 0.f, "%s: window, chunk and soft-cap must not be negative", who);
    RDL_REQUIRE(!a->rel_bias || a->rel_len > 0, "%s: a distance bias needs at least one entry a head", who);
    RDL_REQUIRE(!(a->rel_bias && a->sigmoid_bias), "%s: sigmoid weights come without a distance bias", who);
    RDL_REQUIRE(a->q && a->out && a->tok_seq && a->tok_pos && a->seq_start && a->seq_past && a->seq_cached,
                "%s: missing query, output or batch description", who);
    RDL_REQUIRE(a->q_stride >= (long long)a->n_heads * a->head_dim && a->out_stride >= (long long)a->n_heads * a->head_dim,
                "%s: row strides smaller than a row", who);
    if (a->tables) {
        RDL_REQUIRE(a->k_cache && a->v_cache && a->page_size > 0 && a->ring_pages > 0 && a->ring_pages <= a->table_width,
                    "%s: cache given without storage or with bad paging (page_size=%d ring_pages=%d table_width=%d)", who,
                    a->page_size, a->ring_pages, a->table_width);
    }
    RDL_REQUIRE(a->tables || (a->k_new && a->v_new), "%s: neither a cache nor new keys and values", who);
    RDL_REQUIRE(!(a->sigmoid_bias && a->sinks), "%s: sigmoid weights have no denominator for sinks to join", who);
    return 0;
}

extern "C" int rdl_attention_plain(const AttentionArgs* a, void* stream) {
    if (int e = rdl_check_attention_args(a, "attention_plain")) return e;
    RDL_REQUIRE(a->head_dim <= 32 * PLAIN_MAX_CHUNKS, "attention_plain: head_dim %d exceeds %d", a->head_dim, 32 * PLAIN_MAX_CHUNKS);
    if (a->n_tokens == 0) return 0;
    // 16-byte loads: whole rows of chunks, on 16-byte boundaries (the choice rests on the model's layout, not on the step)
    auto quads = [](const void* p, long long stride) { return (uintptr_t)p % 16 == 0 && stride % 4 == 0; };
    if (a->dtype == RDL_F32 && a->head_dim % 4 == 0 && a->head_dim <= 512 && a->n_heads <= 65535 && quads(a->q, a->q_stride) &&
        (!a->tables || (quads(a->k_cache, 0) && quads(a->v_cache, 0))) && (!a->k_new || (quads(a->k_new, a->kv_stride) && quads(a->v_new, a->kv_stride)))) {
        cudaStream_t st = (cudaStream_t)stream;
        const int hd = a->head_dim;
        RDL_CHECK_EX(hd <= 32 ? launch_attention_f32<1>(*a, st) : hd <= 64 ? launch_attention_f32<2>(*a, st) : hd <= 128 ? launch_attention_f32<4>(*a, st)
                     : hd <= 256 ? launch_attention_f32<8>(*a, st) : launch_attention_f32<16>(*a, st), "attention_plain");
        return 0;
    }
    const int warps = 4;
    const long long items = (long long)a->n_tokens * a->n_heads;
    const unsigned blocks = (unsigned)((items + warps - 1) / warps);
    const bool wide = a->head_dim > 32 * 16;      // the accumulator of a head lives in registers: 16 or 32 values a lane
    if (a->dtype == RDL_BF16) {
        if (wide) attention_plain_kernel<__nv_bfloat16, PLAIN_MAX_CHUNKS><<<blocks, warps * 32, 0, (cudaStream_t)stream>>>(*a);
        else attention_plain_kernel<__nv_bfloat16, 16><<<blocks, warps * 32, 0, (cudaStream_t)stream>>>(*a);
    } else {
        if (wide) attention_plain_kernel<float, PLAIN_MAX_CHUNKS><<<blocks, warps * 32, 0, (cudaStream_t)stream>>>(*a);
        else attention_plain_kernel<float, 16><<<blocks, warps * 32, 0, (cudaStream_t)stream>>>(*a);
    }
    RDL_CHECK_LAUNCH("attention_plain");
    return 0;
}
