// Prefill attention in bfloat16: tiled, with an online softmax in float, soft-cap, causal and
// window masks, grouped heads, sequences of unequal length packed in one batch.  Keys and
// values of earlier steps are read from the paged cache, those of this step from the packed
// rows, chosen per key row.  Formulas as in attention_plain.cu.
//
// One block = 64 query rows of one sequence and one head (4 warps, 16 rows each); key tiles of
// 64 positions aligned to absolute multiples of 64; tiles wholly outside the window are skipped.
// Products run on the tensor cores (mma.sync m16n8k16, float accumulators); scores, tanh,
// exponentials, row maxima and row sums are float.
//
// A few new tokens behind a long past (a conversation's next turn) make few blocks with many keys each: 3 x 41 tokens of 8
// heads are 24 blocks that walk 640 to 720 keys one tile after the other.  There a cluster of two, four or eight blocks takes
// a query tile and head (attention_prefill_shared_kernel below).  Its rows are the same bits as the one block's: what a
// row's sums are made of, and in which order, depends on positions alone, not on what else is in the step.
#include "api.h"
#include "common.cuh"
#include "launch.cuh"

#include <algorithm>
#include <type_traits>

namespace {

constexpr int BM = 64, BN = 64, NTHREADS = 128;

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float tanh_fast(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

// shared tile [64 rows][HD] of bf16 in 16-byte chunks, chunk index swizzled by the row
template <int HD>
__device__ __forceinline__ int swizzled_chunk(int row, int chunk) {
    constexpr int CH = HD / 8;
    if (CH >= 8) return chunk ^ (row & 7);
    return chunk ^ ((row >> 1) & (CH - 1));
}
template <int HD>
__device__ __forceinline__ uint32_t tile_addr(uint32_t base, int row, int chunk) {
    return base + (uint32_t)((row * (HD / 8) + swizzled_chunk<HD>(row, chunk)) * 16);
}

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// this block's shared address `addr` as block `rank` of the cluster has it, and loads from such addresses
__device__ __forceinline__ uint32_t in_block(uint32_t addr, int rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void ld_cluster(uint32_t (&v)[4], uint32_t addr) {
    asm volatile("ld.shared::cluster.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr) : "memory");
}

constexpr float LOG2E = 1.4426950408889634f;
constexpr int MAX_RUNS = 8;

// What a block knows of its query tile, and what a thread knows of its two rows (w0 and w0 + 8 of the tile).
struct Tile {
    int h, g, seq, q0, row0, rows, past, cached, hd;
    int p_first, p_last, lo_first;                  // positions of the tile's rows, and the first key any of them sees
    int pr0, pr1, lo0, lo1;                         // the thread's rows: position and first key
    int pw_first, pw_last, low_first, low_last;     // its warp's rows: the same, first and last
    const int* table;
    int ksteps;
    float inv_cap;
    const float* rel;                               // distance bias of the head: entry n for distance n, the last one for all beyond
    __device__ __forceinline__ Tile(const AttentionArgs& a, int tile, int head) {
        h = head;
        seq = a.tile_seq[tile]; q0 = a.tile_q0[tile];
        row0 = a.seq_start[seq];
        rows = min(BM, a.seq_start[seq + 1] - row0 - q0);
        past = a.seq_past[seq]; cached = a.seq_cached[seq];
        hd = a.head_dim;
        g = h / (a.n_heads / a.n_kv_heads);
        table = a.tables ? a.tables + (long long)seq * a.table_width : nullptr;
        ksteps = (hd + 15) / 16;
        inv_cap = a.softcap > 0.f ? 1.0f / a.softcap : 0.f;
        rel = a.rel_bias ? a.rel_bias + (long long)h * a.rel_len : nullptr;
        const int warp = threadIdx.x >> 5, quad = (threadIdx.x & 31) >> 2;
        p_first = past + q0; p_last = past + q0 + rows - 1;
        lo_first = rdl_first_key(p_first, a.window, a.chunk);
        pr0 = p_first + warp * 16 + quad; pr1 = pr0 + 8;
        pw_first = p_first + warp * 16; pw_last = pw_first + 15;
        lo0 = rdl_first_key(pr0, a.window, a.chunk); lo1 = rdl_first_key(pr1, a.window, a.chunk);
        low_first = rdl_first_key(pw_first, a.window, a.chunk); low_last = rdl_first_key(pw_last, a.window, a.chunk);
    }
    // the warp's rows see something of the key tile from kv0 on
    __device__ __forceinline__ bool sees(int kv0) const { return kv0 <= pw_last && kv0 + BN - 1 >= low_first; }
};

template <int HD>
__device__ __forceinline__ void load_queries(const AttentionArgs& a, const Tile& t, unsigned char* gQ) {
    constexpr int CH = HD / 8;          // 16-byte chunks per row
    const __nv_bfloat16* qbase = (const __nv_bfloat16*)a.q;
    for (int idx = threadIdx.x; idx < BM * CH; idx += NTHREADS) {
        const int r = idx / CH, c = idx - r * CH;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (r < t.rows && c * 8 < t.hd)
            v = *(const uint4*)(qbase + (long long)(t.row0 + t.q0 + r) * a.q_stride + (long long)t.h * t.hd + c * 8);
        *(uint4*)(gQ + (r * CH + swizzled_chunk<HD>(r, c)) * 16) = v;
    }
}

// Where a key tile that lies in one page has its rows in the cache (0: it does not, or is not in the cache): looked up once a tile.
__device__ __forceinline__ long long page_place(const AttentionArgs& a, const Tile& t, int kv0) {
    return a.page_size % BN == 0 && kv0 < t.cached ? rdl_cache_offset(t.table, kv0, a.page_size, a.ring_pages, a.n_kv_heads, t.g, t.hd) : 0;
}

// Chunks c0 .. c0 + cn - 1 (cn a constant where CN is not 0) of the 64 rows of keys (which == 0) or values (which == 1) from position kv0 on,
// on their way to shared memory: asynchronous 16-byte copies that bypass the registers, rows beyond the sequence and
// chunks beyond head_dim filled with zeros.  to(row, chunk): the shared address.  page_at: page_place of kv0.
template <int CN, typename To>
__device__ __forceinline__ void copy_rows(const AttentionArgs& a, const Tile& t, int kv0, long long page_at, int which, int c0, int count, To to) {
    const int cn = CN ? CN : count;
    const __nv_bfloat16* cache_base = (const __nv_bfloat16*)(which ? a.v_cache : a.k_cache);
    const __nv_bfloat16* new_base = (const __nv_bfloat16*)(which ? a.v_new : a.k_new);
    const bool whole_pages = a.page_size % BN == 0;
    const __nv_bfloat16* page = cache_base + page_at;
#pragma unroll 4
    for (int idx = threadIdx.x; idx < BN * cn; idx += NTHREADS) {
        const int r = idx / cn, c = c0 + idx - r * cn;
        const int j = kv0 + r;
        const __nv_bfloat16* src = (const __nv_bfloat16*)a.q;       // any valid address: nothing is read when the size is 0
        uint32_t bytes = 0;
        if (j <= t.p_last && c * 8 < t.hd) {
            bytes = 16;
            if (j < t.cached)   // chunks of a cache row are stored swizzled by the row's place in its page
                src = whole_pages ? page + (long long)r * t.hd + rdl_swizzled_chunk(r, c, t.hd / 8) * 8
                                  : cache_base + rdl_cache_offset(t.table, j, a.page_size, a.ring_pages, a.n_kv_heads, t.g, t.hd) +
                                        rdl_swizzled_chunk(j % a.page_size, c, t.hd / 8) * 8;
            else
                src = new_base + (long long)(t.row0 + j - t.past) * a.kv_stride + (long long)t.g * t.hd + c * 8;
        }
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to(r, c)), "l"(src), "r"(bytes) : "memory");
    }
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(LEFT) : "memory"); }

// The warp's scores against a key tile, scaled, soft-capped, biased and masked, in the base-2 domain; mx0, mx1: the rows' maxima.
template <int HD, int MODE, bool AHEAD>
__device__ __forceinline__ void tile_scores(const AttentionArgs& a, const Tile& t, uint32_t sQ, uint32_t sK, int kv0, float (&s)[BN / 8][4],
                                            float& mx0, float& mx1) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tq = lane & 3;
#pragma unroll
    for (int i = 0; i < BN / 8; ++i) { s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f; }
    if (AHEAD) {       // the next 16 values' operands are asked for before this one's products
        uint32_t af[2][4], bf[2][BN / 16][4];
        auto load = [&](int b, int kk) {
            ldmatrix_x4(af[b], tile_addr<HD>(sQ, warp * 16 + (lane & 15), 2 * kk + (lane >> 4)));
#pragma unroll
            for (int np = 0; np < BN / 16; ++np)
                ldmatrix_x4(bf[b][np], tile_addr<HD>(sK, np * 16 + (lane & 7) + 8 * (lane >> 4), 2 * kk + ((lane >> 3) & 1)));
        };
        auto multiply = [&](int b) {
#pragma unroll
            for (int np = 0; np < BN / 16; ++np) {
                mma_bf16(s[2 * np], af[b], bf[b][np][0], bf[b][np][1]);
                mma_bf16(s[2 * np + 1], af[b], bf[b][np][2], bf[b][np][3]);
            }
        };
        load(0, 0);
        for (int kk = 0; kk < t.ksteps; kk += 2) {
            if (kk + 1 < t.ksteps) load(1, kk + 1);
            multiply(0);
            if (kk + 1 < t.ksteps) {
                if (kk + 2 < t.ksteps) load(0, kk + 2);
                multiply(1);
            }
        }
    } else {
        for (int kk = 0; kk < t.ksteps; ++kk) {
            uint32_t af[4];
            ldmatrix_x4(af, tile_addr<HD>(sQ, warp * 16 + (lane & 15), 2 * kk + (lane >> 4)));
#pragma unroll
            for (int np = 0; np < BN / 16; ++np) {
                uint32_t bf[4];
                ldmatrix_x4(bf, tile_addr<HD>(sK, np * 16 + (lane & 7) + 8 * (lane >> 4), 2 * kk + ((lane >> 3) & 1)));
                mma_bf16(s[2 * np], af, bf[0], bf[1]);
                mma_bf16(s[2 * np + 1], af, bf[2], bf[3]);
            }
        }
    }
    const bool need_mask = !(kv0 + BN - 1 <= t.pw_first && kv0 >= t.low_last);
    const bool rel_plain = MODE == 2 && kv0 + BN - 1 <= t.pw_first && t.pw_last - kv0 < a.rel_len;     // every distance of the tile has an entry
    mx0 = mx1 = -INFINITY;
#pragma unroll
    for (int nt = 0; nt < BN / 8; ++nt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            float v = s[nt][e] * a.score_scale;
            if (a.softcap > 0.f) v = a.softcap * tanh_fast(v * t.inv_cap);
            if (MODE == 2) {
                const int dist = ((e < 2) ? t.pr0 : t.pr1) - (kv0 + nt * 8 + 2 * tq + (e & 1));
                v = fmaf(v, LOG2E, __ldg(t.rel + (rel_plain ? dist : min(max(dist, 0), a.rel_len - 1))));
            } else {
                v *= LOG2E;
            }
            if (need_mask) {
                const int key = kv0 + nt * 8 + 2 * tq + (e & 1);
                const bool keep = key <= ((e < 2) ? t.pr0 : t.pr1) && key >= ((e < 2) ? t.lo0 : t.lo1);
                if (!keep) v = -INFINITY;
            }
            s[nt][e] = v;
        }
        mx0 = fmaxf(mx0, fmaxf(s[nt][0], s[nt][1]));
        mx1 = fmaxf(mx1, fmaxf(s[nt][2], s[nt][3]));
    }
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
}

// Sigmoid weights (no softmax): the weight of a kept key is sigmoid(score + bias), formed in float and handed to the tensor cores as
// two bfloat16 terms (its rounding, pf, and what the rounding left, pl), so that 16 bits of it count.
__device__ __forceinline__ void sigmoid_weights(const float (&s)[BN / 8][4], float sig_bias, uint32_t (&pf)[BN / 16][4], uint32_t (&pl)[BN / 16][4]) {
#pragma unroll
    for (int nt = 0; nt < BN / 8; ++nt) {
        float wv[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) wv[e] = 1.0f / (1.0f + exp2f(-(s[nt][e] + sig_bias)));      // masked: exp2(inf) -> 0
        const uint32_t h01 = pack_bf16(wv[0], wv[1]), h23 = pack_bf16(wv[2], wv[3]);
        pf[nt >> 1][(nt & 1) * 2 + 0] = h01;
        pf[nt >> 1][(nt & 1) * 2 + 1] = h23;
        const float2 f01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&h01));
        const float2 f23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&h23));
        pl[nt >> 1][(nt & 1) * 2 + 0] = pack_bf16(wv[0] - f01.x, wv[1] - f01.y);
        pl[nt >> 1][(nt & 1) * 2 + 1] = pack_bf16(wv[2] - f23.x, wv[3] - f23.y);
    }
}
// Softmax weights against the maxima ms0, ms1, and their sums over the tile.
__device__ __forceinline__ void softmax_weights(const float (&s)[BN / 8][4], float ms0, float ms1, float& rs0, float& rs1, uint32_t (&pf)[BN / 16][4]) {
    rs0 = rs1 = 0.f;
#pragma unroll
    for (int nt = 0; nt < BN / 8; ++nt) {
        const float e0 = exp2f(s[nt][0] - ms0), e1 = exp2f(s[nt][1] - ms0);
        const float e2 = exp2f(s[nt][2] - ms1), e3 = exp2f(s[nt][3] - ms1);
        rs0 += e0 + e1;
        rs1 += e2 + e3;
        pf[nt >> 1][(nt & 1) * 2 + 0] = pack_bf16(e0, e1);
        pf[nt >> 1][(nt & 1) * 2 + 1] = pack_bf16(e2, e3);
    }
    rs0 += __shfl_xor_sync(0xffffffffu, rs0, 1);
    rs0 += __shfl_xor_sync(0xffffffffu, rs0, 2);
    rs1 += __shfl_xor_sync(0xffffffffu, rs1, 1);
    rs1 += __shfl_xor_sync(0xffffffffu, rs1, 2);
}
// A key tile's weights take a row's running maximum m along; c: what the sums so far are scaled by, ms: what the tile's scores are
// taken against.
__device__ __forceinline__ void next_maximum(float& m, float mx, float& ms, float& c) {
    const float mn = fmaxf(m, mx);
    ms = mn == -INFINITY ? 0.f : mn;
    c = exp2f(m - ms);
    m = mn;
}

// o: column tiles [first, first + n) of eight values; normalised and stored.
template <int N, int MODE>
__device__ __forceinline__ void store_rows(const AttentionArgs& a, const Tile& t, const float (&o)[N][4], int first, int n, float m0, float m1, float l0, float l1) {
    const int lane = threadIdx.x & 31, r0 = (threadIdx.x >> 5) * 16 + (lane >> 2), r1 = r0 + 8, tq = lane & 3;
    if (a.sinks) {      // a logit without key or value joins each row's denominator (base-2 domain, like m and l)
        const float sink = a.sinks[t.h] * LOG2E;
        l0 += exp2f(sink - m0);
        l1 += exp2f(sink - m1);
    }
    const float i0 = MODE == 1 ? 1.0f : 1.0f / l0, i1 = MODE == 1 ? 1.0f : 1.0f / l1;
    __nv_bfloat16* out = (__nv_bfloat16*)a.out;
#pragma unroll
    for (int nt = 0; nt < N; ++nt) {
        const int d = (first + nt) * 8 + 2 * tq;
        if (nt < n && d < t.hd) {
            if (r0 < t.rows)
                *(__nv_bfloat162*)(out + (long long)(t.row0 + t.q0 + r0) * a.out_stride + (long long)t.h * t.hd + d) =
                    __floats2bfloat162_rn(o[nt][0] * i0, o[nt][1] * i0);
            if (r1 < t.rows)
                *(__nv_bfloat162*)(out + (long long)(t.row0 + t.q0 + r1) * a.out_stride + (long long)t.h * t.hd + d) =
                    __floats2bfloat162_rn(o[nt][2] * i1, o[nt][3] * i1);
        }
    }
}

// MODE 0: softmax; 1: sigmoid weights; 2: softmax with a bias per head and distance (base-2 domain) added to the scores
template <int HD, int MODE>
__global__ void __launch_bounds__(NTHREADS, HD == 64 && MODE == 1 ? 4 : 0) attention_prefill_kernel(AttentionArgs a) {
    constexpr int CH = HD / 8;
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t sQ = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t sK = sQ + BM * HD * 2;
    const uint32_t sV = sK + BN * HD * 2;

    const Tile t(a, a.n_tiles - 1 - (int)blockIdx.x, blockIdx.y);   // later tiles of a sequence have more keys: start them first
    const int lane = threadIdx.x & 31;

    rdl_grid_wait();               // the batch description above is constant; the rows come from the kernel before
    rdl_grid_launch_dependents();
    load_queries<HD>(a, t, smem);

    float o[HD / 8][4];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    constexpr bool sig = MODE == 1;                                             // weights sigmoid(score + bias[h]), not normalised
    const float sig_bias = sig ? a.sigmoid_bias[t.h] * LOG2E : 0.f;       // in the base-2 domain, like the scores

    auto issue = [&](int kv0, int which) {       // one tile of keys or values, one commit group
        const uint32_t sdst = which ? sV : sK;
        copy_rows<CH>(a, t, kv0, page_place(a, t, kv0), which, 0, CH, [&](int r, int c) { return tile_addr<HD>(sdst, r, c); });
        copies_commit();
    };

    const int kv_first = (t.lo_first / BN) * BN;
    if (kv_first <= t.p_last) {
        issue(kv_first, 0);
        issue(kv_first, 1);
    }
    for (int kv0 = kv_first; kv0 <= t.p_last; kv0 += BN) {
        const bool has_next = kv0 + BN <= t.p_last;
        copies_wait<1>();                      // this tile's keys have landed (its values may be on the way)
        __syncthreads();

        // this warp's rows see nothing of the tile: skip its arithmetic (barriers stay outside)
        const bool warp_active = t.sees(kv0);
        uint32_t pf[BN / 16][4];
        uint32_t pl[BN / 16][4];      // sigmoid weights: what the rounding of pf left
        if (warp_active) {
            float s[BN / 8][4], mx0, mx1;
            tile_scores<HD, MODE, false>(a, t, sQ, sK, kv0, s, mx0, mx1);
            if (sig) {
                sigmoid_weights(s, sig_bias, pf, pl);
            } else {
                float ms0, ms1, c0, c1, rs0, rs1;
                next_maximum(m0, mx0, ms0, c0);
                next_maximum(m1, mx1, ms1, c1);
                softmax_weights(s, ms0, ms1, rs0, rs1, pf);
                l0 = l0 * c0 + rs0;
                l1 = l1 * c1 + rs1;
#pragma unroll
                for (int i = 0; i < HD / 8; ++i) {
                    o[i][0] *= c0; o[i][1] *= c0; o[i][2] *= c1; o[i][3] *= c1;
                }
            }
        }
        __syncthreads();                       // every warp is done with the key tile
        if (has_next) issue(kv0 + BN, 0);      // the next keys travel while P V is computed
        if (has_next) copies_wait<1>();
        else copies_wait<0>();
        __syncthreads();                       // this tile's values have landed
        if (warp_active) {
            // ---- O += P V ----
#pragma unroll
            for (int kk = 0; kk < BN / 16; ++kk) {
#pragma unroll
                for (int dp = 0; dp < HD / 16; ++dp) {
                    if (dp * 16 < t.hd) {
                        uint32_t bf[4];
                        ldmatrix_x4_trans(bf, tile_addr<HD>(sV, kk * 16 + (lane & 15), 2 * dp + (lane >> 4)));
                        mma_bf16(o[2 * dp], pf[kk], bf[0], bf[1]);
                        mma_bf16(o[2 * dp + 1], pf[kk], bf[2], bf[3]);
                        if (sig) {
                            mma_bf16(o[2 * dp], pl[kk], bf[0], bf[1]);
                            mma_bf16(o[2 * dp + 1], pl[kk], bf[2], bf[3]);
                        }
                    }
                }
            }
        }
        __syncthreads();                       // every warp is done with the value tile
        if (has_next) issue(kv0 + BN, 1);      // the next values travel while the next scores are computed
    }
    store_rows<HD / 8, MODE>(a, t, o, 0, HD / 8, m0, m1, l0, l1);
}

// ---------------------------------------------------------------------------------------------
// The same by a cluster of `runs` blocks.  The chain of key tiles is what takes the time (a tile's copies, its scores, its
// exponentials, its share of O, one after the other), and it is taken apart without touching a row's order of
// operations.  Every round takes `runs` key tiles: block r forms the scores and weights of the r-th, which need of the
// tiles before it their rows' maxima alone; then every block adds all the round's tiles, in their order, to its own share of
// O's columns.  What passes between the blocks lies in shared memory: a tile's maxima before the first cluster barrier of a
// round, its weights (as the operand fragments of the thread that uses them) and their sums before the second.  What
// bounds it is latency: two barriers and one trip of the weights a round, with little in flight in four warps a block.
// 3 x 41 tokens behind 640 of 8 heads of 256: 31.4 us (150.7 with one block a tile whose copies look their page up row by row, 112 with
// one that looks it up once a tile; 30.9 with runs of keys whose sums are merged at the end, which rounds differently).
// One prompt behind 6,000: 166 us (1,285; 925; 125).  16 heads of 64, 60 tokens behind 500: 21.0 us (36.6; 29.4; 11.6).
// ---------------------------------------------------------------------------------------------
template <int HD, int MODE>
struct SharedLayout {       // bytes
    static constexpr int PARTS = MODE == 1 ? 2 : 1;                              // bfloat16 terms of a weight
    static constexpr int Q = 0, K = BM * HD * 2, P = K + BN * HD * 2, STATS = P + PARTS * BM * BN * 2, V = STATS + 3 * BM * 4;
    // columns in pieces of eight; a row of a block's share is an odd number of them, so that eight rows' reads fall into different banks
    static __host__ __device__ int share(int hd, int runs) { return (hd / 8 + runs - 1) / runs; }
    static __host__ __device__ int total(int hd, int runs) { return V + runs * BN * (share(hd, runs) | 1) * 16; }
};

template <int HD, int MODE>
__global__ void __launch_bounds__(NTHREADS) attention_prefill_shared_kernel(AttentionArgs a, int runs) {
    using L = SharedLayout<HD, MODE>;
    constexpr int CH = HD / 8, MAX_SHARE = CH / 2;          // two blocks at least
    extern __shared__ __align__(128) unsigned char smem[];
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem), sQ = base + L::Q, sK = base + L::K, sV = base + L::V;
    uint4* weights = reinterpret_cast<uint4*>(smem + L::P);                       // [part][16 keys][thread]
    float* maxima = reinterpret_cast<float*>(smem + L::STATS);                    // [round & 1][row]: read while the next round's are written
    float* sums = maxima + 2 * BM;                                                // [row]

    const int run = (int)cluster_rank();
    const Tile t(a, a.n_tiles - 1 - (int)blockIdx.x / runs, blockIdx.y);
    const int tid = threadIdx.x, lane = tid & 31, w0 = (tid >> 5) * 16 + (lane >> 2), w1 = w0 + 8;
    const int share = L::share(t.hd, runs), pitch = (share | 1) * 16;
    const int col0 = min(run * share, t.hd / 8), cols = min(share, t.hd / 8 - col0);      // this block's columns, in pieces of eight

    const bool wanted = (tid >> 5) * 16 < t.rows;            // rows beyond the sequence's are never stored: their warps take part in the barriers only

    float o[MAX_SHARE][4];
#pragma unroll
    for (int i = 0; i < MAX_SHARE; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
    constexpr bool sig = MODE == 1;
    const float sig_bias = sig ? a.sigmoid_bias[t.h] * LOG2E : 0.f;

    const int kv_first = (t.lo_first / BN) * BN, n_kt = (t.p_last - kv_first) / BN + 1;
    // lane i: where tile `first + i` of a round lies, for a round looked up in one trip (constants: before the wait)
    auto places = [&](int first) { return lane < runs && first + lane < n_kt ? page_place(a, t, kv_first + (first + lane) * BN) : 0LL; };
    // One commit group each, empty where there is nothing to copy: the key tile of this block, and its columns of the values of a round.
    auto issue_keys = [&](int first, long long at) {
        const long long page = __shfl_sync(0xffffffffu, at, run);
        if (first + run < n_kt)
            copy_rows<CH>(a, t, kv_first + (first + run) * BN, page, 0, 0, CH, [&](int r, int c) { return tile_addr<HD>(sK, r, c); });
        copies_commit();
    };
    auto issue_values = [&](int first, long long at) {
        for (int i = 0; i < min(runs, n_kt - first); ++i) {
            const long long page = __shfl_sync(0xffffffffu, at, i);
            if (cols > 0)
                copy_rows<0>(a, t, kv_first + (first + i) * BN, page, 1, col0, cols,
                             [&](int r, int c) { return sV + (uint32_t)((i * BN + r) * pitch + (c - col0) * 16); });
        }
        copies_commit();
    };
    long long at = places(0);

    rdl_grid_wait();
    rdl_grid_launch_dependents();
    load_queries<HD>(a, t, smem);
    issue_keys(0, at);
    issue_values(0, at);
    for (int first = 0, parity = 0; first < n_kt; first += runs, parity ^= 1) {
        const int kv0 = kv_first + (first + run) * BN;
        at = places(first + runs);
        const bool mine = first + run < n_kt && wanted && t.sees(kv0);         // this warp's rows see something of the block's tile
        copies_wait<1>();                      // the keys have landed (the values may be on the way)
        __syncthreads();
        float s[BN / 8][4], mx0 = -INFINITY, mx1 = -INFINITY;
        if (mine) tile_scores<HD, MODE, true>(a, t, sQ, sK, kv0, s, mx0, mx1);
        if ((lane & 3) == 0) { maxima[parity * BM + w0] = mx0; maxima[parity * BM + w1] = mx1; }
        __syncwarp();
        cluster_sync();                        // every tile's maxima are there; the key tile, and the weights of the round before, have been read
        issue_keys(first + runs, at);
        float b0 = m0, b1 = m1;                // the rows' maxima before this block's tile
        if (!sig) {
            float v0[MAX_RUNS - 1], v1[MAX_RUNS - 1];
#pragma unroll
            for (int i = 0; i < MAX_RUNS - 1; ++i) {                              // (all asked for at once; its own where there is none)
                const uint32_t there = in_block(base + L::STATS + (uint32_t)(parity * BM * 4), min(i, run));
                v0[i] = ld_cluster(there + w0 * 4);
                v1[i] = ld_cluster(there + w1 * 4);
            }
#pragma unroll
            for (int i = 0; i < MAX_RUNS - 1; ++i) {
                b0 = i < run ? fmaxf(b0, v0[i]) : b0;
                b1 = i < run ? fmaxf(b1, v1[i]) : b1;
            }
        }
        if (mine) {
            uint32_t pf[BN / 16][4], pl[BN / 16][4];
            if (sig) {
                sigmoid_weights(s, sig_bias, pf, pl);
            } else {
                float ms0, ms1, c0, c1, rs0, rs1;
                next_maximum(b0, mx0, ms0, c0);
                next_maximum(b1, mx1, ms1, c1);
                softmax_weights(s, ms0, ms1, rs0, rs1, pf);
                if ((lane & 3) == 0) { sums[w0] = rs0; sums[w1] = rs1; }
            }
#pragma unroll
            for (int kk = 0; kk < BN / 16; ++kk) {
                weights[kk * NTHREADS + tid] = make_uint4(pf[kk][0], pf[kk][1], pf[kk][2], pf[kk][3]);
                if (sig) weights[(BN / 16 + kk) * NTHREADS + tid] = make_uint4(pl[kk][0], pl[kk][1], pl[kk][2], pl[kk][3]);
            }
        }
        copies_wait<1>();                      // the values have landed (the next keys may be on the way)
        __syncwarp();
        cluster_sync();                        // every tile's weights and sums are there, and everybody's values
        // The round's tiles in their order, what is needed of each asked for before the products of the one before.  (A loop: unrolled,
        // the time went into fetching instructions.)
        constexpr int U = MAX_SHARE < 4 ? MAX_SHARE : 4;
        uint32_t pf[BN / 16][4], pl[BN / 16][4], pf_next[BN / 16][4], pl_next[BN / 16][4];
        float stats[4], stats_next[4] = {0.f, 0.f, 0.f, 0.f};
        auto used = [&](int i) { return i < runs && first + i < n_kt && wanted && t.sees(kv_first + (first + i) * BN); };
        auto fetch = [&](int i) {
            const uint32_t there = in_block(base, i);
            if (!sig) {
                stats_next[0] = ld_cluster(there + L::STATS + (parity * BM + w0) * 4);
                stats_next[1] = ld_cluster(there + L::STATS + (parity * BM + w1) * 4);
                stats_next[2] = ld_cluster(there + L::STATS + (2 * BM + w0) * 4);
                stats_next[3] = ld_cluster(there + L::STATS + (2 * BM + w1) * 4);
            }
            if (cols == 0) return;
#pragma unroll
            for (int kk = 0; kk < BN / 16; ++kk) {
                ld_cluster(pf_next[kk], there + L::P + (kk * NTHREADS + tid) * 16);
                if (sig) ld_cluster(pl_next[kk], there + L::P + ((BN / 16 + kk) * NTHREADS + tid) * 16);
            }
        };
        if (used(0)) fetch(0);
#pragma unroll 1
        for (int i = 0; i < min(runs, n_kt - first); ++i) {
#pragma unroll
            for (int kk = 0; kk < BN / 16; ++kk) {
#pragma unroll
                for (int e = 0; e < 4; ++e) { pf[kk][e] = pf_next[kk][e]; if (sig) pl[kk][e] = pl_next[kk][e]; stats[e] = stats_next[e]; }
            }
            if (used(i + 1)) fetch(i + 1);
            if (!used(i)) continue;
            if (!sig) {
                float ms0, ms1, c0, c1;
                next_maximum(m0, stats[0], ms0, c0);
                next_maximum(m1, stats[1], ms1, c1);
                l0 = l0 * c0 + stats[2];
                l1 = l1 * c1 + stats[3];
#pragma unroll
                for (int u = 0; u < MAX_SHARE; ++u) { o[u][0] *= c0; o[u][1] *= c0; o[u][2] *= c1; o[u][3] *= c1; }
            }
#pragma unroll
            for (int k2 = 0; k2 < BN / 32; ++k2) {
#pragma unroll
                for (int ub = 0; ub < MAX_SHARE; ub += U) {
                    if (ub >= cols) break;
                    uint32_t bf[U][4];         // 32 keys of eight columns each
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (ub + u < cols) ldmatrix_x4_trans(bf[u], sV + (uint32_t)((i * BN + k2 * 32 + lane) * pitch + (ub + u) * 16));
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            if (ub + u < cols) mma_bf16(o[ub + u], pf[2 * k2 + half], bf[u][2 * half], bf[u][2 * half + 1]);
                        if (sig) {
#pragma unroll
                            for (int u = 0; u < U; ++u)
                                if (ub + u < cols) mma_bf16(o[ub + u], pl[2 * k2 + half], bf[u][2 * half], bf[u][2 * half + 1]);
                        }
                    }
                }
            }
        }
        __syncthreads();                       // every warp is done with the values
        issue_values(first + runs, at);
    }
    store_rows<MAX_SHARE, MODE>(a, t, o, col0, cols, m0, m1, l0, l1);
    copies_wait<0>();
    __syncwarp();
    cluster_sync();                            // no block leaves while another may still read its weights
}

// Blocks a query tile and head.  More of them shorten the chain of key tiles and split O's columns, so that even one key tile is
// faster with four; eight pay from five key tiles on (that many of them work in a round), and never more than find room at
// once: two a multiprocessor where their shared memory allows it, and of clusters of four and eight about seven eighths
// of that (the multiprocessors come in groups that such clusters do not fill).  Two blocks save less than their
// barriers cost with heads of up to 64.  Microseconds with 1 / 2 / 4 / 8 blocks, T key tiles, P pairs of query tile and head:
//   heads of 256  T 1, P 8     15.8 / 13.0 / 11.6 / 11.8      heads of 128  T 2, P 16    15.8 / 11.1 / 10.0 / 12.0
//                 T 4, P 8     45.4 / 27.2 / 17.1 / 16.4                    T 4, P 16    27.0 / 18.4 / 11.6 / 13.6
//                 T 5, P 8     55.0 / 35.2 / 23.8 / 17.4                    T 9, P 16    54.3 / 34.5 / 21.7 / 19.3
//                 T 11, P 32    113 / 63.0 / 38.0 / 32.0                    T 9, P 64    55.0 / 35.0 / 24.9 / 42.6
//                 T 11, P 40    113 / 63.1 / 40.6 / 57.7                    T 9, P 128   55.1 / 37.0 / 48.4 / 83.9
//                 T 11, P 64    114 / 63.2 / 41.1 / 62.8      heads of 64   T 9, P 16    29.4 / 31.0 / 21.6 / 21.0
//                 T 11, P 72    114 / 63.2 / 74.8 / 86.8                    T 9, P 64    29.6 / 31.7 / 27.7 / 51.1
//                 T 11, P 144   115 / 68.5 / 115 / 149                      T 9, P 128   29.9 / 35.6 / 50.2 / 81.4
// smem(runs): bytes of a block.  max_keys: the host's bound on the keys a query sees (0: not known); it and the rule change times only.
template <typename Smem>
int choose_runs(long long pairs, int head_dim, int max_keys, int sms, Smem smem) {
    const int key_tiles = max_keys > 0 ? (max_keys + BN - 1) / BN : MAX_RUNS;
    for (int runs = key_tiles > 4 ? MAX_RUNS : 4; runs > 1; runs /= 2) {
        if (runs == 2 && head_dim <= 64) continue;
        const long long slots = (long long)sms * std::min(2, 228 * 1024 / (smem(runs) + 1024));
        if (pairs * runs <= (runs == 2 ? slots : slots * 7 / 8)) return runs;
    }
    return 1;
}

// f(HD, MODE) as integral constants: the widths and forms there are kernels for (softmax, sigmoid weights or a distance bias: kernels
// of their own, so that the softmax kernels keep their registers).
template <typename F>
int by_form(int head_dim, bool sigmoid, bool rel, F f) {
    auto mode = [&](auto hd) {
        return sigmoid ? f(hd, std::integral_constant<int, 1>()) : rel ? f(hd, std::integral_constant<int, 2>()) : f(hd, std::integral_constant<int, 0>());
    };
    return head_dim <= 32 ? mode(std::integral_constant<int, 32>()) : head_dim <= 64 ? mode(std::integral_constant<int, 64>())
           : head_dim <= 128 ? mode(std::integral_constant<int, 128>()) : mode(std::integral_constant<int, 256>());
}

template <int HD, int MODE>
int launch_prefill_as(const AttentionArgs* a, cudaStream_t st) {
    const int runs = choose_runs((long long)a->n_tiles * a->n_heads, a->head_dim, a->max_keys, rdl_sm_count(),
                                 [&](int r) { return SharedLayout<HD, MODE>::total(a->head_dim, r); });
    if (runs == 1) {
        const int smem = (BM + 2 * BN) * HD * 2;
        RDL_CUDA((rdl_allow_shared<attention_prefill_kernel<HD, MODE>>(smem)), "attention_prefill");
        dim3 grid(a->n_tiles, a->n_heads);
        RDL_CHECK_EX(rdl_launch(attention_prefill_kernel<HD, MODE>, grid, dim3(NTHREADS), (size_t)smem, st, *a), "attention_prefill");
        return 0;
    }
    using L = SharedLayout<HD, MODE>;
    const int smem = L::total(a->head_dim, runs);
    RDL_CUDA((rdl_allow_shared<attention_prefill_shared_kernel<HD, MODE>>(smem)), "attention_prefill");
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)runs;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)(a->n_tiles * runs), (unsigned)a->n_heads);
    cfg.blockDim = dim3(NTHREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = g_rdl_programmatic_launch ? 2 : 1;
    RDL_CHECK_EX(cudaLaunchKernelEx(&cfg, attention_prefill_shared_kernel<HD, MODE>, *a, runs), "attention_prefill");
    return 0;
}

}  // namespace

extern "C" int rdl_attention_prefill(const AttentionArgs* a, void* stream) {
    if (int e = rdl_check_attention_args(a, "attention_prefill")) return e;
    RDL_REQUIRE(a->dtype == RDL_BF16, "attention_prefill: bfloat16 only (the 32-bit path uses attention_plain)");
    RDL_REQUIRE(a->head_dim % 16 == 0 && a->head_dim <= 256,
                "attention_prefill: head_dim %d must be a multiple of 16 and at most 256", a->head_dim);
    RDL_REQUIRE(a->tile_seq && a->tile_q0 && a->n_tiles >= 0, "attention_prefill: missing query tiles");
    RDL_REQUIRE(a->n_heads <= 65535, "attention_prefill: too many heads for the grid");
    RDL_REQUIRE(a->q_stride % 8 == 0 && a->kv_stride % 8 == 0 && a->out_stride % 2 == 0 &&
                    ((uintptr_t)a->q % 16 == 0) && ((uintptr_t)a->k_new % 16 == 0) && ((uintptr_t)a->v_new % 16 == 0) &&
                    ((uintptr_t)a->k_cache % 16 == 0) && ((uintptr_t)a->v_cache % 16 == 0) && ((uintptr_t)a->out % 4 == 0),
                "attention_prefill: rows must start on 16-byte boundaries");
    if (a->n_tiles == 0 || a->n_tokens == 0) return 0;
    return by_form(a->head_dim, a->sigmoid_bias, a->rel_bias, [&](auto hd, auto mode) { return launch_prefill_as<hd.value, mode.value>(a, (cudaStream_t)stream); });
}

extern "C" int rdl_attention_prefill_blocks(long long pairs, int head_dim, int sigmoid, int max_keys, int sms) {
    return by_form(head_dim, sigmoid != 0, false, [&](auto hd, auto mode) {
        return choose_runs(pairs, head_dim, max_keys, sms, [&](int r) { return SharedLayout<hd.value, mode.value>::total(head_dim, r); });
    });
}
