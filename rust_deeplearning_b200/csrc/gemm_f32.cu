// Matrix product of the 32-bit path: out[m, n] = sum_k x[m, k] * w[n, k], float operands, fused
// multiply-add in float, no tensor cores and no reduced-precision mode.
//
// Every output element is summed in one order that depends on K alone, whatever M, N or the element's
// place in a tile, so a row's result does not depend on which other rows are in the batch: k is cut into
// eight runs of equal length (a multiple of four); inside a run two chains of fused multiply-adds take the
// even and the odd k (the halves of the two-wide instruction) and are added at the run's end; the runs' sums
// are added one after another.  (One chain over all k, as before, is 2.0 to 2.6 times further from the 64-bit
// result.)  Zeros stand in for k beyond a run: they change no chain.
//
// Two kernels share that order.
//   * Up to 16 rows the weights' bytes bound the product (10.4 GB a step at the 2B shape).  A warp takes one run of k
//     of a tile of 32 or 16 weight rows - a lane a row, its sums over all x rows in registers - through a ring of its
//     own in shared memory (cp.async, 16 bytes a lane, rows 144 bytes apart so that a quarter warp's reads fall into
//     different banks); the eight warps of a block are the eight runs, whose sums meet in shared memory once a tile.
//     Blocks are persistent and the ring runs on from tile to tile; weights are asked for before the wait on the
//     kernel before.
//   * Above, the float units bound it.  A block forms a tile of 32, 48, 64 or 128 rows by 128 columns, a thread 4 to 8 by 8
//     of them, both operands' rows in shared memory as they lie in memory (no transposition: the two-wide instruction
//     takes neighbouring k).  Where the tiles alone do not fill the chip, eight blocks (a cluster) share a tile, a run of k
//     each, and add up through distributed shared memory.
//     A thread's 6 or 8 by 8 sums cost 14 or 16 reads of 16 bytes for 96 or 128 two-wide multiply-adds; with 3 by 8 (11 for 48) the
//     reads from shared memory were the bound: 2,304 outputs of 9,216 for 48 rows 125 -> 110 us, 18,432 of 2,304 146 -> 122 (33 TFLOP/s).
// Both take operands that are not 16-byte aligned (or K not a multiple of four) by 4-byte copies.
// (The reference's product is an f32 library GEMM: rustml/core/main/src/core/tensor/ops.rs:806-823;
// y = x W^T with W [out, in]: rustml/nn/main/src/core/linear.rs:12-15, :168-169.)
#include "api.h"
#include "common.cuh"
#include "launch.cuh"

namespace {

constexpr int RUNS = 8;             // runs of k
constexpr int KC = 32;              // k of a chunk in shared memory
constexpr int PITCH = KC + 4;       // floats between the rows of a chunk

// Length of a run of k: a multiple of four, eight of them cover K.
__host__ __device__ __forceinline__ int run_length(int K) { return ((K + RUNS - 1) / RUNS + 3) & ~3; }

__device__ __forceinline__ unsigned long long ffma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float halves_sum(unsigned long long v) {
    return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32));
}
struct Pairs { unsigned long long lo, hi; };        // four neighbouring k
__device__ __forceinline__ Pairs lds_pairs(uint32_t addr) {
    Pairs v;
    asm volatile("ld.shared.v2.u64 {%0,%1}, [%2];" : "=l"(v.lo), "=l"(v.hi) : "r"(addr));
    return v;
}
// Four floats from p (n of them exist, the rest become zero) to shared memory.
template <bool ALIGNED>
__device__ __forceinline__ void copy4(uint32_t dst, const float* p, int n) {
    if (ALIGNED) {
        const int bytes = n > 0 ? 16 : 0;            // K and the runs are multiples of four
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(p), "r"(bytes) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int bytes = i < n ? 4 : 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * i), "l"(i < n ? p + i : p), "r"(bytes) : "memory");
        }
    }
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// ---- few rows ----

// ROWS weight rows a tile (16: half a warp each takes half of the x rows), MT x rows, STAGES chunks of a warp's ring.
template <int ROWS, int MT, int STAGES, bool ALIGNED>
__global__ void __launch_bounds__(RUNS * 32, 1) gemm_f32_few_kernel(float* __restrict__ out, const float* __restrict__ x,
                                                                   const float* __restrict__ w, int M, int N, int K) {
    constexpr int MINE = ROWS == 32 ? MT : MT / 2;           // x rows of a lane
    constexpr int STAGE = ROWS * PITCH + MT * KC;            // floats
    extern __shared__ __align__(16) float ring[];
    __shared__ float part[2][RUNS][MT][ROWS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = ROWS == 32 ? lane : lane & 15, m0 = ROWS == 32 ? 0 : (lane >> 4) * MINE;
    const int run = run_length(K), k_lo = warp * run, k_hi = min(K, k_lo + run);
    const int chunks = k_hi > k_lo ? (k_hi - k_lo + KC - 1) / KC : 0;
    const int n_tiles = (N + ROWS - 1) / ROWS;
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(ring) + (uint32_t)(warp * STAGES * STAGE * 4);

    auto copy_w = [&](int tile, int c, int s) {
        const int k0 = k_lo + c * KC;
#pragma unroll
        for (int i = 0; i < ROWS / 4; ++i) {
            const int r = i * 4 + (lane >> 3), k = k0 + (lane & 7) * 4, n = tile * ROWS + r;
            const bool ok = n < N && k < k_hi;
            copy4<ALIGNED>(mine + (uint32_t)((s * STAGE + r * PITCH + (lane & 7) * 4) * 4), ok ? w + (long long)n * K + k : w, ok ? k_hi - k : 0);
        }
    };
    auto copy_x = [&](int c, int s) {
        const int k0 = k_lo + c * KC;
#pragma unroll
        for (int i = 0; i < (MT * 8 + 31) / 32; ++i) {
            const int r = i * 4 + (lane >> 3), k = k0 + (lane & 7) * 4;
            if (MT < 4 && r >= MT) continue;
            const bool ok = r < M && k < k_hi;
            copy4<ALIGNED>(mine + (uint32_t)((s * STAGE + ROWS * PITCH + r * KC + (lane & 7) * 4) * 4), ok ? x + (long long)r * K + k : x, ok ? k_hi - k : 0);
        }
    };
    // what is asked for next: chunk `ac` of tile `at`
    int at = blockIdx.x, ac = 0;
    auto advance = [&]() { if (++ac == chunks) { ac = 0; at += gridDim.x; } };
    if (chunks > 0) {
        // the weights of the first chunks need nothing of the kernel before
        for (int s = 0; s < STAGES - 1; ++s) {
            if (at < n_tiles) copy_w(at, ac, s);
            advance();
        }
    }
    rdl_grid_wait();
    rdl_grid_launch_dependents();
    if (chunks > 0) {
        int bt = blockIdx.x, bc = 0;
        for (int s = 0; s < STAGES - 1; ++s) {
            if (bt < n_tiles) copy_x(bc, s);
            copies_commit();
            if (++bc == chunks) { bc = 0; bt += gridDim.x; }
        }
    }
    int s = 0, buf = 0;
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        unsigned long long acc[MINE];
#pragma unroll
        for (int m = 0; m < MINE; ++m) acc[m] = 0ull;
        for (int c = 0; c < chunks; ++c) {
            copies_wait<STAGES - 2>();
            __syncwarp();                                    // chunk s is there for the whole warp, and the one before it has been read
            const int into = s == 0 ? STAGES - 1 : s - 1;
            if (at < n_tiles) { copy_w(at, ac, into); copy_x(ac, into); }
            copies_commit();
            advance();
            const uint32_t wa = mine + (uint32_t)((s * STAGE + row * PITCH) * 4), xa = mine + (uint32_t)((s * STAGE + ROWS * PITCH + m0 * KC) * 4);
#pragma unroll
            for (int q = 0; q < KC / 4; ++q) {
                const Pairs b = lds_pairs(wa + q * 16);
#pragma unroll
                for (int m = 0; m < MINE; ++m) {
                    const Pairs a = lds_pairs(xa + (m * KC + q * 4) * 4);
                    acc[m] = ffma2(a.lo, b.lo, acc[m]);
                    acc[m] = ffma2(a.hi, b.hi, acc[m]);
                }
            }
            if (++s == STAGES) s = 0;
        }
#pragma unroll
        for (int m = 0; m < MINE; ++m) part[buf][warp][m0 + m][row] = halves_sum(acc[m]);
        __syncthreads();                                     // (the other buffer was read before this barrier's predecessor was passed)
        for (int i = threadIdx.x; i < M * ROWS; i += RUNS * 32) {
            const int m = i / ROWS, r = i - m * ROWS, n = tile * ROWS + r;
            float v = part[buf][0][m][r];
#pragma unroll
            for (int g = 1; g < RUNS; ++g) v += part[buf][g][m][r];
            if (n < N) out[(long long)m * N + n] = v;
        }
        buf ^= 1;
    }
}

constexpr int FEW_MAX = 16;

template <int ROWS, int MT, bool ALIGNED>
cudaError_t launch_few(float* out, const float* x, const float* w, int M, int N, int K, cudaStream_t st) {
    // the ring takes what shared memory the runs' sums leave: the bytes a multiprocessor has on their way set the rate
    constexpr int STAGE_BYTES = (ROWS * PITCH + MT * KC) * 4;
    constexpr int FIT = (224 * 1024 - 2 * RUNS * MT * ROWS * 4) / (RUNS * STAGE_BYTES), STAGES = FIT > 10 ? 10 : FIT;
    static_assert(STAGES >= 3, "a ring of three chunks at least");
    constexpr size_t smem = (size_t)RUNS * STAGES * STAGE_BYTES;
    const cudaError_t e = rdl_allow_shared<gemm_f32_few_kernel<ROWS, MT, STAGES, ALIGNED>>((int)smem);
    if (e != cudaSuccess) return e;
    const int tiles = (N + ROWS - 1) / ROWS, sms = rdl_sm_count();
    return rdl_launch(gemm_f32_few_kernel<ROWS, MT, STAGES, ALIGNED>, dim3(tiles < sms ? tiles : sms), dim3(RUNS * 32), smem, st, out, x, w, M, N, K);
}

template <bool ALIGNED>
cudaError_t launch_few_rows(float* out, const float* x, const float* w, int M, int N, int K, cudaStream_t st) {
    // Tiles of 16 weight rows where tiles of 32 would leave multiprocessors without one.
    const bool narrow = (N + 31) / 32 <= rdl_sm_count();
    if (M <= 2) return narrow ? launch_few<16, 2, ALIGNED>(out, x, w, M, N, K, st) : launch_few<32, 2, ALIGNED>(out, x, w, M, N, K, st);
    if (M <= 4) return narrow ? launch_few<16, 4, ALIGNED>(out, x, w, M, N, K, st) : launch_few<32, 4, ALIGNED>(out, x, w, M, N, K, st);
    if (M <= 8) return narrow ? launch_few<16, 8, ALIGNED>(out, x, w, M, N, K, st) : launch_few<32, 8, ALIGNED>(out, x, w, M, N, K, st);
    return narrow ? launch_few<16, 16, ALIGNED>(out, x, w, M, N, K, st) : launch_few<32, 16, ALIGNED>(out, x, w, M, N, K, st);
}

// ---- many rows ----

constexpr int TN = 8, BN = 16 * TN;
// Blocks a multiprocessor: what the registers of 16 TY threads with 8 TM sums each and a ring of so many chunks leave room for.  (Forms
// of three chunks held to the 168 registers of three blocks spilled 12 to 40 bytes for it: 32 rows 16.9 us against 15.5 for up to
// 15 tiles of 2,304 terms, 25.2 against 24.5 for 32 tiles.)
__host__ __device__ constexpr int tile_blocks(int tm, int ty, int chunks) { return ty == 16 ? 1 : tm <= 6 && chunks == 2 ? 3 : 2; }
// Clusters of eight blocks that find room at once with 1, 2 or 3 blocks a multiprocessor: 15, 33 and 48 of 148 multiprocessors (the
// runtime's occupancy query; a cluster lies inside one group of multiprocessors, and not every group's number is a multiple of eight).
constexpr long long clusters_at(int blocks, int sms) { return (blocks == 1 ? 15LL : blocks == 2 ? 33LL : 48LL) * sms / 148; }

__device__ __forceinline__ uint32_t f32_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void f32_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float f32_ld_remote(uint32_t addr, uint32_t rank) {
    uint32_t at;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}

// A tile of TY TM rows by 128 columns; thread (ty, tx) has rows ty + TY i and columns tx + 16 j.  SHARED: the block is one of a
// cluster of eight along z, each with a run of k.
template <int TM, int TY, int TILE_STAGES, bool SHARED, bool ALIGNED>
__global__ void __launch_bounds__(16 * TY, tile_blocks(TM, TY, TILE_STAGES)) gemm_f32_tile_kernel(float* __restrict__ out, const float* __restrict__ x,
                                                                            const float* __restrict__ w, int M, int N, int K) {
    constexpr int BM = TY * TM, STAGE = (BM + BN) * PITCH, RP = 2 * TY;      // STAGE: floats of a chunk; RP: rows a pass of copies takes
    static_assert(BM % RP == 0 && BN % RP == 0, "whole passes of copies");
    extern __shared__ __align__(16) float sm[];
    float* sums = sm + TILE_STAGES * STAGE;                       // [BM][BN]: the runs' sums so far (SHARED: this block's run)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (lane & 7) + 8 * (warp & 1), ty = (lane >> 3) + 4 * (warp >> 1);
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const int run = run_length(K);
    const int g_lo = SHARED ? (int)blockIdx.z : 0, g_hi = SHARED ? g_lo + 1 : RUNS;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);

    auto copy = [&](int k, int k_hi, int s, bool weights) {      // the chunk from k on into stage s
        if (weights) {
#pragma unroll
            for (int i = 0; i < BN / RP; ++i) {
                const int r = i * RP + (tid >> 3), kk = k + (tid & 7) * 4, n = n0 + r;
                const bool ok = n < N && kk < k_hi;
                copy4<ALIGNED>(base + (uint32_t)((s * STAGE + (BM + r) * PITCH + (tid & 7) * 4) * 4), ok ? w + (long long)n * K + kk : w, ok ? k_hi - kk : 0);
            }
        } else {
#pragma unroll
            for (int i = 0; i < BM / RP; ++i) {
                const int r = i * RP + (tid >> 3), kk = k + (tid & 7) * 4, m = m0 + r;
                const bool ok = m < M && kk < k_hi;
                copy4<ALIGNED>(base + (uint32_t)((s * STAGE + r * PITCH + (tid & 7) * 4) * 4), ok ? x + (long long)m * K + kk : x, ok ? k_hi - kk : 0);
            }
        }
    };
    auto run_end = [&](int g) { return min(K, (g + 1) * run); };
    // what is asked for next: the chunk from k `ak` on of run `ag`
    int ag = g_lo, ak = g_lo * run;
    auto advance = [&]() { ak += KC; if (ak >= run_end(ag)) { ++ag; ak = ag * run; } };
    auto there = [&]() { return ag < g_hi && ak < run_end(ag); };
    for (int s = 0; s < TILE_STAGES - 1; ++s) {
        if (there()) { copy(ak, run_end(ag), s, true); advance(); }
    }
    rdl_grid_wait();
    rdl_grid_launch_dependents();
    ag = g_lo; ak = g_lo * run;
    for (int s = 0; s < TILE_STAGES - 1; ++s) {
        if (there()) { copy(ak, run_end(ag), s, false); advance(); }
        copies_commit();
    }
    int s = 0;
    for (int g = g_lo; g < g_hi; ++g) {
        unsigned long long acc[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
        for (int k = g * run; k < run_end(g); k += KC) {
            copies_wait<TILE_STAGES - 2>();
            __syncthreads();                                     // chunk s is there, and everybody has read the one before it
            const int into = s == 0 ? TILE_STAGES - 1 : s - 1;
            if (there()) { copy(ak, run_end(ag), into, true); copy(ak, run_end(ag), into, false); advance(); }
            copies_commit();
            const uint32_t xa = base + (uint32_t)((s * STAGE + ty * PITCH) * 4), wa = base + (uint32_t)((s * STAGE + (BM + tx) * PITCH) * 4);
#pragma unroll 2
            for (int q = 0; q < KC / 4; ++q) {
                Pairs b[TN];
#pragma unroll
                for (int j = 0; j < TN; ++j) b[j] = lds_pairs(wa + (j * 16 * PITCH + q * 4) * 4);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const Pairs a = lds_pairs(xa + (i * TY * PITCH + q * 4) * 4);
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        acc[i][j] = ffma2(a.lo, b[j].lo, acc[i][j]);
                        acc[i][j] = ffma2(a.hi, b[j].hi, acc[i][j]);
                    }
                }
            }
            if (++s == TILE_STAGES) s = 0;
        }
        const bool first = SHARED || g == 0, last = !SHARED && g == RUNS - 1;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int r = ty + TY * i;
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int c = tx + 16 * j;
                float v = halves_sum(acc[i][j]);
                if (!first) v = sums[r * BN + c] + v;
                if (!last) sums[r * BN + c] = v;
                else if (m0 + r < M && n0 + c < N) out[(long long)(m0 + r) * N + n0 + c] = v;
            }
        }
    }
    if constexpr (SHARED) {
        f32_cluster_sync();                                      // all eight runs of the tile lie in their blocks' shared memory
        const uint32_t rank = f32_cluster_rank();
        const uint32_t sums_s = base + (uint32_t)(TILE_STAGES * STAGE * 4);
        constexpr int ROWS_EACH = BM / RUNS;
        for (int i = tid; i < ROWS_EACH * BN; i += 16 * TY) {
            const int r = (int)rank * ROWS_EACH + i / BN, c = i % BN;
            float v[RUNS];
#pragma unroll
            for (int g = 0; g < RUNS; ++g) v[g] = f32_ld_remote(sums_s + (uint32_t)((r * BN + c) * 4), g);
#pragma unroll
            for (int g = 1; g < RUNS; ++g) v[0] += v[g];
            if (m0 + r < M && n0 + c < N) out[(long long)(m0 + r) * N + n0 + c] = v[0];
        }
        f32_cluster_sync();                                      // no block leaves while another may still read its sums
    }
}

template <int TM, int TY, int STAGES, bool SHARED, bool ALIGNED>
cudaError_t launch_tile(float* out, const float* x, const float* w, int M, int N, int K, cudaStream_t st) {
    constexpr int BM = TY * TM;
    constexpr size_t smem = (size_t)(STAGES * (BM + BN) * PITCH + BM * BN) * 4;
    const cudaError_t e = rdl_allow_shared<gemm_f32_tile_kernel<TM, TY, STAGES, SHARED, ALIGNED>>((int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((N + BN - 1) / BN, (M + BM - 1) / BM, SHARED ? RUNS : 1);
    cfg.blockDim = dim3(16 * TY);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (SHARED) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = RUNS;
    }
    if (g_rdl_programmatic_launch) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, gemm_f32_tile_kernel<TM, TY, STAGES, SHARED, ALIGNED>, out, x, w, M, N, K);
}

// The form of a product of more than FEW_MAX rows: rows of a tile, chunks of the ring, and whether eight blocks share a tile.
struct TileForm { int rows, chunks; bool shared; };

// What a wave of tiles costs by the blocks a multiprocessor holds of it (1, 2, 3), and a further wave behind full ones, in
// microseconds for eighths of 9,216 terms; a wave of whole tiles costs eight times its entry.  Measured with 2,304 to 28,672 outputs of
// 2,048 to 14,336 terms and 32 to 2,048 rows.  (Whole tiles of 48 rows fill multiprocessors with three while others hold one.)
struct TileCost { int rows, levels, shared[3], shared_on, whole[3], whole_on; };
constexpr TileCost TILE_COSTS[] = {{32, 3, {51, 82, 113}, 105, {51, 83, 115}, 110},
                                   {48, 3, {68, 110, 149}, 138, {69, 155, 165}, 153},
                                   {64, 2, {81, 140, 0}, 134, {82, 141, 0}, 134},
                                   {128, 1, {130, 0, 0}, 139, {132, 0, 0}, 138}};

// In microseconds: the waves, by the k their chunks hold, and for shared tiles what a wave's meeting costs beyond what long sums hide.
inline double tile_cost(const TileCost& c, bool shared, long long tiles, int K, int sms) {
    auto room = [&](int blocks) { return shared ? clusters_at(blocks, sms) : (long long)blocks * sms; };
    const long long full = room(c.levels) > 0 ? room(c.levels) : 1, before = (tiles - 1) / full, last = tiles - before * full;
    // (behind full waves the ring stays at two chunks: from half of a wave on some multiprocessors then hold three blocks)
    auto fits = [&](int blocks) { return shared && before > 0 && blocks == 2 && c.levels == 3 ? room(3) / 2 : room(blocks); };
    int level = 1;
    while (level < c.levels && last > fits(level)) ++level;
    const double held = (double)RUNS * ((run_length(K) + KC - 1) / KC * KC) / 9216;
    return shared ? held * (before * c.shared_on + c.shared[level - 1]) + 0.8 * (before + 1) : held * RUNS * (before * c.whole_on + c.whole[level - 1]);
}

// The form whose waves cost least.  Of 245 products of 96 to 28,672 outputs and 20 to 2,048 rows it takes one within 5 % of the best
// form in 239.  Microseconds by form, s: shared by eight blocks, * what is taken; in brackets what a rule on the rows alone took
// (tiles of 32, 48 or 64 rows up to 96, then 64 or 128 by the multiprocessors that tiles of 128 give one):
//   2,304 outputs of 9,216    32 rows  32s 83*   48 rows  32s 114  48s 109*   64 rows  32s 114* (138)  48s 155  64s 138    90 rows  32s 152  48s 155*  64s 205
//                            120 rows  32s 194* (208)  48s 203  64s 207  128s 258     200 rows  32s 301  48s 306*  64s 334 (334)  128s 386
//                            700 rows  48s 798  64s 811* (1,129)  64 1,131  128 1,053  128s 1,037
//   18,432 outputs of 2,304   48 rows  32s 171  48s 121*  64s 164   64 rows  32s 171  64s 165*  64 173   120 rows  32 317  64 294  128 277*    900 rows  48 1,984* (2,199)
//   3,584 outputs of 14,336   64 rows  32s 235  64s 212*   128 rows  32s 415  64s 429 (429)  128s 396*   160 rows  32s 509* (603)  64s 604   512 rows  48s 1,385* (1,753)  128 1,627
//   8,192 outputs of 3,584    96 rows  48s 165*   256 rows  32s 441  64s 419  128 421* (449)   384 rows  48s 588* (697)  64s 622  128 838
//   256 outputs of 96         64 rows  32s 4.1* (5.9)  64s 5.9          768 outputs of 3,072   600 rows  48s 102  128s 93*
//   8,000 outputs of 300     400 rows  48s 123  64 108*      800 rows  48s 227  128 212*
inline TileForm tile_form(int M, int N, int K, int sms) {
    TileForm best = {0, 0, false};
    double least = 0;
    for (const TileCost& c : TILE_COSTS) {
        const long long down = ((long long)M + c.rows - 1) / c.rows, tiles = (N + (long long)BN - 1) / BN * down;
        if (down > 65535 && c.rows < 64) continue;               // the grid's height
        for (const bool shared : {true, false}) {
            const double cost = tile_cost(c, shared, tiles, K, sms);
            if (best.rows && cost >= least) continue;
            least = cost;
            // Three chunks, which leave room for two blocks a multiprocessor, where all tiles find room in that way and with two chunks
            // some multiprocessors would hold three blocks, others one (48 rows of 2,304 terms: 24 tiles 31.2 us with two chunks, 32.1
            // with three; 25 tiles 41.2 and 32.1, 32 tiles 41.4 and 32.7; fewer tiles take 20 either way).  Five chunks and one block
            // never won: up to 15 tiles 20 us, from 16 on, which are two waves, 38.
            const bool three = c.rows == 128 || (c.rows < 64 && shared && 2 * tiles > clusters_at(3, sms) && tiles <= clusters_at(2, sms));
            best = {c.rows, three ? 3 : 2, shared};
        }
    }
    return best;
}

template <bool ALIGNED>
cudaError_t launch_rows(float* out, const float* x, const float* w, int M, int N, int K, cudaStream_t st) {
    if (M <= FEW_MAX) return launch_few_rows<ALIGNED>(out, x, w, M, N, K, st);
    const TileForm f = tile_form(M, N, K, rdl_sm_count());
    if (f.rows == 32) return !f.shared ? launch_tile<4, 8, 2, false, ALIGNED>(out, x, w, M, N, K, st)
                             : f.chunks == 2 ? launch_tile<4, 8, 2, true, ALIGNED>(out, x, w, M, N, K, st)
                                             : launch_tile<4, 8, 3, true, ALIGNED>(out, x, w, M, N, K, st);
    if (f.rows == 48) return !f.shared ? launch_tile<6, 8, 2, false, ALIGNED>(out, x, w, M, N, K, st)
                             : f.chunks == 2 ? launch_tile<6, 8, 2, true, ALIGNED>(out, x, w, M, N, K, st)
                                             : launch_tile<6, 8, 3, true, ALIGNED>(out, x, w, M, N, K, st);
    if (f.rows == 64) return f.shared ? launch_tile<8, 8, 2, true, ALIGNED>(out, x, w, M, N, K, st) : launch_tile<8, 8, 2, false, ALIGNED>(out, x, w, M, N, K, st);
    return f.shared ? launch_tile<8, 16, 3, true, ALIGNED>(out, x, w, M, N, K, st) : launch_tile<8, 16, 3, false, ALIGNED>(out, x, w, M, N, K, st);
}

}  // namespace

// The form a product takes on so many multiprocessors: 100 x rows of a tile + 10 x chunks of the ring + 1 where eight blocks share a tile;
// 0: the few-row kernel.
extern "C" int rdl_gemm_f32_form(int m, int n, int k, int sms) {
    if (m <= FEW_MAX) return 0;
    const TileForm f = tile_form(m, n, k, sms);
    return 100 * f.rows + 10 * f.chunks + (f.shared ? 1 : 0);
}

extern "C" int rdl_gemm_f32(void* out, const void* x, const void* w, int m, int n, int k, void* stream) {
    RDL_REQUIRE(m >= 0 && n > 0 && k > 0, "gemm_f32: bad sizes m=%d n=%d k=%d", m, n, k);
    RDL_REQUIRE(out && x && w, "gemm_f32: missing operand");
    if (m == 0) return 0;
    RDL_REQUIRE((m + 63) / 64 <= 65535, "gemm_f32: %d rows exceed the grid limit", m);
    const bool aligned = k % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0;
    cudaStream_t st = (cudaStream_t)stream;
    RDL_CHECK_EX(aligned ? launch_rows<true>((float*)out, (const float*)x, (const float*)w, m, n, k, st)
                         : launch_rows<false>((float*)out, (const float*)x, (const float*)w, m, n, k, st), "gemm_f32");
    return 0;
}
