// grouped.cu — persistent grouped FP32 GEMM: many independent (M, N, K)
// problems in one launch, plus its autotuner.
//
// No reference counterpart (the reference launches one GEMM per call,
// src/sgemm.cuh:19-48); every problem keeps sgemm()'s contract.
//
// Design:
//  - The plan flattens every problem into work items (tile_m, tile_n, k
//    split), sorted longest-first so the tail of the launch is short items.
//  - Persistent 4-warp CTAs (2 or 3 per SM) claim items with an atomic
//    counter and run the same FFMA core as the plain path on each: one of three
//    tile shapes and one of three ways to read the operands (load_of), chosen
//    per problem at plan time; the tensor maps are kept in global memory.
//  - A launch is two kernels, chained: one transposes A (and copies rows TMA
//    cannot describe) for the problems that read prepared operands and resets
//    the tickets, the other runs the items.  What bounds the items is the FMA
//    pipe, and with A [row][k] its register reads: a server's 32 requests took
//    9435 us that way (57.9 TFLOP/s), 8486 with A transposed (64.3, the pass
//    included; 86% of the FP32 peak); 24 odd problems of 300..3000 2245 -> 995.
//  - Without memory for the prepared operands every problem is read in place.
//  - Items with split == 1 run the plain path's exact arithmetic, so their
//    results equal sgemm_b200's bit for bit.  Split-K items write partial sums
//    to a workspace; the last split of a tile to finish (atomic ticket) adds
//    the partials in split order 0, 1, 2, ... and applies alpha/beta, so the
//    result is deterministic and independent of scheduling.
//  - The launch is captured once into a CUDA graph
//    and replayed.
//  - Tile shape, split-K and stage count per size bucket come from the
//    autotuner (sgemm_b200_autotune_grouped), persisted as JSON keyed by the
//    device name and SM count.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <mutex>
#include <numeric>
#include <sstream>
#include <string>
#include <type_traits>
#include <vector>

#include "common.h"
#include "ffma_kernel.cuh"
#include "grouped.h"
#include "plain.h"
#include "transpose.cuh"

namespace sgb {
namespace grouped {

using ffma::Operands;

// Three tile shapes of the plain path's 4-warp FFMA core share one kernel
// (same thread count, one 24 KB shared-memory slot per stage): 128 x 64 and
// 64 x 128 with 8 x 8 threads, and 32 x 128 with 8 x 4 threads for problems
// only a few rows tall, whose rows a 64- or 128-row tile would mostly pad
// with zeros.  3 stages fit 3 CTAs per SM, 4 stages fit 2.
template <int S>
using CfgT = ffma::Cfg<128, 64, 4, 1, 8, S, ffma::kLoaderAsync4, (S == 3 ? 3 : 2)>;  // 128 x 64
template <int S>
using CfgW = ffma::Cfg<64, 128, 2, 2, 8, S, ffma::kLoaderAsync4, (S == 3 ? 3 : 2)>;  // 64 x 128
template <int S>
using CfgS = ffma::Cfg<32, 128, 1, 4, 4, S, ffma::kLoaderAsync4, (S == 3 ? 3 : 2)>;  // 32 x 128

// The same tiles on A transposed (compute_stage_kmajor).
template <int S>
using KmT = ffma::Cfg<128, 64, 4, 1, 8, S, ffma::kLoaderTma, (S == 3 ? 3 : 2), 8, true>;
template <int S>
using KmW = ffma::Cfg<64, 128, 2, 2, 8, S, ffma::kLoaderTma, (S == 3 ? 3 : 2), 8, true>;
template <int S>
using KmS = ffma::Cfg<32, 128, 1, 4, 4, S, ffma::kLoaderTma, (S == 3 ? 3 : 2), 8, true>;

constexpr int THREADS = 128;
constexpr int SLOT_BYTES = 24 * 1024;  // 16 KB + 8 KB per 32-deep k block (4 + 16 KB skinny)
static_assert(CfgT<3>::STAGE_BYTES == SLOT_BYTES && CfgW<3>::STAGE_BYTES == SLOT_BYTES &&
                  CfgS<3>::STAGE_BYTES <= SLOT_BYTES && CfgS<3>::THREADS == THREADS &&
                  KmT<3>::STAGE_BYTES == SLOT_BYTES && KmW<3>::STAGE_BYTES == SLOT_BYTES &&
                  KmS<3>::STAGE_BYTES <= SLOT_BYTES && KmS<3>::COMPUTE_THREADS == THREADS,
              "");
enum TileShape { kTileTall = 0, kTileWide = 1, kTileSkinny = 2 };  // 128x64, 64x128, 32x128

inline int tile_bm(int t) { return t == kTileTall ? 128 : t == kTileWide ? 64 : 32; }
inline int tile_bn(int t) { return t == kTileTall ? 64 : 128; }

// Throughput of each tile relative to 128 x 64 on work that fills them
// (measured on a B200 with single-GEMM kernels of the same shapes).  A
// problem leaves its bucket's tile for another when that tile's zero-padded
// area divided by its efficiency is at least 2% smaller.
inline double tile_efficiency(int t) {
    return t == kTileTall ? 1.0 : t == kTileWide ? 0.994 : 0.75;
}

// How a problem's tiles are read: in place by 4-byte cp.async (strides or bases
// TMA cannot describe), in place by TMA, or by TMA from a transposed copy of A
// (and, where needed, a copy of B in aligned rows) that the launch makes first.
enum Load { kLoadAsync4 = 0, kLoadRows = 1, kLoadTransposed = 2 };

struct GProblem {
    Operands op;
    int tile;      // a TileShape: the tile of the problem's rows (all of them,
                   // or the bulk when `rem_tile` covers a remainder strip)
    int rem_tile;  // tile of the last rows when they are a strip of their own, else -1
    int rem_m0;    // first row of that strip
    int shapes;    // bit t: the problem has tiles of shape t (a map pair per shape)
    int load;      // a Load: how the problem's tiles reach shared memory
    int pack_b;    // B is copied to aligned rows first (kLoadTransposed only)
    int split;     // k splits
    int kbps;      // k blocks per split
    int depth;     // k blocks kept in flight through the stage ring (2..S)
    int tiles_n;
    int cnt_base;  // first tile ticket (split > 1)
    long long ws_base;  // first workspace float (split > 1)
};

// One work item: a tile of one problem (its shape, its first row and column)
// and one k split.  tl is the tile's index within its problem (split-K
// tickets and partials), used only when the problem is split.
struct GItem {
    int prob, m0, n0, ks;
    int tile, tl;
};

// One matrix that the launch prepares: A transposed, or B copied to aligned
// rows, by 64 x 64 tiles; its tiles are blocks first, first + 1, ...
struct GPrep {
    ffma::TransposeJob job;
    int copy;
    int first;
};

struct GParams {
    const GProblem* probs;
    const GItem* items;
    const CUtensorMap* maps;  // 6 per problem: (A, B) for each tile shape it uses
    float* ws;
    int* counters;  // [0] work ticket, [1..] split-K tile tickets
    int* status;
    int n_items;
};

template <int S>
constexpr int smem_bytes() {
    return S * SLOT_BYTES + 1024;
}

// One work item on the FFMA core.  Returns false (uniformly across the CTA)
// if a bounded wait expired.
template <class C, int LOAD, int S>
__device__ __forceinline__ bool run_item(const GParams& gp, const GProblem& pr, const GItem& it,
                                         int item_prob, uint8_t* smem, uint64_t* full_bar,
                                         uint32_t& g, int* last_s) {
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const int wm = warp / C::WN, wn = warp % C::WN;
    int lm, ln;
    C::lane_coords(lane, lm, ln);
    const int m0 = it.m0, n0 = it.n0;
    const int nk = (pr.op.k + C::BK - 1) / C::BK;
    const int kb0 = it.ks * pr.kbps;
    const int kb1 = min(nk, kb0 + pr.kbps);
    const int nkb = max(0, kb1 - kb0);

    uint32_t a_base = 0, xa0 = 0, xa1 = 0;  // A's offsets when it stays [row][k]
    if constexpr (!C::KM) ffma::a_coords<C>(wm, lm, a_base, xa0, xa1);
    const uint32_t b_base = static_cast<uint32_t>((wn * 8 * C::TN + ln * 4) * 4);

    float acc[C::TM][C::TN];
#pragma unroll
    for (int i = 0; i < C::TM; ++i)
#pragma unroll
        for (int j = 0; j < C::TN; ++j) acc[i][j] = 0.0f;

    if constexpr (LOAD != kLoadAsync4) {
        const CUtensorMap* tmA = gp.maps + 6 * item_prob + 2 * it.tile;
        const CUtensorMap* tmB = tmA + 1;
        int issued = 0;
        auto issue = [&](int j) {
            const uint32_t gs = g + j;
            const int s = gs % S;
            uint8_t* st = smem + s * SLOT_BYTES;
            mbar_arrive_expect_tx(&full_bar[s], C::A_TX + C::B_BYTES);
            if constexpr (C::KM)
                tma_load_2d(st, tmA, &full_bar[s], m0, (kb0 + j) * C::BK);
            else
                tma_load_2d(st, tmA, &full_bar[s], (kb0 + j) * C::BK, m0);
            tma_load_2d(st + C::A_BYTES, tmB, &full_bar[s], n0, (kb0 + j) * C::BK);
        };
        if (tid == 0) {
            const int depth = min(S, pr.depth);  // the bucket's stage count
            // the previous item's generic reads of the ring (ordered by the CTA
            // barrier between items) before these TMA refills
            fence_proxy_async_shared();
            for (; issued < depth && issued < nkb; ++issued) issue(issued);
        }
        for (int j = 0; j < nkb; ++j) {
            const uint32_t gs = g + j;
            const int s = gs % S;
            const bool ok = mbar_wait(&full_bar[s], (gs / S) & 1);
            if (__syncthreads_or(!ok)) {
                if (tid == 0) {
                    atomicExch(gp.status, SGEMM_B200_ERR_TIMEOUT);
                    for (int q = j; q < issued; ++q)
                        if (!mbar_wait(&full_bar[(g + q) % S], ((g + q) / S) & 1)) break;
                }
                return false;
            }
            if (tid == 0 && j > 0 && issued < nkb) {
                fence_proxy_async_shared();  // generic reads of the stage before its TMA refill
                issue(issued++);
            }
            const uint8_t* st = smem + s * SLOT_BYTES;
            if constexpr (C::KM)
                ffma::compute_stage_kmajor<C>(st, st + C::A_BYTES, wm, lm, b_base, acc);
            else
                ffma::compute_stage<C>(st, st + C::A_BYTES, a_base, xa0, xa1, b_base, acc);
        }
        g += nkb;
    } else {
#pragma unroll
        for (int s = 0; s < S - 1; ++s) {
            if (s < nkb) {
                uint8_t* st = smem + s * SLOT_BYTES;
                ffma::load_stage_async4<C>(pr.op, st, st + C::A_BYTES, m0, n0, (kb0 + s) * C::BK,
                                           tid);
            }
            cp_async_commit();
        }
        for (int j = 0; j < nkb; ++j) {
            cp_async_wait<S - 2>();
            __syncthreads();
            const int nxt = j + S - 1;
            if (nxt < nkb) {
                uint8_t* st = smem + (nxt % S) * SLOT_BYTES;
                ffma::load_stage_async4<C>(pr.op, st, st + C::A_BYTES, m0, n0, (kb0 + nxt) * C::BK,
                                           tid);
            }
            cp_async_commit();
            const uint8_t* st = smem + (j % S) * SLOT_BYTES;
            ffma::compute_stage<C>(st, st + C::A_BYTES, a_base, xa0, xa1, b_base, acc);
        }
        cp_async_wait<0>();
    }

    // epilogue with C read row by row (BATCH 0): batched C loads cost this
    // kernel spills under its register cap
    if (pr.split == 1) {
        ffma::epilogue_any<C, 0>(pr.op, m0, n0, wm, wn, lm, ln, acc, smem);
        return true;
    }

    // ---- split-K: publish the partial, the last split of the tile reduces.
    constexpr int NQ = C::TM * C::TN / 4;
    constexpr int TILE = C::BM * C::BN;
    const int tile_local = it.tl;
    float4* tile_ws = reinterpret_cast<float4*>(gp.ws + pr.ws_base +
                                                (long long)tile_local * pr.split * TILE);
    float4* mine = tile_ws + (long long)it.ks * (TILE / 4);
#pragma unroll
    for (int i = 0; i < C::TM; ++i)
#pragma unroll
        for (int q = 0; q < C::TN / 4; ++q)
            __stcg(&mine[(i * (C::TN / 4) + q) * THREADS + tid],
                   make_float4(acc[i][4 * q], acc[i][4 * q + 1], acc[i][4 * q + 2],
                               acc[i][4 * q + 3]));
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const int prev = atomicAdd(&gp.counters[1 + pr.cnt_base + tile_local], 1);
        *last_s = prev == pr.split - 1;
    }
    __syncthreads();
    if (*last_s) {
        __threadfence();
        for (int s = 0; s < pr.split; ++s) {
            const float4* part = tile_ws + (long long)s * (TILE / 4);
#pragma unroll
            for (int i = 0; i < C::TM; ++i)
#pragma unroll
                for (int q = 0; q < C::TN / 4; ++q) {
                    const float4 v = __ldcg(&part[(i * (C::TN / 4) + q) * THREADS + tid]);
                    if (s == 0) {
                        acc[i][4 * q] = v.x;
                        acc[i][4 * q + 1] = v.y;
                        acc[i][4 * q + 2] = v.z;
                        acc[i][4 * q + 3] = v.w;
                    } else {
                        acc[i][4 * q] = __fadd_rn(acc[i][4 * q], v.x);
                        acc[i][4 * q + 1] = __fadd_rn(acc[i][4 * q + 1], v.y);
                        acc[i][4 * q + 2] = __fadd_rn(acc[i][4 * q + 2], v.z);
                        acc[i][4 * q + 3] = __fadd_rn(acc[i][4 * q + 3], v.w);
                    }
                }
        }
        (void)NQ;
        ffma::epilogue_any<C, 0>(pr.op, m0, n0, wm, wn, lm, ln, acc, smem);
    }
    return true;
}

template <int S>
__global__ void __launch_bounds__(THREADS, (S == 3 ? 3 : 2)) grouped_kernel(const GParams gp) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[S];
    __shared__ int item_s;
    __shared__ int last_s;
    uint8_t* smem = align_smem_1024(smem_raw);
    const int tid = threadIdx.x;
    if (tid == 0) {
        for (int s = 0; s < S; ++s) mbar_init(&full_bar[s], 1);
        fence_barrier_init();
    }
    __syncthreads();
    grid_wait();
    uint32_t g = 0;  // k blocks consumed through the TMA ring (phase tracking)
    // The first item by block index: blocks are spread over the SMs in order, so
    // the longest items do not share one, as they may when the resident CTAs of a
    // chained launch all claim at once (12 uneven problems 349 us, 211 so).
    for (bool first = true;; first = false) {
        if (tid == 0)
            item_s = first ? (int)blockIdx.x : (int)gridDim.x + atomicAdd(&gp.counters[0], 1);
        __syncthreads();
        const int idx = item_s;
        if (idx >= gp.n_items) break;

        const GItem it = gp.items[idx];
        const GProblem& pr = gp.probs[it.prob];
        bool ok;
        auto run = [&](auto* km, auto* rows) {
            using K = std::remove_pointer_t<decltype(km)>;
            using R = std::remove_pointer_t<decltype(rows)>;
            ok = pr.load == kLoadTransposed
                     ? run_item<K, kLoadTransposed, S>(gp, pr, it, it.prob, smem, full_bar, g,
                                                       &last_s)
                 : pr.load == kLoadRows
                     ? run_item<R, kLoadRows, S>(gp, pr, it, it.prob, smem, full_bar, g, &last_s)
                     : run_item<R, kLoadAsync4, S>(gp, pr, it, it.prob, smem, full_bar, g,
                                                   &last_s);
        };
        if (it.tile == kTileTall)
            run((KmT<S>*)nullptr, (CfgT<S>*)nullptr);
        else if (it.tile == kTileSkinny)
            run((KmS<S>*)nullptr, (CfgS<S>*)nullptr);
        else
            run((KmW<S>*)nullptr, (CfgW<S>*)nullptr);
        if (!ok) break;
        __syncthreads();  // stages and item_s are free for the next item
    }
}

// Before the grouped kernel: block 0 resets its tickets, the others prepare a
// 64 x 64 tile each.  HBM-bound.
constexpr int kPrepThreads = 256;
__global__ void __launch_bounds__(kPrepThreads)
    grouped_prepare_kernel(const GPrep* preps, int count, int* counters, int n_counters) {
    __shared__ float tile[ffma::kTrTile][ffma::kTrTile + 1];
    grid_wait();
    if (blockIdx.x == 0) {
        for (int i = threadIdx.x; i < n_counters; i += kPrepThreads) counters[i] = 0;
        return;
    }
    const int b = blockIdx.x - 1;
    int lo = 0, hi = count - 1;  // the last matrix whose first block is <= b
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (preps[mid].first <= b)
            lo = mid;
        else
            hi = mid - 1;
    }
    const GPrep p = preps[lo];
    if (!p.copy) {
        ffma::transpose_tile(p.job, b - p.first, tile);
        return;
    }
    const int tk = (p.job.k + ffma::kTrTile - 1) / ffma::kTrTile;
    const int c = (b - p.first) % tk * ffma::kTrTile + threadIdx.x % 64;
    const int r0 = (b - p.first) / tk * ffma::kTrTile + threadIdx.x / 64;
    float v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i)
        v[i] = c < p.job.k && r0 + 4 * i < p.job.m
                   ? p.job.src[(int64_t)(r0 + 4 * i) * p.job.ld_src + c]
                   : 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i)
        if (c < p.job.k && r0 + 4 * i < p.job.m)
            p.job.dst[(int64_t)(r0 + 4 * i) * p.job.ld_dst + c] = v[i];
}

// ------------------------------------------------------------------ host --

struct Choice {
    int tile = kTileTall;
    int split = 1;
    int depth = 4;  // stage count: k blocks in flight (capped by the launch's ring)
};

// Size buckets: M*N class x K class.
constexpr int kMnClasses = 3, kKClasses = 3, kBuckets = kMnClasses * kKClasses;
inline int bucket_of(int m, int n, int k) {
    const double mn = double(m) * n;
    const int a = mn < 256.0 * 256.0 ? 0 : (mn < 1024.0 * 1024.0 ? 1 : 2);
    const int b = k < 512 ? 0 : (k < 2048 ? 1 : 2);
    return a * kKClasses + b;
}

// The tuning table: the launch's ring size (3 stages and 3 CTAs per SM, or 4
// and 2) and, per size bucket, tile shape, split-K and stage count (how many
// of the ring's stages a problem's items keep in flight).
struct Table {
    int stages = 3;
    Choice c[kBuckets];
};

static bool load_table(const char* path, Table* t) {
    std::ifstream f(path);
    if (!f) return false;
    std::string line, dev_name;
    int sms = -1, stages = -1;
    Table out;
    int seen = 0;
    while (std::getline(f, line)) {
        const size_t d = line.find("\"device\"");
        if (d != std::string::npos) {
            const size_t a = line.find('"', line.find(':', d) + 1);
            const size_t b = line.find('"', a + 1);
            if (a != std::string::npos && b != std::string::npos)
                dev_name = line.substr(a + 1, b - a - 1);
        }
        if (line.find("\"sm_count\"") != std::string::npos)
            std::sscanf(line.c_str() + line.find(':') + 1, "%d", &sms);
        // the launch's ring size (bucket lines carry their own "stages")
        if (line.find("\"stages\"") != std::string::npos &&
            line.find("{\"mn\"") == std::string::npos)
            std::sscanf(line.c_str() + line.find(':') + 1, "%d", &stages);
        int mn, kc, tile, split, depth = 4;
        const size_t p = line.find("{\"mn\"");
        if (p != std::string::npos &&
            std::sscanf(line.c_str() + p,
                        "{\"mn\": %d, \"k\": %d, \"tile\": %d, \"split\": %d, \"stages\": %d", &mn,
                        &kc, &tile, &split, &depth) >= 4 &&
            mn >= 0 && mn < kMnClasses && kc >= 0 && kc < kKClasses && tile >= 0 && tile <= 2 &&
            split >= 1 && split <= 16 && depth >= 2 && depth <= 4) {
            out.c[mn * kKClasses + kc].tile = tile;
            out.c[mn * kKClasses + kc].split = split;
            out.c[mn * kKClasses + kc].depth = depth;
            ++seen;
        }
    }
    const DeviceInfo& di = device_info();
    // A table tuned on another GPU model or SM count does not apply here.
    if (dev_name != di.name || sms != di.sm_count) return false;
    if (stages == 3 || stages == 4) out.stages = stages;
    *t = out;
    return seen > 0;
}

static bool save_table(const char* path, const Table& t) {
    std::ofstream f(path);
    if (!f) return false;
    const DeviceInfo& di = device_info();
    f << "{\n \"format\": \"sgemm_b200 grouped tuning v2\",\n";
    f << " \"device\": \"" << di.name << "\",\n";
    f << " \"sm_count\": " << di.sm_count << ",\n";
    f << " \"stages\": " << t.stages << ",\n";
    f << " \"buckets\": [\n";
    for (int a = 0; a < kMnClasses; ++a)
        for (int b = 0; b < kKClasses; ++b) {
            const Choice& ch = t.c[a * kKClasses + b];
            f << "  {\"mn\": " << a << ", \"k\": " << b << ", \"tile\": " << ch.tile
              << ", \"split\": " << ch.split << ", \"stages\": " << ch.depth << "}"
              << (a == kMnClasses - 1 && b == kKClasses - 1 ? "\n" : ",\n");
        }
    f << " ]\n}\n";
    return bool(f);
}

static bool tma_ok(int k, const float* A, int lda, const float* B, int ldb) {
    return k > 0 && lda % 4 == 0 && ldb % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0 &&
           reinterpret_cast<uintptr_t>(B) % 16 == 0;
}

}  // namespace grouped
}  // namespace sgb

struct sgemm_b200_grouped_plan {
    int device = -1;
    int stages = 4;
    int n_items = 0;
    int n_tiles = 0;
    int grid = 0;
    size_t ws_floats = 0;
    int n_counters = 0;
    uint8_t* d_block = nullptr;  // what follows it, one allocation
    sgb::grouped::GProblem* d_probs = nullptr;
    sgb::grouped::GItem* d_items = nullptr;
    CUtensorMap* d_maps = nullptr;
    float* d_ws = nullptr;
    float* d_scratch = nullptr;  // transposed A (and copied B) of the problems that use them
    size_t scratch_bytes = 0;    // of kScratchKept
    sgb::grouped::GPrep* d_preps = nullptr;
    int n_preps = 0, prep_tiles = 0;
    int* d_counters = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t cap_stream = nullptr;
};

namespace sgb {
namespace grouped {

// Bytes of scratch that a device's plans hold together: at most kScratchKept.
static size_t g_plan_scratch[64];
static std::mutex g_plan_scratch_mu;

static void give_plan_scratch(sgemm_b200_grouped_plan* p) {
    std::lock_guard<std::mutex> lock(g_plan_scratch_mu);
    if (p->scratch_bytes) g_plan_scratch[p->device] -= p->scratch_bytes;
    p->scratch_bytes = 0;
}

static void free_plan(sgemm_b200_grouped_plan* p) {
    if (!p) return;
    if (p->exec) cudaGraphExecDestroy(p->exec);
    if (p->graph) cudaGraphDestroy(p->graph);
    if (p->cap_stream) cudaStreamDestroy(p->cap_stream);
    cudaFree(p->d_block);
    cudaFree(p->d_ws);
    give_plan_scratch(p);
    pool_free(p->d_scratch);  // after the frees that wait for the device
    delete p;
}

// Host-only part of a plan: per-problem choices and the longest-first item list.
struct Schedule {
    std::vector<GProblem> probs;
    std::vector<GItem> items;
    long long ws_floats = 0;
    int tickets = 0;
    int tiles = 0;
    size_t scratch_floats = 0;  // prepared operands (kLoadTransposed)
};

// Which problems read prepared operands (the launch has a pass before its items
// anyway, which resets the tickets).
//  - Aligned operands: A transposed pays from 512 columns on, where the faster
//    FMA loop (64 TFLOP/s from 58) outweighs moving 8 m k bytes.  48 problems of
//    512 x n x 1024, transposed against in place: n = 512 466 us against 489,
//    n = 1024 845 against 907.
//  - Operands TMA cannot describe: the copies beat the 4-byte loader, whose k
//    block costs about 4 us of latency, wherever there is more than one block.
constexpr int kTransposeMinN = 512;
constexpr double kTransposeMinWork = 32.0e6;  // m n k

static int load_of(const sgemm_b200_problem& p) {
    if (p.m == 0 || p.n == 0) return kLoadAsync4;  // no items, and no map over nothing
    const bool in_place = tma_ok(p.k, p.A, p.lda, p.B, p.ldb);
    const double work = double(p.m) * p.n * p.k;
    if (in_place)
        return p.n >= kTransposeMinN && work >= kTransposeMinWork ? kLoadTransposed : kLoadRows;
    return p.k > 32 ? kLoadTransposed : kLoadAsync4;
}

// Floats of a prepared matrix of `rows` rows of `cols` (32-byte rows, 256-byte start).
inline int prep_pitch(int cols) { return div_up(cols, 8) * 8; }
inline size_t prep_floats(int rows, int cols) {
    return ((size_t)rows * prep_pitch(cols) + 63) / 64 * 64;
}

static int make_schedule(const sgemm_b200_problem* probs, int count, const Table& table,
                         Schedule* out) {
    if (count < 0 || (count > 0 && !probs)) return SGEMM_B200_ERR_INVALID_ARG;
    for (int i = 0; i < count; ++i) {
        const sgemm_b200_problem& q = probs[i];
        const int s = check_gemm_args(q.m, q.n, q.k, &q.alpha, q.A, q.lda, q.B, q.ldb, &q.beta,
                                      q.C, q.ldc);
        if (s != SGEMM_B200_OK) return s;
    }
    Schedule sc;
    sc.probs.resize(count);
    struct Weighted {
        GItem it;
        double cost;
    };
    std::vector<Weighted> items;
    for (int i = 0; i < count; ++i) {
        const sgemm_b200_problem& q = probs[i];
        GProblem& g = sc.probs[i];
        g.op.m = q.m;
        g.op.n = q.n;
        g.op.k = q.k;
        g.op.lda = q.lda;
        g.op.ldb = q.ldb;
        g.op.ldc = q.ldc;
        g.op.alpha = q.alpha;
        g.op.beta = q.beta;
        g.op.A = q.A;
        g.op.B = q.B;
        g.op.C = q.C;
        g.op.vec_c = (q.ldc % 4 == 0) && (reinterpret_cast<uintptr_t>(q.C) % 16 == 0);
        const Choice ch = table.c[bucket_of(q.m, q.n, q.k)];
        // Padded area per unit efficiency of covering `rows` rows with tile t.
        auto area = [&](int rows, int t) {
            return double(div_up(rows, tile_bm(t)) * tile_bm(t)) *
                   double(div_up(q.n, tile_bn(t)) * tile_bn(t)) / tile_efficiency(t);
        };
        // Problem geometry: a problem a few rows tall (the 32 x 128 tile) or
        // one whose edges fit the other 8 x 8 tile better loses less work to
        // zero padding on that tile.
        int best = ch.tile;
        for (int t : {kTileTall, kTileWide, kTileSkinny})
            if (area(q.m, t) < 0.98 * area(q.m, ch.tile) && area(q.m, t) < area(q.m, best)) best = t;
        g.tile = best;
        g.rem_tile = -1;
        g.rem_m0 = q.m;
        const int nk = div_up(q.k, 32);
        int split = std::max(1, std::min(ch.split, nk));
        g.kbps = nk > 0 ? div_up(nk, split) : 0;
        if (g.kbps > 0) split = div_up(nk, g.kbps);  // no empty splits
        g.split = split;
        g.depth = ch.depth;
        if (split == 1 && q.m > 0 && q.n > 0) {
            // Rows may also be covered by two tiles: the whole tiles of a
            // taller shape, then the leftover rows as a strip of a shorter
            // one (every element still runs its whole k-ordered chain in one
            // item, so the result is the same).  Taken when it pads at least
            // 2% less than the single tile.
            double best_area = area(q.m, best);
            for (int t : {kTileTall, kTileWide})
                for (int u : {kTileWide, kTileSkinny}) {
                    if (tile_bm(u) >= tile_bm(t)) continue;
                    const int bulk = q.m / tile_bm(t) * tile_bm(t);
                    if (bulk == 0 || bulk == q.m) continue;
                    const double a = area(bulk, t) + area(q.m - bulk, u);
                    if (a < 0.98 * best_area) {
                        best_area = a;
                        g.tile = t;
                        g.rem_tile = u;
                        g.rem_m0 = bulk;
                    }
                }
        }
        g.load = load_of(q);
        g.pack_b = g.load == kLoadTransposed &&
                   (q.ldb % 4 != 0 || reinterpret_cast<uintptr_t>(q.B) % 16 != 0);
        if (g.load == kLoadTransposed)
            sc.scratch_floats +=
                prep_floats(q.k, q.m) + (g.pack_b ? prep_floats(q.k, q.n) : 0);
        g.shapes = (1 << g.tile) | (g.rem_tile >= 0 ? 1 << g.rem_tile : 0);
        const int bm = tile_bm(g.tile), bn = tile_bn(g.tile);
        const int tm = q.m > 0 ? div_up(g.rem_m0, bm) : 0;
        const int tn = q.n > 0 ? div_up(q.n, bn) : 0;
        g.tiles_n = tn;
        g.cnt_base = sc.tickets;
        g.ws_base = sc.ws_floats;
        if (split > 1) {
            sc.tickets += tm * tn;
            sc.ws_floats += (long long)tm * tn * split * bm * bn;
        }
        // cost ~ FMAs of the item plus a fixed pipeline fill / epilogue term
        auto add = [&](int tile, int m0, int n0, int tl, int ks) {
            const int kb = std::min(g.kbps, nk - ks * g.kbps);
            const double c = double(tile_bm(tile)) * tile_bn(tile) * (std::max(kb, 0) + 6) * 32;
            items.push_back({GItem{i, m0, n0, ks, tile, tl}, c});
        };
        for (int a = 0; a < tm; ++a)
            for (int b = 0; b < tn; ++b)
                for (int ks = 0; ks < split; ++ks) add(g.tile, a * bm, b * bn, a * tn + b, ks);
        sc.tiles += tm * tn;
        if (g.rem_tile >= 0) {  // the remainder strip (split == 1 only)
            const int rbm = tile_bm(g.rem_tile), rbn = tile_bn(g.rem_tile);
            const int rtm = div_up(q.m - g.rem_m0, rbm), rtn = div_up(q.n, rbn);
            for (int a = 0; a < rtm; ++a)
                for (int b = 0; b < rtn; ++b) add(g.rem_tile, g.rem_m0 + a * rbm, b * rbn, 0, 0);
            sc.tiles += rtm * rtn;
        }
    }
    std::stable_sort(items.begin(), items.end(),
                     [](const Weighted& x, const Weighted& y) { return x.cost > y.cost; });
    sc.items.resize(items.size());
    for (size_t i = 0; i < items.size(); ++i) sc.items[i] = items[i].it;
    *out = std::move(sc);
    return SGEMM_B200_OK;
}

// The matrices a launch prepares, laid out in `scratch` in problem order; returns
// their 64 x 64 tiles.
static int make_preps(const Schedule& sc, float* scratch, std::vector<GPrep>* out) {
    int tiles = 0;
    size_t used = 0;
    auto add = [&](const float* src, int rows, int cols, int ld, bool copy) {
        GPrep p;
        p.job.src = src;
        p.job.dst = scratch + used;
        p.job.m = rows;
        p.job.k = cols;
        p.job.ld_src = ld;
        p.job.ld_dst = prep_pitch(copy ? cols : rows);
        p.job.sevens = 0;
        p.job.vec = ld % 4 == 0 && reinterpret_cast<uintptr_t>(src) % 16 == 0;
        p.job.blocks = 0;
        p.copy = copy;
        p.first = tiles;
        used += copy ? prep_floats(rows, cols) : prep_floats(cols, rows);
        tiles += div_up(rows, ffma::kTrTile) * div_up(cols, ffma::kTrTile);
        out->push_back(p);
    };
    for (const GProblem& g : sc.probs) {
        if (g.load != kLoadTransposed) continue;
        add(g.op.A, g.op.m, g.op.k, g.op.lda, false);
        if (g.pack_b) add(g.op.B, g.op.k, g.op.n, g.op.ldb, true);
    }
    return tiles;
}

// At most `floats` of scratch: problems whose prepared matrices do not fit beside
// those before them are read in place.
static void limit_scratch(Schedule* sc, size_t floats) {
    size_t used = 0;
    for (GProblem& g : sc->probs) {
        if (g.load != kLoadTransposed) continue;
        const size_t need =
            prep_floats(g.op.k, g.op.m) + (g.pack_b ? prep_floats(g.op.k, g.op.n) : 0);
        if (need <= floats - used) {
            used += need;
            continue;
        }
        const bool ok = tma_ok(g.op.k, g.op.A, g.op.lda, g.op.B, g.op.ldb);
        g.load = ok ? kLoadRows : kLoadAsync4;
        g.pack_b = 0;
    }
    sc->scratch_floats = used;
}

// Scratch for a new plan beside those of the device's other plans.
static void take_plan_scratch(sgemm_b200_grouped_plan* plan, Schedule* sc) {
    if (plan->device < 0 || plan->device >= 64) return limit_scratch(sc, 0);
    std::lock_guard<std::mutex> lock(g_plan_scratch_mu);
    size_t& held = g_plan_scratch[plan->device];
    limit_scratch(sc, (kScratchKept - held) / sizeof(float));
    plan->scratch_bytes = sizeof(float) * sc->scratch_floats;
    held += plan->scratch_bytes;
}

// The tensor maps of one problem: an (A, B) pair for each tile shape it uses,
// at maps[2 * shape] and maps[2 * shape + 1] (six slots per problem).  `prep`:
// the problem's prepared matrices (A, then B if it is copied), or null.
static bool encode_problem_maps(const GProblem& g, const GPrep* prep, CUtensorMap* maps) {
    for (int t = 0; t < 3; ++t) {
        if (!(g.shapes & (1 << t))) continue;
        const bool okA =
            prep ? encode_tensor_map_2d(&maps[2 * t], CU_TENSOR_MAP_DATA_TYPE_FLOAT32,
                                        prep[0].job.dst, (uint64_t)g.op.m, (uint64_t)g.op.k,
                                        (uint64_t)prep[0].job.ld_dst * 4, tile_bm(t), 32,
                                        CU_TENSOR_MAP_SWIZZLE_NONE)
                 : encode_tensor_map_2d(&maps[2 * t], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, g.op.A,
                                        (uint64_t)g.op.k, (uint64_t)g.op.m,
                                        (uint64_t)g.op.lda * 4, 32, tile_bm(t),
                                        CU_TENSOR_MAP_SWIZZLE_128B);
        const float* B = g.pack_b ? prep[1].job.dst : g.op.B;
        const int ldb = g.pack_b ? prep[1].job.ld_dst : g.op.ldb;
        if (!okA || !encode_tensor_map_2d(&maps[2 * t + 1], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, B,
                                          (uint64_t)g.op.n, (uint64_t)g.op.k, (uint64_t)ldb * 4,
                                          tile_bn(t), 32, CU_TENSOR_MAP_SWIZZLE_NONE))
            return false;
    }
    return true;
}

static bool encode_maps(const Schedule& sc, const std::vector<GPrep>& preps, CUtensorMap* maps) {
    size_t next = 0;
    for (size_t i = 0; i < sc.probs.size(); ++i) {
        const GProblem& g = sc.probs[i];
        if (g.load == kLoadAsync4) continue;
        const GPrep* prep = g.load == kLoadTransposed ? &preps[next] : nullptr;
        if (prep) next += 1 + g.pack_b;
        if (!encode_problem_maps(g, prep, maps + 6 * i)) return false;
    }
    return true;
}

// The kernels' dynamic shared-memory attribute, once per device (attributes
// belong to the device's context); a thread that sees the flag also sees the
// attributes set.
static void set_kernel_attributes() {
    static std::atomic<bool> done[64];
    static std::mutex mu;
    const int dev = device_info().device;
    if (dev < 0 || dev >= 64 || done[dev].load(std::memory_order_acquire)) return;
    std::lock_guard<std::mutex> lock(mu);
    if (done[dev].load(std::memory_order_relaxed)) return;
    cudaFuncSetAttribute(grouped_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         smem_bytes<3>());
    cudaFuncSetAttribute(grouped_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         smem_bytes<4>());
    done[dev].store(true, std::memory_order_release);
}

// Persistent CTAs per SM of the kernel variant with `stages` stages.
static int resident_per_sm(int stages) {
    int occ = 0;
    const cudaError_t e =
        stages == 3 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, grouped_kernel<3>,
                                                                    THREADS, smem_bytes<3>())
                    : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, grouped_kernel<4>,
                                                                    THREADS, smem_bytes<4>());
    return (e == cudaSuccess && occ > 0) ? occ : 1;
}

static int build_plan(const sgemm_b200_problem* probs, int count, const Table& table,
                      sgemm_b200_grouped_plan** out) {
    if (!out) return SGEMM_B200_ERR_INVALID_ARG;
    Schedule sc;
    int st = make_schedule(probs, count, table, &sc);
    if (st != SGEMM_B200_OK) return st;
    if (!device_is_sm100()) return SGEMM_B200_ERR_UNSUPPORTED;
    auto* plan = new sgemm_b200_grouped_plan();
    plan->device = device_info().device;
    plan->stages = table.stages;
    plan->n_tiles = sc.tiles;
    plan->n_items = (int)sc.items.size();
    plan->ws_floats = (size_t)sc.ws_floats;
    plan->n_counters = 1 + sc.tickets;

    // Scratch from the scratch pool: a plan made for one launch does not pay a
    // cudaMalloc of its operands' size.  On the null stream, whose copies below
    // end before this call does.  Within what the other plans leave of kScratchKept.
    take_plan_scratch(plan, &sc);
    if (sc.scratch_floats) {
        cudaMemPool_t pool = scratch_pool();
        if (!pool || cudaMallocFromPoolAsync(reinterpret_cast<void**>(&plan->d_scratch),
                                             sizeof(float) * sc.scratch_floats, pool,
                                             (cudaStream_t)0) != cudaSuccess) {
            cudaGetLastError();
            plan->d_scratch = nullptr;
            limit_scratch(&sc, 0);
            give_plan_scratch(plan);
        }
    }
    std::vector<GPrep> preps;
    plan->prep_tiles = make_preps(sc, plan->d_scratch, &preps);
    plan->n_preps = (int)preps.size();
    std::vector<CUtensorMap> maps(6 * (size_t)std::max(count, 1));
    std::memset(maps.data(), 0, maps.size() * sizeof(CUtensorMap));
    if (!encode_maps(sc, preps, maps.data())) {
        free_plan(plan);
        return SGEMM_B200_ERR_CUDA;
    }

    // One block, one copy: maps, problems, prepared matrices, items; then the
    // tickets, which each launch resets.
    const size_t n_maps = sizeof(CUtensorMap) * maps.size(), n_probs = sizeof(GProblem) * count,
                 n_prep = sizeof(GPrep) * preps.size(), n_it = sizeof(GItem) * sc.items.size();
    static_assert(sizeof(CUtensorMap) % 8 == 0 && sizeof(GProblem) % 8 == 0 &&
                      sizeof(GPrep) % 8 == 0 && sizeof(GItem) % 8 == 0,
                  "every part of the block is aligned");
    const size_t copied = n_maps + n_probs + n_prep + n_it;
    cudaError_t e = cudaMalloc(&plan->d_block, copied + sizeof(int) * plan->n_counters);
    if (e == cudaSuccess && plan->ws_floats)
        e = cudaMalloc(&plan->d_ws, sizeof(float) * plan->ws_floats);
    if (e == cudaSuccess) {
        std::vector<uint8_t> h(copied);
        auto put = [&](size_t at, const void* src, size_t bytes) {
            if (bytes) std::memcpy(h.data() + at, src, bytes);
            return plan->d_block + at;
        };
        plan->d_maps = reinterpret_cast<CUtensorMap*>(put(0, maps.data(), n_maps));
        plan->d_probs = reinterpret_cast<GProblem*>(put(n_maps, sc.probs.data(), n_probs));
        plan->d_preps = reinterpret_cast<GPrep*>(put(n_maps + n_probs, preps.data(), n_prep));
        plan->d_items =
            reinterpret_cast<GItem*>(put(n_maps + n_probs + n_prep, sc.items.data(), n_it));
        plan->d_counters = reinterpret_cast<int*>(plan->d_block + copied);
        e = cudaMemcpy(plan->d_block, h.data(), copied, cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess) {
        free_plan(plan);
        return cuda_status(e);
    }
    set_kernel_attributes();
    const int sms = device_info().sm_count;
    plan->grid = std::max(1, std::min(sms * resident_per_sm(plan->stages), plan->n_items));
    *out = plan;
    return SGEMM_B200_OK;
}

// The launch: operands prepared and tickets reset, then the items.
static int enqueue_kernels(const GParams& p, int stages, int grid, const GPrep* preps, int n_preps,
                           int prep_tiles, int n_counters, cudaStream_t stream) {
    cudaError_t e = launch_chained(grouped_prepare_kernel, 1 + prep_tiles, kPrepThreads, 0, stream,
                                   preps, n_preps, p.counters, n_counters);
    if (e == cudaSuccess)
        e = stages == 3 ? launch_chained(grouped_kernel<3>, grid, THREADS, smem_bytes<3>(), stream,
                                         p)
                        : launch_chained(grouped_kernel<4>, grid, THREADS, smem_bytes<4>(), stream,
                                         p);
    return cuda_status(e);
}

static int enqueue(sgemm_b200_grouped_plan* plan, cudaStream_t stream) {
    if (plan->n_items == 0) return SGEMM_B200_OK;
    GParams p;
    p.probs = plan->d_probs;
    p.items = plan->d_items;
    p.maps = plan->d_maps;
    p.ws = plan->d_ws;
    p.counters = plan->d_counters;
    p.status = device_status_ptr();
    p.n_items = plan->n_items;
    if (!p.status) return SGEMM_B200_ERR_CUDA;
    return enqueue_kernels(p, plan->stages, plan->grid, plan->d_preps, plan->n_preps,
                           plan->prep_tiles, plan->n_counters, stream);
}

static int launch(sgemm_b200_grouped_plan* plan, cudaStream_t stream, int use_graph) {
    if (!plan) return SGEMM_B200_ERR_INVALID_ARG;
    if (!use_graph) return enqueue(plan, stream);
    if (!plan->exec) {
        cudaError_t e = cudaSuccess;
        if (!plan->cap_stream) {
            e = cudaStreamCreateWithFlags(&plan->cap_stream, cudaStreamNonBlocking);
            if (e != cudaSuccess) {
                plan->cap_stream = nullptr;
                return cuda_status(e);
            }
        }
        e = cudaStreamBeginCapture(plan->cap_stream, cudaStreamCaptureModeThreadLocal);
        if (e != cudaSuccess) return cuda_status(e);
        const int s = enqueue(plan, plan->cap_stream);
        cudaGraph_t graph = nullptr;
        e = cudaStreamEndCapture(plan->cap_stream, &graph);
        if (s != SGEMM_B200_OK || e != cudaSuccess) {
            if (graph) cudaGraphDestroy(graph);
            return s != SGEMM_B200_OK ? s : cuda_status(e);
        }
        e = cudaGraphInstantiate(&plan->exec, graph, 0);
        if (e != cudaSuccess) {
            plan->exec = nullptr;
            cudaGraphDestroy(graph);
            return cuda_status(e);
        }
        plan->graph = graph;
    }
    return cuda_status(cudaGraphLaunch(plan->exec, stream));
}

// ------------------------------------------------------------ arena path --
// Batch launcher for the serving loop: device buffers and pinned staging
// buffers are allocated once and grown on demand, so a batch costs a host
// schedule, a few async copies and one kernel launch (no cudaMalloc, no
// graph capture).  An arena must not be reused before its previous batch
// completed (the staging buffers feed async copies).  First allocations are
// generous (min_cap elements), because growing pinned staging means
// cudaFreeHost, which waits for the whole device, in the middle of serving.

template <class T>
static cudaError_t grow(T** d, T** h, size_t* cap, size_t need, cudaStream_t s,
                        size_t min_cap, cudaMemPool_t pool, size_t max_cap = SIZE_MAX) {
    if (need <= *cap) return cudaSuccess;
    const size_t n = std::min(std::max({need, *cap * 2, min_cap}), max_cap);
    if (*d) cudaFreeAsync(*d, s);
    *d = nullptr;
    *cap = 0;
    if (h && *h) {
        cudaFreeHost(*h);
        *h = nullptr;
    }
    if (!pool) return cudaErrorMemoryAllocation;
    cudaError_t e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(d), n * sizeof(T), pool, s);
    if (e == cudaSuccess && h) e = cudaMallocHost(reinterpret_cast<void**>(h), n * sizeof(T));
    if (e == cudaSuccess) *cap = n;
    return e;
}

int arena_launch(Arena* a, const sgemm_b200_problem* probs, int count, cudaStream_t stream) {
    if (!device_is_sm100()) return SGEMM_B200_ERR_UNSUPPORTED;
    Table table;  // built-in choices: split-K off, so results equal the plain path's
    Schedule sc;
    const int st = make_schedule(probs, count, table, &sc);
    if (st != SGEMM_B200_OK) return st;
    if (sc.items.empty()) return SGEMM_B200_OK;
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t x) {
        if (e == cudaSuccess) e = x;
    };
    const size_t n_counters = 1 + (size_t)sc.tickets;
    cudaMemPool_t pool = library_pool();
    // first capacities: 256 problems, 64 Ki work items (~1 MB pinned in all)
    chk(grow(&a->d_probs, &a->h_probs, &a->cap_probs, (size_t)count, stream, 256, pool));
    chk(grow(&a->d_items, &a->h_items, &a->cap_items, sc.items.size(), stream, 1 << 16,
             pool));
    chk(grow(&a->d_maps, &a->h_maps, &a->cap_maps, 6 * (size_t)count, stream, 1536, pool));
    chk(grow<int>(&a->d_counters, nullptr, &a->cap_counters, n_counters, stream, 1024, pool));
    chk(grow<float>(&a->d_ws, nullptr, &a->cap_ws, std::max<size_t>(sc.ws_floats, 1), stream,
                    1, pool));
    if (e != cudaSuccess) return cuda_status(e);
    const size_t limit = a->scratch_limit / sizeof(float);
    limit_scratch(&sc, limit);
    if (sc.scratch_floats &&
        grow<float>(&a->d_scratch, nullptr, &a->cap_scratch, sc.scratch_floats, stream,
                    (size_t)1 << 22, scratch_pool(), limit) != cudaSuccess) {
        cudaGetLastError();
        limit_scratch(&sc, 0);
    }
    std::vector<GPrep> preps;
    const int prep_tiles = make_preps(sc, a->d_scratch, &preps);
    chk(grow(&a->d_preps, &a->h_preps, &a->cap_preps, std::max<size_t>(preps.size(), 1), stream,
             512, pool));
    if (e != cudaSuccess) return cuda_status(e);
    std::memcpy(a->h_probs, sc.probs.data(), sizeof(GProblem) * count);
    std::memcpy(a->h_items, sc.items.data(), sizeof(GItem) * sc.items.size());
    std::memset(a->h_maps, 0, sizeof(CUtensorMap) * 6 * count);
    if (!encode_maps(sc, preps, a->h_maps)) return SGEMM_B200_ERR_CUDA;
    if (!preps.empty()) {
        std::memcpy(a->h_preps, preps.data(), sizeof(GPrep) * preps.size());
        chk(cudaMemcpyAsync(a->d_preps, a->h_preps, sizeof(GPrep) * preps.size(),
                            cudaMemcpyHostToDevice, stream));
    }
    chk(cudaMemcpyAsync(a->d_probs, a->h_probs, sizeof(GProblem) * count, cudaMemcpyHostToDevice,
                        stream));
    chk(cudaMemcpyAsync(a->d_items, a->h_items, sizeof(GItem) * sc.items.size(),
                        cudaMemcpyHostToDevice, stream));
    chk(cudaMemcpyAsync(a->d_maps, a->h_maps, sizeof(CUtensorMap) * 6 * count,
                        cudaMemcpyHostToDevice, stream));
    if (e != cudaSuccess) return cuda_status(e);
    set_kernel_attributes();
    GParams p;
    p.probs = a->d_probs;
    p.items = a->d_items;
    p.maps = a->d_maps;
    p.ws = a->d_ws;
    p.counters = a->d_counters;
    p.status = device_status_ptr();
    p.n_items = (int)sc.items.size();
    if (!p.status) return SGEMM_B200_ERR_CUDA;
    static const int per_sm = resident_per_sm(3);  // after the attributes; once, thread-safe
    const int grid = std::max(1, std::min(device_info().sm_count * per_sm, p.n_items));
    return enqueue_kernels(p, 3, grid, a->d_preps, (int)preps.size(), prep_tiles, (int)n_counters,
                           stream);
}

void arena_release(Arena* a) {
    pool_free(a->d_probs);
    pool_free(a->d_items);
    pool_free(a->d_maps);
    pool_free(a->d_counters);
    pool_free(a->d_ws);
    pool_free(a->d_scratch);
    pool_free(a->d_preps);
    cudaFreeHost(a->h_preps);
    cudaFreeHost(a->h_probs);
    cudaFreeHost(a->h_items);
    cudaFreeHost(a->h_maps);
    *a = Arena();
}

// Median device time (ms) of `reps` graph launches of a plan.
static double time_plan(sgemm_b200_grouped_plan* plan, cudaStream_t s, int reps) {
    if (launch(plan, s, 1) != SGEMM_B200_OK) return 1e30;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    std::vector<float> t;
    for (int r = 0; r < reps; ++r) {
        cudaEventRecord(a, s);
        launch(plan, s, 1);
        cudaEventRecord(b, s);
        cudaEventSynchronize(b);
        float ms = 0;
        cudaEventElapsedTime(&ms, a, b);
        t.push_back(ms);
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    std::sort(t.begin(), t.end());
    return t[t.size() / 2];
}

}  // namespace grouped
}  // namespace sgb

// ---------------------------------------------------------------- C ABI --

extern "C" int sgemm_b200_grouped_plan_create(sgemm_b200_grouped_plan** plan,
                                              const sgemm_b200_problem* problems, int count,
                                              const char* tuning_json) {
    sgb::grouped::Table t;
    if (tuning_json) sgb::grouped::load_table(tuning_json, &t);  // falls back to defaults
    const int s = sgb::grouped::build_plan(problems, count, t, plan);
    sgb::set_last_status(s);
    return s;
}

extern "C" int sgemm_b200_grouped_plan_launch(sgemm_b200_grouped_plan* plan,
                                              sgemm_b200_stream_t stream, int use_graph) {
    const int s = sgb::grouped::launch(plan, sgb::as_stream(stream), use_graph);
    sgb::set_last_status(s);
    return s;
}

extern "C" int sgemm_b200_grouped_plan_info(const sgemm_b200_grouped_plan* plan, int* tiles,
                                            int* work_items, int* grid_ctas) {
    if (!plan) return SGEMM_B200_ERR_INVALID_ARG;
    if (tiles) *tiles = plan->n_tiles;
    if (work_items) *work_items = plan->n_items;
    if (grid_ctas) *grid_ctas = plan->grid;
    return SGEMM_B200_OK;
}

extern "C" void sgemm_b200_grouped_plan_destroy(sgemm_b200_grouped_plan* plan) {
    sgb::grouped::free_plan(plan);
}

extern "C" int sgemm_b200_grouped(const sgemm_b200_problem* problems, int count,
                                  sgemm_b200_stream_t stream) {
    sgemm_b200_grouped_plan* plan = nullptr;
    int s = sgemm_b200_grouped_plan_create(&plan, problems, count, nullptr);
    if (s != SGEMM_B200_OK) return s;
    s = sgb::grouped::launch(plan, sgb::as_stream(stream), 0);
    // The plan's buffers must outlive the kernel.
    cudaError_t e = cudaStreamSynchronize(sgb::as_stream(stream));
    if (s == SGEMM_B200_OK && e != cudaSuccess) s = sgb::cuda_status(e);
    sgb::grouped::free_plan(plan);
    sgb::set_last_status(s);
    return s;
}

extern "C" int sgemm_b200_grouped_sequential(const sgemm_b200_problem* problems, int count,
                                             sgemm_b200_stream_t stream) {
    if (count < 0 || (count > 0 && !problems)) return SGEMM_B200_ERR_INVALID_ARG;
    for (int i = 0; i < count; ++i) {
        const sgemm_b200_problem& q = problems[i];
        const int s = sgemm_b200(q.m, q.n, q.k, &q.alpha, q.A, q.lda, q.B, q.ldb, &q.beta, q.C,
                                 q.ldc, stream);
        if (s != SGEMM_B200_OK) return s;
    }
    return SGEMM_B200_OK;
}

extern "C" int sgemm_b200_grouped_schedule(const sgemm_b200_problem* problems, int count,
                                           const char* tuning_json, int* tiles, int* work_items,
                                           size_t* workspace_bytes) {
    sgb::grouped::Table t;
    if (tuning_json) sgb::grouped::load_table(tuning_json, &t);
    sgb::grouped::Schedule sc;
    const int s = sgb::grouped::make_schedule(problems, count, t, &sc);
    if (s != SGEMM_B200_OK) return s;
    if (tiles) *tiles = sc.tiles;
    if (work_items) *work_items = (int)sc.items.size();
    if (workspace_bytes) *workspace_bytes = (size_t)sc.ws_floats * sizeof(float);
    return SGEMM_B200_OK;
}

extern "C" int sgemm_b200_grouped_bucket(int m, int n, int k) {
    return sgb::grouped::bucket_of(m, n, k);
}

extern "C" int sgemm_b200_autotune_grouped(const sgemm_b200_problem* problems, int count,
                                           const char* json_path) {
    using namespace sgb::grouped;
    if (!json_path) return SGEMM_B200_ERR_INVALID_ARG;
    if (!sgb::device_is_sm100()) return SGEMM_B200_ERR_UNSUPPORTED;
    cudaStream_t s;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess)
        return SGEMM_B200_ERR_CUDA;
    bool present[kBuckets] = {false};
    for (int i = 0; i < count; ++i)
        present[bucket_of(problems[i].m, problems[i].n, problems[i].k)] = true;
    Table best;
    auto measure = [&](const Table& t) {
        sgemm_b200_grouped_plan* plan = nullptr;
        if (build_plan(problems, count, t, &plan) != SGEMM_B200_OK) return 1e30;
        const double ms = time_plan(plan, s, 5);
        free_plan(plan);
        return ms;
    };
    double best_ms = measure(best);
    // The launch's ring size, then per bucket present in the workload (by
    // coordinate descent): tile shape x split-K, then the bucket's stage count.
    // A candidate must win by 1% to replace the current choice.
    for (int st : {3, 4}) {
        if (st == best.stages) continue;
        Table t = best;
        t.stages = st;
        const double ms = measure(t);
        if (ms < best_ms) {
            best_ms = ms;
            best = t;
        }
    }
    auto consider = [&](const Table& t) {
        const double ms = measure(t);
        if (ms < best_ms * 0.99) {
            best_ms = ms;
            best = t;
        }
    };
    for (int b = 0; b < kBuckets; ++b) {
        if (!present[b]) continue;
        const int kclass = b % kKClasses, mnclass = b / kKClasses;
        for (int tile : {kTileTall, kTileWide, kTileSkinny}) {
            if (tile == kTileSkinny && mnclass == 2) continue;  // large problems: no
            for (int split : {1, 2, 4, 8, 16}) {
                if (split > 1 && kclass == 0) continue;  // short K: nothing to split
                Table t = best;
                t.c[b].tile = tile;
                t.c[b].split = split;
                if (t.c[b].tile == best.c[b].tile && t.c[b].split == best.c[b].split) continue;
                consider(t);
            }
        }
        for (int depth : {2, 3, 4}) {
            if (depth == best.c[b].depth) continue;
            Table t = best;
            t.c[b].depth = depth;
            consider(t);
        }
    }
    cudaStreamDestroy(s);
    return save_table(json_path, best) ? SGEMM_B200_OK : SGEMM_B200_ERR_INVALID_ARG;
}
