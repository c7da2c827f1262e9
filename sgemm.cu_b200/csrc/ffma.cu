// ffma.cu — plain-path kernel configurations, dispatch and the C ABI entry
// points that replace the reference's sgemm() (src/sgemm.cuh:19-48).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "common.h"
#include "ffma_kernel.cuh"
#include "plain.h"
#include "transpose.cuh"

namespace sgb {
namespace ffma {

// Compiled configurations (the public config id is the position in kConfigs).
//   tile  warps m x n  columns  stages  loader  CTAs/SM  rows  transposed A
//
// Large tiles read A transposed (compute_stage_kmajor).  B200, TFLOP/s at
// beta 0, against the same tiles on A [row][k]: 128 x 64 at 4096^3 66.3 from
// 58.8 and at 8192^3 (beta 0.5) 67.3 from 59.6 (90% of the FP32 peak from 80),
// 28 x 256 at 2048^3 59.1 from 57.6, all with the transpose in the time.
using C0 = Cfg<128, 256, 4, 2, 16, 4, kLoaderTma, 1, 8, true>;
using C1 = Cfg<128, 128, 4, 2, 8, 3, kLoaderTma, 1, 8, true>;
using C2 = Cfg<128, 128, 4, 1, 16, 3, kLoaderTma, 1, 8, true>;
using C3 = Cfg<64, 128, 2, 2, 8, 4, kLoaderTma, 2, 8, true>;
using C4 = Cfg<64, 64, 2, 1, 8, 4, kLoaderTma, 3, 8, true>;
using C5 = Cfg<64, 128, 2, 2, 8, 3, kLoaderTma, 3, 8, true>;
using C6 = Cfg<128, 64, 4, 1, 8, 3, kLoaderTma, 3, 8, true>;
using S0 = Cfg<64, 64, 2, 2, 4, 4, kLoaderTma, 3>;
using S1 = Cfg<32, 64, 1, 2, 4, 4, kLoaderTma, 4>;
using C8 = Cfg<128, 256, 4, 2, 16, 4, kLoaderAsync4, 1>;
using C9 = Cfg<128, 128, 4, 2, 8, 3, kLoaderAsync4, 2>;
using C11 = Cfg<64, 128, 2, 2, 8, 4, kLoaderAsync4, 2>;
using C12 = Cfg<64, 64, 2, 1, 8, 4, kLoaderAsync4, 3>;
using C14 = Cfg<128, 64, 4, 1, 8, 3, kLoaderAsync4, 3>;
using W0 = Cfg<128, 64, 4, 2, 4, 3, kLoaderTma, 2, 8, true>;
using W1 = Cfg<128, 64, 4, 2, 4, 4, kLoaderTma, 2, 8, true>;
using P0 = Cfg<128, 64, 4, 1, 8, 3, kLoaderTma, 3>;
using P1 = Cfg<128, 64, 4, 1, 8, 4, kLoaderTma, 2>;
// 28 x 256 tiles, 7 x 8 outputs per thread: a 1024 x 1024 output is 37 x 4 =
// 148 tiles, one per SM, each thread doing 56 FMAs per k step where the
// 128 x 64 tile (128 tiles, 20 SMs idle) does 64; two CTAs fit an SM with 3
// stages (2048^3: 592 tiles, two full waves).  The one-CTA form keeps A
// [row][k]: at 1024^3 the transpose costs more than it gives (47.8 against
// 41.6 us).
// P0, P1 and T4 keep A [row][k] too, for calls without scratch for the
// transpose, whose other tiles are small or alone on their SM: 8192^3 18.2 ms on
// P1, 2048^3 297 us on T4 (16.3 ms and 290 us with A transposed).  T4 is also the
// faster one for wide A: 8192 x 512 x 8192 1173 us against 1221 on T3.
using T0 = Cfg<28, 256, 1, 4, 8, 4, kLoaderTma, 1, 7>;
using T3 = Cfg<28, 256, 1, 4, 8, 3, kLoaderTma, 2, 7, true>;
using T4 = Cfg<28, 256, 1, 4, 8, 3, kLoaderTma, 2, 7>;
// Small threads (4 x 2 and 4 x 4 outputs) for outputs too few to give every
// scheduler an 8-row one: a few rows against a wide B, and squares below
// ~900.  A 24 x 4096 x 4096 GEMM, whose 64 tiles of 32 x 64 left 84 SMs idle at
// 57 cycles per k step (117.5 us), takes 42 us on 128 tiles of 32 x 32 (19
// cycles); 64 rows 59 us from 118, 512^3 8.9 from 16.2.  Deep rings: these
// stream B from HBM, 4-8 KB per stage.  What bounds them is issue (one warp per
// scheduler, every instruction taking two cycles) and, from two CTAs per SM,
// shared-memory loads (a wavefront carries two floats per lane).
using K1 = Cfg<16, 32, 1, 2, 2, 12, kLoaderTma, 2, 4>;
using K2 = Cfg<32, 32, 2, 2, 2, 10, kLoaderTma, 2, 4>;
using K3 = Cfg<32, 64, 2, 2, 4, 8, kLoaderTma, 2, 4>;
using K4 = Cfg<16, 128, 1, 4, 4, 6, kLoaderTma, 2, 4>;
using K6 = Cfg<64, 64, 4, 2, 4, 6, kLoaderTma, 2, 4>;
using K8 = Cfg<32, 128, 2, 4, 4, 5, kLoaderTma, 2, 4>;
using Q3 = Cfg<32, 64, 2, 2, 4, 8, kLoaderTma, 2, 4, true>;
using Q7 = Cfg<64, 64, 2, 2, 4, 6, kLoaderTma, 2, 8, true>;
using A2 = Cfg<32, 32, 2, 2, 2, 4, kLoaderAsync4, 2, 4>;
using A3 = Cfg<32, 64, 2, 2, 4, 4, kLoaderAsync4, 2, 4>;

// What a launch costs, in microseconds on a B200 at 1965 MHz: with c CTAs on the
// busiest SM a k step takes u c + v cycles, and each of the c rounds w for its
// prologue and epilogue.  u / (BM BN / 128) is the reciprocal of the tile's
// share of the FP32 peak when the SM is full; v is what too few warps leave
// idle.
struct Cost {
    float u, v, w;
};

struct ConfigDesc {
    const char* name;
    int bm, bn, threads, smem, loader;
    bool km;    // reads A transposed
    int a_box;  // rows of an A box (slots when transposed)
    int ctas;   // that an SM's shared memory holds
    Cost cost;
    bool spare;  // only for calls without scratch: its twin on transposed A is faster
    void (*kernel)(const CUtensorMap, const CUtensorMap, const Params);
};

template <class C>
constexpr ConfigDesc describe(const char* name, float u, float v, float w, bool spare = false) {
    return ConfigDesc{name, C::BM, C::BN, C::THREADS, C::SMEM_BYTES, C::LOADER, C::KM,
                      C::A_BOX, 227 * 1024 / (C::SMEM_BYTES + 1024), Cost{u, v, w}, spare,
                      &ffma_gemm_kernel<C>};
}

// u, v, w fitted per configuration to B200 timings of grids of 148 c CTAs,
// c = 1..8, at k = 1024 and 3072 (the slope gives u c + v, the rest w).  T4's w is
// T0's, so that it leaves problems of one tile per SM to T0 (1024^3 1% faster).
static const ConfigDesc kConfigs[] = {
    describe<C0>("tma_128x256_w8_t8x16_s4", 321.6f, 1.6f, 3.6f),
    describe<C1>("tma_128x128_w8_t8x8_s3", 142.2f, 1.3f, 2.9f),
    describe<C2>("tma_128x128_w4_t8x16_s3", 147.4f, 0.6f, 3.0f),
    describe<C3>("tma_64x128_w4_t8x8_s4", 70.2f, 5.5f, 0.8f),
    describe<C4>("tma_64x64_w2_t8x8_s4", 52.0f, 30.0f, 0.8f),
    describe<C5>("tma_64x128_w4_t8x8_s3", 69.4f, 7.3f, 0.8f),
    describe<C6>("tma_128x64_w4_t8x8_s3", 69.2f, 7.3f, 0.8f),
    describe<S0>("tma_64x64_w4_t8x4_s4", 40.7f, 7.0f, 0.5f),
    describe<S1>("tma_32x64_w2_t8x4_s4", 24.0f, 36.0f, 0.5f),
    describe<C8>("cpa_128x256_w8_t8x16_s4", 425.5f, 1.0f, 3.3f),
    describe<C9>("cpa_128x128_w8_t8x8_s3", 225.0f, 12.0f, 1.7f),
    describe<C11>("cpa_64x128_w4_t8x8_s4", 131.0f, 18.0f, 1.2f),
    describe<C12>("cpa_64x64_w2_t8x8_s4", 77.0f, 75.0f, 0.8f),
    describe<C14>("cpa_128x64_w4_t8x8_s3", 118.5f, 27.0f, 1.2f),
    describe<W0>("tma_128x64_w8_t8x4_s3", 75.4f, 1.5f, 0.8f),
    describe<W1>("tma_128x64_w8_t8x4_s4", 75.4f, 1.8f, 0.8f),
    describe<P0>("tma_128x64_w4p_t8x8_s3", 81.2f, 10.5f, 0.8f, true),
    describe<P1>("tma_128x64_w4p_t8x8_s4", 78.1f, 5.4f, 0.8f, true),
    describe<T0>("tma_28x256_w4p_t7x8_s4", 74.5f, 1.0f, 2.4f),
    describe<T3>("tma_28x256_w4p_t7x8_s3", 64.6f, 9.5f, 0.9f),
    describe<K1>("tma_16x32_w2_t4x2", 9.4f, 7.0f, 0.3f),
    describe<K2>("tma_32x32_w4_t4x2", 13.5f, 5.0f, 0.4f),
    describe<K3>("tma_32x64_w4_t4x4", 21.7f, 5.4f, 0.5f),
    describe<K4>("tma_16x128_w4_t4x4", 22.0f, 6.6f, 0.6f),
    describe<K6>("tma_64x64_w8_t4x4", 41.8f, 1.7f, 0.7f),
    describe<K8>("tma_32x128_w8_t4x4", 41.9f, 1.7f, 0.7f),
    describe<Q3>("tma_32x64_w4_t4x4_at", 19.5f, 6.0f, 0.6f),
    describe<Q7>("tma_64x64_w4_t8x4_at", 37.8f, 8.6f, 0.6f),
    describe<A2>("cpa_32x32_w4_t4x2_s4", 26.0f, 16.0f, 0.5f),
    describe<A3>("cpa_32x64_w4_t4x4_s4", 41.5f, 22.0f, 0.5f),
    describe<T4>("tma_28x256_w4p_t7x8_s3_rows", 68.4f, 7.9f, 2.4f),
};
constexpr int kNumConfigs = sizeof(kConfigs) / sizeof(kConfigs[0]);

// The kernel's shared-memory attribute, once per device.
static cudaError_t set_smem_attribute(int cfg) {
    static bool have[64][kNumConfigs];
    static std::mutex mu;
    const DeviceInfo& d = device_info();
    if (d.device < 0 || d.device >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    if (!have[d.device][cfg]) {
        const cudaError_t e =
            cudaFuncSetAttribute(kConfigs[cfg].kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kConfigs[cfg].smem);
        if (e != cudaSuccess) return e;
        have[d.device][cfg] = true;
    }
    return cudaSuccess;
}

// Unaligned operands are copied to aligned rows (one more launch) for the TMA
// kernels from 512^3 multiply-adds on, and below that, from 317^3 on, where the cost
// model finds it faster than the 4-byte cp.async loader on the operands in place: on a
// B200 317^3 takes 10.0 us in place and 321^3 9.4 us copied, 401^3 37.6 and 10.1.  A
// block copies a row per 0.6 us, however short: 36912 x 48 x 36 takes 14.5 us in place
// and 35.9 copied.
constexpr double kPackMinWork = 32.0e6, kPackWork = 134217728.0;  // 317^3, 512^3

static bool tma_ok(const float* A, int lda, const float* B, int ldb) {
    return (lda % 4 == 0) && (ldb % 4 == 0) && (reinterpret_cast<uintptr_t>(A) % 16 == 0) &&
           (reinterpret_cast<uintptr_t>(B) % 16 == 0);
}

}  // namespace ffma

int plain_config_count() { return ffma::kNumConfigs; }
const char* plain_config_name(int cfg) {
    return (cfg >= 0 && cfg < ffma::kNumConfigs) ? ffma::kConfigs[cfg].name : nullptr;
}
int plain_config_tile(int cfg, int* bm, int* bn) {
    if (cfg < 0 || cfg >= ffma::kNumConfigs) return SGEMM_B200_ERR_INVALID_ARG;
    *bm = ffma::kConfigs[cfg].bm;
    *bn = ffma::kConfigs[cfg].bn;
    return SGEMM_B200_OK;
}

// Modelled time of a problem on a configuration, in microseconds.  Tiles go to
// whichever SM is free, so the busiest SM runs ceil(tiles / SMs) of them, and
// once there are many the ends no longer line up.  With few k steps the other CTAs of
// an SM do not hide a CTA's fill (2 us) and epilogue (1 us per 8192 outputs, twice when
// C is read), and each generation of resident CTAs pays what is left of them.
// Against the fastest configuration the pick took 1.8% longer over 286 problems
// of 4 to 2000 k steps, of which 7 were slower than on the tiles of before (2.9% and
// 15 without that: 596 x 19928 x 4 30.5 us from 27.0), and 1.1% over 278 of 64 to 500.
// A configuration that reads A transposed also pays for the transpose (its launch,
// and its bytes at the rate it runs at).
static double modelled_us(const ffma::ConfigDesc& cd, int m, int n, int k, int sms, bool reads_c) {
    const double per_sm = double(div_up(m, cd.bm)) * div_up(n, cd.bn) / sms;
    const double c = per_sm > 8 ? per_sm + 0.5 : std::ceil(per_sm);
    const double step = double(k) * cd.cost.u / 1965.0;  // a CTA's k steps beside others
    double ends = c * cd.cost.w * (reads_c ? 1.6 : 1.0);
    if (cd.ctas > 1 && c > 1) {
        const double latency = 2.0 + 1.0 * (reads_c ? 2.0 : 1.0) * cd.bm * cd.bn / 8192.0;
        const double others = std::min<double>(c, cd.ctas) - 1;
        ends = std::max(ends, std::max(1.0, c / cd.ctas) * (latency - others * step));
    }
    const double t = ends + step * c + double(k) * cd.cost.v / 1965.0;
    return cd.km ? t + 3.0 + 8.0 * double(m) * k / 4.5e6 : t;
}

// The configuration with the smallest modelled time (the first of equals).
// `scratch`: configurations that read A transposed may be taken.
static int select_for_loader(int m, int n, int k, int loader, bool reads_c, bool scratch = true,
                             double* us = nullptr) {
    using namespace ffma;
    const DeviceInfo& d = device_info();
    const int sms = d.sm_count > 0 ? d.sm_count : 148;
    int best = -1;
    double best_t = 1e300;
    for (int c = 0; c < kNumConfigs; ++c) {
        const ConfigDesc& cd = kConfigs[c];
        if (cd.loader != loader || (scratch ? cd.spare : cd.km)) continue;
        const double t = modelled_us(cd, m, n, k, sms, reads_c);
        if (best < 0 || t < best_t) {
            best_t = t;
            best = c;
        }
    }
    if (us) *us = best_t;
    return best;
}

// The same among the configurations that need no scratch: the operands in place.
static int select_in_place(int m, int n, int k, const float* A, int lda, const float* B, int ldb,
                           bool reads_c) {
    using namespace ffma;
    const int loader = (k == 0 || tma_ok(A, lda, B, ldb)) ? kLoaderTma : kLoaderAsync4;
    return select_for_loader(m, n, k, loader, reads_c, false);
}

int plain_select(int m, int n, int k, const float* A, int lda, const float* B, int ldb,
                 bool reads_c) {
    using namespace ffma;
    const int loader = (k == 0 || tma_ok(A, lda, B, ldb)) ? kLoaderTma : kLoaderAsync4;
    return select_for_loader(m, n, k, loader, reads_c);
}

// Slots of a row of A transposed for configuration cfg, and the copy's bytes.
static int km_pitch(int cfg, int m) {
    return ffma::kConfigs[cfg].bm == 28 ? div_up(m, 28) * 32 : (m + 3) / 4 * 4;
}
static size_t km_bytes(int cfg, int m, int k) {
    return sizeof(float) * (size_t)k * km_pitch(cfg, m);
}

// A transposed A larger than kScratchPerCall is made only in the place of a copy.
static bool too_large(int cfg, int mask, int m, int k) {
    return ffma::kConfigs[cfg].km && k > 0 && !(mask & 1) && km_bytes(cfg, m, k) > kScratchPerCall;
}

// The configuration that runs, given the operands copied first (pack_mask).
static int choose(int mask, int m, int n, int k, const float* A, int lda, const float* B, int ldb,
                  bool reads_c) {
    const int cfg = mask ? select_for_loader(m, n, k, ffma::kLoaderTma, reads_c)
                         : plain_select(m, n, k, A, lda, B, ldb, reads_c);
    return too_large(cfg, mask, m, k)
               ? select_for_loader(m, n, k, ffma::kLoaderTma, reads_c, false)
               : cfg;
}

// Whether a call may take scratch.  In a stream capture scratch becomes memory nodes,
// and a graph that has some cannot be a child graph, nor be instantiated twice: a
// captured call reads its operands in place, with the same result.  Only unaligned
// operands from 512^3 multiply-adds on are copied there, too, as they always were.
static bool scratch_allowed(int mask, int m, int n, int k, cudaStream_t stream) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    const cudaError_t e = cudaStreamIsCapturing(stream, &st);
    if (e != cudaSuccess) cudaGetLastError();
    if (e == cudaSuccess && st == cudaStreamCaptureStatusNone) return true;
    return mask && double(m) * n * k >= ffma::kPackWork;
}

namespace ffma {

// Operand preparation, one launch for both operands: A transposed for the
// configurations that read it [k][slot], and row copies into a 16-byte-aligned
// pitch for strides TMA cannot describe.
struct PackJob {
    const float* src;
    float* dst;
    int rows, cols, ld_src, ld_dst;
};

constexpr int kPackThreads = 256;
constexpr int kPackUnroll = 8;
// Blocks of the transpose, then blocks that copy rows: block r of those copies
// rows r, r + their count, ... of a's rows followed by b's (a job with no rows
// is skipped); within a row the threads take consecutive columns (coalesced),
// eight loads in flight per thread before their stores.  The padding columns
// are not written (the TMA kernel reads only the first `cols` of each row).
// HBM-bound.
__global__ void __launch_bounds__(kPackThreads)
    prepare_kernel(const TransposeJob t, const PackJob a, const PackJob b) {
    __shared__ float tile[kTrTile][kTrTile + 1];
    grid_wait();
    if ((int)blockIdx.x < t.blocks) {
        const int tiles = (t.k + kTrTile - 1) / kTrTile * ((t.m + kTrTile - 1) / kTrTile);
        for (int b = blockIdx.x; b < tiles; b += t.blocks) {
            transpose_tile(t, b, tile);
            __syncthreads();  // the next tile overwrites `tile`
        }
        return;
    }
    const int total = a.rows + b.rows;
    for (int r = blockIdx.x - t.blocks; r < total; r += gridDim.x - t.blocks) {
        const bool in_a = r < a.rows;
        const int row = in_a ? r : r - a.rows;
        const int cols = in_a ? a.cols : b.cols;
        const float* __restrict__ src =
            (in_a ? a.src : b.src) + (int64_t)row * (in_a ? a.ld_src : b.ld_src);
        float* __restrict__ dst =
            (in_a ? a.dst : b.dst) + (int64_t)row * (in_a ? a.ld_dst : b.ld_dst);
        for (int c0 = 0; c0 < cols; c0 += kPackUnroll * kPackThreads) {
            float v[kPackUnroll];
#pragma unroll
            for (int u = 0; u < kPackUnroll; ++u) {
                const int c = c0 + u * kPackThreads + (int)threadIdx.x;
                v[u] = c < cols ? src[c] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < kPackUnroll; ++u) {
                const int c = c0 + u * kPackThreads + (int)threadIdx.x;
                if (c < cols) dst[c] = v[u];
            }
        }
    }
}

static double pack_us(double rows, double elements) {
    return 3.0 + 0.6 * std::ceil(rows / (8 * 148)) + 8.0 * elements / 4.5e6;
}

// Operands the plain path copies to aligned rows before its TMA kernel:
// bit 0 A, bit 1 B; 0 when the kernel reads them in place.
static int pack_mask(int m, int n, int k, const float* A, int lda, const float* B, int ldb) {
    const double work = double(m) * n * k;
    if (k <= 0 || tma_ok(A, lda, B, ldb) || work < kPackMinWork) return 0;
    const bool pa = (lda % 4 != 0) || (reinterpret_cast<uintptr_t>(A) % 16 != 0);
    const bool pb = (ldb % 4 != 0) || (reinterpret_cast<uintptr_t>(B) % 16 != 0);
    if (work < kPackWork) {
        // One block of 4 to 31 k steps: the 4-byte loader is as fast as the copies or
        // faster on all of 22 shapes (64 x 65536 x 17 14.6 us, copied 17.8).
        if (k >= 4 && k < 32) return 0;
        double copied = 0, in_place = 0;
        select_for_loader(m, n, k, kLoaderTma, false, true, &copied);
        select_for_loader(m, n, k, kLoaderAsync4, false, true, &in_place);
        copied += pack_us((pa ? double(m) : 0.0) + (pb ? k : 0),
                          (pa ? double(m) * k : 0.0) + (pb ? double(k) * n : 0.0));
        // with few k steps the 4-byte loader takes about 1.25 times what the model says
        if (copied >= 1.25 * in_place) return 0;
    }
    return (pa ? 1 : 0) | (pb ? 2 : 0);
}

// One launch for the jobs given (at least one): about eight blocks per SM,
// shared between transpose and copies in proportion to their size.
static cudaError_t prepare(TransposeJob t, const PackJob& a, const PackJob& b, cudaStream_t s) {
    const int sms = device_info().sm_count > 0 ? device_info().sm_count : 148;
    const int tiles = t.dst ? div_up(t.m, kTrTile) * div_up(t.k, kTrTile) : 0;
    const double wt = t.dst ? double(t.m) * t.k : 0.0;
    const double wp = double(a.rows) * a.cols + double(b.rows) * b.cols;
    const int want = sms * 8, rows = a.rows + b.rows;
    t.blocks = std::min(tiles, std::max(1, int(want * (wt / (wt + wp)))));
    const int copies = std::min(rows, std::max(1, want - t.blocks));
    return launch_chained(prepare_kernel, t.blocks + copies, kPackThreads, 0, s, t, a, b);
}

}  // namespace ffma

// One launch of configuration cfg on operands it can read in place: A is the
// transposed copy (pitch lda) for a configuration that reads it so.
static int launch_config(int cfg, int m, int n, int k, float alpha, const float* A, int lda,
                         const float* B, int ldb, float beta, float* C, int ldc,
                         const float* acc_in, float* acc_out, int ld_acc, cudaStream_t stream) {
    using namespace ffma;
    const ConfigDesc& cd = kConfigs[cfg];
    Params p;
    p.op.m = m;
    p.op.n = n;
    p.op.k = k;
    p.op.lda = lda;
    p.op.ldb = ldb;
    p.op.ldc = ldc;
    p.op.alpha = alpha;
    p.op.beta = beta;
    p.op.A = A;
    p.op.B = B;
    p.op.C = C;
    p.op.vec_c = (ldc % 4 == 0) && (reinterpret_cast<uintptr_t>(C) % 16 == 0);
    p.status = device_status_ptr();
    if (!p.status) return SGEMM_B200_ERR_CUDA;
    p.tiles_m = div_up(m, cd.bm);
    p.tiles_n = div_up(n, cd.bn);
    p.acc_in = acc_in;
    p.acc_out = acc_out;
    p.ld_acc = ld_acc;

    CUtensorMap tmA, tmB;
    std::memset(&tmA, 0, sizeof(tmA));
    std::memset(&tmB, 0, sizeof(tmB));
    if (cd.loader == kLoaderTma && k > 0) {
        const bool okA =
            cd.km ? encode_tensor_map_2d(&tmA, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, A,
                                         (uint64_t)(cd.bm == 28 ? lda : m), (uint64_t)k,
                                         (uint64_t)lda * 4, cd.a_box, 32,
                                         CU_TENSOR_MAP_SWIZZLE_NONE)
                  : encode_tensor_map_2d(&tmA, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, A, (uint64_t)k,
                                         (uint64_t)m, (uint64_t)lda * 4, 32, cd.a_box,
                                         CU_TENSOR_MAP_SWIZZLE_128B);
        if (!okA ||
            !encode_tensor_map_2d(&tmB, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, B, (uint64_t)n,
                                  (uint64_t)k, (uint64_t)ldb * 4, cd.bn, 32,
                                  CU_TENSOR_MAP_SWIZZLE_NONE))
            return SGEMM_B200_ERR_CUDA;
    }
    const cudaError_t e = set_smem_attribute(cfg);
    if (e != cudaSuccess) return cuda_status(e);
    const int grid = p.tiles_m * p.tiles_n;
    return cuda_status(launch_chained(cd.kernel, grid, cd.threads, cd.smem, stream, tmA, tmB,
                                      p));
}


int plain_pack_rows(int a_rows, int a_cols, const float* A, int lda, float* A2, int lda2,
                    int b_rows, int b_cols, const float* B, int ldb, float* B2, int ldb2,
                    cudaStream_t stream) {
    return cuda_status(ffma::prepare(ffma::TransposeJob{},
                                     ffma::PackJob{A, A2, a_rows, a_cols, lda, lda2},
                                     ffma::PackJob{B, B2, b_rows, b_cols, ldb, ldb2}, stream));
}

int plain_launch(int cfg, int m, int n, int k, float alpha, const float* A, int lda,
                 const float* B, int ldb, float beta, float* C, int ldc, cudaStream_t stream) {
    return plain_launch_acc(cfg, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, nullptr, nullptr,
                            0, stream);
}

int plain_launch_acc(int cfg, int m, int n, int k, float alpha, const float* A, int lda,
                     const float* B, int ldb, float beta, float* C, int ldc, const float* acc_in,
                     float* acc_out, int ld_acc, cudaStream_t stream) {
    using namespace ffma;
    if (m == 0 || n == 0) return SGEMM_B200_OK;
    if (!device_is_sm100()) return SGEMM_B200_ERR_UNSUPPORTED;
    if ((acc_in || acc_out) &&
        (ld_acc < n || ld_acc % 4 != 0 || reinterpret_cast<uintptr_t>(acc_in) % 16 != 0 ||
         reinterpret_cast<uintptr_t>(acc_out) % 16 != 0))
        return SGEMM_B200_ERR_INVALID_ARG;
    // carried accumulators: the caller keeps its operands TMA-aligned (no pack step)
    int mask = (cfg < 0 && !acc_in && !acc_out) ? pack_mask(m, n, k, A, lda, B, ldb) : 0;
    if (cfg < 0) cfg = choose(mask, m, n, k, A, lda, B, ldb, beta != 0.0f);
    if (cfg >= kNumConfigs) return SGEMM_B200_ERR_INVALID_ARG;
    if (!mask && kConfigs[cfg].loader == kLoaderTma && k > 0 && !tma_ok(A, lda, B, ldb))
        return SGEMM_B200_ERR_INVALID_ARG;
    if (((kConfigs[cfg].km && k > 0) || mask) && !scratch_allowed(mask, m, n, k, stream)) {
        mask = 0;
        cfg = select_in_place(m, n, k, A, lda, B, ldb, beta != 0.0f);
    }
    if (too_large(cfg, mask, m, k))
        cfg = select_for_loader(m, n, k, kLoaderTma, beta != 0.0f, false);

    // Scratch, stream-ordered: A transposed for a
    // configuration that reads it so, or operands with strides TMA cannot
    // describe copied to aligned rows.  Same arithmetic, same bits.
    float *A2 = nullptr, *B2 = nullptr;
    const bool km = kConfigs[cfg].km && k > 0;
    if (km || mask) {
        const bool sevens = kConfigs[cfg].bm == 28;
        const bool pa = !km && (mask & 1) != 0, pb = (mask & 2) != 0;
        const int lda2 = km ? km_pitch(cfg, m) : (k + 3) / 4 * 4;
        const int ldb2 = pb ? (n + 3) / 4 * 4 : ldb;
        const size_t a_bytes = km ? km_bytes(cfg, m, k)
                                  : pa ? sizeof(float) * (size_t)m * lda2 : 0;
        const size_t b_bytes = pb ? sizeof(float) * (size_t)k * ldb2 : 0;
        // copies too large to keep in the scratch pool are kept by the library's
        cudaMemPool_t pool = a_bytes + b_bytes <= kScratchPerCall ? scratch_pool() : library_pool();
        cudaError_t e = pool ? cudaSuccess : cudaErrorMemoryAllocation;
        if (e == cudaSuccess && a_bytes) e = cudaMallocFromPoolAsync(&A2, a_bytes, pool, stream);
        if (e == cudaSuccess && b_bytes) e = cudaMallocFromPoolAsync(&B2, b_bytes, pool, stream);
        if (e != cudaSuccess) {
            // no scratch: the best configuration that reads the operands in place
            if (A2) cudaFreeAsync(A2, stream);
            if (B2) cudaFreeAsync(B2, stream);
            cudaGetLastError();
            return plain_launch_acc(select_in_place(m, n, k, A, lda, B, ldb, beta != 0.0f), m, n, k,
                                    alpha, A, lda, B, ldb, beta, C, ldc, acc_in, acc_out, ld_acc,
                                    stream);
        }
        TransposeJob jt = {};
        PackJob ja = {}, jb = {};
        if (km)
            jt = TransposeJob{A, A2, m, k, lda, lda2, sevens,
                              lda % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0, 0};
        if (pa) ja = PackJob{A, A2, m, k, lda, lda2};
        if (pb) jb = PackJob{B, B2, k, n, ldb, ldb2};
        e = prepare(jt, ja, jb, stream);
        if (e != cudaSuccess) {
            if (A2) cudaFreeAsync(A2, stream);
            if (B2) cudaFreeAsync(B2, stream);
            return cuda_status(e);
        }
        if (A2) {
            A = A2;
            lda = lda2;
        }
        if (B2) {
            B = B2;
            ldb = ldb2;
        }
    }
    const int st = launch_config(cfg, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, acc_in, acc_out,
                                 ld_acc, stream);
    if (A2) cudaFreeAsync(A2, stream);
    if (B2) cudaFreeAsync(B2, stream);
    return st;
}

}  // namespace sgb

// ---------------------------------------------------------------- C ABI --

extern "C" int sgemm_b200_with_config(int cfg, int m, int n, int k, const float* alpha,
                                      const float* A, int lda, const float* B, int ldb,
                                      const float* beta, float* C, int ldc,
                                      sgemm_b200_stream_t stream) {
    int s = sgb::check_gemm_args(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    if (s == SGEMM_B200_OK)
        s = sgb::plain_launch(cfg, m, n, k, *alpha, A, lda, B, ldb, *beta, C, ldc,
                              sgb::as_stream(stream));
    sgb::set_last_status(s);
    return s;
}

extern "C" int sgemm_b200(int m, int n, int k, const float* alpha, const float* A, int lda,
                          const float* B, int ldb, const float* beta, float* C, int ldc,
                          sgemm_b200_stream_t stream) {
    return sgemm_b200_with_config(-1, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, stream);
}

extern "C" void sgemm(int m, int n, int k, const float* alpha, float* A, int lda, float* B,
                      int ldb, const float* beta, float* C, int ldc) {
    sgemm_b200(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, nullptr);
}

extern "C" int sgemm_b200_config_count(void) { return sgb::plain_config_count(); }

extern "C" const char* sgemm_b200_config_name(int cfg) { return sgb::plain_config_name(cfg); }

extern "C" int sgemm_b200_select_config_beta(int m, int n, int k, const float* A, int lda,
                                             const float* B, int ldb, const float* beta) {
    if (m <= 0 || n <= 0 || k < 0) return -1;
    const bool reads_c = beta == nullptr || *beta != 0.0f;
    const int mask = sgb::ffma::pack_mask(m, n, k, A, lda, B, ldb);
    return sgb::choose(mask, m, n, k, A, lda, B, ldb, reads_c);
}

extern "C" int sgemm_b200_launches(int m, int n, int k, const float* A, int lda, const float* B,
                                   int ldb, const float* beta) {
    if (m <= 0 || n <= 0 || k < 0) return 0;
    const int cfg = sgemm_b200_select_config_beta(m, n, k, A, lda, B, ldb, beta);
    const bool prepares = sgb::ffma::pack_mask(m, n, k, A, lda, B, ldb) != 0 ||
                          (sgb::ffma::kConfigs[cfg].km && k > 0);
    return prepares ? 2 : 1;
}

extern "C" int sgemm_b200_select_config(int m, int n, int k, const float* A, int lda,
                                        const float* B, int ldb, const float* C, int ldc) {
    (void)C;
    (void)ldc;
    return sgemm_b200_select_config_beta(m, n, k, A, lda, B, ldb, nullptr);
}

extern "C" int sgemm_b200_packs(int m, int n, int k, const float* A, int lda, const float* B,
                                int ldb) {
    if (m <= 0 || n <= 0 || k < 0) return 0;
    return sgb::ffma::pack_mask(m, n, k, A, lda, B, ldb);
}
