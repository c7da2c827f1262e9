// split_fused.cuh — the split-precision GEMM without a pre-pass: the operands are
// read as FP32 and split inside the kernel.  Included by split.cu.
//
// For outputs of few 128 x 256 tiles the pre-pass and the idle SMs are most of
// a call's time.  Here one CTA computes a 128 (n) x NT (m, at most 128) tile of
// C^T over a slab of k:  D[n][m] = B^T A^T, so a few rows of C are a narrow MMA
// instead of a padded one, and a slab of k per CTA (its partial sums met over
// the cluster's shared memory) fills the GPU.  Each FP32 element crosses memory
// once; the terms, their order, the 256-deep D1 chunks and the FP32 sums are
// split_gemm_kernel's, so the result has its bits.
//
//   warps 0..15 split: two groups of eight take the k blocks in turn, each with
//               its own operand buffer, since a block's chain of shared loads,
//               conversions and stores is longer than its MMAs.  Warp w owns TMEM
//               lanes 32 (w % 4).. (columns n of B) and half of a block's k: B's
//               planes go to tensor memory, the MMA's first operand; the group
//               splits A into shared memory (K-major, swizzled), its second
//               operand.  Every warp also drains its quarter of D1's columns once
//               a chunk's MMAs are known to be done.
//   warp 16     TMA producer (one lane): FP32 boxes of A [NT m][32 k] and
//               B [32 k][128 n]
//   warp 17     MMA issuer: the whole warp runs the loop, so that descriptors are
//               uniform values, and one lane issues (one lane alone took 90 cycles
//               per MMA, against 16-64 of work)
// TMEM (512 columns): D1 twice and D2 (NT each), then two buffers of B's planes
// (48 columns each, or 64 for TF32).
// What bounds it (B200, SM cycles): a block of 32 k takes ~660 cycles at NT = 32
// and ~1230 at NT = 128, whose MMAs take 200-770; the rest is the split itself
// (ALU issue and the chain load, convert, store) and, at NT = 128, shared memory
// (each element is landed and read, A's planes written and read by every MMA).
// Measured per call, back to back on three inputs in rotation, BF16X6, against pre-pass
// and 128 x 256 tiles: 24 x 4096 x 4096 18.6 us from 161, 136 x 4096 x 4096 42.0 from 164,
// 1000^3 18.2 from 74, 512^3 11.3 from 33, 64 x 64 x 4096 13.4 from 128; at 2048^3 the
// two meet (96 us here, 91 there).
#pragma once

namespace fused {

constexpr int TN = 128;       // columns of C per tile (rows of the MMA)
constexpr int NT_MAX = 128;   // rows of C per tile (columns of the MMA)
constexpr int BK = 32;        // k block
constexpr int CHUNK_BLOCKS = KCHUNK / BK;
constexpr int SPLIT_WARPS = 16, PRODUCER = SPLIT_WARPS, MMA = SPLIT_WARPS + 1;
constexpr int THREADS = 32 * (SPLIT_WARPS + 2);
constexpr int G = 2;          // groups of split warps, each with an operand buffer
constexpr int GROUP_WARPS = SPLIT_WARPS / G;
constexpr int RAWS_MAX = 10;  // landing stages
constexpr int CQ = NT_MAX / 4;  // columns of D a split warp drains, at most

template <int PATH>
struct Lay {
    using T = Traits<PATH>;
    static constexpr int RAW_B = BK * TN * 4;              // 16 KB
    static constexpr int ROW = BK * T::ESZ;                // bytes of a K-major plane row
    static constexpr int BCOLS = BK * T::ESZ / 4;          // TMEM columns of a B plane
    static constexpr int OPCOLS = T::NSPLIT * BCOLS;
    static constexpr int SMEM = 227 * 1024 - 512;          // all of it but the barriers
    static constexpr int op_bytes(int nt) { return T::NSPLIT * nt * ROW; }
    static constexpr int raw_bytes(int nt) { return RAW_B + nt * BK * 4; }
    // Landing stages that fit: a multiple of G, so that a group meets every phase
    // of the stages it waits on (a parity wait may not skip one).
    static constexpr int raws(int nt) {
        const int fit = (SMEM - 1024 - G * op_bytes(nt)) / raw_bytes(nt) / G * G;
        return fit < RAWS_MAX ? fit : RAWS_MAX;
    }
    static constexpr int STEPS = BK / T::KMMA;
    static_assert(3 * NT_MAX + 2 * OPCOLS <= 512, "tensor memory");
    static_assert(raws(NT_MAX) >= 4 && raws(16) >= 4, "landing stages");
    static_assert(TN * NT_MAX * 4 <= raws(NT_MAX) * raw_bytes(NT_MAX),
                  "the partial tile fits the landing ring");
};

struct Params {
    int m, n, k, ldc;
    float alpha, beta;
    float* C;
    int* status;
    int tiles_m, nt;     // row tiles, rows per tile (a multiple of 16)
    int splits, blocks;  // k slabs (= cluster size), k blocks per slab
};

// One problem of a grouped launch, and one of its tiles.
struct GProblem {
    int m, n, k, ldc;
    float alpha, beta;
    float* C;
    int nt, splits, blocks, pad;
};
struct GTile {
    int prob, m0, n0, pad;
};
struct GParams {
    const GProblem* probs;
    const GTile* tiles;
    const CUtensorMap* maps;  // 2 per problem: A, B
    float* sums;              // TN x NT_MAX per CTA, for problems of several slabs
    int* status;
    int n_tiles;
};

// A walk over a ring of stages: the stage and the parity of its current round.
struct Ring {
    int stage = 0, size;
    uint32_t phase = 0;
    __device__ explicit Ring(int n) : size(n) {}
    __device__ __forceinline__ void next() {
        if (++stage == size) {
            stage = 0;
            phase ^= 1;
        }
    }
};

// Split two neighbouring values (k, k + 1): BF16 planes packed as the MMA reads
// them, k in the low half.
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&p)[3]) {
    p[0] = pack_bf16(x, y);
    const float x1 = __fsub_rn(x, __uint_as_float(p[0] << 16));
    const float y1 = __fsub_rn(y, __uint_as_float(p[0] & 0xffff0000u));
    p[1] = pack_bf16(x1, y1);
    p[2] = pack_bf16(__fsub_rn(x1, __uint_as_float(p[1] << 16)),
                     __fsub_rn(y1, __uint_as_float(p[1] & 0xffff0000u)));
}

struct Barriers {
    uint64_t raw_full[RAWS_MAX], raw_empty[RAWS_MAX];
    uint64_t op_full[G], op_empty[G];
    uint64_t d1_full[2], d1_empty[2], d2_empty;
    volatile int gone;  // a wait has expired
};

// A split warp's wait.  A lane whose wait expires (false) stays with its warp, which
// goes on (in bounds, on what it finds) to the chunk's vote on `gone` (convert); waits
// that come before that no longer last.  A vote per wait instead costs 1-2% of a call.
__device__ __forceinline__ bool wait_or_gone(Barriers& b, uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    while (!mbar_try_wait(bar, parity)) {
        if (b.gone || globaltimer_ns() - t0 > kWaitLimitNs) {
            b.gone = 1;
            return false;
        }
    }
    return true;
}

// Where a CTA keeps things: operand buffers, landing stages (A [nt][32 k], then
// B [32 k][128 n]) and tensor-memory columns (D1 at 0 and dcols, D2 at 2 dcols,
// B's planes from 3 dcols).
struct Place {
    uint8_t* ops;
    uint8_t* raw;
    int op_stride, raw_stride, raws;
    uint32_t tmem;
    uint32_t dcols;
};

template <int PATH>
__device__ __forceinline__ Place make_place(uint8_t* smem, int nt, uint32_t tmem) {
    using L = Lay<PATH>;
    Place pl;
    pl.ops = smem;
    pl.op_stride = L::op_bytes(nt);
    pl.raw = smem + G * pl.op_stride;
    pl.raw_stride = L::raw_bytes(nt);
    pl.raws = L::raws(nt);
    pl.tmem = tmem;
    pl.dcols = nt;
    return pl;
}

__device__ __forceinline__ void init_barriers(Barriers& b) {
    for (int s = 0; s < RAWS_MAX; ++s) {
        mbar_init(&b.raw_full[s], 1);
        mbar_init(&b.raw_empty[s], GROUP_WARPS);
    }
    for (int s = 0; s < G; ++s) {
        mbar_init(&b.op_full[s], GROUP_WARPS);
        mbar_init(&b.op_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
        mbar_init(&b.d1_full[s], 1);
        mbar_init(&b.d1_empty[s], SPLIT_WARPS);
    }
    mbar_init(&b.d2_empty, SPLIT_WARPS);
    b.gone = 0;
}

// The roles, each over the nb k blocks of one slab of one tile.  Counters that
// give the barriers' phases run on from slab to slab.  They return false when a
// bounded wait expired, a whole warp's role in all its lanes, by a vote: a lane that
// left alone would leave its warp short in the collective instructions (votes,
// tensor-memory loads and stores) ahead.

// TMA producer (one lane).
template <int PATH>
__device__ __forceinline__ bool produce(const Place& pl, Barriers& b, const CUtensorMap* tmA,
                                        const CUtensorMap* tmB, int nt, int m0, int n0, int kb0,
                                        int nb, Ring& ring, int& issued) {
    const uint32_t bytes = Lay<PATH>::raw_bytes(nt);
    for (int i = 0; i < nb; ++i, ring.next(), ++issued) {
        if (issued >= pl.raws) {
            // A warp arrives also when its wait for the stage expired (wait_or_gone): the
            // copy may be in flight, and raw_full must not be armed twice in a phase.
            if (!mbar_wait(&b.raw_empty[ring.stage], ring.phase ^ 1) || b.gone) return false;
            fence_proxy_async_shared();  // the warps' reads before the TMA refill
        }
        uint8_t* st = pl.raw + ring.stage * pl.raw_stride;
        uint64_t* bar = &b.raw_full[ring.stage];
        mbar_arrive_expect_tx(bar, bytes);
        tma_load_2d(st, tmA, bar, (kb0 + i) * BK, m0);
        tma_load_2d(st + nt * BK * 4, tmB, bar, n0, (kb0 + i) * BK);
    }
    return true;
}

// Copies still in flight land before the CTA ends (the split warps may have
// given up on one).
__device__ __forceinline__ void settle(const Place& pl, Barriers& b, int issued) {
    for (int j = max(0, issued - pl.raws); j < issued; ++j)
        if (!mbar_wait(&b.raw_full[j % pl.raws], (j / pl.raws) & 1)) break;
}

// MMA warp: g blocks and cg D1 chunks issued so far, in `slab` slabs.
template <int PATH>
__device__ __forceinline__ bool multiply(const Place& pl, Barriers& b, int nt, int nb, bool leader,
                                         uint32_t& g, uint32_t& cg, uint32_t slab) {
    using T = Traits<PATH>;
    using L = Lay<PATH>;
    const uint32_t idesc = make_idesc(T::FMT, TN, nt);
    const uint64_t desc0 = L::ROW == 64 ? sw64_kmajor_desc(smem_u32(pl.ops))
                                        : sw128_kmajor_desc(smem_u32(pl.ops));
    const uint32_t plane16 = static_cast<uint32_t>(nt * L::ROW) >> 4;
    const uint32_t d2 = pl.tmem + 2 * pl.dcols;
    if (slab > 0) {  // D2 of the slab before has been read
        const bool ok = mbar_wait(&b.d2_empty, (slab - 1) & 1);
        if (!__all_sync(0xffffffffu, ok)) return false;
        tc_fence_after();
    }
    for (int i = 0; i < nb; ++i, ++g) {
        const int s = g % G;
        const bool start = i % CHUNK_BLOCKS == 0;  // D1 restarts
        bool ok = mbar_wait(&b.op_full[s], (g / G) & 1);
        if (ok && start && cg >= 2) ok = mbar_wait(&b.d1_empty[cg & 1], ((cg >> 1) - 1) & 1);
        if (!__all_sync(0xffffffffu, ok)) return false;
        tc_fence_after();
        const uint64_t ad0 = desc0 + s * (static_cast<uint32_t>(pl.op_stride) >> 4);
        const uint32_t bt = pl.tmem + 3 * pl.dcols + s * L::OPCOLS;
        const uint32_t d1 = pl.tmem + (cg & 1) * pl.dcols;
        const bool end = (i + 1) % CHUNK_BLOCKS == 0 || i + 1 == nb;
        if (leader) {
#pragma unroll
            for (int j = 0; j < L::STEPS; ++j) {
                // corrections first, then hh, as split_gemm_kernel
#pragma unroll
                for (int q = 0; q < T::NPROD; ++q) {
                    const bool hh = q == T::NPROD - 1;
                    const uint64_t ad = ad0 + T::pa(q) * plane16 + j * (T::KMMA * T::ESZ / 16);
                    const uint32_t ba = bt + T::pb(q) * L::BCOLS + j * 8;
                    const uint32_t accum = hh ? (j > 0 || !start) : (i > 0 || j > 0 || q > 0);
                    mma_ts<T::FMT>(hh ? d1 : d2, ba, ad, idesc, accum);
                }
            }
            if (end) mma_commit(&b.d1_full[cg & 1]);
            mma_commit(&b.op_empty[s]);
        }
        if (end) ++cg;
        __syncwarp();
    }
    return true;
}

// A split warp's rows of the tile: a quarter, in eights.
__device__ __forceinline__ void quarter(int nt, int warp, int& r0, int& count) {
    const int cq = (nt + 31) / 32 * 8;
    r0 = (warp >> 2) * cq;
    count = max(0, min(cq, nt - r0));
}

// Split warps: convert the slab's blocks and leave its sums in acc: column
// 32 (w % 4) + lane of the tile, the rows of quarter().  `g` blocks came before
// the slab; `ring` walks the stages of the warp's group.
template <int PATH>
__device__ __forceinline__ bool convert(const Place& pl, Barriers& b, int nt, int nb, int warp,
                                        int lane, Ring& ring, uint32_t& g, uint32_t& cg,
                                        float (&acc)[CQ]) {
    using T = Traits<PATH>;
    using L = Lay<PATH>;
    const int q = warp & 3, h = warp >> 3, group = (warp >> 2) & 1;
    const int gt = h * 128 + q * 32 + lane;  // thread of the group
    const int plane = nt * L::ROW;
    int r0, count;
    quarter(nt, warp, r0, count);
    const uint32_t trow = pl.tmem + (static_cast<uint32_t>(q * 32) << 16);
#pragma unroll
    for (int j = 0; j < CQ; ++j) acc[j] = 0.0f;
    // acc += this warp's columns of the accumulator at column col
    auto drain = [&](uint32_t col) {
#pragma unroll
        for (int g0 = 0; g0 < CQ / 8; g0 += 2) {
            uint32_t v[16];
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if ((g0 + e) * 8 < count)
                    tmem_ld_32x32b_x8(trow + col + r0 + (g0 + e) * 8, &v[e * 8]);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if ((g0 + e) * 8 < count)
#pragma unroll
                    for (int f = 0; f < 8; ++f)
                        acc[(g0 + e) * 8 + f] =
                            __fadd_rn(acc[(g0 + e) * 8 + f], __uint_as_float(v[e * 8 + f]));
        }
    };
    auto drain_chunk = [&] {
        const int gone = b.gone;  // of the waits before; read behind this one it would take 0.5%
        const bool ok = wait_or_gone(b, &b.d1_full[cg & 1], (cg >> 1) & 1) && !gone;
        if (!__all_sync(0xffffffffu, ok)) return false;
        tc_fence_after();
        drain((cg & 1) * pl.dcols);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&b.d1_empty[cg & 1]);
        ++cg;
        return true;
    };
    int left = (nb + CHUNK_BLOCKS - 1) / CHUNK_BLOCKS;  // chunks to drain
    int due = CHUNK_BLOCKS + G - 1;  // the block by which the next chunk is known done
    for (int i = (group ^ g) & 1; i < nb; i += G) {
        wait_or_gone(b, &b.raw_full[ring.stage], ring.phase);
        const uint8_t* ra = pl.raw + ring.stage * pl.raw_stride;
        const float* rb =
            reinterpret_cast<const float*>(ra + nt * BK * 4) + 16 * h * TN + q * 32 + lane;
        // B: 16 k of one column, split and stored four words of each plane at a time.
        // All at once needs three times the registers, which the other roles' limit
        // (96) does not leave: 136 rows of one input, B in L2, BF16X6 41.0 us so, 38.6 in
        // steps, TF32X3 48.7 and 44.7; a grouped table of 22 314 and 263 (it spilled).
        const uint32_t bt = trow + 3 * pl.dcols + group * L::OPCOLS + h * (L::BCOLS / 2);
        constexpr int KS = 16 / T::ESZ;  // k per step
#pragma unroll
        for (int st = 0; st < 16 / KS; ++st) {
            uint32_t w[T::NSPLIT][4];
            const float* rs = rb + st * KS * TN;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                if constexpr (T::ESZ == 2) {
                    uint32_t pr[3];
                    split_pair(rs[2 * t * TN], rs[(2 * t + 1) * TN], pr);
#pragma unroll
                    for (int z = 0; z < 3; ++z) w[z][t] = pr[z];
                } else {
                    float v[3];
                    split_value<PATH>(rs[t * TN], v);
                    w[0][t] = __float_as_uint(v[0]);
                    w[1][t] = __float_as_uint(v[1]);
                }
            }
            if (st == 0 && g + i >= G) {  // the buffer's previous block has been multiplied
                wait_or_gone(b, &b.op_empty[group], (((g + i) / G) - 1) & 1);
                tc_fence_after();
            }
#pragma unroll
            for (int z = 0; z < T::NSPLIT; ++z)
                tmem_st_32x32b_x4(bt + z * L::BCOLS + st * 4, w[z]);
        }
        // A: units of 8 k of one row; a warp takes 8 rows x 4 chunks
        uint8_t* oa = pl.ops + group * pl.op_stride;
#pragma unroll
        for (int e = 0; e < NT_MAX * 4 / (32 * GROUP_WARPS); ++e) {
            const int u = gt + 32 * GROUP_WARPS * e;
            const int row = (u & 7) | ((u >> 5) << 3), c = (u >> 3) & 3;
            if (u >= nt * 4) break;
            const uint8_t* src = ra + row * 128;
            const float4 x = *reinterpret_cast<const float4*>(src + (((2 * c) ^ (row & 7)) << 4));
            const float4 y =
                *reinterpret_cast<const float4*>(src + (((2 * c + 1) ^ (row & 7)) << 4));
            if constexpr (T::ESZ == 2) {
                uint32_t a[4][3];
                split_pair(x.x, x.y, a[0]);
                split_pair(x.z, x.w, a[1]);
                split_pair(y.x, y.y, a[2]);
                split_pair(y.z, y.w, a[3]);
                uint8_t* dst = oa + row * 64 + ((c ^ ((row >> 1) & 3)) << 4);
#pragma unroll
                for (int z = 0; z < 3; ++z)
                    *reinterpret_cast<uint4*>(dst + z * plane) =
                        make_uint4(a[0][z], a[1][z], a[2][z], a[3][z]);
            } else {
                const float f[8] = {x.x, x.y, x.z, x.w,
                                    y.x, y.y, y.z, y.w};
                float v[8][3];
#pragma unroll
                for (int t = 0; t < 8; ++t) split_value<PATH>(f[t], v[t]);
#pragma unroll
                for (int z = 0; z < 2; ++z)
#pragma unroll
                    for (int t = 0; t < 2; ++t)
                        *reinterpret_cast<float4*>(oa + z * plane + row * 128 +
                                                   (((2 * c + t) ^ (row & 7)) << 4)) =
                            make_float4(v[4 * t][z], v[4 * t + 1][z], v[4 * t + 2][z],
                                        v[4 * t + 3][z]);
            }
        }
        fence_proxy_async_shared();  // A's planes before the MMA reads them
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(&b.op_full[group]);
            mbar_arrive(&b.raw_empty[ring.stage]);  // the stage has been read
        }
        ring.next();
        ring.next();
        if (i >= due) {  // the MMAs of block i - G are done, a chunk's last among them
            due += CHUNK_BLOCKS;
            --left;
            if (!drain_chunk()) return false;
        }
    }
    g += nb;
    for (; left > 0; --left)
        if (!drain_chunk()) return false;
    // D2 is complete: the last D1 commit came after every MMA
    if (nb > 0) drain(2 * pl.dcols);
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&b.d2_empty);
    return true;
}

// C rows m0 + r0 .. of a split warp's column, from its sums.
template <class P>
__device__ __forceinline__ void store_column(const P& p, int nt, int m0, int n0, int warp, int lane,
                                             const float (&acc)[CQ]) {
    int r0, count;
    quarter(nt, warp, r0, count);
    r0 += m0;
    const int col = n0 + 32 * (warp & 3) + lane, rows = min(count, p.m - r0);
    if (col >= p.n) return;
    const float alpha = p.alpha, beta = p.beta;
    const int64_t ld = p.ldc;
    float* c = p.C + r0 * ld + col;
#pragma unroll
    for (int j0 = 0; j0 < CQ; j0 += 8) {
        float old[8];
        if (beta != 0.0f) {
#pragma unroll
            for (int e = 0; e < 8; ++e) old[e] = j0 + e < rows ? c[(j0 + e) * ld] : 0.0f;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            if (j0 + e < rows) {
                float v = __fmul_rn(acc[j0 + e], alpha);
                if (beta != 0.0f) v = fmaf(old[e], beta, v);
                c[(j0 + e) * ld] = v;
            }
        }
    }
}

// One problem: CTA b computes slab b % splits of tile b / splits.
template <int PATH>
__global__ void __launch_bounds__(THREADS, 1)
    split_fused_kernel(const __grid_constant__ CUtensorMap tmA,
                       const __grid_constant__ CUtensorMap tmB, const Params p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) Barriers bars;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_s;
    uint8_t* smem = align_smem_1024(smem_raw);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform
    const int tile = blockIdx.x / p.splits, slab = blockIdx.x % p.splits;
    const int n0 = tile / p.tiles_m * TN, m0 = tile % p.tiles_m * p.nt;
    const int kb0 = slab * p.blocks;
    const int nb = max(0, min(p.blocks, (p.k + BK - 1) / BK - kb0));

    if (tid == 0) {
        init_barriers(bars);
        abort_s = 0;
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(&tmem_base_s, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_s, 0);
    const Place pl = make_place<PATH>(smem, p.nt, tmem);
    grid_wait();

    float acc[CQ];
    bool ok = true;
    if (warp == PRODUCER) {
        if (lane == 0) {
            tma_prefetch_desc(&tmA);
            tma_prefetch_desc(&tmB);
            Ring ring(pl.raws);
            int issued = 0;
            ok = produce<PATH>(pl, bars, &tmA, &tmB, p.nt, m0, n0, kb0, nb, ring, issued);
            settle(pl, bars, issued);
        }
    } else if (warp == MMA) {
        uint32_t g = 0, cg = 0;
        ok = multiply<PATH>(pl, bars, p.nt, nb, elect_one(), g, cg, 0);
    } else {
        Ring ring(pl.raws);
        if ((warp >> 2) & 1) ring.next();  // the second group's first stage
        uint32_t g = 0, cg = 0;
        ok = convert<PATH>(pl, bars, p.nt, nb, warp, lane, ring, g, cg, acc);
    }
    if (!ok) {
        abort_s = 1;
        atomicExch(p.status, SGEMM_B200_ERR_TIMEOUT);
    }

    // ------------------------------------------------------------ epilogue --
    if (p.splits == 1) {
        if (warp < SPLIT_WARPS && !abort_s) store_column(p, p.nt, m0, n0, warp, lane, acc);
    } else {
        // Partial sums meet in shared memory: [row][128 columns]; every CTA of the
        // cluster adds its share of the rows over the slabs, in slab order.
        __syncthreads();  // the landing ring is read out
        const bool good = !abort_s;
        float* part = reinterpret_cast<float*>(pl.raw);
        if (warp < SPLIT_WARPS) {
            int r0, count;
            quarter(p.nt, warp, r0, count);
            float* dst = part + r0 * TN + 32 * (warp & 3) + lane;
#pragma unroll
            for (int j = 0; j < CQ; ++j)
                if (j < count) dst[j * TN] = acc[j];
        }
        cluster_sync_all();
        if (good && warp < SPLIT_WARPS) {
            const int share = (p.nt + p.splits - 1) / p.splits;
            const int jend = min(min(p.nt, p.m - m0), (slab + 1) * share);
            const int col = n0 + 4 * lane;
            const bool vec = p.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15) == 0 &&
                             col + 3 < p.n;
            for (int j = slab * share + warp; j < jend; j += SPLIT_WARPS) {
                const uint32_t at = smem_u32(part + j * TN + 4 * lane);
                float4 v = ld_cluster_f4(at, 0);
                for (int s = 1; s < p.splits; ++s) {
                    const float4 w = ld_cluster_f4(at, s);
                    v.x = __fadd_rn(v.x, w.x);
                    v.y = __fadd_rn(v.y, w.y);
                    v.z = __fadd_rn(v.z, w.z);
                    v.w = __fadd_rn(v.w, w.w);
                }
                float o[4] = {__fmul_rn(v.x, p.alpha), __fmul_rn(v.y, p.alpha),
                              __fmul_rn(v.z, p.alpha), __fmul_rn(v.w, p.alpha)};
                float* c = p.C + (int64_t)(m0 + j) * p.ldc + col;
                if (vec) {
                    if (p.beta != 0.0f) {
                        const float4 old = *reinterpret_cast<const float4*>(c);
                        o[0] = fmaf(old.x, p.beta, o[0]);
                        o[1] = fmaf(old.y, p.beta, o[1]);
                        o[2] = fmaf(old.z, p.beta, o[2]);
                        o[3] = fmaf(old.w, p.beta, o[3]);
                    }
                    *reinterpret_cast<float4*>(c) = make_float4(o[0], o[1], o[2], o[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (col + e < p.n) c[e] = p.beta != 0.0f ? fmaf(c[e], p.beta, o[e]) : o[e];
                }
            }
        }
        cluster_sync_all();  // peers have read this CTA's partial
    }
    tc_fence_before();
    __syncthreads();  // every TMEM access is done
    if (warp == 0) {
        __syncwarp();
        tmem_dealloc(tmem, 512);
    }
}

// Many problems: persistent CTAs over the tiles of all of them, each tile's slabs
// one after the other with the slab sums added in slab order (through a scratch
// tile of the CTA's own), so every problem has split_fused_kernel's bits.  CTA c
// takes, in round r, the snake's position (see split_grouped_kernel) in a list
// sorted longest first.
template <int PATH>
__global__ void __launch_bounds__(THREADS, 1) split_fused_grouped_kernel(const GParams gp) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) Barriers bars;
    __shared__ uint32_t tmem_base_s;
    uint8_t* smem = align_smem_1024(smem_raw);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform
    const int grid = gridDim.x, cta = blockIdx.x;

    if (tid == 0) {
        init_barriers(bars);
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(&tmem_base_s, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_s, 0);
    const Place pl = make_place<PATH>(smem, NT_MAX, tmem);  // fits every problem's tiles
    grid_wait();

    // every role walks the same tiles and slabs: f(problem, tile, first block, blocks,
    // slab of the tile), false to stop
    auto walk = [&](auto f) {
        for (int r = 0; r * grid < gp.n_tiles; ++r) {
            const int t = r * grid + ((r & 1) ? grid - 1 - cta : cta);
            if (t >= gp.n_tiles) continue;
            const GTile tl = gp.tiles[t];
            const GProblem& p = gp.probs[tl.prob];
            const int all = (p.k + BK - 1) / BK, blocks = p.blocks, splits = p.splits;
            for (int s = 0; s < splits; ++s)
                if (!f(p, tl, s * blocks, max(0, min(blocks, all - s * blocks)), s)) return false;
        }
        return true;
    };
    bool ok = true;
    if (warp == PRODUCER) {
        if (lane == 0) {
            Ring ring(pl.raws);
            int issued = 0;
            ok = walk([&](const GProblem& p, const GTile& tl, int kb0, int nb, int s) {
                const CUtensorMap* maps = gp.maps + 2 * tl.prob;
                if (s == 0) {
                    tma_prefetch_desc(maps);
                    tma_prefetch_desc(maps + 1);
                }
                return produce<PATH>(pl, bars, maps, maps + 1, p.nt, tl.m0, tl.n0, kb0, nb, ring,
                                     issued);
            });
            settle(pl, bars, issued);
        }
    } else if (warp == MMA) {
        uint32_t g = 0, cg = 0, slab = 0;
        const bool leader = elect_one();
        ok = walk([&](const GProblem& p, const GTile&, int, int nb, int) {
            return multiply<PATH>(pl, bars, p.nt, nb, leader, g, cg, slab++);
        });
    } else {
        Ring ring(pl.raws);
        if ((warp >> 2) & 1) ring.next();  // the second group's first stage
        uint32_t g = 0, cg = 0;
        ok = walk([&](const GProblem& p, const GTile& tl, int, int nb, int s) {
            float acc[CQ];
            const int nt = p.nt, splits = p.splits;
            if (!convert<PATH>(pl, bars, nt, nb, warp, lane, ring, g, cg, acc)) return false;
            if (splits > 1) {  // the running sum over the slabs before
                int r0, count;
                quarter(nt, warp, r0, count);
                float* sum = gp.sums + (int64_t)cta * TN * NT_MAX + r0 * TN + 32 * (warp & 3) +
                             lane;
                // eight loads in flight, and no store between them: a load, an add and
                // a store per row cost a trip to L2 each
                if (s > 0) {
#pragma unroll
                    for (int j0 = 0; j0 < CQ; j0 += 8) {
                        float before[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            before[e] = j0 < count ? __ldcg(sum + (j0 + e) * TN) : 0.0f;
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            acc[j0 + e] = __fadd_rn(before[e], acc[j0 + e]);
                    }
                }
                if (s + 1 < splits) {
#pragma unroll
                    for (int j = 0; j < CQ; ++j)
                        if (j < count) __stcg(sum + j * TN, acc[j]);
                    return true;
                }
            }
            store_column(p, nt, tl.m0, tl.n0, warp, lane, acc);
            return true;
        });
    }
    if (!ok) atomicExch(gp.status, SGEMM_B200_ERR_TIMEOUT);
    tc_fence_before();
    __syncthreads();  // every TMEM access is done
    if (warp == 0) {
        __syncwarp();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace fused
