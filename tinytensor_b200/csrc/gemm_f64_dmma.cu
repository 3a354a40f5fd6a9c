// gemm_f64_dmma.cu -- f64 batched GEMM on the FP64 tensor-core path (DMMA).
//
// There is no f64 kind of tcgen05.mma; double precision runs on warp-level
// mma.sync (m16n8k4, f64 in / f64 accumulate).  The accumulation is IEEE fp64 FMA
// in the tensor core, so results sit within a few ulp of the reference's fp64 sums
// (tinytensor/tensor/backend/cuda/kernel/matmul.cuh:74,131 accumulate in T).
// Replaces matmul_kernel<double> of the reference.
//
// A CTA is 4 warps on a tile of 64 x 64 or 32 x 32, accumulators in registers; cp.async
// brings K blocks of 16 into a ring of shared-memory stages (16 bytes a copy where the view is
// aligned, 8 for any other strides: f64 views never need a copy), and several CTAs share an SM so
// that one keeps the DMMA pipe busy while another waits for its loads.  When the tiles alone leave
// SMs idle, or make a nearly empty last wave, the CTAs of a cluster split K (sums meet through
// distributed shared memory: one launch, no scratch, fixed order).
//
// Bound: the DMMA pipe, 37.1 TFLOP/s measured.  4096^3 runs at 34.6.  Against one 128 x 64 tile shape
// with loads through registers and no split: 4096^3 4.20 -> 3.98 ms; 2048 x 1024 x 1536, 384 such tiles
// on 148 SMs, 293 -> 211 us; 512^3 53 -> 14; 32 x 1024 x 32 97 -> 6.  A 128 x 64 tile in the present
// form was never the fastest of the three (4096^3 4.06 ms, 2048 x 1536 x 1024 219 us against 206).
#include <atomic>

#include "common.cuh"
#include "cp_async_tile.cuh"

namespace ttb {
namespace {

constexpr int BK = 16;
constexpr int THREADS = 128;

struct DmmaArgs {
    const double *a;
    const double *b;
    double *c;
    int N, K, M;
    long long a_sb, a_s, a_k;  // element strides: batch, row of A / column of B, K
    long long b_sb, b_s, b_k;
    long long c_sb, c_si, c_sj;
    int a_vec, b_vec;  // 16-byte loads
    int c_vec;         // rows of C start on a 16-byte boundary
    int splits, k_per_split;
    int col_tiles;     // blockIdx.x = row of tiles * col_tiles + column
    Epilogue ep;
};

__device__ __forceinline__ void dmma_m16n8k4(double (&c)[4], double a0, double a1, double b0) {
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

__device__ __forceinline__ double finish(double v, const Epilogue &ep, long long b, int i, int j) {
    // addend (bias row / column, or C itself): the thread that reads it stores the result
    if (ep.d) v += static_cast<const double *>(ep.d)[b * ep.d_sb + i * ep.d_si + j * ep.d_sj];
    if (ep.act == TTB_ACT_RELU) v = v < 0.0 ? 0.0 : v;
    return v;
}

template <int BM, int BN, int STAGES, bool A_MN, bool B_MN>
struct Tile {
    using LoadA = TileLoader<double, BK, BM, A_MN, THREADS>;
    using LoadB = TileLoader<double, BK, BN, B_MN, THREADS>;
    static constexpr int STAGE_WORDS = LoadA::WORDS + LoadB::WORDS;
    static constexpr int SMEM = STAGES * STAGE_WORDS * 8;
    static_assert(BM * (BN + 2) * 8 <= SMEM, "the sums of a K split reuse the ring");
};

// Two by two warps, each on a quarter of the tile.
template <int BM, int BN, int STAGES, int MIN_CTAS, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(THREADS, MIN_CTAS) gemm_f64_dmma_kernel(const DmmaArgs p) {
    using T = Tile<BM, BN, STAGES, A_MN, B_MN>;
    constexpr int WM = BM / 2, WN = BN / 2, MT = WM / 16, NT = WN / 8;
    constexpr int PA = T::LoadA::PITCH, PB = T::LoadB::PITCH;
    extern __shared__ __align__(16) double smem[];
    after_previous_kernel();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;  // MMA fragment coordinates
    const int wm = (warp >> 1) * WM, wn = (warp & 1) * WN;
    const int row_tile = blockIdx.x / p.col_tiles;
    const int m0 = row_tile * BM, n0 = (blockIdx.x - row_tile * p.col_tiles) * BN;
    const long long batch = blockIdx.y / p.splits;
    const int split = blockIdx.y % p.splits;
    const int k_begin = split * p.k_per_split;
    const int k_end = k_begin + p.k_per_split < p.K ? k_begin + p.k_per_split : p.K;
    const uint32_t ring = smem_addr(smem);

    typename T::LoadA load_a(p.a + batch * p.a_sb, p.a_s, p.a_k, m0, p.N, k_begin, p.a_vec != 0);
    typename T::LoadB load_b(p.b + batch * p.b_sb, p.b_s, p.b_k, n0, p.M, k_begin, p.b_vec != 0);
    int k_left = k_end - k_begin;  // K not yet asked for
    auto load = [&](int stage) {
        const uint32_t dst = ring + stage * (T::STAGE_WORDS * 8);
        load_a.load(dst, k_left);
        load_b.load(dst + T::LoadA::WORDS * 8, k_left);
        k_left -= BK;
    };

    double acc[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;

    const int num_kb = k_end > k_begin ? (k_end - k_begin + BK - 1) / BK : 0;
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < num_kb) load(s);
        cp_commit();
    }
    int stage = 0;
    for (int kb = 0; kb < num_kb; ++kb) {
        cp_wait<STAGES - 2>();
        __syncthreads();
        if (k_left > 0) load(stage == 0 ? STAGES - 1 : stage - 1);
        cp_commit();
        const double *as = smem + stage * T::STAGE_WORDS, *bs = as + T::LoadA::WORDS;
        if (++stage == STAGES) stage = 0;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            // Fragments of m16n8k4: A(row g / g + 8, k t), B(k t, column g).
            double af[MT][2], bf[NT];
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int row = wm + i * 16 + g + 8 * u;
                    af[i][u] = as[A_MN ? (k + t) * PA + row : row * PA + k + t];
                }
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const int col = wn + j * 8 + g;
                bf[j] = bs[B_MN ? (k + t) * PB + col : col * PB + k + t];
            }
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j) dmma_m16n8k4(acc[i][j], af[i][0], af[i][1], bf[j]);
        }
    }

    double *c = p.c + batch * p.c_sb;
    if (p.splits == 1) {
        // C fragment: c0, c1 -> row g, columns 2t, 2t + 1; c2, c3 -> row g + 8.
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = m0 + wm + i * 16 + g + h * 8;
                if (row >= p.N) continue;
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const int col = n0 + wn + j * 8 + 2 * t;
                    if (col >= p.M) continue;
                    double *dst = c + row * p.c_si + col * p.c_sj;
                    const double v0 = finish(acc[i][j][2 * h], p.ep, batch, row, col);
                    if (col + 1 < p.M) {
                        const double v1 = finish(acc[i][j][2 * h + 1], p.ep, batch, row, col + 1);
                        if (p.c_vec) {
                            *reinterpret_cast<double2 *>(dst) = make_double2(v0, v1);
                        } else {
                            dst[0] = v0;
                            dst[p.c_sj] = v1;
                        }
                    } else {
                        dst[0] = v0;
                    }
                }
            }
        return;
    }
    // Sums of the cluster's CTAs: each leaves its tile in shared memory, CTA r finishes rows
    // [r, r + 1) * BM / splits of it.
    constexpr int PS = BN + 2;
    cp_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<double2 *>(&smem[(wm + i * 16 + g + h * 8) * PS + wn + j * 8 + 2 * t]) =
                    make_double2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
    cluster_sync();
    const int rows = BM / p.splits, r0 = static_cast<int>(cluster_rank()) * rows;
    for (int idx = threadIdx.x; idx < rows * (BN / 2); idx += THREADS) {
        const int r = r0 + idx / (BN / 2), cc = (idx % (BN / 2)) * 2;
        const int row = m0 + r, col = n0 + cc;
        if (row >= p.N || col >= p.M) continue;
        double v0 = 0.0, v1 = 0.0;
        for (int q = 0; q < p.splits; ++q) {
            const double2 w = *reinterpret_cast<const double2 *>(in_cta(&smem[r * PS + cc], static_cast<uint32_t>(q)));
            v0 += w.x;
            v1 += w.y;
        }
        double *dst = c + row * p.c_si + col * p.c_sj;
        v0 = finish(v0, p.ep, batch, row, col);
        if (col + 1 < p.M) v1 = finish(v1, p.ep, batch, row, col + 1);
        if (p.c_vec && col + 1 < p.M) {
            *reinterpret_cast<double2 *>(dst) = make_double2(v0, v1);
        } else {
            dst[0] = v0;
            if (col + 1 < p.M) dst[p.c_sj] = v1;
        }
    }
    cluster_sync();  // nobody leaves while its sums are being read
}

template <int BM, int BN, int STAGES, int MIN_CTAS, bool A_MN, bool B_MN>
int launch_tile(const Problem &p, DmmaArgs &args, int splits) {
    constexpr int bytes = Tile<BM, BN, STAGES, A_MN, B_MN>::SMEM;
    auto kernel = gemm_f64_dmma_kernel<BM, BN, STAGES, MIN_CTAS, A_MN, B_MN>;
    if (bytes > 48 * 1024) {
        static std::atomic<bool> ready[64];
        if (!ready[p.device & 63].load(std::memory_order_acquire)) {
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
            if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(smem)");
            ready[p.device & 63].store(true, std::memory_order_release);
        }
    }
    args.splits = splits;
    const int kb = (args.K + BK - 1) / BK;
    args.k_per_split = (kb + splits - 1) / splits * BK;
    args.col_tiles = static_cast<int>((p.M + BN - 1) / BN);
    const dim3 grid(static_cast<unsigned>(args.col_tiles * ((p.N + BM - 1) / BM)), static_cast<unsigned>(p.B * splits));
    const cudaError_t e =
        launch_after(kernel, {grid, THREADS, bytes, p.stream, dim3(1, static_cast<unsigned>(splits), 1)}, args);
    return e == cudaSuccess ? TTB_OK : cuda_fail(e, "gemm_f64_dmma_kernel launch");
}

template <int BM, int BN, int STAGES, int MIN_CTAS>
int launch_layout(const Problem &p, DmmaArgs &args, int splits, bool a_mn, bool b_mn) {
    if (a_mn)
        return b_mn ? launch_tile<BM, BN, STAGES, MIN_CTAS, true, true>(p, args, splits)
                    : launch_tile<BM, BN, STAGES, MIN_CTAS, true, false>(p, args, splits);
    return b_mn ? launch_tile<BM, BN, STAGES, MIN_CTAS, false, true>(p, args, splits)
                : launch_tile<BM, BN, STAGES, MIN_CTAS, false, false>(p, args, splits);
}

// 16-byte loads or stores: unit stride along the moved dim, everything else a multiple of 16 bytes.
bool vec_ok(const void *ptr, long long unit, long long other, long long batch) {
    return unit == 1 && (other & 1) == 0 && (batch & 1) == 0 && (reinterpret_cast<uintptr_t>(ptr) & 15) == 0;
}

constexpr int kTile[2] = {64, 32}, kPerSm[2] = {3, 4};  // rows and columns of a tile, CTAs an SM holds
// Share of the DMMA pipe's rate that 1, 2, ... CTAs of a tile reach on an SM.
constexpr double kRate[2][4] = {{0.71, 0.89, 0.94, 0.94}, {0.52, 0.79, 0.86, 0.87}};

// Tile and K split with the smallest estimate, in cycles of an SM's DMMA pipe (64 multiply-adds a
// cycle): the SM with the most CTAs runs them in rounds of as many as it holds; a round costs its
// first loads, and a split the exchange of the sums.  Rates and costs are fitted to the times of
// 15 shapes (32 to 4096) in all forms: 6 % off on average, and the form it picks takes 1.04 times the
// best one's time at worst.
void choose(const Problem &p, int sms, int *tile, int *splits) {
    double best = 1e300;
    const int want_tile = *tile, want_splits = *splits;
    const long long kb = (p.K + BK - 1) / BK;
    for (int t = 0; t < 2; ++t) {
        const long long tiles = (p.N + kTile[t] - 1) / kTile[t] * ((p.M + kTile[t] - 1) / kTile[t]);
        if ((want_tile >= 0 && t != want_tile) || tiles > 0x7FFFFFFF) continue;
        const double area = kTile[t] * kTile[t];
        for (int s = 1; s <= 8; s *= 2) {
            if ((want_splits > 0 && s != want_splits) || p.B * s > 65535) continue;
            if (want_splits <= 0 && s > 1 && kb < 2 * s) break;
            const double one = area * static_cast<double>((kb + s - 1) / s) * BK / 64.0;
            const long long most = (tiles * p.B * s + sms - 1) / sms;
            const long long full = most / kPerSm[t], rest = most % kPerSm[t];
            const double rounds = static_cast<double>(full + (rest > 0));
            double cost = static_cast<double>(full * kPerSm[t]) * one / kRate[t][kPerSm[t] - 1] + rounds * 950.0;
            if (rest > 0) cost += static_cast<double>(rest) * one / kRate[t][rest - 1];
            if (s > 1) cost += rounds * 1230.0 + static_cast<double>(most) * area / 2.0;
            if (cost < best) {
                best = cost;
                *tile = t;
                *splits = s;
            }
        }
    }
}

// The FP64 tensor-core rate itself: every warp keeps the widest tile's 16 independent 16 x 8
// accumulator tiles in registers and issues m16n8k4 MMAs on register operands, with no memory
// traffic.  What this loop reaches is the ceiling the GEMM kernel's roofline is quoted against.
constexpr int PEAK_THREADS = 256, PEAK_TILES = 16;
__global__ void __launch_bounds__(PEAK_THREADS) dmma_peak_kernel(double *sink, int iters, double a_seed, double b_seed) {
    double acc[PEAK_TILES][4];
#pragma unroll
    for (int j = 0; j < PEAK_TILES; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = 0.0;
    double a0 = a_seed + threadIdx.x * 1e-9, a1 = a_seed - threadIdx.x * 1e-9, b0 = b_seed;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int j = 0; j < PEAK_TILES; ++j) dmma_m16n8k4(acc[j], a0, a1, b0);
        b0 = -b0;  // keeps the sums bounded and the loop from being folded
    }
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < PEAK_TILES; ++j) s += acc[j][0] + acc[j][1] + acc[j][2] + acc[j][3];
    if (s == 123456.789) sink[0] = s;  // never true: the result only has to look used
}

}  // namespace

// Runs dmma_peak_kernel on `device` (two CTAs of 8 warps per SM) and returns the best of three
// launches in TFLOP/s (2 flops per multiply-add of an m16n8k4 MMA).
int measure_fp64_tensor_peak(int device, double *tflops) {
    int sms = 0;
    int rc = sm_count(device, &sms);
    if (rc != TTB_OK) return rc;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    double *sink = nullptr;
    e = cudaMalloc(&sink, sizeof(double));
    if (e != cudaSuccess) return cuda_fail(e, "cudaMalloc");
    cudaEvent_t t0, t1;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
    const int iters = 1 << 14;
    const int ctas = 2 * sms;
    const double flop = 2.0 * 16 * 8 * 4 * (PEAK_TILES) * static_cast<double>(iters) * (PEAK_THREADS / 32) * ctas;
    double best = 0.0;
    for (int rep = 0; rep < 4 && e == cudaSuccess; ++rep) {  // the first launch is the warm-up
        cudaEventRecord(t0, nullptr);
        dmma_peak_kernel<<<ctas, PEAK_THREADS>>>(sink, iters, 1.0000001, 0.9999999);
        cudaEventRecord(t1, nullptr);
        e = cudaEventSynchronize(t1);
        float ms = 0.f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, t0, t1);
        if (e == cudaSuccess && rep > 0 && ms > 0.f && flop / (ms * 1e9) > best) best = flop / (ms * 1e9);
    }
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    cudaFree(sink);
    if (e != cudaSuccess) return cuda_fail(e, "dmma_peak_kernel");
    note_launch(-1, 4);
    *tflops = best;
    return TTB_OK;
}

bool f64_dmma_eligible(const Problem &p) {
    // 32-bit extents inside the kernel, and the launch limits of the grid
    return p.dtype == TTB_F64 && p.N <= 0x3FFFFFFF && p.M <= 0x3FFFFFFF && p.K <= 0x3FFFFFFF &&
           (p.N + kTile[0] - 1) / kTile[0] * ((p.M + kTile[0] - 1) / kTile[0]) <= 0x7FFFFFFF && p.B <= 65535;
}

int launch_f64_dmma(const Problem &p, int tile, int splits) {
    if (!f64_dmma_eligible(p)) {
        set_error("f64 DMMA kernel: extents beyond its launch limits");
        return TTB_ELIMIT;
    }
    int sms = 148;
    sm_count(p.device, &sms);
    int t = tile > 1 ? 1 : tile, s = splits;
    choose(p, sms, &t, &s);
    if (t < 0 || s <= 0) {
        set_error("f64 DMMA kernel: the forced tile or split exceeds the launch limits");
        return TTB_ELIMIT;
    }
    DmmaArgs a{};
    a.a = static_cast<const double *>(p.a);
    a.b = static_cast<const double *>(p.b);
    a.c = static_cast<double *>(p.c);
    a.N = static_cast<int>(p.N);
    a.K = static_cast<int>(p.K);
    a.M = static_cast<int>(p.M);
    a.a_sb = p.a_sb;
    a.a_s = p.a_si;
    a.a_k = p.a_sk;
    a.b_sb = p.b_sb;
    a.b_s = p.b_sj;
    a.b_k = p.b_sk;
    a.c_sb = p.c_sb;
    a.c_si = p.c_si;
    a.c_sj = p.c_sj;
    a.ep = epilogue_of(p);
    // loads walk the dim with the smaller stride
    const bool a_mn = p.a_si < p.a_sk, b_mn = p.b_sj < p.b_sk;
    a.a_vec = a_mn ? vec_ok(p.a, p.a_si, p.a_sk, p.a_sb) : vec_ok(p.a, p.a_sk, p.a_si, p.a_sb);
    a.b_vec = b_mn ? vec_ok(p.b, p.b_sj, p.b_sk, p.b_sb) : vec_ok(p.b, p.b_sk, p.b_sj, p.b_sb);
    a.c_vec = vec_ok(p.c, p.c_sj, p.c_si, p.c_sb);
    const int rc = t == 0 ? launch_layout<64, 64, 3, 3>(p, a, s, a_mn, b_mn) : launch_layout<32, 32, 4, 4>(p, a, s, a_mn, b_mn);
    if (rc == TTB_OK) note_launch(TTB_VARIANT_DMMA_F64, 1);
    return rc;
}

}  // namespace ttb
