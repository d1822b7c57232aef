// Normal equations G = [J r]^T [J r] per run (A = J^T J in the top-left P x P block,
// g = J^T r in column P, r^T r in the corner).
//
// Kernels:
//   gram_exact_kernel -- every entry is one fused multiply-add chain over the rows in ascending
//     order, acc = fma(u_r, v_r, acc) from acc = 0: bit-identical to the reference's
//     normal_equations_host / gram_dot (include/mikroptim/optim/normal_equations.hpp:19,33).
//     One CTA per run and pair of column tiles streams row tiles through shared memory; each
//     thread advances four chains (one in batches of at most eight columns).
//   gram_dmma_kernel -- FP64 tensor cores: mma.sync.m8n8k4 (f64) on 8 x 8 output tiles of the
//     upper triangle, row tiles of J staged in shared memory; fixed k order (deterministic, not
//     bit-identical to the chain). gram_one_tile_kernel: at most eight columns, no staging.
#include "launch.cuh"

namespace mkb {

namespace {

constexpr int kGramThreads = 256;
constexpr int kMaxCols = MKB_MAX_VARIABLES + 1;
// exact kernel: threads, rows of a staged tile, column stride
constexpr int kExactThreads = 64;
constexpr int kExactRows = 32;
constexpr int kExactLd = kExactRows + 2;

// Column c of run `run`: J columns are strided by `stride` per run (the largest P of an uneven
// batch, else P); column P is the residual.
__device__ inline const double* column(const double* J, const double* r, int64_t run, int c,
                                       int P, int stride, int64_t R) {
    return c < P ? J + (run * stride + c) * R : r + run * R;
}

// 8-byte asynchronous copy to shared memory; zero fill (no read) when `in` is false.
__device__ __forceinline__ void copy_async8(double* dst, const double* src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_addr(dst)), "l"(src),
                 "r"(in ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int kPending>
__device__ __forceinline__ void copy_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

// One CTA per run and pair of 8 kSub-column tiles (ta <= tb); thread (ti, tj) advances the kSub^2
// chains of columns {ti, ti + 8} x {tj, tj + 8}, so a row costs it 2 kSub shared loads for kSub^2
// multiply-adds, eight rows' loads ahead of their use. Row tiles come in by 8-byte cp.async (a
// column starts at any multiple of R), kStages deep. What bounds it is the chain itself, R
// dependent multiply-adds, and the shared loads beside it. The column stride of 17 16-byte units
// keeps the two-row loads of eight neighbouring columns on different banks. 48 runs of P = 29 and
// 28,896 rows: one CTA per run with one chain per pair and synchronous tiles took 2,975 us, four
// chains a thread loaded as they go 1,445 us, 128 threads of two chains with loads ahead 525 us,
// this 455 us.
// kSub = 1 for batches of at most eight columns, where three of four chains would be no one's.
// kPacked: for more CTAs than fit the GPU at once. Three stages instead of four (which hide the
// loads better) let seven CTAs of kSub = 2 reside on an SM instead of six. And a last tile of at
// most kTail columns, which leaves half the threads of its pairs idle, has its own chains done by
// them in pair (0, tb), so that pair (tb, tb) does nothing. One CTA per run / kSub = 2 and nothing
// packed / now (us): 512 runs of 900 rows, P = 6 24.7 / 28.7 / 17.2, P = 16 56.9 / 70.0 / 55.4;
// 16,384 runs of 35 rows, P = 16 137 / 157 / 114, P = 64 866 / 901 / 748.
constexpr int kTail = 4;
constexpr int kFewExactCtas = 148 * 6;  // that fit at once with four stages
template <int kSub, bool kPacked>
__global__ void __launch_bounds__(kExactThreads)
gram_exact_kernel(const double* __restrict__ J, const double* __restrict__ r, int P_all,
                  int64_t R, double* __restrict__ gram, const int* __restrict__ run_mask,
                  const VarParams* __restrict__ vt, int stride, int tile_pairs) {
    constexpr int kCols = 8 * kSub, kStages = kPacked ? 3 : 4;
    __shared__ __align__(16) double tile[kStages][2 * kCols * kExactLd];
    // grid (runs, tile pairs), walked so that the pairs of a run are neighbours (their columns
    // are in L2 once)
    const int64_t block = static_cast<int64_t>(blockIdx.y) * gridDim.x + blockIdx.x;
    const int64_t run = block / tile_pairs;
    if (run_mask != nullptr && run_mask[run] == 0) return;
    int ta = static_cast<int>(block - run * tile_pairs), tb = 0;
    while (ta > tb) ta -= ++tb;  // pair index -> (ta, tb), column by column of the triangle
    const int P = vt != nullptr ? vt[run].P : P_all;
    const int n = P + 1;
    if (tb * kCols >= n) return;
    const bool diagonal = ta == tb;
    const bool tail = kPacked && tb > 0 && n - tb * kCols <= kTail;
    if (diagonal && tail) return;
    const int tid = threadIdx.x, ti = tid >> 3, tj = tid & 7;
    // this thread's row of every staged tile and the columns it copies; columns past n and rows
    // past R are filled with zeros
    constexpr int kCopies = 2 * kCols * kExactRows / kExactThreads;
    constexpr int kCopyStep = kExactThreads / kExactRows;
    const int copies = diagonal ? kCopies / 2 : kCopies;
    const int k_in = tid & (kExactRows - 1), c_in = tid / kExactRows;
    const double* src[kCopies];
    bool in[kCopies];
#pragma unroll
    for (int i = 0; i < kCopies; ++i) {
        const int c = c_in + i * kCopyStep;
        const int col = c < kCols ? ta * kCols + c : tb * kCols + c - kCols;
        in[i] = col < n && i < copies;
        src[i] = in[i] ? column(J, r, run, col, P, stride, R) + k_in : r;
    }
    auto load = [&](int64_t step) {
        const int64_t r0 = step * kExactRows;
        double* dst = tile[step % kStages] + c_in * kExactLd + k_in;
        const bool row = r0 + k_in < R;
#pragma unroll
        for (int i = 0; i < kCopies; ++i)
            if (i < copies)
                copy_async8(dst + i * kCopyStep * kExactLd, in[i] && row ? src[i] + r0 : r,
                            in[i] && row);
    };
    const int64_t steps = (R + kExactRows - 1) / kExactRows;
    for (int s = 0; s < kStages - 1; ++s) {
        if (s < steps) load(s);
        copy_async_commit();
    }
    // chains {p, p + 8} x {q, q + 8}; on the diagonal (p + 8, q) is the transposed pair's
    const bool own = tail && ta == 0 && tj >= kTail;  // one of the tail's own chains
    const int p = (own ? tb : ta) * kCols + ti, q = tb * kCols + tj - (own ? kTail : 0);
    const bool mine = p < n && q < n && (!(diagonal || own) || p <= q);
    const int u_at = (own ? kCols + ti : ti) * kExactLd;
    const int v_at = (diagonal ? tj : kCols + tj - (own ? kTail : 0)) * kExactLd;
    constexpr int kNext = 8 * kExactLd;
    double acc[kSub][kSub] = {};
    for (int64_t step = 0; step < steps; ++step) {
        copy_async_wait<kStages - 2>();
        __syncthreads();  // this step's rows are here; the slot of the last one is free
        if (step + kStages - 1 < steps) load(step + kStages - 1);
        copy_async_commit();
        if (!mine) continue;
        const double* u = tile[step % kStages] + u_at;
        const double* v = tile[step % kStages] + v_at;
        const int64_t left = R - step * kExactRows;
        if (left >= kExactRows) {
            // eight rows' loads ahead of their chains
            double2 x[2][kSub][4], y[2][kSub][4];
            auto fetch = [&](int k, int h) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
#pragma unroll
                    for (int c = 0; c < kSub; ++c)
                        x[h][c][i] =
                            *reinterpret_cast<const double2*>(u + c * kNext + k + 2 * i);
#pragma unroll
                    for (int c = 0; c < kSub; ++c)
                        y[h][c][i] =
                            *reinterpret_cast<const double2*>(v + c * kNext + k + 2 * i);
                }
            };
            fetch(0, 0);
#pragma unroll
            for (int k = 0; k < kExactRows; k += 8) {
                const int h = (k >> 3) & 1;
                if (k + 8 < kExactRows) fetch(k + 8, h ^ 1);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
#pragma unroll
                    for (int e = 0; e < kSub * kSub; ++e)
                        acc[e / kSub][e % kSub] = fma(x[h][e / kSub][i].x, y[h][e % kSub][i].x,
                                                      acc[e / kSub][e % kSub]);
#pragma unroll
                    for (int e = 0; e < kSub * kSub; ++e)
                        acc[e / kSub][e % kSub] = fma(x[h][e / kSub][i].y, y[h][e % kSub][i].y,
                                                      acc[e / kSub][e % kSub]);
                }
            }
        } else {
            for (int k = 0; k < left; ++k) {
#pragma unroll
                for (int e = 0; e < kSub * kSub; ++e)
                    acc[e / kSub][e % kSub] = fma(u[e / kSub * kNext + k], v[e % kSub * kNext + k],
                                                  acc[e / kSub][e % kSub]);
            }
        }
    }
    if (!mine) return;
    double* g = gram + run * (stride + 1) * (stride + 1);
#pragma unroll
    for (int i = 0; i < kSub; ++i) {
#pragma unroll
        for (int j = 0; j < kSub; ++j) {
            const int c = p + 8 * i, d = q + 8 * j;
            if (c >= n || d >= n) continue;
            g[static_cast<int64_t>(d) * n + c] = acc[i][j];
            g[static_cast<int64_t>(c) * n + d] = acc[i][j];
        }
    }
}

// ---- DMMA ------------------------------------------------------------------------------------
constexpr int kDmmaRows = 64;                  // rows per shared tile (16 k-steps of 4)
constexpr int kDmmaMaxTiles = (kMaxCols + 7) / 8;  // 9 column tiles of 8 for P <= 64
constexpr int kDmmaMaxPairs = kDmmaMaxTiles * (kDmmaMaxTiles + 1) / 2;  // 45
constexpr int kDmmaWarps = kGramThreads / 32;
constexpr int kDmmaTilesPerWarp = (kDmmaMaxPairs + kDmmaWarps - 1) / kDmmaWarps;  // 6

// D = A * B + C for one 8x8x4 FP64 tile. Fragments (PTX ISA, mma.m8n8k4 .f64): lane l holds
// A[l/4][l%4], B[l%4][l/4] and D[l/4][2(l%4) + {0, 1}].
__device__ inline void dmma_8x8x4(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// The sums of a run of at most eight columns (P <= 7): one 8 x 8 tile, whose two fragments are the
// same entries (lane l: column l / 4, row l % 4), so every warp streams its own rows straight from
// memory, 32 bytes of each column at a time, and the eight warps' sums are added in order. The
// tiles below leave seven warps idle here and wait for a tile at a time; 1,024 runs of P = 4 and
// 900 rows, in L2: 32.5 us there, 6.7 us here. Which way a run goes is decided by its own P alone,
// so that its bits are the same in every batch. part: [kDmmaWarps * 64] in shared memory.
__device__ __forceinline__ void one_tile_sums(const double* J, const double* r, int64_t run, int P,
                                              int stride, int64_t R, double* part, double* gram) {
    const int n = P + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gid = lane >> 2, tig = lane & 3;
    const bool in = gid < n;
    const double* col = in ? column(J, r, run, gid, P, stride, R) : r;
    // a warp's rows: 4 kUnroll at a time, the warps in turn
    constexpr int kUnroll = 4;
    double d0 = 0.0, d1 = 0.0;
    for (int64_t k0 = int64_t(warp) * 4 * kUnroll; k0 < R; k0 += kDmmaWarps * 4 * kUnroll) {
        double x[kUnroll];
#pragma unroll
        for (int i = 0; i < kUnroll; ++i) {
            const int64_t k = k0 + 4 * i + tig;
            x[i] = in && k < R ? col[k] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < kUnroll; ++i) dmma_8x8x4(d0, d1, x[i], x[i]);
    }
    part[warp * 64 + gid * 8 + 2 * tig] = d0;
    part[warp * 64 + gid * 8 + 2 * tig + 1] = d1;
    __syncthreads();
    if (threadIdx.x < 64) {
        const int row = threadIdx.x >> 3, c = threadIdx.x & 7;
        double sum = part[threadIdx.x];
        for (int w = 1; w < kDmmaWarps; ++w) sum += part[w * 64 + threadIdx.x];
        if (row < n && c < n) gram[run * (stride + 1) * (stride + 1) + row * n + c] = sum;
    }
}

__global__ void __launch_bounds__(kGramThreads)
gram_dmma_kernel(const double* __restrict__ J, const double* __restrict__ r, int P_all,
                 int64_t R, double* __restrict__ gram, const int* __restrict__ run_mask,
                 const VarParams* __restrict__ vt, int stride) {
    // tile[k][c] row-major with a padded row stride (columns of the 8-wide tiles are read
    // across lanes)
    constexpr int kStride = kDmmaMaxTiles * 8 + 1;
    __shared__ double tile[kDmmaRows * kStride];
    const int64_t run = blockIdx.x;
    if (run_mask != nullptr && run_mask[run] == 0) return;
    const int P = vt != nullptr ? vt[run].P : P_all;
    const int n = P + 1;
    if (n <= 8) {
        one_tile_sums(J, r, run, P, stride, R, tile, gram);
        return;
    }
    const int T = (n + 7) / 8;
    const int pairs = T * (T + 1) / 2;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int gid = lane >> 2, tig = lane & 3;
    int ti[kDmmaTilesPerWarp], tj[kDmmaTilesPerWarp];
    double c0[kDmmaTilesPerWarp], c1[kDmmaTilesPerWarp];
    int mine = 0;
    for (int e = warp; e < pairs; e += kDmmaWarps) {
        int j = 0, rem = e;
        while (rem >= j + 1) {
            rem -= j + 1;
            ++j;
        }
        ti[mine] = rem;
        tj[mine] = j;
        c0[mine] = c1[mine] = 0.0;
        ++mine;
    }
    for (int64_t r0 = 0; r0 < R; r0 += kDmmaRows) {
        const int rows = static_cast<int>(R - r0 < kDmmaRows ? R - r0 : kDmmaRows);
        __syncthreads();
        for (int i = threadIdx.x; i < T * 8 * kDmmaRows; i += kGramThreads) {
            const int c = i / kDmmaRows;
            const int k = i - c * kDmmaRows;
            double v = 0.0;
            if (c < n && k < rows) v = column(J, r, run, c, P, stride, R)[r0 + k];
            tile[k * kStride + c] = v;
        }
        __syncthreads();
        const int ksteps = (rows + 3) / 4;
#pragma unroll
        for (int m = 0; m < kDmmaTilesPerWarp; ++m) {
            if (m < mine) {
                const int ca = ti[m] * 8 + gid;
                const int cb = tj[m] * 8 + gid;
                double d0 = c0[m], d1 = c1[m];
                for (int ks = 0; ks < ksteps; ++ks) {
                    const int k = ks * 4 + tig;
                    dmma_8x8x4(d0, d1, tile[k * kStride + ca], tile[k * kStride + cb]);
                }
                c0[m] = d0;
                c1[m] = d1;
            }
        }
    }
    double* g = gram + run * (stride + 1) * (stride + 1);
    for (int m = 0; m < mine; ++m) {
        const int row = ti[m] * 8 + gid;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int col = tj[m] * 8 + 2 * tig + h;
            const double v = h == 0 ? c0[m] : c1[m];
            if (row < n && col < n) {
                g[static_cast<int64_t>(col) * n + row] = v;
                g[static_cast<int64_t>(row) * n + col] = v;
            }
        }
    }
}

// Batches of at most eight columns: the one-tile sums without the tiled kernel's shared memory and
// registers. A wider batch's narrow runs take the same sums in gram_dmma_kernel.
__global__ void __launch_bounds__(kGramThreads)
gram_one_tile_kernel(const double* __restrict__ J, const double* __restrict__ r, int P_all,
                     int64_t R, double* __restrict__ gram, const int* __restrict__ run_mask,
                     const VarParams* __restrict__ vt, int stride) {
    __shared__ double part[kDmmaWarps * 64];
    const int64_t run = blockIdx.x;
    if (run_mask != nullptr && run_mask[run] == 0) return;
    one_tile_sums(J, r, run, vt != nullptr ? vt[run].P : P_all, stride, R, part, gram);
}

}  // namespace

int launch_gram(const double* J, const double* r, int runs, int P, int64_t R, double* gram,
                bool exact, cudaStream_t stream, const int* run_mask, RunVars rv) {
    if (runs <= 0) return MKB_OK;
    const int stride = rv.table != nullptr ? rv.stride : P;
    if (exact) {
        const int tiles = stride + 1 <= 8 ? 1 : (stride + 1 + 15) / 16;
        const int tile_pairs = tiles * (tiles + 1) / 2;
        const dim3 grid(static_cast<unsigned>(runs), static_cast<unsigned>(tile_pairs));
        const bool few = static_cast<int64_t>(runs) * tile_pairs <= kFewExactCtas;
        auto kernel = stride + 1 <= 8 ? gram_exact_kernel<1, true>
                      : few           ? gram_exact_kernel<2, false>
                                      : gram_exact_kernel<2, true>;
        kernel<<<grid, kExactThreads, 0, stream>>>(J, r, P, R, gram, run_mask, rv.table, stride,
                                                   tile_pairs);
    } else if (stride + 1 <= 8)
        gram_one_tile_kernel<<<runs, kGramThreads, 0, stream>>>(J, r, P, R, gram, run_mask,
                                                                rv.table, stride);
    else
        gram_dmma_kernel<<<runs, kGramThreads, 0, stream>>>(J, r, P, R, gram, run_mask, rv.table,
                                                            stride);
    count_launch();
    return cuda_status(cudaGetLastError(), "normal equations launch");
}

MKB_DEFINE_ERROR_READER(gram_device_error)

}  // namespace mkb

extern "C" int mkb_normal_equations_device(const double* J, const double* r, int32_t runs,
                                           int32_t P, int64_t R, double* gram, int32_t exact,
                                           void* stream) {
    using namespace mkb;
    if (runs < 0 || P < 1 || P > MKB_MAX_VARIABLES || R < 0) {
        set_error("normal equations: runs %d, P %d (1..%d) or R %lld out of range", runs, P,
                  MKB_MAX_VARIABLES, static_cast<long long>(R));
        return MKB_ERR_ARGUMENT;
    }
    if (runs > 0 && (J == nullptr || r == nullptr || gram == nullptr)) {
        set_error("normal equations: null pointer");
        return MKB_ERR_ARGUMENT;
    }
    return launch_gram(J, r, runs, P, R, gram, exact != 0, static_cast<cudaStream_t>(stream));
}
