// Broyden modified-second mixing on the device, with deterministic
// reductions (fixed-shape block trees, fixed-order partial sums).
//
// Reference: Source/Solver/Transport/Broyden_Second_Parallel.cpp:213-486
// (GPU branch; its CPU twin :9-211 defines the same arithmetic) and
// Broyden_Parallel_General.cpp:68-355.  The reference accumulates
// V^T x with one atomic per element (:355-365, :412-422) and finishes the
// norms with atomics (:268-272); here each dot product is one block-level
// tree reduction, so repeated runs are bitwise identical.
//
// Storage: V^T and W as [max_step][S] row-major (row `it` = iteration it),
// so every dot product and row update is a coalesced sweep over sites.

#include <cooperative_groups.h>

#include "negf_internal.h"

namespace negf {
namespace {

constexpr int kThreads = 256;

// Device-resident iterations (BroydenDev::step_dev set): the iteration index
// m = step - 1 is read on the device and `flags` (int[4]: converged,
// iterations, error, skip) makes every kernel of a finished solve return at
// entry, so a captured sequence of iterations needs no host round trip.
__device__ __forceinline__ bool skipped(const int* flags) { return flags && flags[3]; }
__device__ __forceinline__ int iter_m(const BroydenDev& b, int m_host) {
    return b.step_dev ? *b.step_dev - 1 : m_host;
}
// Seeded rows, read on the device so that captured launches see later seeds.
__device__ __forceinline__ int seeded(const BroydenDev& b) { return b.step_dev ? b.step_dev[1] : b.base; }

// max that keeps a NaN (a non-finite residual must not read as converged)
__device__ __forceinline__ double nanmax(double a, double b) { return (a != a || b != b) ? a + b : fmax(a, b); }

// Block reduction of (max, sum, sum) in a fixed order.
__device__ __forceinline__ void block_reduce3(double& a, double& b, double& c) {
    __shared__ double sh[3][kThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        a = nanmax(a, __shfl_xor_sync(0xffffffffu, a, o));
        b += __shfl_xor_sync(0xffffffffu, b, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if (lane == 0) {
        sh[0][wid] = a;
        sh[1][wid] = b;
        sh[2][wid] = c;
    }
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
        a = lane < nw ? sh[0][lane] : 0.0;
        b = lane < nw ? sh[1][lane] : 0.0;
        c = lane < nw ? sh[2][lane] : 0.0;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            a = nanmax(a, __shfl_xor_sync(0xffffffffu, a, o));
            b += __shfl_xor_sync(0xffffffffu, b, o);
            c += __shfl_xor_sync(0xffffffffu, c, o);
        }
    }
}

__device__ __forceinline__ double block_sum(double v) {
    __shared__ double sh[kThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    v = 0.0;
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
        v = lane < nw ? sh[lane] : 0.0;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    return v;
}

// Broyden_Second_Parallel.cpp:243-315: F, |F| (or relative), dF, and the
// three scalars (max norm, sum of squares, dF^T dF) as block partials.
__global__ void norm_kernel(BroydenDev b, const double* __restrict__ n_out, const int* flags) {
    if (skipped(flags)) return;
    double mx = 0.0, s1 = 0.0, s2 = 0.0;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < b.S; s += gridDim.x * blockDim.x) {
        const double nin = b.n_in[s], nout = n_out[s];
        const double Fc = nin - nout;
        double nr, sq;
        if (b.norm_type == 0) {
            nr = fabs(Fc);
            sq = Fc * Fc;
        } else {
            nr = fabs(Fc / (nin + nout));
            sq = nr * nr;
        }
        b.norm[s] = nr;
        const double d = Fc - b.F[s];
        b.dF[s] = d;
        b.F[s] = Fc;
        b.sum[s] = 0.0;
        mx = nanmax(mx, nr);
        s1 += sq;
        s2 += d * d;
    }
    block_reduce3(mx, s1, s2);
    if (threadIdx.x == 0) {
        b.part[3 * blockIdx.x + 0] = mx;
        b.part[3 * blockIdx.x + 1] = s1;
        b.part[3 * blockIdx.x + 2] = s2;
    }
}

__global__ void norm_finalize(BroydenDev b, const int* flags) {
    if (threadIdx.x != 0 || skipped(flags)) return;
    double mx = 0.0, s1 = 0.0, s2 = 0.0;
    for (int i = 0; i < b.nblocks; ++i) {
        mx = nanmax(mx, b.part[3 * i]);
        s1 += b.part[3 * i + 1];
        s2 += b.part[3 * i + 2];
    }
    b.scal[0] = mx;
    b.scal[1] = sqrt(s1);
    b.scal[2] = s2;
}

// c[it] = sum_s V[it][s] x[s] for it = 1..rows (one block per row);
// rows = seeded + m - 1 + which with m from the host or the device (rows
// 1..seeded: a seeded initial inverse Jacobian).  With segments the sum runs
// over each segment's sites separately (blockIdx.y = segment, c[it][g]).
__global__ void dots_kernel(BroydenDev b, const double* __restrict__ x, int m_host, int which, const int* flags) {
    if (skipped(flags)) return;
    const int rows = seeded(b) + iter_m(b, m_host) - 1 + which;
    const int it = blockIdx.x + 1;
    if (it > rows) return;
    const int g = blockIdx.y;
    const int lo = b.nseg > 1 ? b.seg_off[g] : 0, hi = b.nseg > 1 ? b.seg_off[g + 1] : b.S;
    const double* v = b.V + (size_t)it * b.S;
    double acc = 0.0;
    for (int s = lo + threadIdx.x; s < hi; s += blockDim.x) acc += v[s] * x[s];
    acc = block_sum(acc);
    if (threadIdx.x == 0) b.c[(size_t)it * b.nseg + g] = acc;
}

// Per-segment dF^T dF (the denominators of the new V row when segmented).
__global__ void segsq_kernel(BroydenDev b, int m_host, const int* flags) {
    if (skipped(flags) || iter_m(b, m_host) <= 0) return;
    const int g = blockIdx.x;
    double acc = 0.0;
    for (int s = b.seg_off[g] + threadIdx.x; s < b.seg_off[g + 1]; s += blockDim.x) acc += b.dF[s] * b.dF[s];
    acc = block_sum(acc);
    if (threadIdx.x == 0) b.dd[g] = acc;
}

// Broyden_Second_Parallel.cpp:381-403: sum = W c (it < m), new V and W rows at m
// (after the seeded rows).
__global__ void newrow_kernel(BroydenDev b, int m_host, const int* flags) {
    if (skipped(flags)) return;
    const int m = iter_m(b, m_host);
    if (m <= 0) return;
    const int row = seeded(b) + m;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < b.S; s += gridDim.x * blockDim.x) {
        const int g = b.nseg > 1 ? b.seg_of[s] : 0;
        const double denom = b.nseg > 1 ? b.dd[g] : b.scal[2];
        double acc = 0.0;
        for (int it = 1; it <= row - 1; ++it) acc += b.W[(size_t)it * b.S + s] * b.c[(size_t)it * b.nseg + g];
        const double dF = b.dF[s];
        const double dn = b.n_in[s] - b.n_prev[s];
        // a zero step (identical consecutive residuals) adds no direction: the
        // reference would divide by zero here
        b.V[(size_t)row * b.S + s] = denom > 0.0 ? dF / denom : 0.0;
        b.W[(size_t)row * b.S + s] = -b.fraction * dF + dn - acc;
    }
}

// Broyden_Second_Parallel.cpp:455-481: sum = W c (it <= m, after the seeded
// rows), then the new input.
__global__ void final_kernel(BroydenDev b, int m_host, const int* flags) {
    if (skipped(flags)) return;
    const int rows = seeded(b) + iter_m(b, m_host);
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < b.S; s += gridDim.x * blockDim.x) {
        const int g = b.nseg > 1 ? b.seg_of[s] : 0;
        double acc = 0.0;
        for (int it = 1; it <= rows; ++it) acc += b.W[(size_t)it * b.S + s] * b.c[(size_t)it * b.nseg + g];
        b.sum[s] = acc;
        const double prev = b.n_in[s];
        b.n_prev[s] = prev;
        b.n_in[s] = prev - b.scalar * b.fraction * b.F[s] - b.scalar * acc;
    }
}

// End of a device-resident step: the loop predicate of Transport.cpp:385-505
// (stop when the norm is not above max_norm), the step count, and the
// MaxStep abort of :389-393 as an error flag for the host.
// switch_norm > 0 (precision switching, flags int[8]): until flags[4] is set
// the charge came from the low-precision plan; the first norm below
// switch_norm sets flags[4] and later steps use the FP64 plan, and only an
// FP64 charge can end the solve.  flags[5] / flags[6] are the skip words of
// the low-precision and FP64 plans; flags[7] counts low-precision steps.
__device__ __forceinline__ void end_step(const BroydenDev& b, double nrm, double max_norm, double switch_norm,
                                         int* flags) {
    flags[1] += 1;
    const int step = *b.step_dev + 1;
    *b.step_dev = step;
    const int limit = b.max_step - seeded(b);  // seeded rows take history capacity
    const bool fp64_charge = !(switch_norm > 0) || flags[4];
    if (!fp64_charge) flags[7] += 1;  // steps on a low-precision charge
    if (!isfinite(nrm))
        flags[2] = 2;
    else if (fp64_charge && !(nrm > max_norm))
        flags[0] = 1;
    else if (step > limit)
        flags[2] = 1;
    flags[3] = (flags[0] || flags[2]) ? 1 : 0;
    if (switch_norm > 0) {
        if (!flags[4] && nrm < switch_norm) flags[4] = 1;
        flags[5] = (flags[3] || flags[4]) ? 1 : 0;
        flags[6] = (flags[3] || !flags[4]) ? 1 : 0;
    }
}

__global__ void step_kernel(BroydenDev b, double max_norm, double switch_norm, int* flags) {
    if (flags[3]) return;
    end_step(b, b.scal[0], max_norm, switch_norm, flags);
}

// A whole step of one segment in one launch (flags null: iteration m_host of a
// step that the host ends): a cluster of 8 blocks, block r holding sites [r chunk,
// (r + 1) chunk).  The dot products of the rows with dF and with F are formed in
// one pass over V (those of the new row dF / |dF|^2 with F from dF . F), the
// partial sums are added over the cluster in rank order, and one pass over W gives
// the new row and the new input.  The seven kernels of the general path (norm,
// finish, dots, row, dots, input, step) are bound by their launches and by chains
// of one block each; a cluster moves V and W at 8 SMs' rate.  us a step, general /
// here, at 30 rows: 2800 sites 35 / 13, 16384 sites 63 / 25, 65536 sites 163 / 74;
// at 60 rows 38 / 15, 69 / 36, 172 / 171; 12000 sites at 100, 200 and 500 rows 66 /
// 49, 78 / 80, 149 / 287, 4000 sites at 500 and 1000 rows 102 / 82, 166 / 177: the
// general path beyond kMixSites sites or kMixWork sites x rows, which a long history
// reaches.
constexpr int kMixBlocks = 8, kMixThreads = 512, kMixSites = 16384;
constexpr long long kMixWork = 200LL * kMixSites;
namespace cg = cooperative_groups;
__global__ void __cluster_dims__(kMixBlocks, 1, 1) __launch_bounds__(kMixThreads)
    mix_kernel(BroydenDev b, const double* __restrict__ n_out, double max_norm, double switch_norm, int* flags,
               int m_host, int chunk) {
    if (skipped(flags)) return;  // written by rank 0 after the last read of every block (cluster.sync)
    extern __shared__ double sh[];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int m = flags ? *b.step_dev - 1 : m_host, row = (flags ? b.step_dev[1] : b.base) + m;
    const int R = m > 0 ? row - 1 : row;  // rows in hand
    double* const mine = sh;              // max, sum of squares, dF.dF, dF.F, then V.dF, V.F per row
    double* const tot = mine + 4 + 2 * b.max_step;
    double* const Fs = tot + 4 + 2 * b.max_step;
    double* const dFs = Fs + chunk;
    const int lo = min(rank * chunk, b.S), n = min(chunk, b.S - lo);
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (int i = t; i < n; i += kMixThreads) {
        const int s = lo + i;
        const double nin = b.n_in[s], nout = n_out[s];
        const double Fc = nin - nout;
        double nr, sq;
        if (b.norm_type == 0) {
            nr = fabs(Fc);
            sq = Fc * Fc;
        } else {
            nr = fabs(Fc / (nin + nout));
            sq = nr * nr;
        }
        const double d = Fc - b.F[s];
        b.norm[s] = nr;
        b.dF[s] = d;
        b.F[s] = Fc;
        Fs[i] = Fc;
        dFs[i] = d;
        v[0] = nanmax(v[0], nr);
        v[1] += sq;
        v[2] += d * d;
        v[3] += d * Fc;
    }
    __shared__ double red[4][kMixThreads / 32];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        v[0] = nanmax(v[0], __shfl_xor_sync(0xffffffffu, v[0], o));
#pragma unroll
        for (int k = 1; k < 4; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    }
    if (lane == 0)
        for (int k = 0; k < 4; ++k) red[k][wid] = v[k];
    __syncthreads();  // F, dF and the warps' sums
    if (t < 4) {
        double a = red[t][0];
        for (int w = 1; w < kMixThreads / 32; ++w) a = t ? a + red[t][w] : nanmax(a, red[t][w]);
        mine[t] = a;
    }
    for (int it = 1 + wid; it <= R; it += kMixThreads / 32) {
        const double* __restrict__ V = b.V + (size_t)it * b.S + lo;
        double a1 = 0.0, a2 = 0.0;
#pragma unroll 4
        for (int i = lane; i < n; i += 32) {
            const double x = V[i];
            a1 += x * dFs[i];
            a2 += x * Fs[i];
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            a1 += __shfl_xor_sync(0xffffffffu, a1, o);
            a2 += __shfl_xor_sync(0xffffffffu, a2, o);
        }
        if (lane == 0) {
            mine[2 + 2 * it] = a1;
            mine[3 + 2 * it] = a2;
        }
    }
    cluster.sync();
    for (int i = t; i < 4 + 2 * R; i += kMixThreads) {
        double a = *cluster.map_shared_rank(mine + i, 0);
        for (int r = 1; r < kMixBlocks; ++r) {
            const double x = *cluster.map_shared_rank(mine + i, r);
            a = i ? a + x : nanmax(a, x);
        }
        tot[i] = a;
    }
    __syncthreads();
    const double denom = tot[2], cn = denom > 0.0 ? tot[3] / denom : 0.0;
    for (int i = t; i < n; i += kMixThreads) {
        const int s = lo + i;
        const double* __restrict__ W = b.W + s;
        double a1 = 0.0, a2 = 0.0;
#pragma unroll 8
        for (int it = 1; it <= R; ++it) {
            const double x = W[(size_t)it * b.S];
            a1 += x * tot[2 + 2 * it];
            a2 += x * tot[3 + 2 * it];
        }
        const double nin = b.n_in[s];
        if (m > 0) {
            const double dF = dFs[i];
            // a zero step adds no direction (newrow_kernel)
            const double w = -b.fraction * dF + (nin - b.n_prev[s]) - a1;
            b.V[(size_t)row * b.S + s] = denom > 0.0 ? dF / denom : 0.0;
            b.W[(size_t)row * b.S + s] = w;
            a2 += w * cn;
        }
        b.sum[s] = a2;
        b.n_prev[s] = nin;
        b.n_in[s] = nin - b.scalar * b.fraction * Fs[i] - b.scalar * a2;
    }
    if (rank == 0) {
        for (int it = 1 + t; it <= row; it += kMixThreads) b.c[it] = it <= R ? tot[3 + 2 * it] : cn;
        if (t == 0) {
            b.scal[0] = tot[0];
            b.scal[1] = sqrt(tot[1]);
            b.scal[2] = tot[2];
            if (flags) end_step(b, tot[0], max_norm, switch_norm, flags);
        }
    }
    cluster.sync();  // no block leaves while its sums are read
}

__global__ void set_int_kernel(int* p, int v) { *p = v; }

__global__ void set_kernel(double* p, double v, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = v;
}

// U[i] = U0[i] + sum_j K[i][j] Q[j]: one warp per row, fixed-order lane tree.
__global__ void affine_kernel(const double* __restrict__ K, const double* __restrict__ U0,
                              const double* __restrict__ Q, double* __restrict__ U, int n, const int* skip) {
    if (skip && *skip) return;
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= n) return;
    const double* k = K + (size_t)row * n;
    double acc = 0.0;
    for (int j = lane; j < n; j += 32) acc += k[j] * Q[j];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) U[row] = U0[row] + acc;
}

// U[i] = U0[i] + sum_j tab[|idx[i] - idx[j]|] Q[j]: the same operator for a
// kernel that depends on the lattice distance only (a ring lattice: zigzag
// tubes), read from a table instead of an n x n matrix.  One warp per row;
// the block stages idx and Q in shared memory in chunks of 1024 sites, and
// consecutive sites give consecutive table entries (coalesced gathers).
constexpr int kToeChunk = 1024;
__global__ void __launch_bounds__(256) toeplitz_kernel(const double* __restrict__ tab, int ntab,
                                                       const int* __restrict__ idx, const double* __restrict__ U0,
                                                       const double* __restrict__ Q, double* __restrict__ U, int n,
                                                       const int* skip) {
    if (skip && *skip) return;
    __shared__ double sq[kToeChunk];
    __shared__ int si[kToeChunk];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int row = blockIdx.x * (blockDim.x >> 5) + wib;
    const int ir = row < n ? idx[row] : 0;
    double acc = 0.0;
    for (int c0 = 0; c0 < n; c0 += kToeChunk) {
        const int cn = min(kToeChunk, n - c0);
        __syncthreads();
        for (int t = threadIdx.x; t < cn; t += blockDim.x) {
            sq[t] = Q[c0 + t];
            si[t] = idx[c0 + t];
        }
        __syncthreads();
        if (row < n) {
            for (int t = lane; t < cn; t += 32) {
                int d = ir - si[t];
                d = d < 0 ? -d : d;
                acc = fma(d < ntab ? __ldg(tab + d) : 0.0, sq[t], acc);
            }
        }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (row < n && lane == 0) U[row] = U0[row] + acc;
}

// Batched form: every row of every tube in one launch.  Block b covers rows
// [first, first + 8) of tube tube_of[b] (blocks never straddle tubes), so the
// tubes' potentials are formed concurrently instead of one launch each.
__global__ void __launch_bounds__(256) toeplitz_batch_kernel(const ToeplitzOp* __restrict__ ops,
                                                             const int2* __restrict__ blocks, const int* skip) {
    if (skip && *skip) return;
    __shared__ double sq[kToeChunk];
    __shared__ int si[kToeChunk];
    const int2 bt = blocks[blockIdx.x];  // (tube, first row)
    const ToeplitzOp op = ops[bt.x];
    const int n = op.n;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int row = bt.y + wib;
    const int ir = row < n ? op.idx[row] : 0;
    double acc = 0.0;
    for (int c0 = 0; c0 < n; c0 += kToeChunk) {
        const int cn = min(kToeChunk, n - c0);
        __syncthreads();
        for (int t = threadIdx.x; t < cn; t += blockDim.x) {
            sq[t] = op.Q[c0 + t];
            si[t] = op.idx[c0 + t];
        }
        __syncthreads();
        if (row < n) {
            for (int t = lane; t < cn; t += 32) {
                int d = ir - si[t];
                d = d < 0 ? -d : d;
                acc = fma(d < op.ntab ? __ldg(op.tab + d) : 0.0, sq[t], acc);
            }
        }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (row < n && lane == 0) op.U[row] = op.U0[row] + acc;
}

}  // namespace

cudaError_t affine_toeplitz_batch(const ToeplitzOp* d_ops, const int2* d_blocks, int num_blocks, cudaStream_t s,
                                  const int* skip) {
    if (num_blocks <= 0) return cudaSuccess;
    toeplitz_batch_kernel<<<num_blocks, 256, 0, s>>>(d_ops, d_blocks, skip);
    return cudaGetLastError();
}

cudaError_t affine_toeplitz(const double* tab, int ntab, const int* idx, const double* U0, const double* Q, double* U,
                            int n, cudaStream_t s, const int* skip) {
    if (n <= 0) return cudaSuccess;
    toeplitz_kernel<<<(n + 7) / 8, 256, 0, s>>>(tab, ntab, idx, U0, Q, U, n, skip);
    return cudaGetLastError();
}

namespace {
// One cluster while it is the faster form (see mix_kernel) and the rows' sums fit its shared memory; rows: the
// most that the launch may find.
constexpr int kMixShared = 200 * 1024;
bool mix_fits(const BroydenDev& b, int rows, int& chunk, size_t& smem) {
    chunk = (b.S + kMixBlocks - 1) / kMixBlocks;
    smem = sizeof(double) * (2 * (4 + 2 * (size_t)b.max_step) + 2 * (size_t)chunk);
    return b.nseg == 1 && b.S <= kMixSites && (long long)b.S * rows <= kMixWork && smem <= kMixShared;
}
cudaError_t mix(const BroydenDev& b, const double* n_out, double max_norm, double switch_norm, int* flags, int m_host,
                int chunk, size_t smem, cudaStream_t s) {
    // the limit belongs to the kernel, not to the launch: the same for every mixer, since other threads launch theirs
    const cudaError_t e = cudaFuncSetAttribute(mix_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMixShared);
    if (e != cudaSuccess) return e;
    mix_kernel<<<kMixBlocks, kMixThreads, smem, s>>>(b, n_out, max_norm, switch_norm, flags, m_host, chunk);
    return cudaGetLastError();
}
void norm(const BroydenDev& b, const double* n_out, const int* flags, cudaStream_t s) {
    norm_kernel<<<b.nblocks, kThreads, 0, s>>>(b, n_out, flags);
    norm_finalize<<<1, 32, 0, s>>>(b, flags);
}
}  // namespace

cudaError_t broyden_step(const BroydenDev& b, const double* n_out, int m, cudaStream_t s) {
    int chunk;
    size_t smem;
    if (mix_fits(b, b.base + m, chunk, smem)) return mix(b, n_out, 0.0, 0.0, nullptr, m, chunk, smem, s);
    norm(b, n_out, nullptr, s);
    if (m > 0) {
        if (b.base + m - 1 >= 1) dots_kernel<<<dim3(b.base + m - 1, b.nseg), kThreads, 0, s>>>(b, b.dF, m, 0, nullptr);
        if (b.nseg > 1) segsq_kernel<<<b.nseg, kThreads, 0, s>>>(b, m, nullptr);
        newrow_kernel<<<b.nblocks, kThreads, 0, s>>>(b, m, nullptr);
    }
    if (b.base + m >= 1) dots_kernel<<<dim3(b.base + m, b.nseg), kThreads, 0, s>>>(b, b.F, m, 1, nullptr);
    final_kernel<<<b.nblocks, kThreads, 0, s>>>(b, m, nullptr);
    return cudaGetLastError();
}

cudaError_t broyden_step_device(const BroydenDev& b, const double* n_out, double max_norm, double switch_norm, int* flags,
                                cudaStream_t s) {
    int chunk;
    size_t smem;
    if (mix_fits(b, b.max_step, chunk, smem)) return mix(b, n_out, max_norm, switch_norm, flags, 0, chunk, smem, s);
    norm(b, n_out, flags, s);
    // shapes cover every m up to max_step, rows above m return
    const dim3 g(b.max_step > 1 ? b.max_step : 1, b.nseg);
    dots_kernel<<<g, kThreads, 0, s>>>(b, b.dF, 0, 0, flags);
    if (b.nseg > 1) segsq_kernel<<<b.nseg, kThreads, 0, s>>>(b, 0, flags);
    newrow_kernel<<<b.nblocks, kThreads, 0, s>>>(b, 0, flags);
    dots_kernel<<<g, kThreads, 0, s>>>(b, b.F, 0, 1, flags);
    final_kernel<<<b.nblocks, kThreads, 0, s>>>(b, 0, flags);
    step_kernel<<<1, 1, 0, s>>>(b, max_norm, switch_norm, flags);
    return cudaGetLastError();
}

cudaError_t set_int(int* p, int v, cudaStream_t s) {
    set_int_kernel<<<1, 1, 0, s>>>(p, v);
    return cudaGetLastError();
}

cudaError_t broyden_set(double* p, double v, int n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int blocks = (n + kThreads - 1) / kThreads;
    set_kernel<<<blocks < 1024 ? blocks : 1024, kThreads, 0, s>>>(p, v, n);
    return cudaGetLastError();
}

cudaError_t affine_potential(const double* K, const double* U0, const double* Q, double* U, int n, cudaStream_t s,
                             const int* skip) {
    if (n <= 0) return cudaSuccess;
    const int warps_per_block = 8;
    affine_kernel<<<(n + warps_per_block - 1) / warps_per_block, 32 * warps_per_block, 0, s>>>(K, U0, Q, U, n, skip);
    return cudaGetLastError();
}

}  // namespace negf
