// Real-space ring-block RGF of a zigzag (m,0) tube (FP64, or mixed FP32/FP64).
//
// Blocks of two rings (2m atoms, m <= 16): ring a = 2k and ring b = 2k+1 are
// joined by the double bond (atom j of a to atoms j and j+1 mod m of b:
// E - H has -gamma C with C[j][j] = C[j][j+1] = 1), ring b of block k and
// ring a of block k+1 by the single bond (atom j to atom j, -gamma I).  In
// mode space these are beta_J = 2 gamma cos(pi J/m) and gamma
// (CNT.cpp:288-336), so a ring-uniform potential reproduces the sum of the m
// mode chains.  The dense 2m x 2m block is
//     M_k = [[A, -gamma C], [-gamma C^T, D]],
// A = diag(E - U_a) - Sigma_a, D = diag(E - U_b) - Sigma_b, where the
// self-energies of the neighbours touch one ring each.  The block algebra
// works on m x m ring corners with Schur complements instead of 2m x 2m
// inversions:
//   forward  (Sigma_b = 0, D diagonal): X_k = g_L[a][a] = S^-1 with
//            S = A - gamma^2 C D^-1 C^T (C D^-1 C^T has three diagonals);
//            g_L[b][b] = D^-1 + gamma^2 Y^T X Y and g_L[a][b] = gamma X Y,
//            Y = C D^-1, follow from X with O(m^2) work; X_k is kept.
//   backward G_kk = g_L + gamma^2 g_L[:, b] G_{k+1}[a][a] g_L[b, :] gives
//            G[a][a] = X + gamma^4 X (Y G' Y^T) X  and
//            tr G[b][b] = tr g_L[b][b] + gamma^2 tr(g_L[b][b] G' g_L[b][b])
//            with G' = G_{k+1}[a][a]: three m x m products per block (two in
//            FP64, see rs_side).  The right lead enters through G_K[a][a] =
//            (I - gamma^2 s_R g_L[b][b])^-1 s_R of its first ring.
// One block update costs one m x m inversion and two or three m x m products
// instead of three 2m x 2m inversions (about 10x fewer operations).
//
// Leads: a lead is uniform (the contact potential on every atom), so the
// ring Fourier modes decouple it into the mode chains of the mode-space pass;
// the ring corner of its surface Green's function is the circulant of the
// per-mode surface values (rs_lead_kernel).

// Kernels (m x m complex tiles in shared memory, row-major; m x m products on
// the FP64 tensor cores, mma.sync m8n8k4, with the results staged in registers
// so that outputs may alias inputs):
//   rs_lead_kernel   both lead corners s_L = g[b][b], s_R = g[a][a] (ring
//                    Fourier modes, per-mode surface values);
//   rs_pair_kernel   an energy's FP64 chain by two warps from its two ends:
//                    forward sweeps (X_k to global scratch), backward sweeps with
//                    the ring sums of c G_jj written per energy; at a real-axis
//                    energy of a biased tube the sweeps carry the source and
//                    drain columns of G in ring corners: ring sums of the contact
//                    spectral functions (the non-equilibrium term);
//   rs_chain_kernel  an energy's FP32 chain of mixed mode, a warp and a helper;
//   rs_reduce_kernel sum over energies per ring in a fixed order (Kahan).
// The U = 0 pass (Rho0) and, in FP64, ring-uniform potentials do not come
// here: the ring's Fourier modes decouple them (ring_modes_charge in
// negf_api.cpp).
// Inversions: FP64 blocks by symmetric sweeps on 2 x 2 pivots, the others by
// Gauss-Jordan on [S | I] (lane = column); on the diagonal pivots with a
// fall-back to partial pivoting when a pivot is small.
//
// Mixed precision: the chain of an energy runs in FP32 when its tube is in
// mixed mode and the point lies at least mixed_fp64_band above the real axis
// (the rule of the mode-space pass); the leads, the other energies, the ring
// sums per energy and their Kahan sum stay FP64.  In FP32 the m x m
// products run on the tensor cores: mma.sync m16n8k8 TF32 with each operand
// split into a TF32 high part and a TF32 remainder (three products per
// pair, about FP32 accuracy) and the complex product in the three-multiply
// form Re = ArBr - AiBi, Im = (Ar + Ai)(Br + Bi) - ArBr - AiBi; the
// inversion runs on the FP32 cores.  The FP32 chains run beside the FP64 ones,
// on a side stream.

#include "negf_internal.h"

namespace negf {
namespace {

constexpr int kMaxM = 16;  // atoms per ring: [S | I] has one lane per column

#include "negf_sgf.cuh"  // cd, sgf_analytic, sgf_decimation (lead mode chains)

template <typename R>
struct __align__(2 * sizeof(R)) cplx {
    R x, y;
};
using cplxd = cplx<double>;
using cplxf = cplx<float>;
template <typename R>
__device__ __forceinline__ cplx<R> cmk(R a, R b) {
    return {a, b};
}
template <typename R>
__device__ __forceinline__ cplx<R> cadd(cplx<R> a, cplx<R> b) {
    return {a.x + b.x, a.y + b.y};
}
template <typename R>
__device__ __forceinline__ cplx<R> csub(cplx<R> a, cplx<R> b) {
    return {a.x - b.x, a.y - b.y};
}
template <typename R>
__device__ __forceinline__ cplx<R> cscale(cplx<R> a, R s) {
    return {a.x * s, a.y * s};
}
template <typename R>
__device__ __forceinline__ cplx<R> cmul(cplx<R> a, cplx<R> b) {
    return {fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x)};
}
// acc + a b
template <typename R>
__device__ __forceinline__ cplx<R> cfma(cplx<R> a, cplx<R> b, cplx<R> acc) {
    return {fma(a.x, b.x, fma(-a.y, b.y, acc.x)), fma(a.x, b.y, fma(a.y, b.x, acc.y))};
}
// acc - a b
template <typename R>
__device__ __forceinline__ cplx<R> cfms(cplx<R> a, cplx<R> b, cplx<R> acc) {
    return {fma(-a.x, b.x, fma(a.y, b.y, acc.x)), fma(-a.x, b.y, fma(-a.y, b.x, acc.y))};
}
// Reciprocal: hardware approximation y0 = rcp.approx.ftz(x) with relative
// error e = 1 - x y0 (|e| <= 2^-20 or better), corrected by the truncated
// series 1/x = y0 (1 + e + e^2 + ...) to a relative error of order e^3 (FP64)
// or e^2 (FP32).  Arguments are squared moduli of pivots and of E - U.
__device__ __forceinline__ double rcp_r(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ float rcp_r(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return fmaf(y, fmaf(-x, y, 1.0f), y);
}
// 1 / b = conj(b) / |b|^2
template <typename R>
__device__ __forceinline__ cplx<R> crcp(cplx<R> b) {
    const R q = rcp_r(fma(b.x, b.x, b.y * b.y));
    return {b.x * q, -b.y * q};
}

// Complex tile, row-major with compile-time leading dimension LD
template <int LD, typename R>
struct Mat {
    cplx<R>* a;
    __device__ __forceinline__ cplx<R>& at(int r, int c) const { return a[r * LD + c]; }
};

template <int M>
__device__ __forceinline__ int wrap(int i) { return i < 0 ? i + M : (i >= M ? i - M : i); }

// FP64 tensor-core product D += A B of an 8 x 8 x 4 tile (mma.sync m8n8k4,
// FP64).  Fragments, g = lane / 4, t = lane % 4: a = A[g][t]; b = B[t][g];
// d = D[g][2t], D[g][2t+1].
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

// op(A) op(B) of m x m tiles in FP64 on the tensor cores: w = val(r, c, v) of all
// entries v, then put(r, c, w, off) of those inside the tile, by the lanes that
// hold them (loads belong into val: behind a store of put they would wait for
// it).  2 x 2 output tiles of 8 x 8 (rows and columns past m are clamped
// duplicates), k in steps
// of 4, complex products in the three-multiply form Re = ArBr - AiBi, Im = (Ar +
// Ai)(Br + Bi) - ArBr - AiBi.  One or two indices left over by the steps of 4
// are rank-one updates on the FP64 cores: 60 issue cycles each at 2 x 2 tiles
// where a padded step takes 192 (an m8n8k4 runs 16 cycles: the tensor cores
// have the FP64 cores' rate here).  SYM: the product is symmetric, and the tile
// above the diagonal is left out: the entries of tile (1, 0) come with off =
// true and stand for (c, r) too.  put may overwrite A and B.
template <int m, bool TA, bool TB, bool SYM, class F, class P>
__device__ __forceinline__ void mm_each(Mat<m, double> A, Mat<m, double> B, int lane, F&& val, P&& put) {
    const int g = lane >> 2, t = lane & 3;
    constexpr int NT = (m + 7) / 8;  // 8 x 8 output tiles per dimension
    constexpr int KD = m % 4 == 3 ? m + 1 : m - (m % 4 <= 2 ? m % 4 : 0);
    double p1[NT][NT][2], p2[NT][NT][2], p3[NT][NT][2];  // Ar Br, Ai Bi, (Ar + Ai)(Br + Bi)
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int q = 0; q < 2; ++q) p1[i][j][q] = p2[i][j][q] = p3[i][j][q] = 0.0;
#pragma unroll
    for (int k0 = 0; k0 < KD; k0 += 4) {
        const int k = min(k0 + t, m - 1);
        cplxd a[NT], b[NT];
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int r = min(8 * i + g, m - 1);
            a[i] = TA ? A.at(k, r) : A.at(r, k);
            b[i] = TB ? B.at(r, k) : B.at(k, r);  // column 8 i + g of B
            if (k0 + 4 > m && k0 + t >= m) a[i] = b[i] = cmk(0.0, 0.0);
        }
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const double as = a[i].x + a[i].y;
#pragma unroll
            for (int j = 0; j < (SYM ? i + 1 : NT); ++j) {
                dmma(p1[i][j], a[i].x, b[j].x);
                dmma(p2[i][j], a[i].y, b[j].y);
                dmma(p3[i][j], as, b[j].x + b[j].y);
            }
        }
    }
#pragma unroll
    for (int k = KD; k < m; ++k) {
        cplxd a[NT], b[NT][2];
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int r = min(8 * i + g, m - 1);
            a[i] = TA ? A.at(k, r) : A.at(r, k);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int c = min(8 * i + 2 * t + q, m - 1);
                b[i][q] = TB ? B.at(c, k) : B.at(k, c);
            }
        }
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const double as = a[i].x + a[i].y;
#pragma unroll
            for (int j = 0; j < (SYM ? i + 1 : NT); ++j)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    p1[i][j][q] = fma(a[i].x, b[j][q].x, p1[i][j][q]);
                    p2[i][j][q] = fma(a[i].y, b[j][q].y, p2[i][j][q]);
                    p3[i][j][q] = fma(as, b[j][q].x + b[j][q].y, p3[i][j][q]);
                }
        }
    }
    __syncwarp();
    cplxd w[NT][NT][2];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < (SYM ? i + 1 : NT); ++j)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const double re = p1[i][j][q] - p2[i][j][q], im = p3[i][j][q] - p1[i][j][q] - p2[i][j][q];
                w[i][j][q] = val(min(8 * i + g, m - 1), min(8 * j + 2 * t + q, m - 1), cmk(re, im));
            }
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < (SYM ? i + 1 : NT); ++j)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int r = 8 * i + g, c = 8 * j + 2 * t + q;
                if (r < m && c < m) put(r, c, w[i][j][q], SYM && i != j);
            }
    __syncwarp();
}

// C = s op(A) op(B) (+ D when ADD); C may alias any operand.
template <int m, bool TA, bool TB, bool ADD>
__device__ __forceinline__ void mm(Mat<m, double> C, Mat<m, double> A, Mat<m, double> B, Mat<m, double> D, double s,
                                   int lane) {
    mm_each<m, TA, TB, false>(
        A, B, lane,
        [&](int r, int c, cplxd v) {
            v = cscale(v, s);
            return ADD ? cadd(v, D.at(r, c)) : v;
        },
        [&](int r, int c, cplxd v, bool) { C.at(r, c) = v; });
}

// TF32 tensor-core product D += A B of a 16 x 8 x 8 tile (mma.sync
// m16n8k8, FP32 accumulate).  Fragments, g = lane / 4, t = lane % 4:
// a = A[g][t], A[g+8][t], A[g][t+4], A[g+8][t+4]; b = B[t][g], B[t+4][g];
// d = D[g][2t], D[g][2t+1], D[g+8][2t], D[g+8][2t+1].
__device__ __forceinline__ void mma_tf32(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// x = hi + lo with hi the TF32 rounding of x and lo the TF32 rounding of the rest
__device__ __forceinline__ void split_tf32(float x, unsigned& hi, unsigned& lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    const float rest = x - __uint_as_float(hi);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(rest));
}
// D += A B in three tensor-core products: lo hi + hi lo + hi hi
__device__ __forceinline__ void mma3(float (&d)[4], const unsigned (&ah)[4], const unsigned (&al)[4],
                                     const unsigned (&bh)[2], const unsigned (&bl)[2]) {
    mma_tf32(d, al, bh);
    mma_tf32(d, ah, bl);
    mma_tf32(d, ah, bh);
}

// s op(A) op(B) of m x m tiles in FP32 on the tensor cores, with val and put as
// above: the tiles are read as zero-padded 16 x 16 operands, the complex product
// in the three-multiply form.
template <int m, bool TA, bool TB, class F, class P>
__device__ __forceinline__ void mm_each(Mat<m, float> A, Mat<m, float> B, float s, int lane, F&& val, P&& put) {
    const int g = lane >> 2, t = lane & 3;
    float t1[2][4], t2[2][4], t3[2][4];  // Ar Br, Ai Bi, (Ar + Ai)(Br + Bi) per 8-column tile
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) t1[n][q] = t2[n][q] = t3[n][q] = 0.0f;
#pragma unroll
    for (int k0 = 0; k0 < m; k0 += 8) {
        unsigned arh[4], arl[4], aih[4], ail[4], ash[4], asl[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = g + ((q & 1) ? 8 : 0), k = k0 + t + ((q & 2) ? 4 : 0);
            cplxf v = cmk(0.0f, 0.0f);
            if (r < m && k < m) v = TA ? A.at(k, r) : A.at(r, k);
            split_tf32(v.x, arh[q], arl[q]);
            split_tf32(v.y, aih[q], ail[q]);
            split_tf32(v.x + v.y, ash[q], asl[q]);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            if (8 * n < m) {
                unsigned brh[2], brl[2], bih[2], bil[2], bsh[2], bsl[2];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int k = k0 + t + 4 * q, c = 8 * n + g;
                    cplxf v = cmk(0.0f, 0.0f);
                    if (k < m && c < m) v = TB ? B.at(c, k) : B.at(k, c);
                    split_tf32(v.x, brh[q], brl[q]);
                    split_tf32(v.y, bih[q], bil[q]);
                    split_tf32(v.x + v.y, bsh[q], bsl[q]);
                }
                mma3(t1[n], arh, arl, brh, brl);
                mma3(t2[n], aih, ail, bih, bil);
                mma3(t3[n], ash, asl, bsh, bsl);
            }
        }
    }
    __syncwarp();
    cplxf w[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q)
            w[n][q] = val(min(g + ((q & 2) ? 8 : 0), m - 1), min(8 * n + 2 * t + (q & 1), m - 1),
                          cmk((t1[n][q] - t2[n][q]) * s, (t3[n][q] - t1[n][q] - t2[n][q]) * s));
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = g + ((q & 2) ? 8 : 0), c = 8 * n + 2 * t + (q & 1);
            if (r < m && c < m) put(r, c, w[n][q]);
        }
    __syncwarp();
}

// C = s op(A) op(B) (+ D when ADD); C may alias any operand.
template <int m, bool TA, bool TB, bool ADD>
__device__ __forceinline__ void mm(Mat<m, float> C, Mat<m, float> A, Mat<m, float> B, Mat<m, float> D, float s,
                                   int lane) {
    mm_each<m, TA, TB>(
        A, B, s, lane, [&](int r, int c, cplxf v) { return ADD ? cadd(v, D.at(r, c)) : v; },
        [&](int r, int c, cplxf v) { C.at(r, c) = v; });
}

// max(|Re|, |Im|)
template <typename R>
__device__ __forceinline__ R cmaxabs(cplx<R> a) {
    return fmax(fabs(a.x), fabs(a.y));
}

// out = S^-1 by Gauss-Jordan with partial pivoting (largest |.|^2 over the
// rows below, lowest row on ties).  Lane c < 2m holds column c of [S | I] in
// registers; the pivot column reaches every lane through buf (m complex in
// shared memory), every lane finds the pivot row by a tournament over it.
// out may alias S.  Returns false on a zero pivot.
template <int m, typename R>
__device__ __noinline__ bool invert_pivoted(Mat<m, R> out, Mat<m, R> S, cplx<R>* buf, int lane) {
    constexpr int n2 = 2 * m;
    __syncwarp();  // S complete
    cplx<R> col[m];
#pragma unroll
    for (int r = 0; r < m; ++r) col[r] = lane < m ? S.at(r, lane) : cmk<R>(lane - m == r ? R(1) : R(0), R(0));
    bool ok = true;
#pragma unroll
    for (int p = 0; p < m; ++p) {
        __syncwarp();  // every lane is done with buf (and with S on the first pivot)
        if (lane == p) {
#pragma unroll
            for (int r = 0; r < m; ++r) buf[r] = col[r];
        }
        __syncwarp();
        R bv[m];
        int bi[m];
#pragma unroll
        for (int r = 0; r < m; ++r) {
            bi[r] = r;
            bv[r] = R(-1);
            if (r >= p) {
                const cplx<R> x = buf[r];
                bv[r] = fma(x.x, x.x, x.y * x.y);
            }
        }
#pragma unroll
        for (int st = 1; st < m; st *= 2) {
#pragma unroll
            for (int r = 0; r + st < m; r += 2 * st) {
                if (bv[r + st] > bv[r]) {
                    bv[r] = bv[r + st];
                    bi[r] = bi[r + st];
                }
            }
        }
        const int idx = bi[0];
        if (!(bv[0] > R(0))) ok = false;
        if (idx != p) {
#pragma unroll
            for (int r = p + 1; r < m; ++r) {
                if (r == idx) {
                    const cplx<R> t = col[r];
                    col[r] = col[p];
                    col[p] = t;
                }
            }
        }
        // multiplier of row r after the swap: buf[r], but buf[p] for row idx
        const cplx<R> rp = cmul(col[p], crcp(buf[idx]));
#pragma unroll
        for (int r = 0; r < m; ++r) {
            if (r == 8) asm volatile("" ::: "memory");  // two batches of multiplier loads
            if (r != p) col[r] = cfms(buf[r == idx ? p : r], rp, col[r]);
        }
        col[p] = rp;
    }
    __syncwarp();
    if (lane >= m && lane < n2) {
#pragma unroll
        for (int r = 0; r < m; ++r) out.at(r, lane - m) = col[r];
    }
    __syncwarp();
    return ok;
}

// out = S^-1 by Gauss-Jordan on the diagonal pivots, falling back to partial
// pivoting (invert_pivoted, from S, which stays untouched until the result
// is written) when any pivot is small: max(|Re|, |Im|) of a pivot below tau
// (1e-3 in FP64, 1e-2 in FP32) times the largest such value of the entries
// of S.  For E - H - Sigma with Im E > 0, S is complex symmetric with a
// positive definite imaginary part, so its leading minors never vanish and
// the diagonal pivots are the usual case; the search and the row swaps of
// partial pivoting (about half the cost of the inversion) leave the common
// path.  Lane c < 2m holds column c of [S | I] in registers, the pivot
// column and its pivot's reciprocal (formed by the pivot's lane beside the rest
// of the previous step) reach every lane through buf (kMaxM + 2 complex, 16-byte
// aligned).  out may alias S.  Returns false on
// a zero pivot.
template <int m, typename R>
__device__ __forceinline__ bool invert(Mat<m, R> out, Mat<m, R> S, cplx<R>* buf, int lane) {
    constexpr int n2 = 2 * m;
    const R tau = sizeof(R) == 8 ? R(1e-3) : R(1e-2);
    __syncwarp();  // S complete
    cplx<R> col[m];
    R smax = R(0), pmin;
#pragma unroll
    for (int r = 0; r < m; ++r) {
        col[r] = lane < m ? S.at(r, lane) : cmk<R>(lane - m == r ? R(1) : R(0), R(0));
        if (lane < m) smax = fmax(smax, cmaxabs(col[r]));
    }
    cplx<R> ip = crcp(col[0]);  // of this lane's next diagonal entry: lane p's is the pivot's
#pragma unroll
    for (int p = 0; p < m; ++p) {
        __syncwarp();  // every lane is done with buf
        if (lane == p) {
            if constexpr (sizeof(R) == 4) {
#pragma unroll
                for (int r = 0; r + 1 < m; r += 2)
                    *reinterpret_cast<float4*>(buf + r) = make_float4(col[r].x, col[r].y, col[r + 1].x, col[r + 1].y);
                if (m & 1) buf[m - 1] = col[m - 1];
            } else {
#pragma unroll
                for (int r = 0; r < m; ++r) buf[r] = col[r];
            }
            buf[kMaxM] = ip;
        }
        __syncwarp();
        const cplx<R> rp = cmul(col[p], buf[kMaxM]), piv = buf[p];
        // the next pivot's row first, and its reciprocal beside the others
        if (p + 1 < m) {
            const int n = p + 1 < m ? p + 1 : p;
            col[n] = cfms(buf[n], rp, col[n]);
            ip = crcp(col[n]);
        }
        pmin = p == 0 ? cmaxabs(piv) : fmin(pmin, cmaxabs(piv));
        if constexpr (sizeof(R) == 4) {
#pragma unroll
            for (int r = 0; r < m; r += 2) {
                float4 b;
                if (r + 1 < m) {
                    b = *reinterpret_cast<const float4*>(buf + r);
                } else {
                    b.x = buf[r].x;
                    b.y = buf[r].y;
                }
                if (r != p && r != p + 1) col[r] = cfms(cmk(b.x, b.y), rp, col[r]);
                if (r + 1 < m && r + 1 != p && r != p) {
                    const int q = r + 1 < m ? r + 1 : r;
                    col[q] = cfms(cmk(b.z, b.w), rp, col[q]);
                }
            }
        } else {
#pragma unroll
            for (int r = 0; r < m; ++r) {
                if (r == 8) asm volatile("" ::: "memory");  // two batches of multiplier loads
                if (r != p && r != p + 1) col[r] = cfms(buf[r], rp, col[r]);
            }
        }
        col[p] = rp;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) smax = fmax(smax, __shfl_xor_sync(0xffffffffu, smax, o));
    if (!(pmin >= tau * smax)) return invert_pivoted<m, R>(out, S, buf, lane);
    __syncwarp();
    if (lane >= m && lane < n2) {
#pragma unroll
        for (int r = 0; r < m; ++r) out.at(r, lane - m) = col[r];
    }
    __syncwarp();
    return true;
}

// Row layout of the FP64 chains: two lanes per row r = lane / 2, the pairs of
// columns (2q, 2q + 1) on the lanes in turn: lane parity h holds column col(h, j)
// as its j-th (columns past m - 1 are padding, whose values go nowhere).
template <int m>
struct RowLay {
    static constexpr int H = 2 * (m / 4) + (m % 4 < 2 ? m % 4 : 2);
    static constexpr int kBuf = 6 * kMaxM;  // column pairs of the sweeps: three buffers
    __device__ static __forceinline__ int col(int h, int j) { return 4 * (j >> 1) + 2 * h + (j & 1); }
};

// a = -S of a complex symmetric m x m matrix S in the row layout; S^-1 in place,
// by symmetric sweeps on 2 x 2 diagonal blocks B (a 1 x 1 one at the end of an
// odd m).  A sweep keeps the matrix symmetric, so the block's rows are its
// columns: with u_r the two entries of row r under B and t_r = u_r B^-1,
//   a_rc -= t_r . u_c,  a_r,block = t_r   (rows outside the block)
// and the same with u_r = -e_r on a zeroed row for the block's own rows.  Only the
// two columns travel through shared memory (one __syncwarp per block; buf: three
// buffers, as the rest of a sweep overlaps the next one's start), and the next
// block's columns are updated first.  Bound by the chain store - load -
// determinant - reciprocal - two products of a block and, near it, by FP64 issue:
// 2640 cycles at m = 13 with one warp per scheduler, against 3100 for single
// pivots with a broadcast row and 3900 for 2 x 2 blocks with broadcast rows.
// Returns false (a is then garbage) when a multiplier t_r outside the block
// reaches 256 or is no number: the caller falls back to partial pivoting.
template <int m>
__device__ __forceinline__ bool invert_sym(cplxd (&a)[RowLay<m>::H], cplxd* buf, int lane) {
    constexpr int H = RowLay<m>::H;
    const int r = lane >> 1, h = lane & 1;
    int bad = 0;
    // the high words of |doubles| order like the doubles
    auto check = [&](cplxd t, int lim) {
        const int x = __double2hiint(t.x) & 0x7fffffff, y = __double2hiint(t.y) & 0x7fffffff;
        bad |= max(x, y) >= lim;
    };
    auto publish = [&](int p) {
        cplxd* b = buf + (p >> 1) % 3 * 2 * kMaxM + 2 * r;
        const int jp = 2 * (p >> 2), j1 = jp + 1 < H ? jp + 1 : jp;
        if (h == ((p >> 1) & 1)) {
            b[0] = a[jp];
            if (p + 1 < m) b[1] = a[j1];
        }
        __syncwarp();
    };
    publish(0);
#pragma unroll
    for (int p = 0; p < m; p += 2) {
        const bool two = p + 1 < m;
        const int hp = (p >> 1) & 1, jp = 2 * (p >> 2), j1 = jp + 1 < H ? jp + 1 : jp;
        const cplxd* b = buf + (p >> 1) % 3 * 2 * kMaxM;
        const bool own = two ? (r >> 1) == (p >> 1) : r == p;
        const int lim = own ? 0x7ff00000 : 0x40700000;  // 256 outside the block
        cplxd u0 = b[2 * r], u1 = two ? b[2 * r + 1] : cmk(0.0, 0.0), t0, t1 = cmk(0.0, 0.0);
        if (own) {
            u0 = cmk(r == p ? -1.0 : 0.0, 0.0);
            u1 = cmk(r == p ? 0.0 : -1.0, 0.0);
        }
        if (two) {
            const cplxd B00 = b[2 * p], B01 = b[2 * p + 1], B11 = b[2 * p + 3];
            const cplxd rd = crcp(cfms(B01, B01, cmul(B00, B11)));
            t0 = cmul(cfms(u1, B01, cmul(u0, B11)), rd);
            t1 = cmul(cfms(u0, B01, cmul(u1, B00)), rd);
            check(t1, lim);
        } else {
            t0 = cmul(u0, crcp(b[2 * p]));
        }
        check(t0, lim);
        auto update = [&](int j) {
            const cplxd* uc = b + 2 * RowLay<m>::col(h, j);
            cplxd v = own ? cmk(0.0, 0.0) : a[j];
            v = cfms(t0, uc[0], v);
            if (two) v = cfms(t1, uc[1], v);
            if (j == jp) v = h == hp ? t0 : v;
            if (two && j == jp + 1) v = h == hp ? t1 : v;
            a[j] = v;
        };
        const int jn = 2 * ((p + 2) >> 2);  // the next block's columns first
        if (p + 2 < m) {
            update(jn);
            if (jn + 1 < H) update(jn + 1 < H ? jn + 1 : jn);
            publish(p + 2);
        }
#pragma unroll
        for (int j = 0; j < H; ++j)
            if (p + 2 >= m || (j != jn && j != jn + 1)) update(j);
    }
    return !__any_sync(0xffffffffu, bad && r < m);
}

// S^-1 of a complex symmetric matrix in the row layout, build() forming a = -S: by
// invert_sym, or, after a large multiplier, with partial pivoting (a second
// build(), in `tile`; col_buf: pivot column).  Returns false on a zero pivot.
template <int m, class F>
__device__ __forceinline__ bool invert_rows(cplxd (&a)[RowLay<m>::H], F&& build, Mat<m, double> tile, cplxd* sym_buf,
                                            cplxd* col_buf, int lane) {
    build();
    if (invert_sym<m>(a, sym_buf, lane)) return true;
    const int r = lane >> 1, h = lane & 1;
    build();
#pragma unroll
    for (int j = 0; j < RowLay<m>::H; ++j)
        if (r < m && RowLay<m>::col(h, j) < m) tile.at(r, RowLay<m>::col(h, j)) = a[j];
    __syncwarp();
    const bool ok = invert_pivoted<m, double>(tile, tile, col_buf, lane);
#pragma unroll
    for (int j = 0; j < RowLay<m>::H; ++j)
        a[j] = cscale(tile.at(min(r, m - 1), min(RowLay<m>::col(h, j), m - 1)), -1.0);
    __syncwarp();  // every lane has read the tile
    return ok;
}

// Asynchronous global -> shared copy of one complex value (cp.async, 8 or 16
// bytes, both addresses aligned to the size) and the wait for all of them.
template <typename T>
__device__ __forceinline__ void cp_async(T* smem_dst, const T* gsrc) {
    static_assert(sizeof(T) == 8 || sizeof(T) == 16, "cp.async copies 8 or 16 bytes here");
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    if constexpr (sizeof(T) == 16)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gsrc) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Lead kernel: block e -> energy e, lanes 0-15 the left lead, 16-31 the
// right one.  A lead is uniform (the contact potential u on every atom), so
// the Fourier vectors of a ring, v_k[j] = exp(2 pi i k j / m) / sqrt(m),
// decouple it: C v_k = (1 + exp(2 pi i k / m)) v_k, and with a gauge phase
// per ring mode k is the chain of alternating hoppings
// beta_k = 2 gamma cos(pi k / m) (the double bond) and gamma (the single
// bond), the surface ring's first bond being beta_k on both sides (left:
// surface ring b bonded to ring a of its cell; right: surface ring a bonded
// to ring b).  These are the mode chains of the mode-space pass
// (CNT.cpp:288-336), so the ring corner of the lead's surface Green's
// function is the circulant
//   s[j][l] = (1/m) sum_k cos(2 pi k (j - l) / m) s_k,
// s_k the mode chain's surface value by the mode-space formula
// (sgf_analytic, CNT.cpp:354-393, or the reference's decimation when the
// tube uses it).  Exact in O(m^2) per energy and lead, with no matrix
// iteration (an iterated decimation on the 2m-atom cell loses accuracy on
// the real axis, where its Schur complements divide by E - u).
// corners[e][side] = g_surface[s][s] (m x m, row-major).
template <int m>
__global__ void __launch_bounds__(32) rs_lead_kernel(double gamma, const double* __restrict__ Ere,
                                                     const double* __restrict__ Eim, int num_e, double Uc0,
                                                     double Uc1,
                                                     int use_decimation, int dec_layers, int dec_iters,
                                                     cplxd* __restrict__ corners) {
    __shared__ cd sk[2][kMaxM], cdiff[2][kMaxM];
    const int lane = threadIdx.x;
    const int e = blockIdx.x;
    if (e >= num_e) return;
    const int side = lane >> 4, k = lane & 15;
    const double u = side == 0 ? Uc0 : Uc1;
    const cd EmU = {Ere[e] - u, Eim[e]};
    if (k < m) {
        const double beta = 2.0 * gamma * cospi((double)k / m);
        sk[side][k] = use_decimation ? sgf_decimation(EmU, beta, gamma, dec_layers, dec_iters)
                                     : sgf_analytic(EmU, beta, gamma);
    }
    __syncwarp();
    if (k < m) {  // circulant value of ring-index difference d = k
        cd acc = {0.0, 0.0};
        for (int q = 0; q < m; ++q) acc = cadd(acc, cscale(cospi(2.0 * (double)((q * k) % m) / m), sk[side][q]));
        cdiff[side][k] = cscale(1.0 / m, acc);
    }
    __syncwarp();
    cplxd* out = corners + ((size_t)e * 2 + side) * m * m;
    for (int i = k; i < m * m; i += 16) {
        const int j = i / m, l = i % m;
        const cd v = cdiff[side][j >= l ? j - l : j - l + m];
        out[i] = cmk(v.x, v.y);
    }
}

// Gamma = i (Sigma - Sigma^dagger) = -2 gamma^2 Im s of a contact (s: the
// lead's surface corner, a symmetric circulant), factored as L L^T: Gamma is
// diagonal in the ring's real Fourier vectors, so column q of L is the vector of
// mode q (the cosine for q <= m / 2, the sine of m - q else) times the root of
// its eigenvalue; eigenvalues below 1e-13 of Gamma's diagonal give a zero
// column.  O(m^2) over the warp (a Cholesky factor on one lane took 0.19 ms per
// energy at m = 13, a tenth of a biased chain).  tab: 2 kMaxM of shared memory.
template <int m>
__device__ __forceinline__ void gamma_factor(const cplxd* __restrict__ s, double g2, Mat<m, double> L, cplxd* tab,
                                             int lane) {
    if (lane < m) {
        double sn, cs;
        sincospi(2.0 * lane / m, &sn, &cs);
        tab[lane] = cmk(cs, sn);
        tab[kMaxM + lane].x = -2.0 * g2 * s[lane * m].y;  // Gamma[d][0]
    }
    __syncwarp();
    double w = 0.0;
    if (lane < m) {
        double lam = 0.0;
        for (int d = 0; d < m; ++d) lam = fma(tab[(lane * d) % m].x, tab[kMaxM + d].x, lam);
        const double norm = lane == 0 || 2 * lane == m ? 1.0 : 2.0;
        if (lam > 1e-13 * tab[kMaxM].x) w = sqrt(lam * norm / m);
    }
    __syncwarp();
    if (lane < m) tab[kMaxM + lane].x = w;
    __syncwarp();
    for (int i = lane; i < m * m; i += 32) {
        const int j = i / m, q = i % m;
        const cplxd v = tab[(q * j) % m];
        L.a[i] = cmk((2 * q <= m ? v.x : v.y) * tab[kMaxM + q].x, 0.0);
    }
    __syncwarp();
}

// Entries of an m x m tile over T threads (16 columns x T / 16 rows at a time):
// all values first (indices past m - 1 are clamped, so that the loads of a pass
// overlap), then the stores.
template <int m, int T, class F>
__device__ __forceinline__ void for_tile(Mat<m, float> out, int t, F&& f) {
    constexpr int S = T / 16, NR = (m + S - 1) / S;
    const int c = min(t & 15, m - 1), h = t >> 4;
    cplxf v[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) v[i] = f(min(h + S * i, m - 1), c);
#pragma unroll
    for (int i = 0; i < NR; ++i)
        if ((t & 15) < m && h + S * i < m) out.at(h + S * i, c) = v[i];
}

// Complex values of shared memory of an FP32 chain: tiles, the pivot column, D^-1
// of two rings b, E - U of two rings a.
template <int m>
__host__ __device__ constexpr int chain_complex() {
    return 7 * m * m + 5 * kMaxM + 2;
}

// One energy's FP32 chain of mixed mode (block of two warps): atom potentials
// Ua, lead corners (FP64, m x m, row-major), scratch myX for X_k (K m^2
// complex), row of 2K ring sums Im(c sum_j G_jj) written in FP64.  Bound by the
// dependent steps of a block update.  Forward, both warps share the O(m^2)
// passes and one inverts; backward, one warp runs the recursion G' -> X + gamma^4
// (X Z) X while the other forms g_L[b][b], W = g_L[b][b] G' and the traces of the
// step, loads X_{k-1} and D^-1 (G' and X alternate between two tiles, one
// barrier a step).  A block's warps sit on schedulers (0, 1) or (2, 3) by turns;
// every other pair of waves of 148 blocks swaps the roles, so that the inverting
// warps, with twice the work, do not share two schedulers.  Charge of a 57-cell
// (13,0) tube, us, one warp per energy / here: 526 FP32 energies 1200 / 653, with
// 128 real-axis points 1428 / 1045; 2062 with 512: 2302 / 2391 (start 3900).  The
// arithmetic of every FP32 value is that of the one-warp form.
constexpr int kFlip = 2 * 148;
template <int m>
__device__ __forceinline__ bool rs_chain(int K, float gamma, cplxf E, cplxd cc, const double* __restrict__ Ua,
                                         const cplxd* __restrict__ sL, const cplxd* __restrict__ sR,
                                         cplxf* __restrict__ myX, double* __restrict__ row, cplxf* sh) {
    using C = cplxf;
    constexpr int mm2 = m * m;
    const int t = threadIdx.x, lane = t & 31;
    const bool helper = (t >= 32) != (blockIdx.x / kFlip % 2 != 0);
    const float g2 = gamma * gamma, g4 = g2 * g2;
    C* buf = sh;              // pivot column (16-byte aligned)
    C* dv = buf + kMaxM + 2;  // D^-1 of ring b of block k: dv + (k & 1) kMaxM
    C* da = dv + 2 * kMaxM;   // E - U of ring a of block k, in the same way
    C* tiles = da + 2 * kMaxM;
    const Mat<m, float> X{tiles}, X1{tiles + mm2}, Gbb{tiles + 2 * mm2}, G0{tiles + 3 * mm2}, G1{tiles + 4 * mm2},
        Z{tiles + 5 * mm2}, H{tiles + 6 * mm2};
    bool ok = true;
    // thread j < m: potentials of atom j on rings a and b of the next block
    float ua_n = 0.0f, ub_n = 0.0f;
    auto fetch_u = [&](int k) {
        if (lane < m) {
            ua_n = (float)__ldg(Ua + (size_t)(2 * k) * m + lane);
            ub_n = (float)__ldg(Ua + (size_t)(2 * k + 1) * m + lane);
        }
    };
    // g_L[b][b] = D^-1 + gamma^2 Y^T X Y, entry (r, c)
    auto gbb = [&](Mat<m, float> Xt, const C* d, int r, int c) {
        const int r0 = wrap<m>(r - 1), c0 = wrap<m>(c - 1);
        const C q = cadd(cadd(Xt.at(r, c), Xt.at(r, c0)), cadd(Xt.at(r0, c), Xt.at(r0, c0)));
        C v = cscale(cmul(cmul(d[r], d[c]), q), g2);
        if (r == c) v = cadd(v, d[r]);
        return v;
    };
    // left lead corner as g_L[b][b] of block -1
    for (int i = t; i < mm2; i += 64) Gbb.a[i] = cmk((float)sL[i].x, (float)sL[i].y);
    // D^-1 and E - U of block k by the helper, beside the inversion of block k - 1
    auto enter = [&](int k) {
        if (lane < m) {
            dv[(k & 1) * kMaxM + lane] = crcp(cmk(E.x - ub_n, E.y));
            da[(k & 1) * kMaxM + lane] = cmk(E.x - ua_n, E.y);
        }
        if (k + 1 < K) fetch_u(k + 1);
    };
    fetch_u(0);
    if (helper) enter(0);
    for (int k = 0; k < K; ++k) {
        const C *d = dv + (k & 1) * kMaxM, *dk = da + (k & 1) * kMaxM;
        __syncthreads();
        // S = diag(E - U_a) - gamma^2 g_L[b][b]_{k-1} - gamma^2 C D^-1 C^T
        for_tile<m, 64>(X, t, [&](int r, int c) {
            const int r1 = wrap<m>(r + 1), c1 = wrap<m>(c + 1);
            C cd = cmk(0.0f, 0.0f);
            if (r == c) cd = cadd(cd, d[r]);
            if (r == c1) cd = cadd(cd, d[r]);
            if (r1 == c) cd = cadd(cd, d[r1]);
            if (r1 == c1) cd = cadd(cd, d[r1]);
            C v = cscale(cadd(Gbb.at(r, c), cd), -g2);
            if (r == c) v = cadd(v, dk[r]);
            return v;
        });
        __syncthreads();
        if (!helper)
            ok = invert<m>(X, X, buf, lane) && ok;
        else if (k + 1 < K)
            enter(k + 1);
        __syncthreads();
        C* dst = myX + (size_t)k * mm2;
        for (int i = t; i < mm2; i += 64) dst[i] = X.a[i];
        for_tile<m, 64>(Gbb, t, [&](int r, int c) { return gbb(X, d, r, c); });
    }
    __syncthreads();
    // G_K[a][a] of the right lead's first ring: (I - gamma^2 s_R g_L[b][b])^-1 s_R
    if (!helper) {
        for (int i = lane; i < mm2; i += 32) X.a[i] = cmk((float)sR[i].x, (float)sR[i].y);
        __syncwarp();
        mm<m, false, false, false>(G0, X, Gbb, G0, -g2, lane);
        if (lane < m) G0.at(lane, lane) = cadd(G0.at(lane, lane), cmk(1.0f, 0.0f));
        ok = invert<m>(G0, G0, buf, lane) && ok;
        mm<m, false, false, false>(G0, G0, X, G0, 1.0f, lane);
    }
    __syncthreads();
    // Backward
    fetch_u(K - 1);
    if (helper && lane < m) dv[((K - 1) & 1) * kMaxM + lane] = crcp(cmk(E.x - ub_n, E.y));
    for (int i = t; i < mm2; i += 64) X.a[i] = myX[(size_t)(K - 1) * mm2 + i];
    __syncthreads();
    Mat<m, float> Xc = X, Xo = X1, Gn = G0, Go = G1;
    // Im(c G_jj), j = lane, of a diagonal
    auto diag = [&](Mat<m, float> G) {
        const C v = G.at(min(lane, m - 1), min(lane, m - 1));
        return lane < m ? fma(cc.x, (double)v.y, cc.y * (double)v.x) : 0.0;
    };
    // lanes 0-15 sum a into row[ra], 16-31 b into row[rb]
    auto write = [&](double a, int ra, double b, int rb) {
        double w = (lane < 16 ? a : b) + __shfl_xor_sync(0xffffffffu, lane < 16 ? b : a, 16);
#pragma unroll
        for (int o = 8; o >= 1; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if ((lane & 15) == 0 && (lane ? rb : ra) < 2 * K) row[lane ? rb : ra] = w;
    };
    for (int k = K - 1; k >= 0; --k) {
        const C* d = dv + (k & 1) * kMaxM;
        if (helper) {
            if (k > 0) {
                const C* src = myX + (size_t)(k - 1) * mm2;
                for (int i = lane; i < mm2; i += 32) cp_async(Xo.a + i, src + i);
                cp_async_commit();
                fetch_u(k - 1);
            }
            for_tile<m, 32>(Gbb, lane, [&](int r, int c) { return gbb(Xc, d, r, c); });
            __syncwarp();
            // W = g_L[b][b] G'; tr G[b][b] = tr g_L[b][b] + gamma^2 sum_rc W[r][c] g_L[b][b][c][r]
            const double ta = diag(Gn);
            double tb = diag(Gbb);
            cplxd tw = cmk(0.0, 0.0);
            mm_each<m, false, false>(
                Gbb, Gn, 1.0f, lane, [&](int r, int c, C v) { return cmul(cscale(v, g2), Gbb.at(c, r)); },
                [&](int, int, C v) { tw = cadd(tw, cmk((double)v.x, (double)v.y)); });
            tb += fma(cc.x, tw.y, cc.y * tw.x);
            write(ta, 2 * k + 2, tb, 2 * k + 1);
            if (k > 0 && lane < m) dv[((k - 1) & 1) * kMaxM + lane] = crcp(cmk(E.x - ub_n, E.y));
            cp_async_wait_all();
        } else {
            // Z = Y G' Y^T = C (D^-1 G' D^-1) C^T, Y = C D^-1: H = D^-1 G' D^-1, then
            // four neighbours of H per entry
            for_tile<m, 32>(H, lane, [&](int r, int c) { return cmul(cmul(d[r], Gn.at(r, c)), d[c]); });
            __syncwarp();
            for_tile<m, 32>(Z, lane, [&](int r, int c) {
                const int r1 = wrap<m>(r + 1), c1 = wrap<m>(c + 1);
                return cadd(cadd(H.at(r, c), H.at(r, c1)), cadd(H.at(r1, c), H.at(r1, c1)));
            });
            __syncwarp();
            // G[a][a] = X + gamma^4 (X Z) X
            mm<m, false, false, false>(Z, Xc, Z, Z, 1.0f, lane);
            mm<m, false, false, true>(Go, Z, Xc, Xc, g4, lane);
        }
        __syncthreads();
        Mat<m, float> tt = Xc;
        Xc = Xo;
        Xo = tt;
        tt = Gn;
        Gn = Go;
        Go = tt;
    }
    if (helper) write(diag(Gn), 0, 0.0, 2 * K);
    return ok;
}

// FP32 chain kernel: block i -> energy e = e_off + i.
// gX: [energy][K][m*m] FP64-complex slots (an FP32 chain uses the first half
// of its slot); rows: [energy][N].
template <int m>
__global__ void __launch_bounds__(64, 8) rs_chain_kernel(int K, double gamma, const double* __restrict__ Ere,
                                                         const double* __restrict__ Eim,
                                                         const double* __restrict__ cre,
                                                         const double* __restrict__ cim, int e_off, int num,
                                                         const double* __restrict__ Ua,
                                                         const cplxd* __restrict__ corners, cplxd* __restrict__ gX,
                                                         double* __restrict__ rows, int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char sh_raw[];
    if ((int)blockIdx.x >= num) return;
    const int e = e_off + blockIdx.x;
    constexpr int mm2 = m * m;
    const cplxd* sL = corners + (size_t)e * 2 * mm2;
    const bool ok = rs_chain<m>(K, (float)gamma, cmk((float)Ere[e], (float)Eim[e]), cmk(cre[e], cim[e]), Ua, sL,
                                sL + mm2, reinterpret_cast<cplxf*>(gX + (size_t)e * K * mm2),
                                rows + (size_t)e * 2 * K, reinterpret_cast<cplxf*>(sh_raw));
    if (!ok && (threadIdx.x & 31) == 0) atomicExch(status, 1);
}

// Complex values of shared memory of one warp of a pair: tiles, then D^-1 of
// the current and the previous ring b, the pivot column of the fall-back and the
// column pairs of the sweeps.
template <int m, bool NEQ>
__host__ __device__ constexpr int pair_complex() {
    return (NEQ ? 7 : 5) * m * m + 3 * kMaxM + 2 + RowLay<m>::kBuf;
}

// One half of an energy's chain in FP64.  The two warps of a block take the
// chain from its two ends and meet in the middle: side 0 runs blocks 0 .. KS -
// 1 from the left lead; side 1 the others from the right lead, on the chain
// read backwards.  Read backwards with the atoms of every ring reflected, j ->
// -j mod m, the chain has the same bonds (ring b comes first, its atom j bonded
// to atoms j and j - 1 of ring a), and the lead corners are symmetric
// circulants, so both sides run the same code; only the potentials' addresses,
// the rows and the contacts' roles differ.  Each side
//   sweeps forward over its KS blocks (X_k kept in myX),
//   takes the other side's end corner s = g[b][b], reflected, as its right lead:
//     G' = G_K[a][a] = (s^-1 - gamma^2 g_L[b][b])^-1 of the other side's last ring,
//   and runs the backward recursion over its blocks, with V = X Y, Y = C D^-1:
//     M = V G'                            gamma^2 M = G_{k,k+1}[a][a]
//     G_kk[a][a] = X + gamma^4 M V^T      (symmetric: three of four tiles)
//     G_kk[b][b]_rr = d_r + gamma^2 d_r^2 (C^T G_kk[a][a] C + 2 gamma^2 C^T M + G')_rr
//   (the last from (E - H) G = 1 in the rows and columns of ring b): two products
//   per block and O(m^2).  The diagonal formula loses a factor gamma^2 |d|^2 of
//   the working precision, so a ring with an atom within gamma / 100 of E (no
//   energy at 300 K: the lowest pole lies 0.08 eV off the axis) takes
//   tr G[b][b] = tr(g_L[b][b]) + gamma^2 tr(g_L[b][b]^2 G') instead.
// The work is that of one chain, its length in dependent steps is halved.
//
// NEQ (a real-axis energy): the row holds the ring sums of the contact
// spectral functions, b0 A^L + b1 A^R with (b0, b1) = cc and
// A^c_ring = sum_{n in ring} [G_{n,c} Gamma_c G_{n,c}^dagger]_nn
// = || G_{ring,c} L_c ||_F^2 (Gamma_c = L_c L_c^T).  The columns of G times L
// come by block substitution, for the side's own lead (S_k = G_{a_k,a_0} L) and
// the other one (T_k):
//   forward   P_k = gamma X_k Q_{k-1}, Q_k = gamma Y^T P_k, Q_{-1} = L / gamma
//             (Q_k = g_L[k]_{b_k, a_0} L; P_k kept in myP);
//   middle    S_K = gamma G' Q_{KS-1}; T_K = G' s^-1 Q', Q' the other side's last Q,
//             reflected (not (I + gamma^2 G' g_L[b][b]) Q': where E passes the potential
//             of whole rings, s and g_L[b][b] are as large as 1 / Im E in some modes and
//             G' = -1 / (gamma^2 g_L[b][b]) there to the last digit; a (13,0) tube of 10
//             blocks at that energy and Im E = 1e-8 came out 1e9 times too large);
//   backward  S_k = P_k + gamma^2 V S_{k+1}, T_k = gamma^2 V T_{k+1}, and on ring b
//             the rows of (E - H) G = 1: D^-1 gamma (C^T S_k + S_{k+1}), the same for T.
// Three products per block; no G_jj sums (the real-axis energies carry no
// contour term).
//
// Bound by the dependent steps of one block update up to one warp per scheduler
// (8000 cycles at m = 13: inversion 2640, products 2000, passes over tiles the
// rest), by FP64 issue and shared memory beyond.  Charge of a 75-cell tube, us,
// with one warp per energy, three products and single pivots / here:
//   m = 13, 64 + 64 + 128 contour points   1425 / 377
//   m = 13, 128 + 128 + 256                1514 / 548
//   m = 13, 512 + 512 + 1024               3366 / 1826
//   m = 16, 128 + 128 + 256                1912 / 759
//   m = 7,  128 + 128 + 256                 600 / 272
//   m = 13, 64 real-axis points            3529 / 758
//   m = 13, 2048 real-axis points          7920 / 2774
template <int m, bool NEQ>
__device__ __forceinline__ bool rs_side(int side, int K, int KS, double gamma, cplxd E, cplxd cc,
                                        const double* __restrict__ Ua, const cplxd* __restrict__ sL,
                                        cplxd* __restrict__ myX, cplxd* __restrict__ myP, double* __restrict__ row,
                                        cplxd* sh, const cplxd* other, int lane) {
    using C = cplxd;
    constexpr int mm2 = m * m, H = (m + 1) / 2, HR = RowLay<m>::H;
    using Tile = Mat<m, double>;
    const double g2 = gamma * gamma, g4 = g2 * g2;
    const Tile X{sh}, B{sh + mm2}, V{sh + 2 * mm2}, Gn{sh + 3 * mm2}, Q{sh + 4 * mm2};
    C* dv = sh + (NEQ ? 7 : 5) * mm2;  // D^-1 of the current ring b
    C* dp = dv + kMaxM;                // D^-1 of the previous ring b
    C* buf = dp + kMaxM;               // pivot column of the fall-back
    C* inv_buf = buf + kMaxM + 2;      // column pairs of the sweeps
    const int N = 2 * K;
    bool ok = true;
    // Row layout (two lanes per row) of the forward sweep, column layout (lane &
    // 15 = column, rows h H ..) of the tile passes; rows and columns past m - 1
    // are clamped, so that no load is conditional and the loads of a pass overlap.
    const int rr = min(lane >> 1, m - 1), hr = lane & 1;
    const bool rv = (lane >> 1) < m;
    auto col = [&](int j) { return min(RowLay<m>::col(hr, j), m - 1); };
    const int pc = min(lane & 15, m - 1), pr = (lane >> 4) * H;
    const bool pv = (lane & 15) < m;
    // potentials of atom rr (of the reflected ring on side 1) on rings a and b of the next block
    const int atom = side && rr > 0 ? m - rr : rr;
    double ua_n = 0.0, ub_n = 0.0;
    auto fetch_u = [&](int k) {
        const int ra = side ? N - 1 - 2 * k : 2 * k, rb = side ? ra - 1 : ra + 1;
        ua_n = __ldg(Ua + (size_t)ra * m + atom);
        ub_n = __ldg(Ua + (size_t)rb * m + atom);
    };
    // g_L[b][b] = D^-1 + gamma^2 Y^T X Y of tile Xt into B
    auto form_gbb = [&](Tile Xt, Tile out, const C* d) {
        const int c0 = wrap<m>(pc - 1);
        const C dc = cscale(d[pc], g2);
        C s[H + 1];
#pragma unroll
        for (int i = 0; i <= H; ++i) {
            const int r = min(wrap<m>(pr - 1 + i), m - 1);
            s[i] = cadd(Xt.at(r, pc), Xt.at(r, c0));
        }
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const int r = min(pr + i, m - 1);
            C v = cmul(cmul(d[r], dc), cadd(s[i], s[i + 1]));
            if (r == pc) v = cadd(v, d[r]);
            if (pv && pr + i < m) out.at(r, pc) = v;
        }
        __syncwarp();
    };
    if constexpr (NEQ) {
        gamma_factor<m>(sL, g2, Q, dv, lane);  // dv, dp: scratch
#pragma unroll
        for (int i = lane; i < mm2; i += 32) Q.a[i] = cscale(Q.a[i], 1.0 / gamma);
    }
    fetch_u(0);
    // E - U_a and D^-1 of this lane's row, one block ahead; D^-1 of the ring in dv, dp (the previous ring's) in turn
    C da = cmk(E.x - ua_n, E.y), db = crcp(cmk(E.x - ub_n, E.y));
    if (KS > 1) fetch_u(1);
    __syncwarp();
    if (rv && hr == 0) dv[rr] = db;
    __syncwarp();
    for (int k = 0; k < KS; ++k) {
        // -S, S = diag(E - U_a) - gamma^2 g_L[b][b]_{k-1} - gamma^2 C D^-1 C^T, in the row layout straight
        // from X_{k-1} (the lead's corner at k = 0): no pass over a tile between two inversions
        C a[HR];
        auto build = [&]() {
            const int r0 = wrap<m>(rr - 1), r1 = wrap<m>(rr + 1);
            const C lo = cscale(db, g2), hi = cscale(dv[r1], g2);
            C dg = csub(cadd(lo, hi), da);
            if (k == 0) {
#pragma unroll
                for (int j = 0; j < HR; ++j) a[j] = cscale(sL[rr * m + col(j)], g2);
            } else {
                const C dr = cscale(dp[rr], g2);
                const C dq = cscale(dr, g2);
                dg = cadd(dg, dr);
#pragma unroll
                for (int j = 0; j < HR; j += 2) {
                    const int c = col(j), c0 = wrap<m>(c - 1);
                    const C s0 = cadd(X.at(rr, c0), X.at(r0, c0)), s1 = cadd(X.at(rr, c), X.at(r0, c));
                    a[j] = cmul(cmul(dq, dp[c]), cadd(s0, s1));
                    if (j + 1 < HR) {
                        const int c1 = col(j + 1);
                        const C s2 = cadd(X.at(rr, c1), X.at(r0, c1));
                        a[j + 1 < HR ? j + 1 : j] = cmul(cmul(dq, dp[c1]), cadd(s1, s2));
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < HR; ++j) {
                const int c = col(j), c1 = wrap<m>(c + 1);
                if (rr == c) a[j] = cadd(a[j], dg);
                if (rr == c1) a[j] = cadd(a[j], lo);  // column r - 1
                if (r1 == c) a[j] = cadd(a[j], hi);   // column r + 1
            }
        };
        ok = invert_rows<m>(a, build, V, inv_buf, buf, lane) && ok;
        __syncwarp();  // every lane is done with X_{k-1} and dp
        C* dst = myX + (size_t)k * mm2;
#pragma unroll
        for (int j = 0; j < HR; ++j) {
            const int c = RowLay<m>::col(hr, j);
            if (rv && c < m) {
                X.at(rr, c) = a[j];
                dst[rr * m + c] = a[j];
            }
        }
        if (k + 1 < KS) {
            da = cmk(E.x - ua_n, E.y);
            db = crcp(cmk(E.x - ub_n, E.y));
            if (rv && hr == 0) dp[rr] = db;
            if (k + 2 < KS) fetch_u(k + 2);
        }
        __syncwarp();
        if constexpr (NEQ) {
            // P_k = gamma X_k Q_{k-1} (in V); Q_k = gamma Y^T P_k, (Y^T P)[r][c] = D^-1_r (P[r][c] + P[r-1][c])
            C* pd = myP + (size_t)k * mm2;
            mm_each<m, false, false, false>(
                X, Q, lane, [&](int, int, C v) { return cscale(v, gamma); },
                [&](int r, int c, C v, bool) { V.at(r, c) = pd[r * m + c] = v; });
            C s[H + 1];
#pragma unroll
            for (int i = 0; i <= H; ++i) s[i] = V.at(min(wrap<m>(pr - 1 + i), m - 1), pc);
#pragma unroll
            for (int i = 0; i < H; ++i) {
                const int r = min(pr + i, m - 1);
                const C v = cmul(cscale(dv[r], gamma), cadd(s[i], s[i + 1]));
                if (pv && pr + i < m) Q.at(r, pc) = v;
            }
            __syncwarp();  // every lane is done with dv
        }
        if (k + 1 < KS) {
            C* const t = dv;
            dv = dp;
            dp = t;
        }
    }
    form_gbb(X, B, dv);
    // the other side's end corner, reflected, into X, its Q into T
    const Tile T{sh + (NEQ ? 5 : 0) * mm2}, P{sh + (NEQ ? 6 : 0) * mm2};
    __syncthreads();
    for (int i = lane; i < mm2; i += 32) {
        const int r = i / m, c = i % m, r1 = r ? m - r : 0, c1 = c ? m - c : 0;
        X.a[i] = other[mm2 + r1 * m + c1];
        if constexpr (NEQ) T.a[i] = other[4 * mm2 + r1 * m + c];
    }
    __syncthreads();  // both have read: B and Q may change
    // s^-1 in place of s, then G' = (s^-1 - gamma^2 g_L[b][b])^-1: on checked pivots, as s can be as near to
    // singular as Im E (invert_sym's multipliers of up to 256 cost the charge 1e-7 at Im E = 1e-8)
    ok = invert<m>(X, X, buf, lane) && ok;
    if constexpr (NEQ) mm<m, false, false, false>(P, X, T, P, 1.0, lane);  // s^-1 Q'
    for (int i = lane; i < mm2; i += 32) Gn.a[i] = csub(X.a[i], cscale(B.a[i], g2));
    ok = invert<m>(Gn, Gn, buf, lane) && ok;
    fetch_u(KS - 1);
    if constexpr (!NEQ) {
        // X_{k-1} is copied into the other of two tiles while step k runs
        Tile Xc = X, Xo = B;
        const Tile M = Q;
        auto fetch_x = [&](Tile to, int k) {
            const C* src = myX + (size_t)k * mm2;
            for (int i = lane; i < mm2; i += 32) cp_async(to.a + i, src + i);
            cp_async_commit();
        };
        // X_k has landed: D^-1 and V of block k; true when its ring b needs the product formula
        auto enter = [&](int k) {
            const C db = crcp(cmk(E.x - ub_n, E.y));
            if (k > 0) fetch_u(k - 1);
            if (rv && hr == 0) dv[rr] = db;
            cp_async_wait_all();
            __syncwarp();
            const int c0 = wrap<m>(pc - 1);
            const C dc = dv[pc];
#pragma unroll
            for (int i = 0; i < H; ++i) {
                const int r = min(pr + i, m - 1);
                const C v = cmul(dc, cadd(Xc.at(r, pc), Xc.at(r, c0)));
                if (pv && pr + i < m) V.at(r, pc) = v;
            }
            return __any_sync(0xffffffffu, g2 * fma(db.x, db.x, db.y * db.y) > 1e4);
        };
        fetch_x(Xc, KS - 1);
        bool near = enter(KS - 1);
        for (int k = KS - 1; k >= 0; --k) {
            __syncwarp();
            if (k > 0) fetch_x(Xo, k - 1);
            const int t = min(lane & 15, m - 1), t0 = wrap<m>(t - 1);
            const C gp = Gn.at(t, t);
            C tr = cmk(0.0, 0.0);  // ring b by products: this lane's part of tr G[b][b]
            if (near) {
                form_gbb(Xc, M, dv);
                if (lane < m) tr = M.at(lane, lane);
                mm_each<m, false, false, true>(
                    M, M, lane, [&](int r, int c, C v) { return cmul(cscale(v, g2), Gn.at(c, r)); },
                    [&](int, int, C v, bool off) { tr = cadd(tr, cscale(v, off ? 2.0 : 1.0)); });
            }
            mm<m, false, false, false>(M, V, Gn, M, 1.0, lane);
            mm_each<m, false, true, true>(
                M, V, lane, [&](int r, int c, C v) { return cadd(cscale(v, g4), Xc.at(r, c)); },
                [&](int r, int c, C v, bool off) {
                    Gn.at(r, c) = v;
                    if (off) Gn.at(c, r) = v;
                });
            // diagonals: lanes 0-15 ring a, 16-31 ring b
            const C g11 = Gn.at(t, t);
            C v = g11;
            if (lane >= 16) {
                const C d = dv[t], d2 = cscale(cmul(d, d), g2);
                const C o = cadd(cadd(Gn.at(t0, t), Gn.at(t0, t)), cadd(g11, Gn.at(t0, t0)));
                const C q = cadd(cadd(o, gp), cscale(cadd(M.at(t, t), M.at(t0, t)), 2.0 * g2));
                v = cfma(d2, q, d);
            }
            double w = (lane & 15) < m ? fma(cc.x, v.y, cc.y * v.x) : 0.0;  // Im(c G_jj)
            if (near) {
                const double wb = fma(cc.x, tr.y, cc.y * tr.x);
                const double other_half = __shfl_xor_sync(0xffffffffu, wb, 16);
                if (lane >= 16) w = wb + other_half;
            }
            const int2 rg = side ? make_int2(N - 1 - 2 * k, N - 2 - 2 * k) : make_int2(2 * k, 2 * k + 1);
            if (k > 0) {
                const Tile tt = Xc;
                Xc = Xo;
                Xo = tt;
                __syncwarp();  // every lane is done with dv
                near = enter(k - 1);
            }
#pragma unroll
            for (int o = 8; o >= 1; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
            if (lane == 0) row[rg.x] = w;
            if (lane == 16) row[rg.y] = w;
        }
    } else {
        // S_K and T_K; then S and T alternate between two tiles each
        Tile Sc = Q, So = B, Tc = T, To = Gn;
        mm<m, false, false, false>(T, Gn, P, T, 1.0, lane);
        mm<m, false, false, false>(Q, Gn, Q, Q, gamma, lane);
        auto fetch = [&](Tile to, const C* src) {
            for (int i = lane; i < mm2; i += 32) cp_async(to.a + i, src + i);
        };
        fetch(X, myX + (size_t)(KS - 1) * mm2);
        fetch(P, myP + (size_t)(KS - 1) * mm2);
        cp_async_commit();
        for (int k = KS - 1; k >= 0; --k) {
            const C db = crcp(cmk(E.x - ub_n, E.y));
            if (k > 0) fetch_u(k - 1);
            if (rv && hr == 0) dv[rr] = db;
            cp_async_wait_all();
            __syncwarp();
            const int c0 = wrap<m>(pc - 1);
            const C dc = dv[pc];
#pragma unroll
            for (int i = 0; i < H; ++i) {
                const int r = min(pr + i, m - 1);
                const C v = cmul(dc, cadd(X.at(r, pc), X.at(r, c0)));
                if (pv && pr + i < m) V.at(r, pc) = v;
            }
            __syncwarp();
            if (k > 0) fetch(X, myX + (size_t)(k - 1) * mm2);
            double sa = 0.0, sb = 0.0;  // this lane's part of the two ring sums
            mm_each<m, false, false, false>(
                V, Sc, lane, [&](int r, int c, C v) { return cadd(cscale(v, g2), P.at(r, c)); },
                [&](int r, int c, C v, bool) {
                    So.at(r, c) = v;
                    sa = fma(v.x, v.x, fma(v.y, v.y, sa));
                });
            sa *= cc.x;
            if (k > 0) fetch(P, myP + (size_t)(k - 1) * mm2);
            cp_async_commit();
            double ta = 0.0, tb = 0.0;
            mm_each<m, false, false, false>(
                V, Tc, lane, [&](int, int, C v) { return cscale(v, g2); },
                [&](int r, int c, C v, bool) {
                    To.at(r, c) = v;
                    ta = fma(v.x, v.x, fma(v.y, v.y, ta));
                });
            sa = fma(cc.y, ta, sa);
            // ring b: gamma D^-1 (C^T S_k + S_{k+1}), (C^T S)[r][c] = S[r][c] + S[r-1][c]
            C s[H + 1], u[H + 1];
#pragma unroll
            for (int i = 0; i <= H; ++i) {
                const int r = min(wrap<m>(pr - 1 + i), m - 1);
                s[i] = So.at(r, pc);
                u[i] = To.at(r, pc);
            }
#pragma unroll
            for (int i = 0; i < H; ++i) {
                const int r = min(pr + i, m - 1);
                const C d = dv[r];
                const C x = cadd(cadd(s[i], s[i + 1]), Sc.at(r, pc)), y = cadd(cadd(u[i], u[i + 1]), Tc.at(r, pc));
                double q = fma(d.x, d.x, d.y * d.y);
                if (!(pv && pr + i < m)) q = 0.0;
                sb = fma(q, fma(x.x, x.x, x.y * x.y), sb);
                tb = fma(q, fma(y.x, y.x, y.y * y.y), tb);
            }
            sb = g2 * fma(cc.x, sb, cc.y * tb);
            // lanes 0-15 sum ring a, 16-31 ring b
            double w = (lane < 16 ? sa : sb) + __shfl_xor_sync(0xffffffffu, lane < 16 ? sb : sa, 16);
#pragma unroll
            for (int o = 8; o >= 1; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
            const int2 rg = side ? make_int2(N - 1 - 2 * k, N - 2 - 2 * k) : make_int2(2 * k, 2 * k + 1);
            if (lane == 0) row[rg.x] = w;
            if (lane == 16) row[rg.y] = w;
            Tile tt = Sc;
            Sc = So;
            So = tt;
            tt = Tc;
            Tc = To;
            To = tt;
            __syncwarp();  // every lane is done with dv and V
        }
    }
    return ok;
}

// FP64 chains: block i -> energy e = e_off + i, one warp per side.  gX: contour
// and pole energies [e][K][m*m] (X_k of side 0, then of side 1); real-axis
// energies [i][2][K][m*m] (X_k, P_k).  Four blocks per SM leave 255 registers a
// thread; six (168, spills) take 369 us against 345 for 64 contour points at m =
// 13 and gain 5 % at 2048.
template <int m, bool NEQ>
__global__ void __launch_bounds__(64, 4) rs_pair_kernel(int K, double gamma, const double* __restrict__ Ere,
                                                        const double* __restrict__ Eim,
                                                        const double* __restrict__ cre,
                                                        const double* __restrict__ cim, int e_off, int num,
                                                        const double* __restrict__ Ua,
                                                        const cplxd* __restrict__ corners, cplxd* __restrict__ gX,
                                                        double* __restrict__ rows, int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char sh_raw[];
    if ((int)blockIdx.x >= num) return;
    constexpr int mm2 = m * m, per = pair_complex<m, NEQ>();
    cplxd* sh = reinterpret_cast<cplxd*>(sh_raw);
    const int lane = threadIdx.x & 31, side = threadIdx.x >> 5;
    const int e = e_off + blockIdx.x, K0 = K / 2, KS = side ? K - K0 : K0;
    cplxd* X = gX + ((size_t)(NEQ ? 2 * blockIdx.x : e) * K + (side ? K0 : 0)) * mm2;
    const cplxd cc = NEQ && side ? cmk(cim[e], cre[e]) : cmk(cre[e], cim[e]);
    const bool ok = rs_side<m, NEQ>(side, K, KS, gamma, cmk(Ere[e], Eim[e]), cc, Ua,
                                    corners + ((size_t)e * 2 + side) * mm2, X, X + (size_t)K * mm2,
                                    rows + (size_t)e * 2 * K, sh + side * per, sh + (1 - side) * per, lane);
    if (!ok && lane == 0) atomicExch(status, 1);
}

// Self-test of the tile primitives: warp w takes matrix w (inversion: mode 0;
// symmetric, as the FP64 chains do: mode 2) or the pair (A, B) w (product: mode 1)
// from in (complex, re/im interleaved, row-major m x m, FP64), computes in
// precision R and writes the m x m result to out.
template <int m, typename R>
__global__ void __launch_bounds__(32) rs_selftest_kernel(int mode, int count, const double* __restrict__ in,
                                                         double* __restrict__ out) {
    __shared__ __align__(16) cplx<R> sh[3 * m * m + kMaxM + 2];
    const int lane = threadIdx.x, w = blockIdx.x;
    if (w >= count) return;
    constexpr int mm2 = m * m;
    cplx<R>* buf = sh;
    const Mat<m, R> A{sh + kMaxM + 2}, B{A.a + mm2}, C{B.a + mm2};
    const bool product = mode == 1;
    const double* src = in + (size_t)w * (product ? 2 : 1) * 2 * mm2;
    for (int i = lane; i < mm2; i += 32) {
        A.a[i] = cmk((R)src[2 * i], (R)src[2 * i + 1]);
        if (product) B.a[i] = cmk((R)src[2 * mm2 + 2 * i], (R)src[2 * mm2 + 2 * i + 1]);
    }
    __syncwarp();
    bool ok = true;
    if (product)
        mm<m, false, false, false>(C, A, B, C, R(1), lane);
    else if (mode == 0)
        ok = invert<m>(C, A, buf, lane);
    else if constexpr (sizeof(R) == 8) {
        __shared__ cplxd sym_buf[RowLay<m>::kBuf];
        constexpr int H = RowLay<m>::H;
        const int r = lane >> 1, h = lane & 1;
        cplxd a[H];
        auto col = [&](int j) { return min(RowLay<m>::col(h, j), m - 1); };
        ok = invert_rows<m>(
            a,
            [&]() {
#pragma unroll
                for (int j = 0; j < H; ++j) a[j] = cscale(A.at(min(r, m - 1), col(j)), -1.0);
            },
            B, sym_buf, buf, lane);
#pragma unroll
        for (int j = 0; j < H; ++j)
            if (r < m && RowLay<m>::col(h, j) < m) C.at(r, RowLay<m>::col(h, j)) = a[j];
        __syncwarp();
    }
    double* dst = out + (size_t)w * 2 * mm2;
    for (int i = lane; i < mm2; i += 32) {
        dst[2 * i] = ok ? (double)C.a[i].x : NAN;
        dst[2 * i + 1] = ok ? (double)C.a[i].y : NAN;
    }
}

// Q[r] = sum over energies of rows[e][r] (minus sub[r]): block = 32 rings x kRsGroups
// energy groups; each thread sums energies g, g + kRsGroups, ... (Kahan),
// then the groups are combined in a fixed order (deterministic).  Bound by the
// serial Kahan steps of a thread: 530 energies of 300 rings 9 us with 32 groups, 19
// us with 8.
constexpr int kRsGroups = 32;
__global__ void __launch_bounds__(32 * kRsGroups) rs_reduce_kernel(const double* __restrict__ rows, int num_e, int N,
                                                                   const double* __restrict__ sub,
                                                                   double* __restrict__ Q) {
    __shared__ double sh_s[kRsGroups][32], sh_c[kRsGroups][32];
    const int r = blockIdx.x * 32 + threadIdx.x, g = threadIdx.y;
    double s = 0.0, comp = 0.0;
    if (r < N) {
#pragma unroll 4
        for (int e = g; e < num_e; e += kRsGroups) {
            const double y = rows[(size_t)e * N + r] - comp;
            const double t = s + y;
            comp = (t - s) - y;
            s = t;
        }
    }
    sh_s[g][threadIdx.x] = s;
    sh_c[g][threadIdx.x] = comp;
    __syncthreads();
    if (g == 0 && r < N) {
        double tot = 0.0, c = 0.0;
        for (int i = 0; i < kRsGroups; ++i) {
            const double y = (sh_s[i][threadIdx.x] - sh_c[i][threadIdx.x]) - c;
            const double t = tot + y;
            c = (t - tot) - y;
            tot = t;
        }
        Q[r] = sub ? tot - sub[r] : tot;
    }
}

// Uatoms[r][j] = U[r] (ring-uniform potential on the atoms).
__global__ void rs_expand_kernel(const double* __restrict__ U, int N, int m, double* __restrict__ Ua) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N * m) Ua[i] = U[i / m];
}

}  // namespace

cudaError_t rs_expand(const double* d_U, int N, int m, double* d_Ua, cudaStream_t stream) {
    if (N * m <= 0) return cudaSuccess;
    rs_expand_kernel<<<(N * m + 255) / 256, 256, 0, stream>>>(d_U, N, m, d_Ua);
    return cudaGetLastError();
}

int rs_max_atoms_per_block() { return 2 * kMaxM; }

cudaError_t rs_selftest(int which, int m, int count, const double* d_in, double* d_out, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    const int product = which == 6 ? 2 : which >= 4;  // the kernel's mode
    const bool fp32 = which == 3 || which == 5;
#define RS_ST(M)                                                                                                   \
    case M:                                                                                                        \
        if (fp32)                                                                                                  \
            rs_selftest_kernel<M, float><<<count, 32, 0, stream>>>(product, count, d_in, d_out);                   \
        else                                                                                                       \
            rs_selftest_kernel<M, double><<<count, 32, 0, stream>>>(product, count, d_in, d_out);                  \
        break;
    switch (m) {
        RS_ST(1) RS_ST(2) RS_ST(3) RS_ST(4) RS_ST(5) RS_ST(6) RS_ST(7) RS_ST(8)
        RS_ST(9) RS_ST(10) RS_ST(11) RS_ST(12) RS_ST(13) RS_ST(14) RS_ST(15) RS_ST(16)
        default:
            return cudaErrorInvalidValue;
    }
#undef RS_ST
    return cudaGetLastError();
}

namespace {
template <int m>
cudaError_t launch_rs(int K, double gamma, const double* d_Ere, const double* d_Eim, const double* d_cre,
                      const double* d_cim, int num_e, int num_64, int num_neq, const RsParallel& par,
                      const double* d_Uatoms, double Uc0, double Uc1, const RsLeads& leads, void* d_corners,
                      void* d_gL, void* d_gLn, double* d_rows, double* d_Q, const double* d_sub, int* d_status,
                      cudaStream_t stream) {
    const int smem = (int)(2 * sizeof(cplxd) * pair_complex<m, false>());
    const int smem_neq = (int)(2 * sizeof(cplxd) * pair_complex<m, true>());
    cudaError_t e = cudaFuncSetAttribute(rs_pair_kernel<m, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(rs_pair_kernel<m, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_neq);
    if (e != cudaSuccess) return e;
    const int num_eq = num_e - num_neq, num_32 = num_eq - num_64;
    const cplxd* corners = static_cast<const cplxd*>(d_corners);
    cplxd* gX = static_cast<cplxd*>(d_gL);
    if (num_e > 0) {
        rs_lead_kernel<m><<<num_e, 32, 0, stream>>>(gamma, d_Ere, d_Eim, num_e, Uc0, Uc1, leads.use_decimation,
                                                    leads.dec_layers, leads.dec_iters, static_cast<cplxd*>(d_corners));
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    // the FP32 chains beside the FP64 ones
    const bool fork = num_32 > 0 && num_e > num_32;
    if (fork) {
        e = cudaEventRecord(par.fork, stream);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(par.side, par.fork, 0);
        if (e != cudaSuccess) return e;
    }
    // the longer chains first; the real-axis ones before the FP32 ones, whose blocks fit beside a whole
    // wave of them (512 points and 270 FP32 energies of a (10,0) tube: 944 us against 1277)
    if (num_neq > 0)
        rs_pair_kernel<m, true><<<num_neq, 64, smem_neq, stream>>>(K, gamma, d_Ere, d_Eim, d_cre, d_cim, num_eq, num_neq,
                                                                   d_Uatoms, corners, static_cast<cplxd*>(d_gLn),
                                                                   d_rows, d_status);
    if (num_32 > 0)
        rs_chain_kernel<m><<<num_32, 64, sizeof(cplxf) * chain_complex<m>(), fork ? par.side : stream>>>(
            K, gamma, d_Ere, d_Eim, d_cre, d_cim, num_64, num_32, d_Uatoms, corners, gX, d_rows, d_status);
    if (num_64 > 0)
        rs_pair_kernel<m, false><<<num_64, 64, smem, stream>>>(K, gamma, d_Ere, d_Eim, d_cre, d_cim, 0, num_64, d_Uatoms,
                                                               corners, gX, d_rows, d_status);
    e = cudaGetLastError();
    if (fork) {
        // joined also after a failed launch, so that a capture ends whole
        cudaError_t j = cudaEventRecord(par.join, par.side);
        if (j == cudaSuccess) j = cudaStreamWaitEvent(stream, par.join, 0);
        if (e == cudaSuccess) e = j;
    }
    if (e != cudaSuccess) return e;
    const int N = 2 * K;
    rs_reduce_kernel<<<(N + 31) / 32, dim3(32, kRsGroups), 0, stream>>>(d_rows, num_e, N, d_sub, d_Q);
    return cudaGetLastError();
}
}  // namespace

cudaError_t launch_realspace(int m, int K, double gamma, const double* d_Ere, const double* d_Eim,
                             const double* d_cre, const double* d_cim, int num_e, int num_64, int num_neq, const RsParallel& par,
                             const double* d_Uatoms, double Uc0, double Uc1, const RsLeads& leads,
                             void* d_corners, void* d_gL, void* d_gLn, double* d_rows, double* d_Q,
                             const double* d_sub, int* d_status, cudaStream_t stream) {
    if (num_64 < 0 || num_neq < 0 || num_64 + num_neq > num_e || K < 2) return cudaErrorInvalidValue;
#define RS_CASE(M)                                                                                                 \
    case M:                                                                                                        \
        return launch_rs<M>(K, gamma, d_Ere, d_Eim, d_cre, d_cim, num_e, num_64, num_neq, par, d_Uatoms, Uc0,      \
                            Uc1, leads, d_corners, d_gL, d_gLn, d_rows, d_Q, d_sub, d_status, stream);
    switch (m) {
        RS_CASE(1) RS_CASE(2) RS_CASE(3) RS_CASE(4) RS_CASE(5) RS_CASE(6) RS_CASE(7) RS_CASE(8)
        RS_CASE(9) RS_CASE(10) RS_CASE(11) RS_CASE(12) RS_CASE(13) RS_CASE(14) RS_CASE(15) RS_CASE(16)
        default:
            return cudaErrorInvalidValue;
    }
#undef RS_CASE
}

}  // namespace negf
