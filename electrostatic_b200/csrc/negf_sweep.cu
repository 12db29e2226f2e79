// FP64 mode-space passes on sm_100a: boundary states, then segments.
//
// Reference path replaced: Compute_RhoEq, Compute_GR_atPoles, Compute_Rho0 and
// Compute_RhoNonEq of Source/Solver/Transport/NEGF/NEGF_Common.cpp:3115-4092,
// and the per-energy recursions of Compute_DensityOfStates and
// Compute_Current (:2390-2847, :4321-4816).
//
// A chain is one (tube, mode, energy): a scalar complex recursion over N
// sites.  Everything below runs in units of the hopping gamma: a_n = (E -
// U_n) / gamma, rho_n = h_n^2 / gamma^2 = r = beta^2 / gamma^2 for even n and
// 1 for odd n (h_n joins sites n and n + 1; N is even).  The two recursions
//   y_{n+1} = rho_n / (a_n - y_n),      y_0     = Sigma_0 / gamma
//   x_{n-1} = rho_{n-1} / (a_n - x_n),  x_{N-1} = Sigma_1 / gamma
// carry the contacts as their initial values, so no site is special, and
// G_nn = 1 / (gamma (a_n - x_n - y_n)).  In projective form (y = p / q,
// x = R / s) a step is linear:
//   forward   q_{n+1} = a_n q_n - p_n,  p_{n+1} = rho_n q_n
//   backward  s_{n-1} = a_n s_n - R_n,  R_{n-1} = rho_{n-1} s_n
// and half of the products with rho are products with 1: 6 FP64 instructions
// a site on average, against 7 with both hoppings kept.  D = s_n q_{n+1} -
// R_n q_n is the same at every site of a segment (Wronskian) and
//   G_nn = q_n s_n / (gamma D),
//   |G_n0|^2   = lambda_n |G_nn|^2 = lambda_{n0} prod rho |s_n / D|^2 / gamma^2,
//   |G_n,N-1|^2 = rho_e prod rho |q_n / D|^2 / gamma^2
// with lambda_{n+1} = lambda_n rho_n / |a_n - y_n|^2 and its mirror image.
//
// Two phases.  First the boundary states (y, lambda) at the first site and
// (x, rho) at the last site of every K-site segment, by one of
//   sweep_kernel  lane = chain, one warp per 32 chains and direction: 6 FP64
//                 instructions a site, N dependent steps (many chains); or one
//                 per piece of the tube as well, behind range_kernel, which
//                 forms the pieces' transfer matrices (long tubes);
//   scan_kernel   thread = segment, one block per chain: the 2 x 2 transfer
//                 matrix of every segment, a scan over them in registers
//                 (parallel in length: few chains).
// Then seg_kernel: lane = segment, a warp loops over chains.  The site sums
// over the chains stay in the lane's registers, so no reduction over lanes
// and no per-chain traffic but the boundary states is left (the fused
// schedule of negf_rgf.cu spends 9 FP64 additions, 18 shuffles and 28 selects
// per 8 sites on the sum over the 32 chains of a warp).  Inside a segment the
// two recursions start from both ends and meet in the middle: the first
// halves are kept in registers, D comes out there, and the second halves form
// the site values as they go.
//
// The last segment of a tube whose N is not a multiple of K is [N - K, N): it
// overlaps its neighbour, whose sites it does not write.  Tubes of fewer than
// kSweepSeg sites use K = 2.

#include "negf_internal.h"

namespace negf {
namespace {

#include "negf_sgf.cuh"  // cd, sgf_analytic, sgf_decimation

constexpr unsigned kFull = 0xffffffffu;

// Reciprocal by the hardware approximation and the series 1/x = y (1 + e +
// e^2 + ...), e = 1 - x y, |e| <= 2^-20: relative error of order e^3.
__device__ __forceinline__ double rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ const GroupDev& group(const GroupSet& gs, int i) { return gs.ext ? gs.ext[i] : gs.g[i]; }

// Group of block b by the groups' first blocks (ascending): bisection over the
// parameters, which hold every stride-th one, then over the table between two of
// them (512 tubes of 120 sites, 1024 groups: 54 us a charge pass, 442 us with a walk
// of the table, 56 us by the warp tables of negf_rgf.cu).
template <int GroupDev::*Base>
__device__ __forceinline__ int find_group(const GroupSet& gs, const int (&base)[kMaxBases], int b) {
    int i = 0;
    for (int n = gs.nbases; n > 1;) {
        const int h = n / 2;
        if (b >= base[i + h]) i += h;
        n -= h;
    }
    i *= gs.stride;
    for (int n = min(gs.stride, gs.ng - i); n > 1;) {
        const int h = n / 2;
        if (b >= gs.ext[i + h].*Base) i += h;
        n -= h;
    }
    return i;
}

__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async16(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// waits until at most n groups are in flight
template <int n>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(n) : "memory");
}

// Boundary states in memory: blocks of 8 segments x 32 chains of one
// component, [chains / 32][segments / 8][component][32][8], the segment's
// place inside its 64 bytes swizzled by the chain.  A sweep warp (lane =
// chain) fills such blocks in shared memory without bank conflicts and stores
// them by one bulk copy; a seg_kernel warp (lane = segment) reads whole
// 64-byte pieces, the components at constant offsets.
constexpr int kBlk = 256;  // doubles of a block
template <int NC>
__device__ __forceinline__ long long state_at(const GroupDev& g, int c, int seg) {
    return g.ck_off + ((long long)(c >> 5) * g.nblk + (seg >> 3)) * (NC * kBlk) + (c & 31) * 8 + ((seg ^ c) & 7);
}

struct ChainIn {
    EnergyRec e;
    double beta, deg;
};
__device__ __forceinline__ ChainIn load_chain(const GroupDev& g, int c) {
    const int code = g.chains[c];
    ChainIn r;
    r.e = g.items[code >> kModeBits];
    const int mode = code & ((1 << kModeBits) - 1);
    r.beta = g.beta[mode];
    r.deg = g.degen[mode];
    return r;
}

// Self-energy of contact `side` in units of gamma: gamma g (Sigma = gamma^2 g,
// NEGF_Common.cpp:4165-4177).
__device__ __forceinline__ cd sigma_over_gamma(const GroupDev& g, const ChainIn& c, int side) {
    const double Uc = g.uc_from_U ? g.U[side ? g.N - 1 : 0] : (side ? g.Uc1 : g.Uc0);
    const cd EmU = {c.e.Er - Uc, c.e.Ei};
    const cd s = g.use_decimation ? sgf_decimation(EmU, c.beta, g.gamma, g.dec_layers, g.dec_iters)
                                  : sgf_analytic(EmU, c.beta, g.gamma);
    return cscale(g.gamma, s);
}

// Chain constants read by seg_kernel, kConst doubles per chain: E / gamma
// (2), r, the two real-axis weights (-2 Im Sigma_k b_k deg / gamma^2), then
// c deg / gamma (contour) or the two Gamma_k (real axis).  Side 0 writes the
// shared ones.
__device__ __forceinline__ void write_constants(const GroupDev& g, const ChainIn& c, cd sig, int side,
                                                double* __restrict__ o) {
    const double ig = 1.0 / g.gamma, gam = -2.0 * sig.y * g.gamma;
    const double w = gam * (side ? c.e.b1 : c.e.b0) * c.deg * ig * ig;
    if (side == 0) {
        o[0] = c.e.Er * ig;
        o[1] = c.e.Ei * ig;
        o[2] = c.beta * c.beta * ig * ig;
        o[3] = w;
        o[5] = g.kind == kRealAxis ? gam : c.e.cr * c.deg * ig;
    } else {
        o[4] = w;
        o[6] = g.kind == kRealAxis ? gam : c.e.ci * c.deg * ig;
    }
}

// One step of either direction; odd: the hopping behind the step is gamma
// (factor 1), else beta (factor r).
struct Lin {
    double pr, pi, qr, qi;
};
__device__ __forceinline__ void lin_step(Lin& s, double ar, double ai, double r, bool odd) {
    const double nqr = fma(ar, s.qr, fma(-ai, s.qi, -s.pr));
    const double nqi = fma(ar, s.qi, fma(ai, s.qr, -s.pi));
    s.pr = odd ? s.qr : r * s.qr;
    s.pi = odd ? s.qi : r * s.qi;
    s.qr = nqr;
    s.qi = nqi;
}

// ------------------------------------------------------------------ transfer matrices
// Transfer matrix of a run of sites, scaled to determinant 1 (by the
// square root of its product of rho, so that lambda needs no powers of r) and
// then to entries of order 1 by 2^-e:
//   forward  (p, q) <- [[-D, C], [-B, A]] (p, q),
//   backward (R, s) <- [[-D, B], [-C, A]] (R, s)  (the same continuants).
struct Tm {
    cd A, B, C, D;
    int e;
};
__device__ __forceinline__ cd cms(cd a, cd b, cd c) {  // a b - c
    return {fma(a.x, b.x, fma(-a.y, b.y, -c.x)), fma(a.x, b.y, fma(a.y, b.x, -c.y))};
}
__device__ __forceinline__ double pow2d(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
// A power of two f with f^2 x in [1/4, 2), from the exponent of x >= 0.
__device__ __forceinline__ double inv_root2(double x) {
    return __hiloint2double((int)((0xbfd00000u - (unsigned)__double2hiint(x)) >> 1 & 0x7ff00000u), 0);
}
// Returns the exponent taken out (0: none).
__device__ __forceinline__ int tm_normalise(Tm& m) {
    const double s = fmax(fmax(fabs(m.A.x) + fabs(m.A.y), fabs(m.B.x) + fabs(m.B.y)),
                          fmax(fabs(m.C.x) + fabs(m.C.y), fabs(m.D.x) + fabs(m.D.y)));
    const int be = (int)((__double_as_longlong(s) >> 52) & 0x7ff);
    if (be == 0 || be >= 0x7fe) return 0;  // zero, subnormal, inf or NaN: leave as is
    const double f = pow2d(1023 - be);
    m.A = cscale(f, m.A);
    m.B = cscale(f, m.B);
    m.C = cscale(f, m.C);
    m.D = cscale(f, m.D);
    m.e += be - 1023;
    return be - 1023;
}
// later o earlier: [[-D2, C2], [-B2, A2]] [[-D1, C1], [-B1, A1]].  drop: the least
// exponent of a result of normalised operands so far; a small one is what is left
// of larger terms.
__device__ __forceinline__ Tm tm_mul(const Tm& m2, const Tm& m1, int& drop) {
    Tm o;
    o.D = cms(m2.C, m1.B, cmul(m2.D, m1.D));
    o.C = cms(m2.C, m1.A, cmul(m2.D, m1.C));
    o.B = cms(m2.A, m1.B, cmul(m2.B, m1.D));
    o.A = cms(m2.A, m1.A, cmul(m2.B, m1.C));
    o.e = m1.e + m2.e;
    drop = min(drop, tm_normalise(o));
    return o;
}
__device__ __forceinline__ Tm tm_identity() { return Tm{{1.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {-1.0, 0.0}, 0}; }
// State (Z, 1) with lambda through m: Z = (-D Z + K1) / (-K2 Z + A), (K1, K2) = (C, B) forward, (B, C) backward
__device__ __forceinline__ void tm_apply(const Tm& m, bool back, cd& Z, double& lam, int& drop) {
    const cd k1 = back ? m.B : m.C, k2 = back ? m.C : m.B;
    const cd num = {fma(-m.D.x, Z.x, fma(m.D.y, Z.y, k1.x)), fma(-m.D.x, Z.y, fma(-m.D.y, Z.x, k1.y))};
    const cd den = {fma(-k2.x, Z.x, fma(k2.y, Z.y, m.A.x)), fma(-k2.x, Z.y, fma(-k2.y, Z.x, m.A.y))};
    auto hi = [](cd z) { return max(__double2hiint(z.x) & 0x7fffffff, __double2hiint(z.y) & 0x7fffffff) >> 20; };
    drop = min(drop, max(hi(num), hi(den)) - max(hi(Z), 1023));
    const double iq = rcp(fma(den.x, den.x, den.y * den.y));
    Z = {fma(num.x, den.x, num.y * den.y) * iq, fma(num.y, den.x, -num.x * den.y) * iq};
    lam *= iq;
    const int e2 = -2 * m.e;  // lambda 2^(-2 e), in two factors inside the exponent range
    const int h = max(-1000, min(1000, e2 / 2)), h2 = max(-1000, min(1000, e2 - e2 / 2));
    lam *= pow2d(h);
    lam *= pow2d(h2);
}

// Pieces of a group's chains (pieces > 1): [chains / 32][piece][9][32] matrices,
// then [2][2][32] contact self-energies.
__device__ __forceinline__ long long tm_at(const GroupDev& g, int w, int piece) {
    return g.tm_off + ((long long)w * (g.pieces * 9 + 4) + piece * 9) * 32;
}
// The state before a piece: the contact's through the n pieces between, their
// matrices in a ring of kCarry shared stages (an L2 latency from load to use).  The
// state stays a pair (P, Q), scaled by the exponent of the pair before, so that an
// application is a chain of four FMAs and a product; one division at the end.
constexpr int kCarry = 8, kCarryStage = 9 * 32;
template <bool BACK, bool RA>
__device__ __forceinline__ void carry(const GroupDev& g, int w, int n, const double* __restrict__ tm, cd& Z,
                                      double& lam) {
    extern __shared__ __align__(16) double carry_ring[];
    const int lane = threadIdx.x;
    auto copy = [&](int j) {
        if (j < n) {
            const double* src = tm + tm_at(g, w, BACK ? g.pieces - 1 - j : j) + 2 * lane;
            double* dst = carry_ring + j % kCarry * kCarryStage + 2 * lane;
#pragma unroll
            for (int q = 0; q < 4; ++q) cp_async16(dst + 64 * q, src + 64 * q);
            if (lane < 16) cp_async16(dst + 256, src + 256);
        }
        cp_async_commit();
    };
    for (int j = 0; j < kCarry; ++j) copy(j);
    const double* sig = tm + tm_at(g, w, g.pieces) + (BACK ? 64 : 0) + lane;
    cd P = {sig[0], sig[32]}, Q = {1.0, 0.0};
    auto exponent = [&]() {  // of the larger of P and Q, 0 when there is none
        auto hi = [](double x) { return __double2hiint(x) & 0x7fffffff; };
        const int be = max(max(hi(P.x), hi(P.y)), max(hi(Q.x), hi(Q.y))) >> 20;
        return be > 0 && be < 0x7fe ? be - 1023 : 0;
    };
    int e = 0;  // the pair times 2^e
    for (int j = 0; j < n; ++j) {
        cp_async_wait<kCarry - 1>();
        __syncwarp();
        const double* q = carry_ring + j % kCarry * kCarryStage + lane;
        const cd A = {q[0], q[32]}, D = {q[192], q[224]};
        const cd k1 = BACK ? cd{q[64], q[96]} : cd{q[128], q[160]}, k2 = BACK ? cd{q[128], q[160]} : cd{q[64], q[96]};
        const int x = exponent();
        const double f = pow2d(-x);
        e += x + (int)q[256];
        const cd p = cms(k1, Q, cmul(D, P)), d = cms(A, Q, cmul(k2, P));
        P = cscale(f, p);
        Q = cscale(f, d);
        __syncwarp();
        copy(j + kCarry);
    }
    cp_async_wait<0>();
    const int x = exponent();
    P = cscale(pow2d(-x), P);
    Q = cscale(pow2d(-x), Q);
    const double iq = rcp(fma(Q.x, Q.x, Q.y * Q.y));
    Z = {fma(P.x, Q.x, P.y * Q.y) * iq, fma(P.y, Q.x, -P.x * Q.y) * iq};
    // lambda = 2^(-2 e) / |Q|^2, the power in two factors inside the exponent range
    const int e2 = -2 * (e + x), h = max(-1000, min(1000, e2 / 2)), h2 = max(-1000, min(1000, e2 - e2 / 2));
    lam = RA ? iq * pow2d(h) * pow2d(h2) : 1.0;
}

// ------------------------------------------------------------------ boundary states: sweeps
// A warp sweeps 32 chains of one group in one direction (even block: forward,
// odd: backward), stores the normalised state of every segment boundary in a
// shared tile of 8 segments and writes full 64-byte pieces of the chains' rows
// [component][segment], the layout that seg_kernel reads with lane = segment.
// Bound: 7 FP64 instructions a site and chain (6 of the step, 1 of the
// boundary); one direction per warp doubles the warps of the pass (the
// dependent chain of a step is two FMAs, 16 cycles against 12 issue cycles,
// so it takes two or more warps per scheduler to fill the FP64 pipe).
// The potentials travel through a shared ring of four tiles of 64 steps
// (cp.async, one 16-byte pair of sites per lane and tile), since ptxas moves
// loads into registers to their use: a lone warp then took 63 cycles a site.
constexpr int kRing = 256, kTile = 64;
struct __align__(128) SweepShared {
    double tile[3 * kBlk];
    double ring[kRing];
};
// Bulk copy of shared memory to global memory (16-byte aligned, a multiple of
// 16 bytes) by one lane, after the other lanes' writes were made visible to
// the async proxy; bulk_read_done: the shared source may be rewritten.
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void bulk_store(double* dst, const double* src, unsigned bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                 "r"((unsigned)__cvta_generic_to_shared(src)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_read_done() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_done() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

template <int K, bool BACK, bool RA>
__device__ __forceinline__ void sweep_chain(const GroupDev& g, int w, int piece, SweepShared& sm,
                                            double* __restrict__ ck, double* __restrict__ cc,
                                            const double* __restrict__ tm) {
    constexpr int NC = RA ? 6 : 4, ROWS = NC / 2;
    const int lane = threadIdx.x;
    const int N = g.N, nseg = g.nseg, nblk = g.nblk;
    const int c = min(w * kWarp + lane, g.nch - 1);
    const double* __restrict__ U = g.U;
    const int tail = N - (nseg - 1) * K;  // sites of the natural last segment, in [2, K]
    const bool cut = tail < K;
    // Step m of a sweep: forward at site m, backward at site N - 1 - m (the parities agree since N is
    // even).  Position m + off of the ring holds it, pairs of steps in site order; off makes every full
    // segment start at a multiple of K, so that its loads have constant offsets.
    const int off = BACK && cut ? K - tail : 0;
    auto fetch = [&](int t) {
        const int p = t * kTile + 2 * lane, m = p - off;
        if (m >= 0 && m < N) cp_async16(&sm.ring[p & (kRing - 1)], U + (BACK ? N - 2 - m : m));
        cp_async_commit();
    };
    // this piece: segments [s_lo, s_hi), from the contact or from the pieces before it
    const int W = g.pieces, s_lo = piece * g.piece_segs;
    const bool last = piece == W - 1;
    const int s_hi = last ? nseg : s_lo + g.piece_segs;
    int pos = BACK ? (last ? off : (nseg - s_hi) * K) : s_lo * K, tile = pos / kTile;
    for (int t = 0; t < 3; ++t) fetch(tile + t);
    const ChainIn ch = load_chain(g, c);
    cd start;
    double lam = 1.0;
    if (W > 1) {
        carry<BACK, RA>(g, w, BACK ? W - 1 - piece : piece, tm, start, lam);
    } else {
        start = sigma_over_gamma(g, ch, BACK);
        if (w * kWarp + lane < g.nch) write_constants(g, ch, start, BACK, cc + g.cc_off + (long long)c * kConst);
    }
    const double ig = 1.0 / g.gamma, Eg = ch.e.Er * ig, ei = ch.e.Ei * ig, r = ch.beta * ch.beta * ig * ig;
    double* __restrict__ out = ck + g.ck_off + ((long long)w * nblk * NC + (BACK ? ROWS : 0)) * kBlk;
    Lin s{start.x, start.y, 1.0, 0.0};
    // The record (p / q, lambda) of a boundary is formed beside the first half of the next segment's
    // steps and the running state is scaled by f, a power of two next to 1 / |q_b|, after them: issue is
    // in order, so a record formed at the boundary itself would hold up the recurrence for its whole
    // chain.  The moduli telescope to lambda_b = mu_b / |q_b|^2, mu_{b+1} = mu_b f_b^2 prod(rho).
    // (Scaled by 1 / |q_b|^2, a step would take |q_b| to G_b / |q_b|: standing waves of the period of two
    // segments, G_b large and small by turns, then grow it without bound, to inf after some 100 of them: 396 us for 33 488 chains of 4000
    // sites, 400 us so.)
    double f = 1.0, mu = lam, yr, yi;
    auto record = [&](const Lin& t, double rprod) {
        const double q2 = fma(t.qr, t.qr, t.qi * t.qi), q1 = rcp(q2);
        yr = fma(t.pr, t.qr, t.pi * t.qi) * q1;
        yi = fma(t.pi, t.qr, -t.pr * t.qi) * q1;
        f = inv_root2(q2);
        if (RA) {
            mu *= rprod;
            lam = mu * q1;
            mu *= f;
            mu *= f;
        }
    };
    auto scale = [&]() {
        s.pr *= f;
        s.pi *= f;
        s.qr *= f;
        s.qi *= f;
    };
    bool first = true;  // the tile's first segment: the bulk copy of the previous tile must have read it
    auto store = [&](int seg) {
        if (first) {
            if (lane == 0) bulk_read_done();
            __syncwarp();
            first = false;
        }
        double* t = sm.tile + lane * 8 + ((seg ^ lane) & 7);
        t[0] = yr;
        t[kBlk] = yi;
        if (RA) t[2 * kBlk] = lam;
        if (BACK ? (seg & 7) == 0 : ((seg & 7) == 7 || seg == nseg - 1)) {
            fence_async_proxy();
            __syncwarp();
            if (lane == 0) bulk_store(out + (long long)(seg >> 3) * (NC * kBlk), sm.tile, ROWS * kBlk * sizeof(double));
            first = true;
        }
    };
    // tiles T and T + 1 are complete while the sweep is in tile T
    auto enter = [&]() {
        if (pos / kTile > tile) {
            tile = pos / kTile;
            __syncwarp();  // every lane has left the tile whose slot is filled next
            fetch(tile + 2);
            cp_async_wait<1>();
            __syncwarp();
        }
    };
    cp_async_wait<1>();
    __syncwarp();
    double rseg = 1.0;  // product of rho over a full segment
#pragma unroll
    for (int j = 0; j < K / 2; ++j) rseg *= r;
    // a of the two steps at position p
    auto pair = [&](int p) {
        const double2 v = *reinterpret_cast<const double2*>(&sm.ring[p & (kRing - 1)]);
        return make_double2(fma(BACK ? -v.y : -v.x, ig, Eg), fma(BACK ? -v.x : -v.y, ig, Eg));
    };
    double rprod = 1.0;  // product of rho since the previous boundary
    // the shortened step to (forward) or from (backward) the last segment
    auto shorter = [&]() {
        enter();
        record(s, rprod);
        scale();
        rprod = 1.0;
        for (int j = 0; j < tail; j += 2) {
            const double2 a = pair(pos + j);
            lin_step(s, a.x, ei, r, false);
            lin_step(s, a.y, ei, r, true);
            rprod *= r;
        }
        pos += tail;
    };
    int seg = BACK ? s_hi - 1 : s_lo;
    const bool end = cut && last;
    if (BACK && end) {
        shorter();
        store(seg--);
    }
    double2 a = pair(pos);  // one pair ahead
    for (int k = s_hi - s_lo - 1 - (end ? 1 : 0); k > 0; --k) {
        enter();
        const Lin t = s;
        const double* at = &sm.ring[pos & (kRing - 1)];
        auto two = [&](int j) {
            const double2 v = *reinterpret_cast<const double2*>(j + 2 < K ? at + j + 2 : &sm.ring[(pos + K) & (kRing - 1)]);
            lin_step(s, a.x, ei, r, false);
            lin_step(s, a.y, ei, r, true);
            a = make_double2(fma(BACK ? -v.y : -v.x, ig, Eg), fma(BACK ? -v.x : -v.y, ig, Eg));
        };
#pragma unroll
        for (int j = 0; j < K / 2; j += 2) two(j);
        record(t, rprod);
        scale();
#pragma unroll
        for (int j = (K / 2 + 1) / 2 * 2; j < K; j += 2) two(j);
        store(seg);
        rprod = rseg;
        pos += K;
        seg += BACK ? -1 : 1;
    }
    if (!BACK && end) {  // from (nseg - 2) K to N - K
        shorter();
        store(seg++);
    }
    record(s, rprod);
    store(seg);
    cp_async_wait<0>();
    if (lane == 0) bulk_done();  // the copies read this block's shared memory
}

template <int K>
__global__ void __launch_bounds__(32, 16) sweep_kernel(const __grid_constant__ GroupSet gs, double* __restrict__ ck,
                                                       double* __restrict__ cc, const double* __restrict__ tm,
                                                       const int* __restrict__ skip) {
    if (skip && *skip) return;
    __shared__ __align__(16) SweepShared sm;
    const GroupDev& g = group(gs, find_group<&GroupDev::sweep_base>(gs, gs.sweep_base, blockIdx.x));
    const int rel = blockIdx.x - g.sweep_base, w = (rel >> 1) / g.pieces, piece = (rel >> 1) % g.pieces;
    if (g.kind == kRealAxis) {
        if (rel & 1)
            sweep_chain<K, true, true>(g, w, piece, sm, ck, cc, tm);
        else
            sweep_chain<K, false, true>(g, w, piece, sm, ck, cc, tm);
    } else {
        if (rel & 1)
            sweep_chain<K, true, false>(g, w, piece, sm, ck, cc, tm);
        else
            sweep_chain<K, false, false>(g, w, piece, sm, ck, cc, tm);
    }
}

// ------------------------------------------------------------------ boundary states: sweeps in pieces
// Transfer matrix of one piece (lane = chain, a warp per 32 chains and piece): two
// columns a site, 11 FP64 instructions, normalised at every segment with its part
// of the determinant.  Two more warps form the contact self-energies and the
// chain constants.  Bound by the steps of a piece, 12 ns a site, behind 4 us of
// start.  64000 sites and 230 chains: 20 us and 40 us of sweeps in pieces, against
// 153 us of scan_kernel and 1120 us of whole sweeps.
template <int K>
__global__ void __launch_bounds__(32, 16) range_kernel(const __grid_constant__ GroupSet gs, double* __restrict__ cc,
                                                       double* __restrict__ tm, const int* __restrict__ skip) {
    if (skip && *skip) return;
    __shared__ __align__(16) double ring[kRing];
    const GroupDev& g = group(gs, find_group<&GroupDev::range_base>(gs, gs.range_base, blockIdx.x));
    const int rel = blockIdx.x - g.range_base, w = rel / (g.pieces + 2), piece = rel % (g.pieces + 2);
    const int lane = threadIdx.x, N = g.N, c = min(w * kWarp + lane, g.nch - 1);
    const int s_lo = piece * g.piece_segs, s_hi = piece == g.pieces - 1 ? g.nseg : s_lo + g.piece_segs;
    const ChainIn ch = load_chain(g, c);
    if (piece >= g.pieces) {  // contact self-energies and chain constants, beside the matrices
        const int side = piece - g.pieces;
        const cd sig = sigma_over_gamma(g, ch, side);
        if (w * kWarp + lane < g.nch) write_constants(g, ch, sig, side, cc + g.cc_off + (long long)c * kConst);
        double* o = tm + tm_at(g, w, g.pieces) + 64 * side + lane;
        o[0] = sig.x;
        o[32] = sig.y;
        return;
    }
    auto fetch = [&](int t) {
        const int p = t * kTile + 2 * lane;
        if (p < N) cp_async16(&ring[p & (kRing - 1)], g.U + p);
        cp_async_commit();
    };
    int tile = s_lo * K / kTile;
    for (int t = 0; t < 3; ++t) fetch(tile + t);
    const double ig = 1.0 / g.gamma, Eg = ch.e.Er * ig, ei = ch.e.Ei * ig, r = ch.beta * ch.beta * ig * ig;
    // r^(-1/2), bounded: a vanishing beta decouples the sites and its lambda is 0 to working precision;
    // its power over a segment as mantissa and exponent
    const double hs = 1.0 / fmax(fabs(ch.beta) * ig, 1e-30);
    auto part = [&](int len, double& mant, int& ex) {
        double f = 1.0;
        for (int j = 0; j < len / 2; ++j) f *= hs;
        const long long b = __double_as_longlong(f);
        ex = (int)((b >> 52) & 0x7ff) - 1023;
        mant = __longlong_as_double((b & 0xfffffffffffffll) | (1023ll << 52));
    };
    double mant;
    int ex, e = 0;
    part(K, mant, ex);
    Lin c1{1.0, 0.0, 0.0, 0.0}, c2{0.0, 0.0, 1.0, 0.0};
    auto normalise = [&]() {
        auto hi = [](double x) { return __double2hiint(x) & 0x7fffffff; };
        const int be = max(max(max(hi(c1.pr), hi(c1.pi)), max(hi(c1.qr), hi(c1.qi))),
                           max(max(hi(c2.pr), hi(c2.pi)), max(hi(c2.qr), hi(c2.qi)))) >> 20;
        const bool scale = be > 0 && be < 0x7fe;  // else zero, subnormal, inf or NaN: leave as is
        const double f = scale ? mant * pow2d(1023 - be) : mant;
        e += ex + (scale ? be - 1023 : 0);
        c1 = {c1.pr * f, c1.pi * f, c1.qr * f, c1.qi * f};
        c2 = {c2.pr * f, c2.pi * f, c2.qr * f, c2.qi * f};
    };
    cp_async_wait<1>();
    __syncwarp();
    for (int s = s_lo; s < s_hi; ++s) {
        const int n0 = s * K;
        if (n0 / kTile > tile) {
            tile = n0 / kTile;
            __syncwarp();  // every lane has left the tile whose slot is filled next
            fetch(tile + 2);
            cp_async_wait<1>();
            __syncwarp();
        }
        const double* at = &ring[n0 & (kRing - 1)];
        auto two = [&](int j) {
            const double2 v = *reinterpret_cast<const double2*>(at + j);
            const double a0 = fma(-v.x, ig, Eg), a1 = fma(-v.y, ig, Eg);
            lin_step(c1, a0, ei, r, false);
            lin_step(c2, a0, ei, r, false);
            lin_step(c1, a1, ei, r, true);
            lin_step(c2, a1, ei, r, true);
        };
        if (n0 + K <= N) {
#pragma unroll
            for (int j = 0; j < K; j += 2) two(j);
        } else {
            for (int j = 0; j < N - n0; j += 2) two(j);
            part(N - n0, mant, ex);
        }
        normalise();
    }
    cp_async_wait<0>();
    const double v[9] = {c2.qr, c2.qi, -c1.qr, -c1.qi, c2.pr, c2.pi, -c1.pr, -c1.pi, (double)e};
    double* o = tm + tm_at(g, w, piece) + lane;
#pragma unroll
    for (int k = 0; k < 9; ++k) o[32 * k] = v[k];
}

// ------------------------------------------------------------------ boundary states: scan over segments
__device__ __forceinline__ Tm tm_shfl(const Tm& m, int src) {
    Tm o;
    o.A = {__shfl_sync(kFull, m.A.x, src), __shfl_sync(kFull, m.A.y, src)};
    o.B = {__shfl_sync(kFull, m.B.x, src), __shfl_sync(kFull, m.B.y, src)};
    o.C = {__shfl_sync(kFull, m.C.x, src), __shfl_sync(kFull, m.C.y, src)};
    o.D = {__shfl_sync(kFull, m.D.x, src), __shfl_sync(kFull, m.D.y, src)};
    o.e = __shfl_sync(kFull, m.e, src);
    return o;
}
constexpr int kScanMaxThreads = 512;

template <int K>
__device__ __forceinline__ Tm seg_matrix(const double* __restrict__ U, int n0, int len, double ig, double Eg, double ei,
                                         double r, double hs) {
    // columns from (1, 0) and (0, 1); the a_n are shared: 11 FP64 instructions a site
    Lin c1{1.0, 0.0, 0.0, 0.0}, c2{0.0, 0.0, 1.0, 0.0};
    if (len == K) {
        double u[K];
#pragma unroll
        for (int j = 0; j < K; j += 2) {
            const double2 v = __ldg(reinterpret_cast<const double2*>(U + n0 + j));
            u[j] = v.x;
            u[j + 1] = v.y;
        }
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const double ar = fma(-u[j], ig, Eg);
            lin_step(c1, ar, ei, r, j & 1);
            lin_step(c2, ar, ei, r, j & 1);
        }
    } else {
        for (int j = 0; j < len; ++j) {
            const double ar = fma(-__ldg(U + n0 + j), ig, Eg);
            lin_step(c1, ar, ei, r, j & 1);
            lin_step(c2, ar, ei, r, j & 1);
        }
    }
    Tm m;
    m.D = {-c1.pr, -c1.pi};
    m.B = {-c1.qr, -c1.qi};
    m.C = {c2.pr, c2.pi};
    m.A = {c2.qr, c2.qi};
    m.e = 0;
    tm_normalise(m);
    // determinant 1: product of rho = r^(len/2), hs = r^(-1/2)
    double f = 1.0;
    for (int j = 0; j < len / 2; ++j) f *= hs;
    m.A = cscale(f, m.A);
    m.B = cscale(f, m.B);
    m.C = cscale(f, m.C);
    m.D = cscale(f, m.D);
    tm_normalise(m);
    return m;
}

// One chain's boundary states by sweeps, for the chains whose scan loses digits:
// lane 0 forward, lane 1 backward (the same steps), potentials staged by the block.
// 30 ns a site.
constexpr int kStage = 256;
template <int K>
__device__ __noinline__ void sweep_states(const GroupDev& g, int c, double* __restrict__ ck, const cd* sig, double Eg,
                                          double ei, double ig, double r, double (*stage)[kStage]) {
    const bool ra = g.kind == kRealAxis, back = threadIdx.x == 1;
    const int N = g.N, nseg = g.nseg;
    Lin s{sig[back].x, sig[back].y, 1.0, 0.0};
    double mu = 1.0, h = 1.0;  // mu = lambda |q|^2, h: product of rho since the last boundary
    for (int m0 = 0; m0 < N; m0 += kStage) {
        const int len = min(kStage, N - m0);
        __syncthreads();
        for (int i = threadIdx.x; i < len; i += blockDim.x) {
            stage[0][i] = g.U[m0 + i];
            stage[1][i] = g.U[N - 1 - m0 - i];
        }
        __syncthreads();
        if (threadIdx.x > 1) continue;
        for (int i = 0; i < len; ++i) {
            const int m = m0 + i, n = back ? N - 1 - m : m;
            // boundaries: the first site of a segment forward, its last one backward
            int seg = -1;
            if (back)
                seg = n == N - 1 ? nseg - 1 : (n + 1) % K == 0 && n / K < nseg - 1 ? n / K : -1;
            else
                seg = n == N - K ? nseg - 1 : n % K == 0 && n < N - K ? n / K : -1;
            if (seg >= 0) {
                const double q2 = fma(s.qr, s.qr, s.qi * s.qi), q1 = rcp(q2), f = inv_root2(q2);
                double* o = ck + (ra ? state_at<6>(g, c, seg) : state_at<4>(g, c, seg)) +
                            (back ? (ra ? 3 : 2) : 0) * kBlk;
                mu *= h;
                h = 1.0;
                o[0] = fma(s.pr, s.qr, s.pi * s.qi) * q1;
                o[kBlk] = fma(s.pi, s.qr, -s.pr * s.qi) * q1;
                if (ra) o[2 * kBlk] = mu * q1;
                mu = mu * f * f;
                s = {s.pr * f, s.pi * f, s.qr * f, s.qi * f};
            }
            const bool odd = m & 1;
            lin_step(s, fma(-stage[back][i], ig, Eg), ei, r, odd);
            if (!odd) h *= r;
        }
    }
}

// One block per chain.  Thread t owns segments [t gper, (t + 1) gper): their
// matrices (kept in `tm` when gper > 1), their product, an inclusive scan over
// the warp in both directions by shuffles, the warps' totals through shared
// memory, then the boundary states of its own segments.  A product of
// matrices, or one with a state, that comes out small against its factors (2^kDrop:
// an evanescent wave that decays, a resonance) has lost as many digits; its chain
// is swept instead, at 30 ns a site.  (Periodic potentials at Im E = 2e-6: charges off
// by 1e-7 of their largest value without this, by 1e-11 with it.  Chains of the
// benchmark's potentials come down to 2^-6.)
constexpr int kDrop = -8;
template <int K>
__global__ void __launch_bounds__(kScanMaxThreads) scan_kernel(const __grid_constant__ GroupSet gs,
                                                               double* __restrict__ ck, double* __restrict__ cc,
                                                               double* __restrict__ tm,
                                                               const int* __restrict__ skip) {
    if (skip && *skip) return;
    __shared__ Tm tot[kScanMaxThreads / 32];
    __shared__ cd sh_sig[2];
    __shared__ double stage[2][kStage];
    const GroupDev& g = group(gs, find_group<&GroupDev::chain_base>(gs, gs.chain_base, blockIdx.x));
    const int c = blockIdx.x - g.chain_base;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5, W = blockDim.x >> 5;
    const int N = g.N, nseg = g.nseg, gper = (nseg + blockDim.x - 1) / blockDim.x;
    const bool ra = g.kind == kRealAxis;
    const ChainIn ch = load_chain(g, c);
    if (t < 2) {
        const cd sig = sigma_over_gamma(g, ch, t);
        sh_sig[t] = sig;
        write_constants(g, ch, sig, t, cc + g.cc_off + (long long)c * kConst);
    }
    const double ig = 1.0 / g.gamma, Eg = ch.e.Er * ig, ei = ch.e.Ei * ig, r = ch.beta * ch.beta * ig * ig;
    // r^(-1/2), bounded: a vanishing beta decouples the sites and its lambda is 0 to working precision
    const double hs = 1.0 / fmax(fabs(ch.beta) * ig, 1e-30);
    const double* __restrict__ U = g.U;
    const int s0 = min(t * gper, nseg), s1 = min(s0 + gper, nseg);
    double* __restrict__ mine = tm + ((long long)blockIdx.x * g.tm_segs) * 9;
    int drop = 0;
    Tm own = tm_identity(), first = own;
    for (int s = s0; s < s1; ++s) {
        const Tm m = seg_matrix<K>(U, s * K, min(K, N - s * K), ig, Eg, ei, r, hs);
        if (gper > 1) {
            const double v[9] = {m.A.x, m.A.y, m.B.x, m.B.y, m.C.x, m.C.y, m.D.x, m.D.y, (double)m.e};
#pragma unroll
            for (int k = 0; k < 9; ++k) mine[(long long)k * g.tm_segs + s] = v[k];
        } else {
            first = m;
        }
        own = s == s0 ? m : tm_mul(m, own, drop);
    }
    Tm pre = own, suf = own;  // inclusive products: pre over lanes <= mine, suf over lanes >= mine
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const Tm a = tm_shfl(pre, max(lane - d, 0)), b = tm_shfl(suf, min(lane + d, 31));
        if (lane >= d) pre = tm_mul(pre, a, drop);
        if (lane + d < 32) suf = tm_mul(b, suf, drop);
    }
    if (lane == 31) tot[wid] = pre;
    Tm ex = tm_shfl(pre, max(lane - 1, 0)), sx = tm_shfl(suf, min(lane + 1, 31));
    if (lane == 0) ex = tm_identity();
    if (lane == 31) sx = tm_identity();
    __syncthreads();
    cd Y = sh_sig[0], X = sh_sig[1];
    double lam = 1.0, rho = 1.0;
    for (int w = 0; w < wid; ++w) tm_apply(tot[w], false, Y, lam, drop);
    for (int w = W - 1; w > wid; --w) tm_apply(tot[w], true, X, rho, drop);
    tm_apply(ex, false, Y, lam, drop);
    tm_apply(sx, true, X, rho, drop);
    auto load = [&](int s) {
        if (gper == 1) return first;
        const double* q = mine + s;
        const long long st = g.tm_segs;
        return Tm{{q[0], q[st]}, {q[2 * st], q[3 * st]}, {q[4 * st], q[5 * st]}, {q[6 * st], q[7 * st]}, (int)q[8 * st]};
    };
    auto put = [&](int s, int comp, cd z, double l) {
        double* o = ck + (ra ? state_at<6>(g, c, s) : state_at<4>(g, c, s)) + comp * kBlk;
        o[0] = z.x;
        o[kBlk] = z.y;
        if (ra) o[2 * kBlk] = l;
    };
    auto put_y = [&](int s, cd y, double l) { put(s, 0, y, l); };
    const int tail = N - (nseg - 1) * K;
    for (int s = s0; s < s1; ++s) {
        if (s < nseg - 1 || tail == K) put_y(s, Y, lam);
        if (s == nseg - 2 && tail < K) {  // the last segment starts at N - K
            Lin q{Y.x, Y.y, 1.0, 0.0};
            double rp = 1.0;
            for (int j = 0; j < tail; ++j) {
                lin_step(q, fma(-__ldg(U + s * K + j), ig, Eg), ei, r, j & 1);
                if (!(j & 1)) rp *= r;
            }
            const double rq = rcp(fma(q.qr, q.qr, q.qi * q.qi));
            put_y(nseg - 1, {fma(q.pr, q.qr, q.pi * q.qi) * rq, fma(q.pi, q.qr, -q.pr * q.qi) * rq}, lam * rp * rq);
        }
        if (s + 1 < s1) tm_apply(load(s), false, Y, lam, drop);
    }
    for (int s = s1 - 1; s >= s0; --s) {
        put(s, ra ? 3 : 2, X, rho);
        if (s > s0) tm_apply(load(s), true, X, rho, drop);
    }
    if (__syncthreads_or(drop < kDrop)) sweep_states<K>(g, c, ck, sh_sig, Eg, ei, ig, r, stage);
}

// ------------------------------------------------------------------ segments
// Boundary states and constants of one chain at this lane's segment.
struct SegIn {
    double yr, yi, lam, xr, xi, rho;
    double Eg, ei, r, k0, k1, c0, c1;
};
// A warp's chains travel through a ring of kStages shared stages filled by
// cp.async (8 bytes per lane and component, 16-byte pieces of the constants):
// the next chains' boundary states arrive from DRAM while this chain is
// computed without holding registers.  (Loaded into registers one chain
// ahead, the compiler moves the loads to their use: half of the cycles were
// long-scoreboard stalls.)
constexpr int kStages = 3;
struct SegStage {
    double rec[6][32];
    double con[32][kConst];
};
// One chain's K-site segment; u(p): U / gamma of sites 2 p and 2 p + 1;
// site(j, a, x, b, y) receives for every site two
// products a x and b y: on the real axis the source and the drain term (k0
// lambda |G|^2 and k1 rho |G|^2), on the contour the two whose sum is Im(c G_nn).
template <int K, bool RA, class P, class F>
__device__ __forceinline__ void segment(const SegIn& v, P&& u, F&& site) {
    constexpr int H = K / 2;
    Lin f{v.yr, v.yi, 1.0, 0.0}, b{v.xr, v.xi, 1.0, 0.0};
    // first halves: sites 0 .. H-1 forward, K-1 .. H backward (steps of equal parity run side by side)
    double fr[H], fi[H], br[H], bi[H];  // real axis: fr = |q|^2, br = |s|^2; contour: q and s
    double2 uf, ub;  // potentials of the current pair of sites, forward and backward
#pragma unroll
    for (int i = 0; i < H; ++i) {
        if (RA) {
            fr[i] = fma(f.qr, f.qr, f.qi * f.qi);
            br[i] = fma(b.qr, b.qr, b.qi * b.qi);
        } else {
            fr[i] = f.qr;
            fi[i] = f.qi;
            br[i] = b.qr;
            bi[i] = b.qi;
        }
        if (!(i & 1)) {
            uf = u(i / 2);
            ub = u((K - 1 - i) / 2);
        }
        lin_step(f, v.Eg - (i & 1 ? uf.y : uf.x), v.ei, v.r, i & 1);
        lin_step(b, v.Eg - (i & 1 ? ub.x : ub.y), v.ei, v.r, i & 1);
    }
    // D = s_{H-1} q_H - R_{H-1} q_{H-1}; for even H the hopping between the
    // halves is gamma, so p_H = q_{H-1}; for H = 1, q_0 = 1
    double dr, di;
    if (H % 2 == 0) {
        dr = fma(b.qr, f.qr, fma(-b.qi, f.qi, fma(-b.pr, f.pr, b.pi * f.pi)));
        di = fma(b.qr, f.qi, fma(b.qi, f.qr, fma(-b.pr, f.pi, -b.pi * f.pr)));
    } else {
        static_assert(H % 2 == 0 || H == 1, "K is 2 or a multiple of 4");
        dr = fma(b.qr, f.qr, fma(-b.qi, f.qi, -b.pr));
        di = fma(b.qr, f.qi, fma(b.qi, f.qr, -b.pi));
    }
    const double inv = rcp(fma(dr, dr, di * di));
    // second halves, step i: forward from site H + i, backward from site H - 1 - i
    auto next = [&](int i) {
        if (!(i & 1)) {
            uf = u((H + i) / 2);
            ub = u((H - 1 - i) / 2);
        }
        lin_step(f, v.Eg - (i & 1 ? uf.y : uf.x), v.ei, v.r, i & 1);
        lin_step(b, v.Eg - (i & 1 ? ub.x : ub.y), v.ei, v.r, i & 1);
    };
    if (RA) {
        // weights of |s_j|^2: A r^ceil(j/2); of |q_j|^2: B r^floor((K-j)/2)
        double A[H / 2 + 1], B[H / 2 + 1];
        A[0] = v.lam * v.k0 * inv;
        B[0] = v.rho * v.k1 * inv;
#pragma unroll
        for (int k = 1; k <= H / 2; ++k) {
            A[k] = A[k - 1] * v.r;
            B[k] = B[k - 1] * v.r;
        }
        double ah = A[H / 2], bh = B[H / 2];  // running powers past the middle
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const int j = H + i, m = H - 1 - i;
            if (H == 1 || (i & 1)) {  // ceil(j/2) and floor((K-m)/2) step up at odd i (at once for H = 1)
                ah *= v.r;
                bh *= v.r;
            }
            const double q2 = fma(f.qr, f.qr, f.qi * f.qi), s2 = fma(b.qr, b.qr, b.qi * b.qi);
            site(j, ah, br[K - 1 - j], B[(K - j) / 2], q2);
            site(m, A[(m + 1) / 2], s2, bh, fr[m]);
            if (i + 1 < H) next(i);
        }
    } else {
        // c conj(D) / |D|^2 folded into the two running states: Im(c q s / D) is then
        // Im(q s) with one factor running and one kept
        const double gr = fma(v.c0, dr, v.c1 * di) * inv, gi = fma(v.c1, dr, -v.c0 * di) * inv;
        auto fold = [&](Lin& s) {
            const Lin t = s;
            s.pr = fma(gr, t.pr, -gi * t.pi);
            s.pi = fma(gr, t.pi, gi * t.pr);
            s.qr = fma(gr, t.qr, -gi * t.qi);
            s.qi = fma(gr, t.qi, gi * t.qr);
        };
        fold(f);
        fold(b);
#pragma unroll
        for (int i = 0; i < H; ++i) {
            const int j = H + i, m = H - 1 - i;
            site(j, f.qr, bi[K - 1 - j], f.qi, br[K - 1 - j]);
            site(m, b.qr, fi[m], b.qi, fr[m]);
            if (i + 1 < H) next(i);
        }
    }
}

// Chains c0 .. c1 - 1 of one unit: each(v) before a chain's segment, then its
// site terms.
template <int K, bool RA, class P, class E, class F>
__device__ __forceinline__ void seg_loop(const GroupDev& g, SegStage* __restrict__ ring, const double* __restrict__ ck,
                                         const double* __restrict__ cc, int c0, int c1, int sub, int seg,
                                         P&& u, E&& each, F&& site) {
    constexpr int NC = RA ? 6 : 4;
    const int lane = threadIdx.x, cpw = 32 / g.lanes;
    const double* __restrict__ con0 = cc + g.cc_off;
    // stage of the chains first .. first + cpw - 1 (past the unit's last chain: the last one again)
    auto fetch = [&](int slot, int first) {
        if (first < c1) {
            SegStage& st = ring[slot];
            const double* p = ck + state_at<NC>(g, min(first + sub, c1 - 1), seg);
#pragma unroll
            for (int k = 0; k < NC; ++k) cp_async8(&st.rec[k][lane], p + k * kBlk);
            for (int i = lane; i < 4 * cpw; i += 32)
                cp_async16(&st.con[i >> 2][2 * (i & 3)], con0 + (long long)min(first + (i >> 2), c1 - 1) * kConst + 2 * (i & 3));
        }
        cp_async_commit();
    };
#pragma unroll
    for (int k = 0; k < kStages - 1; ++k) fetch(k, c0 + k * cpw);
    int slot = 0;
    for (int c = c0; c < c1; c += cpw) {
        cp_async_wait<kStages - 2>();
        __syncwarp();
        const SegStage& st = ring[slot];
        SegIn v;
        v.yr = st.rec[0][lane];
        v.yi = st.rec[1][lane];
        v.lam = RA ? st.rec[2][lane] : 1.0;
        v.xr = st.rec[RA ? 3 : 2][lane];
        v.xi = st.rec[RA ? 4 : 3][lane];
        v.rho = RA ? st.rec[5][lane] : 1.0;
        const double2* q = reinterpret_cast<const double2*>(st.con[sub]);
        const double2 a = q[0], b = q[1], d = q[2], e = q[3];
        v.Eg = a.x;
        v.ei = a.y;
        v.r = b.x;
        v.k0 = b.y;
        v.k1 = d.x;
        v.c0 = d.y;
        v.c1 = e.x;
        if (c + sub >= c1) v.k0 = v.k1 = v.c0 = v.c1 = 0.0;  // lanes past the unit's last chain
        // the slot read in the previous iteration is free: every lane has passed the __syncwarp above
        fetch(slot == 0 ? kStages - 1 : slot - 1, c + (kStages - 1) * cpw);
        slot = slot == kStages - 1 ? 0 : slot + 1;
        each(v);
        segment<K, RA>(v, u, site);
    }
}

// Bound: the FP64 pipe (16.5 FP64 of 25 instructions a site: 12 for the two
// steps, 7 for the real axis or 2 for the contour, 1 per site of the segment's
// D and weights).  168 registers hold the half states and the site sums; the
// potentials sit in shared memory (in registers they spill: 218 us against
// 196 us).  4000 sites, 33 488 chains: 197 us, 0.63 of the pipe; the sweeps
// 202 us, 0.57 of the pipe (14 warps per SM).  The fused schedule's single
// kernel took 467 us for the same pass.
template <int K>
__global__ void __launch_bounds__(32, 11) seg_kernel(const __grid_constant__ GroupSet gs,
                                                     const double* __restrict__ ck, const double* __restrict__ cc,
                                                     double* __restrict__ partial, const int* __restrict__ skip) {
    if (skip && *skip) return;
    __shared__ __align__(16) SegStage ring[kStages];
    const GroupDev& g = group(gs, find_group<&GroupDev::seg_base>(gs, gs.seg_base, blockIdx.x));
    const int rel = blockIdx.x - g.seg_base, sb = rel % g.nsb, cu = rel / g.nsb;
    const int lane = threadIdx.x, G = g.lanes, sg = lane & (G - 1), sub = lane / G;
    const int N = g.N, seg = min(sb * G + sg, g.nseg - 1);
    const int n0 = min(seg * K, N - K);
    const int c0 = cu * g.chains_per_unit, c1 = min(c0 + g.chains_per_unit, g.nch);
    const double ig = 1.0 / g.gamma;
    double acc[K];
    __shared__ double2 usm[K / 2][32];  // potentials / gamma, pairs of sites: 32 registers less per lane
#pragma unroll
    for (int j = 0; j < K; j += 2) {
        const double2 v = __ldg(reinterpret_cast<const double2*>(g.U + n0 + j));
        usm[j / 2][lane] = make_double2(v.x * ig, v.y * ig);
        acc[j] = acc[j + 1] = 0.0;
    }
    auto u = [&](int p) { return usm[p][lane]; };
    auto add = [&](int j, double a, double x, double b, double y) { acc[j] = fma(a, x, fma(b, y, acc[j])); };
    auto none = [](const SegIn&) {};
    if (g.kind == kRealAxis)
        seg_loop<K, true>(g, ring, ck, cc, c0, c1, sub, seg, u, none, add);
    else
        seg_loop<K, false>(g, ring, ck, cc, c0, c1, sub, seg, u, none, add);
    for (int o = G; o < 32; o <<= 1) {
#pragma unroll
        for (int j = 0; j < K; ++j) acc[j] += __shfl_xor_sync(kFull, acc[j], o);
    }
    if (sub == 0 && sb * G + sg < g.nseg) {
        double* __restrict__ row = partial + g.row_base + (long long)cu * N;
#pragma unroll
        for (int j = 0; j < K; j += 2)
            if (n0 + j >= seg * K) *reinterpret_cast<double2*>(row + n0 + j) = make_double2(acc[j], acc[j + 1]);
    }
}

// Transport characteristics (Compute_DensityOfStates, NEGF_Common.cpp:2390-2847;
// Compute_Current's integrand, :4321-4816) of one tube: block = (energy, block
// of 32 segments), the warp loops over the energy's M modes (real-axis chains
// with b0 = b1 = 1, in order; the energy record's cr, ci are Re f_0, Re f_1)
// and keeps the mode sums of a_n = deg Gamma_0 |G_n0|^2 and b_n = deg Gamma_1
// |G_n,N-1|^2 of its sites in registers: deg A_nn = a_n + b_n needs no scratch
// per site and chain.  red[e][8] (zeroed by the caller): [1] Gamma_0 b_0 and [2]
// Gamma_1 a_{N-1} summed over the modes (transmission from either end), then
// a_n f_0 + b_n f_1 at n = N/2, else 0, else N-1 (the current's probes,
// :4684-4714), and at n = N/4, else 3N/4 after N/2 (the charge integrand's,
// :3467-3496).  part[e][segment block]: sum of a_n + b_n; ldos[e][n] (may be
// null): (a_n + b_n) / 2 pi.
template <int K>
__global__ void __launch_bounds__(32, 8) transport_kernel(const __grid_constant__ GroupSet gs, int M,
                                                          const double* __restrict__ ck,
                                                          const double* __restrict__ cc, double* __restrict__ part,
                                                          double* __restrict__ red, double* __restrict__ ldos) {
    __shared__ __align__(16) SegStage ring[kStages];
    __shared__ double2 usm[K / 2][32];
    const GroupDev& g = group(gs, 0);
    const int e = blockIdx.x / g.nsb, sb = blockIdx.x % g.nsb;
    const int lane = threadIdx.x, N = g.N, nseg = g.nseg;
    const int seg = min(sb * 32 + lane, nseg - 1), n0 = min(seg * K, N - K);
    const double ig = 1.0 / g.gamma;
    double A[K], B[K];
#pragma unroll
    for (int j = 0; j < K; j += 2) {
        const double2 v = __ldg(reinterpret_cast<const double2*>(g.U + n0 + j));
        usm[j / 2][lane] = make_double2(v.x * ig, v.y * ig);
        A[j] = A[j + 1] = B[j] = B[j + 1] = 0.0;
    }
    double g0 = 0.0, g1 = 0.0, t0 = 0.0, t1 = 0.0;
    seg_loop<K, true>(
        g, ring, ck, cc, e * M, (e + 1) * M, 0, seg, [&](int p) { return usm[p][lane]; },
        [&](const SegIn& v) {
            g0 = v.c0;
            g1 = v.c1;
        },
        [&](int j, double a, double x, double b, double y) {
            A[j] = fma(a, x, A[j]);
            B[j] = fma(b, y, B[j]);
            if (j == 0) t0 = fma(g0, b * y, t0);
            if (j == K - 1) t1 = fma(g1, a * x, t1);
        });
    const bool real = sb * 32 + lane < nseg;
    const double f0 = g.items[e].cr, f1 = g.items[e].ci;
    double* __restrict__ out = red + (long long)e * 8;
    double sum = 0.0;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int n = n0 + j;
        if (!real || n < seg * K) continue;  // the overlapping last segment leaves its neighbour's sites alone
        const double ab = A[j] + B[j], v = fma(A[j], f0, B[j] * f1);
        sum += ab;
        if (ldos) ldos[(long long)e * N + n] = ab / (2.0 * 3.14159265358979323846);
        if (n == N / 2)
            out[3] = v;
        else if (n == 0)
            out[4] = v;
        else if (n == N - 1)
            out[5] = v;
        if (n != N / 2) {
            if (n == N / 4)
                out[6] = v;
            else if (n == (N * 3) / 4)
                out[7] = v;
        }
    }
    if (real && seg == 0) out[1] = t0;
    if (real && seg == nseg - 1) out[2] = t1;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
    if (lane == 0) part[blockIdx.x] = sum;
}

template <int K>
cudaError_t launch_states(const GroupSet& gs, const SweepShape& sh, double* ck, double* cc, double* tm,
                          const int* skip, cudaStream_t s) {
    if (sh.scan)
        scan_kernel<K><<<sh.chains, sh.scan_threads, 0, s>>>(gs, ck, cc, tm, skip);
    else
    {
        const size_t smem = sh.range_blocks > 0 ? sizeof(double) * kCarry * kCarryStage : 0;
        if (sh.range_blocks > 0) range_kernel<K><<<sh.range_blocks, 32, 0, s>>>(gs, cc, tm, skip);
        sweep_kernel<K><<<sh.sweep_blocks, 32, smem, s>>>(gs, ck, cc, tm, skip);
    }
    return cudaGetLastError();
}
template <int K>
cudaError_t launch_k(const GroupSet& gs, const SweepShape& sh, double* ck, double* cc, double* tm, double* partial,
                     const int* skip, cudaStream_t s, cudaEvent_t mid) {
    const cudaError_t e = launch_states<K>(gs, sh, ck, cc, tm, skip, s);
    if (e != cudaSuccess) return e;
    if (mid) cudaEventRecord(mid, s);
    seg_kernel<K><<<sh.seg_blocks, 32, 0, s>>>(gs, ck, cc, partial, skip);
    return cudaGetLastError();
}
template <int K>
cudaError_t launch_transport_k(const GroupSet& gs, const SweepShape& sh, int M, double* ck, double* cc, double* tm,
                               double* part, double* red, double* ldos, cudaStream_t s) {
    const cudaError_t e = launch_states<K>(gs, sh, ck, cc, tm, nullptr, s);
    if (e != cudaSuccess) return e;
    transport_kernel<K><<<gs.g[0].nch / M * gs.g[0].nsb, 32, 0, s>>>(gs, M, ck, cc, part, red, ldos);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_sweep(const GroupSet& gs, const SweepShape& sh, double* ck, double* cc, double* tm, double* partial,
                         const int* skip, cudaStream_t s, cudaEvent_t mid) {
    if (gs.ng <= 0) return cudaSuccess;
    return sh.K == kSweepSeg ? launch_k<kSweepSeg>(gs, sh, ck, cc, tm, partial, skip, s, mid)
                             : launch_k<2>(gs, sh, ck, cc, tm, partial, skip, s, mid);
}

cudaError_t launch_transport(const GroupSet& gs, const SweepShape& sh, int M, double* ck, double* cc, double* tm,
                             double* part, double* red, double* ldos, cudaStream_t s) {
    if (gs.ng != 1 || M < 1 || gs.g[0].lanes != 32) return cudaErrorInvalidValue;
    return sh.K == kSweepSeg ? launch_transport_k<kSweepSeg>(gs, sh, M, ck, cc, tm, part, red, ldos, s)
                             : launch_transport_k<2>(gs, sh, M, ck, cc, tm, part, red, ldos, s);
}

}  // namespace negf
