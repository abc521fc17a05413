// FP64 translations as tensor-core products (mma.sync f64), four units (source spheres) at a time.
//
// The seven stages of a translation (k_direct.cu) are chains of small real matrices times complex
// vectors.  One pair alone gives a product only four columns (two parts, real and imaginary); here a
// warp takes one degree of four units at once, so that the 16 rows of an m16n8k8 product are
// (unit, part) x (re, im), its contraction index is the order of the input and its columns are the
// orders of the output:
//
//   rotation, one warp per degree n:  load and fold x (or y'), product with Delta^n, the diagonal
//   e^{-i s theta}, product with Delta^n again, store -- in registers from end to end.  Orders are
//   split by parity (the four blocks of Delta's quarter, each padded to 8 x 4), input order
//   i = 4 j + q sits in k-step j of lane quad position q, and the columns of the table's fragments
//   are permuted so that output order i' = 8 t + 4 e + q of accumulator (t, e) is k-step 2t + e of the
//   next product in the same lane: the two products chain without a shuffle or a trip through shared
//   memory.
//   coaxial step, one warp per (unit, order k):  rows are degrees n, the contraction index is mu,
//   the eight columns are (a', b') x (+k, -k) x (re, im); S is read from the pair table straight
//   into the fragments, and w(mu) is formed from x' as its fragment is loaded.  Real and imaginary part
//   of S are two products on the same columns, the second with (-im, re).
//
// A warp owns its degrees in both rotations and its orders in the coaxial step, which rewrites x' as y'
// in place, so a batch of four translations needs two block barriers (the one-pair kernel: 28).
//
// mma.sync f64 runs at the FP64 pipe's full rate here (measured 64 FMA per clock and SM from four warps with one
// chain each), so the products themselves take a quarter of the time; the rest is forming w, the phases and
// the loads around them (L1 data pipe half busy, instruction fetch where the code outgrows its cache).
// One application: 1000 lognormal spheres (orders 11..28) 47.8 -> 21.4 ms, 64 spheres of order 15
// 0.222 -> 0.111 ms, 40 of order 5 78 -> 47 us (k_direct before, this after; copies included).
#pragma once

#include "k_common.cuh"
#include "k_special.cuh"

namespace foggy {
namespace mma {

constexpr int kUnits = 4;
constexpr int kPlanInts = 4 * 32;   // make_plan
constexpr int kRecs = 32;   // unit records made at a time, one per lane: eight batches

__device__ __forceinline__ void mma16x8x8(double (&c)[4], double a0, double a1, double a2, double a3, double b0,
                                          double b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}
__device__ __forceinline__ void mma16x8x4(double (&c)[4], double a0, double a1, double b0) {
    asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a0), "d"(a1), "d"(b0));
}
__device__ __forceinline__ void mma8x8x4(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

// ---- the Delta fragments --------------------------------------------------------------------------
// degree n has n/2 + 1 even and (n+1)/2 odd orders >= 0: steps of 4 for either, output tiles of 8
__host__ __device__ inline int steps_of(int n) { return (n / 2 + 4) / 4; }
// fragments of degree n, in doubles: output parity, tile, input parity, k-steps (32 lanes each; a pair's two values side
// by side in a lane)
__host__ __device__ inline int frags_of(int n) {
    const int k = steps_of(n);
    return 4 * ((k + 1) / 2) * k * 32;
}

// ---- shared memory ----------------------------------------------------------------------------------
// what a batch knows of a unit
struct Unit {
    const double2* x;    // source coefficients, or null: the unit is empty
    const double2* s;    // its coaxial block
    int p;               // source degree
    int km;              // min(source, target degree)
    double rho;          // translation length; 0: the source is added unchanged
};

// Direction of a translation: e^{i phi} and e^{i theta} by their cosine and sine, and its length.
struct Dir {
    double cp, sp, ct, st, rho;
};

// The direction of t = (d0, d1, d2), |t| = r.  The reference evaluates its Legendre functions at
// x = cos(theta), theta = acos(t_z / r), with sqrt(|1 - x^2|) as the sine (LPMNS,
// lib_math_legendre.f90:68-126), so near-axial directions take that x's sine, which is 0 where x
// rounds to +-1.
__device__ inline Dir direction(double d0, double d1, double d2, double r) {
    Dir g{1.0, 0.0, 1.0, 0.0, r};
    const double m = fmax(fabs(d0), fabs(d1));
    if (m > 0.0) {
        const double a = d0 / m, b = d1 / m, h = sqrt(a * a + b * b);
        g.cp = a / h;
        g.sp = b / h;
    }
    if (r != 0.0) {
        g.ct = cos(acos(d2 / r));
        g.st = sqrt(fabs(1.0 - g.ct * g.ct));
    }
    return g;
}

// z^m for m < 32 by binary powers: no more than nine products, so closer to e^{i m phi} than the sine and
// cosine of the rounded product m phi, at a third of the instructions
__device__ __forceinline__ cplx zpow(cplx z, int m) {
    cplx p = (m & 1) ? z : mk(1.0, 0.0);
#pragma unroll
    for (int b = 1; b < 5; ++b) {
        z = z * z;
        if ((m >> b) & 1) p = p * z;
    }
    return p;
}

// x' / y' of one unit by order: order k = 0..pp holds degrees max(1, k)..pp, four complex values each
// (a +k, b +k, a -k, b -k).  Offsets are padded so that the eight lanes of a quarter warp, four orders
// apart by two and both parts, hit distinct banks when they store one degree's orders.
__host__ __device__ inline int order_block(int k, int pp) { return 4 * (pp + 1 - (k < 1 ? 1 : k)); }
__host__ __device__ inline int order_pad(int off, int k) {
    const int lo = k < 1 ? 1 : k;
    return (((2 * ((k >> 1) & 3)) - (off - 4 * lo)) & 7);
}
__host__ __device__ inline int unit_size(int pp) {
    int o = 0;
    for (int k = 0; k <= pp; ++k) o += order_pad(o, k) + order_block(k, pp);
    return o;
}
// table stride of the phases: orders up to 8 NI - 1 are read (those past the degree times zero)
template <int NI>
__host__ __device__ constexpr int phase_ld() {
    return 8 * NI;
}

template <int NI>
__host__ __device__ inline size_t smem_bytes(int pp) {
    return ((size_t)kUnits * unit_size(pp) + (size_t)2 * pp * (pp + 2) + (size_t)2 * 2 * kUnits * phase_ld<NI>() + 4 + 4 * NI + 4) * 16 +
           2 * kRecs * (sizeof(Unit) + sizeof(Dir)) + kPlanInts * sizeof(int);
}

struct Shared {
    double2* buf;     // [unit][unit_size]
    double2* acc;     // target accumulator, a then b
    double2* eps;     // [2][unit][ld] e^{i m (phi + pi/2)}
    double2* eth;     // [2][unit][ld] (-1)^s (2 cos s theta, 2 sin s theta), (1, 0) at s = 0
    Unit* un;         // [2][kRecs] their units
    Dir* dir;         // [2][kRecs] directions of the translations
    int* blk;         // [pp + 1] order offsets
    int* ord;         // degrees by warp
    int* wfirst;      // [warps + 1] into ord
    int* fo;          // first Delta fragment of a degree
    double2* zero;    // four zero values
    double* rn;       // 1 / (2n(n+1)), n < 8 NI + 8
    int us;           // unit stride
};

template <int NI>
__device__ inline Shared carve(void* base, int pp, int us) {
    Shared s;
    double2* d = static_cast<double2*>(base);
    s.us = us;
    s.buf = d;   d += (size_t)kUnits * us;
    s.acc = d;   d += 2 * pp * (pp + 2);
    s.eps = d;   d += 2 * kUnits * phase_ld<NI>();
    s.eth = d;   d += 2 * kUnits * phase_ld<NI>();
    s.zero = d;  d += 4;
    s.rn = reinterpret_cast<double*>(d);  d += 4 * NI + 4;
    s.dir = reinterpret_cast<Dir*>(d);
    s.un = reinterpret_cast<Unit*>(s.dir + 2 * kRecs);
    s.blk = reinterpret_cast<int*>(s.un + 2 * kRecs);
    s.ord = s.blk + 32;
    s.wfirst = s.ord + 32;
    s.fo = s.wfirst + 32;
    return s;
}

// What a launch of largest degree pp lays out in shared memory, made on the host: the order offsets, the degrees
// 1..pp dealt to the warps (largest first, each to the warp with the least work so far), each warp's first, and the first
// fragment of a degree.
constexpr int kDegreeCost[4] = {10, 14, 26, 33};   // by k-steps: products, phases and load latencies, 100 cycles
inline void make_plan(int pp, int warps, int* out) {
    int o = 0;
    for (int k = 0; k <= pp; ++k) {
        o += order_pad(o, k);
        out[k] = o;
        o += order_block(k, pp);
    }
    int load[16] = {0}, own[32] = {0};
    for (int n = pp; n >= 1; --n) {
        int b = 0;
        for (int w = 1; w < warps; ++w)
            if (load[w] < load[b]) b = w;
        load[b] += kDegreeCost[steps_of(n) - 1];
        own[n] = b;
    }
    o = 0;
    for (int w = 0; w < warps; ++w) {
        out[64 + w] = o;
        for (int n = pp; n >= 1; --n)
            if (own[n] == w) out[32 + o++] = n;
    }
    out[64 + warps] = o;
    o = 0;
    for (int n = 1; n <= pp; ++n) {
        out[96 + n] = o;
        o += frags_of(n);
    }
}
// warps of a launch's CTAs (by_degree); with S summed (sum) the radial functions leave no room for a second CTA on an
// SM above order 19, so that one has twice the warps up to 23
__host__ __device__ constexpr int warps_of(int pp, bool sum) { return pp <= 7 ? 4 : pp <= 19 ? 8 : pp <= 23 ? (sum ? 16 : 8) : 12; }

// ---- rotation -----------------------------------------------------------------------------------------
// Products of one degree's fragments with the folded input: for every output order i' = 8t + 4e + q
// of parity P, f(P, 2t + e, E, O) gets the sums over even and odd input orders.  A0 holds the input
// for even output orders, A1 for odd ones, [input parity][k-step][re, im].
template <int N, class F>
__device__ __forceinline__ void delta_mul(const double* __restrict__ frag, int lane, const double (&A0)[2][N][2],
                                          const double (&A1)[2][N][2], F f) {
    int at = 0;
#pragma unroll
    for (int P = 0; P < 2; ++P)
#pragma unroll
        for (int t = 0; t < (N + 1) / 2; ++t) {
            double acc[2][4];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.0;
#pragma unroll
                for (int j = 0; j < N; j += 2) {
                    const double a0 = P ? A1[r][j][0] : A0[r][j][0], a1 = P ? A1[r][j][1] : A0[r][j][1];
                    if (j + 1 < N) {
                        const double a2 = P ? A1[r][j + 1][0] : A0[r][j + 1][0];
                        const double a3 = P ? A1[r][j + 1][1] : A0[r][j + 1][1];
                        const double2 b = __ldg(reinterpret_cast<const double2*>(frag + 32 * at) + lane);
                        mma16x8x8(acc[r], a0, a1, a2, a3, b.x, b.y);
                        at += 2;
                    } else {
                        mma16x8x4(acc[r], a0, a1, __ldg(frag + 32 * at + lane));
                        at += 1;
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (2 * t + e < N) f(P, 2 * t + e, mk(acc[0][e], acc[0][2 + e]), mk(acc[1][e], acc[1][2 + e]));
        }
}

// sign bit of a double flipped where the mask has it
__device__ __forceinline__ double flip(double v, int mask) {
    return __hiloint2double(__double2hiint(v) ^ mask, __double2loint(v));
}

// What a lane keeps through the kernel: its row (unit, part), quad position and, for the orders
// k = 2 (4 j + q) + P of its k-steps, the place of degree n in x' at 4 n + at[P][j].
template <int NI>
struct Lane {
    int q, u, part, lane;
    int at[2][NI];
    __device__ __forceinline__ Lane(const Shared& s, int pp, int lane_) {
        lane = lane_;
        q = lane & 3;
        part = (lane >> 2) & 1;
        u = lane >> 3;
#pragma unroll
        for (int P = 0; P < 2; ++P)
#pragma unroll
            for (int j = 0; j < NI; ++j) {
                const int k = 2 * (4 * j + q) + P;
                at[P][j] = k <= pp ? u * s.us + part + s.blk[k] - 4 * (k < 1 ? 1 : k) : 0;
            }
    }
};

// One degree n of the four units.  out = false: the sources to the axis of their translations, from x into buf.
// out = true: the translated fields from buf back to the common frame, summed over the units and added to acc
// (the warp owns the degree: no other warp touches these entries).  Of the two orders +-m a lane forms, it
// keeps -m where its unit bit 1 is set, +m elsewhere, and gives the other to the lane 16 away; then even or
// odd orders by unit bit 0, eight lanes away.  One function for both directions: the kernel's code has to
// stay within the instruction cache.
template <int NI, int N>
__device__ __forceinline__ void rotate(const Shared& s, const Lane<NI>& L, const double* __restrict__ frag, int n,
                                       int pj, const Unit& un, int cur, bool out) {
    const int q = L.q;
    const double2* eps = s.eps + (cur * kUnits + L.u) * phase_ld<NI>() + 2 * q;
    const double2* eth = s.eth + (cur * kUnits + L.u) * phase_ld<NI>();
    const int pm = n << 31;                   // sign of (-1)^n
    const int ktop = min(un.km, n) - 2 * q;   // orders left of this lane's first; km = -1: empty or coincident
    double2* X = s.buf + 4 * n;
    double A0[2][N][2], A1[2][N][2];
    if (!out) {
        const int pl = un.p;
        const double2* xs = un.x + (L.part * pl * (pl + 2) + n * n - 1 + n);
        const double2* xq = xs + 2 * q;
        const double2* xr = xs - 2 * q;
        const int mtop = n <= pl ? n - 2 * q : -1;   // an empty unit has degree 0
#pragma unroll
        for (int P = 0; P < 2; ++P)
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const int o = 8 * j + P;   // m - 2q
                double2 xp{0, 0}, xm{0, 0};
                if (o <= mtop) {
                    xp = __ldg(xq + o);
                    xm = __ldg(xr - o);
                }
                if (o == 0 && q == 0) xm = double2{0, 0};   // order 0 counts once
                const double2 e = eps[o];
                const double ux = e.x * xp.x - e.y * xp.y, uy = e.x * xp.y + e.y * xp.x;
                const double vx = flip(e.x * xm.x + e.y * xm.y, pm), vy = flip(e.x * xm.y - e.y * xm.x, pm);
                A0[P][j][0] = ux + vx;
                A0[P][j][1] = uy + vy;
                A1[P][j][0] = ux - vx;
                A1[P][j][1] = uy - vy;
            }
    } else {
#pragma unroll
        for (int P = 0; P < 2; ++P)
#pragma unroll
            for (int j = 0; j < N; ++j) {
                double2 yp{0, 0}, ym{0, 0};
                if (8 * j + P <= ktop) {
                    const double2* d = X + L.at[P][j];
                    yp = d[0];
                    ym = d[2];
                }
                if (8 * j + P == 0 && q == 0) ym = double2{0, 0};
                const double mx = flip(ym.x, pm), my = flip(ym.y, pm);
                A0[P][j][0] = yp.x + mx;
                A0[P][j][1] = yp.y + my;
                A1[P][j][0] = yp.x - mx;
                A1[P][j][1] = yp.y - my;
            }
    }
    // folded input of the second product from the sums of the first:
    //   even outputs (-1)^s (2 cos E - 2i sin O), odd ones (-1)^s (2 cos O - 2i sin E)
    double B0[2][N][2], B1[2][N][2];
    delta_mul<N>(frag, L.lane, A0, A1, [&](int P, int j, cplx E, cplx O) {
        const double2 h = eth[2 * (4 * j + q) + P];
        B0[P][j][0] = fma(h.y, O.y, h.x * E.x);
        B0[P][j][1] = fma(-h.y, O.x, h.x * E.y);
        B1[P][j][0] = fma(h.y, E.y, h.x * O.x);
        B1[P][j][1] = fma(-h.y, E.x, h.x * O.y);
    });
    // sums of the second product, over the first's input
    delta_mul<N>(frag, L.lane, B0, B1, [&](int P, int j, cplx E, cplx O) {
        A0[P][j][0] = E.x;
        A0[P][j][1] = E.y;
        A1[P][j][0] = O.x;
        A1[P][j][1] = O.y;
    });
    if (!out) {
#pragma unroll
        for (int P = 0; P < 2; ++P)
#pragma unroll
            for (int j = 0; j < N; ++j)
                if (8 * j + P <= ktop) {
                    double2* d = X + L.at[P][j];
                    d[0] = make_double2(A0[P][j][0] + A1[P][j][0], A0[P][j][1] + A1[P][j][1]);
                    d[2] = make_double2(flip(A0[P][j][0] - A1[P][j][0], pm), flip(A0[P][j][1] - A1[P][j][1], pm));
                }
    } else {
        const bool neg = (L.lane & 16) != 0, odd = (L.lane & 8) != 0;
        const int nm = neg ? 0x80000000 : 0;
        const int first = 2 * q + (odd ? 1 : 0);
        double2* d = s.acc + (L.part * pj * (pj + 2) + n * n - 1 + n) + (neg ? -first : first);
        const int sm = neg ? pm : 0;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            double R[2][2];   // [parity][re, im] of the sign this lane keeps
#pragma unroll
            for (int P = 0; P < 2; ++P) {
                const double2 e = eps[8 * j + P];
                // kept: conj(e) (E + O) at +m, e (E - O) at -m; given: the other (the sign (-1)^n of -m comes last)
                const double ey = flip(e.y, nm), ox = flip(A1[P][j][0], nm), oy = flip(A1[P][j][1], nm);
                const double kx = A0[P][j][0] + ox, ky = A0[P][j][1] + oy, gx = A0[P][j][0] - ox, gy = A0[P][j][1] - oy;
                const double hx = __shfl_xor_sync(0xffffffffu, e.x * gx - ey * gy, 16);
                const double hy = __shfl_xor_sync(0xffffffffu, e.x * gy + ey * gx, 16);
                R[P][0] = fma(e.x, kx, ey * ky) + hx;
                R[P][1] = fma(e.x, ky, -ey * kx) + hy;
            }
            const double gx = __shfl_xor_sync(0xffffffffu, odd ? R[0][0] : R[1][0], 8);
            const double gy = __shfl_xor_sync(0xffffffffu, odd ? R[0][1] : R[1][1], 8);
            const double vx = flip((odd ? R[1][0] : R[0][0]) + gx, sm);
            const double vy = flip((odd ? R[1][1] : R[0][1]) + gy, sm);
            const int m = first + 8 * j;
            if (m <= n && !(neg && m == 0)) {
                double2* dj = d + (neg ? -8 * j : 8 * j);
                double2 v = *dj;
                v.x += vx;
                v.y += vy;
                *dj = v;
            }
        }
    }
}

// degrees of one warp
template <int NI>
__device__ __forceinline__ void rotate_all(const Shared& s, const Lane<NI>& L, const double* __restrict__ frag, int warp,
                                           int top, int pj, const Unit& un, int cur, bool out) {
#pragma unroll 1
    for (int i = s.wfirst[warp]; i < s.wfirst[warp + 1]; ++i) {
        const int n = s.ord[i];
        if (n > top) continue;
        const double* f = frag + s.fo[n];
        switch (steps_of(n)) {
            case 1: rotate<NI, 1>(s, L, f, n, pj, un, cur, out); break;
            case 2: if constexpr (NI >= 2) rotate<NI, 2>(s, L, f, n, pj, un, cur, out); break;
            case 3: if constexpr (NI >= 3) rotate<NI, 3>(s, L, f, n, pj, un, cur, out); break;
            case 4: if constexpr (NI >= 4) rotate<NI, 4>(s, L, f, n, pj, un, cur, out); break;
        }
    }
}

// pair_block_offset(k, M2, M2) in 32 bits: sum over k' < k of (M2 - k')^2
__device__ __forceinline__ int block_offset(int k, int M2) {
    return k * M2 * (M2 - k + 1) + (k - 1) * k * (2 * k - 1) / 6;
}

// ---- coaxial step ---------------------------------------------------------------------------------------
// order k of one unit: y'(n, +-k) = (-1)^k / (2n(n+1)) sum_mu S(k; n, mu) w(mu), x' replaced by y'.
// The rows of a product are eight degrees of Re S over the same eight of Im S, so one complex load
// is two fragment entries and the two products with w's real and imaginary columns meet in one lane.
// S is read along mu (the square is symmetric): a quarter warp then touches two rows of 64 bytes, where
// reading along n it would touch four lines; the L1's lookups are what bounds this kernel.
// wf[mu] (row k): 2 (mu-1) sqrt(mu^2 - k^2), 2 (mu+2) sqrt((mu+1)^2 - k^2); the other two factors of w are
// polynomials of mu.  x' comes without its (2 nu + 1), which is folded into all of them.
__device__ __forceinline__ double2 ld_stream(const double2* p) {
    double2 v;
    asm("ld.global.nc.L1::evict_first.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}

// S fragments of a tile of degrees n0 + r (clamped to pj: rows past it are not stored): k-steps mu = k + 4t + q, clamped
// to pl + 1 in the last two steps (the next order may have a step less).
// One order of one unit, tiles of eight degrees.  sv holds the first tile's fragments on entry and those of order
// k + dk on exit.  One instantiation per number of k-steps NT = ceil((pl + 2 - k) / 4), so that the loops over
// them carry no conditions.
template <int NI, int NT, int KT>
__device__ __forceinline__ void coaxial_k(const Shared& s, const Unit& un, int u, int k, int dk, int pj,
                                          const double2* __restrict__ wf, int lane, double2 (&sv)[KT]) {
    const int r = lane >> 2, q = lane & 3;
    const int pl = un.p, lo = k < 1 ? 1 : k;
    // w(mu) of column r: component r / 2, real or imaginary part.  Degrees above pl read the zero entry, those
    // below lo the entry of lo: their factors are zero.
    const int c = r >> 1, im = r & 1;
    double2* X = s.buf + u * s.us + s.blk[k];
    const double* xd = reinterpret_cast<const double*>(X);
    const int zo = (int)(reinterpret_cast<const double*>(s.zero) - xd);
    const int ca = 2 * c + im, cb = (2 * c + im) ^ 3, co = (2 * c + im) ^ 1;
    const int row = k + q - lo;                 // row of mu at step 0 (-1 at k = q = 0)
    const int d = pl - k - q;                   // degrees above mu at step 0
    const double rho = im ? un.rho : -un.rho;
    const double kk = (c & 2) ? -(double)k : (double)k;   // -k columns
    double m = (double)(k + q);
    const double2* f = wf + (k + q);
    double w[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t, m += 4.0) {
        int ra = 8 * (row + 4 * t), rm = ra - 8, rp = ra + 8;
        if (t == 0) {
            ra = max(ra, 0);
            rm = max(rm, 0);
        }
        if (t == NT - 1) {
            ra = d >= 4 * t ? ra : zo;
            rm = d >= 4 * t - 1 ? rm : zo;
        }
        if (t >= NT - 2) rp = d > 4 * t ? rp : zo;
        const double a = xd[ra + ca], b = xd[ra + cb], am = xd[rm + co], ap = xd[rp + co];
        const double2 g = __ldg(f + 4 * t);
        const double h = fma(4.0, m, 2.0);      // 2 (2 mu + 1)
        double v = fma(g.x, am, -g.y * ap);
        v = fma(kk * h, b, v);
        w[t] = fma(rho, v, fma(m, m, m) * h * a);
    }
    __syncwarp();
    const int fm = k << 31;
    double2* Y = X + 4 * r + q;
#pragma unroll 1
    for (int n0 = lo; n0 <= pj; n0 += 8, Y += 32) {
        // the next tile's fragments, or the next order's first tile's, follow each product that frees theirs
        const bool more = n0 + 8 <= pj, go = more || k + dk <= un.km;
        const int kn = more ? k : k + dk, top = pl + 1 - kn;
        const int M2 = (pj > pl ? pj : pl) + 2, Wk = M2 - kn;
        const double2* S = un.s + (block_offset(kn, M2) + (min((more ? n0 + 8 : kn) + r, pj) - kn) * Wk);
        auto reload = [&](int t) { sv[t] = ld_stream(t >= NT - 2 ? S + min(4 * t + q, top) : S + q + 4 * t); };
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int t = 0; t + 1 < NT; t += 2) {
            mma16x8x8(acc, sv[t].x, sv[t].y, sv[t + 1].x, sv[t + 1].y, w[t], w[t + 1]);
            if (go) {
                reload(t);
                reload(t + 1);
            }
        }
        if (NT & 1) {
            mma16x8x4(acc, sv[NT - 1].x, sv[NT - 1].y, w[NT - 1]);
            if (go) reload(NT - 1);
        }
        const int n = n0 + r;
        const double g = flip(s.rn[n], fm);
        if (n <= pj) Y[0] = make_double2(g * (acc[0] - acc[3]), g * (acc[1] + acc[2]));
    }
}

// orders k0, k0 + dk, ... (dk <= 4) of one unit
template <int NI>
__device__ __forceinline__ void coaxial(const Shared& s, const Unit un, int u, int k0, int dk, int pj,
                                        const double2* __restrict__ wf, int ld, int lane) {
    constexpr int KT = 2 * NI + 1;
    if (k0 > un.km) return;
    double2 sv[KT];
    {
        const int q = lane & 3;
        const int M2 = (pj > un.p ? pj : un.p) + 2, Wk = M2 - k0, top = un.p + 1 - k0;
        const double2* S = un.s + (block_offset(k0, M2) + (min((k0 < 1 ? 1 : k0) + (lane >> 2), pj) - k0) * Wk);
#pragma unroll
        for (int t = 0; t < KT; ++t) sv[t] = ld_stream(S + min(4 * t + q, top));
    }
#pragma unroll 1
    for (int k = k0; k <= un.km; k += dk) {
        const int nt = (un.p + 5 - k) >> 2;
        const double2* f = wf + k * ld;
        switch (nt) {
            case 1: coaxial_k<NI, 1>(s, un, u, k, dk, pj, f, lane, sv); break;
            case 2: coaxial_k<NI, 2>(s, un, u, k, dk, pj, f, lane, sv); break;
            case 3: coaxial_k<NI, 3>(s, un, u, k, dk, pj, f, lane, sv); break;
            case 4: if constexpr (NI >= 2) coaxial_k<NI, 4>(s, un, u, k, dk, pj, f, lane, sv); break;
            case 5: if constexpr (NI >= 2) coaxial_k<NI, 5>(s, un, u, k, dk, pj, f, lane, sv); break;
            case 6: if constexpr (NI >= 3) coaxial_k<NI, 6>(s, un, u, k, dk, pj, f, lane, sv); break;
            case 7: if constexpr (NI >= 3) coaxial_k<NI, 7>(s, un, u, k, dk, pj, f, lane, sv); break;
            case 8: if constexpr (NI >= 4) coaxial_k<NI, 8>(s, un, u, k, dk, pj, f, lane, sv); break;
            case 9: if constexpr (NI >= 4) coaxial_k<NI, 9>(s, un, u, k, dk, pj, f, lane, sv); break;
        }
    }
}

// ---- coaxial step without tables -----------------------------------------------------------------------
// Radial functions of the four units of a batch, zeta_p = i^p z_p for p = 0..pj + pl + 1 and zero around them (kZetaPad
// entries before: the sums run past an entry's own last term, where the coefficients are zero), by one warp: j_n and
// y_n each on its own lane, then all lanes.
constexpr int kZetaPad = 16;
__device__ __forceinline__ void radial(const Unit* un, int pj, int z, double2* zeta, int zl, double* scratch, int lane) {
    if (lane < 2 * kUnits) {
        const int u = lane % kUnits, P = pj + un[u].p + 1;
        double* o = scratch + lane * zl;
        if (un[u].km >= 0) {
            if (lane < kUnits) dev_sph_jn(un[u].rho, P, o);
            else if (z != 1) dev_sph_yn(un[u].rho, P, o);
        }
    }
    __syncwarp();
    for (int t = lane; t < kUnits * zl; t += 32) {
        const int u = t / zl, p = t - u * zl - kZetaPad;
        cplx v = mk(0.0, 0.0);
        if (un[u].km >= 0 && p >= 0 && p <= pj + un[u].p + 1)
            v = zeta_of(z, p, scratch + u * zl, scratch + (kUnits + u) * zl);
        zeta[t] = make_double2(v.x, v.y);
    }
}

// Orders k0, k0 + dk, ... of units u0 and u0 + 1, with S(k; n, mu) = sum_q G_q(k; mu, n) zeta_{n + mu - 2q} summed for each
// fragment entry: one Gaunt coefficient serves both units, and the tiles' accumulators stay in registers so that w is
// formed once.  Bound by the L1's lookups for G and zeta.
template <int NI>
__device__ __forceinline__ void coaxial_sum(const Shared& s, const Unit* un, int u0, int k0, int dk, int pj,
                                            const double2* __restrict__ wf, int ld, const SGaunt& g, const double2* zeta,
                                            int zl, int lane) {
    const int r = lane >> 2, q = lane & 3, c = r >> 1, im = r & 1;
    const int km = max(un[u0].km, un[u0 + 1].km);
    const int ca = 2 * c + im, cb = (2 * c + im) ^ 3, co = (2 * c + im) ^ 1;
#pragma unroll 1
    for (int k = k0; k <= km; k += dk) {
        const int lo = k < 1 ? 1 : k, W = g.NM - k + 1;
        const size_t plane = (size_t)W * W;
        const double* G0 = g.gs + g.koff[k];
        const double kk = (c & 2) ? -(double)k : (double)k;
        int pl[2];
        double rho[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const Unit& u = un[u0 + e];
            pl[e] = k <= u.km ? u.p : -2;   // a unit without this order reads zeros
            rho[e] = im ? u.rho : -u.rho;
        }
        const int top = max(pl[0], pl[1]) + 1;
        double acc[NI][2][4];
#pragma unroll
        for (int i = 0; i < NI; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) acc[i][e][0] = acc[i][e][1] = acc[i][e][2] = acc[i][e][3] = 0.0;
        double m = (double)(k + q);
#pragma unroll 1
        for (int mu0 = k; mu0 <= top; mu0 += 4, m += 4.0) {
            const int mu = mu0 + q;
            const double2 gf = __ldg(wf + k * ld + mu);
            const double h = fma(4.0, m, 2.0), c0 = fma(m, m, m) * h;
            double w[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const double* xd = reinterpret_cast<const double*>(s.buf + (u0 + e) * s.us + s.blk[k]);
                const int zo = (int)(reinterpret_cast<const double*>(s.zero) - xd);
                const int row = 8 * (mu - lo);
                const int ra = mu >= lo && mu <= pl[e] ? row : zo, rm = mu - 1 >= lo && mu - 1 <= pl[e] ? row - 8 : zo;
                const int rp = mu + 1 <= pl[e] ? row + 8 : zo;
                double v = fma(gf.x, xd[rm + co], -gf.y * xd[rp + co]);
                v = fma(kk * h, xd[ra + cb], v);
                w[e] = fma(rho[e], v, c0 * xd[ra + ca]);
            }
            const int mc = min(mu, top);
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                if (lo + 8 * i > pj) break;
                const int n = min(lo + 8 * i + r, pj);
                const double* G = G0 + (size_t)(mc - k) * W + (n - k);
                // past the entry's own min(n, mu) the coefficients are zero
                const int qm = min(min(lo + 8 * i + 7, pj), min(mu0 + 3, top));
                double sx[2] = {0.0, 0.0}, sy[2] = {0.0, 0.0};
                const double2* z0 = zeta + u0 * zl + kZetaPad + n + mc;
                const double2* z1 = z0 + zl;
#pragma unroll 4
                for (int qq = 0; qq <= qm; ++qq, z0 -= 2, z1 -= 2) {
                    const double gq = __ldg(G);
                    G += plane;
                    const double2 za = *z0, zb = *z1;
                    sx[0] = fma(gq, za.x, sx[0]);
                    sy[0] = fma(gq, za.y, sy[0]);
                    sx[1] = fma(gq, zb.x, sx[1]);
                    sy[1] = fma(gq, zb.y, sy[1]);
                }
#pragma unroll
                for (int e = 0; e < 2; ++e) mma16x8x4(acc[i][e], sx[e], sy[e], w[e]);
            }
        }
        __syncwarp();
        const int fm = k << 31;
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int n = lo + 8 * i + r;
            if (n > pj) break;
            const double f = flip(s.rn[n], fm);
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (pl[e] >= 0)
                    s.buf[(u0 + e) * s.us + s.blk[k] + 4 * (n - lo) + q] =
                        make_double2(f * (acc[i][e][0] - acc[i][e][3]), f * (acc[i][e][1] + acc[i][e][2]));
        }
        __syncwarp();
    }
}
// entries of a unit's zeta, and the shared memory of two batches' tables and one's scratch
template <int NI>
__host__ __device__ constexpr int zeta_ld() {
    return 16 * NI + 2 + kZetaPad;
}
template <int NI>
__host__ __device__ constexpr size_t sum_smem_bytes() {
    return (size_t)kUnits * zeta_ld<NI>() * (2 * 16 + 2 * 8);
}

}  // namespace mma
}  // namespace foggy
