// FP64 2D retriangulate pass: one-sided, work-compacted, deterministic integer sums.
//
// The same split as the mixed pass (passes_mix.cuh): one warp per outer element T taken from a
// global counter, 32 pairs (T, b) per batch, each pair's geometry computed once from T, the
// mirrored termNonloc from the symmetric completion, every diagonal entry from its row's sum
// (kernels of |x - y| only; integrate_retriangulate, integration.cpp:345-540). All quadrature
// arithmetic is FP64, and GB300 runs FP64 at 1/64 of its FP32 rate, so the FP64 pipe bounds the
// kernel and everything that can leave it does:
//   * The (pair, outer point) classes come from the certified FP32 test (certified.cuh): a ball
//     holding the partner or missing it with a margin. All else is a cut item. Its polygon's structure
//     comes from the certified FP32 run too, only its points are FP64 (f64_polygon).
//   * Constant kernels: inside items need no quadrature loop. A pair's inside mask indexes a table
//     (shared memory, one entry per mask byte) of the rule's outer sums over the mask; its blocks
//     are those times kc |T| |b| and the rule's inner sums.
//   * Cut items (and, for other kernels, inside items) are listed pair by pair, so a pair's items
//     are neighbours: full warps integrate the items, then full warps fold them, one (pair, output)
//     per lane, instead of every lane walking all outer points.
// Measured (quadrature phase, against the two-sided colored pass): constant kernel, 2 * 128^2
// triangles, delta = 0.1, 2.56e7 pairs: 19.3 ms against 1740 ms; 2 * 32^2 triangles: 0.45 against 66.6 ms;
// parabola, 2 * 57^2, delta = 0.12: 5.2 against 257 ms; fractional, 2 * 40^2: 8.1 and 5.1 for the close
// pairs against 568 ms. The FP64 pipe is 70 to 90% busy in these. With one integer per slot the first
// took 18.6 ms: 0.4 ms of the rest are the second integers' sums, 0.3 the moments' origin.
//
// Sums. Every contribution is cut into 64-bit integers that are added with integer atomics, so the
// result does not depend on the order of the warps. The unit of a slot (t, v) of termNonloc
// follows from a bound of that slot: the blocks' sum over the elements at t and at v is at most
// 2^xN |patch t| |patch v|, with |patch| the elements' |det| sum at a vertex. Exponents are kept
// in eighths of a bit (vexp = 8 log2 |patch|, rounded up), so that only their sum is rounded to a
// whole power: the unit 2^((xN + vexp[t] + vexp[v]) / 8 - 62) is near 2^-55 of a pair that fills the
// ball, whatever the mesh grading. A contribution near the bound is a whole number of units; of a
// smaller one a second integer, 40 bits below the first, holds what is left, and of one below about
// 2^-50 of the bound (a sliver that the sphere cuts off) a third, 40 bits lower again. So a slot holds
// all bits of its contributions however small they are against the bound: the smallest entries of a matrix
// are 1e-24 of the largest. Most batches have no second and almost all no third parts, and skip them.
// The sums with many more terms have two integers: termLocal in the diagonal-block slots (unit
// 2^(xD + vexp[t] - 62)), and per partner element its termLocalPrime, of which a constant kernel's
// inside part is one number, the |T| weighted sum of the outer rule over the inside masks. A nonzero
// contribution counts at least one of the last units, so a slot is zero only when all its
// contributions are (the reference drops exact zeros).
#pragma once
#include "passes_mix.cuh"

namespace nlg {

constexpr int F64_WARPS = 4;
constexpr int F64_THREADS = 32 * F64_WARPS;
constexpr int F64_CAP = 128;   // items integrated before their pairs are folded (>= MAXQ)
constexpr int F64_RN = 7;      // per item: innerLocal, innerNonloc[3], off-diagonal termLocalPrime sums[3]
constexpr int F64_OUT = 15;    // per pair: termNonloc[9], off-diagonal termLocal[3] and termLocalPrime[3]
constexpr int F64_BITS = 62;   // a bound of 2^x has the unit 2^(x - 62)
constexpr int F64_WIDE = 40;   // bits from one integer of a sum to the next
constexpr int F64_ERR_THIRD = 12;   // err[]: some slot has a third integer
constexpr int F64_ELP = 8;     // per element: inside sum (two integers), cut termLocalPrime[3], second integers[3]

struct F64Args {
    MixArgs m;                  // m.elp: F64_ELP integers per element
    const int *vexp;            // per vertex, 8 log2 of its elements' |det| sum, rounded up
    long long *valslo;          // second integers of vals
    long long *valsNt;          // third integers of valsN (m.valsN: two integers per slot)
    const double *idet;         // per element, 1 / det (signed)
    const double *mtab;         // constant kernels: the mask table (k_mask_table)
    const double *pw;           // singular kernels: power tables (primitives.cuh)
    int exact;                  // the inner rule integrates degree two (bit 0), four (bit 1) exactly (see f64_item)
};

struct F64Warp {
    long long rhb[3], rrb[3];   // T's rows (see MixWarp)
    unsigned rmask[3];
    int rlo[3], tvs[3];
    int te[3];                  // vexp of T's vertices
    int pid[32];                // partner element
    int pe[32];                 // its eexp
    int pve[32][3];             // vexp of its vertices
    F2 pc[32][3];               // its vertices relative to T's vertex 0, FP32
    unsigned short list[F64_CAP];           // items, pair by pair: lane << 6 | inside << 5 | outer point
    unsigned char order[F64_CAP];           // the inside items, then the cut items (kernels that list both)
    unsigned char pl[32], ps[32], pn[32];   // chunk's pairs: owner lane, first item, item count
};
struct F64Entry {   // one partner vertex of a batch and its integer sums over T's rows
    int col, pad;
    long long v[6];   // first integers, second integers
};
// per-pair sums of the folded items (15, and termLocalPrime's second integers), then the item results;
// the scatter list lies over both
constexpr int F64_ACC = F64_OUT + 3;
constexpr size_t F64_WORK_BYTES = (size_t)(32 * F64_ACC + F64_CAP * F64_RN) * 8;
static_assert(F64_WORK_BYTES >= 96 * sizeof(F64Entry), "the scatter list lies over the item results");
__host__ __device__ constexpr size_t f64_warp_bytes(int nPx) {
    return (sizeof(F64Warp) + 15) / 16 * 16 + (size_t)nPx * (24 + 56) + F64_WORK_BYTES + 16;
}
// mask sums of the outer rule: one table of up to 256 entries per 8 outer points
__host__ __device__ constexpr int f64_tab_entries(int nPx) { return 256 * (nPx / 8) + (nPx % 8 ? 1 << (nPx % 8) : 0); }
__host__ __device__ constexpr size_t f64_smem_bytes(int kind, int nPx) {
    return (kind == MIX_CONST ? (size_t)f64_tab_entries(nPx) * 7 * 8 : 0) +
           F64_WARPS * ((f64_warp_bytes(nPx) + 15) / 16 * 16) + 16;
}

// 2^e, e in [-1022, 1023]
__device__ __forceinline__ double pow2i(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
// v 2^e by its exponent field, off the FP64 pipe (results below the normal range become 0, above it inf)
__device__ __forceinline__ double scale2(double v, int e) {
    const int hi = __double2hiint(v), x = (hi >> 20) & 0x7ff, y = x + e;
    if (x == 0 || y <= 0) return 0.0;
    return y >= 0x7ff ? __longlong_as_double(0x7ff0000000000000LL) : __hiloint2double(hi + (e << 20), __double2loint(v));
}
// e with |x| < 2^e (x normal; at least -900 for zeros and subnormals)
__device__ __forceinline__ int exp_above(double x) {
    const int e = ((__double2hiint(x) >> 20) & 0x7ff) - 1022;
    return e < -900 ? -900 : e;
}
// q (a number of units) = hi + lo 2^-40 + rest, all of q's sign, by its bits: the conversions of the FP64
// pipe are as slow as its arithmetic. rest is set where bits are left over (|q| < 2^12); f64_third holds
// those. |q| >= 2^lim or NaN sets bad: rigorous bounds (all but singular kernels) leave a sum its 62 bits;
// without one lim is what keeps the sum from wrapping.
__device__ __forceinline__ void f64_split(double q, int lim, bool &bad, long long &hi, long long &lo, bool &rest) {
    const long long b = __double_as_longlong(q);
    const int x = (int)(b >> 52) & 0x7ff, n = 1075 - x;   // |q| = m 2^-n
    const long long m = x ? (b & 0xfffffffffffffLL) | 1LL << 52 : 0;
    bad |= x >= 1023 + lim;
    long long h, l = 0;
    if (n <= 0) {
        h = m << min(-n, 63);
    } else {
        h = m >> min(n, 63);
        const long long f = m - (h << min(n, 63));
        const int k = min(n - F64_WIDE, 63);
        l = k <= 0 ? f << -k : f >> k;
        rest |= k > 0 && (l << k) != f;
    }
    hi = b < 0 ? -h : h;
    lo = b < 0 ? -l : l;
}
// The third integer: the bits of |q| < 2^13 below 2^-40, in units of 2^-80 (a nonzero rest never to zero).
__device__ __forceinline__ long long f64_third(double q) {
    const long long b = __double_as_longlong(q);
    const int n = 1075 - ((int)(b >> 52) & 0x7ff), k = min(n - F64_WIDE, 63);
    const long long a = (b & 0xfffffffffffffLL) | 1LL << 52, g = a - ((a >> k) << k);
    const long long t = n <= 2 * F64_WIDE ? g << (2 * F64_WIDE - n) : max(g >> min(n - 2 * F64_WIDE, 63), 1LL);
    return b < 0 ? -t : t;
}
// The sums of two integers: a nonzero contribution counts at least one of the second's units.
__device__ __forceinline__ void f64_split2(double q, int lim, bool &bad, long long &hi, long long &lo) {
    bool rest = false;
    f64_split(q, lim, bad, hi, lo, rest);
    if (rest && (hi | lo) == 0) lo = __double2hiint(q) < 0 ? -1 : 1;
}
// Their value: the lower integers' carries go up first, so that no cancellation is left between them.
__device__ __forceinline__ double f64_join(long long hi, long long lo, long long third = 0) {
    constexpr double W = 1.0 / (double)(1LL << F64_WIDE);
    lo += (third + (1LL << (F64_WIDE - 1))) >> F64_WIDE;
    third -= (third + (1LL << (F64_WIDE - 1))) >> F64_WIDE << F64_WIDE;
    hi += (lo + (1LL << (F64_WIDE - 1))) >> F64_WIDE;
    lo -= (lo + (1LL << (F64_WIDE - 1))) >> F64_WIDE << F64_WIDE;
    return (double)hi + W * ((double)lo + W * (double)third);
}

// s + c += x y, c the low part of the sum (product and sum without loss to second order)
__device__ __forceinline__ void f64_acc2(double &s, double &c, double x, double y) {
    const double p = x * y, t = s + p, z = t - s;
    c += ((s - (t - z)) + (p - z)) + fma(x, y, -p);
    s = t;
}
// Outer sum over the mask byte of table entry i (8 outer points from 8 (i >> 8) on) of dx_k f_k, f a
// product of up to two basis functions: r < 0 leaves out the first, c < 0 the second. Every entry of
// the matrix takes these sums, so they are summed with compensation.
__device__ __forceinline__ double f64_mask_sum(const Rule &rule, int dV, int i, int r, int c) {
    double s = 0, e = 0;
    for (int b = 0; b < 8; b++) {
        const int k = 8 * (i >> 8) + b;
        if (!((i >> b) & 1) || k >= rule.nPx) continue;
        const double pr = r < 0 ? 1.0 : rule.psix[dV * k + r], pc = c < 0 ? 1.0 : rule.psix[dV * k + c];
        const double w = rule.dx[k] * pr;
        f64_acc2(s, e, w, pc);
        e += fma(rule.dx[k], pr, -w) * pc;
    }
    return s + e;
}

// Mask table of the rule, TS numbers per entry: the sums over dx psi_r, then over dx psi_r psi_c (r < c),
// and in 2D over dx. Built once per assembly: the compensated sums on the FP64 pipe would cost each
// block of the pass 0.2 ms with 11 points, copying them costs it a few microseconds.
__global__ void k_mask_table(Rule rule, int dV, int TS, int n, double *__restrict__ tab) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * TS) return;
    const int m = i / TS;
    int q = i - TS * m, r = q, c = -1;
    if (q >= dV) {   // (r, c) of the q-th product, or past them
        r = 0;
        for (q -= dV; r < dV - 1 && q >= dV - 1 - r; r++) q -= dV - 1 - r;
        c = r + 1 + q;
        if (r == dV - 1) r = c = -1;
    }
    tab[i] = f64_mask_sum(rule, dV, m, r, c);
}

// Square root, quotient and reciprocal square root by Newton's iteration from an FP32 seed (22 bits or
// more, so two steps reach FP64; the last step of the square root and of the quotient is the residual
// correction). The seed's conversions go through the integer pipe (conversions from and to FP64 run
// at its rate). CUDA's division and square root, which keep the FP64 pipe busy about twice as long,
// serve arguments outside [2^-98, 2^98], where the seed would leave the FP32 range.
__device__ __forceinline__ bool f64_seedable(double v) {   // v > 0
    return (unsigned)((__double2hiint(v) >> 20) - (1023 - 98)) < 196u;
}
__device__ __forceinline__ float f64_to_seed(double v) {
    const int hi = __double2hiint(v);
    return __int_as_float(((hi - (896 << 20)) << 3) | (int)((unsigned)__double2loint(v) >> 29));
}
__device__ __forceinline__ double f64_from_seed(float s) {
    const int b = __float_as_int(s);
    return __hiloint2double((b >> 3) + (896 << 20), b << 29);
}
__device__ __forceinline__ double f64_rsqrt_step(double v, double y) { return fma(0.5 * y, fma(-(v * y), y, 1.0), y); }
__device__ __forceinline__ double f64_rsqrt(double v) {
    if (!f64_seedable(v)) return 1.0 / sqrt(v);
    return f64_rsqrt_step(v, f64_rsqrt_step(v, f64_from_seed(rsqrtf(f64_to_seed(v)))));
}
__device__ __forceinline__ double f64_sqrt(double v) {
    if (!f64_seedable(v)) return sqrt(v);
    const double y = f64_rsqrt_step(v, f64_from_seed(rsqrtf(f64_to_seed(v)))), g = v * y;
    return fma(0.5 * y, fma(-g, g, v), g);
}
__device__ __forceinline__ double f64_div(double a, double b) {
    const double m = fabs(b);
    if (!f64_seedable(m)) return a / b;
    double y = f64_from_seed(__fdividef(1.f, f64_to_seed(m)));
    y = __hiloint2double(__double2hiint(y) | (__double2hiint(b) & 0x80000000), __double2loint(y));
    y = fma(y, fma(-b, y, 1.0), y);
    const double q = a * y;
    return fma(y, fma(-b, q, a), q);
}

// Classes by FP64 tests, for problems outside the certified FP32 range (precision "fp64-onesided" only;
// "fp64" takes the general pass there): triangle Q relative to the ball's center, inside and outside with a
// margin of 2^-40, far above the tests' rounding for elements up to 512 horizons; the rest is cut.
constexpr double MARG_D64 = 1.0 / 1099511627776.0;
__device__ __noinline__ int f64_class(double sq, const double *x, const double *Eb) {
    const double sqlo = sq * (1.0 - MARG_D64), sqhi = sq * (1.0 + MARG_D64);
    bool in = true, out = true;
    for (int i = 0; i < 3; i++) {
        const int j = i == 2 ? 0 : i + 1;
        const double px = Eb[2 * i] - x[0], py = Eb[2 * i + 1] - x[1], ux = Eb[2 * j] - Eb[2 * i], uy = Eb[2 * j + 1] - Eb[2 * i + 1];
        const double pp = px * px + py * py, pu = px * ux + py * uy, uu = ux * ux + uy * uy, cr = px * uy - py * ux;
        in = in && pp < sqlo;
        out = out && pp > sqhi && (!(pu < 0.0 && -pu < uu) || cr * cr > sqhi * uu);   // the end point, then the side
    }
    return in ? CLS_IN : (out ? CLS_OUT : CLS_CUT);
}

// Kernel value from r2 = |x - y|^2; pw the problem's power table (singular kernels).
template <int KIND>
__device__ __forceinline__ double f64_kernel(const ProbParams &P, const double *pw, double r2) {
    if (KIND == MIX_CONST) return P.kc;
    if (KIND == MIX_SINGULAR) return pw_eval(pw, r2);
    if (P.kernel == KER_PARABOLA) return P.kc * (P.sqdelta - r2);
    return P.kc * exp2(-0.5 * P.expo * log2(r2));
}

// A cut item in the general pass's arithmetic (out_retri_f64, in_retri_f64), step by step in absolute
// coordinates: the rare items whose polygon the certified run leaves open and which is tiny (a sphere
// through a vertex, a near-tangent edge). Such a polygon may lie below the rounding of the partner's
// reference coordinates, and which of its sums vanish decides which matrix entries exist.
template <int KIND>
__device__ __forceinline__ void f64_item_exact(const ProbParams &P, const Rule &rule, const double *pw, const double *x,
                                            const double *Eb, double *res, unsigned &nsub) {
    double R[18], S0 = 0, S1[3] = {0, 0, 0}, S2[3] = {0, 0, 0};
    const int n = xretriangulate(x, Eb, P.sqdelta, P.caps, R);
    for (int r = 0; r + 2 < n; r++) {
        nsub++;
        const double tri[6] = {R[0], R[1], R[2 * r + 2], R[2 * r + 3], R[2 * r + 4], R[2 * r + 5]};
        const double rTdet = xabsDet2(tri);
        for (int i = 0; i < rule.nPy; i++) {
            double y[2], ref[2] = {0, 0};
            y[0] = (tri[2] - tri[0]) * rule.Py[2 * i] + (tri[4] - tri[0]) * rule.Py[2 * i + 1] + tri[0];
            y[1] = (tri[3] - tri[1]) * rule.Py[2 * i] + (tri[5] - tri[1]) * rule.Py[2 * i + 1] + tri[1];
            const double z0 = x[0] - y[0], z1 = x[1] - y[1];
            const double w = f64_kernel<KIND>(P, pw, z0 * z0 + z1 * z1) * rule.dy[i] * rTdet;
            xtoRef(Eb, y, ref);
            const double l0 = 1.0 - ref[0] - ref[1];
            S0 += w;
            S1[0] += l0 * w;
            S1[1] += ref[0] * w;
            S1[2] += ref[1] * w;
            S2[0] += l0 * ref[0] * w;
            S2[1] += l0 * ref[1] * w;
            S2[2] += ref[0] * ref[1] * w;
        }
    }
    res[0] = S0;
#pragma unroll
    for (int q = 0; q < 3; q++) { res[1 + q] = S1[q]; res[4 + q] = S2[q]; }
}

// Polygon of a cut item: points relative to the ball's center in R, and in the partner's reference
// coordinates in L (n of each, at most 9).
struct F64Poly {
    double R[18], L[18];
    int n;
};

// The polygon of B(x) and the triangle Q (relative to x), e1, e2 its edges from Q0. The certified FP32
// run fixes what the points are (which vertices, which roots of which edges, which caps: the
// reference's branches); only the points themselves are FP64: per crossing a square root and a
// quotient, per cap a reciprocal square root. In reference coordinates vertices are constants and
// a crossing is its root. Against the exact routine, which takes both roots of all three edges with
// their divisions for every item, that is about a third of the FP64 instructions: with the closed
// moments of f64_item the pass went from 51.5 to 20.5 ms on 2 * 128^2 triangles (constant kernel) when
// this came. False where a decision
// is within its margin. LATE takes such an item's polygon from the exact routine instead, and is false
// where that holds less than 1e-5 of the partner (f64_item_exact then; above, every sum of the item is
// far above its rounding).
template <bool PHYS, bool LATE>
__device__ __forceinline__ bool f64_polygon(const ProbParams &P, const double *x, const double *Eb, const F2 *Qf, const double *Q,
                                            const double *e, double adet, double idet, F64Poly &Y) {
    auto to_ref = [&](double yx, double yy, double *l) {
        const double dx = yx - Q[0], dy = yy - Q[1];
        l[0] = (e[3] * dx - e[2] * dy) * idet;
        l[1] = (e[0] * dy - e[1] * dx) * idet;
    };
    if (LATE) {
        Y.n = xretriangulate(x, Eb, P.sqdelta, P.caps, Y.R);
        double area = 0;
        for (int j = 0; j < Y.n; j++) {
            Y.R[2 * j] -= x[0];
            Y.R[2 * j + 1] -= x[1];
            to_ref(Y.R[2 * j], Y.R[2 * j + 1], &Y.L[2 * j]);
            if (j >= 2)
                area += fabs((Y.R[2 * j - 2] - Y.R[0]) * (Y.R[2 * j + 1] - Y.R[1]) - (Y.R[2 * j - 1] - Y.R[1]) * (Y.R[2 * j] - Y.R[0]));
        }
        return Y.n < 3 || area >= 1e-5 * adet;
    }
    bool amb = false;
    unsigned long long codes = 0;
    Y.n = fretriangulate<true>(Qf, P.sqdelta_f, P.caps, nullptr, amb, nullptr, &codes);
    if (amb) return false;
    unsigned xm = 0, cm = 0;
    for (int j = 0; j < Y.n; j++) {
        const int c = (int)(codes >> (4 * j)) & 15;
        xm |= (unsigned)(c >= FCODE_X && c < FCODE_CAP) << j;
        cm |= (unsigned)(c == FCODE_CAP) << j;
        if (c < 3) {
            Y.L[2 * j] = c == 1 ? 1.0 : 0.0;
            Y.L[2 * j + 1] = c == 2 ? 1.0 : 0.0;
            if (PHYS) {
                Y.R[2 * j] = c == 0 ? Q[0] : (c == 1 ? Q[2] : Q[4]);
                Y.R[2 * j + 1] = c == 0 ? Q[1] : (c == 1 ? Q[3] : Q[5]);
            }
        }
    }
#pragma unroll 1
    for (; xm; xm &= xm - 1) {
        const int j = __ffs(xm) - 1, c = ((int)(codes >> (4 * j)) & 15) - FCODE_X, k = c >> 1, r = c & 1;
        const double px = k == 0 ? Q[0] : (k == 1 ? Q[2] : Q[4]), py = k == 0 ? Q[1] : (k == 1 ? Q[3] : Q[5]);
        const double qx = k == 0 ? Q[2] : (k == 1 ? Q[4] : Q[0]), qy = k == 0 ? Q[3] : (k == 1 ? Q[5] : Q[1]);
        const double bx = px - qx, by = py - qy;
        const double ab = qx * bx + qy * by, aad = (qx * qx + qy * qy) - P.sqdelta, bb = bx * bx + by * by;
        const double v = ab * ab - aad * bb, sv = __double2hiint(v) > 0 ? f64_sqrt(v) : 0.0;
        // the root of larger size has no cancellation, the other is aad / bb over it (as the reference)
        const bool pos = ab < 0.0;
        const double big = pos ? sv - ab : -(ab + sv);
        const bool direct = pos == (r == 0);
        const double lam = f64_div(direct ? big : aad, direct ? bb : big);
        Y.R[2 * j] = fma(lam, bx, qx);
        Y.R[2 * j + 1] = fma(lam, by, qy);
        Y.L[2 * j] = k == 0 ? 1.0 - lam : (k == 1 ? lam : 0.0);
        Y.L[2 * j + 1] = k == 0 ? 0.0 : (k == 1 ? 1.0 - lam : lam);
    }
#pragma unroll 1
    for (; cm; cm &= cm - 1) {   // between two crossings (placePointOnCap, integration.cpp:1353-1377)
        const int j = __ffs(cm) - 1, i = j ? j - 1 : 0, h = j + 1 < Y.n ? j + 1 : 0;
        const double o = idet > 0 ? -1.0 : 1.0;
        const double nx = (Y.R[2 * i + 1] - Y.R[2 * h + 1]) * o, ny = (Y.R[2 * h] - Y.R[2 * i]) * o;
        const double s = P.delta * f64_rsqrt(nx * nx + ny * ny);
        Y.R[2 * j] = nx * s;
        Y.R[2 * j + 1] = ny * s;
        to_ref(Y.R[2 * j], Y.R[2 * j + 1], &Y.L[2 * j]);
    }
    return true;
}

// Inner sums of one item into res (see F64_RN), without the factor |T|: the quadrature over the
// partner (inside) or over the fan of its polygon with the ball (cut).
// Polynomial kernels need no inner points. An inside item of the parabola kernel is a combination of
// the rule's moments to degree four. Where the inner rule integrates the polynomials exactly (degree two
// for constant kernels, four for the parabola), the sums over the fan are the polygon's integrals,
// taken from its sides in reference coordinates about its first point: closed forms per side for constant
// kernels; for the parabola the integral over the triangle (0, P0, P1) of a monomial of degree d is
// (P0 x P1) / (d + 2) times its mean over the side, by the 3-point Gauss rule (exact to degree five). The
// polygon's own point as the origin keeps the digits of a small one, whose sides are short against their
// distance from any other origin (taken from the partner's vertex 0, the smallest entries of a parabola
// matrix were off by 1e-5 of themselves; the sides that lie on the edges through that vertex and add
// nothing are about as many as the two through the first point).
// Returns false for a cut item whose polygon the certified run leaves open, which takes LATE.
template <int KIND, bool LATE>
__device__ __forceinline__ bool f64_item(const ProbParams &P, const Rule &rule, const PassRuleT<double> &pr, bool inside,
                                         int exact, const double *pw, const double *x, const F2 *Qf, const double *Eb, double adet, double idet,
                                         double *res, unsigned &nsub) {
    const double Q[6] = {Eb[0] - x[0], Eb[1] - x[1], Eb[2] - x[0], Eb[3] - x[1], Eb[4] - x[0], Eb[5] - x[1]};
    const double e[4] = {Eb[2] - Eb[0], Eb[3] - Eb[1], Eb[4] - Eb[0], Eb[5] - Eb[1]};
    double S0 = 0, S1[3] = {0, 0, 0}, S2[3] = {0, 0, 0};
    const bool parab = KIND == MIX_REGULAR && P.kernel == KER_PARABOLA;
    // parabola: kernel kc (k0 - k1 . u - (ka u1^2 + 2 kb u1 u2 + kd u2^2)) in reference coordinates u about the
    // point that lies at (yx, yy) from x
    double k0 = 0, k1x = 0, k1y = 0, ka = 0, kb2 = 0, kd = 0;
    auto parab_at = [&](double yx, double yy) {
        k0 = P.sqdelta - (yx * yx + yy * yy);
        k1x = 2.0 * (yx * e[0] + yy * e[1]);
        k1y = 2.0 * (yx * e[2] + yy * e[3]);
        ka = e[0] * e[0] + e[1] * e[1];
        kb2 = 2.0 * (e[0] * e[2] + e[1] * e[3]);
        kd = e[2] * e[2] + e[3] * e[3];
    };
    auto from_moments = [&](double f, const double *I) {   // I: integrals of the kernel times 1, r1, r2, r1^2, r1 r2, r2^2
        S0 = f * I[0];
        S1[0] = f * (I[0] - I[1] - I[2]); S1[1] = f * I[1]; S1[2] = f * I[2];
        S2[0] = f * (I[1] - I[3] - I[4]); S2[1] = f * (I[2] - I[4] - I[5]); S2[2] = f * I[4];
    };
    auto from_moments_at = [&](double o1, double o2, const double *I) {   // the same of u = r - (o1, o2)
        const double o0 = 1.0 - o1 - o2, i12 = I[1] + I[2];
        S0 = I[0];
        S1[0] = o0 * I[0] - i12; S1[1] = o1 * I[0] + I[1]; S1[2] = o2 * I[0] + I[2];
        S2[0] = o0 * S1[1] - o1 * i12 - (I[3] + I[4]);
        S2[1] = o0 * S1[2] - o2 * i12 - (I[4] + I[5]);
        S2[2] = o1 * S1[2] + (o2 * I[1] + I[4]);
    };
    auto sum_point = [&](double k, int i, double *I) {   // inner point i with kernel value k
        I[0] += k * rule.dy[i];
        I[1] += k * pr.cy[3 * i + 1];
        I[2] += k * pr.cy[3 * i + 2];
        I[3] += k * pr.cyy[6 * i + 3];
        I[4] += k * pr.cyy[6 * i + 4];
        I[5] += k * pr.cyy[6 * i + 5];
    };
    if (KIND == MIX_REGULAR && parab && inside) {
        nsub++;
        parab_at(Q[0], Q[1]);
        const double *m = pr.mom, *h = pr.mom4;
        auto sum = [&](double c, double cx, double cy, double cxx, double cxy, double cyy) {
            return k0 * c - (k1x * cx + k1y * cy) - (ka * cxx + kb2 * cxy + kd * cyy);
        };
        const double I[6] = {sum(m[0], m[1], m[2], m[3], m[4], m[5]), sum(m[1], m[3], m[4], h[0], h[1], h[2]),
                             sum(m[2], m[4], m[5], h[1], h[2], h[3]), sum(m[3], h[0], h[1], h[4], h[5], h[6]),
                             sum(m[4], h[1], h[2], h[5], h[6], h[7]), sum(m[5], h[2], h[3], h[6], h[7], h[8])};
        from_moments(P.kc * adet, I);
    } else if (KIND != MIX_CONST && inside) {
        nsub++;
        double I[6] = {0, 0, 0, 0, 0, 0};
        for (int i = 0; i < rule.nPy; i++) {
            const double yx = Q[0] + e[0] * rule.Py[2 * i] + e[2] * rule.Py[2 * i + 1];
            const double yy = Q[1] + e[1] * rule.Py[2 * i] + e[3] * rule.Py[2 * i + 1];
            sum_point(f64_kernel<KIND>(P, pw, yx * yx + yy * yy), i, I);
        }
        from_moments(adet, I);
    } else {
        F64Poly Y;
        if (!f64_polygon<KIND != MIX_CONST, LATE>(P, x, Eb, Qf, Q, e, adet, idet, Y)) {
            if (LATE) f64_item_exact<KIND>(P, rule, pw, x, Eb, res, nsub);
            return LATE;
        }
        if (Y.n >= 3) nsub += Y.n - 2;
        if ((KIND == MIX_CONST && (exact & 1)) || (KIND == MIX_REGULAR && parab && (exact & 2))) {
            double I[6] = {0, 0, 0, 0, 0, 0};
            const double o1 = Y.L[0], o2 = Y.L[1];
            if (KIND != MIX_CONST && Y.n >= 3) parab_at(Y.R[0], Y.R[1]);
            const double k02 = 0.5 * k0, k03 = (1.0 / 3.0) * k0, k04 = 0.25 * k0;
            double x1 = Y.L[2] - o1, y1 = Y.L[3] - o2;
#pragma unroll 1
            for (int j = 2; j < Y.n; j++) {
                const double x0 = x1, y0 = y1;
                x1 = Y.L[2 * j] - o1;
                y1 = Y.L[2 * j + 1] - o2;
                const double c = fabs(x0 * y1 - x1 * y0);
                if (KIND == MIX_CONST) {
                    const double sx = x0 + x1, sy = y0 + y1;
                    I[0] += c;
                    I[1] = fma(c, sx, I[1]);
                    I[2] = fma(c, sy, I[2]);
                    I[3] = fma(c, fma(sx, sx, -(x0 * x1)), I[3]);
                    I[4] = fma(c, fma(sx, sy, fma(x0, y0, x1 * y1)), I[4]);
                    I[5] = fma(c, fma(sy, sy, -(y0 * y1)), I[5]);
                } else {
                    const double dx = x1 - x0, dy = y1 - y0;
#pragma unroll
                    for (int g = 0; g < 3; g++) {
                        const double t = g == 1 ? 0.5 : (g == 0 ? 0.11270166537925831 : 0.8872983346207417);
                        const double zx = fma(t, dx, x0), zy = fma(t, dy, y0), cg = c * (g == 1 ? 4.0 / 9.0 : 5.0 / 18.0);
                        const double k1 = k1x * zx + k1y * zy, k2 = zx * (ka * zx) + zy * (kb2 * zx + kd * zy);
                        const double w0 = cg * (k02 - (1.0 / 3.0) * k1 - 0.25 * k2), w1 = cg * (k03 - 0.25 * k1 - 0.2 * k2);
                        const double w2 = cg * (k04 - 0.2 * k1 - (1.0 / 6.0) * k2), tx = w2 * zx;
                        I[0] += w0;
                        I[1] += w1 * zx;
                        I[2] += w1 * zy;
                        I[3] += tx * zx;
                        I[4] += tx * zy;
                        I[5] += (w2 * zy) * zy;
                    }
                }
            }
            const double f = P.kc * adet;
            I[0] *= KIND == MIX_CONST ? 0.5 * f : f;
#pragma unroll
            for (int q = 1; q < 6; q++) I[q] *= KIND != MIX_CONST ? f : (q < 3 ? (1.0 / 6.0) * f : (q == 4 ? (1.0 / 24.0) * f : (1.0 / 12.0) * f));
            if (Y.n >= 3) from_moments_at(o1, o2, I);
        } else if (KIND == MIX_CONST) {   // the rule's moments on each fan triangle (see item_cut_const)
            const double m0 = pr.mom[0], mx = pr.mom[1], my = pr.mom[2], mxx = pr.mom[3], mxy = pr.mom[4], myy = pr.mom[5];
            const double la[3] = {1.0 - Y.L[0] - Y.L[1], Y.L[0], Y.L[1]};
            for (int r = 0; r + 2 < Y.n; r++) {
                const double *b = &Y.L[2 * r + 2], *c = &Y.L[2 * r + 4];
                double be[3], ga[3];
                be[1] = b[0] - la[1]; be[2] = b[1] - la[2]; be[0] = -be[1] - be[2];
                ga[1] = c[0] - la[1]; ga[2] = c[1] - la[2]; ga[0] = -ga[1] - ga[2];
                const double rT = adet * P.kc * fabs(be[1] * ga[2] - be[2] * ga[1]);
                double t0[3], t1[3], t2[3];
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    t0[q] = la[q] * m0 + (be[q] * mx + ga[q] * my);
                    t1[q] = la[q] * mx + (be[q] * mxx + ga[q] * mxy);
                    t2[q] = la[q] * my + (be[q] * mxy + ga[q] * myy);
                    S1[q] += rT * t0[q];
                }
                S0 += rT * m0;
                S2[0] += rT * (la[0] * t0[1] + (be[0] * t1[1] + ga[0] * t2[1]));
                S2[1] += rT * (la[0] * t0[2] + (be[0] * t1[2] + ga[0] * t2[2]));
                S2[2] += rT * (la[1] * t0[2] + (be[1] * t1[2] + ga[1] * t2[2]));
            }
        } else {
            double M[6] = {0, 0, 0, 0, 0, 0};
            for (int r = 0; r + 2 < Y.n; r++) {
                const double Bx = Y.R[2 * r + 2] - Y.R[0], By = Y.R[2 * r + 3] - Y.R[1];
                const double Cx = Y.R[2 * r + 4] - Y.R[0], Cy = Y.R[2 * r + 5] - Y.R[1];
                const double rT = fabs(Bx * Cy - By * Cx);
                double I[6] = {0, 0, 0, 0, 0, 0};   // in the fan triangle's own reference coordinates
                for (int i = 0; i < rule.nPy; i++) {
                    const double px = rule.Py[2 * i], py = rule.Py[2 * i + 1];
                    const double yx = Y.R[0] + Bx * px + Cx * py, yy = Y.R[1] + By * px + Cy * py;
                    sum_point(f64_kernel<KIND>(P, pw, yx * yx + yy * yy), i, I);
                }
                // r1, r2 of the partner are affine in them
                const double a1 = Y.L[0], a2 = Y.L[1], b1 = Y.L[2 * r + 2] - a1, b2 = Y.L[2 * r + 3] - a2;
                const double c1 = Y.L[2 * r + 4] - a1, c2 = Y.L[2 * r + 5] - a2;
                const double u0 = a1 * I[0] + b1 * I[1] + c1 * I[2], v0 = a2 * I[0] + b2 * I[1] + c2 * I[2];
                const double ux = a1 * I[1] + b1 * I[3] + c1 * I[4], vx = a2 * I[1] + b2 * I[3] + c2 * I[4];
                const double uy = a1 * I[2] + b1 * I[4] + c1 * I[5], vy = a2 * I[2] + b2 * I[4] + c2 * I[5];
                M[0] += rT * I[0];
                M[1] += rT * u0;
                M[2] += rT * v0;
                M[3] += rT * (a1 * u0 + b1 * ux + c1 * uy);
                M[4] += rT * (a1 * v0 + b1 * vx + c1 * vy);
                M[5] += rT * (a2 * v0 + b2 * vx + c2 * vy);
            }
            from_moments(1.0, M);
        }
    }
    res[0] = S0;
#pragma unroll
    for (int q = 0; q < 3; q++) { res[1 + q] = S1[q]; res[4 + q] = S2[q]; }
    return true;
}
// About one cut item in 400 on the mesh above. Out of line, after the others of its chunk: inlined, the
// exact routines' registers and code cost the ordinary items 5 to 10%.
template <int KIND>
__device__ __noinline__ unsigned f64_item_late(const ProbParams *P, const Rule &rule, const PassRuleT<double> &pr, int exact,
                                               const double *pw, const double *x, const double *Eb, double adet, double idet,
                                               double *res) {
    unsigned nsub = 0;
    f64_item<KIND, true>(*P, rule, pr, false, exact, pw, x, nullptr, Eb, adet, idet, res, nsub);
    return nsub;
}

template <int KIND>
__global__ void __launch_bounds__(F64_THREADS, 3) k_pass_f64(F64Args fa, Rule rule, PassRuleT<double> pr) {
    constexpr bool CK = KIND == MIX_CONST;
    extern __shared__ __align__(16) unsigned char s_raw[];
    const PassArgs &a = fa.m.p;
    const SlotMap &sm = fa.m.m;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int nPx = rule.nPx;
    double *tab = reinterpret_cast<double *>(s_raw);   // mask sums (constant kernels)
    unsigned char *wbase = reinterpret_cast<unsigned char *>(tab + (CK ? 7 * f64_tab_entries(nPx) : 0));
    wbase = s_raw + ((wbase - s_raw) + 15) / 16 * 16 + (size_t)wib * ((f64_warp_bytes(nPx) + 15) / 16 * 16);
    F64Warp &W = *reinterpret_cast<F64Warp *>(wbase);
    double *x64 = reinterpret_cast<double *>(wbase + (sizeof(F64Warp) + 15) / 16 * 16);   // [nPx][2]
    F2 *xf = reinterpret_cast<F2 *>(x64 + 2 * nPx);                                       // [nPx]
    double *coef = reinterpret_cast<double *>(xf + nPx);   // [nPx][7]: |T| dx times psi_r, psi_r psi_c (r < c), 1
    unsigned char *work = reinterpret_cast<unsigned char *>(coef + 7 * nPx);
    long long *acc = reinterpret_cast<long long *>(work);                                 // [32][F64_ACC]
    double *res = reinterpret_cast<double *>(acc + 32 * F64_ACC);                   // [F64_CAP][F64_RN]
    F64Entry *slist = reinterpret_cast<F64Entry *>(work);
    if (CK) {
        for (int i = threadIdx.x; i < 7 * f64_tab_entries(nPx); i += F64_THREADS) tab[i] = fa.mtab[i];
        __syncthreads();
    }
    long long *vals = reinterpret_cast<long long *>(a.vals);
    bool bad = false;   // a contribution outside the fixed-point range (reported at the end)
    bool miss = false;  // a matrix slot not found (reported at the end)
    unsigned nsub = 0, nclose = 0, nitin = 0, nitcut = 0;
    for (;;) {
        int idx = 0;
        if (lane == 0) idx = atomicAdd(fa.m.work, 1);
        idx = __shfl_sync(FULL, idx, 0);
        if (idx >= a.count) break;
        const int T = a.list ? a.list[idx] : idx;
        const long long lb = a.out_ptr[T], le = a.out_cnt ? lb + a.out_cnt[T] : a.out_ptr[T + 1];
        const long long ln = lb + (a.near_cnt ? a.near_cnt[T] : 0);   // near pairs come first
        if (lb == le || a.labT[T] == 0) continue;
        int tv[3];
        unsigned keepmask = 0;   // bit r: the row of T's vertex r exists
#pragma unroll
        for (int r = 0; r < 3; r++) {
            tv[r] = a.T32[(long long)T * 3 + r];
            if (a.labV[tv[r]] > 0) keepmask |= 1u << r;
        }
        if (lane < 3) {   // T's rows, for the lookups of every batch
            const int u = sel3(tv, lane);
            RowHash h;
            h.hb = h.rb = 0;
            h.mask = 0xffffffffu;
            h.lo = 0;
            if (keepmask & (1u << lane)) h = row_hash(sm, u);
            W.rhb[lane] = h.hb;
            W.rrb[lane] = h.rb;
            W.rmask[lane] = h.mask;
            W.rlo[lane] = h.lo;
            W.tvs[lane] = u;
            W.te[lane] = fa.vexp[u];
        }
        const ProbParams P = a.probs[a.eprob[T]];
        const double *pw = KIND == MIX_SINGULAR ? fa.pw + (long long)a.eprob[T] * PW_N : nullptr;
        const double *ET64 = &a.EC[(long long)T * 6];
        const float ohi0 = a.EChi[(long long)T * 6], ohi1 = a.EChi[(long long)T * 6 + 1];
        const float olo0 = a.EClo[(long long)T * 6], olo1 = a.EClo[(long long)T * 6 + 1];
        const double dT = a.adet[T];
        for (int k = lane; k < nPx; k += 32) {
            xtoPhys<2>(ET64, &rule.Px[2 * k], &x64[2 * k]);
            xf[k] = f2((float)(x64[2 * k] - ET64[0]), (float)(x64[2 * k + 1] - ET64[1]));
        }
        for (int i = lane; i < 7 * nPx; i += 32) {
            const int k = i / 7, q = i - 7 * k;
            coef[i] = dT * (q < 3 ? pr.cx[3 * k + q] : (q < 6 ? pr.cxx[6 * k + (q == 5 ? 4 : q - 2)] : pr.dxf[k]));
        }
        __syncwarp();
        int et[3];   // eighths of a bit: the unit exponent of T's rows
#pragma unroll
        for (int r = 0; r < 3; r++) et[r] = 8 * F64_BITS - P.xN - W.te[r];
        const double dTs = scale2(dT, F64_BITS - P.xS);
        const int limN = CK ? F64_BITS : P.limN, limE = CK ? F64_BITS : P.limE;
        double D[3] = {0, 0, 0};   // termLocal of T's pairs, off-diagonal
        const bool frac_close = KIND == MIX_SINGULAR && duffy_close(P);
        int part_next = lb + lane < le ? a.pB[lb + lane] : T;   // partners one batch ahead
        for (long long p0 = lb; p0 < le; p0 += 32) {
            const long long p = p0 + lane;
            const bool act = p < le;
            const bool near = min(p0 + 32, le) <= ln;   // the whole batch: no classes to find
            const int part = part_next;
            part_next = p + 32 < le ? a.pB[p + 32] : T;
            int pv[3];
#pragma unroll
            for (int r = 0; r < 3; r++) pv[r] = a.T32[(long long)part * 3 + r];
            bool close = false;
            if (frac_close && act) {
                close = (part == T);
#pragma unroll
                for (int i = 0; i < 3; i++)
#pragma unroll
                    for (int j = 0; j < 3; j++) close |= (tv[i] == pv[j]);
            }
            const double rb = a.adet[part];
            const int eb = exp_above(rb);
            int ve[3];
#pragma unroll
            for (int c = 0; c < 3; c++) ve[c] = fa.vexp[pv[c]];
            W.pid[lane] = part;
            W.pe[lane] = eb;
#pragma unroll
            for (int c = 0; c < 3; c++) W.pve[lane][c] = ve[c];
            unsigned inm = 0, cutm = 0;
            if (act && near) inm = nPx >= 32 ? 0xffffffffu : (1u << nPx) - 1u;
            if (act && !close && !(CK && near)) {
                float pc[6];
#pragma unroll
                for (int j = 0; j < 6; j++)
                    pc[j] = (a.EChi[(long long)part * 6 + j] - ((j & 1) ? ohi1 : ohi0)) + (a.EClo[(long long)part * 6 + j] - ((j & 1) ? olo1 : olo0));
#pragma unroll
                for (int j = 0; j < 3; j++) W.pc[lane][j] = f2(pc[2 * j], pc[2 * j + 1]);
                for (int k = 0; k < (near ? 0 : nPx); k++) {
                    const F2 x = xf[k];
                    const F2 Q[3] = {f2(pc[0] - x.x, pc[1] - x.y), f2(pc[2] - x.x, pc[3] - x.y), f2(pc[4] - x.x, pc[5] - x.y)};
                    const int c = P.cert ? fclassify(Q, P.sqdelta_f) : f64_class(P.sqdelta, &x64[2 * k], &a.EC[(long long)part * 6]);
                    inm |= (unsigned)(c == CLS_IN) << k;
                    cutm |= (unsigned)(c == CLS_CUT) << k;
                }
            }
            nitin += __popc(inm);
            nitcut += __popc(cutm);
            if (CK) nsub += __popc(inm);
            // items, pair by pair, in chunks of whole pairs; inside and cut items are integrated apart,
            // so that a warp does not run both paths
            const unsigned itm = CK ? cutm : inm | cutm;
            const int cnt = __popc(itm), cin = CK ? 0 : __popc(inm);
            const int sc = warp_incl_scan(cnt | cin << 16, lane);
            const int incl = sc & 0xffff, off = incl - cnt, offin = (sc >> 16) - cin;
            const int total = __shfl_sync(FULL, incl, 31);
            for (int base = 0, basein = 0; base < total;) {
                const bool mine = cnt > 0 && off >= base && off + cnt <= base + F64_CAP;
                const unsigned who = __ballot_sync(FULL, mine);
                const int last = 31 - __clz(who);
                const int end = __shfl_sync(FULL, incl, last), endin = __shfl_sync(FULL, sc >> 16, last);
                const int n = end - base, nin = endin - basein;
                if (mine) {
                    int w = off - base, wi = offin - basein, wc = nin + w - wi;
                    const int r = __popc(who & lanemask_lt());
                    W.pl[r] = (unsigned char)lane;
                    W.ps[r] = (unsigned char)w;
                    W.pn[r] = (unsigned char)cnt;
                    for (unsigned mm = itm; mm; mm &= mm - 1) {
                        const int k = __ffs(mm) - 1;
                        const unsigned in = (inm >> k) & 1u;
                        if (!CK) W.order[in ? wi++ : wc++] = (unsigned char)w;
                        W.list[w++] = (unsigned short)(lane << 6 | in << 5 | k);
                    }
                }
                __syncwarp();
                unsigned late = 0;   // bit r: this lane's r-th item of the chunk needs the exact routine
                for (int part0 = 0; part0 < (CK ? 1 : 2); part0++) {   // inside items, then cut items
                    const int first = CK || part0 == 0 ? 0 : nin, past = CK || part0 ? n : nin;
                    for (int i0 = first + lane, r = 0; i0 < past; i0 += 32, r++) {
                        const int i = CK ? i0 : W.order[i0], it = W.list[i], k = it & 31, j = it >> 6, b = W.pid[j];
                        const F2 xk = xf[k], Qf[3] = {W.pc[j][0] - xk, W.pc[j][1] - xk, W.pc[j][2] - xk};
                        const bool inside = !CK && part0 == 0;
                        if ((!P.cert && !inside) || !f64_item<KIND, false>(P, rule, pr, inside, fa.exact, pw, &x64[2 * k], Qf, &a.EC[(long long)b * 6],
                                                   a.adet[b], fa.idet[b], &res[i * F64_RN], nsub))
                            late |= 1u << r;
                    }
                }
                for (; late; late &= late - 1) {
                    const int i0 = (CK ? 0 : nin) + lane + 32 * (__ffs(late) - 1);
                    const int i = CK ? i0 : W.order[i0], it = W.list[i], b = W.pid[it >> 6];
                    nsub += f64_item_late<KIND>(&a.probs[a.eprob[T]], rule, pr, fa.exact, pw, &x64[2 * (it & 31)],
                                                &a.EC[(long long)b * 6], a.adet[b], fa.idet[b], &res[i * F64_RN]);
                }
                __syncwarp();
                const int nun = __popc(who) * F64_OUT;
                for (int u = lane; u < nun; u += 32) {
                    const int r = u / F64_OUT, o = u - r * F64_OUT, pl = W.pl[r];
                    const int ci = o < 9 ? o / 3 : (o < 12 ? o - 6 : 6);
                    const int ri = o < 9 ? 1 + o % 3 : (o < 12 ? 0 : o - 8);
                    double v = 0;
                    for (int i = W.ps[r], e = i + W.pn[r]; i < e; i++) v += coef[7 * (W.list[i] & 31) + ci] * res[i * F64_RN + ri];
                    long long *A = &acc[pl * F64_ACC];
                    if (o < 12) A[o] = __double_as_longlong(v);
                    else f64_split2(scale2(v, F64_BITS - P.xD - W.pe[pl]), limE, bad, A[o], A[o + 3]);
                }
                __syncwarp();
                base = end;
                basein = endin;
            }
            // owner: the pair's termNonloc (termLocal is summed per lane)
            const long long *A = &acc[lane * F64_ACC];
            double nx[9];
#pragma unroll
            for (int i = 0; i < 9; i++) nx[i] = cnt ? __longlong_as_double(A[i]) : 0.0;
            long long *ep = &fa.m.elp[(long long)part * F64_ELP];
            if (CK && inm) {   // inside items: kc |T| |b| times the rule's sums
                double m[7];
#pragma unroll
                for (int q = 0; q < 7; q++) m[q] = tab[7 * (inm & 255u) + q];
                for (int b = 1; 8 * b < nPx; b++)
#pragma unroll
                    for (int q = 0; q < 7; q++) m[q] += tab[7 * (256 * b + ((inm >> (8 * b)) & 255u)) + q];
                const double kr = P.kc * dT * rb;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const double iN = kr * pr.insum[1 + c];
#pragma unroll
                    for (int r = 0; r < 3; r++) nx[3 * r + c] = fma(m[r], iN, nx[3 * r + c]);
                }
                const double kl = kr * pr.insum[0];
#pragma unroll
                for (int q = 0; q < 3; q++) D[q] += m[3 + q] * kl;
                long long hi, lo;
                f64_split2(m[6] * dTs, limE, bad, hi, lo);
                red_add(ep, 0, hi);
                if (lo) red_add(ep, 1, lo);
            }
            if (cnt) {
#pragma unroll
                for (int q = 0; q < 3; q++) D[q] += __longlong_as_double(A[9 + q]);
#pragma unroll
                for (int q = 0; q < 6; q++) red_add(ep, 2 + q, A[12 + q]);
            }
            if (KIND == MIX_SINGULAR && close) {   // Duffy blocks (their termNonlocPrime is termNonloc)
                nclose++;
                const long long cs = close_slot(a.xadj, a.adj, T, part);
                if (cs < 0) {
                    miss = true;
                } else {
                    const double *cb = &a.closebuf[cs * 36];
                    D[0] += cb[1]; D[1] += cb[2]; D[2] += cb[5];
#pragma unroll
                    for (int q = 0; q < 3; q++) {
                        long long hi, lo;
                        f64_split2(scale2(cb[q == 2 ? 23 : 19 + q], F64_BITS - P.xD - eb), limE, bad, hi, lo);
                        red_add(ep, 2 + q, hi);
                        red_add(ep, 5 + q, lo);
                    }
#pragma unroll
                    for (int i = 0; i < 9; i++) nx[i] = cb[9 + i];
                }
            }
            // termNonloc into T's own rows: lanes sharing a partner vertex add their integers, all
            // lanes share the (vertex, row) lookups; the mirrored entries come from k_sym_add_f64
            __syncwarp();
            int nent = 0;
            auto slot_of = [&](int r, int col) {   // of T's row r; -2: no such entry is kept
                RowHash h;
                h.hb = W.rhb[r]; h.rb = W.rrb[r]; h.mask = W.rmask[r]; h.lo = W.rlo[r];
                if (col == W.tvs[r]) return -2LL;   // the matrix diagonal: from the row sum
                if (h.mask != 0xffffffffu) return slot_find_row(sm, h, col);
                if (a.labV[col] > 0) return slot_find(sm, col, W.tvs[r]);   // T's vertex has no row: the mirror
                return -2LL;
            };
#pragma unroll 1
            for (int c = 0; c < 3; c++) {
                const int col = act ? sel3(pv, c) : -1;
                long long o[3], ol[3], s[3], sl[3];
                double q[3];
                unsigned rests = 0;
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    bool rest = false;
                    q[r] = scale2(sel3(&nx[3 * r], c), (et[r] - sel3(ve, c)) >> 3);
                    f64_split(q[r], limN, bad, o[r], ol[r], rest);
                    rests |= (unsigned)rest << r;
                    s[r] = o[r];
                    sl[r] = ol[r];
                }
                if (__any_sync(FULL, rests)) {   // slivers (about one cut item in 1000): third integers
#pragma unroll
                    for (int r = 0; r < 3; r++) {
                        const long long st = (rests >> r) & 1u ? slot_of(r, col) : -1;
                        if (st < 0) continue;   // the scatter below reports what is missing
                        red_add(fa.valsNt, st, f64_third(q[r]));
                        a.err[F64_ERR_THIRD] = 1;
                    }
                }
                const bool wide = __any_sync(FULL, ol[0] | ol[1] | ol[2]);
                const unsigned grp = __match_any_sync(FULL, col);
                const bool leader = (__ffs(grp) - 1) == lane;
                const int maxn = __reduce_max_sync(FULL, (unsigned)__popc(grp));
                unsigned rest = grp & ~(1u << lane);
                for (int it = 1; it < maxn; it++) {
                    const int src = rest ? __ffs(rest) - 1 : lane;
                    const bool use = rest != 0;
                    if (rest) rest &= rest - 1;
#pragma unroll
                    for (int r = 0; r < 3; r++) {
                        const long long t = shfl64(o[r], src);
                        if (use) s[r] += t;
                    }
                    if (!wide) continue;
#pragma unroll
                    for (int r = 0; r < 3; r++) {
                        const long long t = shfl64(ol[r], src);
                        if (use) sl[r] += t;
                    }
                }
                const bool put = leader && col >= 0;
                const unsigned m = __ballot_sync(FULL, put);
                if (put) {
                    F64Entry &e = slist[nent + __popc(m & lanemask_lt())];
                    e.col = col;
#pragma unroll
                    for (int r = 0; r < 3; r++) { e.v[r] = s[r]; e.v[3 + r] = sl[r]; }
                }
                nent += __popc(m);
            }
            __syncwarp();
            for (int w = lane; w < 3 * nent; w += 32) {
                const int e = w / 3, r = w - 3 * e;
                const long long st = slot_of(r, slist[e].col);
                if (st < 0) { miss |= st == -1; continue; }
                red_add(fa.m.valsN, 2 * st, slist[e].v[r]);
                if (slist[e].v[3 + r]) red_add(fa.m.valsN, 2 * st + 1, slist[e].v[3 + r]);
            }
            __syncwarp();
        }
        // termLocal of all of T's pairs into T's diagonal block
#pragma unroll
        for (int i = 0; i < 3; i++) D[i] = warp_sum(D[i]);
        if (lane < 9 && lane / 3 != lane % 3) {   // off-diagonal entries (the diagonal: k_sym_add_f64)
            const int r = lane / 3, c = lane % 3;
            const int s = sm.dslot[(long long)T * 9 + lane];
            const double d = r + c == 1 ? D[0] : (r + c == 2 ? D[1] : D[2]);
            if (s >= 0) {
                long long hi, lo;
                f64_split2(scale2(d, F64_BITS - P.xD - ((W.te[r] + 7) >> 3)), CK ? F64_BITS : P.limD, bad, hi, lo);
                red_add(vals, s, hi);
                red_add(fa.valslo, s, lo);
            } else if (keepmask & (1u << r)) miss = true;
        }
        __syncwarp();
    }
    if (__any_sync(FULL, bad) && lane == 0) atomicOr(&a.err[5], 1);
    if (__any_sync(FULL, miss) && lane == 0) atomicOr(&a.err[3], 1);
    nsub = warp_sum(nsub);
    nclose = warp_sum(nclose);
    nitin = warp_sum(nitin);
    nitcut = warp_sum(nitcut);
    if (lane == 0) {
        if (nsub && a.n_subtri) atomicAdd(a.n_subtri, (unsigned long long)nsub);
        if (nclose && a.n_close) atomicAdd(a.n_close, (unsigned long long)nclose);
        if (nitin && a.n_in) atomicAdd(a.n_in, (unsigned long long)nitin);
        if (nitcut && a.n_cut) atomicAdd(a.n_cut, (unsigned long long)nitcut);
    }
}

// vexp of every vertex: 8 log2 of its elements' |det| sum, rounded up (with a margin far above the
// logarithm's rounding).
__global__ void k_vexp(const long long *__restrict__ vptr, const int *__restrict__ vel, const double *__restrict__ adet,
                       long long nV, int *__restrict__ vexp) {
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nV) return;
    double s = 0;
    for (long long i = vptr[v]; i < vptr[v + 1]; i++) s += adet[vel[i]];
    vexp[v] = s > 1e-270 ? (int)ceil(8.0 * log2(s) + 1e-3) : -7200;
}

// termLocalPrime sums of each element into its diagonal-block slots, in their rows' units. The
// inside part of a constant kernel is kc |b| times its summed outer weights times the inner rule's
// sums in01, in02, in12 of psi_r psi_c.
__global__ void k_elem_blocks_f64(const long long *__restrict__ elp, const double *__restrict__ adet,
                                  const int *__restrict__ vexp, const int *__restrict__ dslot,
                                  const int *__restrict__ T32, const int *__restrict__ labV,
                                  const int *__restrict__ eprob, const ProbParams *__restrict__ probs, double in01,
                                  double in02, double in12, long long nE, long long *__restrict__ vals,
                                  long long *__restrict__ valslo, int *__restrict__ err) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nE) return;
    const long long *p = &elp[e * F64_ELP];
    if ((p[0] | p[1] | p[2] | p[3] | p[4] | p[5] | p[6] | p[7]) == 0) return;
    const ProbParams &P = probs[eprob[e]];
    const double in[3] = {in01, in02, in12};
    const double kin = scale2(f64_join(p[0], p[1]), P.xS - F64_BITS) * (P.kc * adet[e]);
    const int eb = exp_above(adet[e]);
    double b[3];
#pragma unroll
    for (int q = 0; q < 3; q++) b[q] = kin * in[q] + scale2(f64_join(p[2 + q], p[5 + q]), P.xD + eb - F64_BITS);
    bool bad = false;
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) {
            if (r == c) continue;   // the diagonal comes from the row sum (k_sym_add_f64)
            const int v = T32[e * 3 + r], s = dslot[e * 9 + 3 * r + c];
            if (s >= 0) {
                long long hi, lo;
                f64_split2(scale2(b[r + c - 1], F64_BITS - P.xD - ((vexp[v] + 7) >> 3)), P.limD, bad, hi, lo);
                red_add(vals, s, hi);
                red_add(valslo, s, lo);
            } else if (labV[v] > 0) {
                atomicOr(&err[3], 1);
            }
        }
    if (bad) atomicOr(&err[5], 1);
}

// The FP64 matrix from the sums: entry (t, v) is the diagonal blocks' part minus the termNonloc sums
// of the slot and of its transposed slot (tpos null: rules without Prime blocks have none); each diagonal entry is minus its row's other entries. vals
// is replaced in place by FP64 values. One warp per row; HBM-bound (each slot's sums are read
// twice).
__global__ void k_sym_add_f64(const long long *__restrict__ rowptr, const int *__restrict__ cols,
                              const int *__restrict__ tpos, const long long *__restrict__ valsN,
                              const long long *__restrict__ valsNt, const long long *__restrict__ valslo,
                              const int *__restrict__ vexp, const int *__restrict__ vprob,
                              const ProbParams *__restrict__ probs, long long nrows, const int *__restrict__ err,
                              double *__restrict__ vals) {
    const int lane = threadIdx.x & 31;
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    const bool third = err[F64_ERR_THIRD] != 0;
    const longlong2 *N = reinterpret_cast<const longlong2 *>(valsN);
    auto sum_of = [&](long long s) {
        const longlong2 q = N[s];
        return f64_join(q.x, q.y, third ? valsNt[s] : 0);
    };
    for (long long t = gw; t < nrows; t += nw) {
        const long long b = rowptr[t], e = rowptr[t + 1];
        if (b == e) continue;
        const ProbParams &P = probs[vprob[t]];
        const int et = vexp[t], eN = 8 * F64_BITS - P.xN - et, eD = P.xD + ((et + 7) >> 3) - F64_BITS;
        double off = 0;
        long long dslot = -1;
        for (long long s = b + lane; s < e; s += 32) {
            const int v = cols[s];
            if (v == (int)t) { dslot = s; continue; }
            const int tp = tpos ? tpos[s] : -1;
            const long long ts = tp >= 0 ? rowptr[v] + tp : -1;
            double q = sum_of(s);
            if (ts >= 0) q += sum_of(ts);
            const long long dh = reinterpret_cast<const long long *>(vals)[s];
            double x = -scale2(q, -((eN - vexp[v]) >> 3));
            if (dh | valslo[s]) x += scale2(f64_join(dh, valslo[s]), eD);   // a slot of a diagonal block
            vals[s] = x;
            off += x;
        }
        off = warp_sum(off);
        if (dslot >= 0) vals[dslot] = -off;   // the row sums to zero
    }
}

}  // namespace nlg
