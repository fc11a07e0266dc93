// Mixed-precision 2D retriangulate pass: one-sided, work-compacted, fixed-point scatter.
//
// One warp per outer element T (taken from a global work counter, so no coloring is needed).
// For each batch of 32 interacting pairs (T, b), every lane classifies its pair's outer points
// (ball contains b / misses it / cuts it); the (pair, outer point) items are compacted into an
// "inside" list and a "cut" list and processed 32 at a time, each item writing its inner sums to
// its own shared-memory slot; the owning lane then folds the slots into the pair's blocks in a
// fixed order (integrate_retriangulate, integration.cpp:345-540):
//   termLocal L (T x T), termNonloc N (T x b), termLocalPrime LP (b x b).
// All kernels of this path are functions of |x - y|, so k(y, x) = k(x, y) and
// termNonlocPrime = termNonloc exactly; the pair therefore contributes
//   A[T, T] += L,  A[T, b] -= N,  A[b, T] -= N^T,  A[b, b] += LP
// (Cassemble.cpp:737-766) and the inner element's side of the pair needs no second geometry.
// Close pairs of the singular kernel take their four FP64 blocks from closebuf instead.
// Contributions are added to the CSR values as 64-bit fixed-point integers (slots.cuh), so the
// matrix does not depend on the order in which warps finish.
#pragma once
#include "passes.cuh"
#include "slots.cuh"

namespace nlg {

constexpr int MIX_WARPS = 4;
constexpr int MIX_THREADS = 32 * MIX_WARPS;
constexpr int RES_N = 7;    // per item: innerLocal, innerNonloc[3], off-diagonal termLocalPrime sums[3] (the matrix
                            // diagonal comes from the row sums); the odd stride keeps the banks apart
// upper-triangle positions of the off-diagonal entries (0, 1), (0, 2), (1, 2)
__host__ __device__ __forceinline__ constexpr int off3(int q) { return q == 2 ? 4 : q + 1; }
constexpr int SCAT_U = 1;   // slot lookups per lane whose first accesses are issued together (more
                            // unrolling overflows the instruction cache of this kernel)

// Per-warp shared scratch; nPx-dependent arrays follow the struct in dynamic shared memory:
// the outer points of T (FP64, exact; FP32 relative to T's vertex 0), the item results and the
// item lists.
struct MixWarp {
    float pc[32][6];            // partner element, local coordinates
    float prt[32];              // partner |det|
    int pid[32];            // partner element
    long long rhb[3], rrb[3];   // T's rows: slot map start, CSR row start
    unsigned rmask[3];          // T's rows: slot map size field (0xffffffff: no row), see RowHash
    int rlo[3];                 // T's rows: first window word (window-rank map)
    int tvs[3];                 // T's vertices
};
// The vertices of a batch's partners, each with the lanes that hold it: per entry its vertex and, for
// every local vertex c, the lanes whose c-th vertex it is. Vertices meet in a small table in shared
// memory: every (lane, c) writes itself at its vertex's low bits, and who finds its own vertex there
// joins that writer's entry. Others (two vertices with the same low bits) have an entry of their own: a
// vertex may have several entries, and the users' integer sums allow that. Against one __match_any_sync
// per local vertex a vertex has one entry instead of up to three; k_pass_near2d at n = 256, delta = 0.1:
// 18.8 against 19.7 ms (9.8 since the lists came in element order).
constexpr int GROUP_TAB = 512;
template <int DV>
struct VertexGroups {
    int col[32 * DV];              // every (c, lane)'s vertex
    int vert[32 * DV];             // entries: vertex
    unsigned lanes[32 * DV][DV];   // entries: lanes by local vertex
    unsigned char id[32 * DV];     // entry of a leading (c, lane)
    unsigned char tab[GROUP_TAB];
};
// The entries of pv (DV vertices of every active lane); returns their number. A barrier of the warp
// lies between this and the last readers of g before, and at its end.
template <int DV>
__device__ __forceinline__ int group_vertices(VertexGroups<DV> &g, const int *pv, bool act) {
    const int lane = threadIdx.x & 31;
    if (act) {
#pragma unroll
        for (int c = 0; c < DV; c++) {
            g.col[32 * c + lane] = pv[c];
            g.tab[pv[c] & (GROUP_TAB - 1)] = (unsigned char)(32 * c + lane);
        }
    }
    __syncwarp();
    int n = 0, lead[DV];
#pragma unroll
    for (int c = 0; c < DV; c++) {
        lead[c] = 32 * c + lane;
        if (act) {
            const int w = g.tab[pv[c] & (GROUP_TAB - 1)];
            if (g.col[w] == pv[c]) lead[c] = w;
        }
        const bool put = act && lead[c] == 32 * c + lane;
        const unsigned m = __ballot_sync(FULL, put);
        if (put) {
            const int e = n + __popc(m & lanemask_lt());
            g.id[32 * c + lane] = (unsigned char)e;
            g.vert[e] = pv[c];
#pragma unroll
            for (int i = 0; i < DV; i++) g.lanes[e][i] = 0;
        }
        n += __popc(m);
    }
    __syncwarp();
    if (act) {
#pragma unroll
        for (int c = 0; c < DV; c++) atomicOr(&g.lanes[g.id[lead[c]]][c], 1u << lane);
    }
    __syncwarp();
    return n;
}

struct VertexGroup {   // lanes of a batch whose partners share a vertex (as local vertex c)
    int col, c;
    unsigned lanes;
};
// One column group of a batch: the partner vertex and the integer sums of its three rows
// (termNonloc into A[T, v], termNonlocPrime into A[v, T]). Stored over the item results.
struct ScatEntry {
    int col, pad;
    long long v[6];
};
__host__ __device__ constexpr size_t mix_res_bytes(int nPx) {
    return (size_t)32 * nPx * RES_N * sizeof(float) > 96 * sizeof(ScatEntry) ? (size_t)32 * nPx * RES_N * sizeof(float)
                                                                          : 96 * sizeof(ScatEntry);
}
__host__ __device__ constexpr size_t mix_warp_bytes(int nPx) {
    // MixWarp + x64[nPx * 2] doubles + xf[nPx] 2-vectors + res[32][nPx][RES_N] (or the scatter
    // list) + lists[2][32 * nPx] shorts
    return ((sizeof(MixWarp) + 15) / 16) * 16 + (size_t)nPx * 16 + ((size_t)nPx * 2 * sizeof(float) + 15) / 16 * 16 +
           mix_res_bytes(nPx) + (size_t)2 * 32 * nPx * 2 + 16;
}


struct MixArgs {
    PassArgs p;
    SlotMap m;
    int *work;   // global element counter
    // one-sided retriangulate pass only:
    long long *valsN;   // termNonloc of each outer element into its own rows; the transposed
                        // contributions come from k_sym_add (the matrix is symmetric)
    long long *elp;     // termLocalPrime per partner element, upper triangle (k_elem_blocks adds
                        // it to the diagonal-block slots)
};

// Inner sums of one "inside" item: the ball around x contains the partner element b.
__device__ __forceinline__ void item_in(const ProbParams &P, const Rule &rule, const PassRule &pr,
                                        const float *pc, float rT, F2 x, float *res) {
    const float *Py = rule.Pyf, *dy = rule.dyf;
    const F2 p0 = f2(pc[0] - x.x, pc[1] - x.y);
    const F2 e1 = f2(pc[2] - pc[0], pc[3] - pc[1]), e2 = f2(pc[4] - pc[0], pc[5] - pc[1]);
    float iL = 0, i0 = 0, i1 = 0, i2 = 0;
    float lp[3] = {0, 0, 0};
#pragma unroll 1   // the compiler's unrolling cost the parabola instance 9% (instruction cache)
    for (int i = 0; i < rule.nPy; i++) {
        const float px = Py[2 * i], py = Py[2 * i + 1];
        const float yx = p0.x + e1.x * px + e2.x * py;
        const float yy = p0.y + e1.y * px + e2.y * py;
        const float kw = kernel_f32(P, -yx, -yy) * rT;
        iL = fmaf(kw, dy[i], iL);
        i0 = fmaf(kw, pr.cy[3 * i + 0], i0);
        i1 = fmaf(kw, pr.cy[3 * i + 1], i1);
        i2 = fmaf(kw, pr.cy[3 * i + 2], i2);
#pragma unroll
        for (int q = 0; q < 3; q++) lp[q] = fmaf(kw, pr.cyy[6 * i + off3(q)], lp[q]);
    }
    res[0] = iL; res[1] = i0; res[2] = i1; res[3] = i2;
#pragma unroll
    for (int q = 0; q < 3; q++) res[4 + q] = lp[q];
}

// Inner sums of one "cut" item: polygon of B(x) and b (certified FP32 with the exact FP64
// fallback, or the exact FP64 routine), fan sub-triangles, basis of b by the inverse affine map.
__device__ __forceinline__ void item_cut(const ProbParams &P, const Rule &rule, const float *pc, F2 x,
                                         const double *x64, const double *Eb64, float *res,
                                         unsigned &nsub, unsigned &namb) {
    const float *Py = rule.Pyf, *dy = rule.dyf;
    const F2 Q[3] = {f2(pc[0] - x.x, pc[1] - x.y), f2(pc[2] - x.x, pc[3] - x.y), f2(pc[4] - x.x, pc[5] - x.y)};
    const F2 e1 = Q[1] - Q[0], e2 = Q[2] - Q[0];
    const float idet = 1.f / (e1.x * e2.y - e1.y * e2.x);
    F2 Rp[9];
    const int n = cut_polygon(Q, P.sqdelta_f, P, x64, Eb64, Rp, namb);
    float iL = 0, i0 = 0, i1 = 0, i2 = 0;
    float lp[3] = {0, 0, 0};
    for (int r = 0; r + 2 < n; r++) {
        nsub++;
        const F2 Av = Rp[0], B = Rp[r + 1] - Rp[0], C = Rp[r + 2] - Rp[0];
        const float rT = fabsf(B.x * C.y - B.y * C.x);
#pragma unroll 1
        for (int i = 0; i < rule.nPy; i++) {
            const float px = Py[2 * i], py = Py[2 * i + 1];
            const float yx = Av.x + B.x * px + C.x * py;
            const float yy = Av.y + B.y * px + C.y * py;
            const float kw = kernel_f32(P, -yx, -yy) * rT * dy[i];
            const float dxr = yx - Q[0].x, dyr = yy - Q[0].y;
            const float r0 = (e2.y * dxr - e2.x * dyr) * idet;
            const float r1 = (e1.x * dyr - e1.y * dxr) * idet;
            const float s0 = 1.f - r0 - r1;
            iL += kw;
            i0 = fmaf(kw, s0, i0);
            i1 = fmaf(kw, r0, i1);
            i2 = fmaf(kw, r1, i2);
            lp[0] = fmaf(kw, s0 * r0, lp[0]);
            lp[1] = fmaf(kw, s0 * r1, lp[1]);
            lp[2] = fmaf(kw, r0 * r1, lp[2]);
        }
    }
    res[0] = iL; res[1] = i0; res[2] = i1; res[3] = i2;
#pragma unroll
    for (int q = 0; q < 3; q++) res[4 + q] = lp[q];
}

// Inner sums of one "cut" item for a constant kernel. The kernel weight of every inner point is
// kc |S| dy_i, and the basis functions of b are affine, so on a fan sub-triangle S = (A, B, C)
// psi_a(y_i) = psi_a(A) + (psi_a(B) - psi_a(A)) px_i + (psi_a(C) - psi_a(A)) py_i, and the rule's
// sums over S follow from its moments m = sum_i dy_i (1, px, py, px^2, px py, py^2):
//   sum_i dy_i psi_a = al_a m0 + be_a mx + ga_a my,
//   sum_i dy_i psi_a psi_b = al_a t0_b + be_a t1_b + ga_a t2_b  (t_b the first sums of psi_b with
//   weights (1, px, py)).
// This equals the quadrature sum of the general item for any rule. The basis values come from the
// polygon's points (one evaluation per point instead of per inner point), and every sum stays in
// the basis functions' own range, so no cancellation enters where a basis function is small.
__device__ __forceinline__ void item_cut_const(const ProbParams &P, const PassRule &pr, const float *pc,
                                               F2 x, const double *x64, const double *Eb64, float *res,
                                               unsigned &nsub, unsigned &namb) {
    const F2 Q[3] = {f2(pc[0] - x.x, pc[1] - x.y), f2(pc[2] - x.x, pc[3] - x.y), f2(pc[4] - x.x, pc[5] - x.y)};
    const F2 e1 = Q[1] - Q[0], e2 = Q[2] - Q[0];
    const float idet = 1.f / (e1.x * e2.y - e1.y * e2.x);
    F2 Rp[9];
    const int n = cut_polygon(Q, P.sqdelta_f, P, x64, Eb64, Rp, namb);
    const float m0 = pr.mom[0], mx = pr.mom[1], my = pr.mom[2], mxx = pr.mom[3], mxy = pr.mom[4], myy = pr.mom[5];
    auto basis = [&](F2 y, float *l) {   // psi_0..2 of b at y (as the general item evaluates them)
        const float dxr = y.x - Q[0].x, dyr = y.y - Q[0].y;
        l[1] = (e2.y * dxr - e2.x * dyr) * idet;
        l[2] = (e1.x * dyr - e1.y * dxr) * idet;
        l[0] = 1.f - l[1] - l[2];
    };
    float S0 = 0, S1[3] = {0, 0, 0}, S2[3] = {0, 0, 0};
    float la[3], lb[3], lc[3];
    if (n >= 3) {
        basis(Rp[0], la);
        basis(Rp[1], lb);
    }
    for (int r = 0; r + 2 < n; r++) {
        nsub++;
        const F2 B = Rp[r + 1] - Rp[0], C = Rp[r + 2] - Rp[0];
        const float rT = fabsf(B.x * C.y - B.y * C.x);
        basis(Rp[r + 2], lc);
        float t0[3], t1[3], t2[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const float al = la[q], be = lb[q] - la[q], ga = lc[q] - la[q];
            t0[q] = fmaf(al, m0, fmaf(be, mx, ga * my));
            t1[q] = fmaf(al, mx, fmaf(be, mxx, ga * mxy));
            t2[q] = fmaf(al, my, fmaf(be, mxy, ga * myy));
        }
        S0 = fmaf(rT, m0, S0);
#pragma unroll
        for (int q = 0; q < 3; q++) {
            S1[q] = fmaf(rT, t0[q], S1[q]);
            const float al = la[q], be = lb[q] - la[q], ga = lc[q] - la[q];
#pragma unroll
            for (int q2 = q + 1; q2 < 3; q2++)
                S2[q + q2 - 1] = fmaf(rT, fmaf(al, t0[q2], fmaf(be, t1[q2], ga * t2[q2])), S2[q + q2 - 1]);
        }
#pragma unroll
        for (int q = 0; q < 3; q++) lb[q] = lc[q];
    }
    const float kc = P.kc_f;
    res[0] = kc * S0;
#pragma unroll
    for (int q = 0; q < 3; q++) res[1 + q] = kc * S1[q];
#pragma unroll
    for (int q = 0; q < 3; q++) res[4 + q] = kc * S2[q];
}

// Appends this lane's items of class cls (one per outer point k with that class) to list, in
// (k, lane) order; returns the list length (uniform).
__device__ __forceinline__ int build_list(const unsigned char *mycls, int nPx, int cls,
                                          unsigned short *list) {
    const int lane = threadIdx.x & 31;
    int n = 0;
    for (int k = 0; k < nPx; k++) {
        const bool mine = mycls[k] == cls;
        const unsigned m = __ballot_sync(FULL, mine);
        if (mine) list[n + __popc(m & lanemask_lt())] = (unsigned short)(k * 32 + lane);
        n += __popc(m);
    }
    __syncwarp();
    return n;
}

// The same from a bit mask of the lane's outer points (bit k: item (k, lane) is in the list).
__device__ __forceinline__ int build_list_mask(unsigned mask, int nPx, unsigned short *list) {
    const int lane = threadIdx.x & 31;
    int n = 0;
    for (int k = 0; k < nPx; k++) {
        const bool mine = (mask >> k) & 1u;
        const unsigned m = __ballot_sync(FULL, mine);
        if (mine) list[n + __popc(m & lanemask_lt())] = (unsigned short)(k * 32 + lane);
        n += __popc(m);
    }
    __syncwarp();
    return n;
}

// a[i] for i in {0, 1, 2} as register selects (no dynamic indexing of register arrays)
template <typename X>
__device__ __forceinline__ X sel3(const X *v, int i) {
    return i == 0 ? v[0] : (i == 1 ? v[1] : v[2]);
}

__device__ __forceinline__ long long shfl64(long long v, int src) {
    return (long long)__shfl_sync(FULL, (unsigned long long)v, src);
}

// KIND: the kernel class of the launch's problems. MIX_CONST: constant kernels; inside items take
// the rule's precomputed element sums and cut items the moment form (item_cut_const). MIX_REGULAR:
// other kernels without close pairs. MIX_SINGULAR: singular kernels whose close pairs come from
// the Duffy blocks. Each instance holds only its class's code, which keeps the kernel small (it is
// bound by instruction fetch as much as by anything else).
enum { MIX_CONST = 0, MIX_REGULAR = 1, MIX_SINGULAR = 2 };
template <int KIND>
__global__ void __launch_bounds__(MIX_THREADS, 4) k_pass_mix2d(MixArgs ma, Rule rule, PassRule pr) {
    constexpr bool CK = KIND == MIX_CONST;
    extern __shared__ __align__(16) unsigned char s_raw[];
    const PassArgs &a = ma.p;
    const SlotMap &sm = ma.m;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int nPx = rule.nPx;
    unsigned char *wbase = s_raw + (size_t)wib * mix_warp_bytes(nPx);
    MixWarp &W = *reinterpret_cast<MixWarp *>(wbase);
    double *x64 = reinterpret_cast<double *>(wbase + ((sizeof(MixWarp) + 15) / 16) * 16);   // [nPx * 2]
    F2 *xf = reinterpret_cast<F2 *>(x64 + 2 * nPx);                                              // [nPx]
    float *res = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(xf) + ((size_t)nPx * 2 * sizeof(float) + 15) / 16 * 16);   // [32][nPx][RES_N]
    unsigned short *lst = reinterpret_cast<unsigned short *>(reinterpret_cast<unsigned char *>(res) + mix_res_bytes(nPx));   // [2][32*nPx]
    ScatEntry *slist = reinterpret_cast<ScatEntry *>(res);   // scatter list, after the fold
    long long *vals = reinterpret_cast<long long *>(a.vals);
    int *ovf = &a.err[5];
    bool bad = false;   // a contribution outside the fixed-point range (reported at the end)
    bool miss = false;  // a matrix slot not found (reported at the end)
    unsigned nsub = 0, namb = 0, nclose = 0, nitin = 0, nitcut = 0;
    for (;;) {
        int idx = 0;
        if (lane == 0) idx = atomicAdd(ma.work, 1);
        idx = __shfl_sync(FULL, idx, 0);
        if (idx >= a.count) break;
        const int T = a.list ? a.list[idx] : idx;
        const long long l0 = a.out_ptr[T], le = a.out_cnt ? l0 + a.out_cnt[T] : a.out_ptr[T + 1];
        const long long ln = l0 + (a.near_cnt ? a.near_cnt[T] : 0);   // near pairs come first
        const long long lb = CK ? ln : l0;   // constant kernels: k_pass_near2d takes them
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
        }
        const ProbParams P = a.probs[a.eprob[T]];
        const double *ET64 = &a.EC[(long long)T * 6];
        const float ohi0 = a.EChi[(long long)T * 6], ohi1 = a.EChi[(long long)T * 6 + 1];
        const float olo0 = a.EClo[(long long)T * 6], olo1 = a.EClo[(long long)T * 6 + 1];
        const float rTT = a.adetf[T];
        for (int k = lane; k < nPx; k += 32) {
            xtoPhys<2>(ET64, &rule.Px[2 * k], &x64[2 * k]);
            xf[k] = f2((float)(x64[2 * k] - ET64[0]), (float)(x64[2 * k + 1] - ET64[1]));
        }
        __syncwarp();
        long long D[6];   // termLocal of T's pairs, integer sums
#pragma unroll
        for (int i = 0; i < 6; i++) D[i] = 0;
        const bool frac_close = KIND == MIX_SINGULAR && duffy_close(P);   // fractional or weakSingular close blocks
        const float sqf = P.sqdelta_f;
        int part_next = lb + lane < le ? a.pB[lb + lane] : T;   // partners one batch ahead
        for (long long p0 = lb; p0 < le; p0 += 32) {
            const long long p = p0 + lane;
            const bool act = p < le;
            const bool near = !CK && min(p0 + 32, le) <= ln;   // the whole batch: no classes to find
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
            // owner: partner data and classes
            float pc[6];
#pragma unroll
            for (int j = 0; j < 6; j++) {
                pc[j] = (a.EChi[(long long)part * 6 + j] - ((j & 1) ? ohi1 : ohi0)) + (a.EClo[(long long)part * 6 + j] - ((j & 1) ? olo1 : olo0));
            }
#pragma unroll
            for (int j = 0; j < 6; j++) W.pc[lane][j] = pc[j];
            W.prt[lane] = a.adetf[part];
            W.pid[lane] = part;
            // classes as bit masks over the outer points: inm (ball contains the partner), cutm
            // (ball cuts it). Only cut items (and, for other kernels, inside items) write their
            // sums into res; the fold reads res for those items only.
            const unsigned fullm = nPx >= 32 ? 0xffffffffu : (1u << nPx) - 1u;
            unsigned inm = near && act ? fullm : 0, cutm = 0;
            for (int k = 0; k < (near ? 0 : nPx); k++) {
                int c = CLS_OUT;
                if (act && !close) {
                    const F2 x = xf[k];
                    const F2 Q[3] = {f2(pc[0] - x.x, pc[1] - x.y), f2(pc[2] - x.x, pc[3] - x.y), f2(pc[4] - x.x, pc[5] - x.y)};
                    c = fclassify(Q, sqf);
                }
                inm |= (unsigned)(c == CLS_IN) << k;
                cutm |= (unsigned)(c == CLS_CUT) << k;
            }
            nitin += __popc(inm);
            nitcut += __popc(cutm);
            if (CK) nsub += __popc(inm);
            __syncwarp();
            const int nin = CK ? 0 : build_list_mask(inm, nPx, lst);
            const int ncut = near ? 0 : build_list_mask(cutm, nPx, lst + 32 * nPx);
            for (int c0 = 0; c0 < nin; c0 += 32) {
                if (c0 + lane < nin) {
                    const int it = lst[c0 + lane];
                    const int k = it >> 5, j = it & 31;
                    nsub++;
                    item_in(P, rule, pr, W.pc[j], W.prt[j], xf[k], &res[(j * nPx + k) * RES_N]);
                }
            }
            for (int c0 = 0; c0 < ncut; c0 += 32) {
                if (c0 + lane < ncut) {
                    const int it = lst[32 * nPx + c0 + lane];
                    const int k = it >> 5, j = it & 31;
                    if (CK)
                        item_cut_const(P, pr, W.pc[j], xf[k], &x64[2 * k], &a.EC[(long long)W.pid[j] * 6],
                                       &res[(j * nPx + k) * RES_N], nsub, namb);
                    else
                        item_cut(P, rule, W.pc[j], xf[k], &x64[2 * k], &a.EC[(long long)W.pid[j] * 6],
                                 &res[(j * nPx + k) * RES_N], nsub, namb);
                }
            }
            __syncwarp();
            // owner: fold the item sums into the pair's blocks, in fixed point from here on
            long long nx[9], mx[9], lpx[6], lx[6];
#pragma unroll
            for (int i = 0; i < 9; i++) nx[i] = mx[i] = 0;
#pragma unroll
            for (int i = 0; i < 6; i++) lpx[i] = lx[i] = 0;
            // constant kernel: a pair with every outer point inside takes the precomputed sums
            // (lanefull), so its blocks do not depend on the other pairs of its batch; when that
            // holds for every active pair (a warp vote, taken here where all lanes are present)
            // the outer-point loop is skipped
            const bool lanefull = CK && inm == fullm;
            const bool allin = CK && __all_sync(FULL, !act || close || lanefull);
            if (act) {
                if (close) {
                    nclose++;
                    const long long cs = close_slot(a.xadj, a.adj, T, part);
                    if (cs < 0) {
                        miss = true;
                    } else {
                        const double *cb = &a.closebuf[cs * 36];
#pragma unroll
                        for (int i = 0; i < 3; i++)
#pragma unroll
                            for (int j = i + 1; j < 3; j++) lx[sym_idx<3>(i, j)] = fx64d(cb[3 * i + j], P.fx_mul, bad);
#pragma unroll
                        for (int i = 0; i < 9; i++) {
                            nx[i] = fx64d(cb[9 + i], P.fx_mul, bad);    // termNonloc [T vertex][b vertex]
                            mx[i] = fx64d(cb[27 + i], P.fx_mul, bad);   // termNonlocPrime [T vertex][b vertex]
                        }
#pragma unroll
                        for (int i = 0; i < 3; i++)
#pragma unroll
                            for (int j = i + 1; j < 3; j++) lpx[sym_idx<3>(i, j)] = fx64d(cb[18 + 3 * i + j], P.fx_mul, bad);
                    }
                } else {
                    float L[6] = {0, 0, 0, 0, 0, 0}, N[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
                    float LP[3] = {0, 0, 0};
                    // the outer-point loop is warp-uniform (the rule's constants are read at one
                    // address per warp); each lane adds the items its classes select
                    float Axx[6] = {0, 0, 0, 0, 0, 0}, Ax[3] = {0, 0, 0}, Ad = 0;   // inside items (constant kernel)
                    if (lanefull) {   // every item inside: the rule's sums over all outer points
#pragma unroll
                        for (int ab = 0; ab < 6; ab++) Axx[ab] = pr.xsum[ab];
#pragma unroll
                        for (int r = 0; r < 3; r++) Ax[r] = pr.xsum[6 + r];
                        Ad = pr.xsum[9];
                    }
                    if (!allin) {
                        for (int k = 0; k < nPx; k++) {
                            if (lanefull) continue;
                            if (CK && ((inm >> k) & 1u)) {
#pragma unroll
                                for (int ab = 0; ab < 6; ab++) Axx[ab] += pr.cxx[6 * k + ab];
#pragma unroll
                                for (int r = 0; r < 3; r++) Ax[r] += pr.cx[3 * k + r];
                                Ad += pr.dxf[k];
                                continue;
                            }
                            if (!(((inm | cutm) >> k) & 1u)) continue;
                            const float *rr = &res[(lane * nPx + k) * RES_N];
                            const float dk = pr.dxf[k];
#pragma unroll
                            for (int ab = 0; ab < 6; ab++) L[ab] = fmaf(pr.cxx[6 * k + ab], rr[0], L[ab]);
#pragma unroll
                            for (int r = 0; r < 3; r++) {
                                const float c = pr.cx[3 * k + r];
                                N[3 * r + 0] = fmaf(c, rr[1], N[3 * r + 0]);
                                N[3 * r + 1] = fmaf(c, rr[2], N[3 * r + 1]);
                                N[3 * r + 2] = fmaf(c, rr[3], N[3 * r + 2]);
                            }
#pragma unroll
                            for (int q = 0; q < 3; q++) LP[q] = fmaf(dk, rr[4 + q], LP[q]);
                        }
                    }
                    if (CK) {   // an inside item's sums are kc |b| times the rule's element sums
                        float inv[RES_N];   // innerLocal, innerNonloc[3], off-diagonal termLocalPrime[3]
                        const float kr = P.kc_f * W.prt[lane];
#pragma unroll
                        for (int q = 0; q < RES_N; q++) inv[q] = kr * pr.insum[q < 4 ? q : 4 + off3(q - 4)];
#pragma unroll
                        for (int ab = 0; ab < 6; ab++) L[ab] = fmaf(Axx[ab], inv[0], L[ab]);
#pragma unroll
                        for (int r = 0; r < 3; r++) {
                            N[3 * r + 0] = fmaf(Ax[r], inv[1], N[3 * r + 0]);
                            N[3 * r + 1] = fmaf(Ax[r], inv[2], N[3 * r + 1]);
                            N[3 * r + 2] = fmaf(Ax[r], inv[3], N[3 * r + 2]);
                        }
#pragma unroll
                        for (int q = 0; q < 3; q++) LP[q] = fmaf(Ad, inv[4 + q], LP[q]);
                    }
#pragma unroll
                    for (int i = 0; i < 6; i++)   // the diagonal entries come from the row sums (k_sym_add)
                        if (i != 0 && i != 3 && i != 5) lx[i] = fx64(L[i] * rTT, P.fx_mul, bad);
#pragma unroll
                    for (int i = 0; i < 9; i++) mx[i] = nx[i] = fx64(N[i] * rTT, P.fx_mul, bad);
#pragma unroll
                    for (int q = 0; q < 3; q++) lpx[off3(q)] = fx64(LP[q] * rTT, P.fx_mul, bad);
                }
                // Only off-diagonal entries of the matrix are accumulated: every kept row of the
                // assembled operator sums to zero (for kernels of |x - y| each pair's blocks do, the
                // basis functions summing to one), so k_sym_add sets each diagonal entry to minus
                // its row's off-diagonal sum. The integers are those a per-pair balance of the
                // block diagonals would give, so the matrix is the same bit for bit.
#pragma unroll
                for (int i = 0; i < 6; i++) D[i] += lx[i];
                // termLocalPrime (off-diagonal part) into the partner's block accumulator
                red_add(ma.elp, (long long)part * 6 + 1, lpx[1]);
                red_add(ma.elp, (long long)part * 6 + 2, lpx[2]);
                red_add(ma.elp, (long long)part * 6 + 4, lpx[4]);
            }
            // termNonloc into A[T, b] (minus sign): lanes sharing a partner vertex add their
            // integers, the first of them lists the sums (over the item results, read by now); then
            // all lanes share the (vertex, row) lookups. The mirror A[b, T] -= N^T comes from the
            // symmetric completion (k_sym_add), except where T's vertex has no row (written here
            // into the partner vertex's row) and for close pairs, whose termNonlocPrime block is
            // its own FP64 result (the difference to N^T is added here).
            __syncwarp();
            const bool anyclose = KIND == MIX_SINGULAR && __any_sync(FULL, close);
            int nent = 0;
#pragma unroll 1
            for (int c = 0; c < 3; c++) {
                const int col = act ? sel3(pv, c) : -1;
                const unsigned grp = __match_any_sync(FULL, col);
                const bool leader = (__ffs(grp) - 1) == lane;
                const int maxn = __reduce_max_sync(FULL, (unsigned)__popc(grp));
                const long long o0 = sel3(&nx[0], c), o1 = sel3(&nx[3], c), o2 = sel3(&nx[6], c);
                const long long p0v = sel3(&mx[0], c), p1v = sel3(&mx[3], c), p2v = sel3(&mx[6], c);
                long long sn0 = o0, sn1 = o1, sn2 = o2, sq0 = p0v, sq1 = p1v, sq2 = p2v;
                unsigned rest = grp & ~(1u << lane);
                for (int it = 1; it < maxn; it++) {
                    const int src = rest ? __ffs(rest) - 1 : lane;
                    const bool use = rest != 0;
                    if (rest) rest &= rest - 1;
                    const long long t0 = shfl64(o0, src), t1 = shfl64(o1, src), t2 = shfl64(o2, src);
                    if (use) { sn0 += t0; sn1 += t1; sn2 += t2; }
                    if (anyclose) {
                        const long long u0 = shfl64(p0v, src), u1 = shfl64(p1v, src), u2 = shfl64(p2v, src);
                        if (use) { sq0 += u0; sq1 += u1; sq2 += u2; }
                    }
                }
                if (!anyclose) { sq0 = sn0; sq1 = sn1; sq2 = sn2; }
                const bool put = leader && col >= 0;
                const unsigned m = __ballot_sync(FULL, put);
                if (put) {
                    ScatEntry &e = slist[nent + __popc(m & lanemask_lt())];
                    e.col = col;
                    e.v[0] = sn0; e.v[1] = sn1; e.v[2] = sn2;
                    e.v[3] = sq0; e.v[4] = sq1; e.v[5] = sq2;
                }
                nent += __popc(m);
            }
            __syncwarp();
            // (row, column) lookups, SCAT_U per lane at a time: the first memory access of each is
            // issued before any is examined, so their latencies overlap
            const int nit = 3 * nent;
            for (int w0 = 0; w0 < nit; w0 += 32 * SCAT_U) {
                SlotProbe pb[SCAT_U];
#pragma unroll
                for (int u = 0; u < SCAT_U; u++) {
                    const int w = w0 + lane + 32 * u;
                    pb[u].e = HEMPTY;
                    pb[u].i = 0;
                    if (w < nit) {
                        const int e = w / 3, r = w - 3 * e;
                        RowHash h;
                        h.hb = W.rhb[r]; h.rb = W.rrb[r]; h.mask = W.rmask[r]; h.lo = W.rlo[r];
                        pb[u] = slot_probe_begin(sm, h, slist[e].col);
                    }
                }
#pragma unroll
                for (int u = 0; u < SCAT_U; u++) {
                    const int w = w0 + lane + 32 * u;
                    if (w >= nit) continue;
                    const int e = w / 3, r = w - 3 * e;
                    const int col = slist[e].col;
                    if (col == W.tvs[r]) continue;   // the matrix diagonal: from the row sum
                    const long long sn = slist[e].v[r], sq = slist[e].v[3 + r];
                    RowHash h;
                    h.hb = W.rhb[r]; h.rb = W.rrb[r]; h.mask = W.rmask[r]; h.lo = W.rlo[r];
                    if (h.mask != 0xffffffffu) {
                        const long long s = slot_probe_end(sm, h, col, pb[u]);
                        if (s < 0) { miss = true; continue; }
                        red_add(ma.valsN, s, -sn);
                        if (anyclose && sq != sn && a.labV[col] > 0) {
                            const int tp = sm.tpos[s];
                            if (tp < 0) miss = true;
                            else red_add(vals, sm.rowptr[col] + tp, sn - sq);
                        }
                    } else if (a.labV[col] > 0) {
                        const long long q = slot_find(sm, col, W.tvs[r]);
                        if (q < 0) miss = true;
                        else red_add(vals, q, -sq);
                    }
                }
            }
            __syncwarp();
        }
        // termLocal of all of T's pairs into T's diagonal block
#pragma unroll
        for (int i = 0; i < 6; i++)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) D[i] += (long long)__shfl_xor_sync(FULL, (unsigned long long)D[i], o);
        if (lane < 9 && lane / 3 != lane % 3) {   // off-diagonal entries (the diagonal: k_sym_add)
            const int r = lane / 3, c = lane % 3;
            const int s = sm.dslot[(long long)T * 9 + lane];
            const int si = r <= c ? sym_idx<3>(r, c) : sym_idx<3>(c, r);
            long long d = 0;
#pragma unroll
            for (int i = 0; i < 6; i++)
                if (i == si) d = D[i];
            if (s >= 0) red_add(vals, s, d);
            else if (keepmask & (1u << r)) miss = true;
        }
        __syncwarp();
    }
    if (__any_sync(FULL, bad) && lane == 0) atomicOr(ovf, 1);
    if (__any_sync(FULL, miss) && lane == 0) atomicOr(&a.err[3], 1);
    nsub = warp_sum(nsub);
    namb = warp_sum(namb);
    nclose = warp_sum(nclose);
    nitin = warp_sum(nitin);
    nitcut = warp_sum(nitcut);
    if (lane == 0) {
        if (nsub && a.n_subtri) atomicAdd(a.n_subtri, (unsigned long long)nsub);
        if (namb && a.n_amb) atomicAdd(a.n_amb, (unsigned long long)namb);
        if (nclose && a.n_close) atomicAdd(a.n_close, (unsigned long long)nclose);
        if (nitin && a.n_in) atomicAdd(a.n_in, (unsigned long long)nitin);
        if (nitcut && a.n_cut) atomicAdd(a.n_cut, (unsigned long long)nitcut);
    }
}

// Near pairs of constant kernels (the first near_cnt[T] of every element's list: all of the partner is in
// every outer point's ball), 80% and more of the pairs where the horizon is many elements wide. Their
// blocks need the two elements' measures only, so this kernel has no geometry, no classes and no items;
// it forms the same FP32 values in the same order as k_pass_mix2d does for a pair with every point
// inside. Bound by instruction issue and the latency of its lookups, so it stands apart from the general
// kernel: 64 registers instead of 128, 32 warps per SM instead of 16. Per pair nine integers go to
// shared memory; the lanes then share the batch's vertices (VertexGroups), each lane summing one
// vertex's integers for T's three rows. n = 256, delta = 0.1 (3.8e8 pairs, 3.1e8 of them near), the
// whole pass: 54.1 ms with the near pairs in k_pass_mix2d, 47.2 with this kernel, 37.1 when the lists
// came in element order (k_bfs).
struct NearWarp {
    long long val[32 * 9];      // termNonloc [row r][vertex c] of each lane's pair
    VertexGroups<3> g;
    long long rhb[3], rrb[3];   // T's rows (see MixWarp)
    unsigned rmask[3];
    int rlo[3], tvs[3];
};
constexpr int NEAR_BLOCKS = 8;
__global__ void __launch_bounds__(MIX_THREADS, NEAR_BLOCKS) k_pass_near2d(MixArgs ma, PassRule pr, int nPx) {
    __shared__ NearWarp s_w[MIX_WARPS];
    const PassArgs &a = ma.p;
    const SlotMap &sm = ma.m;
    const int lane = threadIdx.x & 31;
    NearWarp &W = s_w[threadIdx.x >> 5];
    long long *vals = reinterpret_cast<long long *>(a.vals);
    bool miss = false;   // as in k_pass_mix2d
    float most = 0.f;                 // largest magnitude of a contribution in units
    unsigned long long npair = 0;
    for (;;) {
        int idx = 0;
        if (lane == 0) idx = atomicAdd(ma.work, 1);
        idx = __shfl_sync(FULL, idx, 0);
        if (idx >= a.count) break;
        const int T = a.list ? a.list[idx] : idx;
        const int nn = a.near_cnt[T];
        if (nn == 0 || a.labT[T] == 0) continue;
        const long long lb = a.out_ptr[T], le = lb + nn;
        npair += nn;
        if (lane < 3) {
            const int u = a.T32[(long long)T * 3 + lane];
            RowHash h;
            h.hb = h.rb = 0;
            h.mask = 0xffffffffu;
            h.lo = 0;
            if (a.labV[u] > 0) h = row_hash(sm, u);
            W.rhb[lane] = h.hb;
            W.rrb[lane] = h.rb;
            W.rmask[lane] = h.mask;
            W.rlo[lane] = h.lo;
            W.tvs[lane] = u;
        }
        const ProbParams &P = a.probs[a.eprob[T]];
        const float kc = P.kc_f, mul = P.fx_mul, rTT = a.adetf[T];
        long long D[3] = {0, 0, 0};   // termLocal of T's pairs, off-diagonal
        int part_next = lb + lane < le ? a.pB[lb + lane] : T;   // partners one batch ahead
        for (long long p0 = lb; p0 < le; p0 += 32) {
            const long long p = p0 + lane;
            const bool act = p < le;
            const int part = part_next;
            part_next = p + 32 < le ? a.pB[p + 32] : T;
            int pv[3];
#pragma unroll
            for (int c = 0; c < 3; c++) pv[c] = act ? a.T32[(long long)part * 3 + c] : -1;
            if (act) {
                const float kr = kc * a.adetf[part];
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    D[q] += fx64(pr.xsum[off3(q)] * (kr * pr.insum[0]) * rTT, mul, most);
                    // termLocalPrime (off-diagonal part) into the partner's block accumulator
                    red_add(ma.elp, (long long)part * 6 + off3(q), fx64(pr.xsum[9] * (kr * pr.insum[4 + off3(q)]) * rTT, mul, most));
#pragma unroll
                    for (int c = 0; c < 3; c++)
                        W.val[lane * 9 + 3 * q + c] = fx64(pr.xsum[6 + q] * (kr * pr.insum[1 + c]) * rTT, mul, most);
                }
            }
            const int nent = group_vertices<3>(W.g, pv, act);
            for (int e = lane; e < nent; e += 32) {
                const int col = W.g.vert[e];
                SlotProbe pb[3];
                RowHash h[3];
#pragma unroll
                for (int r = 0; r < 3; r++) {   // in flight while the members are summed
                    h[r].hb = W.rhb[r]; h[r].rb = W.rrb[r]; h[r].mask = W.rmask[r]; h[r].lo = W.rlo[r];
                    pb[r] = slot_probe_begin(sm, h[r], col);
                }
                long long sn[3] = {0, 0, 0};
#pragma unroll
                for (int c = 0; c < 3; c++)
                    for (unsigned mm = W.g.lanes[e][c]; mm; mm &= mm - 1) {
                        const long long *v = &W.val[(__ffs(mm) - 1) * 9 + c];
#pragma unroll
                        for (int r = 0; r < 3; r++) sn[r] += v[3 * r];
                    }
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    if (col == W.tvs[r]) continue;   // the matrix diagonal: from the row sum
                    if (h[r].mask != 0xffffffffu) {
                        const long long s = slot_probe_end(sm, h[r], col, pb[r]);
                        if (s < 0) miss = true;
                        else red_add(ma.valsN, s, -sn[r]);
                    } else if (a.labV[col] > 0) {   // T's vertex has no row: into the partner vertex's row
                        const long long q = slot_find(sm, col, W.tvs[r]);
                        if (q < 0) miss = true;
                        else red_add(vals, q, -sn[r]);
                    }
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int q = 0; q < 3; q++) D[q] = (long long)warp_sum((unsigned long long)D[q]);
        if (lane < 9 && lane / 3 != lane % 3) {   // termLocal into T's diagonal block, off-diagonal entries
            const int r = lane / 3, c = lane % 3, q = r + c - 1;   // (0, 1), (0, 2), (1, 2)
            const int s = sm.dslot[(long long)T * 9 + lane];
            if (s >= 0) red_add(vals, s, sel3(D, q));
            else if (W.rmask[r] != 0xffffffffu) miss = true;
        }
        __syncwarp();
    }
    const bool bad = !(most < 4.0e18f);
    if (__any_sync(FULL, bad) && lane == 0) atomicOr(&a.err[5], 1);
    if (__any_sync(FULL, miss) && lane == 0) atomicOr(&a.err[3], 1);
    if (lane == 0 && npair) {
        if (a.n_subtri) atomicAdd(a.n_subtri, npair * nPx);
        if (a.n_in) atomicAdd(a.n_in, npair * nPx);
    }
}

// Symmetric completion of the one-sided retriangulate pass: every slot (t, v) adds the
// termNonloc sums of the transposed slot (v, t) when v has a row. Integer sums, so the completed
// matrix is exactly symmetric in these contributions, as the reference's A[b, T] -= termNonlocPrime
// = termNonloc^T (kernels of |x - y|) makes it. Then the row's diagonal entry is set to minus the
// sum of its other entries, which the pass left out (every kept row sums to zero). One warp per row.
__global__ void k_sym_add(const long long *__restrict__ rowptr, const int *__restrict__ cols,
                          const int *__restrict__ tpos, const long long *__restrict__ valsN, long long nrows,
                          long long *__restrict__ vals) {
    const int lane = threadIdx.x & 31;
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long t = gw; t < nrows; t += nw) {
        const long long b = rowptr[t], e = rowptr[t + 1];
        long long off = 0, dslot = -1;
        for (long long s = b + lane; s < e; s += 32) {
            if (cols[s] == (int)t) { dslot = s; continue; }
            long long v = valsN[s];
            const int tp = tpos[s];
            if (tp >= 0) v += valsN[rowptr[cols[s]] + tp];
            v += vals[s];
            vals[s] = v;
            off += v;
        }
        off = (long long)warp_sum((unsigned long long)off);
        if (dslot >= 0) vals[dslot] = -off;   // the row sums to zero
    }
}

// termLocalPrime blocks accumulated per partner element into its diagonal-block slots.
__global__ void k_elem_blocks(const long long *__restrict__ elp, const int *__restrict__ dslot,
                              const int *__restrict__ T32, const int *__restrict__ labV, long long nE,
                              long long *__restrict__ vals, int *__restrict__ err) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nE) return;
    long long b[6];
    bool any = false;
#pragma unroll
    for (int q = 0; q < 6; q++) {
        b[q] = elp[e * 6 + q];
        any |= b[q] != 0;
    }
    if (!any) return;
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) {
            if (r == c) continue;   // the diagonal comes from the row sum (k_sym_add)
            const int s = dslot[e * 9 + 3 * r + c];
            if (s >= 0) red_add(vals, s, b[r <= c ? sym_idx<3>(r, c) : sym_idx<3>(c, r)]);
            else if (labV[T32[e * 3 + r]] > 0) atomicOr(&err[3], 1);
        }
}

}  // namespace nlg
