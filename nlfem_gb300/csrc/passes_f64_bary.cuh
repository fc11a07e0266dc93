// FP64 barycenter pass for constant kernels (integrate_baryCenter, integration.cpp:910-1018), 2D and 3D.
//
// One-sided like the mixed barycenter pass (passes_bary.cuh): each element writes its own rows. A
// pair's items (outer points whose ball holds the partner's barycenter) all have the same inner
// sums, kc |b| times the rule's, so its blocks are those times the outer rule's sums over the inside
// mask, read from a table with one entry per mask byte. The mask comes from the certified FP32
// distance (the exact FP64 test inside its margin). That leaves about 45 FP64 instructions per 3D
// pair: products and conversions of its (dim + 1)^2 termNonloc entries. The general pass runs the
// outer x inner point loop (121 kernel values per pair with 11-point rules) on the FP64 pipe instead.
// Sums and their units are those of passes_f64.cuh (two integers per sum, third ones for what is far
// below the units); k_sym_add_f64 without transposed slots completes the rows.
#pragma once
#include "passes_f64.cuh"

namespace nlg {

template <int DIM>
struct F64BaryWarp {
    double x64[MAXQ * DIM];                 // outer points of T
    float xf[MAXQ * DIM];                   // relative to T's vertex 0
    long long rhb[DIM + 1], rrb[DIM + 1];   // T's rows (see MixWarp)
    unsigned rmask[DIM + 1];
    int rlo[DIM + 1], tvs[DIM + 1], te[DIM + 1];
    long long val[32 * bary_vals(DIM)];     // a batch's integers,
    long long low[32 * bary_vals(DIM)];     // their second integers, and the groups of its partner vertices
    VertexGroup list[32 * (DIM + 1)];         // (see k_pass_bary)
};
// outer sums per mask: psi_r, then psi_r psi_c off the diagonal; an odd stride keeps the banks apart
template <int DIM>
__host__ __device__ constexpr int f64_bary_tab() { return DIM == 2 ? 7 : 11; }
template <int DIM>
__host__ __device__ constexpr size_t f64_bary_smem(int nPx) {
    return ((size_t)f64_tab_entries(nPx) * f64_bary_tab<DIM>() * 8 + 15) / 16 * 16 + F64_WARPS * ((sizeof(F64BaryWarp<DIM>) + 15) / 16 * 16);
}

template <int DIM>
__global__ void __launch_bounds__(F64_THREADS, 3) k_pass_bary_f64(F64Args fa, Rule rule, PassRuleT<double> pr) {
    constexpr int dV = DIM + 1, NO = dV * (dV - 1) / 2, TS = f64_bary_tab<DIM>(), VS = bary_vals(DIM);
    extern __shared__ __align__(16) unsigned char s_raw[];
    const PassArgs &a = fa.m.p;
    const SlotMap &sm = fa.m.m;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int nPx = rule.nPx;
    double *tab = reinterpret_cast<double *>(s_raw);
    F64BaryWarp<DIM> &W = *reinterpret_cast<F64BaryWarp<DIM> *>(
        s_raw + ((size_t)f64_tab_entries(nPx) * TS * 8 + 15) / 16 * 16 + (size_t)wib * ((sizeof(F64BaryWarp<DIM>) + 15) / 16 * 16));
    for (int i = threadIdx.x; i < TS * f64_tab_entries(nPx); i += F64_THREADS) tab[i] = fa.mtab[i];
    __syncthreads();
    long long *vals = reinterpret_cast<long long *>(a.vals);
    bool bad = false, miss = false;
    unsigned namb = 0, nitin = 0;
    for (;;) {
        int idx = 0;
        if (lane == 0) idx = atomicAdd(fa.m.work, 1);
        idx = __shfl_sync(FULL, idx, 0);
        if (idx >= a.count) break;
        const int T = a.list ? a.list[idx] : idx;
        const long long lb = a.out_ptr[T], le = a.out_cnt ? lb + a.out_cnt[T] : a.out_ptr[T + 1];
        const long long ln = lb + (a.near_cnt ? a.near_cnt[T] : 0);   // near pairs come first
        if (lb == le || a.labT[T] == 0) continue;
        if (lane < dV) {
            const int u = a.T32[(long long)T * dV + lane];
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
            W.te[lane] = fa.vexp[u];
        }
        const ProbParams P = a.probs[a.eprob[T]];
        const double *ET64 = &a.EC[(long long)T * DIM * dV];
        float ohi[DIM], olo[DIM];
#pragma unroll
        for (int j = 0; j < DIM; j++) {
            ohi[j] = a.EChi[(long long)T * DIM * dV + j];
            olo[j] = a.EClo[(long long)T * DIM * dV + j];
        }
        for (int k = lane; k < nPx; k += 32) {
            xtoPhys<DIM>(ET64, &rule.Px[DIM * k], &W.x64[DIM * k]);
#pragma unroll
            for (int j = 0; j < DIM; j++) W.xf[DIM * k + j] = (float)(W.x64[DIM * k + j] - ET64[j]);
        }
        __syncwarp();
        int et[dV];
#pragma unroll
        for (int r = 0; r < dV; r++) et[r] = 8 * F64_BITS - P.xN - W.te[r];
        const double kT = 2.0 * P.kc * a.adet[T];   // weight 2 (integration.cpp:1001-1013)
        double D[NO];   // termLocal of T's pairs, off-diagonal
#pragma unroll
        for (int q = 0; q < NO; q++) D[q] = 0;
        const float sqlo = P.sqdelta_f * (1.f - MARG_D), sqhi = P.sqdelta_f * (1.f + MARG_D);
        int part_next = lb + lane < le ? a.pB[lb + lane] : T;   // partners one batch ahead
        for (long long p0 = lb; p0 < le; p0 += 32) {
            const long long p = p0 + lane;
            const bool act = p < le;
            const bool near = min(p0 + 32, le) <= ln;   // the whole batch: no classes to find
            const int part = part_next;
            part_next = p + 32 < le ? a.pB[p + 32] : T;
            int pv[dV];
#pragma unroll
            for (int c = 0; c < dV; c++) pv[c] = a.T32[(long long)part * dV + c];
            unsigned inm = 0;
            if (act && near) inm = nPx == 32 ? 0xffffffffu : (1u << nPx) - 1u;
            else if (act) {
                float bf[DIM];
                bary_offset<DIM>(a.BCf, part, ohi, olo, bf);
                unsigned und = 0;
                for (int k = 0; k < nPx; k++) {
                    float d2 = 0.f;
#pragma unroll
                    for (int j = 0; j < DIM; j++) {
                        const float d = W.xf[DIM * k + j] - bf[j];
                        d2 = fmaf(d, d, d2);
                    }
                    inm |= (unsigned)(d2 < sqlo) << k;
                    und |= (unsigned)(d2 >= sqlo && d2 <= sqhi) << k;
                }
                if (und) {   // inside the margin: the exact test decides
                    double b64[DIM];
                    xbary<DIM>(&a.EC[(long long)part * DIM * dV], b64);
                    namb += __popc(und);
                    for (; und; und &= und - 1) {
                        const int k = __ffs(und) - 1;
                        if (xbaryInside<DIM>(&W.x64[DIM * k], b64, P.sqdelta)) inm |= 1u << k;
                    }
                }
            }
            nitin += __popc(inm);
            double nx[dV * dV];
#pragma unroll
            for (int i = 0; i < dV * dV; i++) nx[i] = 0;
            if (inm) {
                double m[dV + NO];
#pragma unroll
                for (int q = 0; q < dV + NO; q++) m[q] = tab[TS * (inm & 255u) + q];
                for (int b = 1; 8 * b < nPx; b++)
#pragma unroll
                    for (int q = 0; q < dV + NO; q++) m[q] += tab[TS * (256 * b + ((inm >> (8 * b)) & 255u)) + q];
                const double kr = kT * a.adet[part];
#pragma unroll
                for (int c = 0; c < dV; c++) {
                    const int ve = fa.vexp[pv[c]];
                    const double iN = kr * pr.insum[1 + c];
#pragma unroll
                    for (int r = 0; r < dV; r++) nx[dV * r + c] = scale2(m[r] * iN, (et[r] - ve) >> 3);
                }
                const double kl = kr * pr.insum[0];
#pragma unroll
                for (int q = 0; q < NO; q++) D[q] += m[dV + q] * kl;
            }
            // termNonloc into T's rows: sums per partner vertex and lookups shared by the lanes
            bool rest = false, low = false;
#pragma unroll
            for (int i = 0; i < dV * dV; i++) {
                f64_split(nx[i], F64_BITS, bad, W.val[lane * VS + i], W.low[lane * VS + i], rest);
                low |= W.low[lane * VS + i] != 0;
            }
            low = __any_sync(FULL, low);
            if (__any_sync(FULL, rest)) {   // elements far smaller than their neighbours
                for (int i = 0; rest && i < dV * dV; i++) {
                    const int r = i / dV, c = i - dV * r, col = a.T32[(long long)part * dV + c];
                    double q = 0;
#pragma unroll
                    for (int j = 0; j < dV * dV; j++) q = j == i ? nx[j] : q;
                    long long hi, lo;
                    bool third = false, dummy = false;
                    f64_split(q, F64_BITS, dummy, hi, lo, third);
                    RowHash h;
                    h.hb = W.rhb[r]; h.rb = W.rrb[r]; h.mask = W.rmask[r]; h.lo = W.rlo[r];
                    if (!third || h.mask == 0xffffffffu || col == W.tvs[r]) continue;
                    const long long s = slot_find_row(sm, h, col);
                    if (s < 0) continue;   // the scatter below reports it
                    red_add(fa.valsNt, s, f64_third(q));
                    a.err[F64_ERR_THIRD] = 1;
                }
                __syncwarp();
            }
            int nent = 0;
#pragma unroll
            for (int c = 0; c < dV; c++) {
                const int col = act ? pv[c] : -1;
                const unsigned grp = __match_any_sync(FULL, col);
                const bool put = (__ffs(grp) - 1) == lane && col >= 0;
                const unsigned m = __ballot_sync(FULL, put);
                if (put) {
                    VertexGroup &e = W.list[nent + __popc(m & lanemask_lt())];
                    e.col = col;
                    e.c = c;
                    e.lanes = grp;
                }
                nent += __popc(m);
            }
            __syncwarp();
            for (int w = lane; w < dV * nent; w += 32) {
                const int e = w / dV, r = w - dV * e;
                RowHash h;
                h.hb = W.rhb[r]; h.rb = W.rrb[r]; h.mask = W.rmask[r]; h.lo = W.rlo[r];
                const int col = W.list[e].col;
                if (h.mask == 0xffffffffu || col == W.tvs[r]) continue;   // no row; the matrix diagonal: from the row sum
                const SlotProbe pb = slot_probe_begin(sm, h, col);
                const long long *v = &W.val[dV * r + W.list[e].c], *vl = &W.low[dV * r + W.list[e].c];
                long long sn = 0, sl = 0;
                for (unsigned mm = W.list[e].lanes; mm; mm &= mm - 1) sn += v[(__ffs(mm) - 1) * VS];
                if (low)
                    for (unsigned mm = W.list[e].lanes; mm; mm &= mm - 1) sl += vl[(__ffs(mm) - 1) * VS];
                const long long s = slot_probe_end(sm, h, col, pb);
                if (s < 0) {
                    miss = true;
                } else {
                    red_add(fa.m.valsN, 2 * s, sn);
                    if (sl) red_add(fa.m.valsN, 2 * s + 1, sl);
                }
            }
            __syncwarp();
        }
        // termLocal of all of T's pairs: off-diagonal entries of T's block
#pragma unroll
        for (int q = 0; q < NO; q++) D[q] = warp_sum(D[q]);
        if (lane < dV * dV && lane / dV != lane % dV) {
            const int r = lane / dV, c = lane % dV, lo = r < c ? r : c, up = r < c ? c : r;
            RowHash h;
            h.hb = W.rhb[r]; h.rb = W.rrb[r]; h.mask = W.rmask[r]; h.lo = W.rlo[r];
            if (h.mask != 0xffffffffu) {
                const int qi = sym_idx<dV>(lo, up) - lo - 1;   // off-diagonal entries in table order
                double d = 0;
#pragma unroll
                for (int q = 0; q < NO; q++)
                    if (q == qi) d = D[q];
                const long long s = slot_find_row(sm, h, W.tvs[c]);
                if (s < 0) {
                    miss = true;
                } else {
                    long long hi, lo;
                    f64_split2(scale2(d, F64_BITS - P.xD - ((W.te[r] + 7) >> 3)), F64_BITS, bad, hi, lo);
                    red_add(vals, s, hi);
                    red_add(fa.valslo, s, lo);
                }
            }
        }
        __syncwarp();
    }
    if (__any_sync(FULL, bad) && lane == 0) atomicOr(&a.err[5], 1);
    if (__any_sync(FULL, miss) && lane == 0) atomicOr(&a.err[3], 1);
    namb = warp_sum(namb);
    nitin = warp_sum(nitin);
    if (lane == 0) {
        if (nitin && a.n_subtri) atomicAdd(a.n_subtri, (unsigned long long)nitin);
        if (namb && a.n_amb) atomicAdd(a.n_amb, (unsigned long long)namb);
        if (nitin && a.n_in) atomicAdd(a.n_in, (unsigned long long)nitin);
    }
}

}  // namespace nlg
