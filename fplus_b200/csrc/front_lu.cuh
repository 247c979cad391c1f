// front_lu.cuh -- the pivot-block LU of a front that one CTA's shared memory holds, in 8-column panels.
#pragma once
#include "kernels.cuh"

namespace fpl {

// Partial-pivot LU of a front's pivot block (nrows x npiv) in shared memory, one CTA.  The panel group (one thread per row,
// ceil(nrows / 32) warps) pivots panel p, columns [c0, c0 + 8), with its rows' panel entries in registers, while the update
// group (the other warps) applies panel p - 1 to the columns from c0 + 8 on.
//   a pivot step: every warp posts its best candidate (the largest pivot key, ties to the smaller row of B) with the
//     candidate row's panel entries and reciprocal; one barrier of the panel group; every thread takes the same winner and
//     eliminates.  The elimination carries the row operations along (Gauss-Jordan on the panel's identity): entry k of a
//     row ends as the coefficient E[row, k] of the panel's k-th pivot row in that row, so that every later column c takes
//     A[row, c] += sum_k E[row, k] A_old[pivot row k, c], for the rows below the pivots (E = -L21 L11^-1) and the pivot rows
//     themselves (E = L11^-1 - I) alike: no triangular solve stands between a panel and the columns after it.
//   the next panel's columns: each panel-group thread applies the panel to its own row (E in its registers), no wait for
//     the update group.
//   the columns after those: the update group copies the pivot rows' old values, then takes 8 x 8 tiles as FP64 mma
//     products of depth 8 (complex: four real ones).
// One CTA-wide barrier per panel.  Rows never move: a row pivoted at step j is tagged j, and the block goes out in the
// final order at the end.
//
// What bounds it (B200): the npiv dependent pivot steps, about 700 cycles each (complex) or 650 (real): the key, one 32-bit
// warp reduction and a ballot, the post, the barrier, the choice among the warps' words, the winner's loads, the update of
// the next column.  Only the leading 30 bits of a pivot key are compared on that path; equal leading bits, border rows and
// values at the edge of the range take the whole keys (a uniform branch that is rarely taken: with the full tie and threshold
// tests on the path a complex step took 1,090 cycles).  The update's multiply-adds (0.8 M for 120 x 64 complex, 7 us at 64 a
// cycle) run beside the steps.  Measured against the one-barrier-per-step form k_front_lu2, one launch: 120 x 64 complex
// 43 against 84 us, 80 x 64 complex 39 / 70, 120 x 64 real 35 / 60, 128 x 128 real 63 / 152, 213 x 64 real 45 / 115, 25 x 24
// real 14.7 / 20.9, 3 x 2 real 4.6 / 6.4.
constexpr int LU6_PB = 8, LU6_UPD = 256;

__host__ __device__ constexpr int lu6_ld(int nrows, bool cplx) { return cplx ? (nrows | 3) + 2 : ((nrows + 7) & ~7) + 2; }   // 1 mod 4; 2 mod 8
__host__ __device__ constexpr int lu6_eld(int nrows) { return ((nrows + 15) & ~15) + 4; }                                    // 4 mod 16
// dynamic shared memory: the block, the coefficients (two buffers; two planes for complex), the pivot rows' old values,
// row ids, thresholds and their keys, tags, final order
static inline size_t front_lu6_smem(int64_t nrows, int64_t npiv, int64_t vs)
{
    const bool cp = vs == 16;
    return (size_t)(lu6_ld((int)nrows, cp) * npiv * vs + 2 * LU6_PB * lu6_eld((int)nrows) * vs + LU6_PB * lu6_eld((int)npiv) * vs +
                    nrows * 8 + npiv * 16 + nrows * 8);
}
// the warps of the panel group in the two forms of the kernel: up to 128 rows, and up to what shared memory holds of at
// least nine columns
__host__ __device__ constexpr int lu6_tallw(bool cplx) { return cplx ? 7 : 16; }
// panel-group warps for the rows, and the update group (none needed for at most two panels)
static inline int front_lu6_threads(int64_t nrows, int64_t npiv)
{
    return (int)(((nrows + 31) & ~(int64_t)31) + (npiv > 2 * LU6_PB ? LU6_UPD : 32));
}

// the panel group's posts of a step (two, used in turn), a slot per warp (MW): the candidate's word (lu6_word), row,
// reciprocal and panel entries, and the whole key and row of B where those decide; u holds the posts of a panel's steps
// (two panels), from which the update group takes the pivot rows' U entries of the panel's own columns
template <typename T, int MW> struct __align__(16) Lu6Post {
    unsigned word[2][MW];
    int row[2][MW];
    unsigned long long key[MW];
    long long rid[MW];
    T inv[2][MW];
    T u[2][LU6_PB][MW][LU6_PB];
    int prow[2][LU6_PB], win[2][LU6_PB];
    int cnt[MW];
    int stop;
};

// the most dynamic shared memory of a launch (227 KB a block, less the posts)
template <typename T, int MW> constexpr int lu6_smem_max() { return 227 * 1024 - (int)sizeof(Lu6Post<T, MW>); }
template <typename T> static inline bool front_lu6_fits(int64_t nrows, int64_t npiv)
{
    constexpr int TW = lu6_tallw(VT<T>::cplx_);
    if (npiv < 1 || npiv > nrows || nrows > 32 * TW) return false;
    const int64_t sm = (int64_t)front_lu6_smem(nrows, npiv, sizeof(T));
    return sm <= (nrows <= 128 ? lu6_smem_max<T, 4>() : lu6_smem_max<T, TW>());
}

// The top 30 bits of a value's pivot key (0 for a row that is not live; LU6_ODD for a value whose key or reciprocal needs the
// scaled arithmetic: at the edges of the range, infinities, NaN), and its reciprocal.  No branch.
constexpr unsigned LU6_ODD = 0x7fffffffu;
template <typename T> struct Key30;
template <> struct Key30<double> {
    unsigned key;
    bool in;
    __device__ __forceinline__ Key30(double v, bool live)
    {
        const unsigned h = (unsigned)__double2hiint(v) & 0x7fffffffu;
        in = h - 0x00200000u < 0x7fb00000u;                        // 2^-1021 <= |v| < 2^1022
        const unsigned k = in ? h >> 1 : (h | (unsigned)__double2loint(v)) == 0u ? 0u : LU6_ODD;
        key = live ? k : 0u;
    }
    __device__ __forceinline__ double inverse(double v) const { return __drcp_rn(in ? v : 1.0); }
};
template <> struct Key30<cplx> {
    unsigned key;
    bool in;
    double q;
    __device__ __forceinline__ Key30(cplx v, bool live)
    {
        q = __dadd_rn(__dmul_rn(v.x, v.x), __dmul_rn(v.y, v.y));
        const unsigned h = (unsigned)__double2hiint(q);
        in = h - 0x01b00000u < 0x7c900000u;                        // 2^-996 <= |v|^2 < 2^997
        const bool zero = ((__double2hiint(v.x) | __double2hiint(v.y)) & 0x7fffffff) == 0 && (__double2loint(v.x) | __double2loint(v.y)) == 0;
        const unsigned k = in ? (h >> 3) + (unsigned)(PIVKEY_OFF << 17) : zero ? 0u : LU6_ODD;
        key = live ? k : 0u;
    }
    __device__ __forceinline__ cplx inverse(cplx v) const
    {
        const double d = __drcp_rn(in ? q : 1.0);
        return cplx{v.x * d, -v.y * d};
    }
};

template <typename T, int MW>
__device__ __forceinline__ void front_lu6_body(const T *__restrict__ W, int64_t ld, int nrows, int npiv, int nri,
                                               int64_t fcol, const double *__restrict__ colmax, double pivot_rel,
                                               int64_t *__restrict__ rowid, T *__restrict__ Lout, int *__restrict__ perm,
                                               int64_t *__restrict__ p_lu, DevStatus *st, int64_t front, const PivotAsm &pa)
{
    constexpr bool CP = VT<T>::cplx_;
    constexpr int PB = LU6_PB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ Lu6Post<T, MW> P;
    const int lda = lu6_ld(nrows, CP), eld = lu6_eld(nrows), bld = lu6_eld(npiv);
    T *A = reinterpret_cast<T *>(smem_raw);                        // column-major: A[c * lda + i]
    double *E = reinterpret_cast<double *>(A + (size_t)npiv * lda);                    // buffer b, plane z, coefficient k, row i:
    const int ebuf = (CP ? 2 : 1) * PB * eld;                                          //   E[b * ebuf + (z * PB + k) * eld + i]
    double *Bp = E + 2 * ebuf;                                                         // plane z, pivot k, column c: (z * PB + k) * bld + c
    int64_t *rid = reinterpret_cast<int64_t *>(Bp + (CP ? 2 : 1) * PB * bld);
    double *thr = reinterpret_cast<double *>(rid + nrows);
    unsigned long long *thk = reinterpret_cast<unsigned long long *>(thr + npiv);
    int *tag = reinterpret_cast<int *>(thk + npiv);
    int *sperm = tag + nrows;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
    const int pgw = (nrows + 31) >> 5, npg = pgw * 32, nug = nt - npg;
    if (tid == 0) P.stop = st->code != 0;
    for (int c = tid; c < npiv; c += nt) { thr[c] = pivot_rel * colmax[fcol + c]; thk[c] = pivkey_of_modulus<T>(2.0 * thr[c]); }
    for (int i = tid; i < nrows; i += nt) tag[i] = INT_MAX;
    if (tid < 2 * MW) { P.word[tid / MW][tid % MW] = 0u; P.row[tid / MW][tid % MW] = 0; }
    // the block: from the working block, or assembled here (the sources of PivotAsm); a warp per column
    if (!pa.on) {
        pdl_wait();
        for (int i = tid; i < nrows; i += nt) rid[i] = rowid[i];
        for (int c = warp; c < npiv; c += nw) {
            const T *w = W + (int64_t)c * ld;
            for (int i0 = lane; i0 < nrows; i0 += 128) {
                T v[4];
#pragma unroll
                for (int q = 0; q < 4; q++) v[q] = i0 + 32 * q < nrows ? w[i0 + 32 * q] : VT<T>::zero();
#pragma unroll
                for (int q = 0; q < 4; q++) if (i0 + 32 * q < nrows) A[c * lda + i0 + 32 * q] = v[q];
            }
        }
    } else {
        for (int e = tid; e < npiv * lda; e += nt) A[e] = VT<T>::zero();
        for (int i = tid; i < nrows; i += nt) rid[i] = pa.rowinit[i];
        __syncthreads();
        const T *Bx = reinterpret_cast<const T *>(pa.Bx);
        for (int e = tid; e < (int)pa.acnt; e += nt) {
            const int d = (int)pa.adst[e];
            A[(d / nrows) * lda + d % nrows] = Bx[pa.asrc[e]];
        }
        pdl_wait();                                   // the child's CB columns (the launch before) are written
        for (int t = tid; t < (int)pa.nslot; t += nt) rid[pa.slot + t] = pa.child_rowid[t];
        __syncthreads();
        const T *cb = reinterpret_cast<const T *>(pa.cb);
        const int cbr = (int)pa.cbr, nsl = (int)pa.nslot, sl = (int)pa.slot, tb = (int)pa.tau_base;
        for (int c0 = warp; c0 < (int)pa.h; c0 += 4 * nw)     // a warp per column, four columns' loads in flight
            for (int t = lane; t < cbr; t += 32) {
                const int pr = t < nsl ? sl + t : tb + (t - nsl);
                T v[4];
#pragma unroll
                for (int q = 0; q < 4; q++) v[q] = c0 + q * nw < (int)pa.h ? cb[t + (int64_t)(c0 + q * nw) * cbr] : VT<T>::zero();
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (c0 + q * nw < (int)pa.h) {
                        T *a = A + (int)pa.relcol[c0 + q * nw] * lda + pr;
                        *a = add(*a, v[q]);
                    }
            }
    }
    __syncthreads();
    if (P.stop) return;
    const bool pg = warp < pgw;
    const int i = tid;
    const bool inrow = pg && i < nrows;
    const long long myrid = inrow ? (long long)rid[i] : LLONG_MAX;
    bool live = inrow;
    int mytag = INT_MAX;
    T pv[PB];                                          // panel group: the row's panel entries, rotated: pv[0] is the step's column
#pragma unroll
    for (int q = 0; q < PB; q++) pv[q] = inrow && q < npiv ? A[q * lda + i] : VT<T>::zero();
    bool fresh = false;                                // pivoted in the panel before: pv holds its U entries of this panel
    int buf = 0;
    for (int c0 = 0; c0 < npiv; c0 += PB, buf ^= 1) {
        const int w = npiv - c0 < PB ? npiv - c0 : PB;
        if (pg) {
            T *lcol = A + c0 * lda + i;                // where this row's multiplier of the step goes
            if (c0 > 0) {
                named_bar(1, npg);                     // everyone has read the pivot rows' old values
                if (fresh)
#pragma unroll
                    for (int q = 0; q < PB; q++) if (q < w) lcol[q * lda] = pv[q];
            }
            for (int s = 0; s < w; s++, lcol += lda) {
                const int par = s & 1, j = c0 + s;
                const unsigned tk = (unsigned)(thk[j] >> 33);
                const Key30<T> kv(pv[0], live);
                const unsigned k30 = kv.key, m30 = __reduce_max_sync(0xffffffffu, k30);
                const T xinv = kv.inverse(pv[0]);      // (in the shadow of the reduction)
                const unsigned cnd = __ballot_sync(0xffffffffu, k30 == m30);
                if (lane == __ffs(cnd) - 1) {
                    // (the word's low bit: the candidate needs the careful choice below, should it win)
                    P.word[par][warp] = (m30 << 1) | (unsigned)((cnd & (cnd - 1u)) != 0u || m30 == LU6_ODD || i >= nri);
                    P.row[par][warp] = i;
                    T *uo = P.u[buf][s][warp];
#pragma unroll
                    for (int q = 0; q < PB; q++) uo[q] = pv[q];
                    P.inv[par][warp] = xinv;
                }
                named_bar(1, npg);
                // the winner, the same for every thread of the group
                int bs, ties;
                unsigned bw;
                if constexpr (MW == 4) {               // (the slots past the last warp stay empty)
                    const uint4 k = *reinterpret_cast<const uint4 *>(P.word[par]);
                    bw = max(max(k.x, k.y), max(k.z, k.w));
                    const unsigned b1 = bw >> 1;
                    const bool e0 = k.x >> 1 == b1, e1 = k.y >> 1 == b1, e2 = k.z >> 1 == b1, e3 = k.w >> 1 == b1;
                    bs = e0 ? 0 : e1 ? 1 : e2 ? 2 : 3;
                    ties = e0 + e1 + e2 + e3;
                } else {
                    const unsigned k = lane < pgw ? P.word[par][lane] : 0u;
                    bw = __reduce_max_sync(0xffffffffu, k);
                    const unsigned c2 = __ballot_sync(0xffffffffu, k >> 1 == bw >> 1 && lane < pgw);
                    bs = __ffs(c2) - 1;
                    ties = __popc(c2);
                }
                int bi = P.row[par][bs];
                T inv = P.inv[par][bs];
                T u[PB];
#pragma unroll
                for (int q = 0; q < PB; q++) u[q] = P.u[buf][s][bs][q];
                if ((bw & 1u) || ties > 1 || bw >> 1 <= tk) {
                    // The careful choice, the same for every thread of the group: equal leading bits, a border row, a
                    // value at the edge of the range or near the singular threshold.  The whole keys, ties to the smaller
                    // row of B, the singular test of the reference (FPLUS src/factor_sn_panel.inc:232-233): no candidate,
                    // a zero modulus, or a modulus below thr (a key at or above that of 2 thr is clear of it).
                    const unsigned long long key = live ? pivkey(pv[0]) : 0ull;
                    const unsigned long long mk = warp_max_key(key);
                    const bool top = key != 0ull && key == mk;
                    const unsigned long long rm = warp_min_u64(top ? (unsigned long long)myrid : ~0ull);
                    named_bar(1, npg);                 // the posts of the quick choice have been read
                    if (mk == 0ull && lane == 0) { P.key[warp] = 0ull; P.rid[warp] = LLONG_MAX; }
                    if (top && (unsigned long long)myrid == rm) {
                        T *uo = P.u[buf][s][warp];
                        P.row[par][warp] = i;
#pragma unroll
                        for (int q = 0; q < PB; q++) uo[q] = pv[q];
                        P.inv[par][warp] = recip(pv[0]);
                        P.key[warp] = mk;
                        P.rid[warp] = myrid;
                    }
                    named_bar(1, npg);
                    bs = 0;
                    unsigned long long bk = P.key[0];
                    for (int q = 1; q < pgw; q++) {
                        const unsigned long long k = P.key[q];
                        if (k > bk || (k == bk && P.rid[q] < P.rid[bs])) { bk = k; bs = q; }
                    }
                    bi = P.row[par][bs];
                    inv = P.inv[par][bs];
#pragma unroll
                    for (int q = 0; q < PB; q++) u[q] = P.u[buf][s][bs][q];
                    int stop = 0;
                    if (bk == 0ull || (bk < thk[j] && vabs(u[0]) < thr[j])) stop = 1;
                    else if (bi >= nri) stop = 2;
                    if (stop) {
                        if (tid == 0) {
                            if (stop == 1) set_status(st, ST_SINGULAR, fcol + j, bk != 0ull ? vabs(u[0]) : 0.0, thr[j]);
                            else set_status(st, ST_BORDER, front, vabs(u[0]), thr[j]);
                            P.stop = 1;
                        }
                        break;
                    }
                }
                if (tid == 0) { P.prow[buf][s] = bi; P.win[buf][s] = bs; }
                if (i == bi) { mytag = j; live = false; }
                const T l = live ? mul(pv[0], inv) : VT<T>::zero();
#pragma unroll
                for (int q = 1; q < PB; q++) pv[q - 1] = msub(pv[q], l, u[q]);
                pv[PB - 1] = scal(l, -1.0);
                if (live) *lcol = l;
            }
            if (inrow) tag[i] = mytag;
            if (w == PB) {
                // the coefficients: a row pivoted at step s of this panel keeps those of the pivots before it; rows
                // pivoted before the panel have none
#pragma unroll
                for (int k = 0; k < PB; k++) {
                    if (!live && !(mytag >= c0 && k < mytag - c0)) pv[k] = VT<T>::zero();
                    double *e = E + buf * ebuf + k * eld + i;
                    if constexpr (CP) { if (i < eld) { e[0] = pv[k].x; e[PB * eld] = pv[k].y; } } else { if (i < eld) e[0] = pv[k]; }
                }
            }
        }
        __syncthreads();
        if (P.stop) return;
        // the pivot rows' U entries of the panel's own columns, from the posts
        const int c1 = c0 + PB;
        if (!pg || c1 >= npiv) {
            const int b0 = c1 >= npiv ? tid : tid - npg, bn = c1 >= npiv ? nt : nug;
            for (int e = b0; e < w * PB; e += bn) {
                const int s = e >> 3, q = e & (PB - 1);
                if (q < w - s) A[(c0 + s + q) * lda + P.prow[buf][s]] = P.u[buf][s][P.win[buf][s]][q];
            }
        }
        if (c1 >= npiv) break;
        if (pg) {
            // this row's entries of the next panel
            T nv[PB];
            int co[PB];
#pragma unroll
            for (int q = 0; q < PB; q++) {
                co[q] = (c1 + q < npiv ? c1 + q : npiv - 1) * lda;
                nv[q] = inrow ? A[co[q] + i] : VT<T>::zero();
            }
#pragma unroll
            for (int k = 0; k < PB; k++) {
                const T e = scal(pv[k], -1.0);
                const T *ap = A + P.prow[buf][k];
#pragma unroll
                for (int q = 0; q < PB; q++) nv[q] = msub(nv[q], e, ap[co[q]]);
            }
            fresh = mytag >= c0 && mytag < c1;
#pragma unroll
            for (int q = 0; q < PB; q++) pv[q] = c1 + q < npiv ? nv[q] : VT<T>::zero();
        } else if (c1 + PB < npiv) {
            const int ut = tid - npg, uw = warp - pgw, nuw = nug >> 5;
            const int t0 = c1 + PB;                    // the columns after the next panel
            for (int e = ut; e < PB * (npiv - t0); e += nug) {
                const int k = e & (PB - 1), c = t0 + (e >> 3);
                const T v = A[c * lda + P.prow[buf][k]];
                if constexpr (CP) { Bp[k * bld + c] = v.x; Bp[(PB + k) * bld + c] = v.y; } else Bp[k * bld + c] = v;
            }
            named_bar(2, nug);
            // items: an 8-column block by two 8-row blocks (neighbouring warps share the columns)
            const int rf = (nrows + 15) >> 4, cf = (npiv - t0 + PB - 1) >> 3;
            const int r = lane >> 2, kq = lane & 3;
            const double *Eb = E + buf * ebuf;
            for (int p = uw; p < rf * cf; p += nuw) {
                const int cb = t0 + PB * (p / rf), r0 = 16 * (p % rf);
                double cr[2][2], ci[2][2];
                bool ok[2][2];
                const int cc = cb + 2 * kq;
#pragma unroll
                for (int a = 0; a < 2; a++) {
                    const int row = r0 + 8 * a + r;
                    const bool rok = row < nrows && tag[row < nrows ? row : 0] >= c0;   // not a row pivoted before the panel
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        ok[a][h] = rok && cc + h < npiv;
                        const T v = ok[a][h] ? A[(cc + h) * lda + row] : VT<T>::zero();
                        if constexpr (CP) { cr[a][h] = v.x; ci[a][h] = v.y; } else cr[a][h] = v;
                    }
                }
#pragma unroll
                for (int ks = 0; ks < PB; ks += 4) {
                    const int k = ks + kq;
                    const bool bok = cb + r < npiv;
                    const double br = bok ? Bp[k * bld + cb + r] : 0.0;
                    const double bi_ = CP && bok ? Bp[(PB + k) * bld + cb + r] : 0.0;
#pragma unroll
                    for (int a = 0; a < 2; a++) {
                        const int row = r0 + 8 * a + r;
                        const double er = row < nrows ? Eb[k * eld + row] : 0.0;
                        dmma(cr[a][0], cr[a][1], er, br);
                        if constexpr (CP) {
                            const double ei = row < nrows ? Eb[(PB + k) * eld + row] : 0.0;
                            dmma(ci[a][0], ci[a][1], er, bi_);
                            dmma(cr[a][0], cr[a][1], -ei, bi_);
                            dmma(ci[a][0], ci[a][1], ei, br);
                        }
                    }
                }
#pragma unroll
                for (int a = 0; a < 2; a++)
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        if (ok[a][h]) {
                            T *x = A + (cc + h) * lda + r0 + 8 * a + r;
                            if constexpr (CP) *x = cplx{cr[a][h], ci[a][h]}; else *x = cr[a][h];
                        }
            }
        }
    }
    // the final order: pivot rows at their step, the others after them in block order
    if (pg) {
        const bool un = inrow && mytag == INT_MAX;
        const unsigned bal = __ballot_sync(0xffffffffu, un);
        if (lane == 0) P.cnt[warp] = __popc(bal);
        named_bar(1, npg);
        int k0 = npiv;
        for (int q = 0; q < warp; q++) k0 += P.cnt[q];
        if (inrow) {
            const int k = un ? k0 + __popc(bal & ((1u << lane) - 1u)) : mytag;
            sperm[k] = i;
            perm[k] = i;
            rowid[k] = myrid;
            if (k < npiv) p_lu[fcol + k] = myrid;
        }
    }
    __syncthreads();
    // a warp per column, four rows per lane (and two columns) in flight
    for (int k0 = lane; k0 < nrows; k0 += 128) {
        int sp[4];
#pragma unroll
        for (int q = 0; q < 4; q++) sp[q] = k0 + 32 * q < nrows ? sperm[k0 + 32 * q] : 0;
#pragma unroll 2
        for (int c = warp; c < npiv; c += nw) {
            T v[4];
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = A[c * lda + sp[q]];
#pragma unroll
            for (int q = 0; q < 4; q++) if (k0 + 32 * q < nrows) Lout[(int64_t)c * nrows + k0 + 32 * q] = v[q];
        }
    }
}

// MW: the most warps of the panel group (4: blocks of at most 128 rows, with more registers per thread)
template <typename T, int MW>
__global__ void __launch_bounds__(32 * MW + LU6_UPD, 1) k_front_lu6(const T *__restrict__ W, int64_t ld, int nrows, int npiv, int nri,
                                                    int64_t fcol, const double *__restrict__ colmax, double pivot_rel,
                                                    int64_t *__restrict__ rowid, T *__restrict__ Lout, int *__restrict__ perm,
                                                    int64_t *__restrict__ p_lu, DevStatus *st, int64_t front, PivotAsm pa)
{
    front_lu6_body<T, MW>(W, ld, nrows, npiv, nri, fcol, colmax, pivot_rel, rowid, Lout, perm, p_lu, st, front, pa);
}

// the pivot-block LU of a level's batched fronts, a CTA each
template <typename T>
__global__ void __launch_bounds__(128 + LU6_UPD, VT<T>::cplx_ ? 1 : 2) k_bat_lu6(const FcFront *__restrict__ fc, const int *__restrict__ list,
                                                 const T *__restrict__ Wbase, const double *__restrict__ colmax, double pivot_rel,
                                                 int64_t *__restrict__ rowid_all, T *__restrict__ La, int *__restrict__ permall,
                                                 int64_t *__restrict__ p_lu, DevStatus *st)
{
    const int fi = list[blockIdx.x];
    const FcFront F = fc[fi];
    PivotAsm pa;
    pa.on = 0;
    front_lu6_body<T, 4>(Wbase + F.wofs, F.nr, (int)F.nr, (int)F.np, (int)F.nri, F.f, colmax, pivot_rel, rowid_all + F.row_off,
                      La + F.L_off, permall + F.row_off, p_lu, st, fi, pa);
}

}  // namespace fpl
