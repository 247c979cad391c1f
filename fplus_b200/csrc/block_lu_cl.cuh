// block_lu_cl.cuh -- the pivot block of a tall front (too large for one CTA's shared memory) by one thread-block cluster.
#pragma once
#include <cstddef>
#include "kernels.cuh"
#include "front_lu.cuh"
#include "chain_solve.cuh"

namespace fpl {

// Partial-pivot LU of a front's pivot block (nrows x npiv) in one launch of one cluster of G CTAs (the interface and the
// outputs of k_block_lu_mc: rows never move, chosen[j] = the position of step j's pivot row, U12 beyond a row's own panel in
// Ub; k_mc_order and k_mc_lout follow).  CTA b owns the rows [b * per, b * per + per), a thread per row with its entries of
// the panel (32 columns; 16 complex) in registers and its multipliers in shared memory.  A pivot step:
//   1. every warp elects its best row by the leading 30 bits of the pivot key (one warp reduction, one ballot) and leaves
//      that row's panel entries, its reciprocal and position in shared memory; after a block barrier every warp takes the
//      CTA's best and stores its word and row into one or two CTAs of the cluster, by asynchronous stores that complete on
//      the receiver's barrier for the step (mbarrier, the expected bytes of all CTAs);
//   2. everyone waits for the step's posts;
//   3. every warp takes the same winner from the G words in its own shared memory, and every row its multiplier and update.
// The posts alternate by the step's parity: a CTA posts step j + 2 only after every CTA's post of step j + 1, which is sent
// after that CTA's reads of step j.
// Equal leading bits, border rows, values at the edge of the range or near the singular threshold go through whole keys and
// row ids with two more barriers, the same for all (rare).  After a panel every CTA forms U12 of the panel's pivot rows and
// applies the panel's update to its live rows as FP64 mma products.
//
// What bounds it (B200): the npiv dependent steps, and 2 npiv^2 nrows / G flops of trailing updates per CTA (a quarter of
// the time at 1,500 rows).  Cycles of a real step at 1,500 rows: 5,000 reading the winner's row from its CTA after a
// cluster barrier; 3,750 with the rows pushed before it (2,270 of them in the barrier's release); 2,990 with asynchronous
// stores; 2,240 with the panel in registers (in shared memory its updates were loads and stores that had to keep their
// order), 910 of them between the stores and their arrival.  1,500 x 256: 597 -> 445 us real against the form with the
// cluster barrier, 829 -> 835 us complex; 5,000 x 256 real: 783 -> 637 us.  A complex panel is 16 columns: 32 took 1,020 us
// (an update of every step covers the whole panel).  Trailing entries are loaded before the products that change them
// (912 -> 835 us complex).  U12 formed once by shares of the columns and read back from Ub, instead of by every CTA for
// itself: 452 us real, 865 complex.
constexpr int CL_MAXG = 16, CL_MAXW = 16, CL_SLOTS = CL_MAXG + CL_MAXW;
template <typename T> __host__ __device__ constexpr int cl_pw() { return VT<T>::cplx_ ? 16 : 32; }    // panel columns
template <typename T> __host__ __device__ constexpr int cl_cw() { return VT<T>::cplx_ ? 64 : 128; }
// leading dimensions of the panel (rows) and of a chunk of U12 (columns): the mma fragments of a half-warp hit all banks
template <typename T> __host__ __device__ constexpr int cl_ld(int m) { return VT<T>::cplx_ ? ((m + 7) & ~7) + 2 : ((m + 15) & ~15) + 4; }
template <typename T> struct __align__(16) ClPost {
    T v[cl_pw<T>()];           // the candidate row's panel values (the CTAs' posts: in column order, L11's before the step's column)
    T inv;                     // 1 / its value in the step's column
    long long rid;             // (the careful choice: its row of B, its whole key)
    unsigned long long key;
    int pos;                   // (at a multiple of eight bytes: one store takes pos and word)
    unsigned word;             // the key's leading bits, and a flag for the careful choice
    int pad[2];
};
// the address of a shared-memory object in CTA `rank` of the cluster, and an asynchronous store there that completes on a
// barrier of that CTA
__device__ __forceinline__ unsigned cl_map(const void *p, int rank)
{
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void st_async(unsigned dst, double v, unsigned bar)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];"
                 ::"r"(dst), "l"(__double_as_longlong(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async(unsigned dst, cplx v, unsigned bar) { st_async(dst, v.x, bar); st_async(dst + 8, v.y, bar); }
template <typename T> __host__ __device__ constexpr size_t cl_smem(int per)
{
    return (size_t)(cl_pw<T>() * (cl_ld<T>(per) + cl_pw<T>() + 1 + cl_ld<T>(cl_cw<T>()))) * sizeof(T) +
           (size_t)(2 * CL_SLOTS + 1) * sizeof(ClPost<T>) + (size_t)per * 8 + (size_t)2 * ((per + 15) & ~15) +
           cl_pw<T>() * sizeof(T);      // (a row's entries are read past the last post's end)
}

template <typename T>
__global__ void __launch_bounds__(VT<T>::cplx_ ? 256 : 512) k_block_lu_cl(T *W, int64_t ld, int nrows, int npiv, int nri, int per, int64_t fcol,
                                                     const double *__restrict__ colmax, double pivot_rel,
                                                     const int64_t *__restrict__ rowid, int64_t *__restrict__ chosen,
                                                     T *__restrict__ Ub, DevStatus *st, int64_t front)
{
    namespace cg = cooperative_groups;
    constexpr bool CP = VT<T>::cplx_;
    constexpr int CW = cl_cw<T>(), UL = cl_ld<T>(CW), CL_PW = cl_pw<T>(), CL_LB = CL_PW + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int sl = cl_ld<T>(per);
    T *S = reinterpret_cast<T *>(smem_raw);              // the panel's multipliers (a pivot row: its U entries too): S[c * sl + r]
    T *Lb = S + CL_PW * sl;                              // the panel's pivot rows: Lb[k * CL_LB + c] (L11 \ U11)
    T *Uc = Lb + CL_PW * CL_LB;                          // a chunk of U12: Uc[k * UL + c]
    ClPost<T> *post = reinterpret_cast<ClPost<T> *>(reinterpret_cast<unsigned char *>(S) +
        ((size_t)(CL_PW * sl + CL_PW * CL_LB + CL_PW * UL) * sizeof(T)));           // [parity][the CTAs', then the own warps']
    long long *rid_s = reinterpret_cast<long long *>(post + 2 * CL_SLOTS + 1);
    unsigned char *live = reinterpret_cast<unsigned char *>(rid_s + per), *was = live + ((per + 15) & ~15);     // (was: live at the panel's start)
    __shared__ int s_piv[CL_PW];
    __shared__ double s_thr[CL_PW];
    __shared__ unsigned s_tk[CL_PW];
    __shared__ int s_stop, s_late, s_far;                // (s_late, s_far: a wait of this CTA, of another one, ran out)
    __shared__ unsigned long long bars[2];               // the posts of the steps of each parity
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
    const int G = gridDim.x, b = blockIdx.x;
    const int r_lo = b * per, r_hi = r_lo + per < nrows ? r_lo + per : nrows, nmine = r_hi > r_lo ? r_hi - r_lo : 0;
    const int npr = npiv < nrows ? npiv : nrows;
    if (tid == 0) {
        s_stop = st->code != 0;
        s_late = s_far = 0;
        bar_init(bars, 1);
        bar_init(bars + 1, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int r = tid; r < per; r += nt) {
        live[r] = r < nmine;
        rid_s[r] = r < nmine ? rowid[r_lo + r] : LLONG_MAX;
    }
    // every CTA of the cluster starts from CTA 0's reading of the status word (the barrier counts must agree)
    cl.sync();
    if (tid == 0) s_stop = *cl.map_shared_rank(&s_stop, 0);
    __syncthreads();
    bool stopped = s_stop != 0;                          // the same in every thread (every decision below is)
    const int nwr = (nmine + 31) >> 5;                   // the warps with rows of their own
    for (int p0 = 0; p0 < npr && !stopped; p0 += CL_PW) {
        const int w = npr - p0 < CL_PW ? npr - p0 : CL_PW;
        if (tid < w) { const double t = pivot_rel * colmax[fcol + p0 + tid]; s_thr[tid] = t; s_tk[tid] = (unsigned)(pivkey_of_modulus<T>(2.0 * t) >> 33); }
        bool mine = tid < nmine && live[tid];
        T pv[CL_PW];                                     // this row's entries from the step's column on, pv[0] the step's
#pragma unroll
        for (int q = 0; q < CL_PW; q++) pv[q] = mine && q < w ? W[(r_lo + tid) + (int64_t)(p0 + q) * ld] : VT<T>::zero();
        if (tid < per) was[tid] = mine;
        __syncthreads();
        for (int kk = 0; kk < w; kk++) {
            const int j = p0 + kk, par = j & 1;
            const unsigned tk = s_tk[kk];
            if (tid == 0) bulk_expect(bars + par, (unsigned)G * (unsigned)((w + 1) * sizeof(T) + 8));
            // 1. the warp's candidate
            const Key30<T> kv(pv[0], mine);
            const unsigned m30 = __reduce_max_sync(0xffffffffu, kv.key);
            const T xinv = kv.inverse(pv[0]);
            const unsigned cnd = __ballot_sync(0xffffffffu, kv.key == m30);
            const int wl = __ffs(cnd) - 1, row = (warp << 5) + wl;       // (a warp without live rows posts an empty word)
            ClPost<T> *all = post + par * CL_SLOTS, *my = all + CL_MAXG + warp;
            if (lane == wl && warp < nwr) {
#pragma unroll
                for (int q = 0; q < CL_PW; q++) my->v[q] = pv[q];
                my->inv = xinv;
                my->pos = r_lo + row;
                const bool odd = (cnd & (cnd - 1u)) != 0u || m30 == LU6_ODD || r_lo + row >= nri;
                my->word = (m30 << 1) | (unsigned)(odd && m30 != 0u);
            }
            __syncthreads();
            if (*(volatile int *)&s_late) { stopped = true; break; }      // (a wait ran out: the same for the whole CTA)
            {
                // the CTA's best (the same for every warp), into the CTAs d = warp, warp + nw, ..
                const unsigned k = lane < nwr ? all[CL_MAXG + lane].word : 0u, mb = __reduce_max_sync(0xffffffffu, k);
                const unsigned c2 = __ballot_sync(0xffffffffu, k >> 1 == mb >> 1 && lane < nwr);
                const ClPost<T> *bst = all + CL_MAXG + (c2 ? __ffs(c2) - 1 : 0);
                const T vi = bst->inv;
                const int vp = mb != 0u ? bst->pos : r_lo;       // (no candidate: any row)
                // (lane: an entry from the step's column on, or one of the row's multipliers before it)
                const int rem = w - kk, col = lane < rem ? kk + lane : lane - rem;
                const T v = lane >= w ? VT<T>::zero() : lane < rem ? bst->v[lane] : S[col * sl + (vp - r_lo)];
                const unsigned word = mb | (unsigned)((c2 & (c2 - 1u)) != 0u && mb != 0u);
                for (int d = warp; d < G; d += nw) {
                    const unsigned bar = cl_map(bars + par, d), dst = cl_map(all + b, d);
                    if (lane < w) st_async(dst + (unsigned)(col * sizeof(T)), v, bar);
                    if (lane == 0) {
                        st_async(dst + (unsigned)offsetof(ClPost<T>, inv), vi, bar);
                        st_async(dst + (unsigned)offsetof(ClPost<T>, pos), __hiloint2double((int)word, vp), bar);     // (pos, then word)
                    }
                }
            }
            // 2. the posts
            const bool late = !bar_wait(bars + par, (unsigned)(j >> 1) & 1u);
            if (late) {                                  // (leaves at the next block barrier, with its CTA)
                set_status(st, ST_WAIT, front, 0.0, 0.0);
                s_late = 1;
                for (int d = 0; d < G; d++) *(volatile int *)cl.map_shared_rank(&s_far, d) = 1;
            }
            // 3. the winner, the same for every warp
            const unsigned kq = lane < G ? all[lane].word : 0u;
            const unsigned bw = __reduce_max_sync(0xffffffffu, kq);
            const unsigned c3 = __ballot_sync(0xffffffffu, kq >> 1 == bw >> 1 && lane < G);
            const bool ties = (c3 & (c3 - 1u)) != 0u;
            const ClPost<T> *win = all + (c3 ? __ffs(c3) - 1 : 0);
            T inv = win->inv;
            int gp = late ? r_lo : win->pos;
            if (!late && ((bw & 1u) || ties || bw >> 1 <= tk)) {
                // the careful choice: whole keys, ties to the smaller row of B, the reference's singular test
                // (FPLUS src/factor_sn_panel.inc:232-233); the same for every thread of the cluster
                const unsigned long long key = mine ? pivkey(pv[0]) : 0ull;
                const unsigned long long mk = warp_max_key(key);
                const bool top = key != 0ull && key == mk;
                const unsigned long long myr = mine ? (unsigned long long)rid_s[tid] : ~0ull;
                const unsigned long long rm = warp_min_u64(top ? myr : ~0ull);
                const unsigned tb = __ballot_sync(0xffffffffu, top && myr == rm);
                const int tl = tb ? __ffs(tb) - 1 : -1;
                __syncthreads();
                if (*(volatile int *)&s_late) { stopped = true; break; }
                cl.sync();                               // every warp has read the quick choice's posts
                if (*(volatile int *)&s_far) { stopped = true; break; }       // (another CTA has left)
                if (tl >= 0) {
                    // (in column order, as the CTAs' posts)
                    if (lane < kk) my->v[lane] = S[lane * sl + (warp << 5) + tl];
                    if (lane == tl) {
#pragma unroll
                        for (int q = 0; q < CL_PW; q++) if (kk + q < w) my->v[kk + q] = pv[q];
                        my->inv = recip(pv[0]);
                        my->pos = r_lo + tid;
                    }
                }
                if (lane == 0) { my->key = mk; my->rid = tl >= 0 ? (long long)rm : LLONG_MAX; }
                cl.sync();
                unsigned long long gk = 0ull;
                long long gr = LLONG_MAX;
                int gi = -1;
                for (int i = lane; i < G * nw; i += 32) {
                    const ClPost<T> *c = cl.map_shared_rank(all + CL_MAXG + i % nw, i / nw);
                    const unsigned long long k = c->key;
                    const long long r = c->rid;
                    if (k != 0ull && (k > gk || (k == gk && r < gr))) { gk = k; gr = r; gi = i; }
                }
                const int src = warp_argbest(gi >= 0 ? (long long)gk : -1, gr);
                gi = src >= 0 ? __shfl_sync(0xffffffffu, gi, src) : -1;
                gk = src >= 0 ? __shfl_sync(0xffffffffu, gk, src) : 0ull;
                if (gi >= 0) {
                    // (a copy of the winner's row in this CTA, as the quick choice's)
                    const ClPost<T> *far = cl.map_shared_rank(all + CL_MAXG + gi % nw, gi / nw);
                    ClPost<T> *near = post + 2 * CL_SLOTS;
                    if (warp == 0 && lane < w) near->v[lane] = far->v[lane];
                    inv = far->inv;
                    gp = far->pos;
                    win = near;
                }
                cl.sync();                               // (nobody leaves, or posts again, while posts are being read)
                const T pvt = win->v[kk];
                const double t = s_thr[kk];
                int stop = 0;
                if (gi < 0 || gk == 0ull || (gk < pivkey_of_modulus<T>(2.0 * t) && vabs(pvt) < t)) stop = 1;
                else if (gp >= nri) stop = 3;
                if (stop) {
                    if (tid == 0 && b == 0) {
                        if (stop == 1) set_status(st, ST_SINGULAR, fcol + j, gi >= 0 ? vabs(pvt) : 0.0, t);
                        else set_status(st, ST_BORDER, front, vabs(pvt), t);
                    }
                    stopped = true;
                    break;
                }
            }
            if (tid == 0) { if (b == 0) chosen[j] = gp; s_piv[kk] = gp; }
            if (warp == nw - 1 && lane < w) Lb[kk * CL_LB + lane] = win->v[lane];        // row kk of L11 \ U11
            const bool own = gp >= r_lo && gp < r_hi;
            if (own && warp == (gp - r_lo) >> 5 && lane >= kk && lane < w) S[lane * sl + (gp - r_lo)] = win->v[lane];
            // the pivot row leaves the search; a live row takes its multiplier and the update of its later columns
            if (r_lo + tid == gp) mine = false;
            const T l = mine ? mul(pv[0], inv) : VT<T>::zero();
            if (mine) S[kk * sl + tid] = l;
            // (entries beyond the panel's end, read past the row, only ever meet each other)
            const T *u = win->v + kk;
#pragma unroll
            for (int q = 1; q < CL_PW; q++) pv[q - 1] = msub(pv[q], l, u[q]);
        }
        if (tid < per) live[tid] = mine ? 1 : 0;
        if (stopped) break;
        __syncthreads();
        for (int r = tid; r < nmine; r += nt)            // (the rows that took part: live ones and this panel's pivots)
            if (was[r]) for (int c = 0; c < w; c++) W[(r_lo + r) + (int64_t)(p0 + c) * ld] = S[c * sl + r];
        if (p0 + w >= npiv) continue;
        // the owners' updates of the pivot rows' later columns are visible to every CTA
        __threadfence();
        cl.sync();
        // the trailing columns [p0 + w, npiv) by chunks
        for (int c0 = p0 + w; c0 < npiv; c0 += CW) {
            const int cw = npiv - c0 < CW ? npiv - c0 : CW;
            for (int e0 = tid; e0 < CL_PW * cw; e0 += 8 * nt) {          // eight loads in flight per thread
                T u[8];
#pragma unroll
                for (int z = 0; z < 8; z++) {
                    const int e = e0 + z * nt, k = e & (CL_PW - 1);
                    u[z] = e < CL_PW * cw && k < w ? ldcg_v(W + s_piv[k] + (int64_t)(c0 + (e / CL_PW)) * ld) : VT<T>::zero();
                }
#pragma unroll
                for (int z = 0; z < 8; z++) {
                    const int e = e0 + z * nt;
                    if (e < CL_PW * cw) Uc[(e & (CL_PW - 1)) * UL + (e / CL_PW)] = u[z];
                }
            }
            __syncthreads();
            // U12 = L11^-1 A12: a thread per column, 8-row blocks in registers
            for (int c = tid; c < cw; c += nt) {
                for (int r0 = 0; r0 < w; r0 += 8) {
                    T y[8];
#pragma unroll
                    for (int z = 0; z < 8; z++) y[z] = r0 + z < w ? Uc[(r0 + z) * UL + c] : VT<T>::zero();
#pragma unroll 4
                    for (int i = 0; i < r0; i++) {
                        const T xi = Uc[i * UL + c];
#pragma unroll
                        for (int z = 0; z < 8; z++) y[z] = msub(y[z], Lb[(r0 + z) * CL_LB + i], xi);
                    }
#pragma unroll
                    for (int z = 1; z < 8; z++)
#pragma unroll
                        for (int zz = 0; zz < z; zz++) y[z] = msub(y[z], Lb[(r0 + z) * CL_LB + r0 + zz], y[zz]);
#pragma unroll
                    for (int z = 0; z < 8; z++) if (r0 + z < w) Uc[(r0 + z) * UL + c] = y[z];
                }
            }
            __syncthreads();
            if (b == (c0 / CW) % G)
                for (int e = tid; e < CL_PW * cw; e += nt) {
                    const int k = e & (CL_PW - 1), c = e / CL_PW;
                    if (k < w) Ub[(p0 + k) + (int64_t)(c0 + c) * npiv] = Uc[k * UL + c];
                }
            // A22 -= L21 U12 on this CTA's live rows: 16-row x 32-column items, a warp each
            constexpr int NF = CP ? 2 : 4;               // 8-column fragments per item
            const int tr = (nmine + 15) >> 4, tc = (cw + 8 * NF - 1) / (8 * NF);
            const int fr_ = lane >> 2, fk = lane & 3;
            for (int it = warp; it < tr * tc; it += nw) {
                const int rb = 16 * (it % tr), cb = 8 * NF * (it / tr);
                // (the entries to update are loaded before the products: their latency is behind these)
                T o[2][NF][2];
                T *x0 = W + (r_lo + rb + fr_) + (int64_t)(c0 + cb + 2 * fk) * ld;
                bool ok[2];
#pragma unroll
                for (int a = 0; a < 2; a++) {
                    ok[a] = rb + 8 * a + fr_ < nmine && live[rb + 8 * a + fr_];
#pragma unroll
                    for (int f = 0; f < NF; f++)
#pragma unroll
                        for (int h = 0; h < 2; h++)
                            o[a][f][h] = ok[a] && cb + 8 * f + 2 * fk + h < cw ? x0[8 * a + (int64_t)(8 * f + h) * ld] : VT<T>::zero();
                }
                double ar[2][NF][2], ai[2][NF][2];
#pragma unroll
                for (int a = 0; a < 2; a++)
#pragma unroll
                    for (int f = 0; f < NF; f++) { ar[a][f][0] = ar[a][f][1] = 0.0; if constexpr (CP) ai[a][f][0] = ai[a][f][1] = 0.0; }
#pragma unroll 2
                for (int ks = 0; ks < w; ks += 4) {
                    const int k = ks + fk;
                    T la[2], ub[NF];
#pragma unroll
                    for (int a = 0; a < 2; a++) {
                        const int r = rb + 8 * a + fr_;
                        la[a] = k < w && r < nmine ? S[k * sl + r] : VT<T>::zero();
                    }
#pragma unroll
                    for (int f = 0; f < NF; f++) {
                        const int c = cb + 8 * f + fr_;
                        ub[f] = k < w && c < cw ? Uc[k * UL + c] : VT<T>::zero();
                    }
#pragma unroll
                    for (int a = 0; a < 2; a++)
#pragma unroll
                        for (int f = 0; f < NF; f++) {
                            if constexpr (CP) {
                                dmma(ar[a][f][0], ar[a][f][1], la[a].x, ub[f].x);
                                dmma(ai[a][f][0], ai[a][f][1], la[a].x, ub[f].y);
                                dmma(ar[a][f][0], ar[a][f][1], -la[a].y, ub[f].y);
                                dmma(ai[a][f][0], ai[a][f][1], la[a].y, ub[f].x);
                            } else dmma(ar[a][f][0], ar[a][f][1], la[a], ub[f]);
                        }
                }
#pragma unroll
                for (int a = 0; a < 2; a++)
#pragma unroll
                    for (int f = 0; f < NF; f++)
#pragma unroll
                        for (int h = 0; h < 2; h++)
                            if (ok[a] && cb + 8 * f + 2 * fk + h < cw) {
                                T *x = x0 + 8 * a + (int64_t)(8 * f + h) * ld;
                                if constexpr (CP) *x = cplx{o[a][f][h].x - ar[a][f][h], o[a][f][h].y - ai[a][f][h]};
                                else *x = o[a][f][h] - ar[a][f][h];
                            }
            }
            __syncthreads();
        }
    }
    cl.sync();                                           // no CTA leaves while another may still read its shared memory
}

}  // namespace fpl
