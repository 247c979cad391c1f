// block_lu_cl.cuh -- the pivot block of a tall front (too large for one CTA's shared memory) by one thread-block cluster.
#pragma once
#include "kernels.cuh"
#include "front_lu.cuh"

namespace fpl {

// Partial-pivot LU of a front's pivot block (nrows x npiv) in one launch of one cluster of G CTAs (the interface and the
// outputs of k_block_lu_mc: rows never move, chosen[j] = the position of step j's pivot row, U12 beyond a row's own panel in
// Ub; k_mc_order and k_mc_lout follow).  CTA b owns the rows [b * per, b * per + per), a thread per row, and keeps their
// 32-column panel in shared memory.  A pivot step:
//   1. every warp elects its best row by the leading 30 bits of the pivot key (one warp reduction, one ballot) and leaves
//      that row's panel values (with the update the row still lacks), its reciprocal and position in shared memory; after a
//      block barrier every warp takes the CTA's best and stores its word and values into one or two CTAs of the cluster;
//   2. cluster barrier; the threads apply the last pivot's update to their rows' later columns meanwhile;
//   3. every warp takes the same winner from the G words in its own shared memory.
// Equal leading bits, border rows, values at the edge of the range or near the singular threshold go through whole keys and
// row ids with two more barriers, the same for all (rare).  After a panel every CTA forms U12 of the panel's pivot rows and
// applies the rank-32 update to its live rows as FP64 mma products.
//
// What bounds it (B200): the npiv dependent steps, each a cluster barrier with its remote stores (about 500 cycles by itself;
// reading the winner's values from its CTA after the barrier instead took 700 more), and 2 npiv^2 nrows / G flops of trailing updates per CTA.
constexpr int CL_PW = 32, CL_LB = CL_PW + 1, CL_MAXG = 16, CL_MAXW = 16, CL_SLOTS = CL_MAXG + CL_MAXW;
template <typename T> __host__ __device__ constexpr int cl_cw() { return VT<T>::cplx_ ? 64 : 128; }
// leading dimensions of the panel (rows) and of a chunk of U12 (columns): the mma fragments of a half-warp hit all banks
template <typename T> __host__ __device__ constexpr int cl_ld(int m) { return VT<T>::cplx_ ? ((m + 7) & ~7) + 2 : ((m + 15) & ~15) + 4; }
template <typename T> struct __align__(16) ClPost {
    T v[CL_PW];                // the candidate row's panel values
    T inv;                     // 1 / its value in the step's column
    long long rid;             // (the careful choice: its row of B, its whole key)
    unsigned long long key;
    int pos;
    unsigned word;             // the key's leading bits, and a flag for the careful choice
    int pad[2];
};
template <typename T> __host__ __device__ constexpr size_t cl_smem(int per)
{
    return (size_t)(CL_PW * cl_ld<T>(per) + CL_PW * CL_LB + CL_PW * cl_ld<T>(cl_cw<T>())) * sizeof(T) +
           (size_t)2 * CL_SLOTS * sizeof(ClPost<T>) + (size_t)per * 8 + (size_t)((per + 15) & ~15);
}

template <typename T>
__global__ void __launch_bounds__(512) k_block_lu_cl(T *W, int64_t ld, int nrows, int npiv, int nri, int per, int64_t fcol,
                                                     const double *__restrict__ colmax, double pivot_rel,
                                                     const int64_t *__restrict__ rowid, int64_t *__restrict__ chosen,
                                                     T *__restrict__ Ub, DevStatus *st, int64_t front)
{
    namespace cg = cooperative_groups;
    constexpr bool CP = VT<T>::cplx_;
    constexpr int CW = cl_cw<T>(), UL = cl_ld<T>(CW);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int sl = cl_ld<T>(per);
    T *S = reinterpret_cast<T *>(smem_raw);              // the panel: S[c * sl + r]
    T *Lb = S + CL_PW * sl;                              // the panel's pivot rows: Lb[k * CL_LB + c] (L11 \ U11)
    T *Uc = Lb + CL_PW * CL_LB;                          // a chunk of U12: Uc[k * UL + c]
    ClPost<T> *post = reinterpret_cast<ClPost<T> *>(reinterpret_cast<unsigned char *>(S) +
        ((size_t)(CL_PW * sl + CL_PW * CL_LB + CL_PW * UL) * sizeof(T)));           // [parity][the CTAs', then the own warps']
    long long *rid_s = reinterpret_cast<long long *>(post + 2 * CL_SLOTS);
    unsigned char *live = reinterpret_cast<unsigned char *>(rid_s + per);
    __shared__ int s_piv[CL_PW];
    __shared__ double s_thr[CL_PW];
    __shared__ unsigned s_tk[CL_PW];
    __shared__ int s_stop;
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
    const int G = gridDim.x, b = blockIdx.x;
    const int r_lo = b * per, r_hi = r_lo + per < nrows ? r_lo + per : nrows, nmine = r_hi > r_lo ? r_hi - r_lo : 0;
    const int npr = npiv < nrows ? npiv : nrows;
    if (tid == 0) s_stop = st->code != 0;
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
        for (int c = warp; c < w; c += nw)               // a warp per column
            for (int r = lane; r < nmine; r += 32) S[c * sl + r] = W[(r_lo + r) + (int64_t)(p0 + c) * ld];
        __syncthreads();
        bool mine = tid < nmine && live[tid];
        T x = mine ? S[tid] : VT<T>::zero();             // this row's value in the step's column
        for (int kk = 0; kk < w; kk++) {
            const int j = p0 + kk, par = j & 1;
            const unsigned tk = s_tk[kk];
            // 1. the warp's candidate
            const Key30<T> kv(x, mine);
            const unsigned m30 = __reduce_max_sync(0xffffffffu, kv.key);
            const T xinv = kv.inverse(x);
            const unsigned cnd = __ballot_sync(0xffffffffu, kv.key == m30);
            const int wl = __ffs(cnd) - 1, row = (warp << 5) + wl;       // (a warp without live rows posts an empty word)
            ClPost<T> *all = post + par * CL_SLOTS, *my = all + CL_MAXG + warp;
            __syncwarp();                                // (the warp's own rows of S, as their threads left them)
            if (warp < nwr) {
                // the row's panel values (its multipliers before this column), with the previous pivot's update after it
                if (row < nmine && lane < w) {
                    T v = S[lane * sl + row];
                    if (kk >= 1 && lane > kk) v = msub(v, S[(kk - 1) * sl + row], Lb[(kk - 1) * CL_LB + lane]);
                    my->v[lane] = v;
                }
                if (lane == wl) {
                    my->inv = xinv;
                    my->pos = r_lo + row;
                    const bool odd = (cnd & (cnd - 1u)) != 0u || m30 == LU6_ODD || r_lo + row >= nri;
                    my->word = (m30 << 1) | (unsigned)(odd && m30 != 0u);
                }
            }
            __syncthreads();
            {
                // the CTA's best (the same for every warp), into the CTAs d = warp, warp + nw, ..
                const unsigned k = lane < nwr ? all[CL_MAXG + lane].word : 0u, mb = __reduce_max_sync(0xffffffffu, k);
                const unsigned c2 = __ballot_sync(0xffffffffu, k >> 1 == mb >> 1 && lane < nwr);
                const ClPost<T> *bst = all + CL_MAXG + (c2 ? __ffs(c2) - 1 : 0);
                const T v = lane < w ? bst->v[lane] : VT<T>::zero();
                const T vi = bst->inv;
                const int vp = bst->pos;
                for (int d = warp; d < G; d += nw) {
                    ClPost<T> *dst = cl.map_shared_rank(all + b, d);
                    if (lane < w) dst->v[lane] = v;
                    if (lane == 0) { dst->inv = vi; dst->pos = vp; dst->word = mb | (unsigned)((c2 & (c2 - 1u)) != 0u && mb != 0u); }
                }
            }
            // 2. the barrier; meanwhile the previous pivot's update of this row's later columns
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            if (mine && kk >= 1) {
                const T l = S[(kk - 1) * sl + tid];
                const T *lb = Lb + (kk - 1) * CL_LB;
                for (int c0 = kk + 1; c0 < w; c0 += 8) {         // (loads first: the stores could alias them)
                    T xv[8], uv[8];
#pragma unroll
                    for (int z = 0; z < 8; z++) { const int c = c0 + z < w ? c0 + z : w - 1; xv[z] = S[c * sl + tid]; uv[z] = lb[c]; }
#pragma unroll
                    for (int z = 0; z < 8; z++) if (c0 + z < w) S[(c0 + z) * sl + tid] = msub(xv[z], l, uv[z]);
                }
            }
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
            // 3. the winner, the same for every warp
            const unsigned kq = lane < G ? all[lane].word : 0u;
            const unsigned bw = __reduce_max_sync(0xffffffffu, kq);
            const unsigned c3 = __ballot_sync(0xffffffffu, kq >> 1 == bw >> 1 && lane < G);
            const bool ties = (c3 & (c3 - 1u)) != 0u;
            const ClPost<T> *win = all + (c3 ? __ffs(c3) - 1 : 0);
            T v = lane < w ? win->v[lane] : VT<T>::zero();
            T inv = win->inv;
            int gp = win->pos;
            if ((bw & 1u) || ties || bw >> 1 <= tk) {
                // the careful choice: whole keys, ties to the smaller row of B, the reference's singular test
                // (FPLUS src/factor_sn_panel.inc:232-233); the same for every thread of the cluster
                const unsigned long long key = mine ? pivkey(x) : 0ull;
                const unsigned long long mk = warp_max_key(key);
                const bool top = key != 0ull && key == mk;
                const unsigned long long myr = mine ? (unsigned long long)rid_s[tid] : ~0ull;
                const unsigned long long rm = warp_min_u64(top ? myr : ~0ull);
                const unsigned tb = __ballot_sync(0xffffffffu, top && myr == rm);
                const int tl = tb ? __ffs(tb) - 1 : -1;
                cl.sync();                               // every warp has read the quick choice's posts
                if (tl >= 0) {
                    // (the row's later columns have had the previous pivot's update by now)
                    if (lane < w) my->v[lane] = S[lane * sl + (warp << 5) + tl];
                    if (lane == tl) { my->inv = recip(x); my->pos = r_lo + tid; }
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
                    win = cl.map_shared_rank(all + CL_MAXG + gi % nw, gi / nw);
                    v = lane < w ? win->v[lane] : VT<T>::zero();
                    inv = win->inv;
                    gp = win->pos;
                }
                const T pv = shfl_v<T>(v, kk);
                const double t = s_thr[kk];
                int stop = 0;
                if (gi < 0 || gk == 0ull || (gk < pivkey_of_modulus<T>(2.0 * t) && vabs(pv) < t)) stop = 1;
                else if (gp >= nri) stop = 3;
                cl.sync();                               // (nobody leaves, or posts again, while posts are being read)
                if (stop) {
                    if (tid == 0 && b == 0) {
                        if (stop == 1) set_status(st, ST_SINGULAR, fcol + j, gi >= 0 ? vabs(pv) : 0.0, t);
                        else set_status(st, ST_BORDER, front, vabs(pv), t);
                    }
                    stopped = true;
                    break;
                }
            }
            if (tid == 0) { if (b == 0) chosen[j] = gp; s_piv[kk] = gp; }
            // every warp keeps the winner's row of L11 \ U11 (the same values) for the deferred update
            if (lane < w) Lb[kk * CL_LB + lane] = v;
            const T un = shfl_v<T>(v, kk + 1 < w ? kk + 1 : kk);
            // the pivot row leaves the search; a live row takes its multiplier and the next column's update
            if (mine) {
                if (r_lo + tid == gp) mine = false;
                else {
                    const T l = mul(x, inv);
                    S[kk * sl + tid] = l;
                    if (kk + 1 < w) { x = msub(S[(kk + 1) * sl + tid], l, un); S[(kk + 1) * sl + tid] = x; }
                }
            }
            __syncwarp();
        }
        if (tid < per) live[tid] = mine ? 1 : 0;
        if (stopped) break;
        __syncthreads();
        for (int c = warp; c < w; c += nw)
            for (int r = lane; r < nmine; r += 32) W[(r_lo + r) + (int64_t)(p0 + c) * ld] = S[c * sl + r];
        if (p0 + w >= npiv) continue;
        // (the pivot rows' values right of the panel are read from W: their owners wrote them before the panel's barriers)
        // the trailing columns [p0 + w, npiv) by chunks
        for (int c0 = p0 + w; c0 < npiv; c0 += CW) {
            const int cw = npiv - c0 < CW ? npiv - c0 : CW;
            for (int e0 = tid; e0 < CL_PW * cw; e0 += 8 * nt) {          // eight loads in flight per thread
                T u[8];
#pragma unroll
                for (int z = 0; z < 8; z++) {
                    const int e = e0 + z * nt, k = e & (CL_PW - 1);
                    u[z] = e < CL_PW * cw && k < w ? ldcg_v(W + s_piv[k] + (int64_t)(c0 + (e >> 5)) * ld) : VT<T>::zero();
                }
#pragma unroll
                for (int z = 0; z < 8; z++) {
                    const int e = e0 + z * nt;
                    if (e < CL_PW * cw) Uc[(e & (CL_PW - 1)) * UL + (e >> 5)] = u[z];
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
                    const int k = e & (CL_PW - 1), c = e >> 5;
                    if (k < w) Ub[(p0 + k) + (int64_t)(c0 + c) * npiv] = Uc[k * UL + c];
                }
            // A22 -= L21 U12 on this CTA's live rows: 16-row x 32-column items, a warp each
            constexpr int NF = CP ? 2 : 4;               // 8-column fragments per item
            const int tr = (nmine + 15) >> 4, tc = (cw + 8 * NF - 1) / (8 * NF);
            const int fr_ = lane >> 2, fk = lane & 3;
            for (int it = warp; it < tr * tc; it += nw) {
                const int rb = 16 * (it % tr), cb = 8 * NF * (it / tr);
                double ar[2][NF][2], ai[2][NF][2];
#pragma unroll
                for (int a = 0; a < 2; a++)
#pragma unroll
                    for (int f = 0; f < NF; f++) { ar[a][f][0] = ar[a][f][1] = 0.0; if constexpr (CP) ai[a][f][0] = ai[a][f][1] = 0.0; }
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
                for (int a = 0; a < 2; a++) {
                    const int r = rb + 8 * a + fr_;
                    const bool ok = r < nmine && live[r < per ? r : 0];
                    T *x0 = W + (r_lo + r) + (int64_t)(c0 + cb + 2 * fk) * ld;
                    T o[NF][2];
#pragma unroll
                    for (int f = 0; f < NF; f++)
#pragma unroll
                        for (int h = 0; h < 2; h++)
                            o[f][h] = ok && cb + 8 * f + 2 * fk + h < cw ? x0[(int64_t)(8 * f + h) * ld] : VT<T>::zero();
#pragma unroll
                    for (int f = 0; f < NF; f++)
#pragma unroll
                        for (int h = 0; h < 2; h++)
                            if (ok && cb + 8 * f + 2 * fk + h < cw) {
                                if constexpr (CP) x0[(int64_t)(8 * f + h) * ld] = cplx{o[f][h].x - ar[a][f][h], o[f][h].y - ai[a][f][h]};
                                else x0[(int64_t)(8 * f + h) * ld] = o[f][h] - ar[a][f][h];
                            }
                }
            }
            __syncthreads();
        }
    }
    cl.sync();                                           // no CTA leaves while another may still read its shared memory
}

}  // namespace fpl
