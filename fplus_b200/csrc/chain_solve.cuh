// chain_solve.cuh -- the triangular sweeps through the dense chain (fronts of at most 64 pivots whose columns are all of
// [f, n), each front's contribution block the next one's only child).
//
// The chain is one dependency: K blocks of nb unknowns, each needing every one before it.  The column sweeps (U, U^T) read
// n^2 / 2 entries of U12 (8.6 GB for n = 32,768 complex), the row sweeps (L, L^T) K blocks of at most 256 x 64.
//
//   k_chain_u  U x = y (TR 0, from the last front) or U^T z = w (TR 1, 2, from the first): one launch.  CTA 0 solves block
//              after block; the other CTAs own blocks of unknowns and subtract the solved blocks' products from them as
//              these appear, two or more blocks ahead of the solver (which takes the product with the block just solved
//              itself, from shared memory).  U12's 64 x 64 blocks are contiguous and stream through a ring of shared
//              memory without waiting for x.  Cross-CTA order: a counter of the blocks solved and a flag per block whose
//              products are all in, release / acquire, waits bounded.  A cooperative launch, so all CTAs are resident.
//   k_chain_l  L (TR 0) or L^T (TR 1, 2) by one CTA per group of right-hand sides, the front's row vector in shared
//              memory from front to front (no global round trip), L streamed in 16-column pieces.
// Both solve a front's triangle by 16 x 16 diagonal blocks inverted once per factorization (k_chain_dinv): four dependent
// products instead of 64 dependent steps.
#pragma once
#include "kernels.cuh"

namespace fpl {

constexpr int CH_THREADS = 256, CH_NB = 64, CH_MAXNR = 256, CH_STAGES = 3;
constexpr unsigned CH_SPIN = 1u << 22;          // polls before a wait gives up (about a second)

// a chain front as the sweeps read it; nslot, slot, tau: where the previous chain front's contribution rows enter (its row t
// at initial row slot + t, t < nslot, or tau + t - nslot)
struct ChainFront {
    long long f, np, nr, L_off, U_off, row_off, nslot, slot, tau;
};

// the inverses of the 16 x 16 diagonal blocks of a chain front's U11 (dinv[0 .. 4)) and unit-lower L11 (dinv[4 .. 8)),
// column-major, identity beyond the front's pivots; a thread per column
template <typename T>
__global__ void __launch_bounds__(128) k_chain_dinv(const ChainFront *__restrict__ fr, const T *__restrict__ La, T *__restrict__ dinv,
                                                    const DevStatus *st)
{
    if (st->code) return;
    const ChainFront F = fr[blockIdx.x];
    const int lower = threadIdx.x >> 6, b = (threadIdx.x >> 4) & 3, c = threadIdx.x & 15;
    const int np = (int)F.np, k0 = 16 * b;
    const T *L = La + F.L_off;
    T x[16];
    auto at = [&](int i, int k) -> T { return k0 + i < np && k0 + k < np ? L[(k0 + i) + (int64_t)(k0 + k) * F.nr] : VT<T>::zero(); };
    if (lower) {
#pragma unroll
        for (int i = 0; i < 16; i++) {
            T s = i == c ? VT<T>::one() : VT<T>::zero();
#pragma unroll
            for (int k = 0; k < i; k++) s = msub(s, at(i, k), x[k]);
            x[i] = s;
        }
    } else {
#pragma unroll
        for (int i = 15; i >= 0; i--) {
            T s = i == c ? VT<T>::one() : VT<T>::zero();
#pragma unroll
            for (int k = 15; k > i; k--) s = msub(s, at(i, k), x[k]);
            const T d = at(i, i);
            x[i] = k0 + i < np ? (is_zero(d) ? VT<T>::zero() : mul(s, recip(d))) : s;
        }
    }
    T *o = dinv + ((int64_t)blockIdx.x * 8 + 4 * lower + b) * 256 + c * 16;
#pragma unroll
    for (int i = 0; i < 16; i++) o[i] = x[i];
}

template <int N> __device__ __forceinline__ void cp_async_wait_n() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void st_release_u32(unsigned *p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// one thread waits until *p >= v; false when the wait ran out
__device__ __forceinline__ bool chain_wait(const unsigned *p, unsigned v)
{
    for (unsigned k = 0; k < CH_SPIN; k++)
        if (ld_acquire_u32(p) >= v) return true;
    return false;
}
template <typename T> __device__ __forceinline__ T madd(T a, T l, T p);
template <> __device__ __forceinline__ double madd<double>(double a, double l, double p) { return fma(l, p, a); }
template <> __device__ __forceinline__ cplx madd<cplx>(cplx a, cplx l, cplx p)
{
    return cplx{fma(-l.y, p.y, fma(l.x, p.x, a.x)), fma(l.y, p.x, fma(l.x, p.y, a.y))};
}
template <int TR> __device__ __forceinline__ double opv(double v) { return v; }
template <int TR> __device__ __forceinline__ cplx opv(cplx v) { return TR == 2 ? cplx{v.x, -v.y} : v; }

// acc[r] = sum over this lane's share of the inner index k < kn of M(o, k) x[k + r * xld], four lanes (q) per output o,
// then summed over the four lanes.  M(o, k) = Mp[k * ld + o] (plain), or op(Mp[o * ld + k]) (transposed; the lanes of
// neighbouring outputs start two apart, so that they read other banks)
template <typename T, int TR, int RB>
__device__ __forceinline__ void quad_mv(T (&acc)[RB], const T *Mp, int ld, int o, int q, int kn, const T *x, int xld, int rb)
{
#pragma unroll
    for (int r = 0; r < RB; r++) acc[r] = VT<T>::zero();
    const int ne = (kn + 3) >> 2;
#pragma unroll 4
    for (int e = 0; e < ne; e++) {
        int k;
        if (TR == 0) k = q + 4 * e;
        else { int ee = e + (o & 1); if (ee >= ne) ee -= ne; k = q + 4 * ee; }
        if (k < kn) {
            const T m = TR == 0 ? Mp[k * ld + o] : opv<TR>(Mp[o * ld + k]);
#pragma unroll
            for (int r = 0; r < RB; r++) if (r < rb) acc[r] = madd<T>(acc[r], m, x[k + r * xld]);
        }
    }
#pragma unroll
    for (int r = 0; r < RB; r++) {
        acc[r] = add(acc[r], shfl_xor_v<T>(acc[r], 1));
        acc[r] = add(acc[r], shfl_xor_v<T>(acc[r], 2));
    }
}

// dynamic shared memory of k_chain_u for `own` blocks per worker and rb right-hand sides (the larger of the two roles)
static inline size_t chain_u_smem(int64_t own, int64_t rb, int64_t vs)
{
    const size_t worker = (size_t)(CH_STAGES * CH_NB * CH_NB + CH_NB * rb * (1 + own)) * vs;
    const size_t solver = (size_t)(2 * CH_NB * CH_NB + 2 * 2560 + 2 * CH_NB * rb) * vs;
    return worker > solver ? worker : solver;
}

// t = 0 .. K - 1: the blocks in solve order (TR 0: front K - 1 - t, else front t).  Y: the right-hand sides (pivot order,
// overwritten), X: the solution; both n x nrhs.  sync[0]: blocks solved; sync[1 + t]: block t has every product but that of
// block t - 1.  RB >= rb right-hand sides.
template <typename T, int TR, int RB>
__global__ void __launch_bounds__(CH_THREADS) k_chain_u(const ChainFront *__restrict__ fr, int K, int nb, const T *__restrict__ La,
                                                        const T *__restrict__ Ua, const T *__restrict__ dinv, T *Y, T *X, int64_t n,
                                                        int rb, unsigned *sync, DevStatus *st)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_ok;
    const int tid = threadIdx.x, o = tid >> 2, q = tid & 3;
    auto front_of = [&](int t) -> int { return TR == 0 ? K - 1 - t : t; };
    const int np_last = (int)fr[K - 1].np;
    auto np_of = [&](int t) -> int { return front_of(t) == K - 1 ? np_last : nb; };
    // the 64 x 64 block of U12 that couples block t to block s < t in solve order, and its column count
    auto block_ptr = [&](int t, int s) -> const T * {
        const int a = TR == 0 ? front_of(t) : front_of(s), c = TR == 0 ? front_of(s) : front_of(t);    // rows of front a, columns of front c > a
        return Ua + fr[a].U_off + (int64_t)(c - a - 1) * nb * nb;
    };
    auto block_size = [&](int t, int s) -> int { return nb * (TR == 0 ? np_of(s) : np_of(t)); };
    auto copy = [&](T *dst, const T *src, int cnt) { for (int e = tid; e < cnt; e += CH_THREADS) cp_async_el(dst + e, src + e); };
    if (st->code) return;
    if (blockIdx.x > 0) {
        // a worker: owns the blocks t = w, w + W, .. (w = blockIdx.x - 1)
        const int w = blockIdx.x - 1, W = gridDim.x - 1;
        T *ring = reinterpret_cast<T *>(smem_raw);
        T *xs = ring + CH_STAGES * CH_NB * CH_NB;      // x of the block being subtracted: xs[k + r * CH_NB]
        T *acc = xs + CH_NB * rb;                      // owned block j's sums: acc[(j * rb + r) * CH_NB + o]
        const int own = w < K ? (K - 1 - w) / W + 1 : 0;
        for (int e = tid; e < own * rb * CH_NB; e += CH_THREADS) acc[e] = VT<T>::zero();
        // tasks in order: s ascending, the owned t >= s + 2 ascending
        auto first_t = [&](int s) -> int { const int m = s + 2; return m <= w ? w : w + (m - w + W - 1) / W * W; };
        int ps = 0, pt = 0;                            // the next task to load
        auto settle = [&](int &s, int &t) { while (s <= K - 3 && t >= K) { s++; t = first_t(s); } };
        pt = first_t(0);
        settle(ps, pt);
        int cs = ps, ct = pt;                          // the task to compute
        auto load_next = [&](int slot) {
            if (ps <= K - 3) {
                copy(ring + slot * CH_NB * CH_NB, block_ptr(pt, ps), block_size(pt, ps));
                pt += W;
                settle(ps, pt);
            }
            cp_async_commit();
        };
        for (int k = 0; k < CH_STAGES - 1; k++) load_next(k);
        int slot = 0, have = -1;
        while (cs <= K - 3) {
            if (have != cs) {                          // a new solved block: wait for it, its x into shared memory
                if (tid == 0) s_ok = chain_wait(sync, (unsigned)cs + 1u);
                __syncthreads();
                if (!s_ok) { if (tid == 0) set_status(st, ST_WAIT, cs, 0, 0); break; }
                const int64_t f = fr[front_of(cs)].f;
                const int np = np_of(cs);
                for (int e = tid; e < np * rb; e += CH_THREADS) { const int k = e % np, r = e / np; xs[k + r * CH_NB] = ldcg_v(X + f + k + r * n); }
                have = cs;
            }
            cp_async_wait_n<CH_STAGES - 2>();
            __syncthreads();                           // the block and x are in; the slot before is free
            load_next((slot + CH_STAGES - 1) % CH_STAGES);
            const int no = TR == 0 ? nb : np_of(ct), kn = TR == 0 ? np_of(cs) : nb;
            T a[RB];
            quad_mv<T, TR, RB>(a, ring + slot * CH_NB * CH_NB, nb, o < no ? o : 0, q, kn, xs, CH_NB, rb);
            T *ao = acc + (int64_t)((ct - w) / W) * rb * CH_NB + o;
            if (q == 0 && o < no) {
#pragma unroll
                for (int r = 0; r < RB; r++) if (r < rb) ao[r * CH_NB] = add(ao[r * CH_NB], a[r]);
                if (cs == ct - 2) {                    // the last product this worker takes for block ct
                    T *y = Y + fr[front_of(ct)].f + o;
#pragma unroll
                    for (int r = 0; r < RB; r++) if (r < rb) y[r * n] = sub(y[r * n], ao[r * CH_NB]);
                    __threadfence();
                }
            }
            if (cs == ct - 2) {
                __syncthreads();
                if (tid == 0) st_release_u32(sync + 1 + ct, 1u);
            }
            slot = (slot + 1) % CH_STAGES;
            ct += W;
            settle(cs, ct);
        }
        cp_async_wait_n<0>();
        return;
    }
    // the solver
    T *off = reinterpret_cast<T *>(smem_raw);          // two stages: the block coupling t to t - 1
    T *tri = off + 2 * CH_NB * CH_NB;                  // two stages: U11's 16-column panels above the diagonal blocks (panel b: 16b rows,
                                                       // at 256 b (b - 1) / 2), then the four inverted diagonal blocks (at 1536)
    T *ys = tri + 2 * 2560, *xs = ys + CH_NB * rb;
    auto load = [&](int t) {
        if (t < K) {
            const int sl = t & 1, k = front_of(t), np = np_of(t);
            T *tr = tri + sl * 2560;
            const T *L = La + fr[k].L_off;
            const int64_t nr = fr[k].nr;
            if (t > 0) copy(off + sl * CH_NB * CH_NB, block_ptr(t, t - 1), block_size(t, t - 1));
            const T *dv = dinv + (int64_t)k * 8 * 256;
            copy(tr + 1536, dv, 1024);
            for (int e = tid; e < 1536; e += CH_THREADS) {
                const int b = e < 256 ? 1 : e < 768 ? 2 : 3, p = e - 128 * b * (b - 1), rows = 16 * b, r = p % rows, c = 16 * b + p / rows;
                if (c < np) cp_async_el(tr + e, L + r + (int64_t)c * nr);
            }
        }
        cp_async_commit();
    };
    load(0);
    for (int t = 0; t < K; t++) {
        const int sl = t & 1, k = front_of(t), np = np_of(t), nbk = (np + 15) >> 4;
        const int64_t f = fr[k].f;
        if (tid == 0) s_ok = t < 2 || chain_wait(sync + 1 + t, 1u);
        cp_async_wait_n<0>();
        __syncthreads();
        if (!s_ok) { if (tid == 0) set_status(st, ST_WAIT, t, 0, 0); break; }
        load(t + 1);                                   // (into the stage that block t - 1 used)
        T a[RB];
        if (t > 0) quad_mv<T, TR, RB>(a, off + sl * CH_NB * CH_NB, nb, o < np ? o : 0, q, np_of(t - 1), xs, CH_NB, rb);
        if (q == 0 && o < np) {
            const T d = La[fr[k].L_off + o + (int64_t)o * fr[k].nr];
            if (is_zero(d)) set_status(st, ST_SOLVE_ZERO, f + o, 0, 0);
#pragma unroll
            for (int r = 0; r < RB; r++)
                if (r < rb) {
                    const T y = ldcg_v(Y + f + o + r * n);
                    ys[o + r * CH_NB] = t > 0 ? sub(y, a[r]) : y;
                }
        }
        __syncthreads();
        const T *tr = tri + sl * 2560;
        for (int bb = 0; bb < nbk; bb++) {
            const int b = TR == 0 ? nbk - 1 - bb : bb, k0 = 16 * b;
            const T *pan = tr + 128 * b * (b - 1);     // panel b (16b rows)
            if (TR != 0 && b > 0) {
                // w_b -= U[0 .. 16b, b]^T z
                if (o < 16) {
                    quad_mv<T, TR, RB>(a, pan, 16 * b, k0 + o < np ? o : 0, q, k0, xs, CH_NB, rb);
                    if (q == 0 && k0 + o < np)
#pragma unroll
                        for (int r = 0; r < RB; r++) if (r < rb) ys[k0 + o + r * CH_NB] = sub(ys[k0 + o + r * CH_NB], a[r]);
                }
                __syncthreads();
            }
            const int w16 = np - k0 < 16 ? np - k0 : 16;
            if (o < 16) {
                quad_mv<T, TR, RB>(a, tr + 1536 + 256 * b, 16, o < w16 ? o : 0, q, w16, ys + k0, CH_NB, rb);
                if (q == 0 && o < w16)
#pragma unroll
                    for (int r = 0; r < RB; r++) if (r < rb) { xs[k0 + o + r * CH_NB] = a[r]; X[f + k0 + o + r * n] = a[r]; }
            }
            __syncthreads();
            if (TR == 0 && b > 0) {
                // y[0 .. 16b) -= U[0 .. 16b, b] x_b
                if (o < k0) {
                    quad_mv<T, 0, RB>(a, pan, 16 * b, o, q, w16, xs + k0, CH_NB, rb);
                    if (q == 0)
#pragma unroll
                        for (int r = 0; r < RB; r++) if (r < rb) ys[o + r * CH_NB] = sub(ys[o + r * CH_NB], a[r]);
                }
                __syncthreads();
            }
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) st_release_u32(sync, (unsigned)t + 1u);
    }
    cp_async_wait_n<0>();
}

// dynamic shared memory of k_chain_l: CH_LSTAGES pieces of 16 columns (with the inverted diagonal block), two row vectors
constexpr int CH_LSTAGES = 4;
static inline size_t chain_l_smem(int64_t maxnr, int64_t rb, int64_t vs)
{
    return (size_t)(CH_LSTAGES * (16 * maxnr + 256) + 2 * maxnr * rb) * vs;
}

// The L sweep (TR 0: v0 = the first front's gathered vector in its final row order, VB; later fronts' entering rows from R
// in row space; y into S2 in pivot order) or the L^T sweep (TR 1, 2: z = R in pivot order; x into S2).  blockIdx.x: the
// group of RB right-hand sides.
template <typename T, int TR, int RB>
__global__ void __launch_bounds__(CH_THREADS) k_chain_l(const ChainFront *__restrict__ fr, int K, int maxnr, const T *__restrict__ La,
                                                        const T *__restrict__ dinv, const int *__restrict__ permall,
                                                        const int64_t *__restrict__ rowinit, const T *__restrict__ VB0, int64_t vstride,
                                                        const T *__restrict__ R, T *__restrict__ S2, int64_t n, int nrhs)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = blockIdx.x * RB, rb = nrhs - r0 < RB ? nrhs - r0 : RB;
    const int psz = 16 * maxnr + 256;
    T *ring = reinterpret_cast<T *>(smem_raw);         // piece: L[row, 16b + c] at c * maxnr + row, then the inverted diagonal block
    T *v = ring + CH_LSTAGES * psz, *vn = v + maxnr * rb;      // the front's row vector: v[pos + r * maxnr]
    R += (int64_t)r0 * n; S2 += (int64_t)r0 * n; VB0 += (int64_t)r0 * vstride;
    // the pieces in order: TR 0: fronts and blocks ascending, else descending
    int pk = TR == 0 ? 0 : K - 1, pb = TR == 0 ? 0 : ((int)fr[K - 1].np + 15) / 16 - 1;
    auto load_next = [&](int slot) {
        if (pk >= 0 && pk < K) {
            const ChainFront F = fr[pk];
            const int np = (int)F.np, nr = (int)F.nr, k0 = 16 * pb, w = np - k0 < 16 ? np - k0 : 16;
            T *d = ring + slot * psz;
            for (int c = warp; c < w; c += CH_THREADS / 32)
                for (int row = k0 + 16 + lane; row < nr; row += 32) cp_async_el(d + c * maxnr + row, La + F.L_off + row + (int64_t)(k0 + c) * F.nr);
            // (a last block of fewer than 16 pivots: the rows from its end on)
            if (w < 16) for (int c = warp; c < w; c += CH_THREADS / 32)
                for (int row = k0 + w + lane; row < nr && row < k0 + 16; row += 32) cp_async_el(d + c * maxnr + row, La + F.L_off + row + (int64_t)(k0 + c) * F.nr);
            cp_async_el(d + 16 * maxnr + tid, dinv + ((int64_t)pk * 8 + 4 + pb) * 256 + tid);
            if (TR == 0) { if (k0 + 16 < np) pb++; else { pk++; pb = 0; } }
            else { if (pb > 0) pb--; else { pk--; if (pk >= 0) pb = ((int)fr[pk].np + 15) / 16 - 1; } }
        }
        cp_async_commit();
    };
    for (int k = 0; k < CH_LSTAGES - 1; k++) load_next(k);
    int slot = 0;
    if (TR == 0) {
        for (int e = tid; e < (int)fr[0].nr * rb; e += CH_THREADS) { const int p = e % (int)fr[0].nr, r = e / (int)fr[0].nr; v[p + r * maxnr] = VB0[p + r * vstride]; }
    } else {
        const ChainFront F = fr[K - 1];
        for (int e = tid; e < (int)F.np * rb; e += CH_THREADS) { const int p = e % (int)F.np, r = e / (int)F.np; v[p + r * maxnr] = R[F.f + p + r * n]; }
    }
    for (int kk = 0; kk < K; kk++) {
        const int k = TR == 0 ? kk : K - 1 - kk;
        const ChainFront F = fr[k];
        const int np = (int)F.np, nr = (int)F.nr, nbk = (np + 15) >> 4;
        // for the next front: this thread's row position there (TR 0), or here (TR 1, 2: where it came from)
        int pm = -1;
        T ent[RB];
        const int kn = TR == 0 ? k + 1 : k - 1;        // the next front
        const ChainFront G = TR == 0 ? fr[kn < K ? kn : k] : F;        // the front whose rows enter from the one below it
        const bool more = TR == 0 ? kn < K : kn >= 0;
        if (more && tid < (int)G.nr) pm = permall[G.row_off + tid];
        for (int bb = 0; bb < nbk; bb++) {
            const int b = TR == 0 ? bb : nbk - 1 - bb, k0 = 16 * b, w = np - k0 < 16 ? np - k0 : 16;
            cp_async_wait_n<CH_LSTAGES - 2>();
            __syncthreads();
            load_next((slot + CH_LSTAGES - 1) % CH_LSTAGES);
            const T *Lp = ring + slot * psz, *D = Lp + 16 * maxnr;
            slot = (slot + 1) % CH_LSTAGES;
            T a[RB];
            if (TR == 0) {
                if (tid < 64) {
                    const int o = tid >> 2, q = tid & 3;
                    quad_mv<T, 0, RB>(a, D, 16, o, q, w, v + k0, maxnr, rb);
                    __syncwarp();
                }
                __syncthreads();
                if (tid < 64 && (tid & 3) == 0 && (tid >> 2) < w) {
                    const int o = tid >> 2;
#pragma unroll
                    for (int r = 0; r < RB; r++) if (r < rb) { v[k0 + o + r * maxnr] = a[r]; S2[F.f + k0 + o + r * n] = a[r]; }
                }
                __syncthreads();
                // the rows below: two lanes per row, eight columns each
                for (int i0 = k0 + w; i0 < nr; i0 += CH_THREADS / 2) {
                    const int row = i0 + (tid >> 1), h = tid & 1;
                    T s[RB];
#pragma unroll
                    for (int r = 0; r < RB; r++) s[r] = VT<T>::zero();
                    if (row < nr) {
#pragma unroll
                        for (int c = 0; c < 8; c++) {
                            const int cc = 2 * c + h;
                            if (cc < w) {
                                const T l = Lp[cc * maxnr + row];
#pragma unroll
                                for (int r = 0; r < RB; r++) if (r < rb) s[r] = madd<T>(s[r], l, v[k0 + cc + r * maxnr]);
                            }
                        }
                    }
#pragma unroll
                    for (int r = 0; r < RB; r++) {
                        s[r] = add(s[r], shfl_xor_v<T>(s[r], 1));
                        if (r < rb && row < nr && h == 0) v[row + r * maxnr] = sub(v[row + r * maxnr], s[r]);
                    }
                }
            } else {
                // s_b = z_b - L[rows below, b]^T x: sixteen lanes per column
                const int c = tid >> 4, l16 = tid & 15;
                T s[RB];
#pragma unroll
                for (int r = 0; r < RB; r++) s[r] = VT<T>::zero();
                if (c < w)
                    for (int row = k0 + w + l16; row < nr; row += 16) {
                        const T l = opv<TR>(Lp[c * maxnr + row]);
#pragma unroll
                        for (int r = 0; r < RB; r++) if (r < rb) s[r] = madd<T>(s[r], l, v[row + r * maxnr]);
                    }
#pragma unroll
                for (int r = 0; r < RB; r++) {
#pragma unroll
                    for (int m = 8; m > 0; m >>= 1) s[r] = add(s[r], shfl_xor_v<T>(s[r], m));
                    if (r < rb && c < w && l16 == 0) v[k0 + c + r * maxnr] = sub(v[k0 + c + r * maxnr], s[r]);
                }
                __syncthreads();
                if (tid < 64) quad_mv<T, TR, RB>(a, D, 16, tid >> 2, tid & 3, w, v + k0, maxnr, rb);
                __syncthreads();
                if (tid < 64 && (tid & 3) == 0 && (tid >> 2) < w) {
                    const int o = tid >> 2;
#pragma unroll
                    for (int r = 0; r < RB; r++) if (r < rb) { v[k0 + o + r * maxnr] = a[r]; S2[F.f + k0 + o + r * n] = a[r]; }
                }
            }
        }
        if (!more) break;
        // the next front's vector
        int t = -1;                                    // the contribution row (of the front below G) at this position of G
        if (pm >= 0) t = pm >= (int)G.slot && pm < (int)(G.slot + G.nslot) ? pm - (int)G.slot : pm >= (int)G.tau ? (int)G.nslot + pm - (int)G.tau : -1;
        if (TR == 0) {
            if (pm >= 0 && t < 0) {
                const int64_t g = rowinit[G.row_off + pm];
#pragma unroll
                for (int r = 0; r < RB; r++) if (r < rb) ent[r] = g >= 0 ? R[g + r * n] : VT<T>::zero();
            }
            __syncthreads();
            if (pm >= 0)
#pragma unroll
                for (int r = 0; r < RB; r++) if (r < rb) vn[tid + r * maxnr] = t >= 0 ? v[np + t + r * maxnr] : ent[r];
        } else {
            const ChainFront H = fr[kn];
            T z[RB];
            if (tid < (int)H.np)
#pragma unroll
                for (int r = 0; r < RB; r++) if (r < rb) z[r] = R[H.f + tid + r * n];
            __syncthreads();
            if (t >= 0)
#pragma unroll
                for (int r = 0; r < RB; r++) if (r < rb) vn[(int)H.np + t + r * maxnr] = v[tid + r * maxnr];
            if (tid < (int)H.np)
#pragma unroll
                for (int r = 0; r < RB; r++) if (r < rb) vn[tid + r * maxnr] = z[r];
        }
        T *sw = v; v = vn; vn = sw;
        // (the next piece's barrier orders these writes before they are read)
    }
    cp_async_wait_n<0>();
}

}  // namespace fpl
