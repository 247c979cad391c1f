// sweeps.cuh -- the level-scheduled triangular sweeps (trans 0) of the fronts below the dense chain.
#pragma once
#include "chain_solve.cuh"

namespace fpl {

constexpr int SW_THREADS = 256;

// A front's triangle applied to the vector x (x[k * RB + r], k up to np and zero from there to the next sixteen, shared
// memory; overwritten; sd: the side of the front's diagonal blocks, less than 16 only for a single one), the result in xs (the same layout): xs = L11^-1 x (UPPER false) or U11^-1 x.  By 16-column blocks: the
// block's 16 unknowns (diag_solve), then the rows beyond it updated from the block's
// columns; the packed pieces (at pk, see k_front_pack) stream through a ring of STG stages of psz elements by bulk copies
// ahead of the chain.  The pipe (its barriers, initialised, and the pieces taken so far) serves several calls of a CTA of
// SW_THREADS.  Ends with a barrier; false (for every thread) when a copy did not land.
//
// What bounds it: np / 16 dependent block steps (two small products, two barriers).
struct TriPipe { unsigned long long *bars; int done; };
__host__ __device__ constexpr int tri_pad(int np) { return (np + 15) & ~15; }
template <typename T, bool UPPER, int RB, int STG>
__device__ __forceinline__ bool tri16(const T *__restrict__ pk, int sd, int np, T *x, T *xs, T *ring, int psz, TriPipe &pipe)
{
    const int tid = threadIdx.x, nbk = (np + 15) >> 4;
    int issued = 0;
    auto blk = [&](int i) -> int { return UPPER ? nbk - 1 - i : i; };
    auto load_next = [&]() {                           // one thread
        if (issued >= nbk) return;
        const int b = blk(issued), k0 = 16 * b, w = np - k0 < 16 ? np - k0 : 16, sl = (pipe.done + issued) % STG;
        const unsigned bytes = (unsigned)((sd * sd + 16 * (UPPER ? k0 : np - k0 - w)) * sizeof(T));
        bulk_expect(pipe.bars + sl, bytes);
        bulk_load(ring + sl * psz, pk + (UPPER ? pk_u(b) : pk_l(b, np)), bytes, pipe.bars + sl);
        issued++;
    };
    if (tid == SW_THREADS - 1) for (int k = 0; k < STG - 1; k++) load_next();
    bool ok = true;
    for (int i = 0; i < nbk; i++) {
        const int b = blk(i), k0 = 16 * b, w = np - k0 < 16 ? np - k0 : 16, d = pipe.done + i;
        ok = bar_wait(pipe.bars + d % STG, (unsigned)(d / STG) & 1u) && ok;
        __syncthreads();                               // (the piece before is no longer read; x is as its updates left it)
        const T *D = ring + (d % STG) * psz, *Lp = D + 256;
        if (tid == SW_THREADS - 1) load_next();
        if (tid < diag_threads(RB))
            diag_solve<T, 0, UPPER, !UPPER, RB, false>(D, sd, w, x + k0 * RB, [&](int i, int r, T v) { xs[(k0 + i) * RB + r] = v; });
        __syncthreads();
        // the rows beyond the block: two lanes per row, eight columns each (columns beyond the pivots are zero)
        const int ra = UPPER ? 0 : k0 + w, rl = UPPER ? k0 : np - k0 - w;
        for (int i0 = 0; i0 < rl; i0 += SW_THREADS / 2) {
            const int ii = i0 + (tid & 15) + 16 * (tid >> 5), h = (tid >> 4) & 1, row = ii < rl ? ii : 0;
            T s[RB];
#pragma unroll
            for (int r = 0; r < RB; r++) s[r] = VT<T>::zero();
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const T l = Lp[(2 * c + h) * rl + row];
                const T *xv = xs + (k0 + 2 * c + h) * RB;
#pragma unroll
                for (int r = 0; r < RB; r++) s[r] = madd<T>(s[r], l, xv[r]);
            }
#pragma unroll
            for (int r = 0; r < RB; r++) {
                s[r] = add(s[r], shfl_xor_v<T>(s[r], 16));
                if (ii < rl && h == 0) x[(ra + ii) * RB + r] = sub(x[(ra + ii) * RB + r], s[r]);
            }
        }
    }
    pipe.done += nbk;
    return !__syncthreads_or(!ok);
}
// the barriers of a pipe (ends with a barrier)
template <int STG> __device__ __forceinline__ TriPipe tri_pipe(unsigned long long *bars)
{
    if (threadIdx.x == 0) {
        for (int k = 0; k < STG; k++) bar_init(bars + k, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    return TriPipe{bars, 0};
}
// shared memory of tri16 (x, xs and the ring), in elements
static inline int64_t tri16_elems(int64_t np, int64_t rb, int stg) { return 2 * tri_pad((int)np) * rb + stg * (16 * np + 256); }

// L sweep of a level's small fronts, a CTA each: the front's vector in its final row order, x =
// L11^-1 v (into Y in pivot order), then the contribution u = v[np:] - L21 x into VB, a thread per row with L's row read
// once for all of the pass's right-hand sides
template <typename T, int RB>
__global__ void __launch_bounds__(SW_THREADS) k_sw_fwdL(const SvFront *__restrict__ fr, const int *__restrict__ list,
                                                        const T *__restrict__ La, const T *__restrict__ pk,
                                                        const int64_t *__restrict__ rowinit, const int *__restrict__ permall,
                                                        const int64_t *__restrict__ rsp, const int64_t *__restrict__ rsi,
                                                        const T *__restrict__ R, T *__restrict__ Y, T *__restrict__ VB, int64_t vstride,
                                                        int64_t n, int nrhs, DevStatus *st)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const SvFront F = fr[list[blockIdx.x]];
    const int nr = (int)F.nr, np = (int)(F.np < F.nr ? F.np : F.nr), nri = (int)F.nri, tid = threadIdx.x, m = nr - np;
    const int npd = tri_pad(np), psz = 16 * np + 256;
    T *ring = reinterpret_cast<T *>(smem_raw), *x = ring + 2 * psz, *xs = x + npd * RB, *v = xs + npd * RB;       // v: the rows below the pivots, v[t + r * m]
    __shared__ unsigned long long bars[2];
    TriPipe pipe = tri_pipe<2>(bars);
    for (int e = tid; e < npd * RB; e += SW_THREADS) x[e] = VT<T>::zero();
    __syncthreads();
    const T *L = La + F.L_off;
    const int *perm = permall + F.row_off;
    pdl_wait();
    pdl_trigger();
    for (int r0 = 0; r0 < nrhs; r0 += RB) {
        const int rc = nrhs - r0 < RB ? nrhs - r0 : RB;
        for (int e = tid; e < nr * rc; e += SW_THREADS) {
            const int k = e % nr, r = e / nr, i = F.np > 0 ? perm[k] : k;     // (a front without pivots keeps its order)
            const int64_t g = F.row_off + i, ri = rowinit[g], q0 = rsp[g], q1 = rsp[g + 1];
            T val = (i < nri && ri >= 0) ? R[ri + (int64_t)(r0 + r) * n] : VT<T>::zero();
            for (int64_t q = q0; q < q1; q++) val = add(val, VB[rsi[q] + (int64_t)(r0 + r) * vstride]);
            if (k < np) x[k * RB + r] = val; else v[k - np + r * m] = val;
        }
        __syncthreads();
        if (!tri16<T, false, RB, 2>(pk + F.l_pk, (int)F.pk_s, np, x, xs, ring, psz, pipe)) { if (tid == 0) set_status(st, ST_WAIT, F.f, 0, 0); return; }
        for (int e = tid; e < np * rc; e += SW_THREADS) { const int k = e % np, r = e / np; Y[F.f + k + (int64_t)(r0 + r) * n] = xs[k * RB + r]; }
        for (int t = tid; t < m; t += SW_THREADS) {
            T acc[RB];
#pragma unroll
            for (int r = 0; r < RB; r++) acc[r] = VT<T>::zero();
            for (int k0 = 0; k0 < np; k0 += 16) {
                T lv[16];
#pragma unroll
                for (int q = 0; q < 16; q++) lv[q] = k0 + q < np ? L[np + t + (int64_t)(k0 + q) * nr] : VT<T>::zero();
#pragma unroll
                for (int q = 0; q < 16; q++)
                    if (k0 + q < np)
#pragma unroll
                        for (int r = 0; r < RB; r++) acc[r] = madd<T>(acc[r], lv[q], xs[(k0 + q) * RB + r]);
            }
#pragma unroll
            for (int r = 0; r < RB; r++)
                if (r < rc) VB[F.row_off + np + t + (int64_t)(r0 + r) * vstride] = sub(v[t + r * m], acc[r]);
        }
        __syncthreads();
        if (r0 + RB < nrhs) for (int e = tid; e < npd * RB; e += SW_THREADS) x[e] = VT<T>::zero();
        __syncthreads();
    }
}
static inline int64_t sw_fwdL_elems(int64_t nr, int64_t np, int64_t rb) { return nr * rb + tri16_elems(np, rb, 2); }

// U sweep of a level's small fronts, a CTA each: the CB columns' x gathered into shared memory,
// the product with U12 split over column groups (each U12 entry read once for all of the pass's right-hand sides; the
// groups' sums added in order), then x = U11^-1 (y - the product)
template <typename T, int RB>
__global__ void __launch_bounds__(SW_THREADS) k_sw_bwdU(const SvFront *__restrict__ fr, const int *__restrict__ list,
                                                        const T *__restrict__ La, const T *__restrict__ Ua, const T *__restrict__ pk,
                                                        const int64_t *__restrict__ cols, const T *__restrict__ Y, T *__restrict__ X,
                                                        int64_t n, int nrhs, DevStatus *st)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const SvFront F = fr[list[blockIdx.x]];
    const int np = (int)F.np, ncb = (int)(F.nc - F.np), tid = threadIdx.x;
    if (np == 0) { pdl_wait(); return; }
    const int G = SW_THREADS / np;                     // column groups (np <= 64)
    const int npd = tri_pad(np), psz = 16 * np + 256;
    T *ring = reinterpret_cast<T *>(smem_raw), *x = ring + 2 * psz, *xs = x + npd * RB, *xc = xs + npd * RB, *red = xc + ncb * RB;
    __shared__ unsigned long long bars[2];
    TriPipe pipe = tri_pipe<2>(bars);
    for (int e = tid; e < npd * RB; e += SW_THREADS) x[e] = VT<T>::zero();
    for (int e = tid; e < ncb * RB; e += SW_THREADS) xc[e] = VT<T>::zero();
    __syncthreads();
    const T *U12 = Ua + F.U_off;
    const int64_t *cb = cols + F.col_off + np;
    pdl_wait();
    pdl_trigger();
    for (int r0 = 0; r0 < nrhs; r0 += RB) {
        const int rc = nrhs - r0 < RB ? nrhs - r0 : RB;
        for (int t = tid; t < ncb; t += SW_THREADS) {
            const T *xr = X + cb[t] + (int64_t)r0 * n;
#pragma unroll
            for (int r = 0; r < RB; r++) if (r < rc) xc[t * RB + r] = xr[(int64_t)r * n];
        }
        __syncthreads();
        const int i = tid % np, g = tid / np;
        if (g < G) {
            T acc[RB];
#pragma unroll
            for (int r = 0; r < RB; r++) acc[r] = VT<T>::zero();
            for (int t0 = g; t0 < ncb; t0 += 8 * G) {
                T u[8];
#pragma unroll
                for (int q = 0; q < 8; q++) u[q] = t0 + q * G < ncb ? U12[i + (int64_t)(t0 + q * G) * np] : VT<T>::zero();
#pragma unroll
                for (int q = 0; q < 8; q++)
                    if (t0 + q * G < ncb)
#pragma unroll
                        for (int r = 0; r < RB; r++) acc[r] = madd<T>(acc[r], u[q], xc[(t0 + q * G) * RB + r]);
            }
#pragma unroll
            for (int r = 0; r < RB; r++) red[(g * RB + r) * np + i] = acc[r];
        }
        __syncthreads();
        for (int e = tid; e < np * rc; e += SW_THREADS) {
            const int ii = e % np, r = e / np;
            T s = VT<T>::zero();
            for (int gg = 0; gg < G; gg++) s = add(s, red[(gg * RB + r) * np + ii]);
            x[ii * RB + r] = sub(Y[F.f + ii + (int64_t)(r0 + r) * n], s);
        }
        __syncthreads();
        if (!tri16<T, true, RB, 2>(pk + F.u_pk, (int)F.pk_s, np, x, xs, ring, psz, pipe)) { if (tid == 0) set_status(st, ST_WAIT, F.f, 0, 0); return; }
        for (int e = tid; e < np * rc; e += SW_THREADS) { const int k = e % np, r = e / np; X[F.f + k + (int64_t)(r0 + r) * n] = xs[k * RB + r]; }
        __syncthreads();
    }
}
static inline int64_t sw_bwdU_elems(int64_t nc, int64_t np, int64_t rb) { return nc * rb + SW_THREADS * rb + tri16_elems(np, rb, 2); }

// The larger fronts.  x = L11^-1 v[:np], a CTA per front (blockIdx.x) and group of RB right-hand sides (blockIdx.y); x into
// VB in place and into Y in pivot order
template <typename T, int RB, int STG>
__global__ void __launch_bounds__(SW_THREADS) k_swb_L11(const SvFront *__restrict__ fr, const int *__restrict__ list,
                                                        const T *__restrict__ pk, T *__restrict__ VB,
                                                        int64_t vstride, T *__restrict__ Y, int64_t n, int nrhs, DevStatus *st)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const SvFront F = fr[list[blockIdx.x]];
    const int np = (int)(F.np < F.nr ? F.np : F.nr), tid = threadIdx.x, r0 = blockIdx.y * RB, rc = nrhs - r0 < RB ? nrhs - r0 : RB;
    if (np == 0) return;
    const int npd = tri_pad(np), psz = 16 * np + 256;
    T *ring = reinterpret_cast<T *>(smem_raw), *x = ring + STG * psz, *xs = x + npd * RB;
    __shared__ unsigned long long bars[STG];
    TriPipe pipe = tri_pipe<STG>(bars);
    for (int e = tid; e < npd * RB; e += SW_THREADS) {
        const int k = e % npd, r = e / npd;
        x[k * RB + r] = k < np && r < rc ? VB[F.row_off + k + (int64_t)(r0 + r) * vstride] : VT<T>::zero();
    }
    __syncthreads();
    if (!tri16<T, false, RB, STG>(pk + F.l_pk, (int)F.pk_s, np, x, xs, ring, psz, pipe)) { if (tid == 0) set_status(st, ST_WAIT, F.f, 0, 0); return; }
    for (int e = tid; e < np * rc; e += SW_THREADS) {
        const int k = e % np, r = e / np;
        VB[F.row_off + k + (int64_t)(r0 + r) * vstride] = xs[k * RB + r];
        Y[F.f + k + (int64_t)(r0 + r) * n] = xs[k * RB + r];
    }
}

// u = v[np:] - L21 x, 32 rows per CTA (blockIdx.x; blockIdx.y: the front): eight groups of threads take the pivot columns
// k = g, g + 8, .. (sixteen loads in flight each), their sums added in order.  RB right-hand sides per pass over L
template <typename T, int RB>
__global__ void __launch_bounds__(SW_THREADS) k_swb_L21(const SvFront *__restrict__ fr, const int *__restrict__ list,
                                                        const T *__restrict__ La, T *__restrict__ VB, int64_t vstride, int nrhs)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const SvFront F = fr[list[blockIdx.y]];
    const int np = (int)(F.np < F.nr ? F.np : F.nr), tid = threadIdx.x, rl = tid & 31, g = tid >> 5;
    const int64_t row = np + (int64_t)blockIdx.x * 32 + rl;
    if (np == 0 || np + (int64_t)blockIdx.x * 32 >= F.nr) return;
    T *xs = reinterpret_cast<T *>(smem_raw), *red = xs + np * RB;      // x: xs[k * RB + r]; red[(g * RB + r) * 32 + rl]
    const T *L = La + F.L_off + row;
    const bool on = row < F.nr;
    for (int r0 = 0; r0 < nrhs; r0 += RB) {
        const int rc = nrhs - r0 < RB ? nrhs - r0 : RB;
        for (int e = tid; e < np * RB; e += SW_THREADS) { const int k = e % np, r = e / np; xs[k * RB + r] = r < rc ? VB[F.row_off + k + (int64_t)(r0 + r) * vstride] : VT<T>::zero(); }
        __syncthreads();
        T acc[RB];
#pragma unroll
        for (int r = 0; r < RB; r++) acc[r] = VT<T>::zero();
        for (int k0 = g; k0 < np; k0 += 128) {
            T lv[16];
#pragma unroll
            for (int q = 0; q < 16; q++) lv[q] = on && k0 + 8 * q < np ? L[(int64_t)(k0 + 8 * q) * F.nr] : VT<T>::zero();
#pragma unroll
            for (int q = 0; q < 16; q++)
                if (k0 + 8 * q < np)
#pragma unroll
                    for (int r = 0; r < RB; r++) acc[r] = madd<T>(acc[r], lv[q], xs[(k0 + 8 * q) * RB + r]);
        }
#pragma unroll
        for (int r = 0; r < RB; r++) red[(g * RB + r) * 32 + rl] = acc[r];
        __syncthreads();
        for (int e = tid; e < 32 * rc; e += SW_THREADS) {
            const int l = e & 31, r = e >> 5;
            const int64_t rw = np + (int64_t)blockIdx.x * 32 + l;
            T s = VT<T>::zero();
#pragma unroll
            for (int gg = 0; gg < 8; gg++) s = add(s, red[(gg * RB + r) * 32 + l]);
            if (rw < F.nr) { T *o = VB + F.row_off + rw + (int64_t)(r0 + r) * vstride; *o = sub(*o, s); }
        }
        __syncthreads();
    }
}

// The partial products U12 x[CB columns] of chunk blockIdx.x of a front's CB columns (F.nch chunks; blockIdx.y: the front;
// blockIdx.z: 64 rows of U12): four column groups (sixteen loads in flight each), their sums added in order, into part
// (the front's partial sums start at F.poff * nrhs).  RB right-hand sides per pass over U12
template <typename T, int RB>
__global__ void __launch_bounds__(SW_THREADS) k_swb_u12(const SvFront *__restrict__ fr, const int *__restrict__ list,
                                                        const T *__restrict__ Ua, const int64_t *__restrict__ cols,
                                                        const T *__restrict__ X, int64_t n, int nrhs, T *__restrict__ part)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const SvFront F = fr[list[blockIdx.y]];
    const int np = (int)F.np, tid = threadIdx.x, rl = tid & 63, g = tid >> 6, i0 = 64 * blockIdx.z;
    if (blockIdx.x >= F.nch || i0 >= np) return;
    const int64_t ncb = F.nc - F.np, chunk = (ncb + F.nch - 1) / F.nch, c0 = blockIdx.x * chunk;
    const int cc = (int)(c0 + chunk < ncb ? chunk : ncb - c0);
    T *Xs = reinterpret_cast<T *>(smem_raw), *red = Xs + chunk * RB;   // Xs[k * RB + r]; red[(g * RB + r) * 64 + rl]
    const bool on = i0 + rl < np;
    const T *U = Ua + F.U_off + i0 + rl + c0 * np;
    const int64_t *cb = cols + F.col_off + np + c0;
    T *pp = part + F.poff * nrhs + (int64_t)blockIdx.x * np * nrhs;
    for (int r0 = 0; r0 < nrhs; r0 += RB) {
        const int rc = nrhs - r0 < RB ? nrhs - r0 : RB;
        for (int k = tid; k < cc; k += SW_THREADS) {
            const T *xr = X + cb[k] + (int64_t)r0 * n;
#pragma unroll
            for (int r = 0; r < RB; r++) Xs[k * RB + r] = r < rc ? xr[(int64_t)r * n] : VT<T>::zero();
        }
        __syncthreads();
        T acc[RB];
#pragma unroll
        for (int r = 0; r < RB; r++) acc[r] = VT<T>::zero();
        for (int k0 = g; k0 < cc; k0 += 64) {
            T u[16];
#pragma unroll
            for (int q = 0; q < 16; q++) u[q] = on && k0 + 4 * q < cc ? U[(int64_t)(k0 + 4 * q) * np] : VT<T>::zero();
#pragma unroll
            for (int q = 0; q < 16; q++)
                if (k0 + 4 * q < cc)
#pragma unroll
                    for (int r = 0; r < RB; r++) acc[r] = madd<T>(acc[r], u[q], Xs[(k0 + 4 * q) * RB + r]);
        }
#pragma unroll
        for (int r = 0; r < RB; r++) red[(g * RB + r) * 64 + rl] = acc[r];
        __syncthreads();
        for (int e = tid; e < 64 * rc; e += SW_THREADS) {
            const int l = e & 63, r = e >> 6;
            const T s = add(add(red[r * 64 + l], red[(RB + r) * 64 + l]), add(red[(2 * RB + r) * 64 + l], red[(3 * RB + r) * 64 + l]));
            if (i0 + l < np) pp[i0 + l + (int64_t)(r0 + r) * np] = s;
        }
        __syncthreads();
    }
}

// x = U11^-1 (y - the partial products, in chunk order), a CTA per front (blockIdx.x) and group of RB right-hand sides
// (blockIdx.y); presummed: k_svb_psum left y - the products in the front's first partial sum
template <typename T, int RB, int STG>
__global__ void __launch_bounds__(SW_THREADS) k_swb_bwdU(const SvFront *__restrict__ fr, const int *__restrict__ list,
                                                         const T *__restrict__ pk, const T *__restrict__ part,
                                                         const T *__restrict__ Y, T *__restrict__ X, int64_t n, int nrhs, int presummed, DevStatus *st)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const SvFront F = fr[list[blockIdx.x]];
    const int np = (int)F.np, tid = threadIdx.x, r0 = blockIdx.y * RB, rc = nrhs - r0 < RB ? nrhs - r0 : RB;
    if (np == 0) return;
    const int npd = tri_pad(np), psz = 16 * np + 256;
    T *ring = reinterpret_cast<T *>(smem_raw), *x = ring + STG * psz, *xs = x + npd * RB;
    const T *pp = part + F.poff * nrhs;
    __shared__ unsigned long long bars[STG];
    TriPipe pipe = tri_pipe<STG>(bars);
    for (int e = tid; e < npd * RB; e += SW_THREADS) {
        const int i = e % npd, rr = e / npd;
        const int64_t r = r0 + rr;
        T v = VT<T>::zero();
        if (i < np && rr < rc) {
            if (presummed && F.nch > 0) v = pp[i + r * np];
            else {
                v = Y[F.f + i + r * n];
                for (int64_t q0 = 0; q0 < F.nch; q0 += 16) {     // sixteen loads in flight, the sum in chunk order
                    T pv[16];
#pragma unroll
                    for (int q = 0; q < 16; q++) pv[q] = q0 + q < F.nch ? pp[(q0 + q) * np * nrhs + i + r * np] : VT<T>::zero();
#pragma unroll
                    for (int q = 0; q < 16; q++) if (q0 + q < F.nch) v = sub(v, pv[q]);
                }
            }
        }
        x[i * RB + rr] = v;
    }
    __syncthreads();
    if (!tri16<T, true, RB, STG>(pk + F.u_pk, (int)F.pk_s, np, x, xs, ring, psz, pipe)) { if (tid == 0) set_status(st, ST_WAIT, F.f, 0, 0); return; }
    for (int e = tid; e < np * rc; e += SW_THREADS) { const int k = e % np, r = e / np; X[F.f + k + (int64_t)(r0 + r) * n] = xs[k * RB + r]; }
}

}  // namespace fpl
