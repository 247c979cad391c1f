// chain_solve.cuh -- the triangular sweeps through the dense chain (fronts of at most 64 pivots whose columns are all of
// [f, n), each front's contribution block the next one's only child), and the packed triangles that all sweeps read.
//
// The chain is one dependency: K blocks of nb unknowns, each needing every one before it.  The column sweeps (U, U^T) read
// n^2 / 2 entries of U12 (8.6 GB for n = 32,768 complex), the row sweeps (L, L^T) K blocks of at most 197 x 64.
//
//   k_chain_u  U x = y (TR 0, from the last front) or U^T z = w (TR 1, 2, from the first): one launch.  CTA 0 solves block
//              after block; the other CTAs own blocks of unknowns and subtract the solved blocks' products from them as
//              these appear, two or more blocks ahead of the solver (which takes the product with the block just solved
//              itself, from shared memory).  U12's 64 x 64 blocks are contiguous and stream through a ring of shared
//              memory without waiting for x.  Cross-CTA order: a counter of the blocks solved and a flag per block whose
//              products are all in, release / acquire, waits bounded.  All CTAs are resident together: a
//              cooperative launch.
//   k_chain_l  L (TR 0) or L^T (TR 1, 2) by one CTA per group of right-hand sides, the front's row vector in shared
//              memory from front to front (no global round trip), L streamed in 16-column pieces.
// Both solve a front's triangle by 16 x 16 diagonal blocks (diag_solve): one product with the inverted block where that is as
// accurate as the 16 steps of a substitution, else the substitution.  All streams are bulk copies (cp.async.bulk) of
// contiguous, packed pieces: element-wise cp.async issued 26 cycles a warp and held the shared-memory loads of the chain up
// behind it (a 16 x 16 product took 2,800 cycles).
#pragma once
#include "kernels.cuh"

namespace fpl {

constexpr int CH_THREADS = 256, CH_NB = 64, CH_MAXNR = 256, CH_STAGES = 3, CH_UTHREADS = CH_THREADS + 64;
constexpr unsigned CH_SPIN = 1u << 22;          // polls before a wait for another CTA gives up (about a second)
constexpr long long CH_CYCLES = 4000000000ll;   // the longest wait for a bulk copy (about two seconds)
constexpr int CH_BLK = CH_NB * CH_NB + 2;       // a ring stage (two elements more: see load_block)

// a chain front as the sweeps read it; nslot, slot, tau: where the previous chain front's contribution rows enter (its row t
// at initial row slot + t, t < nslot, or tau + t - nslot); u_pk, l_pk: its packed pieces
struct ChainFront {
    long long f, np, nr, row_off, nslot, slot, tau, u_pk, l_pk;
};

// Packed pieces of a front's triangles, one per 16 pivots (block b, k0 = 16 b): the diagonal block (256 elements, element
// (i, k) at pk_e(i, k): rows and columns both read without bank conflicts), then the 16 columns' other entries (zero beyond
// the pivots):
//   U piece b: rows [0, k0) of U11's columns (leading dimension k0), at u_pk + pk_u(b)
//   L piece b: rows [k0 + w, R) of L's columns (w pivots in the block, leading dimension R - k0 - w), at l_pk + pk_l(b, R);
//              R = the front's rows on the dense chain, its pivots elsewhere
// The diagonal block is kept as its inverse D (identity beyond the pivots) or as the triangle itself (U: with the reciprocals
// of the pivots on its diagonal; one beyond the pivots); which, says the far corner of the other triangle (pk_flag: zero for
// the inverse).  A tree front of at most 8 pivots has a block of 2, 4 or 8 rows and columns (side s) instead of 16: with 256
// elements for every one-pivot front a diagonal matrix's packed triangles were 512 times its factors.
// x = D y leaves a residual of up to about u |U| |D| |U| |x| where substitution leaves u |U| |x|.  So the inverse stands only where
// the 1-norms of R^-1 |U| |D| R and of C^-1 |U|^T |D|^T C (the transposed sweeps) are at most PACK_GROWTH; R and C hold the
// block's row and column sums, so that a scaling of the rows or columns changes nothing.  Measured over blocks with a column
// within 1 to 1e-8.5 of the ones before it, rows scaled over up to 16 decades: the largest row's |r| / (|U| |x| + |y|) is at
// most 1.4e-16 times the norm for x = D y (where D stands: 7e-15, 1.5e-16 in the middle), 2.3e-16 for substitution.  The norms
// (of |re| + |im|) are at most 7 on the stencils' and the random matrices' fronts; on the pencils' chains about 22 in the
// middle, at most 33 (L), 1 block of 100 above 128 (U); on narrow complex bands' 33 to 51 in the middle, 1 to 25 of 100 above.
__host__ __device__ constexpr int64_t pk_u(int64_t b) { return 256 * b + 128 * b * (b - 1); }
__host__ __device__ constexpr int64_t pk_l(int64_t b, int64_t R) { return 256 * b + 16 * b * R - 128 * b * (b + 1); }
__host__ __device__ constexpr int pk_e(int i, int k, int s = 16) { return s * k + ((i + k) & (s - 1)); }
__host__ __device__ constexpr int pk_flag(bool lower, int s = 16) { return lower ? pk_e(0, s - 1, s) : pk_e(s - 1, 0, s); }
__host__ __device__ constexpr int pk_side(int64_t np) { return np > 8 ? 16 : np > 4 ? 8 : np > 2 ? 4 : 2; }
constexpr double PACK_GROWTH = 128.0;
__device__ __forceinline__ double abs1(double v) { return fabs(v); }
__device__ __forceinline__ double abs1(cplx v) { return fabs(v.x) + fabs(v.y); }

template <typename T>
__global__ void __launch_bounds__(128) k_front_pack(const SvFront *__restrict__ fr, const int *__restrict__ dfront, const T *__restrict__ La,
                                                    T *__restrict__ pk, const DevStatus *st)
{
    if (st->code) return;
    const int64_t blk = blockIdx.x;
    const SvFront F = fr[dfront[blk]];
    const int np = (int)(F.np < F.nr ? F.np : F.nr), b = (int)(blk - F.d_off), k0 = 16 * b, w = np - k0 < 16 ? np - k0 : 16;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sd = (int)F.pk_s;
    const T *L = La + F.L_off;
    T *du = pk + F.u_pk + pk_u(b), *dl = pk + F.l_pk + pk_l(b, F.l_rows);
    if (warp == 0) {                                    // the diagonal blocks: a lane per column (U's, then L's)
        const int lower = lane >> 4, c = lane & 15;
        T x[16];
        auto at = [&](int i, int k) -> T { return i < w && k < w ? L[(k0 + i) + (int64_t)(k0 + k) * F.nr] : VT<T>::zero(); };
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
                const T d = at(i, i);                   // (never zero: the factorization reports such a column as singular)
                x[i] = i < w ? (is_zero(d) ? VT<T>::zero() : mul(s, recip(d))) : s;
            }
        }
        // the two norms (of the block and of its transpose): lane c has row c's sum of moduli and column c's, then the sums over
        // the other direction's divided by them, then one entry of each norm; an inverse, a sum or a quotient out of range
        // makes it infinite or NaN
        auto mod = [&](int i, int k) -> double { return i == k && (lower || i >= w) ? 1.0 : (lower ? i >= k : i <= k) ? abs1(at(i, k)) : 0.0; };
        double rs = 0.0, cs = 0.0, rq = 0.0, cq = 0.0, g = 0.0, gt = 0.0;
        for (int k = 0; k < 16; k++) { rs += mod(c, k); cs += mod(k, c); }
        const double ri = 1.0 / rs, ci = 1.0 / cs;
        for (int k = 0; k < 16; k++) {
            cq += mod(k, c) * __shfl_sync(0xffffffffu, ri, k, 16);
            rq += mod(c, k) * __shfl_sync(0xffffffffu, ci, k, 16);
        }
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const double m = abs1(x[k]);
            g += __shfl_sync(0xffffffffu, cq, k, 16) * m;
            double t = m * rq;
            for (int h = 8; h > 0; h >>= 1) t += __shfl_xor_sync(0xffffffffu, t, h);
            if (k == c) gt = t;
        }
        g *= rs;
        gt *= cs;
        const unsigned good = __ballot_sync(0xffffffffu, g <= PACK_GROWTH && gt <= PACK_GROWTH);
        const bool inv = (lower ? good >> 16 : good & 0xffffu) == 0xffffu;
        T *o = lower ? dl : du;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            if (!inv) {
                x[i] = (lower ? i > c : i < c) ? at(i, c) : VT<T>::zero();
                if (!lower && i == c) { const T d = at(c, c); x[i] = c >= w ? VT<T>::one() : is_zero(d) ? VT<T>::zero() : recip(d); }
                if (lower ? i == 0 && c == sd - 1 : i == sd - 1 && c == 0) x[i] = VT<T>::one();      // (pk_flag)
            }
            if (i < sd && c < sd) o[pk_e(i, c, sd)] = x[i];
        }
    }
    const int rl = (int)F.l_rows - k0 - w;
    for (int c = warp; c < 16; c += 4) {
        const bool in = c < w;
        const T *src = L + (int64_t)(k0 + (in ? c : 0)) * F.nr;
        for (int r = lane; r < k0; r += 32) du[256 + c * k0 + r] = in ? src[r] : VT<T>::zero();
        for (int r = lane; r < rl; r += 32) dl[256 + c * rl + r] = in ? src[k0 + w + r] : VT<T>::zero();
    }
}

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(unsigned long long *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// a bulk copy of `bytes` (a multiple of 16; both addresses 16-byte aligned) that completes on `bar`
__device__ __forceinline__ void bulk_expect(unsigned long long *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned long long *bar, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// waits for the phase; false when the wait ran out of time
__device__ __forceinline__ bool bar_wait(unsigned long long *bar, unsigned parity)
{
    if (bar_try(bar, parity)) return true;
    const long long t0 = clock64();
    while (!bar_try(bar, parity))
        if (clock64() - t0 > CH_CYCLES) return false;
    return true;
}

__device__ __forceinline__ void st_release_u32(unsigned *p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// arrive at a named barrier without waiting
__device__ __forceinline__ void named_arrive(int id, int count) { asm volatile("barrier.arrive %0, %1;" ::"r"(id), "r"(count) : "memory"); }
// one thread waits until *p >= v; false when the wait ran out.  It polls with relaxed loads (an acquiring load each time
// invalidates the SM's L1, which slowed the other warps' products threefold) and acquires once
__device__ __forceinline__ bool chain_wait(const unsigned *p, unsigned v)
{
    for (unsigned k = 0; k < CH_SPIN; k++) {
        unsigned c;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(p) : "memory");
        if (c >= v) { (void)ld_acquire_u32(p); return true; }
        __nanosleep(20);
    }
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

// The sum over k < kn (a multiple of 16) of M(o, k) x[k * RB + r] by four lanes per output, each with four of every sixteen k,
// then summed over the four lanes.  The output o and the lane's share q of thread tid (a warp: eight outputs, lane = o + 8 q,
// so that the eight lanes of a shared-memory phase read eight neighbouring elements: with the shares in neighbouring lanes a
// 64 x 64 product took 2,700 cycles).  M(o, k) = Mp[k * ld + o] (plain), or op(Mp[o * ld + k]) (transposed; neighbouring
// outputs start one apart)
__device__ __forceinline__ int quad_o(int tid) { return (tid & 7) + 8 * (tid >> 5); }
__device__ __forceinline__ int quad_q(int tid) { return (tid >> 3) & 3; }
template <typename T, int RB> __device__ __forceinline__ void quad_sum(T (&acc)[RB])
{
#pragma unroll
    for (int r = 0; r < RB; r++) {
        acc[r] = add(acc[r], shfl_xor_v<T>(acc[r], 8));
        acc[r] = add(acc[r], shfl_xor_v<T>(acc[r], 16));
    }
}
template <typename T, int TR, int RB>
__device__ __forceinline__ void quad_mv(T (&acc)[RB], const T *Mp, int ld, int o, int q, int kn, const T *x)
{
#pragma unroll
    for (int r = 0; r < RB; r++) acc[r] = VT<T>::zero();
    const T *m = TR == 0 ? Mp + q * ld + o : Mp + o * ld;
    const int ms = 4 * ld;
    for (int e = 0; e < kn; e += 16) {
        T v[4];
        int k[4];
#pragma unroll
        for (int z = 0; z < 4; z++) {
            k[z] = TR == 0 ? e + q + 4 * z : e + ((4 * q + z + o) & 15);
            v[z] = TR == 0 ? m[z * ms] : opv<TR>(m[k[z]]);
        }
        if (TR == 0) m += 4 * ms;
#pragma unroll
        for (int z = 0; z < 4; z++)
#pragma unroll
            for (int r = 0; r < RB; r++) acc[r] = madd<T>(acc[r], v[z], x[k[z] * RB + r]);
    }
    quad_sum<T, RB>(acc);
}

// x = M^-1 y for a packed 16 x 16 diagonal block D of w <= 16 unknowns: M = L (unit lower) or U (TR 0), or its transpose (TR 1, 2
// with conj); BACK: M is upper triangular; UNIT: it has a unit diagonal; sd: the block's side (w <= sd).  y: [k * RB + r], finite
// or not, from w on zero or not part of the block.  By the threads tid < diag_threads(RB); put(o, r, x) takes unknown o < 16 of right-hand side r, zero from
// w on (INPLACE: after every thread has read y; named barrier 2).
//
// What bounds it (B200, one right-hand side, from y in shared memory to x there, two barriers included): the product 373
// cycles real, 481 complex (263 and 461 without the flag and the terms left out; 1,238 and 1,066 with 8 and 4 right-hand
// sides); the substitution, a lane per unknown and one exchange per step, 970 (unit) and 1,480 real, 1,630 and 1,890 complex (a dependent FP64 operation takes about 25 cycles, a shuffle 27).  Four unknowns at a time, solved by every
// lane for itself, took 1,180 to 1,200 real and 1,780 to 1,890 complex; the whole block in one lane 960 to 3,080.
__host__ __device__ constexpr int sub_warps(int rb) { return (rb + 1) / 2; }
__host__ __device__ constexpr int diag_threads(int rb) { return 32 * sub_warps(rb) > 64 ? 32 * sub_warps(rb) : 64; }
__device__ __forceinline__ double shfl16_v(double v, int src) { return __shfl_sync(0xffffffffu, v, src, 16); }
__device__ __forceinline__ cplx shfl16_v(cplx v, int src) { return cplx{shfl16_v(v.x, src), shfl16_v(v.y, src)}; }
// the substitution (its own function: the product's path keeps the registers): unknown o = tid % 16 of two right-hand sides
// per warp
template <typename T, int TR, bool BACK, bool UNIT, int RB>
__device__ __noinline__ T diag_sub(const T *D, int sd, int w, const T *y)
{
    auto at = [&](int i, int k) -> T { return i < sd && k < sd ? (TR == 0 ? D[pk_e(i, k, sd)] : opv<TR>(D[pk_e(k, i, sd)])) : VT<T>::zero(); };
    const int o = threadIdx.x & 15, r = RB == 1 ? 0 : 2 * (threadIdx.x >> 5) + ((threadIdx.x >> 4) & 1);
    T a = o < w ? y[o * RB + r] : VT<T>::zero();
    const T inv = UNIT ? VT<T>::one() : at(o, o);
#pragma unroll
    for (int s = 0; s < 16; s++) {
        const int k = BACK ? 15 - s : s;
        const T x = UNIT ? a : mul(a, inv), v = shfl16_v(x, k), u = msub(a, at(o, k), v);
        a = o == k ? x : (BACK ? o < k : o > k) ? u : a;
    }
    return o < w ? a : VT<T>::zero();
}
template <typename T, int TR, bool BACK, bool UNIT, int RB, bool INPLACE, typename PUT>
__device__ __forceinline__ void diag_solve(const T *D, int sd, int w, const T *y, PUT put)
{
    const int tid = threadIdx.x;
    if (is_zero(D[pk_flag((TR == 0) != BACK, sd)])) {
        if (tid >= 64) return;
        // four lanes per unknown; the terms outside the triangle are left out, not multiplied by zero (an infinity in y
        // reaches the unknowns that depend on it, as in a substitution)
        const int o = quad_o(tid), q = quad_q(tid);
        T a[RB];
#pragma unroll
        for (int r = 0; r < RB; r++) a[r] = VT<T>::zero();
#pragma unroll
        for (int z = 0; z < 4; z++) {
            const int k = 8 * (q & 1) + 4 * (q >> 1) + z;         // (no bank conflicts in either order)
            const bool in = BACK ? k >= o && k < w : k <= o && o < w;
            const T m = o >= sd || k >= sd ? VT<T>::zero() : TR == 0 ? D[pk_e(o, k, sd)] : opv<TR>(D[pk_e(k, o, sd)]);
#pragma unroll
            for (int r = 0; r < RB; r++) a[r] = madd<T>(a[r], m, in ? y[k * RB + r] : VT<T>::zero());
        }
        quad_sum<T, RB>(a);
        if (INPLACE) named_bar(2, 64);
        if (q == 0)
#pragma unroll
            for (int r = 0; r < RB; r++) put(o, r, o < w ? a[r] : VT<T>::zero());
        return;
    }
    if (tid >= 32 * sub_warps(RB)) return;
    const T x = diag_sub<T, TR, BACK, UNIT, RB>(D, sd, w, y);
    if (RB > 1 || tid < 16) put(tid & 15, RB == 1 ? 0 : 2 * (tid >> 5) + ((tid >> 4) & 1), x);
}

// right-hand sides per pass of the multiple-right-hand-side forms
template <typename T> __host__ __device__ constexpr int ch_rb() { return VT<T>::cplx_ ? 4 : 8; }
// dynamic shared memory of k_chain_u for `own` blocks' sums per worker (the larger of the two roles)
static inline size_t chain_u_smem(int64_t own, int64_t rb, int64_t vs)
{
    const size_t worker = (size_t)(CH_STAGES * CH_BLK + CH_NB * rb * (1 + own)) * vs;
    const size_t solver = (size_t)(2 * CH_BLK + 2 * 2560 + 4 * CH_NB * rb) * vs;
    return worker > solver ? worker : solver;
}

// x = U11^-1 y (TR 0) or U11^-T y of one chain front (np pivots) from its packed pieces tr, by CH_THREADS threads (o, q: quad_o,
// quad_q; ys and x: [k * RB + r], zero beyond the pivots; ys is overwritten); ends without a barrier after the last writes of x but
// the named barrier 1 of its steps
template <typename T, int TR, int RB>
__device__ __forceinline__ void chain_tri(const T *tr, T *ys, T *x, int np, int o, int q)
{
    const int nbk = (np + 15) >> 4;
    T a[RB];
    for (int bb = 0; bb < nbk; bb++) {
        const int b = TR == 0 ? nbk - 1 - bb : bb, k0 = 16 * b;
        const T *D = tr + pk_u(b), *pan = D + 256;         // (16 columns, leading dimension k0)
        if (TR != 0 && b > 0) {
            // w_b -= U[0 .. 16b, b]^T z
            if (o < 16) {
                quad_mv<T, TR, RB>(a, pan, k0, o, q, k0, x);
                if (q == 0)
#pragma unroll
                    for (int r = 0; r < RB; r++) ys[(k0 + o) * RB + r] = sub(ys[(k0 + o) * RB + r], a[r]);
            }
            named_bar(1, CH_THREADS);
        }
        if (threadIdx.x < diag_threads(RB))
            diag_solve<T, TR, TR == 0, false, RB, false>(D, 16, np - k0 < 16 ? np - k0 : 16, ys + k0 * RB,
                                                         [&](int i, int r, T v) { x[(k0 + i) * RB + r] = v; });
        named_bar(1, CH_THREADS);
        if (TR == 0 && b > 0) {
            // y[0 .. 16b) -= U[0 .. 16b, b] x_b
            if (o < k0) {
                quad_mv<T, 0, RB>(a, pan, k0, o, q, 16, x + k0 * RB);
                if (q == 0)
#pragma unroll
                    for (int r = 0; r < RB; r++) ys[o * RB + r] = sub(ys[o * RB + r], a[r]);
            }
            named_bar(1, CH_THREADS);
        }
    }
}

// the product of a 64 x 64 block with the kn values of xs (quad_mv, the last front's odd lengths included); oo: this
// thread's output, or 0 beyond the outputs
template <typename T, int TR, int RB>
__device__ __forceinline__ void block_mv(T (&a)[RB], const T *M, int nb, int oo, int q, int kn, const T *xs)
{
    if ((kn & 15) == 0) { quad_mv<T, TR, RB>(a, M, nb, oo, q, kn, xs); return; }
#pragma unroll
    for (int r = 0; r < RB; r++) a[r] = VT<T>::zero();
    for (int k = q; k < kn; k += 4) {
        const T m = TR == 0 ? M[k * nb + oo] : opv<TR>(M[oo * nb + k]);
#pragma unroll
        for (int r = 0; r < RB; r++) a[r] = madd<T>(a[r], m, xs[k * RB + r]);
    }
    quad_sum<T, RB>(a);
}

// t = 0 .. K - 1: the blocks in solve order (TR 0: front K - 1 - t, else front t); front k's pivots are [f0 + k nb, ..) and
// its U12 starts at U0 + sum of the fronts' before it.  Y: the right-hand sides (pivot order, overwritten), X: the
// solution; both n x nrhs.  sync[0]: blocks solved; sync[1 + t]: block t has every product but that of block t - 1.
// rb <= RB right-hand sides.
//
// What bounds it: at small K the solver's step (the 64 x 64 product with the block just solved, then four 16 x 16
// solves and their updates) and the round trip solver - worker - solver; at large K the stream of U12.
template <typename T, int TR, int RB>
__global__ void __launch_bounds__(CH_UTHREADS) k_chain_u(const ChainFront *__restrict__ fr, int K, int nb, int64_t f0, int64_t U0,
                                                         int np_last, const T *__restrict__ Ua, const T *__restrict__ pk, T *Y, T *X,
                                                         int64_t n, int rb, unsigned *sync, T *gacc, DevStatus *st)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned long long bars[CH_STAGES];
    __shared__ int s_ok;
    const int tid = threadIdx.x, o = quad_o(tid), q = quad_q(tid);
    auto front_of = [&](int t) -> int { return TR == 0 ? K - 1 - t : t; };
    auto np_of = [&](int t) -> int { return front_of(t) == K - 1 ? np_last : nb; };
    auto f_of = [&](int t) -> int64_t { return f0 + (int64_t)front_of(t) * nb; };
    // the block of U12 that couples block t to block s < t in solve order (rows of front a, columns of front c > a); where
    // its start is not 16-byte aligned the copy takes one element more before and after it, and sh is 1
    const int sh = VT<T>::cplx_ ? 0 : (int)(U0 & 1);
    auto load_block = [&](T *dst, int t, int s, unsigned long long *bar) {
        const int a = TR == 0 ? front_of(t) : front_of(s), c = TR == 0 ? front_of(s) : front_of(t);
        const int64_t off = U0 + (int64_t)nb * ((int64_t)a * (n - f0) - (int64_t)nb * a * (a + 1) / 2) + (int64_t)(c - a - 1) * nb * nb;
        const int cnt = nb * (c == K - 1 ? np_last : nb);
        // (an odd count of 8-byte elements, in the last front only, is rounded up: the arena has room behind it)
        const unsigned bytes = (unsigned)((((size_t)(cnt + 2 * sh) * sizeof(T)) + 15) & ~(size_t)15);
        bulk_expect(bar, bytes);
        bulk_load(dst, Ua + off - sh, bytes, bar);
    };
    if (tid == 0) {
        s_ok = st->code == 0;
        for (int k = 0; k < CH_STAGES; k++) bar_init(bars + k, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (!*(volatile int *)&s_ok) return;
    if (blockIdx.x > 0) {
        if (tid >= CH_THREADS) return;                 // (the solver's helper warps)
        // a worker: owns the blocks t = w, w + W, .. (w = blockIdx.x - 1)
        const int w = blockIdx.x - 1, W = gridDim.x - 1;
        T *ring = reinterpret_cast<T *>(smem_raw);
        T *xs = ring + CH_STAGES * CH_BLK;             // x of the block being subtracted: xs[k * RB + r]
        // owned block j's sums, in shared memory (after x), or in global memory (gacc, block t's at t): [o * RB + r] from
        // acc + j * ajs on; each entry is its thread's own
        const int own = w < K ? (K - 1 - w) / W + 1 : 0;
        T *acc = gacc ? gacc + (int64_t)w * CH_NB * RB : xs + CH_NB * RB;
        const int64_t ajs = (gacc ? (int64_t)W : 1) * CH_NB * RB;
        if (q == 0) for (int j = 0; j < own; j++)
#pragma unroll
            for (int r = 0; r < RB; r++) acc[j * ajs + o * RB + r] = VT<T>::zero();
        for (int e = tid; e < RB * CH_NB; e += CH_THREADS) xs[e] = VT<T>::zero();
        // tasks in order: s ascending, the owned t >= s + 2 ascending (t = w + j W, j from j0(s))
        auto first_j = [&](int s) -> int { const int m = s + 2 - w; return m <= 0 ? 0 : (m + W - 1) / W; };
        int ps = 0, pj = first_j(0), cs, cj, issued = 0, done = 0;
        while (ps <= K - 3 && pj >= own) { ps++; pj = first_j(ps); }
        cs = ps; cj = pj;
        auto load_next = [&]() {                       // one thread
            if (ps <= K - 3) {
                load_block(ring + (issued % CH_STAGES) * CH_BLK, w + pj * W, ps, bars + issued % CH_STAGES);
                issued++;
                pj++;
                while (ps <= K - 3 && pj >= own) { ps++; pj = first_j(ps); }
            }
        };
        if (tid == CH_THREADS - 1) for (int k = 0; k < CH_STAGES; k++) load_next();
        int have = -1;
        while (cs <= K - 3) {
            if (have != cs) {                          // a new solved block: wait for it, its x into shared memory
                if (tid == 0 && !chain_wait(sync, (unsigned)cs + 1u)) s_ok = 0;
                named_bar(1, CH_THREADS);
                const int64_t f = f_of(cs);
                const int np = np_of(cs);
                if (*(volatile int *)&s_ok)
                    for (int e = tid; e < CH_NB * rb; e += CH_THREADS) {
                        const int k = e & (CH_NB - 1), r = e / CH_NB;
                        xs[k * RB + r] = k < np ? ldcg_v(X + f + k + r * n) : VT<T>::zero();
                    }
                have = cs;
                named_bar(1, CH_THREADS);
            }
            const int slot = done % CH_STAGES, ct = w + cj * W;
            if (!bar_wait(bars + slot, (unsigned)(done / CH_STAGES) & 1u)) s_ok = 0;
            const int no = TR == 0 ? nb : np_of(ct);
            // (the inner length in whole sixteens: x is zero beyond the block; nb is one, and so are U12's columns but in the
            // last front, whose block's copy may hold less: those columns are not read)
            const int kn = TR == 0 ? np_of(cs) : nb;
            T a[RB];
            const T *M = ring + slot * CH_BLK + sh;
            block_mv<T, TR, RB>(a, M, nb, o < no ? o : 0, q, kn, xs);
            T *ao = acc + cj * ajs + o * RB;
            const bool last = cs == ct - 2;            // the last product this worker takes for block ct
            if (q == 0 && o < no) {
#pragma unroll
                for (int r = 0; r < RB; r++) a[r] = add(ao[r], a[r]);
                if (last) {
                    T *y = Y + f_of(ct) + o;
#pragma unroll
                    for (int r = 0; r < RB; r++) if (r < rb) y[r * n] = sub(y[r * n], a[r]);
                    __threadfence();
                } else {
#pragma unroll
                    for (int r = 0; r < RB; r++) ao[r] = a[r];
                }
            }
            named_bar(1, CH_THREADS);                  // the stage is free, the sums are out
            if (!*(volatile int *)&s_ok) { if (tid == 0) set_status(st, ST_WAIT, cs, 0, 0); break; }
            if (last && tid == 0) st_release_u32(sync + 1 + ct, 1u);
            if (tid == CH_THREADS - 1) load_next();
            done++;
            cj++;
            while (cs <= K - 3 && cj >= own) { cs++; cj = first_j(cs); }
        }
        // the copies in flight (after a wait that ran out)
        if (tid == CH_THREADS - 1) for (; done < issued; done++) (void)bar_wait(bars + done % CH_STAGES, (unsigned)(done / CH_STAGES) & 1u);
        return;
    }
    // the solver: 256 threads on the critical path and two helper warps, one that waits for the workers' part of the next
    // block's right-hand side and brings it in, one that publishes the solved block (the stores, the fence, the counter)
    T *off = reinterpret_cast<T *>(smem_raw);          // two stages: the block coupling t to t - 1
    T *tri = off + 2 * CH_BLK;                         // two stages: the front's packed U pieces
    T *yin = tri + 2 * 2560, *xs = yin + 2 * CH_NB * RB;       // right-hand sides and solutions, two blocks each in turn: [k * RB + r]
    for (int e = tid; e < 4 * CH_NB * RB; e += CH_UTHREADS) yin[e] = VT<T>::zero();
    __syncthreads();
    if (tid >= CH_THREADS) {
        const int lane = tid & 31;
        if (tid < CH_THREADS + 32) {                   // right-hand sides in
            for (int t = 0; t < K; t++) {
                const int np = np_of(t);
                int ok = 1;
                if (t >= 2 && lane == 0) ok = chain_wait(sync + 1 + t, 1u);
                ok = __shfl_sync(0xffffffffu, ok, 0);
                const int64_t f = f_of(t);
                if (ok) for (int e = lane; e < CH_NB * rb; e += 32) {
                    const int p = e & (CH_NB - 1), r = e / CH_NB;
                    yin[((t & 1) * CH_NB + p) * RB + r] = p < np ? ldcg_v(Y + f + p + r * n) : VT<T>::zero();
                }
                else if (lane == 0) { set_status(st, ST_WAIT, t, 0, 0); s_ok = 0; }
                __syncwarp();
                named_bar(3, CH_THREADS + 32);         // block t's right-hand side is in
                if (!*(volatile int *)&s_ok) return;
            }
        } else {                                       // solved blocks out
            for (int t = 0; t < K; t++) {
                named_bar(4 + (t & 1), CH_THREADS + 32);       // block t is solved (or a wait ran out)
                if (!*(volatile int *)&s_ok) return;
                const int np = np_of(t);
                const int64_t f = f_of(t);
                for (int e = lane; e < np * rb; e += 32) { const int p = e % np, r = e / np; X[f + p + r * n] = xs[((t & 1) * CH_NB + p) * RB + r]; }
                __threadfence();
                __syncwarp();
                if (lane == 0) st_release_u32(sync, (unsigned)t + 1u);
            }
        }
        return;
    }
    long long upk = tid == CH_THREADS - 1 ? fr[front_of(0)].u_pk : 0;      // the loading thread: the next block's packed pieces
    auto load = [&](int t) {
        if (t < K) {
            const int sl = t & 1, np = np_of(t);
            unsigned long long *bar = bars + sl;
            const unsigned bytes = (unsigned)(pk_u((np + 15) >> 4) * sizeof(T));
            if (t > 0) {
                const int s = t - 1, a = TR == 0 ? front_of(t) : front_of(s), c = TR == 0 ? front_of(s) : front_of(t);
                const int64_t uo = U0 + (int64_t)nb * ((int64_t)a * (n - f0) - (int64_t)nb * a * (a + 1) / 2);
                const unsigned ub = (unsigned)((((size_t)(nb * (c == K - 1 ? np_last : nb) + 2 * sh) * sizeof(T)) + 15) & ~(size_t)15);
                bulk_expect(bar, bytes + ub);
                bulk_load(off + sl * CH_BLK, Ua + uo - sh, ub, bar);
            } else bulk_expect(bar, bytes);
            bulk_load(tri + sl * 2560, pk + upk, bytes, bar);
            if (t + 1 < K) upk = fr[front_of(t + 1)].u_pk;
        }
    };
    if (tid == CH_THREADS - 1) load(0);
    for (int t = 0; t < K; t++) {
        const int sl = t & 1, np = np_of(t);
        T *ys = yin + sl * CH_NB * RB, *x = xs + sl * CH_NB * RB;
        const T *xp = xs + (sl ^ 1) * CH_NB * RB;
        if (tid == CH_THREADS - 1) load(t + 1);        // (into the stage that block t - 1 used: everyone is past it)
        if (!bar_wait(bars + sl, (unsigned)(t >> 1) & 1u)) { set_status(st, ST_WAIT, t, 0, 0); s_ok = 0; }
        named_bar(3, CH_THREADS + 32);                 // the copies, and the right-hand side
        if (!*(volatile int *)&s_ok) {
            // (the copies in flight land first)
            if (tid == CH_THREADS - 1) { (void)bar_wait(bars + sl, (unsigned)(t >> 1) & 1u); if (t + 1 < K) (void)bar_wait(bars + (sl ^ 1), (unsigned)((t + 1) >> 1) & 1u); }
            named_bar(4 + (t & 1), CH_THREADS + 32);
            break;
        }
        T a[RB];
        if (t > 0) {
            const int kn = np_of(t - 1);
            const T *M = off + sl * CH_BLK + sh;
            block_mv<T, TR, RB>(a, M, nb, o < np ? o : 0, q, kn, xp);
            if (q == 0 && o < np)
#pragma unroll
                for (int r = 0; r < RB; r++) ys[o * RB + r] = sub(ys[o * RB + r], a[r]);
        }
        named_bar(1, CH_THREADS);
        chain_tri<T, TR, RB>(tri + sl * 2560, ys, x, np, o, q);
        named_arrive(4 + (t & 1), CH_THREADS + 32);    // x is in shared memory: out it goes (two barriers in turn: block t + 2
                                                       // cannot be done before block t is out)
    }
}

// One step of the same sweep as a launch of its own (s = -1 .. K - 2): CTA 0 solves block s + 1, the others add the product
// with block s to the sums of the blocks from s + 2 on (gacc: block t's at t CH_NB RB).  Every value is formed as k_chain_u
// forms it, so the results are the same bit for bit.  For captured graphs: a branch of a graph shares the SMs with the other
// matrices' branches, and a launch that needs several whole SMs at once holds those up.
static inline size_t chain_ustep_smem(int64_t rb, int64_t vs) { return (size_t)(CH_NB * CH_NB + 2560 + 3 * CH_NB * rb) * vs; }
template <typename T, int TR, int RB>
__global__ void __launch_bounds__(CH_THREADS) k_chain_ustep(const ChainFront *__restrict__ fr, int K, int nb, int64_t f0, int64_t U0,
                                                            int np_last, const T *__restrict__ Ua, const T *__restrict__ pk, T *Y, T *X,
                                                            int64_t n, int rb, int s, T *gacc, const DevStatus *st)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, o = quad_o(tid), q = quad_q(tid), t = s + 1 + blockIdx.x;
    T *M = reinterpret_cast<T *>(smem_raw), *tr = M + CH_NB * CH_NB, *xp = tr + 2560, *ys = xp + CH_NB * RB, *x = ys + CH_NB * RB;
    auto front_of = [&](int u) -> int { return TR == 0 ? K - 1 - u : u; };
    auto np_of = [&](int u) -> int { return front_of(u) == K - 1 ? np_last : nb; };
    auto f_of = [&](int u) -> int64_t { return f0 + (int64_t)front_of(u) * nb; };
    auto stage = [&](T *dst, const T *src, int cnt) {
        for (int e0 = tid; e0 < cnt; e0 += 16 * CH_THREADS) {
            T v[16];
#pragma unroll
            for (int z = 0; z < 16; z++) v[z] = e0 + z * CH_THREADS < cnt ? src[e0 + z * CH_THREADS] : VT<T>::zero();
#pragma unroll
            for (int z = 0; z < 16; z++) if (e0 + z * CH_THREADS < cnt) dst[e0 + z * CH_THREADS] = v[z];
        }
    };
    const int np = np_of(t);
    if (s >= 0) {                                      // (the factors do not change during the solve: before the wait)
        const int a = TR == 0 ? front_of(t) : front_of(s), c = TR == 0 ? front_of(s) : front_of(t);
        stage(M, Ua + U0 + (int64_t)nb * ((int64_t)a * (n - f0) - (int64_t)nb * a * (a + 1) / 2) + (int64_t)(c - a - 1) * nb * nb,
              nb * (c == K - 1 ? np_last : nb));
    }
    if (blockIdx.x == 0) stage(tr, pk + fr[front_of(t)].u_pk, (int)pk_u((np + 15) >> 4));
    pdl_wait();
    pdl_trigger();
    if (st->code) return;
    for (int e = tid; e < CH_NB * RB; e += CH_THREADS) {
        const int k = e & (CH_NB - 1), r = e / CH_NB;
        xp[k * RB + r] = s >= 0 && r < rb && k < np_of(s) ? ldcg_v(X + f_of(s) + k + r * n) : VT<T>::zero();
        if (blockIdx.x == 0) {
            ys[k * RB + r] = r < rb && k < np ? ldcg_v(Y + f_of(t) + k + r * n) : VT<T>::zero();
            x[k * RB + r] = VT<T>::zero();
        }
    }
    __syncthreads();
    T a[RB];
    if (s >= 0) {
        const int no = TR == 0 ? (blockIdx.x == 0 ? np : nb) : np, kn = blockIdx.x == 0 ? np_of(s) : TR == 0 ? np_of(s) : nb;
        block_mv<T, TR, RB>(a, M, nb, o < no ? o : 0, q, kn, xp);
        if (q == 0 && o < no) {
            if (blockIdx.x == 0) {
#pragma unroll
                for (int r = 0; r < RB; r++) ys[o * RB + r] = sub(ys[o * RB + r], a[r]);
            } else {
                T *ao = gacc + ((int64_t)t * CH_NB + o) * RB;
#pragma unroll
                for (int r = 0; r < RB; r++) a[r] = add(s > 0 ? ao[r] : VT<T>::zero(), a[r]);
                if (s == t - 2) {
#pragma unroll
                    for (int r = 0; r < RB; r++) if (r < rb) { T *y = Y + f_of(t) + o + r * n; *y = sub(*y, a[r]); }
                } else {
#pragma unroll
                    for (int r = 0; r < RB; r++) ao[r] = a[r];
                }
            }
        }
    }
    if (blockIdx.x > 0) return;
    __syncthreads();
    chain_tri<T, TR, RB>(tr, ys, x, np, o, q);
    __syncthreads();
    for (int e = tid; e < np * rb; e += CH_THREADS) { const int k = e % np, r = e / np; X[f_of(t) + k + r * n] = x[k * RB + r]; }
}

// dynamic shared memory of k_chain_l: CH_LSTAGES packed pieces, two row vectors
constexpr int CH_LSTAGES = 4;
__host__ __device__ constexpr int ch_lpiece(int maxnr) { return 256 + 16 * maxnr; }
static inline size_t chain_l_smem(int64_t maxnr, int64_t rb, int64_t vs)
{
    return (size_t)(CH_LSTAGES * ch_lpiece((int)maxnr) + 2 * (maxnr + 16) * rb) * vs;
}

// The L sweep (TR 0: v0 = the first front's gathered vector in its final row order, VB; later fronts' entering rows from R
// in row space; y into S2 in pivot order) or the L^T sweep (TR 1, 2: z = R in pivot order; x into S2).  blockIdx.x: the
// group of RB right-hand sides.
template <typename T, int TR, int RB>
__global__ void __launch_bounds__(CH_THREADS) k_chain_l(const ChainFront *__restrict__ fr, int K, int maxnr, const T *__restrict__ pk,
                                                        const int *__restrict__ permall, const int64_t *__restrict__ rowinit,
                                                        const T *__restrict__ VB0, int64_t vstride, const T *__restrict__ R,
                                                        T *__restrict__ S2, int64_t n, int nrhs, DevStatus *st)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned long long bars[CH_LSTAGES];
    __shared__ int s_ok;
    const int tid = threadIdx.x;
    const int r0 = blockIdx.x * RB, rb = nrhs - r0 < RB ? nrhs - r0 : RB;
    const int psz = ch_lpiece(maxnr), vld = maxnr + 16;
    T *ring = reinterpret_cast<T *>(smem_raw);
    T *v = ring + CH_LSTAGES * psz, *vn = v + vld * RB;        // the front's row vector: v[pos * RB + r]
    R += (int64_t)r0 * n; S2 += (int64_t)r0 * n; VB0 += (int64_t)r0 * vstride;
    if (tid == 0) {
        s_ok = st->code == 0;
        for (int k = 0; k < CH_LSTAGES; k++) bar_init(bars + k, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int e = tid; e < 2 * vld * RB; e += CH_THREADS) v[e] = VT<T>::zero();
    __syncthreads();
    if (!*(volatile int *)&s_ok) return;
    // the pieces in order: TR 0: fronts and blocks ascending, else descending (the loading thread; the front after the
    // one being loaded is read ahead)
    const bool loader = tid == CH_THREADS - 1;
    const int step = TR == 0 ? 1 : -1;
    int pkf = TR == 0 ? 0 : K - 1, issued = 0;
    ChainFront PF = fr[pkf], PN = fr[K > 1 ? pkf + step : pkf];
    int pb = TR == 0 ? 0 : ((int)PF.np + 15) / 16 - 1;
    auto load_next = [&]() {
        if (pkf < 0 || pkf >= K) return;
        const int np = (int)PF.np, k0 = 16 * pb, w = np - k0 < 16 ? np - k0 : 16;
        const unsigned bytes = (unsigned)((256 + 16 * ((int)PF.nr - k0 - w)) * sizeof(T));
        unsigned long long *bar = bars + issued % CH_LSTAGES;
        bulk_expect(bar, bytes);
        bulk_load(ring + (issued % CH_LSTAGES) * psz, pk + PF.l_pk + pk_l(pb, PF.nr), bytes, bar);
        issued++;
        const bool end = TR == 0 ? k0 + 16 >= np : pb == 0;
        if (!end) { pb += step; return; }
        pkf += step;
        PF = PN;
        pb = TR == 0 ? 0 : ((int)PF.np + 15) / 16 - 1;
        if (pkf + step >= 0 && pkf + step < K) PN = fr[pkf + step];
    };
    if (loader) for (int k = 0; k < CH_LSTAGES - 1; k++) load_next();
    ChainFront F = fr[TR == 0 ? 0 : K - 1];
    {
        const int m = TR == 0 ? (int)F.nr : (int)F.np;
        for (int e = tid; e < m * rb; e += CH_THREADS) { const int p = e % m, r = e / m; v[p * RB + r] = TR == 0 ? VB0[p + r * vstride] : R[F.f + p + r * n]; }
    }
    int done = 0;
    for (int kk = 0; kk < K; kk++) {
        const int k = TR == 0 ? kk : K - 1 - kk;
        const int np = (int)F.np, nr = (int)F.nr, nbk = (np + 15) >> 4;
        const bool more = kk + 1 < K;
        const ChainFront N = fr[more ? k + step : k];  // the next front
        // G: the front whose rows enter from the one below it (the next one, TR 0; this one otherwise); this thread's row there
        const int gnr = TR == 0 ? (int)N.nr : nr, gsl = (int)(TR == 0 ? N.slot : F.slot), gns = (int)(TR == 0 ? N.nslot : F.nslot),
                  gta = (int)(TR == 0 ? N.tau : F.tau);
        const int64_t gro = TR == 0 ? N.row_off : F.row_off;
        int pm = more && tid < gnr ? permall[gro + tid] : -1, t = -1;
        int64_t g = -1;
        T ent[RB];
#pragma unroll
        for (int r = 0; r < RB; r++) ent[r] = VT<T>::zero();
        if (TR != 0 && more && tid < (int)N.np)
#pragma unroll
            for (int r = 0; r < RB; r++) if (r < rb) ent[r] = R[N.f + tid + r * n];
        for (int bb = 0; bb < nbk; bb++, done++) {
            const int b = TR == 0 ? bb : nbk - 1 - bb, k0 = 16 * b, w = np - k0 < 16 ? np - k0 : 16, rl = nr - k0 - w;
            if (!bar_wait(bars + done % CH_LSTAGES, (unsigned)(done / CH_LSTAGES) & 1u)) s_ok = 0;
            __syncthreads();                           // (the piece before is no longer read: its stage is the next to load)
            if (!*(volatile int *)&s_ok) {
                if (tid == 0) set_status(st, ST_WAIT, k, 0, 0);
                if (loader) for (; done < issued; done++) (void)bar_wait(bars + done % CH_LSTAGES, (unsigned)(done / CH_LSTAGES) & 1u);
                return;
            }
            const T *D = ring + (done % CH_LSTAGES) * psz, *Lp = D + 256;      // Lp[c * rl + (row - k0 - w)]
            if (TR == 0) {
                if (tid < diag_threads(RB))
                    diag_solve<T, 0, false, true, RB, true>(D, 16, w, v + k0 * RB, [&](int i, int r, T a) {
                        if (i < w) { v[(k0 + i) * RB + r] = a; if (r < rb) S2[F.f + k0 + i + r * n] = a; }
                    });
                else if (loader) load_next();
                // the next front's rows, a block step after the load each needs (so that none waits)
                if (bb == (nbk > 1 ? 1 : 0) && pm >= 0) {
                    t = pm >= gsl && pm < gsl + gns ? pm - gsl : pm >= gta ? gns + pm - gta : -1;
                    if (t < 0) g = rowinit[gro + pm];
                }
                if (bb == nbk - 1 && pm >= 0 && t < 0 && g >= 0)
#pragma unroll
                    for (int r = 0; r < RB; r++) if (r < rb) ent[r] = R[g + r * n];
                __syncthreads();
                // the rows below: two lanes per row, eight columns each
                for (int i0 = 0; i0 < rl; i0 += CH_THREADS / 2) {
                    const int i = i0 + (tid & 15) + 16 * (tid >> 5), h = (tid >> 4) & 1, ii = i < rl ? i : 0;
                    T s[RB];
#pragma unroll
                    for (int r = 0; r < RB; r++) s[r] = VT<T>::zero();
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        const T l = Lp[(2 * c + h) * rl + ii];
                        const T *xv = v + (k0 + (2 * c + h < w ? 2 * c + h : 0)) * RB;
#pragma unroll
                        for (int r = 0; r < RB; r++) s[r] = madd<T>(s[r], l, xv[r]);
                    }
#pragma unroll
                    for (int r = 0; r < RB; r++) {
                        s[r] = add(s[r], shfl_xor_v<T>(s[r], 16));
                        if (i < rl && h == 0) v[(k0 + w + i) * RB + r] = sub(v[(k0 + w + i) * RB + r], s[r]);
                    }
                }
            } else {
                if (loader) load_next();
                if (bb == (nbk > 1 ? 1 : 0) && pm >= 0) t = pm >= gsl && pm < gsl + gns ? pm - gsl : pm >= gta ? gns + pm - gta : -1;
                // s_b = z_b - L[rows below, b]^T x: sixteen lanes per column
                const int c = tid >> 4, l16 = tid & 15;
                T s[RB];
#pragma unroll
                for (int r = 0; r < RB; r++) s[r] = VT<T>::zero();
                for (int i = l16; i < rl; i += 16) {
                    const T l = opv<TR>(Lp[c * rl + i]);
#pragma unroll
                    for (int r = 0; r < RB; r++) s[r] = madd<T>(s[r], l, v[(k0 + w + i) * RB + r]);
                }
#pragma unroll
                for (int r = 0; r < RB; r++) {
#pragma unroll
                    for (int m = 8; m > 0; m >>= 1) s[r] = add(s[r], shfl_xor_v<T>(s[r], m));
                    if (c < w && l16 == 0) v[(k0 + c) * RB + r] = sub(v[(k0 + c) * RB + r], s[r]);
                }
                __syncthreads();
                if (tid < diag_threads(RB))
                    diag_solve<T, TR, true, true, RB, true>(D, 16, w, v + k0 * RB, [&](int i, int r, T a) {
                        if (i < w) { v[(k0 + i) * RB + r] = a; if (r < rb) S2[F.f + k0 + i + r * n] = a; }
                    });
            }
        }
        if (!more) break;
        // the next front's vector
        __syncthreads();
        if (TR == 0) {
            if (pm >= 0)
#pragma unroll
                for (int r = 0; r < RB; r++) vn[tid * RB + r] = t >= 0 ? v[(np + t) * RB + r] : ent[r];
        } else {
            if (t >= 0)
#pragma unroll
                for (int r = 0; r < RB; r++) vn[((int)N.np + t) * RB + r] = v[tid * RB + r];
            if (tid < (int)N.np)
#pragma unroll
                for (int r = 0; r < RB; r++) vn[tid * RB + r] = ent[r];
        }
        T *sw = v; v = vn; vn = sw;
        F = N;
        // (the next piece's barrier orders these writes before they are read)
    }
}

}  // namespace fpl
