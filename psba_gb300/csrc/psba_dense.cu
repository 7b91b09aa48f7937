// Dense FP64 reduced-camera solve on sm_103a.
//
// S (Np x Np, lower triangle, Np a multiple of TILE) is factored S = L L^T
// by one cooperative persistent kernel over TILE x TILE lower tiles.  CTA 0
// (the panel) walks the diagonal: it applies the last update to each
// diagonal tile, factors it (panel_factor, with the forward solve of rhs carried
// along) and forms the sub-diagonal tile below it, which it keeps for the
// next step.  The other CTAs (helpers) accumulate every other update
// (left-looking) and solve the remaining tiles against the diagonal
// inverses, in a fixed dependency order; waits are bounded spins on per-tile
// flags in global memory (acquire/release) or on the values themselves, sent
// with the launch's epoch (mail).  After the factor, the back
// solve L^T x = y runs on a thread-block cluster (k_tri_cluster).  On request
// one step of iterative refinement follows: r = b - S x in FP64 against a copy of S taken before
// the factor (k_refine_residual), then both triangular solves of r with the
// factor, added into x (the same kernels with their forward part on).
//
// This replaces the reference's explicit inverse (SPD_inv.cl: 3x3-block
// Cholesky chain, kern_trigMat_inv, kern_trigMat_mul, then matVec_mul) with
// two triangular solves.  The failure test is the reference's: a non-positive
// or non-finite pivot (SPD_inv.cl:66-107) sets status 1; every flag is still
// raised and waits for mail end at the status, so nothing waits forever.  A spin that runs out of its
// iteration budget sets status 2 and the kernel completes.
#include <cfloat>
#include <cooperative_groups.h>
#include <mutex>
#include <vector>

#include "psba_internal.h"

namespace psba {

namespace cg = cooperative_groups;

constexpr int T = TILE;
constexpr int TT = TILE * TILE;
// Launch shape (compile-time tuning knobs): threads per CTA, update steps
// staged per batch, and a cap on CTAs per SM (0: as many as fit).
#ifndef PSBA_CHOL_THREADS
#define PSBA_CHOL_THREADS 256
#endif
#ifndef PSBA_CHOL_BJ
#define PSBA_CHOL_BJ 8
#endif
#ifndef PSBA_CHOL_PER_SM
#define PSBA_CHOL_PER_SM 1  // the panel's FP64 chain runs alone on its SM
#endif
constexpr int CF_THREADS = PSBA_CHOL_THREADS;
// Polls per wait (each one L2 round trip; the default, 2^22, is a second or
// two) come from the launch: a handle can shorten the bound
// (psba_set_wait_limit).  Thread 0 of each CTA stores it here at entry.
__shared__ long long s_spin_limit;
constexpr int BJ = PSBA_CHOL_BJ;             // update steps staged per batch in a tile task
static_assert(BJ >= 5, "the panel keeps its tiles in the staging area");

__device__ __forceinline__ int ld_acquire(const int *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ int ld_relaxed(const int *p)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(int *p, int v)
{
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// One thread's wait for flag == epoch.  The polls are relaxed loads (an acquire
// a poll slows down the SM's other warps' loads) and the last one an acquire;
// the status word is looked at every 16 polls, so a poll is one L2 round trip.
// Returns false when the budget ran out or another task already reported a
// timeout.
__device__ __forceinline__ bool poll_flag(const int *flag, int epoch, int *status)
{
    const long long limit = s_spin_limit;
    for (long long it = 0; it < limit; ++it) {
        if (ld_relaxed(flag) == epoch && ld_acquire(flag) == epoch) return true;
        if ((it & 15) == 15 && ld_relaxed(status) == 2) break;
        __nanosleep(20);
    }
    atomicExch(status, 2);
    return false;
}

// Threads 0 and 32 wait for a flag each; the block then proceeds.
__device__ void block_wait(const int *fa, const int *fb, int epoch, int *status)
{
    if (threadIdx.x == 0) poll_flag(fa, epoch, status);
    if (threadIdx.x == 32) poll_flag(fb, epoch, status);
    __syncthreads();
}

// Mail.  What the chain of panel steps waits for goes from CTA to CTA as
// 16-byte packets, a value and the launch's epoch, each written and read whole
// (one 128-bit access).  A packet is its own flag: the reader polls the values
// themselves, so a hand-off is a store and a poll, ~1 us less than store, fence,
// flag, poll and load.  Per block column K: L_KK^-1 and PD(K) by lower triangle
// rows (PD's b behind it), L_{K+1,K}, SUB(K) and the pre-solve (K+2, K) by rows, y_K.
constexpr int TRI = T * (T + 1) / 2;
constexpr int ML_INV = 0, ML_PD = ML_INV + TRI, ML_SUBD = ML_PD + TRI + T, ML_SUB = ML_SUBD + TT, ML_PRE = ML_SUB + TT,
              ML_Y = ML_PRE + TT, ML_COLUMN = ML_Y + T;
static_assert(ML_COLUMN == CHOL_MAIL, "the packets of a block column");

__device__ __forceinline__ int tri_at(int r, int c) { return r * (r + 1) / 2 + c; }

// row and column of entry e of a lower triangle by rows
__device__ __forceinline__ void tri_of(int e, int &r, int &c)
{
    r = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
    while ((r + 1) * (r + 2) / 2 <= e) ++r;
    while (r * (r + 1) / 2 > e) --r;
    c = e - r * (r + 1) / 2;
}

__device__ __forceinline__ void mail_put(ulonglong2 *p, double v, int epoch)
{
    asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"((long long)epoch)
                 : "memory");
}

// The thread's n <= N packets p[0], p[stride], ...; waits for all.  False when the
// budget ran out, or another task failed or timed out.
template <int N>
__device__ __forceinline__ bool mail_get(const ulonglong2 *p, int stride, int n, double (&v)[N], int epoch, int *status)
{
    const long long limit = s_spin_limit;
    for (long long it = 0; it < limit; ++it) {
        bool ok = true;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            long long x = 0, tag = epoch;
            if (j < n)
                asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                             : "=l"(x), "=l"(tag)
                             : "l"(p + j * stride)
                             : "memory");
            v[j] = __longlong_as_double(x);
            ok = ok && tag == epoch;
        }
        if (ok) return true;
        if ((it & 15) == 15 && ld_relaxed(status) != 0) return false;
    }
    atomicCAS(status, 0, 2);
    return false;
}

__device__ __forceinline__ int tile_task(int I, int K, int nb)
{
    return K * nb - (K * (K - 1)) / 2 + (I - K);  // column-major over the lower triangle
}

__device__ __forceinline__ void load_tile(double (*dst)[T + 1], const double *S, int Np, int I, int K)
{
    for (int e = threadIdx.x; e < TT; e += CF_THREADS) {
        const int r = e / T, c = e % T;
        dst[r][c] = __ldcg(S + (size_t)(I * T + r) * Np + K * T + c);
    }
}

// ---------------------------------------------------------------------------
// Diagonal-tile factor and inverse.  An FP64 result is ready ~64 cycles after
// issue, so the time of a 16 x 16 tile is the number of dependent FP64 steps of
// its columns, and what stands between them.  A Gauss-Jordan elimination without
// division has two per column: with the pivot p_s, every entry (r, c) of a row
// r > s takes
//     q <- p_s q - a_rs o,   o = a_cs for c > s, x_sc for c < s,
// where a is what is left of the tile and x, in the places of the columns
// already eliminated, the rows of its unit factor's inverse (x_rs starts as
// -a_rs).  Row r of a carries the factor sigma_r = p_0 ... p_(r-1), x_rc the
// factor sigma_r / sigma_c, and at the end
//     L_rc = a_rc t_c,  (L^-1)_rc = x_rc sigma_c t_r,  t_c = 1 / sqrt(p_c sigma_c).
// The only square roots are the 16 of t, all at once.
// Range: rows and columns are first scaled by 2^-H_r, H_r = floor(log2(a_rr) / 2) of
// the tile before its last update, which puts the diagonal below 4, and every
// four columns all entries are scaled by the power of two that brings sigma
// back to one.  In between sigma grows to 2^30 at most, and four columns of
// pivots D_0 ... D_3 (scaled) shrink it to D_0^8 D_1^4 D_2^2 D_3: it takes four
// in a row below 2^-60, far under the rounding errors of the tile, to underflow,
// and the tile is then refused.
//
// Roles: warps 0-3 hold one entry of rows 4-15 a thread (and one sigma), warp 4
// those of rows 0-3, whose columns end early; they meet once a column.  Column
// s of all is in q[s]: a_is for i >= s, x_si for i < s, so that in the end
// everything is there.  Warp 5 takes b's update and y, warp 7 the step's fetches.
// Cycles a tile (N = 528): 1,850 for the last update (at the SM's FP64 rate: one
// warp instruction per ~19 cycles), 4,150 for 15 columns (277 each, of which
// the two FP64 steps ~150, the shared-memory round and the barrier ~90), 400 to
// the inverse but for t, and 1,800 for the sub-diagonal tile, beside which the
// roots (770 by themselves) are taken.  A panel step is 8,900 of these; with an
// LDL^T elimination, a reciprocal a column and the inverse behind it, the tile
// alone took 15,000.  What a column does not need is kept out of it: a branch
// costs ~30 cycles, a sign flip or a comparison in FP64 60.
// Beside the 16 entries, q[s] has sigma_s, a zero (sigma's a) and a place for the
// stores of threads that have nothing to publish: a store under a condition
// on row and column cost 170 cycles a column in branches.
constexpr int PF_SIGMA = T, PF_ZERO = T + 1, PF_NONE = T + 2, PF_ROW = T + 3;
struct PfWork {
    double (*q)[PF_ROW];  // (q[s][PF_ZERO] = 0 set by the caller)
    double *t;
};

// The entry of a thread of warps 0-4: row r, column c (row 0 takes no step).
// Warp 4 has three lanes an entry for the update; the first goes on with it.
struct PfEntry {
    int r, c;
    bool own;
};
__device__ __forceinline__ PfEntry pf_entry()
{
    const int tid = threadIdx.x, lane = tid & 31;
    PfEntry e{tid < 128 ? 4 : 0, tid < 128 ? tid : lane % 10, tid < 128 ? tid < 126 : lane < 10};
    for (; e.c > e.r; ++e.r) e.c -= e.r + 1;
    if (e.r >= T || tid >= 160) e.r = e.c = 0;
    return e;
}

// Named barriers.  The instructions count whole warps, so the warp's lanes come
// together first (roles split warps here, and a warp that arrives in two
// parts would be counted twice).
template <int ID, int N>
__device__ __forceinline__ void pf_bar()
{
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
template <int ID, int N>
__device__ __forceinline__ void pf_arrive()
{
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(N) : "memory");
}

// x 2^n by the exponent field: what would be subnormal is zero, what would
// overflow infinite; infinities and NaN stay
__device__ __forceinline__ double pf_ldexp(double x, int n)
{
    const int h = __double2hiint(x), e = (h >> 20) & 0x7ff, ne = e + n;
    if (e == 0x7ff) return x;
    if (e == 0 || ne <= 0) return 0.0;
    if (ne >= 0x7ff) return __hiloint2double((h & 0x80000000) | 0x7ff00000, 0);
    return __hiloint2double(h + (n << 20), __double2loint(x));
}

// The tile's scale H, by one warp
__device__ __forceinline__ void tile_exp(const double (*a)[T + 1], int *H)
{
    const int l = threadIdx.x & (T - 1);
    H[l] = (((__double2hiint(a[l][l]) >> 20) & 0x7ff) - 1023) >> 1;
}

// The same without a branch, and n in the exponent field's place
__device__ __forceinline__ double pf_shift(double x, int n)
{
    const int h = __double2hiint(x);
    const unsigned e = h & 0x7ff00000, ne = e + (unsigned)n;
    const bool in = ne - 1 < 0x7fefffffu && e != 0x7ff00000u, nan = e == 0x7ff00000u;
    const int edge = nan ? h : n > 0 && e != 0 ? (h & (int)0x80000000) | 0x7ff00000 : 0;
    return __hiloint2double(in && e != 0 ? h + n : edge, (in && e != 0) || nan ? __double2loint(x) : 0);
}

// Warps 0-6 (224 threads): the last update of the diagonal tile a and of b with
// the previous step's sub-diagonal tile lsub and y (first: none), then the
// elimination.  X gets the inverse but for t (rows r to be multiplied by t_r),
// w.q the rest.
__device__ __forceinline__ void panel_factor(const double (*a)[T + 1], const int *H, const double (*lsub)[T + 1], double *b,
                                             const double *y, bool first, double (*X)[T + 1], const PfWork &w,
                                             const PfEntry &e)
{
    static_assert(CF_THREADS == 256 && T == 16, "the factor is laid out for eight warps and 16 x 16 tiles");
    constexpr int NE = 160, NT = CF_THREADS - 32;  // threads of warps 0-4 and of warps 0-6
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp >= 5) {
        // b (warp 5, two lanes a row), when the columns leave the FP64 units room for it
        pf_bar<4, NT>();
        if (!first && warp == 5) {
            const int r = lane >> 1, k0 = lane & 1;
            double v = 0.0;
#pragma unroll
            for (int k = 0; k < T; k += 2) v = fma(lsub[r][k0 + k], y[k0 + k], v);
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            if (k0 == 0) b[r] -= v;
        }
        pf_bar<1, NT>();
        return;
    }
    int r = e.r, c = e.c;
    const bool own = e.own, sig = tid == 127;
    double q;
    if (warp < 4) {
        q = a[r][c];
        if (!first)
#pragma unroll
            for (int k = 0; k < T; ++k) q = fma(-lsub[r][k], lsub[c][k], q);
    } else {
        const int k0 = lane / 10;  // three lanes an entry
        double v = 0.0;
        if (!first && lane < 30)
#pragma unroll
            for (int k = 0; k < T; k += 3)
                if (k0 + k < T) v = fma(lsub[r][k0 + k], lsub[c][k0 + k], v);
        const double v1 = __shfl_down_sync(0xffffffffu, v, 10), v2 = __shfl_down_sync(0xffffffffu, v, 20);
        q = a[r][c] - (v + (v1 + v2));
        if (!own) r = c = 0;
    }
    q = pf_shift(q, -(H[r] + H[c]) * (1 << 20));
    if (sig) {
        c = PF_SIGMA;
        q = 1.0;
    }
    const int ra = sig ? PF_ZERO : r, to = sig ? PF_SIGMA : PF_NONE;
    w.q[0][own && c == 0 ? r : to] = q;
    const int steps = warp == 0 ? 8 : warp == 1 ? 11 : warp == 2 ? 14 : warp == 3 ? 15 : 3;  // the warp's last row
    pf_bar<2, NE>();
    const double *qs = w.q[0];
    double *qn = w.q[1];
#pragma unroll
    for (int g = -1; g < T - 1; g += 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int s = g + j;
            if (s < 0) continue;
            if (s < steps) {
                // (past its row's steps a thread goes on with values that nobody reads)
                const double p = qs[s], ar = qs[ra];
                const double f = fma(p, q, -(ar * qs[c]));  // (the smaller product is the rounded one)
                // a sign flip in FP64 arithmetic would be one more dependent step
                q = c == s ? __hiloint2double(__double2hiint(ar) ^ (int)0x80000000, __double2loint(ar)) : f;
                if (j == 3) {
                    const int e = (__double2hiint(p) & 0x7ff00000) + (__double2hiint(qs[PF_SIGMA]) & 0x7ff00000);
                    q = pf_shift(q, (2046 << 20) - e);
                }
                qn[c == s + 1 ? r : r == s + 1 ? c : to] = q;
            }
            qs += PF_ROW;
            qn += PF_ROW;
            pf_bar<2, NE>();
        }
        if (g == 7) pf_arrive<4, NT>();
    }
    if (own) {
        const double sc = w.q[c][PF_SIGMA];
        X[r][c] = pf_shift(r == c ? sc : w.q[r][c] * sc, -H[c] * (1 << 20));
    }
    pf_bar<1, NT>();
}

// y = L^-1 b by warp 5, two lanes a row
__device__ __forceinline__ void panel_y(const double (*X)[T + 1], const double *b, const double *t, double *y, double *yg,
                                        ulonglong2 *mail, int epoch)
{
    const int r = (threadIdx.x & 31) >> 1, k0 = threadIdx.x & 1;
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < T; k += 2) v = fma(k0 + k <= r ? X[r][k0 + k] : 0.0, b[k0 + k], v);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v *= t[r];
    if (k0 == 0) {
        y[r] = v;
        mail_put(mail + ML_Y + r, v, epoch);
        yg[r] = v;
    }
}

// Warps 4-6 after it, beside the others' sub-diagonal tile: t (warp 4), then the
// inverse, to the mail and Ig (lower triangle), and y (warp 5).  (The solves use
// the diagonal tiles' inverses only: L_II itself is not kept.)  True in warp 4
// when a pivot was not a positive normal number.  t is announced on barrier 5
// to warps 0-3 (if they wait).
struct PfOut {
    int r[2], c[2];  // the thread's entries of the triangle
};

__device__ __forceinline__ bool panel_finish(const double (*X)[T + 1], const int *H, const double *b, double *y, bool waited,
                                             double *Ig, double *yg, ulonglong2 *mail, int epoch,
                                             const PfWork &w, const PfOut &o)
{
    const int tid = threadIdx.x, lane = tid & 31;
    bool bad = false;
    if (tid < 160) {
        const int l = lane & (T - 1);
        const double p = w.q[l][l], sg = w.q[l][PF_SIGMA], d = p * sg;
        w.t[l] = rsqrt(d);
        if (waited) pf_arrive<5, 160>();
        // the pivot itself is p 2^2H / sigma
        bad = __any_sync(0xffffffffu,
                         !(p > 0.0 && d >= DBL_MIN && pf_ldexp(p, 2 * H[l]) >= DBL_MIN * sg && d <= DBL_MAX));
    }
    pf_bar<6, 96>();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int r = o.r[j], c = o.c[j];
        if (r >= T) continue;
        const double xr = X[r][c] * w.t[r];
        mail_put(mail + ML_INV + tri_at(r, c), xr, epoch);
        Ig[r * T + c] = xr;
    }
    if (tid >= 160 && tid < 192) panel_y(X, b, w.t, y, yg, mail, epoch);
    return bad;
}

// Dealt-out tile products.  A tile operation costs the largest number of
// FP64 instructions any thread of a warp runs, so the products below are
// spread evenly over the CTA.

// a[r][c] -= sum_k L[r][k] L[c][k] for c <= r and
// b[r] -= sum_k L[r][k] y[k]: the NE x T products (element, k) are cut into
// consecutive runs of PER, one per thread; a run spans at most NACC
// elements, whose partial sums go to part[NACC t ...].  Each element then
// subtracts its partial sums in k order.  The accumulator and operands of a
// product are picked by selects, so a warp issues one FMA per product.
struct LowerUpdate {
    static constexpr int NT = CF_THREADS;
    static constexpr int NTRI = T * (T + 1) / 2;
    static constexpr int NE = NTRI + T;
    static constexpr int PER = (NE * T + NT - 1) / NT;
    static constexpr int NACC = (T - 1 + PER + T - 1) / T;  // elements one run can touch
    static constexpr int PART = NACC * NT;                  // doubles of partial sums
};

__device__ void update_lower(double (*a)[T + 1], const double (*L)[T + 1], double *b, const double *y, double *part)
{
    constexpr int NT = CF_THREADS;
    using U = LowerUpdate;
    constexpr int NTRI = U::NTRI, NE = U::NE, PER = U::PER, NACC = U::NACC;
    auto sync = [] { __syncthreads(); };
    const int tid = threadIdx.x;
    const int f0 = tid * PER, e0 = f0 / T;
    const double *xs[NACC], *ys[NACC];
    double p[NACC];
#pragma unroll
    for (int j = 0; j < NACC; ++j) {
        const int ej = min(e0 + j, NE - 1);
        int r, c;
        if (ej < NTRI) {
            tri_of(ej, r, c);
            xs[j] = L[r];
            ys[j] = L[c];
        } else {
            xs[j] = L[ej - NTRI];
            ys[j] = y;
        }
        p[j] = 0.0;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int f = f0 + i;
        const int k = f % T, idx = f / T - e0;
        const bool valid = f < NE * T;
        const double *xp = xs[0], *yp = ys[0];
        double acc = p[0];
#pragma unroll
        for (int j = 1; j < NACC; ++j) {
            xp = idx == j ? xs[j] : xp;
            yp = idx == j ? ys[j] : yp;
            acc = idx == j ? p[j] : acc;
        }
        const double v = fma(valid ? xp[k] : 0.0, valid ? yp[k] : 0.0, acc);
#pragma unroll
        for (int j = 0; j < NACC; ++j) p[j] = idx == j ? v : p[j];
    }
#pragma unroll
    for (int j = 0; j < NACC; ++j) part[NACC * tid + j] = p[j];
    sync();
    for (int e2 = tid; e2 < NE; e2 += NT) {
        const int tlo = (e2 * T) / PER, thi = (e2 * T + T - 1) / PER;
        int r = 0, c = 0;
        if (e2 < NTRI) tri_of(e2, r, c);
        double v = e2 < NTRI ? a[r][c] : b[e2 - NTRI];
        for (int t = tlo; t <= thi; ++t) v -= part[NACC * t + (e2 - (t * PER) / T)];
        if (e2 < NTRI) a[r][c] = v;
        else b[e2 - NTRI] = v;
    }
    sync();
}

// A Linv^T with the lower triangle of Linv: v_rc = sum_{k <= c} A[r][k] Linv[c][k],
// columns c0 and c1 = T-1-c0 of a row to one thread, T + 1 products, which
// out(r, c0, c1, v0, v1) gets.  Called by the first TT / 2 threads (the products are at one FP64
// warp instruction per 64 cycles and SM quarter either way, ~1,100 cycles).
template <typename Out>
__device__ __forceinline__ void tile_trsm(const double (*A)[T + 1], const double (*Li)[T + 1], Out out)
{
    const int r = threadIdx.x / (T / 2), c0 = threadIdx.x % (T / 2), c1 = T - 1 - c0;
    double x[T + 1], y[T + 1];
    // the products' factors first, so that the chain waits for no load
#pragma unroll
    for (int i = 0; i <= T; ++i) {
        const bool first = i <= c0;
        const int c = first ? c0 : c1, k = first ? i : i - c0 - 1;
        x[i] = A[r][k];
        y[i] = Li[c][k];
    }
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int i = 0; i <= T; ++i) {
        const bool first = i <= c0;
        const double v = fma(x[i], y[i], first ? s0 : s1);
        s0 = first ? v : s0;
        s1 = first ? s1 : v;
    }
    out(r, c0, c1, s0, s1);
}

// After the CTA barrier, thread 0's release store orders every thread's
// earlier writes (the barrier puts them before it) ahead of the flag.
__device__ __forceinline__ void block_release(int *flag, int epoch)
{
    __syncthreads();
    if (threadIdx.x == 0) st_release(flag, epoch);
}

// Flags: tile (I, K), I > K, at tile_task(I, K), raised when it is stored (and
// y_K with (K+1, K)).  By mail go, beside that, the diagonal inverses, the
// sub-diagonal tiles and y, the partial diagonal PD(I) =
// A_II - sum_{J <= I-2} L_IJ L_IJ^T (with b_I likewise), the partial sub-diagonal
// SUB(I) = A_{I+1,I} - sum_{J <= I-1} L_{I+1,J} L_IJ^T, and the
// second-subdiagonal tile (K+2, K) after its accumulation, before its solve.
//
// The factor with the forward solve of rhs carried along.  CTA 0 (the panel)
// walks the diagonal: step I applies the last update to PD(I) with L_{I,I-1}
// (its own, kept in shared memory), factors the tile (panel_factor), stores
// Linv_II (panel_finish; nothing reads L_II) and forms L_{I+1,I} = SUB(I) Linv_II^T, which it keeps, and
// y_I.  The other CTAs (helpers) run the task list: the tiles (I, K) with
// I >= K + 2 (left-looking updates, then the triangular solve with Linv_KK),
// and the PD and SUB accumulations, in the order
//   P(0), C(0), PD(2), SUB(1), P(1), C(1), PD(3), SUB(2), P(2), ...
// (P = panel step, C(K) = the tiles of column K) -- every task depends only on
// tasks before it, each helper takes every (G-1)-th task in that order and
// the panel its steps in order, so with all CTAs resident (cooperative
// launch) the first unfinished task can always run: no deadlock.
__global__ void __launch_bounds__(CF_THREADS, 1) k_chol_dataflow(int Np, int nb, int n_tasks,
                                                              const int2 *__restrict__ tasks,
                                                              double *__restrict__ S,
                                                              double *__restrict__ Linv,
                                                              double *__restrict__ rhs,
                                                              ulonglong2 *__restrict__ mail,
                                                              int *__restrict__ flags, int epoch,
                                                              int *__restrict__ status, long long spin_limit)
{
    static_assert(LowerUpdate::PART <= BJ * T * (T + 1), "update_lower's partial sums fit in the staging area");
    __shared__ double a[T][T + 1], linv[T][T + 1];
    __shared__ double bi[BJ][T][T + 1], bk[BJ][T][T + 1], by[BJ][T];
    __shared__ double bvec[T];
    __shared__ int ready_n;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    double *part = &bk[0][0][0];
    if (tid == 0) s_spin_limit = spin_limit;
    __syncthreads();
    if (blockIdx.x == 0) {
        // ---- panel.  Step I: warps 0-6 update and factor the diagonal tile;
        // warps 0-3 form L_{I+1,I} (the columns' factor t last, so that its
        // roots are not waited for), while warps 4-6 finish the tile's outputs and
        // y_I; warp 7, which raises L_{I+1,I}'s flag when the next step begins,
        // fetches SUB(I) and then PD(I+1) with its b as they come.  The panel tracks failure
        // itself (a bad pivot, a wait that ran out): it then leaves the loop
        // and raises all flags that are left.
        double(*lsub)[T + 1] = bi[2], (*asub)[T + 1] = bi[3], (*wli)[T + 1] = bi[4];
        double(*pfq)[PF_ROW] = reinterpret_cast<double(*)[PF_ROW]>(&bk[0][0][0]);
        const PfWork pw{pfq, by[3]};
        const PfEntry pe = pf_entry();
        __shared__ int hexp[2][T], stop[2];  // by the step's parity
        if (tid < 2) stop[tid] = 0;
        if (tid < T) pfq[tid][PF_ZERO] = 0.0;
        load_tile(bi[0], S, Np, 0, 0);
        if (tid < T) by[0][tid] = __ldcg(rhs + tid);
        __syncthreads();
        if (warp == 7) tile_exp(bi[0], hexp[0]);
        __syncthreads();
        PfOut po{{T, T}, {0, 0}};
#pragma unroll
        for (int j = 0; j < 2; ++j)
            if (warp >= 4 && warp < 7 && tid - 128 + 96 * j < TRI) tri_of(tid - 128 + 96 * j, po.r[j], po.c[j]);
        int pd_r[5], pd_c[5];  // warp 7's places in PD's mail
#pragma unroll
        for (int q = 0; q < 5; ++q) tri_of(min(lane + 32 * q, TRI - 1), pd_r[q], pd_c[q]);
        bool failed = false;
        int I = 0;
        for (; I < nb && !failed; ++I) {
            const int cur = I & 1;
            double *wy = by[2];
            if (warp == 7) {
                if (I >= 1 && lane == 0) st_release(flags + tile_task(I, I - 1, nb), epoch);
                if (I + 1 < nb) {
                    double(*an)[T + 1] = bi[cur ^ 1], *bn = by[cur ^ 1];
                    bool ok = true;
                    if (I == 0) {  // no updates before these
                        for (int e = lane; e < TT; e += 32) {
                            const double *src = S + (size_t)(T + e / T) * Np + e % T;
                            asub[e / T][e % T] = __ldcg(src);
                            an[e / T][e % T] = __ldcg(src + T);
                        }
                        if (lane < T) bn[lane] = __ldcg(rhs + T + lane);
                        pf_arrive<3, 160>();
                    } else {
                        double v[8];
                        ok = mail_get(mail + (size_t)I * ML_COLUMN + ML_SUB + lane, 32, 8, v, epoch, status);
#pragma unroll
                        for (int q = 0; q < 8; ++q) asub[2 * q + (lane >> 4)][lane & 15] = v[q];
                        pf_arrive<3, 160>();
                        double u[5];
                        ok = mail_get(mail + (size_t)(I + 1) * ML_COLUMN + ML_PD + lane, 32, lane < 24 ? 5 : 4, u, epoch, status) && ok;
#pragma unroll
                        for (int q = 0; q < 5; ++q) {
                            const int e = lane + 32 * q;
                            if (e < TRI) an[pd_r[q]][pd_c[q]] = u[q];
                            else if (e < TRI + T) bn[e - TRI] = u[q];
                        }
                    }
                    __syncwarp();
                    tile_exp(bi[cur ^ 1], hexp[cur ^ 1]);
                    if (!ok) stop[cur] = 1;
                }
            } else {
                ulonglong2 *mc = mail + (size_t)I * ML_COLUMN;
                panel_factor(bi[cur], hexp[cur], lsub, by[cur], wy, I == 0, wli, pw, pe);
                if (warp >= 4) {
                    const bool bad = panel_finish(wli, hexp[cur], by[cur], wy, I + 1 < nb, Linv + (size_t)I * TT,
                                                  rhs + I * T, mc, epoch, pw, po);
                    if (tid == 128 && bad) {
                        atomicCAS(status, 0, 1);
                        stop[cur] = 1;
                    }
                } else if (I + 1 < nb) {
                    pf_bar<3, 160>();  // SUB(I) is there
                    double *Lg = S + (size_t)((I + 1) * T) * Np + I * T;
                    double v0, v1;
                    int r, c0, c1;
                    tile_trsm(asub, wli, [&](int i, int j0, int j1, double x0, double x1) {
                        r = i;
                        c0 = j0;
                        c1 = j1;
                        v0 = x0;
                        v1 = x1;
                    });
                    pf_bar<5, 160>();  // t
                    v0 *= pw.t[c0];
                    v1 *= pw.t[c1];
                    mail_put(mc + ML_SUBD + r * T + c0, v0, epoch);
                    mail_put(mc + ML_SUBD + r * T + c1, v1, epoch);
                    lsub[r][c0] = v0;
                    lsub[r][c1] = v1;
                    Lg[(size_t)r * Np + c0] = v0;
                    Lg[(size_t)r * Np + c1] = v1;
                }
            }
            __syncthreads();
            failed = stop[cur] != 0;
        }
        if (tid == 0 && failed)
            for (int J = I - 1; J + 1 < nb; ++J) st_release(flags + tile_task(J + 1, J, nb), epoch);
        return;
    }
    // ---- helpers
    int inv_r, inv_c;  // the thread's place in an inverse's mail
    tri_of(min(tid, TRI - 1), inv_r, inv_c);
    for (int t = blockIdx.x - 1; t < n_tasks; t += gridDim.x - 1) {
        const int I = tasks[t].x, K = tasks[t].y;
        const int kind = I - K;  // 0: PD(I), 1: SUB(K), >= 2: tile (I, K)
        load_tile(a, S, Np, I, K);
        if (kind == 0 && tid < T) bvec[tid] = __ldcg(rhs + I * T + tid);
        __syncthreads();
        // Updates J = 0 .. n_upd-1 in order.  The flags of the next BJ steps
        // are polled at once (one L2 round trip); the ready ones have all their
        // tiles loaded together and are applied from shared memory.  Each
        // element is updated in the same order as one step at a time would.
        const int n_upd = kind == 0 ? I - 1 : K;
        const int n_main = kind <= 1 ? n_upd - 1 : n_upd;  // PD and SUB take their last step below
        int J = 0;
        while (J < n_main) {
            const int nmax = min(BJ, n_main - J);
            if (tid == 0) ready_n = nmax;
            __syncthreads();
            if (tid < nmax) {
                // the diagonal's other flag is that of y_J
                const int fi = ld_acquire(flags + tile_task(I, J + tid, nb));
                const int fk = ld_acquire(flags + tile_task(kind != 0 ? K : J + tid + 1, J + tid, nb));
                if (fi != epoch || fk != epoch) atomicMin(&ready_n, tid);
            }
            __syncthreads();
            int n = ready_n;
            if (n == 0) {  // the next step is not done yet: wait for it alone
                block_wait(flags + tile_task(I, J, nb), flags + tile_task(kind != 0 ? K : J + 1, J, nb), epoch, status);
                n = 1;
            }
            for (int e2 = tid; e2 < n * TT; e2 += CF_THREADS) {
                const int q = e2 / TT, r = (e2 % TT) / T, c = e2 % T;
                bi[q][r][c] = __ldcg(S + (size_t)(I * T + r) * Np + (J + q) * T + c);
                if (kind != 0) bk[q][r][c] = __ldcg(S + (size_t)(K * T + r) * Np + (J + q) * T + c);
            }
            if (kind == 0)
                for (int e2 = tid; e2 < n * T; e2 += CF_THREADS) by[e2 / T][e2 % T] = __ldcg(rhs + (J + e2 / T) * T + e2 % T);
            __syncthreads();
            if (kind == 0) {
                // the partial sums use bk, which the diagonal accumulation leaves free
                for (int q = 0; q < n; ++q) update_lower(a, bi[q], bvec, by[q], part);
            } else {
                for (int q = 0; q < n; ++q)
                    for (int e2 = tid; e2 < TT; e2 += CF_THREADS) {
                        const int r = e2 / T, c = e2 % T;
                        double sacc = a[r][c];
#pragma unroll
                        for (int k = 0; k < T; ++k) sacc = fma(-bi[q][r][k], bk[q][c][k], sacc);
                        a[r][c] = sacc;
                    }
            }
            __syncthreads();
            J += n;
        }
        if (kind <= 1) {
            // Last step, J = I - 2: L_{I,J} is the second-subdiagonal tile, whose
            // own task mails it before its solve and solves it for the others
            // once the panel raises Linv_JJ.  PD and SUB solve it here themselves
            // (the same arithmetic, so the same bits) as soon as Linv_JJ is
            // there, which saves the panel a hand-off per step.
            // Warps 0-3 solve it, the others meanwhile fetch L_{K,J} or y_J.
            const int Jl = I - 2;
            const ulonglong2 *from = mail + (size_t)Jl * ML_COLUMN;
            if (warp < 4) {
                double v[2];
                mail_get(from + ML_PRE + tid, TT / 2, 2, v, epoch, status);
                bi[1][tid / T][tid % T] = v[0];
                bi[1][tid / T + T / 2][tid % T] = v[1];
                mail_get(from + ML_INV + tid, TT / 2, tid < TRI - TT / 2 ? 2 : 1, v, epoch, status);
                linv[inv_r][inv_c] = v[0];
                if (tid < TRI - TT / 2) linv[T - 1][tid + TT / 2 - tri_at(T - 1, 0)] = v[1];
                pf_bar<3, TT / 2>();
                tile_trsm(bi[1], linv, [&](int i, int j0, int j1, double x0, double x1) {
                    bi[0][i][j0] = x0;
                    bi[0][i][j1] = x1;
                });
            } else {
                const int u = tid - TT / 2;
                double v[2];
                if (kind == 1) {
                    mail_get(from + ML_SUBD + u, TT / 2, 2, v, epoch, status);
                    bi[2][u / T][u % T] = v[0];
                    bi[2][u / T + T / 2][u % T] = v[1];
                } else if (u < T) {
                    mail_get(from + ML_Y + u, 0, 1, v, epoch, status);
                    by[0][u] = v[0];
                }
            }
            __syncthreads();
            const int r = tid / T, c = tid % T;
            if (kind == 0) {
                update_lower(a, bi[0], bvec, by[0], part);
                ulonglong2 *to = mail + (size_t)I * ML_COLUMN + ML_PD;
                if (c <= r) mail_put(to + tri_at(r, c), a[r][c], epoch);
                if (tid < T) mail_put(to + TRI + tid, bvec[tid], epoch);
            } else {
                double sacc = a[r][c];
#pragma unroll
                for (int k = 0; k < T; ++k) sacc = fma(-bi[0][r][k], bi[2][c][k], sacc);
                mail_put(mail + (size_t)K * ML_COLUMN + ML_SUB + tid, sacc, epoch);
            }
        } else {
            // the second-subdiagonal tile before its solve, for PD(K + 2) and SUB(K + 1)
            if (kind == 2) mail_put(mail + (size_t)K * ML_COLUMN + ML_PRE + tid, a[tid / T][tid % T], epoch);
            if (tid < TRI) {
                double v[1];
                mail_get(mail + (size_t)K * ML_COLUMN + ML_INV + tid, 0, 1, v, epoch, status);
                linv[inv_r][inv_c] = v[0];
            }
            __syncthreads();
            if (warp < 4)
                tile_trsm(a, linv, [&](int r, int c0, int c1, double v0, double v1) {
                    double *row = S + (size_t)(I * T + r) * Np + K * T;
                    row[c0] = v0;
                    row[c1] = v1;
                });
            block_release(flags + tile_task(I, K, nb), epoch);
        }
        __syncthreads();
    }
}

// Helper tasks in dependency order (see k_chol_dataflow): after panel step K
// come the tiles (I, K), I >= K + 2, then PD(K + 2) and SUB(K + 1).
void chol_task_list(int nb, std::vector<int2> &tasks)
{
    tasks.clear();
    for (int K = 0; K < nb; ++K) {
        for (int I = K + 2; I < nb; ++I) tasks.push_back(make_int2(I, K));
        if (K + 2 < nb) {
            tasks.push_back(make_int2(K + 2, K + 2));  // PD(K + 2)
            tasks.push_back(make_int2(K + 2, K + 1));  // SUB(K + 1)
        }
    }
}

int chol_grid(int n_tasks, int grid_cap)
{
    // CTAs per SM and SMs, per device (handles on several devices and
    // several host threads share this cache)
    static std::mutex mu;
    static int per_sm_dev[MAX_DEVICES], sms_dev[MAX_DEVICES];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= MAX_DEVICES) dev = 0;
    int per_sm, sms;
    {
        std::lock_guard<std::mutex> lk(mu);
        if (sms_dev[dev] == 0) {
            int p = 0, n = 0;
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p, k_chol_dataflow, CF_THREADS, 0);
            if (p < 1) p = 1;
            if (PSBA_CHOL_PER_SM > 0 && p > PSBA_CHOL_PER_SM) p = PSBA_CHOL_PER_SM;
            per_sm_dev[dev] = p;
            sms_dev[dev] = n > 0 ? n : 1;
        }
        per_sm = per_sm_dev[dev];
        sms = sms_dev[dev];
    }
    int cap = per_sm * sms;
    if (grid_cap > 0 && grid_cap < cap) cap = grid_cap;
    if (cap < 2) cap = 2;  // the panel and at least one helper
    return n_tasks < cap ? n_tasks : cap;
}

// ---------------------------------------------------------------------------
// The triangular solves on a thread-block cluster of TC_CTAS CTAs (one SM
// each): the back solve after the factor, or (refine = 1) both solves of a
// refinement residual, added into x.  Block after block, x_p = D_p y_p with the
// diagonal inverse, then y_r -= C_pr x_p for every later block r: a chain of nb
// steps, each two 16 x 16 products long when nothing else is waited for.
// CTA 0 keeps that chain to itself.  Two pairs of its warps take the diagonal
// product and the update of the next block in turns (four lanes an entry, four
// terms each, a fixed tree), warps 2 and 3 the update of the block after that,
// from x_p as soon as it is known.  All blocks from the third on take x_p in the other
// CTAs: block p is CTA 1 + p mod 7's, which sends it to CTA 0 with all its
// updates but the last two, two chain steps before it is needed.  x_p and these
// blocks travel as st.async stores that complete an mbarrier of their own (one
// per block and pass, used once), ~350 cycles, where one cluster barrier per
// step, with the solving CTA changing every step, made a step of 3,300
// cycles.  Each entry takes its updates in step order: results do not depend on
// timing.  A step is 1,500 cycles, two products of ~500 (six dependent FP64
// instructions and two shuffles each) and ~500 of barriers and shared memory:
// N = 528 takes 28 us, with a barrier of the cluster a step 56.
constexpr int TC_CTAS = 8, TC_THREADS = 256, TC_OWNERS = TC_CTAS - 1;
constexpr int TC_NEAR = 3;           // blocks up to p + TC_NEAR - 1 take x_p in CTA 0
constexpr int TC_SPIN = 1 << 12;     // polls without a pause (~60 us, longer than any wait of a solve that runs)
constexpr int TC_DRAIN = 1 << 20;    // polls for what is still under way to a CTA that gave up

__device__ __forceinline__ unsigned smem_at(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mb_init(unsigned long long *b, int count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_at(b)), "r"(count) : "memory");
}

__device__ __forceinline__ void mb_expect(unsigned long long *b, int bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_at(b)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mb_arrive(unsigned long long *b)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_at(b)) : "memory");
}

// Waits for the barrier's first phase, `limit` polls at most; false if they ran
// out.  (test_wait: try_wait suspends the thread for as long as the device likes,
// a hint of 100 ns notwithstanding, so its polls bound nothing.)
__device__ __forceinline__ bool mb_poll(unsigned long long *b, long long limit)
{
    for (long long it = 0; it < limit; ++it) {
        int ok;
        asm volatile("{ .reg .pred q; mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 q, [%1], 0; selp.s32 %0, 1, 0, q; }"
                     : "=r"(ok)
                     : "r"(smem_at(b))
                     : "memory");
        if (ok) return true;
        if (it >= TC_SPIN) __nanosleep(200);
    }
    return false;
}

// The waits of a thread: after one that ran out, nothing is waited for any more
struct TriWait {
    long long limit;
    bool dead;
    __device__ __forceinline__ void operator()(unsigned long long *b)
    {
        if (!dead) dead = !mb_poll(b, limit);
    }
};

// The address of p's place in the shared memory of CTA `rank`
__device__ __forceinline__ unsigned peer_at(const void *p, int rank)
{
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_at(p)), "r"(rank));
    return a;
}

// v to another CTA's shared memory, 8 bytes of what its barrier there waits for
__device__ __forceinline__ void send(unsigned place, unsigned bar, double v)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(place),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}

// Four lanes of one output: their sum in all of them
__device__ __forceinline__ double quad_sum(double s)
{
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    return s + __shfl_xor_sync(0xffffffffu, s, 2);
}

__device__ __forceinline__ double dot4(const double (&cf)[4], const double *v)
{
    double s = cf[0] * v[0];
#pragma unroll
    for (int j = 1; j < 4; ++j) s = fma(cf[j], v[j], s);
    return quad_sum(s);
}

// The matrix as the chain sees it, by positions (0 is solved first)
template <bool FWD>
struct TriView {
    const double *S, *Linv;
    int Np, nb;
    __device__ __forceinline__ int block(int p) const { return FWD ? p : nb - 1 - p; }
    // terms 4 g .. 4 g + 3 of entry c of the diagonal product at p: a place that
    // moves by diag_step from one p to the next
    __device__ __forceinline__ const double *diag_at(int p, int c, int g) const
    {
        return Linv + (size_t)block(p) * TT + (FWD ? c * T + 4 * g : 4 * g * T + c);
    }
    __device__ __forceinline__ ptrdiff_t diag_step() const { return FWD ? TT : -TT; }
    __device__ __forceinline__ static void diag(const double *L, int c, int g, double (&v)[4])
    {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = (FWD ? 4 * g + j <= c : 4 * g + j >= c) ? __ldcg(L + (FWD ? j : j * T)) : 0.0;
    }
    // terms of what entry c of the block at r takes of x_p; moves by coef_step when
    // both move on
    __device__ __forceinline__ const double *coef_at(int p, int r, int c, int g) const
    {
        const int P = block(p) * T, R = block(r) * T;
        return S + (FWD ? (size_t)(R + c) * Np + P + 4 * g : (size_t)(P + 4 * g) * Np + R + c);
    }
    __device__ __forceinline__ ptrdiff_t coef_step() const { return (ptrdiff_t)(FWD ? T : -T) * (Np + 1); }
    __device__ __forceinline__ void coef(const double *L, double (&v)[4]) const
    {
        const unsigned st = FWD ? 1 : Np;
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = __ldcg(L + j * st);
    }
};

// One solve: base (Np) is the right-hand side, xs takes the solution in every
// CTA, far (Np) is CTA 0's inbox and the others' blocks, bars 2 nb barriers.
template <bool FWD>
__device__ __forceinline__ void tri_pass(const TriView<FWD> &m, int rank, const double *base, double *xs, double *far,
                                         unsigned long long *bars, double (*yb)[T], double (*near2)[T], TriWait &wait)
{
    const int tid = threadIdx.x, lane = tid & 31, g = tid & 3, nb = m.nb;
    if (rank == 0) {
        unsigned long long *bfar = bars, *bx = bars + nb;
        const int c = (tid & 63) >> 2;
        if (tid < 64 || (tid >= 128 && tid < 192)) {
            // the chain: even p by warps 0 and 1, odd p by warps 4 and 5, so that
            // what follows a step (x to the others, the next coefficients' loads,
            // ~500 cycles) goes beside the next one
            const int set = tid >= 128;
            double dg[4] = {}, cr[4] = {};
            const double *dp = m.diag_at(min(set, nb - 1), c, g), *cp = m.coef_at(min(set, nb - 1), min(set + 1, nb - 1), c, g);
            const ptrdiff_t ds = 2 * m.diag_step(), cs = 2 * m.coef_step();
            if (set < nb) m.diag(dp, c, g, dg);
            if (set + 1 < nb) m.coef(cp, cr);
            int at = m.block(set) * T + c;
            // where x goes: CTAs 1 + g and 5 + g (whose barrier p is x_p's)
            unsigned to0 = peer_at(xs, 1 + g) + at * (int)sizeof(double), to1 = peer_at(xs, g < 3 ? 5 + g : 0) + at * (int)sizeof(double);
            unsigned tb0 = peer_at(bars + set, 1 + g), tb1 = peer_at(bars + set, g < 3 ? 5 + g : 0);
            if (set == 0) {
                if (g == 0) yb[0][c] = base[at];
                pf_bar<1, 64>();
            }
            for (int p = set; p < nb; p += 2) {
                if (set) pf_bar<5, 128>();  // y_p is there
                else if (p > 0) pf_bar<4, 128>();
                const double x = dot4(dg, yb[set] + 4 * g);
                if (g == 0) xs[at] = x;
                if (set) pf_bar<6, 64>();
                else pf_bar<1, 64>();
                if (p + 1 < nb) {
                    const double u = dot4(cr, xs + (at - c) + 4 * g);
                    double b;
                    if (p > 0) {
                        if (set) pf_bar<2, 128>();
                        else pf_bar<3, 128>();
                        b = near2[set ^ 1][c];
                    } else {
                        b = base[m.block(1) * T + c];
                    }
                    if (g == 0) yb[set ^ 1][c] = b - u;
                    if (set) pf_arrive<4, 128>();
                    else pf_arrive<5, 128>();
                }
                if (lane == 0) mb_arrive(bx + p);
                send(to0, tb0, x);
                if (g < 3) send(to1, tb1, x);
                if (p + 2 < nb) m.diag(dp += ds, c, g, dg);
                if (p + 3 < nb) m.coef(cp += cs, cr);
                constexpr int ahead = 2 * (FWD ? T : -T);
                at += ahead;
                to0 += (unsigned)(ahead * (int)sizeof(double));
                to1 += (unsigned)(ahead * (int)sizeof(double));
                tb0 += 2 * sizeof(unsigned long long);
                tb1 += 2 * sizeof(unsigned long long);
            }
        } else if (tid >= 64 && tid < 128) {
            double cf[4], cn[4] = {}, cm[4] = {};
            const double *cp = m.coef_at(0, min(2, nb - 1), c, g);
            const ptrdiff_t cs = m.coef_step();
            if (nb > 2) m.coef(cp, cf);
            if (nb > 3) m.coef(cp += cs, cn);
            for (int p = 2; p < nb; ++p) {
                if (p + 2 < nb) m.coef(cp += cs, cm);
                if (p >= TC_NEAR) wait(bfar + p);
                const double b = (p >= TC_NEAR ? far : base)[m.block(p) * T + c];
                wait(bx + p - 2);
                const double v = b - dot4(cf, xs + m.block(p - 2) * T + 4 * g);
                if (g == 0) near2[p & 1][c] = v;
                // a barrier per parity: the next but one, p + 2, needs an x_p that
                // the chain has only after it has taken this one
                if (p & 1) pf_arrive<3, 128>();
                else pf_arrive<2, 128>();
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    cf[j] = cn[j];
                    cn[j] = cm[j];
                }
            }
        }
    } else {
        // entry c of this CTA's blocks k, k + 4, k + 8, ... (four lanes)
        const int c = (tid >> 2) & (T - 1), k = tid >> 6;
        const int p0 = rank - 1 + TC_OWNERS * k, step = TC_OWNERS * (TC_THREADS / 64);
        auto next = [&](int q) {  // the first of them at q or later
            return q <= p0 ? p0 : p0 + (q - p0 + step - 1) / step * step;
        };
        if (g == 0)
            for (int p = p0; p < nb; p += step) far[m.block(p) * T + c] = base[m.block(p) * T + c];
        double cf[4] = {}, cn[4] = {}, cm[4] = {};
        auto coef = [&](int q, int p, double (&v)[4]) { m.coef(m.coef_at(q, p, c, g), v); };
        if (next(TC_NEAR) < nb) coef(0, next(TC_NEAR), cf);
        if (next(TC_NEAR + 1) < nb) coef(1, next(TC_NEAR + 1), cn);
        for (int q = 0; q < nb; ++q) {
            int p = next(q + TC_NEAR);
            const int pn = next(q + 2 + TC_NEAR);
            if (pn < nb) coef(q + 2, pn, cm);
            wait(bars + q);
            const double *xq = xs + m.block(q) * T + 4 * g;
            if (p < nb) {
                const double s = dot4(cf, xq);
                double *mine = far + m.block(p) * T + c;
                if (g == 0) {
                    const double v = *mine - s;
                    if (p == q + TC_NEAR) send(peer_at(mine, 0), peer_at(bars + p, 0), v);
                    else *mine = v;
                }
                for (p += step; p < nb; p += 2 * step) {
                    double c0[4], c1[4] = {};
                    const int p1 = p + step;
                    coef(q, p, c0);
                    if (p1 < nb) coef(q, p1, c1);
                    const double s0 = dot4(c0, xq), s1 = dot4(c1, xq);
                    if (g == 0) {
                        far[m.block(p) * T + c] -= s0;
                        if (p1 < nb) far[m.block(p1) * T + c] -= s1;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                cf[j] = cn[j];
                cn[j] = cm[j];
            }
        }
    }
}

__device__ __forceinline__ void cl_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

size_t tri_smem(int Np, int refine)
{
    const size_t passes = refine ? 2 : 1;
    return passes * (2 * sizeof(double) * Np + 2 * sizeof(unsigned long long) * (Np / T));
}

__global__ void __launch_bounds__(TC_THREADS, 1) k_tri_cluster(int refine, int Np, int nb,
                                                            const double *__restrict__ S,
                                                            const double *__restrict__ Linv,
                                                            const double *__restrict__ rhs,
                                                            double *__restrict__ x, float2 *__restrict__ x2,
                                                            int *__restrict__ status, long long spin_limit)
{
    static_assert(T == 16 && TC_CTAS == 8, "two sends a lane reach the other CTAs");
    extern __shared__ double tri_sm[];  // per pass: x, inbox; then the barriers
    __shared__ double yb[2][T], near2[2][T];
    const int rank = (int)cg::this_cluster().block_rank(), tid = threadIdx.x, passes = refine ? 2 : 1;
    if (*status != 0) return;  // the same word for every CTA: all leave together
    unsigned long long *bars = reinterpret_cast<unsigned long long *>(tri_sm + (size_t)2 * passes * Np);
    for (int i = tid; i < passes * nb; i += TC_THREADS) {
        unsigned long long *b = bars + (i >= nb ? nb + i : i);
        mb_init(b, 1);  // a block on its way here: x_p, or in CTA 0 the block at p
        mb_init(b + nb, 2);  // x_p in CTA 0, from its two warps
        if (rank != 0 || i % nb >= TC_NEAR) mb_expect(b, T * sizeof(double));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    cl_sync();
    TriWait wait{spin_limit, false};
    double *xs = tri_sm, *far = tri_sm + (size_t)passes * Np;
    if (refine) {
        tri_pass(TriView<true>{S, Linv, Np, nb}, rank, rhs, xs, far, bars, yb, near2, wait);
        __syncthreads();
        tri_pass(TriView<false>{S, Linv, Np, nb}, rank, xs, xs + Np, far + Np, bars + 2 * nb, yb, near2, wait);
        xs += Np;
    } else {
        tri_pass(TriView<false>{S, Linv, Np, nb}, rank, rhs, xs, far, bars, yb, near2, wait);
    }
    if (wait.dead) atomicCAS(status, 0, 2);
    // Every block sent to a CTA has been waited for there, or (all are sent, if
    // late, whoever gave up) is waited for now: a store under way must not outlive
    // the CTA whose shared memory it goes to.
    if (__syncthreads_or(wait.dead))
        for (int i = tid; i < passes * nb; i += TC_THREADS)
            if (rank != 0 || i % nb >= TC_NEAR) mb_poll(bars + (i >= nb ? nb + i : i), TC_DRAIN);
    cl_sync();
    if (rank == 0)
        for (int i = tid; i < Np; i += TC_THREADS) {
            const double xv = refine ? x[i] + xs[i] : xs[i];
            x[i] = xv;
            if (x2) x2[i] = split2f(xv);
        }
}

// The triangular solves after the factor: the back solve of d.rhs into x
// (refine = 0), or both solves of d.rhs added into x (refine = 1).
void launch_tri(const DeviceProblem &d, int refine, double *x, cudaStream_t s)
{
    const int nb = d.Np / T, Np = d.Np;
    // the solution also as FP32 pairs for the mixed form's eb sums (x is dpa
    // on every path that reaches them)
    float2 *x2 = d.prec == PSBA_PREC_MIXED && d.cnp == 6 ? d.dpa2f : nullptr;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(TC_CTAS);
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = tri_smem(Np, refine);
    cfg.stream = s;
    if (cfg.dynamicSmemBytes > 40 * 1024)  // above the default limit (as for k_cholmod: the same value always)
        cudaFuncSetAttribute(k_tri_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tri_smem(4096, 1));
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = TC_CTAS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const double *S = d.S, *Linv = d.Linv, *rhs = d.rhs;
    cudaLaunchKernelEx(&cfg, k_tri_cluster, refine, Np, nb, S, Linv, rhs, x, x2, d.status, d.wait_limit);
    note_launch(1);
}

void launch_chol_dataflow(const DeviceProblem &d, int epoch, double *x_out, cudaStream_t s)
{
    int nb = d.Np / T;
    int Np = d.Np;
    {
        int n_tasks = d.chol_n_tasks;
        const int grid = chol_grid(n_tasks + 1, d.chol_grid_cap);
        const int2 *tasks = d.chol_tasks;
        double *S = d.S, *Linv = d.Linv, *rhs = d.rhs;
        ulonglong2 *mail = d.chol_mail;
        int *flags = d.chol_flags, *status = d.status;
        long long spin = d.wait_limit;
        void *args[] = {&Np, &nb, &n_tasks, (void *)&tasks, &S, &Linv, &rhs, &mail, &flags, &epoch, &status, &spin};
        cudaMemsetAsync(d.status, 0, 2 * sizeof(int), s);
        cudaLaunchCooperativeKernel((const void *)k_chol_dataflow, dim3(grid), dim3(CF_THREADS), args, 0, s);
        note_launch(1);
    }
    launch_tri(d, 0, x_out, s);
}

// r = b - S x over the Np rows (S symmetric, its lower triangle in Sc with
// leading dimension ld), each row's sum as Dot2 of Ogita, Rump and Oishi
// ("Accurate sum and dot product", SIAM J. Sci. Comput. 26(6), 2005): every
// product split exactly by an FMA, the running sum carried with Knuth's
// TwoSum and the rounding errors summed beside it, so the residual is as
// accurate as if S x were formed in twice the working precision.  A residual
// formed in plain FP64 is mostly the rounding of S x (S x matches b to the
// last bits after a backward-stable solve), so a refinement step on it
// leaves the forward error where it was; on this one it falls from ~cond(S)
// eps to ~eps.  One warp a row: the row's part left of the diagonal and the
// column's part below it, each lane's terms in order, then a fixed xor tree
// of the (sum, error) pairs.  A failed factor (status != 0) leaves r
// untouched.
constexpr int RR_THREADS = 256;

// s + e = a + b exactly (Knuth's TwoSum)
__device__ __forceinline__ void two_sum(double a, double b, double &s, double &e)
{
    s = __dadd_rn(a, b);
    const double z = __dsub_rn(s, a);
    e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, z)), __dsub_rn(b, z));
}

// (hi, lo) += a x
__device__ __forceinline__ void dot2_add(double a, double x, double &hi, double &lo)
{
    const double p = __dmul_rn(a, x);
    const double pe = fma(a, x, -p);  // a x - p exactly
    double t;
    two_sum(hi, p, hi, t);
    lo = __dadd_rn(lo, __dadd_rn(t, pe));
}

__global__ void __launch_bounds__(RR_THREADS) k_refine_residual(int Np, const double *__restrict__ Sc, int ld,
                                                                 const double *__restrict__ b,
                                                                 const double *__restrict__ x, double *__restrict__ r,
                                                                 const int *__restrict__ status)
{
    const int i = (int)((blockIdx.x * (size_t)RR_THREADS + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (i >= Np || *status != 0) return;
    const double *row = Sc + (size_t)i * ld;
    double hi = 0.0, lo = 0.0;
    for (int j = lane; j <= i; j += 32) dot2_add(row[j], x[j], hi, lo);
    for (int j = i + 1 + lane; j < Np; j += 32) dot2_add(Sc[(size_t)j * ld + i], x[j], hi, lo);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double oh = __shfl_xor_sync(0xffffffffu, hi, off), ol = __shfl_xor_sync(0xffffffffu, lo, off);
        double t;
        two_sum(hi, oh, hi, t);
        lo = __dadd_rn(__dadd_rn(lo, ol), t);
    }
    if (lane == 0) {
        double s, t;
        two_sum(b[i], -hi, s, t);
        r[i] = __dadd_rn(s, __dsub_rn(t, lo));
    }
}

// One refinement step of the solve x of S x = b just made: S and b were saved
// (Sc with leading dimension ld, bc) before the factor overwrote them; the
// residual goes to d.rhs, and its solve is added into x.
void launch_refine(const DeviceProblem &d, const double *Sc, int ld, const double *bc, double *x, cudaStream_t s)
{
    const int blocks = (int)(((size_t)d.Np * 32 + RR_THREADS - 1) / RR_THREADS);
    k_refine_residual<<<blocks, RR_THREADS, 0, s>>>(d.Np, Sc, ld, bc, x, d.rhs, d.status);
    note_launch(1);
    launch_tri(d, 1, x, s);
}

// ---------------------------------------------------------------------------
// Modified Cholesky (trust-region lambda fallback), restating cholmod_blk.cl
// with get_delta_beta (cl_cholmod.cpp:109-165) and kern_cholmod_E: block
// columns of 3 are factored as plain 3x3 blocks when the pivots are positive
// and every entry below is <= beta; otherwise their columns are redone one
// at a time with d = max(|c|, delta) and the theta/beta bound.
//
// One cooperative launch, right-looking, one grid barrier per block step.  Row i
// belongs to CTA i mod G, which keeps its rows in shared memory from the first
// step to the last (where they do not fit, in S itself).  Per step every CTA
// reads the step's three columns (n x 3, published by the rows' owners) and
// forms the whole panel in shared memory, with the 3x3 factor, the test against
// beta and, where it fails, the column-at-a-time path, so nothing of the
// step's decisions goes between CTAs; it then updates its own rows with the
// rank-3 product and publishes their next three columns.  Each entry takes
// the same sequence of 3-term subtractions, in the same block order, as the
// reference's left-looking sums; the column-at-a-time path subtracts the
// earlier blocks in those 3-term groups and the block's own columns one at a
// time.
//
// Bound by a step's chain: the columns' L2 round trip, the 3x3 factor's
// divisions and roots (a warp issues an FP64 instruction per 64 cycles, so
// they are dealt to lanes, five rounds deep), the panel and the barrier.  At
// N = 528: 33 ms on one CTA; 4.65 ms with four barriers a step, a one-thread 3x3
// factor and the flags of all CTAs read by every thread; 1.83 ms with one
// barrier and the rows in S (each thread's updates waited for one another's
// loads); 1.35 ms with the rows resident.
constexpr int CM_THREADS = 256;

__device__ double cta_max(double v, double *red)
{
    for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, off));
    __syncthreads();  // the last result is read
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = red[0];
    for (int w = 1; w < CM_THREADS / 32; ++w) r = fmax(r, red[w]);
    return r;
}

// The 3x3 factor of the block t (row-major, lower read) and its inverse by one
// warp: L 00 10 11 20 21 22 and Li row-major; false if a pivot is not
// positive and finite or an entry not finite (cholmod_blk.cl:135-191).
__device__ bool cm_block(const double *t, double *L, double *Li, int lane)
{
    const double t0 = t[0], t3 = t[3], t4 = t[4], t6 = t[6], t7 = t[7], t8 = t[8];
    auto from = [](double v, int src) { return __shfl_sync(0xffffffffu, v, src); };
    // round 1
    const double q1 = (lane == 0 ? t3 * t3 : t3 * t6) / t0;
    const double p1 = t4 - from(q1, 0), cross = t7 - from(q1, 1);
    const double a1 = -t8 * t3 * t3, a2 = 2 * t7 * t3 * t6, a3 = -t4 * t6 * t6;
    const double a4 = t0 * (t4 * t8 - t7 * t7), a5 = -t3 * t3 + t0 * t4;
    // round 2
    const double q2 = (lane == 0 ? a1 + a2 + a3 + a4 : t0) / a5;
    const double p2 = from(q2, 0), w4 = from(q2, 1);
    // round 3
    const double root = sqrt(lane == 0 ? t0 : lane == 1 ? p1 : lane == 2 ? p2 : w4);
    const double l0 = from(root, 0), l2 = from(root, 1), l5 = from(root, 2), l4 = from(root, 3) * cross;
    // round 4
    const double q4 = (lane == 0 ? t3 : lane == 1 ? t6 : 1.0) / (lane <= 2 ? l0 : lane == 3 ? l2 : l5);
    const double l1 = from(q4, 0), l3 = from(q4, 1);
    // round 5
    const double q5 = (lane == 0 ? -l1 : lane == 1 ? l1 * l4 - l2 * l3 : -l4) /
                      (lane == 0 ? l0 * l2 : lane == 1 ? l0 * l2 * l5 : l2 * l5);
    const double i0 = from(q4, 2), i4 = from(q4, 3), i8 = from(q4, 4), i3 = from(q5, 0), i6 = from(q5, 1), i7 = from(q5, 2);
    if (lane == 0) {
        L[0] = l0; L[1] = l1; L[2] = l2; L[3] = l3; L[4] = l4; L[5] = l5;
        Li[0] = i0; Li[1] = 0; Li[2] = 0;
        Li[3] = i3; Li[4] = i4; Li[5] = 0;
        Li[6] = i6; Li[7] = i7; Li[8] = i8;
    }
    return isfinite(t0) && t0 > 0 && isfinite(p1) && p1 > 0 && isfinite(p2) && p2 > 0 && isfinite(l1) && isfinite(l3) &&
           isfinite(l4);
}

// work: diag (n), then gmax[2 G], then the published columns, twice 3 n.
// resident: the CTA's rows in shared memory (rows x n doubles after the panel's
// 3 n), else in S; panel_stride > 0: the panel does not fit either and is a
// slice of `panel` per CTA.
__global__ void __launch_bounds__(CM_THREADS) k_cholmod(double *S, int n, int ld, double *E, double *work, int resident,
                                                        double *panel, size_t panel_stride)
{
    cg::grid_group grid = cg::this_grid();
    extern __shared__ double cm_sm[];
    __shared__ double dred[CM_THREADS / 32];
    __shared__ double sh_t[9], sh_L[6], sh_Li[9], sh_lxx;
    __shared__ int sh_ok;
    const int G = gridDim.x, b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double *P = panel_stride ? panel + (size_t)b * panel_stride : cm_sm;  // row r of the step's panel at 3 r
    double *diag = work, *gmax = work + n, *cols = gmax + 2 * G;
    // this CTA's rows b, b + G, ...: row b + q G at R + q pitch
    double *R = resident ? cm_sm + 3 * (size_t)n : S + (size_t)b * ld;
    const size_t pitch = resident ? (size_t)n : (size_t)G * ld;
    const int n_rows = b < n ? (n - b + G - 1) / G : 0;
    // xi = max |offdiag|, gamma = max |diag| over the symmetric matrix (lower read)
    double xi = 0.0, gam = 0.0;
    for (int q = 0; q < n_rows; ++q) {
        const int r = b + q * G;
        for (int k = tid; k < n; k += CM_THREADS) {
            double *s = S + (size_t)r * ld + k;
            if (k > r) {
                *s = 0.0;
                continue;
            }
            const double v = *s;
            if (resident) R[q * pitch + k] = v;
            if (k < 3) __stcg(cols + 3 * (size_t)r + k, v);
            if (k == r) {
                gam = fmax(gam, fabs(v));
                diag[r] = v;
            } else {
                xi = fmax(xi, fabs(v));
            }
        }
    }
    xi = cta_max(xi, dred);
    gam = cta_max(gam, dred);
    if (tid == 0) {
        gmax[2 * b] = xi;
        gmax[2 * b + 1] = gam;
    }
    grid.sync();
    xi = 0.0;
    gam = 0.0;
    for (int q = tid; q < G; q += CM_THREADS) {
        xi = fmax(xi, __ldcg(gmax + 2 * q));
        gam = fmax(gam, __ldcg(gmax + 2 * q + 1));
    }
    xi = cta_max(xi, dred);
    gam = cta_max(gam, dred);
    const double delta = 1e-15 * fmax(xi + gam, 1.0);
    double beta = fmax(gam, 1e-15);
    beta = fmax(beta, xi / sqrt((double)n * (double)n - 1.0));
    beta = sqrt(beta);
    const int nb = n / 3;
    for (int j = 0; j < nb; ++j) {
        const int j3 = 3 * j, t0 = j3 + 3;
        const double *in = cols + 3 * (size_t)n * (j & 1);
        double *out = cols + 3 * (size_t)n * ((j + 1) & 1);
        // the step's columns, updated by the earlier steps: the 3x3 block for
        // warp 0, all of them into the panel
        if (warp == 0) {
            if (lane < 9) {
                const int u = lane / 3, v = lane % 3;
                sh_t[lane] = __ldcg(in + 3 * (size_t)(j3 + max(u, v)) + min(u, v));
            }
            __syncwarp();
            const bool ok = cm_block(sh_t, sh_L, sh_Li, lane);
            if (lane == 0) sh_ok = ok;
        } else {
            for (int e = 3 * t0 + tid - 32; e < 3 * n; e += CM_THREADS - 32) P[e] = __ldcg(in + e);
        }
        __syncthreads();
        int big = sh_ok ? 0 : 1;
        if (!big) {
            // L_ij = T_ij Li^T, tested before it is kept
            const double i0 = sh_Li[0], i3 = sh_Li[3], i4 = sh_Li[4], i6 = sh_Li[6], i7 = sh_Li[7], i8 = sh_Li[8];
            for (int r = t0 + tid; r < n; r += CM_THREADS) {
                const double x0 = P[3 * (size_t)r], x1 = P[3 * (size_t)r + 1], x2 = P[3 * (size_t)r + 2];
                if (x0 * i0 > beta || x0 * i3 + x1 * i4 > beta || x0 * i6 + x1 * i7 + x2 * i8 > beta) big = 1;
            }
            big = __syncthreads_or(big);
            if (!big) {
                for (int r = t0 + tid; r < n; r += CM_THREADS) {
                    const double x0 = P[3 * (size_t)r], x1 = P[3 * (size_t)r + 1], x2 = P[3 * (size_t)r + 2];
                    P[3 * (size_t)r] = x0 * i0;
                    P[3 * (size_t)r + 1] = x0 * i3 + x1 * i4;
                    P[3 * (size_t)r + 2] = x0 * i6 + x1 * i7 + x2 * i8;
                }
                if (tid == 0) {
                    double *d = P + 3 * (size_t)j3;
                    d[0] = sh_L[0]; d[1] = 0; d[2] = 0;
                    d[3] = sh_L[1]; d[4] = sh_L[2]; d[5] = 0;
                    d[6] = sh_L[3]; d[7] = sh_L[4]; d[8] = sh_L[5];
                }
            }
        }
        if (big) {
            // the block's columns one at a time, from the values read above
            if (tid < 9) P[3 * (size_t)j3 + tid] = tid / 3 >= tid % 3 ? sh_t[tid] : 0.0;
            __syncthreads();
            for (int col = 0; col < 3; ++col) {
                const int x = j3 + col;
                const double *px = P + 3 * (size_t)x;
                if (tid == 0) {
                    double sum = px[col];
                    for (int k = 0; k < col; ++k) sum -= px[k] * px[k];
                    sh_lxx = sqrt(fmax(fabs(sum), delta));
                }
                __syncthreads();
                double lxx = sh_lxx, th = 0.0;
                int over = 0;
                for (int r = x + 1 + tid; r < n; r += CM_THREADS) {
                    double *pr = P + 3 * (size_t)r;
                    double c = pr[col];
                    for (int k = 0; k < col; ++k) c = c - (pr[k] * px[k]);
                    pr[col] = c;
                    th = fmax(th, fabs(c));
                    if (c / lxx > beta) over = 1;
                }
                if (__syncthreads_or(over)) lxx = cta_max(th, dred) / beta;
                for (int r = x + 1 + tid; r < n; r += CM_THREADS) P[3 * (size_t)r + col] /= lxx;
                if (tid == 0) P[3 * (size_t)x + col] = lxx;
                __syncthreads();
            }
        }
        __syncthreads();
        // this CTA's rows from j3 on: their L (into S, and their copy), then
        // the rank-3 update S_ic -= L_i,j3.. L_c,j3.., c <= i, a warp per row
        // and pass of 32 columns; the next step's columns go out first
        const int q0 = j3 > b ? (j3 - b + G - 1) / G : 0;
        for (int e = tid; e < 3 * (n_rows - q0); e += CM_THREADS) {
            const int q = q0 + e / 3, c = e % 3, r = b + q * G;
            if (r - j3 < c) continue;
            const double v = P[3 * (size_t)r + c];
            S[(size_t)r * ld + j3 + c] = v;
            if (resident) R[q * pitch + j3 + c] = v;
        }
        for (int q = q0; q < n_rows; ++q) {
            const int i = b + q * G;
            if (i < t0) continue;
            const double a0 = P[3 * (size_t)i], a1 = P[3 * (size_t)i + 1], a2 = P[3 * (size_t)i + 2];
            double *row = R + q * pitch;
            for (int c = t0 + tid; c <= i; c += CM_THREADS) {
                const double v = row[c] - (a0 * P[3 * (size_t)c] + a1 * P[3 * (size_t)c + 1] + a2 * P[3 * (size_t)c + 2]);
                row[c] = v;
                if (c < t0 + 3) __stcg(out + 3 * (size_t)i + (c - t0), v);
            }
        }
        grid.sync();
    }
    // E_i = sum_k L_ik^2 - A_ii, a warp per row
    for (int q = warp; q < n_rows; q += CM_THREADS / 32) {
        const int i = b + q * G;
        double sum = 0.0;
        for (int k = lane; k <= i; k += 32) {
            const double v = R[q * pitch + k];
            sum = fma(v, v, sum);
        }
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (lane == 0) E[i] = sum - diag[i];
    }
}

// Dynamic shared memory at most (the rest of a CTA's 227 KB holds the static part)
constexpr size_t CM_SMEM = 218 * 1024;

// doubles of work the modified Cholesky needs at size n
size_t cholmod_work(int n)
{
    const size_t panel = 3 * (size_t)n * sizeof(double) > CM_SMEM ? 3 * (size_t)n * CM_MAX_CTAS : 0;
    return 7 * (size_t)n + 2 * (size_t)CM_MAX_CTAS + 8 + panel;
}

void launch_cholmod(double *S, int n, int ld, double *E, double *work, cudaStream_t s, int grid_cap)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int G = sms < CM_MAX_CTAS ? sms : CM_MAX_CTAS;
    if (grid_cap > 0 && grid_cap < G) G = grid_cap;
    const int rows = (n + 7) / 8;  // no more CTAs than the trailing rows can use
    if (rows < G) G = rows;
    if (G < 1) G = 1;
    // the panel (24 bytes a row) and the CTA's rows: resident up to n of about
    // 1,700 on 152 CTAs, the panel alone up to 9,300
    size_t smem = 3 * (size_t)n * sizeof(double), stride = 0;
    const size_t all = smem + (size_t)((n + G - 1) / G) * n * sizeof(double);
    int resident = all <= CM_SMEM;
    if (resident) {
        smem = all;
    } else if (smem > CM_SMEM) {
        smem = 0;
        stride = 3 * (size_t)n;
    }
    if (smem > 40 * 1024)  // above the default limit (an attribute of the kernel on this device; the same value always)
        cudaFuncSetAttribute(k_cholmod, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CM_SMEM);
    double *panel = work + 7 * (size_t)n + 2 * CM_MAX_CTAS + 8;
    void *args[] = {&S, &n, &ld, &E, &work, &resident, &panel, &stride};
    cudaLaunchCooperativeKernel((const void *)k_cholmod, dim3(G), dim3(CM_THREADS), args, smem, s);
    note_launch(1);
}

}  // namespace psba

// ---------------------------------------------------------------------------
// Diagnostic entry points for the parity tests: the dense solve on a caller
// matrix, and the projections' reciprocal.
namespace psba {

__global__ void k_pivot_reciprocal(int n, const double *__restrict__ x, double *__restrict__ y)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = rcp_fast(x[i]);
}

}  // namespace psba

extern "C" int psba_eval_pivot_reciprocal(int n, const double *x, double *y)
{
    using namespace psba;
    if (n < 0 || (n > 0 && (!x || !y))) return set_error("psba_eval_pivot_reciprocal: bad arguments"), PSBA_ERR_ARG;
    if (n == 0) return PSBA_OK;
    double *dx = nullptr, *dy = nullptr;
    cudaError_t e = cudaMalloc(&dx, sizeof(double) * (size_t)n);
    if (e == cudaSuccess) e = cudaMalloc(&dy, sizeof(double) * (size_t)n);
    if (e == cudaSuccess) e = cudaMemcpy(dx, x, sizeof(double) * (size_t)n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_pivot_reciprocal<<<(n + 255) / 256, 256>>>(n, dx, dy);
        note_launch(1);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(y, dy, sizeof(double) * (size_t)n, cudaMemcpyDeviceToHost);
    cudaFree(dx);
    cudaFree(dy);
    if (e != cudaSuccess) return set_error(std::string("CUDA error: ") + cudaGetErrorString(e)), PSBA_ERR_CUDA;
    return PSBA_OK;
}

// The handle's dense solve (k_chol_dataflow + the back solve) on an n x n
// matrix given by the caller: S row-major, lower triangle read; padded to a
// multiple of TILE with an identity block.
extern "C" int psba_eval_dense_solve(int n, const double *S, const double *b, double *x, int *status)
{
    using namespace psba;
    if (n <= 0 || n > 4096 || !S || !b || !x || !status)
        return set_error("psba_eval_dense_solve: n must be in 1..4096 and every pointer set"), PSBA_ERR_ARG;
    DeviceProblem d;
    d.Np = ((n + TILE - 1) / TILE) * TILE;
    const int Np = d.Np, nb = Np / TILE;
    std::vector<int2> tasks;
    chol_task_list(nb, tasks);
    d.chol_n_tasks = (int)tasks.size();
    d.chol_n_flags = nb * (nb + 1) / 2;
    std::vector<double> hS((size_t)Np * Np, 0.0), hb(Np, 0.0);
    for (int r = 0; r < Np; ++r)
        for (int c = 0; c <= r; ++c) hS[(size_t)r * Np + c] = (r < n && c < n) ? S[(size_t)r * n + c] : (r == c ? 1.0 : 0.0);
    for (int r = 0; r < n; ++r) hb[r] = b[r];
    cudaStream_t st = nullptr;
    std::vector<void *> mem;
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    auto get = [&](auto **p, size_t count) {
        if (e != cudaSuccess) return;
        e = cudaMalloc((void **)p, sizeof(**p) * (count ? count : 1));
        if (e == cudaSuccess) mem.push_back((void *)*p);
    };
    get(&d.S, (size_t)Np * Np);
    get(&d.rhs, (size_t)Np);
    get(&d.xsol, (size_t)Np);
    get(&d.Linv, (size_t)Np * TILE);
    get(&d.chol_mail, (size_t)nb * CHOL_MAIL);
    get(&d.chol_tasks, tasks.size());
    get(&d.chol_flags, (size_t)d.chol_n_flags);
    get(&d.status, 4);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.S, hS.data(), sizeof(double) * hS.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(d.rhs, hb.data(), sizeof(double) * Np, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && !tasks.empty())
        e = cudaMemcpyAsync(d.chol_tasks, tasks.data(), sizeof(int2) * tasks.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d.chol_flags, 0, sizeof(int) * d.chol_n_flags, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d.chol_mail, 0, sizeof(*d.chol_mail) * nb * CHOL_MAIL, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d.status, 0, sizeof(int) * 4, st);
    if (e == cudaSuccess) {
        launch_chol_dataflow(d, 1, d.xsol, st);
        e = cudaGetLastError();
    }
    int hst[4] = {0, 0, 0, 0};
    if (e == cudaSuccess) e = cudaMemcpyAsync(hst, d.status, sizeof(hst), cudaMemcpyDeviceToHost, st);
    std::vector<double> hx(Np);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hx.data(), d.xsol, sizeof(double) * Np, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    for (void *p : mem) cudaFree(p);
    if (st) cudaStreamDestroy(st);
    if (e != cudaSuccess) return set_error(std::string("CUDA error: ") + cudaGetErrorString(e)), PSBA_ERR_CUDA;
    *status = hst[0];
    if (hst[0] == 0)
        for (int r = 0; r < n; ++r) x[r] = hx[r];
    return PSBA_OK;
}
