// The Schur complement's products on limb rows (psba_fixed.h): the pieces that
// the single-problem kernels (psba_schurfx.cu) and the batched engine share.
#pragma once

#include "psba_fixed.h"
#include "psba_internal.h"

#ifdef __CUDACC__
namespace psba {

constexpr int FX_CHUNK = 32;  // entries aligned to one exponent at a time

// What the product kernels read.
struct FxArgs {
    const int *pa, *pb;    // pair entries: observation of camera k, of camera l
    const int *cam_obs;    // observations by camera
    const int *obs_pt;
    const int2 *Yq, *Wq, *ex;
    const double *W, *Vinv;  // for entries with an infinity or a NaN
    const double *U, *gb;
    const int *pair_kl;
    double *off_partial, *diag_partial;
};

// One output of a chunk that holds an infinity or a NaN, in plain FP64:
// sum_t Y_t[r] . (W_t[c], or gb for column CNP), Y formed as in k_limb_rows.
template <int CNP>
__device__ __noinline__ double fx_plain(const FxArgs &g, const int *pa, const int *pb, int n, int r, int c, double acc)
{
    for (int t = 0; t < n; ++t) {
        const int a = pa[t], i = g.obs_pt[a];
        const double *w = g.W + 3 * CNP * (size_t)a + 3 * r, *s = g.Vinv + 6 * (size_t)i;
        const double *x = c < CNP ? g.W + 3 * CNP * (size_t)pb[t] + 3 * c : g.gb + 3 * (size_t)i;
        acc = fma(w[0] * s[0] + w[1] * s[1] + w[2] * s[2], x[0], acc);
        acc = fma(w[0] * s[1] + w[1] * s[3] + w[2] * s[4], x[1], acc);
        acc = fma(w[0] * s[2] + w[1] * s[4] + w[2] * s[5], x[2], acc);
    }
    return acc;
}

// The (r, c) of output v: row-major blocks, or (DIAG) the lower triangle, then ea as column CNP
template <int CNP, bool DIAG>
__device__ __forceinline__ void out_rc(int v, int &r, int &c)
{
    constexpr int NL = CNP * (CNP + 1) / 2;
    if (!DIAG) {
        r = v / CNP;
        c = v % CNP;
    } else if (v >= NL) {
        r = v - NL;
        c = CNP;
    } else {
        r = 0;
        c = v;
        while (c > r) c -= ++r;
    }
}
template <int CNP, bool DIAG>
__host__ __device__ constexpr int n_out()
{
    return DIAG ? CNP * (CNP + 1) / 2 + CNP : CNP * CNP;
}

// The exponent that output (r, c) of a block of cameras k, l adds to its chunks'
template <int CNP>
__device__ __forceinline__ int out_weight(const FxArgs &g, int k, int l, int r, int c)
{
    int e = fx_weight(g.U[CNP * CNP * (size_t)k + (CNP + 1) * r]);
    if (c < CNP) e += fx_weight(g.U[CNP * CNP * (size_t)l + (CNP + 1) * c]);
    return e;
}

// N neighbouring limb words, as 16-byte loads where N is even
template <int N>
__device__ __forceinline__ void ld_limbs(const int2 *p, int2 *out)
{
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int k = 0; k < N; k += 2) {
            const int4 v = *reinterpret_cast<const int4 *>(p + k);
            out[k] = make_int2(v.x, v.y);
            out[k + 1] = make_int2(v.z, v.w);
        }
    } else {
#pragma unroll
        for (int k = 0; k < N; ++k) out[k] = p[k];
    }
}

// A TR x TC tile of entry t's products, summed over the NJ inner columns
template <int TR, int TC, int RP, int CP, int NJ = 3>
__device__ __forceinline__ void fx_tile(const int2 *y, const int2 *w, long long (&hh)[TR][TC], long long (&hl)[TR][TC])
{
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        int2 a[TR], b[TC];
        ld_limbs<TR>(y + j * RP, a);
        ld_limbs<TC>(w + j * CP, b);
#pragma unroll
        for (int p = 0; p < TR; ++p)
#pragma unroll
            for (int q = 0; q < TC; ++q) fx_mad(a[p], b[q], hh[p][q], hl[p][q]);
    }
}

// ---------------------------------------------------------------------------
// 6-parameter cameras: a warp per unit, no block barriers.  Per 32 entries:
// the entries' rows come into the warp's shared memory by 16-byte
// asynchronous copies (the next chunk's are under way during the sums' end);
// lane t moves entry t's W row (and gb, DIAG) to the chunk's exponent; lane
// 4 g + q takes entries g, g + 8, g + 16, g + 24 and quadrant q of the block in
// two 64-bit integers per output; the eight lane groups' totals meet in
// shared memory, and a lane per output adds them to its FP64 sum.
// Camera block (k, l), sy and sw: F6_SY and F6_SW words of the warp's shared
// memory; emit(v, r, c, sum) is called by one lane per output v at (r, c).  NC:
// the limb rows and gb come from an earlier launch (read-only cache loads).
constexpr int F6_SY = FX_CHUNK * 18, F6_SW = FX_CHUNK * 26;

template <bool DIAG, bool NC, typename Emit>
__device__ void fx6_unit(const FxArgs &g, const SchurUnit u, int k, int l, int2 *sy, int2 *sw, Emit &&emit)
{
    constexpr int CNP = 6, TC = DIAG ? 4 : 3, CP = 2 * TC;  // columns: 6, or 6 + gb + a pad
    constexpr int SY = 18, SW = DIAG ? 26 : 18;             // words from entry to entry: no bank conflicts
    constexpr int NV = n_out<CNP, DIAG>(), PER = (NV + 31) / 32;
    const int lane = threadIdx.x & 31, q = lane & 3, r0 = 3 * (q >> 1), c0 = TC * (q & 1);
    long long *st = reinterpret_cast<long long *>(sy);  // the totals, over the rows that are read
    static_assert(8 * 6 * CP <= FX_CHUNK * SY, "the totals fit");
    double acc[PER];
    int at[PER], we[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        acc[p] = 0.0;
        at[p] = -1;
        we[p] = 0;
        const int v = lane + 32 * p;
        if (v < NV) {
            int r, c;
            out_rc<CNP, DIAG>(v, r, c);
            at[p] = r * CP + c;
            we[p] = out_weight<CNP>(g, k, l, r, c);
        }
    }
    const int *pa = DIAG ? g.cam_obs + u.begin : g.pa + u.begin, *pb = DIAG ? pa : g.pb + u.begin;
    // entry lane of a chunk: its observations, its exponents and (DIAG) its
    // point; while a chunk is summed, the next one's
    int an = 0, bn = 0, ey = 0, ew = 0, pt = 0;
    auto indices = [&](int t0) {
        const int t = min(t0 + lane, u.count - 1);
        an = __ldg(pa + t);
        bn = DIAG ? an : __ldg(pb + t);
    };
    auto exponents = [&](int &y, int &w, int &i) {
        const int2 x = NC ? __ldg(g.ex + an) : g.ex[an];
        y = x.x;
        w = DIAG ? x.y : NC ? __ldg(&g.ex[bn].y) : g.ex[bn].y;
        if (DIAG) i = __ldg(g.obs_pt + an);
    };
    auto rows = [&]() {
#pragma unroll
        for (int m = 0; m < 9; ++m) {  // piece p of 9 x 32: row p / 9, 16 bytes p % 9
            const int p = lane + 32 * m, r = p / 9, part = p - 9 * r;
            const int ra = __shfl_sync(0xffffffffu, an, r), rb = __shfl_sync(0xffffffffu, bn, r);
            const int wd = DIAG ? (part / 3) * CP + 2 * (part % 3) : 2 * part;
            cp_async16(sy + r * SY + 2 * part, g.Yq + 18 * (size_t)ra + 2 * part);
            cp_async16(sw + r * SW + wd, g.Wq + 18 * (size_t)rb + 2 * part);
        }
    };
    indices(0);
    exponents(ey, ew, pt);
    rows();
    for (int t0 = 0; t0 < u.count; t0 += FX_CHUNK) {
        const int n = min(FX_CHUNK, u.count - t0);
        const bool more = t0 + FX_CHUNK < u.count;
        if (more) indices(t0 + FX_CHUNK);
        const int e = lane < n ? ey + ew : -(1 << 20);
        const int E = __reduce_max_sync(0xffffffffu, e);
        bool bad = E >= FX_NAN / 2;
        int Eg = 0;
        double gv[3] = {0.0, 0.0, 0.0};
        if (DIAG) {
            int eg = -(1 << 20), nf = 0;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const double *gj = g.gb + 3 * (size_t)pt + j;
                gv[j] = NC ? __ldg(gj) : *gj;
                eg = max(eg, fx_exp(gv[j]));
                nf |= fx_nonfinite(gv[j]);
            }
            Eg = __reduce_max_sync(0xffffffffu, lane < n ? ey + eg : -(1 << 20));
            bad |= __any_sync(0xffffffffu, nf);
        }
        const int eyt = ey;
        cp_async_wait();
        __syncwarp();
        if (more) exponents(ey, ew, pt);
        if (!bad) {
            // entry lane's W row, d bits down
            if (lane < n) {
                const int d = E - e;
                int4 *row = reinterpret_cast<int4 *>(sw + lane * SW);
#pragma unroll
                for (int m = 0; m < 9; ++m) {
                    int4 &x = row[DIAG ? (m / 3) * (CP / 2) + m % 3 : m];
                    const int2 s0 = fx_shift(make_int2(x.x, x.y), d), s1 = fx_shift(make_int2(x.z, x.w), d);
                    x = make_int4(s0.x, s0.y, s1.x, s1.y);
                }
                if (DIAG)
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        const int2 s = fx_limbs(gv[j], Eg - eyt - fx_exp(gv[j]));
                        row[j * (CP / 2) + 3] = make_int4(s.x, s.y, 0, 0);
                    }
            }
            __syncwarp();
            long long hh[3][TC], hl[3][TC];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j) hh[i][j] = hl[i][j] = 0;
#pragma unroll
            for (int m = 0; m < FX_CHUNK / 8; ++m) {
                const int t = (lane >> 2) + 8 * m;
                if (t < n) fx_tile<3, TC, 6, CP>(sy + t * SY + r0, sw + t * SW + c0, hh, hl);
            }
            __syncwarp();  // the rows are read
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j)
                    st[(lane >> 2) * 6 * CP + (r0 + i) * CP + c0 + j] = fx_total(hh[i][j], hl[i][j]);
            __syncwarp();
#pragma unroll
            for (int p = 0; p < PER; ++p) {
                if (at[p] < 0) continue;
                long long T = 0;
#pragma unroll
                for (int s = 0; s < 8; ++s) T += st[s * 6 * CP + at[p]];
                acc[p] = fx_add(acc[p], T, we[p] + (DIAG && at[p] % CP == CNP ? Eg : E));
            }
        } else {
#pragma unroll
            for (int p = 0; p < PER; ++p)
                if (at[p] >= 0) acc[p] = fx_plain<CNP>(g, pa + t0, pb + t0, n, at[p] / CP, at[p] % CP, acc[p]);
        }
        __syncwarp();
        if (more) rows();
    }
#pragma unroll
    for (int p = 0; p < PER; ++p)
        if (at[p] >= 0) emit(lane + 32 * p, at[p] / CP, at[p] % CP, acc[p]);
}

}  // namespace psba
#endif
