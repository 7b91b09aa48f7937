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
    const int2 *Yq, *Wq;   // limbs
    const int2 *Yl, *Wl;   // third pieces
    const int2 *ex;
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

// The N <= 4 third pieces of a group
template <int N>
__device__ __forceinline__ void ld_lows(const int2 *p, float (&out)[N])
{
    const uint2 v = *reinterpret_cast<const uint2 *>(p);
    out[0] = (float)(v.x & 0xffffu);
    if (N > 1) out[1] = (float)(v.x >> 16);
    if (N > 2) out[2] = (float)(v.y & 0xffffu);
    if (N > 3) out[3] = (float)(v.y >> 16);
}

// ---------------------------------------------------------------------------
// 6-parameter cameras: a warp per unit, no block barriers.  Per 32 entries:
// the entries' rows come into the warp's shared memory by 16-byte
// asynchronous copies (the next chunk's are under way during the sums' end);
// lane t moves entry t's W row (and gb, DIAG) to the chunk's exponent; lane
// 4 g + q takes entries g, g + 8, g + 16, g + 24 and quadrant q of the block in
// two 64-bit integers and an FP32 number per output (DIAG: and gb as a fourth
// column); the eight lane groups' totals meet in shared memory, and a lane per
// output adds them to its FP64 sum.
// Camera block (k, l), sm: F6_WORDS of the warp's shared memory; emit(v, r, c,
// sum) is called by one lane per output v at (r, c).  SOLO: an observation's
// limbs and third pieces are one row, and they and gb come from an earlier
// launch (read-only cache loads); else limbs and third pieces are apart.
constexpr int F6_L = 18, F6_F = 6, F6_G = 4;  // int2 words an entry: limbs, third pieces, gb (three limbs, third pieces)
constexpr int F6_WORDS = FX_CHUNK * (2 * (F6_L + F6_F) + F6_G);

template <bool DIAG, bool SOLO, typename Emit>
__device__ void fx6_unit(const FxArgs &g, const SchurUnit u, int k, int l, int2 *sm, Emit &&emit)
{
    constexpr int CNP = 6, TC = DIAG ? 4 : 3, CP = 2 * TC;  // totals of a row: 6, or 6 and each half's gb column
    constexpr int NV = n_out<CNP, DIAG>(), PER = (NV + 31) / 32;
    constexpr size_t ROW_L = SOLO ? F6_L + F6_F : F6_L, ROW_F = SOLO ? F6_L + F6_F : F6_F;
    int2 *yl = sm, *wl = yl + FX_CHUNK * F6_L, *yf = wl + FX_CHUNK * F6_L, *wf = yf + FX_CHUNK * F6_F,
         *sg = wf + FX_CHUNK * F6_F;
    const int lane = threadIdx.x & 31, q = lane & 3, rg = q >> 1, cg = q & 1;
    // the totals, over the rows that are read
    long long *sH = reinterpret_cast<long long *>(yl);
    unsigned *sL = reinterpret_cast<unsigned *>(sH + 8 * 6 * CP);
    static_assert(8 * 6 * CP * 12 <= FX_CHUNK * F6_L * 8, "the totals fit");
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
        const int2 x = SOLO ? __ldg(g.ex + an) : g.ex[an];
        y = x.x;
        w = DIAG ? x.y : SOLO ? __ldg(&g.ex[bn].y) : g.ex[bn].y;
        if (DIAG) i = __ldg(g.obs_pt + an);
    };
    auto rows = [&]() {
#pragma unroll
        for (int m = 0; m < 12; ++m) {  // piece p of 12 x 32: row p / 12, 16 bytes p % 12
            const int p = lane + 32 * m, r = p / 12, part = p - 12 * r;
            const int ra = __shfl_sync(0xffffffffu, an, r), rb = __shfl_sync(0xffffffffu, bn, r);
            const bool lim = part < 9;
            const int d = lim ? r * F6_L + 2 * part : 2 * FX_CHUNK * F6_L + r * F6_F + 2 * (part - 9);
            const int dw = d + (lim ? FX_CHUNK * F6_L : FX_CHUNK * F6_F);
            cp_async16(sm + d, lim ? g.Yq + ROW_L * ra + 2 * part : g.Yl + ROW_F * ra + 2 * (part - 9));
            cp_async16(sm + dw, lim ? g.Wq + ROW_L * rb + 2 * part : g.Wl + ROW_F * rb + 2 * (part - 9));
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
                gv[j] = SOLO ? __ldg(gj) : *gj;
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
                int4 *row = reinterpret_cast<int4 *>(wl + lane * F6_L), *low = reinterpret_cast<int4 *>(wf + lane * F6_F);
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const int4 f = low[j];
                    Fx3 s[6];
#pragma unroll
                    for (int m = 0; m < 3; ++m) {
                        const int4 x = row[3 * j + m];
                        const unsigned f0 = m == 0 ? f.x & 0xffff : m == 1 ? f.y & 0xffff : (unsigned)f.z >> 16;
                        const unsigned f1 = m == 0 ? (unsigned)f.x >> 16 : m == 1 ? f.z & 0xffff : f.w & 0xffff;
                        s[2 * m] = fx_shift(make_int2(x.x, x.y), f0, d);
                        s[2 * m + 1] = fx_shift(make_int2(x.z, x.w), f1, d);
                        row[3 * j + m] = make_int4(s[2 * m].v.x, s[2 * m].v.y, s[2 * m + 1].v.x, s[2 * m + 1].v.y);
                    }
                    low[j] = make_int4(s[0].f | s[1].f << 16, s[2].f, s[3].f | s[4].f << 16, s[5].f);
                }
                if (DIAG) {
                    Fx3 s[3];
#pragma unroll
                    for (int j = 0; j < 3; ++j) s[j] = fx_limbs3(gv[j], Eg - eyt - fx_exp(gv[j]));
                    int4 *gr = reinterpret_cast<int4 *>(sg + lane * F6_G);
                    gr[0] = make_int4(s[0].v.x, s[0].v.y, s[1].v.x, s[1].v.y);
                    gr[1] = make_int4(s[2].v.x, s[2].v.y, s[0].f | s[1].f << 16, s[2].f);
                }
            }
            __syncwarp();
            long long hh[3][TC], hl[3][TC];
            float cr[3][TC];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j) {
                    hh[i][j] = hl[i][j] = 0;
                    cr[i][j] = 0.0f;
                }
#pragma unroll 1
            for (int m = 0; m < FX_CHUNK / 8; ++m) {
                const int t = (lane >> 2) + 8 * m;
                if (t >= n) break;
                float fg[3];
                if (DIAG) ld_lows<3>(sg + t * F6_G + 3, fg);
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    int2 a[3], b[TC];
                    float fa[3], fb[TC], fw[3];
                    ld_limbs<3>(yl + t * F6_L + 6 * j + 3 * rg, a);
                    ld_limbs<3>(wl + t * F6_L + 6 * j + 3 * cg, b);
                    ld_lows<3>(yf + t * F6_F + 2 * j + rg, fa);
                    ld_lows<3>(wf + t * F6_F + 2 * j + cg, fw);
#pragma unroll
                    for (int c = 0; c < 3; ++c) fb[c] = fw[c];
                    if (DIAG) {
                        b[TC - 1] = sg[t * F6_G + j];
                        fb[TC - 1] = fg[j];
                    }
                    fx_products<3, TC>(a, fa, b, fb, hh, hl, cr);
                }
            }
            __syncwarp();  // the rows are read
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j) {
                    const int to = (lane >> 2) * 6 * CP + (3 * rg + i) * CP + (j < 3 ? 3 * cg + j : 6 + cg);
                    fx_carry(hh[i][j], hl[i][j], cr[i][j], sH[to], sL[to]);
                }
            __syncwarp();
#pragma unroll
            for (int p = 0; p < PER; ++p) {
                if (at[p] < 0) continue;
                long long H = 0;
                unsigned L = 0;
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    H += sH[s * 6 * CP + at[p]];
                    L += sL[s * 6 * CP + at[p]];
                }
                acc[p] = fx_add(acc[p], H, L, we[p] + (DIAG && at[p] % CP == CNP ? Eg : E));
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
