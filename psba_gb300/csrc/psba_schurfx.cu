// The FP64 Schur complement's products in block fixed point (psba_fixed.h):
// S's off-diagonal blocks sum_i Y_ik W_il^T and the diagonal blocks with ea's
// sums Y gb (compute_S.cl:39-77, compute_ea.cl:21-36).
//
// k_limb_rows forms Y = W V^-1 (compute_Yblks.cl:26-37) and cuts each
// observation's Y and W rows into limbs and third pieces (psba_fixed.h),
// relative to the observation's own largest value after the camera's row
// weights (fx_weight).  The sums then need one more shift per pair entry, of
// its W row, to the largest eY + eW among the 32 entries taken together: a point
// close to one camera has a W row there 10^4 times the others' and Y rows as
// much smaller, and only what lies 73 bits below the largest product is lost.  Cutting both rows at every
// use instead (a point is in about six pairs per observation) cost 1,560
// instructions per warp and 32 entries, twice the products' own.
#include "psba_fixed_schur.h"
#include "psba_internal.h"

namespace psba {

namespace {

inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// ---------------------------------------------------------------------------
// Y and the limb rows.  A CTA takes LR_THREADS / TPO consecutive observations
// (their W rows are contiguous), TPO threads each, TR rows a thread; rows go
// through shared memory so that global loads and stores are coalesced.
// Bound by the FP64 pipe (9 multiply-adds a row) and the ~35 integer
// instructions that cut a value (88 cameras: 51 us).
constexpr int LR_THREADS = 128;

template <int CNP>
__global__ void __launch_bounds__(LR_THREADS) k_limb_rows(int no, const int *__restrict__ obs_pt,
                                                          const int *__restrict__ obs_cam,
                                                          const double *__restrict__ W,
                                                          const double *__restrict__ Vinv,
                                                          const double *__restrict__ U, int2 *__restrict__ Yq,
                                                          int2 *__restrict__ Wq, int2 *__restrict__ ex)
{
    constexpr int RP = fx_rows(CNP), TPO = CNP == 6 ? 2 : 4, TR = RP / TPO, OB = LR_THREADS / TPO, WORDS = fx_words(CNP);
    static_assert(TR == fx_group(CNP), "a thread's rows are a group of third pieces");
    __shared__ __align__(16) double sw[OB * 3 * CNP];
    __shared__ __align__(16) int2 sq[2][OB * WORDS];
    const int o0 = blockIdx.x * OB, n = min(OB, no - o0), tid = threadIdx.x;
    for (int e = tid; e < n * 3 * CNP; e += LR_THREADS) sw[e] = __ldg(W + 3 * CNP * (size_t)o0 + e);
    const int t = tid / TPO, q = tid % TPO, o = o0 + min(t, n - 1);
    const double *vi = Vinv + 6 * (size_t)__ldg(obs_pt + o);
    const double *u = U + CNP * CNP * (size_t)__ldg(obs_cam + o);
    const double s00 = __ldg(vi), s01 = __ldg(vi + 1), s02 = __ldg(vi + 2), s11 = __ldg(vi + 3), s12 = __ldg(vi + 4),
                 s22 = __ldg(vi + 5);
    int rho[TR];
#pragma unroll
    for (int a = 0; a < TR; ++a) {
        const int r = q * TR + a;
        rho[a] = r < CNP ? fx_weight(__ldg(u + (CNP + 1) * r)) : 0;
    }
    __syncthreads();
    double w[TR][3], y[TR][3];
    int ew = -4096, ey = -4096, bw = 0, by = 0;
#pragma unroll
    for (int a = 0; a < TR; ++a) {
        const int r = q * TR + a;
        if (r >= CNP) {
#pragma unroll
            for (int j = 0; j < 3; ++j) w[a][j] = y[a][j] = 0.0;
            continue;
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) w[a][j] = sw[min(t, n - 1) * 3 * CNP + 3 * r + j];
        y[a][0] = w[a][0] * s00 + w[a][1] * s01 + w[a][2] * s02;
        y[a][1] = w[a][0] * s01 + w[a][1] * s11 + w[a][2] * s12;
        y[a][2] = w[a][0] * s02 + w[a][1] * s12 + w[a][2] * s22;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            ew = max(ew, fx_exp(w[a][j]) - rho[a]);
            ey = max(ey, fx_exp(y[a][j]) - rho[a]);
            bw |= fx_nonfinite(w[a][j]);
            by |= fx_nonfinite(y[a][j]);
        }
    }
#pragma unroll
    for (int x = 1; x < TPO; x *= 2) {
        ew = max(ew, __shfl_xor_sync(0xffffffffu, ew, x));
        ey = max(ey, __shfl_xor_sync(0xffffffffu, ey, x));
        bw |= __shfl_xor_sync(0xffffffffu, bw, x);
        by |= __shfl_xor_sync(0xffffffffu, by, x);
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        unsigned fy[4] = {}, fw[4] = {};
#pragma unroll
        for (int a = 0; a < TR; ++a) {
            const int at = t * WORDS + j * RP + q * TR + a;
            const Fx3 vy = fx_limbs3(y[a][j], ey + rho[a] - fx_exp(y[a][j])), vw = fx_limbs3(w[a][j], ew + rho[a] - fx_exp(w[a][j]));
            sq[0][at] = vy.v;
            sq[1][at] = vw.v;
            fy[a] = vy.f;
            fw[a] = vw.f;
        }
        const int at = t * WORDS + fx_limb_words(CNP) + j * TPO + q;
        sq[0][at] = make_int2(fy[0] | fy[1] << 16, fy[2] | fy[3] << 16);
        sq[1][at] = make_int2(fw[0] | fw[1] << 16, fw[2] | fw[3] << 16);
    }
    if (q == 0 && t < n) ex[o] = make_int2(by ? FX_NAN : ey, bw ? FX_NAN : ew);
    __syncthreads();
    int4 *yd = reinterpret_cast<int4 *>(Yq + WORDS * (size_t)o0), *wd = reinterpret_cast<int4 *>(Wq + WORDS * (size_t)o0);
    const int4 *ys = reinterpret_cast<const int4 *>(sq[0]), *ws = reinterpret_cast<const int4 *>(sq[1]);
    for (int e = tid; e < n * WORDS / 2; e += LR_THREADS) {
        yd[e] = ys[e];
        wd[e] = ws[e];
    }
}

constexpr int F6_WARPS = 4, F6_CTAS = 4;  // resident CTAs per SM: 287 / 283 us with 3 / 4 at 88 cameras
constexpr int F6_SMEM = F6_WARPS * F6_WORDS * (int)sizeof(int2);  // dynamic: 52 KB

// The diagonal units' blocks first (more work per entry), then the pairs'.
__global__ void __launch_bounds__(32 * F6_WARPS, F6_CTAS) k_schur_fx6(FxArgs g, int n_diag, const SchurUnit *__restrict__ diag,
                                                             int n_off, const SchurUnit *__restrict__ off)
{
    extern __shared__ __align__(16) int2 fx_sm[];
    const int warp = threadIdx.x >> 5, diag_ctas = (n_diag + F6_WARPS - 1) / F6_WARPS;
    int2 *sm = fx_sm + warp * F6_WORDS;
    if ((int)blockIdx.x < diag_ctas) {
        const int uid = blockIdx.x * F6_WARPS + warp;
        if (uid < n_diag) {
            const SchurUnit u = diag[uid];
            fx6_unit<true, true>(g, u, u.slot, u.slot, sm,
                           [&](int v, int, int, double x) { g.diag_partial[(size_t)u.out * 27 + v] = x; });
        }
    } else {
        const int uid = (blockIdx.x - diag_ctas) * F6_WARPS + warp;
        if (uid < n_off) {
            const SchurUnit u = off[uid];
            fx6_unit<false, true>(g, u, __ldg(g.pair_kl + 2 * u.slot), __ldg(g.pair_kl + 2 * u.slot + 1), sm,
                            [&](int v, int, int, double x) { g.off_partial[(size_t)u.out * 36 + v] = x; });
        }
    }
}

// ---------------------------------------------------------------------------
// 11- and 16-parameter cameras: a CTA of four warps per unit, the same steps;
// half-warps take the entries in turn, 4 x 4 threads with a TR x TR tile each
// (diagonal blocks: and gb, as the 12th column's pad, or as a fifth column).
constexpr int FV_THREADS = 128;

// Shared memory of a CTA in int2 words: per entry limbs (two words of padding)
// and third pieces of Y and of W and gb's three limbs and third pieces, then the warps' totals.
template <int CNP, bool DIAG>
struct FvShape {
    static constexpr int RP = fx_rows(CNP), TR = RP / 4, NL = fx_limb_words(CNP), NF = fx_low_words(CNP), NW = FV_THREADS / 32;
    static constexpr int XG = DIAG && CNP == RP ? 1 : 0;  // gb is a column more
    static constexpr int TC = TR + XG, CP = RP + 4 * XG;
    static constexpr int SL = NL + 2, ENTRY = 2 * (SL + NF) + 4 * XG;
    static constexpr int ROWS = FX_CHUNK * ENTRY, TOTALS = NW * RP * CP;
    static constexpr int BYTES = ROWS * 8 + TOTALS * 12;
    // CTAs an SM: as many as the tile's registers leave (without the bound the 16-parameter
    // diagonal blocks take 242 registers, with it 166: 21 cameras 154 -> 142 us both launches)
    static constexpr int CTAS = CNP == 11 ? 4 : 3;
};

template <int CNP, bool DIAG>
__global__ void __launch_bounds__(FV_THREADS, FvShape<CNP, DIAG>::CTAS)
    k_schur_fxv(FxArgs g, const SchurUnit *__restrict__ units)
{
    using F = FvShape<CNP, DIAG>;
    constexpr int RP = F::RP, TR = F::TR, TC = F::TC, CP = F::CP, SL = F::SL, NF = F::NF, NW = F::NW, G = fx_group(CNP);
    constexpr int NV = n_out<CNP, DIAG>(), PER = (NV + FV_THREADS - 1) / FV_THREADS;
    constexpr int LIMBS = F::NL / 2, PIECES = LIMBS + NF / 2;  // 16-byte pieces of a row
    static_assert(TR == G, "a thread's rows are a group of third pieces");
    extern __shared__ __align__(16) int2 fx_sm[];
    long long *sH = reinterpret_cast<long long *>(fx_sm + F::ROWS);
    unsigned *sL = reinterpret_cast<unsigned *>(sH + F::TOTALS);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const SchurUnit u = units[blockIdx.x];
    const int *pa = DIAG ? g.cam_obs + u.begin : g.pa + u.begin, *pb = DIAG ? pa : g.pb + u.begin;
    double acc[PER];
    int at[PER], we[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        acc[p] = 0.0;
        at[p] = -1;
        we[p] = 0;
        const int v = tid + FV_THREADS * p;
        if (v < NV) {
            int r, c;
            out_rc<CNP, DIAG>(v, r, c);
            at[p] = r * CP + c;
            we[p] = out_weight<CNP>(g, DIAG ? u.slot : __ldg(g.pair_kl + 2 * u.slot),
                                    DIAG ? u.slot : __ldg(g.pair_kl + 2 * u.slot + 1), r, c);
        }
    }
    // entry lane of a chunk, in every warp: its observations two chunks ahead,
    // its exponents and (DIAG) its point one chunk ahead, with the rows
    int an = 0, bn = 0, eyn = 0, en = 0, ptn = 0;
    auto indices = [&](int t0) {
        const int t = min(t0 + lane, u.count - 1);
        an = __ldg(pa + t);
        bn = DIAG ? an : __ldg(pb + t);
    };
    // (a second buffer for the next chunk's rows, 58 KB a CTA, left too few CTAs: 52
    // cameras, 11 parameters, 642 us for both launches instead of 580)
    int2 *yl = fx_sm, *wl = yl + FX_CHUNK * SL, *yf = wl + FX_CHUNK * SL, *wf = yf + FX_CHUNK * NF, *sg = wf + FX_CHUNK * NF;
    auto fetch = [&](int t0) {
        const int n = min(FX_CHUNK, u.count - t0);
#pragma unroll
        for (int m = 0; m < (FX_CHUNK * PIECES + FV_THREADS - 1) / FV_THREADS; ++m) {
            const int p = tid + FV_THREADS * m, t = p / PIECES, part = p % PIECES;
            const int ia = __shfl_sync(0xffffffffu, an, t & 31), ib = DIAG ? ia : __shfl_sync(0xffffffffu, bn, t & 31);
            if (t >= n) continue;
            const bool lim = part < LIMBS;
            const int to = lim ? t * SL + 2 * part : t * NF + 2 * (part - LIMBS);
            cp_async16((lim ? yl : yf) + to, g.Yq + fx_words(CNP) * (size_t)ia + 2 * part);
            cp_async16((lim ? wl : wf) + to, g.Wq + fx_words(CNP) * (size_t)ib + 2 * part);
        }
        en = -(1 << 20);
        if (lane < n) {
            const int2 xa = __ldg(g.ex + an);
            eyn = xa.x;
            en = eyn + (DIAG ? xa.y : __ldg(&g.ex[bn].y));
            if (DIAG) ptn = __ldg(g.obs_pt + an);
        }
        if (t0 + FX_CHUNK < u.count) indices(t0 + FX_CHUNK);
    };
    indices(0);
    fetch(0);
    for (int t0 = 0; t0 < u.count; t0 += FX_CHUNK) {
        const int n = min(FX_CHUNK, u.count - t0), e = en, ey = eyn, pt = ptn;
        const int E = __reduce_max_sync(0xffffffffu, e);
        const int d = E - e;
        bool bad = E >= FX_NAN / 2;  // the same in every warp
        int Eg = 0;
        double gv[3] = {0.0, 0.0, 0.0};
        if (DIAG) {
            int eg = -(1 << 20), nf = 0;
            if (lane < n)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    gv[j] = __ldg(g.gb + 3 * (size_t)pt + j);
                    eg = max(eg, fx_exp(gv[j]));
                    nf |= fx_nonfinite(gv[j]);
                }
            Eg = __reduce_max_sync(0xffffffffu, lane < n ? ey + eg : -(1 << 20));
            bad |= __any_sync(0xffffffffu, nf);
        }
        cp_async_wait();
        __syncthreads();
        if (!bad) {
            if (lane < n) {
                // entry lane's W row, d bits down; the warps share out its groups
#pragma unroll
                for (int m = 0; m < NF / NW; ++m) {
                    const int gr = warp + NW * m;  // column gr / 4, rows of group gr % 4
                    int2 *v = wl + lane * SL + (gr / 4) * RP + (gr % 4) * G;
                    int2 &f = wf[lane * NF + gr];
                    const int2 f0 = f;
                    Fx3 x[4] = {};
#pragma unroll
                    for (int k = 0; k < G; ++k) {
                        const unsigned w = k < 2 ? f0.x : f0.y;
                        x[k] = fx_shift(v[k], k & 1 ? w >> 16 : w & 0xffff, d);
                        v[k] = x[k].v;
                    }
                    if (DIAG && F::XG == 0 && gr % 4 == 3) {
                        // the group of the padding row, whose place gb takes
                        const double gj = gr / 4 == 0 ? gv[0] : gr / 4 == 1 ? gv[1] : gv[2];
                        x[CNP % G] = fx_limbs3(gj, Eg - ey - fx_exp(gj));
                        v[CNP % G] = x[CNP % G].v;
                    }
                    f = make_int2(x[0].f | x[1].f << 16, x[2].f | x[3].f << 16);
                }
                if (F::XG && warp == 0) {
                    Fx3 x[3];
#pragma unroll
                    for (int j = 0; j < 3; ++j) {
                        x[j] = fx_limbs3(gv[j], Eg - ey - fx_exp(gv[j]));
                        sg[lane * 4 + j] = x[j].v;
                    }
                    sg[lane * 4 + 3] = make_int2(x[0].f | x[1].f << 16, x[2].f);
                }
            }
        }
        __syncthreads();
        if (!bad) {
            const int l = tid & 15, rg = l >> 2, cg = l & 3;
            long long hh[TR][TC], hl[TR][TC];
            float cr[TR][TC];
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j) {
                    hh[i][j] = hl[i][j] = 0;
                    cr[i][j] = 0.0f;
                }
#pragma unroll 1
            for (int t = tid >> 4; t < n; t += FV_THREADS / 16) {
                float fg[3] = {};
                if (F::XG) ld_lows<3>(sg + t * 4 + 3, fg);
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    int2 a[TR], b[TC], bw[TR];
                    float fa[TR], fb[TC], fw[TR];
                    ld_limbs<TR>(yl + t * SL + j * RP + rg * TR, a);
                    ld_limbs<TR>(wl + t * SL + j * RP + cg * TR, bw);
                    ld_lows<TR>(yf + t * NF + 4 * j + rg, fa);
                    ld_lows<TR>(wf + t * NF + 4 * j + cg, fw);
#pragma unroll
                    for (int c = 0; c < TR; ++c) {
                        b[c] = bw[c];
                        fb[c] = fw[c];
                    }
                    if (F::XG) {
                        b[TC - 1] = sg[t * 4 + j];
                        fb[TC - 1] = fg[j];
                    }
                    fx_products<TR, TC>(a, fa, b, fb, hh, hl, cr);
                }
            }
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j) {
                    long long H;
                    unsigned L;
                    fx_carry(hh[i][j], hl[i][j], cr[i][j], H, L);
                    H += __shfl_xor_sync(0xffffffffu, H, 16);
                    L += __shfl_xor_sync(0xffffffffu, L, 16);
                    if (lane < 16) {
                        const int to = (warp * RP + rg * TR + i) * CP + (j < TR ? cg * TR + j : RP + cg);
                        sH[to] = H;
                        sL[to] = L;
                    }
                }
        }
        __syncthreads();
        if (t0 + FX_CHUNK < u.count) fetch(t0 + FX_CHUNK);
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            if (at[p] < 0) continue;
            const int r = at[p] / CP, c = at[p] % CP;
            if (bad) {
                acc[p] = fx_plain<CNP>(g, pa + t0, pb + t0, n, r, c, acc[p]);
                continue;
            }
            long long H = 0;
            unsigned L = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                H += sH[w * RP * CP + at[p]];
                L += sL[w * RP * CP + at[p]];
            }
            acc[p] = fx_add(acc[p], H, L, we[p] + (DIAG && c == CNP ? Eg : E));
        }
    }
    double *out = (DIAG ? g.diag_partial : g.off_partial) + (size_t)u.out * NV;
#pragma unroll
    for (int p = 0; p < PER; ++p)
        if (at[p] >= 0) out[tid + FV_THREADS * p] = acc[p];
}

// ---------------------------------------------------------------------------
// U_j = sum A^T A (upper triangle) and ga_j = sum A^T e of a camera unit,
// 11/16-parameter cameras: a Gram matrix of the observations' two rows of
// [A | e], 32 observations at a time, each column cut relative to its largest
// value among them (U_cc holds that value's square, so nothing that counts
// against sqrt(U_rr U_cc) is lost), e as column CNP.  In FP64 the sums were two
// multiply-adds per output and observation on the FP64 pipe.
template <int CNP>
__global__ void __launch_bounds__(FV_THREADS) k_camera_fx(const CamUnit *__restrict__ units,
                                                          const int *__restrict__ cam_obs,
                                                          const double *__restrict__ A, const double *__restrict__ ex,
                                                          double *__restrict__ partial)
{
    constexpr int RP = fx_rows(CNP), TR = RP / 4, NC = CNP + 1, TC = (NC + 3) / 4, CP = 4 * TC, NW = FV_THREADS / 32;
    constexpr int ST = 2 * CP + 2;  // words from observation to observation
    constexpr int NU = CNP * (CNP + 1) / 2, NV = NU + CNP, PER = (NV + FV_THREADS - 1) / FV_THREADS;
    __shared__ __align__(16) long long sa[FX_CHUNK * ST];
    __shared__ float sf[FX_CHUNK * 2 * CP];  // third pieces
    __shared__ long long sH[NW][RP * CP];
    __shared__ unsigned sL[NW][RP * CP];
    __shared__ int s_E[CP];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const CamUnit u = units[blockIdx.x];
    for (int e = tid; e < FX_CHUNK * ST; e += FV_THREADS) sa[e] = 0;  // the padding columns
    for (int e = tid; e < FX_CHUNK * 2 * CP; e += FV_THREADS) sf[e] = 0.0f;
    double acc[PER];
    int at[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        acc[p] = 0.0;
        at[p] = -1;
        const int v = tid + FV_THREADS * p;
        if (v < NU) {  // row-major upper triangle
            int r = 0, c = v;
            while (c >= CNP - r) c -= CNP - r++;
            at[p] = r * CP + r + c;
        } else if (v < NV) {
            at[p] = (v - NU) * CP + CNP;
        }
    }
    // the thread's LD values of a chunk: the next chunk's are on their way while
    // this one is summed, and their observations' indices one chunk before that
    // (52 cameras, two limbs a factor: 99.4 -> 81.9 us; with the third piece 109)
    constexpr int LD = (FX_CHUNK * 2 * NC + FV_THREADS - 1) / FV_THREADS;
    int oi[LD];
    double v[LD];
    auto indices = [&](int t0) {
#pragma unroll
        for (int m = 0; m < LD; ++m) {
            const int t = t0 + (tid + FV_THREADS * m) / (2 * NC);
            oi[m] = t < min(u.count, t0 + FX_CHUNK) ? __ldg(cam_obs + u.begin + t) : -1;
        }
    };
    auto values = [&] {
#pragma unroll
        for (int m = 0; m < LD; ++m) {
            const int k = (tid + FV_THREADS * m) % (2 * NC), i = k / NC, c = k % NC;
            if (oi[m] >= 0) v[m] = c < CNP ? __ldg(A + 2 * CNP * (size_t)oi[m] + i * CNP + c) : __ldg(ex + 2 * (size_t)oi[m] + i);
        }
    };
    indices(0);
    values();
    if (FX_CHUNK < u.count) indices(FX_CHUNK);
    for (int t0 = 0; t0 < u.count; t0 += FX_CHUNK) {
        const int n = min(FX_CHUNK, u.count - t0);
        __syncthreads();  // the last chunk's limbs are read
#pragma unroll
        for (int m = 0; m < LD; ++m) {
            const int e = tid + FV_THREADS * m, t = e / (2 * NC), k = e % (2 * NC);
            if (t < n) sa[t * ST + k / NC * CP + k % NC] = __double_as_longlong(v[m]);
        }
        if (t0 + FX_CHUNK < u.count) {
            values();
            if (t0 + 2 * FX_CHUNK < u.count) indices(t0 + 2 * FX_CHUNK);
        }
        __syncthreads();
        // a warp per column, a lane per observation
        int bad = 0, E[TC];
        double x[TC][2];
#pragma unroll
        for (int q = 0; q < TC; ++q) {
            const int c = warp + NW * q;
            int e = 1;
            x[q][0] = x[q][1] = 0.0;
            if (c < NC && lane < n) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    x[q][i] = __longlong_as_double(sa[lane * ST + i * CP + c]);
                    e = max(e, fx_exp(x[q][i]));
                    bad |= fx_nonfinite(x[q][i]);
                }
            }
            E[q] = __reduce_max_sync(0xffffffffu, e);
            if (lane == 0) s_E[c] = E[q];
        }
        if (__syncthreads_or(bad)) {  // an infinity or a NaN: plain FP64 sums
#pragma unroll
            for (int p = 0; p < PER; ++p)
                if (at[p] >= 0)
                    for (int t = 0; t < n; ++t)
#pragma unroll
                        for (int i = 0; i < 2; ++i)
                            acc[p] = fma(__longlong_as_double(sa[t * ST + i * CP + at[p] / CP]),
                                         __longlong_as_double(sa[t * ST + i * CP + at[p] % CP]), acc[p]);
            continue;
        }
#pragma unroll
        for (int q = 0; q < TC; ++q) {
            const int c = warp + NW * q;
            if (c < NC && lane < n)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const Fx3 v = fx_limbs3(x[q][i], E[q] - fx_exp(x[q][i]));
                    *reinterpret_cast<int2 *>(sa + lane * ST + i * CP + c) = v.v;
                    sf[lane * 2 * CP + i * CP + c] = (float)v.f;
                }
        }
        __syncthreads();
        const int l = tid & 15, r0 = (l >> 2) * TR, c0 = (l & 3) * TC;
        long long hh[TR][TC], hl[TR][TC];
        float cr[TR][TC];
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) {
                hh[i][j] = hl[i][j] = 0;
                cr[i][j] = 0.0f;
            }
        for (int t = tid >> 4; t < n; t += FV_THREADS / 16) {
            const int2 *row = reinterpret_cast<const int2 *>(sa) + t * ST;
            const float *low = sf + t * 2 * CP;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                int2 a[TR], b[TC];
                float fa[TR], fb[TC];
                ld_limbs<TR>(row + i * CP + r0, a);
                ld_limbs<TC>(row + i * CP + c0, b);
#pragma unroll
                for (int k = 0; k < TR; ++k) fa[k] = low[i * CP + r0 + k];
#pragma unroll
                for (int k = 0; k < TC; ++k) fb[k] = low[i * CP + c0 + k];
                fx_products<TR, TC>(a, fa, b, fb, hh, hl, cr);
            }
        }
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) {
                long long H;
                unsigned L;
                fx_carry(hh[i][j], hl[i][j], cr[i][j], H, L);
                H += __shfl_xor_sync(0xffffffffu, H, 16);
                L += __shfl_xor_sync(0xffffffffu, L, 16);
                if (lane < 16) {
                    sH[warp][(r0 + i) * CP + c0 + j] = H;
                    sL[warp][(r0 + i) * CP + c0 + j] = L;
                }
            }
        __syncthreads();
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            if (at[p] < 0) continue;
            long long H = 0;
            unsigned L = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                H += sH[w][at[p]];
                L += sL[w][at[p]];
            }
            acc[p] = fx_add(acc[p], H, L, s_E[at[p] / CP] + s_E[at[p] % CP]);
        }
    }
#pragma unroll
    for (int p = 0; p < PER; ++p)
        if (at[p] >= 0) partial[(size_t)blockIdx.x * NV + tid + FV_THREADS * p] = acc[p];
}

template <int CNP>
void limb_rows_t(const DeviceProblem &d, cudaStream_t s)
{
    constexpr int OB = LR_THREADS / (CNP == 6 ? 2 : 4);
    k_limb_rows<CNP><<<ceil_div(d.no, OB), LR_THREADS, 0, s>>>(d.no, d.obs_pt, d.obs_cam, d.W, d.Vinv, d.U,
                                                               d.Yq, d.Wq, d.fx_ex);
}

template <int CNP, bool DIAG>
void schur_fxv_t(const FxArgs &g, int n, const SchurUnit *units, cudaStream_t s)
{
    constexpr int bytes = FvShape<CNP, DIAG>::BYTES;
    if (n == 0) return;
    if (bytes > 40 * 1024)  // above the default limit (as for k_schur_fx6)
        cudaFuncSetAttribute(k_schur_fxv<CNP, DIAG>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    k_schur_fxv<CNP, DIAG><<<n, FV_THREADS, bytes, s>>>(g, units);
    note_launch(1);
}

}  // namespace

void launch_limb_rows(const DeviceProblem &d, cudaStream_t s)
{
    if (d.no == 0) return;
    if (d.cnp == 6) limb_rows_t<6>(d, s);
    else if (d.cnp == 11) limb_rows_t<11>(d, s);
    else limb_rows_t<16>(d, s);
    note_launch(1);
}

void launch_camera_fx(const DeviceProblem &d, cudaStream_t s)
{
    if (d.n_cam_units == 0) return;
    if (d.cnp == 11) k_camera_fx<11><<<d.n_cam_units, FV_THREADS, 0, s>>>(d.cam_units, d.cam_obs, d.A, d.ex, d.cam_partial);
    else k_camera_fx<16><<<d.n_cam_units, FV_THREADS, 0, s>>>(d.cam_units, d.cam_obs, d.A, d.ex, d.cam_partial);
    note_launch(1);
}

void launch_schur_fx(const DeviceProblem &d, double *diag_partial, cudaStream_t s)
{
    const int low = fx_limb_words(d.cnp);
    FxArgs g{d.pair_a, d.pair_b, d.cam_obs, d.obs_pt, d.Yq, d.Wq, d.Yq + low, d.Wq + low, d.fx_ex, d.W, d.Vinv,
             d.U, d.g + d.N, d.pair_kl, d.schur_partial, diag_partial};
    if (d.cnp == 6) {
        const int ctas = ceil_div(d.n_fx_diag_units, F6_WARPS) + ceil_div(d.n_off_units, F6_WARPS);
        if (ctas == 0) return;
        // above the default limit (an attribute of the kernel on this device; the same value always)
        cudaFuncSetAttribute(k_schur_fx6, cudaFuncAttributeMaxDynamicSharedMemorySize, F6_SMEM);
        k_schur_fx6<<<ctas, 32 * F6_WARPS, F6_SMEM, s>>>(g, d.n_fx_diag_units, d.fx_diag_units, d.n_off_units, d.off_units);
        note_launch(1);
        return;
    }
    if (d.cnp == 11) {
        schur_fxv_t<11, true>(g, d.n_diag_units, d.diag_units, s);
        schur_fxv_t<11, false>(g, d.n_off_units, d.off_units, s);
    } else {
        schur_fxv_t<16, true>(g, d.n_diag_units, d.diag_units, s);
        schur_fxv_t<16, false>(g, d.n_off_units, d.off_units, s);
    }
}

}  // namespace psba
