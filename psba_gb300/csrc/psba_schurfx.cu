// The FP64 Schur complement's products in block fixed point (psba_fixed.h):
// S's off-diagonal blocks sum_i Y_ik W_il^T and the diagonal blocks with ea's
// sums Y gb (compute_S.cl:39-77, compute_ea.cl:21-36).
//
// k_limb_rows forms Y = W V^-1 (compute_Yblks.cl:26-37) and cuts each
// observation's Y and W rows into limbs, relative to the observation's own
// largest value after the camera's row weights (fx_weight).  The sums then
// need one more shift per pair entry, of its W row, to the largest
// eY + eW among the 32 entries taken together: a point close to one camera has a W
// row there 10^4 times the others' and Y rows as much smaller, and only what
// lies 57 bits below the largest product is lost.  Cutting both rows at every
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
// Bound by the FP64 pipe (9 multiply-adds a row) and the ~25 integer
// instructions that cut a value.
constexpr int LR_THREADS = 128;

template <int CNP>
__global__ void __launch_bounds__(LR_THREADS) k_limb_rows(int no, const int *__restrict__ obs_pt,
                                                          const int *__restrict__ obs_cam,
                                                          const double *__restrict__ W,
                                                          const double *__restrict__ Vinv,
                                                          const double *__restrict__ U, int2 *__restrict__ Yq,
                                                          int2 *__restrict__ Wq, int2 *__restrict__ ex)
{
    constexpr int RP = fx_rows(CNP), TPO = CNP == 6 ? 2 : 4, TR = RP / TPO, OB = LR_THREADS / TPO, WORDS = 3 * RP;
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
    for (int a = 0; a < TR; ++a)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int at = t * WORDS + j * RP + q * TR + a;
            sq[0][at] = fx_limbs(y[a][j], ey + rho[a] - fx_exp(y[a][j]));
            sq[1][at] = fx_limbs(w[a][j], ew + rho[a] - fx_exp(w[a][j]));
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

constexpr int F6_WARPS = 4, F6_CTAS = 4;  // resident CTAs per SM: 188 / 173 / 185 us with 3 / 4 / 5 at 88 cameras

// The diagonal units' blocks first (more work per entry), then the pairs'.
__global__ void __launch_bounds__(32 * F6_WARPS, F6_CTAS) k_schur_fx6(FxArgs g, int n_diag, const SchurUnit *__restrict__ diag,
                                                             int n_off, const SchurUnit *__restrict__ off)
{
    __shared__ __align__(16) int2 sy[F6_WARPS][F6_SY], sw[F6_WARPS][F6_SW];
    const int warp = threadIdx.x >> 5, diag_ctas = (n_diag + F6_WARPS - 1) / F6_WARPS;
    if ((int)blockIdx.x < diag_ctas) {
        const int uid = blockIdx.x * F6_WARPS + warp;
        if (uid < n_diag) {
            const SchurUnit u = diag[uid];
            fx6_unit<true, true>(g, u, u.slot, u.slot, sy[warp], sw[warp],
                           [&](int v, int, int, double x) { g.diag_partial[(size_t)u.out * 27 + v] = x; });
        }
    } else {
        const int uid = (blockIdx.x - diag_ctas) * F6_WARPS + warp;
        if (uid < n_off) {
            const SchurUnit u = off[uid];
            fx6_unit<false, true>(g, u, __ldg(g.pair_kl + 2 * u.slot), __ldg(g.pair_kl + 2 * u.slot + 1), sy[warp], sw[warp],
                            [&](int v, int, int, double x) { g.off_partial[(size_t)u.out * 36 + v] = x; });
        }
    }
}

// ---------------------------------------------------------------------------
// 11- and 16-parameter cameras: a CTA of four warps per unit, the same steps;
// half-warps take the entries in turn, 4 x 4 threads with a TR x TC tile each.
constexpr int FV_THREADS = 128;

template <int CNP, bool DIAG>
__global__ void __launch_bounds__(FV_THREADS) k_schur_fxv(FxArgs g, const SchurUnit *__restrict__ units)
{
    constexpr int RP = fx_rows(CNP), TR = RP / 4, TC = DIAG && CNP == 16 ? 5 : TR, CP = 4 * TC;
    constexpr int SY = 3 * RP + 2, SW = 3 * CP + 2, NW = FV_THREADS / 32;
    constexpr int NV = n_out<CNP, DIAG>(), PER = (NV + FV_THREADS - 1) / FV_THREADS;
    constexpr int PIECES = 3 * RP / 2;  // 16-byte pieces of a row
    // this chunk's rows and, where 48 KB hold them (CNP 11), the next one's, which
    // are then under way while this one is summed; else they are fetched after it
    constexpr int NB = 2 * 8 * FX_CHUNK * (SY + SW) + 8 * NW * RP * CP <= 48 * 1024 ? 2 : 1;
    __shared__ __align__(16) int2 sys[NB][FX_CHUNK * SY], sws[NB][FX_CHUNK * SW];
    __shared__ long long st[NW][RP * CP];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const SchurUnit u = units[blockIdx.x];
    const int *pa = DIAG ? g.cam_obs + u.begin : g.pa + u.begin, *pb = DIAG ? pa : g.pb + u.begin;
    for (int e = tid; e < NB * FX_CHUNK * SW; e += FV_THREADS) sws[0][e] = make_int2(0, 0);  // the padding columns
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
    auto fetch = [&](int t0) {
        const int n = min(FX_CHUNK, u.count - t0);
        int2 *sy = sys[(t0 / FX_CHUNK) & (NB - 1)], *sw = sws[(t0 / FX_CHUNK) & (NB - 1)];
#pragma unroll
        for (int m = 0; m < (FX_CHUNK * PIECES + FV_THREADS - 1) / FV_THREADS; ++m) {
            const int p = tid + FV_THREADS * m, t = p / PIECES, part = p % PIECES;
            const int ia = __shfl_sync(0xffffffffu, an, t & 31), ib = DIAG ? ia : __shfl_sync(0xffffffffu, bn, t & 31);
            if (t >= n) continue;
            const int wd = (part / (RP / 2)) * CP + 2 * (part % (RP / 2));
            cp_async16(sy + t * SY + 2 * part, g.Yq + 3 * RP * (size_t)ia + 2 * part);
            cp_async16(sw + t * SW + wd, g.Wq + 3 * RP * (size_t)ib + 2 * part);
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
    __syncthreads();
    fetch(0);
    for (int t0 = 0; t0 < u.count; t0 += FX_CHUNK) {
        const int n = min(FX_CHUNK, u.count - t0), e = en, ey = eyn, pt = ptn;
        int2 *sy = sys[(t0 / FX_CHUNK) & (NB - 1)], *sw = sws[(t0 / FX_CHUNK) & (NB - 1)];
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
        if (NB == 2 && t0 + FX_CHUNK < u.count) fetch(t0 + FX_CHUNK);
        if (!bad) {
            if (lane < n) {
                // entry lane's W row, d bits down; the warps share out the row
#pragma unroll
                for (int m = 0; m < (PIECES + NW - 1) / NW; ++m) {
                    const int part = warp + NW * m;
                    if (part < PIECES) {
                        int4 &x = *reinterpret_cast<int4 *>(sw + lane * SW + (part / (RP / 2)) * CP + 2 * (part % (RP / 2)));
                        const int2 s0 = fx_shift(make_int2(x.x, x.y), d), s1 = fx_shift(make_int2(x.z, x.w), d);
                        x = make_int4(s0.x, s0.y, s1.x, s1.y);
                    }
                }
            }
            if (DIAG) {
                if (CNP < RP) __syncthreads();  // gb takes the place of the padding column that the shift has rewritten
                if (lane < n && warp < 3)
                    sw[lane * SW + warp * CP + CNP] = fx_limbs(gv[warp], Eg - ey - fx_exp(gv[warp]));
            }
        }
        __syncthreads();
        if (!bad) {
            const int l = tid & 15, r0 = (l >> 2) * TR, c0 = (l & 3) * TC;
            long long hh[TR][TC], hl[TR][TC];
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j) hh[i][j] = hl[i][j] = 0;
            for (int t = tid >> 4; t < n; t += FV_THREADS / 16)
                fx_tile<TR, TC, RP, CP>(sy + t * SY + r0, sw + t * SW + c0, hh, hl);
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
                for (int j = 0; j < TC; ++j) {
                    long long T = fx_total(hh[i][j], hl[i][j]);
                    T += __shfl_xor_sync(0xffffffffu, T, 16);
                    if (lane < 16) st[warp][(r0 + i) * CP + c0 + j] = T;
                }
        }
        __syncthreads();
        if (NB == 1 && t0 + FX_CHUNK < u.count) fetch(t0 + FX_CHUNK);
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            if (at[p] < 0) continue;
            const int r = at[p] / CP, c = at[p] % CP;
            if (bad) {
                acc[p] = fx_plain<CNP>(g, pa + t0, pb + t0, n, r, c, acc[p]);
                continue;
            }
            long long T = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) T += st[w][at[p]];
            acc[p] = fx_add(acc[p], T, we[p] + (DIAG && c == CNP ? Eg : E));
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
    __shared__ long long st[NW][RP * CP];
    __shared__ int s_E[CP];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const CamUnit u = units[blockIdx.x];
    for (int e = tid; e < FX_CHUNK * ST; e += FV_THREADS) sa[e] = 0;  // the padding columns
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
    // (52 cameras: 99.4 -> 81.9 us)
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
                for (int i = 0; i < 2; ++i)
                    *reinterpret_cast<int2 *>(sa + lane * ST + i * CP + c) = fx_limbs(x[q][i], E[q] - fx_exp(x[q][i]));
        }
        __syncthreads();
        const int l = tid & 15, r0 = (l >> 2) * TR, c0 = (l & 3) * TC;
        long long hh[TR][TC], hl[TR][TC];
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) hh[i][j] = hl[i][j] = 0;
        for (int t = tid >> 4; t < n; t += FV_THREADS / 16) {
            const int2 *row = reinterpret_cast<const int2 *>(sa) + t * ST;
            fx_tile<TR, TC, CP, CP, 2>(row + r0, row + c0, hh, hl);
        }
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) {
                long long T = fx_total(hh[i][j], hl[i][j]);
                T += __shfl_xor_sync(0xffffffffu, T, 16);
                if (lane < 16) st[warp][(r0 + i) * CP + c0 + j] = T;
            }
        __syncthreads();
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            if (at[p] < 0) continue;
            long long T = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) T += st[w][at[p]];
            acc[p] = fx_add(acc[p], T, s_E[at[p] / CP] + s_E[at[p] % CP]);
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
                                                               reinterpret_cast<int2 *>(d.Y), d.Wq, d.fx_ex);
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
    FxArgs g{d.pair_a, d.pair_b, d.cam_obs, d.obs_pt, reinterpret_cast<const int2 *>(d.Y), d.Wq, d.fx_ex, d.W, d.Vinv,
             d.U, d.g + d.N, d.pair_kl, d.schur_partial, diag_partial};
    if (d.cnp == 6) {
        const int ctas = ceil_div(d.n_fx_diag_units, F6_WARPS) + ceil_div(d.n_off_units, F6_WARPS);
        if (ctas == 0) return;
        k_schur_fx6<<<ctas, 32 * F6_WARPS, 0, s>>>(g, d.n_fx_diag_units, d.fx_diag_units, d.n_off_units, d.off_units);
        note_launch(1);
        return;
    }
    if (d.n_diag_units > 0) {
        if (d.cnp == 11) k_schur_fxv<11, true><<<d.n_diag_units, FV_THREADS, 0, s>>>(g, d.diag_units);
        else k_schur_fxv<16, true><<<d.n_diag_units, FV_THREADS, 0, s>>>(g, d.diag_units);
        note_launch(1);
    }
    if (d.n_off_units > 0) {
        if (d.cnp == 11) k_schur_fxv<11, false><<<d.n_off_units, FV_THREADS, 0, s>>>(g, d.off_units);
        else k_schur_fxv<16, false><<<d.n_off_units, FV_THREADS, 0, s>>>(g, d.off_units);
        note_launch(1);
    }
}

}  // namespace psba
