// lg_batched.cu -- thousands of independent least-squares problems
// min ||A_t x - b_t|| (A_t m_t x n_t, m_t >= n_t, nrhs right-hand sides) in
// up to three launches side by side: a persistent one, and before it one of
// clusters of eight CTAs and one of four for the large instances that would
// outlast the rest (batches of up to 32 instances per SM).
//
// Per instance the algorithm is the reference's least-squares driver
// (least-squares/main_ls_qr3.c:94-119): Householder QR of A, Q^T applied to
// the right-hand sides, R x = (Q^T b)(0:n).  Here each reflector is applied to
// the right-hand sides as soon as it is formed, so no T factor is needed, and
// x overwrites B(0:n, :) (LAPACK dgels convention); A holds V and R on exit.
// CTAs take instances from a device counter (largest first, order prepared on
// the host), so uneven sizes balance without any inter-CTA waiting.
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include <cooperative_groups.h>

#include "lg_house.cuh"
#include "../../include/lila_gpu.h"

namespace lg {
namespace bat {

namespace cg = cooperative_groups;

struct Inst {
    int m, n, lda, ldb;
};

constexpr int NB = 8;    // panel width
constexpr int UW = 4;    // trailing columns of one warp's pass
constexpr int TIERS = 3; // launches by team: clusters of 8 and of 4 CTAs, single CTAs
__host__ __device__ constexpr int tier_ctas(int tier) { return tier == 0 ? 8 : (tier == 1 ? 4 : 1); }
constexpr int MAXG = 34; // column groups exchanged at a time in a cluster (n + nrhs <= 136 in one go)

// Blocked Householder least squares of one instance by a CTA (CS = 1) or by a
// cluster of CS CTAs, each on its own block of rows.
//
// Bound: the FP64 pipe (2 lanes per clock per SM, 64 clocks of a sub-partition
// per warp instruction whatever its lanes carry).  So no FP64 instruction is
// spent on what is not a product of the algorithm where that can be avoided:
//  * a panel of NB columns takes one pass over its rows per column: the pass
//    scales v, updates the panel's later columns and accumulates the next
//    column's products with all panel columns (those before it give T), the
//    eight sums reduced by a transposing butterfly (9 additions per warp, not
//    40); plain sums of squares (no maximum, no division per element), a
//    column whose squares leave the FP64 range is taken again scaled by a
//    power of two;
//  * a warp owns UW trailing columns: W = V^T C over all rows needs no other
//    warp, its 32 sums land one per lane (31 additions, not 160), W := T^T W
//    by shuffles, C -= V W, without a block barrier;
//  * the back substitution runs one warp per right-hand side from registers
//    with the reciprocals of R's diagonal formed beforehand.
// 5,000 uneven instances (m 64..4096, n 8..128): 195 -> 140 ms (920 GFLOP/s,
// 73 % of the DFMA peak); 400 took 47 ms in the previous form (one column's
// dot products per pass over the block, five shuffle additions per accumulator
// in every warp, scaled norms by division, one CTA per instance).
//
// In a cluster each CTA publishes its partial sums in every CTA's shared
// memory (distributed shared memory) and one cluster barrier later all add
// them in CTA order; the trailing W of column group q is added up and
// multiplied by T^T in CTA q mod CS.  Slots alternate with the column so that
// one barrier per column is enough.
template <int TH, int CS>
struct Shared {
    static constexpr int NW = TH / 32;
    double red[NW][NB];          // per warp sums of a column's products
    double x[2][CS][NB];         // per CTA sums, written by every CTA of the cluster
    double piv[2][NB], own[NB];  // the pivot row's panel entries; as its owner has them
    double w[NB], f[NB], g[NB];  // update factors of the panel columns, V^T v
    double T[NB][NB], tau[NB];
    double sc, beta;
    double wb[NW][NB * UW];
    double part[CS > 1 ? MAXG : 1][NB * UW], wt[CS > 1 ? MAXG : 1][NB * UW];
    int emax[CS], nz[CS];
    int exp2, below, redo, idx;
};

__device__ __forceinline__ double *colp(double *A, int lda, double *B, int ldb, int n, int c)
{
    return c < n ? A + (size_t)c * lda : B + (size_t)(c - n) * ldb;
}

template <int CS>
__device__ __forceinline__ void team_sync()
{
    if (CS > 1)
        cg::this_cluster().sync();
    else
        __syncthreads();
}

// `p` of this CTA's shared memory in CTA `rank` of the cluster.
template <int CS, typename V>
__device__ __forceinline__ V *remote(V *p, int rank)
{
    return CS > 1 ? cg::this_cluster().map_shared_rank(p, rank) : p;
}

// Eight sums over the warp: lane l returns sum number l / 4.
__device__ __forceinline__ double reduce8(double (&a)[NB], int lane)
{
#pragma unroll
    for (int h = NB / 2, o = 16; h > 0; h /= 2, o /= 2)
#pragma unroll
        for (int i = 0; i < h; i++) {
            const double send = (lane & o) ? a[i] : a[i + h], keep = (lane & o) ? a[i + h] : a[i];
            a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    double v = a[0];
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}

// 32 sums over the warp: lane l returns sum number l.
__device__ __forceinline__ double reduce32(double (&a)[NB * UW], int lane)
{
#pragma unroll
    for (int h = 16; h > 0; h /= 2)
#pragma unroll
        for (int i = 0; i < h; i++) {
            const double send = (lane & h) ? a[i] : a[i + h], keep = (lane & h) ? a[i + h] : a[i];
            a[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    return a[0];
}

template <int TH, int CS>
struct Solver {
    using S = Shared<TH, CS>;
    static constexpr int NW = TH / 32;
    S &s;
    double *A, *B;
    int m, n, lda, ldb, nrhs;
    int rank, lo, hi;  // this CTA's rows [lo, hi)
    int tid, warp, lane;

    __device__ Solver(S &sh) : s(sh) {}

    // a pivot-row entry; in a cluster the owner's warp 0 passes it on (reflect)
    __device__ __forceinline__ void put_pivot(int par, int c, double v)
    {
        if (CS > 1)
            s.own[c] = v;
        else
            s.piv[par][c] = v;
    }

    // products of column kk of the panel at j0 (rows below its pivot) with the
    // panel's columns; the pivot row into slot par
    __device__ void dots(int j0, int jb, int kk, int par, double (&acc)[NB])
    {
        const int k = j0 + kk;
        const double *P = A + (size_t)j0 * lda, *xk = A + (size_t)k * lda;
#pragma unroll
        for (int c = 0; c < NB; c++) acc[c] = 0.0;
        for (int r = lo + (max(k - lo, 0)) / TH * TH + tid; r < hi; r += TH) {
            if (r < k) continue;
            if (r == k) {
#pragma unroll
                for (int c = 0; c < NB; c++)
                    if (c < jb) put_pivot(par, c, P[(size_t)r + (size_t)c * lda]);
                continue;
            }
            const double y = xk[r];
#pragma unroll
            for (int c = 0; c < NB; c++)
                if (c < jb) acc[c] = fma(y, P[(size_t)r + (size_t)c * lda], acc[c]);
        }
    }

    // the pass of column KK: v, the update of the panel's later columns and
    // the products of column KK + 1
    template <int KK>
    __device__ void pass(int j0, int jb, int par, double (&acc)[NB])
    {
        const int k = j0 + KK;
        double *P = A + (size_t)j0 * lda;
        const double sc = s.sc, beta = s.beta;
        double f[NB];
#pragma unroll
        for (int c = KK + 1; c < NB; c++) f[c] = s.f[c];
        const bool next = KK + 1 < jb;
#pragma unroll
        for (int c = 0; c < NB; c++) acc[c] = 0.0;
        for (int r = lo + (max(k - lo, 0)) / TH * TH + tid; r < hi; r += TH) {
            if (r < k) continue;
            double *row = P + r;
            if (r == k) {
                row[(size_t)KK * lda] = beta;
#pragma unroll
                for (int c = KK + 1; c < NB; c++)
                    if (c < jb) row[(size_t)c * lda] -= s.w[c];
                continue;
            }
            double a[NB];
#pragma unroll
            for (int c = 0; c < NB; c++) a[c] = (c < jb && (next || c == KK)) ? row[(size_t)c * lda] : 0.0;
            const double x = a[KK];
            a[KK] = x * sc;
            row[(size_t)KK * lda] = a[KK];
            if (!next) continue;
#pragma unroll
            for (int c = KK + 1; c < NB; c++)
                if (c < jb) {
                    a[c] = fma(-f[c], x, a[c]);
                    row[(size_t)c * lda] = a[c];
                }
            constexpr int K1 = KK + 1 < NB ? KK + 1 : KK;
            if (r == k + 1) {
#pragma unroll
                for (int c = 0; c < NB; c++)
                    if (c < jb) put_pivot(par, c, a[c]);
            } else {
                const double y = a[K1];
#pragma unroll
                for (int c = 0; c < NB; c++)
                    if (c < jb) acc[c] = fma(y, a[c], acc[c]);
            }
        }
    }

    // sums of acc over the team, then the reflector of column kk (by warp 0);
    // on return (block barrier passed) s.sc, s.beta, s.w, s.f, s.tau[kk], T's
    // column kk and s.redo are set
    __device__ void reflect(int j0, int jb, int kk, int par, double (&acc)[NB], bool scaled)
    {
        // a warp without rows spends no additions
        const double mine = lo + 32 * warp < hi ? reduce8(acc, lane) : 0.0;
        if ((lane & 3) == 0) s.red[warp][lane >> 2] = mine;
        __syncthreads();
        const int c = lane >> 2, q = lane & 3;
        double d = 0.0;
        if (warp == 0) {
            for (int u = q; u < NW; u += 4) d += s.red[u][c];
            d += __shfl_xor_sync(0xffffffffu, d, 1);
            d += __shfl_xor_sync(0xffffffffu, d, 2);
        }
        if (CS > 1) {
            if (warp == 0) {
                const bool owner = j0 + kk >= lo && j0 + kk < hi;
                for (int u = q; u < CS; u += 4) {
                    *remote<CS>(&s.x[par][rank][c], u) = d;
                    if (owner) *remote<CS>(&s.piv[par][c], u) = s.own[c];
                }
            }
            team_sync<CS>();
            if (warp == 0) {
                d = 0.0;
                for (int u = q; u < CS; u += 4) d += s.x[par][u][c];
                d += __shfl_xor_sync(0xffffffffu, d, 1);
                d += __shfl_xor_sync(0xffffffffu, d, 2);
            }
        }
        if (warp == 0) {
            const double p = s.piv[par][c];
            const double alpha = __shfl_sync(0xffffffffu, p, 4 * kk), ss = __shfl_sync(0xffffffffu, d, 4 * kk);
            const int k = j0 + kk;
            const bool last = k == m - 1;
            const bool redo = !scaled && !last && !house_in_range(alpha, ss);
            const Reflector h = house_reflector(alpha, ss, scaled ? s.below != 0 : !last);
            const double sc = h.sc, tau = h.tau;
            // A(k, c) + sc d_c: v^T of the column for c > kk, V^T v for c < kk
            const double e = fma(sc, d, p), w = tau * e;
            if (q == 0) {
                s.w[c] = w;
                s.f[c] = sc * w;
                s.g[c] = e;
            }
            if (lane == 0) {
                s.sc = sc;
                s.beta = scaled ? scalbn(h.beta, s.exp2) : h.beta;
                s.tau[kk] = tau;
                s.redo = redo;
            }
            __syncwarp();
            // T(:, kk) = -tau T(:, 0:kk) g
            if (lane < NB) {
                double t = 0.0;
                for (int u = lane; u < kk; u++) t = fma(s.T[lane][u], s.g[u], t);
                s.T[lane][kk] = lane < kk ? (tau == 0.0 ? 0.0 : -tau * t) : (lane == kk ? tau : 0.0);
            }
        }
        __syncthreads();
    }

    // rare: scale rows k.. of column k by a power of two taken from their
    // largest exponent
    __device__ void rescale(int k)
    {
        double *x = A + (size_t)k * lda;
        if (tid == 0) s.emax[rank] = s.nz[rank] = 0;
        __syncthreads();
        int e = 0, nz = 0;
        for (int r = lo + tid; r < hi; r += TH) {
            if (r < k) continue;
            const int xe = house_exponent(x[r]);
            if (r > k && xe) nz = 1;
            e = max(e, xe);
        }
        atomicMax(&s.emax[rank], e);
        if (nz) atomicOr(&s.nz[rank], 1);
        __syncthreads();
        if (CS > 1) {
            const int te = s.emax[rank], tn = s.nz[rank];
            __syncthreads();
            if (tid < CS) {
                *remote<CS>(&s.emax[rank], tid) = te;
                *remote<CS>(&s.nz[rank], tid) = tn;
            }
            team_sync<CS>();
        }
        int ex = 0, any = 0;
        for (int u = 0; u < CS; u++) {
            ex = max(ex, s.emax[u]);
            any |= s.nz[u];
        }
        const int sh = house_shift(ex);
        for (int r = lo + tid; r < hi; r += TH)
            if (r >= k) x[r] = scalbn(x[r], -sh);
        team_sync<CS>();  // all have read emax and nz
        if (tid == 0) {
            s.exp2 = sh;
            s.below = any;
        }
        __syncthreads();
    }

    template <int KK>
    __device__ void columns(int j0, int jb, double (&acc)[NB])
    {
        if (KK >= jb) return;
        const int k = j0 + KK;
        reflect(j0, jb, KK, k & 1, acc, false);
        if (s.redo) {
            rescale(k);
            dots(j0, jb, KK, k & 1, acc);
            reflect(j0, jb, KK, k & 1, acc, true);
        }
        pass<KK>(j0, jb, (k + 1) & 1, acc);
        if constexpr (KK + 1 < NB) columns<KK + 1>(j0, jb, acc);
    }

    // V(r, 0..7) of the panel: rows above j0 + 7 need the unit lower mask
    __device__ __forceinline__ void load_v(int j0, int jb, int r, bool top, double (&v)[NB])
    {
        const double *row = A + (size_t)j0 * lda + r;
#pragma unroll
        for (int i = 0; i < NB; i++) {
            v[i] = i < jb ? row[(size_t)i * lda] : 0.0;
            if (top) v[i] = (i >= jb || r < j0 + i) ? 0.0 : (r == j0 + i ? 1.0 : v[i]);
        }
    }

    // W(i, j) of one column group over this CTA's rows, sum i UW + j in lane i UW + j
    __device__ double group_w(int j0, int jb, int c0, int nc)
    {
        double acc[NB * UW];
#pragma unroll
        for (int u = 0; u < NB * UW; u++) acc[u] = 0.0;
        const double *col[UW];
#pragma unroll
        for (int j = 0; j < UW; j++) col[j] = colp(A, lda, B, ldb, n, c0 + min(j, nc - 1));
        for (int r0 = lo + max(j0 - lo, 0) / 32 * 32; r0 < hi; r0 += 32) {
            const int r = r0 + lane;
            if (r >= hi) continue;
            double v[NB];
            load_v(j0, jb, r, r0 < j0 + NB, v);
#pragma unroll
            for (int j = 0; j < UW; j++) {
                const double cv = r >= j0 ? col[j][r] : 0.0;
#pragma unroll
                for (int i = 0; i < NB; i++) acc[i * UW + j] = fma(v[i], cv, acc[i * UW + j]);
            }
        }
        __syncwarp();
        return reduce32(acc, lane);
    }

    // T^T W, W's entries one per lane
    __device__ __forceinline__ double times_t(double w)
    {
        const int i = lane / UW, j = lane % UW;
        double x = 0.0;
#pragma unroll
        for (int p = 0; p < NB; p++) x = fma(s.T[p][i], __shfl_sync(0xffffffffu, w, p * UW + j), x);
        return x;
    }

    // C -= V W of one column group over this CTA's rows
    __device__ void group_update(int j0, int jb, int c0, int nc, const double *w)
    {
        double ww[NB * UW];
#pragma unroll
        for (int u = 0; u < NB * UW; u++) ww[u] = w[u];
        double *col[UW];
#pragma unroll
        for (int j = 0; j < UW; j++) col[j] = colp(A, lda, B, ldb, n, c0 + min(j, nc - 1));
        for (int r0 = lo + max(j0 - lo, 0) / 32 * 32; r0 < hi; r0 += 32) {
            const int r = r0 + lane;
            if (r < j0 || r >= hi) continue;
            double v[NB];
            load_v(j0, jb, r, r0 < j0 + NB, v);
#pragma unroll
            for (int j = 0; j < UW; j++) {
                if (j >= nc) break;
                double x = col[j][r];
#pragma unroll
                for (int i = 0; i < NB; i++) x = fma(-v[i], ww[i * UW + j], x);
                col[j][r] = x;
            }
        }
        __syncwarp();
    }

    __device__ void trailing(int j0, int jb)
    {
        const int ncol = n + nrhs, first = j0 + jb, groups = (ncol - first + UW - 1) / UW;
        if (CS == 1) {
            for (int q = warp; q < groups; q += NW) {
                const int c0 = first + UW * q, nc = min(UW, ncol - c0);
                s.wb[warp][lane] = times_t(group_w(j0, jb, c0, nc));
                __syncwarp();
                group_update(j0, jb, c0, nc, s.wb[warp]);
            }
            return;
        }
        for (int g0 = 0; g0 < groups; g0 += MAXG) {
            const int ng = min(MAXG, groups - g0);
            for (int q = warp; q < ng; q += NW) {
                const int c0 = first + UW * (g0 + q);
                s.part[q][lane] = group_w(j0, jb, c0, min(UW, ncol - c0));
            }
            team_sync<CS>();
            for (int q = rank + CS * warp; q < ng; q += CS * NW) {
                double w = 0.0;
#pragma unroll
                for (int u = 0; u < CS; u++) w += *remote<CS>(&s.part[q][lane], u);
                w = times_t(w);
#pragma unroll
                for (int u = 0; u < CS; u++) *remote<CS>(&s.wt[q][lane], u) = w;
            }
            team_sync<CS>();
            for (int q = warp; q < ng; q += NW) {
                const int c0 = first + UW * (g0 + q);
                group_update(j0, jb, c0, min(UW, ncol - c0), s.wt[q]);
            }
        }
    }

    // R x = y for one right-hand side by one warp, x over B(0:n, j); returns
    // k + 1 of the smallest k with a zero or non-finite R(k, k), 0 if none
    __device__ int back_substitute(int j)
    {
        double *b = B + (size_t)j * ldb;
        int bad = 0;
        // row blocks of 32 from the bottom: the block's own triangle from
        // registers, then the rows above it
        for (int q = (n - 1) / 32; q >= 0; q--) {
            const int r = 32 * q + lane, nk = min(32, n - 32 * q);
            const bool on = r < n;
            double y = on ? b[r] : 0.0;
            const double d = on ? A[(size_t)r + (size_t)r * lda] : 1.0;
            const double ad = fabs(d);
            const bool plain = ad >= 1e-290 && ad <= 1e290;
            const double inv = plain ? copysign(rcp_nr(ad), d) : 1.0 / d;
            const bool is_bad = d == 0.0 || !isfinite(d);
            const unsigned bm = __ballot_sync(0xffffffffu, on && is_bad);
            if (bm) bad = 32 * q + __ffs(bm);
            double col = nk > 1 && r < n ? A[(size_t)r + (size_t)(32 * q + nk - 1) * lda] : 0.0;
            for (int k = nk - 1; k >= 0; k--) {
                const double cur = col;
                if (k > 0 && on) col = A[(size_t)r + (size_t)(32 * q + k - 1) * lda];
                // lane k: y / d, the quotient corrected by one residual step (an
                // infinite one has none)
                double x = y * inv;
                if (plain && bexp_of(x) != 0x7FF)
                    x = fma(fma(-x, d, y), inv, x);
                else
                    x = is_bad ? NAN : y / d;
                x = __shfl_sync(0xffffffffu, x, k);
                if (lane == k) y = x;
                if (lane < k) y = fma(-cur, x, y);
            }
            if (on) b[r] = y;
            // rows above: b(0:32 q) -= R(0:32 q, block) x
            for (int rr = lane; rr < 32 * q; rr += 32) {
                double z = b[rr];
                for (int k = 0; k < nk; k++) {
                    // x_k from lane k: every lane takes part (32 q is a multiple of 32)
                    const double xk = __shfl_sync(0xffffffffu, y, k);
                    z = fma(-A[(size_t)rr + (size_t)(32 * q + k) * lda], xk, z);
                }
                b[rr] = z;
            }
            __syncwarp();
        }
        return bad;
    }

    __device__ void solve(const Inst &I, double *a, double *b, int nr, int *info)
    {
        m = I.m;
        n = I.n;
        lda = I.lda;
        ldb = I.ldb;
        A = a;
        B = b;
        nrhs = nr;
        const int rows = ((m + CS - 1) / CS + 31) / 32 * 32;  // whole warps, coalesced
        lo = min(m, rank * rows);
        hi = min(m, lo + rows);
        for (int j0 = 0; j0 < n; j0 += NB) {
            const int jb = min(NB, n - j0);
            for (int u = tid; u < NB * NB; u += TH) s.T[u / NB][u % NB] = 0.0;
            double acc[NB];
            dots(j0, jb, 0, j0 & 1, acc);
            columns<0>(j0, jb, acc);
            __syncthreads();
            trailing(j0, jb);
            __syncthreads();
        }
        team_sync<CS>();
        for (int j = rank + CS * warp; j < nrhs; j += CS * NW) {
            const int bad = back_substitute(j);
            if (j == 0 && lane == 0) *info = bad;
        }
        team_sync<CS>();
    }
};

// Persistent: teams of CS CTAs take instances order[*from .. *to) from the
// tier's counter, largest first (null: from the first, to the last).  A tier's
// launch starts beside the one
// before it (programmatic launch) and ends after it.
template <int TH, int CS>
__global__ void __launch_bounds__(TH, TH <= 256 ? 512 / TH : 1)
    k_gels(int count, int nrhs, const Inst *inst, double *const *Aptr, double *const *Bptr, const int *order,
           int *counter, const int *from, const int *to, int *info)
{
    __shared__ Shared<TH, CS> s;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    Solver<TH, CS> v(s);
    v.tid = threadIdx.x;
    v.warp = threadIdx.x >> 5;
    v.lane = threadIdx.x & 31;
    v.rank = CS > 1 ? (int)cg::this_cluster().block_rank() : 0;
    const int first = from ? *from : 0, last = to ? *to : count;
    if (CS > 1) team_sync<CS>();  // every CTA of the cluster runs before its memory is written
    for (;;) {
        if (v.rank == 0 && threadIdx.x == 0) {
            const int idx = atomicAdd(counter, 1);
            for (int u = 0; u < CS; u++) *remote<CS>(&s.idx, u) = idx;
        }
        team_sync<CS>();
        const int at = first + s.idx;
        if (at >= last) break;
        const int t = order[at];
        v.solve(inst[t], Aptr[t], Bptr[t], nrhs, info + t);
    }
    if (CS > 1) team_sync<CS>();  // no CTA leaves while its memory may still be written
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace bat

struct BatchMeta {
    int count, nrhs;
    bat::Inst *inst;
    double **Aptr, **Bptr;
    int *order, *counter;  // counter[0 .. TIERS): the launches' queues, then TIERS + 1 bounds of their instances
};

constexpr double kTier8 = 1.0, kTier4 = 0.16;  // of the work per SM

static long long batch_bytes(int count)
{
    return 256 + (long long)count * ((long long)sizeof(bat::Inst) + 2 * sizeof(double *) + sizeof(int)) + 256;
}

static BatchMeta carve_meta(void *work, int count)
{
    BatchMeta b;
    uint8_t *p = (uint8_t *)work;
    b.counter = (int *)p;
    p += 256;
    b.inst = (bat::Inst *)p;
    p += (size_t)count * sizeof(bat::Inst);
    b.Aptr = (double **)p;
    p += (size_t)count * sizeof(double *);
    b.Bptr = (double **)p;
    p += (size_t)count * sizeof(double *);
    b.order = (int *)p;
    b.count = count;
    b.nrhs = 0;
    return b;
}

// launch configuration (threads, CTAs per SM), chosen by lila_gpu_gels_autotune
static int g_gels_threads = 256, g_gels_per_sm = 2;

// One tier's launch over order[*from .. *to): as many clusters as are resident
// at once (the next tier starts beside it only when all its CTAs have
// started).  False (nothing enqueued) when the device refuses such clusters.
template <int TH, int CS>
static bool launch_tier(const BatchMeta &b, int nrhs, int *info, int tier, const int *from, const int *to, bool beside)
{
    cudaLaunchAttribute at[2];
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(sm_count() * g_gels_per_sm);
    cfg.blockDim = dim3(TH);
    cfg.stream = stream();
    cfg.attrs = at;
    if (CS > 1) {
        at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        at[cfg.numAttrs++].val.clusterDim = {CS, 1, 1};
        int n = 0;
        cfg.gridDim = dim3(CS);
        if (cudaOccupancyMaxActiveClusters(&n, bat::k_gels<TH, CS>, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            return false;
        }
        cfg.gridDim = dim3(CS * n);
    }
    if (beside) {
        at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cudaLaunchKernelEx(&cfg, bat::k_gels<TH, CS>, b.count, nrhs, (const bat::Inst *)b.inst,
                           (double *const *)b.Aptr, (double *const *)b.Bptr, (const int *)b.order, b.counter + tier,
                           from, to, info) == cudaSuccess)
        return true;
    if (CS > 1) cudaGetLastError();  // the single CTAs take these instances
    return false;
}

static void launch_gels(const BatchMeta &b, int nrhs, int *info)
{
    cudaMemsetAsync(b.counter, 0, bat::TIERS * sizeof(int), stream());
    trace_break();
    trace_begin();
    // the instances that would keep one SM busy long after the others go to
    // clusters (prepare bounds the tiers; none in a batch of over 32 per SM;
    // always CTAs of 256 threads); what a refused cluster launch leaves goes
    // to the single CTAs
    const int *bound = b.counter + bat::TIERS, *from = nullptr;
    if (b.count <= 32 * sm_count() && launch_tier<256, 8>(b, nrhs, info, 0, bound, bound + 1, false)) {
        from = bound + 1;
        note_launch("gels_batched_clusters");
        trace_begin();
        if (launch_tier<256, 4>(b, nrhs, info, 1, bound + 1, bound + 2, true)) {
            from = bound + 2;
            note_launch("gels_batched_clusters");
            trace_begin();
        }
    }
    const bool beside = from != nullptr;
    if (g_gels_threads == 128)
        launch_tier<128, 1>(b, nrhs, info, 2, from, nullptr, beside);
    else if (g_gels_threads == 512)
        launch_tier<512, 1>(b, nrhs, info, 2, from, nullptr, beside);
    else
        launch_tier<256, 1>(b, nrhs, info, 2, from, nullptr, beside);
    note_launch("gels_batched");
}

}  // namespace lg

using namespace lg;

extern "C" {

long long lila_query_dgels_batched(int count) { return batch_bytes(count); }

int lila_dgels_batched_prepare(int count, const int *m, const int *n, int nrhs, double *const *A, const int *lda,
                               double *const *B, const int *ldb, void *work, long long work_bytes)
{
    if (count < 0) return -1;
    if (nrhs < 1 || nrhs > 8) return -4;
    if (work_bytes < batch_bytes(count)) return -10;
    std::vector<bat::Inst> inst(count);
    std::vector<int> order(count);
    for (int t = 0; t < count; t++) {
        if (m[t] < n[t] || n[t] < 1) return -2;
        if (lda[t] < m[t] || ldb[t] < m[t]) return -6;
        inst[t] = bat::Inst{m[t], n[t], lda[t], ldb[t]};
        order[t] = t;
    }
    // largest work first: m n^2
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return (double)inst[a].m * inst[a].n * inst[a].n > (double)inst[b].m * inst[b].n * inst[b].n;
    });
    // An instance's team: a cluster of 8 CTAs when its FMAs exceed what the
    // whole batch spread over all SMs leaves for one, a cluster of 4 from a
    // sixth of that, provided its columns carry enough rows to pay for the
    // cluster's exchange; smaller teams waste fewer FP64 slots on reductions.
    // 500 instances (m up to 4096, n up to 128; 10 ms of FMAs on all SMs): one
    // CTA each 34 ms (the largest takes that long alone), clusters of 8 or one
    // 20.6 ms, these tiers 18.7 ms; 60 instances 33.6, 4.6 and 5.2 ms.  An
    // eighth instead of a sixth gains 5 % there and loses 4 % at 2,000
    // instances, a quarter the other way round.
    auto fma = [&](int t) { return (double)inst[t].m * inst[t].n * (inst[t].n + 2.0 * nrhs); };
    double total = 0.0;
    for (int t = 0; t < count; t++) total += fma(t);
    const double share[bat::TIERS - 1] = {kTier8, kTier4};
    int head[2 * bat::TIERS + 1] = {};
    for (int tier = 0, at = 0; tier < bat::TIERS - 1; tier++) {
        while (at < count && fma(order[at]) > share[tier] * total / sm_count() &&
               (long long)inst[order[at]].m * inst[order[at]].n >= 16384)
            at++;
        head[bat::TIERS + tier + 1] = at;
    }
    head[2 * bat::TIERS] = count;
    BatchMeta b = carve_meta(work, count);
    cudaStream_t st = stream();
    cudaMemcpyAsync(b.counter, head, sizeof head, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b.inst, inst.data(), sizeof(bat::Inst) * count, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b.Aptr, A, sizeof(double *) * count, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b.Bptr, B, sizeof(double *) * count, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b.order, order.data(), sizeof(int) * count, cudaMemcpyHostToDevice, st);
    cudaStreamSynchronize(st);  // host vectors go out of scope
    return 0;
}

// Up to three launches over the prepared instances (stream-capturable).
int lila_dgels_batched_run(int count, int nrhs, void *work, int *info)
{
    if (count <= 0) return 0;
    BatchMeta b = carve_meta(work, count);
    launch_gels(b, nrhs, info);
    return 0;
}

// Captures lila_dgels_batched_run into a CUDA graph (on a private stream) and
// returns its executable handle; lila_gpu_graph_launch replays it on the
// library stream.
void *lila_dgels_batched_graph(int count, int nrhs, void *work, int *info)
{
    cudaStream_t cap;
    if (cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
    void *prev = lila_gpu_get_stream();
    lila_gpu_set_stream(cap);
    cudaGraph_t g = nullptr;
    cudaGraphExec_t ge = nullptr;
    if (cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
        lila_dgels_batched_run(count, nrhs, work, info);
        if (cudaStreamEndCapture(cap, &g) == cudaSuccess && g) {
            if (cudaGraphInstantiate(&ge, g, 0) != cudaSuccess) ge = nullptr;
            cudaGraphDestroy(g);
        }
    }
    lila_gpu_set_stream(prev);
    cudaStreamDestroy(cap);
    return (void *)ge;
}

int lila_gpu_graph_launch(void *exec)
{
    if (!exec) return -1;
    return cudaGraphLaunch((cudaGraphExec_t)exec, lg::stream()) == cudaSuccess ? 0 : -2;
}

int lila_gpu_graph_destroy(void *exec)
{
    if (!exec) return 0;
    return cudaGraphExecDestroy((cudaGraphExec_t)exec) == cudaSuccess ? 0 : -1;
}

// Times (threads, CTAs per SM) candidates on the prepared batch (its A and B
// are overwritten: call on a scratch copy) and keeps the fastest for later
// launches.  Returns threads * 100 + CTAs per SM.
int lila_gpu_gels_autotune(int count, int nrhs, void *work, int *info, double *const *Asave, double *const *A,
                           const long long *bytesA, double *const *Bsave, double *const *B, const long long *bytesB)
{
    const int cand_th[3] = {128, 256, 512};
    const int cand_sm[3] = {1, 2, 4};
    float best = 1e30f;
    int bth = 256, bsm = 2;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    for (int a = 0; a < 3; a++)
        for (int c = 0; c < 3; c++) {
            if (cand_th[a] * cand_sm[c] > 1024) continue;
            for (int t = 0; t < count; t++) {
                cudaMemcpyAsync(A[t], Asave[t], bytesA[t], cudaMemcpyDeviceToDevice, lg::stream());
                cudaMemcpyAsync(B[t], Bsave[t], bytesB[t], cudaMemcpyDeviceToDevice, lg::stream());
            }
            g_gels_threads = cand_th[a];
            g_gels_per_sm = cand_sm[c];
            cudaEventRecord(e0, lg::stream());
            lila_dgels_batched_run(count, nrhs, work, info);
            cudaEventRecord(e1, lg::stream());
            cudaEventSynchronize(e1);
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (ms < best) {
                best = ms;
                bth = cand_th[a];
                bsm = cand_sm[c];
            }
        }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    g_gels_threads = bth;
    g_gels_per_sm = bsm;
    return bth * 100 + bsm;
}

int lila_gpu_gels_config(int threads, int per_sm)
{
    if (threads != 128 && threads != 256 && threads != 512) return -1;
    if (per_sm < 1 || per_sm > 8) return -2;
    g_gels_threads = threads;
    g_gels_per_sm = per_sm;
    return 0;
}

}  // extern "C"
