// lg_tsqr.cu -- TSQR reduction tree for the tall-skinny leaf (FP64).
//
// The reference's only tree QR is LAPACK's dlatsqr with Q built by dlarfb /
// dtprfb sweeps (tsqr/main_test_tsqr.c:234-395); its lila leaf for tall
// panels is Cholesky QR + Householder reconstruction
// (lila-c/lila_dgeqrf_w03_mt_hr.c:3-33).  This leaf combines the two: a
// row-block Householder tree gives an orthonormal Q and R at any condition
// number, and the reconstruction tile loop of the Cholesky leaf turns them
// into the w03 outputs (V and S R in A, T tiles, Q S in Q).
//
//   level 0: the ml x n block is cut into row blocks of mb rows (mb <= 256);
//            one CTA factors a block in shared memory (Householder, LAPACK
//            dlarfg convention), writes its reflectors over the block of A
//            and its n x n R into the level-1 stack.
//   level l: the stack of R factors is cut into groups of `arity` R's (their
//            rows interleaved, see RowMap); each group is factored the same way (reflectors in place in the
//            stack), its R going to the next stack, until one R remains.
//   Q:       from I_n at the root, each level applies its groups'
//            reflectors to [Q_parent_block; 0] (backward sweep); level 0
//            writes Q.
#include "lg_house.cuh"
#include "../../include/lila_gpu.h"

namespace lg {

void hr_tiles(int m, int n, int i, int mt, double *A, int lda, double *T, int ldt, double *Q, int ldq,
              double *S, double *work, long long lwork);

namespace tsqr {

// Both kernels hold a block (rows x n <= 16,384 entries) with its columns in
// registers: column c belongs to LG lanes, lane g holds rows g, g + LG, ..
// (RPL of them), so a dot product or an update is RPL FMAs per lane against
// one shared column, with only log2(LG) shuffle additions; the FP64 pipe (64
// clocks of a sub-partition per warp instruction) is what bounds them.  Against
// the block in shared memory, one warp per column and a five-step shuffle
// reduction per dot product, 131,072 x 32 (512 blocks of 256 rows, groups of 4):
// QR 2.10 -> 0.82 ms, backward sweep 1.96 -> 0.80 ms; the 512 blocks run with
// the FP64 pipe 73 % (QR) and 95 % (sweep) busy, the five levels above them are
// bound by their columns' chains (91 us per level, 150 before the interleaving
// and 35 us per sweep).
constexpr int CH = 4;  // registers skipped together

// f(u, v[u LG]) for the registers u of the first `left` rows, in chunks of CH;
// a chunk's loads are issued before the previous chunk's FMAs, so that the
// branch between them does not expose the shared-memory latency.
template <int LG, int RPL, typename F>
__device__ __forceinline__ void run_chunks(const double *v, int left, F &&f)
{
    double cur[CH], nxt[CH];
#pragma unroll
    for (int i = 0; i < CH; i++) cur[i] = v[i * LG];
#pragma unroll
    for (int q = 0; q < RPL; q += CH) {
        if (q * LG >= left) break;
#pragma unroll
        for (int i = 0; i < CH; i++) nxt[i] = q + CH < RPL ? v[(q + CH + i) * LG] : 0.0;
#pragma unroll
        for (int i = 0; i < CH; i++) f(q + i, cur[i]);
#pragma unroll
        for (int i = 0; i < CH; i++) cur[i] = nxt[i];
    }
}

// Where row r of block b's n x n factor stands in the next level's stack: the
// factors of a group are interleaved row by row, so that column k of the group
// has its entries (a upper triangles of n rows) in its first a (k + 1) rows and
// the kernels run over those only: n^3 FMAs per group of four instead of 3.7
// n^3, 3 n^2 instead of 7 n^2 per column of the backward sweep.
struct RowMap {
    int n, arity, blocks;
    __device__ __forceinline__ int row(int b, int r) const
    {
        const int group = b / arity, first = group * arity;
        return first * n + r * min(arity, blocks - first) + (b - first);
    }
};

// Householder QR of rows [b rb, min((b+1) rb, total)) of X (ld ldx, n columns;
// stacked: interleaved triangles, see RowMap).  Reflectors overwrite the block
// below its diagonal, tau goes to tau[b n + k], R (n x n upper, zero below; rows
// past a short block are zero) to the rows that `map` gives in R (ld ldr).
//
// Per column: its group leaves it in shared memory (zero down to the pivot), one
// barrier, every later group's dot product and the reflector, one barrier, the
// updates x_c -= tau sc (A(k, c) + sc d_c) u with u the column and alpha - beta
// in its pivot row.  Register 0 always holds the LG rows around the pivot: when
// all of them are done they go out (R above the diagonal, the scaled column
// below it) and the registers move up by one, so neither the pivot nor the rows
// above it have to be picked out of the registers (353 instructions per warp and
// column, most of them selects, before that: one warp per sub-partition has
// nothing to hide them behind).
template <int LG, int RPL>
__global__ void __launch_bounds__(512) k_block_qr(double *X, int ldx, int total, int rb, int n, bool stacked,
                                                  double *tau, double *R, int ldr, RowMap map)
{
    __shared__ double xk[2][RPL * LG];
    __shared__ double s_sc, s_f, s_u;
    __shared__ int s_redo;
    const int b = blockIdx.x, r0 = b * rb, rows = min(rb, total - r0);
    const int lane = threadIdx.x & 31, c = threadIdx.x / LG, g = threadIdx.x % LG;
    const bool mine = c < n;
    const int wc1 = (threadIdx.x / 32 + 1) * (32 / LG);  // one past the warp's last column
    double x[RPL];
    double *col = X + r0 + (size_t)(mine ? c : 0) * ldx;
#pragma unroll
    for (int u = 0; u < RPL; u++) x[u] = (mine && g + u * LG < rows) ? col[g + u * LG] : 0.0;
    double my_tau = 0.0, my_sc = 0.0, my_beta = 0.0;
    const int kmax = min(rows, n), tri = stacked ? rows / n : rows;
    int base = 0;  // row of lane 0's register 0
    // register 0 goes out (R on and above the diagonal, the reflector below
    // it) and the others move up
    double *rout = R + map.row(b, 0) + (size_t)(mine ? c : 0) * ldr;
    const int rstep = map.row(b, 1) - map.row(b, 0);
    auto next = [&] {
        const int r = base + g;
        if (mine && r < n) rout[r * rstep] = r >= rows ? 0.0 : (r < c ? x[0] : (r == c ? my_beta : 0.0));
        if (mine && r > c && r < rows) col[r] = x[0] * my_sc;
#pragma unroll
        for (int u = 0; u + 1 < RPL; u++) x[u] = x[u + 1];
        x[RPL - 1] = 0.0;
        base += LG;
    };
    for (int k = 0; k < kmax; k++) {
        const int left = min(rows, tri * (k + 1)) - base;  // column k is zero from row base + left
        double *xs = xk[k & 1];
        auto leave = [&] {
            xs[g] = base + g > k ? x[0] : 0.0;
#pragma unroll
            for (int u = 1; u < RPL; u++) xs[g + u * LG] = x[u];
        };
        if (c == k) leave();
        __syncthreads();
        double d = 0.0, p = 0.0;
        // dot products with column k, the pivot row's entry, and (column k's
        // group) the reflector
        auto products = [&](bool scaled, bool below, int sh) {
            d = 0.0;
            run_chunks<LG, RPL>(xs + g, left, [&](int u, double v) { d = fma(v, x[u], d); });
            d = group_sum<LG>(d);
            p = __shfl_sync(0xffffffffu, x[0], (lane & ~(LG - 1)) | (k - base));
            if (c == k) {
                const bool last = k == rows - 1;
                const Reflector h = house_reflector(p, d, scaled ? below : !last);
                my_tau = h.tau;
                my_sc = h.sc;
                my_beta = scaled ? scalbn(h.beta, sh) : h.beta;
                if (g == 0) {
                    s_sc = h.sc;
                    s_f = h.tau * h.sc;
                    s_u = h.u;
                    s_redo = !scaled && !last && !house_in_range(p, d);
                }
            }
        };
        if (wc1 > k) products(false, false, 0);
        __syncthreads();
        if (s_redo) {  // rare: the column again, scaled by a power of two
            __syncthreads();
            int e = 0, nz = 0;
            if (wc1 > k) {
#pragma unroll
                for (int u = 0; u < RPL; u++)
                    if (base + g + u * LG >= k) {
                        const int xe = house_exponent(x[u]);
                        e = max(e, xe);
                        if (base + g + u * LG > k) nz |= xe;
                    }
#pragma unroll
                for (int o = LG / 2; o > 0; o >>= 1) {
                    e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
                    nz |= __shfl_xor_sync(0xffffffffu, nz, o);
                }
            }
            const int sh = house_shift(e);
            if (c == k) {
#pragma unroll
                for (int u = 0; u < RPL; u++)
                    if (base + g + u * LG >= k) x[u] = scalbn(x[u], -sh);
                leave();
            }
            __syncthreads();
            if (wc1 > k) products(true, nz != 0, sh);
            __syncthreads();
        }
        if (c > k) {
            // a zero column has s_f = 0 and an all-zero xs: nothing changes
            const double f = s_f * fma(s_sc, d, p), pivot = s_u;
            const bool at = base + g == k;
            run_chunks<LG, RPL>(xs + g, left, [&](int u, double v) { x[u] = fma(-f, u == 0 && at ? pivot : v, x[u]); });
        }
        if (k - base == LG - 1) next();
    }
    if (mine && g == 0) tau[(size_t)b * n + c] = my_tau;
    const int end = max(rows, n);
#pragma unroll 1
    while (base < end) next();
}

// Leading dimension of the reflectors in shared memory (whole chunks of rows).
__host__ __device__ constexpr int block_ld(int rb, int lg) { return (rb + CH * lg - 1) / (CH * lg) * (CH * lg); }

// Y = H_0 ... H_{n-1} [Qin_b; 0] for block b (rows as in k_block_qr), written
// to Y rows [b rb, ...) (ld ldy).  Qin_b = the rows of Qin that `map` gives.  The
// reflectors stand in shared memory (unit lower, zeros above); every lane group
// runs its column through all of them without a block barrier, so the columns
// of a block may be split over blockIdx.y (nc each) where there are few blocks.
template <int LG, int RPL>
__global__ void __launch_bounds__(512) k_block_apply(const double *X, int ldx, int total, int rb, int n, bool stacked,
                                                     const double *tau, const double *Qin, int ldqin, RowMap map,
                                                     double *Y, int ldy, int nc)
{
    extern __shared__ double V[];  // rows x n, then tau
    const int b = blockIdx.x, r0 = b * rb, rows = min(rb, total - r0);
    const int kmax = min(rows, n), ld = block_ld(rb, LG);
    double *s_tau = V + (size_t)ld * n;
    for (int k = threadIdx.x >> 5; k < kmax; k += blockDim.x >> 5)
#pragma unroll 4
        for (int r = threadIdx.x & 31; r < ld; r += 32)
            V[r + (size_t)k * ld] = r > k && r < rows ? X[(size_t)(r0 + r) + (size_t)k * ldx] : (r == k ? 1.0 : 0.0);
    for (int k = threadIdx.x; k < kmax; k += blockDim.x) s_tau[k] = tau[(size_t)b * n + k];
    const int g = threadIdx.x % LG, c = blockIdx.y * nc + threadIdx.x / LG;
    const bool mine = threadIdx.x / LG < nc && c < n;
    double y[RPL];
#pragma unroll
    for (int u = 0; u < RPL; u++) {
        const int r = g + u * LG;
        y[u] = mine && r < n && r < rows ? Qin[(size_t)map.row(b, r) + (size_t)c * ldqin] : 0.0;
    }
    __syncthreads();
    const int tri = stacked ? rows / n : rows;
    for (int k = kmax - 1; k >= 0; k--) {
        const double tk = s_tau[k];
        if (tk == 0.0) continue;
        const int top = min(rows, tri * (k + 1));
        const double *v = V + (size_t)k * ld + g;
        double d = 0.0;
#pragma unroll
        for (int q = 0; q < RPL; q += CH) {
            if (q * LG >= top || (q + CH) * LG <= k) continue;
#pragma unroll
            for (int u = q; u < q + CH; u++) d = fma(v[u * LG], y[u], d);
        }
        const double f = tk * group_sum<LG>(d);
#pragma unroll
        for (int q = 0; q < RPL; q += CH) {
            if (q * LG >= top || (q + CH) * LG <= k) continue;
#pragma unroll
            for (int u = q; u < q + CH; u++) y[u] = fma(-f, v[u * LG], y[u]);
        }
    }
    if (!mine) return;
#pragma unroll
    for (int u = 0; u < RPL; u++) {
        const int r = g + u * LG;
        if (r < rows) Y[(size_t)(r0 + r) + (size_t)c * ldy] = y[u];
    }
}

static int round32(int t) { return (t + 31) / 32 * 32; }

template <int LG, int RPL>
struct Lanes {
    static constexpr int lg = LG, rpl = RPL;
};

// Lanes per column and rows per lane for blocks of rb rows whose n columns
// have at most 512 threads (rb n <= 16,384): 32 rows per lane spend the fewest
// shuffle additions; 64 (with spills) hold the wide blocks in between.  The
// backward sweep of few blocks (its columns split over CTAs) is bound by its
// chain of dot products instead and takes 16 lanes where 32 columns or fewer
// leave the threads for them (a 128 x 32 block: 40 us against 77 on 4 lanes).
template <typename F>
static void with_lanes(int rb, int n, bool chain, F &&f)
{
    if (chain && n <= 32 && rb <= 128)
        f(Lanes<16, 8>{});
    else if (chain && n <= 32 && rb <= 256)
        f(Lanes<16, 16>{});
    else if (rb <= 128)
        f(Lanes<4, 32>{});
    else if (rb <= 256 && n <= 64)
        f(Lanes<8, 32>{});
    else if (rb <= 256)
        f(Lanes<4, 64>{});
    else if (n <= 32)
        f(Lanes<16, 32>{});
    else
        f(Lanes<8, 64>{});
}

static void launch_qr(int nb, double *X, int ldx, int total, int rb, int n, bool stacked, double *tau, double *R,
                      int ldr, RowMap map)
{
    with_lanes(rb, n, false, [&](auto l) {
        constexpr int lg = decltype(l)::lg, rpl = decltype(l)::rpl;
        k_block_qr<lg, rpl><<<nb, round32(n * lg), 0, stream()>>>(X, ldx, total, rb, n, stacked, tau, R, ldr, map);
    });
}

static void launch_apply(int nb, const double *X, int ldx, int total, int rb, int n, bool stacked, const double *tau,
                         const double *Qin, int ldqin, RowMap map, double *Y, int ldy)
{
    // few blocks: their columns over about two CTAs per SM, 32 at most each
    int split = 2 * sm_count() / nb;
    if (split < 1) split = 1;
    int nc = (n + split - 1) / split;
    nc = (nc + 7) / 8 * 8;
    with_lanes(rb, nc, split > 1, [&](auto l) {
        constexpr int lg = decltype(l)::lg, rpl = decltype(l)::rpl;
        const size_t smem = ((size_t)block_ld(rb, lg) * n + n) * sizeof(double);
        cudaFuncSetAttribute(k_block_apply<lg, rpl>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k_block_apply<lg, rpl><<<dim3(nb, (n + nc - 1) / nc), round32(nc * lg), smem, stream()>>>(
            X, ldx, total, rb, n, stacked, tau, Qin, ldqin, map, Y, ldy, nc);
    });
}

}  // namespace tsqr

struct TsqrPlan {
    int levels, arity;
    int nb[32];     // blocks at each level
    int rows[32];   // rows of the matrix factored at each level
    int rb[32];     // rows per block at each level
    long long stack_off[32], tau_off[32];
    long long ybuf, yalt, ylen, total;
};

static TsqrPlan plan_tsqr(int ml, int n, int mb, int arity)
{
    TsqrPlan p{};
    p.arity = arity;
    long long off = 0;
    int rows = ml, rb = mb, lvl = 0;
    while (true) {
        p.rows[lvl] = rows;
        p.rb[lvl] = rb;
        p.nb[lvl] = (rows + rb - 1) / rb;
        p.tau_off[lvl] = off;
        off += (long long)p.nb[lvl] * n;
        p.stack_off[lvl] = off;  // R stack produced by this level
        off += (long long)p.nb[lvl] * n * n;
        if (p.nb[lvl] == 1) break;
        rows = p.nb[lvl] * n;
        rb = arity * n;
        lvl++;
    }
    p.levels = lvl + 1;
    long long ymax = n;  // root identity rows
    for (int l = 1; l < p.levels; l++) ymax = ymax > p.rows[l] ? ymax : p.rows[l];
    p.ylen = ymax * n;
    p.ybuf = off;
    off += p.ylen;
    p.yalt = off;
    off += p.ylen;
    p.total = off + 64;  // + S
    return p;
}

long long need_tsqr(int ml, int n, int mb, int arity)
{
    TsqrPlan p = plan_tsqr(ml, n, mb, arity);
    return p.total;
}

// Q (ml x n, ldq) and R (upper n x n into A's leaf top, lda) of A(i:m, i:i+n).
static void tsqr_qr(int ml, int n, double *Aii, int lda, double *Qii, int ldq, double *work, const TsqrPlan &p)
{
    // upward: factor level by level
    for (int l = 0; l < p.levels; l++) {
        double *X = l == 0 ? Aii : work + p.stack_off[l - 1];
        const int ldx = l == 0 ? lda : p.rows[l];
        double *Rs = work + p.stack_off[l];
        const int ldr = p.nb[l] * n;
        trace_begin();
        tsqr::launch_qr(p.nb[l], X, ldx, p.rows[l], p.rb[l], n, l > 0, work + p.tau_off[l], Rs, ldr,
                        tsqr::RowMap{n, p.arity, p.nb[l]});
        note_launch("tsqr_block_qr");
    }
    // downward: Qin of the top level is I_n
    double *yin = work + p.ybuf, *yout = work + p.yalt;
    set2d(n, n, 0.0, 1.0, yin, n, 0);
    int ldin = n;
    for (int l = p.levels - 1; l >= 0; l--) {
        const double *X = l == 0 ? Aii : work + p.stack_off[l - 1];
        const int ldx = l == 0 ? lda : p.rows[l];
        double *Y = l == 0 ? Qii : yout;
        const int ldy = l == 0 ? ldq : p.rows[l];
        trace_begin();
        tsqr::launch_apply(p.nb[l], X, ldx, p.rows[l], p.rb[l], n, l > 0, work + p.tau_off[l], yin, ldin,
                           tsqr::RowMap{n, p.arity, p.nb[l]}, Y, ldy);
        note_launch("tsqr_block_apply");
        double *t = yin;
        yin = yout;
        yout = t;
        ldin = ldy;
    }
    // R: the root's factor, written over the leaf's top block only now that
    // level 0's reflectors stored there have been applied
    copy2d(n, n, work + p.stack_off[p.levels - 1], n, Aii, lda);
}

// Autotuned (mb, arity) per (ml, n), cached: candidates are timed once on the
// caller's own data shape with a scratch copy.
struct TuneEntry {
    int ml, n, mb, arity;
};
static TuneEntry g_tune[16];
static int g_ntune = 0;

static bool tune_lookup(int ml, int n, int &mb, int &arity)
{
    for (int k = 0; k < g_ntune; k++)
        if (g_tune[k].ml == ml && g_tune[k].n == n) {
            mb = g_tune[k].mb;
            arity = g_tune[k].arity;
            return true;
        }
    return false;
}

}  // namespace lg

using namespace lg;

extern "C" {

int lila_query_dgeqrf_w03_tsqr(int mb, int arity, int m, int n, int i, int mt)
{
    if (mb <= 0) mb = 256;
    if (arity <= 0) arity = 4;
    if (n <= 0 || m - i < 1) return 1;
    long long v = need_tsqr(m - i, n, mb, arity);
    // after the tree: S (global index, i + n) and the reconstruction tile
    // loop's scratch ((j - i) * n_tile <= n * n doubles)
    const long long hr = (long long)i + n + (long long)n * n;
    if (hr > v) v = hr;
    return v > 0x7fffffffLL ? 0x7fffffff : (int)v;
}

int lila_dgeqrf_w03_tsqr(int mb, int arity, int m, int n, int i, int mt, double *A, int lda, double *T, int ldt,
                         double *Q, int ldq, double *work, int lwork)
{
    if (mb < 0 || mb > 256) return -1;
    if (arity < 0 || arity > 16) return -2;
    if (m < 0) return -3;
    if (n < 0 || i + n > m) return -4;
    if (i < 0) return -5;
    if (mt <= 0) return -6;
    if (lda < (m > 1 ? m : 1)) return -8;
    if (ldt < mt) return -10;
    if (ldq < (m > 1 ? m : 1)) return -12;
    if (n == 0) return 0;
    if (mb == 0 || arity == 0) {
        int tmb = 256, tar = 4;
        if (tune_lookup(m - i, n, tmb, tar)) {
            if (mb == 0) mb = tmb;
            if (arity == 0) arity = tar;
        } else {
            if (mb == 0) mb = 256;
            if (arity == 0) arity = 4;
        }
    }
    if (mb < n) mb = n;
    if ((long long)mb * n > 16384 || (long long)arity * n * n > 16384 || arity < 2) return -2;
    if (lwork < lila_query_dgeqrf_w03_tsqr(mb, arity, m, n, i, mt)) return -14;
    const int ml = m - i;
    double *Aii = A + i + (size_t)i * lda;
    double *Qii = Q + i + (size_t)i * ldq;
    TsqrPlan p = plan_tsqr(ml, n, mb, arity);
    tsqr_qr(ml, n, Aii, lda, Qii, ldq, work, p);
    double *S = work;  // tree buffers are dead once Q is formed
    // S is indexed by the global column: S + i holds the leaf's signs
    hr_tiles(m, n, i, mt, A, lda, T, ldt, Q, ldq, S, work + i + n, (long long)lwork - (i + n));
    return 0;
}

// Times the (mb, arity) candidates on a matrix of the given shape (scratch
// buffers are the caller's: A, Q, T and work of the usual sizes) and caches the
// fastest for later calls with mb = arity = 0.  Returns the chosen mb * 100 + arity.
int lila_gpu_tsqr_autotune(int m, int n, double *A, int lda, double *T, int ldt, double *Q, int ldq,
                           double *work, int lwork)
{
    const int cand_mb[2] = {128, 256};
    const int cand_ar[2] = {2, 4};
    float best = 1e30f;
    int bmb = 256, bar = 4;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    for (int a = 0; a < 2; a++)
        for (int b = 0; b < 2; b++) {
            const int mb = cand_mb[a] < n ? n : cand_mb[a];
            if ((long long)mb * n > 16384 || (long long)cand_ar[b] * n * n > 16384) continue;
            if (lwork < lila_query_dgeqrf_w03_tsqr(mb, cand_ar[b], m, n, 0, ldt)) continue;
            cudaEventRecord(e0, stream());
            TsqrPlan p = plan_tsqr(m, n, mb, cand_ar[b]);
            tsqr_qr(m, n, A, lda, Q, ldq, work, p);
            cudaEventRecord(e1, stream());
            cudaEventSynchronize(e1);
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            if (ms < best) {
                best = ms;
                bmb = mb;
                bar = cand_ar[b];
            }
        }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (g_ntune < 16) g_tune[g_ntune++] = TuneEntry{m, n, bmb, bar};
    (void)T;
    return bmb * 100 + bar;
}

}  // extern "C"
