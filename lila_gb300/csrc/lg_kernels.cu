// lg_kernels.cu -- FP64 building blocks of the GB300 LILA library.
//
// These are the general, shape-agnostic kernels every lila routine can be
// expressed with (masked GEMM with split-K, small triangular solves, one-CTA
// Cholesky / sign-choice LU / Householder generation).  FP64 on GB300 runs
// at roughly 2 DFMA per clock per SM, so one resident warp already keeps an
// SM's FP64 pipe busy: the kernels below are sized to put work on all 152
// SMs (split-K for the tall reductions) rather than for register reuse.
#include <math.h>

#include "lg_common.cuh"

namespace lg {

// ---------------------------------------------------------------------------
// masked GEMM
// ---------------------------------------------------------------------------
__device__ __forceinline__ double op_elem(const Operand &X, int r, int k)
{
    int sr = X.trans == NT ? r : k;
    int sc = X.trans == NT ? k : r;
    switch (X.mask) {
    case M_UNIT_LOWER:
        if (sr < sc) return 0.0;
        if (sr == sc) return 1.0;
        break;
    case M_UPPER:
        if (sr > sc) return 0.0;
        break;
    case M_LOWER:
        if (sr < sc) return 0.0;
        break;
    case M_UNIT_UPPER:
        if (sr > sc) return 0.0;
        if (sr == sc) return 1.0;
        break;
    default:
        break;
    }
    return X.p[(size_t)sr + (size_t)sc * (size_t)X.ld];
}

__device__ __forceinline__ void epilogue_store(double v, int r, int c, double *C, int ldc,
                                               const GemmEpi &e)
{
    if (e.upper_only && r > c) return;
    double out = e.alpha * v;
    if (e.add_diag && r == c) out += 1.0;
    size_t off = (size_t)r + (size_t)c * (size_t)ldc;
    if (e.beta != 0.0 && r >= e.zero_rows) out += e.beta * C[off];
    C[off] = out;
}

// One BM x BN output tile over the K slice blockIdx.z.  The FP64 pipe retires
// two FMA per clock per SM, so a tile's FMAs, not its loads, bound it: the
// micro-tile is only as large as the load count asks (1 x 1 at 16 x 16), the
// next K step's operands are loaded into registers while the current one is
// multiplied from a two-stage shared buffer (one block barrier per step), and
// what the masks or the matrix's edge leave out is not multiplied:
// the K range is cut to what triangular masks leave nonzero, a warp whose
// outputs all lie outside the matrix skips its FMAs, and with upper_only a
// tile below the diagonal returns at once.  (So a NaN or an infinity opposite a
// mask's zeros does not spread past its tile, as in BLAS' dtrmm.)  Against the same kernel on fixed
// 32 x 32 tiles with 256-deep K slices and unpipelined loads: the 617 products
// of a 1413 x 692 recursive QR 22.1 -> 7.1 ms, the 133 of 4000 x 1000 (tiles
// of 256) 21.6 -> 16.1 ms, the upper 64 x 64 Gram of 262,144 rows 2.23 -> 1.4 ms.
// PARTS (K > 512, slices of more than SUB terms): an output is summed in chains
// of SUB terms, whose rounding errors grow with the chain.  The plan takes K
// slices for their time alone, so without this the Gram's chains were as long as
// 4,384 and a product of 520 terms was one chain.  Errors with it against
// double-double products (root mean square, of the largest entry): Q^T C of 520 x
// 600 x 33 in tiles of 32 7.7e-17 -> 6.5e-17, 775 x 1852 x 40 6.4e-17 -> 5.4e-17,
// the Cholesky QR leaf of 262,144 x 64 a quarter less (A 3.3e-16 -> 2.4e-16).  It
// costs nothing (3.62 and 3.63 ms, 1413 x 692 8.09 ms both), as the additions are
// outside the loop over K steps; inside it the leaf took 3.66 ms.  Chains of 160
// take 3.634 ms, of 256 lose what is gained at 520 terms.  The 64 x 64 tile has
// no registers for a second set of sums; it is taken where the output has many
// tiles.
constexpr int SUB = 192;
constexpr int UPPER_TILES = 2;  // upper_only on a grid without the tiles below the diagonal
template <int BM, int BN, int BK, int TM, int TN, bool PARTS>
__global__ void __launch_bounds__(256)
    k_gemm(int M, int N, int K, int kchunk, Operand A, Operand B, double *C, int ldc, GemmEpi e,
           double *part)
{
    constexpr int RT = BM / TM, CT = BN / TN;  // threads along rows, columns
    constexpr int NTH = 256;
    static_assert(RT * CT == NTH, "one micro-tile per thread");
    constexpr int LA = BM * BK / NTH, LB = BN * BK / NTH;
    // rows of As and Bs are padded to an odd length: a transposed operand's
    // stores walk a column of them
    __shared__ double As[2][BK][BM + 1];
    __shared__ double Bs[2][BK][BN + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // a warp covers 8 row threads x 4 column threads
    const int tr = (lane & 7) + 8 * (warp % (RT / 8)), tc = (lane >> 3) + 4 * (warp / (RT / 8));
    int bx = blockIdx.x, by = blockIdx.y;
    if (e.upper_only == UPPER_TILES)  // blockIdx.x counts the tiles on and above the diagonal
        for (by = 0; bx > by; by++) bx -= by + 1;
    const int row0 = bx * BM, col0 = by * BN;
    if (e.upper_only && row0 > col0 + BN - 1) return;
    int kbeg = blockIdx.z * kchunk;
    int kend = min(K, kbeg + kchunk);
    // rows [row0, row0 + BM) of op(A) and columns [col0, col0 + BN) of op(B)
    // are zero outside [kbeg, kend) under the stored operand's triangular mask
    {
        const bool lowA = A.mask == M_UNIT_LOWER || A.mask == M_LOWER, upA = A.mask == M_UPPER || A.mask == M_UNIT_UPPER;
        const bool lowB = B.mask == M_UNIT_LOWER || B.mask == M_LOWER, upB = B.mask == M_UPPER || B.mask == M_UNIT_UPPER;
        if (A.trans == NT ? lowA : upA) kend = min(kend, row0 + BM);
        if (A.trans == NT ? upA : lowA) kbeg = max(kbeg, row0 / BK * BK);
        if (B.trans == NT ? upB : lowB) kend = min(kend, col0 + BN);
        if (B.trans == NT ? lowB : upB) kbeg = max(kbeg, col0 / BK * BK);
    }
    const bool live = row0 + 8 * (warp % (RT / 8)) < M && col0 + 4 * (warp / (RT / 8)) < N;
    double acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0.0;

    // PARTS: sums of SUB terms, added up in `sum`
    double sum[PARTS ? TM : 1][PARTS ? TN : 1] = {};
    auto add_up = [&] {
        if constexpr (PARTS) {
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) {
                    sum[i][j] += acc[i][j];
                    acc[i][j] = 0.0;
                }
        }
    };

    double ra[LA], rb[LB];
    chain_wait();
    auto load = [&](int k0) {
#pragma unroll
        for (int u = 0; u < LA; u++) {
            const int idx = tid + u * NTH;
            const int r = A.trans == NT ? idx % BM : idx / BK, k = A.trans == NT ? idx / BM : idx % BK;
            const int gr = row0 + r, gk = k0 + k;
            ra[u] = (gr < M && gk < kend) ? op_elem(A, gr, gk) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < LB; u++) {
            const int idx = tid + u * NTH;
            const int c = B.trans == NT ? idx / BK : idx % BN, k = B.trans == NT ? idx % BK : idx / BN;
            const int gc = col0 + c, gk = k0 + k;
            rb[u] = (gc < N && gk < kend) ? op_elem(B, gk, gc) : 0.0;
        }
    };
    load(kbeg);
    int buf = 0;
    int kstop = PARTS ? min(kend, kbeg + SUB) : kend;
    for (int k0 = kbeg;;) {
        for (; k0 < kstop; k0 += BK, buf ^= 1) {
#pragma unroll
            for (int u = 0; u < LA; u++) {
                const int idx = tid + u * NTH;
                if (A.trans == NT)
                    As[buf][idx / BM][idx % BM] = ra[u];
                else
                    As[buf][idx % BK][idx / BK] = ra[u];
            }
#pragma unroll
            for (int u = 0; u < LB; u++) {
                const int idx = tid + u * NTH;
                if (B.trans == NT)
                    Bs[buf][idx % BK][idx / BK] = rb[u];
                else
                    Bs[buf][idx / BN][idx % BN] = rb[u];
            }
            // one barrier per step: the buffer written two steps later was last
            // read before the barrier of the step between
            __syncthreads();
            if (k0 + BK < kend) load(k0 + BK);
            if (live) {
#pragma unroll
                for (int k = 0; k < BK; k++) {
                    double a[TM], b[TN];
#pragma unroll
                    for (int i = 0; i < TM; i++) a[i] = As[buf][k][tr + i * RT];
#pragma unroll
                    for (int j = 0; j < TN; j++) b[j] = Bs[buf][k][tc + j * CT];
#pragma unroll
                    for (int i = 0; i < TM; i++)
#pragma unroll
                        for (int j = 0; j < TN; j++) acc[i][j] = fma(a[i], b[j], acc[i][j]);
                }
            }
        }
        if (!PARTS) break;
        add_up();
        if (kstop == kend) break;
        kstop = min(kend, kstop + SUB);
    }
    if constexpr (PARTS) {
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int j = 0; j < TN; j++) acc[i][j] = sum[i][j];
    }
    // Only now: blocks of the next kernel let in before would be placed where
    // this one's blocks have left room, several to some SMs and none to others
    // (opened at the start: 4000 x 1000 in tiles of 256 21.4 -> 22.3 ms).
    chain_open();
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) {
            int r = row0 + tr + i * RT, c = col0 + tc + j * CT;
            if (r < M && c < N) {
                if (part)
                    part[(size_t)blockIdx.z * M * N + (size_t)r + (size_t)c * M] = acc[i][j];
                else
                    epilogue_store(acc[i][j], r, c, C, ldc, e);
            }
        }
}

// Sum of the K slices' partial products in slice order, eight loads in flight
// per thread.
__global__ void k_splitk_reduce(int M, int N, int splits, const double *part, double *C, int ldc,
                                GemmEpi e)
{
    chain_wait();
    size_t total = (size_t)M * N;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int r = (int)(idx % M), c = (int)(idx / M);
        if (e.upper_only && r > c) continue;
        double s = 0.0;
        const double *p = part + idx;
        int z = 0;
        for (; z + 8 <= splits; z += 8, p += 8 * total) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = p[(size_t)u * total];
#pragma unroll
            for (int u = 0; u < 8; u++) s += v[u];
        }
        for (; z < splits; z++, p += total) s += *p;
        epilogue_store(s, r, c, C, ldc, e);
    }
    chain_open();
}

// SM count of the current device (queried once), for the grid heuristics
static int num_sm() { return sm_count(); }

static inline int ceil_div(long long a, long long b) { return (int)((a + b - 1) / b); }

// Tile and K split of an M x N x K product.  The FP64 pipe makes every tile
// cost BM BN kchunk / 2 clocks of its SM whatever its shape, so the plan with
// the least work on the busiest SM wins: small tiles and fine K slices when
// the output has few tiles, 64 x 64 when it has many (fewer loads).  A split
// adds the reduction launch (~3 us) and splits / 2 clocks per output.  A 32 x
// 350 x 1316 product: 106 us on 66 CTAs (32 x 32 x 264, FP64 pipe 21 % busy),
// its FMAs take 23 us on all SMs.
struct GemmPlan {
    int tile, splits, kchunk;
};

static GemmPlan gemm_plan(int M, int N, int K, long long part_len, bool upper_only)
{
    const double sm = num_sm();
    const long long out = (long long)M * N;
    GemmPlan best{32, 1, K > 0 ? K : 1};
    double best_t = 1e300;
    for (int t = 16; t <= 64; t *= 2) {
        if (t < 64 && ceil_div(N, t) > 65535) continue;  // grid.y limit
        double tiles = (double)ceil_div(M, t) * ceil_div(N, t);
        // upper_only: the tiles below the diagonal return at once
        if (upper_only) {
            const double d = ceil_div(M < N ? M : N, t);
            tiles -= 0.5 * d * (d - 1) + (double)(ceil_div(M, t) - d) * ceil_div(N, t);
        }
        // clocks of a K step of 16 that the pipe does not cover: the loads'
        // latency and the barrier
        const double step = 700.0;
        for (int per = 0; per <= 8; per++) {
            // about `per` CTAs on every SM (0: no split)
            int splits = 1;
            if (per > 0) {
                splits = (int)(per * sm / tiles);
                if (splits > K / 32) splits = K / 32;
                if (splits > 128) splits = 128;
                if ((long long)splits * out > part_len) splits = (int)(part_len / out);
                if (splits < 2) continue;
            }
            int kchunk = K > 0 ? K : 1;
            if (splits > 1) {
                kchunk = ceil_div(ceil_div(K, splits), 16) * 16;
                splits = ceil_div(K, kchunk);
                if (splits < 2) continue;
            }
            const double ctas = tiles * splits;
            const double waves = ceil(ctas / sm);
            const double work = 0.5 * t * t * kchunk;  // clocks of one CTA alone on its SM
            // co-resident CTAs share the pipe and hide each other's latency
            const double lat = ceil_div(kchunk, 16) * step + 1500.0;
            double time = waves * work > lat ? waves * work + 0.1 * lat : lat + 0.1 * waves * work;
            if (splits > 1) time += 6000.0 + 0.5 * splits * out / sm;
            // wider tiles load less per FMA: prefer them when equal
            time *= t == 16 ? 1.06 : (t == 32 ? 1.02 : 1.0);
            if (time < best_t) {
                best_t = time;
                best = GemmPlan{t, splits, kchunk};
            }
        }
    }
    return best;
}

int gemm_splits(int M, int N, int K, long long part_len)
{
    if (M <= 0 || N <= 0) return 1;
    return gemm_plan(M, N, K, part_len, false).splits;
}

// Whether a product goes to the tensor cores in split precision: its time there
// (38 us of latency, then 0.175 us per million multiply-adds of the padded 128 x
// 64 x 32 tiles) against the FP64 pipe's (10 us, 1.65 us per million).  128 x 64
// x 3000: FP64 54 us, split 44; 3000 x 128 x 64: 50 and 35; 128 x 256 x 512: 38
// and 44; 128 x 3000 x 6000: 3,795 and 403.  Thin tiles count at their padded
// size: 34 reflectors on 6000 x 3000 take the FP64 pipe 970 us.
static bool split_pays(int M, int N, int K)
{
    if (precision() != 1 || M < 16 || N < 16 || K < 16) return false;
    const double fma = 1e-6 * M * N * K;
    const double pad = 1e-6 * (128.0 * ceil_div(M, 128)) * (64.0 * ceil_div(N, 64)) * (32.0 * ceil_div(K, 32));
    return 38.0 + 0.175 * pad < 10.0 + 1.65 * fma;
}

// The product, or (more than one slice returned) its K slices in `part`.
static int gemm_parts(int M, int N, int K, Operand A, Operand B, double *C, int ldc, const GemmEpi &e, double *part,
                      long long part_len, const char *tag)
{
    const GemmPlan p = gemm_plan(M, N, K, part ? part_len : 0, e.upper_only != 0);
    double *pp = p.splits > 1 ? part : nullptr;
    dim3 grid(ceil_div(M, p.tile), ceil_div(N, p.tile), p.splits);
    GemmEpi ek = e;
    if (e.upper_only && M == N) {
        // no CTAs for the tiles below the diagonal: they would leave the others
        // unevenly spread (64 x 64 x 262,144: 1.42 ms with them, 1.14 without)
        ek.upper_only = UPPER_TILES;
        grid.x = grid.x * (grid.x + 1) / 2;
        grid.y = 1;
    }
    trace_begin();
    auto launch = [&](auto kern) { launch_chained(kern, grid, 256, 0, M, N, K, p.kchunk, A, B, C, ldc, ek, pp); };
    const bool parts = K > 512 && p.kchunk > SUB;
    if (p.tile == 64)
        launch(k_gemm<64, 64, 16, 4, 4, false>);
    else if (p.tile == 32)
        parts ? launch(k_gemm<32, 32, 16, 2, 2, true>) : launch(k_gemm<32, 32, 16, 2, 2, false>);
    else
        parts ? launch(k_gemm<16, 16, 32, 1, 1, true>) : launch(k_gemm<16, 16, 32, 1, 1, false>);
    note_launch(tag);
    return p.splits;
}

void gemm(int M, int N, int K, Operand A, Operand B, double *C, int ldc, const GemmEpi &e,
          double *part, long long part_len, const char *tag)
{
    if (M <= 0 || N <= 0) return;
    if (split_pays(M, N, K)) {
        ozgemm(M, N, K, A, B, C, ldc, e, part, part_len, "ozgemm");
        return;
    }
    const int splits = gemm_parts(M, N, K, A, B, C, ldc, e, part, part_len, tag);
    if (splits > 1) splitk_reduce(M, N, splits, part, C, ldc, e);
}

// The sum of the product's K slices (vb x n partials; one: the product itself)
// times op(T), `cols` columns per CTA: the sums go to shared memory, next to
// T's triangle.  Latency bounds it (rounds of loads, then chains of up to vb
// FMAs), so a CTA has one column while there are SMs for it, four at most, and
// threads left over share an output's terms.  One launch instead of the slices'
// reduction and a product of its own (6.5 + 5.8 us at 32 x 31, 6.8 us together).
constexpr int RT_COLS = 4, RT_NTH = 128;
__global__ void __launch_bounds__(RT_NTH) k_reduce_times_tri(int vb, int n, int cols, int splits, const double *part,
                                                             const double *T, int ldt, int trans, double *W2)
{
    __shared__ double Ws[64 * RT_COLS], Ts[64 * 65], Ps[2][RT_NTH];
    chain_wait();
    const int c0 = blockIdx.x * cols, nc = min(cols, n - c0), out = vb * nc;
    const size_t total = (size_t)vb * n;
    // T's triangle as rows of op(T): Ts[r + k * 65] = op(T)(r, k)
    {
        const int r = threadIdx.x & 63;
#pragma unroll 4
        for (int c = threadIdx.x >> 6; c < vb; c += RT_NTH / 64)
            if (r <= c) Ts[trans == TR ? c + r * 65 : r + c * 65] = T[(size_t)r + (size_t)c * ldt];
    }
    // P threads to an output, part p of its terms each; with P > 1 there is
    // one round of outputs
    const int P = out <= RT_NTH / 4 ? 4 : out <= RT_NTH / 2 ? 2 : 1;
    const int me = P == 1 ? threadIdx.x : threadIdx.x % (RT_NTH / P), p = P == 1 ? 0 : threadIdx.x / (RT_NTH / P);
    auto combine = [&](double *ps, double s) {
        if (P == 1) return s;
        ps[threadIdx.x] = s;
        __syncthreads();
        if (p) return 0.0;
        s += ps[me + RT_NTH / P];
        if (P == 4) s += ps[me + 2 * (RT_NTH / 4)] + ps[me + 3 * (RT_NTH / 4)];
        return s;
    };
    for (int idx = me; idx < (P == 1 ? out : RT_NTH / P); idx += RT_NTH / P) {
        double s = 0.0;
        if (idx < out) {
            const double *q = part + (size_t)c0 * vb + idx;
            int z = p;
            for (; z + 3 * P < splits; z += 4 * P) {
                double v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) v[u] = q[(size_t)(z + u * P) * total];
                s += (v[0] + v[1]) + (v[2] + v[3]);
            }
            for (; z < splits; z += P) s += q[(size_t)z * total];
        }
        s = combine(Ps[0], s);
        if (p == 0 && idx < out) Ws[idx] = s;
    }
    __syncthreads();
    chain_open();
    for (int idx = me; idx < (P == 1 ? out : RT_NTH / P); idx += RT_NTH / P) {
        double s = 0.0;
        if (idx < out) {
            const int r = idx % vb, c = idx / vb;
            const int k0 = trans == TR ? 0 : r, k1 = trans == TR ? r + 1 : vb;
            for (int k = k0 + p; k < k1; k += P) s = fma(Ts[r + k * 65], Ws[k + c * vb], s);
        }
        s = combine(Ps[1], s);
        if (p == 0 && idx < out) W2[(size_t)c0 * vb + idx] = s;
    }
}

void gemm_times_tri(int vb, int n, int K, Operand A, Operand B, const double *T, int ldt, int trans, double *W1,
                    double *W2, double *part, long long part_len)
{
    if (vb <= 0 || n <= 0) return;
    GemmEpi e;
    if (vb > 64 || split_pays(vb, n, K)) {
        gemm(vb, n, K, A, B, W1, vb, e, part, part_len);
        gemm(vb, n, vb, opnd(T, ldt, trans, M_UPPER), opnd(W1, vb), W2, vb, e);
        return;
    }
    const int splits = gemm_parts(vb, n, K, A, B, W1, vb, e, part, part_len, "gemm");
    trace_begin();
    const int cols = std::min(ceil_div(n, num_sm()), RT_COLS);
    launch_chained(k_reduce_times_tri, dim3(ceil_div(n, cols)), 128, 0, vb, n, cols, splits, splits > 1 ? part : W1, T,
                   ldt, trans, W2);
    note_launch("reduce_times_tri");
}

void splitk_reduce(int M, int N, int splits, const double *part, double *C, int ldc, const GemmEpi &e)
{
    long long total = (long long)M * N;
    int blocks = ceil_div(total, 128);
    if (blocks > 8 * num_sm()) blocks = 8 * num_sm();
    trace_begin();
    launch_chained(k_splitk_reduce, dim3(blocks), 128, 0, M, N, splits, part, C, ldc, e);
    note_launch("splitk_reduce");
}

// ---------------------------------------------------------------------------
// element-wise helpers
// ---------------------------------------------------------------------------
__global__ void k_copy2d(int m, int n, const double *src, int lds, double *dst, int ldd)
{
    chain_wait();
    size_t total = (size_t)m * n;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        size_t r = idx % m, c = idx / m;
        dst[r + c * ldd] = src[r + c * lds];
    }
}

__global__ void k_copy2d_trans(int m, int n, const double *src, int lds, double *dst, int ldd)
{
    size_t total = (size_t)m * n;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        size_t r = idx % m, c = idx / m;
        dst[c + r * ldd] = src[r + c * lds];
    }
}

__global__ void k_set2d(int m, int n, double off, double diag, double *dst, int ldd, int uplo)
{
    chain_wait();
    size_t total = (size_t)m * n;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        int r = (int)(idx % m), c = (int)(idx / m);
        if (uplo == 1 && r > c) continue;
        if (uplo == 2 && r <= c) continue;
        dst[(size_t)r + (size_t)c * ldd] = (r == c) ? diag : off;
    }
}

__global__ void k_sub2d(int m, int n, const double *src, int lds, double *dst, int ldd)
{
    size_t total = (size_t)m * n;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        size_t r = idx % m, c = idx / m;
        dst[r + c * ldd] -= src[r + c * lds];
    }
}

__global__ void k_flip_rows(int nrows, int n, const double *S, double *X, int ldx, int upper)
{
    chain_wait();
    size_t total = (size_t)nrows * n;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        int k = (int)(idx % nrows), c = (int)(idx / nrows);
        if (upper && c < k) continue;
        if (S[k] == -1.0) X[(size_t)k + (size_t)c * ldx] = -X[(size_t)k + (size_t)c * ldx];
    }
}

__global__ void k_flip_cols(int m, int n, const double *S, double *X, int ldx)
{
    chain_wait();
    size_t total = (size_t)m * n;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        size_t r = idx % m, c = idx / m;
        if (S[c] == -1.0) X[r + c * ldx] = -X[r + c * ldx];
    }
}

static inline int ew_blocks(long long total)
{
    int b = ceil_div(total > 0 ? total : 1, 256);
    return b > 8 * num_sm() ? 8 * num_sm() : b;
}

void copy2d(int m, int n, const double *src, int lds, double *dst, int ldd)
{
    if (m <= 0 || n <= 0) return;
    trace_begin();
    launch_chained(k_copy2d, dim3(ew_blocks((long long)m * n)), 256, 0, m, n, src, lds, dst, ldd);
    note_launch("copy2d");
}
void copy2d_trans(int m, int n, const double *src, int lds, double *dst, int ldd)
{
    if (m <= 0 || n <= 0) return;
    k_copy2d_trans<<<ew_blocks((long long)m * n), 256, 0, stream()>>>(m, n, src, lds, dst, ldd);
    note_launch("copy2d_trans");
}
void set2d(int m, int n, double off, double diag, double *dst, int ldd, int uplo)
{
    if (m <= 0 || n <= 0) return;
    launch_chained(k_set2d, dim3(ew_blocks((long long)m * n)), 256, 0, m, n, off, diag, dst, ldd, uplo);
    note_launch("set2d");
}
void sub2d(int m, int n, const double *src, int lds, double *dst, int ldd)
{
    if (m <= 0 || n <= 0) return;
    k_sub2d<<<ew_blocks((long long)m * n), 256, 0, stream()>>>(m, n, src, lds, dst, ldd);
    note_launch("sub2d");
}
void flip_rows(int nrows, int n, const double *S, double *X, int ldx, int upper)
{
    if (nrows <= 0 || n <= 0) return;
    launch_chained(k_flip_rows, dim3(ew_blocks((long long)nrows * n)), 256, 0, nrows, n, S, X, ldx, upper);
    note_launch("flip_rows");
}
void flip_cols(int m, int n, const double *S, double *X, int ldx)
{
    if (m <= 0 || n <= 0) return;
    trace_begin();
    launch_chained(k_flip_cols, dim3(ew_blocks((long long)m * n)), 256, 0, m, n, S, X, ldx);
    note_launch("flip_cols");
}

// ---------------------------------------------------------------------------
// triangular solves
// ---------------------------------------------------------------------------
__global__ void k_trsm_left_lower_unit(int M, int N, const double *L, int ldl, double *B, int ldb)
{
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    double *b = B + (size_t)c * ldb;
    for (int r = 1; r < M; r++) {
        double s = b[r];
        for (int p = 0; p < r; p++) s -= L[(size_t)r + (size_t)p * ldl] * b[p];
        b[r] = s;
    }
}

// The same for M <= 64, a warp per column: the column's rows two per lane, each
// solved entry broadcast to the rows below it (M dependent steps of one or two
// FMAs instead of M^2 / 2 dependent global loads on one thread).
__global__ void __launch_bounds__(128) k_trsm_left_lower_unit_warp(int M, int N, const double *L, int ldl, double *B,
                                                                   int ldb)
{
    chain_wait();
    const int lane = threadIdx.x & 31, c = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (c >= N) return;
    double *b = B + (size_t)c * ldb;
    double b0 = lane < M ? b[lane] : 0.0, b1 = lane + 32 < M ? b[lane + 32] : 0.0;
    for (int p = 0; p + 1 < M; p++) {
        const double l0 = lane > p && lane < M ? L[(size_t)lane + (size_t)p * ldl] : 0.0;
        const double l1 = lane + 32 > p && lane + 32 < M ? L[(size_t)(lane + 32) + (size_t)p * ldl] : 0.0;
        const double x = __shfl_sync(0xffffffffu, p < 32 ? b0 : b1, p & 31);
        b0 = lane > p ? fma(-x, l0, b0) : b0;
        b1 = lane + 32 > p ? fma(-x, l1, b1) : b1;
    }
    if (lane < M) b[lane] = b0;
    if (lane + 32 < M) b[lane + 32] = b1;
}

void trsm_left_lower_unit(int M, int N, const double *L, int ldl, double *B, int ldb)
{
    if (M <= 1 || N <= 0) return;
    if (M <= 64) {
        launch_chained(k_trsm_left_lower_unit_warp, dim3(ceil_div(N, 4)), 128, 0, M, N, L, ldl, B, ldb);
        note_launch("trsm_left_lower_unit");
        return;
    }
    k_trsm_left_lower_unit<<<ceil_div(N, 64), 64, 0, stream()>>>(M, N, L, ldl, B, ldb);
    note_launch("trsm_left_lower_unit");
}

// Row r of B solves x * U = alpha * S.*b, any N: the row's solved prefix is
// re-read from global memory (coalesced across the threads of a warp, which own
// consecutive rows).
__global__ void k_trsm_right_upper(int M, int N, double alpha, const double *U, int ldu, double *B,
                                   int ldb, const double *S)
{
    for (size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x; r < (size_t)M;
         r += (size_t)gridDim.x * blockDim.x) {
        for (int c = 0; c < N; c++) {
            double s = alpha * B[r + (size_t)c * ldb];
            if (S && S[c] == -1.0) s = -s;
            for (int p = 0; p < c; p++) s -= B[r + (size_t)p * ldb] * U[(size_t)p + (size_t)c * ldu];
            B[r + (size_t)c * ldb] = s / U[(size_t)c + (size_t)c * ldu];
        }
    }
}

// The same solve for few rows (N <= 64): one warp per row, row r's 64
// values held two per lane; column c's dot product with the solved columns
// is split over the lanes and reduced by shuffles, so a row costs N
// reduction steps instead of N^2 / 2 dependent FMAs on one thread.
__global__ void __launch_bounds__(128) k_trsm_right_upper_warp(int M, int N, double alpha, const double *U, int ldu,
                                                                double *B, int ldb, const double *S)
{
    __shared__ double Us[64 * 64];
    for (int idx = threadIdx.x; idx < N * N; idx += blockDim.x) {
        const int r = idx % N, c = idx / N;
        Us[r + 64 * c] = (r <= c) ? U[(size_t)r + (size_t)c * ldu] : 0.0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= M) return;
    double b0 = lane < N ? B[(size_t)row + (size_t)lane * ldb] : 0.0;
    double b1 = lane + 32 < N ? B[(size_t)row + (size_t)(lane + 32) * ldb] : 0.0;
    double x0 = 0.0, x1 = 0.0;
    for (int c = 0; c < N; c++) {
        double s = alpha * __shfl_sync(0xffffffffu, c < 32 ? b0 : b1, c & 31);
        if (S && S[c] == -1.0) s = -s;
        double d = (lane < c ? x0 * Us[lane + 64 * c] : 0.0) + (lane + 32 < c ? x1 * Us[lane + 32 + 64 * c] : 0.0);
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        const double x = (s - d) / Us[c + 64 * c];
        if (c < 32) {
            if (lane == c) x0 = x;
        } else if (lane == c - 32) {
            x1 = x;
        }
    }
    if (lane < N) B[(size_t)row + (size_t)lane * ldb] = x0;
    if (lane + 32 < N) B[(size_t)row + (size_t)(lane + 32) * ldb] = x1;
}

// The same solve for many rows (N <= 64): a row per thread, held in registers, U
// broadcast from shared memory, the divisions by U's diagonal as products with
// its reciprocal corrected by the residual (3 FP64 operations instead of ~10).
// Bound by the FP64 pipe: N^2 / 2 FMAs per row (0.85 ms for 262,144 x 64).  262,144
// x 64: 1.26 -> 1.12 ms against rows re-read from global memory; the
// reconstruction's copy, sign pass and solve 1.44 -> 1.09 ms in one pass.
// Optionally the source rows come from another matrix (X, ldx), whose columns with
// S = -1 are then negated in place: the reconstruction's V = Q S U^-1 with Q := Q S
// in one pass.
template <bool FROM>
__global__ void __launch_bounds__(128) k_trsm_right_upper_rows(int M, int N, double alpha, const double *U, int ldu,
                                                                double *B, int ldb, const double *S, double *X, int ldx)
{
    __shared__ __align__(16) double Us[64 * 64];
    __shared__ double s_d[64], s_inv[64];
    __shared__ int s_neg[64], s_plain[64];
    for (int idx = threadIdx.x; idx < 64 * 64; idx += 128) {
        const int r = idx & 63, c = idx >> 6;
        Us[idx] = r < c && c < N ? U[(size_t)r + (size_t)c * ldu] : 0.0;
    }
    if (threadIdx.x < N) {
        const double d = U[(size_t)threadIdx.x * (ldu + 1)];
        s_d[threadIdx.x] = d;
        s_inv[threadIdx.x] = 1.0 / d;
        const int ex = (__double2hiint(d) >> 20) & 0x7FF;
        s_plain[threadIdx.x] = ex > 40 && ex < 2007;  // d and 1 / d normal
        s_neg[threadIdx.x] = S && S[threadIdx.x] == -1.0;
    }
    __syncthreads();
    for (size_t row = blockIdx.x * (size_t)128 + threadIdx.x; row < (size_t)M; row += (size_t)gridDim.x * 128) {
        double *b = B + row, *x = FROM ? X + row : b;
        const int ld = FROM ? ldx : ldb;
        double v[64];
#pragma unroll
        for (int c = 0; c < 64; c++) {
            v[c] = 0.0;
            if (c < N) v[c] = x[(size_t)c * ld];
        }
        if (alpha != 1.0) {
#pragma unroll
            for (int c = 0; c < 64; c++) v[c] *= alpha;
        }
#pragma unroll
        for (int c = 0; c < 64; c++) {
            if (c >= N) break;
            if (s_neg[c]) {
                v[c] = __longlong_as_double(__double_as_longlong(v[c]) ^ (long long)0x8000000000000000ull);
                if (FROM) x[(size_t)c * ld] = v[c];
            }
            double t = v[c];
#pragma unroll
            for (int p = 0; p < c; p++) t = fma(-v[p], Us[p + c * 64], t);
            const double inv = s_inv[c], d = s_d[c], q = t * inv;
            // the residual of an infinite quotient is no number
            if (s_plain[c] && ((__double2hiint(q) >> 20) & 0x7FF) != 0x7FF)
                v[c] = fma(fma(-q, d, t), inv, q);
            else
                v[c] = t / d;
            b[(size_t)c * ldb] = v[c];
        }
    }
}

// V = Q S U^-1 of M rows into B, Q := Q S (N <= 64).
void trsm_right_upper_from(int M, int N, const double *U, int ldu, double *Q, int ldq, double *B, int ldb,
                           const double *S, const char *tag)
{
    if (M <= 0 || N <= 0) return;
    trace_begin();
    k_trsm_right_upper_rows<true><<<ceil_div(M, 128), 128, 0, stream()>>>(M, N, 1.0, U, ldu, B, ldb, S, Q, ldq);
    note_launch(tag);
}

void trsm_right_upper(int M, int N, double alpha, const double *U, int ldu, double *B, int ldb,
                      const double *S, const char *tag)
{
    if (M <= 0 || N <= 0) return;
    if (N <= 64 && M <= 2048) {
        trace_begin();
        k_trsm_right_upper_warp<<<ceil_div(M, 4), 128, 0, stream()>>>(M, N, alpha, U, ldu, B, ldb, S);
        note_launch(tag);
        return;
    }
    int blocks = ceil_div(M, 128);
    trace_begin();
    if (N <= 64) {
        k_trsm_right_upper_rows<false><<<blocks, 128, 0, stream()>>>(M, N, alpha, U, ldu, B, ldb, S, nullptr, 0);
    } else {
        if (blocks > 16 * num_sm()) blocks = 16 * num_sm();
        k_trsm_right_upper<<<blocks, 128, 0, stream()>>>(M, N, alpha, U, ldu, B, ldb, S);
    }
    note_launch(tag);
}

// Row r: x * L^T = alpha * b with L unit lower (so L^T unit upper).
__global__ void k_trsm_right_lower_unit_trans(int M, int N, double alpha, const double *L, int ldl,
                                              double *B, int ldb)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= M) return;
    for (int c = 0; c < N; c++) {
        double s = alpha * B[(size_t)r + (size_t)c * ldb];
        for (int p = 0; p < c; p++) s -= B[(size_t)r + (size_t)p * ldb] * L[(size_t)c + (size_t)p * ldl];
        B[(size_t)r + (size_t)c * ldb] = s;
    }
}

// The same for N <= 64, a warp per row (its values two per lane, each solved one
// broadcast to the later ones), L in shared memory: 64 x 64 in 110 -> 20 us.
__global__ void __launch_bounds__(256) k_trsm_right_lower_unit_trans_warp(int M, int N, double alpha, const double *L,
                                                                          int ldl, double *B, int ldb)
{
    chain_wait();
    __shared__ double Ls[64 * 64];
    for (int idx = threadIdx.x; idx < N * N; idx += 256) {
        const int r = idx % N, c = idx / N;
        if (r > c) Ls[r + 64 * c] = L[(size_t)r + (size_t)c * ldl];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= M) return;
    double *b = B + row;
    double b0 = lane < N ? alpha * b[(size_t)lane * ldb] : 0.0, b1 = lane + 32 < N ? alpha * b[(size_t)(lane + 32) * ldb] : 0.0;
    for (int p = 0; p + 1 < N; p++) {
        const double x = __shfl_sync(0xffffffffu, p < 32 ? b0 : b1, p & 31);
        if (x == 0.0) continue;  // left of an upper triangular row's diagonal, whatever L holds there
        if (lane > p && lane < N) b0 = fma(-x, Ls[lane + 64 * p], b0);
        if (lane + 32 > p && lane + 32 < N) b1 = fma(-x, Ls[lane + 32 + 64 * p], b1);
    }
    if (lane < N) b[(size_t)lane * ldb] = b0;
    if (lane + 32 < N) b[(size_t)(lane + 32) * ldb] = b1;
}

void trsm_right_lower_unit_trans(int M, int N, double alpha, const double *L, int ldl, double *B,
                                 int ldb)
{
    if (M <= 0 || N <= 0) return;
    if (N <= 64) {
        launch_chained(k_trsm_right_lower_unit_trans_warp, dim3(ceil_div(M, 8)), 256, 0, M, N, alpha, L, ldl, B, ldb);
        note_launch("trsm_right_lower_unit_trans");
        return;
    }
    k_trsm_right_lower_unit_trans<<<ceil_div(M, 64), 64, 0, stream()>>>(M, N, alpha, L, ldl, B, ldb);
    note_launch("trsm_right_lower_unit_trans");
}

// ---------------------------------------------------------------------------
// one-CTA factorizations
// ---------------------------------------------------------------------------
// Block-wide reduction; `ident` is the identity of `op` (0 for sums, 0 for
// maxima of absolute values), used for the lanes beyond the block's warps.
template <typename Op>
__device__ double block_reduce(double v, Op op, double *red, double ident = 0.0)
{
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    int w = threadIdx.x / 32, l = threadIdx.x % 32;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    int nw = (blockDim.x + 31) / 32;
    if (w == 0) {
        v = (l < nw) ? red[l] : ident;
        for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (l == 0) red[32] = v;
    }
    __syncthreads();
    return red[32];
}

struct OpSum {
    __device__ double operator()(double a, double b) const { return a + b; }
};
struct OpMax {
    __device__ double operator()(double a, double b) const { return a > b ? a : b; }
};

// Cholesky G = U^T U (upper, in place), left-looking by rows.  On a
// non-positive pivot the status bit is set and the factorization stops
// (LAPACK dpotrf leaves the matrix partially factored the same way).
__global__ void k_potrf_upper(int n, double *A, int lda, int *status)
{
    __shared__ double red[33];
    __shared__ int bad;
    if (threadIdx.x == 0) bad = 0;
    for (int j = 0; j < n; j++) {
        double part = 0.0;
        for (int p = threadIdx.x; p < j; p += blockDim.x) {
            double a = A[(size_t)p + (size_t)j * lda];
            part += a * a;
        }
        double s = block_reduce(part, OpSum(), red);
        if (threadIdx.x == 0) {
            double d = A[(size_t)j + (size_t)j * lda] - s;
            if (!(d > 0.0)) {
                A[(size_t)j + (size_t)j * lda] = d;
                bad = 1;
                atomicOr(status, ST_CHOL_BREAKDOWN);
            } else {
                A[(size_t)j + (size_t)j * lda] = sqrt(d);
            }
        }
        __syncthreads();
        if (bad) return;
        double d = A[(size_t)j + (size_t)j * lda];
        for (int c = j + 1 + threadIdx.x; c < n; c += blockDim.x) {
            double t = A[(size_t)j + (size_t)c * lda];
            for (int p = 0; p < j; p++)
                t -= A[(size_t)p + (size_t)j * lda] * A[(size_t)p + (size_t)c * lda];
            A[(size_t)j + (size_t)c * lda] = t / d;
        }
        __syncthreads();
    }
}

constexpr int SLD = 65;  // leading dimension of the 64 x 64 blocks in shared memory

// The same for n <= 64 in shared memory, the pivot one step ahead: while the
// other warps subtract row j from the rows after j + 1, warp 0 subtracts it from
// row j + 1, takes that row's pivot (1 / sqrt by rsqrt_nr) and scales it; one
// block barrier per step.  64 x 64: 141 us for the kernel above (every step a
// reduction and columns of dependent global loads), 64 us here.
__global__ void __launch_bounds__(512) k_potrf_small(int n, double *A, int lda, int *status)
{
    chain_open();
    chain_wait();
    extern __shared__ double G[];  // (r, c) at r * SLD + c: a warp's lanes run along a row
    __shared__ int s_bad;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int idx = threadIdx.x; idx < n * n; idx += 512) {
        const int r = idx % n, c = idx / n;
        if (r <= c) G[r * SLD + c] = A[(size_t)r + (size_t)c * lda];
    }
    if (threadIdx.x == 0) s_bad = n;
    __syncthreads();
    // row j by warp 0: the pivot and the scaling; false on a non-positive pivot
    auto scale_row = [&](int j) {
        const double d = G[j * SLD + j];
        if (!(d > 0.0)) {
            if (lane == 0) s_bad = j;
            return;
        }
        // an infinite pivot is its own root, and the row then holds what t / inf is
        const bool finite = __double2hiint(d) != 0x7FF00000;
        const double y = finite ? rsqrt_nr(d) : 0.0;
        double root = d;
        if (finite) {
            root = d * y;
            root = fma(0.5 * y, fma(-root, root, d), root);
        }
        __syncwarp();
        for (int c = j + lane; c < n; c += 32) {
            const double t = G[j * SLD + c];
            double u = t * y;
            // t / root to rounding level (an infinite quotient has no residual)
            if (finite && ((__double2hiint(u) >> 20) & 0x7FF) != 0x7FF) u = fma(fma(-u, root, t), y, u);
            G[j * SLD + c] = c == j ? root : u;
        }
    };
    if (warp == 0) scale_row(0);
    __syncthreads();
    for (int j = 0; j < n; j++) {
        if (s_bad <= j) break;
        if (warp == 0) {
            if (j + 1 < n) {
                const double l = G[j * SLD + j + 1];
                for (int c = j + 1 + lane; c < n; c += 32) G[(j + 1) * SLD + c] = fma(-l, G[j * SLD + c], G[(j + 1) * SLD + c]);
                __syncwarp();
                scale_row(j + 1);
            }
        } else {
            for (int r = j + 1 + warp; r < n; r += 15) {
                const double l = G[j * SLD + r];
                for (int c = r + lane; c < n; c += 32) G[r * SLD + c] = fma(-l, G[j * SLD + c], G[r * SLD + c]);
            }
        }
        __syncthreads();
    }
    const int bad = s_bad;
    for (int idx = threadIdx.x; idx < n * n; idx += 512) {
        const int r = idx % n, c = idx / n;
        if (r <= c && (r < bad || (r == bad && c == bad))) A[(size_t)r + (size_t)c * lda] = G[r * SLD + c];
    }
    if (threadIdx.x == 0 && bad < n) atomicOr(status, ST_CHOL_BREAKDOWN);
}

__device__ int d_potrf_sink;

void potrf_upper(int n, double *A, int lda, bool record_breakdown)
{
    if (n <= 0) return;
    int *st = status_ptr();
    if (!record_breakdown) {
        void *p = nullptr;
        cudaGetSymbolAddress(&p, d_potrf_sink);
        st = (int *)p;
    }
    if (n <= 64)
        launch_chained(k_potrf_small, dim3(1), 512, 64 * SLD * sizeof(double), n, A, lda, st);
    else
        k_potrf_upper<<<1, 256, 0, stream()>>>(n, A, lda, st);
    note_launch("potrf_upper");
}

// LU without pivoting of (T S - I), S(k) = -1 when |1 - t_kk| < |1 + t_kk|
// (t_kk the partially eliminated diagonal), as in lila_dorgh2_3: column k is
// negated for S(k) = -1, the pivot is t_kk - 1, L below, U on/above.
__global__ void k_lu_sign(int n, double *T, int ldt, double *S, int *status)
{
    __shared__ double sgn, piv;
    for (int k = 0; k < n; k++) {
        if (threadIdx.x == 0) {
            double t = T[(size_t)k + (size_t)k * ldt];
            sgn = (fabs(1.0 - t) < fabs(1.0 + t)) ? -1.0 : 1.0;
            S[k] = sgn;
        }
        __syncthreads();
        if (sgn == -1.0)
            for (int r = threadIdx.x; r < n; r += blockDim.x)
                T[(size_t)r + (size_t)k * ldt] = -T[(size_t)r + (size_t)k * ldt];
        __syncthreads();
        if (threadIdx.x == 0) {
            double p = T[(size_t)k + (size_t)k * ldt] - 1.0;
            T[(size_t)k + (size_t)k * ldt] = p;
            piv = p;
            if (p == 0.0) atomicOr(status, ST_LU_ZERO_PIVOT);
        }
        __syncthreads();
        for (int r = k + 1 + threadIdx.x; r < n; r += blockDim.x)
            T[(size_t)r + (size_t)k * ldt] /= piv;
        __syncthreads();
        int w = n - k - 1;
        for (int idx = threadIdx.x; idx < w * w; idx += blockDim.x) {
            int r = k + 1 + idx % w, c = k + 1 + idx / w;
            T[(size_t)r + (size_t)c * ldt] -= T[(size_t)r + (size_t)k * ldt] * T[(size_t)k + (size_t)c * ldt];
        }
        __syncthreads();
    }
}

// Rare cases kept out of line: inline, the compiler issues their FP64 instructions
// for every pivot (131,072 x 32 leaf 1.865 -> 1.870 ms).
static __device__ __noinline__ bool sign_of_wide(double t) { return fabs(1.0 - t) < fabs(1.0 + t); }
static __device__ __noinline__ double quotient(double a, double p) { return a / p; }

// The same for n <= 64 in shared memory, the pivot column one step ahead of the
// others (as in k_potrf_small).  The pivot is -(1 + |t_kk|), so its reciprocal
// needs no division.  64 x 64: 73 us with the two launches it replaces.  With A given, the reconstruction's other small steps too:
// the strict lower part goes to A (and leaves zeros in T), and A's rows k with
// S(k) = -1 are negated from the diagonal on.
__global__ void __launch_bounds__(512) k_lu_sign_small(int n, double *T, int ldt, double *S, double *A, int lda,
                                                       int *status)
{
    chain_open();
    chain_wait();
    extern __shared__ double G[];  // column-major, SLD
    __shared__ double s_sgn[64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int idx = threadIdx.x; idx < n * n; idx += 512) {
        const int r = idx % n, c = idx / n;
        G[r + c * SLD] = T[(size_t)r + (size_t)c * ldt];
    }
    __syncthreads();
    auto pivot_col = [&](int k) {  // warp 0
        double *g = G + k * SLD;
        const double t = g[k];
        // |1 - t| < |1 + t| in FP64 is t > 2^-54, an integer comparison, up to
        // 2^53; past that the rounding of both sides decides
        const long long tb = __double_as_longlong(t);
        const bool wide = ((tb >> 52) & 0x7FF) >= 1023 + 53;
        bool neg = tb > 0x3C90000000000000ll;
        if (wide) neg = sign_of_wide(t);
        const long long flip = neg ? (long long)0x8000000000000000ull : 0ll;
        const double p = __longlong_as_double(tb ^ flip) - 1.0, inv = -rcp_nr(-p);
        __syncwarp();
        for (int r0 = 0; r0 < n; r0 += 32) {
            const int r = r0 + lane;
            if (r >= n) continue;
            const double a = __longlong_as_double(__double_as_longlong(g[r]) ^ flip);
            double l = a;
            if (r0 + 31 > k) {  // some row of the warp below the pivot
                l = a * inv;
                if (wide)
                    l = quotient(a, p);
                else if (((__double2hiint(l) >> 20) & 0x7FF) != 0x7FF)  // an infinity has no residual
                    l = fma(fma(-l, p, a), inv, l);
            }
            g[r] = r < k ? a : (r == k ? p : l);
        }
        if (lane == 0) {
            s_sgn[k] = neg ? -1.0 : 1.0;
            if (p == 0.0) atomicOr(status, ST_LU_ZERO_PIVOT);
        }
    };
    if (warp == 0) pivot_col(0);
    __syncthreads();
    for (int k = 0; k + 1 < n; k++) {
        const double *l = G + k * SLD;
        if (warp == 0) {
            double *g = G + (k + 1) * SLD;
            const double u = g[k];
            for (int r = (k + 1) / 32 * 32 + lane; r < n; r += 32)
                if (r > k) g[r] = fma(-l[r], u, g[r]);
            __syncwarp();
            pivot_col(k + 1);
        } else {
            for (int c = k + 1 + warp; c < n; c += 15) {
                double *g = G + c * SLD;
                const double u = g[k];
                for (int r = (k + 1) / 32 * 32 + lane; r < n; r += 32)
                    if (r > k) g[r] = fma(-l[r], u, g[r]);
            }
        }
        __syncthreads();
    }
    for (int idx = threadIdx.x; idx < n * n; idx += 512) {
        const int r = idx % n, c = idx / n;
        const double v = G[r + c * SLD];
        T[(size_t)r + (size_t)c * ldt] = A && r > c ? 0.0 : v;
        if (A) {
            double *a = A + (size_t)r + (size_t)c * lda;
            if (r > c)
                *a = v;
            else if (s_sgn[r] == -1.0)
                *a = -*a;
        }
    }
    if (threadIdx.x < n) S[threadIdx.x] = s_sgn[threadIdx.x];
}

void lu_sign(int n, double *T, int ldt, double *S)
{
    if (n <= 0) return;
    if (n <= 64)
        launch_chained(k_lu_sign_small, dim3(1), 512, 64 * SLD * sizeof(double), n, T, ldt, S, nullptr, 0, status_ptr());
    else
        k_lu_sign<<<1, 256, 0, stream()>>>(n, T, ldt, S, status_ptr());
    note_launch("lu_sign");
}

bool lu_sign_tile(int n, double *T, int ldt, double *S, double *A, int lda)
{
    if (n > 64) return false;
    if (n <= 0) return true;
    launch_chained(k_lu_sign_small, dim3(1), 512, 64 * SLD * sizeof(double), n, T, ldt, S, A, lda, status_ptr());
    note_launch("lu_sign");
    return true;
}

// LAPACK dlarfg on x(0:m): beta = -sign(alpha)*||x||, tau = (beta-alpha)/beta,
// v = x(1:m)/(alpha-beta); norm by max-scaled sum of squares.
__global__ void k_larfg(int m, double *x, double *tau)
{
    __shared__ double red[33];
    __shared__ double s_scale_inv;
    const double safmin = 2.2250738585072014e-308 / 1.1102230246251565e-16;
    int len = m - 1;
    double alpha = x[0];
    double *xs = x + 1;
    double mx = 0.0;
    for (int i = threadIdx.x; i < len; i += blockDim.x) mx = fmax(mx, fabs(xs[i]));
    double scale = block_reduce(mx, OpMax(), red);
    if (len <= 0 || scale == 0.0) {
        if (threadIdx.x == 0) *tau = 0.0;
        return;
    }
    double part = 0.0;
    for (int i = threadIdx.x; i < len; i += blockDim.x) {
        double t = xs[i] / scale;
        part += t * t;
    }
    double ssq = block_reduce(part, OpSum(), red);
    double xnorm = scale * sqrt(ssq);
    double beta = -copysign(hypot(alpha, xnorm), alpha);
    int knt = 0;
    if (fabs(beta) < safmin) {
        const double rsafmn = 1.0 / safmin;
        while (fabs(beta) < safmin && knt < 20) {
            knt++;
            for (int i = threadIdx.x; i < len; i += blockDim.x) xs[i] *= rsafmn;
            beta *= rsafmn;
            alpha *= rsafmn;
            __syncthreads();
        }
        mx = 0.0;
        for (int i = threadIdx.x; i < len; i += blockDim.x) mx = fmax(mx, fabs(xs[i]));
        scale = block_reduce(mx, OpMax(), red);
        part = 0.0;
        for (int i = threadIdx.x; i < len; i += blockDim.x) {
            double t = xs[i] / scale;
            part += t * t;
        }
        ssq = block_reduce(part, OpSum(), red);
        xnorm = scale * sqrt(ssq);
        beta = -copysign(hypot(alpha, xnorm), alpha);
    }
    if (threadIdx.x == 0) s_scale_inv = 1.0 / (alpha - beta);
    __syncthreads();
    double sc = s_scale_inv;
    for (int i = threadIdx.x; i < len; i += blockDim.x) xs[i] *= sc;
    if (threadIdx.x == 0) {
        *tau = (beta - alpha) / beta;
        for (int j = 0; j < knt; j++) beta *= safmin;
        x[0] = beta;
    }
}

void larfg(int m, double *x, double *tau)
{
    if (m <= 0) return;
    int th = m > 4096 ? 1024 : 256;
    k_larfg<<<1, th, 0, stream()>>>(m, x, tau);
    note_launch("larfg");
}

// dlarft recurrence from the Gram G = V^T V (only G(r, j), r < j used):
// T(j,j) = tau_j ; T(0:j, j) = T(0:j,0:j) * (-tau_j * G(0:j, j)).
__global__ void k_larft_from_gram(int k, const double *G, int ldg, const double *tau, double *T,
                                  int ldt)
{
    extern __shared__ double tmp[];
    for (int j = 0; j < k; j++) {
        double tj = tau[j];
        for (int r = threadIdx.x; r < j; r += blockDim.x)
            tmp[r] = (tj == 0.0) ? 0.0 : -tj * G[(size_t)r + (size_t)j * ldg];
        __syncthreads();
        for (int r = threadIdx.x; r < j; r += blockDim.x) {
            double s = 0.0;
            for (int c = r; c < j; c++) s += T[(size_t)r + (size_t)c * ldt] * tmp[c];
            T[(size_t)r + (size_t)j * ldt] = s;
        }
        if (threadIdx.x == 0) T[(size_t)j + (size_t)j * ldt] = tj;
        __syncthreads();
    }
}

// The same T for k <= 64 by doubling, T12 = -T11 (G12 T22) for blocks of 1, 2,
// 4, .. columns (dlarft's recurrence regrouped, as lila_dlarft_connect does):
// 2 log2(k) block barriers instead of 2 k, all operands in shared memory.
// The column recurrence on global memory took ~110 us for k = 64, this ~20.
constexpr int LARFT_LD = 65;
__global__ void __launch_bounds__(512) k_larft_small(int k, const double *G, int ldg, const double *tau, double *T,
                                                     int ldt)
{
    extern __shared__ double lf[];
    double *Gs = lf, *Ts = lf + 64 * LARFT_LD, *Ys = lf + 2 * 64 * LARFT_LD;
    chain_wait();
    for (int idx = threadIdx.x; idx < k * k; idx += blockDim.x) {
        const int r = idx % k, c = idx / k;
        if (r < c) Gs[r + c * LARFT_LD] = G[(size_t)r + (size_t)c * ldg];
        if (r == c) Ts[r + c * LARFT_LD] = tau[c];
    }
    __syncthreads();
    for (int b = 1; b < k; b *= 2) {
        const int pairs = (k + 2 * b - 1) / (2 * b), total = pairs * b * b;
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
            const int r0 = 2 * b * (idx / (b * b)), r = r0 + idx % b, c0 = r0 + b, c = c0 + idx / b % b;
            if (c >= k) continue;
            double s = 0.0;
            for (int q = c0; q <= c; q++) s = fma(Gs[r + q * LARFT_LD], Ts[q + c * LARFT_LD], s);
            Ys[r + c * LARFT_LD] = s;
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
            // rows by the slow index: a warp's sums have the same length
            const int r0 = 2 * b * (idx / (b * b)), r = r0 + idx / b % b, c = r0 + b + idx % b;
            if (c >= k) continue;
            double s = 0.0;
            for (int q = r; q < r0 + b; q++) s = fma(Ts[r + q * LARFT_LD], Ys[q + c * LARFT_LD], s);
            Ts[r + c * LARFT_LD] = -s;
        }
        __syncthreads();
    }
    chain_open();
    for (int idx = threadIdx.x; idx < k * k; idx += blockDim.x) {
        const int r = idx % k, c = idx / k;
        if (r <= c) T[(size_t)r + (size_t)c * ldt] = Ts[r + c * LARFT_LD];
    }
}

void larft_from_gram(int k, const double *G, int ldg, const double *tau, double *T, int ldt)
{
    if (k <= 0) return;
    trace_begin();
    if (k <= 64) {
        constexpr int smem = 3 * 64 * LARFT_LD * (int)sizeof(double);
        cudaFuncSetAttribute(k_larft_small, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        launch_chained(k_larft_small, dim3(1), 512, smem, k, G, ldg, tau, T, ldt);
    } else {
        k_larft_from_gram<<<1, 256, (size_t)k * sizeof(double), stream()>>>(k, G, ldg, tau, T, ldt);
    }
    note_launch("larft_from_gram");
}

__global__ void k_diag_to_vec(int n, const double *T, int ldt, double *out)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = T[(size_t)i + (size_t)i * ldt];
}

void diag_to_vec(int n, const double *T, int ldt, double *out)
{
    if (n <= 0) return;
    k_diag_to_vec<<<ceil_div(n, 256), 256, 0, stream()>>>(n, T, ldt, out);
    note_launch("diag_to_vec");
}

}  // namespace lg
