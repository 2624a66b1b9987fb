// lg_panel.cu -- Householder QR of panels and of small matrices in one launch,
// column by column out of shared memory (the reflectors of dgeqr3,
// lila-c/dgeqr3.c:3-114, LAPACK dlarfg conventions).
//
// What bounds both kernels is the FP64 pipe (2 lanes per clock per SM: a warp
// instruction holds its sub-partition for 64 clocks whether its lanes carry
// work or not) and the chain from one column to the next.  So a group of LG
// lanes owns a column: its dot products and updates run down the rows with
// full warps and only the last log2(LG) additions are shuffles, the reflector
// is formed by one lane with Newton-Raphson reciprocals, and the column is not
// scaled into v before its trailing columns are updated (v_r = x_r sc enters
// through the factor sc w_c; the scaling happens on the way out).
//
// k_panel (m x nb, nb <= 64, a block of rows per CTA, cooperative launch).
// For column j every CTA publishes, from its rows below the pivot, its dot
// products d_c = sum_r x_j(r) A(r, c) with every column (c = j: the sum of
// squares; c < j: for T), and the CTA that owns row j the pivot row A(j, c).
// One warp per column, spread over the CTAs, adds the CTAs' partials of its
// column in a fixed order and publishes the total (so all CTAs get the same
// beta, tau bit for bit); then every CTA updates its rows with w_c = A(j, c) +
// sc d_c.  Adding the partials in every CTA instead saves one trip through L2
// but costs G FP64 additions per column and CTA: 7.1 us per column at 4000 x
// 64 against 4.8 us this way (11.7 us before, with 5 shuffle additions per
// column and a counter barrier).
// The exchange has no separate barrier: a value travels as two 64-bit words
// of (32 data bits, 32-bit column tag), and its reader polls until both tags
// are column j's.  Slots alternate between two buffers: a slot of column j is
// written again for column j + 2 only by a CTA that has every total of column
// j + 1, to which every CTA contributed after it had read column j's.  The
// slots are zeroed before the launch; every wait is bounded (clock limit); one
// that gives up sets ST_WAIT_TIMEOUT and the CTA returns.
//
// k_qr_small: the whole matrix in one CTA's shared memory, V, R, the T tiles
// and (optionally) the explicit Q in one launch.
#include <math.h>

#include "lg_house.cuh"

namespace lg {
namespace pnl {

constexpr int NT = 256, MAXNB = 64;  // threads of a panel CTA, most columns
constexpr int NTS = 512;              // threads of the one-CTA kernel

// Lanes per column for n columns in a CTA of `threads`: as few as cover the
// block, since every doubling adds a shuffle addition per dot product.  128
// threads would spend fewer still, but one warp per sub-partition does not
// hide its loads (87 x 53 in one CTA: 504 us with 128 threads, 349 with 256,
// 322 with 512; the 4000 x 64 panel 317 us with 128, 309 with 256).
__host__ __device__ inline int lanes_for(int threads, int n)
{
    return threads / 64 * (n > 32 ? 1 : (n > 16 ? 2 : 4));
}
// The leading dimension in shared memory: lanes modulo 16, so the 16 / lanes
// columns that a half warp reads fall into different banks.
__host__ __device__ inline int pad_ld(int rows, int lanes) { return ((rows - lanes + 15) / 16 * 16) + lanes; }

// ---- tagged slots -----------------------------------------------------------
// A slot is two 64-bit words, (tag, low half) and (tag, high half) of the value:
// flags travelling in the data words, as NCCL's published low-latency (LL)
// protocol has them.  The vector accesses are of 64-bit elements because only an
// element is a single access (PTX, vector data types): a word comes with its own
// tag or not at all, whereas four 32-bit elements may be seen one without the
// other.
struct __align__(16) Slot {
    unsigned long long lo, hi;
};
__device__ __forceinline__ void slot_put(Slot *p, double v, uint32_t tag)
{
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.volatile.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | (uint32_t)__double2loint(v)),
                 "l"(t | (uint32_t)__double2hiint(v))
                 : "memory");
}
__device__ __forceinline__ Slot slot_get(const Slot *p)
{
    Slot w;
    asm volatile("ld.volatile.global.v2.b64 {%0, %1}, [%2];" : "=l"(w.lo), "=l"(w.hi) : "l"(p) : "memory");
    return w;
}
__device__ __forceinline__ bool slot_ready(const Slot &w, uint32_t tag)
{
    return (uint32_t)(w.lo >> 32) == tag && (uint32_t)(w.hi >> 32) == tag;
}
__device__ __forceinline__ double slot_value(const Slot &w) { return __hiloint2double((int)w.hi, (int)w.lo); }

// The value of slot p once it holds `tag`; false when the wait gave up.
__device__ __forceinline__ bool slot_wait(const Slot *p, uint32_t tag, long long limit, double &v)
{
    Slot w = slot_get(p);
    if (!slot_ready(w, tag)) {
        const long long t0 = clock64();
        do {
            if (clock64() - t0 > limit) return false;
            w = slot_get(p);
        } while (!slot_ready(w, tag));
    }
    v = slot_value(w);
    return true;
}

// Sum over the warp of the slots p[0 .. G) once each holds `tag` (lane l adds
// p[l], p[l + 32], .., then a butterfly); false when the wait gave up.
__device__ __forceinline__ bool slots_sum(const Slot *p, int lane, int G, uint32_t tag, long long limit, double &sum)
{
    constexpr int B = 5;  // loads in flight: 160 CTAs
    sum = 0.0;
    bool ok = true;
    for (int q0 = 0; q0 < G && ok; q0 += B * 32) {
        Slot w[B];
        const long long t0 = clock64();
        for (;;) {
            bool ready = true;
#pragma unroll
            for (int u = 0; u < B; u++) {
                w[u] = Slot{(unsigned long long)tag << 32, (unsigned long long)tag << 32};
                if (q0 + u * 32 + lane < G) w[u] = slot_get(p + q0 + u * 32 + lane);
            }
#pragma unroll
            for (int u = 0; u < B; u++) ready = ready && slot_ready(w[u], tag);
            if (__all_sync(0xffffffffu, ready)) break;
            if (__any_sync(0xffffffffu, clock64() - t0 > limit)) {
                ok = false;
                break;
            }
        }
#pragma unroll
        for (int u = 0; u < B; u++)
            if (q0 + u * 32 < G) sum += slot_value(w[u]);
    }
    sum = group_sum<32>(sum);
    return ok;
}

// Slots of one buffer: column c's partial of CTA q at c G + q, its total at
// nb G + c, the pivot row's entry at nb (G + 1) + c.
__host__ __device__ inline long long slot_buffer(int nb, int G) { return (long long)nb * (G + 2); }
// Behind the two buffers those of a column taken again: partials and totals as
// above, then the CTAs' largest exponents.  One set is enough: the next column
// taken again writes it after that column's own exchange, so after every CTA has
// left this one.
__host__ __device__ inline long long slot_count(int nb, int G) { return 2 * slot_buffer(nb, G) + (long long)nb * (G + 1) + G; }

template <int LG>
__global__ void __launch_bounds__(NT, 1)
    k_panel(int m, int nb, int rpb, double *A, int lda, double *tau, double *Gram, Slot *slots, int *status,
            long long limit, uint32_t tag_skew)
{
    extern __shared__ double X[];  // nb columns, ld
    __shared__ double s_tau, s_f, s_sc[MAXNB], s_beta[MAXNB], s_d[MAXNB], s_p[MAXNB];
    constexpr int NW = NT / 32;
    __shared__ int s_shift, s_below, s_e[NW], s_nz[NW];
    __shared__ int2 s_stop;  // a wait gave up; the column has to be taken again
    const int G = gridDim.x, b = blockIdx.x;
    const int r0 = b * rpb, nr = min(m - r0, rpb), ld = pad_ld(rpb, LG);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = threadIdx.x / LG, g = threadIdx.x % LG;  // this thread's column and its lane in the group
    if (threadIdx.x == 0) s_stop = make_int2(0, 0);
    for (int cc = warp; cc < nb; cc += NW)
        for (int r = lane; r < nr; r += 32) X[r + cc * ld] = A[(size_t)(r0 + r) + (size_t)cc * lda];
    __syncthreads();
    const bool mine = c < nb;
    double *xc = X + (mine ? c : 0) * ld;
    // one past the warp's last column, 0 for a warp without columns
    const int wc1 = warp * (32 / LG) < nb ? min(nb, (warp + 1) * (32 / LG)) : 0;
    for (int j = 0; j < nb; j++) {
        Slot *buf = slots + (size_t)(j & 1) * slot_buffer(nb, G);
        Slot *total = buf + (size_t)nb * G, *pivot = total + nb;
        const uint32_t tag = j + 1 + tag_skew;
        const bool owner = j >= r0 && j < r0 + nr;
        double *xj = X + j * ld;
        const int first = max(0, j + 1 - r0);
        // this CTA's partials (the warps of columns before j would be idle
        // now: the products for T cost nothing extra)
        auto product = [&] {
            double d = 0.0;
#pragma unroll 4
            for (int r = first + g; r < nr; r += LG) d = fma(xj[r], xc[r], d);
            return group_sum<LG>(d);
        };
        if (wc1 > 0) {
            const double d = product();
            if (mine && g == 0) {
                slot_put(buf + (size_t)c * G + b, d, j + 1);
                if (owner) slot_put(pivot + c, xc[j - r0], j + 1);
            }
        }
        // the totals of the columns this warp adds up
        bool ok = true;
        for (int cc = b + warp * G; cc < nb; cc += NW * G) {
            double d, p = 0.0;
            ok = slots_sum(buf + (size_t)cc * G, lane, G, tag, limit, d) && ok;
            if (cc >= j) {
                if (lane == 0) slot_put(total + cc, d, j + 1);
            } else {
                ok = slot_wait(pivot + cc, tag, limit, p) && ok;
                if (lane == 0) {
                    s_d[cc] = d;
                    s_p[cc] = p;
                }
            }
        }
        double d = 0.0, pr = 0.0;
        if (wc1 > j) {
            if (mine && c >= j) ok = slot_wait(pivot + c, tag, limit, pr) && slot_wait(total + c, tag, limit, d) && ok;
            if (c == j && g == 0) {
                // house_in_range by the exponents alone, beside the reflector's
                // chain (an FP64 compare in it cost 80 ns per column); a sum of
                // zero is out of range, so there is something below here
                s_stop.y = bexp_of(d) < 1023 - 930 || bexp_of(d) > 1023 + 929 || bexp_of(pr) > 1023 + 463;
                const Reflector h = house_reflector(pr, d, true);
                s_tau = h.tau;
                s_f = h.tau * h.sc;
                s_sc[j] = h.sc;
                s_beta[j] = h.beta;
                if (owner) tau[j] = h.tau;
            }
        }
        if (!ok) s_stop.x = 1;
        __syncthreads();
        const int2 stop = s_stop;
        if (stop.x) {
            if (threadIdx.x == 0) atomicOr(status, ST_WAIT_TIMEOUT);
            return;
        }
        if (stop.y) {
            // rare, and the same in every CTA (they have the same total and pivot):
            // rows j.. of the column by 2^-k, k its largest exponent, and the column
            // again, as in k_qr_small
            Slot *part = slots + 2 * slot_buffer(nb, G), *sum = part + (size_t)nb * G, *exps = sum + nb;
            int e = 0, nz = 0;
            for (int r = max(0, j - r0) + threadIdx.x; r < nr; r += NT) {
                const int x = house_exponent(xj[r]);
                if (r0 + r > j && x) nz = 1;
                e = max(e, x);
            }
            e = __reduce_max_sync(0xffffffffu, e);
            nz = __any_sync(0xffffffffu, nz);
            if (lane == 0) {
                s_e[warp] = e;
                s_nz[warp] = nz;
            }
            __syncthreads();
            if (warp == 0) {
                e = __reduce_max_sync(0xffffffffu, lane < NW ? s_e[lane] : 0);
                nz = __any_sync(0xffffffffu, lane < NW && s_nz[lane]);
                if (lane == 0) slot_put(exps + b, __hiloint2double(nz, e), j + 1);
                for (int q = lane; q < G && ok; q += 32) {
                    double v = 0.0;
                    ok = slot_wait(exps + q, tag, limit, v);
                    e = max(e, __double2loint(v));
                    nz |= __double2hiint(v);
                }
                e = __reduce_max_sync(0xffffffffu, e);
                nz = __any_sync(0xffffffffu, nz);
                if (lane == 0) {
                    s_shift = house_shift(e);
                    s_below = nz;
                }
                if (!ok) s_stop.x = 1;
            }
            __syncthreads();
            const int k = s_shift;
            for (int r = max(0, j - r0) + threadIdx.x; r < nr; r += NT) xj[r] = scalbn(xj[r], -k);
            __syncthreads();
            if (wc1 > 0 && !s_stop.x) {
                const double dk = product();
                if (mine && g == 0) slot_put(part + (size_t)c * G + b, dk, j + 1);
            }
            for (int cc = b + warp * G; cc < nb && !s_stop.x; cc += NW * G) {
                double dk;
                ok = slots_sum(part + (size_t)cc * G, lane, G, tag, limit, dk) && ok;
                if (lane == 0) {
                    if (cc >= j)
                        slot_put(sum + cc, dk, j + 1);
                    else
                        s_d[cc] = dk;
                }
            }
            if (wc1 > j && !s_stop.x) {
                if (mine && c >= j) ok = slot_wait(sum + c, tag, limit, d) && ok;
                if (c == j && g == 0) {
                    const Reflector h = house_reflector(scalbn(pr, -k), d, s_below != 0);
                    s_tau = h.tau;
                    s_f = h.tau * h.sc;
                    s_sc[j] = h.sc;
                    s_beta[j] = scalbn(h.beta, k);
                    if (owner) tau[j] = h.tau;
                }
            }
            __syncthreads();
            if (!ok) s_stop.x = 1;
            __syncthreads();
            if (s_stop.x) {
                if (threadIdx.x == 0) atomicOr(status, ST_WAIT_TIMEOUT);
                return;
            }
        }
        const double tj = s_tau, sc = s_sc[j];
        if (wc1 > j + 1 && tj != 0.0 && mine && c > j) {
            const double e = fma(sc, d, pr), f = s_f * e;
#pragma unroll 4
            for (int r = first + g; r < nr; r += LG) xc[r] = fma(-f, xj[r], xc[r]);
            if (owner && g == 0) xc[j - r0] = fma(-tj, e, pr);
        }
        // (V^T V)(cc, j) = v_cc(j) + sum_{r > j} v_cc(r) v_j(r)
        for (int cc = b + warp * G; cc < j; cc += NW * G)
            if (lane == 0) Gram[cc + (size_t)j * nb] = s_sc[cc] * fma(sc, s_d[cc], s_p[cc]);
        __syncthreads();
    }
    for (int cc = warp; cc < nb; cc += NW) {
        const double sc = s_sc[cc], beta = s_beta[cc];
        for (int r = lane; r < nr; r += 32) {
            const int gr = r0 + r;
            const double x = X[r + cc * ld];
            A[(size_t)gr + (size_t)cc * lda] = gr > cc ? x * sc : (gr == cc ? beta : x);
        }
    }
}

// Householder QR of an m x n matrix (m >= n) held in one CTA's shared memory:
// V and R in A, the T tiles (reflector c belongs to the tile floor((i + c) /
// mt); i = 0 and mt >= n give the one n x n T of a panel) and, when Q is
// given, Q = H_0 .. H_{n-1} [I; 0].
//
// Per column two block barriers: the dot products of column j with the columns
// of its T tile before it (for T) and all columns from it on, the reflector by
// one lane of column j's group while the other groups finish; then each group
// updates its columns.  T(:, j) = -tau_j T(:, 0:j) (V^T v_j) runs beside the
// next column's dot products.  A sum of squares outside [1e-280, 1e280] takes
// the column again scaled by a power of two (dlarfg's scaled norm).  Q is
// formed in place of V from the last reflector to the first; a column is
// touched by its own group only, so one barrier per step.
template <int LG>
__global__ void __launch_bounds__(NTS, 1)
    k_qr_small(int m, int n, int ld, double *A, int lda, double *T, int ldt, int i, int mt, double *Q, int ldq)
{
    extern __shared__ double sm[];
    constexpr int NW = NTS / 32, NG = NTS / LG;
    const int tw = min(mt, n);
    double *X = sm, *Ts = X + (size_t)ld * n, *s_d = Ts + tw * (tw + 1), *s_g = s_d + n, *s_sc = s_g + n,
           *s_tau = s_sc + n, *s_beta = s_tau + n;
    __shared__ double s_f;
    __shared__ int s_redo, s_exp, s_nz;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cg = threadIdx.x / LG, g = threadIdx.x % LG;
    for (int c = warp; c < n; c += NW)
        for (int r = lane; r < m; r += 32) X[r + c * ld] = A[(size_t)r + (size_t)c * lda];
    __syncthreads();

    // dot products of column j's rows below the pivot with the columns lo ..,
    // column j itself first; its group's first lane forms the reflector
    auto dots = [&](int j, int lo, bool scaled) {
        const double *xj = X + j * ld;
        auto one = [&](int c) {
            const double *xc = X + (size_t)min(c, n - 1) * ld;
            double d = 0.0;
#pragma unroll 4
            for (int r = j + 1 + g; r < m; r += LG) d = fma(xj[r], xc[r], d);
            return group_sum<LG>(d);
        };
        const int jg = j % NG;
        if (cg / (32 / LG) == jg / (32 / LG)) {  // the warp of column j: all its groups take the same turn
            const int c = j - jg + cg;
            const double d = one(c);
            if (g == 0 && c < n && c >= lo) {
                s_d[c] = d;
                if (c == j) {
                    const double alpha = xj[j];
                    const bool last = j == m - 1;
                    if (!scaled) s_redo = !last && !house_in_range(alpha, d);
                    const Reflector h = house_reflector(alpha, d, scaled ? s_nz != 0 : !last);
                    s_tau[j] = h.tau;
                    s_f = h.tau * h.sc;
                    if (scaled || !s_redo) X[j + j * ld] = h.u;  // u's pivot entry, until V goes out
                    s_sc[j] = h.sc;
                    s_beta[j] = scaled ? scalbn(h.beta, s_exp) : h.beta;
                }
            }
        }
        for (int c0 = lo - lo % NG; c0 < n; c0 += NG) {
            if (c0 == j - jg && cg / (32 / LG) == jg / (32 / LG)) continue;
            if (c0 + (warp + 1) * (32 / LG) <= lo || c0 + warp * (32 / LG) >= n) continue;
            const int c = c0 + cg;
            const double d = one(c);
            if (g == 0 && c < n && c >= lo) s_d[c] = d;
        }
    };
    // T(:, j) of j's tile from g_c = v_c^T v_j (s_g), rows ts .. j
    auto t_column = [&](int j, int ts) {
        const double tj = s_tau[j];
        double *gt = T + (i + ts) % mt + (size_t)j * ldt;
        for (int r0 = ts; r0 < j; r0 += NG) {
            if (r0 + warp * (32 / LG) >= j) break;
            const int r = r0 + cg;
            double s = 0.0;
            if (r < j)
                for (int c = r + g; c < j; c += LG) s = fma(Ts[(r - ts) + (c - ts) * (tw + 1)], s_g[c], s);
            s = group_sum<LG>(s);
            if (r < j && g == 0) {
                const double t = tj == 0.0 ? 0.0 : -tj * s;
                Ts[(r - ts) + (j - ts) * (tw + 1)] = t;
                gt[r - ts] = t;
            }
        }
        if (threadIdx.x == 0) {
            Ts[(j - ts) + (j - ts) * (tw + 1)] = tj;
            gt[j - ts] = tj;
        }
    };
    // first column of j's tile
    auto tile_start = [&](int j) { return max(0, (i + j) / mt * mt - i); };

    for (int j = 0; j < n; j++) {
        const int ts = tile_start(j);
        double *xj = X + j * ld;
        dots(j, ts, false);
        // the previous column's T beside this column's dot products
        if (j > 0) t_column(j - 1, tile_start(j - 1));
        __syncthreads();
        if (s_redo) {
            // rare: scale rows j.. of column j by 2^-e, e the largest exponent,
            // and take the column again
            if (threadIdx.x == 0) {
                s_exp = 0;
                s_nz = 0;
            }
            __syncthreads();
            int e = 0, nz = 0;
            for (int r = j + threadIdx.x; r < m; r += NTS) {
                const int x = house_exponent(xj[r]);
                if (r > j && x) nz = 1;
                e = max(e, x);
            }
            atomicMax(&s_exp, e);
            if (nz) atomicOr(&s_nz, 1);
            __syncthreads();
            const int k = house_shift(s_exp);
            __syncthreads();
            if (threadIdx.x == 0) s_exp = k;
            for (int r = j + threadIdx.x; r < m; r += NTS) xj[r] = scalbn(xj[r], -k);
            __syncthreads();
            dots(j, ts, true);
            __syncthreads();
        }
        const double tj = s_tau[j], sc = s_sc[j];
        for (int c0 = ts - ts % NG; c0 < n; c0 += NG) {
            if (c0 + (warp + 1) * (32 / LG) <= ts || c0 + warp * (32 / LG) >= n) continue;
            const int c = c0 + cg;
            const bool on = c >= ts && c < n && c != j, right = on && c > j && tj != 0.0;
            double *xc = X + (on ? c : j) * ld;
            const double e = on ? fma(sc, s_d[c], xc[j]) : 0.0;
            __syncwarp();  // the group has read its pivot entry
            if (right) {
                const double f = s_f * e;
#pragma unroll 4
                for (int r = j + g; r < m; r += LG) xc[r] = fma(-f, xj[r], xc[r]);
            }
            if (on && c < j && g == 0) s_g[c] = s_sc[c] * e;
        }
        __syncthreads();
    }
    t_column(n - 1, tile_start(n - 1));
    // V and R out; V stays, scaled, where Q is formed
    for (int c = warp; c < n; c += NW) {
        const double sc = s_sc[c], beta = s_beta[c];
        for (int r = lane; r < m; r += 32) {
            double x = X[r + c * ld];
            x = r > c ? x * sc : (r == c ? beta : x);
            A[(size_t)r + (size_t)c * lda] = x;
            X[r + c * ld] = r > c ? x : 0.0;
        }
    }
    if (!Q) return;
    __syncthreads();
    for (int j = n - 1; j >= 0; j--) {
        const double tj = s_tau[j];
        double *xj = X + j * ld;
        for (int c0 = (j + 1) - (j + 1) % NG; c0 < n; c0 += NG) {
            if (c0 + (warp + 1) * (32 / LG) <= j + 1 || c0 + warp * (32 / LG) >= n) continue;
            const int c = c0 + cg;
            const bool on = c > j && c < n;
            double *xc = X + (on ? c : j) * ld;
            double d = 0.0;
#pragma unroll 4
            for (int r = j + 1 + g; r < m; r += LG) d = fma(xj[r], xc[r], d);
            d = tj * group_sum<LG>(d);
            if (on) {
#pragma unroll 4
                for (int r = j + 1 + g; r < m; r += LG) xc[r] = fma(-d, xj[r], xc[r]);
                if (g == 0) xc[j] = -d;
            }
        }
        __syncthreads();
        if (cg == j % NG) {
            for (int r = j + 1 + g; r < m; r += LG) xj[r] *= -tj;
            if (g == 0) xj[j] = 1.0 - tj;
        }
        __syncwarp();  // the next step reads the column by other lanes of its group
    }
    __syncthreads();
    for (int c = warp; c < n; c += NW)
        for (int r = lane; r < m; r += 32) Q[(size_t)r + (size_t)c * ldq] = X[r + c * ld];
}

}  // namespace pnl

// Doubles of workspace panel_coop needs for an nb-column panel (tau, the
// Gram V^T V and the 16-byte exchange slots; the rest is kept so that the workspace queries' answers stay).
long long panel_coop_work(int nb)
{
    const long long G = sm_count();
    return (long long)nb + (long long)nb * nb + 2 * ((pnl::MAXNB + 2) * G + pnl::MAXNB) + 8 + 64LL * nb * nb;
}

// Whether the cooperative panel applies to an m x nb panel.
bool panel_coop_fits(int m, int nb)
{
    if (nb < 2 || nb > pnl::MAXNB || m < 2 * nb || m < 256) return false;
    const int G = sm_count();
    const int rpb = (m + G - 1) / G;
    return (size_t)rpb * nb * sizeof(double) <= 200 * 1024;
}

// V (unit lower, below the diagonal), R (on and above) in A and the nb x nb T
// of the panel's compact-WY form (forward, columnwise), as dgeqr3 gives them.
// Returns false when the cooperative launch was refused (nothing enqueued).
// tag_skew: added to the tag every reader waits for (0; a test passes one that
// no CTA writes, so that every wait runs out, see lila_prim_panel_phantom).
static bool panel_coop_launch(int m, int nb, double *A, int lda, double *T, int ldt, double *work, uint32_t tag_skew)
{
    if (!panel_coop_fits(m, nb)) return false;
    const int Gmax = sm_count();
    // every SM takes part from 16 rows each on
    int rpb = (m + Gmax - 1) / Gmax;
    if (rpb < 16) rpb = 16;
    const int G = (m + rpb - 1) / rpb;
    double *tau = work;
    double *Gram = tau + nb;
    // slots on a 16-byte boundary (work is at least 8-byte aligned)
    pnl::Slot *slots = (pnl::Slot *)(((uintptr_t)(Gram + (size_t)nb * nb) + 15) & ~(uintptr_t)15);
    const long long nslots = pnl::slot_count(nb, G);
    const int lg = pnl::lanes_for(pnl::NT, nb);
    const size_t smem = (size_t)pnl::pad_ld(rpb, lg) * nb * sizeof(double);
    const void *kern = lg == 4 ? (const void *)pnl::k_panel<4>
                               : (lg == 8 ? (const void *)pnl::k_panel<8> : (const void *)pnl::k_panel<16>);
    cudaStream_t st = stream();
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    trace_break();
    cudaMemsetAsync(slots, 0, (size_t)nslots * sizeof(pnl::Slot), st);
    int *status = status_ptr();
    long long limit = wait_limit();
    void *args[] = {(void *)&m,    (void *)&nb,    (void *)&rpb,    (void *)&A,     (void *)&lda,     (void *)&tau,
                    (void *)&Gram, (void *)&slots, (void *)&status, (void *)&limit, (void *)&tag_skew};
    trace_begin();
    if (cudaLaunchCooperativeKernel(kern, dim3(G), dim3(pnl::NT), args, smem, st) != cudaSuccess) {
        cudaGetLastError();  // refused (e.g. not all CTAs can be resident): nothing ran
        trace_cancel();
        return false;
    }
    note_launch("panel_coop");
    larft_from_gram(nb, Gram, nb, tau, T, ldt);
    return true;
}

bool panel_coop(int m, int nb, double *A, int lda, double *T, int ldt, double *work)
{
    return panel_coop_launch(m, nb, A, lda, T, ldt, work, 0);
}

// Shared memory of k_qr_small, 0 when the matrix does not fit.
static size_t qr_small_smem(int m, int n, int mt)
{
    const long long tw = mt < n ? mt : n;
    const long long b = 8LL * ((long long)pnl::pad_ld(m, pnl::lanes_for(pnl::NTS, n)) * n + tw * (tw + 1) + 5LL * n);
    return b <= 220 * 1024 ? (size_t)b : 0;
}

bool qr_small(int m, int n, double *A, int lda, double *T, int ldt, int i, int mt, double *Q, int ldq)
{
    const size_t smem = n < 1 || m < n ? 0 : qr_small_smem(m, n, mt);
    if (!smem) return false;
    cudaStream_t st = stream();
    auto launch = [&](auto kern) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        trace_begin();
        kern<<<1, pnl::NTS, smem, st>>>(m, n, pnl::pad_ld(m, pnl::lanes_for(pnl::NTS, n)), A, lda, T, ldt, i, mt, Q, ldq);
        note_launch("qr_small");
        return true;
    };
    if (pnl::lanes_for(pnl::NTS, n) == 8) return launch(pnl::k_qr_small<8>);
    if (pnl::lanes_for(pnl::NTS, n) == 16) return launch(pnl::k_qr_small<16>);
    return launch(pnl::k_qr_small<32>);
}

}  // namespace lg

extern "C" {
// Failure-path test of the exchange's bounded waits: the panel of an m x nb
// matrix with every reader waiting for a tag that is never written (extra > 0),
// so each CTA's wait runs out after the lila_gpu_set_wait_limit cycles, sets
// LILA_ST_WAIT_TIMEOUT and returns (A and T are then meaningless).  1 when
// the cooperative launch ran, 0 when the panel does not apply.
int lila_prim_panel_phantom(int m, int nb, double *A, int lda, double *T, int ldt, double *work, int extra)
{
    if (extra < 0) return -8;
    return lg::panel_coop_launch(m, nb, A, lda, T, ldt, work, extra ? 0x40000000u : 0u) ? 1 : 0;
}
long long lila_prim_panel_work(int nb) { return lg::panel_coop_work(nb); }
}
