/*
 * facp_power.cuh -- the power iterations of the convex QP solver (sigma_max of
 * A, the extreme eigenvalues of Q) in a resident kernel of their own (sm_103a).
 *
 * What bounds a step is latency: two grid barriers, the gathers between them,
 * and FP64 instructions, which hold the pipe for 19 cycles however many lanes are
 * active and make a dependent one wait 64 (counters at 50,000 variables: warps at
 * a barrier 27 of 38 cycles, FP64 pipe 22% busy, L2 22%; at 200,000 FP64 33%, L2
 * 43%).  So a lane owns a row: 32 rows of about equal length make a slice (rows
 * sorted by length within a window of 2,048), stored entry by entry, whose
 * products and whose epilogue then run with all lanes active, four gathers in
 * flight per lane, and no shared memory or block barrier in between; what is one
 * number for the grid is computed in one lane.  The persistent iteration kernel
 * (k_facp) sums a row in two to four lanes after staging the products; it keeps
 * the matrices with a row of more than kPowerChain entries, whose lane would be a
 * chain of dependent gathers.
 * A step for sigma_max of a random 25,000 x 50,000 A with 500,000 nonzeros: 23 ->
 * 14.7 us, 100,000 x 200,000 with 2M: 57 -> 28 us (1,024 threads or two, eight
 * gathers in flight: 10 to 30% slower).
 */
#pragma once

#include "facp_kernels.cuh"

namespace pdal {
namespace facp {

constexpr int kPowerThreads = 512; /* one block per SM: as few barrier arrivals as can be */
constexpr int kPowerWindow = 2048;
constexpr int kPowerChain = 96;

/* rows in slices: slice s is entries[s].x + 32 j + lane, j < entries[s].y */
struct PowerMat {
    int ns;
    const int2 *entries;
    const int2 *rows; /* per lane: row (-1: none), its entries */
    const int *ci;
    const double *v;
};

struct PowerArgs {
    PowerMat a, at; /* Q: at */
    int m, n;       /* A: rows and columns; Q: both n */
    double *v, *vn, *last, *dp;
    double *part; /* three windows x grid x kSlot */
    GridBar *bar;
    Ctl *ctl;
    int bar_extra, max_iter, shifted;
    long long spin_limit;
    double tol, tol2, lam_max; /* tol2 = tol^2, or 0 for a tol of 0 or less */
};

/* HostPowerMat's arrays from the rows of a CSR matrix; a warp per slice */
static __global__ void k_power_pack(int ns, const int2 *__restrict__ entries, const int2 *__restrict__ rows,
                                    const int *__restrict__ rp, const int *__restrict__ ci,
                                    const double *__restrict__ v, int *pci, double *pv) {
    const int lane = threadIdx.x & 31;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < ns; s += (gridDim.x * blockDim.x) >> 5) {
        const int2 e = rows[(size_t)s * 32 + lane];
        if (e.x < 0) continue;
        const size_t to = (size_t)entries[s].x + lane;
        const int k = rp[e.x];
        for (int j = 0; j < e.y; ++j) {
            pci[to + 32 * j] = ci[k + j];
            pv[to + 32 * j] = v[k + j];
        }
    }
}

/* The rows of M times gat, epi(row, sum, red) in the row's lane.  The entries of
 * the next group, of this slice or the next, are loaded while this group's
 * gathers are in flight. */
template <class Epi, class R>
__device__ __forceinline__ void power_rows(const PowerMat &M, const double *gat, const Epi &epi, R &red) {
    constexpr int U = 4;
    const int lane = threadIdx.x & 31, step = (int)gridDim.x * (kPowerThreads / 32);
    int s = (int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x;
    if (s >= M.ns) return;
    int c[U];
    double w[U];
    auto entries = [&](const int2 &d, int len, int j, int (&ci)[U], double (&v)[U]) {
        const size_t at = (size_t)d.x + lane;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (j + u < len) {
                ci[u] = __ldg(M.ci + at + (j + u) * 32);
                v[u] = __ldg(M.v + at + (j + u) * 32);
            }
    };
    int2 d = __ldg(M.entries + s), e = __ldg(M.rows + (size_t)s * 32 + lane);
    entries(d, e.y, 0, c, w);
    while (s < M.ns) {
        int2 dn = make_int2(0, 0), en = make_int2(-1, 0);
        if (s + step < M.ns) {
            dn = __ldg(M.entries + s + step);
            en = __ldg(M.rows + (size_t)(s + step) * 32 + lane);
        }
        typename Epi::In in;
        if (e.x >= 0) in = epi.fetch(e.x);
        double sum = 0.0;
        int j = 0;
        do {
            double g[U], wn[U];
            int cn[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j + u < e.y) g[u] = __ldcg(gat + c[u]);
            const bool more = j + U < d.y;
            entries(more ? d : dn, more ? e.y : en.y, more ? j + U : 0, cn, wn);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j + u < e.y) sum = fma(w[u], g[u], sum);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                c[u] = cn[u];
                w[u] = wn[u];
            }
            j += U;
        } while (j < d.y);
        if (e.x >= 0) epi.finish(e.x, sum, in, red);
        s += step;
        d = dn;
        e = en;
    }
}

/* Grid sums of r, the same in every block, through of(term, sum): a warp per term
 * over the blocks' slots in a fixed order.  One lane applies `of`: a reciprocal
 * square root in all sixteen warps takes the FP64 pipe 3 us.  Three windows of slots in turn: the one of the
 * reduction before last is read by nobody when it is written again. */
template <int NS, class Of>
__device__ bool power_sums(const PowerArgs &a, Red<NS, 0> &r, unsigned &sense, int &window, double *smem, int *sok,
                           double (&tot)[NS], Of of) {
    constexpr int NW = kPowerThreads / 32;
    double *buf = a.part + (size_t)window * gridDim.x * kSlot;
    window = window == 2 ? 0 : window + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    static_assert(NS <= NW, "a warp per term");
    /* lane by lane over the warps first: NW + 5 FP64 instructions a term, where
     * a sum per warp would take 5 NW */
#pragma unroll
    for (int i = 0; i < NS; ++i) smem[(size_t)i * kPowerThreads + threadIdx.x] = r.s[i];
    __syncthreads();
    if (warp < NS) {
        const double *t = smem + (size_t)warp * kPowerThreads + lane;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int w = 0; w < NW; ++w) acc[w & 3] += t[32 * w];
        const double sum = warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
        if (lane == 0) buf[(size_t)blockIdx.x * kSlot + warp] = sum;
    }
    if (!grid_barrier(a.bar, gridDim.x, a.bar_extra, a.spin_limit, sense, sok)) return false;
    if (warp < NS) {
        double acc = 0.0;
        for (int b = lane; b < (int)gridDim.x; b += 32) acc += __ldcg(buf + (size_t)b * kSlot + warp);
        acc = warp_sum(acc);
        if (lane == 0) smem[warp] = of(warp, acc);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NS; ++i) tot[i] = smem[i];
    __syncthreads();
    return true;
}

struct PowerColEpi {
    struct In {};
    double *dp, inv;
    __device__ __forceinline__ In fetch(int) const { return In{}; }
    __device__ __forceinline__ void finish(int j, double s, const In &, Red<1, 0> &) const { dp[j] = inv * s; }
};
/* as EpiPowerRows; the quotient is inv s[0] */
struct PowerRowEpi {
    struct In {
        double v, last;
    };
    const double *v, *last;
    double *vn;
    double back; /* s2 last_inv */
    __device__ __forceinline__ In fetch(int i) const { return In{__ldcg(v + i), last ? __ldcg(last + i) : 0.0}; }
    __device__ __forceinline__ void finish(int i, double s, const In &in, Red<3, 0> &r) const {
        vn[i] = s;
        r.s[0] = fma(in.v, s, r.s[0]);
        r.s[1] = fma(s, s, r.s[1]);
        const double w = fma(-back, in.last, in.v);
        r.s[2] = fma(w, w, r.s[2]);
    }
};
/* as EpiPowerQ */
struct PowerQEpi {
    struct In {
        double v;
    };
    const double *v;
    double *av;
    double inv, lmax;
    int shifted;
    /* the quotient is inv s[0] */
    __device__ __forceinline__ In fetch(int i) const { return In{__ldcg(v + i)}; }
    __device__ __forceinline__ void finish(int j, double s, const In &in, Red<2, 0> &r) const {
        const double q = inv * (shifted ? fma(lmax, in.v, -s) : s);
        av[j] = q;
        r.s[0] = fma(in.v, q, r.s[0]);
        r.s[1] = fma(q, q, r.s[1]);
    }
};

/* Q: the extreme eigenvalues (run_power_q); otherwise sigma_max(A)
 * (run_power_a), in the same steps and with the same tests. */
template <bool Q>
__global__ void __launch_bounds__(kPowerThreads, 1) k_facp_power(PowerArgs a) {
    __shared__ double smem[(Q ? 2 : 3) * kPowerThreads];
    __shared__ int sok;
    unsigned sense = 0u;
    int window = 0;
    double *v = a.v, *vn = a.vn, *last = a.last;
    double inv;
    auto sweep = [&](int len, auto term, auto of) {
        Red<1, 0> r;
        r.zero();
        for (int i = blockIdx.x * kPowerThreads + threadIdx.x; i < len; i += gridDim.x * kPowerThreads) {
            const double t = term(i);
            r.s[0] = fma(t, t, r.s[0]);
        }
        double t[1];
        const bool ok = power_sums<1>(a, r, sense, window, smem, &sok, t, of);
        return ok ? t[0] : -1.0;
    };
    inv = sweep(a.m, [&](int i) { return __ldcg(v + i); }, [](int, double x) { return rsqrt(x); });
    bool ok = !(inv < 0.0);
    double value = Q ? 0.0 : 1.0, back = 0.0;
    int it = 0;
    for (; ok && it < a.max_iter; ++it) {
        if constexpr (Q) {
            Red<2, 0> r;
            r.zero();
            PowerQEpi e{v, vn, inv, a.lam_max, a.shifted};
            power_rows(a.at, v, e, r);
            double t[2];
            ok = power_sums<2>(a, r, sense, window, smem, &sok, t,
                               [&](int q, double x) { return q == 0 ? inv * x : rsqrt(x); });
            if (!ok) break;
            const double old = value;
            value = t[0];
            if (it > 0 && fabs(value - old) < a.tol) break;
            inv = t[1];
            double *w = v;
            v = vn;
            vn = w;
        } else {
            Red<1, 0> none;
            PowerColEpi ec{a.dp, inv};
            power_rows(a.at, v, ec, none);
            ok = grid_barrier(a.bar, gridDim.x, a.bar_extra, a.spin_limit, sense, &sok);
            if (!ok) break;
            Red<3, 0> r;
            r.zero();
            PowerRowEpi er{v, it > 0 ? last : nullptr, vn, back};
            power_rows(a.a, a.dp, er, r);
            double t[3];
            ok = power_sums<3>(a, r, sense, window, smem, &sok, t,
                               [&](int q, double x) { return q == 0 ? inv * x : q == 1 ? rsqrt(x) : x; });
            if (!ok) break;
            if (it > 0 && t[2] < a.tol2) {
                --it;
                break;
            }
            value = t[0];
            back = value * inv;
            inv = t[1];
            double *w = last;
            last = v;
            v = vn;
            vn = w;
        }
    }
    if (!Q && ok && it == a.max_iter && it > 0) { /* the last step's residual */
        const double res = sweep(a.m, [&](int i) { return fma(-back, __ldcg(last + i), __ldcg(v + i)); },
                                 [](int, double x) { return x; });
        ok = !(res < 0.0);
        if (ok && res < a.tol2) --it;
    }
    if (threadIdx.x != 0) return;
    if (!ok) {
        atomicExch(&a.ctl->status, 1);
    } else if (blockIdx.x == 0) {
        a.ctl->power_value = Q ? (a.shifted ? a.lam_max - value : value) : sqrt(value);
        a.ctl->power_iters = it;
    }
}

} // namespace facp
} // namespace pdal
