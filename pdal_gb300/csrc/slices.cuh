/*
 * slices.cuh -- lane-major ("sliced") copies of a CSR matrix, and the LP
 * iteration and sigma_max estimate of a problem that fits on the chip as one
 * resident launch whose warps hand the iterates to each other entry by entry
 * (sm_103a).
 *
 * A slice is what one warp sums: 32 lanes, each with its own list of
 * nonzeros, stored entry by entry (entry j of every lane side by side), so a
 * warp's loads of column indices and values are whole 128-byte lines and no
 * staging, row pointers or block barriers stand between a load and its
 * product.  Rows are sorted by length within a window, so the lanes of a
 * slice end together.  Lanes cost and save: a lane's entries are dependent
 * rounds of gathers, but an FP64 instruction holds an SM's FP64 pipe for 19
 * cycles however many lanes are active, and a dependent one waits 64 (measured),
 * so the epilogues of many lanes a row, in a few lanes of a warp, bound the
 * iteration of an LP that fills the SMs with one (CpalSolver::plan_flow draws
 * the line).  persistent_loop = 1 keeps the row-block engine's lanes and
 * summation order: bit-identical sums.
 *
 * k_flow runs the iterations of one evaluation block, with the matrices in
 * the shared memory of one CTA per SM, in one of two forms:
 *
 * tagged   Every entry of x-bar and u is stored together with the number of
 *          the iteration that made it (one 64-bit word in FP32, two in FP64),
 *          and a warp that gathers an entry polls it until it carries the
 *          number it needs.  An exchange is one store and the polls that see
 *          it, about 1,800 cycles over the whole GPU, where a grid barrier
 *          takes 2,300, without the gather behind it, and a launch more.  One buffer
 *          per vector is enough: an entry x-bar_j is gathered exactly by the
 *          rows with a nonzero in column j, and the next x-bar_j is made from
 *          the u of those rows, each stored after its row has gathered
 *          x-bar_j; the same holds for u with the roles exchanged.  No warp
 *          waits for a later one: waits are for the previous product only,
 *          all CTAs are resident (cooperative launch), every poll is bounded.
 * barrier  Plain vectors and a grid barrier between the products: polling
 *          rounds repeat every gather, which costs more than it saves once
 *          the gathers themselves, 32-byte sectors of L2, take the time.
 *
 * Microseconds per iteration (random LPs, k nonzeros per column, 0.4 rows per
 * column, GB300):
 *   nonzeros  k  form    launches  tagged  barrier
 *     20,000  8  FP64       7.8      5.1     6.8
 *                FP32       5.5      2.9     4.7
 *     60,000  1  FP64      10.4      7.5     8.6
 *                FP32       5.9      5.6     5.0
 *     60,000  8  FP64      10.9      5.3     7.5
 *                FP32       6.1      3.0     5.1
 *    100,000  8  FP64      14.1      7.6     9.0
 *                FP32       6.6      3.3     5.8
 *    200,000  1  FP64      17.2     18.4    20.1
 *                FP32       7.7     10.0     8.1
 *    200,000  8  FP64      15.0     10.4    10.8
 *                FP32       7.0      9.3     7.0
 *    400,000  8  FP64      16.9     12.4    12.6
 *                FP32       8.7     12.5     8.9
 *    700,000  8  FP64      29.4     25.1    18.8
 *                FP32      14.2     22.4    13.4
 *  1,000,000  2  FP64      55.3     39.6    40.0
 *                FP32      18.0     21.3    17.0
 *  1,000,000  8  FP64      38.8     27.8    20.8
 *                FP32      17.8     23.5    14.6
 *  1,000,000 20  FP64      34.2     21.0    20.2
 *                FP32      15.5     20.8    17.6
 * (CpalSolver::flow_form holds the lines drawn from these.)  The tagged power
 * iteration, k_power_flow, takes 6.7 / 7.0 / 8.0 / 10.5 / 24.2 us a step at
 * 20,000 / 100,000 / 200,000 / 400,000 / 1,000,000 nonzeros of k = 8, where five
 * launches take 17.0 / 20.9 / 22.6 / 25.2 / 37.8.
 */
#pragma once

#include "cpal_kernels.cuh"

namespace pdal {

constexpr int kFlowWarps = 16; /* warps of a CTA that work on slices, at most (the launch says how many) */

/* ------------------------------------------------------------------ */
/* tagged words                                                        */
/* ------------------------------------------------------------------ */
template <typename T>
struct Tagged;
template <>
struct Tagged<float> {
    using Word = unsigned long long;
    static __device__ __forceinline__ void store(Word *p, float v, unsigned tag) {
        const Word w = ((Word)tag << 32) | __float_as_uint(v);
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
    }
    static __device__ __forceinline__ Word load(const Word *p) {
        Word w;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
        return w;
    }
    static __device__ __forceinline__ bool is(const Word &w, unsigned tag) { return (unsigned)(w >> 32) == tag; }
    static __device__ __forceinline__ float value(const Word &w) { return __uint_as_float((unsigned)w); }
};
/* each half of the double carries the tag, so the two 64-bit words need not
 * be written or read together */
template <>
struct Tagged<double> {
    using Word = ulonglong2;
    static __device__ __forceinline__ void store(Word *p, double v, unsigned tag) {
        const unsigned long long t = (unsigned long long)tag << 32, b = (unsigned long long)__double_as_longlong(v);
        asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(t | (b & 0xffffffffull)),
                     "l"(t | (b >> 32))
                     : "memory");
    }
    static __device__ __forceinline__ Word load(const Word *p) {
        Word w;
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w.x), "=l"(w.y) : "l"(p) : "memory");
        return w;
    }
    static __device__ __forceinline__ bool is(const Word &w, unsigned tag) {
        return (unsigned)(w.x >> 32) == tag && (unsigned)(w.y >> 32) == tag;
    }
    static __device__ __forceinline__ double value(const Word &w) {
        return __longlong_as_double((long long)((w.y << 32) | (w.x & 0xffffffffull)));
    }
};

/* a vector of tagged words, its entries 1 << shift words apart */
template <typename T>
struct TaggedVec {
    typename Tagged<T>::Word *p;
    int shift;
    __device__ __forceinline__ typename Tagged<T>::Word *at(int i) const { return p + ((size_t)i << shift); }
};

/* a poll loop that runs out, or sees that another one did, gives up */
struct FlowGuard {
    int *err;
    int limit;
    /* `weight`: polls of this wait in the time of an L2 round trip */
    __device__ __forceinline__ bool expired(int &spins, int weight = 1) const {
        ++spins;
        if (spins > limit * weight) {
            atomicExch(err, 2);
            return true;
        }
        return (spins & 255) == 0 && *(volatile int *)err != 0;
    }
};

/* Grid barrier (for the problems whose gathers are too
 * many to poll): one release-add per CTA on a counter that is zero at launch,
 * then an acquire poll until all CTAs of this barrier have arrived.  All
 * warps of a CTA call every wait(), a warp whose own work gave up (!good) with
 * them: a warp that left by itself would leave its CTA's others in bar.sync for
 * good.  The same wait() then returns false in all of them, without polling. */
struct FlowBarrier {
    unsigned *count;
    int *ok;     /* shared */
    int *failed; /* shared, zero at first */
    FlowGuard guard;
    unsigned target;
    __device__ __forceinline__ bool wait(bool good_so_far) {
        target += gridDim.x;
        if (!good_so_far) *(volatile int *)failed = 1;
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
            int spins = 0, good = *(volatile int *)failed == 0;
            while (good) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
                if (v >= target) break;
                if (guard.expired(spins)) {
                    good = 0;
                    break;
                }
            }
            *ok = good;
        }
        __syncthreads();
        return *ok != 0;
    }
};

/* ------------------------------------------------------------------ */
/* slices                                                              */
/* ------------------------------------------------------------------ */
/* One matrix in slices; cta[b]..cta[b+1] are the slices of CTA b. */
template <typename T>
struct SliceDev {
    const int4 *__restrict__ desc; /* {first entry, entries of the longest lane, g, slot}: g lanes per
                                      row, or g = 0 for a part of a long row (slot of its sum) */
    const int2 *__restrict__ rl;   /* per lane: row (g = 0: long row id; -1: none), its entries */
    const int *__restrict__ ci;
    const T *__restrict__ val;
    const int *__restrict__ cta;
    const int4 *__restrict__ linfo; /* RowPlanDev's */
    const int *__restrict__ rp;
    typename Tagged<T>::Word *part; /* eight per piece of a long row */
    int nslices, nlong, S;
    bool chain; /* row sums in the row-block product's order */
};

/* position in the CSR arrays of a lane's entry 0, and the step between its
 * entries */
__device__ __forceinline__ int slice_source(const int4 &d, const int2 &rl, int lane, const int *__restrict__ rp,
                                            const int4 *__restrict__ linfo, int S, int &step) {
    if (d.z > 0) {
        step = d.z;
        return rp[rl.x] + (lane & (d.z - 1));
    }
    const int4 li = linfo[rl.x];
    step = kThreads;
    return li.w + (d.w / 8 - li.z) * S + (d.w & 7) * 32 + lane;
}

/* column indices (once) and values (after the equilibration) of every slice
 * from the CSR arrays; a warp per slice */
template <typename Src, typename Dst>
__global__ void k_slice_pack(int nslices, const int4 *__restrict__ desc, const int2 *__restrict__ rl,
                             const int4 *__restrict__ linfo, int S, const int *__restrict__ rp,
                             const Src *__restrict__ src, Dst *dst) {
    const int lane = threadIdx.x & 31;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslices; s += (gridDim.x * blockDim.x) >> 5) {
        const int4 d = desc[s];
        const int2 e = rl[(size_t)s * 32 + lane];
        if (e.y == 0) continue;
        int step;
        const int k = slice_source(d, e, lane, rp, linfo, S, step);
        for (int j = 0; j < e.y; ++j) dst[d.x + j * 32 + lane] = (Dst)src[k + j * step];
    }
}

/* gathers in flight per lane (FP64 has half the registers to hold them) */
template <typename T>
constexpr int kSliceUnroll = sizeof(T) == 4 ? 8 : 4;

/* the vector a product gathers, complete before the launch */
template <typename T>
struct PlainSource {
    const T *p;
    template <int U>
    __device__ __forceinline__ bool gather(const int (&c)[U], int n, T (&g)[U]) const {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u < n) g[u] = __ldcg(p + c[u]);
        return true;
    }
};
/* the vector a product gathers, entry by entry as its tag becomes `tag` */
template <typename T>
struct TaggedSource {
    TaggedVec<T> v;
    unsigned tag;
    FlowGuard guard;
    template <int U>
    __device__ __forceinline__ bool gather(const int (&c)[U], int n, T (&g)[U]) const {
        typename Tagged<T>::Word w[U];
        unsigned need = n >= U ? (1u << U) - 1u : (n > 0 ? (1u << n) - 1u : 0u);
        int spins = 0;
        bool ok = true;
        while (need) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (need & (1u << u)) w[u] = Tagged<T>::load(v.at(c[u]));
#pragma unroll
            for (int u = 0; u < U; ++u)
                if ((need & (1u << u)) && Tagged<T>::is(w[u], tag)) {
                    g[u] = Tagged<T>::value(w[u]);
                    need &= ~(1u << u);
                }
            if (need && guard.expired(spins)) {
                ok = false;
                break;
            }
        }
        return ok;
    }
};

/* A lane's sum over its entries: a chain of fused multiply-adds in entry
 * order, or (FP64, chain = false) four chains, since a dependent FP64
 * instruction takes 64 cycles.  False when a gather gave up. */
template <typename T, class Src>
__device__ __forceinline__ bool slice_dot(const int *ci, const T *val, int L, int len, const Src &src, bool chain,
                                          T &acc) {
    constexpr int U = kSliceUnroll<T>;
    acc = T(0);
    T part[3] = {T(0), T(0), T(0)};
    bool ok = true;
    for (int j = 0; j < L; j += U) {
        int c[U];
        T v[U], g[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            g[u] = T(0);
            if (j + u < len) {
                c[u] = ci[(j + u) * 32];
                v[u] = val[(j + u) * 32];
            }
        }
        ok = src.template gather<U>(c, len - j, g) && ok;
        if (sizeof(T) == 4 || chain) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j + u < len) acc = vfma(v[u], g[u], acc);
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (j + u < len) {
                    T &a = (u & 3) ? part[(u & 3) ? (u & 3) - 1 : 0] : acc;
                    a = vfma(v[u], g[u], a);
                }
        }
    }
    if (!(sizeof(T) == 4 || chain)) acc = (acc + part[0]) + (part[1] + part[2]);
    return ok;
}

/* the CTA's share of the packed matrix, copied to shared memory at `at` */
template <typename T>
struct SliceShare {
    const int *ci;
    const T *val;
    int base, s0, s1;
    int4 d; /* the warp's first slice and the lane's entry in it */
    int2 e;
};
template <typename T>
__device__ __forceinline__ SliceShare<T> slice_share(const SliceDev<T> &M, unsigned char *&at) {
    SliceShare<T> r;
    r.s0 = M.cta[blockIdx.x];
    r.s1 = M.cta[blockIdx.x + 1];
    r.base = r.s0 < r.s1 ? M.desc[r.s0].x : 0;
    int end = r.base;
    if (r.s0 < r.s1) {
        const int4 last = M.desc[r.s1 - 1];
        end = last.x + 32 * last.y;
    }
    const int len = end - r.base; /* a multiple of 32: every copy below is of whole 16-byte vectors */
    T *v = reinterpret_cast<T *>(at);
    int *c = reinterpret_cast<int *>(at + (size_t)len * sizeof(T));
    at += (size_t)len * (sizeof(T) + sizeof(int));
    const int4 *gc = reinterpret_cast<const int4 *>(M.ci + r.base);
    const int4 *gv = reinterpret_cast<const int4 *>(M.val + r.base);
    for (int i = threadIdx.x; i < len / 4; i += blockDim.x) reinterpret_cast<int4 *>(c)[i] = gc[i];
    for (int i = threadIdx.x; i < (int)(len * sizeof(T) / 16); i += blockDim.x) reinterpret_cast<int4 *>(v)[i] = gv[i];
    r.ci = c;
    r.val = v;
    const int s = r.s0 + (int)(threadIdx.x >> 5);
    r.d = make_int4(0, 0, 0, -1);
    r.e = make_int2(-1, 0);
    if (s < r.s1) {
        r.d = M.desc[s];
        r.e = M.rl[(size_t)s * 32 + (threadIdx.x & 31)];
    }
    return r;
}

/* The sum of long row `li` of `len` entries from its parts, as they are
 * published under `tag`: eight per piece in order, then the pieces in FP64 in
 * order.  Not inlined: its registers would spill into the products' loops. */
template <typename T>
__device__ __noinline__ bool flow_long_sum(const typename Tagged<T>::Word *part, int4 li, int len, int S, unsigned tag,
                                           FlowGuard guard, T &sum) {
    const int lane = threadIdx.x & 31;
    double tot = 0.0;
    bool ok = true;
    for (int q0 = 0; q0 < li.y; q0 += 32) {
        T t = T(0);
        if (q0 + lane < li.y) {
            /* the piece's parts polled together: one after the other they take
             * a round trip to L2 each */
            const int parts = min(8, (min(S, len - (q0 + lane) * S) + 31) / 32);
            const typename Tagged<T>::Word *p = part + (size_t)(li.z + q0 + lane) * 8;
            T v[8];
            unsigned need = (1u << parts) - 1u;
            int spins = 0;
            while (need) {
                typename Tagged<T>::Word w[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (need & (1u << u)) w[u] = Tagged<T>::load(p + u);
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if ((need & (1u << u)) && Tagged<T>::is(w[u], tag)) {
                        v[u] = Tagged<T>::value(w[u]);
                        need &= ~(1u << u);
                    }
                if (need && guard.expired(spins)) {
                    ok = false;
                    break;
                }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (u < parts) t += v[u];
        }
        const int n = min(32, li.y - q0);
        for (int k = 0; k < n; ++k) tot += (double)__shfl_sync(0xffffffffu, t, k);
    }
    sum = (T)tot;
    return !__any_sync(0xffffffffu, !ok);
}

/* One product over the slices of this warp: every row's sum goes to
 * epi.finish(row, sum, epi.fetch(row)), whose inputs are loaded before the
 * gathers wait.  The parts of a long row publish their sums under `tag`; the
 * warp that holds the row's first part collects them after its own slices, in
 * the order of rowblock_run_at.  A part without entries publishes nothing (it
 * waits for nothing and could run ahead).  Without LONG there are no long rows:
 * their code costs the products' loops registers (20,000 x 50,000 in FP64 with
 * it 16.5 us an iteration and 17.4 a power step, without 14.9 and 14.5).  wait()
 * returns when a plain source is complete (a tagged one waits by itself).
 * Returns false for the whole warp when a wait gave up. */
template <bool LONG, typename T, class Src, class Epi, class Wait>
__device__ __forceinline__ bool flow_phase(const SliceDev<T> &M, const SliceShare<T> &sh, const Src &src, Epi &epi,
                                           unsigned tag, const FlowGuard &guard, int warps, Wait wait) {
    const int lane = threadIdx.x & 31, first = sh.s0 + (int)(threadIdx.x >> 5);
    int4 d = sh.d;
    int2 e = sh.e;
    bool lead = d.z > 0 && e.x >= 0 && (lane & (d.z - 1)) == 0;
    typename Epi::In in;
    if (lead) in = epi.fetch(e.x);
    if (!wait()) return false;
    for (int s = first; s < sh.s1; s += warps) {
        if (s != first) {
            d = M.desc[s];
            e = M.rl[(size_t)s * 32 + lane];
            lead = d.z > 0 && e.x >= 0 && (lane & (d.z - 1)) == 0;
            if (lead) in = epi.fetch(e.x);
        }
        const int at = d.x - sh.base + lane;
        T acc;
        const bool ok = slice_dot<T>(sh.ci + at, sh.val + at, d.y, e.y, src, M.chain, acc);
        if (__any_sync(0xffffffffu, !ok)) return false;
        if (d.z > 0) {
            for (int o = d.z >> 1; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, d.z);
            if (lead) epi.finish(e.x, acc, in);
        } else if (LONG && d.y > 0) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) Tagged<T>::store(M.part + d.w, acc, tag);
        }
    }
    if constexpr (LONG) {
        if (M.nlong == 0) return true;
        for (int s = first; s < sh.s1; s += warps) {
            const int4 d = M.desc[s];
            if (d.z > 0) continue;
            const int4 li = M.linfo[M.rl[(size_t)s * 32].x]; /* {row, pieces, first piece, first entry} */
            if (d.w != 8 * li.z) continue;
            typename Epi::In in;
            if (lane == 0) in = epi.fetch(li.x);
            T tot;
            if (!flow_long_sum<T>(M.part, li, M.rp[li.x + 1] - li.w, M.S, tag, guard, tot)) return false;
            if (lane == 0) epi.finish(li.x, tot, in);
        }
    }
    return true;
}

/* ------------------------------------------------------------------ */
/* the iterations of one evaluation block                              */
/* ------------------------------------------------------------------ */
template <typename T>
struct FlowArgs {
    SliceDev<T> at, a;
    PrimalArgs<T> pa;
    DualArgs<T> da;
    const T *gat; /* gathered by the first primal product: u (beta > 0) or y */
    TaggedVec<T> xt, ut; /* x-bar and u (or y); no tag in 1..F before the launch but F */
    CpalState *st;
    const typename WeightT<T>::type *wt;
    int F;
    FlowGuard guard;
    unsigned *bar; /* the barrier form's counter */
};

/* r v + (1 - r) old; with the default r = 1 that is v */
template <typename T>
__device__ __forceinline__ T reflected(T r, T v, T old) {
    return r == T(1) ? v : r * v + (T(1) - r) * old;
}

/* PrimalEpi with x-bar published; the plain x-bar, x^ and lambda are written
 * in the block's last iteration, for the evaluation */
template <typename T, bool BAR>
struct FlowPrimalEpi {
    struct In {
        T x, c, lb, ub;
        typename AnchorT<T>::type x0;
    };
    const FlowArgs<T> &L;
    const Coefs<T> &k;
    T w, omw;
    unsigned tag;
    __device__ __forceinline__ In fetch(int j) const {
        const PrimalArgs<T> &a = L.pa;
        return In{a.x[j], a.c[j], a.lb[j], a.ub[j], a.x0[j]};
    }
    __device__ __forceinline__ void finish(int j, T s, const In &i) const {
        const T t = i.x - k.tau * (i.c - s);
        const T proj = vmax(i.lb, vmin(t, i.ub));
        const T xb = T(2) * proj - i.x;
        if (BAR)
            L.pa.xbar[j] = xb;
        else
            Tagged<T>::store(L.xt.at(j), xb, tag);
        if (tag == (unsigned)L.F) {
            if (!BAR) L.pa.xbar[j] = xb;
            L.pa.xh[j] = proj;
            L.pa.lam[j] = (proj - t) * k.inv_tau;
        }
        const T refl = reflected(k.r, xb, i.x);
        L.pa.x[j] = halpern(w, omw, refl, i.x0);
    }
};

/* DualEpi with u (y when beta = 0) published */
template <typename T, bool BETA, bool BAR>
struct FlowDualEpi {
    using In = DualIn<T>;
    const FlowArgs<T> &L;
    const Coefs<T> &k;
    T w, omw;
    unsigned tag;
    __device__ __forceinline__ In fetch(int i) const {
        DualEpi<T, false, BETA> e;
        e.a = L.da;
        e.k = k;
        return e.fetch(i);
    }
    __device__ __forceinline__ void finish(int i, T p, const In &d) const {
        const DualArgs<T> &a = L.da;
        const T yi = d.y;
        const T zb = vmax(d.lo, vmin(p - yi * k.inv_prox, d.hi));
        const T yn = yi - k.rho * (p - zb);
        const T yb = T(2) * yn - yi;
        const T refl = reflected(k.r, yb, yi);
        const T ynew = halpern(w, omw, refl, d.y0);
        if (!BETA && !BAR) Tagged<T>::store(L.ut.at(i), ynew, tag);
        const bool major = tag == (unsigned)L.F;
        if (BETA) {
            const T axn = halpern(w, omw, reflected(k.r, p, d.ax), d.ax0);
            const T z2 = vmax(d.lo, vmin(axn - ynew * k.inv_beta, d.hi));
            const T un = ynew - k.beta * (axn - z2);
            if (!BAR) Tagged<T>::store(L.ut.at(i), un, tag);
            if (BAR || major) a.u[i] = un;
            a.ax[i] = axn;
        }
        a.y[i] = ynew;
        if (major) {
            a.yh[i] = yn;
            a.ybar[i] = yb;
        }
    }
};

template <typename T, bool BETA, bool BAR, bool LONG>
__global__ void __launch_bounds__(kFlowWarps * 32, 1) k_flow(FlowArgs<T> L) {
    extern __shared__ __align__(16) unsigned char flow_smem[];
    __shared__ int bar_ok, bar_failed;
    /* one read for the CTA: a CTA that gives up sets the status while others
     * start, and a CTA of which a part left would not get through its barriers */
    if (__syncthreads_or(threadIdx.x == 0 ? L.st->status : 0)) return;
    if (threadIdx.x == 0) bar_failed = 0;
    unsigned char *at = flow_smem;
    const SliceShare<T> sp = slice_share(L.at, at), sd = slice_share(L.a, at);
    Coefs<T> k;
    load_coefs(L.st, k);
    __syncthreads();
    FlowBarrier bar{L.bar, &bar_ok, &bar_failed, L.guard, 0u};
    auto none = [] { return true; };
    const int warps = (int)(blockDim.x >> 5);
    bool good = true; /* no wait of this warp has given up */
    for (int i = 1; i <= L.F; ++i) {
        const T w = L.wt[i].w, omw = L.wt[i].omw;
        const unsigned tag = (unsigned)i;
        FlowPrimalEpi<T, BAR> ep{L, k, w, omw, tag};
        FlowDualEpi<T, BETA, BAR> ed{L, k, w, omw, tag};
        if constexpr (BAR) {
            /* a phase is false where its barrier failed, in every warp of the
             * CTA, or where this warp gave up on a long row's parts: then the
             * next barrier takes the CTA out */
            bool left = false;
            auto wait = [&] {
                left = !bar.wait(good);
                return !left;
            };
            auto wait_next = [&] { return i == 1 || wait(); };
            good = flow_phase<LONG, T>(L.at, sp, PlainSource<T>{L.gat}, ep, tag, L.guard, warps, wait_next);
            if (!left) good = flow_phase<LONG, T>(L.a, sd, PlainSource<T>{L.pa.xbar}, ed, tag, L.guard, warps, wait);
            if (left) break;
        } else {
            if (i == 1)
                good = flow_phase<LONG, T>(L.at, sp, PlainSource<T>{L.gat}, ep, tag, L.guard, warps, none);
            else
                good = flow_phase<LONG, T>(L.at, sp, TaggedSource<T>{L.ut, tag - 1, L.guard}, ep, tag, L.guard, warps, none);
            good = good && flow_phase<LONG, T>(L.a, sd, TaggedSource<T>{L.xt, tag, L.guard}, ed, tag, L.guard, warps, none);
            if (!good) break;
        }
    }
    if (!good && (threadIdx.x & 31) == 0) atomicExch(&L.st->status, kStatusDeviceError);
}

/* ------------------------------------------------------------------ */
/* sums over the grid, one step behind                                 */
/* ------------------------------------------------------------------ */
/* Each warp with rows adds its lanes' four sums, the last warp of a CTA to
 * do so adds the warps' in order and publishes the CTA's; one service warp
 * per CTA collects the grid's in a fixed order and hands the totals to its
 * own CTA through shared memory.  Four records may be under way: a CTA
 * publishes record r + 4 after it has seen the totals of record r + 2 or a
 * later one, so every CTA has published r + 2, which its warps do after they
 * have seen the totals of r -- the slots of r are free.  (A warp that takes
 * part publishes, or makes entries that publishing warps wait for; one
 * without either leaves at once, flow_idle.) */
struct FlowSums {
    double warp[4][kFlowWarps][4]; /* [record & 3] */
    int arrived[4];
    volatile int ready[4]; /* record whose totals are in the slot (0: none yet) */
};

/* four sums over a warp in eleven shuffles and six additions: halves of the
 * warp take different sums; lane 8q ends with sum q */
__device__ __forceinline__ double warp_sum4(double a, double b, double c, double d) {
    const int lane = threadIdx.x & 31;
    const bool hi = lane & 16;
    const double k0 = hi ? c : a, k1 = hi ? d : b, o0 = hi ? a : c, o1 = hi ? b : d;
    const double p = k0 + __shfl_xor_sync(0xffffffffu, o0, 16), q = k1 + __shfl_xor_sync(0xffffffffu, o1, 16);
    const bool h2 = lane & 8;
    double r = (h2 ? q : p) + __shfl_xor_sync(0xffffffffu, h2 ? p : q, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    return r;
}

/* `active` warps of the CTA call this for every record */
__device__ __forceinline__ void flow_publish(FlowSums &f, int active, unsigned rec, const double (&s)[4],
                                             Tagged<double>::Word *out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, slot = rec & 3;
    const double r = warp_sum4(s[0], s[1], s[2], s[3]);
    if ((lane & 7) == 0) f.warp[slot][warp][lane >> 3] = r;
    __syncwarp();
    int last = 0;
    if (lane == 0) {
        __threadfence_block();
        last = atomicAdd(&f.arrived[slot], 1) == active - 1;
    }
    if (!__shfl_sync(0xffffffffu, last, 0)) return;
    __threadfence_block();
    if (lane < 4) {
        double t = 0.0;
        for (int w = 0; w < active; ++w) t += f.warp[slot][w][lane];
        Tagged<double>::store(out + (size_t)blockIdx.x * 4 + lane, t, rec);
    }
    if (lane == 0) f.arrived[slot] = 0;
}

/* a warp with no rows of A to publish for and no entries in its columns */
template <typename T>
__device__ __forceinline__ bool flow_idle(const SliceDev<T> &at, const SliceShare<T> &sp, int active, int warps) {
    const int warp = threadIdx.x >> 5;
    if (warp < active) return false;
    for (int s = sp.s0 + warp; s < sp.s1; s += warps)
        if (at.desc[s].y > 0) return false;
    return true;
}

/* Service warp: the totals of record `rec`, lane q & 3 holding total q.
 * CTA 0's collects every CTA's sums -- several loads of a lane in flight, four
 * chains of additions -- and gives each CTA a copy of the totals to poll: 152
 * warps polling the same 152 CTAs' lines take turns at them in L2 (measured:
 * 9.1 us a power step of a 2,000 x 5,000 LP instead of 7.1). */
__device__ __forceinline__ bool flow_collect(Tagged<double>::Word *sums, unsigned rec, const FlowGuard &guard,
                                             double &tot) {
    using W = Tagged<double>;
    const int lane = threadIdx.x & 31, ctas = (int)gridDim.x;
    const W::Word *in = sums + (size_t)(rec & 3) * ctas * 4;
    W::Word *out = sums + (size_t)(4 + (rec & 3)) * ctas * 4;
    bool ok = true;
    int spins = 0;
    if (blockIdx.x != 0) {
        tot = 0.0;
        if (lane < 4) {
            const W::Word *p = out + (size_t)blockIdx.x * 4 + lane;
            W::Word w = W::load(p);
            while (!W::is(w, rec)) {
                if (guard.expired(spins)) {
                    ok = false;
                    break;
                }
                w = W::load(p);
            }
            tot = W::value(w);
        }
        if (__any_sync(0xffffffffu, !ok)) return false;
        tot = __shfl_sync(0xffffffffu, tot, lane & 3);
        return true;
    }
    constexpr int U = 4;
    double acc[U] = {0.0, 0.0, 0.0, 0.0};
    for (int b0 = lane >> 2; b0 < ctas && ok; b0 += 8 * U) {
        unsigned need = 0;
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (b0 + 8 * u < ctas) need |= 1u << u;
        while (need) {
            W::Word w[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (need & (1u << u)) w[u] = W::load(in + (size_t)(b0 + 8 * u) * 4 + (lane & 3));
#pragma unroll
            for (int u = 0; u < U; ++u)
                if ((need & (1u << u)) && W::is(w[u], rec)) {
                    acc[u] += W::value(w[u]);
                    need &= ~(1u << u);
                }
            if (need && guard.expired(spins)) {
                ok = false;
                break;
            }
        }
    }
    if (__any_sync(0xffffffffu, !ok)) return false;
    tot = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
    for (int o = 16; o >= 4; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    for (int b = lane >> 2; b < ctas; b += 8) W::store(out + (size_t)b * 4 + (lane & 3), tot, rec);
    return true;
}

__device__ __forceinline__ void flow_ready(FlowSums &f, unsigned rec) {
    __threadfence_block();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) f.ready[rec & 3] = (int)rec;
}
__device__ __forceinline__ bool flow_wait(FlowSums &f, unsigned rec, const FlowGuard &guard) {
    int spins = 0;
    bool ok = true;
    /* of shared memory, tens of cycles a poll: as long as the service warp may
     * wait for the other CTAs, whose verdict this one would otherwise preempt */
    while (f.ready[rec & 3] != (int)rec)
        if (guard.expired(spins, 32)) {
            ok = false;
            break;
        }
    __threadfence_block();
    return !__any_sync(0xffffffffu, !ok);
}

/* ------------------------------------------------------------------ */
/* sigma_max(A)^2                                                      */
/* ------------------------------------------------------------------ */
struct FlowPowerArgs {
    SliceDev<double> at, a;
    double *v0;         /* the start vector, plain */
    double *hist[4];    /* the last vectors, each read by the thread that wrote it */
    TaggedVec<double> dt, vt; /* A^T v and v, tags zero before the launch */
    Tagged<double>::Word *sums; /* [CTAs' sums, totals][record & 3][CTA][4], tags zero before the launch */
    PowerState *ps;
    FlowGuard guard;
};

struct FlowStoreEpi {
    struct In {};
    TaggedVec<double> out;
    unsigned tag;
    double scale; /* the vector's, once per row: FP64 products bound the step */
    __device__ __forceinline__ In fetch(int) const { return In{}; }
    __device__ __forceinline__ void finish(int j, double s, const In &) const {
        Tagged<double>::store(out.at(j), scale * s, tag);
    }
};

/* Row i of step k: v_{k+1} = s.  The sums v_k . v_{k+1} and |v_{k+1}|^2, and
 * step k-2's share |v_{k-1} a - v_{k-2} b|^2 of the residual. */
struct FlowPowerEpi {
    struct In {
        double v, v1, v2;
    };
    const FlowPowerArgs &L;
    unsigned k;
    double a, b;
    double *s;
    __device__ __forceinline__ In fetch(int i) const {
        return In{L.hist[k & 3][i], k > 2 ? L.hist[(k - 1) & 3][i] : 0.0, k > 2 ? L.hist[(k - 2) & 3][i] : 0.0};
    }
    __device__ __forceinline__ void finish(int i, double x, const In &in) const {
        Tagged<double>::store(L.vt.at(i), x, k);
        L.hist[(k + 1) & 3][i] = x;
        s[0] += in.v * x;
        s[1] += x * x;
        if (k > 2) {
            const double d = in.v1 * a - b * in.v2;
            s[2] += d * d;
        }
    }
};

/*
 * The power iteration of k_power_* in one launch.  Step k = 1, 2, ...:
 * dp = c_k A^T v_k, v_{k+1} = A dp.  Any c_k keeps the vectors' direction and
 * the Rayleigh quotient
 *   s2_k = v_k . v_{k+1} / (c_k |v_k|^2),
 * so 1/|v_k| is foretold from the sums of step k-2, which takes the grid's sums
 * off the critical path: with the growth g = |v_{k-1}| / (c_{k-2} |v_{k-2}|) of
 * that step, |v_k| is about c_{k-1} g |v_{k-1}|.  Then |v_{k+1}| = g_k g_{k-1} /
 * g_{k-2}, about the largest eigenvalue, as with 1/|v_k| itself (c_1 and c_2
 * are that, c_3 = c_2; 1/|v_{k-1}| for c_k, one scalar less, swings the norm up
 * to the eigenvalue's square, whose own square leaves the range of a double for
 * entries of 1e39).  The residual of step k, |v_{k+1} / (c_k |v_k|) - s2_k v_k / |v_k||,
 * is added element by element in step k+2 and tested in step k+4; the steps
 * run in excess change nothing, s2 is that of the step whose residual passed.
 * One warp more than the workers (the service warp) collects the sums.
 */
struct FlowScalars {
    double c, a, b; /* scale of step rec + 2 (rec = 1: of step 2 too); the residual's coefficients of step rec */
    int done;
};

template <bool LONG>
__global__ void __launch_bounds__(kFlowWarps * 32 + 32, 1) k_power_flow(FlowPowerArgs L, int max_steps) {
    extern __shared__ __align__(16) unsigned char flow_smem[];
    __shared__ FlowSums f;
    __shared__ FlowScalars sc[4];
    if (L.ps->done) return; /* written at the end of a launch only */
    if (threadIdx.x < 4) {
        f.arrived[threadIdx.x] = 0;
        f.ready[threadIdx.x] = 0;
    }
    unsigned char *at = flow_smem;
    const SliceShare<double> sp = slice_share(L.at, at), sd = slice_share(L.a, at);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double c1 = L.ps->inv, n1 = L.ps->vsq, tol = L.ps->tol;
    const int warps = (int)(blockDim.x >> 5) - 1;
    const int active = max(1, min(sd.s1 - sd.s0, warps)); /* warps that publish sums */
    /* every step whose residual may be wanted, plus the four that follow it */
    const int last = max_steps + 4;
    if (warp == warps) {
        double ck[4], nk[4], s2k[4]; /* by step & 3 */
        ck[1] = c1;
        nk[1] = n1;
        for (int rec = 1; rec <= last; ++rec) {
            double tot;
            if (!flow_collect(L.sums, (unsigned)rec, L.guard, tot)) return;
            const double dot = __shfl_sync(0xffffffffu, tot, 0), nn = __shfl_sync(0xffffffffu, tot, 1),
                         rr = __shfl_sync(0xffffffffu, tot, 2);
            const double c = ck[rec & 3], n = nk[rec & 3];
            nk[(rec + 1) & 3] = nn;
            if (rec == 1) ck[2] = 1.0 / sqrt(nn);
            ck[(rec + 2) & 3] = c * sqrt(n) / (ck[(rec + 1) & 3] * nn);
            const double s2 = dot / (c * n), inv_n = 1.0 / sqrt(n);
            /* the residual of step rec - 2 */
            const int step = rec - 2;
            int done = 0;
            if (step >= 1 && (sqrt(rr) < tol || step >= max_steps)) {
                done = 1;
                if (blockIdx.x == 0 && lane == 0) {
                    L.ps->s2 = s2k[step & 3];
                    L.ps->res = sqrt(rr);
                    L.ps->iters = step;
                    L.ps->done = 1;
                }
            }
            s2k[rec & 3] = s2;
            if (lane == 0) sc[rec & 3] = FlowScalars{ck[(rec + 2) & 3], inv_n / c, s2 * inv_n, done};
            flow_ready(f, (unsigned)rec);
            if (done) return;
        }
        return;
    }
    if (flow_idle(L.at, sp, active, warps)) return;
    auto none = [] { return true; };
    for (int k = 1; k <= last; ++k) {
        double c = c1, a = 0.0, b = 0.0;
        if (k > 1) {
            const int rec = max(k - 2, 1); /* c_3 = c_2 */
            if (!flow_wait(f, (unsigned)rec, L.guard)) return;
            const FlowScalars s = sc[rec & 3];
            if (s.done) return;
            c = s.c;
            a = s.a;
            b = s.b;
        }
        FlowStoreEpi ec{L.dt, (unsigned)k, c};
        bool ok;
        if (k == 1)
            ok = flow_phase<LONG, double>(L.at, sp, PlainSource<double>{L.v0}, ec, (unsigned)k, L.guard, warps, none);
        else
            ok = flow_phase<LONG, double>(L.at, sp, TaggedSource<double>{L.vt, (unsigned)(k - 1), L.guard}, ec, (unsigned)k,
                               L.guard, warps, none);
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        FlowPowerEpi er{L, (unsigned)k, a, b, s};
        ok = ok && flow_phase<LONG, double>(L.a, sd, TaggedSource<double>{L.dt, (unsigned)k, L.guard}, er, (unsigned)k,
                                 L.guard, warps, none);
        if (!ok) return;
        if (warp < active) flow_publish(f, active, (unsigned)k, s, L.sums + (size_t)(k & 3) * gridDim.x * 4);
    }
}

} // namespace pdal
