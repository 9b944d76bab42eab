// fit_cluster.cu -- a mid-size graph's fit in one launch of one thread-block
// cluster, every CTA with the whole state in its own shared memory.
//
// Reference: libdress/src/dress.c:546-608 (the iteration), :500-529 (the merge
// walk that pairs the common neighbours of an edge).
//
// Each CTA owns a range of vertices and one of edges (ranges, so that a warp's
// 32 remote stores are neighbours).  It gathers from its own copy of the values
// and norms and writes what it updates into all copies; a cluster barrier ends
// each phase.
// What bounds it is latency: a sweep is two phases of one dependent chain each
// (ids, gathers, additions, root or quotient) and their barriers, and a gather
// from another SM's memory takes several times as long as a local one.
// Measured on G(2000, 10000), 22 sweeps: 353 us with the state spread over the
// cluster and every term gathered from its owner, plus 93 us for the pairs on
// one block of another launch; 150 us in all this way (287 us with items dealt
// out in turn: a warp's remote stores then touch 32 places).
//
// Sums are the batch kernel's: products checked once a value against a range in
// which all additions of rounding errors are exact in any order
// (fast_range, delta_nabla.cpp), so a row's partial sums over several lanes
// merge to the reference's bits.  TwoSum instead of Fast2Sum: a lane's partial
// sum may start with its smallest term.  A product outside the range ends the
// kernel with ST_FITS = 0.
//
// Graphs whose products leave the range are fitted with a certificate per sum
// (CERT: CSum, common.cuh), from the start, by the same kernel; another launch
// over the whole device finds the pairs first, whose walks would otherwise be a
// part of eight SMs' work.  (Going on from the sweep that left, instead, saved a
// few microseconds and cost the uncertified kernel 4 to 8 % through its
// registers.)  G(2000, 10000) with one weight of zero: 314 us a
// call; 1,503 through the multi-kernel fit, 564 by an earlier certified cluster
// kernel that gathered every term from its owner.
#include <algorithm>
#include <climits>
#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>

#include "batch.h"
#include "common.cuh"

namespace dress {
namespace {

constexpr int CTAS = 8, THREADS = 1024;
constexpr int OWN = 4;                       // edges a thread owns, at most
constexpr size_t CLUSTER_SMEM = 227 * 1024;

__device__ __forceinline__ unsigned cta_rank()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// the address of another CTA's copy of a shared-memory word
__device__ __forceinline__ unsigned at_rank(unsigned a, unsigned r)
{
    unsigned d;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(r));
    return d;
}
__device__ __forceinline__ void put(unsigned a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ double take(unsigned a)
{
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void put_u32(unsigned a, unsigned v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// s + c = the exact sum so far (TwoSum; c is exact within the fast range)
struct ExactSum {
    double s, c;
    __device__ __forceinline__ void init() { s = c = 0.0; }
    __device__ __forceinline__ void start(double x) { s = x; }
    __device__ __forceinline__ void add(double x)
    {
        const double t = dadd(s, x), b = dsub(t, s);
        c = dadd(c, dadd(dsub(s, dsub(t, b)), dsub(x, b)));
        s = t;
    }
    __device__ __forceinline__ void merge_lanes(int width)
    {
        for (int o = width >> 1; o > 0; o >>= 1) {
            const double os = __shfl_xor_sync(0xffffffffu, s, o), oc = __shfl_xor_sync(0xffffffffu, c, o);
            c = dadd(c, oc);
            add(os);
        }
    }
    __device__ __forceinline__ double value() const { return dadd(s, c); }
};
struct CertSum : CSum {
    __device__ __forceinline__ void start(double x) { add(x); }
};

struct Args {
    int N, E, fwd, max_iter, lpv, twice;     // lanes to a vertex; both value buffers fit
    int spread;                              // a norm is held by its vertex's CTA only
    int slot_room;                           // slot ids there is room for
    double eps;
    ImageShape img;
    const unsigned char *data;
    unsigned *pairs, *cursor;                // room for every pair; words taken (CERT: edge_pairs first)
    double *values;
    unsigned long long *stats;
};

// CERT: every edge's first pair and their count, ahead of the pairs.  (In their
// place rather than by a pointer of its own: 8 bytes more of arguments change the
// other kernel's registers, and it took 3 % longer.)
__device__ __forceinline__ uint2 *edge_pairs(const Args &A) { return (uint2 *)A.pairs; }
template <bool CERT>
__device__ __forceinline__ unsigned *all_pairs(const Args &A)
{
    return CERT ? A.pairs + 2 * A.E : A.pairs;
}

// CERT: the pairs of every edge, a thread each (the merge walk of the kernel below).
constexpr int PAIR_THREADS = 64;
__global__ void __launch_bounds__(PAIR_THREADS) k_cluster_pairs(const Args A)
{
    const ClusterLayout L = cluster_layout(A.N, A.E, A.img.Q, A.img.uniform, A.img.has_nw, A.img.has_dinit);
    const unsigned short *off = (const unsigned short *)(A.data + L.off), *tgt = (const unsigned short *)(A.data + L.tgt);
    const unsigned short *eid = (const unsigned short *)(A.data + L.eid);
    const int e = blockIdx.x * PAIR_THREADS + threadIdx.x, lane = threadIdx.x & 31;
    int iu0 = 0, iv0 = 0, iu_end = 0, iv_end = 0;
    unsigned count = 0;
    if (e < A.E) {
        const unsigned uv = ((const unsigned *)(A.data + L.uv))[e], u = uv & 0xffffu, v = uv >> 16;
        iu0 = off[u], iu_end = off[u + 1];
        iv0 = off[v], iv_end = off[v + 1];
        for (int iu = iu0, iv = iv0; iu < iu_end && iv < iv_end;) {
            const unsigned x = tgt[iu], y = tgt[iv];
            count += x == y;
            iu += x <= y;
            iv += x >= y;
        }
    }
    unsigned at = count;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += y;
    }
    unsigned base = 0;
    if (lane == 31 && at) base = atomicAdd(A.cursor, at);
    at += __shfl_sync(0xffffffffu, base, 31) - count;
    if (e >= A.E) return;
    edge_pairs(A)[e] = make_uint2(at, count);
    unsigned *pairs = all_pairs<true>(A);
    const unsigned end = at + count;
    for (int iu = iu0, iv = iv0; at < end;) {
        const unsigned x = tgt[iu], y = tgt[iv];
        if (x == y) pairs[at++] = (unsigned)eid[iu] | (unsigned)eid[iv] << 16;
        iu += x <= y;
        iv += x >= y;
    }
}

// One CTA's shared memory: values (twice where they fit), norms; control words.
struct Ctl {
    unsigned long long largest;
    double maxima[CTAS];                     // every CTA's, on rank 0
    unsigned far[3], bad, part[33], base;
};

template <bool CERT>
__global__ void __launch_bounds__(THREADS, 1) k_fit_cluster(const Args A)
{
    extern __shared__ __align__(16) unsigned char smem[];
    Ctl *ctl = (Ctl *)smem;
    double *x0 = (double *)(smem + 256);
    double *x1 = A.twice ? x0 + A.E : x0;
    double *vd = x1 + A.E;
    const unsigned rank = cta_rank();
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, N = A.N, E = A.E;
    const ClusterLayout L = cluster_layout(N, E, A.img.Q, A.img.uniform, A.img.has_nw, A.img.has_dinit);
    const unsigned *uv = (const unsigned *)(A.data + L.uv);
    const unsigned short *off = (const unsigned short *)(A.data + L.off);
    const unsigned short *eid = (const unsigned short *)(A.data + L.eid);
    const double *w = (const double *)(A.data + L.w);
    const double *nw = A.img.has_nw ? (const double *)(A.data + L.nw) : nullptr;
    const bool one_w = A.img.uniform != 0;
    // sums in units of the weight where that is one power of two; certified sums
    // take every product in full (units could over- or underflow)
    const bool uni = one_w && !CERT;
    const int nv = (N + CTAS - 1) / CTAS, ne = (E + CTAS - 1) / CTAS;
    const int u0 = min(N, (int)rank * nv), u1 = min(N, u0 + nv), e0 = min(E, (int)rank * ne), e1 = min(E, e0 + ne);
    const double wc = A.img.wc, base4 = uni ? ddiv(4.0, wc) : 4.0;

    // ---- pairs of this thread's edges, by merge walks over staged rows -------------
    unsigned own_uv[OWN], first[OWN], count[OWN];
    if (t == 0) {
        ctl->bad = ctl->far[0] = ctl->far[1] = ctl->far[2] = 0;
        ctl->largest = 0ULL;
    }
    if (CERT) {
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            const int e = e0 + j * THREADS + t;
            own_uv[j] = e < e1 ? uv[e] : 0u;
            const uint2 r = e < e1 ? edge_pairs(A)[e] : make_uint2(0u, 0u);
            first[j] = r.x;
            count[j] = r.y;
        }
    } else {
        unsigned short *so = (unsigned short *)x0, *st = so + ((N + 2) & ~1);
        const unsigned short *tgt = (const unsigned short *)(A.data + L.tgt);
        for (int i = t; i <= N; i += THREADS) so[i] = off[i];
        for (int i = t; i < A.img.Q; i += THREADS) st[i] = tgt[i];
        __syncthreads();
        unsigned mine = 0;
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            const int e = e0 + j * THREADS + t;
            count[j] = 0;
            own_uv[j] = 0;
            if (e < e1) {
                own_uv[j] = uv[e];
                const int u = own_uv[j] & 0xffffu, v = own_uv[j] >> 16;
                int iu = so[u], iv = so[v];
                const int iu_end = so[u + 1], iv_end = so[v + 1];
                while (iu < iu_end && iv < iv_end) {
                    const unsigned x = st[iu], y = st[iv];
                    count[j] += x == y;
                    iu += x <= y;
                    iv += x >= y;
                }
            }
            mine += count[j];
        }
        unsigned incl = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) ctl->part[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            unsigned v = ctl->part[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += y;
            }
            ctl->part[lane] = v;
            if (lane == 31) ctl->base = atomicAdd(A.cursor, v);
        }
        __syncthreads();
        unsigned at = ctl->base + incl - mine + (warp > 0 ? ctl->part[warp - 1] : 0u);
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            first[j] = at;
            if (count[j]) {
                const int u = own_uv[j] & 0xffffu, v = own_uv[j] >> 16;
                int iu = so[u], iv = so[v];
                const unsigned end = at + count[j];
                while (at < end) {
                    const unsigned x = st[iu], y = st[iv];
                    if (x == y) A.pairs[at++] = (unsigned)eid[iu] | (unsigned)eid[iv] << 16;
                    iu += x <= y;
                    iv += x >= y;
                }
            }
        }
        __syncthreads();                     // the rows make room for the values
    }
    // this CTA's slot ids, behind the norms where they fit
    const int s0 = off[u0], s1 = off[u1];
    unsigned short *slots = (unsigned short *)(vd + (A.spread ? nv : N));
    const bool held = s1 - s0 <= A.slot_room;
    if (held)
        for (int i = t; i < s1 - s0; i += THREADS) slots[i] = eid[s0 + i];
    const unsigned slots_a = (unsigned)__cvta_generic_to_shared(slots);
    const auto slot = [&](int k) -> int {
        if (!held) return eid[k];
        unsigned short v;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(slots_a + 2u * (unsigned)(k - s0)));
        return v;
    };

    // ---- initial values -------------------------------------------------------------
    {
        const double *dinit = (const double *)(A.data + L.dinit);
        bool out = false;
        for (int e = t; e < E; e += THREADS) {
            const double d = A.img.has_dinit ? dinit[e] : 1.0;
            const double p = uni ? d : dmul(CERT && one_w ? wc : w[e], d);
            x0[e] = p;
            out |= !CERT && (unsigned)__double2hiint(p) - A.img.lo >= A.img.span;
        }
        if (__syncthreads_or(out)) {         // every CTA checks every value: all leave
            if (rank == 0 && t == 0) A.stats[ST_FITS] = 0ULL;
            return;
        }
    }
    double val[OWN];                         // values of this thread's edges
#pragma unroll
    for (int j = 0; j < OWN; ++j) {
        const int e = e0 + j * THREADS + t;
        val[j] = e < e1 ? (A.img.has_dinit ? ((const double *)(A.data + L.dinit))[e] : 1.0) : 0.0;
    }
    const unsigned vd_a = (unsigned)__cvta_generic_to_shared(vd);
    const unsigned far_a = (unsigned)__cvta_generic_to_shared(ctl->far);
    const unsigned bad_a = (unsigned)__cvta_generic_to_shared(&ctl->bad);
    cluster_sync();                          // every CTA runs and has its copy

    // ---- sweeps ------------------------------------------------------------------------
    using Sum = std::conditional_t<CERT, CertSum, ExactSum>;
    const int lpv = A.lpv, sub = t & (lpv - 1);
    int it = 0;
    double lmax = 0.0;
    for (; it < A.max_iter; ++it) {
        for (int b = u0; b < u1; b += THREADS / lpv) {
            const int u = b + t / lpv;
            Sum q;
            q.init();
            if (u < u1) {
                if (sub == 0) q.start(nw ? dmul(base4, nw[u]) : base4);
                int k = off[u] + sub;
                const int end = off[u + 1];
                for (; k + 3 * lpv < end; k += 4 * lpv) {
                    const int i0 = slot(k), i1 = slot(k + lpv), i2 = slot(k + 2 * lpv), i3 = slot(k + 3 * lpv);
                    const double v0 = x0[i0], v1 = x0[i1], v2 = x0[i2], v3 = x0[i3];
                    q.add(v0);
                    q.add(v1);
                    q.add(v2);
                    q.add(v3);
                }
                const int i0 = k < end ? slot(k) : 0, i1 = k + lpv < end ? slot(k + lpv) : 0;
                const int i2 = k + 2 * lpv < end ? slot(k + 2 * lpv) : 0;
                const double v0 = x0[i0], v1 = x0[i1], v2 = x0[i2];
                if (k < end) q.add(v0);
                if (k + lpv < end) q.add(v1);
                if (k + 2 * lpv < end) q.add(v2);
            }
            q.merge_lanes(lpv);
            if (u < u1) {
                double S;
                if constexpr (CERT) {
                    if (!q.result(S)) {      // every lane of the vertex
                        const double *x = x0;
                        const unsigned short *id = eid + off[u];
                        S = sorted_sum_select(nw ? dmul(base4, nw[u]) : base4, off[u + 1] - off[u],
                                              [=](int k, double &v) { return v = x[id[k]], true; });
                    }
                } else {
                    S = q.value();
                }
                const double v = dsqrt(uni ? dmul(wc, S) : S);
                if (A.spread) {
                    if (sub == 0) vd[u - u0] = v;
                } else {
                    for (unsigned r = sub; r < CTAS; r += lpv) put(at_rank(vd_a + 8u * (unsigned)u, r), v);
                }
            }
        }
        cluster_sync();
        bool far = false, out = false;
        lmax = 0.0;
        double p[OWN];
        const unsigned x1_a = (unsigned)__cvta_generic_to_shared(x1);
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
            const int e = e0 + j * THREADS + t;
            p[j] = 0.0;
            if (e < e1) {
                const int u = own_uv[j] & 0xffffu, v = own_uv[j] >> 16;
                const double own = x0[e];
                double nu, nn;
                if (A.spread) {
                    const int ru = u / nv, rv = v / nv;
                    nu = take(at_rank(vd_a + 8u * (unsigned)(u - ru * nv), ru));
                    nn = take(at_rank(vd_a + 8u * (unsigned)(v - rv * nv), rv));
                } else {
                    nu = vd[u];
                    nn = vd[v];
                }
                const double den = dmul(nu, nn);
                double s0 = nw ? dmul(base4, nw[u]) : base4;
                if (!A.fwd) s0 = dadd(s0, nw ? dmul(base4, nw[v]) : base4);
                const double self = dadd(s0, A.fwd ? own : dadd(own, own));
                Sum q;
                q.init();
                q.start(self);
                for (unsigned k = 0; k < count[j]; ++k) {
                    const unsigned pr = all_pairs<CERT>(A)[first[j] + k];
                    q.add(dadd(x0[pr & 0xffffu], x0[pr >> 16]));
                }
                double S;
                if constexpr (CERT) {
                    if (!q.result(S)) {
                        const double *x = x0;
                        const unsigned *pp = all_pairs<CERT>(A) + first[j];
                        S = sorted_sum_select(self, (int)count[j], [=](int k, double &v) {
                            return v = dadd(x[pp[k] & 0xffffu], x[pp[k] >> 16]), true;
                        });
                    }
                } else {
                    S = q.value();
                }
                double r = ddiv(uni ? dmul(wc, S) : S, den);
                if (CERT) r = den > 0.0 ? r : 0.0;           // (positive in the range)
                p[j] = uni ? r : dmul(CERT && one_w ? wc : w[e], r);
                out |= !CERT && (unsigned)__double2hiint(p[j]) - A.img.lo >= A.img.span;
                const double dd = fabs(dsub(val[j], r));
                val[j] = r;
                far |= dd >= A.eps;
                if (dd > lmax) lmax = dd;
                if (A.twice)
#pragma unroll
                    for (unsigned c = 0; c < CTAS; ++c) put(at_rank(x1_a + 8u * (unsigned)e, c), p[j]);
            }
        }
        if (__any_sync(0xffffffffu, far) && lane < CTAS) put_u32(at_rank(far_a + 4u * (unsigned)(it % 3), lane), 1u);
        if (__any_sync(0xffffffffu, out) && lane < CTAS) put_u32(at_rank(bad_a, lane), 1u);
        cluster_sync();
        if (ctl->bad) break;
        far = ctl->far[it % 3] != 0;
        // written again two sweeps on, after the barriers of the next one
        if (t == 0) ctl->far[(it + 2) % 3] = 0u;
        if (A.twice) {
            double *s = x0;
            x0 = x1;
            x1 = s;
        } else {                             // every CTA is past its gathers
#pragma unroll
            for (int j = 0; j < OWN; ++j) {
                const int e = e0 + j * THREADS + t;
                if (e < e1)
#pragma unroll
                    for (unsigned c = 0; c < CTAS; ++c) put(at_rank(x1_a + 8u * (unsigned)e, c), p[j]);
            }
            cluster_sync();
        }
        if (!far && 0.0 < A.eps) break;
    }
    if (ctl->bad) {
        if (rank == 0 && t == 0) A.stats[ST_FITS] = 0ULL;
        cluster_sync();
        return;
    }
#pragma unroll
    for (int j = 0; j < OWN; ++j) {
        const int e = e0 + j * THREADS + t;
        if (e < e1) A.values[e] = val[j];
    }
    for (int u = u0 + t; u < u1; u += THREADS) A.values[E + u] = vd[A.spread ? u - u0 : u];
    // the last sweep's largest |delta|: within the CTA, then on rank 0
    if (lmax > 0.0) atomicMax(&ctl->largest, (unsigned long long)__double_as_longlong(lmax));
    __syncthreads();
    if (t == 0)
        put(at_rank((unsigned)__cvta_generic_to_shared(ctl->maxima), 0) + 8 * rank,
            __longlong_as_double((long long)ctl->largest));
    cluster_sync();
    if (rank == 0 && t == 0) {
        const int sweeps = it < A.max_iter ? it + 1 : A.max_iter;
        A.stats[ST_SWEEPS] = (unsigned long long)sweeps;
        A.stats[ST_EDGE_ITERS] = (unsigned long long)E * (unsigned long long)sweeps;
        A.stats[ST_FITS] = 1ULL;
        A.stats[ST_ITERATIONS] = (unsigned long long)(it < A.max_iter ? it : A.max_iter);
        double m = 0.0;
        for (int r = 0; r < CTAS; ++r) m = fmax(m, ctl->maxima[r]);
        A.stats[ST_DELTA] = (unsigned long long)__double_as_longlong(m);
    }
}

size_t smem_bytes(int E, int N, bool twice, bool spread)
{
    return 256 + 8 * ((size_t)E * (twice ? 2 : 1) + (size_t)(spread ? (N + CTAS - 1) / CTAS : N));
}

// the staged rows, which the values later replace
size_t rows_bytes(int N, int S)
{
    return 256 + 2 * ((size_t)S + (size_t)N + 2);
}

}  // namespace

bool cluster_fits(int E, int N, int S)
{
    static_assert(sizeof(Ctl) <= 256, "control words");
    return E <= OWN * THREADS * CTAS && E < 65536 && N < 65536 && S < 65536 && smem_bytes(E, N, false, true) <= CLUSTER_SMEM &&
           rows_bytes(N, S) <= CLUSTER_SMEM;
}

Status launch_cluster_fit(const ClusterFit &f, cudaStream_t st)
{
    Args a{};
    a.N = f.N;
    a.E = f.E;
    a.fwd = f.fwd;
    a.max_iter = f.max_iter;
    a.eps = f.eps;
    a.img = f.img;
    a.data = f.data;
    a.pairs = f.pairs;
    a.cursor = f.cursor;
    a.values = f.values;
    a.stats = f.stats;
    // as many lanes to a vertex as there are threads, up to one for every two
    // slots of a mean row
    a.lpv = 1;
    const int mean = f.N > 0 ? f.img.Q / f.N : 1;
    while (a.lpv < 8 && 2LL * a.lpv * f.N <= (long long)CTAS * THREADS && 4 * a.lpv <= mean) a.lpv <<= 1;
    // the values twice and all norms where they fit, then the values once and all
    // norms, then the values once (G(8000, 22000))
    a.twice = smem_bytes(f.E, f.N, true, false) <= CLUSTER_SMEM;
    a.spread = !a.twice && smem_bytes(f.E, f.N, false, false) > CLUSTER_SMEM;
    // room for 1.5 times a CTA's mean share of the slots
    size_t smem = smem_bytes(f.E, f.N, a.twice != 0, a.spread != 0);
    a.slot_room = (int)std::min<size_t>((size_t)f.img.Q / CTAS * 3 / 2 + 64, (CLUSTER_SMEM - smem) / 2);
    smem = std::max(smem + 2 * (size_t)a.slot_room, rows_bytes(f.N, f.img.Q));
    // the attribute, and whether such a cluster can be placed, once per device
    static std::mutex mu;
    static std::map<int, int> placeable;
    int dev = 0;
    DRESS_CUDA_TRY(cudaGetDevice(&dev));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(CTAS);
    cfg.blockDim = dim3(THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CTAS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    {
        std::lock_guard<std::mutex> lk(mu);
        auto it = placeable.find(dev);
        if (it == placeable.end()) {
            int clusters = INT_MAX;
            for (void (*k)(const Args) : {k_fit_cluster<false>, k_fit_cluster<true>}) {
                DRESS_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CLUSTER_SMEM));
                int n = 0;
                cfg.dynamicSmemBytes = CLUSTER_SMEM;
                if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
                    cudaGetLastError();
                    n = 0;
                }
                clusters = std::min(clusters, n);
            }
            it = placeable.emplace(dev, clusters).first;
        }
        if (it->second < 1) return Status::Err(DRESSX_EUNSUPPORTED, "cluster fit does not fit the device");
    }
    if (f.certified) {
        count_launch(), k_cluster_pairs<<<(f.E + PAIR_THREADS - 1) / PAIR_THREADS, PAIR_THREADS, 0, st>>>(a);
        DRESS_CUDA_TRY(cudaGetLastError());
    }
    cfg.dynamicSmemBytes = smem;
    count_launch();
    DRESS_CUDA_TRY(cudaLaunchKernelEx(&cfg, f.certified ? k_fit_cluster<true> : k_fit_cluster<false>, a));
    return Status::Ok();
}

}  // namespace dress
