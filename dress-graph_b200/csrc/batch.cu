// batch.cu -- one persistent launch fits many small subgraphs.
//
// Reference behaviour: the Delta^k / Nabla^k drivers
// (libdress/src/delta_dress_impl.c:171-318, nabla_dress_impl.c:142-311)
// rebuild a CSR per subgraph on the host and call the fit
// (libdress/src/dress.c:546-608) once per subgraph.  Here:
//   * a CTA grabs a chunk of subgraphs of one parent graph from a global
//     counter, copies the parent's packed image (endpoints, rows,
//     common-neighbour pairs, weights) into shared memory once, and its thread
//     groups (one group per subgraph) pull subgraphs from the chunk;
//   * a subgraph is the parent plus a mask: Delta deletes the k vertices of
//     the combination with lexicographic rank s, Nabla gives the k vertices of
//     the ordered tuple with rank s the marker weights sqrt(prime_i); both are
//     unranked in the kernel.  The values of dead edges are zero, so the sums
//     run over the parent's rows and pairs without asking which are alive: a
//     zero term changes no bit of a sum;
//   * each group iterates its subgraph to its own convergence (values, vertex
//     norms in shared memory) and appends the live edges' values to the
//     request's value segment (the histogram is built afterwards, hist.cu).
//
// What bounds it: issue slots (67 % busy) and the gathers of values by edge id,
// which random ids spread over the shared-memory banks (1.6 wavefronts of 3 are
// conflicts); the FP64 pipe is at 35 %.  So a term is one gather and four
// additions (FastSum), ids take 16 bits and come four to a load, and edges with
// as many pairs are neighbours, which keeps 28 of 32 lanes busy.  115,425
// Delta^1 subgraphs of 2,000 regular graphs (16 to 100 vertices): 12.5 ms with
// a liveness test, a weight and a certificate per term and item, 3.2 ms now;
// 61 subgraphs of one graph, on one CTA before and one a CTA now: 735 -> 35 us.
#include <algorithm>
#include <map>
#include <mutex>

#include "batch.h"
#include "common.cuh"

namespace dress {
namespace {

__device__ __forceinline__ long long binom_d(int n, int k)
{
    if (k < 0 || k > n) return 0;
    if (k > n - k) k = n - k;
    long long r = 1;
    for (int i = 0; i < k; ++i) r = r * (n - i) / (i + 1);
    return r;
}

__device__ __forceinline__ long long perm_d(int n, int k)
{
    if (k < 0 || k > n) return 0;
    long long r = 1;
    for (int i = 0; i < k; ++i) r *= (n - i);
    return r;
}

__constant__ int c_primes[16] = {2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53};

// sqrt of the (i+1)-th prime for i < 16, sqrt(2i+3) beyond
// (libdress/src/nabla_dress_impl.c:33-46)
__device__ __forceinline__ double marker_weight(int i)
{
    return dsqrt((double)(i < 16 ? c_primes[i] : 2 * i + 3));
}

// ---- subgraphs in shared memory -------------------------------------------------
// An array in shared memory by its 32-bit address: the kernel holds a dozen of
// them at 64 registers a thread, and a spill would go to L2 (the shared memory
// leaves almost no L1).
template <class T>
struct SArr;
template <>
struct SArr<double> {
    unsigned a;
    __device__ __forceinline__ double operator[](unsigned i) const
    {
        double v;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a + 8 * i));
        return v;
    }
    __device__ __forceinline__ void set(unsigned i, double v) const
    {
        asm volatile("st.shared.f64 [%0], %1;" ::"r"(a + 8 * i), "d"(v) : "memory");
    }
    __device__ __forceinline__ double *ptr() const { return (double *)__cvta_shared_to_generic(a); }
};
template <>
struct SArr<unsigned> {
    unsigned a;
    __device__ __forceinline__ unsigned operator[](unsigned i) const
    {
        unsigned v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a + 4 * i));
        return v;
    }
    __device__ __forceinline__ unsigned *ptr() const { return (unsigned *)__cvta_shared_to_generic(a); }
};
template <>
struct SArr<uint2> {
    unsigned a;
    __device__ __forceinline__ uint2 operator[](unsigned i) const
    {
        uint2 v;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a + 8 * i));
        return v;
    }
    __device__ __forceinline__ uint2 *ptr() const { return (uint2 *)__cvta_shared_to_generic(a); }
};

// a parent's image in global memory (read through L2), the same interface
template <class T>
struct GArr {
    const T *p;
    __device__ __forceinline__ T operator[](unsigned i) const { return p[i]; }
    __device__ __forceinline__ const T *ptr() const { return p; }
};

template <template <class> class A>
struct ImageView {
    A<uint2> edge;
    A<unsigned> row;
    A<uint2> eid, pairs;
    A<double> w, nw, dinit;
};

__device__ __forceinline__ ImageLayout image_of(const ParentDesc &P)
{
    return image_layout(P.N, P.E, P.img.Q, P.img.P2, P.img.uniform, P.img.has_nw, P.img.has_dinit);
}
__device__ __forceinline__ ImageView<SArr> image_shared(unsigned b, const ImageLayout &L)
{
    return {{b + (unsigned)L.edge},  {b + (unsigned)L.row}, {b + (unsigned)L.eid},
            {b + (unsigned)L.pairs}, {b + (unsigned)L.w},   {b + (unsigned)L.nw}, {b + (unsigned)L.dinit}};
}
__device__ __forceinline__ ImageView<GArr> image_global(const unsigned char *b, const ImageLayout &L)
{
    return {{(const uint2 *)(b + L.edge)}, {(const unsigned *)(b + L.row)}, {(const uint2 *)(b + L.eid)},
            {(const uint2 *)(b + L.pairs)}, {(const double *)(b + L.w)}, {(const double *)(b + L.nw)},
            {(const double *)(b + L.dinit)}};
}

// The threads of one subgraph: one warp, or several with a named barrier.
struct Group {
    int gid, t, size;
    __device__ __forceinline__ void sync() const
    {
        if (size == 32) __syncwarp();
        else asm volatile("bar.sync %0, %1;" ::"r"(gid + 1), "r"(size) : "memory");
    }
    // barrier and vote in one
    __device__ __forceinline__ bool any(bool p) const
    {
        if (size == 32) {
            const bool r = __any_sync(0xffffffffu, p) != 0;
            __syncwarp();
            return r;
        }
        int r;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\t"
                     "barrier.cta.red.or.pred q, %2, %3, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                     : "=r"(r)
                     : "r"((int)p), "r"(gid + 1), "r"(size)
                     : "memory");
        return r != 0;
    }
};

// One subgraph's shared memory (state_bytes).
struct State {
    SArr<double> x0, x1, dv, vd, mw;
    SArr<unsigned> ctl;             // [0] live edges, then the emission cursor; [1] a product
                                    // is out of the fast range; [2..3] one 64-bit word
    SArr<unsigned> ks, eb;
};

template <int MODE>
__device__ __forceinline__ State state_at(unsigned b, int E, int N, int k)
{
    State s;
    const unsigned kk = k > 0 ? k : 1, e8 = 8u * (unsigned)(E + 1);
    s.x0.a = b;
    s.x1.a = b + e8;
    s.dv.a = b + 2 * e8;
    s.vd.a = s.dv.a + (MODE == STATE_PRODUCT ? e8 : 0);
    s.ctl.a = s.vd.a + 8u * (unsigned)N;
    s.mw.a = s.ctl.a + 16;
    s.ks.a = s.mw.a + 8 * kk;
    s.eb.a = s.ks.a + 4 * kk;
    return s;
}

// Neumaier's sum when every term is non-negative and no term's exponent is
// above the running sum's: the rounding error of each addition is then
// x - (t - s), without choosing the larger operand.  The caller knows from
// the range of the products (fast_range, delta_nabla.cpp) that this holds for
// every item of the subgraph and that every addition into c is exact in any
// order, so s + c rounds to the bits of the reference's sorted sum
// (libdress/src/dress.c:51-66) without a certificate per item: the "exact
// compensation" case of CSum (common.cuh), decided once a sweep for all items.
// Four additions a term; CSum takes eight FP64 operations and eight selects.
// WIDE: TwoSum, six additions a term, which needs no order of the exponents, so
// the range may reach above the running sums: products of 8 and more (edge
// weights of 4 and more, vertex weights below 1).  Such parents took the slow
// sums otherwise: a whole-graph fit of 300 edges with weights 1 to 10 228 us,
// 163 so; the Delta^1 kernel of 60 graphs of 16 to 100 vertices with them 787 us,
// 387 so (166 by the narrow sums at weights of 0.5 to 2).
template <bool WIDE>
struct FastSum {
    double s, c;
    __device__ __forceinline__ void add(double x)
    {
        const double t = dadd(s, x);
        if (WIDE) {
            const double b = dsub(t, s);
            c = dadd(c, dadd(dsub(s, dsub(t, b)), dsub(x, b)));
        } else {
            c = dadd(c, dsub(x, dsub(t, s)));
        }
        s = t;
    }
};

// high word of a product inside the fast range (zero, negative, infinite and
// NaN products are outside)
__device__ __forceinline__ bool in_range(double x, unsigned lo, unsigned span)
{
    return (unsigned)__double2hiint(x) - lo < span;
}

// The sums of a subgraph whose products leave the fast range, and of tests of
// the sorted path: each item by item_sum over its live terms.
template <int MODE>
struct SlowTerms {
    const unsigned short *ids;
    const double *x, *w;
    const unsigned *eb;
    double wc;
    int E;
    __device__ __forceinline__ double prod(int e) const
    {
        return MODE == STATE_UNIFORM ? dmul(wc, x[e]) : MODE == STATE_PRODUCT ? x[e] : dmul(w[e], x[e]);
    }
    __device__ __forceinline__ bool alive(int e) const { return e < E && ((eb[e >> 5] >> (e & 31)) & 1u); }
};
template <int MODE>
struct SlowRow : SlowTerms<MODE> {
    __device__ __forceinline__ bool operator()(int j, double &t) const
    {
        const int e = this->ids[j];
        if (!this->alive(e)) return false;
        t = this->prod(e);
        return true;
    }
};
template <int MODE>
struct SlowPairs : SlowTerms<MODE> {
    __device__ __forceinline__ bool operator()(int j, double &t) const
    {
        const int ex = this->ids[2 * j], ey = this->ids[2 * j + 1] & 0x7fff;
        if (!this->alive(ex)) return false;
        t = dadd(this->prod(ex), this->prod(ey));
        return true;
    }
};
// 4 nw of a vertex as the sums take it (in units of the weight where that is
// one power of two)
template <template <class> class A>
__device__ __forceinline__ double four_nw(const ParentDesc &P, const State &st, const ImageView<A> &G, double base4, int x)
{
    double r = base4;
    if (P.kind == ITEM_NABLA) {
        for (int i = 0; i < P.k; ++i)
            if ((int)st.ks[i] == x) r = st.mw[i];
    } else if (P.kind == ITEM_PLAIN && P.img.has_nw) {
        r = dmul(base4, G.nw[x]);
    }
    return r;
}

// A sweep's two phases off the fast path.
template <int MODE, template <class> class A>
struct SlowSweep {
    const ParentDesc &P;
    const ImageView<A> &G;
    const State &st;
    double *x0, *x1;
    __device__ __forceinline__ double a4(int x) const
    {
        const double r = four_nw(P, st, G, MODE == STATE_UNIFORM ? ddiv(4.0, P.img.wc) : 4.0, x);
        return MODE == STATE_UNIFORM ? dmul(P.img.wc, r) : r;
    }
    template <class T>
    __device__ __forceinline__ void terms(T &q, const uint2 *ids) const
    {
        q.ids = (const unsigned short *)ids;
        q.x = x0, q.w = G.w.ptr(), q.eb = st.eb.ptr(), q.wc = P.img.wc, q.E = P.E;
    }
};

template <int MODE, template <class> class A>
__device__ __forceinline__ void slow_vertices(const ParentDesc &P, const ImageView<A> &G, const State &st, unsigned x0, int t,
                                           int size)
{
    const SlowSweep<MODE, A> S{P, G, st, SArr<double>{x0}.ptr(), nullptr};
    for (int u = t; u < P.N; u += size) {
        const unsigned row = G.row[u], b = row & 0xffffu, e = row >> 16;
        SlowRow<MODE> q;
        S.terms(q, G.eid.ptr() + b);
        st.vd.set(u, dsqrt(item_sum(S.a4(u), 4 * (int)(e - b), q, P.force_exact != 0)));
    }
}

// the largest |delta| (NaN ignored, as in the reference's max)
template <int MODE, template <class> class A>
__device__ __forceinline__ double slow_edges(const ParentDesc &P, const ImageView<A> &G, const State &st, unsigned x0,
                                          unsigned x1, int t, int size)
{
    const SlowSweep<MODE, A> S{P, G, st, SArr<double>{x0}.ptr(), SArr<double>{x1}.ptr()};
    double lmax = 0.0;
    for (int e = t; e < P.E; e += size) {
        if (!((st.eb[e >> 5] >> (e & 31)) & 1u)) continue;
        const uint2 rec = G.edge[e];
        const int u = rec.x & 0xffffu, v = rec.x >> 16;
        unsigned n = 0;                            // groups of pairs
        if (rec.y != NO_PAIRS)
            while (!(G.pairs[rec.y + n++].y >> 31)) {}
        SlowPairs<MODE> q;
        S.terms(q, G.pairs.ptr() + (n ? rec.y : 0));
        const double own = q.prod(e), old = MODE == STATE_PRODUCT ? st.dv[e] : S.x0[e];
        const double self = P.fwd ? dadd(S.a4(u), own) : dadd(dadd(S.a4(u), S.a4(v)), dmul(2.0, own));
        const double num = item_sum(self, 2 * (int)n, q, P.force_exact != 0);
        const double den = dmul(st.vd[u], st.vd[v]);
        const double r = den > 0.0 ? ddiv(num, den) : 0.0;
        S.x1[e] = MODE == STATE_PRODUCT ? dmul(G.w[e], r) : r;
        if (MODE == STATE_PRODUCT) st.dv.set(e, r);
        const double dd = fabs(dsub(old, r));
        if (dd > lmax) lmax = dd;
    }
    return lmax;
}

// Unranking by the group's first warp: 32 candidates of the next vertex at a
// time, the lexicographic blocks' sizes summed across the lanes.
__device__ __forceinline__ void unrank(const ParentDesc &P, long long r, int *ks, int lane)
{
    const int N = P.N, k = P.k;
    if (P.kind == ITEM_DELTA) {
        int c = 0;
        for (int i = 0; i < k; ++i) {
            if (i == k - 1) {                      // blocks of one
                c += (int)r;
                if (lane == 0) ks[i] = c;
                break;
            }
            for (; c < N; c += 32) {
                const long long cnt = binom_d(N - c - lane - 1, k - i - 1);
                long long sum = cnt;
                for (int o = 1; o < 32; o <<= 1) {
                    const long long y = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += y;
                }
                const unsigned m = __ballot_sync(0xffffffffu, r < sum);
                if (m) {
                    const int l = __ffs(m) - 1;
                    r -= __shfl_sync(0xffffffffu, sum - cnt, l);
                    c += l;
                    break;
                }
                r -= __shfl_sync(0xffffffffu, sum, 31);
            }
            if (lane == 0) ks[i] = c;
            ++c;
        }
        return;
    }
    if (lane) return;
    for (int i = 0; i < k; ++i) {
        const long long per = perm_d(N - i - 1, k - i - 1), idx = r / per;
        r -= idx * per;
        // the idx-th vertex not taken yet: idx plus the taken ones up to it
        int v = (int)idx;
        for (;;) {
            int n = (int)idx;
            for (int j = 0; j < i; ++j) n += ks[j] <= v;
            if (n == v) break;
            v = n;
        }
        ks[i] = v;
    }
}

// The four ids of a group of slots, or of two pairs, and their values.
struct Four {
    unsigned i0, i1, i2, i3;
    __device__ __forceinline__ explicit Four(uint2 id)
        : i0(id.x & 0xffffu), i1(id.x >> 16), i2(id.y & 0xffffu), i3((id.y >> 16) & 0x7fffu) {}
};
template <int MODE, template <class> class A>
__device__ __forceinline__ double term(const SArr<double> x, const ImageView<A> &G, unsigned i)
{
    const double v = x[i];
    if (MODE != STATE_VALUE) return v;
    return v != 0.0 ? dmul(G.w[i], v) : 0.0;       // the padding id has no weight
}

// One subgraph.  SUM_NARROW, SUM_WIDE: by FastSum; false, with nothing emitted,
// when a live product leaves the range.  SUM_SLOW: every sum by item_sum.
enum { SUM_NARROW = 0, SUM_WIDE = 1, SUM_SLOW = 2 };
template <int MODE, template <class> class A, int SUM>
__device__ __forceinline__ bool fit_item(const ParentDesc &P, const ImageView<A> &G, long long item, const Group &g,
                                         unsigned mem)
{
    constexpr bool FAST = SUM != SUM_SLOW;
    using RangeSum = FastSum<SUM == SUM_WIDE>;
    const State st = state_at<MODE>(mem, P.E, P.N, P.k);
    unsigned *ctl = st.ctl.ptr();
    SArr<double> x0 = st.x0, x1 = st.x1;
    const double wc = P.img.wc;
    // 4 nw, in units of the weight where that is one power of two
    const double base4 = MODE == STATE_UNIFORM ? ddiv(4.0, wc) : 4.0;
    int live;
    {
        const int E = P.E, k = P.kind == ITEM_PLAIN ? 0 : P.k;
        if (g.t < 32 && k > 0) unrank(P, P.ranks ? P.ranks[item] : P.offset + item * P.stride, (int *)st.ks.ptr(), g.t);
        if (g.t == 0) {
            ctl[0] = ctl[1] = 0;
            x0.set(E, 0.0);                        // the id that pads rows and pairs
            x1.set(E, 0.0);
        }
        if (P.kind == ITEM_NABLA)
            for (int i = g.t; i < k; i += g.size) st.mw.set(i, dmul(base4, marker_weight(i)));
        g.sync();
        if (k > 0) {                               // the image's ids of the mask vertices
            if (g.t < k) {
                const unsigned short *vmap = (const unsigned short *)(P.data + image_of(P).vmap);
                for (int i = g.t; i < k; i += g.size) st.ks.ptr()[i] = vmap[st.ks[i]];
            }
            g.sync();
        }

        // ---- live edges, initial values -----------------------------------------
        // a warp's lanes take 32 consecutive edges, so a ballot is a word of bits
        bool out = false;
        int n = 0;
        for (int b0 = g.t & ~31; b0 < E; b0 += g.size) {
            const int e = b0 + (g.t & 31);
            bool al = e < E;
            if (al) {
                if (P.kind == ITEM_DELTA) {
                    const unsigned uv = G.edge[e].x;
                    for (int i = 0; i < k; ++i) {
                        const unsigned x = st.ks[i];
                        if ((uv & 0xffffu) == x || (uv >> 16) == x) al = false;
                    }
                }
                const double d = P.img.has_dinit ? G.dinit[e] : 1.0;
                const double p = MODE == STATE_UNIFORM ? d : dmul(G.w[e], d);
                x0.set(e, al ? (MODE == STATE_PRODUCT ? p : d) : 0.0);
                if (!al) x1.set(e, 0.0);
                if (MODE == STATE_PRODUCT) st.dv.set(e, d);
                out |= al && !in_range(p, SUM == SUM_WIDE ? P.img.wide_lo : P.img.lo,
                                       SUM == SUM_WIDE ? P.img.wide_span : P.img.span);
            }
            const unsigned word = __ballot_sync(0xffffffffu, al);
            if ((g.t & 31) == 0) st.eb.ptr()[b0 >> 5] = word;
            n += __popc(word);
        }
        if ((g.t & 31) == 0 && n) atomicAdd(&ctl[0], (unsigned)n);
        if (out) ctl[1] = 1;
        g.sync();                                  // the bits, counts and initial values, group-wide
        live = (int)st.ctl[0];
        const bool off = FAST && st.ctl[1];
        if (off || (live == 0 && P.kind != ITEM_PLAIN)) {   // the reference skips edgeless subgraphs
            g.sync();
            return !off;
        }
    }

    // Without a sweep no barrier lies between the reads of ctl[0] and ctl[1] above
    // and thread 0's reset of them below.
    if (P.max_iter <= 0) g.sync();

    // ---- sweeps ------------------------------------------------------------------
    // Live products are positive on the fast path, so a zero marks a dead edge.
    const bool ones = P.kind == ITEM_DELTA || (P.kind == ITEM_PLAIN && !P.img.has_nw);   // every nw is 1.0
    const bool fwd = P.fwd != 0, plain = P.kind == ITEM_PLAIN;
    const unsigned lo = SUM == SUM_WIDE ? P.img.wide_lo : P.img.lo, span = SUM == SUM_WIDE ? P.img.wide_span : P.img.span;
    const double eps = P.eps;
    const int N = P.N, E = P.E;
    int it = 0;
    double lmax = 0.0;
    for (; it < P.max_iter; ++it) {
        if (FAST) {
            for (int u = g.t; u < N; u += g.size) {
                RangeSum q{ones ? base4 : four_nw(P, st, G, base4, u), 0.0};
                const unsigned row = G.row[u];
                for (unsigned b = row & 0xffffu, e = row >> 16; b < e; ++b) {
                    const Four f(G.eid[b]);
                    const double v0 = term<MODE>(x0, G, f.i0), v1 = term<MODE>(x0, G, f.i1);
                    const double v2 = term<MODE>(x0, G, f.i2), v3 = term<MODE>(x0, G, f.i3);
                    q.add(v0);
                    q.add(v1);
                    q.add(v2);
                    q.add(v3);
                }
                const double S = dadd(q.s, q.c);
                st.vd.set(u, dsqrt(MODE == STATE_UNIFORM ? dmul(wc, S) : S));
            }
        } else {
            slow_vertices<MODE, A>(P, G, st, x0.a, g.t, g.size);
        }
        g.sync();
        bool far = false;
        lmax = 0.0;
        if (FAST) {
            bool out = false;
            for (int e = g.t; e < E; e += g.size) {
                const double xe = x0[e];
                if (xe == 0.0) continue;
                const uint2 rec = G.edge[e];
                const unsigned u = rec.x & 0xffffu, v = rec.x >> 16;
                const double den = dmul(st.vd[u], st.vd[v]);      // the norms are positive
                const double own = MODE == STATE_VALUE ? dmul(G.w[e], xe) : xe;
                double s0 = base4;
                if (ones) {
                    if (!fwd) s0 = dadd(base4, base4);
                } else {
                    s0 = four_nw(P, st, G, base4, u);
                    if (!fwd) s0 = dadd(s0, four_nw(P, st, G, base4, v));
                }
                RangeSum q{dadd(s0, fwd ? own : dadd(own, own)), 0.0};      // 2 own is exact
                if (rec.y != NO_PAIRS) {
                    uint2 id;
                    unsigned b = rec.y;
                    do {
                        id = G.pairs[b++];
                        const Four f(id);
                        const double v0 = term<MODE>(x0, G, f.i0), v1 = term<MODE>(x0, G, f.i1);
                        const double v2 = term<MODE>(x0, G, f.i2), v3 = term<MODE>(x0, G, f.i3);
                        q.add(dadd(v0, v1));
                        q.add(dadd(v2, v3));
                    } while (!(id.y >> 31));
                }
                const double S = dadd(q.s, q.c);
                const double r = ddiv(MODE == STATE_UNIFORM ? dmul(wc, S) : S, den);
                const double p = MODE == STATE_UNIFORM ? r : dmul(G.w[e], r);
                const double old = MODE == STATE_PRODUCT ? st.dv[e] : xe;
                x1.set(e, MODE == STATE_PRODUCT ? p : r);
                if (MODE == STATE_PRODUCT) st.dv.set(e, r);
                out |= !in_range(p, lo, span);
                const double dd = fabs(dsub(old, r));
                far |= dd >= eps;
                if (plain && dd > lmax) lmax = dd;
            }
            if (out) ctl[1] = 1;
        } else {
            lmax = slow_edges<MODE, A>(P, G, st, x0.a, x1.a, g.t, g.size);
            far = lmax >= eps;
        }
        // One barrier orders this sweep's writes of x1 and its reads of vd and
        // x0 before the next sweep's writes, and carries the vote: the sweep's
        // max |delta| is below eps exactly when no |delta| reaches it.
        far = g.any(far);
        if (FAST && st.ctl[1]) {
            g.sync();                              // every thread has seen it
            return false;
        }
        const SArr<double> t = x0;
        x0 = x1;
        x1 = t;
        if (!far && 0.0 < eps) break;
    }
    const int sweeps = it < P.max_iter ? it + 1 : P.max_iter;
    const SArr<double> val = MODE == STATE_PRODUCT ? st.dv : x0;
    unsigned long long *word64 = (unsigned long long *)(ctl + 2);

    // ---- plain fit: the final state in edge / vertex order -------------------------
    if (P.kind == ITEM_PLAIN) {
        const unsigned short *vmap = (const unsigned short *)(P.data + image_of(P).vmap);
        const unsigned short *emap = (const unsigned short *)(P.data + image_of(P).emap);
        for (int e = g.t; e < E; e += g.size) P.values[e] = val[emap[e]];
        if (P.max_iter > 0)     // the norms of the last sweep (none without sweeps)
            for (int u = g.t; u < P.N; u += g.size) P.values[E + u] = st.vd[vmap[u]];
        if (g.t == 0) *word64 = 0ULL;
        g.sync();
        if (lmax > 0.0) atomicMax(word64, (unsigned long long)__double_as_longlong(lmax));
        g.sync();
        if (g.t == 0) {
            const int done = P.max_iter > 0 ? sweeps : 0;
            P.stats[ST_SWEEPS] = (unsigned long long)done;
            P.stats[ST_EDGE_ITERS] = (unsigned long long)E * (unsigned long long)done;
            P.stats[ST_FITS] = 1ULL;
            P.stats[ST_ITERATIONS] = (unsigned long long)(it < P.max_iter ? it : P.max_iter);
            P.stats[ST_DELTA] = *word64;
        }
        g.sync();
        return true;
    }

    // ---- emit the live values -------------------------------------------------------
    if (g.t == 0) {
        *word64 = atomicAdd(&P.stats[ST_CURSOR], (unsigned long long)live);
        ctl[0] = 0;
        atomicAdd(&P.stats[ST_SWEEPS], (unsigned long long)sweeps);
        atomicAdd(&P.stats[ST_EDGE_ITERS], (unsigned long long)live * (unsigned long long)sweeps);
        atomicAdd(&P.stats[ST_FITS], 1ULL);
    }
    g.sync();
    double *out = P.values + (long long)*word64;
    const int lane = g.t & 31;
    for (int b0 = g.t & ~31; b0 < E; b0 += g.size) {
        const unsigned word = st.eb[b0 >> 5];
        unsigned at = 0;
        if (lane == 0) at = atomicAdd(&ctl[0], (unsigned)__popc(word));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(word & ((1u << lane) - 1));
        if ((word >> lane) & 1u) out[at] = val[b0 + lane];
    }
    if (P.multisets) {
        const unsigned short *emap = (const unsigned short *)(P.data + image_of(P).emap);
        double *row = P.multisets + (P.ranks ? P.ranks[item] : P.offset + item * P.stride) * (long long)E;
        for (int e = g.t; e < E; e += g.size) {
            const int i = emap[e];
            row[e] = (st.eb[i >> 5] >> (i & 31)) & 1u ? val[i] : __longlong_as_double(0x7ff8000000000000LL);
        }
    }
    g.sync();
    return true;
}

// The same by the other sums, as calls of their own: what they need in registers
// does not weigh on the narrow loops.
template <int MODE, template <class> class A, int SUM>
__device__ __noinline__ bool fit_item_call(const ParentDesc &P, const ImageView<A> G, long long item, const Group g,
                                           unsigned mem)
{
    return fit_item<MODE, A, SUM>(P, G, item, g, mem);
}
template <int MODE, template <class> class A>
__device__ __noinline__ void fit_item_rest(const ParentDesc &P, const ImageView<A> G, long long item, const Group g,
                                           unsigned mem)
{
    if (!P.force_exact && P.img.wide_span && fit_item_call<MODE, A, SUM_WIDE>(P, G, item, g, mem)) return;
    fit_item_call<MODE, A, SUM_SLOW>(P, G, item, g, mem);
}

// Every group of the CTA takes subgraphs of the chunk until none is left.
template <int MODE, template <class> class A>
__device__ __forceinline__ void fit_chunk(const ParentDesc &P, const Chunk &ch, const Geometry &q, const ImageView<A> &G,
                                          unsigned states, int *next)
{
    const int warp = (int)threadIdx.x >> 5, gid = warp / q.warps;
    if (gid >= q.groups) return;
    const Group g{gid, (int)threadIdx.x - gid * q.warps * 32, q.warps * 32};
    const unsigned mem = states + (unsigned)(gid * q.state);
    for (;;) {
        int item = 0;
        if (g.size == 32) {
            if (g.t == 0) item = atomicAdd(next, 1);
            item = __shfl_sync(0xffffffffu, item, 0);
        } else {
            unsigned *ctl = state_at<MODE>(mem, P.E, P.N, P.k).ctl.ptr();
            if (g.t == 0) ctl[2] = (unsigned)atomicAdd(next, 1);
            g.sync();
            item = (int)ctl[2];
            g.sync();
        }
        if (item >= ch.count) return;
        // the cheapest sums whose range the parent's first products are in, then
        // what a product that leaves it on the way needs
        if (P.force_exact || P.img.span == 0 || !fit_item<MODE, A, SUM_NARROW>(P, G, ch.first + item, g, mem))
            fit_item_rest<MODE, A>(P, G, ch.first + item, g, mem);
    }
}

// One CTA per slot of the device, L.ctas to an SM; 64 registers a thread keep
// 32 warps on an SM.  Nothing is spilled inside the sweep loops: the images and
// states leave almost no L1, and with 30 spilled loads there the 2,000-graph
// batch took 5.6 ms, without them 3.7 (3.2 since items are sorted by length).
// The chunk's geometry -- state mode,
// staging, warps per subgraph -- follows from the parent's sizes alone, so a
// launch mixes parents of any sizes and memory is divided by each parent's
// own state, not by the largest of the batch.
__global__ void __launch_bounds__(32 * BATCH_SM_WARPS, 1) k_batch(BatchLaunch L)
{
    extern __shared__ __align__(16) unsigned char smem[];
    int *s_chunk = (int *)smem, *s_next = s_chunk + 1;
    Chunk *s_ch = (Chunk *)(smem + 16);
    ParentDesc *s_desc = (ParentDesc *)(smem + 16 + sizeof(Chunk));
    unsigned char *room = smem + BATCH_HEADER;
    int staged = -1;
    for (;;) {
        if (threadIdx.x == 0) {
            *s_chunk = atomicAdd(L.chunk_counter, 1);
            *s_next = 0;
        }
        __syncthreads();
        const int c = *s_chunk;
        if (c >= L.nchunks) break;
        if (threadIdx.x < sizeof(Chunk) / 4) ((int *)s_ch)[threadIdx.x] = ((const int *)(L.chunks + c))[threadIdx.x];
        const int parent = L.chunks[c].parent;
        if (threadIdx.x < sizeof(ParentDesc) / 4)
            ((int *)s_desc)[threadIdx.x] = ((const int *)(L.parents + parent))[threadIdx.x];
        __syncthreads();
        const ParentDesc &P = *s_desc;
        const Geometry q = chunk_geometry(P.N, P.E, P.kind == ITEM_PLAIN ? 0 : P.k, P.img, batch_room(L.smem), (int)blockDim.x >> 5,
                                          s_ch->warps);
        if (q.staged && parent != staged) {
            const int4 *src = (const int4 *)P.data;
            int4 *dst = (int4 *)room;
            for (int i = threadIdx.x; i < (int)(q.image / 16); i += blockDim.x) dst[i] = src[i];
            staged = parent;
        }
        if (!q.staged) staged = -1;                // the states take the image's place
        __syncthreads();
        const ImageLayout IL = image_of(P);
        const unsigned base = (unsigned)__cvta_generic_to_shared(room), states = base + (unsigned)q.image;
        if (q.staged) {
            const ImageView<SArr> G = image_shared(base, IL);
            if (q.mode == STATE_UNIFORM) fit_chunk<STATE_UNIFORM>(P, *s_ch, q, G, states, s_next);
            else if (q.mode == STATE_PRODUCT) fit_chunk<STATE_PRODUCT>(P, *s_ch, q, G, states, s_next);
            else fit_chunk<STATE_VALUE>(P, *s_ch, q, G, states, s_next);
        } else {
            const ImageView<GArr> G = image_global(P.data, IL);
            if (q.mode == STATE_UNIFORM) fit_chunk<STATE_UNIFORM>(P, *s_ch, q, G, states, s_next);
            else if (q.mode == STATE_PRODUCT) fit_chunk<STATE_PRODUCT>(P, *s_ch, q, G, states, s_next);
            else fit_chunk<STATE_VALUE>(P, *s_ch, q, G, states, s_next);
        }
        __syncthreads();
    }
}

}  // namespace

Status batch_smem(int device, int ctas, int *bytes)
{
    int optin = 0, per_sm = 0, reserved = 0;
    DRESS_CUDA_TRY(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
    DRESS_CUDA_TRY(cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device));
    DRESS_CUDA_TRY(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, device));
    *bytes = std::min(optin, per_sm / ctas - reserved) & ~15;
    return Status::Ok();
}

Status launch_batch(const BatchLaunch &L, int sms, cudaStream_t st)
{
    if (L.nchunks <= 0) return Status::Ok();
    // the attribute is set once per device, to the most the device allows
    int dev = 0;
    DRESS_CUDA_TRY(cudaGetDevice(&dev));
    static std::mutex mu;
    static std::map<int, int> cap;
    int most = 0;
    {
        std::lock_guard<std::mutex> lk(mu);
        auto it = cap.find(dev);
        if (it == cap.end()) {
            DRESS_TRY(batch_smem(dev, 1, &most));
            DRESS_CUDA_TRY(cudaFuncSetAttribute(k_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
            cap[dev] = most;
        } else {
            most = it->second;
        }
    }
    if (L.smem > most || L.smem <= BATCH_HEADER || L.ctas < 1 || L.ctas > 8)
        return Status::Err(DRESSX_EUNSUPPORTED, "batch kernel does not fit on an SM");
    const int grid = std::min(L.nchunks, L.ctas * sms);
    count_launch(), k_batch<<<grid, 32 * (BATCH_SM_WARPS / L.ctas), L.smem, st>>>(L);
    DRESS_CUDA_TRY(cudaGetLastError());
    return Status::Ok();
}

}  // namespace dress
