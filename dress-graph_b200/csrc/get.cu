// get.cu -- batched virtual-edge queries on a fitted graph.
//
// Reference: dress_get (libdress/src/dress.c:651-739) answers one (u, v)
// pair: the stored value of an existing edge, or, for a non-edge, the fixed
// point of the pair's own value with every other value frozen -- the sorted
// KBN sum of its common-neighbour terms w_ux d_ux + w_vx d_vx plus the
// self-loop constant, then a scalar iteration.  Here many pairs run at once:
//   k_get_sums    a warp per pair: the edge lookup (binary search of u's row),
//                 else the shorter row's neighbours looked up in the longer one,
//                 32 at a time, their terms in a certified sum (CSum);
//   k_get_iterate one thread per pair: the scalar iteration;
//   k_get_fill / segmented_sort / k_get_exact   the pairs whose certificate
//                 failed (none on ordinary weights): the terms go to a slot per
//                 pair, are sorted by the exact-histogram radix sort and summed
//                 one thread each.
// Every operation is the reference's, in the same order, separately rounded.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "engine.h"
#include "hist.h"

namespace dress {
namespace {

struct GetGraph {
    int N, fwd, undirected;
    const int *off, *tgt, *eidx;
    const double *w, *d, *vd, *nw;       // nw null: unit vertex weights
};

__device__ __forceinline__ double ordered_to_double(unsigned long long k)
{
    unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffULL) : ~k;
    return __longlong_as_double((long long)b);
}

__device__ __forceinline__ double self_loop(const GetGraph &G, int u, int v)
{
    const double nu = G.nw ? G.nw[u] : 1.0, nv = G.nw ? G.nw[v] : 1.0;
    return G.fwd ? dmul(4.0, nu) : dadd(dmul(4.0, nu), dmul(4.0, nv));
}

// the pair's own fixed point from its intercept A (dress.c:713-738)
__device__ double iterate_pair(const GetGraph &G, int u, int v, double A, double ew, int max_iter, double eps)
{
    const double cf = G.fwd ? 1.0 : 2.0;
    const double cw = G.undirected ? dmul(2.0, ew) : ew;
    const double du2 = dmul(G.vd[u], G.vd[u]);
    const double dv2 = dmul(G.vd[v], G.vd[v]);
    if (du2 <= 0.0 || dv2 <= 0.0) return 0.0;
    double d = 1.0;
    for (int it = 0; it < max_iter; ++it) {
        const double wd = dmul(cw, d);
        const double den = dmul(dsqrt(dadd(du2, wd)), dsqrt(dadd(dv2, wd)));
        if (den <= 0.0) return 0.0;
        const double nx = ddiv(dadd(A, dmul(cf, wd)), den);
        if (fabs(dsub(nx, d)) <= eps) {
            d = nx;
            break;
        }
        d = nx;
    }
    return d;
}

__device__ __forceinline__ double term_of(const GetGraph &G, int eu, int ev)
{
    return dadd(dmul(G.w[eu], G.d[eu]), dmul(G.w[ev], G.d[ev]));
}

// first index in [lo, hi) with tgt[index] >= x
__device__ __forceinline__ int lower_bound(const int *tgt, int lo, int hi, int x)
{
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (tgt[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// A warp per pair.  The lanes look up the shorter row's neighbours in the
// longer row, each lane's search starting where the last round's ended; the
// i-th of a run of parallel edges meets the i-th of the other row's run, as in
// the reference's merge walk.  What it waits for is the chain of dependent
// loads of a search, so a warp has 32 of them in flight; a thread per pair
// walked both rows to their ends, hubs' too, twice (100,003 pairs of a
// 200,003-edge power-law graph: 4.3 ms of kernels and 0.7 ms of sorting, now
// 540 us).
// cnt[i]: -1 an existing edge (answered here), 0 the sum is in sum[i], else the
// number of terms of a pair left to the exact path (counted in todo[1]).
__global__ void __launch_bounds__(256) k_get_sums(GetGraph G, long long n, const int *qu, const int *qv, int *cnt,
                                                  double *sum, double *out, int *todo, int force_exact)
{
    const int lane = threadIdx.x & 31;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; i < n; i += nw) {
        const int u = qu[i], v = qv[i];
        if (u < 0 || u >= G.N || v < 0 || v >= G.N) {
            if (lane == 0) {
                atomicExch(&todo[0], 1);
                cnt[i] = -1;
                out[i] = 0.0;
            }
            continue;
        }
        // the probes of the reference's search, so parallel edges give the same one
        int lo = G.off[u], hi = G.off[u + 1] - 1, found = -1;
        while (lo <= hi) {
            const int mid = lo + (hi - lo) / 2;
            const int nb = G.tgt[mid];
            if (nb == v) {
                found = mid;
                break;
            }
            if (nb < v) lo = mid + 1;
            else hi = mid - 1;
        }
        if (found >= 0) {
            if (lane == 0) {
                out[i] = G.d[G.eidx[found]];
                cnt[i] = -1;
            }
            continue;
        }
        const bool swap = G.off[u + 1] - G.off[u] > G.off[v + 1] - G.off[v];
        const int a = swap ? v : u, b = swap ? u : v;
        const int s0 = G.off[a], s1 = G.off[a + 1], l1 = G.off[b + 1];
        int from = G.off[b], terms = 0;
        CSum q;
        q.init();
        if (lane == 0) q.add(self_loop(G, u, v));
        for (int k0 = s0; k0 < s1 && from < l1; k0 += 32) {
            const int k = k0 + lane;
            int at = l1;
            if (k < s1) {
                const int x = G.tgt[k];
                at = lower_bound(G.tgt, from, l1, x);
                // place in a run of parallel edges, by search: a run of r would
                // take r steps in each of its lanes
                const int r = k > s0 && G.tgt[k - 1] == x ? k - lower_bound(G.tgt, s0, k, x) : 0;
                if (r < l1 - at && G.tgt[at + r] == x) {
                    q.add(term_of(G, G.eidx[k], G.eidx[at + r]));
                    ++terms;
                }
            }
            // the last lane's target bounds the next round's from below
            from = __shfl_sync(0xffffffffu, at, min(31, s1 - 1 - k0));
        }
        terms = __reduce_add_sync(0xffffffffu, terms);
        q.merge_lanes(32);
        if (lane == 0) {
            double r;
            if (!force_exact && q.result(r)) {
                sum[i] = r;
                cnt[i] = 0;
            } else {
                cnt[i] = terms + 1;
                atomicAdd(&todo[1], 1);
            }
        }
    }
}

__global__ void k_get_iterate(GetGraph G, long long n, const int *qu, const int *qv, const int *cnt, const double *sum,
                              const double *ew, double ew0, int max_iter, double eps, double *out)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        if (cnt[i] == 0) out[i] = iterate_pair(G, qu[i], qv[i], sum[i], ew ? ew[i] : ew0, max_iter, eps);
}

// the terms of the pairs left to the exact path, into their slots
__global__ void k_get_fill(GetGraph G, long long n, const int *qu, const int *qv, const int *cnt,
                           const long long *slot, unsigned long long *keys)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int c = cnt[i];
        if (c <= 0) continue;
        const int u = qu[i], v = qv[i];
        unsigned long long *k = keys + slot[i];
        int m = 0;
        int iu = G.off[u], iu_end = G.off[u + 1];
        int iv = G.off[v], iv_end = G.off[v + 1];
        while (iu < iu_end && iv < iv_end) {
            const int x = G.tgt[iu], y = G.tgt[iv];
            if (x == y) k[m++] = (unsigned long long)__double_as_longlong(term_of(G, G.eidx[iu], G.eidx[iv]));
            iu += (x <= y);
            iv += (x >= y);
        }
        k[m] = (unsigned long long)__double_as_longlong(self_loop(G, u, v));
    }
}

__global__ void k_get_exact(GetGraph G, long long n, const int *qu, const int *qv, const int *cnt,
                            const long long *slot, const unsigned long long *sorted, const double *ew, double ew0,
                            int max_iter, double eps, double *out)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int c = cnt[i];
        if (c <= 0) continue;
        const unsigned long long *k = sorted + slot[i];
        double s = ordered_to_double(k[0]), cc = 0.0;
        for (int t = 1; t < c; ++t) kbn_step(s, cc, ordered_to_double(k[t]));
        out[i] = iterate_pair(G, qu[i], qv[i], dadd(s, cc), ew ? ew[i] : ew0, max_iter, eps);
    }
}

}  // namespace

Status get_batch(p_dress_graph_t g, const int *u, const int *v, long long n, int max_iterations, double epsilon,
                 const double *edge_weights, double edge_weight, double *out, const Ctx &ctx)
{
    if (!g || n < 0 || (n > 0 && (!u || !v || !out))) return Status::Err(DRESSX_EINVAL, "bad arguments");
    if (n == 0) return Status::Ok();
    const int N = g->N, E = g->E;
    const long long S = N > 0 ? g->adj_offset[N] : 0;
    if (N <= 0) return Status::Err(DRESSX_EINVAL, "query on an empty graph");
    cudaStream_t st = ctx.st;
    const int sms = ctx.num_sms;
    DRESS_CUDA_TRY(cudaSetDevice(ctx.device));
    // one device block: the graph, the queries, the results
    const auto al = [](size_t x) { return (x + 15) & ~(size_t)15; };
    size_t total = 0;
    const auto place = [&](size_t bytes) {
        const size_t o = total;
        total = al(total + bytes);
        return o;
    };
    const size_t o_w = place(8 * (size_t)E), o_d = place(8 * (size_t)E), o_vd = place(8 * (size_t)N);
    const size_t o_nw = place(g->NW ? 8 * (size_t)N : 0), o_ew = place(edge_weights ? 8 * (size_t)n : 0);
    const size_t o_off = place(4 * ((size_t)N + 1)), o_tgt = place(4 * (size_t)S), o_eidx = place(4 * (size_t)S);
    const size_t o_u = place(4 * (size_t)n), o_v = place(4 * (size_t)n), o_cnt = place(4 * (size_t)n);
    const size_t o_sum = place(8 * (size_t)n), o_out = place(8 * (size_t)n), o_todo = place(8);
    DevBuf<unsigned char> dev;
    DRESS_TRY(dev.alloc(total, st));
    unsigned char *p = dev.get();
    {
        std::vector<HostSpan> up = {{g->edge_weight, p + o_w, 8 * (size_t)E}, {g->edge_dress, p + o_d, 8 * (size_t)E},
                                    {g->vertex_dress, p + o_vd, 8 * (size_t)N}};
        if (g->NW) up.push_back({g->NW, p + o_nw, 8 * (size_t)N});
        if (edge_weights) up.push_back({(void *)edge_weights, p + o_ew, 8 * (size_t)n});
        up.push_back({g->adj_offset, p + o_off, 4 * ((size_t)N + 1)});
        up.push_back({g->adj_target, p + o_tgt, 4 * (size_t)S});
        up.push_back({g->adj_edge_idx, p + o_eidx, 4 * (size_t)S});
        up.push_back({(void *)u, p + o_u, 4 * (size_t)n});
        up.push_back({(void *)v, p + o_v, 4 * (size_t)n});
        DRESS_TRY(staged_upload(up.data(), (int)up.size(), ctx));
    }
    const int *d_u = (const int *)(p + o_u), *d_v = (const int *)(p + o_v);
    int *d_cnt = (int *)(p + o_cnt), *d_todo = (int *)(p + o_todo);
    double *d_sum = (double *)(p + o_sum), *d_out = (double *)(p + o_out);
    const double *d_ew = edge_weights ? (const double *)(p + o_ew) : nullptr;
    DRESS_CUDA_TRY(cudaMemsetAsync(d_todo, 0, 8, st));
    GetGraph G{N, g->variant == DRESS_VARIANT_FORWARD || g->variant == DRESS_VARIANT_BACKWARD,
               g->variant == DRESS_VARIANT_UNDIRECTED, (const int *)(p + o_off), (const int *)(p + o_tgt),
               (const int *)(p + o_eidx), (const double *)(p + o_w), (const double *)(p + o_d),
               (const double *)(p + o_vd), g->NW ? (const double *)(p + o_nw) : nullptr};
    const unsigned wgrid = (unsigned)std::min<long long>((n + 7) / 8, 64LL * sms);
    const unsigned grid = (unsigned)std::min<long long>((n + 127) / 128, 16LL * sms);
    count_launch(), k_get_sums<<<wgrid, 256, 0, st>>>(G, n, d_u, d_v, d_cnt, d_sum, d_out, d_todo,
                                                      ctx.cfg->exact_sums != 0);
    count_launch(), k_get_iterate<<<grid, 128, 0, st>>>(G, n, d_u, d_v, d_cnt, d_sum, d_ew, edge_weight, max_iterations,
                                                        epsilon, d_out);
    DRESS_CUDA_TRY(cudaGetLastError());
    int todo[2] = {0, 0};
    DRESS_CUDA_TRY(counted_memcpy(todo, d_todo, sizeof todo, cudaMemcpyDeviceToHost, st));
    DRESS_CUDA_TRY(cudaStreamSynchronize(st));
    if (todo[0]) return Status::Err(DRESSX_EINVAL, "query vertex out of range");
    if (todo[1]) {
        // pairs whose certificate failed: slots, per-slot sort, sums
        std::vector<int> cnt((size_t)n);
        DRESS_CUDA_TRY(counted_memcpy(cnt.data(), d_cnt, (size_t)n * sizeof(int), cudaMemcpyDeviceToHost, st));
        DRESS_CUDA_TRY(cudaStreamSynchronize(st));
        std::vector<long long> slot((size_t)n, 0), begin, len;
        long long terms = 0;
        for (long long i = 0; i < n; ++i)
            if (cnt[(size_t)i] > 0) {
                slot[(size_t)i] = terms;
                begin.push_back(terms);
                len.push_back(cnt[(size_t)i]);
                terms += cnt[(size_t)i];
            }
        DevBuf<long long> d_slot;
        DevBuf<unsigned long long> d_keys, d_alt;
        DRESS_TRY(d_slot.alloc((size_t)n, st));
        DRESS_CUDA_TRY(counted_memcpy(d_slot.get(), slot.data(), (size_t)n * sizeof(long long), cudaMemcpyHostToDevice, st));
        DRESS_TRY(d_keys.alloc((size_t)terms, st));
        DRESS_TRY(d_alt.alloc((size_t)terms, st));
        count_launch(), k_get_fill<<<grid, 128, 0, st>>>(G, n, d_u, d_v, d_cnt, d_slot.get(), d_keys.get());
        unsigned long long *sorted = nullptr;
        DRESS_TRY(segmented_sort(d_keys.get(), d_alt.get(), begin, len, &sorted, st, sms));
        count_launch(), k_get_exact<<<grid, 128, 0, st>>>(G, n, d_u, d_v, d_cnt, d_slot.get(), sorted, d_ew, edge_weight,
                                                          max_iterations, epsilon, d_out);
        DRESS_CUDA_TRY(cudaGetLastError());
        DRESS_CUDA_TRY(cudaStreamSynchronize(st));
    }
    const HostSpan down[1] = {{out, d_out, 8 * (size_t)n}};
    return staged_download(down, 1, ctx);
}

}  // namespace dress

using namespace dress;

extern "C" int dressx_get_batch(p_dress_graph_t g, const int *u, const int *v, int64_t n, int max_iterations,
                                double epsilon, const double *edge_weights, double edge_weight, double *out)
{
    Engine &en = engine();
    std::lock_guard<std::mutex> lk(en.mu);
    Status s = en.init();
    if (s.ok()) s = get_batch(g, u, v, (long long)n, max_iterations, epsilon, edge_weights, edge_weight, out, en.ctx);
    set_last_error(s);
    return s.code;
}
