// fit_small.cu -- the single-graph fit of a small or mid-size graph in one launch.
//
// Reference: libdress/src/dress.c:546-608 (the iteration driver) with the
// vertex and edge phases of :556-591.  A graph of up to SMALL_MAX_EDGES edges
// whose fit state and packed image fit one SM's shared memory, with rows of at
// most 256 neighbours, is fitted by one CTA of the batch kernel as a single
// whole-graph item: every sweep, the convergence test and the final values in
// one launch, without per-sweep kernels or host round trips.  Graphs of up to
// CLUSTER_MAX_EDGES edges run on a thread-block cluster whose CTAs hold the
// values each (fit_cluster.cu), in two launches where products are out of range.  Larger graphs, and graphs that carry their own
// intercept tables, take the multi-kernel fit in fit_graph.cu.  Bit-identical
// to the reference all.
#include <algorithm>
#include <climits>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "batch.h"
#include "engine.h"

namespace dress {

namespace {
// One CTA up to this many edges, a cluster of 8 beyond (fit_cluster.cu).
// Measured per dress_fit_cuda call on G(n, m), one CTA against the cluster:
// 76 / 104 us at 300 edges, 102 / 112 at 600, 116 / 119 at 1000, 147 / 126 at
// 1500, 184 / 142 at 2047.
constexpr int SMALL_MAX_EDGES = 1024;
// Beyond this the multi-kernel fit takes over; it pays about 1 ms of fixed
// cost: 495 us against 870 before and about 1000 at G(4000, 20000).
constexpr int CLUSTER_MAX_EDGES = 24576;
// Rows up to this many neighbours: one thread sums an item's terms, so a
// longer row would make one thread's serial loop the whole sweep; the
// multi-kernel fit gives such rows a warp or a block.
constexpr int SMALL_MAX_DEG = 256;

// Graphs of more vertices than 16-bit ids name are fitted without the isolated
// ones, up to these sizes: 2,000 edges of 100,000 vertices 869 us by the
// multi-kernel fit, 481 so; 4,000 of 262,144 1,250 and 1,056; 8,000 of 262,144
// 1,238 and 1,485 where few edges share a vertex.
constexpr int COMPACT_MAX_VERTICES = 1 << 18, COMPACT_MAX_EDGES = 4096;

// The checks of fit_graph's device validation, on the host: rows in order
// and in range, edge ids and endpoints in range.
bool small_graph_ok(p_dress_graph_t g, int &maxdeg)
{
    const int N = g->N, E = g->E;
    maxdeg = 0;
    for (int u = 0; u < N; ++u) {
        const int b = g->adj_offset[u], e = g->adj_offset[u + 1];
        if (e < b) return false;
        maxdeg = std::max(maxdeg, e - b);
        for (int s = b; s < e; ++s) {
            const int x = g->adj_target[s], ei = g->adj_edge_idx[s];
            if (x < 0 || x >= N || ei < 0 || ei >= E) return false;
            if (s > b && x < g->adj_target[s - 1]) return false;
        }
    }
    for (int e = 0; e < E; ++e)
        if (g->U[e] < 0 || g->U[e] >= N || g->V[e] < 0 || g->V[e] >= N) return false;
    return true;
}

// The fit of a graph's vertices that have a row or an edge, in their order; the
// others' norms are the root of their own term.
Status fit_compact(p_dress_graph_t g, int max_iterations, double epsilon, int *iterations, double *delta,
                   FitStats *stats, const Ctx &ctx, bool &used)
{
    const int N = g->N, E = g->E, S = g->adj_offset[N];
    int maxdeg = 0;
    if (N > COMPACT_MAX_VERTICES || E > COMPACT_MAX_EDGES || !small_graph_ok(g, maxdeg)) return Status::Ok();
    std::vector<int> id((size_t)N, 0), vertex, off, tgt((size_t)S), U((size_t)E), V((size_t)E);
    for (int e = 0; e < E; ++e) id[(size_t)g->U[e]] = id[(size_t)g->V[e]] = 1;
    for (int u = 0; u < N; ++u) {
        if (!id[(size_t)u] && g->adj_offset[u + 1] == g->adj_offset[u]) continue;
        id[(size_t)u] = (int)vertex.size();
        vertex.push_back(u);
        off.push_back(g->adj_offset[u]);
    }
    const int n = (int)vertex.size();
    if (n > UINT16_MAX) return Status::Ok();
    off.push_back(S);
    for (int q = 0; q < S; ++q) tgt[(size_t)q] = id[(size_t)g->adj_target[q]];
    for (int e = 0; e < E; ++e) {
        U[(size_t)e] = id[(size_t)g->U[e]];
        V[(size_t)e] = id[(size_t)g->V[e]];
    }
    std::vector<double> norms((size_t)n), nw;
    if (g->NW)
        for (int u : vertex) nw.push_back(g->NW[u]);
    dress_graph_t h = *g;
    h.N = n;
    h.U = U.data();
    h.V = V.data();
    h.adj_offset = off.data();
    h.adj_target = tgt.data();
    h.NW = g->NW ? nw.data() : nullptr;
    h.vertex_dress = norms.data();
    DRESS_TRY(fit_small(&h, max_iterations, epsilon, iterations, delta, stats, ctx, used));
    if (!used || max_iterations <= 0) return Status::Ok();
    for (int u = 0; u < N; ++u) g->vertex_dress[u] = std::sqrt(4.0 * (g->NW ? g->NW[u] : 1.0));
    for (int i = 0; i < n; ++i) g->vertex_dress[vertex[(size_t)i]] = norms[(size_t)i];
    return Status::Ok();
}

}  // namespace

Status fit_small(p_dress_graph_t g, int max_iterations, double epsilon, int *iterations, double *delta,
                 FitStats *stats, const Ctx &ctx, bool &used)
{
    used = false;
    const auto t0 = std::chrono::steady_clock::now();
    const int N = g->N, E = g->E;
    const int max_edges = ctx.cfg->one_launch_max_edges == 0 ? CLUSTER_MAX_EDGES : ctx.cfg->one_launch_max_edges;
    if (E < 1 || E > max_edges || N < 1 || (g->precompute_intercepts && g->intercept_offset))
        return Status::Ok();
    const long long S = g->adj_offset[N];
    if (g->adj_offset[0] != 0 || S < 0) return Status::Ok();      // fit_graph reports it
    if (N > UINT16_MAX) return fit_compact(g, max_iterations, epsilon, iterations, delta, stats, ctx, used);

    // one CTA that holds the state and the staged graph, else one cluster
    // whose CTAs hold the values and norms each
    bool one_cta = E <= SMALL_MAX_EDGES && batch_fits(E, N, S, 0);
    const bool cluster = cluster_fits(E, N, (int)std::min<long long>(S, INT_MAX)) && ctx.cfg->exact_sums == 0;
    if (!one_cta && !cluster) return Status::Ok();
    int maxdeg = 0;
    if (!small_graph_ok(g, maxdeg)) return Status::Ok();       // fit_graph reports it
    if (maxdeg > SMALL_MAX_DEG) return Status::Ok();

    BatchLaunch L{};
    ImageShape img;
    std::vector<int> ioff, pairs;
    long long T = 0;
    if (one_cta) {
        // On one CTA the graph itself must be staged in shared memory too: read
        // through L2 by a single SM, the sweeps are latency-bound.  Its pairs
        // come from the host, the cluster finds its own.
        bool dup = false;                    // repeated neighbours: the merge walk pairs them as the reference does
        merge_walk_pairs(g, ioff, pairs, maxdeg, dup);
        img = plan_image(g, ioff, ITEM_PLAIN, 0, g->NW != nullptr, true);
        L.ctas = 1;
        DRESS_TRY(batch_smem(ctx.device, 1, &L.smem));
        one_cta = chunk_geometry(N, E, 0, img, batch_room(L.smem), BATCH_SM_WARPS, BATCH_SM_WARPS).staged != 0;
        if (!one_cta && !cluster) return Status::Ok();
        T = (long long)(pairs.size() / 2);
    }
    long long image = 0;
    if (one_cta) {
        image = image_layout(N, E, img.Q, img.P2, img.uniform, img.has_nw, 1).bytes;
    } else {
        img = plan_cluster(g, maxdeg);
        image = cluster_layout(N, E, img.Q, img.uniform, img.has_nw, img.has_dinit).bytes;
        T = 0;
        for (int e = 0; e < E; ++e)          // room for every pair
            T += std::min(g->adj_offset[g->U[e] + 1] - g->adj_offset[g->U[e]],
                          g->adj_offset[g->V[e] + 1] - g->adj_offset[g->V[e]]);
    }

    // One device block holds everything: the packed image, the descriptor, the
    // chunk, the counter, the statistics and the results (and a cluster's
    // pairs and where each edge's begin).  The host writes the inputs once, into the context's pinned
    // stage, and one copy each way moves them.
    auto al = [](size_t x) { return (x + 15) & ~(size_t)15; };
    const size_t off_desc = al((size_t)image);
    const size_t off_chunk = al(off_desc + sizeof(ParentDesc));
    const size_t off_ctr = al(off_chunk + sizeof(Chunk));
    const size_t off_stats = al(off_ctr + sizeof(int));
    const size_t off_vals = al(off_stats + ST_WORDS * sizeof(unsigned long long));
    const size_t total = off_vals + ((size_t)E + N) * sizeof(double);
    cudaStream_t st = ctx.st;
    DevBuf<unsigned char> d_blob;
    const size_t off_pairs = al(total);
    DRESS_TRY(d_blob.alloc(one_cta ? total : off_pairs + 8 * (size_t)E + 4 * (size_t)T, st));
    DRESS_TRY(ctx.stage->reserve(total));
    unsigned char *h = (unsigned char *)ctx.stage->ptr();
    unsigned char *dv = d_blob.get();
    const int fwd = g->variant == DRESS_VARIANT_FORWARD || g->variant == DRESS_VARIANT_BACKWARD;
    std::memset(h + off_ctr, 0, off_vals - off_ctr);           // counter and statistics
    if (one_cta) {
        pack_image(g, ioff, pairs, img, h);
        ParentDesc P{};
        P.N = N;
        P.E = E;
        P.kind = ITEM_PLAIN;
        P.k = 0;
        P.fwd = fwd;
        P.force_exact = ctx.cfg->exact_sums != 0;
        P.max_iter = max_iterations;
        P.eps = epsilon;
        P.img = img;
        P.data = dv;
        P.values = (double *)(dv + off_vals);
        P.stats = (unsigned long long *)(dv + off_stats);
        P.offset = 0;
        P.stride = 1;
        const Chunk ch{0, 1, 0, std::max(1, std::min(BATCH_SM_WARPS, (E + 31) / 32)), 0};
        std::memcpy(h + off_desc, &P, sizeof P);
        std::memcpy(h + off_chunk, &ch, sizeof ch);
    } else {
        pack_cluster(g, img, h);
    }
    DRESS_CUDA_TRY(counted_memcpy(dv, h, off_vals, cudaMemcpyHostToDevice, st));
    L.parents = (const ParentDesc *)(dv + off_desc);
    L.chunks = (const Chunk *)(dv + off_chunk);
    L.nchunks = 1;
    L.chunk_counter = (int *)(dv + off_ctr);

    cudaEvent_t e0, e1;
    DRESS_CUDA_TRY(cudaEventCreate(&e0));
    DRESS_CUDA_TRY(cudaEventCreate(&e1));
    struct EvGuard {
        cudaEvent_t a, b;
        ~EvGuard() { cudaEventDestroy(a); cudaEventDestroy(b); }
    } guard{e0, e1};
    const double setup_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    DRESS_CUDA_TRY(cudaEventRecord(e0, st));
    // A cluster sums within the range that the host knows the products to begin
    // in; where they are outside, or leave it on the way, with certificates.
    bool certified = img.span == 0;
    unsigned long long sv[ST_WORDS];
    for (;;) {
        if (one_cta) {
            DRESS_TRY(launch_batch(L, ctx.num_sms, st));
        } else {
            const ClusterFit cf{N, E, fwd, max_iterations, epsilon, img, dv, (unsigned *)(dv + off_pairs),
                                (unsigned *)(dv + off_ctr), certified, (double *)(dv + off_vals),
                                (unsigned long long *)(dv + off_stats)};
            Status ls = launch_cluster_fit(cf, st);
            if (ls.code == DRESSX_EUNSUPPORTED) return Status::Ok();     // the multi-kernel fit takes it
            DRESS_TRY(ls);
        }
        DRESS_CUDA_TRY(cudaEventRecord(e1, st));

        // statistics and results come back in one copy through the stage
        DRESS_CUDA_TRY(counted_memcpy(h + off_stats, dv + off_stats, total - off_stats, cudaMemcpyDeviceToHost, st));
        DRESS_CUDA_TRY(cudaStreamSynchronize(st));
        std::memcpy(sv, h + off_stats, sizeof sv);
        if (sv[ST_FITS] != 0) break;
        if (one_cta || certified) return Status::Ok();               // (neither gives up)
        certified = true;
        DRESS_CUDA_TRY(cudaMemsetAsync(dv + off_ctr, 0, sizeof(int), st));
    }
    std::memcpy(g->edge_dress, h + off_vals, (size_t)E * sizeof(double));
    // the norms of the last sweep (none without sweeps), as fit_graph leaves them
    if (sv[ST_SWEEPS] > 0) std::memcpy(g->vertex_dress, h + off_vals + (size_t)E * sizeof(double), (size_t)N * sizeof(double));
    float it_ms = 0.f;
    cudaEventElapsedTime(&it_ms, e0, e1);
    if (iterations) *iterations = (int)(long long)sv[ST_ITERATIONS];
    if (delta && sv[ST_SWEEPS] > 0) std::memcpy(delta, &sv[ST_DELTA], sizeof(double));
    if (stats) {
        *stats = FitStats{};
        stats->T = T;
        stats->sweeps = (int)sv[ST_SWEEPS];
        stats->setup_ms = setup_ms;
        stats->iterate_ms = it_ms;
    }
    used = true;
    return Status::Ok();
}

}  // namespace dress
