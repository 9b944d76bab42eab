// batch.h -- persistent batched fit of many small subgraphs (batch.cu).
#pragma once
#include <stdint.h>

#include <vector>

#include "engine.h"

namespace dress {

enum { ITEM_DELTA = 0, ITEM_NABLA = 1, ITEM_PLAIN = 2 };

// Packed images are staged into shared memory with 16-byte copies: every
// section starts on a 16-byte boundary.
__host__ __device__ inline long long pl_align(long long b) { return (b + 15) & ~15LL; }

// The graph as the cluster fit reads it: endpoints (u | v << 16), row offsets,
// slot targets and edge ids (u16), weights (absent when all are one power of
// two), vertex weights, initial values (absent when all are 1.0).
struct ClusterLayout {
    long long uv, off, tgt, eid, w, nw, dinit, bytes;
};

__host__ __device__ inline ClusterLayout cluster_layout(int N, int E, int S, int uniform, int has_nw, int has_dinit)
{
    ClusterLayout L;
    long long o = 0;
    L.uv = o;      o = pl_align(o + 4LL * E);
    L.off = o;     o = pl_align(o + 2LL * (N + 1));
    L.tgt = o;     o = pl_align(o + 2LL * S);
    L.eid = o;     o = pl_align(o + 2LL * S);
    L.w = o;       o = pl_align(o + (uniform ? 0 : 8LL * E));
    L.nw = o;      o = pl_align(o + (has_nw ? 8LL * N : 0));
    L.dinit = o;   o = pl_align(o + (has_dinit ? 8LL * E : 0));
    L.bytes = o;
    return L;
}

// The image of one parent graph as the batch kernel reads it.  Ids take 15
// bits (a batched graph's state fits one SM's shared memory, so it has fewer
// than 2^15 edges).  Rows are padded to whole groups of four slots and pair
// lists to whole groups of two, with the id E, whose product is zero: one
// 8-byte load brings four slots or two pairs, and no loop has a remainder.
//   edge   [E]    endpoints, u | v << 16, and the first group of the edge's
//                 pairs (NO_PAIRS: it has none)
//   row    [N]    the row's groups, first | end << 16
//   eid    [Q]    four slot edge ids, 4 x u16
//   pairs  [P2]   two pairs (u,x),(v,x), 4 x u16; bit 15 of the last id marks
//                 an edge's last group
//   w      [E]    variant weights (absent when all are one power of two)
//   nw, dinit     vertex weights, initial values, where the item has them
// Vertices and edges are renumbered, longest rows and pair lists first, so the
// lanes of a warp take items of one length.  Past the part that is staged:
//   vmap   [N], emap [E]   the image's ids of the caller's vertices and edges, u16
struct ImageLayout {
    long long edge, row, eid, pairs, w, nw, dinit, staged, vmap, emap, bytes;
};
constexpr unsigned NO_PAIRS = 0xffffffffu;

__host__ __device__ inline ImageLayout image_layout(int N, int E, int Q, int P2, int uniform, int has_nw, int has_dinit)
{
    ImageLayout L;
    long long o = 0;
    L.edge = o;    o = pl_align(o + 8LL * E);
    L.row = o;     o = pl_align(o + 4LL * N);
    L.eid = o;     o = pl_align(o + 8LL * Q);
    L.pairs = o;   o = pl_align(o + 8LL * P2);
    L.w = o;       o = pl_align(o + (uniform ? 0 : 8LL * E));
    L.nw = o;      o = pl_align(o + (has_nw ? 8LL * N : 0));
    L.dinit = o;   o = pl_align(o + (has_dinit ? 8LL * E : 0));
    L.staged = o;
    L.vmap = o;    o = pl_align(o + 2LL * N);
    L.emap = o;    o = pl_align(o + 2LL * E);
    L.bytes = o;
    return L;
}

// What the host knows of a parent's image (plan_image) and passes on.
struct ImageShape {
    int Q = 0, P2 = 0;           // groups of slots and of pairs
    int uniform = 0;             // every weight is the same power of two, wc
    int has_nw = 0, has_dinit = 0;
    double wc = 1.0;
    // high words a live product may have on the fast path (fast_range), and on
    // the wide one (batch kernel); span 0: not to be tried
    unsigned lo = 0, span = 0, wide_lo = 0, wide_span = 0;
};

// Per-request statistics record written by the kernel.
enum { ST_CURSOR = 0, ST_SWEEPS, ST_EDGE_ITERS, ST_FITS, ST_ITERATIONS, ST_DELTA, ST_WORDS };

// One parent graph of a launch and the subgraphs to fit on it.  Every
// pointer addresses device memory owned by the request, so requests of one
// launch may live in unrelated allocations.
struct ParentDesc {
    int N, E;
    int kind;            // ITEM_*
    int k;
    int fwd;             // FORWARD/BACKWARD self term
    int max_iter;
    double eps;
    ImageShape img;      // shape of the image at data
    const unsigned char *data;   // packed arrays (image_layout)
    double *values;      // DELTA/NABLA: live values in completion order;
                         // PLAIN: E final edge values, then N vertex norms
    unsigned long long *stats;   // ST_WORDS counters
    double *multisets;   // C(N,k) x E row-major matrix, or null
    const long long *ranks;      // sampled ranks (item i -> ranks[i]), or null ...
    long long offset, stride;    // ... else rank of item i = offset + i*stride
    int force_exact;             // every sum by the exact sorted path (tests of that path)
};

struct Chunk {
    int parent;
    int count;
    long long first;     // first item index within the parent
    int warps;           // warps per subgraph, at least (chunk_geometry)
    int pad = 0;
};

struct BatchLaunch {
    const ParentDesc *parents;
    const Chunk *chunks;
    int nchunks;
    int *chunk_counter;
    int ctas;                        // CTAs to an SM: 1, 2, 4 or 8, of 32 / ctas warps each
    int smem;                        // dynamic shared memory of a CTA (batch_smem)
};

constexpr int BATCH_SM_WARPS = 32;   // batch warps of an SM (64 registers a thread)
constexpr int BATCH_HEADER = 320;    // bytes ahead of the image: chunk, descriptor, counters
static_assert(sizeof(ParentDesc) + sizeof(Chunk) + 16 <= BATCH_HEADER, "descriptor header");

// How the state of a subgraph holds its values.
//   STATE_UNIFORM  two value buffers; the weight is one power of two, so sums
//                  are taken of the values and scaled at the end (exact)
//   STATE_PRODUCT  two buffers of products w*d, and the values: a term is one
//                  gather
//   STATE_VALUE    two value buffers, products formed per term: weighted
//                  graphs whose products do not fit beside the values
enum { STATE_UNIFORM = 0, STATE_PRODUCT = 1, STATE_VALUE = 2 };

// Shared memory of one subgraph's state: the value buffers with one dummy
// entry each, the vertex norms, the control words, the k mask vertices and
// their marker weights, the live-edge bits.
__host__ __device__ inline long long state_bytes(int E, int N, int k, int mode)
{
    const long long d = (mode == STATE_PRODUCT ? 3LL : 2LL) * (E + 1) + N + 2;
    return pl_align(8 * d + 12LL * (k > 0 ? k : 1) + 4LL * ((E + 31) / 32));
}

// A chunk's schedule on a CTA of `cta` warps with `room` bytes for images and states.
struct Geometry {
    int mode;            // STATE_*
    int staged;          // the image is copied into shared memory
    int warps, groups;   // warps per subgraph, subgraphs at once
    long long image, state;
};

// As many subgraphs at once as memory holds, at `warps` warps each; the image
// is staged unless that costs half of them.  Where memory holds fewer than
// the warps would serve, the idle warps are shared out among them.
__host__ __device__ inline Geometry chunk_geometry(int N, int E, int k, const ImageShape &s, long long room, int cta,
                                                   int warps)
{
    Geometry q;
    const long long image = image_layout(N, E, s.Q, s.P2, s.uniform, s.has_nw, s.has_dinit).staged;
    q.mode = s.uniform ? STATE_UNIFORM : state_bytes(E, N, k, STATE_PRODUCT) <= room ? STATE_PRODUCT : STATE_VALUE;
    q.state = state_bytes(E, N, k, q.mode);
    int want = cta / warps > 1 ? cta / warps : 1;
    if (warps > 1 && want > 15) want = 15;   // a named barrier each
    const long long in = image < room ? (room - image) / q.state : 0, out = room / q.state;
    const int gin = in < want ? (int)in : want, gout = out < want ? (int)out : want;
    q.staged = gin > 0 && 2 * gin >= gout;
    q.groups = q.staged ? gin : gout;
    q.image = q.staged ? image : 0;
    if (q.groups < 1) q.groups = 1;          // (the callers have checked that one state fits)
    q.warps = cta / q.groups;
    if (q.warps > 1 && q.groups > 15) q.warps = 1;
    const int useful = (E + 31) / 32 > warps ? (E + 31) / 32 : warps;
    if (q.warps > useful) q.warps = useful;
    return q;
}

Status launch_batch(const BatchLaunch &L, int sms, cudaStream_t st);
// The dynamic shared memory of a batch CTA with `ctas` to an SM, and the room
// that it leaves for images and states.
Status batch_smem(int device, int ctas, int *bytes);
__host__ __device__ inline long long batch_room(int smem) { return smem - BATCH_HEADER; }
// One whole-graph fit by one cluster (fit_cluster.cu).  img: Q = the row slots.
struct ClusterFit {
    int N, E, fwd, max_iter;
    double eps;
    ImageShape img;
    const unsigned char *data;           // cluster_layout
    unsigned *pairs, *cursor;            // room for 2 E + sum_e min(deg u, deg v) words, 8-byte aligned; zero
    int certified;                       // sums with certificates; 0: within img's range
    double *values;                      // E final edge values, then N vertex norms
    unsigned long long *stats;           // ST_FITS 0: a product left the range, nothing was fitted
};
// Whether one CTA's memory holds the values and norms.
bool cluster_fits(int E, int N, int S);
Status launch_cluster_fit(const ClusterFit &f, cudaStream_t st);
// A graph is batchable when one subgraph's smallest state fits and the image can
// name it: ids below 2^15 and 2^16, at most 65,535 groups of row slots (S slots of
// rows padded to groups of four).  Rows of two slots an edge stay far below; a
// caller's own rows may hold more.
constexpr long long BATCH_STATE_MAX = 227 * 1024 - BATCH_HEADER;
inline bool batch_fits(int E, int N, long long S, int k)
{
    return E < 32768 && N < 65536 && S + 3LL * N <= 4 * 65535LL &&
           state_bytes(E, N, k, STATE_VALUE) <= BATCH_STATE_MAX;
}

// ---- host planning helpers (delta_nabla.cpp) ------------------------------------
long long binom_h(int n, int k);
long long perm_h(int n, int k);
// Common-neighbour pairs of every edge by the reference's merge walk
// (libdress/src/dress.c:307-363): pairs[2t], pairs[2t+1] are the (u,x) and
// (v,x) edge ids of pair t, ioff[e]..ioff[e+1] the pairs of edge e.  Also the
// largest row and whether any row repeats a neighbour.
void merge_walk_pairs(p_dress_graph_t g, std::vector<int> &ioff, std::vector<int> &pairs, int &maxdeg, bool &dup);
// The shape of a graph's image for items of one kind and order, and the image
// itself at dst (image_layout bytes).  has_nw, has_dinit: PLAIN items.
ImageShape plan_image(p_dress_graph_t g, const std::vector<int> &ioff, int kind, int k, bool has_nw, bool has_dinit);
void pack_image(p_dress_graph_t g, const std::vector<int> &ioff, const std::vector<int> &pairs, const ImageShape &s,
                unsigned char *dst);
// The range of products (lo, span) for sums of up to `most` terms in any order.
ImageShape plan_products(double nw_min, double nw_max, long long most, bool fwd, double w_max);
// The same for the cluster fit (max_deg: the longest row).
ImageShape plan_cluster(p_dress_graph_t g, int max_deg);
void pack_cluster(p_dress_graph_t g, const ImageShape &s, unsigned char *dst);
// Chunks of a launch: the parents' items, divided so that every SM has work.
struct ChunkSource {
    int parent, N, E, k;
    long long first, items;
    ImageShape img;
};
void build_chunks(const std::vector<ChunkSource> &src, int min_warps, int sms, int ctas, int smem,
                  std::vector<Chunk> &chunks);

}  // namespace dress
