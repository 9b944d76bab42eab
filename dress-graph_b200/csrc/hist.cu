// hist.cu -- exact (value, count) histograms of many value segments.
//
// Reference: libdress/src/dress_histogram.c:40-155 -- a hash map keyed on the
// exact double (equality by ==) flattened to [bits, count] pairs sorted
// ascending by value.  Here every request's converged edge values sit in one
// contiguous segment of a device buffer; all segments are divided into buckets
// that a block sorts by the order-preserving 64-bit image of the double and
// run-length encodes in shared memory.  A run is
// one bit pattern, as the reference's map keys values by their bits (its
// hash reads the pattern) and merges them by ==: the only ==-equal values it
// can keep apart, +0 and -0, hash to different slots and merge only when
// one's probe run reaches the other; here they are two entries, -0 first.
// Every NaN is a run of its own (never == itself), as in the map.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <thread>
#include <condition_variable>
#include <vector>

#include "engine.h"
#include "hist.h"
#include "host_par.h"

namespace dress {
namespace {

constexpr int HT = 512;                 // threads per tile block
constexpr int HI = 16;                  // keys per thread per tile
constexpr int TILE = HT * HI;           // 8192 keys per tile
constexpr int RADIX = 256;

__device__ __forceinline__ unsigned long long to_ordered(unsigned long long b)
{
    return (b >> 63) ? ~b : (b | 0x8000000000000000ULL);
}
__device__ __forceinline__ unsigned long long from_ordered(unsigned long long k)
{
    return (k >> 63) ? (k & 0x7fffffffffffffffULL) : ~k;
}

__device__ __forceinline__ unsigned lanemask_lt_h()
{
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

struct Tile {
    long long begin, end;   // key range
    int seg;
};

__global__ void k_to_ordered(long long n, unsigned long long *k)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        k[i] = to_ordered(k[i]);
}

// per-tile digit counts
__global__ void __launch_bounds__(HT) k_tile_hist(const Tile *tiles, const unsigned long long *keys,
                                                  int shift, int *counts)
{
    __shared__ int c[RADIX];
    Tile t = tiles[blockIdx.x];
    for (int d = threadIdx.x; d < RADIX; d += HT) c[d] = 0;
    __syncthreads();
    for (long long i = t.begin + threadIdx.x; i < t.end; i += HT)
        atomicAdd(&c[(keys[i] >> shift) & 0xff], 1);
    __syncthreads();
    for (int d = threadIdx.x; d < RADIX; d += HT) counts[(long long)blockIdx.x * RADIX + d] = c[d];
}

// per segment: scatter offsets of every (tile, digit); flags a pass that moves keys
__global__ void __launch_bounds__(RADIX) k_seg_offsets(const long long *seg_begin, const int *seg_tile0,
                                                       const int *counts, long long *offs, int *moves)
{
    __shared__ long long base[RADIX];
    __shared__ int nonzero;
    int s = blockIdx.x, d = threadIdx.x;
    int t0 = seg_tile0[s], t1 = seg_tile0[s + 1];
    long long tot = 0;
    for (int t = t0; t < t1; ++t) tot += counts[(long long)t * RADIX + d];
    if (d == 0) nonzero = 0;
    base[d] = tot;
    __syncthreads();
    if (tot > 0) atomicAdd(&nonzero, 1);
    if (d == 0) {
        long long run = seg_begin[s];
        for (int k = 0; k < RADIX; ++k) {
            long long c = base[k];
            base[k] = run;
            run += c;
        }
    }
    __syncthreads();
    if (nonzero > 1 && d == 0) *moves = 1;
    long long run = base[d];
    for (int t = t0; t < t1; ++t) {
        offs[(long long)t * RADIX + d] = run;
        run += counts[(long long)t * RADIX + d];
    }
}

// The same offsets for one long segment, in parallel: per chunk of
// OFF_CHUNK tiles the digit sums (k_chunk_sums), then the digit bases and
// every chunk's base per digit (k_chunk_bases, one block over the chunks),
// then each chunk's tiles (k_chunk_fill).  k_seg_offsets walks every tile of
// its segment with one block, which makes a segment of 10^8 keys (12K tiles)
// cost milliseconds per pass.
constexpr int OFF_CHUNK = 64;

__global__ void __launch_bounds__(RADIX) k_chunk_sums(int nt, const int *counts, long long *csum)
{
    const int c = blockIdx.x, d = threadIdx.x;
    const int t1 = min(nt, (c + 1) * OFF_CHUNK);
    long long sum = 0;
    for (int t = c * OFF_CHUNK; t < t1; ++t) sum += counts[(long long)t * RADIX + d];
    csum[(long long)c * RADIX + d] = sum;
}

__global__ void __launch_bounds__(RADIX) k_chunk_bases(int nch, const long long *seg_begin, long long *csum,
                                                       int *moves)
{
    __shared__ long long base[RADIX];
    __shared__ int nonzero;
    const int d = threadIdx.x;
    long long tot = 0;
    for (int c = 0; c < nch; ++c) tot += csum[(long long)c * RADIX + d];
    if (d == 0) nonzero = 0;
    base[d] = tot;
    __syncthreads();
    if (tot > 0) atomicAdd(&nonzero, 1);
    if (d == 0) {
        long long run = seg_begin[0];
        for (int k = 0; k < RADIX; ++k) {
            const long long c = base[k];
            base[k] = run;
            run += c;
        }
    }
    __syncthreads();
    if (nonzero > 1 && d == 0) *moves = 1;
    long long run = base[d];
    for (int c = 0; c < nch; ++c) {
        const long long v = csum[(long long)c * RADIX + d];
        csum[(long long)c * RADIX + d] = run;
        run += v;
    }
}

__global__ void __launch_bounds__(RADIX) k_chunk_fill(int nt, const int *counts, const long long *cbase,
                                                      long long *offs)
{
    const int c = blockIdx.x, d = threadIdx.x;
    const int t1 = min(nt, (c + 1) * OFF_CHUNK);
    long long run = cbase[(long long)c * RADIX + d];
    for (int t = c * OFF_CHUNK; t < t1; ++t) {
        offs[(long long)t * RADIX + d] = run;
        run += counts[(long long)t * RADIX + d];
    }
}

// stable scatter of one tile: rounds of HT consecutive keys, each key ranked
// by (its rank among equal digits in its warp) + (same digit in earlier warps
// of the round) + (same digit in earlier rounds of the tile)
__global__ void __launch_bounds__(HT) k_tile_scatter(const Tile *tiles, const unsigned long long *src,
                                                     unsigned long long *dst, int shift,
                                                     const long long *offs, const unsigned *psrc, unsigned *pdst)
{
    constexpr int W = HT / 32;
    __shared__ int wcnt[W][RADIX];
    __shared__ int rtot[RADIX];
    __shared__ long long dbase[RADIX];
    Tile t = tiles[blockIdx.x];
    int wid = threadIdx.x >> 5;
    for (int d = threadIdx.x; d < RADIX; d += HT) dbase[d] = offs[(long long)blockIdx.x * RADIX + d];
    for (long long r0 = t.begin; r0 < t.end; r0 += HT) {
        for (int q = threadIdx.x; q < W * RADIX; q += HT) (&wcnt[0][0])[q] = 0;
        __syncthreads();
        long long i = r0 + threadIdx.x;
        bool valid = i < t.end;
        unsigned long long key = valid ? src[i] : 0ULL;
        int dg = valid ? (int)((key >> shift) & 0xff) : RADIX;      // RADIX: no key
        unsigned peers = __match_any_sync(0xffffffffu, dg);
        int rank = __popc(peers & lanemask_lt_h());
        if (valid && rank == 0) wcnt[wid][dg] = __popc(peers);
        __syncthreads();
        for (int d = threadIdx.x; d < RADIX; d += HT) {
            int run = 0;
            for (int w = 0; w < W; ++w) {
                int c = wcnt[w][d];
                wcnt[w][d] = run;
                run += c;
            }
            rtot[d] = run;
        }
        __syncthreads();
        if (valid) {
            const long long pos = dbase[dg] + wcnt[wid][dg] + rank;
            dst[pos] = key;
            if (pdst) pdst[pos] = psrc[i];          // payload moves with its key
        }
        __syncthreads();
        for (int d = threadIdx.x; d < RADIX; d += HT) dbase[d] += rtot[d];
        __syncthreads();
    }
}

// Tiles of the segments, uploaded, and the keys sorted (order-preserving
// image) within every segment; `out` is the buffer holding the result.
struct SortPlan {
    DevBuf<Tile> tiles;
    DevBuf<long long> seg_begin, seg_end;
    int nt = 0, nseg = 0;
    unsigned long long *out = nullptr;
    unsigned *pout = nullptr;
};

// ordered: keys are raw double bits, sorted by value through their
// order-preserving image (left in place); otherwise they are unsigned
// integers.  vals/valt (nullable): a 32-bit payload moved with the keys.
// key_bits < 64: the keys are below 2^key_bits, so only the passes over those
// bits run, each unconditionally (no host check of whether it moves keys).
Status sort_segments(unsigned long long *keys, unsigned long long *alt, const std::vector<long long> &begin,
                     const std::vector<long long> &len, SortPlan &sp, cudaStream_t st, int sms,
                     bool ordered = true, unsigned *vals = nullptr, unsigned *valt = nullptr, int key_bits = 64)
{
    const int nseg = (int)begin.size();
    sp.nseg = nseg;
    sp.out = keys;
    sp.pout = vals;
    std::vector<Tile> tiles;
    std::vector<int> seg_tile0((size_t)nseg + 1, 0);
    std::vector<long long> seg_end((size_t)nseg);
    long long total = 0, lo = -1, hi = 0;
    for (int s = 0; s < nseg; ++s) {
        seg_tile0[(size_t)s] = (int)tiles.size();
        seg_end[(size_t)s] = begin[(size_t)s] + len[(size_t)s];
        for (long long b = begin[(size_t)s]; b < seg_end[(size_t)s]; b += TILE)
            tiles.push_back({b, b + TILE < seg_end[(size_t)s] ? b + TILE : seg_end[(size_t)s], s});
        total += len[(size_t)s];
        if (len[(size_t)s] > 0) {
            if (lo < 0 || begin[(size_t)s] < lo) lo = begin[(size_t)s];
            if (seg_end[(size_t)s] > hi) hi = seg_end[(size_t)s];
        }
    }
    seg_tile0[(size_t)nseg] = (int)tiles.size();
    sp.nt = (int)tiles.size();
    if (total == 0) return Status::Ok();
    const int nt = sp.nt;

    DevBuf<int> d_seg_tile0, d_counts, d_moves;
    DevBuf<long long> d_offs;
    DRESS_TRY(sp.tiles.alloc((size_t)nt, st));
    DRESS_TRY(d_seg_tile0.alloc((size_t)nseg + 1, st));
    DRESS_TRY(sp.seg_begin.alloc((size_t)nseg, st));
    DRESS_TRY(sp.seg_end.alloc((size_t)nseg, st));
    DRESS_TRY(d_counts.alloc((size_t)nt * RADIX, st));
    DRESS_TRY(d_offs.alloc((size_t)nt * RADIX, st));
    DRESS_TRY(d_moves.alloc(1, st));
    DRESS_CUDA_TRY(counted_memcpy(sp.tiles.get(), tiles.data(), (size_t)nt * sizeof(Tile), cudaMemcpyHostToDevice, st));
    DRESS_CUDA_TRY(counted_memcpy(d_seg_tile0.get(), seg_tile0.data(), ((size_t)nseg + 1) * sizeof(int),
                                   cudaMemcpyHostToDevice, st));
    DRESS_CUDA_TRY(counted_memcpy(sp.seg_begin.get(), begin.data(), (size_t)nseg * sizeof(long long),
                                   cudaMemcpyHostToDevice, st));
    DRESS_CUDA_TRY(counted_memcpy(sp.seg_end.get(), seg_end.data(), (size_t)nseg * sizeof(long long),
                                   cudaMemcpyHostToDevice, st));

    // order-preserving image of the doubles over the used span
    if (ordered)
        count_launch(), k_to_ordered<<<(unsigned)((hi - lo + 255) / 256 < 64 * sms ? (hi - lo + 255) / 256 : 64 * sms), 256, 0, st>>>(
            hi - lo, keys + lo);
    unsigned long long *a = keys, *b = alt;
    unsigned *pa = vals, *pb = valt;
    const bool chunked = nseg == 1 && nt >= 4 * OFF_CHUNK;
    const int nch = (nt + OFF_CHUNK - 1) / OFF_CHUNK;
    DevBuf<long long> d_csum;
    if (chunked) DRESS_TRY(d_csum.alloc((size_t)nch * RADIX, st));
    const bool check = key_bits >= 64;
    const int passes = check ? 8 : std::max(1, (key_bits + 7) / 8);
    for (int pass = 0; pass < passes; ++pass) {
        int shift = 8 * pass;
        count_launch(), k_tile_hist<<<nt, HT, 0, st>>>(sp.tiles.get(), a, shift, d_counts.get());
        if (check) DRESS_CUDA_TRY(cudaMemsetAsync(d_moves.get(), 0, sizeof(int), st));
        if (chunked) {
            count_launch(), k_chunk_sums<<<nch, RADIX, 0, st>>>(nt, d_counts.get(), d_csum.get());
            count_launch(), k_chunk_bases<<<1, RADIX, 0, st>>>(nch, sp.seg_begin.get(), d_csum.get(), d_moves.get());
            count_launch(), k_chunk_fill<<<nch, RADIX, 0, st>>>(nt, d_counts.get(), d_csum.get(), d_offs.get());
        } else {
            count_launch(), k_seg_offsets<<<nseg, RADIX, 0, st>>>(sp.seg_begin.get(), d_seg_tile0.get(),
                                                                  d_counts.get(), d_offs.get(), d_moves.get());
        }
        if (check) {
            int moves = 0;
            DRESS_CUDA_TRY(counted_memcpy(&moves, d_moves.get(), sizeof(int), cudaMemcpyDeviceToHost, st));
            DRESS_CUDA_TRY(cudaStreamSynchronize(st));
            if (!moves) continue;
        }
        count_launch(), k_tile_scatter<<<nt, HT, 0, st>>>(sp.tiles.get(), a, b, shift, d_offs.get(), pa, pb);
        unsigned long long *t = a;
        a = b;
        b = t;
        unsigned *tp = pa;
        pa = pb;
        pb = tp;
    }
    DRESS_CUDA_TRY(cudaGetLastError());
    sp.out = a;
    sp.pout = pa;
    return Status::Ok();
}

// ---- histograms -----------------------------------------------------------------
// A bucket is a range of values that one block sorts in shared memory and
// run-length encodes on the spot: a short segment is one bucket, a long one is
// first divided at splitters drawn from a sample of its values
// (k_split_sample, k_split_count, k_split_scan, k_split_scatter).  Values
// equal to a splitter are counted apart (eq), so a value that fills much of a
// segment makes no bucket long, and no run crosses two buckets.  Every bucket
// leaves its runs at its own place (values in A, counts in B); the bases
// follow from the run counts (k_run_bases), then the runs are packed into
// [bits, count] pairs in order (k_run_pairs).
//
// Each key is read twice and written once on the way through a split (from L2
// up to about 10^7 keys) and goes through the radix passes in registers and
// shared memory only.  The passes over global memory that this replaces moved
// every key eight times through 8-byte scattered stores, with a host check
// between passes.  29.2 M values in 2,000 segments: 3.9 -> 2.0 ms; one segment of
// 2^20 values: 503 -> 133 us; 8 segments of 280,000: 750 -> 270 us.
struct Bucket {
    long long begin;
    unsigned len, eq;            // keys to sort, keys equal to the splitter above them
    int raw;                     // still double bits, in the source buffer
    int pad;
};

struct LongSeg {
    long long begin, len;
    int bk0, nb;                 // its buckets, a power of two of them
    int slot0;                   // first of its splitters and counters
    int pad;
};

constexpr int BT = 512, BI = 16, BUCKET_CAP = BT * BI;            // 8,192 keys a block
constexpr int SPLIT_T = 512, SPLIT_I = 16, SPLIT_TILE = SPLIT_T * SPLIT_I;
constexpr int MAX_SPLIT = 4096;

// Lanes of the warp with the same 8-bit digit.
__device__ __forceinline__ unsigned same_digit(unsigned d)
{
    unsigned peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const unsigned v = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? v : ~v;
    }
    return peers;
}

// Sort of n <= BUCKET_CAP keys by one block of BT threads, `items` =
// ceil(n / BT) to a thread: item i of lane l of warp w at place
// (w items + i) 32 + l, padding (~0) from place n on.  LSD radix passes of 8
// bits; a key is ranked among the equal digits before it in its warp
// (ballots), and its warp's digit counts are scanned across the warps.  The
// passes first take only the highest 24 of the bits in which the keys differ:
// for a few thousand values of a fit that leaves at most a few ties, which are
// ordered by insertion.  Where a group of ties is unordered and longer than
// TIES, all bits are sorted, lowest first.  (The bucket sorts of 2^20
// values: 120 us with all bits always, 46 us this way.)  Ends with the keys in `keys`
// in order.  cnt: BT/32 x 256 words, aux: AUX_WORDS.
constexpr int AUX_WORDS = 296, TIES = 24;

__device__ __forceinline__ void block_sort(unsigned long long (&k)[BI], int n, int items, unsigned long long *keys,
                                           unsigned *cnt, unsigned *aux)
{
    constexpr int W = BT / 32;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    unsigned *dbase = aux, *part = aux + 256, *flag = aux + 290;
    unsigned long long *diff = (unsigned long long *)(aux + 288);
    unsigned *mine = cnt + warp * 256;
    const unsigned lt = lanemask_lt_h();
    const int p0 = warp * items * 32 + lane;               // place of item 0
    if (t == 0) {
        *diff = 0ULL;
        *flag = 0u;
        keys[0] = k[0];
    }
    __syncthreads();
    {
        const unsigned long long first = keys[0];
        unsigned long long m = 0;
#pragma unroll
        for (int i = 0; i < BI; ++i)
            if (i < items && p0 + 32 * i < n) m |= k[i] ^ first;
        const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)m), hi = __reduce_or_sync(0xffffffffu, (unsigned)(m >> 32));
        if (lane == 0 && (lo | hi)) atomicOr(diff, (unsigned long long)hi << 32 | lo);
    }
    __syncthreads();
    const unsigned long long m = *diff;
    if (m == 0) {                                          // one value
#pragma unroll
        for (int i = 0; i < BI; ++i)
            if (i < items) keys[p0 + 32 * i] = k[i];
        __syncthreads();
        return;
    }
    const int high = 63 - __clzll((long long)m), low = __ffsll((long long)m) - 1;
    int from = max(low, high - 23);
    for (;;) {
        for (int shift = from; shift <= high; shift += 8) {
            if (((m >> shift) & 255u) == 0) continue;
            for (int d = lane; d < 256; d += 32) mine[d] = 0;
            __syncwarp();
            unsigned rank[BI / 2];
#pragma unroll
            for (int i = 0; i < BI; ++i)
                if (i < items) {
                    const unsigned d = (unsigned)(k[i] >> shift) & 255u;
                    const unsigned peers = same_digit(d);
                    const unsigned r = __popc(peers & lt), base = mine[d];
                    __syncwarp();
                    if (r == 0) mine[d] = base + __popc(peers);
                    __syncwarp();
                    if (i & 1) rank[i / 2] |= (base + r) << 16;
                    else rank[i / 2] = base + r;
                }
            __syncthreads();
            if (t < 256) {
                unsigned tot = 0;
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    const unsigned c = cnt[w * 256 + t];
                    cnt[w * 256 + t] = tot;
                    tot += c;
                }
                unsigned x = tot;
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (lane == 31) part[warp] = x;
                dbase[t] = x - tot;
            }
            __syncthreads();
            if (t < 256 && warp > 0) {
                unsigned before = 0;
#pragma unroll
                for (int w = 0; w < 8; ++w)
                    if (w < warp) before += part[w];
                dbase[t] += before;
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < BI; ++i)
                if (i < items) {
                    const unsigned d = (unsigned)(k[i] >> shift) & 255u;
                    keys[dbase[d] + mine[d] + ((rank[i / 2] >> (16 * (i & 1))) & 0xffffu)] = k[i];
                }
            __syncthreads();
            if (shift + 8 <= high) {
#pragma unroll
                for (int i = 0; i < BI; ++i)
                    if (i < items) k[i] = keys[p0 + 32 * i];
                __syncthreads();
            }
        }
        if (from == low) return;
        // ties of the high bits: inversions among neighbours
        unsigned inv = 0;
#pragma unroll
        for (int i = 0; i < BI; ++i)
            if (i < items && p0 + 32 * i + 1 < n && keys[p0 + 32 * i + 1] < keys[p0 + 32 * i]) inv |= 1u << i;
        if (__syncthreads_or(inv != 0) == 0) return;
        unsigned act = 0;                                  // the first inversion of a short group
        for (unsigned x = inv; x; x &= x - 1) {
            const int i = __ffs((int)x) - 1, p = p0 + 32 * i;
            const unsigned long long top = keys[p] >> from;
            int h = p, e = p + 1;
            bool first = true;
            while (h > 0 && p - h <= TIES && (keys[h - 1] >> from) == top) {
                first &= keys[h - 1] <= keys[h];
                --h;
            }
            while (e + 1 < n && e - h <= TIES && (keys[e + 1] >> from) == top) ++e;
            if (e - h + 1 > TIES) *flag = 1u;
            else if (first) act |= 1u << i;
        }
        __syncthreads();
        if (*flag == 0) {
            for (unsigned x = act; x; x &= x - 1) {
                const int i = __ffs((int)x) - 1, p = p0 + 32 * i;
                const unsigned long long top = keys[p] >> from;
                int h = p;
                while (h > 0 && (keys[h - 1] >> from) == top) --h;
                for (int q = h + 1; q < n && (keys[q] >> from) == top; ++q) {
                    const unsigned long long v = keys[q];
                    int r = q;
                    for (; r > h && keys[r - 1] > v; --r) keys[r] = keys[r - 1];
                    keys[r] = v;
                }
            }
            __syncthreads();
            return;
        }
#pragma unroll
        for (int i = 0; i < BI; ++i)
            if (i < items) k[i] = keys[p0 + 32 * i];
        __syncthreads();
        from = low;
    }
}

__device__ __forceinline__ bool is_nan_key(unsigned long long k)
{
    const double a = __longlong_as_double((long long)from_ordered(k));
    return a != a;
}

constexpr size_t BUCKET_SMEM = (size_t)BUCKET_CAP * 8 + (size_t)(BT / 32) * 1024 + 4 * AUX_WORDS;

// Exclusive position of this thread's `v` among the block's, and the total.
template <int T>
__device__ __forceinline__ unsigned block_offset(unsigned v, unsigned *part, unsigned &total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) part[warp] = x;
    __syncthreads();
    unsigned before = 0;
    total = 0;
    for (int w = 0; w < T / 32; ++w) {
        if (w < warp) before += part[w];
        total += part[w];
    }
    return before + x - v;
}

// One bucket beyond a block's capacity: radix passes over global memory between
// A and B by one block, then the runs tile by tile.  Returns the runs.  Rare up to
// 6*10^6 distinct values a segment, 15 % of the buckets at 2*10^7 and nearly all
// from 6*10^7 on (k_split_sample), with 4,096 of them at work: a segment of
// 19.5 M, 66 M, 158 M and 536 M values takes 2.3, 8.9, 22 and 76 ms, the passes
// over global memory by the whole device that this replaces 2.7, 8.9, 23 and 82.
__device__ __noinline__ unsigned long_bucket(long long begin, unsigned n, unsigned long long *A, unsigned long long *B,
                                             unsigned *cnt, unsigned *aux)
{
    constexpr int I = BI, W = BT / 32;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    unsigned *mine = cnt + warp * 256, *dbase = aux, *part = aux + 256;
    const unsigned lt = lanemask_lt_h();
    unsigned long long *src = A + begin, *dst = B + begin;
    for (int shift = 0; shift < 64; shift += 8) {          // an even number: the result is in A
        for (int d = t; d < 256; d += BT) dbase[d] = 0;
        __syncthreads();
        for (unsigned i = t; i < n; i += BT) atomicAdd(&dbase[(unsigned)(src[i] >> shift) & 255u], 1u);
        __syncthreads();
        {
            unsigned total;
            const unsigned c = t < 256 ? dbase[t] : 0u;
            const unsigned o = block_offset<BT>(c, part, total);
            if (t < 256) dbase[t] = o;
        }
        for (unsigned t0 = 0; t0 < n; t0 += BUCKET_CAP) {
            for (int d = lane; d < 256; d += 32) mine[d] = 0;
            __syncwarp();
            unsigned long long k[I];
            unsigned rank[I];
#pragma unroll
            for (int i = 0; i < I; ++i) {
                const unsigned p = t0 + (warp * I + i) * 32 + lane;
                k[i] = p < n ? src[p] : ~0ULL;             // padding ranks after every key
            }
#pragma unroll
            for (int i = 0; i < I; ++i) {
                const unsigned d = (unsigned)(k[i] >> shift) & 255u;
                const unsigned peers = same_digit(d), r = __popc(peers & lt), base = mine[d];
                __syncwarp();
                if (r == 0) mine[d] = base + __popc(peers);
                __syncwarp();
                rank[i] = base + r;
            }
            __syncthreads();
            unsigned tot = 0;
            if (t < 256)
                for (int w = 0; w < W; ++w) {
                    const unsigned c = cnt[w * 256 + t];
                    cnt[w * 256 + t] = tot;
                    tot += c;
                }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < I; ++i) {
                const unsigned p = t0 + (warp * I + i) * 32 + lane, d = (unsigned)(k[i] >> shift) & 255u;
                if (p < n) dst[dbase[d] + mine[d] + rank[i]] = k[i];
            }
            __syncthreads();
            if (t < 256) dbase[t] += tot;                  // the last tile's padding is never used again
            __syncthreads();
        }
        unsigned long long *s = src;
        src = dst;
        dst = s;
    }
    // runs in place: values to A, starts to B, then counts from the starts
    unsigned long long prev = 0;
    unsigned runs = 0;
    for (unsigned t0 = 0; t0 < n; t0 += BT) {
        const unsigned p = t0 + t;
        const unsigned long long k = p < n ? src[p] : 0ULL;
        const unsigned long long before = p == 0 || p >= n ? 0ULL : t == 0 ? prev : src[p - 1];
        const bool h = p < n && (p == 0 || k != before || is_nan_key(k));
        prev = t == 0 && t0 + BT <= n ? src[t0 + BT - 1] : 0ULL;
        __syncthreads();                                   // the tile is read before its places are written
        unsigned total;
        const unsigned at = runs + block_offset<BT>(h, part, total);
        if (h) {
            src[at] = from_ordered(k);
            dst[at] = p;
        }
        runs += total;
        __syncthreads();
    }
    for (unsigned t0 = 0; t0 < runs; t0 += BT) {
        const unsigned r = t0 + t;
        unsigned long long c = 0;
        if (r < runs) c = (r + 1 < runs ? dst[r + 1] : (unsigned long long)n) - dst[r];
        __syncthreads();
        if (r < runs) dst[r] = c;
        __syncthreads();
    }
    return runs;
}

// One block per bucket: its keys sorted, its runs written.
__global__ void __launch_bounds__(BT, 2) k_bucket_runs(const Bucket *bk, const unsigned long long *src,
                                                       unsigned long long *A, unsigned long long *B, unsigned *runs)
{
    extern __shared__ __align__(16) unsigned char hsm[];
    const Bucket b = bk[blockIdx.x];
    // the splitter's run is sorted along when all fits
    const bool all = (unsigned long long)b.len + b.eq <= BUCKET_CAP;
    const unsigned n = all ? b.len + b.eq : b.len, eq = all ? 0u : b.eq;
    unsigned long long *keys = (unsigned long long *)hsm;
    unsigned *cnt = (unsigned *)(keys + BUCKET_CAP), *aux = cnt + (BT / 32) * 256, *part = aux + 256;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    unsigned R = 0;
    const unsigned long long sv = eq ? A[b.begin + n] : 0ULL;      // the splitter's value
    if (n > BUCKET_CAP) {
        R = long_bucket(b.begin, n, A, B, cnt, aux);
    } else if (n) {
        const int items = (int)((n + BT - 1) / BT), p0 = warp * items * 32 + lane;
        unsigned long long k[BI];
        const unsigned long long *in = b.raw ? src : A;
#pragma unroll
        for (int i = 0; i < BI; ++i) {
            const unsigned p = p0 + 32 * i;
            k[i] = ~0ULL;
            if (i < items && p < n) {
                k[i] = in[b.begin + p];
                if (b.raw) k[i] = to_ordered(k[i]);
            }
        }
        block_sort(k, (int)n, items, keys, cnt, aux);
        // run heads, their starts in order (u16, over the counters)
        unsigned heads = 0, own = 0;                       // one bit an item; the warp's heads
#pragma unroll
        for (int i = 0; i < BI; ++i)
            if (i < items) {
                const unsigned p = p0 + 32 * i;
                const unsigned long long x = keys[p];
                const bool h = p < n && (p == 0 || x != keys[p - 1] || is_nan_key(x));
                if (h) heads |= 1u << i;
                own += __popc(__ballot_sync(0xffffffffu, h));
            }
        if (lane == 0) part[warp] = own;
        __syncthreads();
        unsigned at = 0;
        for (int w = 0; w < BT / 32; ++w) {
            if (w < warp) at += part[w];
            R += part[w];
        }
        unsigned short *starts = (unsigned short *)cnt;
#pragma unroll
        for (int i = 0; i < BI; ++i)
            if (i < items) {
                const bool h = (heads >> i) & 1u;
                const unsigned m = __ballot_sync(0xffffffffu, h);
                if (h) starts[at + __popc(m & lanemask_lt_h())] = (unsigned short)(p0 + 32 * i);
                at += __popc(m);
            }
        __syncthreads();
        for (unsigned r = t; r < R; r += BT) {
            const unsigned p = starts[r], e = r + 1 < R ? starts[r + 1] : n;
            A[b.begin + r] = from_ordered(keys[p]);
            B[b.begin + r] = e - p;
        }
    }
    if (eq) {
        __syncthreads();
        const bool nan = is_nan_key(sv);
        const unsigned m = nan ? eq : 1u;                  // every NaN is a run
        for (unsigned r = t; r < m; r += BT) {
            A[b.begin + R + r] = from_ordered(sv);
            B[b.begin + R + r] = nan ? 1u : eq;
        }
        R += m;
    }
    if (t == 0) runs[blockIdx.x] = R;
}

// Splitters of a long segment: every (samples / buckets)-th of a sorted sample
// of up to BUCKET_CAP values at jittered places (a plain stride would meet the
// same edge of every subgraph), equal ones once.  Eight samples a bucket, up to
// 1,024 buckets (3*10^6 values), keep nearly every bucket below 2.5 times the
// mean; beyond, four and then two, and from 1.3*10^7 values on the mean grows:
// what a block cannot hold goes to long_bucket.
__global__ void __launch_bounds__(BT) k_split_sample(const LongSeg *segs, const unsigned long long *src,
                                                     unsigned long long *split, int *nsplit)
{
    extern __shared__ __align__(16) unsigned char hsm[];
    unsigned long long *keys = (unsigned long long *)hsm;
    unsigned *cnt = (unsigned *)(keys + BUCKET_CAP), *aux = cnt + (BT / 32) * 256;
    const LongSeg s = segs[blockIdx.x];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int ns = min(BUCKET_CAP, 8 * s.nb), items = (ns + BT - 1) / BT;
    const unsigned long long step = (unsigned long long)s.len / ns;
    unsigned long long k[BI];
#pragma unroll
    for (int i = 0; i < BI; ++i) {
        const unsigned p = (warp * items + i) * 32 + lane;
        k[i] = ~0ULL;
        if (i < items && (int)p < ns) {
            unsigned h = p * 2654435761u;
            h ^= h >> 15;
            h *= 2246822519u;
            h ^= h >> 13;
            k[i] = to_ordered(src[s.begin + (long long)(step * p + h % step)]);
        }
    }
    block_sort(k, ns, items, keys, cnt, aux);
    const int per = ns / s.nb;                             // a power of two, at least 2
    unsigned total = 0;
    for (int j0 = 0; j0 < s.nb - 1; j0 += BT) {
        const int j = j0 + t;
        bool h = false;
        unsigned long long x = 0;
        if (j < s.nb - 1) {
            x = keys[(j + 1) * per];
            h = j == 0 || x != keys[j * per];
        }
        unsigned m;
        const unsigned at = total + block_offset<BT>(h, aux + 256, m);
        if (h) split[s.slot0 + at] = x;
        total += m;
    }
    if (t == 0) nsplit[blockIdx.x] = (int)total;
}

// Bucket of every key of a tile: 2 j between splitters j-1 and j, 2 j + 1 equal
// to splitter j; the tile's counts are added up in shared memory first.
__global__ void __launch_bounds__(SPLIT_T) k_split_count(const LongSeg *segs, const Tile *tiles,
                                                         const unsigned long long *src, const unsigned long long *split,
                                                         const int *nsplit, unsigned short *ids, unsigned *counts)
{
    extern __shared__ __align__(16) unsigned char hsm[];
    const Tile tl = tiles[blockIdx.x];
    const LongSeg s = segs[tl.seg];
    unsigned long long *sp = (unsigned long long *)hsm;
    unsigned *c = (unsigned *)(sp + s.nb);
    const int m = nsplit[tl.seg];
    for (int j = threadIdx.x; j < m; j += SPLIT_T) sp[j] = split[s.slot0 + j];
    for (int j = threadIdx.x; j < 2 * s.nb; j += SPLIT_T) c[j] = 0;
    __syncthreads();
#pragma unroll 4
    for (int i = 0; i < SPLIT_I; ++i) {
        const long long p = tl.begin + i * SPLIT_T + threadIdx.x;
        if (p >= tl.end) break;
        const unsigned long long k = to_ordered(src[p]);
        int j = 0;                                         // splitters at or below k
        for (int st = s.nb >> 1; st > 0; st >>= 1)
            if (j + st <= m && sp[j + st - 1] <= k) j += st;
        const unsigned id = j > 0 && sp[j - 1] == k ? 2 * j - 1 : 2 * j;
        ids[p] = (unsigned short)id;
        atomicAdd(&c[id], 1u);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < 2 * s.nb; j += SPLIT_T)
        if (c[j]) atomicAdd(&counts[2 * s.slot0 + j], c[j]);
}

// Buckets and cursors of a long segment from its counts.
__global__ void __launch_bounds__(1024) k_split_scan(const LongSeg *segs, unsigned *counts, Bucket *bk)
{
    __shared__ unsigned part[32];
    const LongSeg s = segs[blockIdx.x];
    unsigned run = 0;
    for (int j0 = 0; j0 < s.nb; j0 += 1024) {
        const int j = j0 + threadIdx.x;
        unsigned a = 0, e = 0;
        if (j < s.nb) {
            a = counts[2 * (s.slot0 + j)];
            e = counts[2 * (s.slot0 + j) + 1];
        }
        unsigned total;
        const unsigned at = run + block_offset<1024>(a + e, part, total);
        if (j < s.nb) {
            counts[2 * (s.slot0 + j)] = at;
            counts[2 * (s.slot0 + j) + 1] = at + a;
            bk[s.bk0 + j] = {s.begin + at, a, e, 0, 0};
        }
        run += total;
    }
}

__global__ void __launch_bounds__(SPLIT_T) k_split_scatter(const LongSeg *segs, const Tile *tiles,
                                                           const unsigned long long *src, const unsigned short *ids,
                                                           unsigned *cursor, unsigned long long *A)
{
    extern __shared__ __align__(16) unsigned char hsm[];
    const Tile tl = tiles[blockIdx.x];
    const LongSeg s = segs[tl.seg];
    unsigned *c = (unsigned *)hsm;
    for (int j = threadIdx.x; j < 2 * s.nb; j += SPLIT_T) c[j] = 0;
    __syncthreads();
    unsigned id[SPLIT_I], rk[SPLIT_I];
#pragma unroll
    for (int i = 0; i < SPLIT_I; ++i) {
        const long long p = tl.begin + i * SPLIT_T + threadIdx.x;
        id[i] = p < tl.end ? ids[p] : 0xffffffffu;
        if (p < tl.end) rk[i] = atomicAdd(&c[id[i]], 1u);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < 2 * s.nb; j += SPLIT_T)
        if (c[j]) c[j] = atomicAdd(&cursor[2 * s.slot0 + j], c[j]);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < SPLIT_I; ++i) {
        const long long p = tl.begin + i * SPLIT_T + threadIdx.x;
        if (p < tl.end) A[s.begin + c[id[i]] + rk[i]] = to_ordered(src[p]);
    }
}

// First run of every bucket, and of every segment (seg_bk: its first bucket).
__global__ void __launch_bounds__(1024) k_run_bases(int nbk, const unsigned *runs, long long *base, int nseg,
                                                    const int *seg_bk, long long *seg_runs)
{
    __shared__ unsigned part[32];
    long long run = 0;
    for (int b0 = 0; b0 < nbk; b0 += 4096) {
        unsigned v[4], sum = 0;
        const int b = b0 + 4 * (int)threadIdx.x;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i] = b + i < nbk ? runs[b + i] : 0u;
            sum += v[i];
        }
        unsigned total;
        long long at = run + block_offset<1024>(sum, part, total);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (b + i < nbk) base[b + i] = at;
            at += v[i];
        }
        run += total;
    }
    if (threadIdx.x == 0) base[nbk] = run;
    __syncthreads();
    for (int s = threadIdx.x; s <= nseg; s += 1024) seg_runs[s] = base[seg_bk[s]];
}

__global__ void __launch_bounds__(128) k_run_pairs(const Bucket *bk, const unsigned *runs, const long long *base,
                                                   const unsigned long long *A, const unsigned long long *B,
                                                   long long *pairs, int aligned, long long *num_runs)
{
    if (num_runs && blockIdx.x == 0 && threadIdx.x == 0) *num_runs = base[gridDim.x];
    const long long b0 = bk[blockIdx.x].begin, o = base[blockIdx.x];
    const unsigned R = runs[blockIdx.x];
    for (unsigned r = threadIdx.x; r < R; r += 128) {
        const longlong2 q = make_longlong2((long long)A[b0 + r], (long long)B[b0 + r]);
        if (aligned) {
            ((longlong2 *)pairs)[o + r] = q;
        } else {                                           // a caller's buffer may start at any int64
            pairs[2 * (o + r)] = q.x;
            pairs[2 * (o + r) + 1] = q.y;
        }
    }
}

// Buckets for a segment's length: 1,536 to 3,072 keys each (a block holds 8,192).
inline int split_buckets(long long len)
{
    int nb = 4;
    while (nb < MAX_SPLIT && (long long)nb * 3072 < len) nb <<= 1;
    return nb;
}

size_t split_count_bytes(int nb) { return (size_t)nb * 16; }

// The attributes of the kernels above, once per device.
// always: also where they were set before (a device reset drops them)
Status hist_attributes(bool always)
{
    static std::mutex mu;
    static unsigned long long done[2] = {0, 0};            // devices 0..127
    int dev = 0;
    DRESS_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    if (!always && dev < 128 && ((done[dev >> 6] >> (dev & 63)) & 1ULL)) return Status::Ok();
    const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
    DRESS_CUDA_TRY(cudaFuncSetAttribute(k_bucket_runs, at, (int)BUCKET_SMEM));
    DRESS_CUDA_TRY(cudaFuncSetAttribute(k_split_sample, at, (int)BUCKET_SMEM));
    DRESS_CUDA_TRY(cudaFuncSetAttribute(k_split_count, at, (int)split_count_bytes(MAX_SPLIT)));
    if (dev < 128) done[dev >> 6] |= 1ULL << (dev & 63);
    return Status::Ok();
}

// The device side of a set of segments, in order; see the section's head.
// Everything it points to is device memory.
struct HistLaunch {
    int nseg, nbk, nlong, ntiles, max_nb;
    const unsigned long long *src;
    unsigned long long *A, *B;
    Bucket *bk;
    const LongSeg *segs;
    const Tile *tiles;
    const int *seg_bk;
    unsigned long long *split;
    int *nsplit;
    unsigned *counts;                                      // zero on entry
    unsigned short *ids;
    unsigned *runs;
    long long *base, *seg_runs;
};

Status launch_hist_runs(const HistLaunch &h, cudaStream_t st, bool attributes = false)
{
    DRESS_TRY(hist_attributes(attributes));
    if (h.nlong) {
        count_launch(), k_split_sample<<<h.nlong, BT, BUCKET_SMEM, st>>>(h.segs, h.src, h.split, h.nsplit);
        count_launch(), k_split_count<<<h.ntiles, SPLIT_T, split_count_bytes(h.max_nb), st>>>(
            h.segs, h.tiles, h.src, h.split, h.nsplit, h.ids, h.counts);
        count_launch(), k_split_scan<<<h.nlong, 1024, 0, st>>>(h.segs, h.counts, h.bk);
        count_launch(), k_split_scatter<<<h.ntiles, SPLIT_T, (size_t)h.max_nb * 8, st>>>(h.segs, h.tiles, h.src, h.ids,
                                                                                        h.counts, h.A);
    }
    count_launch(), k_bucket_runs<<<h.nbk, BT, BUCKET_SMEM, st>>>(h.bk, h.src, h.A, h.B, h.runs);
    count_launch(), k_run_bases<<<1, 1024, 0, st>>>(h.nbk, h.runs, h.base, h.nseg, h.seg_bk, h.seg_runs);
    DRESS_CUDA_TRY(cudaGetLastError());
    return Status::Ok();
}

Status launch_hist_pairs(const HistLaunch &h, long long *pairs, cudaStream_t st, long long *num_runs = nullptr)
{
    const int aligned = ((uintptr_t)pairs & 15) == 0;
    count_launch(), k_run_pairs<<<h.nbk, 128, 0, st>>>(h.bk, h.runs, h.base, h.A, h.B, pairs, aligned,
                                                  num_runs);
    DRESS_CUDA_TRY(cudaGetLastError());
    return Status::Ok();
}

}  // namespace

Status segmented_sort(unsigned long long *keys, unsigned long long *alt, const std::vector<long long> &begin,
                      const std::vector<long long> &len, unsigned long long **sorted, cudaStream_t st, int sms)
{
    SortPlan sp;
    DRESS_TRY(sort_segments(keys, alt, begin, len, sp, st, sms));
    *sorted = sp.out;
    return Status::Ok();
}

Status sort_pairs(unsigned long long *keys, unsigned long long *alt, unsigned *vals, unsigned *valt, long long n,
                  unsigned long long **sorted_keys, unsigned **sorted_vals, cudaStream_t st, int sms, int key_bits)
{
    SortPlan sp;
    DRESS_TRY(sort_segments(keys, alt, std::vector<long long>{0}, std::vector<long long>{n}, sp, st, sms, false,
                            vals, valt, key_bits));
    *sorted_keys = sp.out;
    *sorted_vals = sp.pout;
    return Status::Ok();
}

// Counts and places within a segment take 32 bits: a longer segment is taken in
// pieces, whose lists are merged on the host (a result of some 10^9 runs would
// not fit the device beside the values; the usual one of so many values is short).
constexpr long long SEGMENT_MAX = 1LL << 31;

static Status histogram_pieces(unsigned long long *keys, unsigned long long *alt, const std::vector<long long> &begin,
                               const std::vector<long long> &len, HistResult &res, cudaStream_t st)
{
    const int nseg = (int)begin.size();
    std::vector<long long> pb, pl, first;                  // pieces, and every segment's first
    for (int s = 0; s < nseg; ++s) {
        first.push_back((long long)pb.size());
        for (long long o = 0; o < len[(size_t)s]; o += SEGMENT_MAX) {
            pb.push_back(begin[(size_t)s] + o);
            pl.push_back(std::min(SEGMENT_MAX, len[(size_t)s] - o));
        }
    }
    first.push_back((long long)pb.size());
    std::vector<long long> all;
    try {
        std::vector<std::vector<long long>> lists;
        {
            HistResult part;
            DRESS_TRY(histogram_device(keys, alt, pb, pl, part, st));
            DRESS_TRY(histogram_download(part, lists, st));
        }
        for (int s = 0; s < nseg; ++s) {
            std::vector<const int64_t *> p;
            std::vector<int64_t> n;
            for (long long i = first[(size_t)s]; i < first[(size_t)s + 1]; ++i) {
                p.push_back((const int64_t *)lists[(size_t)i].data());
                n.push_back((int64_t)lists[(size_t)i].size());
            }
            int64_t *out = nullptr, out_len = 0;
            if (dressx_hist_merge(p.data(), n.data(), (int)p.size(), &out, &out_len) != DRESSX_OK) throw std::bad_alloc();
            const std::unique_ptr<int64_t, void (*)(void *)> own(out, std::free);
            all.insert(all.end(), out, out + out_len);
            res.seg_runs[(size_t)s + 1] = (long long)all.size() / 2;
        }
    } catch (const std::bad_alloc &) {
        return Status::Err(DRESSX_ENOMEM, "host allocation of the histograms failed");
    }
    res.R = res.seg_runs[(size_t)nseg];
    DRESS_TRY(res.pairs.alloc(all.size(), st));
    DRESS_CUDA_TRY(counted_memcpy(res.pairs.get(), all.data(), all.size() * 8, cudaMemcpyHostToDevice, st));
    DRESS_CUDA_TRY(cudaStreamSynchronize(st));
    return Status::Ok();
}

Status histogram_device(unsigned long long *keys, unsigned long long *alt, const std::vector<long long> &begin,
                        const std::vector<long long> &len, HistResult &res, cudaStream_t st)
{
    const int nseg = (int)begin.size();
    res.nseg = nseg;
    res.R = 0;
    res.seg_runs.assign((size_t)nseg + 1, 0);
    for (long long n : len)
        if (n > SEGMENT_MAX) return histogram_pieces(keys, alt, begin, len, res, st);
    // descriptors of the launch, packed into one upload
    std::vector<Bucket> bk;
    std::vector<LongSeg> segs;
    std::vector<Tile> tiles;
    std::vector<int> seg_bk((size_t)nseg + 1);
    HistLaunch h{};
    int slots = 0;
    long long ids_lo = -1, ids_hi = 0;
    for (int s = 0; s < nseg; ++s) {
        const long long b = begin[(size_t)s], n = len[(size_t)s];
        seg_bk[(size_t)s] = (int)bk.size();
        if (n <= 0) continue;
        if (n <= BUCKET_CAP) {
            bk.push_back({b, (unsigned)n, 0u, 1, 0});
            continue;
        }
        const int nb = split_buckets(n);
        for (long long t = b; t < b + n; t += SPLIT_TILE)
            tiles.push_back({t, std::min(t + SPLIT_TILE, b + n), (int)segs.size()});
        segs.push_back({b, n, (int)bk.size(), nb, slots, 0});
        bk.resize(bk.size() + (size_t)nb, Bucket{b, 0u, 0u, 0, 0});
        slots += nb;
        h.max_nb = std::max(h.max_nb, nb);
        if (ids_lo < 0) ids_lo = b;
        ids_lo = std::min(ids_lo, b);
        ids_hi = std::max(ids_hi, b + n);
    }
    seg_bk[(size_t)nseg] = (int)bk.size();
    if (bk.empty()) return Status::Ok();
    h.nseg = nseg;
    h.nbk = (int)bk.size();
    h.nlong = (int)segs.size();
    h.ntiles = (int)tiles.size();
    h.src = keys;
    h.A = alt;
    h.B = keys;
    const auto al = [](size_t x) { return (x + 15) & ~(size_t)15; };
    const size_t o_seg = al(bk.size() * sizeof(Bucket)), o_tile = al(o_seg + segs.size() * sizeof(LongSeg));
    const size_t o_sbk = al(o_tile + tiles.size() * sizeof(Tile)), up = al(o_sbk + seg_bk.size() * sizeof(int));
    const size_t o_split = up, o_ns = al(o_split + 8 * (size_t)slots), o_cnt = al(o_ns + 4 * segs.size());
    const size_t o_runs = al(o_cnt + 8 * (size_t)slots), o_base = al(o_runs + 4 * bk.size());
    const size_t o_sr = al(o_base + 8 * (bk.size() + 1)), all = al(o_sr + 8 * ((size_t)nseg + 1));
    std::vector<unsigned char> host(up);
    std::memcpy(host.data(), bk.data(), bk.size() * sizeof(Bucket));
    if (!segs.empty()) std::memcpy(host.data() + o_seg, segs.data(), segs.size() * sizeof(LongSeg));
    if (!tiles.empty()) std::memcpy(host.data() + o_tile, tiles.data(), tiles.size() * sizeof(Tile));
    std::memcpy(host.data() + o_sbk, seg_bk.data(), seg_bk.size() * sizeof(int));
    DevBuf<unsigned char> work;
    DevBuf<unsigned short> ids;
    DRESS_TRY(work.alloc(all, st));
    unsigned char *w = work.get();
    DRESS_CUDA_TRY(counted_memcpy(w, host.data(), up, cudaMemcpyHostToDevice, st));
    h.bk = (Bucket *)w;
    h.segs = (const LongSeg *)(w + o_seg);
    h.tiles = (const Tile *)(w + o_tile);
    h.seg_bk = (const int *)(w + o_sbk);
    h.split = (unsigned long long *)(w + o_split);
    h.nsplit = (int *)(w + o_ns);
    h.counts = (unsigned *)(w + o_cnt);
    h.runs = (unsigned *)(w + o_runs);
    h.base = (long long *)(w + o_base);
    h.seg_runs = (long long *)(w + o_sr);
    if (slots) {
        DRESS_TRY(ids.alloc((size_t)(ids_hi - ids_lo), st));
        h.ids = ids.get() - ids_lo;
        DRESS_CUDA_TRY(cudaMemsetAsync(h.counts, 0, 8 * (size_t)slots, st));
    }
    DRESS_TRY(launch_hist_runs(h, st));
    DRESS_CUDA_TRY(counted_memcpy(res.seg_runs.data(), h.seg_runs, 8 * ((size_t)nseg + 1), cudaMemcpyDeviceToHost, st));
    DRESS_CUDA_TRY(cudaStreamSynchronize(st));
    res.R = res.seg_runs[(size_t)nseg];
    DRESS_TRY(res.pairs.alloc(2 * (size_t)res.R, st));
    return launch_hist_pairs(h, res.pairs.get(), st);
}

Status histogram_fetch(HistResult &res, std::vector<int64_t *> &outs, std::vector<long long> &lens, Pinned *stage,
                       cudaStream_t st, int max_threads)
{
    const int nseg = res.nseg;
    outs.assign((size_t)nseg, nullptr);
    lens.assign((size_t)nseg, 0);
    const long long R = res.R;
    if (R == 0) return Status::Ok();
    std::vector<long long> first((size_t)nseg, 0);
    for (int sg = 0; sg < nseg; ++sg) {
        first[(size_t)sg] = res.seg_runs[(size_t)sg];
        lens[(size_t)sg] = 2 * (res.seg_runs[(size_t)sg + 1] - res.seg_runs[(size_t)sg]);
    }
    const size_t bytes = 2 * (size_t)R * sizeof(long long);
    long long *host = nullptr;
    std::vector<long long> pageable;
    const bool pinned = stage && stage->reserve(bytes).ok();
    if (pinned) {
        host = (long long *)stage->ptr();
    } else {
        pageable.resize(2 * (size_t)R);
        host = pageable.data();
    }
    // The output, runs [0, R) in segment order, is cut into one part per host
    // thread, balanced by bytes; each part is its own download.  A thread
    // allocates the arrays of the segments that start in its part, and after
    // a barrier (a segment may reach into later parts) maps the pages of its
    // part's share of the arrays while the downloads stream in -- the page
    // faults of fresh memory cost more than the copy -- then copies its
    // share once its part landed.  From 4 MiB on a thread per MiB: 14 MB took
    // one thread 4.3 ms.  Below, the caller's thread does it all and waits by
    // spinning: an event's blocking wait costs 0.3 ms.
    const int nthr = pinned && bytes > (4u << 20) ? std::min(max_threads, host_threads((long long)(bytes >> 20))) : 1;
    const int parts = std::max(1, nthr);
    std::vector<long long> pcut((size_t)parts + 1);
    for (int t = 0; t <= parts; ++t) pcut[(size_t)t] = R * t / parts;
    std::vector<cudaEvent_t> ev((size_t)parts, nullptr);
    Status err;
    for (int t = 0; t < parts && err.ok(); ++t) {
        const long long r0 = pcut[(size_t)t], r1 = pcut[(size_t)t + 1];
        if (r1 <= r0) continue;
        if (parts > 1 &&
            cudaEventCreateWithFlags(&ev[(size_t)t], cudaEventDisableTiming | cudaEventBlockingSync) != cudaSuccess) {
            ev[(size_t)t] = nullptr;
            err = Status::Err(DRESSX_ECUDA, "event creation failed");
            break;
        }
        cudaError_t e = counted_memcpy(host + 2 * r0, res.pairs.get() + 2 * r0, 2 * (size_t)(r1 - r0) * sizeof(long long),
                                       cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess && parts > 1) e = cudaEventRecord(ev[(size_t)t], st);
        if (e != cudaSuccess) err = Status::Err(DRESSX_ECUDA, std::string("histogram download: ") + cudaGetErrorString(e));
    }
    // segments in part order: the first segment whose runs reach into each part
    std::vector<int> seg0((size_t)parts + 1, nseg);
    {
        int sg = 0;
        for (int t = 0; t < parts; ++t) {
            while (sg < nseg && (lens[(size_t)sg] == 0 || first[(size_t)sg] + lens[(size_t)sg] / 2 <= pcut[(size_t)t]))
                ++sg;
            seg0[(size_t)t] = sg;
        }
    }
    std::atomic<bool> nomem{false};
    std::mutex mu;
    std::condition_variable cv;
    int ready = 0;                               // parts landed; -1 once the downloads failed
    int arrived = 0;                             // parts whose arrays are allocated
    auto barrier = [&] {
        std::unique_lock<std::mutex> lk(mu);
        if (++arrived == parts) cv.notify_all();
        else cv.wait(lk, [&] { return arrived == parts; });
    };
    auto part_work = [&](int t) {
        const long long p0 = pcut[(size_t)t], p1 = pcut[(size_t)t + 1];
        // the segments starting in this part
        for (int sg = seg0[(size_t)t]; sg < nseg && first[(size_t)sg] < p1; ++sg) {
            const size_t n = (size_t)lens[(size_t)sg] * sizeof(int64_t);
            if (!n || first[(size_t)sg] < p0) continue;
            outs[(size_t)sg] = (int64_t *)std::malloc(n);
            if (!outs[(size_t)sg]) nomem = true;
        }
        barrier();
        // this part's share of segment sg: runs [a, b)
        auto share = [&](int sg, long long &a, long long &b) {
            a = std::max(p0, first[(size_t)sg]);
            b = std::min(p1, first[(size_t)sg] + lens[(size_t)sg] / 2);
        };
        for (int sg = seg0[(size_t)t]; sg < nseg && first[(size_t)sg] < p1; ++sg) {
            long long a, b;
            share(sg, a, b);
            char *o = (char *)outs[(size_t)sg];
            if (b <= a || !o) continue;
            const size_t lo_b = (size_t)(a - first[(size_t)sg]) * 16, hi_b = (size_t)(b - first[(size_t)sg]) * 16;
            for (size_t x = lo_b; x < hi_b; x += 4096) ((volatile char *)o)[x] = 0;
        }
        bool ok;
        if (parts == 1) {
            ok = err.ok() && cudaStreamSynchronize(st) == cudaSuccess;
            if (!ok && err.ok()) err = Status::Err(DRESSX_ECUDA, "histogram download failed");
        } else {
            std::unique_lock<std::mutex> lk(mu);
            cv.wait(lk, [&] { return ready < 0 || ready > t; });
            ok = ready > t;
        }
        if (ok)
            for (int sg = seg0[(size_t)t]; sg < nseg && first[(size_t)sg] < p1; ++sg) {
                long long a, b;
                share(sg, a, b);
                int64_t *o = outs[(size_t)sg];
                if (b <= a || !o) continue;
                // (a small result stays in the cache for its reader)
                if (parts == 1) std::memcpy(o + 2 * (a - first[(size_t)sg]), host + 2 * a, (size_t)(b - a) * 16);
                else copy_nt(o + 2 * (a - first[(size_t)sg]), host + 2 * a, (size_t)(b - a) * 16);
            }
    };
    std::vector<std::thread> th;
    if (parts > 1)
        for (int t = 0; t < parts; ++t) th.emplace_back(part_work, t);
    // this thread waits for the downloads in order and releases the parts
    for (int t = 0; parts > 1 && t < parts && err.ok(); ++t) {
        if (ev[(size_t)t] && cudaEventSynchronize(ev[(size_t)t]) != cudaSuccess) {
            err = Status::Err(DRESSX_ECUDA, "histogram download failed");
        } else {
            std::lock_guard<std::mutex> lk(mu);
            ready = t + 1;
            cv.notify_all();
        }
    }
    if (!err.ok()) {
        std::lock_guard<std::mutex> lk(mu);
        ready = -1;
        cv.notify_all();
    }
    if (parts == 1) part_work(0);
    for (auto &t : th) t.join();
    for (cudaEvent_t e : ev)
        if (e) cudaEventDestroy(e);
    if (err.ok() && nomem) err = Status::Err(DRESSX_ENOMEM, "host allocation of the histograms failed");
    if (!err.ok()) {
        for (auto &o : outs) std::free(o);
        outs.assign((size_t)nseg, nullptr);
    }
    return err;
}

Status histogram_download(HistResult &res, std::vector<std::vector<long long>> &out, cudaStream_t st)
{
    out.assign((size_t)res.nseg, std::vector<long long>());
    const long long R = res.R;
    if (R == 0) return Status::Ok();
    std::vector<long long> pairs(2 * (size_t)R);
    DRESS_CUDA_TRY(counted_memcpy(pairs.data(), res.pairs.get(), 2 * (size_t)R * sizeof(long long),
                                   cudaMemcpyDeviceToHost, st));
    DRESS_CUDA_TRY(cudaStreamSynchronize(st));
    for (int sg = 0; sg < res.nseg; ++sg)
        out[(size_t)sg].assign(pairs.begin() + 2 * res.seg_runs[(size_t)sg], pairs.begin() + 2 * res.seg_runs[(size_t)sg + 1]);
    return Status::Ok();
}

Status histogram_segments(unsigned long long *keys, unsigned long long *alt, const std::vector<long long> &begin,
                          const std::vector<long long> &len, std::vector<std::vector<long long>> &out,
                          cudaStream_t st)
{
    HistResult res;
    DRESS_TRY(histogram_device(keys, alt, begin, len, res, st));
    return histogram_download(res, out, st);
}

}  // namespace dress

// ---------------------------------------------------------------------------
// Histogram without any allocation (dressx_histogram_noalloc)
//
// Some callers cannot allocate device memory at the moment they need a
// histogram: code running while a CUDA graph is being captured, frameworks
// whose caching allocator owns all device memory, or real-time loops that
// forbid allocation after start-up.  For them the pipeline above runs on one
// segment of at most NOALLOC_MAX values with every scratch buffer carved out
// of the file-scope array below.  Every GPU that loads this library holds the
// array (about 16 MiB) until the process exits.  The call only enqueues work
// on the caller's stream (no host synchronisation), so results are ready when the stream reaches that point.  All
// calls share the one array: calls whose work overlaps on the GPU race.
// ---------------------------------------------------------------------------
namespace dress {
namespace {

constexpr long long NOALLOC_MAX = DRESSX_NOALLOC_MAX_VALUES;
constexpr int NA_BUCKETS = 512;                                     // split_buckets(NOALLOC_MAX)
constexpr int NA_TILES = (int)(NOALLOC_MAX / SPLIT_TILE);
static_assert(NOALLOC_MAX % SPLIT_TILE == 0 && NOALLOC_MAX <= 3072LL * NA_BUCKETS, "whole tiles and buckets");

// byte offsets of the carved buffers
constexpr long long NA_A = 0;                                       // u64 keys, then run values
constexpr long long NA_B = NA_A + 8 * NOALLOC_MAX;                  // u16 bucket ids, then u64 run counts
constexpr long long NA_BK = NA_B + 8 * NOALLOC_MAX;                 // Bucket [buckets]
constexpr long long NA_TILESB = NA_BK + 32LL * NA_BUCKETS;          // Tile [tiles]
constexpr long long NA_SPLIT = NA_TILESB + 32LL * NA_TILES;         // u64 [buckets]
constexpr long long NA_COUNTS = NA_SPLIT + 8LL * NA_BUCKETS;        // u32 [2 buckets]
constexpr long long NA_RUNS = NA_COUNTS + 8LL * NA_BUCKETS;         // u32 [buckets]
constexpr long long NA_BASE = NA_RUNS + 4LL * NA_BUCKETS;           // i64 [buckets+1]
constexpr long long NA_SEG = NA_BASE + 8LL * (NA_BUCKETS + 1) + 8;  // LongSeg, i64 [2], i32 [2], i32
constexpr long long NA_BYTES = NA_SEG + 128;
static_assert(sizeof(Tile) <= 32 && sizeof(Bucket) <= 32 && sizeof(LongSeg) <= 64 && NA_SEG % 16 == 0, "descriptor slots");

static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_BYTES];

// single segment [0, n) of nb buckets (one: a short segment)
__global__ void k_na_setup(long long n, int nb, int nt, Bucket *bk, Tile *tiles, LongSeg *seg, int *seg_bk,
                           unsigned *counts)
{
    for (int t = threadIdx.x; t < nt; t += blockDim.x) {
        const long long b = (long long)t * SPLIT_TILE;
        tiles[t].begin = b;
        tiles[t].end = b + SPLIT_TILE < n ? b + SPLIT_TILE : n;
        tiles[t].seg = 0;
    }
    for (int j = threadIdx.x; j < 2 * nb; j += blockDim.x) counts[j] = 0;
    if (threadIdx.x == 0) {
        if (nb == 1) bk[0] = {0, (unsigned)n, 0u, 1, 0};
        *seg = {0, n, 0, nb, 0, 0};
        seg_bk[0] = 0;
        seg_bk[1] = nb;
    }
}

}  // namespace
}  // namespace dress

namespace dress {
namespace {

constexpr int NA_MAX_DEVICES = 128;
std::mutex g_na_mu;
unsigned char *g_na_base[NA_MAX_DEVICES];      // device address of the array, per device

// The array's name is a host-side stand-in in host code; its device address
// comes from cudaGetSymbolAddress with the device current.  Outside stream
// capture every call looks it up afresh (a cudaDeviceReset or another
// context made current then cannot leave a stale address behind); while
// `st` is being captured the address of the device's last call outside
// capture is used, so the first call on a device must come before any
// capture.
cudaError_t noalloc_scratch(cudaStream_t st, unsigned char **out, bool *fresh)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= NA_MAX_DEVICES) return cudaErrorInvalidDevice;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) {
        cudaGetLastError();
        cs = cudaStreamCaptureStatusActive;
    }
    std::lock_guard<std::mutex> lk(g_na_mu);
    *fresh = cs == cudaStreamCaptureStatusNone || !g_na_base[dev];
    if (*fresh) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_na_base[dev] = (unsigned char *)p;
    }
    *out = g_na_base[dev];
    return cudaSuccess;
}

}  // namespace
}  // namespace dress

extern "C" int dressx_histogram_noalloc(const double *values, int64_t n, int64_t *pairs, int64_t *num_runs,
                                        void *stream)
{
    using namespace dress;
    if (n < 0 || (n > 0 && (!values || !pairs)) || !num_runs) {
        std::fprintf(stderr, "dress_b200: dressx_histogram_noalloc: bad arguments\n");
        return DRESSX_EINVAL;
    }
    if (n > NOALLOC_MAX) {
        std::fprintf(stderr, "dress_b200: dressx_histogram_noalloc: %lld values exceed the maximum of %lld\n",
                     (long long)n, (long long)NOALLOC_MAX);
        return DRESSX_EUNSUPPORTED;
    }
    cudaStream_t st = (cudaStream_t)stream;
    unsigned char *base = nullptr;
    bool fresh = true;                                // the kernels' attributes too are set afresh
    cudaError_t e = noalloc_scratch(st, &base, &fresh);
    if (e != cudaSuccess) {
        std::fprintf(stderr, "dress_b200: dressx_histogram_noalloc: scratch address: %s\n", cudaGetErrorString(e));
        return DRESSX_ECUDA;
    }
    if (n == 0) {
        e = cudaMemsetAsync(num_runs, 0, sizeof(int64_t), st);
        return e == cudaSuccess ? DRESSX_OK : DRESSX_ECUDA;
    }
    // every scratch word read below is written first in this call, so the
    // array needs no clearing between calls
    const int nb = n <= BUCKET_CAP ? 1 : split_buckets(n);
    const int nt = n <= BUCKET_CAP ? 0 : (int)((n + SPLIT_TILE - 1) / SPLIT_TILE);
    unsigned char *tail = base + NA_SEG;
    HistLaunch h{};
    h.nseg = 1;
    h.nbk = nb;
    h.nlong = n > BUCKET_CAP;
    h.ntiles = nt;
    h.max_nb = nb;
    h.src = (const unsigned long long *)values;
    h.A = (unsigned long long *)(base + NA_A);
    h.B = (unsigned long long *)(base + NA_B);
    h.bk = (Bucket *)(base + NA_BK);
    h.segs = (const LongSeg *)tail;
    h.tiles = (const Tile *)(base + NA_TILESB);
    h.seg_runs = (long long *)(tail + 64);
    h.seg_bk = (const int *)(tail + 80);
    h.nsplit = (int *)(tail + 88);
    h.split = (unsigned long long *)(base + NA_SPLIT);
    h.counts = (unsigned *)(base + NA_COUNTS);
    h.ids = (unsigned short *)(base + NA_B);          // read for the last time before the counts are written
    h.runs = (unsigned *)(base + NA_RUNS);
    h.base = (long long *)(base + NA_BASE);
    count_launch(), k_na_setup<<<1, 256, 0, st>>>(n, nb, nt, h.bk, (Tile *)h.tiles, (LongSeg *)h.segs, (int *)h.seg_bk,
                                                  h.counts);
    Status s = launch_hist_runs(h, st, fresh);
    if (s.ok()) s = launch_hist_pairs(h, (long long *)pairs, st, (long long *)num_runs);
    if (!s.ok()) {
        std::fprintf(stderr, "dress_b200: dressx_histogram_noalloc: launch: %s\n", s.msg.c_str());
        return DRESSX_ECUDA;
    }
    return DRESSX_OK;
}
