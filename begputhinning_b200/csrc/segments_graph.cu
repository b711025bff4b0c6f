// segments_graph.cu -- ExtractSegmentsV as one cooperative launch
// (2D/ExtractSegments.cpp:16-127, 3D/ExtractSegments.cpp:135-251), bit-exact
// in content and order, with no sequential part left.
//
// The reference visits the nodes (points without exactly two foreground
// neighbours) in raster order; a visit walks -v branches, each along a run of
// two-neighbour points (a chain) or one step to a neighbouring node, zeroes
// what it walks over and adds 1 to the value of the node it ends at.  Two
// facts make every node's output independent of the others' visits:
//  * an edge (a chain, or two adjacent nodes) is always walked by the node
//    that comes first in raster order.  A node starts with one unit of budget
//    per neighbour; each earlier neighbour's walk takes exactly one of them
//    and exactly one of its edges, so at its visit the budget equals the
//    edges that are left, and all of them are walked;
//  * hence the arrivals at a node before its visit are its edges to earlier
//    nodes, and its segments, in the scan order of its neighbours, are its
//    edges to later nodes, chains that lead nowhere, and chains back to
//    itself, followed by one single-point segment per unit of budget left
//    over (neighbours on the frame, an isolated point).
// A walk that meets no nonzero point stays where it is and ends on the same
// point again: at the end of a chain that leads to the frame, and at the far
// end of a chain back to its own node, whose far end then counts as one more
// (two-point) segment of that node.  tests/test_segment_edges.py checks this
// closed form against the oracle on thinned and on raw masks.
//
// What is left is list ranking: every chain point has to know the two ends
// of its chain and its distance to them.  Each chain point is two half-edges
// (leaving it through its first or second neighbour); pointer jumping over
// the half-edges takes at most log5(longest chain) rounds, after which every
// point writes its own coordinates at its place in the output.  Phases (grid
// barriers in between):
//   A  node and chain masks per packed word (bit-sliced neighbour counts)
//   B  block prefix sums -> raster-ordered node and chain lists
//   C  half-edges: successor or, next to a node or the frame, terminal
//   J  pointer jumping until no half-edge finishes any more (the rest are
//      cycles without a node, which the reference never walks)
//   D  segments and points per node;  E  prefix sums, node outputs
//   F  chain points write their coordinates
//   G, H (CenterlineExtraction only) pruning, smoothing and flattening
//      (2D/CenterlineExtraction.cpp:51-131, 3D/CenterlineExtraction.cpp:56-144),
//      so the whole path needs one readback and no count on the host
//
// Bound: latency -- about 7 + log5(longest chain) grid barriers of 1-2 us and
// as many chains of dependent loads.  Measured on a B200, this kernel alone:
// 2048^2 stroke image (214 k points) 62 us, 256^3 volume (3.9 k points) 47 us
// (84 and 57 us with one half-edge, one node and one strided word per thread at
// a time).  Against a walk that followed each chain with one thread and ran the
// nodes from a queue in the order of their dependences, whole ExtractSegmentsV
// calls: 5.72 -> 0.29 ms and 0.86 -> 0.10 ms.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "host.h"
#include "kernels.cuh"

namespace bgt {

namespace {
constexpr int kSegThreads = 512;
constexpr int kSegWarps = kSegThreads / 32;
constexpr uint32_t kFin = 0x80000000u;      // half-edge pair: the pointer is a terminal half-edge
constexpr uint32_t kNone = 0xffffffffu;     // no exit node / not walked from this end
constexpr int kMaxRounds = 64;
constexpr size_t kSegHeaderBytes = 64;
// sync block: [0] barrier arrivals, [1] status, then per jump round: finished, left over
constexpr int kSyncInts = 2 + 2 * kMaxRounds;

__host__ __device__ inline size_t seg_up16(size_t v) { return (v + 15) & ~size_t(15); }

// Output block: header, start[S + 1], is_end[S], x[N], y[N], z[N].
struct SegLayout {
    size_t start, is_end, x, y, z, total;
};
__host__ __device__ inline SegLayout seg_layout(unsigned S, unsigned N, int dims)
{
    SegLayout L;
    L.start = kSegHeaderBytes;
    L.is_end = L.start + seg_up16((size_t)(S + 1) * 4);
    L.x = L.is_end + seg_up16(S);
    L.y = L.x + seg_up16((size_t)N * 2);
    L.z = L.y + seg_up16((size_t)N * 2);
    L.total = L.z + (dims == 3 ? seg_up16((size_t)N * 2) : 0);
    return L;
}

// Output block of the centreline tail: header, I[nsegs + 1], X[N], Y[N], Z[N].
struct TailLayout {
    size_t idx, x, y, z, total;
};
__host__ __device__ inline TailLayout tail_layout(unsigned S, unsigned N, int dims)
{
    TailLayout L;
    L.idx = kSegHeaderBytes;
    L.x = L.idx + seg_up16((size_t)(S + 1) * 4);
    L.y = L.x + seg_up16((size_t)N * 4);
    L.z = L.y + seg_up16((size_t)N * 4);
    L.total = L.z + (dims == 3 ? seg_up16((size_t)N * 4) : 0);
    return L;
}

struct SegArgs {
    const uint32_t *buf;  // packed image, P words per row
    int W, H, D, P;
    uint32_t ww, nw;      // used words per row, used words in all
    FastDiv dww, dH;
    uint4 *rec;           // per used word with foreground: node mask, chain mask, node rank, chain index
    // chain points
    uint2 *cpt;           // row, x
    uint16_t *cdir;       // its two neighbours (window cells): low | high << 8
    unsigned long long *pair;  // per half-edge: steps << 32 | kFin? | half-edge reached
    uint32_t *cexit;      // terminal half-edge -> rank of its node (kNone: the chain leads nowhere)
    uint32_t *cbase;      // terminal half-edge -> output index of the chain's first point walked from its node
    uint32_t cap_c;
    // nodes
    uint2 *npt;           // row, x
    uint8_t *ndeg;        // foreground neighbours
    uint2 *ncnt;          // segments, points
    uint32_t cap_n;
    uint2 *bsum, *bsum2, *bsum3;  // per block: nodes and chain points; segments and points; kept ones
    int *sync;
    uint8_t *out;
    unsigned long long out_bytes;
    long long timeout_ns;
    // centreline tail
    uint32_t *keep;       // segment -> its first output point, kNone: pruned
    uint32_t cap_s;       // segments it holds
    uint8_t *tail;
    unsigned long long tail_bytes, maxlen;
    int span;
    const int *check[2];  // status words of the kernels before this one (or null)
};

// Header of the output blocks.
struct SegHeader {
    uint32_t nodes, chains, segs, pts;
    int status;   // 0 done, 1 lists too small, 2 output too small, 4 a wait ran out, 8 sums past 32 bits
    int checked;  // the status words, OR-ed
    uint32_t kept, kept_pts;
};

// Grid barrier (cooperative launch: every block is resident).  Bounded; false
// once any block gave up (bit 30 of the arrivals, which ends every wait).  One
// word says all, so that a block that arrives last reads once (a status word
// of its own, read behind the wait: CenterlineExtraction of a 512^2 image 152 us
// instead of 148, segments of a 256^3 volume 96.1 instead of 95.6).
__device__ bool seg_barrier(const SegArgs &a, unsigned &gen)
{
    constexpr int kGaveUp = 1 << 30;
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        gen++;
        __threadfence();
        atomicAdd(a.sync, 1);
        const int target = (int)(gen * gridDim.x);
        const unsigned long long t_end = globaltimer() + (unsigned long long)a.timeout_ns;
        int v = ld_acquire(a.sync);
        for (int spin = 0; v < target; v = ld_acquire(a.sync), spin++)
            if ((spin & 255) == 255 && globaltimer() > t_end) {
                atomicOr(a.sync, kGaveUp);
                atomicOr(&reinterpret_cast<SegHeader *>(a.tail ? a.tail : a.out)->status, 4);
                v = kGaveUp;
                break;
            }
        ok = !(v & kGaveUp);
    }
    __syncthreads();
    return ok;  // (thread 0 writes it again behind the next barrier's first __syncthreads)
}

// Exclusive prefix sum over the block of two counters packed in 64 bits.
__device__ unsigned long long seg_exscan(unsigned long long v, unsigned long long *total)
{
    __shared__ unsigned long long wsum[kSegWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    unsigned long long before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kSegWarps; w++) {
        const unsigned long long s = wsum[w];
        if (w < warp) before += s;
        all += s;
    }
    __syncthreads();
    *total = all;
    return before + x - v;
}

// Sums of the per-block totals before this block, and of all blocks.
__device__ void seg_block_prefix(const uint2 *sums, unsigned long long (&before)[2], unsigned long long (&all)[2])
{
    __shared__ unsigned long long part[kSegWarps][4];
    unsigned long long v[4] = {0, 0, 0, 0};
    for (unsigned k = threadIdx.x; k < gridDim.x; k += kSegThreads) {
        const uint2 u = __ldcg(sums + k);
        v[2] += u.x;
        v[3] += u.y;
        if (k < blockIdx.x) {
            v[0] += u.x;
            v[1] += u.y;
        }
    }
    const int warps = min(kSegWarps, (int)(gridDim.x + 31) >> 5);  // warps that hold any
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < warps) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] += __shfl_xor_sync(kFull, v[i], o);
        if (lane < 4) part[warp][lane] = lane == 0 ? v[0] : lane == 1 ? v[1] : lane == 2 ? v[2] : v[3];
    }
    __syncthreads();
    before[0] = before[1] = all[0] = all[1] = 0;
    for (int w = 0; w < warps; w++) {
        before[0] += part[w][0];
        before[1] += part[w][1];
        all[0] += part[w][2];
        all[1] += part[w][3];
    }
    __syncthreads();
}

template <int DIMS>
struct Win {
    static constexpr int C = DIMS == 2 ? 4 : 13;  // centre cell; a cell before it precedes the point in raster order
};

// Foreground bits of the 3x3 (x3) window of the interior point (row, x),
// cells in the reference's scan order, the centre cleared.
template <int DIMS>
__device__ __forceinline__ uint32_t seg_window(const SegArgs &a, uint32_t row, uint32_t x)
{
    const uint32_t j0 = (x - 1) >> 5, j1 = (x + 1) >> 5, sh = (x - 1) & 31u;
    uint32_t w = 0;
#pragma unroll
    for (int k = 0; k < (DIMS == 2 ? 3 : 9); k++) {
        const int dz = DIMS == 2 ? 0 : k / 3 - 1, dy = DIMS == 2 ? k - 1 : k % 3 - 1;
        const uint32_t *p = a.buf + (size_t)((long long)row + (long long)dz * a.H + dy) * a.P;
        w |= (__funnelshift_r(__ldg(p + j0), __ldg(p + j1), sh) & 7u) << (3 * k);
    }
    return w & ~(1u << Win<DIMS>::C);
}

// Cells of the window that are interior (points when they are foreground).
template <int DIMS>
__device__ __forceinline__ uint32_t seg_interior(const SegArgs &a, uint32_t row, uint32_t x)
{
    constexpr uint32_t all = DIMS == 2 ? 0x1FFu : 0x7FFFFFFu;
    constexpr uint32_t xl = DIMS == 2 ? 0x49u : 0x1249249u, yl = DIMS == 2 ? 0x7u : 0x1C0E07u;
    uint32_t y = row, m = all;
    if (DIMS == 3) {
        const uint32_t z = fdiv(a.dH, row);
        y = row - z * (uint32_t)a.H;
        if (z == 1) m &= ~0x1FFu;
        if (z + 2 == (uint32_t)a.D) m &= ~(0x1FFu << 18);
    }
    if (x == 1) m &= ~xl;
    if (x + 2 == (uint32_t)a.W) m &= ~(xl << 2);
    if (y == 1) m &= ~yl;
    if (y + 2 == (uint32_t)a.H) m &= ~(yl << 6);
    return m;
}

// The point in window cell q of (row, x): true for a node (id = its rank),
// false for a chain point (id = its index).
__device__ __forceinline__ bool seg_point(const SegArgs &a, uint32_t row, uint32_t x, int q, uint32_t &id)
{
    const int dz = q / 9, dy = (q / 3) % 3, dx = q % 3;  // 2D callers add 9 (the middle plane)
    const uint32_t r = (uint32_t)((long long)row + (long long)(dz - 1) * a.H + (dy - 1));
    const uint32_t xx = x + (uint32_t)dx - 1u;
    const uint4 w = __ldcg(a.rec + (size_t)r * a.ww + (xx >> 5));
    const uint32_t b = 1u << (xx & 31u);
    const bool node = (w.x & b) != 0u;
    id = node ? w.z + __popc(w.x & (b - 1u)) : w.w + __popc(w.y & (b - 1u));
    return node;
}

// Phases A and B: masks, counts, lists.
template <int DIMS>
__device__ __forceinline__ void seg_masks(const SegArgs &a, uint32_t i, uint32_t c, uint32_t &nodes, uint32_t &chains)
{
    const uint32_t row = fdiv(a.dww, i), j = i - row * a.ww;
    uint32_t y = row, z = 0;
    if (DIMS == 3) {
        z = fdiv(a.dH, row);
        y = row - z * (uint32_t)a.H;
    }
    nodes = chains = 0;
    if (y == 0 || y + 1 >= (uint32_t)a.H || (DIMS == 3 && (z == 0 || z + 1 >= (uint32_t)a.D))) return;
    uint32_t pts = c;
    if (j == 0) pts &= ~1u;
    const int last = a.W - 2 - (int)(j * 32);  // highest interior bit of the word
    if (last < 0) return;
    if (last < 31) pts &= (2u << last) - 1u;
    if (!pts) return;
    // counts modulo 2, and "at least two", "at least four": exactly two = the second and neither of the others
    uint32_t c0 = 0, c1 = 0, big = 0;
    auto add = [&](uint32_t v) {
        const uint32_t t = c0 & v;
        c0 ^= v;
        big |= c1 & t;
        c1 ^= t;
    };
#pragma unroll
    for (int k = 0; k < (DIMS == 2 ? 3 : 9); k++) {
        const int dz = DIMS == 2 ? 0 : k / 3 - 1, dy = DIMS == 2 ? k - 1 : k % 3 - 1;
        const uint32_t *p = a.buf + (size_t)((long long)row + (long long)dz * a.H + dy) * a.P + j;
        const uint32_t m = __ldg(p), l = j > 0 ? __ldg(p - 1) : 0u, r = j + 1 < a.ww ? __ldg(p + 1) : 0u;
        add(at_xm1(m, l));
        if (dz != 0 || dy != 0) add(m);
        add(at_xp1(m, r));
    }
    const uint32_t two = c1 & ~c0 & ~big;
    nodes = pts & ~two;
    chains = pts & two;
}

// What node r does at its visit, by a group of kSegGroup lanes that take its
// neighbours side by side (a neighbour costs six dependent loads); with EMIT
// its segments and end points are written from segment si and point pi on (and
// the chains it walks learn where their points go), else only counted.  Whole
// warps call it; lanes of groups without a node pass live = false.  Returns
// the node's segments and points in every lane of its group.
template <int DIMS>
struct Group {
    static constexpr int N = DIMS == 2 ? 4 : 8;
};
template <int DIMS, bool EMIT>
__device__ __forceinline__ uint2 seg_visit(const SegArgs &a, bool live, uint32_t r, uint32_t si, uint32_t pi,
                                           int32_t *start, uint8_t *is_end, int16_t *px, int16_t *py, int16_t *pz)
{
    constexpr int C = Win<DIMS>::C, q0 = DIMS == 2 ? 9 : 0, G = Group<DIMS>::N;
    const int g = threadIdx.x & (G - 1);
    const uint2 at = live ? __ldcg(a.npt + r) : make_uint2(0u, 0u);
    const uint32_t win = live ? seg_window<DIMS>(a, at.x, at.y) : 0u;
    uint32_t todo = live ? win & seg_interior<DIMS>(a, at.x, at.y) : 0u;
    const int n = __popc(win);
    const uint32_t pi0 = pi, si0 = si;
    uint32_t arrivals = 0;
    auto put = [&](uint32_t k, uint2 p) {
        uint32_t y = p.x, z = 0;
        if (DIMS == 3) {
            z = fdiv(a.dH, p.x);
            y = p.x - z * (uint32_t)a.H;
            pz[k] = (int16_t)z;
        }
        px[k] = (int16_t)p.y;
        py[k] = (int16_t)y;
    };
    while (__any_sync(kFull, todo != 0u)) {
        // this lane's neighbour: the g-th of those left
        uint32_t m = todo;
        for (int i = 0; i < g; i++) m &= m - 1;
#pragma unroll
        for (int i = 0; i < G; i++) todo &= todo - 1;
        // what it gives: an arrival, or a segment of `len` chain points that ends at `end`
        bool arrival = false, seg = false, end1 = false;
        uint32_t len = 0, home = kNone;  // home: terminal half-edge of this end of the chain
        uint2 end = at;
        bool walked = false;
        if (m) {
            const int q = __ffs(m) - 1;
            uint32_t id;
            if (seg_point(a, at.x, at.y, q + q0, id)) {
                arrival = q < C;
                seg = !arrival;
                if (EMIT && seg) {
                    end = __ldcg(a.npt + id);
                    end1 = __ldcg(a.ndeg + id) < 2;
                }
            } else {
                const int back = 2 * C - q;
                const int sr = (__ldcg(a.cdir + id) & 0xff) == back ? 0 : 1;  // the side of the chain point that r is on
                const unsigned long long pr = __ldcg(a.pair + 2 * (size_t)id + (1 - sr));
                const uint32_t t = (uint32_t)pr & ~kFin;
                const uint32_t e = __ldcg(a.cexit + t);
                home = 2 * id + sr;
                seg = true;
                walked = true;
                len = (uint32_t)(pr >> 32) + 1;
                if (e == kNone) {  // leads to the frame: the last point again
                    if (EMIT) end = __ldcg(a.cpt + (t >> 1));
                } else if (e == r) {
                    const uint16_t fd = __ldcg(a.cdir + (t >> 1));
                    const int far_q = 2 * C - ((t & 1) ? fd >> 8 : fd & 0xff);  // the cell of r that holds the far end
                    walked = q < far_q;
                    if (!walked) len = 0;
                    if (EMIT) end = __ldcg(a.cpt + (walked ? t >> 1 : id));
                } else if (e > r) {
                    if (EMIT) {
                        end = __ldcg(a.npt + e);
                        end1 = __ldcg(a.ndeg + e) < 2;
                    }
                } else {
                    seg = walked = false;
                    arrival = true;
                }
            }
        }
        // places in the order of the neighbours
        uint32_t segs = seg, pts = seg ? len + 2 : 0u;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const uint32_t s1 = __shfl_up_sync(kFull, segs, o, G), p1 = __shfl_up_sync(kFull, pts, o, G);
            if (g >= o) {
                segs += s1;
                pts += p1;
            }
        }
        if (EMIT && m) {
            const uint32_t k = si + segs - 1, p = pi + pts - (len + 2);
            if (home != kNone) a.cbase[home] = walked ? p + 1 : kNone;
            if (seg) {
                start[k] = (int32_t)p;
                is_end[k] = end1 || n < 2;
                put(p, at);
                put(p + 1 + len, end);
            }
        }
        si += __shfl_sync(kFull, segs, G - 1, G);
        pi += __shfl_sync(kFull, pts, G - 1, G);
        const unsigned arr = __ballot_sync(kFull, arrival);
        arrivals += __popc((arr >> (threadIdx.x & 31 & ~(G - 1))) & ((1u << G) - 1u));
    }
    // the rest of the budget: single points
    const int left = live ? max(n, 1) - (int)arrivals - (int)(si - si0) : 0;
    if (EMIT)
        for (int k = g; k < left; k += G) {
            start[si + k] = (int32_t)(pi + k);
            is_end[si + k] = n < 2;
            put(pi + k, at);
        }
    if (!EMIT && live && g == 0) a.ndeg[r] = (uint8_t)n;
    return make_uint2(si - si0 + max(left, 0), pi - pi0 + max(left, 0));
}

// A kept segment's points, smoothed, by one warp.  Point q is the mean of the
// points within min(span, q, n - 1 - q) of it.  The reference keeps a float
// running sum of integer coordinates, which is exact while it stays below
// 2^24 (spans up to kTailSpan: 2 * span + 2 coordinates of 15 bits), so the
// sum is taken as an integer here and the quotient is the same.
constexpr int kTailSpan = 255;
template <int DIMS>
__device__ __forceinline__ void tail_segment(const SegArgs &a, const int16_t *px, const int16_t *py, const int16_t *pz,
                                             int first, int n, uint32_t to, float *X, float *Y, float *Z)
{
    const int span = min(a.span, (n - 1) / 2);
    for (int q = threadIdx.x & 31; q < n; q += 32) {
        const int h = min(span, min(q, n - 1 - q));
        int x = 0, y = 0, z = 0;
        for (int k = first + q - h; k <= first + q + h; k++) {
            x += __ldcg(px + k);
            y += __ldcg(py + k);
            if (DIMS == 3) z += __ldcg(pz + k);
        }
        const float c = (float)(2 * h + 1);
        X[to + q] = __fdiv_rn((float)x, c);
        Y[to + q] = __fdiv_rn((float)y, c);
        if (DIMS == 3) Z[to + q] = __fdiv_rn((float)z, c);
    }
}

template <int DIMS, bool TAIL>
__global__ void __launch_bounds__(kSegThreads, 1) segments_graph_kernel(const SegArgs a)
{
    unsigned gen = 0;
    const uint32_t tid = blockIdx.x * kSegThreads + threadIdx.x, nthr = gridDim.x * kSegThreads;
    SegHeader *hdr = reinterpret_cast<SegHeader *>(TAIL ? a.tail : a.out);
    unsigned long long total, before[2], all[2];

    // A: masks and counts of this thread's range of words
    const uint32_t per = (a.nw + nthr - 1) / nthr;
    const uint32_t w0 = min(a.nw, per * tid), w1 = min(a.nw, w0 + per);
    unsigned long long cnt = 0;
    for (uint32_t i = w0; i < w1; i++) {
        const uint32_t row = fdiv(a.dww, i);
        const uint32_t c = __ldg(a.buf + (size_t)row * a.P + (i - row * a.ww));
        if (!c) continue;
        uint32_t nodes, chains;
        seg_masks<DIMS>(a, i, c, nodes, chains);
        a.rec[i] = make_uint4(nodes, chains, 0u, 0u);
        cnt += (unsigned long long)__popc(nodes) << 32 | __popc(chains);
    }
    const unsigned long long mine = seg_exscan(cnt, &total);
    if (threadIdx.x == 0) a.bsum[blockIdx.x] = make_uint2((uint32_t)(total >> 32), (uint32_t)total);
    if (!seg_barrier(a, gen)) return;

    // B: lists in raster order
    seg_block_prefix(a.bsum, before, all);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        hdr->nodes = (uint32_t)min(all[0], (unsigned long long)kNone);
        hdr->chains = (uint32_t)min(all[1], (unsigned long long)kNone);
        hdr->checked = (a.check[0] ? __ldcg(a.check[0]) : 0) | (a.check[1] ? __ldcg(a.check[1]) : 0);
        if (all[0] > a.cap_n || all[1] > a.cap_c) atomicOr(&hdr->status, 1);
    }
    if (all[0] > a.cap_n || all[1] > a.cap_c) return;
    const uint32_t nn = (uint32_t)all[0], nc = (uint32_t)all[1];
    if (cnt) {
        uint32_t ni = (uint32_t)before[0] + (uint32_t)(mine >> 32), ci = (uint32_t)before[1] + (uint32_t)mine;
        for (uint32_t i = w0; i < w1; i++) {
            const uint32_t row = fdiv(a.dww, i);
            if (!__ldg(a.buf + (size_t)row * a.P + (i - row * a.ww))) continue;
            const uint4 rc = a.rec[i];  // written by this thread
            if (!(rc.x | rc.y)) continue;
            a.rec[i] = make_uint4(rc.x, rc.y, ni, ci);
            const uint32_t x0 = (i - row * a.ww) * 32;
            for (uint32_t m = rc.x; m; m &= m - 1) a.npt[ni++] = make_uint2(row, x0 + __ffs(m) - 1);
            for (uint32_t m = rc.y; m; m &= m - 1) a.cpt[ci++] = make_uint2(row, x0 + __ffs(m) - 1);
        }
    }
    if (!seg_barrier(a, gen)) return;

    // C: half-edges
    constexpr int C = Win<DIMS>::C, q0 = DIMS == 2 ? 9 : 0;
    for (uint32_t k = tid; k < nc; k += nthr) {
        const uint2 at = __ldcg(a.cpt + k);
        const uint32_t win = seg_window<DIMS>(a, at.x, at.y), in = seg_interior<DIMS>(a, at.x, at.y);
        const int q2[2] = {__ffs(win) - 1, 31 - __clz(win)};
        a.cdir[k] = (uint16_t)(q2[0] | q2[1] << 8);
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const int q = q2[s];
            const uint32_t h = 2 * k + s;
            uint32_t id = kNone;
            const bool inner = (in >> q) & 1u;
            if (!inner || seg_point(a, at.x, at.y, q + q0, id)) {
                a.pair[h] = kFin | h;
                a.cexit[h] = id;
                a.cbase[h] = kNone;
                continue;
            }
            // the neighbour's side that does not lead back here
            const int qq = q + q0;
            const uint32_t r = (uint32_t)((long long)at.x + (long long)(qq / 9 - 1) * a.H + ((qq / 3) % 3 - 1));
            const uint32_t nwin = seg_window<DIMS>(a, r, at.y + (uint32_t)(qq % 3) - 1u);
            const uint32_t s2 = (__ffs(nwin) - 1) == 2 * C - q ? 1u : 0u;
            a.pair[h] = 1ull << 32 | (2 * id + s2);
        }
    }
    if (!seg_barrier(a, gen)) return;

    // J: pointer jumping.  Pairs are read and written whole (8 bytes), so a
    // reader sees an older or a newer pair, both true.  Of the half-edges of
    // a path that are not finished the one nearest its terminal points at a
    // finished one, so a round in which none finishes leaves only cycles.
    for (int round = 0; round < kMaxRounds; round++) {
        bool fin = false, left = false;
        // several half-edges of a thread at a time, so that their loads overlap
        constexpr int U = 4;
        for (uint32_t h0 = tid; h0 < 2 * nc; h0 += U * nthr) {
            uint32_t p[U], d[U];
            bool open[U];
#pragma unroll
            for (int i = 0; i < U; i++) {
                const uint32_t h = h0 + i * nthr;
                const unsigned long long v = h < 2 * nc ? __ldcg(a.pair + h) : (unsigned long long)kFin;
                p[i] = (uint32_t)v;
                d[i] = (uint32_t)(v >> 32);
                open[i] = !(p[i] & kFin);
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                unsigned long long u[U];
#pragma unroll
                for (int i = 0; i < U; i++) u[i] = p[i] & kFin ? (unsigned long long)p[i] : __ldcg(a.pair + p[i]);
#pragma unroll
                for (int i = 0; i < U; i++) {
                    p[i] = (uint32_t)u[i];
                    d[i] += (uint32_t)(u[i] >> 32);
                }
            }
#pragma unroll
            for (int i = 0; i < U; i++) {
                if (!open[i]) continue;
                __stcg(a.pair + h0 + i * nthr, (unsigned long long)d[i] << 32 | p[i]);
                if (p[i] & kFin) fin = true;
                else left = true;
            }
        }
        const int any_left = __syncthreads_or(left), any_fin = __syncthreads_or(fin);
        if (threadIdx.x == 0) {
            if (any_fin) atomicOr(a.sync + 2 + 2 * round, 1);
            if (any_left) atomicOr(a.sync + 3 + 2 * round, 1);
        }
        if (!seg_barrier(a, gen)) return;
        if (!__ldcg(a.sync + 2 + 2 * round) || !__ldcg(a.sync + 3 + 2 * round)) break;
    }

    // D: segments and points per node (a contiguous range of nodes per block)
    const uint32_t nper = (nn + gridDim.x - 1) / gridDim.x;
    const uint32_t n0 = min(nn, nper * blockIdx.x), n1 = min(nn, n0 + nper);
    constexpr uint32_t G = Group<DIMS>::N;
    const uint32_t group = threadIdx.x / G, groups = kSegThreads / G;
    const bool lead = threadIdx.x % G == 0;
    unsigned long long s0 = 0, s1 = 0;
    for (uint32_t base = n0; base < n1; base += groups) {
        const uint32_t r = base + group;
        const uint2 v = seg_visit<DIMS, false>(a, r < n1, r, 0, 0, nullptr, nullptr, nullptr, nullptr, nullptr);
        if (r < n1 && lead) {
            a.ncnt[r] = v;
            s0 += v.x;
            s1 += v.y;
        }
    }
    seg_exscan(s0, &total);
    s0 = total;
    seg_exscan(s1, &total);
    s1 = total;
    if (threadIdx.x == 0) {
        a.bsum2[blockIdx.x] = make_uint2((uint32_t)s0, (uint32_t)s1);
        if (s0 >> 31 || s1 >> 31) atomicOr(a.sync + 1, 8);
    }
    if (!seg_barrier(a, gen)) return;

    // E: output ranges, node outputs
    seg_block_prefix(a.bsum2, before, all);
    const bool wide = (ld_acquire(a.sync + 1) & 8) || all[0] >> 31 || all[1] >> 31;
    const SegLayout L = seg_layout((unsigned)all[0], (unsigned)all[1], DIMS);
    // (many segments of few points fit the output block, but not `keep`)
    const bool small = L.total > a.out_bytes || (TAIL && all[0] > a.cap_s);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        hdr->segs = (uint32_t)all[0];
        hdr->pts = (uint32_t)all[1];
        if (wide || small) atomicOr(&hdr->status, wide ? 8 : 2);
    }
    if (wide || small) return;
    int32_t *start = reinterpret_cast<int32_t *>(a.out + L.start);
    uint8_t *is_end = a.out + L.is_end;
    int16_t *px = reinterpret_cast<int16_t *>(a.out + L.x), *py = reinterpret_cast<int16_t *>(a.out + L.y),
            *pz = reinterpret_cast<int16_t *>(a.out + L.z);
    if (blockIdx.x == 0 && threadIdx.x == 0) start[all[0]] = (int32_t)all[1];
    uint32_t so = (uint32_t)before[0], po = (uint32_t)before[1];
    for (uint32_t base = n0; base < n1; base += groups) {
        const uint32_t r = base + group;
        const uint2 v = r < n1 && lead ? __ldcg(a.ncnt + r) : make_uint2(0u, 0u);
        unsigned long long o = seg_exscan((unsigned long long)v.x << 32 | v.y, &total);
        o = __shfl_sync(kFull, o, 0, G);  // the group's
        seg_visit<DIMS, true>(a, r < n1, r, so + (uint32_t)(o >> 32), po + (uint32_t)o, start, is_end, px, py, pz);
        so += (uint32_t)(total >> 32);
        po += (uint32_t)total;
    }
    if (!seg_barrier(a, gen)) return;

    // F: chain points
    for (uint32_t k = tid; k < nc; k += nthr) {
        uint32_t pos = kNone;
#pragma unroll
        for (int s = 0; s < 2; s++) {
            const unsigned long long v = __ldcg(a.pair + 2 * (size_t)k + s);
            if (!((uint32_t)v & kFin)) continue;  // a cycle without a node
            const uint32_t b = __ldcg(a.cbase + ((uint32_t)v & ~kFin));
            if (b != kNone) pos = b + (uint32_t)(v >> 32);
        }
        if (pos == kNone) continue;
        const uint2 at = __ldcg(a.cpt + k);
        uint32_t y = at.x;
        if (DIMS == 3) {
            const uint32_t z = fdiv(a.dH, at.x);
            y = at.x - z * (uint32_t)a.H;
            pz[pos] = (int16_t)z;
        }
        px[pos] = (int16_t)at.y;
        py[pos] = (int16_t)y;
    }
    if constexpr (TAIL) {
        if (!seg_barrier(a, gen)) return;
        // G: segments kept (more than maxlen points, or not an end segment)
        const uint32_t S = (uint32_t)all[0];
        const uint32_t sper = (S + gridDim.x - 1) / gridDim.x;
        const uint32_t k0 = min(S, sper * blockIdx.x), k1 = min(S, k0 + sper);
        auto points = [&](uint32_t k) {
            const uint32_t n = (uint32_t)(__ldcg(start + k + 1) - __ldcg(start + k));
            return (unsigned long long)n > a.maxlen || !__ldcg(is_end + k) ? n : 0u;
        };
        unsigned long long kept = 0;
        for (uint32_t k = k0 + threadIdx.x; k < k1; k += kSegThreads) {
            const uint32_t n = points(k);
            kept += n ? 1ull << 32 | n : 0ull;
        }
        seg_exscan(kept, &total);
        if (threadIdx.x == 0) a.bsum3[blockIdx.x] = make_uint2((uint32_t)(total >> 32), (uint32_t)total);
        if (!seg_barrier(a, gen)) return;
        seg_block_prefix(a.bsum3, before, all);
        const TailLayout T = tail_layout((unsigned)all[0], (unsigned)all[1], DIMS);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            hdr->kept = (uint32_t)all[0];
            hdr->kept_pts = (uint32_t)all[1];
            if (T.total > a.tail_bytes) atomicOr(&hdr->status, 2);
        }
        if (T.total > a.tail_bytes) return;
        uint32_t *I = reinterpret_cast<uint32_t *>(a.tail + T.idx);
        float *X = reinterpret_cast<float *>(a.tail + T.x), *Y = reinterpret_cast<float *>(a.tail + T.y),
              *Z = reinterpret_cast<float *>(a.tail + T.z);
        if (blockIdx.x == 0 && threadIdx.x == 0) I[all[0]] = (uint32_t)all[1];
        uint32_t to = (uint32_t)before[0], pt = (uint32_t)before[1];
        for (uint32_t base = k0; base < k1; base += kSegThreads) {
            const uint32_t k = base + threadIdx.x;
            const uint32_t n = k < k1 ? points(k) : 0u;
            const unsigned long long o = seg_exscan(n ? 1ull << 32 | n : 0ull, &total);
            if (k < k1) a.keep[k] = n ? pt + (uint32_t)o : kNone;
            if (n) I[to + (uint32_t)(o >> 32)] = pt + (uint32_t)o;
            to += (uint32_t)(total >> 32);
            pt += (uint32_t)total;
        }
        __syncthreads();
        // H: the block's segments, a warp each
        for (uint32_t k = k0 + (threadIdx.x >> 5); k < k1; k += kSegWarps) {
            const uint32_t p = a.keep[k];
            if (p == kNone) continue;
            const int first = __ldcg(start + k), n = __ldcg(start + k + 1) - first;
            tail_segment<DIMS>(a, px, py, pz, first, n, p, X, Y, Z);
        }
    }
}
}  // namespace

// Device segment extraction of a packed image and, with `tail`, the rest of
// CenterlineExtraction.  Returns BGT_OK with *r filled, 1 when the image is
// beyond this path's index range, or an error.  The lists and the outputs
// live in scratch sized by what the context has met so far; an image that
// needs more reports its counts and is run once more.  The results are read
// back to pinned memory: with the header as much as the last result had, the
// rest, if any, by a second copy.
int segments_graph(bgt_ctx *c, int dims, const uint32_t *d_buf, int W, int H, int D, int P, const SegTail *tail,
                   SegResult *r)
{
    *r = SegResult();
    const long long rows = (long long)H * D, ww = (W + 31) / 32, nw = rows * ww, npx = (long long)W * rows;
    if (nw >= (1LL << 31) || rows >= (1LL << 31) || (tail && tail->span > kTailSpan)) return 1;
    cudaStream_t st = c->stream;
    SegArgs a{};
    a.buf = d_buf;
    a.W = W;
    a.H = H;
    a.D = D;
    a.P = P;
    a.ww = (uint32_t)ww;
    a.nw = (uint32_t)nw;
    a.dww = make_fastdiv((uint32_t)ww);
    a.dH = make_fastdiv((uint32_t)H);
    a.timeout_ns = 2000000000LL;
    // about two words per thread, one block per SM at most (a barrier costs more with more blocks)
    const int grid = (int)std::max<long long>(1, std::min<long long>(c->sms, (nw + 2 * kSegThreads - 1) / (2 * kSegThreads)));
    c->seg_chains = std::max(c->seg_chains, std::max<size_t>(16384, (size_t)npx / (dims == 2 ? 16 : 64)));
    c->seg_nodes = std::max(c->seg_nodes, std::max<size_t>(4096, (size_t)npx / (dims == 2 ? 64 : 256)));
    void *p_rec, *p_out, *p_list, *p_sync, *h_pin;
    int rc;
    if ((rc = ctx_scratch(c, 30, (size_t)nw * sizeof(uint4), &p_rec)) ||
        (rc = ctx_scratch(c, 33, kSyncInts * sizeof(int) + 3 * (size_t)c->sms * sizeof(uint2), &p_sync)))
        return rc;
    a.rec = (uint4 *)p_rec;
    a.sync = (int *)p_sync;
    a.bsum = (uint2 *)((char *)p_sync + kSyncInts * sizeof(int));
    a.bsum2 = a.bsum + c->sms;
    a.bsum3 = a.bsum2 + c->sms;
    size_t out_segs = 0, out_pts = 0;
    for (int attempt = 0; attempt < 5; attempt++) {
        const size_t nc = c->seg_chains, nn = c->seg_nodes;
        if (nc >= (1u << 30) || nn >= (1u << 31)) return 1;
        // points: the chain points and two per segment, about two segments per node
        out_segs = std::max(out_segs, std::min<size_t>(4 * nn, 1u << 30));
        out_pts = std::max(out_pts, std::min<size_t>(nc + 8 * nn, 1u << 30));
        size_t off = 0;
        auto take = [&](size_t bytes) {
            const size_t o = off;
            off += (bytes + 255) / 256 * 256;
            return o;
        };
        const size_t o_cpt = take(nc * 8), o_cdir = take(nc * 2), o_pair = take(nc * 16), o_exit = take(nc * 8),
                     o_base = take(nc * 8), o_npt = take(nn * 8), o_deg = take(nn), o_cnt = take(nn * 8),
                     o_keep = take(tail ? out_segs * 4 : 0);
        if ((rc = ctx_scratch(c, 31, off, &p_list))) return rc;
        char *l = (char *)p_list;
        a.cpt = (uint2 *)(l + o_cpt);
        a.cdir = (uint16_t *)(l + o_cdir);
        a.pair = (unsigned long long *)(l + o_pair);
        a.cexit = (uint32_t *)(l + o_exit);
        a.cbase = (uint32_t *)(l + o_base);
        a.npt = (uint2 *)(l + o_npt);
        a.ndeg = (uint8_t *)(l + o_deg);
        a.ncnt = (uint2 *)(l + o_cnt);
        a.keep = (uint32_t *)(l + o_keep);
        a.cap_s = (uint32_t)out_segs;
        a.cap_c = (uint32_t)nc;
        a.cap_n = (uint32_t)nn;
        a.out_bytes = seg_layout((unsigned)out_segs, (unsigned)out_pts, dims).total;
        if ((rc = ctx_scratch(c, 19, a.out_bytes, &p_out))) return rc;
        a.out = (uint8_t *)p_out;
        uint8_t *block = a.out;
        size_t block_bytes = a.out_bytes;
        if (tail) {
            void *p_tail;
            block_bytes = a.tail_bytes = tail_layout((unsigned)out_segs, (unsigned)out_pts, dims).total;
            if ((rc = ctx_scratch(c, 22, block_bytes, &p_tail))) return rc;
            block = a.tail = (uint8_t *)p_tail;
            a.maxlen = (unsigned long long)(long long)tail->max_segment_length;
            a.span = std::max(0, tail->span);
            a.check[0] = tail->check[0];
            a.check[1] = tail->check[1];
        }
        const size_t first = std::min(block_bytes, std::min<size_t>(std::max<size_t>(c->seg_read, 32 << 10), 2 << 20));
        if ((rc = ctx_pinned(c, first, &h_pin))) return rc;
        cudaError_t e = cudaMemsetAsync(a.sync, 0, kSyncInts * sizeof(int), st);
        if (e == cudaSuccess) e = cudaMemsetAsync(block, 0, sizeof(SegHeader), st);
        if (e != cudaSuccess) return cuda_fail(e, "segment sync reset");
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(kSegThreads);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = dims == 2 ? (tail ? cudaLaunchKernelEx(&cfg, segments_graph_kernel<2, true>, a)
                              : cudaLaunchKernelEx(&cfg, segments_graph_kernel<2, false>, a))
                      : (tail ? cudaLaunchKernelEx(&cfg, segments_graph_kernel<3, true>, a)
                              : cudaLaunchKernelEx(&cfg, segments_graph_kernel<3, false>, a));
        if (e != cudaSuccess) return cuda_fail(e, "segment kernel");
        e = cudaMemcpyAsync(h_pin, block, first, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return cuda_fail(e, "segment extraction");
        const SegHeader h = *(const SegHeader *)h_pin;
        r->checked = h.checked;
        if (h.checked) return BGT_OK;  // the image is not valid: the caller reports why
        if (h.status & 4) return fail(BGT_ERR_TIMEOUT, "segment extraction: a device wait gave up");
        if (h.status & 8) return fail(BGT_ERR_LIMIT, "segment output bound exceeds 2^31 entries");
        if (h.status & 1) {
            c->seg_chains = std::max(c->seg_chains, (size_t)h.chains + h.chains / 8);
            c->seg_nodes = std::max(c->seg_nodes, (size_t)h.nodes + h.nodes / 8);
            continue;
        }
        if (h.status & 2) {
            out_segs = std::max(out_segs, (size_t)h.segs);
            out_pts = std::max(out_pts, (size_t)h.pts);
            continue;
        }
        const SegLayout L = seg_layout(h.segs, h.pts, dims);
        const TailLayout T = tail_layout(h.kept, h.kept_pts, dims);
        const size_t total = tail ? T.total : L.total;
        c->seg_read = total + total / 8;
        if (total > first) {
            if ((rc = ctx_pinned(c, total, &h_pin))) return rc;
            e = cudaMemcpyAsync(h_pin, block, total, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) return cuda_fail(e, "segment readback");
        }
        const char *o = (const char *)h_pin;
        if (tail) {
            r->nseg = (int)h.kept;
            r->npts = (int)h.kept_pts;
            r->idx = (const uint32_t *)(o + T.idx);
            r->fx = (const float *)(o + T.x);
            r->fy = (const float *)(o + T.y);
            r->fz = (const float *)(o + T.z);
            return BGT_OK;
        }
        r->nseg = (int)h.segs;
        r->npts = (int)h.pts;
        r->start = (const int32_t *)(o + L.start);
        r->is_end = (const uint8_t *)(o + L.is_end);
        r->px = (const int16_t *)(o + L.x);
        r->py = (const int16_t *)(o + L.y);
        r->pz = (const int16_t *)(o + L.z);
        DevSegs &d = r->dev;
        d.nseg = r->nseg;
        d.npts = r->npts;
        if (h.segs == 0) return BGT_OK;
        d.start = (int32_t *)(a.out + L.start);
        d.is_end = a.out + L.is_end;
        d.px = (int16_t *)(a.out + L.x);
        d.py = (int16_t *)(a.out + L.y);
        d.pz = dims == 3 ? (int16_t *)(a.out + L.z) : nullptr;
        return BGT_OK;
    }
    return fail(BGT_ERR_NOMEM, "segment extraction: the counts kept growing");
}

}  // namespace bgt
