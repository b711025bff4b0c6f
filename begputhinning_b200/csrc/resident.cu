// resident.cu -- the resident engine: every work item (an instance, or one
// band of rows of a 2D image too large for one CTA) is loaded once into one
// CTA's shared memory and thinned there from its first subiteration to its
// fixed point; only the bands of a large image (every fourth iteration) and
// the slabs of a large volume (every iteration) meet to trade boundary rows
// through global memory.
// One CTA of 768 threads per SM holds up to 225 KB (measured against two
// CTAs of 384 threads with 111 KB each: larger bands and slabs won).
//
// 2D band (dense).  Rows of the band (core plus `halo` rows on each side,
// clamped to the image) lie twice in shared memory (subiteration t reads one
// copy and writes the other) with an odd pitch of 2*ceil(wl/2)+3 words
// (wl = ceil(W/32); a zero word left of every row and zero words right of
// it).  A subiteration hands units (a strip of 32 rows x a chunk of words,
// chunks sized so that there are about two units per warp) to warps
// dynamically; lane = row, walking the chunk in pairs of words: each lane
// loads its own row and the rows above and below straight from shared
// memory and forms the x-neighbours by funnel shifts.  A unit whose 3x3
// neighbourhood of units did not change during the last four subiterations
// -- one of each direction -- is a fixed point for the next one and is
// skipped (a unit processed without a change wrote identical data to both
// copies, so a skipped unit is current in both).  A
// single band stops after four consecutive subiterations without a deletion
// (a fixed point of N, S, E and W: the reference's result, whatever the
// alignment).  Bands of one image run their iterations (N, S, E, W) in
// lockstep, meeting after every kResPassesPerExchange-th one: then a band
// writes its first and last `halo` core rows to global memory, meets the
// other bands at a per-image counter, stops if no band's core changed in
// that iteration, and otherwise reads its halo rows from its neighbours.
// With halo = 4 rows per iteration of the period, wrong values entering at a
// band's outer edge between two meetings (4 rows per iteration at most)
// reach at most its halo rows; if an iteration before the meeting was
// already a fixed point, the one at the meeting is too.
//
// 3D volume (dense boxes, word lists).  A box of the volume (rows x planes,
// full width) lies once in shared memory.  Deletion never adds foreground,
// so the words that are empty at the start are never looked at: each
// iteration goes over the list of the others, keeps the active ones (a word
// next to one that changed in the previous iteration: otherwise its union is
// empty, the argument of the tile engine at word granularity), evaluates the
// pre-test and U on them, one word per thread, and the words with a non-empty
// union are the candidates of the five other subiterations.  A subiteration
// finds its deletions, meets, and applies them, so the state needs no second
// copy.  A large volume is cut into boxes on several CTAs that trade the
// words changed near their edges after every iteration.  A box with more
// non-empty words than the lists hold goes over all of its words instead.
//
// Rules, order of directions and termination are those of the tile engine
// (2D/CUDA_ThinningKernelMultiBlock2D.cuh:104-135,
// 3D/CUDA_ThinningKernel3D_Linear.cuh:746-782); every wait is bounded.
#include <algorithm>

#include "kernels.cuh"
#include "pixels.cuh"
#include "rules.cuh"
#include "tiles.cuh"

namespace bgt {

namespace {
constexpr int kWarps = kResThreads / 32;
constexpr int kSmemBytes = kResSmemBytes;  // dynamic shared memory per CTA

__host__ __device__ inline size_t up16(size_t v) { return (v + 15) & ~size_t(15); }
}  // namespace

// ------------------------------------------------------------ geometry ----
#ifndef BGT_RES_LANE_ROWS
#define BGT_RES_LANE_ROWS 1
#endif
constexpr int kLaneRows = BGT_RES_LANE_ROWS;  // rows of a 2D unit per lane (1 or 2)
constexpr int kUnitRowsH = 32 * kLaneRows - 8, kUnitWordsH = 8;  // 2D unit (see the 2D section)

// words of shared memory a 2D band of nrows rows needs: zero row, two row
// copies and the activity record of its units
__host__ __device__ inline size_t res_words2d(int W, int nrows)
{
    const int wl = (W + 31) >> 5;
    const int nch = (wl + kUnitWordsH - 1) / kUnitWordsH;
    const int pp = (nch * kUnitWordsH + 2) | 1;
    const int ns = (nrows + kUnitRowsH - 1) / kUnitRowsH;
    return (size_t)pp * (1 + 2 * (size_t)nrows) + (size_t)ns * nch;
}

// bytes of shared memory a box of ny x nz rows of wl words (halo included)
// needs: its state, the rows' masks and, in the dense form, two more words
// per word (the lists take what they find there, up to 44% non-empty words)
constexpr size_t kBoxListBytes = 4 + 4 + 4 + 4 + 2;  // list, candidate, union, deletions, active list
__host__ __device__ inline size_t res_bytes3d(int wl, int ny, int nz)
{
    const size_t rows2 = (size_t)(ny + 2) * (nz + 2), words = rows2 * (wl + 1) + 1;
    return up16(words * 4) + 2 * up16(rows2 * 4) + 2 * words * 4 + 80;
}

int res_smem_bytes() { return kSmemBytes; }

int res_rows_fit2d(int W)
{
    int lo = 0, hi = 32767;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (res_words2d(W, mid) * 4 <= (size_t)kSmemBytes) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

bool res_fits3d(int W, int ny, int nz)
{
    const int wl = (W + 31) / 32;
    // words are indexed by 16 bits
    return (long long)(ny + 2) * (nz + 2) * (wl + 1) < 65535 && res_bytes3d(wl, ny, nz) <= (size_t)kSmemBytes;
}

// ------------------------------------------------------------ helpers -----
// The CTAs of one instance meet for the k-th time: each adds 1 to the low half
// of meet[k & 1], and 1 to its high half when something of its own changed
// since the last meeting; the wait (bounded) ends when all `bands` arrived.
// Two words in turn, so that a CTA that is already at the next meeting leaves
// what a late one reads here alone (it cannot get to the one after that).
// One thread per CTA calls it, after a __syncthreads that follows the CTA's
// writes to global memory.  Returns 0 when nobody changed anything, 1 when
// somebody did, 2 when the wait ran out.
struct MeetState {
    unsigned k = 0, seen0 = 0, seen1 = 0;  // meetings so far, high halves after the last one of either word
};
__device__ __forceinline__ int res_meet(unsigned long long *meet, unsigned bands, bool changed, MeetState &m,
                                        long long timeout_ns)
{
    unsigned long long *w = meet + (m.k & 1);
    const unsigned arrivals = bands * (m.k / 2 + 1);
    __threadfence();
    atomicAdd(w, changed ? (1ull << 32) + 1ull : 1ull);
    const unsigned long long t_end = globaltimer() + (unsigned long long)timeout_ns;
    for (int spin = 0;; spin++) {
        const unsigned long long v = ld_acquire64(w);
        if ((unsigned)v >= arrivals) {
            const unsigned n = (unsigned)(v >> 32);
            const bool some = n != ((m.k & 1) ? m.seen1 : m.seen0);
            if (m.k & 1) m.seen1 = n;
            else m.seen0 = n;
            m.k++;
            return some ? 1 : 0;
        }
        if ((spin & 63) == 63 && globaltimer() > t_end) return 2;
        if (spin >= 4096) __nanosleep(64);  // partners that have not started yet
    }
}

// Next work unit of a subiteration for this warp (dynamic distribution over
// the CTA's warps): lane 0 takes a ticket of counter `c`.
__device__ __forceinline__ int res_take(int *c)
{
    int k = 0;
    if ((threadIdx.x & 31) == 0) k = atomicAdd(c, 1);
    return __shfl_sync(kFull, k, 0);
}

// Positions of the words of an ny x nz grid of rows of wl words, in raster
// order, for a thread that takes every kResThreads-th one.
struct WordPos {
    int x, y, z;
};
struct WordWalk {
    int wl, ny, dx, dy, dz;
    __device__ __forceinline__ WordWalk(int wl_, int ny_) : wl(wl_), ny(ny_)
    {
        const int q = kResThreads / wl;
        dx = kResThreads - q * wl;
        dz = q / ny;
        dy = q - dz * ny;
    }
    __device__ __forceinline__ WordPos first() const
    {
        const int r = (int)threadIdx.x / wl;
        return WordPos{(int)threadIdx.x - r * wl, r % ny, r / ny};
    }
    __device__ __forceinline__ void next(WordPos &q) const
    {
        q.x += dx;
        q.y += dy;
        q.z += dz;
        if (q.x >= wl) {
            q.x -= wl;
            q.y++;
        }
        if (q.y >= ny) {
            q.y -= ny;
            q.z++;
        }
    }
};

// Where an instance's words come from and go to: its pixels, or (pix false)
// its packed buffer.
struct ResIO {
    const IODesc *d;
    bool pix;
};

// put(pos, word) for every word of the grid of rows whose first pixel row and
// plane are y0, z0 (warps stay together: put may hold warp-wide votes; `live`
// is false for lanes past the end, whose word is 0).  U words of a thread are
// in flight at once: at 768 threads and 48 bytes per word of one-byte pixels,
// two cover the latency of HBM.
template <int U, class Fetch, class Put>
__device__ __forceinline__ void res_load_loop(const WordWalk &walk, int n, Fetch fetch, Put put)
{
    const int lane = threadIdx.x & 31;
    WordPos q = walk.first();
    for (int i = threadIdx.x; i - lane < n; i += U * kResThreads) {
        uint32_t v[U];
        WordPos at[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
            at[k] = q;
            v[k] = fetch(i + k * kResThreads < n, q);
            walk.next(q);
        }
#pragma unroll
        for (int k = 0; k < U; k++) put(i + k * kResThreads < n, at[k], v[k]);
    }
}
template <class Put>
__device__ __forceinline__ void res_load(const Inst &in, const ResIO &io, const WordWalk &walk, int n, int y0, int z0,
                                         Put put)
{
    if (!io.pix) {
        const uint32_t *g = in.buf[0];
        const int H = in.H, P = in.P;
        res_load_loop<4>(walk, n, [&](bool live, const WordPos &q) {
            return live ? __ldcg(g + ((size_t)(z0 + q.z) * H + (y0 + q.y)) * P + q.x) : 0u;
        }, put);
        return;
    }
    const IODesc &d = *io.d;
    const int inW = d.inW, inH = d.inH, inD = d.inD;
    auto count = [&](bool live, const WordPos &q, uint32_t &off) {
        const int y = y0 + q.y, z = z0 + q.z;
        off = ((uint32_t)z * (uint32_t)inH + (uint32_t)y) * (uint32_t)inW + 32u * (uint32_t)q.x;
        return live && y < inH && z < inD ? max(0, min(32, inW - 32 * q.x)) : 0;
    };
    if (dtype_bytes(d.dtype) == 1) {
        const uint32_t neg = pixel_neg(d);
        res_load_loop<2>(walk, n, [&](bool live, const WordPos &q) {
            uint32_t off;
            const int cnt = count(live, q, off);
            return pixel_bytes(d, off, cnt, neg);
        }, put);
    } else {
        res_load_loop<1>(walk, n, [&](bool live, const WordPos &q) {
            uint32_t off;
            const int cnt = count(live, q, off);
            return pixel_word_wide(d, off, cnt);
        }, put);
    }
}

// The way back for rows [y0, y0 + ny) of planes [z0, z0 + nz): row(y, z) = the
// packed words of grid row y of grid plane z.
template <class Row>
__device__ __forceinline__ void res_store(const Inst &in, const ResIO &io, int ny, int nz, int y0, int z0, Row row)
{
    const int lane = threadIdx.x & 31, wl = (in.W + 31) >> 5;
    const WordWalk walk(wl, ny);
    const int n = nz * ny * wl;
    if (!io.pix || !io.d->out) {
        uint32_t *g = in.buf[0];
        WordPos q = walk.first();
        for (int i = threadIdx.x; i < n; i += kResThreads, walk.next(q))
            g[((size_t)(z0 + q.z) * in.H + (y0 + q.y)) * in.P + q.x] = row(q.y, q.z)[q.x];
        return;
    }
    const IODesc &d = *io.d;
    if (dtype_bytes(d.dtype) == 1) {
        const uint32_t per = ((uint32_t)ny * (uint32_t)in.W + 31u) / 32u + 1u;  // chunks a plane's rows touch at most
        for (uint32_t i = threadIdx.x; i < per * (uint32_t)nz; i += kResThreads) {
            const uint32_t z = nz == 1 ? 0u : i / per;
            uint8_t *out = (uint8_t *)d.out + ((size_t)(z0 + (int)z) * in.H + y0) * in.W;
            pixel_chunk(out, (uint32_t)ny, in.W, d.dW, i - z * per, [&](uint32_t r) { return row((int)r, (int)z); });
        }
        return;
    }
    WordPos q = walk.first();
    for (int i = threadIdx.x; i - lane < n; i += kResThreads, walk.next(q)) {
        const bool live = i < n;
        const uint32_t off = ((uint32_t)(z0 + q.z) * (uint32_t)in.H + (uint32_t)(y0 + q.y)) * (uint32_t)in.W + 32u * (uint32_t)q.x;
        pixel_store_wide(d, off, live ? min(32, in.W - 32 * q.x) : 0, live ? row(q.y, q.z)[q.x] : 0u);
    }
}

// ------------------------------------------------------------ 2D ----------
// A pass is one iteration (N, S, E, W) run on register tiles: a warp loads a
// unit -- 24 core rows plus 4 halo rows above and below (lane = row) by 8
// core words plus one halo word on either side -- from the pass-start copy,
// runs the four subiterations in registers (rows above and below by
// shuffles, x-neighbours by funnel shifts) and writes its core to the other
// copy.  Wrong values entering at a unit's edge move one row (or bit) per
// subiteration, so after four they reach only its halo.
// BGT_RES_LANE_ROWS=2 builds units of 56 core rows, two adjacent rows per
// lane (each other's vertical neighbours, half the shuffles per row, less
// halo): measured slower on stroke images (1.13 against 1.06 ms for 512
// images), as the larger units stay active for longer.
constexpr int kUnitRows = 32 * kLaneRows - 2 * 4;  // core rows of a unit (K = 4)
constexpr int kUnitWords = 8;                      // core words of a unit
constexpr int kHaloLanes = 4 / kLaneRows;          // lanes holding the top (or bottom) halo rows

// The rule on word j of a lane's two rows a (upper) and b (lower): o the
// words, n/p the words after/before them (pass-start values).
template <int DIR>
__device__ __forceinline__ void word2d_pair(uint32_t oa, uint32_t na, uint32_t pa, uint32_t ob, uint32_t nb,
                                            uint32_t pb, uint32_t &ra, uint32_t &rb)
{
    const uint32_t xpa = at_xp1(oa, na), xma = at_xm1(oa, pa);
    const uint32_t xpb = at_xp1(ob, nb), xmb = at_xm1(ob, pb);
    uint32_t A[8], B[8];
    A[0] = __shfl_up_sync(kFull, ob, 1);   // row above a: the lower row of the lane above
    A[1] = __shfl_up_sync(kFull, xpb, 1);
    A[7] = __shfl_up_sync(kFull, xmb, 1);
    A[2] = xpa;
    A[6] = xma;
    A[4] = ob;
    A[3] = xpb;
    A[5] = xmb;
    B[4] = __shfl_down_sync(kFull, oa, 1);  // row below b: the upper row of the lane below
    B[3] = __shfl_down_sync(kFull, xpa, 1);
    B[5] = __shfl_down_sync(kFull, xma, 1);
    B[2] = xpb;
    B[6] = xmb;
    B[0] = oa;
    B[1] = xpa;
    B[7] = xma;
    ra = keep2d<DIR>(oa, A);
    rb = keep2d<DIR>(ob, B);
}

// One subiteration on the lane's two rows of S+2 words (words j0..j1-1 are
// processed; the rest keep their values).  Words that are empty in both
// rows of every lane are skipped.
template <int S, int DIR, int J0, int J1>
__device__ __forceinline__ void subit2d_pair(uint32_t (&a)[S + 2], uint32_t (&b)[S + 2])
{
    uint32_t pa = J0 > 0 ? a[J0 - 1] : 0u, pb = J0 > 0 ? b[J0 - 1] : 0u;
#pragma unroll
    for (int j = J0; j < J1; j++) {
        const uint32_t oa = a[j], ob = b[j];
        const uint32_t na = j + 1 < S + 2 ? a[j + 1] : 0u, nb = j + 1 < S + 2 ? b[j + 1] : 0u;
        if (__any_sync(kFull, (oa | ob) != 0u)) word2d_pair<DIR>(oa, na, pa, ob, nb, pb, a[j], b[j]);
        pa = oa;
        pb = ob;
    }
}

// K subiterations from phase PH; the last one only on the core words.
template <int K, int S, int PH, int I = 0>
__device__ __forceinline__ void run_subits2d_pair(uint32_t (&a)[S + 2], uint32_t (&b)[S + 2])
{
    if constexpr (I + 1 < K) {
        subit2d_pair<S, (PH + I) & 3, 0, S + 2>(a, b);
        run_subits2d_pair<K, S, PH, I + 1>(a, b);
    } else if constexpr (I + 1 == K) {
        subit2d_pair<S, (PH + I) & 3, 1, S + 1>(a, b);
    }
}

__host__ __device__ inline int res_pitch2d_tiles(int W)
{
    const int wl = (W + 31) >> 5;
    const int nch = (wl + kUnitWords - 1) / kUnitWords;
    return (nch * kUnitWords + 2) | 1;  // zero word left, zero words right, odd
}

struct Band2D {
    uint32_t *zero;     // pp zero words
    uint32_t *buf0, *buf1;  // nrows x pp each: pass q reads buf[q & 1], writes buf[(q + 1) & 1]
    int *until;         // [nstrips][nchunks]: the unit is processed while q <= until (a unit in
                        // its 3x3 neighbourhood deleted something in the previous pass)
    int pp, wl, nrows, nstrips, nchunks;
    int a;              // image row of the band's first row in shared memory
    int r0, r1;         // core rows (image coordinates)
};

// One pass q over the band's units.  A unit none of whose inputs for the
// pass -- its core and the 4-pixel border bands of its 3x3 neighbours -- had
// a deletion in the previous pass (one subiteration of every direction) is
// skipped: that region is a fixed point, and a unit processed without a
// change wrote identical data to both copies.  A unit that deletes something
// extends `until` to q + 1 for itself and for each neighbour whose border
// band the deletions reach (a reader in the same pass may see the new value:
// it then processes a unit it could have skipped).
// Returns this thread's deleted core bits (band core rows only).
__device__ uint32_t res_pass2d(const Band2D &b, int q, int *take, unsigned long long *words)
{
    const int lane = threadIdx.x & 31;
    const uint32_t *IN = (q & 1) ? b.buf1 : b.buf0;
    uint32_t *OUT = (q & 1) ? b.buf0 : b.buf1;
    const int nunits = b.nstrips * b.nchunks;
    uint32_t core = 0;
    for (;;) {
        const int u = res_take(take);
        if (u >= nunits) break;
        if (b.until[u] < q) continue;
        const int s = u / b.nchunks, c = u - s * b.nchunks;
        const int x0 = 1 + kUnitWords * c;
        const int rbase = kUnitRows * s - 4 + kLaneRows * lane;  // band row of the lane's first row
        uint32_t v[kLaneRows][kUnitWords + 2];
        const uint32_t *in[kLaneRows];
        bool valid[kLaneRows];
#pragma unroll
        for (int i = 0; i < kLaneRows; i++) {
            const int r = rbase + i;
            valid[i] = r >= 0 && r < b.nrows;
            in[i] = valid[i] ? IN + (size_t)r * b.pp : b.zero;
#pragma unroll
            for (int k = 0; k < kUnitWords + 2; k++) v[i][k] = in[i][x0 - 1 + k];
        }
        if constexpr (kLaneRows == 2) run_subits2d_pair<4, kUnitWords, 0>(v[0], v[1]);
        else run_subits2d<4, kUnitWords, 0>(v[0]);
        const bool core_lane = lane >= kHaloLanes && lane < 32 - kHaloLanes;
        uint32_t chg = 0, lft = 0, rgt = 0;
#pragma unroll
        for (int i = 0; i < kLaneRows; i++) {
            if (!(valid[i] && core_lane)) continue;
            uint32_t *out = OUT + (size_t)(rbase + i) * b.pp;
            uint32_t ci = 0;
#pragma unroll
            for (int k = 0; k < kUnitWords; k++) {
                const uint32_t d = v[i][1 + k] ^ in[i][x0 + k];
                ci |= d;
                if (k == 0) lft |= d & 0xFu;                     // within 4 pixels of the left edge
                if (k == kUnitWords - 1) rgt |= d & 0xF0000000u;  // ... of the right edge
                out[x0 + k] = v[i][1 + k];
            }
            chg |= ci;
            const int gy = b.a + rbase + i;
            if (gy >= b.r0 && gy < b.r1) core |= ci;
        }
        // The next pass of a neighbour depends on this unit only through the
        // 4 pixels next to their common border (four subiterations reach 4
        // pixels): activate the neighbours whose border band changed
        // (border bands, as the tile engine does).
        const unsigned m_any = __ballot_sync(kFull, chg != 0u);
        if (m_any) {
            const unsigned m_l = __ballot_sync(kFull, lft != 0u), m_r = __ballot_sync(kFull, rgt != 0u);
            // lanes holding the first and last 4 core rows
            constexpr unsigned band_top = ((1u << kHaloLanes) - 1u) << kHaloLanes;
            constexpr unsigned band_bot = ((1u << kHaloLanes) - 1u) << (32 - 2 * kHaloLanes);
            if (lane < 9) {
                const int dy = lane / 3 - 1, dx = lane % 3 - 1;
                const unsigned rows = dy < 0 ? band_top : dy > 0 ? band_bot : ~0u;
                const unsigned cols = dx < 0 ? m_l : dx > 0 ? m_r : m_any;
                const int ns = s + dy, nc = c + dx;
                if ((rows & cols & m_any) && ns >= 0 && ns < b.nstrips && nc >= 0 && nc < b.nchunks)
                    b.until[ns * b.nchunks + nc] = q + 1;
            }
        }
        if (lane == 0)
            *words += (unsigned long long)min(kUnitRows, b.nrows - kUnitRows * s) *
                      min(kUnitWords, b.wl - kUnitWords * c);
    }
    return core;
}

__device__ void res_run2d(Inst &in, const ResIO &io, const ResItem &it, uint32_t *sm, ResSched *S, int *take)
{
    __shared__ int s_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Band2D b;
    b.wl = (in.W + 31) >> 5;
    b.pp = res_pitch2d_tiles(in.W);
    b.nchunks = (b.wl + kUnitWords - 1) / kUnitWords;
    b.r0 = it.r0;
    b.r1 = it.r1;
    b.a = max(0, it.r0 - it.halo);
    const int bend = min(in.H, it.r1 + it.halo);
    b.nrows = bend - b.a;
    b.nstrips = (b.nrows + kUnitRows - 1) / kUnitRows;
    b.zero = sm;
    b.buf0 = sm + b.pp;
    b.buf1 = b.buf0 + (size_t)b.nrows * b.pp;
    b.until = reinterpret_cast<int *>(b.buf1 + (size_t)b.nrows * b.pp);
    const int pp = b.pp;
    const int nunits = b.nstrips * b.nchunks;

    // zero row and row copies (their words left and right of the image stay zero)
    {
        const int total = pp * (1 + 2 * b.nrows);
        for (int i = threadIdx.x; i < total / 4; i += kResThreads)
            reinterpret_cast<uint4 *>(sm)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (threadIdx.x < (total & 3)) sm[(total & ~3) + threadIdx.x] = 0u;
    }
    for (int i = threadIdx.x; i < nunits; i += kResThreads) b.until[i] = -1;
    if (threadIdx.x < 2) take[threadIdx.x] = 0;
    __syncthreads();
    res_load(in, io, WordWalk(b.wl, b.nrows), b.nrows * b.wl, b.a, 0, [&](bool, const WordPos &q, uint32_t v) {
        if (!v) return;
        const int w = q.y * pp + q.x + 1;
        b.buf0[w] = v;
        b.buf1[w] = v;
        // units holding foreground start active
        b.until[(q.y / kUnitRows) * b.nchunks + q.x / kUnitWords] = 0;
    });
    __syncthreads();

    int result = 0;  // 1 converged, -1 pass cap or failed wait
    MeetState meet;
    unsigned long long words = 0;
    int q = 0;
    for (;; q++) {
        // the counter of this pass was cleared during the previous one;
        // clear the next one's (nobody uses it before the barrier below)
        if (threadIdx.x == 0) take[(q + 1) & 1] = 0;
        const uint32_t core = res_pass2d(b, q, take + (q & 1), &words);
        const bool any = __syncthreads_or(core != 0u);
        if (it.bands == 1) {
            if (!any) {
                result = 1;
                break;
            }
        } else if (q % kResPassesPerExchange == kResPassesPerExchange - 1) {
            // end of pass q (state in buf[(q+1)&1]), the last of an exchange
            // period: trade boundary rows with the neighbouring bands
            const int h = it.halo;
            const int e = q / kResPassesPerExchange;  // exchange index
            uint32_t *cur = (q & 1) ? b.buf0 : b.buf1;
            uint32_t *gx = in.buf[(e + 1) & 1];  // buf[0] holds the start state other bands may still load
            for (int k = warp; k < 2 * h; k += kWarps) {
                const bool top = k < h;
                if (top ? it.band == 0 : it.band + 1 == it.bands) continue;
                const int gy = top ? b.r0 + k : b.r1 - 2 * h + k;
                const uint32_t *srow = cur + (size_t)(gy - b.a) * pp;
                uint32_t *grow = gx + (size_t)gy * in.P;
                for (int w = lane; w < b.wl; w += 32) grow[w] = srow[w + 1];
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                s_flag = res_meet(in.res_meet, it.bands, any, meet, S->timeout_ns);
                if (s_flag == 2) atomicOr(&S->status, kErrQueueTimeout);
            }
            __syncthreads();
            const int f = s_flag;
            if (f != 1) {
                result = f == 0 ? 1 : -1;
                break;
            }
            // halo rows: the neighbours' boundary core rows after pass q
            const int ntop = b.r0 - b.a, nh = ntop + (bend - b.r1);
            uint32_t hc = 0;
            for (int k = warp; k < nh; k += kWarps) {
                const int r = k < ntop ? k : (b.r1 - b.a) + (k - ntop);
                const uint32_t *grow = gx + (size_t)(b.a + r) * in.P;
                uint32_t *srow = cur + (size_t)r * pp;
                for (int w = lane; w < b.wl; w += 32) {
                    const uint32_t v = __ldcg(grow + w);
                    hc |= v ^ srow[w + 1];
                    srow[w + 1] = v;
                }
            }
            if (__syncthreads_or(hc != 0u)) {
                // units within reach of the halo rows go on next pass
                for (int u = threadIdx.x; u < nunits; u += kResThreads) {
                    const int st = u / b.nchunks;
                    const int ga = b.a + kUnitRows * st - kUnitRows, gb = b.a + kUnitRows * st + 2 * kUnitRows;
                    if (ga < b.r0 || gb > b.r1) b.until[u] = q + 1;
                }
                __syncthreads();
            }
        }
        if (q >= in.pass_cap) {
            if (threadIdx.x == 0) atomicOr(&S->status, kErrPassLimit);
            result = -1;
            break;
        }
    }
    // the converged core rows (in buf[(q+1)&1])
    __syncthreads();
    const uint32_t *fin = ((q & 1) ? b.buf0 : b.buf1) + (size_t)(b.r0 - b.a) * pp + 1;
    res_store(in, io, b.r1 - b.r0, 1, b.r0, 0, [&](int y, int) { return fin + (size_t)y * pp; });
    if (lane == 0 && words) atomicAdd(&in.work_words, words);  // core words per pass (one iteration)
    if (threadIdx.x == 0) {
        if (it.band == 0) in.passes_run = q + 1;
        if (result < 0) atomicMin(&in.converged, -1);
        atomicAdd(&in.tiles_run, 1ull);
    }
    __syncthreads();
}

// ------------------------------------------------------------ 3D ----------
// Entry of a box's word list: word index in shared memory (16 bits), its
// column in the rows' change masks (5 bits), its distance from the box's core
// (3 bits, 0 = core), and, in the candidate list, whether it changed.
constexpr uint32_t kEntChanged = 1u << 24;
__device__ __forceinline__ uint32_t ent_idx(uint32_t e) { return e & 0xffffu; }
__device__ __forceinline__ uint32_t ent_col(uint32_t e) { return (e >> 16) & 31u; }
__device__ __forceinline__ int ent_dist(uint32_t e) { return (int)((e >> 21) & 7u); }

struct Box3D {
    uint32_t *state;      // [nz + 2][ny + 2] rows of wl words, a zero word between rows, a zero word at the end
    uint32_t *cidx, *cU, *cdel;  // candidates of this iteration: entry, union, deletions of the subiteration
    int p, ps;            // words between rows, between planes
};

// The 3x3x3 neighbourhood words of the word at s.
__device__ __forceinline__ void box_window(const uint32_t *s, int p, int ps, uint32_t (&g)[27])
{
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const uint32_t *r = s + (k / 3 - 1) * ps + (k % 3 - 1) * p;
        const uint32_t l = r[-1], c = r[0], n = r[1];
        g[3 * k] = at_xm1(c, l);
        g[3 * k + 1] = c;
        g[3 * k + 2] = at_xp1(c, n);
    }
}

// Position of this lane's element in a list the warp appends to (-1: none).
__device__ __forceinline__ int warp_append(bool take, int *count)
{
    const unsigned m = __ballot_sync(kFull, take);
    int base = 0;
    if ((threadIdx.x & 31) == 0 && m) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(kFull, base, 0);
    return take ? base + __popc(m & ((1u << (threadIdx.x & 31)) - 1u)) : -1;
}

// Subiteration J (1..5: N, E, D, S, W) on the candidates: find the deletions,
// meet, apply them, meet.  Words farther than 5 - J from the core are left
// alone: what they read may be wrong by now, and nothing reads them before
// their owner sends them.
template <int J>
__device__ __forceinline__ uint32_t box_deletions(const Box3D &b, uint32_t e, uint32_t cand)
{
    if (ent_dist(e) > 5 - J || cand == 0u) return 0u;
    uint32_t g[27];
    box_window(b.state + ent_idx(e), b.p, b.ps, g);
    return cand & rule3d<J>(g);
}

// ... with any number of candidates per thread
template <int J>
__device__ __forceinline__ void box_subiteration(const Box3D b, int nc, unsigned &words)
{
    bool any = false;
    for (int c = threadIdx.x; c < nc; c += kResThreads) {
        const uint32_t e = b.cidx[c];
        const uint32_t del = box_deletions<J>(b, e, b.state[ent_idx(e)] & b.cU[c]);
        words += ent_dist(e) == 0;
        any |= del != 0u;
        b.cdel[c] = del;
    }
    if (!__syncthreads_or(any)) return;
    for (int c = threadIdx.x; c < nc; c += kResThreads) {
        const uint32_t del = b.cdel[c];
        if (del) {
            const uint32_t e = b.cidx[c];
            b.state[ent_idx(e)] &= ~del;
            b.cidx[c] = e | kEntChanged;
        }
    }
    __syncthreads();
}

// ... with at most one: its word, union and entry stay in registers
template <int J>
__device__ __forceinline__ void box_subiteration1(const Box3D b, uint32_t e, uint32_t un, uint32_t &val, unsigned &words)
{
    const uint32_t del = box_deletions<J>(b, e, val & un);
    words += un != 0u && ent_dist(e) == 0;
    if (!__syncthreads_or(del != 0u)) return;
    if (del) {
        val &= ~del;
        b.state[ent_idx(e)] = val;
    }
    __syncthreads();
}

// One volume, or one box of it: rows [c0, c1) of planes [r0, r1) are the
// core; `halo` rows and planes around it (clamped to the volume) are held
// too.  Boxes run whole iterations (pre-test, U, N, E, D, S, W) in lockstep.
// A wrong value moves one row or plane per subiteration (the pre-test reads
// the same neighbours as U), so with six halo rows and planes the core is
// exact after an iteration; then every box sends the words near its core's
// edge that changed to a list in global memory, the boxes meet, and each
// takes over what lies in its halo from its neighbours' lists.
//
// Bound: the latency of an iteration (about 10 us: six dependent subiterations
// with two barriers each, then the meeting), not throughput: a box has some
// hundred active words.  Against warps marching through sparse bricks of
// 32 x 32 x 4 voxels, every brick of the neighbourhood of a change evaluated
// whole (24 us per iteration): a 97 x 75 x 66 tree volume 214 -> 72 us, a
// 187 x 203 x 161 one 955 -> 150 us, a 256^3 one, whose bricks did not fit,
// 1330 us on the tile rings -> 176 us.
__device__ void res_run3d(Inst &in, const ResIO &io, const ResItem &it, uint8_t *smb, ResSched *S)
{
    __shared__ int s_n[4];  // lengths: word list, active words, candidates, messages
    __shared__ int s_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int H = in.H, D = in.D, wl = (in.W + 31) >> 5;
    const bool team = it.bands > 1;
    const int z0 = max(0, it.r0 - it.halo), z1 = min(D, it.r1 + it.halo);
    const int y0 = max(0, it.c0 - it.halo), y1 = min(H, it.c1 + it.halo);
    const int nz = z1 - z0, ny = y1 - y0, ny2 = ny + 2, rows2 = (nz + 2) * ny2;
    int xs = 0;  // words per column of the change masks: 1 << xs
    while (((wl - 1) >> xs) > 31) xs++;
    Box3D b;
    b.p = wl + 1;
    b.ps = ny2 * b.p;
    const uint32_t mp = 0xffffffffu / (uint32_t)b.p + 1u;
    const uint32_t mny = 0xffffffffu / (uint32_t)ny2 + 1u;
    const int nwords = rows2 * b.p + 1;
    size_t off = 0;
    b.state = reinterpret_cast<uint32_t *>(smb);
    off += up16((size_t)nwords * 4);
    uint32_t *const act = reinterpret_cast<uint32_t *>(smb + off);
    off += up16((size_t)rows2 * 4);
    uint32_t *const chg = reinterpret_cast<uint32_t *>(smb + off);
    off += up16((size_t)rows2 * 4);
    uint32_t *const list = reinterpret_cast<uint32_t *>(smb + off);
    const int list_cap = (int)(((size_t)kSmemBytes - off) / 4);

    for (size_t i = threadIdx.x; i < off / 16; i += kResThreads) reinterpret_cast<uint4 *>(smb)[i] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x < 4) s_n[threadIdx.x] = 0;
    __syncthreads();
    const int nbox = nz * ny * wl;
    const WordWalk walk(wl, ny);
    auto dist_of = [&](const WordPos &q) {
        const int y = y0 + q.y, z = z0 + q.z;
        return max(max(max(it.c0 - y, y - it.c1 + 1), max(it.r0 - z, z - it.r1 + 1)), 0);
    };
    auto index_of = [&](const WordPos &q) { return ((q.z + 1) * ny2 + q.y + 1) * b.p + 1 + q.x; };
    res_load(in, io, walk, nbox, y0, z0, [&](bool, const WordPos &q, uint32_t v) {
        const int d = dist_of(q), idx = v ? index_of(q) : 0;
        if (v) b.state[idx] = v;
        const int pos = warp_append(v != 0u && d <= 5, &s_n[0]);
        if (pos >= 0 && pos < list_cap) list[pos] = (uint32_t)idx | (uint32_t)(q.x >> xs) << 16 | (uint32_t)d << 21;
    });
    __syncthreads();
    const int nl = s_n[0];
    MeetState meet;
    // more non-empty words than the lists hold: go over all words of the box,
    // with the union and the deletions stored per word
    const bool dense = off + (size_t)nl * kBoxListBytes + 64 > (size_t)kSmemBytes;
    b.cidx = list + nl;
    b.cU = dense ? list : b.cidx + nl;
    b.cdel = b.cU + (dense ? nwords : nl);
    uint16_t *const alist = reinterpret_cast<uint16_t *>(b.cdel + nl);
    for (int r = threadIdx.x; r < rows2; r += kResThreads) act[r] = kFull;
    __syncthreads();

    const int gy = in.res_gy;  // boxes along y
    const int bz = it.band / gy, by = it.band - bz * gy, gz = it.bands / gy;
    int iter = 0, result = 0;
    unsigned words = 0, entries = 0;
    const int cap_it = in.pass_cap / 6 + 1;
    // a word of the core changed: mark it, and tell the boxes around when it lies near the core's edge
    auto changed = [&](uint32_t idx, uint32_t col, uint2 *msg) {
        const uint32_t row = __umulhi(idx, mp);
        atomicOr(&chg[row], 1u << col);
        if (!team) return;
        const int zz = (int)__umulhi(row, mny), y = y0 + (int)row - zz * ny2 - 1, z = z0 + zz - 1;
        const int h = it.halo;
        if ((it.r0 > 0 && z < it.r0 + h) || (it.r1 < D && z >= it.r1 - h) || (it.c0 > 0 && y < it.c0 + h) ||
            (it.c1 < H && y >= it.c1 - h)) {
            const int x = (int)idx - (int)row * b.p - 1;
            msg[atomicAdd(&s_n[3], 1)] =
                make_uint2(((uint32_t)z * (uint32_t)H + (uint32_t)y) * (uint32_t)wl + (uint32_t)x, b.state[idx]);
        }
    };
    for (;; iter++) {
        bool core = false;
        uint2 *msg = nullptr;
        if (team) msg = in.res_msg + ((size_t)(iter & 1) * it.bands + it.band) * in.res_stride;
        if (!dense) {
            // active words: a word of the row's 3x3 rows that is at most one
            // column away changed in the previous iteration (otherwise its union
            // is empty), and some voxel of it misses one of its face neighbours
            for (int base = warp * 32; base < nl; base += kResThreads) {
                const int k = base + lane;
                bool on = false;
                if (k < nl) {
                    const uint32_t e = list[k], idx = ent_idx(e);
                    if ((act[__umulhi(idx, mp)] >> ent_col(e)) & 1u) {
                        const uint32_t *s = b.state + idx;
                        const uint32_t c = *s;
                        const uint32_t faces = at_xm1(c, s[-1]) & at_xp1(c, s[1]) & s[b.p] & s[-b.p] & s[b.ps] & s[-b.ps];
                        on = (c & ~faces) != 0u;
                    }
                }
                const int pos = warp_append(on, &s_n[1]);
                if (pos >= 0) alist[pos] = (uint16_t)k;
            }
            __syncthreads();
            const int na = s_n[1];
            // pre-test and U
            for (int base = warp * 32; base < na; base += kResThreads) {
                const int k = base + lane;
                uint32_t e = 0, un = 0, du = 0;
                if (k < na) {
                    e = list[alist[k]];
                    const uint32_t *s = b.state + ent_idx(e);
                    uint32_t g[27];
                    box_window(s, b.p, b.ps, g);
                    du = rule3d<0>(g) & g[13];
                    un = (du | rule3d<1>(g) | rule3d<2>(g) | rule3d<3>(g) | rule3d<4>(g) | rule3d<5>(g)) & g[13];
                    words += ent_dist(e) == 0;
                    entries++;
                }
                const int c = warp_append(un != 0u, &s_n[2]);
                if (c >= 0) {
                    b.cidx[c] = e;
                    b.cU[c] = un;
                    b.cdel[c] = du;
                }
            }
            __syncthreads();
            const int nc = s_n[2];
            if (nc > kResThreads) {
                for (int c = threadIdx.x; c < nc; c += kResThreads) {
                    const uint32_t del = b.cdel[c];
                    if (del) {
                        const uint32_t e = b.cidx[c];
                        b.state[ent_idx(e)] &= ~del;
                        b.cidx[c] = e | kEntChanged;
                    }
                }
                __syncthreads();
                box_subiteration<1>(b, nc, words);
                box_subiteration<2>(b, nc, words);
                box_subiteration<3>(b, nc, words);
                box_subiteration<4>(b, nc, words);
                box_subiteration<5>(b, nc, words);
            } else if (nc > 0) {
                const int c = threadIdx.x;
                uint32_t e = 0, un = 0, val = 0, del = 0;
                if (c < nc) {
                    e = b.cidx[c];
                    un = b.cU[c];
                    del = b.cdel[c];
                    val = b.state[ent_idx(e)];
                }
                const uint32_t before = val;
                if (del) {
                    val &= ~del;
                    b.state[ent_idx(e)] = val;
                }
                __syncthreads();
                box_subiteration1<1>(b, e, un, val, words);
                box_subiteration1<2>(b, e, un, val, words);
                box_subiteration1<3>(b, e, un, val, words);
                box_subiteration1<4>(b, e, un, val, words);
                box_subiteration1<5>(b, e, un, val, words);
                if (val != before) b.cidx[c] = e | kEntChanged;
            }
            for (int c = threadIdx.x; c < nc; c += kResThreads) {
                const uint32_t e = b.cidx[c];
                if (!(e & kEntChanged) || ent_dist(e) != 0) continue;
                core = true;
                changed(ent_idx(e), ent_col(e), msg);
            }
        } else {
            WordPos q = walk.first();
            for (int i = threadIdx.x; i < nbox; i += kResThreads, walk.next(q)) {
                const int idx = index_of(q), d = dist_of(q);
                const uint32_t *s = b.state + idx;
                uint32_t un = 0, du = 0;
                if (d <= 5 && *s && ((act[(q.z + 1) * ny2 + q.y + 1] >> (q.x >> xs)) & 1u)) {
                    uint32_t g[27];
                    box_window(s, b.p, b.ps, g);
                    du = rule3d<0>(g) & g[13];
                    un = (du | rule3d<1>(g) | rule3d<2>(g) | rule3d<3>(g) | rule3d<4>(g) | rule3d<5>(g)) & g[13];
                    words += d == 0;
                    entries++;
                }
                b.cU[idx] = un;
                b.cdel[idx] = du;
            }
            __syncthreads();
#pragma unroll 1
            for (int j = 0; j < 6; j++) {
                // deletions of subiteration j were found: apply them, then find the next one's
                q = walk.first();
                for (int i = threadIdx.x; i < nbox; i += kResThreads, walk.next(q)) {
                    const int idx = index_of(q);
                    const uint32_t del = b.cdel[idx];
                    if (del) b.state[idx] &= ~del;
                }
                __syncthreads();
                if (j == 5) break;
                q = walk.first();
                for (int i = threadIdx.x; i < nbox; i += kResThreads, walk.next(q)) {
                    const int idx = index_of(q), d = dist_of(q);
                    const uint32_t cand = b.state[idx] & b.cU[idx];
                    uint32_t del = 0;
                    if (cand && d <= 4 - j) {
                        uint32_t g[27];
                        box_window(b.state + idx, b.p, b.ps, g);
                        del = cand & (j == 0   ? rule3d<1>(g)
                                      : j == 1 ? rule3d<2>(g)
                                      : j == 2 ? rule3d<3>(g)
                                      : j == 3 ? rule3d<4>(g)
                                               : rule3d<5>(g));
                        words += d == 0;
                    }
                    b.cdel[idx] = del;
                }
                __syncthreads();
            }
            // only voxels of the union were deleted: a word changed when it lost some of its union
            q = walk.first();
            for (int i = threadIdx.x; i < nbox; i += kResThreads, walk.next(q)) {
                const int idx = index_of(q);
                if (!(b.cU[idx] & ~b.state[idx]) || dist_of(q) != 0) continue;
                core = true;
                changed((uint32_t)idx, (uint32_t)(q.x >> xs), msg);
            }
        }
        const bool any = __syncthreads_or(core);
        bool any_chg = any;
        if (!team) {
            if (!any) {
                result = 1;
                break;
            }
        } else {
            if (threadIdx.x == 0) {
                in.res_cnt[(iter & 1) * it.bands + it.band] = s_n[3];
                s_flag = res_meet(in.res_meet, it.bands, any, meet, S->timeout_ns);
                if (s_flag == 2) atomicOr(&S->status, kErrQueueTimeout);
            }
            __syncthreads();
            const int f = s_flag;
            if (f != 1) {
                result = f == 0 ? 1 : -1;
                break;
            }
            // three warps per neighbouring box take over its messages
            const int k8 = warp & 7, k9 = k8 < 4 ? k8 : k8 + 1;
            const int nbz = bz + k9 / 3 - 1, nby = by + k9 % 3 - 1;
            if (nbz >= 0 && nbz < gz && nby >= 0 && nby < gy) {
                const int nb = nbz * gy + nby;
                const uint2 *m = in.res_msg + ((size_t)(iter & 1) * it.bands + nb) * in.res_stride;
                const int k0 = (warp >> 3) * 32 + lane;
                // the first message is loaded beside the count, whether it is one or not
                uint2 v = k0 < in.res_stride ? __ldcg(m + k0) : make_uint2(0u, 0u);
                const int n = __ldcg(in.res_cnt + (iter & 1) * it.bands + nb);
                for (int k = k0; k < n;) {
                    const int r = (int)(v.x / (uint32_t)wl), x = (int)v.x - r * wl, z = r / H, y = r - z * H;
                    if (z >= z0 && z < z1 && y >= y0 && y < y1) {
                        const int row = (z - z0 + 1) * ny2 + (y - y0 + 1);
                        b.state[row * b.p + 1 + x] = v.y;
                        atomicOr(&chg[row], 1u << (x >> xs));
                        any_chg = true;
                    }
                    k += (kWarps / 8) * 32;
                    if (k < n) v = __ldcg(m + k);
                }
            }
            any_chg = __syncthreads_or(any_chg);
        }
        if (iter + 1 >= cap_it) {
            if (threadIdx.x == 0) atomicOr(&S->status, kErrPassLimit);
            result = -1;
            break;
        }
        // rows to look at in the next iteration
        for (int r = threadIdx.x + ny2; r < rows2 - ny2; r += kResThreads) {
            uint32_t m = 0;
            if (any_chg) {
                const uint32_t *c = chg + r;
#pragma unroll
                for (int k = 0; k < 9; k++) m |= c[(k / 3 - 1) * ny2 + (k % 3 - 1)];
            }
            act[r] = m | m << 1 | m >> 1;
        }
        if (threadIdx.x >= 1 && threadIdx.x < 4) s_n[threadIdx.x] = 0;
        __syncthreads();
        if (any_chg)
            for (int r = threadIdx.x; r < rows2; r += kResThreads) chg[r] = 0u;
        // (chg is next written after the barriers of the next iteration)
    }
    __syncthreads();
    // the converged core
    res_store(in, io, it.c1 - it.c0, it.r1 - it.r0, it.c0, it.r0, [&](int y, int z) {
        return b.state + ((z + it.r0 - z0 + 1) * ny2 + (y + it.c0 - y0 + 1)) * b.p + 1;
    });
    words = __reduce_add_sync(kFull, words);
    entries = __reduce_add_sync(kFull, entries);
    if (lane == 0 && words) {
        atomicAdd(&in.work_words, (unsigned long long)words);
        atomicAdd(&in.tiles_run, (unsigned long long)entries);
    }
    if (threadIdx.x == 0) {
        if (it.band == 0) in.passes_run = 6 * (iter + 1);
        if (result < 0) atomicMin(&in.converged, -1);
    }
    __syncthreads();
}

// ------------------------------------------------------------ kernels -----
__global__ void resident_reset_kernel(Inst *insts, int n, ResSched *S, int nitems, long long timeout_ns)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        Inst &in = insts[i];
        in.res_meet[0] = in.res_meet[1] = 0;
        if (in.res) {
            in.converged = 1;  // lowered to -1 by a band that fails
            in.passes_run = 0;
            in.tiles_run = 0;
            in.work_words = 0;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        S->head = 0;
        S->nitems = nitems;
        S->status = 0;
        S->timeout_ns = timeout_ns;
    }
}

__device__ __forceinline__ int res_smid()
{
    int v;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(v));
    return v;
}

__global__ void __launch_bounds__(kResThreads, kResCtasPerSm)
    resident_kernel(Inst *insts, const ResItem *items, ResSched *S, ResTrace *trace, const IODesc *ios, bool pix,
                    const __grid_constant__ IODesc one)
{
    extern __shared__ __align__(16) uint8_t res_smem[];
    __shared__ int s_item;
    __shared__ int s_take[2];
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(&S->head, 1);
        __syncthreads();
        const int k = s_item;
        __syncthreads();
        if (k >= S->nitems) break;
        const ResItem it = items[k];
        Inst &in = insts[it.inst];
        const long long t0 = (long long)globaltimer();
        const ResIO io{ios ? ios + it.inst : &one, pix};
        if (in.dims == 2)
            res_run2d(in, io, it, reinterpret_cast<uint32_t *>(res_smem), S, s_take);
        else
            res_run3d(in, io, it, res_smem, S);
        if (threadIdx.x == 0) trace[k] = ResTrace{t0, (long long)globaltimer(), res_smid(), 0};
    }
}

cudaError_t res_occupancy(int *per_sm)
{
    cudaError_t e = cudaFuncSetAttribute(resident_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(resident_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, resident_kernel, kResThreads, kSmemBytes);
}

cudaError_t launch_resident(int grid, Inst *d_insts, int ninst, const ResItem *d_items, int nitems,
                            ResSched *d_rs, ResTrace *d_trace, long long timeout_ns, const IODesc *d_io,
                            const IODesc *one, bool pixels, cudaStream_t st)
{
    if (nitems == 0) return cudaSuccess;
    static bool attr_done = false;
    if (!attr_done) {
        cudaError_t e = cudaFuncSetAttribute(resident_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(resident_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        if (e != cudaSuccess) return e;
        attr_done = true;
    }
    resident_reset_kernel<<<std::max(1, std::min(64, (ninst + 255) / 256)), 256, 0, st>>>(d_insts, ninst, d_rs, nitems,
                                                                                       timeout_ns);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // cooperative: all CTAs are resident at once, which the bands of an image
    // (waiting for one another) rely on
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(grid, nitems));
    cfg.blockDim = dim3(kResThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, resident_kernel, d_insts, d_items, d_rs, d_trace, one ? nullptr : d_io, pixels,
                              one ? *one : IODesc{});
}

}  // namespace bgt
