// resident.cu -- the resident engine: every work item (an instance, or one
// box of it) is loaded once into one
// CTA's shared memory and thinned there from its first subiteration to its
// fixed point; only the boxes of a large image (every few iterations) and of
// a large volume (every iteration) meet to trade their edges through global
// memory.
// One CTA of 768 threads per SM holds up to 225 KB (measured against two
// CTAs of 384 threads with 111 KB each: larger bands and slabs won).
//
// 2D image (dense).  The rows of the image, or of a box of it (core plus halo),
// lie twice in shared memory (pass q reads one copy and writes the other) with
// an odd pitch and zero words left and right of every row.  A pass hands units
// (24 rows x 2, 4 or 8 words) to warps dynamically; units whose surroundings
// did not change in the previous pass are skipped.  One box stops after a pass
// without a deletion: a fixed point of N, S, E and W, the reference's result.
// The boxes of a larger image meet after every few passes.
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
constexpr int kUnitRows = 24;  // core rows of a 2D unit (see the 2D section)

// Core words of the units of a 2D box of nrows rows of wl words: the width
// whose pass is shortest when every unit is active.  A unit of UW words costs
// UW + 1 word steps (one for its halo); a pass of few units takes as long as
// the units of one warp one after the other, a pass of many is bound by the
// ALU, which takes about kUnitLatency units in the time of one.  Widths of 8,
// 4 and 2 words for all boxes took the mixed batch 1.20, 1.23 and 1.38 ms, 16
// images of 1024^2 120, 116 and 121 us, a 200 x 160 image 21.1, 20.6 and 19.3 us.
constexpr int kUnitLatency = 11;
__host__ __device__ inline long long res_unit_cost(int nrows, int wl, int uw)
{
    const long long units = (long long)((nrows + kUnitRows - 1) / kUnitRows) * ((wl + uw - 1) / uw);
    const long long lat = (units + kWarps - 1) / kWarps * kUnitLatency * (uw + 1), alu = units * (uw + 1);
    return lat > alu ? lat : alu;
}
__host__ __device__ inline int res_unit_words(int nrows, int wl)
{
    int best = 8;
    for (int uw = 4; uw >= 2; uw /= 2)
        if (res_unit_cost(nrows, wl, uw) < res_unit_cost(nrows, wl, best)) best = uw;
    return best;
}
__host__ __device__ inline int res_pitch2d(int wl, int uw)
{
    return ((wl + uw - 1) / uw * uw + 2) | 1;  // zero word left, zero words right, odd
}
// words of shared memory a 2D box of nrows rows of wl words (halo included)
// needs with units of uw words: zero row, two row copies and the activity
// record of its units
inline size_t res_words2d(int wl, int nrows, int uw)
{
    return (size_t)res_pitch2d(wl, uw) * (1 + 2 * (size_t)nrows) +
           (size_t)((nrows + kUnitRows - 1) / kUnitRows) * ((wl + uw - 1) / uw);
}

// A 3D box of ny x nz rows of wl words (halo included) holds its state and the
// rows' masks in shared memory, and lists of its non-empty words; the planner
// leaves room for kListFill of the words.  A box with more non-empty words
// than its lists hold goes over all of its words, at most kDenseWords per
// thread, whose unions and deletions that thread keeps (in local memory).
constexpr size_t kBoxListBytes = 4 + 4 + 4 + 4 + 2;  // list, candidate, union, deletions, active list
constexpr double kListFill = 0.25;
constexpr int kDenseWords = 32;

int res_smem_bytes() { return kSmemBytes; }

double res_cost2d(int wl, int nrows) { return (double)res_unit_cost(nrows, wl, res_unit_words(nrows, wl)); }

bool res_fits2d(int wl, int nrows)
{
    // with units of any width: the boxes of an image differ in size (those at
    // its edges have less halo), so a smaller one may take wider units
    for (int uw = 2; uw <= 8; uw *= 2)
        if (res_words2d(wl, nrows, uw) * 4 > (size_t)kSmemBytes) return false;
    return true;
}

bool res_fits3d(int W, int ny, int nz)
{
    const int wl = (W + 31) / 32;
    const double rows2 = (double)(ny + 2) * (nz + 2), held = rows2 * (wl + 1) + 1, words = (double)wl * ny * nz;
    // words are indexed by 16 bits
    return held < 65535 && words <= (double)kDenseWords * kResThreads &&
           held * 4 + rows2 * 8 + kListFill * words * kBoxListBytes + 128 <= (double)kSmemBytes;
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

// put(pos, word) for every word of the grid of rows whose first word, row and
// plane are x0, y0, z0 (warps stay together: put may hold warp-wide votes; `live`
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
__device__ __forceinline__ void res_load(const Inst &in, const ResIO &io, const WordWalk &walk, int n, int x0, int y0, int z0,
                                         Put put)
{
    if (!io.pix) {
        const uint32_t *g = in.buf[0];
        const int H = in.H, P = in.P;
        res_load_loop<4>(walk, n, [&](bool live, const WordPos &q) {
            return live ? __ldcg(g + ((size_t)(z0 + q.z) * H + (y0 + q.y)) * P + (x0 + q.x)) : 0u;
        }, put);
        return;
    }
    const IODesc &d = *io.d;
    const int inW = d.inW, inH = d.inH, inD = d.inD;
    auto count = [&](bool live, const WordPos &q, uint32_t &off) {
        const int x = 32 * (x0 + q.x), y = y0 + q.y, z = z0 + q.z;
        off = ((uint32_t)z * (uint32_t)inH + (uint32_t)y) * (uint32_t)inW + (uint32_t)x;
        return live && y < inH && z < inD ? max(0, min(32, inW - x)) : 0;
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

// The way back for words [x0, x1) of rows [y0, y0 + ny) of planes [z0, z0 + nz):
// row(y, z) = the packed words from x0 on of grid row y of grid plane z.
template <class Row>
__device__ __forceinline__ void res_store(const Inst &in, const ResIO &io, int x0, int x1, int ny, int nz, int y0,
                                          int z0, Row row)
{
    const int lane = threadIdx.x & 31, wl = x1 - x0;
    const WordWalk walk(wl, ny);
    const int n = nz * ny * wl;
    if (!io.pix || !io.d->out) {
        uint32_t *g = in.buf[0];
        WordPos q = walk.first();
        for (int i = threadIdx.x; i < n; i += kResThreads, walk.next(q))
            g[((size_t)(z0 + q.z) * in.H + (y0 + q.y)) * in.P + x0 + q.x] = row(q.y, q.z)[q.x];
        return;
    }
    const IODesc &d = *io.d;
    const int np = min(in.W, 32 * x1) - 32 * x0;  // pixels per row
    if (dtype_bytes(d.dtype) == 1 && np == in.W) {
        // whole rows: one run of pixels per plane
        const uint32_t per = ((uint32_t)ny * (uint32_t)in.W + 31u) / 32u + 1u;  // chunks it touches at most
        for (uint32_t i = threadIdx.x; i < per * (uint32_t)nz; i += kResThreads) {
            const uint32_t z = nz == 1 ? 0u : i / per;
            uint8_t *out = (uint8_t *)d.out + ((size_t)(z0 + (int)z) * in.H + y0) * in.W;
            pixel_chunk(out, (uint32_t)ny, in.W, d.dW, i - z * per, [&](uint32_t r) { return row((int)r, (int)z); });
        }
        return;
    }
    if (dtype_bytes(d.dtype) == 1) {
        // parts of rows: a run per row (wl + 1 aligned chunks hold it)
        const WordWalk chunks(wl + 1, ny);
        WordPos q = chunks.first();
        for (int i = threadIdx.x; i < nz * ny * (wl + 1); i += kResThreads, chunks.next(q)) {
            uint8_t *out = (uint8_t *)d.out + ((size_t)(z0 + q.z) * in.H + (y0 + q.y)) * in.W + 32 * x0;
            const uint32_t *s = row(q.y, q.z);
            pixel_run_chunk(out, np, (uint32_t)q.x, s);
        }
        return;
    }
    WordPos q = walk.first();
    for (int i = threadIdx.x; i - lane < n; i += kResThreads, walk.next(q)) {
        const bool live = i < n;
        const int x = 32 * (x0 + q.x);
        const uint32_t off = ((uint32_t)(z0 + q.z) * (uint32_t)in.H + (uint32_t)(y0 + q.y)) * (uint32_t)in.W + (uint32_t)x;
        pixel_store_wide(d, off, live ? min(32, in.W - x) : 0, live ? row(q.y, q.z)[q.x] : 0u);
    }
}

// ------------------------------------------------------------ 2D ----------
// A pass is one iteration (N, S, E, W) run on register tiles: a warp loads a
// unit -- 24 core rows plus 4 halo rows above and below (lane = row) by UW
// core words plus a halo word -- from the pass-start copy, runs the four
// subiterations in registers (rows above and below by shuffles, x-neighbours
// by funnel shifts) and writes its core to the other copy.  Wrong values
// entering at a unit's edge move one row (or bit) per subiteration, so after
// four they reach only its halo.  Of the words left and right of the unit
// only the four pixels next to it matter, so one halo word holds both: its
// low half is the right one's, its high half the left one's, and the words
// form a ring (wrong values from the seam in its middle stay 12 bits away):
// 9 word steps per subiteration for 8 core words instead of 10.

// One subiteration on the ring of UW core words and the halo word v[UW];
// pairs of words empty in every lane are skipped.  The last subiteration
// leaves the halo word alone.
template <int UW, int DIR, bool LAST>
__device__ __forceinline__ void subit2d_ring(uint32_t (&v)[UW + 1])
{
    const uint32_t first = v[0];
    uint32_t prev = v[UW];
#pragma unroll
    for (int j = 0; j < UW; j += 2) {
        const uint32_t o0 = v[j], o1 = v[j + 1], on = v[j + 2];
        if (__any_sync(kFull, (o0 | o1) != 0u)) {
            v[j] = word2d<DIR>(o0, o1, prev);
            v[j + 1] = word2d<DIR>(o1, on, o0);
        }
        prev = o1;
    }
    if constexpr (!LAST) {
        const uint32_t o = v[UW];
        if (__any_sync(kFull, o != 0u)) v[UW] = word2d<DIR>(o, first, prev);
    }
}

struct Box2D {
    uint32_t *zero;         // pp zero words
    uint32_t *buf0, *buf1;  // nrows x pp each: pass q reads buf[q & 1], writes buf[(q + 1) & 1]
    int *until;             // [nstrips][nchunks]: the unit is processed while q <= until (a unit in
                            // its 3x3 neighbourhood deleted something in the previous pass)
    int pp, wl, nrows, nstrips, nchunks;
    int rlo, rhi;           // core rows and words, within the box
    int wlo, whi;
};

// One pass q over the box's units.  A unit none of whose inputs for the
// pass -- its core and the 4-pixel border bands of its 3x3 neighbours -- had
// a deletion in the previous pass (one subiteration of every direction) is
// skipped: that region is a fixed point, and a unit processed without a
// change wrote identical data to both copies.  A unit that deletes something
// extends `until` to q + 1 for itself and for each neighbour whose border
// band the deletions reach (a reader in the same pass may see the new value:
// it then processes a unit it could have skipped).
// Returns this thread's deleted core bits (of the box's core only).
template <int UW>
__device__ uint32_t res_pass2d(const Box2D &b, int q, int *take, unsigned long long *words)
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
        const int x0 = 1 + UW * c;
        const int r = kUnitRows * s - 4 + lane;  // box row of this lane
        const bool valid = r >= 0 && r < b.nrows;
        const uint32_t *in = (valid ? IN + (size_t)r * b.pp : b.zero) + x0;
        uint32_t v[UW + 1];
#pragma unroll
        for (int k = 0; k < UW; k++) v[k] = in[k];
        v[UW] = (in[-1] & 0xFFFF0000u) | (in[UW] & 0xFFFFu);
        subit2d_ring<UW, 0, false>(v);
        subit2d_ring<UW, 1, false>(v);
        subit2d_ring<UW, 2, false>(v);
        subit2d_ring<UW, 3, true>(v);
        uint32_t chg = 0, lft = 0, rgt = 0;
        if (valid && lane >= 4 && lane < 28) {
            uint32_t *out = OUT + (size_t)r * b.pp + x0;
            const int klo = b.wlo - UW * c, khi = b.whi - UW * c;
            uint32_t cc = 0;
#pragma unroll
            for (int k = 0; k < UW; k++) {
                const uint32_t d = v[k] ^ in[k];
                chg |= d;
                if (k >= klo && k < khi) cc |= d;
                if (k == 0) lft = d & 0xFu;                 // within 4 pixels of the left edge
                if (k == UW - 1) rgt = d & 0xF0000000u;     // ... of the right edge
                out[k] = v[k];
            }
            if (r >= b.rlo && r < b.rhi) core |= cc;
        }
        // The next pass of a neighbour depends on this unit only through the
        // 4 pixels next to their common border (four subiterations reach 4
        // pixels): activate the neighbours whose border band changed
        // (border bands, as the tile engine does).
        const unsigned m_any = __ballot_sync(kFull, chg != 0u);
        if (m_any) {
            const unsigned m_l = __ballot_sync(kFull, lft != 0u), m_r = __ballot_sync(kFull, rgt != 0u);
            // lanes holding the first and last 4 core rows
            constexpr unsigned band_top = 0xF0u, band_bot = 0x0F000000u;
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
            *words += (unsigned long long)min(kUnitRows, b.nrows - kUnitRows * s) * min(UW, b.wl - UW * c);
    }
    return core;
}

// Bound: in a large batch the ALU (13 half-rate operations per word step) and
// the passes' tails; for a lone image the latency of its passes (1.5 us each
// in a box of a 512^2 image) and meetings (4 us with the exchange).  Boxes of
// rows and words against bands of full-width rows: a 4096^2 image 127 -> 102 us,
// a 1501 x 1003 float image 154 -> 92 us, a 512^2 one 59 -> 43 us, the mixed
// batch (with the exchange flattened over the threads) 1.24 -> 1.19 ms.
//
// One image, or one box of it: rows [r0, r1) of words [c0, c1) are the core;
// `halo` rows above and below it and one word left and right (clamped to the
// image) are held too.  Boxes run passes in lockstep and meet after every
// halo / 4-th one: then a box writes the edge of its core to global memory,
// meets the others, stops if no box's core changed in that pass, and reads
// its halo.  Wrong values entering at a box's outer edge move at most 4 rows
// or pixels per pass, so halo rows (and the 32 pixels of a word, for up to 8
// passes) keep the core exact; if a pass before the meeting was a fixed point
// already, the one at the meeting is too.
template <int UW>
__device__ void res_run2d(Inst &in, const ResIO &io, const ResItem &it, uint32_t *sm, ResSched *S, int *take)
{
    __shared__ int s_flag;
    const int lane = threadIdx.x & 31;
    const int wl_img = (in.W + 31) >> 5;
    const int a = max(0, it.r0 - it.halo), e0 = it.halo ? max(0, it.c0 - 1) : 0;  // first row and word held
    const int aend = min(in.H, it.r1 + it.halo), e1 = it.halo ? min(wl_img, it.c1 + 1) : wl_img;
    Box2D b;
    b.wl = e1 - e0;
    b.pp = res_pitch2d(b.wl, UW);
    b.nchunks = (b.wl + UW - 1) / UW;
    b.nrows = aend - a;
    b.nstrips = (b.nrows + kUnitRows - 1) / kUnitRows;
    b.rlo = it.r0 - a;
    b.rhi = it.r1 - a;
    b.wlo = it.c0 - e0;
    b.whi = it.c1 - e0;
    b.zero = sm;
    b.buf0 = sm + b.pp;
    b.buf1 = b.buf0 + (size_t)b.nrows * b.pp;
    b.until = reinterpret_cast<int *>(b.buf1 + (size_t)b.nrows * b.pp);
    const int pp = b.pp;
    const int nunits = b.nstrips * b.nchunks;

    // zero row and row copies (their words left and right of the box stay zero)
    {
        const int total = pp * (1 + 2 * b.nrows);
        for (int i = threadIdx.x; i < total / 4; i += kResThreads)
            reinterpret_cast<uint4 *>(sm)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (threadIdx.x < (total & 3)) sm[(total & ~3) + threadIdx.x] = 0u;
    }
    for (int i = threadIdx.x; i < nunits; i += kResThreads) b.until[i] = -1;
    if (threadIdx.x < 2) take[threadIdx.x] = 0;
    __syncthreads();
    res_load(in, io, WordWalk(b.wl, b.nrows), b.nrows * b.wl, e0, a, 0, [&](bool, const WordPos &q, uint32_t v) {
        if (!v) return;
        const int w = q.y * pp + q.x + 1;
        b.buf0[w] = v;
        b.buf1[w] = v;
        // units holding foreground start active
        b.until[(q.y / kUnitRows) * b.nchunks + q.x / UW] = 0;
    });
    __syncthreads();

    int result = 0;  // 1 converged, -1 pass cap or failed wait
    MeetState meet;
    unsigned long long words = 0;
    const int period = it.halo / 4;
    int q = 0, since = 0, e = 0;  // pass, passes since the last meeting, meetings
    for (;; q++) {
        // the counter of this pass was cleared during the previous one;
        // clear the next one's (nobody uses it before the barrier below)
        if (threadIdx.x == 0) take[(q + 1) & 1] = 0;
        const uint32_t core = res_pass2d<UW>(b, q, take + (q & 1), &words);
        const bool any = __syncthreads_or(core != 0u);
        if (it.bands == 1) {
            if (!any) {
                result = 1;
                break;
            }
        } else if (++since == period) {
            since = 0;
            uint32_t *cur = (q & 1) ? b.buf0 : b.buf1;
            uint32_t *gx = in.buf[(e + 1) & 1];  // buf[0] may hold the start state other boxes still load
            // the edge of the core: its first and last `halo` rows, its first and last words
            const int cw = it.c1 - it.c0, ch = it.r1 - it.r0;
            const int top = it.r0 > 0 ? min(it.halo, ch) : 0, bot = it.r1 < in.H ? min(it.halo, ch - top) : 0;
            for (int i = threadIdx.x; i < (top + bot) * cw; i += kResThreads) {
                const int r = i / cw, w = it.c0 + i - r * cw, y = r < top ? it.r0 + r : it.r1 - bot + (r - top);
                gx[(size_t)y * in.P + w] = cur[(y - a) * pp + 1 + w - e0];
            }
            for (int i = threadIdx.x; i < 2 * ch; i += kResThreads) {
                const int y = it.r0 + (i >> 1), w = (i & 1) ? it.c1 - 1 : it.c0;
                if ((i & 1) ? it.c1 < wl_img : it.c0 > 0) gx[(size_t)y * in.P + w] = cur[(y - a) * pp + 1 + w - e0];
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
            e++;
            // the halo: a word that changed makes its unit, and the units it is within 4 pixels of, active
            auto take_over = [&](int y, int w, uint32_t v) {
                const int r = y - a, x = w - e0;
                uint32_t *p = cur + r * pp + 1 + x;
                if (*p == v) return;
                *p = v;
                const int s = r / kUnitRows, c = x / UW, rr = r - s * kUnitRows, cc = x - c * UW;
                for (int dy = rr < 4 && s > 0 ? -1 : 0; dy <= (rr >= kUnitRows - 4 && s + 1 < b.nstrips ? 1 : 0); dy++)
                    for (int dx = cc == 0 && c > 0 ? -1 : 0; dx <= (cc == UW - 1 && c + 1 < b.nchunks ? 1 : 0); dx++)
                        b.until[(s + dy) * b.nchunks + c + dx] = q + 1;
            };
            const int htop = it.r0 - a, hrows = htop + (aend - it.r1);
            for (int i = threadIdx.x; i < hrows * b.wl; i += kResThreads) {
                const int r = i / b.wl, w = e0 + i - r * b.wl, y = r < htop ? a + r : it.r1 + (r - htop);
                take_over(y, w, __ldcg(gx + (size_t)y * in.P + w));
            }
            for (int i = threadIdx.x; i < 2 * ch; i += kResThreads) {
                const int y = it.r0 + (i >> 1), w = (i & 1) ? it.c1 : e0;
                if ((i & 1) ? e1 > it.c1 : e0 < it.c0) take_over(y, w, __ldcg(gx + (size_t)y * in.P + w));
            }
            __syncthreads();
        }
        if (q >= in.pass_cap) {
            if (threadIdx.x == 0) atomicOr(&S->status, kErrPassLimit);
            result = -1;
            break;
        }
    }
    // the converged core (in buf[(q+1)&1])
    __syncthreads();
    const uint32_t *fin = ((q & 1) ? b.buf0 : b.buf1) + (size_t)b.rlo * pp + 1 + b.wlo;
    res_store(in, io, it.c0, it.c1, it.r1 - it.r0, 1, it.r0, 0, [&](int y, int) { return fin + (size_t)y * pp; });
    if (lane == 0 && words) atomicAdd(&in.work_words, words);  // words per pass (one iteration)
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
    res_load(in, io, walk, nbox, 0, y0, z0, [&](bool, const WordPos &q, uint32_t v) {
        const int d = dist_of(q), idx = v ? index_of(q) : 0;
        if (v) b.state[idx] = v;
        const int pos = warp_append(v != 0u && d <= 5, &s_n[0]);
        if (pos >= 0 && pos < list_cap) list[pos] = (uint32_t)idx | (uint32_t)(q.x >> xs) << 16 | (uint32_t)d << 21;
    });
    __syncthreads();
    const int nl = s_n[0];
    MeetState meet;
    // more non-empty words than the lists hold: go over all words of the box
    const bool dense = off + (size_t)nl * kBoxListBytes + 64 > (size_t)kSmemBytes;
    b.cidx = list + nl;
    b.cU = b.cidx + nl;
    b.cdel = b.cU + nl;
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
            uint32_t un[kDenseWords], del[kDenseWords];  // of this thread's words
            WordPos q = walk.first();
            int k = 0;
            for (int i = threadIdx.x; i < nbox; i += kResThreads, walk.next(q), k++) {
                const int d = dist_of(q);
                const uint32_t *s = b.state + index_of(q);
                un[k] = del[k] = 0;
                if (d <= 5 && *s && ((act[(q.z + 1) * ny2 + q.y + 1] >> (q.x >> xs)) & 1u)) {
                    uint32_t g[27];
                    box_window(s, b.p, b.ps, g);
                    const uint32_t du = rule3d<0>(g) & g[13];
                    del[k] = du;
                    un[k] = (du | rule3d<1>(g) | rule3d<2>(g) | rule3d<3>(g) | rule3d<4>(g) | rule3d<5>(g)) & g[13];
                    words += d == 0;
                    entries++;
                }
            }
            __syncthreads();
#pragma unroll 1
            for (int j = 0; j < 6; j++) {
                // deletions of subiteration j were found: apply them, then find the next one's
                q = walk.first();
                k = 0;
                for (int i = threadIdx.x; i < nbox; i += kResThreads, walk.next(q), k++)
                    if (del[k]) b.state[index_of(q)] &= ~del[k];
                __syncthreads();
                if (j == 5) break;
                q = walk.first();
                k = 0;
                for (int i = threadIdx.x; i < nbox; i += kResThreads, walk.next(q), k++) {
                    del[k] = 0;
                    if (!un[k] || dist_of(q) > 4 - j) continue;
                    const uint32_t *s = b.state + index_of(q);
                    const uint32_t cand = *s & un[k];
                    if (!cand) continue;
                    uint32_t g[27];
                    box_window(s, b.p, b.ps, g);
                    del[k] = cand & (j == 0   ? rule3d<1>(g)
                                     : j == 1 ? rule3d<2>(g)
                                     : j == 2 ? rule3d<3>(g)
                                     : j == 3 ? rule3d<4>(g)
                                              : rule3d<5>(g));
                    words += dist_of(q) == 0;
                }
                __syncthreads();
            }
            // only voxels of the union were deleted: a word changed when it lost some of its union
            q = walk.first();
            k = 0;
            for (int i = threadIdx.x; i < nbox; i += kResThreads, walk.next(q), k++) {
                const int idx = index_of(q);
                if (!(un[k] & ~b.state[idx]) || dist_of(q) != 0) continue;
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
            // kWarps / 8 warps per neighbouring box take over its messages
            const int k8 = warp & 7, k9 = k8 < 4 ? k8 : k8 + 1;
            const int nbz = bz + k9 / 3 - 1, nby = by + k9 % 3 - 1;
            if (warp < kWarps / 8 * 8 && nbz >= 0 && nbz < gz && nby >= 0 && nby < gy) {
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
    res_store(in, io, 0, wl, it.c1 - it.c0, it.r1 - it.r0, it.c0, it.r0, [&](int y, int z) {
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
        if (in.dims == 2) {
            const int wl = (in.W + 31) >> 5;
            const int nw = it.halo ? min(wl, it.c1 + 1) - max(0, it.c0 - 1) : wl;
            const int nr = min(in.H, it.r1 + it.halo) - max(0, it.r0 - it.halo);
            uint32_t *sm = reinterpret_cast<uint32_t *>(res_smem);
            switch (res_unit_words(nr, nw)) {
            case 2: res_run2d<2>(in, io, it, sm, S, s_take); break;
            case 4: res_run2d<4>(in, io, it, sm, S, s_take); break;
            default: res_run2d<8>(in, io, it, sm, S, s_take); break;
            }
        } else
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
