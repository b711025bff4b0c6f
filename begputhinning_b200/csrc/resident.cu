// resident.cu -- the resident engine: every work item (an instance, or one
// box of it) is loaded once into one
// CTA's shared memory and thinned there from its first subiteration to its
// fixed point; only the boxes of a large image (every few iterations) and of
// a large volume (every iteration) meet to trade their edges through global
// memory.
// One CTA of 768 threads per SM holds up to 225 KB (measured against two
// CTAs of 384 threads with 111 KB each: larger boxes won).
//
// 2D image (dense).  The rows of the image, or of a box of it (core plus halo),
// lie twice in shared memory (pass q reads one copy and writes the other) with
// an odd pitch and zero words left and right of every row.  A pass hands units
// (24 rows x 2, 4 or 8 words) to warps dynamically; words whose surroundings
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
// non-empty words than the lists hold looks for candidates among all of its
// words instead.
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
// than its lists hold has the candidates of an iteration in that room; where even
// they do not fit, it goes over all of its words, at most kDenseWords per
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

int res_words3d(int W) { return (W + 29) / 30; }

bool res_fits3d(int W, int ny, int nz)
{
    const int wl = res_words3d(W);
    const double held = (double)(((ny + 2) * (wl | 1)) | 1) * (nz + 2), words = (double)wl * ny * nz;
    const double rows2 = (double)((ny + 5) & ~3) * (nz + 2);
    // words are indexed by 16 bits
    return held < 65535 && words <= (double)kDenseWords * kResThreads &&
           held * 4 + rows2 * 2 + kListFill * words * kBoxListBytes + 128 <= (double)kSmemBytes;
}

// ------------------------------------------------------------ helpers -----
extern __shared__ __align__(16) uint8_t res_smem[];  // dynamic shared memory of the CTA

// The CTAs of one image meet for the k-th time: each adds 1 to the low half
// of meet[k & 1], and 1 to its high half when something of its own changed
// since the last meeting; the wait (bounded) ends when all `bands` arrived.
// Two words in turn, so that a CTA that is already at the next meeting leaves
// what a late one reads here alone (it cannot get to the one after that).
// One thread per CTA calls it, after a __syncthreads that follows the CTA's
// writes to global memory.  Returns 0 when nobody changed anything, 1 when
// somebody did, 2 when the wait ran out.
struct MeetState {
    unsigned k, seen0, seen1;  // meetings so far, high halves after the last one of either word
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

// put(pos, word) for every word (W30: the 30-voxel words of full rows, see the
// 3D section) of the grid of rows whose first word, row and
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
template <bool W30, class Put>
__device__ __forceinline__ void res_load(const Inst &in, const ResIO &io, const WordWalk &walk, int n, int x0, int y0, int z0,
                                         Put put)
{
    if (!io.pix) {
        const uint32_t *g = in.buf[0];
        const int H = in.H, P = in.P;
        res_load_loop<4>(walk, n, [&](bool live, const WordPos &q) {
            if (!live) return 0u;
            const uint32_t *r = g + ((size_t)(z0 + q.z) * H + (y0 + q.y)) * P;
            if (!W30) return __ldcg(r + x0 + q.x);
            if (q.x == 0) return __ldcg(r) << 1;
            const int x = 30 * q.x - 1, j = x >> 5;
            return __funnelshift_r(__ldcg(r + j), j + 1 < P ? __ldcg(r + j + 1) : 0u, x & 31);
        }, put);
        return;
    }
    const IODesc &d = *io.d;
    const int inW = d.inW, inH = d.inH, inD = d.inD;
    // first pixel and number of pixels of a word; a row's first 30-voxel word starts one pixel late
    auto count = [&](bool live, const WordPos &q, uint32_t &off) {
        const bool late = W30 && q.x == 0;
        const int x = late ? 0 : W30 ? 30 * q.x - 1 : 32 * (x0 + q.x), y = y0 + q.y, z = z0 + q.z;
        off = ((uint32_t)z * (uint32_t)inH + (uint32_t)y) * (uint32_t)inW + (uint32_t)x;
        return live && y < inH && z < inD ? max(0, min(late ? 31 : 32, inW - x)) : 0;
    };
    auto place = [&](const WordPos &q, uint32_t w) { return W30 && q.x == 0 ? w << 1 : w; };
    if (dtype_bytes(d.dtype) == 1) {
        const uint32_t neg = pixel_neg(d);
        res_load_loop<2>(walk, n, [&](bool live, const WordPos &q) {
            uint32_t off;
            const int cnt = count(live, q, off);
            return place(q, pixel_bytes(d, off, cnt, neg));
        }, put);
    } else {
        res_load_loop<1>(walk, n, [&](bool live, const WordPos &q) {
            uint32_t off;
            const int cnt = count(live, q, off);
            return place(q, pixel_word_wide(d, off, cnt));
        }, put);
    }
}

// The way back for words [x0, x1) of rows [y0, y0 + ny) of planes [z0, z0 + nz):
// bits(y, z, x) = 32 pixels from the x-th one on of grid row y of grid plane z
// (what lies past the row's last pixel, or word x1, does not matter).
template <class Bits>
__device__ __forceinline__ void res_store(const Inst &in, const ResIO &io, int x0, int x1, int ny, int nz, int y0,
                                          int z0, Bits bits)
{
    const int lane = threadIdx.x & 31, wl = x1 - x0;
    const WordWalk walk(wl, ny);
    const int n = nz * ny * wl;
    if (!io.pix || !io.d->out) {
        uint32_t *g = in.buf[0];
        WordPos q = walk.first();
        for (int i = threadIdx.x; i < n; i += kResThreads, walk.next(q)) {
            const int left = in.W - 32 * (x0 + q.x);  // pixels from the word's first one on
            const uint32_t w = bits(q.y, q.z, 32 * q.x);
            g[((size_t)(z0 + q.z) * in.H + (y0 + q.y)) * in.P + x0 + q.x] = left >= 32 ? w : w & ((1u << left) - 1u);
        }
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
            pixel_chunk(out, (uint32_t)ny, in.W, d.dW, i - z * per,
                        [&](uint32_t r, int x) { return bits((int)r, (int)z, x); });
        }
        return;
    }
    if (dtype_bytes(d.dtype) == 1) {
        // parts of rows: a run per row (wl + 1 aligned chunks hold it)
        const WordWalk chunks(wl + 1, ny);
        WordPos q = chunks.first();
        for (int i = threadIdx.x; i < nz * ny * (wl + 1); i += kResThreads, chunks.next(q)) {
            uint8_t *out = (uint8_t *)d.out + ((size_t)(z0 + q.z) * in.H + (y0 + q.y)) * in.W + 32 * x0;
            pixel_run_chunk(out, np, (uint32_t)q.x, [&](int x) { return bits(q.y, q.z, x); });
        }
        return;
    }
    WordPos q = walk.first();
    for (int i = threadIdx.x; i - lane < n; i += kResThreads, walk.next(q)) {
        const bool live = i < n;
        const int x = 32 * (x0 + q.x);
        const uint32_t off = ((uint32_t)(z0 + q.z) * (uint32_t)in.H + (uint32_t)(y0 + q.y)) * (uint32_t)in.W + (uint32_t)x;
        pixel_store_wide(d, off, live ? min(32, in.W - x) : 0, live ? bits(q.y, q.z, 32 * q.x) : 0u);
    }
}

// An item is done: its outcome and work (words and tiles: this thread's share)
// go to its record, and the last CTA of an instance clears the meetings for
// the next run.  All threads call it; ends with a barrier.
__device__ void res_done(Inst &in, const ResItem &it, int result, int passes, unsigned long long words,
                         unsigned long long tiles, ResTrace *tr)
{
    __shared__ unsigned long long s_work[2];
    if (threadIdx.x < 2) s_work[threadIdx.x] = 0;
    __syncthreads();
    // one add per warp: a 64-bit add to shared memory is a loop that 768 threads would take 40 us for
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        words += __shfl_xor_sync(kFull, words, o);
        tiles += __shfl_xor_sync(kFull, tiles, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&s_work[0], words);
        atomicAdd(&s_work[1], tiles);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        tr->result = result;
        tr->passes = passes;
        tr->words = s_work[0];
        tr->tiles = s_work[1];
        if (it.bands > 1 && atomicAdd(&in.res_left, 1) == it.bands - 1) {
            in.res_meet[0] = in.res_meet[1] = 0;
            in.res_left = 0;
            in.res_run++;
        }
    }
    __syncthreads();
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

// One subiteration on the ring of UW core words and the halo word v[UW], for
// the active words only (bits of `act`, the same in every lane; a pair at a
// time, so that two chains of operations overlap).  The last
// subiteration leaves the halo word alone.
template <int UW, int DIR, bool LAST>
__device__ __forceinline__ void subit2d_ring(uint32_t (&v)[UW + 1], uint32_t act)
{
    const uint32_t first = v[0];
    uint32_t prev = v[UW];
#pragma unroll
    for (int j = 0; j < UW; j += 2) {
        const uint32_t o0 = v[j], o1 = v[j + 1], on = v[j + 2];
        if (act & (3u << j)) {
            v[j] = word2d<DIR>(o0, o1, prev);
            v[j + 1] = word2d<DIR>(o1, on, o0);
        }
        prev = o1;
    }
    if constexpr (!LAST) {
        const uint32_t o = v[UW];
        if (act & (1u << UW)) v[UW] = word2d<DIR>(o, first, prev);
    }
}

struct Box2D {
    uint32_t *zero;         // pp zero words
    uint32_t *buf0, *buf1;  // nrows x pp each: pass q reads buf[q & 1], writes buf[(q + 1) & 1]
    uint32_t *act;          // [nstrips][nchunks]: the unit's active words, bit k (pass q even) or
                            // 16 + k (odd) for word k
    int pp, wl, nrows, nstrips, nchunks;
    int rlo, rhi;           // core rows and words, within the box
    int wlo, whi;
};

// One pass q over the box's units.  Word k of a unit is active when the
// previous pass deleted something in it or within 4 pixels or rows of it (one
// subiteration of every direction reaches that far).  The others, and the
// words next to them as far as the pass looks, are a fixed point: no
// subiteration of the pass changes them, and both copies hold them already.
// A pass that deletes something in a word makes the word active in the next
// one, and each of its eight neighbours within 4 pixels or rows of the deletions.
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
        const int sh = (q & 1) * 16;
        const uint32_t act = (b.act[u] >> sh) & 0xffu;
        if (!act) continue;
        __syncwarp();
        if (lane == 0) atomicAnd(b.act + u, 0xffff0000u >> sh);  // for pass q + 2
        const int s = u / b.nchunks, c = u - s * b.nchunks;
        const int x0 = 1 + UW * c;
        const int r = kUnitRows * s - 4 + lane;  // box row of this lane
        const bool valid = r >= 0 && r < b.nrows;
        const uint32_t *in = (valid ? IN + (size_t)r * b.pp : b.zero) + x0;
        uint32_t v[UW + 1];
#pragma unroll
        for (int k = 0; k < UW; k++) v[k] = in[k];
        v[UW] = (in[-1] & 0xFFFF0000u) | (in[UW] & 0xFFFFu);
        // active words that are not empty by now, and the halo word where a word next to it is one
        uint32_t some = v[UW] ? 1u << UW : 0u;
#pragma unroll
        for (int k = 0; k < UW; k++) some |= v[k] ? 1u << k : 0u;
        some = __reduce_or_sync(kFull, some);
        const uint32_t m = some & ((some & act & (1u | 1u << (UW - 1))) ? act | 1u << UW : act);
        subit2d_ring<UW, 0, false>(v, m);
        subit2d_ring<UW, 1, false>(v, m);
        subit2d_ring<UW, 2, false>(v, m);
        subit2d_ring<UW, 3, true>(v, m);
        uint32_t chg = 0;  // bit 1 + k: word k to be active for the rows around, 0 and 1 + UW: the words left and right
        if (valid && lane >= 4 && lane < 28) {
            uint32_t *out = OUT + (size_t)r * b.pp + x0;
            const int klo = b.wlo - UW * c, khi = b.whi - UW * c;
            uint32_t cc = 0;
#pragma unroll
            for (int k = 0; k < UW; k++) {
                if (!(act & (1u << k))) continue;
                const uint32_t d = v[k] ^ in[k];
                if (d) chg |= 2u << k;
                if (d & 0xFu) chg |= 1u << k;
                if (d & 0xF0000000u) chg |= 4u << k;
                if (k >= klo && k < khi) cc |= d;
                out[k] = v[k];
            }
            if (r >= b.rlo && r < b.rhi) core |= cc;
        }
        // what changed in any row, in the first four and in the last four: ten bits each
        chg = __reduce_or_sync(kFull, chg | (lane < 8 ? chg << 10 : 0u) | (lane >= 24 ? chg << 20 : 0u));
        if (chg && lane < 9) {
            const int dy = lane / 3 - 1, dx = lane % 3 - 1;
            const uint32_t f = (chg >> (dy < 0 ? 10 : dy > 0 ? 20 : 0)) & 0x3ffu;
            const uint32_t on = dx < 0 ? (f & 1u) << (UW - 1) : dx > 0 ? f >> (UW + 1) : (f >> 1) & ((1u << UW) - 1u);
            const int ns = s + dy, nc = c + dx;
            if (on && ns >= 0 && ns < b.nstrips && nc >= 0 && nc < b.nchunks)
                atomicOr(b.act + ns * b.nchunks + nc, on << (16 - sh));
        }
        if (lane == 0)
            *words += (unsigned long long)min(kUnitRows, b.nrows - kUnitRows * s) * __popc(m & ((1u << UW) - 1u));
    }
    return core;
}

// Bound: in a large batch the latency of a word step's chain (6 warps per
// scheduler issue on half of the cycles, the ALU is half busy) and the
// passes' tails (27 % of the warps' time); for a lone image the latency of its passes (1.5 us each
// in a box of a 512^2 image) and meetings (4 us with the exchange).  Boxes of
// rows and words against bands of full-width rows: a 4096^2 image 127 -> 102 us,
// a 1501 x 1003 float image 154 -> 92 us, a 512^2 one 59 -> 43 us, the mixed
// batch (with the exchange flattened over the threads) 1.24 -> 1.19 ms.
// Words active one by one against whole units with a vote per pair and
// subiteration: 4096^2 103 -> 97 us, 16 images of 1024^2 121 -> 117 us, the
// mixed batch 1.19 -> 1.17 ms (a branch per word instead of per pair: 1.21 ms;
// 1024 threads: 1.18 ms).
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
__device__ void res_run2d(Inst &in, const ResIO &io, const ResItem &it, uint32_t *sm, ResSched *S, int *take,
                          ResTrace *tr)
{
    __shared__ int s_flag;
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
    b.act = b.buf1 + (size_t)b.nrows * b.pp;
    const int pp = b.pp;
    const int nunits = b.nstrips * b.nchunks;

    // zero row and row copies (their words left and right of the box stay zero)
    {
        const int total = pp * (1 + 2 * b.nrows);
        for (int i = threadIdx.x; i < total / 4; i += kResThreads)
            reinterpret_cast<uint4 *>(sm)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (threadIdx.x < (total & 3)) sm[(total & ~3) + threadIdx.x] = 0u;
    }
    for (int i = threadIdx.x; i < nunits; i += kResThreads) b.act[i] = 0;
    if (threadIdx.x < 2) take[threadIdx.x] = 0;
    __syncthreads();
    res_load<false>(in, io, WordWalk(b.wl, b.nrows), b.nrows * b.wl, e0, a, 0, [&](bool, const WordPos &q, uint32_t v) {
        if (!v) return;
        const int w = q.y * pp + q.x + 1;
        b.buf0[w] = v;
        b.buf1[w] = v;
        // words with foreground start active, in the units within 4 rows of it
        const int s = q.y / kUnitRows, rr = q.y - s * kUnitRows, c = q.x / UW;
        volatile uint32_t *act = b.act + s * b.nchunks + c;
        const uint32_t bit = 1u << (q.x - c * UW);
        if (!(*act & bit)) atomicOr((uint32_t *)act, bit);
        if (rr < 4 && s > 0 && !(act[-b.nchunks] & bit)) atomicOr((uint32_t *)act - b.nchunks, bit);
        if (rr >= kUnitRows - 4 && s + 1 < b.nstrips && !(act[b.nchunks] & bit)) atomicOr((uint32_t *)act + b.nchunks, bit);
    });
    __syncthreads();

    int result = 0;  // 1 converged, -1 pass cap or failed wait
    MeetState meet{0, 0, 0};
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
            // the halo: a word that changed becomes active, and the words it is within 4 pixels or rows of
            auto take_over = [&](int y, int w, uint32_t v) {
                const int r = y - a, x = w - e0;
                uint32_t *p = cur + r * pp + 1 + x;
                const uint32_t d = *p ^ v;
                if (!d) return;
                *p = v;
                const int s = r / kUnitRows, rr = r - s * kUnitRows;
                const int s0 = rr < 4 && s > 0 ? s - 1 : s, s1 = rr >= kUnitRows - 4 && s + 1 < b.nstrips ? s + 1 : s;
                const int x0 = (d & 0xFu) && x > 0 ? x - 1 : x, x1 = (d & 0xF0000000u) && x + 1 < b.wl ? x + 1 : x;
                for (int t = s0; t <= s1; t++)
                    for (int k = x0; k <= x1; k++)
                        atomicOr(b.act + t * b.nchunks + k / UW, 1u << ((q & 1 ? 0 : 16) + k % UW));
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
    res_store(in, io, it.c0, it.c1, it.r1 - it.r0, 1, it.r0, 0, [&](int y, int, int x) {
        const uint32_t *s = fin + y * pp + (x >> 5);
        return __funnelshift_r(s[0], s[1], x & 31);
    });
    res_done(in, it, result, q + 1, words, threadIdx.x == 0, tr);
}

// ------------------------------------------------------------ 3D ----------
// Entry of a box's word list: word index in shared memory (16 bits), its
// column in the rows' change masks (3 bits), its distance from the box's core
// (3 bits, 0 = core), whether its row goes on to its left and right, and, in
// the candidate list, whether it changed.
constexpr uint32_t kEntChanged = 1u << 24, kEntLeft = 1u << 25, kEntRight = 1u << 26;
__device__ __forceinline__ uint32_t ent_idx(uint32_t e) { return e & 0xffffu; }
__device__ __forceinline__ uint32_t ent_col(uint32_t e) { return (e >> 16) & 7u; }
__device__ __forceinline__ int ent_dist(uint32_t e) { return (int)((e >> 21) & 7u); }

// Words of a 3D box hold 30 voxels: bit 1 + k of word j is voxel x = 30 j + k, and
// bits 0 and 31 repeat the voxels next to them, which are the neighbouring
// words' bits 30 and 1.  A word's 3x3x3 neighbourhood is then 9 words of
// shared memory instead of 27 (whose loads, at two to four lanes per bank, set
// the time of a subiteration), and a deletion at either end of a word is
// applied to the neighbour's copy as well.
constexpr int kVox = 30;
constexpr uint32_t kCoreBits = 0x7FFFFFFEu;

// Everything about the box that all threads share lies in shared memory and is
// read where it is needed: at 80 registers a thread, 27 of them the window,
// values kept over an iteration would be spilled to local memory, and every
// acquire of a meeting empties the L1 that holds the spills.
struct Box3D {
    ResItem it;
    int H, D, wl;              // volume rows, planes; words per row
    int y0, y1, z0, z1;        // rows and planes held
    int p, ps;                 // words between rows, between planes
    uint32_t mp, mps;          // reciprocals of p and ps: see box_plane_row
    int my, mrows;             // rows of the masks: per plane (a multiple of 4), in all
    int xs;                    // words per column of the masks: 1 << xs
    int act, chg, list;        // offsets of the masks and of the word list
    int nl;                    // its length (0: the box goes over all of its words)
    int cand, cap;             // offset of the candidates' lists, candidates they hold
    int gy, gz, by, bz;        // boxes along y and z; this box
    int stride;                // messages a box may send
    uint4 *msgs, *heads;
    unsigned run;              // tags of this run's messages and headers
    int n[4];                  // lengths: word list, active words, candidates, messages
    int flag;
};

__device__ __forceinline__ uint32_t *box_state() { return reinterpret_cast<uint32_t *>(res_smem); }
__device__ __forceinline__ uint32_t *box_words(int off) { return reinterpret_cast<uint32_t *>(res_smem + off); }
// the candidates' entries, unions and deletions, one list behind the other
__device__ __forceinline__ uint32_t *box_cand(const Box3D &v, int k) { return box_words(v.cand) + k * v.cap; }

// Plane and row of a word, padding included.  n / d = mulhi(2 n, m) with
// m = ceil(2^31 / d) = (2^31 + e) / d, e < d: the product exceeds n / d by
// n e / (d 2^31), less than 1 / d for n < 2^16 and d <= 2^15 (a box has fewer than
// 2^16 words in at least three planes of at least three rows).  2^31 and not
// 2^32, whose quotient by 1 (rows of one word) does not fit 32 bits.
__device__ __forceinline__ uint32_t box_plane_row(const Box3D &v, uint32_t idx, uint32_t &y2)
{
    const uint32_t z2 = __umulhi(2 * idx, v.mps);
    y2 = __umulhi(2 * (idx - z2 * (uint32_t)v.ps), v.mp);
    return z2;
}
__device__ __forceinline__ int box_index(const Box3D &v, const WordPos &q)
{
    return (q.z + 1) * v.ps + (q.y + 1) * v.p + q.x;
}
__device__ __forceinline__ int box_dist(const Box3D &v, const WordPos &q)
{
    const int y = v.y0 + q.y, z = v.z0 + q.z;
    return max(max(max(v.it.c0 - y, y - v.it.c1 + 1), max(v.it.r0 - z, z - v.it.r1 + 1)), 0);
}
__device__ __forceinline__ uint32_t box_entry(const Box3D &v, const WordPos &q, int idx, int d)
{
    return (uint32_t)idx | (uint32_t)(q.x >> v.xs) << 16 | (uint32_t)d << 21 | (q.x > 0 ? kEntLeft : 0u) |
           (q.x + 1 < v.wl ? kEntRight : 0u);
}
__device__ __forceinline__ void box_mark(const Box3D &v, int row, int col)
{
    atomicOr(box_words(v.chg) + (row >> 2), 1u << (8 * (row & 3) + col));
}
// a word of the core changed: mark it, and tell the boxes around when it lies near the core's edge
__device__ __forceinline__ void box_changed(Box3D &v, uint32_t idx, uint32_t col, int iter)
{
    uint32_t y2;
    const uint32_t z2 = box_plane_row(v, idx, y2);
    box_mark(v, (int)(z2 * (uint32_t)v.my + y2), (int)col);
    if (v.it.bands == 1) return;
    const int y = v.y0 + (int)y2 - 1, z = v.z0 + (int)z2 - 1, h = v.it.halo;
    if ((v.it.r0 > 0 && z < v.it.r0 + h) || (v.it.r1 < v.D && z >= v.it.r1 - h) || (v.it.c0 > 0 && y < v.it.c0 + h) ||
        (v.it.c1 < v.H && y >= v.it.c1 - h)) {
        const int x = (int)idx - (int)z2 * v.ps - (int)y2 * v.p;
        uint4 *msg = v.msgs + ((size_t)(iter & 1) * v.it.bands + v.it.band) * v.stride;
        st_relaxed128(msg + atomicAdd(&v.n[3], 1),
                      make_uint4(((uint32_t)z * (uint32_t)v.H + (uint32_t)y) * (uint32_t)v.wl + (uint32_t)x,
                                 box_state()[idx], v.run, (uint32_t)iter + 1u));
    }
}

// The 3x3x3 neighbourhood of the word at s; returns its own voxels.
__device__ __forceinline__ uint32_t box_window(const uint32_t *s, int p, int ps, uint32_t (&g)[27])
{
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const uint32_t c = s[(k / 3 - 1) * ps + (k % 3 - 1) * p];
        g[3 * k] = c << 1;
        g[3 * k + 1] = c;
        g[3 * k + 2] = c >> 1;
    }
    return g[13] & kCoreBits;
}

// Delete voxels of the word of entry e (other threads may do so to the copies in it).
__device__ __forceinline__ void box_delete(uint32_t e, uint32_t del)
{
    uint32_t *s = box_state() + ent_idx(e);
    atomicAnd(s, ~del);
    if ((del & 2u) && (e & kEntLeft)) atomicAnd(s - 1, ~(1u << 31));
    if ((del & (1u << kVox)) && (e & kEntRight)) atomicAnd(s + 1, ~1u);
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
__device__ __forceinline__ uint32_t box_deletions(const Box3D &v, uint32_t e, uint32_t un)
{
    const uint32_t *s = box_state() + ent_idx(e);
    if (ent_dist(e) > 5 - J || !(*s & un)) return 0u;
    uint32_t g[27];
    return box_window(s, v.p, v.ps, g) & un & rule3d<J>(g);
}

// ... with any number of candidates per thread
template <int J>
__device__ __forceinline__ void box_subiteration(const Box3D &v, int nc, unsigned &words)
{
    bool any = false;
    for (int c = threadIdx.x; c < nc; c += kResThreads) {
        const uint32_t e = box_cand(v, 0)[c];
        const uint32_t del = box_deletions<J>(v, e, box_cand(v, 1)[c]);
        words += ent_dist(e) == 0;
        any |= del != 0u;
        box_cand(v, 2)[c] = del;
    }
    if (!__syncthreads_or(any)) return;
    for (int c = threadIdx.x; c < nc; c += kResThreads) {
        const uint32_t del = box_cand(v, 2)[c];
        if (del) {
            const uint32_t e = box_cand(v, 0)[c];
            box_delete(e, del);
            box_cand(v, 0)[c] = e | kEntChanged;
        }
    }
    __syncthreads();
}

// ... with at most one: its union and entry stay in registers
template <int J>
__device__ __forceinline__ void box_subiteration1(const Box3D &v, uint32_t &e, uint32_t un, unsigned &words)
{
    const uint32_t del = un ? box_deletions<J>(v, e, un) : 0u;
    words += un != 0u && ent_dist(e) == 0;
    if (!__syncthreads_or(del != 0u)) return;
    if (del) {
        box_delete(e, del);
        e |= kEntChanged;
    }
    __syncthreads();
}

// Voxels of the word c at s with all six face neighbours: no direction deletes them.
__device__ __forceinline__ uint32_t box_faces(const Box3D &v, const uint32_t *s, uint32_t c)
{
    return (c << 1) & (c >> 1) & s[v.p] & s[-v.p] & s[v.ps] & s[-v.ps];
}

// Candidates of an iteration from the word list: pre-test and U on the active words.
__device__ __forceinline__ void box_collect(Box3D &v, unsigned &words, unsigned &entries)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *const list = box_words(v.list);
    uint16_t *const alist = reinterpret_cast<uint16_t *>(box_cand(v, 3));  // active words: positions in `list`
    const int nl = v.nl;
    // active words: a word of the row's 3x3 rows that is at most one column
    // away changed in the previous iteration (otherwise its union is empty),
    // and some voxel of it misses one of its face neighbours
    for (int base = warp * 32; base < nl; base += kResThreads) {
        const int k = base + lane;
        bool on = false;
        if (k < nl) {
            const uint32_t e = list[k], idx = ent_idx(e);
            uint32_t y2;
            const uint32_t z2 = box_plane_row(v, idx, y2);
            if ((res_smem[v.act + (int)(z2 * (uint32_t)v.my + y2)] >> ent_col(e)) & 1u) {
                const uint32_t *s = box_state() + idx;
                const uint32_t c = *s;
                on = (c & kCoreBits & ~box_faces(v, s, c)) != 0u;
            }
        }
        const int pos = warp_append(on, &v.n[1]);
        if (pos >= 0) alist[pos] = (uint16_t)k;
    }
    __syncthreads();
    const int na = v.n[1];
    // pre-test and U
    for (int base = warp * 32; base < na; base += kResThreads) {
        const int k = base + lane;
        uint32_t e = 0, un = 0, du = 0;
        if (k < na) {
            e = list[alist[k]];
            uint32_t g[27];
            const uint32_t val = box_window(box_state() + ent_idx(e), v.p, v.ps, g);
            du = rule3d<0>(g) & val;
            un = (du | rule3d<1>(g) | rule3d<2>(g) | rule3d<3>(g) | rule3d<4>(g) | rule3d<5>(g)) & val;
            words += ent_dist(e) == 0;
            entries++;
        }
        const int c = warp_append(un != 0u, &v.n[2]);
        if (c >= 0) {
            box_cand(v, 0)[c] = e;
            box_cand(v, 1)[c] = un;
            box_cand(v, 2)[c] = du;
        }
    }
    __syncthreads();
}

// ... from all words of the box, for one with more non-empty words than its
// lists hold: most of them lie inside solid parts and are not candidates.  There may
// be more candidates (v.n[2]) than their lists hold.  Returns this thread's work (words
// of the core, words).  Against box_iteration_dense in every iteration: 100 solid 64^3
// volumes 3.45 -> 1.30 ms, a 60 x 130 x 31 one 3.83 -> 1.52 ms, 150 of noise at 100^3, whose
// first iterations have too many candidates, 5.8 -> 3.0 ms.
static __device__ __noinline__ uint2 box_collect_all(Box3D &v)
{
    uint2 work = make_uint2(0u, 0u);
    const int lane = threadIdx.x & 31, nbox = (v.z1 - v.z0) * (v.y1 - v.y0) * v.wl, cap = v.cap;
    const WordWalk walk(v.wl, v.y1 - v.y0);
    WordPos q = walk.first();
    for (int i = threadIdx.x; i - lane < nbox; i += kResThreads, walk.next(q)) {
        const int d = i < nbox ? box_dist(v, q) : 6;
        uint32_t un = 0, du = 0;
        int idx = 0;
        if (d <= 5 && ((res_smem[v.act + (q.z + 1) * v.my + q.y + 1] >> (q.x >> v.xs)) & 1u)) {
            idx = box_index(v, q);
            const uint32_t *s = box_state() + idx;
            const uint32_t c = *s;
            if (c & kCoreBits & ~box_faces(v, s, c)) {
                uint32_t g[27];
                const uint32_t val = box_window(s, v.p, v.ps, g);
                du = rule3d<0>(g) & val;
                un = (du | rule3d<1>(g) | rule3d<2>(g) | rule3d<3>(g) | rule3d<4>(g) | rule3d<5>(g)) & val;
                work.x += d == 0;
                work.y++;
            }
        }
        const int c = warp_append(un != 0u, &v.n[2]);
        if (c >= 0 && c < cap) {
            box_cand(v, 0)[c] = box_entry(v, q, idx, d);
            box_cand(v, 1)[c] = un;
            box_cand(v, 2)[c] = du;
        }
    }
    __syncthreads();
    return work;
}

// The rest of an iteration on its candidates.  Returns whether a word of the core changed.
__device__ __forceinline__ bool box_thin(Box3D &v, int nc, int iter, unsigned &words)
{
    bool core = false;
    if (nc > kResThreads) {
        for (int c = threadIdx.x; c < nc; c += kResThreads) {
            const uint32_t del = box_cand(v, 2)[c];
            if (del) {
                const uint32_t e = box_cand(v, 0)[c];
                box_delete(e, del);
                box_cand(v, 0)[c] = e | kEntChanged;
            }
        }
        __syncthreads();
        box_subiteration<1>(v, nc, words);
        box_subiteration<2>(v, nc, words);
        box_subiteration<3>(v, nc, words);
        box_subiteration<4>(v, nc, words);
        box_subiteration<5>(v, nc, words);
        for (int c = threadIdx.x; c < nc; c += kResThreads) {
            const uint32_t e = box_cand(v, 0)[c];
            if (!(e & kEntChanged) || ent_dist(e) != 0) continue;
            core = true;
            box_changed(v, ent_idx(e), ent_col(e), iter);
        }
    } else if (nc > 0) {
        const int c = threadIdx.x;
        uint32_t e = 0, un = 0;
        if (c < nc) {
            e = box_cand(v, 0)[c];
            un = box_cand(v, 1)[c];
            const uint32_t del = box_cand(v, 2)[c];
            if (del) {
                box_delete(e, del);
                e |= kEntChanged;
            }
        }
        __syncthreads();
        box_subiteration1<1>(v, e, un, words);
        box_subiteration1<2>(v, e, un, words);
        box_subiteration1<3>(v, e, un, words);
        box_subiteration1<4>(v, e, un, words);
        box_subiteration1<5>(v, e, un, words);
        if ((e & kEntChanged) && ent_dist(e) == 0) {
            core = true;
            box_changed(v, ent_idx(e), ent_col(e), iter);
        }
    }
    return core;
}

// An iteration on all words of the box, for one with more candidates than their
// lists hold: a thread keeps the unions and deletions of its words (in local memory, so
// that it takes about 100 us for the 12288 words of a 64^3 box).
static __device__ __noinline__ bool box_iteration_dense(Box3D &v, int iter, unsigned &words, unsigned &entries)
{
    uint32_t un[kDenseWords], del[kDenseWords];
    bool core = false;
    const int nbox = (v.z1 - v.z0) * (v.y1 - v.y0) * v.wl;
    const WordWalk walk(v.wl, v.y1 - v.y0);
    WordPos q = walk.first();
    int k = 0;
    for (int i = threadIdx.x; i < nbox; i += kResThreads, walk.next(q), k++) {
        const int d = box_dist(v, q);
        const uint32_t *s = box_state() + box_index(v, q);
        un[k] = del[k] = 0;
        if (d <= 5 && (*s & kCoreBits) && ((res_smem[v.act + (q.z + 1) * v.my + q.y + 1] >> (q.x >> v.xs)) & 1u)) {
            uint32_t g[27];
            const uint32_t val = box_window(s, v.p, v.ps, g), du = rule3d<0>(g) & val;
            del[k] = du;
            un[k] = (du | rule3d<1>(g) | rule3d<2>(g) | rule3d<3>(g) | rule3d<4>(g) | rule3d<5>(g)) & val;
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
            if (del[k]) box_delete(box_entry(v, q, box_index(v, q), 0), del[k]);
        __syncthreads();
        if (j == 5) break;
        q = walk.first();
        k = 0;
        for (int i = threadIdx.x; i < nbox; i += kResThreads, walk.next(q), k++) {
            del[k] = 0;
            if (!un[k] || box_dist(v, q) > 4 - j) continue;
            const uint32_t *s = box_state() + box_index(v, q);
            if (!(*s & un[k])) continue;
            uint32_t g[27];
            const uint32_t cand = box_window(s, v.p, v.ps, g) & un[k];
            del[k] = cand & (j == 0   ? rule3d<1>(g)
                             : j == 1 ? rule3d<2>(g)
                             : j == 2 ? rule3d<3>(g)
                             : j == 3 ? rule3d<4>(g)
                                      : rule3d<5>(g));
            words += box_dist(v, q) == 0;
        }
        __syncthreads();
    }
    // only voxels of the union were deleted: a word changed when it lost some of its union
    q = walk.first();
    k = 0;
    for (int i = threadIdx.x; i < nbox; i += kResThreads, walk.next(q), k++) {
        const int idx = box_index(v, q);
        if (!(un[k] & ~box_state()[idx]) || box_dist(v, q) != 0) continue;
        core = true;
        box_changed(v, (uint32_t)idx, (uint32_t)(q.x >> v.xs), iter);
    }
    return core;
}

// One volume, or one box of it: rows [c0, c1) of planes [r0, r1) are the
// core; `halo` rows and planes around it (clamped to the volume) are held
// too.  Boxes run whole iterations (pre-test, U, N, E, D, S, W) in lockstep.
// A wrong value moves one row or plane per subiteration (the pre-test reads
// the same neighbours as U), so with six halo rows and planes the core is
// exact after an iteration; then every box sends the words near its core's
// edge that changed to a list in global memory, waits for every box's header
// (its count, and whether its core changed), and takes over what lies in its
// halo from its neighbours' lists.  Headers and messages are 16 bytes, written
// and read in one access, and carry the run and the iteration: each is waited
// for by itself, so that no fence, counter or second trip stands between them
// (97 x 75 x 66: 87 -> 82 us, 256^3: 176 -> 167 us, the int16 volume below 190 ->
// 179 us).  Two sets in turn: a box writes the messages of iteration i + 2 when
// it has every header of i + 1, which a box sends when it is done with those of i.
//
// Bound: the latency of an iteration (8 to 12 us: six dependent subiterations
// with two barriers each, then the meeting), not throughput: a box has some
// hundred active words.  Against warps marching through sparse bricks of
// 32 x 32 x 4 voxels, every brick of the neighbourhood of a change evaluated
// whole (24 us per iteration): a 97 x 75 x 66 tree volume 214 -> 85 us, a
// 187 x 203 x 161 one (16-bit pixels, transfers included) 955 -> 221 us, a
// 256^3 one, whose bricks did not fit, 1330 us on the tile rings -> 179 us
// (both before the headers and messages above; words of 32 voxels took them 238 and 193 us).
__device__ void res_run3d(Inst &in, const ResIO &io, const ResItem &item, ResSched *S, ResTrace *tr)
{
    __shared__ Box3D v;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        v.it = item;
        v.H = in.H;
        v.D = in.D;
        v.wl = (in.W + kVox - 1) / kVox;
        v.z0 = max(0, item.r0 - item.halo);
        v.z1 = min(in.D, item.r1 + item.halo);
        v.y0 = max(0, item.c0 - item.halo);
        v.y1 = min(in.H, item.c1 + item.halo);
        const int nz = v.z1 - v.z0, ny = v.y1 - v.y0;
        v.p = v.wl | 1;  // odd strides: rows and planes start on different banks
        v.ps = ((ny + 2) * v.p) | 1;
        v.mp = 0x7fffffffu / (uint32_t)v.p + 1u;
        v.mps = 0x7fffffffu / (uint32_t)v.ps + 1u;
        v.my = (ny + 5) & ~3;
        v.mrows = (nz + 2) * v.my;
        v.xs = 0;
        while (((v.wl - 1) >> v.xs) > 7) v.xs++;
        v.act = (int)up16((size_t)(nz + 2) * v.ps * 4);
        v.chg = v.act + (int)up16((size_t)v.mrows);
        v.list = v.chg + (int)up16((size_t)v.mrows);
        v.gy = in.res_gy;
        v.gz = item.bands / v.gy;
        v.bz = item.band / v.gy;
        v.by = item.band - v.bz * v.gy;
        v.stride = in.res_stride;
        v.msgs = in.res_msg;
        v.heads = in.res_head;
        v.run = in.res_run;
        v.flag = 0;
        v.nl = 0;
        for (int k = 0; k < 4; k++) v.n[k] = 0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < v.list / 16; i += kResThreads) reinterpret_cast<uint4 *>(res_smem)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    {
        const int list_cap = (kSmemBytes - v.list) / 4, nz = v.z1 - v.z0, ny = v.y1 - v.y0;
        res_load<true>(in, io, WordWalk(v.wl, ny), nz * ny * v.wl, 0, v.y0, v.z0,
                       [&](bool, const WordPos &q, uint32_t w) {
                           const int d = box_dist(v, q), idx = w ? box_index(v, q) : 0;
                           if (w) box_state()[idx] = w;
                           const int pos = warp_append((w & kCoreBits) != 0u && d <= 5, &v.n[0]);
                           if (pos >= 0 && pos < list_cap) box_words(v.list)[pos] = box_entry(v, q, idx, d);
                       });
    }
    for (int r = threadIdx.x; r < v.mrows / 4; r += kResThreads) box_words(v.act)[r] = kFull;
    __syncthreads();
    // more non-empty words than the lists hold: the candidates' lists take all of the room
    if (threadIdx.x == 0) {
        const bool dense = v.list + (size_t)v.n[0] * kBoxListBytes + 64 > (size_t)kSmemBytes;
        v.nl = dense ? 0 : v.n[0];
        v.cand = dense ? v.list : v.list + 4 * v.nl;
        v.cap = dense ? (kSmemBytes - 64 - v.list) / 12 : v.nl;
    }
    __syncthreads();
    const bool dense = v.n[0] > v.nl;

    int iter = 0, result = 0;
    unsigned words = 0, entries = 0;
    for (;; iter++) {
        if (dense) {
            const uint2 work = box_collect_all(v);
            if (v.n[2] <= v.cap) {
                words += work.x;
                entries += work.y;
            }
        } else {
            box_collect(v, words, entries);
        }
        const int nc = v.n[2];
        const bool core = nc > v.cap ? box_iteration_dense(v, iter, words, entries) : box_thin(v, nc, iter, words);
        const bool any = __syncthreads_or(core);
        bool any_chg = any;
        if (v.it.bands == 1) {
            if (!any) {
                result = 1;
                break;
            }
        } else {
            uint4 *const heads = v.heads + (iter & 1) * v.it.bands;
            if (threadIdx.x == 0)
                st_relaxed128(heads + v.it.band, make_uint4((unsigned)v.n[3], any ? 1u : 0u, v.run, (unsigned)iter + 1u));
            const unsigned long long t_end = globaltimer() + (unsigned long long)S->timeout_ns;
            // a header or message of this iteration, once it is there (bounded)
            auto await = [&](const uint4 *p, uint4 w) {
                for (int spin = 0; w.z != v.run || w.w != (unsigned)iter + 1u; w = ld_relaxed128(p), spin++) {
                    if ((spin & 63) == 63 && globaltimer() > t_end) {
                        v.flag = 2;
                        w = make_uint4(0u, 0u, 0u, 0u);
                        break;
                    }
                    if (spin >= 4096) __nanosleep(64);  // partners that have not started yet
                }
                return w;
            };
            // kWarps / 8 warps per neighbouring box take over its messages
            const int k8 = warp & 7, k9 = k8 < 4 ? k8 : k8 + 1;
            const int nbz = v.bz + k9 / 3 - 1, nby = v.by + k9 % 3 - 1;
            const bool next = warp < kWarps / 8 * 8 && nbz >= 0 && nbz < v.gz && nby >= 0 && nby < v.gy;
            const int nb = next ? nbz * v.gy + nby : v.it.band, k0 = (warp >> 3) * 32 + lane;
            const uint4 *m = v.msgs + ((size_t)(iter & 1) * v.it.bands + nb) * v.stride;
            // every thread's first header and message are on their way together, whether they are there or not
            uint4 h = ld_relaxed128(heads + nb), w = ld_relaxed128(m + min(k0, v.stride - 1));
            bool some = false;
            for (int t = threadIdx.x; t < v.it.bands; t += kResThreads) some |= await(heads + t, ld_relaxed128(heads + t)).y != 0u;
            if (next) {
                h = await(heads + nb, h);
                const int n = (int)h.x;
                for (int k = k0; k < n;) {
                    w = await(m + k, w);
                    if (v.flag) break;
                    const int r = (int)(w.x / (uint32_t)v.wl), x = (int)w.x - r * v.wl, z = r / v.H, y = r - z * v.H;
                    if (z >= v.z0 && z < v.z1 && y >= v.y0 && y < v.y1) {
                        uint32_t *s = box_state() + (z - v.z0 + 1) * v.ps + (y - v.y0 + 1) * v.p + x;
                        atomicAnd(s, w.y);
                        if (!(w.y & 2u) && x > 0) atomicAnd(s - 1, ~(1u << 31));
                        if (!(w.y & (1u << kVox)) && x + 1 < v.wl) atomicAnd(s + 1, ~1u);
                        box_mark(v, (z - v.z0 + 1) * v.my + (y - v.y0 + 1), x >> v.xs);
                        any_chg = true;
                    }
                    k += (kWarps / 8) * 32;
                    if (k < n) w = ld_relaxed128(m + k);
                }
            }
            some = __syncthreads_or(some);
            if (v.flag || !some) {
                result = v.flag ? -1 : 1;
                if (v.flag && threadIdx.x == 0) atomicOr(&S->status, kErrQueueTimeout);
                break;
            }
            any_chg = __syncthreads_or(any_chg);
        }
        if (iter + 1 >= in.pass_cap / 6 + 1) {
            if (threadIdx.x == 0) atomicOr(&S->status, kErrPassLimit);
            result = -1;
            break;
        }
        // rows to look at in the next iteration, four at a time, a byte each (my
        // is a multiple of 4; the bytes before the first and after the last row
        // belong to rows of padding)
        const int my4 = v.my / 4;
        for (int w = threadIdx.x + my4; w < v.mrows / 4 - my4; w += kResThreads) {
            uint32_t m = 0;
            if (any_chg) {
                const uint32_t *c = box_words(v.chg) + w;
#pragma unroll
                for (int dz = -1; dz <= 1; dz++) {
                    const uint32_t *r = c + dz * my4;
                    m |= r[0] | __funnelshift_l(r[-1], r[0], 8) | __funnelshift_r(r[0], r[1], 8);
                }
            }
            box_words(v.act)[w] = m | ((m << 1) & 0xFEFEFEFEu) | ((m >> 1) & 0x7F7F7F7Fu);
        }
        if (threadIdx.x >= 1 && threadIdx.x < 4) v.n[threadIdx.x] = 0;
        __syncthreads();
        if (any_chg)
            for (int r = threadIdx.x; r < v.mrows / 4; r += kResThreads) box_words(v.chg)[r] = 0u;
        // (chg is next written after the barriers of the next iteration)
    }
    __syncthreads();
    // the converged core
    res_store(in, io, 0, (in.W + 31) >> 5, v.it.c1 - v.it.c0, v.it.r1 - v.it.r0, v.it.c0, v.it.r0, [&](int y, int z, int x) {
        // 32 voxels from x on: the rest of its word, then the next word's from its second voxel on
        const int j = x / kVox, o = x - j * kVox;
        const uint32_t *s = box_state() + (z + v.it.r0 - v.z0 + 1) * v.ps + (y + v.it.c0 - v.y0 + 1) * v.p + j;
        return s[0] >> (o + 1) | (j + 1 < v.wl ? s[1] >> 2 << (kVox + 1 - o) : 0u);
    });
    res_done(in, v.it, result, 6 * (iter + 1), words, entries, tr);
}

// ------------------------------------------------------------ kernels -----
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
    __shared__ int s_item;
    __shared__ int s_take[2];
    for (;;) {
        if (threadIdx.x == 0) {
            s_item = atomicAdd(&S->head, 1);
            // the run's errors come after its first item was taken: waits of seconds and pass caps
            if (s_item == 0) S->status = 0;
        }
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
            case 2: res_run2d<2>(in, io, it, sm, S, s_take, trace + k); break;
            case 4: res_run2d<4>(in, io, it, sm, S, s_take, trace + k); break;
            default: res_run2d<8>(in, io, it, sm, S, s_take, trace + k); break;
            }
        } else
            res_run3d(in, io, it, S, trace + k);
        if (threadIdx.x == 0) {
            trace[k].t0 = t0;
            trace[k].t1 = (long long)globaltimer();
            trace[k].sm = res_smid();
        }
    }
    // the last CTA leaves the item counter as the next run needs it
    if (threadIdx.x == 0 && atomicAdd(&S->done, 1) == (int)gridDim.x - 1) {
        S->head = 0;
        S->done = 0;
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

cudaError_t launch_resident(int grid, Inst *d_insts, const ResItem *d_items, int nitems, ResSched *d_rs,
                            ResTrace *d_trace, const IODesc *d_io, const IODesc *one, bool pixels, bool teams,
                            cudaStream_t st)
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
    cfg.numAttrs = teams ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, resident_kernel, d_insts, d_items, d_rs, d_trace, one ? nullptr : d_io, pixels,
                              one ? *one : IODesc{});
}

}  // namespace bgt
