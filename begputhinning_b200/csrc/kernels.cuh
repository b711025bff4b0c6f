// kernels.cuh -- declarations shared by the kernel translation unit and the
// host-side batch/engine code.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace bgt {

// Tile configurations.  2D ids 0..7: (K, S) with NW = 4 warps, ids 8..12 the
// same with shared warp edges; 3D ids 16, 17, 19: (NWX = 4, TZ = 8, 16, 4).
// All use 128 threads so the persistent engine can run any mix of them in
// one launch.
struct CfgInfo {
    int id, dims, k, S, NW, NWX, TZ;
    int TW, TH, TZc;  // core tile extent (words, rows, planes)
    int smem;         // dynamic shared memory bytes
    int box[3];       // TMA box (words, rows, planes)
    int ubox[3];      // TMA box of the 3D union (core words, rows, core planes)
};
// Tensor maps per instance: buf[0], buf[1] and (3D) the union.
constexpr int kMapsPerInst = 3;
const CfgInfo *cfg_info(int id);  // nullptr if unknown
int max_cfg_smem();               // largest dynamic shared memory of any configuration
const int *cfg_ids_2d(int *n);
const int *cfg_ids_3d(int *n);

// Scheduler state of the persistent engine (device memory).
struct alignas(128) Ring {
    unsigned head;      // next ticket to claim
    unsigned pad0[31];  // head and tail on separate 128-byte lines
    unsigned tail;      // next ticket to reserve
    unsigned cap;       // slots
    unsigned *seq;      // [cap] slot sequence numbers
    int4 *item;         // [cap] (instance, tile, pass, tiles in the wave)
};

struct Sched {
    Ring ring[2];       // 0: critical-path instances, 1: the rest
    int live;           // instances not yet converged
    int live_prio[2];   // ... per ring (a ring with no live instance gets no more items)
    int gang_budget;    // CTAs that may still join gangs (the rest keep claiming)
    int status;         // error bits
    long long timeout_ns;
};

// Resident engine (resident.cu).  A work item is one instance, or one box of
// it (the boxes of an instance run together and trade what lies along their
// edges through global memory).  Items are taken in order by one fetch-and-add.
struct ResItem {
    int inst;        // instance index
    int band, bands; // box index and number of boxes (1: the whole instance)
    int r0, r1;      // core rows [r0, r1) of the box; 3D: core planes
    int halo;        // rows (3D: and planes) kept on each side of the core (0 for a single box)
    int c0, c1;      // core words of the box; 3D: core rows
};
struct ResSched {
    int head;        // next item
    int done;        // CTAs that have left the kernel (the last one resets both for the next run)
    int nitems;
    int status;      // error bits of the run
    long long timeout_ns;
};
// What became of one work item in the last run: its timeline (global timer,
// ns; SM id), outcome and work.
struct ResTrace {
    long long t0, t1;
    int sm;
    int result;      // 1 converged, -1 pass cap or failed wait
    int passes;      // passes (3D: subiterations) run
    int pad;
    unsigned long long words, tiles;  // packed core words processed; units of work
};
// One CTA per SM: two of 384 threads with 112 KB each took the mixed batch
// from 1.19 to 1.35 ms and three of 256 to 1.52 ms (smaller boxes, more halo),
// lone images and volumes as long or longer; 1024 threads from 1.166 to 1.178 ms.
constexpr int kResThreads = 768;
constexpr int kResCtasPerSm = 1;
constexpr int kResSmemBytes = 230400;  // dynamic shared memory of one CTA
// Dynamic shared memory of the resident kernel (one CTA per SM).
int res_smem_bytes();
// Whether a 2D box of nrows rows of wl words (halo included) fits one CTA.
bool res_fits2d(int wl, int nrows);
// Its cost: word steps of a pass over all of its units.
double res_cost2d(int wl, int nrows);
// Passes between two meetings of the boxes of an image (4 halo rows each): 3,
// 4, 5 and 6 took a 4096^2 image 99, 98, 91 and 101 us, a 512^2 one 47, 44, 51
// and 50 us, a 1501 x 1003 float one 85, 86, 89 and 86 us, the mixed batch 1.165,
// 1.154, 1.156 and 1.175 ms (the passes that images need decide much of it: a
// run ends at a meeting).
constexpr int kResPeriod2D = 4;
// Whether a 3D box (ny rows x nz planes of a volume W wide, halo included) fits one CTA.
bool res_fits3d(int W, int ny, int nz);
// Words of its rows (30 voxels each).
int res_words3d(int W);
constexpr int kResHalo3D = 6;  // one iteration: six subiterations, one row and plane each
cudaError_t res_occupancy(int *per_sm);  // resident CTAs per SM
// Per-instance input/output of a batch-wide pack/unpack launch.
// Unsigned 32-bit division by a divisor fixed per instance, as a multiply
// and shifts (Granlund and Montgomery, "Division by invariant integers using
// multiplication", 1994, section 4): with l = ceil(log2 d),
// m = floor(2^32 (2^l - d) / d) + 1, t = mulhi(m, n):
// n / d = (t + ((n - t) >> min(l, 1))) >> max(l - 1, 0), exact for every
// 32-bit n.
struct FastDiv {
    uint32_t m = 1, s1 = 0, s2 = 0, d = 1;
};
inline FastDiv make_fastdiv(uint32_t d)
{
    FastDiv f;
    f.d = d;
    uint32_t l = 0;
    while (l < 32 && (1ull << l) < d) l++;
    f.m = (uint32_t)(((1ull << 32) * ((1ull << l) - d)) / d + 1);
    f.s1 = l < 1 ? l : 1;
    f.s2 = l > 1 ? l - 1 : 0;
    return f;
}
__device__ __forceinline__ uint32_t fdiv(const FastDiv &f, uint32_t n)
{
    const uint32_t t = __umulhi(f.m, n);
    return (t + ((n - t) >> f.s1)) >> f.s2;
}

struct alignas(16) IODesc {
    const void *in;
    void *out;
    int dtype, mode;         // pixel type; binarisation 0 = 2D rule, 1 = 3D rule, 2 = nonzero
    int inW, inH, inD;       // input extents inside the instance
    int inst;                // instance index
    long long wbegin;        // first global packed-word index of the instance (pack)
    long long gbegin;        // first global unpack-word index (rows x ceil(W/32))
    // dividers of the instance: words per row P, rows H, pixels per row W,
    // used words per row ceil(W/32), and the core tile extents TW, TH, TZ
    FastDiv dP, dH, dW, dWW, dTW, dTH, dTZ;
};

// pixels: instances are read from and written to their pixel arrays (d_io by
// instance, or `one` for a batch of one instance); else buf[0] holds them.
// teams: some instance is cut into several boxes.
cudaError_t launch_resident(int grid, Inst *d_insts, const ResItem *d_items, int nitems,
                            ResSched *d_rs, ResTrace *d_trace, const IODesc *d_io, const IODesc *one, bool pixels,
                            bool teams, cudaStream_t st);

// Launchers (stream-ordered, no host synchronisation).
// bytes: every input is one byte wide and tested "byte != 0" (see pack_all_kernel)
cudaError_t launch_pack_all(const Inst *d_insts, const IODesc *d_io, int n, long long total_words, bool bytes,
                            cudaStream_t st);
cudaError_t launch_unpack_all(const Inst *d_insts, const IODesc *d_io, int n, long long total_words,
                              cudaStream_t st);
// mode 0: 2D binarisation, 1: 3D binarisation, 2: nonzero.  Input extents
// inW x inH x inD (row stride inW) inside the packed W x H x D.
cudaError_t launch_pack(int dtype, int mode, const void *in, int inW, int inH, int inD, int W, int H, int D, int P,
                        uint32_t *buf0, uint32_t *buf1, cudaStream_t st);
cudaError_t launch_unpack(int dtype, const uint32_t *buf, int W, int H, int D, int P, void *out,
                          cudaStream_t st);
// per-tile nonempty marks -> lc (-1 nonempty, kNever empty); counts nonempty tiles into *count
cudaError_t launch_tile_init(const Inst *d_inst, const Inst &h_inst, int *d_count, cudaStream_t st);
cudaError_t launch_plain_pass(int cfg, Inst *d_inst, int ntiles, int q, int *d_flag, int *d_err,
                              cudaStream_t st);
// Device-side pass loop of the plain path (one per instance).
struct PlainLoop {
    int q;            // pass to run next
    int last_change;  // last pass with a change
    int flag;         // set by the pass when a tile changed
    int converged;    // 1 converged, -1 pass cap, 0 running
};
cudaError_t launch_plain_dev_pass(int cfg, Inst *d_inst, int ntiles, PlainLoop *d_loop, int *d_err, cudaStream_t st);
cudaError_t launch_plain_loop_init(PlainLoop *d_loop, cudaStream_t st);
// Records the pass in the loop state and in the instance (passes_run,
// converged; kErrPassLimit in *d_err at the cap) and sets the graph's
// conditional to 1 while another pass is needed.
cudaError_t launch_plain_loop_step(PlainLoop *d_loop, Inst *d_inst, int *d_err, cudaGraphConditionalHandle h,
                                   cudaStream_t st);
cudaError_t launch_engine(int grid, int smem, Inst *d_insts, int ninst, Sched *d_sched, cudaStream_t st);
cudaError_t launch_rule_table(int dims, int dir, uint32_t *d_out, cudaStream_t st);
int engine_max_blocks_per_sm(int smem);
cudaError_t engine_set_smem(int smem);

}  // namespace bgt
