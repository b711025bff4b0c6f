// host.h -- host-side structures behind the C ABI handles.
#pragma once
#include <cstddef>
#include <map>
#include <tuple>
#include <vector>

#include <cuda.h>
#include <cuda_runtime.h>

#include "bgt_capi.h"
#include "common.cuh"
#include "kernels.cuh"

struct bgt_batch;

namespace bgt {
struct Sched;
struct IODesc;

struct Scratch {
    void *ptr = nullptr;
    size_t bytes = 0;
};

struct BatchItem {
    int dims = 2, W = 0, H = 0, D = 1, cfg = -1;
    bool auto_cfg = true;  // added with cfg < 0 (the resident engine may take it)
};

struct IO {
    int dtype = 0;
    const void *in = nullptr;
    void *out = nullptr;
    int inW = 0, inH = 0, inD = 0;  // input extents (0: the instance's own)
    bool packed = false;            // buf[0] already holds the packed input (resident instances)
};

struct Stat {
    int passes = 0, converged = 0;
};

int fail(int code, const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what);
size_t dtype_size(int dtype);
int default_cfg(int dims, int W, int H, int D);
int tuned_cfg(int dims, int W, int H, int D);
int ctx_scratch(bgt_ctx *c, int slot, size_t bytes, void **out);
// Host buffer of at least `bytes`, for readbacks that end before the call returns:
// pinned and kept (grown, never shrunk) up to 256 MB, pageable beyond and given
// back by ctx_pinned_done or the next ctx_pinned.
int ctx_pinned(bgt_ctx *c, size_t bytes, void **out);
void ctx_pinned_done(bgt_ctx *c);
int single_batch(bgt_ctx *c, int dims, int W, int H, int D, bgt_batch **out);
int batch_check(bgt_batch *b);
// Status words of the batch's last run (device pointers, null: none), and
// their bits as an error code.
void batch_status_words(const bgt_batch *b, const int *(&words)[2]);
int batch_status(int bits);
// Packed host transfers of the batch's only instance (w x h x d pixels of
// `dtype` in it): whether they serve it (out: the output array, or null), and the
// upload of its packed input in place of set_io.
bool batch_packs_host(const bgt_batch *b, int dtype, const void *in, const void *out, int w, int h, int d);
int batch_upload_packed(bgt_batch *b, int dtype, const void *in, int w, int h, int d);
int batch_set_input_extent(bgt_batch *b, int id, int inW, int inH, int inD);
size_t batch_pool_bytes(const std::vector<BatchItem> &items);
// Lay a batch out in caller-provided device memory (the serving runtime's
// arena) from the next finalize on; the memory is not freed by the batch.
int batch_use_pool(bgt_batch *b, void *pool, size_t bytes);

// Segment list on the host (malloc'ed arrays), in the reference's emission order.
struct HostSegs {
    int nseg = 0, npts = 0;
    int32_t *start = nullptr;
    uint8_t *is_end = nullptr;
    int16_t *px = nullptr, *py = nullptr, *pz = nullptr;
};
// Segment arrays in device memory (same layout as HostSegs; null when empty).
struct DevSegs {
    int nseg = 0, npts = 0;
    int32_t *start = nullptr;
    uint8_t *is_end = nullptr;
    int16_t *px = nullptr, *py = nullptr, *pz = nullptr;
};
// The rest of CenterlineExtraction: pruning and smoothing; status words of the
// kernels that made the image, read back with the results.
struct SegTail {
    int max_segment_length = 0, span = 0;
    const int *check[2] = {nullptr, nullptr};
};
// Results in the context's pinned memory, valid until its next use (idx, fx,
// fy, fz with a tail, start .. pz without), and the device arrays (without).
struct SegResult {
    int nseg = 0, npts = 0, checked = 0;
    const int32_t *start = nullptr;
    const uint8_t *is_end = nullptr;
    const int16_t *px = nullptr, *py = nullptr, *pz = nullptr;
    const uint32_t *idx = nullptr;
    const float *fx = nullptr, *fy = nullptr, *fz = nullptr;
    DevSegs dev;
};
// One cooperative launch (segments_graph.cu); 1 = beyond its range.
int segments_graph(bgt_ctx *c, int dims, const uint32_t *d_buf, int W, int H, int D, int P, const SegTail *tail,
                   SegResult *r);
// Device ExtractSegmentsV on a packed image (P words per row): arrays left in
// the context's scratch, or copied to host memory.
int segments_device_arrays(bgt_ctx *c, int dims, const uint32_t *d_buf, int W, int H, int D, int P, DevSegs *out);
// ... or in the context's pinned memory.
int segments_result(bgt_ctx *c, int dims, const uint32_t *d_buf, int W, int H, int D, int P, SegResult *r);
int segments_packed(bgt_ctx *c, int dims, const uint32_t *d_buf, int W, int H, int D, int P, HostSegs *out);
// Exclusive prefix sum of n ints on the context's stream (CUB temporary
// storage in scratch slot `slot`).
cudaError_t exscan(bgt_ctx *c, int slot, const int *in, int *out, long long n, cudaStream_t st);
void free_host_segs(HostSegs *s);
}  // namespace bgt

struct bgt_ctx {
    int device = 0;
    int sms = 148;
    cudaStream_t own = nullptr;
    cudaStream_t stream = nullptr;
    std::vector<bgt::Scratch> scratch;
    bgt::Scratch pinned;
    void *large = nullptr; // in its place for results beyond its limit
    bgt::SegResult view;   // segments of bgt_segments_begin, until bgt_segments_take (in `pinned` or `large`)
    int view_dims = 0;     // 0: none
    size_t seg_chains = 0, seg_nodes = 0;  // list sizes of the segment extraction (grown on demand)
    size_t seg_read = 0;                   // bytes its last result took (read back with the header)
    std::map<std::tuple<int, int, int, int>, bgt_batch *> cache;
};

struct bgt_batch {
    bgt_ctx *ctx = nullptr;
    std::vector<bgt::BatchItem> items;
    std::vector<bgt::Inst> h;
    std::vector<bgt::IO> io;
    std::vector<bgt::Stat> stats;
    bool finalized = false;
    bool stats_valid = false;
    bool ran = false;        // since it was finalized: the device holds records of a run
    int last_mode = 0;
    void *pool = nullptr;
    size_t pool_bytes = 0;
    size_t used_bytes = 0;
    bool reserved = false;              // pool pre-allocated by bgt_batch_reserve (or external)
    bool external = false;              // pool owned by the caller (batch_use_pool), never freed here
    int grid_cap = 0;                   // engine CTA cap (0: full device)
    std::vector<CUtensorMap> maps;      // host copies of uploaded tables (kept
    std::vector<bgt::IODesc> io_host;   // alive for stream-ordered uploads)
    bgt::Sched *d_sched = nullptr;
    unsigned *d_seq = nullptr;
    int4 *d_item = nullptr;
    bgt::Inst *d_insts = nullptr;
    CUtensorMap *d_tmaps = nullptr;
    int *d_flag = nullptr;
    void *d_lc = nullptr;         // contiguous per-tile "last change" arrays
    size_t lc_bytes = 0;
    bgt::IODesc *d_io = nullptr;  // per-instance I/O table of the batch-wide pack/unpack
    bool io_dirty = true;
    bool pixels = true;       // the resident kernel reads and writes the pixels itself (no output overlaps another's input)
    bool timed = true;        // record the stage boundaries
    bool bytes_only = false;  // every input one byte wide, tested "byte != 0"
    long long pack_words = 0, unpack_words = 0;
    unsigned cap = 0;
    int smem = 0;
    int grid = 0;
    // stage boundaries of an engine run: pack, resident engine, tile engine, unpack
    cudaEvent_t ev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    // resident engine plan (resident.cu): items in the order they are taken
    int engine_mode = 0;              // 0: resident engine where it fits, tile rings for the rest; 1: rings only
    std::vector<bgt::ResItem> res_items;
    bgt::ResItem *d_res_items = nullptr;
    bgt::ResSched *d_rs = nullptr;
    bgt::ResTrace *d_rtrace = nullptr;  // per-item timeline of the last resident run
    int res_grid = 0;
    bool res_teams = false;           // some instance is cut into several boxes
    bgt::ResSched rs_host{};          // kept alive for its stream-ordered upload
    bool any_ring = false;            // some instance is planned for the tile rings
    cudaGraphExec_t gexec = nullptr;
    bool graph_valid = false;
    // plain path with the pass loop on the device (bgt_batch_run mode 2)
    cudaGraphExec_t pexec = nullptr;
    bool pgraph_valid = false;
    bgt::PlainLoop *d_ploop = nullptr;  // one loop state per instance
};
