// segments.cu -- ExtractSegmentsV on the device (2D/ExtractSegments.cpp:16-127,
// 3D/ExtractSegments.cpp:135-251), bit-exact in content and order.
//
// The whole extraction as one launch is in segments_graph.cu.  Here: its
// counterpart for images beyond that launch's index range (and, selected by
// BGT_SEGMENTS_PIXEL_WALK=1, for tests that compare the two), which replays
// the reference's walk pixel by pixel:
//   1. classify (one thread per packed word, bit-sliced neighbour counts):
//      value map V = 2 for points with exactly two foreground neighbours,
//      -max(n,1) otherwise (nodes), 0 for background and frame pixels;
//   2. node list in raster order (prefix sum over per-word node counts);
//   3. components (union-find with atomics), nodes grouped by component in
//      raster order (stable radix sort), and a warp per component replaying
//      the walk (the lanes read the 8/26 neighbour values, a ballot picks the
//      first nonzero one in the reference's scan order).
#include <cub/cub.cuh>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "host.h"
#include "kernels.cuh"

namespace bgt {

// --------------------------------------------------------- classify -------
// bit-sliced counter: add one bit-word x to the counter c[0..NB)
template <int NB>
__device__ __forceinline__ void csa_add(uint32_t (&c)[NB], uint32_t x)
{
#pragma unroll
    for (int i = 0; i < NB; i++) {
        const uint32_t t = c[i] & x;
        c[i] ^= x;
        x = t;
    }
}

__device__ __forceinline__ uint32_t word_at(const uint32_t *buf, int P, int H, int D, int z, int y, int j)
{
    if (z < 0 || z >= D || y < 0 || y >= H || j < 0 || j >= P) return 0u;
    return __ldg(buf + ((size_t)z * H + y) * P + j);
}

// interior mask of word j of a row: bits with 1 <= x <= W-2
__device__ __forceinline__ uint32_t interior_bits(int W, int j)
{
    const int x0 = j * 32;
    uint32_t m = 0xffffffffu;
    if (x0 == 0) m &= ~1u;
    const int last = W - 2 - x0;  // highest allowed bit
    if (last < 0) return 0u;
    if (last < 31) m &= (2u << last) - 1u;
    return m;
}

template <int DIMS>
__global__ void classify_kernel(const uint32_t *__restrict__ buf, int W, int H, int D, int P,
                                int8_t *__restrict__ V, int *__restrict__ node_count)
{
    const int wwords = (W + 31) >> 5;
    const long long nw = (long long)H * D * wwords;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nw;
         i += (long long)gridDim.x * blockDim.x) {
        const long long row = i / wwords;
        const int j = (int)(i - row * wwords);
        const int y = (int)(row % H), z = (int)(row / H);
        const uint32_t c = word_at(buf, P, H, D, z, y, j);
        uint32_t pts = c & interior_bits(W, j);
        if (y == 0 || y == H - 1) pts = 0;
        if (DIMS == 3 && (z == 0 || z == D - 1)) pts = 0;
        constexpr int NB = DIMS == 2 ? 4 : 5;
        uint32_t cnt[NB] = {};
        const int zlo = DIMS == 3 ? -1 : 0, zhi = DIMS == 3 ? 1 : 0;
        if (pts) {
            for (int dz = zlo; dz <= zhi; dz++)
                for (int dy = -1; dy <= 1; dy++) {
                    const uint32_t l = word_at(buf, P, H, D, z + dz, y + dy, j - 1);
                    const uint32_t m = word_at(buf, P, H, D, z + dz, y + dy, j);
                    const uint32_t r = word_at(buf, P, H, D, z + dz, y + dy, j + 1);
                    csa_add<NB>(cnt, at_xm1(m, l));
                    if (dz != 0 || dy != 0) csa_add<NB>(cnt, m);
                    csa_add<NB>(cnt, at_xp1(m, r));
                }
        }
        // exactly two neighbours
        uint32_t eq2 = ~cnt[0] & cnt[1] & ~cnt[2] & ~cnt[3];
        if (NB == 5) eq2 &= ~cnt[NB - 1];
        const uint32_t nodes = pts & ~eq2;
        node_count[i] = __popc(nodes);
        int8_t *vrow = V + ((size_t)z * H + y) * W + (size_t)j * 32;
        const int nb = min(32, W - j * 32);
        for (int b = 0; b < nb; b++) {
            int8_t v = 0;
            if ((pts >> b) & 1u) {
                int n = 0;
#pragma unroll
                for (int k = 0; k < NB; k++) n |= (int)((cnt[k] >> b) & 1u) << k;
                v = (int8_t)(n == 2 ? 2 : -(n == 0 ? 1 : n));
            }
            vrow[b] = v;
        }
    }
}

// node raster indices in raster order; offs = exclusive scan of node_count
template <int DIMS>
__global__ void emit_nodes_kernel(const uint32_t *__restrict__ buf, int W, int H, int D, int P,
                                  const int8_t *__restrict__ V, const int *__restrict__ offs,
                                  uint32_t *__restrict__ nodes)
{
    const int wwords = (W + 31) >> 5;
    const long long nw = (long long)H * D * wwords;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nw;
         i += (long long)gridDim.x * blockDim.x) {
        const long long row = i / wwords;
        const int j = (int)(i - row * wwords);
        const size_t base = (size_t)row * W + (size_t)j * 32;
        const int nb = min(32, W - j * 32);
        int o = offs[i];
        for (int b = 0; b < nb; b++)
            if (V[base + b] < 0) nodes[o++] = (uint32_t)(base + b);
    }
}

// ------------------------------------------------------------- CCL --------
__device__ __forceinline__ uint32_t uf_find(uint32_t *par, uint32_t x)
{
    for (;;) {
        const uint32_t p = __ldcg(par + x);
        if (p == x) return x;
        const uint32_t g = __ldcg(par + p);
        if (g != p) atomicCAS(par + x, p, g);  // path halving
        x = p;
    }
}

__device__ __forceinline__ void uf_union(uint32_t *par, uint32_t a, uint32_t b)
{
    for (int guard = 0; guard < 1 << 20; guard++) {
        a = uf_find(par, a);
        b = uf_find(par, b);
        if (a == b) return;
        if (a < b) { const uint32_t t = a; a = b; b = t; }  // hook the larger root under the smaller
        const uint32_t old = atomicCAS(par + a, a, b);
        if (old == a) return;
        a = old;
    }
}

__global__ void uf_init_kernel(const int8_t *__restrict__ V, uint32_t *par, long long n)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        par[i] = V[i] != 0 ? (uint32_t)i : 0xffffffffu;
}

// union every point with its point neighbours that precede it in raster order
template <int DIMS>
__global__ void uf_hook_kernel(const int8_t *__restrict__ V, int W, int H, int D, uint32_t *par)
{
    const long long n = (long long)W * H * D;
    const long long slice = (long long)W * H;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        if (V[i] == 0) continue;
        // points are interior, so every neighbour index is in range
        const int zlo = DIMS == 3 ? -1 : 0;
        for (int dz = zlo; dz <= 0; dz++)
            for (int dy = -1; dy <= 1; dy++)
                for (int dx = -1; dx <= 1; dx++) {
                    const long long off = dz * slice + (long long)dy * W + dx;
                    if (off >= 0) continue;  // only predecessors
                    if (V[i + off] != 0) uf_union(par, (uint32_t)i, (uint32_t)(i + off));
                }
    }
}

__global__ void node_keys_kernel(uint32_t *par, const uint32_t *__restrict__ nodes, int nn,
                                 uint32_t *__restrict__ keys)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x)
        keys[i] = uf_find(par, nodes[i]);
}

// component starts in the sorted node list: flags[i] = key changes at i
__global__ void comp_flags_kernel(const uint32_t *__restrict__ keys, int nn, int *__restrict__ flag)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x)
        flag[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

__global__ void comp_starts_kernel(const int *__restrict__ flag, const int *__restrict__ pos, int nn,
                                   int *__restrict__ starts)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x)
        if (flag[i]) starts[pos[i]] = i;
}

// ------------------------------------------------------------- walk -------
struct WalkOut {
    int *nseg;   // [nn] per node (indexed by position in the raster-ordered list)
    int *npts;   // [nn]
    int *tpo;    // [nn] the node's first point in the temporary arrays
    int *tso;    // [nn] the node's first segment in the temporary arrays
    const int *cpb;  // [ncomp+1] each component's first point in the temporary arrays
    const int *csb;  // [ncomp+1] each component's first segment
    int16_t *tx, *ty, *tz;  // temporary points in emission order, per component
    int32_t *trel;          // temporary segment starts (point index within the node's output)
    uint8_t *tend;          // temporary is_end flags
    int *err;               // kErrSegOverflow when a component outgrows its bound
};

// One warp per component replays the reference's walk over the component's
// nodes in raster order (lanes read the 8/26 neighbours, a ballot picks the
// first nonzero one in the reference's scan order).  Writes to the value map
// are kept to the pixels that anything can look at again: a walk along a
// chain zeroes its first and last chain pixels and every original node it
// passes; the chain pixels in between (nn == 2, both neighbours on the same
// walk) are skipped, because only a walk standing next to them could read
// them and the chain is never entered again (its ends are zero).  The walk
// excludes the pixel it came from, which the reference has zeroed.  A stall
// (no nonzero neighbour) zeroes the pixel before it, so that the stalled
// pixel's later walks see it as the reference does.  Coordinates follow the
// steps instead of being divided out of the raster index.
template <int DIMS>
__global__ void walk_kernel(int8_t *V, const int8_t *__restrict__ V0, int W, int H,
                            const uint32_t *__restrict__ sorted_nodes, const uint32_t *__restrict__ sorted_rank,
                            const int *__restrict__ comp_start, int ncomp, int nn, WalkOut out)
{
    constexpr int ND = DIMS == 2 ? 8 : 26;
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    const long long slice = (long long)W * H;
    // this lane's neighbour offset in the reference's scan order, and its
    // (dx, dy, dz) packed as (dz+1)*9 + (dy+1)*3 + (dx+1)
    long long my_off = 0;
    int my_d = 13;
    {
        int q = 0;
        const int zlo = DIMS == 3 ? -1 : 0, zhi = DIMS == 3 ? 1 : 0;
        for (int dz = zlo; dz <= zhi; dz++)
            for (int dy = -1; dy <= 1; dy++)
                for (int dx = -1; dx <= 1; dx++) {
                    if (!dz && !dy && !dx) continue;
                    if (q == lane) {
                        my_off = dz * slice + (long long)dy * W + dx;
                        my_d = (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1);
                    }
                    q++;
                }
    }
    const unsigned lane_ok = lane < ND ? 1u : 0u;
    for (int comp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; comp < ncomp; comp += warps) {
        const int a = comp_start[comp];
        const int b = comp + 1 < ncomp ? comp_start[comp + 1] : nn;
        // the component's outputs go to its own temporary range, in emission order
        int po = out.cpb[comp], so = out.csb[comp];
        const int po_end = out.cpb[comp + 1], so_end = out.csb[comp + 1];
        for (int k = a; k < b; k++) {
            const long long p = sorted_nodes[k];
            const int rank = (int)sorted_rank[k];  // position in raster-ordered node list
            const int vp = V[p];
            __syncwarp();
            if (lane == 0) {
                out.tpo[rank] = po;
                out.tso[rank] = so;
            }
            if (vp >= 0) {
                if (lane == 0) {
                    out.nseg[rank] = 0;
                    out.npts[rank] = 0;
                }
                continue;
            }
            if (lane == 0) V[p] = 0;
            __syncwarp();
            const int p_x = (int)(p % W), p_y = (int)((p / W) % H), p_z = DIMS == 3 ? (int)(p / slice) : 0;
            int ni = -1;
            int segs = 0, pts = 0;
            int cx = p_x, cy = p_y, cz = p_z;
            auto put = [&]() {
                if (lane == 0) {
                    if (po < po_end) {
                        out.tx[po] = (int16_t)cx;
                        out.ty[po] = (int16_t)cy;
                        if (DIMS == 3) out.tz[po] = (int16_t)cz;
                    } else {
                        atomicOr(out.err, kErrSegOverflow);
                    }
                }
                po++;
                pts++;
            };
            auto step = [&](int s) {  // move the coordinates by the delta of scan index s
                const int d = __shfl_sync(kFull, my_d, s);
                cx += d % 3 - 1;
                cy += (d / 3) % 3 - 1;
                cz += d / 9 - 1;
                return __shfl_sync(kFull, my_off, s);
            };
            const int v0p = V0[p];
            for (int br = 0; br < -vp; br++) {
                int is_end = v0p > -2 && v0p < 2;
                const int seg_rel = pts;
                cx = p_x;
                cy = p_y;
                cz = p_z;
                put();
                // first neighbour after ni in scan order with a nonzero value;
                // every lane loads its neighbour's current and original value
                // at once, and the chosen one's reach the warp by shuffles
                int vn = lane_ok ? V[p + my_off] : 0, v0n = lane_ok ? V0[p + my_off] : 0;
                const unsigned m = __ballot_sync(kFull, lane_ok && lane > ni && vn != 0);
                ni = m ? __ffs(m) - 1 : ND;
                if (ni < ND) {
                    long long prev = p;
                    int back = ND - 1 - ni;  // scan index of the step back to prev
                    int vt = __shfl_sync(kFull, vn, ni), v0t = __shfl_sync(kFull, v0n, ni);
                    long long t = p + step(ni);
                    bool first = true, stall = false;
                    for (int guard = 0; guard < (1 << 30); guard++) {
                        if (vt != 2) break;
                        put();
                        vn = lane_ok ? V[t + my_off] : 0;
                        v0n = lane_ok ? V0[t + my_off] : 0;
                        const unsigned m2 = __ballot_sync(kFull, lane_ok && lane != back && vn != 0);
                        if (!m2) {
                            stall = true;
                            break;
                        }
                        if (lane == 0 && (first || v0t != 2)) V[t] = 0;
                        const int s2 = __ffs(m2) - 1;
                        prev = t;
                        back = ND - 1 - s2;
                        vt = __shfl_sync(kFull, vn, s2);
                        v0t = __shfl_sync(kFull, v0n, s2);
                        t += step(s2);
                        first = false;
                        __syncwarp();
                    }
                    __syncwarp();
                    // the last chain pixel (prev, unless the walk never left p) becomes zero in memory too
                    if (lane == 0 && prev != p) V[prev] = 0;
                    __syncwarp();
                    put();
                    if (v0t > -2 && v0t < 2) is_end = 1;
                    // a stalled walk stays on t, which the reference zeroed: it becomes 1
                    if (lane == 0) V[t] = stall ? (int8_t)1 : (int8_t)(vt + 1);
                    __syncwarp();
                }
                if (lane == 0) {
                    if (so < so_end) {
                        out.trel[so] = seg_rel;
                        out.tend[so] = (uint8_t)is_end;
                    } else {
                        atomicOr(out.err, kErrSegOverflow);
                    }
                }
                so++;
                segs++;
            }
            if (lane == 0) {
                out.nseg[rank] = segs;
                out.npts[rank] = pts;
            }
        }
    }
}

// fg pixels per union-find root (the component's pixel count)
__global__ void comp_px_kernel(const int8_t *__restrict__ V, uint32_t *par, long long n, uint32_t *cnt)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        if (V[i] != 0) atomicAdd(cnt + uf_find(par, (uint32_t)i), 1u);
}

// per component: branches = sum of |v| over its nodes (a bound on its
// segments), pixels from its root
__global__ void comp_sums_kernel(const int8_t *__restrict__ V0, const uint32_t *__restrict__ snodes,
                                 const uint32_t *__restrict__ keys_s, const int *__restrict__ flag,
                                 const int *__restrict__ fpos, const uint32_t *__restrict__ cnt, int nn,
                                 int *branches, int *px)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        const int c = fpos[i] + flag[i] - 1;
        atomicAdd(branches + c, -(int)V0[snodes[i]]);
        if (flag[i]) px[c] = (int)cnt[keys_s[i]];
    }
}

// bounds of a component's output: segments <= branches; points <= pixels +
// 3 * branches (each branch adds its start and end point, and a pixel is
// walked through again only after two walks ended on it)
__global__ void comp_bounds_kernel(const int *__restrict__ branches, const int *__restrict__ px, int ncomp,
                                   int *bpts, int *bsegs)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c <= ncomp; c += gridDim.x * blockDim.x) {
        bpts[c] = c < ncomp ? px[c] + 3 * branches[c] : 0;
        bsegs[c] = c < ncomp ? branches[c] : 0;
    }
}

// Move each node's output from its component's temporary range to its place
// in the reference's emission order (one warp per node).
template <int DIMS>
__global__ void place_kernel(const WalkOut w, const int *__restrict__ seg_off, const int *__restrict__ pt_off,
                             int nn, int32_t *start, uint8_t *is_end, int16_t *px, int16_t *py, int16_t *pz)
{
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nn; r += warps) {
        const int np = w.npts[r], ns = w.nseg[r];
        const int ti = w.tpo[r], to = pt_off[r], si = w.tso[r], so = seg_off[r];
        for (int j = lane; j < np; j += 32) {
            px[to + j] = w.tx[ti + j];
            py[to + j] = w.ty[ti + j];
            if (DIMS == 3) pz[to + j] = w.tz[ti + j];
        }
        for (int j = lane; j < ns; j += 32) {
            start[so + j] = to + w.trel[si + j];
            is_end[so + j] = w.tend[si + j];
        }
    }
}

__global__ void iota_kernel(uint32_t *a, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a[i] = (uint32_t)i;
}

__global__ void gather_kernel(const uint32_t *__restrict__ src, const uint32_t *__restrict__ idx,
                              uint32_t *__restrict__ dst, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src[idx[i]];
}

static size_t align16(size_t v) { return (v + 15) / 16 * 16; }

static int grid_of(long long n, int block = 256)
{
    long long g = (n + block - 1) / block;
    return (int)std::max(1LL, std::min(g, 148LL * 16));
}

// Exclusive sum via CUB; temp storage from scratch slot `slot`.
cudaError_t exscan(bgt_ctx *c, int slot, const int *in, int *out, long long n, cudaStream_t st)
{
    size_t tb = 0;
    cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, tb, in, out, (int)n, st);
    if (e != cudaSuccess) return e;
    void *tmp = nullptr;
    if (ctx_scratch(c, slot, tb, &tmp) != BGT_OK) return cudaErrorMemoryAllocation;
    return cub::DeviceScan::ExclusiveSum(tmp, tb, in, out, (int)n, st);
}

// Device segment extraction on a packed image (P words per row, H rows, D
// planes; W x H x D pixels).  The segment arrays stay in the context's
// scratch (slot 19) until the next extraction on the context.
int segments_device_arrays(bgt_ctx *c, int dims, const uint32_t *d_buf, int W, int H, int D, int P, DevSegs *out)
{
    cudaStream_t st = c->stream;
    const long long npx = (long long)W * H * D;
    // BGT_SEGMENTS_PIXEL_WALK=1 selects the per-component pixel walk below (tests compare both)
    if (npx < (1LL << 32) - 1 && !getenv("BGT_SEGMENTS_PIXEL_WALK")) {
        SegResult r;
        const int grc = segments_graph(c, dims, d_buf, W, H, D, P, nullptr, &r);
        *out = r.dev;
        if (grc != 1) return grc;  // done, or an error
    }
    if (npx >= (1LL << 32) - 1) return fail(BGT_ERR_LIMIT, "segment extraction limited to < 2^32 pixels");
    const long long nw = (long long)H * D * ((W + 31) / 32);
    // scratch slots: 1 V, 2 V0, 3 node_count, 4 node offs, 5 nodes, 6 par, 7 keys, 8 keys_sorted,
    // 9 vals(rank), 10 vals_sorted, 11 flags, 12 flag pos, 13 comp starts, 14 cub temp,
    // 15 nseg, 16 npts, 17 seg_off, 18 pt_off, 19 out arrays
    void *p1, *p2, *p3, *p4, *p6;
    int rc;
    if ((rc = ctx_scratch(c, 1, npx, &p1)) || (rc = ctx_scratch(c, 2, npx, &p2)) ||
        (rc = ctx_scratch(c, 3, (nw + 1) * 4, &p3)) || (rc = ctx_scratch(c, 4, (nw + 1) * 4, &p4)) ||
        (rc = ctx_scratch(c, 6, npx * 4, &p6)))
        return rc;
    int8_t *V = (int8_t *)p1, *V0 = (int8_t *)p2;
    int *cnt = (int *)p3, *offs = (int *)p4;
    uint32_t *par = (uint32_t *)p6;
    cudaError_t e;
    if (dims == 2)
        classify_kernel<2><<<grid_of(nw), 256, 0, st>>>(d_buf, W, H, D, P, V, cnt);
    else
        classify_kernel<3><<<grid_of(nw), 256, 0, st>>>(d_buf, W, H, D, P, V, cnt);
    cudaMemcpyAsync(V0, V, npx, cudaMemcpyDeviceToDevice, st);  // the reference's "onn"
    cudaMemsetAsync(cnt + nw, 0, 4, st);
    if ((e = exscan(c, 14, cnt, offs, nw + 1, st)) != cudaSuccess) return cuda_fail(e, "node scan");
    int nn = 0;
    if ((e = cudaMemcpyAsync(&nn, offs + nw, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return cuda_fail(e, "node count");
    *out = DevSegs();
    if (nn == 0) return BGT_OK;
    void *p5, *p7, *p8, *p9, *p10, *p11, *p12, *p13, *p15, *p16, *p17, *p18;
    if ((rc = ctx_scratch(c, 5, (size_t)nn * 4, &p5)) || (rc = ctx_scratch(c, 7, (size_t)nn * 4, &p7)) ||
        (rc = ctx_scratch(c, 8, (size_t)nn * 4, &p8)) || (rc = ctx_scratch(c, 9, (size_t)nn * 4, &p9)) ||
        (rc = ctx_scratch(c, 10, (size_t)nn * 4, &p10)) || (rc = ctx_scratch(c, 11, (size_t)(nn + 1) * 4, &p11)) ||
        (rc = ctx_scratch(c, 12, (size_t)(nn + 1) * 4, &p12)) || (rc = ctx_scratch(c, 13, (size_t)nn * 4, &p13)) ||
        (rc = ctx_scratch(c, 15, (size_t)(nn + 1) * 4, &p15)) || (rc = ctx_scratch(c, 16, (size_t)(nn + 1) * 4, &p16)) ||
        (rc = ctx_scratch(c, 17, (size_t)(nn + 1) * 4, &p17)) || (rc = ctx_scratch(c, 18, (size_t)(nn + 1) * 4, &p18)))
        return rc;
    uint32_t *nodes = (uint32_t *)p5, *keys = (uint32_t *)p7, *keys_s = (uint32_t *)p8;
    uint32_t *rank = (uint32_t *)p9, *rank_s = (uint32_t *)p10;
    int *flag = (int *)p11, *fpos = (int *)p12, *cstart = (int *)p13;
    int *nseg = (int *)p15, *npts = (int *)p16, *seg_off = (int *)p17, *pt_off = (int *)p18;
    if (dims == 2)
        emit_nodes_kernel<2><<<grid_of(nw), 256, 0, st>>>(d_buf, W, H, D, P, V, offs, nodes);
    else
        emit_nodes_kernel<3><<<grid_of(nw), 256, 0, st>>>(d_buf, W, H, D, P, V, offs, nodes);
    // components
    uf_init_kernel<<<grid_of(npx), 256, 0, st>>>(V, par, npx);
    if (dims == 2)
        uf_hook_kernel<2><<<grid_of(npx), 256, 0, st>>>(V, W, H, D, par);
    else
        uf_hook_kernel<3><<<grid_of(npx), 256, 0, st>>>(V, W, H, D, par);
    node_keys_kernel<<<grid_of(nn), 256, 0, st>>>(par, nodes, nn, keys);
    iota_kernel<<<grid_of(nn), 256, 0, st>>>(rank, nn);
    // stable sort of (component, rank): keeps raster order inside a component
    {
        size_t tb = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, tb, keys, keys_s, rank, rank_s, nn, 0, 32, st);
        void *tmp;
        if ((rc = ctx_scratch(c, 14, tb, &tmp))) return rc;
        if ((e = cub::DeviceRadixSort::SortPairs(tmp, tb, keys, keys_s, rank, rank_s, nn, 0, 32, st)) != cudaSuccess)
            return cuda_fail(e, "component sort");
    }
    comp_flags_kernel<<<grid_of(nn), 256, 0, st>>>(keys_s, nn, flag);
    cudaMemsetAsync(flag + nn, 0, 4, st);
    if ((e = exscan(c, 14, flag, fpos, nn + 1, st)) != cudaSuccess) return cuda_fail(e, "component scan");
    comp_starts_kernel<<<grid_of(nn), 256, 0, st>>>(flag, fpos, nn, cstart);
    int ncomp = 0;
    if ((e = cudaMemcpyAsync(&ncomp, fpos + nn, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return cuda_fail(e, "component count");
    // sorted node raster indices nodes[rank_s[k]] (keys are no longer needed)
    uint32_t *snodes = keys;
    gather_kernel<<<grid_of(nn), 256, 0, st>>>(nodes, rank_s, snodes, nn);
    // bounds of every component's output, and its temporary ranges
    void *p23, *p24, *p26;
    if ((rc = ctx_scratch(c, 23, (size_t)npx * 4, &p23)) ||
        (rc = ctx_scratch(c, 24, (size_t)(ncomp + 1) * 6 * 4, &p24)) ||
        (rc = ctx_scratch(c, 26, (size_t)(nn + 1) * 2 * 4, &p26)))
        return rc;
    uint32_t *pxcnt = (uint32_t *)p23;
    int *branches = (int *)p24, *cpx = branches + (ncomp + 1), *bpts = cpx + (ncomp + 1),
        *bsegs = bpts + (ncomp + 1), *cpb = bsegs + (ncomp + 1), *csb = cpb + (ncomp + 1);
    cudaMemsetAsync(pxcnt, 0, (size_t)npx * 4, st);
    cudaMemsetAsync(branches, 0, (size_t)(ncomp + 1) * 4, st);
    comp_px_kernel<<<grid_of(npx), 256, 0, st>>>(V, par, npx, pxcnt);
    comp_sums_kernel<<<grid_of(nn), 256, 0, st>>>(V0, snodes, keys_s, flag, fpos, pxcnt, nn, branches, cpx);
    comp_bounds_kernel<<<grid_of(ncomp + 1), 256, 0, st>>>(branches, cpx, ncomp, bpts, bsegs);
    if ((e = exscan(c, 14, bpts, cpb, ncomp + 1, st)) != cudaSuccess ||
        (e = exscan(c, 14, bsegs, csb, ncomp + 1, st)) != cudaSuccess)
        return cuda_fail(e, "component bounds scan");
    int tb[2] = {0, 0};
    if ((e = cudaMemcpyAsync(&tb[0], cpb + ncomp, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaMemcpyAsync(&tb[1], csb + ncomp, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return cuda_fail(e, "component bounds");
    if (tb[0] < 0 || tb[1] < 0) return fail(BGT_ERR_LIMIT, "segment output bound exceeds 2^31 entries");
    const size_t Tp = (size_t)tb[0], Ts = (size_t)tb[1];
    const size_t t_x = 0, t_y = align16(Tp * 2 + 2), t_z = t_y + align16(Tp * 2 + 2), t_rel = t_z + align16(Tp * 2 + 2),
                 t_end = t_rel + align16(Ts * 4 + 4), t_err = t_end + align16(Ts + 1), t_tot = t_err + 16;
    void *p25;
    if ((rc = ctx_scratch(c, 25, t_tot, &p25))) return rc;
    char *tbuf = (char *)p25;
    WalkOut wo{};
    wo.nseg = nseg;
    wo.npts = npts;
    wo.tpo = (int *)p26;
    wo.tso = wo.tpo + (nn + 1);
    wo.cpb = cpb;
    wo.csb = csb;
    wo.tx = (int16_t *)(tbuf + t_x);
    wo.ty = (int16_t *)(tbuf + t_y);
    wo.tz = (int16_t *)(tbuf + t_z);
    wo.trel = (int32_t *)(tbuf + t_rel);
    wo.tend = (uint8_t *)(tbuf + t_end);
    wo.err = (int *)(tbuf + t_err);
    cudaMemsetAsync(wo.err, 0, 4, st);
    // one walk over every component (a warp each), outputs in emission order per component
    const int wgrid = (int)std::min<long long>(((long long)ncomp * 32 + 255) / 256, 148LL * 16);
    if (dims == 2)
        walk_kernel<2><<<wgrid, 256, 0, st>>>(V, V0, W, H, snodes, rank_s, cstart, ncomp, nn, wo);
    else
        walk_kernel<3><<<wgrid, 256, 0, st>>>(V, V0, W, H, snodes, rank_s, cstart, ncomp, nn, wo);
    cudaMemsetAsync(nseg + nn, 0, 4, st);
    cudaMemsetAsync(npts + nn, 0, 4, st);
    if ((e = exscan(c, 14, nseg, seg_off, nn + 1, st)) != cudaSuccess) return cuda_fail(e, "segment scan");
    if ((e = exscan(c, 14, npts, pt_off, nn + 1, st)) != cudaSuccess) return cuda_fail(e, "point scan");
    int tot[3] = {0, 0, 0};
    if ((e = cudaMemcpyAsync(&tot[0], seg_off + nn, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaMemcpyAsync(&tot[1], pt_off + nn, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaMemcpyAsync(&tot[2], wo.err, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return cuda_fail(e, "segment totals");
    if (tot[2]) return fail(BGT_ERR_LIMIT, "segment output outgrew its bound");
    const int S = tot[0], Np = tot[1];
    // output block: start[S+1] int32, is_end[S] u8, px, py (pz) int16[Np]
    const size_t o_start = 0, o_end = align16((size_t)(S + 1) * 4), o_px = o_end + align16((size_t)S + 1),
                 o_py = o_px + align16((size_t)Np * 2 + 2), o_pz = o_py + align16((size_t)Np * 2 + 2),
                 o_tot = o_pz + align16((size_t)Np * 2 + 2);
    void *p19;
    if ((rc = ctx_scratch(c, 19, o_tot, &p19))) return rc;
    char *ob = (char *)p19;
    int32_t *o_st = (int32_t *)(ob + o_start);
    uint8_t *o_ie = (uint8_t *)(ob + o_end);
    int16_t *o_x = (int16_t *)(ob + o_px), *o_y = (int16_t *)(ob + o_py), *o_z = (int16_t *)(ob + o_pz);
    const int pgrid = (int)std::min<long long>(((long long)nn * 32 + 255) / 256, 148LL * 16);
    if (dims == 2)
        place_kernel<2><<<pgrid, 256, 0, st>>>(wo, seg_off, pt_off, nn, o_st, o_ie, o_x, o_y, o_z);
    else
        place_kernel<3><<<pgrid, 256, 0, st>>>(wo, seg_off, pt_off, nn, o_st, o_ie, o_x, o_y, o_z);
    cudaMemcpyAsync(o_st + S, pt_off + nn, 4, cudaMemcpyDeviceToDevice, st);
    out->nseg = S;
    out->npts = Np;
    out->start = o_st;
    out->is_end = o_ie;
    out->px = o_x;
    out->py = o_y;
    out->pz = dims == 3 ? o_z : nullptr;
    return BGT_OK;
}

// The same, with the segment arrays in the context's pinned memory.
int segments_result(bgt_ctx *c, int dims, const uint32_t *d_buf, int W, int H, int D, int P, SegResult *out)
{
    SegResult &r = *out;
    int rc = 1;
    if ((long long)W * H * D < (1LL << 32) - 1 && !getenv("BGT_SEGMENTS_PIXEL_WALK"))
        rc = segments_graph(c, dims, d_buf, W, H, D, P, nullptr, &r);
    if (rc != 1) return rc;
    // the pixel walk leaves its arrays on the device, one behind the other
    rc = segments_device_arrays(c, dims, d_buf, W, H, D, P, &r.dev);
    if (rc != BGT_OK) return rc;
    r.nseg = r.dev.nseg;
    r.npts = r.dev.npts;
    if (r.nseg == 0) return BGT_OK;
    const char *first = (const char *)r.dev.start;
    const size_t span = (size_t)((const char *)((dims == 3 ? r.dev.pz : r.dev.py) + r.npts) - first);
    void *pin = nullptr;
    if ((rc = ctx_pinned(c, span, &pin))) return rc;
    cudaError_t e = cudaMemcpyAsync(pin, first, span, cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(e, "segment readback");
    auto host = [&](const void *d) { return (const char *)pin + ((const char *)d - first); };
    r.start = (const int32_t *)host(r.dev.start);
    r.is_end = (const uint8_t *)host(r.dev.is_end);
    r.px = (const int16_t *)host(r.dev.px);
    r.py = (const int16_t *)host(r.dev.py);
    r.pz = dims == 3 ? (const int16_t *)host(r.dev.pz) : nullptr;
    return BGT_OK;
}

// The same, with the segment arrays copied to host memory (malloc).
int segments_packed(bgt_ctx *c, int dims, const uint32_t *d_buf, int W, int H, int D, int P, HostSegs *out)
{
    *out = HostSegs();
    SegResult r;
    const int rc = segments_result(c, dims, d_buf, W, H, D, P, &r);
    if (rc != BGT_OK) return rc;
    const int S = r.nseg, Np = r.npts;
    out->nseg = S;
    out->npts = Np;
    out->start = (int32_t *)malloc((size_t)(S + 1) * 4);
    out->is_end = (uint8_t *)malloc((size_t)S + 1);
    out->px = (int16_t *)malloc((size_t)Np * 2 + 2);
    out->py = (int16_t *)malloc((size_t)Np * 2 + 2);
    out->pz = dims == 3 ? (int16_t *)malloc((size_t)Np * 2 + 2) : nullptr;
    if (!out->start || !out->is_end || !out->px || !out->py || (dims == 3 && !out->pz)) {
        free_host_segs(out);
        return fail(BGT_ERR_NOMEM, "host allocation of segment arrays");
    }
    out->start[0] = 0;
    if (S > 0) {
        memcpy(out->start, r.start, (size_t)(S + 1) * 4);
        memcpy(out->is_end, r.is_end, (size_t)S);
        memcpy(out->px, r.px, (size_t)Np * 2);
        memcpy(out->py, r.py, (size_t)Np * 2);
        if (dims == 3) memcpy(out->pz, r.pz, (size_t)Np * 2);
    }
    ctx_pinned_done(c);
    return BGT_OK;
}

void free_host_segs(HostSegs *s)
{
    free(s->start);
    free(s->is_end);
    free(s->px);
    free(s->py);
    free(s->pz);
    *s = HostSegs();
}

}  // namespace bgt
