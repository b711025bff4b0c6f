// pixels.cuh -- pixels <-> bit words: the binarisation of every pixel type on
// the way in, 0/1 in the pixel type on the way out.  Shared by the batch-wide
// pack and unpack kernels and by the resident kernel, which reads and writes
// the pixels of its instances itself.
#pragma once
#include <cstdint>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"

namespace bgt {

// Foreground tests of the reference's binarisation.  2D: (unsigned int)v > 0
// evaluated on the device (2D/CUDA_DeviceHelperFunctions.cuh:101), i.e. a
// saturating conversion for floating types.  3D: int(v) > 0 as the host
// evaluates it (3D/CenterlineExtraction.cpp:44; x86-64 conversion of
// out-of-range floats gives INT_MIN).
template <typename T>
__device__ __forceinline__ bool fg2(T v) { return (unsigned int)v > 0u; }
template <>
__device__ __forceinline__ bool fg2<bool>(bool v) { return v; }

template <typename T>
__device__ __forceinline__ bool fg3(T v) { return (int)v > 0; }
template <>
__device__ __forceinline__ bool fg3<float>(float v) { return v >= 1.0f && v < 2147483648.0f; }
template <>
__device__ __forceinline__ bool fg3<double>(double v) { return v >= 1.0 && v < 2147483648.0; }
template <>
__device__ __forceinline__ bool fg3<bool>(bool v) { return v; }

__device__ __forceinline__ int dtype_bytes(int dtype)
{
    return dtype == BGT_F64 ? 8 : (dtype == BGT_U32 || dtype == BGT_I32 || dtype == BGT_F32) ? 4
                                  : (dtype == BGT_U16 || dtype == BGT_I16) ? 2 : 1;
}

// 4 bytes -> 4 bits "byte != 0" (bit 28 + k for byte k, anything below them) with
// integer ALU ops only: the low seven bits of each byte plus 0x7F carry into
// the byte's MSB exactly when they are nonzero (no carry leaves the byte), and
// OR-ing the byte back in covers the MSB itself; multiplying the MSBs by 0x00204081
// moves bits 7, 15, 23, 31 to 28..31 without carries.  With `neg` all ones, "byte > 0"
// of signed bytes: those whose own MSB is set are taken out again.
__device__ __forceinline__ uint32_t nz4_high(uint32_t c, uint32_t neg = 0u)
{
    return (((((c & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | c) & ~(c & neg)) & 0x80808080u) * 0x00204081u;
}
__device__ __forceinline__ uint32_t nz4_to_bits(uint32_t c, uint32_t neg = 0u) { return nz4_high(c, neg) >> 28; }
// 16 bytes -> 16 bits, the low bits of w above them: a funnel shift per 4 bytes
__device__ __forceinline__ uint32_t nz16_to_bits(const uint4 &c, uint32_t neg, uint32_t w)
{
    w = __funnelshift_l(nz4_high(c.w, neg), w, 4);
    w = __funnelshift_l(nz4_high(c.z, neg), w, 4);
    w = __funnelshift_l(nz4_high(c.y, neg), w, 4);
    return __funnelshift_l(nz4_high(c.x, neg), w, 4);
}

// 4 bits -> 4 bytes of value 0/1 (bit k to byte k): the multiplier places bit
// k at 8k and the mask drops the other partial products (all at distinct bits).
__device__ __forceinline__ uint32_t bits4_to_bytes(uint32_t nib) { return (nib * 0x00204081u) & 0x01010101u; }

// 32 one-byte pixels from p (n < 32 at a row's ragged end) -> "byte != 0"
// bits (neg all ones: "byte > 0", signed), without branches that depend on p's
// alignment: three aligned 16-byte loads (two for an aligned p) cover p .. p+31
// (they may run past the row into the next one, never past the input: `room` =
// bytes readable from p onward, `lead` = bytes readable before p) and are turned
// into bits, 48 of them, which one funnel shift brings into place; bits at and past
// n are cleared.  The load is bound by its instructions (a word takes some
// hundred): shifting the 12 loaded words into place before the conversion
// (two select stages and a funnel shift each) took the resident kernel 1164
// instead of 1154 us on the mixed batch, 96 instead of 94 on a 4096^2 image.  Words too close to either end of the input take the byte loop.
__device__ __forceinline__ uint32_t pack_bytes32(const uint8_t *p, int n, long long room, long long lead,
                                                 uint32_t neg = 0u)
{
    const uintptr_t pa = reinterpret_cast<uintptr_t>(p);
    const unsigned o = (unsigned)(pa & 15u);
    if ((long long)o <= lead && (long long)(o ? 48u - o : 32u) <= room) {
        const uint4 *a16 = reinterpret_cast<const uint4 *>(pa & ~uintptr_t(15));
        const uint4 A = __ldg(a16), B = __ldg(a16 + 1), C = o ? __ldg(a16 + 2) : make_uint4(0, 0, 0, 0);
        const uint32_t w =
            __funnelshift_r(nz16_to_bits(A, neg, nz16_to_bits(B, neg, 0u)), nz16_to_bits(C, neg, 0u), o);
        return n >= 32 ? w : w & ((1u << n) - 1u);
    }
    uint32_t w = 0;
    for (int b = 0; b < n; b++) w |= (uint32_t)(p[b] != 0 && !(p[b] & neg & 0x80u)) << b;
    return w;
}

// The packed word of `cnt` (0..32) one-byte pixels from element `off` of the input.
__device__ __forceinline__ uint32_t pixel_bytes(const IODesc &d, uint32_t off, int cnt, uint32_t neg)
{
    if (cnt <= 0) return 0u;
    const long long total = (long long)d.inW * d.inH * d.inD;
    return pack_bytes32((const uint8_t *)d.in + off, cnt, total - off, off, neg);
}
// the `neg` of an input's pixel type and rule
__device__ __forceinline__ uint32_t pixel_neg(const IODesc &d)
{
    return d.mode == 1 && (d.dtype == BGT_I8 || (d.dtype == BGT_CHAR && std::is_signed<char>::value)) ? 0xffffffffu : 0u;
}

// Wider pixels: the warp builds its 32 lanes' words one after the other, a
// lane per pixel (coalesced whatever the alignment) and a vote per word.  Every
// lane loads, clamped to the input, and each lane masks its own word in the end,
// so that the loads of 16 words are in flight at once (a branch around each
// load left one in flight: the resident kernel on a 1501 x 1003 float image
// 96 -> 85 us, on a 187 x 203 x 161 int16 volume 225 -> 190 us).
template <typename T, int MODE>
__device__ __forceinline__ uint32_t pixel_vote(const T *p, uint32_t last, uint32_t off, int cnt)
{
    constexpr int U = 16;
    const int lane = threadIdx.x & 31;
    uint32_t w = 0;
#pragma unroll
    for (int k0 = 0; k0 < 32; k0 += U) {
        T v[U];
#pragma unroll
        for (int k = 0; k < U; k++) v[k] = __ldg(p + min(__shfl_sync(kFull, off, k0 + k) + (uint32_t)lane, last));
#pragma unroll
        for (int k = 0; k < U; k++) {
            const uint32_t m = __ballot_sync(kFull, MODE == 0 ? fg2<T>(v[k]) : MODE == 1 ? fg3<T>(v[k]) : v[k] != (T)0);
            if (lane == k0 + k) w = m;
        }
    }
    return cnt >= 32 ? w : w & ((1u << cnt) - 1u);
}
template <typename T>
__device__ __forceinline__ uint32_t pixel_vote_mode(const IODesc &d, uint32_t off, int cnt)
{
    const uint32_t last = (uint32_t)d.inW * (uint32_t)d.inH * (uint32_t)d.inD - 1u;
    return d.mode == 0   ? pixel_vote<T, 0>((const T *)d.in, last, off, cnt)
           : d.mode == 1 ? pixel_vote<T, 1>((const T *)d.in, last, off, cnt)
                         : pixel_vote<T, 2>((const T *)d.in, last, off, cnt);
}
// Every lane of the warp calls it (cnt = 0 for none).
static __device__ __noinline__ uint32_t pixel_word_wide(const IODesc &d, uint32_t off, int cnt)
{
    switch (d.dtype) {
    case BGT_U16: return pixel_vote_mode<uint16_t>(d, off, cnt);
    case BGT_I16: return pixel_vote_mode<int16_t>(d, off, cnt);
    case BGT_U32: return pixel_vote_mode<uint32_t>(d, off, cnt);
    case BGT_I32: return pixel_vote_mode<int32_t>(d, off, cnt);
    case BGT_F32: return pixel_vote_mode<float>(d, off, cnt);
    default: return pixel_vote_mode<double>(d, off, cnt);
    }
}

// The same way out: lane l writes pixel l of the warp's k-th word.
template <typename T>
__device__ __forceinline__ void pixel_spread(T *p, uint32_t off, int cnt, uint32_t w)
{
    const int lane = threadIdx.x & 31;
#pragma unroll 4
    for (int k = 0; k < 32; k++) {
        const uint32_t o = __shfl_sync(kFull, off, k), v = __shfl_sync(kFull, w, k);
        const int c = __shfl_sync(kFull, cnt, k);
        if (lane < c) p[(size_t)o + lane] = (T)((v >> lane) & 1u);
    }
}
static __device__ __noinline__ void pixel_store_wide(const IODesc &d, uint32_t off, int cnt, uint32_t w)
{
    switch (dtype_bytes(d.dtype)) {
    case 2: pixel_spread((uint16_t *)d.out, off, cnt, w); break;
    case 4:
        if (d.dtype == BGT_F32) pixel_spread((float *)d.out, off, cnt, w);
        else pixel_spread((uint32_t *)d.out, off, cnt, w);
        break;
    default: pixel_spread((double *)d.out, off, cnt, w); break;
    }
}

// 32-byte-aligned chunk c of the one-byte pixels of `rows` consecutive rows of
// W pixels that start at `out`; bits(r, x) = 32 pixels of row r from x on.  Two 128-bit stores where the chunk lies
// inside the rows and spans at most two of them, bytes otherwise.
template <class Bits>
__device__ __forceinline__ void pixel_chunk(uint8_t *out, uint32_t rows, int W, const FastDiv &dW, uint32_t c, Bits pix)
{
    const uintptr_t o = reinterpret_cast<uintptr_t>(out), end = o + (uintptr_t)rows * W;
    const uintptr_t a = (o & ~uintptr_t(31)) + (uintptr_t)c * 32u;
    const uintptr_t lo = a > o ? a : o, hi = a + 32 < end ? a + 32 : end;
    if (lo >= hi) return;
    const uint32_t f = (uint32_t)(lo - o);
    uint32_t r = fdiv(dW, f);
    int x = (int)(f - r * (uint32_t)W);
    if (hi - lo == 32 && W >= 32) {
        uint32_t bits = pix(r, x);
        if (x + 32 > W) {  // the chunk runs into the next row
            const int n0 = W - x;
            bits = (bits & ((1u << n0) - 1u)) | pix(r + 1, 0) << n0;
        }
        uint4 *q = reinterpret_cast<uint4 *>(a);
        q[0] = make_uint4(bits4_to_bytes(bits & 15u), bits4_to_bytes((bits >> 4) & 15u),
                          bits4_to_bytes((bits >> 8) & 15u), bits4_to_bytes((bits >> 12) & 15u));
        q[1] = make_uint4(bits4_to_bytes((bits >> 16) & 15u), bits4_to_bytes((bits >> 20) & 15u),
                          bits4_to_bytes((bits >> 24) & 15u), bits4_to_bytes(bits >> 28));
        return;
    }
    for (uintptr_t b = lo; b < hi; b++) {
        *reinterpret_cast<uint8_t *>(b) = (uint8_t)(pix(r, x) & 1u);
        if (++x == W) {
            x = 0;
            r++;
        }
    }
}

// Chunk c of a run of n one-byte pixels at `out`; pix(x) = 32 of them from x on.
template <class Bits>
__device__ __forceinline__ void pixel_run_chunk(uint8_t *out, int n, uint32_t c, Bits pix)
{
    const uintptr_t o = reinterpret_cast<uintptr_t>(out), end = o + (uintptr_t)n;
    const uintptr_t a = (o & ~uintptr_t(31)) + (uintptr_t)c * 32u;
    const uintptr_t lo = a > o ? a : o, hi = a + 32 < end ? a + 32 : end;
    if (lo >= hi) return;
    const int x = (int)(lo - o);
    const uint32_t bits = pix(x);
    if (hi - lo == 32) {
        uint4 *q = reinterpret_cast<uint4 *>(a);
        q[0] = make_uint4(bits4_to_bytes(bits & 15u), bits4_to_bytes((bits >> 4) & 15u),
                          bits4_to_bytes((bits >> 8) & 15u), bits4_to_bytes((bits >> 12) & 15u));
        q[1] = make_uint4(bits4_to_bytes((bits >> 16) & 15u), bits4_to_bytes((bits >> 20) & 15u),
                          bits4_to_bytes((bits >> 24) & 15u), bits4_to_bytes(bits >> 28));
        return;
    }
    // an end of the run: whole 4-byte groups, then the bytes left
    for (uintptr_t b = lo; b < hi;) {
        const unsigned k = (unsigned)(b - lo);
        if ((b & 3) == 0 && b + 4 <= hi) {
            *reinterpret_cast<uint32_t *>(b) = bits4_to_bytes((bits >> k) & 15u);
            b += 4;
        } else {
            *reinterpret_cast<uint8_t *>(b) = (uint8_t)((bits >> k) & 1u);
            b++;
        }
    }
}

}  // namespace bgt
