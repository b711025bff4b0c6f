// hostpix.h -- pixels <-> bit words on the host: the binarisation of every pixel
// type and its 0/1 output, on all cores, so that a host array crosses the link
// as one bit per pixel.
#pragma once
#include <cstddef>
#include <cstdint>

namespace bgt {

// Pack the w x h x d array `in` (mode 0: 2D foreground rule, 1: 3D rule) into
// H x D rows of P words: bit b of word j = pixel 32 j + b; rows and planes past
// the array are zero.
void host_pack(int dtype, int mode, const void *in, int w, int h, int d, int H, int D, int P, uint32_t *out);
// The way back: w x h x d values 0/1 of the pixel type.
void host_unpack(int dtype, const uint32_t *words, int w, int h, int d, int P, void *out);

// Whether packing an array of `bytes` bytes in pixels of `pixel` bytes on the host is
// faster than sending it over the link, by where it lies and how many worker
// threads there are.  us per Thinning call packed / sent, by CPUs of the process:
//                        1            2            3            4         16
//   pageable
//     1024^2 uint8     253/279      186/283      175/272      162/277    167/264
//     2048^2 uint8     733/674      509/717      381/680      397/715    376/694
//     4096^2 uint8    2740/2316    1778/2322    1336/2575    1379/2393  1016/2282
//     256^3 uint8     3880/2139    1789/2301    1401/2222    1233/2217   968/2188
//     int16, 12 MB    3004/1726    1797/1681    1256/1734    1062/1744   849/1781
//     2048^2 float    1791/1998    1025/2144     849/2218     775/2122   451/2039
//   pinned
//     2048^2 uint8                  448/296                   355/297    330/297
//     int16, 12 MB                 1603/748                  1032/745    817/744
//     2048^2 float                 1123/758                   600/758    450/756
// A second and a fourth thread that call at the same time, and find the workers
// busy, gain more: 4096^2 uint8 1549/3572 and 2293/7262.
bool host_pack_pays(size_t pixel, size_t bytes, bool pinned, int workers);
// Worker threads beside the caller (started on first use).
int host_workers();

// The worker threads live while some context does (retained and released by each).
void host_pool_retain();
void host_pool_release();

}  // namespace bgt
