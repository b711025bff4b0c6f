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

// The worker threads live while some context does (retained and released by each).
void host_pool_retain();
void host_pool_release();

}  // namespace bgt
