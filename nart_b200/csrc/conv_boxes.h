// Tiles of the persistent convolution kernel whose activations are loaded once for all taps (kernel modes 4 and 5).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

// Tiles whose activations are loaded once for all taps.  One TMA box holds the tile's pixels and the ring around them that the
// window reaches, `pitch` pixels a row, and a tap's operand is the same box from a later row on: the descriptor's start address
// moves, the swizzle being a function of the absolute address.  With a vertical stride there is a box per parity of the rows; columns
// lie side by side (a horizontal stride only with windows of one column).
struct HaloTiles {
    int planes;                        // row parities with a tap, 1 or 2
    int tw, th, pitch;                 // output pixels a tile (one image)
    int tap_row;                       // between the numbers of taps that are neighbours in a plane, along its columns
    int taps_w, dx;                    // taps a row; the box's first column against the tile's
    int taps_h[2], tap0[2];            // per plane: rows of taps, the first tap's number
    int dy[2], rows[2];                // the box's first line against the tile's, its pixels (pitch * lines)
    uint8_t row_parity[2], col_parity;
    int span;                          // pixels that the operands of a box reach over
};
// What the boxes depend on: the window.  row_pixels: the columns of the window that one operand row holds, 0 for one.
struct HaloWindow {
    int r, s, stride_h, stride_w, pad_h, pad_w;
    int width;                         // pixels an operand row holds; 1, or (ConvIgemmPlan::quads) all those of a window's row: s is 1 then
    int ring_w = 0, ring_h = 0;        // pixels beside the tile's, along each axis
    HaloWindow(int r, int s, int stride_h, int stride_w, int pad_h, int pad_w, int row_pixels = 0, int width = 1);
    // (up to sixteen taps and 64 lines of ring: nothing in the kernel asks for it, larger windows have not been measured)
    bool fits() const { return (stride_w == 1 || s == 1) && r * s <= 16 && (r * s >= 2 || width > 1) && ring_h <= 64; }
};
// Planes and taps from h.tw, h.th and h.pitch; the eight-row groups of an operand lie `group` pixels apart.
void halo_planes(const HaloWindow &win, int group, HaloTiles *h);
// The high word of the descriptor of a box's operand, from that of the weights: the eight-row groups `group` pixels of `pitch` bytes
// apart; quads: not swizzled.
__host__ __device__ inline uint32_t halo_desc_hi(uint32_t desc_hi, int group, int pitch, int quads)
{
    return (desc_hi & (quads ? 0x1fffc000u : ~0x3fffu)) | (uint32_t)((group * pitch) >> 4);
}

}  // namespace b200
