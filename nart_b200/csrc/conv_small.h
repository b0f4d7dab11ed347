// The one-tile-per-CTA convolution kernel for launches that do not fill the GPU (conv_small_sm100.cu): its arguments,
// and how a launch is cut for it.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

// Tiles whose activations are loaded once for all taps.  One TMA box holds the tile's pixels and the ring around them that the
// window reaches, `pitch` pixels a row; the accumulator row of output pixel (x, y) of the tile is y * pitch + x, and a tap's
// operand is the same box from a later row on: the descriptor's start address moves, the swizzle being a function of the
// absolute address.  The rows between the tile's lines belong to no pixel.  A strided conv has one box per parity plane.
constexpr int kHaloTaps = 16;
struct HaloTiles {
    int planes;                        // parity planes with a tap, 1 to 4
    int tw, th, pitch;                 // output pixels a tile (one image); (th - 1) * pitch + tw <= 128 in the small kernel
    int tap_row, tap_col;              // between the numbers of taps that are neighbours in a plane, along its rows and columns
    int taps_h[4], taps_w[4], tap0[4]; // per plane: its taps, rows and columns, and the first one's number
    int dx[4], dy[4], rows[4];         // the box's first pixel against the tile's, its pixels (pitch * lines)
    uint8_t parity[4];                 // row parity * 2 + column parity
    int span;                          // pixels that the operands of a box reach over
};
// What the boxes depend on: the window.  row_pixels: the columns of the window that one operand row holds, 0 for one.
struct HaloWindow {
    int r, s, stride_h, stride_w, pad_h, pad_w;
    int width;                         // pixels an operand row holds; 1, or (ConvIgemmPlan::quads) all those of a window's row: s is 1 then
    int ring_w = 0, ring_h = 0;        // pixels beside the tile's, along each axis
    HaloWindow(int r, int s, int stride_h, int stride_w, int pad_h, int pad_w, int row_pixels = 0, int width = 1);
    bool fits() const { return r * s <= kHaloTaps && (r * s >= 2 || width > 1) && ring_h <= 64; }
};
// Planes and taps from h.tw, h.th and h.pitch; the eight-row groups of an operand lie `group` pixels apart.
void halo_planes(const HaloWindow &win, int group, HaloTiles *h);
// The tiles of at most 128 accumulator rows that cover an ow x oh output best; false where there are too many taps.
bool halo_tiles(const HaloWindow &win, int ow, int oh, HaloTiles *h);
// The high word of the descriptor of a box's operand, from that of the weights: the eight-row groups `group` pixels of `pitch` bytes
// apart; quads: not swizzled.
__host__ __device__ inline uint32_t halo_desc_hi(uint32_t desc_hi, int group, int pitch, int quads)
{
    return (desc_hi & (quads ? 0x1fffc000u : ~0x3fffu)) | (uint32_t)((group * pitch) >> 4);
}

struct alignas(64) SmallMaps {
    CUtensorMap a[4];   // activations, one per (row parity, column parity) of a strided conv
    CUtensorMap b;      // weights [kpad][R*S*C], boxes of bn rows
    CUtensorMap ones;   // 16 rows, the first all ones: the window-sum column of a weight zero point other than 128
};

struct SmallArgs {
    int n, oh, ow, cout;
    int r, s, pad_h, pad_w, stride_h, stride_w;
    int tw_sh, th_sh, tn;              // M-tile box (ow, oh, image) of 128 pixels: log2, log2, images
    int tiles_w, tiles_h, n_tiles_n;
    int bk, kblocks, cchunks;          // k-block bytes per pixel, k-blocks of a tile, k-blocks per tap
    int cpad, last_steps;              // weights' pitch per tap; 32-byte steps of a tap's last k-block that hold channels
    int bn;                            // output channels per tile
    int split;                         // CTAs (one cluster) that share a tile's k-blocks: 1, 2, 4 or 8
    int slots;                         // k-blocks in flight
    int a_wide;                        // see IgemmArgs::a_wide
    uint32_t idesc, tmem_cols;
    int form;                          // EpiForm, and its constants (see IgemmArgs)
    const int32_t *off32;              // [n_cls][kpad]
    const int32_t *mul, *shift;        // [kpad]
    int ushift, rnd_hi;
    const uint8_t *row_cls, *col_cls;  // [oh], [ow]
    int n_col_cls, n_cls, kpad;
    int ozp, qmax, relu_lo;
    uint32_t out_flip;                 // 0x80808080 for int8 outputs, else 0
    int wzp_d;                         // weight zero point - 128; not 0: the tile has the window-sum column
    uint8_t *y;
    const uint8_t *res;                // not nullptr: sum = eltwise SUM of y and res (constants as in IgemmArgs)
    uint8_t *sum;
    int r_m[2], r_add[2], r_b[2];
    int r_s0, r_ozp, r_lo;
    int *status;
    const uint8_t *next_ro;            // see IgemmArgs::next_ro
    uint32_t next_ro_bytes;
};

// The kernel with one box of activations for several taps: its boxes in flight, a_slot_bytes of shared memory each, and
// a_pitch, quads as in IgemmBoxArgs.
struct SmallBoxArgs : SmallArgs {
    HaloTiles halo;
    int a_slots, a_pitch, quads;
    uint32_t a_slot_bytes;
};

// How to cut m_tiles x (k output channels) x kblocks for this kernel: channels per tile and CTAs per tile.  taps, box_rows: taps of
// the window and pixels of the boxes of a channel chunk (HaloTiles), 0 for a box per tap.  *cost: the time to beat (0: the
// persistent kernel's, with bn_p channels per tile); false where this kernel does not.
bool conv_small_pick(int m_tiles, int k, int kblocks, int bk, bool wzp, int bn_p, int taps, int box_rows, double *cost, int *bn, int *split);
// Completes bn-dependent fields (slots, idesc, tmem_cols) and launches.
size_t conv_small_smem(SmallBoxArgs &a, bool box, bool act_signed);
int conv_small_launch(const SmallMaps &maps, const SmallBoxArgs &a, bool box, int m_tiles, size_t smem, size_t bytes, cudaStream_t st);
int conv_small_warm();

}  // namespace b200
