// What the convolution entry point (conv_tcgen05.cu) and the persistent kernels
// (conv_persistent_tcgen05.cu) share.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

namespace mdc {

struct ConvShape {
  const float *x, *w, *bias, *add;
  float *out;
  int64_t N, IC, H, W, OC, KH, KW, OH, OW, PHL, PWL, SH, SW, DH, DW;
  bool relu;
};

// The tiles of conv_halo_tcgen05.cu.  A tile is 128 output pixels whose windows lie in one region of the input:
//   rect    16 rows of 8 pixels;
//   flat    128 pixels one after the other in rows `Wv` apart (stride 1 only), the margin between rows included.
// Images follow one another `Hv` input rows apart (`HvO` output rows), the rows between them being padding, so a tile
// may hold the end of one image and the start of the next.  A region is kept by classes of rows and columns modulo the
// stride, in each of which the pixels that a tap reads for neighbouring outputs are neighbours.
struct HaloPlan {
  int flat;
  int Wv, Hv, HvO;
  int IW, px;               // input pixels per row of the region (rect), and in all
  int pitch;                // pixels from one row of a class to the next
  int class_px, plane_px;   // pixels of a class / of all classes
  int tiles_w;              // tiles side by side (1 when flat)
  int64_t m_tiles;
};

// Strides 1 and 2.  False where the form cannot describe the shape.
inline bool halo_plan(const ConvShape &c, bool flat, HaloPlan *h) {
  if (c.SH > 2 || c.SW > 2 || (flat && (c.SH != 1 || c.SW != 1))) return false;
  const int64_t span_h = (c.KH - 1) * c.DH, span_w = (c.KW - 1) * c.DW;
  if (span_h > 1024 || span_w > 1024 || c.PHL > 4096 || c.PWL > 4096) return false;
  // distance between images (rows): what windows reach before the first and past the last element is padding
  auto pitch = [](int64_t size, int64_t out, int64_t before, int64_t span, int64_t stride) {
    const int64_t after = (out - 1) * stride - before + span - (size - 1);
    const int64_t pad = before > after ? before : after, need = size + (pad > 0 ? pad : 0);
    const int64_t outs = (need + stride - 1) / stride;
    return outs > out ? outs : out;
  };
  const int64_t HvO = pitch(c.H, c.OH, c.PHL, span_h, c.SH), Wv = flat ? pitch(c.W, c.OW, c.PWL, span_w, 1) : 0;
  const int64_t rows = (c.N - 1) * HvO + c.OH;  // of outputs, margins between images included
  if ((rows + 16) * c.SH + span_h > (1 << 30)) return false;
  h->flat = flat ? 1 : 0;
  h->Wv = static_cast<int>(Wv), h->HvO = static_cast<int>(HvO), h->Hv = static_cast<int>(HvO * c.SH);
  int64_t px, plane;
  if (flat) {
    if ((rows + 2) * Wv + span_h * Wv > (1 << 30)) return false;
    h->tiles_w = 1, h->m_tiles = ((rows - 1) * Wv + c.OW + 127) / 128;
    h->IW = static_cast<int>(Wv), h->pitch = static_cast<int>(Wv);
    plane = px = 128 + span_h * Wv + span_w;
    h->class_px = static_cast<int>(px);
  } else {
    h->tiles_w = static_cast<int>((c.OW + 7) / 8), h->m_tiles = (rows + 15) / 16 * h->tiles_w;
    const int64_t IW = 7 * c.SW + span_w + 1, IH = 15 * c.SH + span_h + 1;
    h->IW = static_cast<int>(IW), h->pitch = static_cast<int>((IW + c.SW - 1) / c.SW);
    h->class_px = static_cast<int>(h->pitch * ((IH + c.SH - 1) / c.SH));
    px = IW * IH, plane = static_cast<int64_t>(h->class_px) * c.SH * c.SW;
  }
  if (plane > 2048) return false;
  h->px = static_cast<int>(px), h->plane_px = static_cast<int>(plane);
  return true;
}

// A strided 1 x 1 window reads one pixel in SH x SW: makes `c` the convolution without stride or padding on a copy that
// holds the output's pixels only.  False, and nothing changed, for other shapes.
bool conv_sampled(ConvShape &c);

// Launches the rewriting of the operands: the input of `call` as NHWC fp16, channels zero-padded to a multiple of 8, images
// of copy_h x copy_w pixels (zeros beyond the input's, or the output's pixels where `sampled`); the filter as [OC][block of
// 64 channels][tap][64].  `c` is `call`, or what conv_sampled made of it.
bool conv_prepare(const ConvShape &c, const ConvShape &call, bool sampled, int64_t copy_h, int64_t copy_w, void *x16, void *w16,
                  cudaStream_t s);

// Where conv_halo_kernel takes a call, and in which form; `c` after conv_sampled.  The other kernels are the im2col
// kernel (16 channels or more) and the gather kernel.  us a call, inputs changing, theirs / the form's:
//   copy, windows of 25 taps and more   26x192x60x37->32 5x5 73 / 57, 16x32x113x91->32 7x7 105 / 66, 3x352x54x33->165 7x7
//                                       79 / 64: a k-block costs the im2col kernel at least 340 cycles, these 46 to 64 an MMA
//   copy, 1 x 1                         32x64x56x56->256 73 / 58, 45x192x47x35->32 26 / 21, 2x32x179x207->131 38 / 24
//   copy, up to 64 outputs              16x16x112x112->16 31 / 16, 32x64x56x56->64 with residual 26.9 / 25.1
//   copy, few tiles and many channels   17x448x13x9->113 18.2 / 16.4, 1x160x9x7->96 10.3 / 9.2, 32x512x7x7->512 25.0 / 23.1
// A call of one round of tiles and up to ten k-blocks is bound by its launches, and this kernel's parameters are the longer
// ones: 2x32x20x20->32 7.9 / 8.0, 9x96x21x30->32 1x1 stride 2 7.9 / 8.1.
// Elsewhere the im2col kernel's stores win, whose 32 pixels of a warp are neighbours in memory: 32x128x28x28->128 19.2 / 20.4,
// 25x224x38x43->192 49.8 / 54.2, 34x32x23x21->352 22.2 / 23.8.  Rect keeps to whole sectors where rows of the output are
// multiples of eight pixels (32x64x56x56->64 19.2, flat 25.2); flat wastes less elsewhere (32x256x14x14->256 17.4, rect 20.7).
//   direct, up to 15 channels           16x3x224x224->32 7x7 143 / 79, 16x3x128x128->64 5x5 43 / 33, 4x12x100x100->64 5x5 29 / 11.5;
//                                       but 16x3x256x256->64 3x3 64 / 69, 30x3x250x256->32 3x3 stride 2 44 / 57, and windows
//                                       that reach far: 18x3x18x29->96 7x7 dilation 2 12.3 / 12.8
//   direct, stride 2, up to 32 channels 42x32x97x102->32 5x5 54 / 46, 2x32x22x23->32 7x7 15.5 / 13.5; but 1x32x165x248->192 28 / 31
enum class ConvForm { kOther, kCopyRect, kCopyFlat, kDirectRect, kDirectFlat };
inline ConvForm conv_form(const ConvShape &c, int sms) {
  const int64_t taps = c.KH * c.KW, pixels = c.N * c.OH * c.OW;
  const bool unit = c.SH == 1 && c.SW == 1;
  HaloPlan h;
  auto direct = [&]() {
    if (c.SH > 2 || c.SW > 2) return ConvForm::kOther;
    return unit && c.OW < 48 && halo_plan(c, true, &h) ? ConvForm::kDirectFlat : ConvForm::kDirectRect;
  };
  if (c.IC < 16) return taps >= 25 && (c.KH - 1) * c.DH <= 8 && (c.KW - 1) * c.DW <= 8 ? direct() : ConvForm::kOther;
  if (!unit) return c.IC <= 32 && taps >= 25 && (c.OC <= 64 || pixels < 5000) ? direct() : ConvForm::kOther;
  const bool few = (pixels + 127) / 128 * ((c.OC + 63) / 64) <= sms;
  if (few && (c.IC + 63) / 64 * taps <= 10) return ConvForm::kOther;
  if (taps > 1 && c.OC > 64 && c.IC < 384 && !(taps >= 25 && (c.OC <= 128 || c.IC >= 64)) && !(few && c.IC >= 64)) return ConvForm::kOther;
  if (taps > 1 && c.OW % 8 == 0) return ConvForm::kCopyRect;
  return halo_plan(c, true, &h) && h.px <= 512 ? ConvForm::kCopyFlat : ConvForm::kCopyRect;
}

// Runs the convolution on conv_halo_kernel; false (and nothing launched) when the shape is not one for it.
bool conv_halo(const ConvShape &c, cudaStream_t s);

// Whether the shape is one that the persistent kernels take.
bool conv_persistent_takes(const ConvShape &c);

// Runs the convolution on the persistent kernels; false (and nothing launched) when the shape is one
// that they do not take or there is no memory for their operands.
bool conv_persistent(const ConvShape &c, cudaStream_t s);

}  // namespace mdc
