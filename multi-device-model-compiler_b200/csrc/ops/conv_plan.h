// What the convolution entry point (conv_tcgen05.cu) and the persistent kernels
// (conv_persistent_tcgen05.cu) share.
#pragma once

#include <algorithm>
#include <cstddef>
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

// 16 channels fill a quarter of a k-block; below that the gathered patch has fewer k-blocks.
inline bool conv_gathers(const ConvShape &c) { return c.IC < 16; }

// A strided 1 x 1 window reads one pixel in SH x SW: makes `c` the convolution without stride or padding on a copy that
// holds the output's pixels only.  False, and nothing changed, for other shapes.  (33 x 476 x 87 x 56, stride 2: 108 us with
// the whole input rewritten, 65 sampled.)
inline bool conv_sampled(ConvShape &c) {
  if (conv_gathers(c) || c.KH * c.KW != 1 || (c.SH == 1 && c.SW == 1)) return false;
  c.H = c.OH, c.W = c.OW, c.SH = c.SW = c.DH = c.DW = 1, c.PHL = c.PWL = 0;
  return true;
}

// im2col: first and last window origin relative to the first and last column / row of the image.
inline int64_t conv_upper_w(const ConvShape &c) { return (c.OW - 1) * c.SW - c.PWL - (c.W - 1); }
inline int64_t conv_upper_h(const ConvShape &c) { return (c.OH - 1) * c.SH - c.PHL - (c.H - 1); }

constexpr int kDenseMaxOC = 2048;       // bias kept in shared memory
constexpr int kDenseMaxGatherK = 1024;  // entries of the gather's table

// Whether the shape is within the limits of the persistent kernels.
inline bool conv_dense_describes(const ConvShape &call) {
  ConvShape c = call;
  conv_sampled(c);
  const int64_t taps = c.KH * c.KW, span_h = (c.KH - 1) * c.DH, span_w = (c.KW - 1) * c.DW;
  if (c.OC > kDenseMaxOC || taps > 4096 || c.N * c.OH * c.OW * c.OC > (int64_t(1) << 40)) return false;
  if (conv_gathers(c)) return c.IC * taps <= kDenseMaxGatherK && span_h <= 32767 && span_w <= 32767;
  // limits of the im2col tensor map: strides, corners and tap offsets
  const int64_t up_w = conv_upper_w(c), up_h = conv_upper_h(c);
  return c.SW <= 8 && c.SH <= 8 && c.PWL <= 127 && c.PHL <= 127 && up_w >= -128 && up_w <= 127 && up_h >= -128 &&
         up_h <= 127 && span_w <= 255 && span_h <= 255;
}

// Launches the rewriting of the operands: the input of `call` as NHWC fp16, channels zero-padded to a multiple of 8, images
// of copy_h x copy_w pixels (zeros beyond the input's, or the output's pixels where `sampled`); the filter as [OC][block of
// 64 channels][tap][64].  `c` is `call`, or what conv_sampled made of it.
bool conv_prepare(const ConvShape &c, const ConvShape &call, bool sampled, int64_t copy_h, int64_t copy_w, void *x16, void *w16,
                  cudaStream_t s);

// The persistent kernels' tile: width, by the cycles of the busiest CTA: rounds x the slowest of a tile's three engines.
// Loads: about 64 bytes per cycle and SM out of L2 (a gathered k-block about 400 cycles with three
// groups at work, as the gather once was); MMAs: 2 cycles per column and k-block, at least what reading A takes; epilogue:
// about 24 bytes per cycle and SM of HBM.  E.g. 6272 pixels x 256 channels: 147 tiles of 96 columns
// in one round (224 units of load) beat 98 of 128 in one (256) and 49 of 256 (384).
inline int choose_conv_bn(int64_t m_tiles, int64_t OC, int64_t num_kb, bool gather, bool add, int sms) {
  int best = 32;
  double best_cost = 1e300;
  for (int bn = 256; bn >= 32; bn -= 32) {
    if (bn > 32 && bn >= OC + 32) continue;
    const int64_t n_tiles = (OC + bn - 1) / bn;
    const int64_t rounds = (m_tiles * n_tiles + sms - 1) / sms;
    const double load = num_kb * ((gather ? 400.0 : 256.0) + bn * 2.0);
    const double mma = num_kb * (bn < 64 ? 160.0 : bn < 96 ? 192.0 : 2.0 * bn);
    const double epi = bn * (add ? 1024.0 : 512.0) / 24.0;
    double tile = load > mma ? load : mma;
    if (epi > tile) tile = epi;
    const double cost = static_cast<double>(rounds) * tile + epi;
    if (cost < best_cost * 0.97) best_cost = cost, best = bn;
  }
  return best;
}
// The filter stays in shared memory when it is one tile wide, there is a second tile to use it, and it leaves the ring room.
inline bool conv_filter_stays(int64_t num_kb, int bn, int64_t n_tiles, int64_t tiles, int sms) {
  return n_tiles == 1 && tiles > sms && num_kb * bn * 128 <= 100 * 1024;
}

constexpr int kRingMaxStages = 12;
constexpr int kGatherGroups = 3;  // of four warps, that gather alternate k-blocks
// Stages of the persistent kernels' ring in `room` bytes; 0: too few.  Gathered patches are read nine-fold through L1, which
// keeps most of the memory.  A group gathers every third k-block and waits for its stage's previous use by parity alone: it
// knows that the block which its last one replaced has been used, three blocks and the ring back, so with fewer stages than
// groups the use before the previous one would pass for it.
inline int conv_ring_stages(int64_t room, int64_t stage_bytes, bool gather) {
  const int64_t least = gather ? kGatherGroups : 2, most = gather ? 4 : kRingMaxStages;
  const int64_t n = std::min(room / stage_bytes, most);
  return n < least ? 0 : static_cast<int>(n);
}

// Where the values k of a gathered patch lie, as kernel arguments.  Near: in bytes from the window's origin, and which row and
// column of the window have to lie inside the input; one 32-bit sum of an offset and an origin reaches any value, counted from
// `lead` bytes ahead of the input, where the first window may begin.
constexpr int kNearTaps = 256;
struct NearTaps {
  uint32_t lead;
  uint32_t off[kNearTaps];
  uint32_t need[kNearTaps];  // bits 0-15 the row, 16-30 the column; beyond the patch bit 31
};
// Far: in elements from the window's origin, and the row of the input from the origin's << 16 | the column.
struct FarTaps {
  uint32_t off[kDenseMaxGatherK];
  uint32_t pos[kDenseMaxGatherK];
};
inline bool conv_taps_near(const ConvShape &c) {
  return c.IC * c.KH * c.KW <= kNearTaps && c.KH <= 16 && c.KW <= 15 &&
         (c.N * c.IC * c.H * c.W + c.PHL * c.W + c.PWL) * 4 < (int64_t(1) << 32) &&
         (((c.IC - 1) * c.H + (c.KH - 1) * c.DH) * c.W + (c.KW - 1) * c.DW) * 4 < (int64_t(1) << 32);
}
// The tables' entries up to the patch's end in whole eights, which is as far as they are read.  On every call, so counted up: a
// division an entry is time that a small call has no GPU work to hide behind.  Host time of a call with 27 / 135 / 960 values 8.25 /
// 8.88 / 13.9 us with divisions, 8.12 / 8.23 / 8.90 so, 7.97 / 8.00 / 7.89 when the GPU filled a table of its own; the tables' bytes,
// 512 instead of 2048, make no difference.
inline void fill_taps(const ConvShape &c, NearTaps *t) {
  t->lead = static_cast<uint32_t>((c.PHL * c.W + c.PWL) * 4);
  int64_t k = 0;
  for (int64_t ic = 0; ic < c.IC; ++ic)
    for (int64_t kh = 0; kh < c.KH; ++kh) {
      const uint32_t row = static_cast<uint32_t>((ic * c.H + kh * c.DH) * c.W * 4);
      for (int64_t kw = 0; kw < c.KW; ++kw, ++k) t->off[k] = row + static_cast<uint32_t>(kw * c.DW * 4), t->need[k] = 1u << kh | 0x10000u << kw;
    }
  for (; k % 8; ++k) t->off[k] = 0, t->need[k] = 0x80000000u;
}
inline void fill_taps(const ConvShape &c, FarTaps *t) {
  int64_t k = 0;
  for (int64_t ic = 0; ic < c.IC; ++ic)
    for (int64_t kh = 0; kh < c.KH; ++kh) {
      const uint32_t row = static_cast<uint32_t>((ic * c.H + kh * c.DH) * c.W), pos = static_cast<uint32_t>(kh * c.DH << 16);
      for (int64_t kw = 0; kw < c.KW; ++kw, ++k) t->off[k] = row + static_cast<uint32_t>(kw * c.DW), t->pos[k] = pos | static_cast<uint32_t>(kw * c.DW);
    }
  for (; k % 8; ++k) t->off[k] = t->pos[k] = 0;
}

// How conv_halo_kernel runs a call: in a copy of the input or directly (see there), by rect or flat tiles.
enum class ConvForm { kOther, kCopyRect, kCopyFlat, kDirectRect, kDirectFlat };
inline bool form_copies(ConvForm f) { return f == ConvForm::kCopyRect || f == ConvForm::kCopyFlat; }
inline bool form_flat(ConvForm f) { return f == ConvForm::kCopyFlat || f == ConvForm::kDirectFlat; }

constexpr int kHaloMaxOC = 2048;           // bias kept in shared memory
constexpr int kHaloMaxTaps = 64;           // entries of its table of taps, or pairs of them
constexpr int kHaloFilterStages = 12;
constexpr int kHaloInputWarps = 12;        // of the direct forms
constexpr size_t kHaloMaxSmem = 220 * 1024;
constexpr int64_t kHaloAddSmem = 150 * 1024;  // beside a residual, where fewer stages do

// A tile of conv_halo_kernel and what follows from it.
struct HaloTile {
  HaloPlan h;
  int ncb, last_steps;        // blocks of 64 channels; sixteens of the last one's channels
  int pairs;                  // up to eight channels: MMAs of two taps
  int num_kb;                 // filter blocks of 64 k
  int mmas;                   // of a tile
  int chain, splits;          // few channels: MMAs per sum, and sums (see halo_chain)
  int qb;                     // 32-pixel pieces of a region
  int boxes, box_px;          // loads that make up a copy's region, and the pixels of one
  int bn, resident, stages, filter_stages, filter_kbs;
  uint32_t region_bytes, regions_bytes;  // of a stage / of all
  size_t smem;
};

// Shared memory: regions, then the filter whole or a ring of its k-blocks, several to a stage where they are short (a
// hand-over costs as much as the MMAs of 64 columns).  False where it does not fit.
inline bool fit_halo(HaloTile *t, bool copy, bool add, int64_t OC, int bn, int sms) {
  const int64_t fixed = 2048 + (OC + 31) / 32 * 128, room = static_cast<int64_t>(kHaloMaxSmem) - fixed;
  const int64_t num_kb = t->num_kb, b_bytes = bn * 128, filter = num_kb * b_bytes, region = t->region_bytes;
  const int64_t most = region <= 16 * 1024 ? 8 : 4;
  const int64_t tiles = t->h.m_tiles * ((OC + bn - 1) / bn);
  const bool resident = OC <= bn && tiles > sms && filter + 2 * region <= room;
  int64_t kbs = 32 * 1024 / b_bytes;
  if (kbs > 4) kbs = 4;
  if (kbs > num_kb) kbs = num_kb;
  const int64_t blocks = (num_kb + kbs - 1) / kbs, least = blocks < 3 ? blocks : 3;
  int64_t n = (room - (resident ? filter : least * kbs * b_bytes)) / region;
  if (n > most) n = most;
  // as many stages as regions that the input warps' pieces reach over: a stage's barrier is then never two uses behind
  const int64_t reach = copy ? 0 : (kHaloInputWarps + t->qb - 1) / t->qb;
  if (n < 2 || n < reach) return false;
  // No more stages than the busiest CTA fills, so that the next call's CTAs fit beside those of a short one.  In a graph: 33x6x13x14->8
  // 5x5 7.3 -> 6.4 us (8.4 -> 8.3 from the host, which needs that long), 150 direct shapes 0.96 of the time, the slowest 1.02.
  const int64_t rounds = (tiles + sms - 1) / sms;
  n = std::min(n, std::max({int64_t(2), reach, rounds * t->ncb}));
  int64_t fs = (room - n * region) / (kbs * b_bytes);
  fs = std::min({fs, int64_t(kHaloFilterStages), blocks * rounds});
  // A residual's loads in flight hold their lines in L1, four sectors to a line, and 220 KB leave it 30: 32x64x56x56->64 3x3
  // 25.3 -> 24.3 us a call (in a graph 25.1 -> 23.9), -> 256 1x1 58.0 -> 51.6 (57.5 -> 51.4).  Not where the filter streams by for every tile, which then is what
  // takes the time: 1x176x15x14->136 7x7 23.4 -> 24.6, 8x16x89x83->16 7x7 27.8 -> 29.0.
  if (add && copy && (resident || blocks <= 4))
    while (n > 3 && n * region + (resident ? filter : fs * kbs * b_bytes) + fixed > kHaloAddSmem) --n;
  t->bn = bn, t->resident = resident ? 1 : 0, t->stages = static_cast<int>(n);
  t->filter_stages = resident ? 0 : static_cast<int>(fs), t->filter_kbs = static_cast<int>(kbs);
  t->regions_bytes = static_cast<uint32_t>((n * region + 1023) / 1024 * 1024);
  t->smem = static_cast<size_t>(1024 + t->regions_bytes + (resident ? filter : fs * kbs * b_bytes) + (OC + 31) / 32 * 128);
  return true;
}

// The tensor core adds to its fp32 sum once per MMA, and rounds there.  With few channels an MMA holds padding and a sum takes
// more of them than one over a dense patch, as the gather kernel builds it, would: 28 instead of 10 for 7 x 7 x 3, which
// was 5.3e-7 off a sum in 64 bits where the dense one is 2.3e-7 (2-norm, relative).  So such a sum is made in as many
// parts as it takes to have no more MMAs in each, added in the epilogue.  0: one sum (16 channels or more: no other kernel
// is denser).
inline int halo_chain(const ConvShape &c) { return c.IC < 16 ? static_cast<int>((c.IC * c.KH * c.KW + 15) / 16) : 0; }

// The tile of a form, its width by the cycles of the busiest CTA.  False where the form does not take the shape.
inline bool halo_tile(const ConvShape &c, ConvForm form, int sms, HaloTile *best) {
  const bool copy = form_copies(form), flat = form_flat(form);
  const int64_t ncb = (c.IC + 63) / 64, taps = c.KH * c.KW, pair_taps = c.KH * ((c.KW + 1) / 2);
  const bool pairs = c.IC <= 8;
  const int64_t num_kb = pairs ? (pair_taps + 3) / 4 : ncb * taps;
  const int last_steps = static_cast<int>((c.IC - (ncb - 1) * 64 + 15) / 16);
  const int64_t mmas = pairs ? pair_taps : ((ncb - 1) * 4 + last_steps) * taps;
  if (!copy && c.IC > 32) return false;  // one block of channels
  if (c.OC > kHaloMaxOC || (pairs ? pair_taps : taps) > kHaloMaxTaps || ncb * taps > (1 << 16) || c.OH * c.OW > INT32_MAX) return false;
  HaloTile t;
  t.ncb = static_cast<int>(ncb), t.last_steps = last_steps, t.pairs = pairs ? 1 : 0, t.num_kb = static_cast<int>(num_kb);
  t.mmas = static_cast<int>(mmas), t.chain = halo_chain(c);
  t.splits = t.chain ? static_cast<int>((mmas + t.chain - 1) / t.chain) : 1;
  if (!halo_plan(c, flat, &t.h)) return false;
  t.qb = (t.h.px + 31) / 32;
  if (copy) {
    t.boxes = flat ? (t.h.px + 255) / 256 : 1;
    t.box_px = flat ? (t.h.px + t.boxes * 8 - 1) / (t.boxes * 8) * 8 : t.h.px;
    if (!flat && (t.h.IW > 256 || t.h.px / t.h.IW > 256)) return false;
    t.region_bytes = static_cast<uint32_t>((t.boxes * t.box_px * 128 + 1023) / 1024 * 1024);
  } else {
    t.boxes = t.box_px = 0;
    t.region_bytes = static_cast<uint32_t>(t.h.plane_px * 32 * (pairs ? 1 : last_steps));
  }
  double best_cost = 1e300;
  for (int bn = 256; bn >= 32; bn -= 32) {
    if ((bn > 32 && bn >= c.OC + 32) || 2 * t.splits * bn > 512) continue;
    if (!fit_halo(&t, copy, c.add != nullptr, c.OC, bn, sms)) continue;
    const int64_t tiles = t.h.m_tiles * ((c.OC + bn - 1) / bn);
    if (tiles > (1 << 30)) continue;
    const double rounds = static_cast<double>((tiles + sms - 1) / sms);
    // Cycles of a tile's engines: MMAs; bytes out of L2 (regions of a copy, the filter where it does not stay) at 64 a
    // cycle; lines through the load / store unit (pixels of one channel lie in rows of the region's width); stores;
    // instructions of the input warps.
    const double in_lines = flat ? 1.8 : 1.0 + 26.0 / t.h.IW, out_lines = flat ? 1.8 : 4.0;
    const double mma = static_cast<double>(mmas) * (bn < 64 ? 46.0 : bn < 128 ? 54.0 : bn / 2.0);
    const double l2 = (copy ? static_cast<double>(ncb) * t.region_bytes : 0.0) / 64.0 + (t.resident ? 0.0 : num_kb * bn * 2.0);
    const double loads = copy ? 0.0 : t.qb * (pairs ? static_cast<double>(c.IC) : last_steps * 16.0);
    const double work = copy ? 0.0 : t.qb * (last_steps * 100.0 + 60.0);
    const double epi = bn * ((c.add ? 1024.0 : 512.0) / 24.0 + 4.0 * (t.splits - 1));
    const double lsu = loads * in_lines + bn * 4.0 * out_lines * (c.add ? 2.0 : 1.0);
    const double cost = rounds * (std::max({mma, l2, lsu, epi, work}) + 300.0) + epi + (copy ? l2 : 3.0 * loads);
    if (cost < best_cost * 0.98) best_cost = cost, *best = t;
  }
  return best_cost < 1e300;
}

// What a call takes on the persistent kernels, and on conv_halo_kernel, in us: estimates to choose by.  Their constants were
// fitted to 2500 shapes timed on all of these kernels (16 to 1024 channels under 1 x 1 to 7 x 7 windows, 1 to 32 channels
// under 25 to 81 taps; strides 1 and 2, dilations, maps of one row or column and square ones, 1 to 65536 tiles): absolute
// times are met within 10 % for half of them, and what is chosen is rarely the slower one (conv_form).  A CTA's tiles pass
// one after another, each as slow as the slowest of its engines; or all CTAs wait for memory.  Cycles at 1.85 GHz; no call
// is over before its two launches.
constexpr double kConvLaunches = 7.9;
inline double conv_us(double bytes_rewritten, double cycles) {
  return std::max(kConvLaunches, 4.5 + bytes_rewritten / 8.0e6 + cycles / 1850.0);
}
inline double dense_us(const ConvShape &c, int sms) {
  const double out = 4.0 * c.N * c.OC * c.OH * c.OW * (c.add ? 2 : 1);
  const int64_t taps = c.KH * c.KW, ncb = (c.IC + 63) / 64, m_tiles = (c.N * c.OH * c.OW + 127) / 128, Cp8 = (c.IC + 7) / 8;
  const bool gather = conv_gathers(c);
  const int64_t num_kb = gather ? (c.IC * taps + 63) / 64 : ncb * taps;
  const int bn = choose_conv_bn(m_tiles, c.OC, num_kb, gather, c.add != nullptr, sms);
  const int64_t n_tiles = (c.OC + bn - 1) / bn, tiles = m_tiles * n_tiles;
  const double rounds = static_cast<double>((tiles + sms - 1) / sms);
  // instructions of the gather, as they were when this was fitted; it takes about half of that now (see conv_form)
  if (gather) return conv_us(0.0, rounds * num_kb * 2600.0 + 4000.0);
  // an im2col k-block: the hand-over of its stage, or 70 bytes a cycle; rows of the copy that end inside a sector are read
  // at half that rate
  const double kb = std::max(400.0, (16384.0 + (conv_filter_stays(num_kb, bn, n_tiles, tiles, sms) ? 0 : bn * 128)) / 70.0);
  const double loads = kb * (num_kb + (Cp8 % 2 ? 0.8 * taps : 0.0)), epi = bn * (c.add ? 1024.0 : 512.0) / 35.0;
  const double rewritten = 6.0 * (static_cast<double>(c.N) * c.IC * c.H * c.W + static_cast<double>(c.OC) * c.IC * taps);
  const double memory = out / 3000.0 + 2.0 * c.N * c.H * c.W * Cp8 * 8 / 1150.0;
  return conv_us(rewritten, std::max(rounds * (1450.0 + std::max(loads, epi)), memory) + epi);
}
inline double halo_us(const ConvShape &c, ConvForm form, const HaloTile &t, int sms) {
  const bool copy = form_copies(form), flat = form_flat(form);
  const int64_t tiles = t.h.m_tiles * ((c.OC + t.bn - 1) / t.bn);
  const double rounds = static_cast<double>((tiles + sms - 1) / sms);
  const double blocks = t.resident ? 0 : (t.num_kb + t.filter_kbs - 1) / t.filter_kbs;  // stages of the filter
  // rows of eight pixels that do not start on a sector are stored in parts of two
  const double parts = flat || c.OW % 8 == 0 ? 1.0 : 1.5;
  double mma = t.mmas * (t.bn < 64 ? 42.0 : std::max(58.0, t.bn / 2.0));
  if (!copy) {
    mma += blocks * 490.0;
    const double in = t.qb * t.last_steps * 120.0, epi = t.bn * (512.0 * parts * (c.add ? 3.5 : 1.0) / 30.0 + 6.0 * (t.splits - 1));
    return conv_us(0.0, rounds * (1800.0 + std::max({mma, in, epi})) + epi + in);
  }
  mma += blocks * 330.0 + t.ncb * 960.0;
  const double l2 = (static_cast<double>(t.ncb) * t.region_bytes + (t.resident ? 0.0 : t.num_kb * t.bn * 128.0)) / 43.0;
  const double stored = parts * (c.add ? (flat ? 1.5 : 2.0) : 1.0), epi = t.bn * 512.0 * stored / (flat ? 19.0 : 39.0);
  const double rewritten = 6.0 * (static_cast<double>(c.N) * c.IC * c.H * c.W + static_cast<double>(c.OC) * c.IC * c.KH * c.KW);
  const double memory = 4.0 * c.N * c.OC * c.OH * c.OW * stored / 2000.0;
  return conv_us(rewritten, std::max(rounds * (530.0 + std::max({mma, l2, epi})), memory) + epi + t.region_bytes / 43.0);
}

// Where conv_halo_kernel takes a call, in which form and with which tile; `c` after conv_sampled.  dense: whether the
// persistent kernels take it too (im2col with 16 channels or more, gather below).  The quicker one by the estimates above: a
// region's tiles hold the margins between images too, and rect ones whatever 16 rows x 8 pixels leave empty.
// us a call, inputs changing, theirs / rect / flat:
//   a k-block costs im2col 400 cycles or more, a region's MMAs 42 to 58 each below 128 columns:
//     32x64x56x56->64 3x3 24 / 19 / 26, 16x16x77x77->16 20 / 12 / 12, 33x32x55x55->32 5x5 46 / 20 / 22, 33x192x55x55->32 5x5 113 / 90 / 94
//   a block of 64 channels costs a region 960 beside them and 43 bytes a cycle, so wide tiles and many blocks go dense:
//     32x128x28x28->128 3x3 19.1 / 20.0 / 20.7, 32x512x14x14->512 35 / 48 / 46, 8x384x56x56->384 67 / 87 / 101, 32x512x28x28->512 108 / 141 / 137
//   rows of eight pixels off the sectors: 14x64x85x93->448 5x1 67 / 201 / 70, 25x64x52x87->256 1x3 44 / 108 / 51
//   empty tiles: 1x64x1x65536->64 1x3 15 / 56 / 17, 1x64x4x8192->64 3x3 13 / 19, 206x32x2x112->64 5x5 dilation 3 24 / 69
//   1 x 1: 32x64x56x56->256 40 / 34 / 30, 117x128x43x60->32 with residual 91 / 65 / 60, but 10x96x220x8->142 12 / 15 / 15
//   few channels, gather / rect / flat: 16x3x224x224->32 7x7 92 / 76, 16x6x64x64->64 7x7 35 / 14 / 15, 1x16x1x160000->32 1x9 27 / 101 / 15,
//     but 256x1x28x28->32 5x5 12 / 24 / 24, 21x3x29x37->352 5x5 14 / 23 / 23, 1x3x4x40000->32 5x5 18 / 42
//   stride 2, 16 to 32 channels, im2col / rect: 16x24x150x153->32 5x5 78 / 30, 4x32x200x203->32 5x5 27 / 19, but 4x16x120x123->256 7x7 24 / 32
// Below 25 taps few channels and strides stay where they are: nearly all that was measured there is slower (16x3x256x256->64
// 3x3 56 / 87; not 43x6x255x256->8 3x3 dilation 2 134 / 131).  From 25 taps on the line stands too early since the gather takes half of
// what dense_us says: 16x3x128x128->64 5x5 goes to a region that takes 31.6 where the gather would 26.3, 16x4x100x100->128 7x7 48.8 /
// 33.3, 64x3x56x56->64 5x5 24.5 / 21.3, 16x3x224x224->64 7x7 stride 2 35.1 / 31.1, 16x3x18x256->64 7x7 16.4 / 15.4.
// When these estimates were fitted: over 1648 shapes with copies the choice takes 0.901 of the dense kernels' time (geometric mean; always the best one, 0.890)
// and 40 are more than 4 % slower; over 871 others 0.814 (0.804) and 39.  Over 1050 that the estimates were not fitted to,
// 0.910 (0.893), 14 of 700, and 0.804 (0.790), 16 of 350.
inline ConvForm conv_form(const ConvShape &c, int sms, bool dense = true, HaloTile *tile = nullptr) {
  const bool unit = c.SH == 1 && c.SW == 1, direct = c.IC < 16 || (!unit && c.IC <= 32);
  ConvForm best = ConvForm::kOther;
  if (direct ? c.KH * c.KW < 25 : !unit) return best;
  double us = dense ? dense_us(c, sms) : 1e300;
  auto consider = [&](ConvForm form) {
    HaloTile t;
    if (!halo_tile(c, form, sms, &t)) return;
    // The remaining kernel (conv_tcgen05.cu) takes twice a region's time or more (2x48x1x3000->64 1x9 dilation 33 29 us / 15), so
    // not on tiles that are mostly empty.  It packs channels without padding: where a region would pad them, its sums take
    // more MMAs, and are further off 64 bits (17 channels 3.3e-7 against 2.3e-7).
    if (!dense && (t.h.m_tiles > 2 * ((c.N * c.OH * c.OW + 127) / 128) || (c.IC > 16 && c.IC % 16))) return;
    const double e = halo_us(c, form, t, sms);
    if (e >= us) return;
    us = e, best = form;
    if (tile) *tile = t;
  };
  if (c.KH * c.KW > 1) consider(direct ? ConvForm::kDirectRect : ConvForm::kCopyRect);  // (1 x 1 has no margins to read)
  // Where rect wastes little: a copy whose rows are whole sectors is stored as such, which flat tiles do not; a flat region
  // of long rows is read for pixels that most of its tile has no use for.
  HaloPlan rect, flat;
  const bool keep = c.KH * c.KW > 1 && (direct ? c.KH > 1 && c.OW >= 48 : c.OW % 8 == 0) && halo_plan(c, false, &rect) && halo_plan(c, true, &flat) &&
                    rect.m_tiles * 5 <= flat.m_tiles * 6;
  if (unit && !keep) consider(direct ? ConvForm::kDirectFlat : ConvForm::kCopyFlat);
  return best;
}

// Runs the convolution on conv_halo_kernel; false (and nothing launched) when the shape is not one for it.
bool conv_halo(const ConvShape &c, cudaStream_t s);

// Whether the persistent kernels take the shape here: it is within their limits, and the driver makes im2col maps.
bool conv_persistent_takes(const ConvShape &c);

// Runs the convolution on the persistent kernels; false (and nothing launched) when the shape is one
// that they do not take or there is no memory for their operands.
bool conv_persistent(const ConvShape &c, cudaStream_t s);

}  // namespace mdc
