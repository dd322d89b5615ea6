"""The tiles of the convolution kernel whose taps share one region of the input (conv_plan.h), compiled for the host: every
live output's every tap finds its input pixel, or padding, where the kernel looks for it."""
import os
import shutil
import subprocess

import pytest

OPS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multi-device-model-compiler_b200", "csrc", "ops")
CUDA_INCLUDE = "/usr/local/cuda/include"

PROGRAM = r"""
#include "conv_plan.h"
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <vector>
using namespace mdc;
int main() {
  srand(1);
  auto pick = [](int lo, int hi) { return lo + rand() % (hi - lo + 1); };
  int rects = 0, flats = 0, strided = 0;
  for (int i = 0; i < 1500; ++i) {
    ConvShape c = {};
    c.N = pick(1, 4), c.IC = 1, c.OC = 1, c.H = pick(1, 24), c.W = pick(1, 24), c.KH = pick(1, 5), c.KW = pick(1, 5);
    c.SH = pick(1, 3), c.SW = pick(1, 3), c.DH = pick(1, 3), c.DW = pick(1, 3), c.PHL = pick(0, 4), c.PWL = pick(0, 4);
    const int64_t span_h = (c.KH - 1) * c.DH, span_w = (c.KW - 1) * c.DW;
    c.OH = (c.H + c.PHL + pick(0, 4) - span_h - 1) / c.SH + 1, c.OW = (c.W + c.PWL + pick(0, 4) - span_w - 1) / c.SW + 1;
    if (c.OH < 1 || c.OW < 1 || c.H + c.PHL + 4 < span_h + 1 || c.W + c.PWL + 4 < span_w + 1) continue;
    c.OH -= c.OH > 1 ? pick(0, 1) : 0, c.OW -= c.OW > 1 ? pick(0, 1) : 0;
    for (int flat = 0; flat < 2; ++flat) {
      HaloPlan h;
      if (!halo_plan(c, flat, &h)) {
        assert(c.SH > 2 || c.SW > 2 || (flat && (c.SH > 1 || c.SW > 1)));
        continue;
      }
      flat ? ++flats : c.SH * c.SW > 1 ? ++strided : ++rects;
      std::vector<int> seen(c.N * c.OH * c.OW, 0);
      for (int64_t tile = 0; tile < h.m_tiles; ++tile) {
        // the region's pixels by their place, as the input warps write them: image, row, column, or -1 for padding
        std::vector<int64_t> at(h.plane_px, -2);
        for (int64_t q = 0; q < h.px; ++q) {
          int64_t row, col, place = q;
          if (flat) {
            const int64_t px = tile * 128 - c.PHL * h.Wv - c.PWL + q;
            row = px < 0 ? -1 : px / h.Wv, col = px < 0 ? 0 : px % h.Wv;
          } else {
            const int64_t rh = q / h.IW, rw = q % h.IW;
            row = tile / h.tiles_w * 16 * c.SH - c.PHL + rh, col = tile % h.tiles_w * 8 * c.SW - c.PWL + rw;
            place = (rh % c.SH * c.SW + rw % c.SW) * h.class_px + rh / c.SH * h.pitch + rw / c.SW;
          }
          assert(place >= 0 && place < h.plane_px);
          const int64_t img = row < 0 ? c.N : row / h.Hv, y = row < 0 ? 0 : row % h.Hv;
          at[place] = img < c.N && y < c.H && col >= 0 && col < c.W ? (img * c.H + y) * c.W + col : -1;
        }
        for (int64_t r = 0; r < 128; ++r) {
          const int64_t vr = flat ? (tile * 128 + r) / h.Wv : tile / h.tiles_w * 16 + r / 8;
          const int64_t ow = flat ? (tile * 128 + r) % h.Wv : tile % h.tiles_w * 8 + r % 8;
          const int64_t img = vr / h.HvO, oh = vr % h.HvO;
          const bool live = img < c.N && oh < c.OH && ow < c.OW;
          if (live) ++seen[(img * c.OH + oh) * c.OW + ow];
          for (int64_t kh = 0; kh < c.KH; ++kh)
            for (int64_t kw = 0; kw < c.KW; ++kw) {
              const int64_t rh = kh * c.DH, rw = kw * c.DW;
              const int64_t place = (rh % c.SH * c.SW + rw % c.SW) * h.class_px + rh / c.SH * h.pitch + rw / c.SW +
                                    (flat ? r : r / 8 * h.pitch + r % 8);
              assert(place < h.plane_px);  // whatever the pixel: the tensor core reads all 128
              if (!live) continue;
              const int64_t y = oh * c.SH - c.PHL + rh, x = ow * c.SW - c.PWL + rw;
              assert(at[place] == (y >= 0 && y < c.H && x >= 0 && x < c.W ? (img * c.H + y) * c.W + x : -1));
            }
        }
      }
      for (int n : seen) assert(n == 1);
    }
  }
  assert(rects > 50 && flats > 50 && strided > 100);
  // where the kernel takes a call
  ConvShape c = {};
  auto form = [&](int N, int IC, int H, int W, int OC, int K, int S, int KH = 0, int D = 1, bool dense = true) {
    if (!KH) KH = K;
    c.N = N, c.IC = IC, c.H = H, c.W = W, c.OC = OC, c.KH = KH, c.KW = K, c.SH = c.SW = S, c.DH = c.DW = D;
    c.PHL = KH / 2 * D, c.PWL = K / 2 * D;
    c.OH = (H + 2 * c.PHL - (KH - 1) * D - 1) / S + 1, c.OW = (W + 2 * c.PWL - (K - 1) * D - 1) / S + 1;
    return conv_form(c, 148, dense);
  };
  assert(form(16, 3, 256, 256, 64, 3, 1) == ConvForm::kOther && form(16, 3, 224, 224, 32, 7, 1) == ConvForm::kDirectRect);
  assert(form(21, 3, 29, 37, 352, 5, 1) == ConvForm::kOther && form(8, 15, 20, 20, 8, 5, 3) == ConvForm::kOther);
  assert(form(8, 3, 29, 37, 32, 9, 1) == ConvForm::kDirectRect && form(8, 3, 29, 37, 32, 11, 1) == ConvForm::kOther);
  assert(form(32, 64, 56, 56, 64, 3, 1) == ConvForm::kCopyRect && form(32, 64, 57, 57, 64, 3, 1) == ConvForm::kCopyFlat);
  assert(form(32, 128, 28, 28, 128, 3, 1) == ConvForm::kOther && form(32, 512, 14, 14, 512, 3, 1) == ConvForm::kOther);
  assert(form(32, 64, 56, 56, 256, 1, 1) == ConvForm::kCopyFlat && form(1, 160, 9, 7, 96, 3, 1) == ConvForm::kCopyRect);
  assert(form(2, 64, 20, 20, 32, 3, 1) == ConvForm::kOther && form(2, 65, 20, 20, 32, 3, 1) != ConvForm::kOther);
  assert(form(2, 32, 22, 23, 32, 7, 2) == ConvForm::kDirectRect && form(2, 64, 22, 23, 32, 7, 2) == ConvForm::kOther);
  // mostly empty tiles (one or a few rows of many pixels; rect 2 to 16 times the dense tiles), and many channels on large
  // maps: the dense kernels take 0.2 to 0.8 of the region kernel's time on these
  for (int w : {65536, 65535, 49152}) assert(form(1, 64, 1, w, 64, 3, 1, 1) != ConvForm::kCopyRect);
  assert(form(1, 16, 1, 160000, 32, 9, 1, 1) == ConvForm::kCopyFlat && form(4, 64, 1, 16384, 64, 3, 1, 1) == ConvForm::kOther);
  assert(form(1, 64, 4, 8192, 64, 3, 1) == ConvForm::kOther && form(1, 64, 17, 2048, 64, 3, 1) == ConvForm::kOther);
  assert(form(1, 3, 4, 40000, 32, 5, 1) == ConvForm::kOther && form(206, 32, 2, 112, 64, 5, 1, 5, 3) == ConvForm::kOther);
  assert(form(32, 512, 28, 28, 512, 3, 1) == ConvForm::kOther && form(8, 384, 56, 56, 128, 3, 1) == ConvForm::kOther);
  assert(form(14, 64, 85, 93, 448, 1, 1, 5) != ConvForm::kCopyRect && form(4, 16, 120, 123, 256, 7, 2) == ConvForm::kOther);
  // a dilation that the im2col map cannot describe goes to a region, unless most of its tiles were empty
  assert(form(1, 64, 1, 20000, 64, 9, 1, 1, 32, false) == ConvForm::kCopyFlat);
  assert(form(64, 64, 1, 64, 64, 9, 1, 1, 32, false) == ConvForm::kOther);
  // a tile and its memory belong to the form, and keep to the kernel's limits
  for (int i = 0; i < 4000; ++i) {
    const int K = pick(0, 2) ? pick(1, 9) : 1, S = pick(1, 2), size = pick(1, 3) * pick(1, 90) + K;
    if (form(pick(1, 9), i % 2 ? pick(1, 40) : pick(1, 700), size, pick(1, 300) + K, pick(1, 2100), K, S) == ConvForm::kOther) continue;
    HaloTile t;
    const ConvForm f = conv_form(c, 148, true, &t);
    assert(form_flat(f) == (t.h.flat != 0) && (form_copies(f) ? c.IC >= 16 && S == 1 : c.IC <= 32));
    assert(t.smem <= kHaloMaxSmem && t.stages >= 2 && t.bn % 32 == 0 && t.bn <= 256 && 2 * t.splits * t.bn <= 512);
    assert(t.resident ? c.OC <= t.bn : t.filter_stages >= 1 && t.filter_stages <= kHaloFilterStages);
    assert(form_copies(f) || t.stages * t.qb >= kHaloInputWarps);
  }
  printf("ok\n");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INCLUDE), reason="no host compiler or CUDA headers")
def test_halo_tiles_find_every_tap(tmp_path):
    src = tmp_path / "plan.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "plan")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", OPS, "-I", CUDA_INCLUDE, str(src), "-o", exe], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout == "ok\n"


ROUTES = r"""
#include "conv_plan.h"
#include <cstdio>
using namespace mdc;
int main() {  // per call: N IC H W OC KH KW OH OW SH SW DH DW PHL PWL post_add
  const char *names[] = {"kOther", "kCopyRect", "kCopyFlat", "kDirectRect", "kDirectFlat"};
  long v[16];
  static float some;
  for (;;) {
    for (long &x : v)
      if (scanf("%ld", &x) != 1) return 0;
    ConvShape c = {};
    c.N = v[0], c.IC = v[1], c.H = v[2], c.W = v[3], c.OC = v[4], c.KH = v[5], c.KW = v[6], c.OH = v[7], c.OW = v[8];
    c.SH = v[9], c.SW = v[10], c.DH = v[11], c.DW = v[12], c.PHL = v[13], c.PWL = v[14], c.add = v[15] ? &some : nullptr;
    const bool dense = conv_dense_describes(c);
    conv_sampled(c);
    puts(names[static_cast<int>(conv_form(c, 148, dense))]);
  }
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INCLUDE), reason="no host compiler or CUDA headers")
def test_rows_of_the_gpu_tests_reach_their_kernels(tmp_path):
    """The GPU tests compare results, which are the same on every kernel: here each of their rows is held to the kernel that
    it is there for."""
    import test_gpu_conv_pool as gpu
    rows = gpu.CONV_EDGES + gpu.REGION_FORMS
    rows += [(f, (n, ic, 20, w, 9, 5, 5, (1, 1), (2,) * 4, (1, 1), False, False)) for f, n, ic, w in gpu.INFINITIES]
    rows += [(f, (3, ic, size, size, oc, k, k, (st, st), (k // 2,) * 4, (1, 1), False, False)) for f, ic, oc, size, k, st in gpu.OVERLAPS]
    rows.append(("kCopyRect", (12, 32, 2048, 2048, 8, 3, 3, (1, 1), (1,) * 4, (1, 1), False, False)))  # without memory for its copy
    calls = []
    for _, (N, IC, H, W, OC, KH, KW, stride, pad, dil, add, _relu) in rows:
        OH = (H + pad[0] + pad[2] - (KH - 1) * dil[0] - 1) // stride[0] + 1
        OW = (W + pad[1] + pad[3] - (KW - 1) * dil[1] - 1) // stride[1] + 1
        calls.append((N, IC, H, W, OC, KH, KW, OH, OW, *stride, *dil, pad[0], pad[1], int(add)))
    src, exe = tmp_path / "routes.cpp", str(tmp_path / "routes")
    src.write_text(ROUTES)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", OPS, "-I", CUDA_INCLUDE, str(src), "-o", exe], check=True)
    told = subprocess.run([exe], input=" ".join(str(x) for c in calls for x in c), check=True, capture_output=True, text=True).stdout.split()
    assert len(told) == len(rows)
    assert not [(want, got, row) for (want, row), got in zip(rows, told) if want != got]
    assert set(told) == {"kOther", "kCopyRect", "kCopyFlat", "kDirectRect", "kDirectFlat"}


RING = r"""
#include "conv_plan.h"
#include <cassert>
#include <cstdio>
using namespace mdc;
int main() {
  // A group's wait at block b, its last block b - 3 let in: blocks up to b - 3 - stages are known to be used, and any
  // number more.  What passes a wait by parity must be the use that is waited for.
  auto safe = [](int stages) {
    for (int b = 3; b < 200; ++b)
      for (int used = b - kGatherGroups - stages + 1; used <= b; ++used) {
        const int use = b / stages, of = b % stages, done = used <= of ? 0 : (used - of - 1) / stages + 1;  // of b's stage
        if ((done & 1) == (use & 1) && done < use) return false;
      }
    return true;
  };
  assert(!safe(1) && !safe(2) && safe(3) && safe(4));
  for (int64_t room = 0; room < 300 * 1024; room += 512)
    for (int64_t stage : {16384, 16384 + 32 * 128, 16384 + 256 * 128}) {
      const int gather = conv_ring_stages(room, stage, true), im2col = conv_ring_stages(room, stage, false);
      assert(gather == 0 || (safe(gather) && gather * stage <= room && gather <= 4));
      assert(im2col == 0 || (im2col >= 2 && im2col * stage <= room && im2col <= kRingMaxStages));
      assert((gather == 0) == (room / stage < 3) && (im2col == 0) == (room / stage < 2));
    }
  puts("ok");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INCLUDE), reason="no host compiler or CUDA headers")
def test_a_gathered_ring_has_a_stage_for_every_group(tmp_path):
    src, exe = tmp_path / "ring.cpp", str(tmp_path / "ring")
    src.write_text(RING)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", OPS, "-I", CUDA_INCLUDE, str(src), "-o", exe], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout == "ok\n"


TAPS = r"""
#include "conv_plan.h"
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <cstring>
using namespace mdc;
int main() {
  srand(3);
  auto pick = [](int lo, int hi) { return lo + rand() % (hi - lo + 1); };
  int nears = 0, fars = 0;
  for (int i = 0; i < 20000; ++i) {
    ConvShape c = {};
    c.IC = pick(1, 15), c.KH = pick(1, 9) * (i % 7 ? 1 : 2), c.KW = pick(1, 9) * (i % 11 ? 1 : 2), c.DH = pick(1, 40), c.DW = pick(1, 40);
    c.H = pick(1, 300), c.W = pick(1, 300), c.N = pick(1, 5), c.PHL = pick(0, 50), c.PWL = pick(0, 50);
    const int64_t K = c.IC * c.KH * c.KW;
    if (K > kDenseMaxGatherK) continue;
    static NearTaps n;
    static FarTaps f;
    memset(&n, 0xee, sizeof n), memset(&f, 0xee, sizeof f);
    const bool near = conv_taps_near(c);
    assert(near == (K <= 256 && c.KH <= 16 && c.KW <= 15));
    if (near) fill_taps(c, &n), ++nears, assert(n.lead == (c.PHL * c.W + c.PWL) * 4);
    fill_taps(c, &f), ++fars;
    for (int64_t k = 0; k < (K + 7) / 8 * 8; ++k) {
      const int64_t ic = k / (c.KH * c.KW), kh = k / c.KW % c.KH, kw = k % c.KW, off = (ic * c.H + kh * c.DH) * c.W + kw * c.DW;
      assert(f.off[k] == (k < K ? off : 0) && f.pos[k] == (k < K ? (kh * c.DH) << 16 | (kw * c.DW) : 0));
      if (near) assert(n.off[k] == (k < K ? off * 4 : 0) && n.need[k] == (k < K ? 1u << kh | 0x10000u << kw : 0x80000000u));
    }
  }
  assert(nears > 1000 && fars > nears);
  // where 32 bits end: the last value of the input from `lead` bytes ahead of it, and the last tap from a window's origin
  ConvShape c = {};
  c.N = 4, c.IC = 4, c.H = 8192, c.W = 8191, c.KH = c.KW = 3, c.DH = c.DW = 1;
  for (int64_t w = 8191; w <= 8192; ++w)
    for (int64_t ph : {0, 1, 2, 15})
      for (int64_t pw : {0, 1, 7}) {
        c.W = w, c.PHL = ph, c.PWL = pw;
        assert(conv_taps_near(c) == ((c.N * c.IC * c.H * w + ph * w + pw) * 4 <= 0xffffffffll));
      }
  c.PHL = c.PWL = 0, c.W = 8191;
  for (; c.PHL < 32; ++c.PHL) assert(conv_taps_near(c) == (c.PHL <= 16));  // 131072 values of 2^30 left, 16 rows and 16 values
  c.N = 1, c.IC = 15, c.H = 8192, c.W = 8192, c.PHL = 0;
  for (int64_t d : {1, 5000, 8191, 8192, 16383, 16384}) {
    c.DH = d;
    assert(conv_taps_near(c) == (((14 * 8192 + 2 * d) * 8192 + 2) * 4 <= 0xffffffffll));
  }
  puts("ok");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INCLUDE), reason="no host compiler or CUDA headers")
def test_taps_of_a_gathered_patch(tmp_path):
    """The tables are counted up: each entry against the division that defines it, and the line to 64-bit addresses."""
    src, exe = tmp_path / "taps.cpp", str(tmp_path / "taps")
    src.write_text(TAPS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", OPS, "-I", CUDA_INCLUDE, str(src), "-o", exe], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout == "ok\n"
