// The operands that one call has to bring into 16 bits, collected and then converted by ONE launch
// (elementwise.cu): casts of activations and packings of weights.  Host bookkeeping only.
#pragma once

#include <cstdint>

namespace mdc {

struct OperandList {
  static constexpr int kMax = 5;  // a transformer layer: its input and four weights
  static constexpr int64_t kThreads = 256;
  // Elements that a block casts: of a contiguous array, or of rows that are padded (element by element:
  // shorter, so that a few odd rows still spread over the SMs).
  static constexpr int64_t kCastItems = kThreads * 16, kPadItems = kThreads * 4;
  struct Job {
    const float *src;
    void *dst;
    int64_t rows, cols, pitch;  // cast: [rows, cols] -> [rows, pitch]; pack: [rows = K, cols = N] -> [N, pitch]
    int64_t first_block;
    int tiles_n;                // pack: 64-column tiles; 0 marks a cast
    int vec_ok;                 // cast: 16-byte accesses; pack: stores of whole sectors
  };
  Job jobs[kMax];
  int n = 0;
  int64_t blocks = 0;
  bool overflow = false;  // a job more than the list holds: launch() refuses, nothing is converted in part

  // fp32 [R, C] -> 16-bit [R, Cp], zeros in the columns C .. Cp
  void cast(const float *src, void *dst, int64_t R, int64_t C, int64_t Cp) {
    if (R <= 0 || Cp <= 0) return;
    Job *j = add(src, dst, R, C, Cp);
    if (!j) return;
    j->tiles_n = 0;
    j->vec_ok = C == Cp && ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0;
    const int64_t items = j->vec_ok ? kCastItems : kPadItems;
    blocks += (R * Cp + items - 1) / items;
  }
  // weight fp32 [K, N] -> 16-bit [N, Kp], Kp = K rounded up to 8, zero padded
  void pack(const float *w, void *dst, int64_t K, int64_t N) {
    if (K <= 0 || N <= 0) return;
    Job *j = add(w, dst, K, N, (K + 7) / 8 * 8);
    if (!j) return;
    j->tiles_n = static_cast<int>((N + 63) / 64);
    j->vec_ok = j->pitch % 16 == 0 && !(reinterpret_cast<uintptr_t>(dst) & 31u);
    blocks += j->tiles_n * ((j->pitch + 63) / 64);
  }
  void clear() { n = 0, blocks = 0, overflow = false; }
  // Nothing when empty; the list is empty afterwards.  late: the next kernel may start once this one's own
  // dependency is resolved, instead of at once: what is older than this launch is then complete for it.
  void launch(int32_t dtype, void *stream, bool late = false);

 private:
  Job *add(const float *src, void *dst, int64_t rows, int64_t cols, int64_t pitch) {
    if (n == kMax) {
      overflow = true;
      return nullptr;
    }
    Job &j = jobs[n++];
    j.src = src, j.dst = dst, j.rows = rows, j.cols = cols, j.pitch = pitch, j.first_block = blocks;
    return &j;
  }
};

}  // namespace mdc
