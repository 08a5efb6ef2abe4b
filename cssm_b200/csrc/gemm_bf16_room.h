// Column tiles and shared memory of the bf16 GEMM (csrc/gemm_bf16.cu): a pure function of the problem, host code only.
#pragma once
#include <cstddef>

namespace cssm {

constexpr int GB_BM = 128, GB_BK = 64, GB_MAX_STAGES = 8;
constexpr size_t GB_SMEM = 227 * 1024;
constexpr unsigned GB_BAR_BYTES = 320;                     // barriers and the TMEM slot
constexpr unsigned GB_A_BYTES = GB_BM * 128;               // one A stage: 128 rows x 128 bytes
constexpr size_t GB_BOX = 16384;                         // one staged output box: 128 rows x 64 columns
constexpr int GB_BIAS_MAX = 2048;                        // longest bias kept in shared memory

// Columns of a tile: 256, 192, 128 or 64 with the staged output, other multiples of 32 up to 256 as one tile with direct stores; 0: none.
inline int gb_columns(int N) {
  if (N % 256 == 0) return 256;
  if (N % 192 == 0) return 192;
  if (N % 128 == 0) return 128;
  if (N % 64 == 0) return 64;
  return N <= 256 && N % 32 == 0 ? N : 0;
}
// A residual with a short K loop gains more from the TMA residual prefetch (three staging slots, BN <= 128) than it loses in
// operand traffic: 37 against 47 us for M = 100 K, K = 256, N = 256.
inline int gb_columns(int N, int K, bool res) {
  const int bn = gb_columns(N);
  return bn == 256 && res && K < 512 ? 128 : bn;
}
// Few row tiles: narrower column tiles while every tile still gets an SM of its own, so that a CTA has less of an epilogue and
// fewer weights to wait for.  One 224-pixel image: the 23 launches 258 -> 199 us, the pass 405 -> 351 us; 33 images of 256
// pixels 866 -> 842 us.
inline int gb_narrow(int bn, int N, int m_tiles, int sms) {
  for (int n = 128; n >= 64; n /= 2)
    if (bn > n && N % n == 0 && (long long)m_tiles * (N / n) <= sms) bn = n;
  return bn;
}

struct Bf16Room {
  int wres;                  // the weights stay resident
  int stages, ostg;          // ring stages, staging slots of an epilogue half (0: no staging)
  int bias_n;                // bias values kept in shared memory, 0: read from global memory (or none)
  size_t bytes;              // dynamic shared memory; 0: does not fit
};

struct Bf16Form {
  int N, BN, Kpad;
  int rounds;                // tiles a CTA takes
  bool im2col;
  bool staged;               // output through staging slots and TMA stores
  bool res, rtma;            // a residual; its boxes by TMA into the slots (with staged)
  bool act;                  // GELU or SiLU
  bool bias, bias_aligned;   // a bias; it starts on 16 bytes
};

inline Bf16Room gb_room(const Bf16Form& f) {
  Bf16Room r = {};
  // Weights of at most 64 KB that form a single N tile stay resident (a weight tile re-read from L2 for every M tile costs as
  // much operand traffic as the A tile itself).
  const size_t weights = (size_t)f.Kpad * f.BN * 2;
  r.wres = !f.im2col && f.N == f.BN && weights <= 64 * 1024 ? 1 : 0;
  const size_t stage = GB_A_BYTES + (r.wres ? 0 : (size_t)f.BN * 128), held = r.wres ? weights : 0;
  // Residual by TMA: four stages, the rest goes to three or four staging slots a half.  Everything else: as many stages as there
  // is room for beside two slots (sixteen of 4 KB where every warp has its own).
  auto fit = [&](int bias_n, int stages) {
    const size_t fixed = GB_BAR_BYTES + 1024 + (size_t)bias_n * 4, room = GB_SMEM - held;      // 1024: alignment
    r.bias_n = bias_n;
    r.stages = stages;
    while (r.stages > 2 && r.stages * stage + (f.staged ? 4 * GB_BOX : 0) + fixed > room) --r.stages;
    const size_t used = r.stages * stage + fixed;
    r.ostg = !f.staged ? 0 : !f.rtma ? 2 : used > room ? 0 : (int)((room - used) / (2 * GB_BOX));
    if (r.ostg > 4) r.ostg = 4;
    r.bytes = r.ostg < (f.rtma ? 3 : f.staged ? 2 : 0) ? 0 : held + used + r.ostg * 2 * GB_BOX;
    if (r.bytes > GB_SMEM) r.bytes = 0;
  };
  const int most = f.rtma ? 4 : GB_MAX_STAGES;
  fit(0, most);
  if (!f.bias || f.N > GB_BIAS_MAX) return r;
  const Bf16Room without = r;
  fit(f.N, most);
  // The bias takes no staging slot away: four stages of 128 columns and three slots leave room for 432 values, so that a longer one
  // is read from global memory there (100000 x 64 -> 448 + residual in 64-column tiles: 51 us with the bias copied and three slots, 43
  // with four).  One that starts off 16 bytes can only be copied: a stage less then.
  if (f.rtma && r.ostg < without.ostg) {
    if (f.bias_aligned) return without;
    fit(f.N, 3);
  }
  // Nor the fourth stage of 192-column tiles (room for 432 values beside it, too), where long K loops of many tiles need it.  us a
  // launch, bias in global memory and four stages / copied and three: 100352 rows, 576 -> 1152 142 / 162, 384 -> 576 56 / 62, 192 -> 576
  // 42 / 42, 64 -> 576 31 / 28; 576 -> 576 + residual 95 / 90, 768 -> 576 104 / 110; 25088 rows, 384 -> 1344 GELU 40 / 38, 576 -> 1344 48 /
  // 51, 384 -> 960 (six rounds) 28 / 27; 5000 rows 3 % to 20 % the other way at every depth.
  const int deep = f.res ? 12 : f.act ? 9 : 6;
  if (!f.rtma && f.bias_aligned && r.stages < 4 && without.stages >= 4 && f.rounds >= 7 && f.Kpad >= deep * GB_BK) return without;
  return r;
}

}  // namespace cssm
