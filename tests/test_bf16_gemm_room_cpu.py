"""Tiles and shared memory of the bf16 GEMM (csrc/gemm_bf16_room.h), walked over widths, depths, row tiles and forms in a small host
program: every width that has a tile fits, a residual by TMA has its three staging slots, and a bias in shared memory takes none of
the slots that the form has without one, nor a long K loop's fourth stage."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "gemm_bf16_room.h"
using namespace cssm;
int main() {
  long bad = 0, seen = 0;
  auto report = [&](const char* what, int N, int K, int mt, int BN, const Bf16Room& r) {
    if (++bad < 20) std::printf("%s: N %d K %d row tiles %d BN %d stages %d slots %d bias %d bytes %zu\n", what, N, K, mt, BN, r.stages, r.ostg, r.bias_n, r.bytes);
  };
  for (int N = 32; N <= 4096; N += 32)
    for (int K : {32, 64, 96, 128, 192, 256, 320, 448, 512, 640, 1024, 2048, 4096})
      for (int mt : {1, 2, 9, 18, 19, 24, 37, 74, 100, 148, 149, 1000})
        for (int form = 0; form < 32; ++form) {
          const bool res = form & 1, bias = form & 2, aligned = !(form & 4), im2col = form & 8, act = form & 16;
          if (im2col && res) continue;
          const int Kpad = (K + GB_BK - 1) / GB_BK * GB_BK;
          int BN = gb_columns(N, K, res);
          if (BN == 0) {
            if (N % 64 == 0 || N <= 256) report("no tile", N, K, mt, 0, Bf16Room{});
            continue;
          }
          BN = gb_narrow(BN, N, mt, 148);
          const bool staged = BN % 64 == 0, rtma = staged && res && BN <= 128;
          const int rounds = (mt * (N / BN) + 147) / 148;
          const Bf16Room r = gb_room({N, BN, Kpad, rounds, im2col, staged, res, rtma, act, bias, aligned});
          const Bf16Room plain = gb_room({N, BN, Kpad, rounds, im2col, staged, res, rtma, act, false, true});
          ++seen;
          if (N % BN != 0) report("not whole tiles", N, K, mt, BN, r);
          if (r.bytes == 0 || r.bytes > 227 * 1024) report("refused", N, K, mt, BN, r);
          if (r.stages < 2 || r.stages > GB_MAX_STAGES || r.ostg > 4) report("ring", N, K, mt, BN, r);
          if (staged && r.ostg < (rtma ? 3 : 2)) report("slots", N, K, mt, BN, r);
          if (aligned && r.ostg < plain.ostg) report("fewer slots", N, K, mt, BN, r);
          if (aligned && rtma && r.stages < plain.stages) report("fewer stages", N, K, mt, BN, r);
          // long K loops of many tiles keep the fourth stage
          if (aligned && rounds >= 7 && Kpad >= 12 * GB_BK && plain.stages >= 4 && r.stages < 4) report("fourth stage", N, K, mt, BN, r);
          if (r.bias_n != 0 && (!bias || r.bias_n != N)) report("bias", N, K, mt, BN, r);
          // what the kernel lays out: weights, ring, two halves of staging slots, barriers, bias, 1024 bytes of alignment
          const size_t need = (r.wres ? (size_t)Kpad * BN * 2 : 0) + (size_t)r.stages * (GB_A_BYTES + (r.wres ? 0 : BN * 128)) +
                              (size_t)r.ostg * 2 * GB_BOX + GB_BAR_BYTES + (size_t)r.bias_n * 4 + 1024;
          if (r.bytes != 0 && r.bytes != need) report("bytes", N, K, mt, BN, r);
          // a bias that starts off 16 bytes cannot be read from global memory in fours
          if (bias && !aligned && N <= GB_BIAS_MAX && r.bias_n != N) report("bias not copied", N, K, mt, BN, r);
          // slots and stages of a residual without any bias in shared memory: 128 columns 4 and 3, 64 columns 4 and 4
          if (rtma && !r.wres && aligned && (r.stages != 4 || r.ostg != (BN == 128 ? 3 : 4))) report("residual", N, K, mt, BN, r);
        }
  std::printf("%ld cases, %ld bad\n", seen, bad);
  return bad != 0 || seen < 100000;
}
"""


def test_every_width_fits(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "room.cpp", tmp_path / "room"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "cssm_b200", "csrc"), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
