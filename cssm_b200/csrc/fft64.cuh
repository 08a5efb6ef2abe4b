// 64-point complex FFT of one lane, in registers, and the 64x64 plane geometry of the kernel that gives a lane whole rows and
// columns (csrc/gdn_spectral_p64.cu): one plane to a warp.
//
// Rows: lane j packs the real rows 2 j and 2 j + 1 of the plane into one FFT and separates them in its registers.  Columns: the DC and
// Nyquist columns of real rows are real and share one FFT, so a plane has 32 columns and lane = column.  A plane's region of 64 x 33
// entries of 8 bytes holds in turn
//   raw       pairs of rows, 528 bytes apart (16-byte accesses of a lane's pair are free of bank conflicts);
//   rows      [even rows, odd rows][k]: row h at p64_row(h) * 33, entry 0 the real DC and Nyquist values;
//   spectrum  bin (kh, kw) at p64_slot(bin_index(PATH_R64, kh, kw)): the order of the gates and kernel spectra, with the eight kh of a
//             group turned by kw so that lanes of consecutive columns and lanes of consecutive bins both meet 16 different banks.
// Going forward rows and bins are twice the transform (halves are left out), the packed column is not.
#pragma once
#include "fft.cuh"

namespace cssm {

// cos / sin of 2 pi p / 64, p = 0 .. 16; the rest by symmetry (p is a compile-time constant where it is used)
__host__ __device__ constexpr float c64q(int p) {
  return p == 0 ? 1.f : p == 1 ? 0.9951847266721968862448f : p == 2 ? 0.9807852804032304491261f : p == 3 ? 0.9569403357322088649357f
       : p == 4 ? 0.9238795325112867561281f : p == 5 ? 0.8819212643483550297127f : p == 6 ? 0.8314696123025452370787f
       : p == 7 ? 0.7730104533627369608109f : p == 8 ? 0.7071067811865475244008f : p == 9 ? 0.6343932841636454982151f
       : p == 10 ? 0.5555702330196022247428f : p == 11 ? 0.4713967368259976485563f : p == 12 ? 0.3826834323650897717284f
       : p == 13 ? 0.2902846772544623676361f : p == 14 ? 0.1950903220161282678482f : p == 15 ? 0.0980171403295606019941f : 0.f;
}
__host__ __device__ constexpr float c64(int p) { return p <= 16 ? c64q(p) : p <= 32 ? -c64q(32 - p) : p <= 48 ? -c64q(p - 32) : c64q(64 - p); }
__host__ __device__ constexpr float s64(int p) { return c64((p + 48) & 63); }

// x[n] -> X[k], e^{-...}, natural order (unscaled)
__device__ __forceinline__ void fft64_lane(cf (&x)[64]) {
#pragma unroll
  for (int n2 = 0; n2 < 8; ++n2) {
    cf t[8];
#pragma unroll
    for (int n1 = 0; n1 < 8; ++n1) t[n1] = x[8 * n1 + n2];
    dft8<false>(t);
#pragma unroll
    for (int k1 = 0; k1 < 8; ++k1) {
      const int p = n2 * k1;
      if (p == 0) x[8 * k1 + n2] = t[k1];
      else if (p == 16) x[8 * k1 + n2] = mk(t[k1].y, -t[k1].x);
      else {
        const float c = c64(p), s = -s64(p);
        x[8 * k1 + n2] = mk(t[k1].x * c - t[k1].y * s, t[k1].y * c + t[k1].x * s);
      }
    }
  }
  cf y[64];
#pragma unroll
  for (int k1 = 0; k1 < 8; ++k1) {
    cf t[8];
#pragma unroll
    for (int n2 = 0; n2 < 8; ++n2) t[n2] = x[8 * k1 + n2];
    dft8<false>(t);
#pragma unroll
    for (int k2 = 0; k2 < 8; ++k2) y[k1 + 8 * k2] = t[k2];
  }
#pragma unroll
  for (int k = 0; k < 64; ++k) x[k] = y[k];
}

constexpr int P64_PITCH = 33, P64_PLANE_CF = 64 * P64_PITCH;
constexpr int P64_RAW = 32 * 528;

__host__ __device__ constexpr int p64_row(int h) { return (h & 1) * 32 + (h >> 1); }
// i: bin_index(PATH_R64, kh, kw) = ((kh / 8) * 33 + kw) * 8 + kh % 8
__host__ __device__ __forceinline__ int p64_slot(int i) { return i ^ ((((i >> 3) % 33) >> 1) & 7); }

// raw plane -> z[n] = (row 2 j, row 2 j + 1)
__device__ __forceinline__ void p64_load_rows(const unsigned char* raw, int j, cf (&z)[64]) {
  const float4* r = reinterpret_cast<const float4*>(raw + j * 528);
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    const float4 u = r[c], v = r[16 + c];
    z[4 * c] = mk(u.x, v.x); z[4 * c + 1] = mk(u.y, v.y); z[4 * c + 2] = mk(u.z, v.z); z[4 * c + 3] = mk(u.w, v.w);
  }
}
// rows 2 j, 2 j + 1 from (.y, .x) of z
__device__ __forceinline__ void p64_store_rows_swapped(unsigned char* raw, int j, const cf (&z)[64]) {
  float4* r = reinterpret_cast<float4*>(raw + j * 528);
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    r[c] = make_float4(z[4 * c].y, z[4 * c + 1].y, z[4 * c + 2].y, z[4 * c + 3].y);
    r[16 + c] = make_float4(z[4 * c].x, z[4 * c + 1].x, z[4 * c + 2].x, z[4 * c + 3].x);
  }
}
// row spectra of the packed pair -> the rows' places
__device__ __forceinline__ void p64_put_rows(cf* sp, int j, const cf (&z)[64]) {
  cf* a = sp + j * P64_PITCH;
  cf* b = a + 32 * P64_PITCH;
  a[0] = mk(z[0].x, z[32].x);
  b[0] = mk(z[0].y, z[32].y);
#pragma unroll
  for (int k = 1; k < 32; ++k) {
    const cf u = z[k], v = z[64 - k];
    a[k] = mk(u.x + v.x, u.y - v.y);
    b[k] = mk(u.y + v.y, v.x - u.x);
  }
}
// the inverse (rows not doubled) -> packed full spectrum, real and imaginary parts exchanged: the forward FFT of that is the
// inverse one, exchanged
__device__ __forceinline__ void p64_get_rows_swapped(const cf* sp, int j, cf (&z)[64]) {
  const cf* a = sp + j * P64_PITCH;
  const cf* b = a + 32 * P64_PITCH;
  const cf a0 = a[0], b0 = b[0];
  z[0] = mk(b0.x, a0.x);
  z[32] = mk(b0.y, a0.y);
#pragma unroll
  for (int k = 1; k < 32; ++k) {
    const cf e = a[k], o = b[k];
    z[k] = mk(e.y + o.x, e.x - o.y);
    z[64 - k] = mk(o.x - e.y, e.x + o.y);
  }
}
// column kw = 0 .. 31 of a lane -> spectrum places (0: the packed column, for p64_unpack_columns)
__device__ __forceinline__ void p64_put_columns(cf* sp, int kw, const cf (&z)[64]) {
  const int f = (kw >> 1) & 7;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    cf* d = sp + kw * 8 + (j ^ f);
#pragma unroll
    for (int g = 0; g < 8; ++g) d[g * 264] = z[8 * g + j];
  }
}
__device__ __forceinline__ void p64_get_columns_swapped(const cf* sp, int kw, cf (&z)[64]) {
  const int f = (kw >> 1) & 7;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const cf* d = sp + kw * 8 + (j ^ f);
#pragma unroll
    for (int g = 0; g < 8; ++g) { const cf v = d[g * 264]; z[8 * g + j] = mk(v.y, v.x); }
  }
}
// packed column Z = A + i N of the DC and Nyquist columns -> 2 A in column 0, 2 N in column 32 (the whole warp)
__device__ __forceinline__ void p64_unpack_columns(cf* sp, int lane) {
  cf u[2], v[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int k = lane + 32 * q, m = (64 - k) & 63;
    u[q] = sp[(k >> 3) * 264 + (k & 7)];
    v[q] = sp[(m >> 3) * 264 + (m & 7)];
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int k = lane + 32 * q;
    cf* d = sp + (k >> 3) * 264 + (k & 7);
    d[0] = mk(u[q].x + v[q].x, u[q].y - v[q].y);
    d[256] = mk(u[q].y + v[q].y, v[q].x - u[q].x);
  }
}
// columns 0 and 32 -> packed column 0; as irfft2 does, only the parts whose inverse is real enter
__device__ __forceinline__ void p64_pack_columns(cf* sp, int lane) {
  cf z[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int k = lane + 32 * q, m = (64 - k) & 63;
    const cf* d = sp + (k >> 3) * 264 + (k & 7);
    const cf* e = sp + (m >> 3) * 264 + (m & 7);
    const cf a = d[0], ac = e[0], n = d[256], nc = e[256];
    z[q] = mk(0.5f * (a.x + ac.x) - 0.5f * (n.y - nc.y), 0.5f * (a.y - ac.y) + 0.5f * (n.x + nc.x));
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int k = lane + 32 * q;
    sp[(k >> 3) * 264 + (k & 7)] = z[q];
  }
}

}  // namespace cssm
