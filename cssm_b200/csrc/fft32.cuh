// 32-point complex FFT of one lane, in registers, and the 32x32 plane geometry of the kernels that give a lane whole rows and
// columns (csrc/gdn_spectral_p32.cu).
//
// Two planes to a warp.  Rows: lane = (plane, j) packs the real rows j and j + 16 of its plane into one FFT and separates them in
// its registers.  Columns: the DC and Nyquist columns of real rows are real and share one FFT, so a plane has 16 columns and
// lane = (plane, column).  A spectrum is kept as 32 rows of 17 entries (16 used): entry (kh, 0) is A[kh] + i N[kh] of the DC
// and Nyquist columns A, N, entry (kh, kw) the bin itself.  With that odd pitch both the row and the column lanes' 8-byte accesses are
// free of bank conflicts.
#pragma once
#include "fft.cuh"

namespace cssm {

// cos / sin of 2 pi p / 32, p = 0 .. 8; the rest by symmetry (p is a compile-time constant where it is used)
__host__ __device__ constexpr float c32q(int p) {
  return p == 0 ? 1.f : p == 1 ? 0.98078528040323044913f : p == 2 ? 0.92387953251128675613f : p == 3 ? 0.83146961230254523708f
       : p == 4 ? 0.70710678118654752440f : p == 5 ? 0.55557023301960222474f : p == 6 ? 0.38268343236508977173f
       : p == 7 ? 0.19509032201612826785f : 0.f;
}
__host__ __device__ constexpr float c32(int p) { return p <= 8 ? c32q(p) : p <= 16 ? -c32q(16 - p) : p <= 24 ? -c32q(p - 16) : c32q(32 - p); }
__host__ __device__ constexpr float s32(int p) { return c32((p + 24) & 31); }

template <bool INV>
__device__ __forceinline__ void dft4v(cf& a, cf& b, cf& c, cf& d) {
  const cf s0 = a + c, d0 = a - c, s1 = b + d, d1 = b - d;
  const cf r = INV ? mk(-d1.y, d1.x) : mk(d1.y, -d1.x);
  a = s0 + s1; c = s0 - s1; b = d0 + r; d = d0 - r;
}

// x[n] -> X[k], natural order (unscaled); INV: e^{+...}
template <bool INV>
__device__ __forceinline__ void fft32_lane(cf (&x)[32]) {
  cf y[4][8];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    cf t[8];
#pragma unroll
    for (int n1 = 0; n1 < 8; ++n1) t[n1] = x[4 * n1 + n2];
    dft8<INV>(t);
#pragma unroll
    for (int k1 = 0; k1 < 8; ++k1) {
      const int p = n2 * k1;
      if (p == 0) y[n2][k1] = t[k1];
      else if (p == 8) y[n2][k1] = INV ? mk(-t[k1].y, t[k1].x) : mk(t[k1].y, -t[k1].x);
      else {
        const float c = c32(p), s = INV ? s32(p) : -s32(p);
        y[n2][k1] = mk(t[k1].x * c - t[k1].y * s, t[k1].y * c + t[k1].x * s);
      }
    }
  }
#pragma unroll
  for (int k1 = 0; k1 < 8; ++k1) {
    dft4v<INV>(y[0][k1], y[1][k1], y[2][k1], y[3][k1]);
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) x[k1 + 8 * k2] = y[k2][k1];
  }
}

constexpr int P32_PITCH = 17, P32_PLANE_CF = 32 * P32_PITCH;      // one spectrum
constexpr int P32_RAW = 2 * 32 * 128;                              // two planes as TMA leaves them: rows of 128 bytes, 128-byte swizzle

// rows j, j + 16 of the lane's plane from a swizzled pair of planes (64 rows): z[n] = (row j, row j + 16)
__device__ __forceinline__ void p32_load_rows(const unsigned char* raw, int pl, int j, cf (&z)[32]) {
  const unsigned char* r0 = raw + (pl * 32 + j) * 128;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int off = (c ^ (j & 7)) << 4;                            // j and j + 16 have the same low bits
    const float4 u = *reinterpret_cast<const float4*>(r0 + off), v = *reinterpret_cast<const float4*>(r0 + 16 * 128 + off);
    z[4 * c] = mk(u.x, v.x); z[4 * c + 1] = mk(u.y, v.y); z[4 * c + 2] = mk(u.z, v.z); z[4 * c + 3] = mk(u.w, v.w);
  }
}
// rows j, j + 16 from (.y, .x) of z
__device__ __forceinline__ void p32_store_rows_swapped(unsigned char* raw, int pl, int j, const cf (&z)[32]) {
  unsigned char* r0 = raw + (pl * 32 + j) * 128;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int off = (c ^ (j & 7)) << 4;
    *reinterpret_cast<float4*>(r0 + off) = make_float4(z[4 * c].y, z[4 * c + 1].y, z[4 * c + 2].y, z[4 * c + 3].y);
    *reinterpret_cast<float4*>(r0 + 16 * 128 + off) = make_float4(z[4 * c].x, z[4 * c + 1].x, z[4 * c + 2].x, z[4 * c + 3].x);
  }
}
// row spectra of the packed pair -> rows j, j + 16 of the plane's buffer
__device__ __forceinline__ void p32_put_rows(cf* sp, int j, const cf (&z)[32]) {
  cf* a = sp + j * P32_PITCH;
  cf* b = a + 16 * P32_PITCH;
  a[0] = mk(z[0].x, z[16].x);
  b[0] = mk(z[0].y, z[16].y);
#pragma unroll
  for (int k = 1; k < 16; ++k) {
    const cf u = z[k], v = z[32 - k];
    a[k] = mk(0.5f * (u.x + v.x), 0.5f * (u.y - v.y));
    b[k] = mk(0.5f * (u.y + v.y), 0.5f * (v.x - u.x));
  }
}
// the inverse: rows j, j + 16 (entry 0: the real DC and Nyquist values) -> packed full spectrum, real and imaginary parts
// exchanged: the forward FFT of that is the inverse one, exchanged
__device__ __forceinline__ void p32_get_rows_swapped(const cf* sp, int j, cf (&z)[32]) {
  const cf* a = sp + j * P32_PITCH;
  const cf* b = a + 16 * P32_PITCH;
  const cf a0 = a[0], b0 = b[0];
  z[0] = mk(b0.x, a0.x);
  z[16] = mk(b0.y, a0.y);
#pragma unroll
  for (int k = 1; k < 16; ++k) {
    const cf e = a[k], o = b[k];
    z[k] = mk(e.y + o.x, e.x - o.y);
    z[32 - k] = mk(o.x - e.y, e.x + o.y);
  }
}

// Bins of a lane: two of column kw, kh[0] and kh[1].  Threads t = 0 .. 271 in columns of 16 (j = t & 15) in the order 0, 16, 1,
// 2, ... 15: the first warp has the two real columns, with j and 32 - j (0 and 16 for j = 0), the others j and j + 16.
__device__ __forceinline__ void p32_bins(int t, int& kw, int (&kh)[2]) {
  const int c = t >> 4, j = t & 15;
  kw = c == 0 ? 0 : c == 1 ? 16 : c - 1;
  kh[0] = j;
  kh[1] = c >= 2 ? j + 16 : j == 0 ? 16 : 32 - j;
}
// spectrum value of the lane's bin q (real: the lane is of the first warp)
__device__ __forceinline__ cf p32_read1(const cf* sp, bool real, int kw, const int (&kh)[2], int q) {
  if (!real) return sp[kh[q] * P32_PITCH + kw];
  const cf u = sp[kh[0] * P32_PITCH], v = sp[kh[1] * P32_PITCH];
  if (kh[0] == 0) {
    const cf z = q ? v : u;
    return mk(kw ? z.y : z.x, 0.f);
  }
  // A[k] = (Z[k] + conj Z[-k]) / 2, N[k] = (Z[k] - conj Z[-k]) / 2i; the other bin is the conjugate
  const cf x = kw ? mk(0.5f * (u.y + v.y), 0.5f * (v.x - u.x)) : mk(0.5f * (u.x + v.x), 0.5f * (u.y - v.y));
  return q ? mk(x.x, -x.y) : x;
}
// output values of the lane's two bins -> spectrum for the inverse; as irfft2 does, only the part of columns 0 and 16
// whose inverse is real enters.  Called by whole warps where `real`.
__device__ __forceinline__ void p32_write(cf* sp, bool real, int kw, const int (&kh)[2], cf o0, cf o1) {
  if (!real) {
    sp[kh[0] * P32_PITCH + kw] = o0;
    sp[kh[1] * P32_PITCH + kw] = o1;
    return;
  }
  const bool self = kh[0] == 0;
  // this column's Hermitian part at kh[0] (self-paired bins: their real parts, both)
  const cf e = self ? mk(o0.x, o1.x) : mk(0.5f * (o0.x + o1.x), 0.5f * (o0.y - o1.y));
  const cf f = mk(__shfl_xor_sync(0xffffffffu, e.x, 16), __shfl_xor_sync(0xffffffffu, e.y, 16));      // the other column's
  const cf a = kw ? f : e, n = kw ? e : f;
  const int row = kh[kw ? 1 : 0];
  cf m;
  if (self) m = kw ? mk(a.y, n.y) : mk(a.x, n.x);
  else m = kw ? mk(a.x + n.y, n.x - a.y) : mk(a.x - n.y, a.y + n.x);      // conj(A) + i conj(N) : A + i N
  sp[row * P32_PITCH] = m;
}
// half-spectrum sums of |.|^2 of the lane's plane, from the rows (Parseval; columns 0 and 16 count once, the others twice in the
// full sum): lanes 0-15 get plane 0's, 16-31 plane 1's.  xx: sums of squares of the lane's two rows, z: their packed row spectra.
__device__ __forceinline__ float p32_energy(float xx, const cf (&z)[32]) {
  float e = 512.f * xx + 16.f * (z[0].x * z[0].x + z[0].y * z[0].y + z[16].x * z[16].x + z[16].y * z[16].y);
#pragma unroll
  for (int o = 8; o; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  return e;
}

}  // namespace cssm
