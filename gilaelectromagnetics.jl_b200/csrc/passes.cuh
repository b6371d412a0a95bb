// passes.cuh -- kernel parameters of the five matvec passes and the device
// helpers that every form of a pass shares (kernel addressing, tile orders,
// the 3x3 multiply, the Lippmann-Schwinger epilogue).
#pragma once
#include "fft.cuh"
#include "matvec.cuh"

namespace gila {

// Shared-memory row of an x pass: element i sits at i + i/8, which spreads
// the stride-R accesses of the early Stockham stages over all banks.
__host__ __device__ __forceinline__ int row_stride(int P) { return P + (P + 7) / 8; }

// -------------------------------------------------------------------- xfwd
template <typename C>
struct XfParams {
  const C* in;
  C* A;
  const AxisPlan* pl;  // device copy
  int P;
  const C* tw;
  int nin;       // source x cells
  int M;         // rows per CTA
  int64_t rows;  // total rows = 3 * sy * sz * nrhs
  FDiv nind;     // division by nin
};

// ---------------------------------------------------------------------- y
template <typename C>
struct YParams {
  const C* src;
  C* dst;
  const AxisPlan* pl;  // device copy
  int P;
  const C* tw;
  int Px;
  int TX;
  int ntiles;     // ceil(Px / TX)
  int nin, nout;  // rows read / written
  int nz;         // z planes per channel in this pass
  int src_z, dst_z;          // z planes per channel in the src / dst layouts
  int src_rows, dst_rows;    // y rows per plane in the src / dst layouts
  int64_t q0;                // first plane (ch*nz + z) of this launch
  int64_t src_sub, dst_sub;  // plane index of the first plane held by src / dst
  FDiv md;                   // division by the line count TX
  // kx tiles of this launch: nt tiles, the first nlo from lo0 on, the rest
  // from hi0 on (all tiles: nt = nlo = ntiles, lo0 = 0)
  int nt, nlo, lo0, hi0;
};

// ---------------------------------------------------------------------- z
// Kernel address of frequency f on one axis (mirror rules of mulBrnDev!,
// src/glaActSup.jl:789-846), computed arithmetically: branch bit p = f & 1,
// stored index m, mirrored flag (sign flip of the off-diagonal components).
struct AxMap {
  int brn;   // P / 2
  int full;  // stored extent == brn (no mirror)
  int fe;    // forward count of the even branch: ceil(t/2) + iseven(t)
  int fo;    // forward count of the odd branch: ceil(t/2)
};
__device__ __forceinline__ void ax_map(const AxMap& a, int f, int& p, int& m, int& mir) {
  p = f & 1;
  const int k = f >> 1;
  if (a.full) {
    m = k;
    mir = 0;
  } else if (p == 0) {
    mir = k >= a.fe;
    m = mir ? a.brn - k : k;
  } else {
    mir = k >= a.fo;
    m = mir ? a.brn - 1 - k : k;
  }
}

template <typename C>
struct ZParams {
  C* B;
  const C* ker;
  const int* mapx;
  const int* mapy;
  const int* mapz;
  const AxisPlan* pl;  // device copy
  int P;
  const C* tw;
  int Px, Py;
  int TX, ntiles;
  int nin, nout;  // source / target z cells
  int zb;         // z planes per channel in B
  int tx, ty, tz; // stored kernel extents
  int parT;
  int nrhs;
  int zmir;  // fused z pass: one kernel load per mirror pair of z frequencies
  double scale;
  FDiv md;    // division by the tile width TX
  FDiv nind;  // division by nin
  AxMap ax[3];
  int ts0, nts;  // positions [ts0, ts0 + nts) of the mirror tile order (all: 0, ntiles)
  // spectrum rows of this launch: B holds Py rows, which are rows ky0 ..
  // ky0 + Py - 1 of the operator's spectrum (the kernel values and mirror
  // flags follow the operator's row); ky0 = 0 and Py = the full row count
  // except for the slab pieces of a slab-decomposed matvec
  int ky0;
};

// ky order that places each frequency next to its mirror Py - ky, and kx
// tile order that places tile i next to tile ntiles-1-i, so that the four
// CTAs reading the same stored (half-spectrum) kernel values run together and
// the re-reads are served from L2.
__device__ __forceinline__ int mirror_seq(int idx, int n) {
  if (idx == 0) return 0;
  if (n % 2 == 0) {
    if (idx == 1) return n / 2;
    const int k = (idx - 2) / 2 + 1;
    return (idx % 2 == 0) ? k : n - k;
  }
  const int k = (idx - 1) / 2 + 1;
  return (idx % 2 == 1) ? k : n - k;
}
__device__ __forceinline__ int tile_seq(int idx, int n) {
  const int k = idx / 2;
  return (idx % 2 == 0) ? k : n - 1 - k;
}

// FP64 kernel values are read once per column and their L2 lines are shared
// by the CTAs of the mirror columns, not by the threads of one CTA: the loads
// bypass L1 allocation (measured 3% faster z passes at 256x256x128 than
// cached loads, whose fills share the L1 data path with the transposes).
__device__ __forceinline__ double2 ld_nc_na(const double2* g) {
  double2 r;
  asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(r.x), "=d"(r.y) : "l"(g));
  return r;
}
// FP32: cached (measured faster than loads past L1 here), since a line-pair
// thread reads the two x parities of one stored index, which sit side by
// side: one 16-byte load where both are unmirrored, two loads of one line
// otherwise
__device__ __forceinline__ float2 ld_nc_na(const float2* g) { return __ldg(g); }
template <typename C>
__device__ __forceinline__ C ker_ld(const C* __restrict__ g, int c, int tx) {
  return ld_nc_na(g + 2 * c * tx);
}
// Stored kernel layout: target-partition blocks laid out by ker_index
// ([py,pz][tz][ty][6][tx][px]); the threads of a warp (consecutive kx of a
// tile, alternating x parity) read consecutive entries of one component.
// Returns the address of component 0 of entry (eo, iz, iy, ix); component c
// is 2 * c * tx entries further (ker_ld).
template <typename C>
__device__ __forceinline__ const C* ker_at(const C* __restrict__ kpar, int eo, int iz, int iy, int ix, int tx, int ty,
                                           int tz) {
  // one partition holds 8 * tz * ty * 6 * tx < 2^31 entries (host-checked)
  return kpar + (((((eo & 3) * tz + iz) * ty + iy) * 6) * tx + ix) * 2 + (eo >> 2);
}

// -------------------------------------------------------------------- xinv
template <typename C>
struct XiParams {
  const C* A;
  C* out;
  const AxisPlan* pl;  // device copy
  int P;
  const C* tw;
  int nout;  // target x cells
  int M;
  int64_t rows;   // rows in this launch
  int64_t g_off;  // global row index (over all rhs) of the first row
  int ty, tz, parT;
  int part_scatter;  // parT > 1
  int tdiv[3];
  int toff[64][3];
  int64_t full[3];
  C alpha, beta;
  FDiv pd;  // division by P
  // Lippmann-Schwinger epilogue (ls != 0): out = ls_in - chi .* value
  const C* ls_in;
  const C* ls_chi;
  int64_t ls_chi_rs;
  int ls;
  FDiv rows_rhs;  // division by 3 * tz * ty (rows per right-hand side)
  FDiv rows_zy;   // division by tz * ty
};

// the epilogue value at output index o of row gg, column i
template <typename C>
__device__ __forceinline__ C ls_value(const C* __restrict__ in, const C* __restrict__ chi, int64_t chi_rs, FDiv rr,
                                      FDiv rzy, int nout, int64_t gg, int i, int64_t o, C v) {
  const uint32_t rhs = rr.div((uint32_t)gg);
  const uint32_t rem = (uint32_t)gg - rhs * rr.d;
  const uint32_t zy = rem - rzy.div(rem) * rzy.d;
  const C c = chi[(int64_t)rhs * chi_rs + (int64_t)zy * nout + i];
  return csub(in[o], cmul(c, v));
}

// a with both parts' signs flipped when f != 0: a sign-bit XOR on the high
// words, no FP64 instruction
__device__ __forceinline__ double2 cflip(double2 a, int f) {
  const long long m = (long long)(f != 0) << 63;
  return make_double2(__longlong_as_double(__double_as_longlong(a.x) ^ m),
                      __longlong_as_double(__double_as_longlong(a.y) ^ m));
}

// s * (g0 a + g1 b + g2 c) as two FMA chains
__device__ __forceinline__ double2 mac3(const double2& g0, const double2& a, const double2& g1, const double2& b,
                                       const double2& g2, const double2& c, double s) {
  double re = g0.x * a.x;
  re = fma(-g0.y, a.y, re);
  re = fma(g1.x, b.x, re);
  re = fma(-g1.y, b.y, re);
  re = fma(g2.x, c.x, re);
  re = fma(-g2.y, c.y, re);
  double im = g0.x * a.y;
  im = fma(g0.y, a.x, im);
  im = fma(g1.x, b.y, im);
  im = fma(g1.y, b.x, im);
  im = fma(g2.x, c.y, im);
  im = fma(g2.y, c.x, im);
  return make_double2(re * s, im * s);
}

// the 3x3 symmetric multiply of one frequency (stored kernel g: xx, yy, zz,
// xy, xz, yz; mirror flags rx, ry, rz), scaled by s
__device__ __forceinline__ void zmul3f(double2& x0, double2& x1, double2& x2, const double2 (&g)[6], int rx, int ry,
                                       int rz, double s) {
  const double2 gxy = cflip(g[3], rx ^ ry), gxz = cflip(g[4], rx ^ rz), gyz = cflip(g[5], ry ^ rz);
  const double2 a = x0, b = x1, c = x2;
  x0 = mac3(g[0], a, gxy, b, gxz, c, s);
  x1 = mac3(gxy, a, g[1], b, gyz, c, s);
  x2 = mac3(gxz, a, gyz, b, g[2], c, s);
}

__device__ __forceinline__ float2 cflip(float2 a, int f) {
  const int m = (f != 0) << 31;
  return make_float2(__int_as_float(__float_as_int(a.x) ^ m), __int_as_float(__float_as_int(a.y) ^ m));
}

__device__ __forceinline__ float2 mac3(const float2& g0, const float2& a, const float2& g1, const float2& b,
                                      const float2& g2, const float2& c, float s) {
  float re = g0.x * a.x;
  re = fmaf(-g0.y, a.y, re);
  re = fmaf(g1.x, b.x, re);
  re = fmaf(-g1.y, b.y, re);
  re = fmaf(g2.x, c.x, re);
  re = fmaf(-g2.y, c.y, re);
  float im = g0.x * a.y;
  im = fmaf(g0.y, a.x, im);
  im = fmaf(g1.x, b.y, im);
  im = fmaf(g1.y, b.x, im);
  im = fmaf(g2.x, c.y, im);
  im = fmaf(g2.y, c.x, im);
  return make_float2(re * s, im * s);
}

__device__ __forceinline__ void zmul3f(float2& x0, float2& x1, float2& x2, const float2 (&g)[6], int rx, int ry,
                                       int rz, float s) {
  const float2 gxy = cflip(g[3], rx ^ ry), gxz = cflip(g[4], rx ^ rz), gyz = cflip(g[5], ry ^ rz);
  const float2 a = x0, b = x1, c = x2;
  x0 = mac3(g[0], a, gxy, b, gxz, c, s);
  x1 = mac3(gxy, a, g[1], b, gyz, c, s);
  x2 = mac3(gxz, a, gyz, b, g[2], c, s);
}

}  // namespace gila
