// kerbuild.cu -- the FP64 Green-kernel build on the GPU.
//
// Replaces GlaOprMem's kernel section (src/glaMemSup.jl:44-156) and the
// real-space element generation it calls (src/glaGen.jl, src/glaInt.jl,
// src/glaIntSup.jl), which the reference runs on host threads (hours at
// 256x256x128, hence its JLD2 cache).  Everything stays in FP64:
//
//   1. weak (singular) face-pair integrals wekS / wekE / wekV: the DIRECTFN
//      nested Gauss-Legendre sums (src/glaIntSup.jl), one launch per kind of
//      integral, partials reduced in a fixed order (deterministic);
//   2. the 8 near offsets (egoFunSng!, src/glaGen.jl:350-528): corrected
//      pairs from the weak values, the rest by cubature;
//   3. far offsets (egoFunInn! / egoFunOut!, src/glaGen.jl:233-248,322-335):
//      for the 24 face pairs that feed the six stored components the adaptive
//      Genz-Malik degree-7/5 cubature (the algorithm of Cubature.jl's
//      hcubature, src/glaGen.jl:574-576): the rule once per pair and thread,
//      then a warp for each pair that needs more regions;
//   4. external operators: circulant separations by grdSel/sepGrd
//      (src/glaGen.jl:603-645), touching offsets averaged from the contact
//      self circulant (egoCntOut!, src/glaGen.jl:250-306);
//   5. Toeplitz -> circulant embedding (egoToeCrc!, src/glaGen.jl:143-163),
//      FP64 3-D FFT of the six components, parity-branch extraction and
//      symmetric truncation (src/glaMemSup.jl:96-156), cast to the operator
//      dtype, NaN/Inf check.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "internal.h"
#include "matvec_mx.cuh"

namespace gila {
namespace kb {

constexpr double PI = 3.14159265358979323846264338327950288;
constexpr double S3 = 1.7320508075688772935274463415058723669;
constexpr double CUB_RELTOL = 1e-6, CUB_ABSTOL = 1e-9, CNT_TOL = 1e-8;  // src/glaGen.jl:3-8
constexpr int kMaxOrd = 64;

// ------------------------------------------------------------ complex FP64
struct Z {
  double x, y;
};
__host__ __device__ inline Z zmk(double a, double b) { return Z{a, b}; }
__host__ __device__ inline Z zadd(Z a, Z b) { return Z{a.x + b.x, a.y + b.y}; }
__host__ __device__ inline Z zsub(Z a, Z b) { return Z{a.x - b.x, a.y - b.y}; }
__host__ __device__ inline Z zmul(Z a, Z b) { return Z{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
__host__ __device__ inline Z zsc(Z a, double s) { return Z{a.x * s, a.y * s}; }
__host__ __device__ inline Z zdiv(Z a, Z b) {
  const double d = b.x * b.x + b.y * b.y;
  return Z{(a.x * b.x + a.y * b.y) / d, (a.y * b.x - a.x * b.y) / d};
}

struct Consts {
  int ord;
  double x[kMaxOrd], w[kMaxOrd];  // Gauss-Legendre nodes / weights on [-1,1]
  Z f;                            // frqPhz
};

// sclEgo (src/glaInt.jl:41-44): exp(2 pi i d f) / (4 pi d f^2)
__device__ inline Z scl_ego(double d, Z f) {
  const Z z = zsc(f, (2.0 * PI) * d);
  const double e = exp(-z.y);
  double s, c;
  sincos(z.x, &s, &c);
  return zdiv(Z{e * c, e * s}, zsc(zmul(f, f), (4.0 * PI) * d));
}
// sclEgoN (src/glaInt.jl:51-59)
__device__ inline Z scl_ego_n(double d, Z f) {
  if (d > 1e-7) {
    const Z z = zsc(f, (2.0 * PI) * d);
    const double e = exp(-z.y);
    double s, c;
    sincos(z.x, &s, &c);
    return zdiv(Z{e * c - 1.0, e * s}, zsc(zmul(f, f), (4.0 * PI) * d));
  }
  const Z a = zdiv(Z{0.0, 1.0}, f);
  return Z{(a.x - PI * d) / 2.0, a.y / 2.0};
}

__device__ inline double thf(double a, double b, double p) { return 0.5 * ((b - a) * p + a + b); }

struct Tri6 {
  double r[6][3];
};

// Point of a triangle (r0, r1, r2) at (e, x) of the DIRECTFN simplex (spX!,
// src/glaIntSup.jl): affine, C + De e + Dx x.
struct Aff {
  double c[3], e[3], x[3];
};
__device__ inline Aff tri_aff(const double (*r)[3]) {
  Aff a;
  for (int d = 0; d < 3; ++d) {
    a.c[d] = 0.5 * (r[0][d] + r[1][d]);
    a.e[d] = 0.5 * (r[1][d] - r[0][d]);
    a.x[d] = (r[2][d] - a.c[d]) / S3;
  }
  return a;
}

// Along the innermost variable z of every weak integral the two points move
// on straight lines, so their difference is A + B z, and the integrand is
// z^k times the (regularised) kernel at its length.  One kernel value: for a
// real frequency a sine / cosine pair of the half phase, and e^{i t} - 1 =
// -2 sin^2(t/2) + 2 i sin(t/2) cos(t/2), which does not cancel at small t; the
// division by the length is one reciprocal root.  `rq` holds f.x and 1 / (4 pi
// f.x^2); a frequency with an imaginary part takes scl_ego / scl_ego_n.
struct RealF {
  double f, s;
};
// (out of line: the registers of its range reduction would count in every
// kernel below)
static __device__ __noinline__ double2 sincos_pi_any(double x) {
  double2 r;
  sincospi(x, &r.x, &r.y);
  return r;
}
// sin(pi x), cos(pi x).  Phases of up to a quarter half-turn -- every weak
// integral of cells below 1/8 wavelength -- take the Taylor sums to x^15 and
// x^16 (the next terms are below 5e-17): 16 multiply-adds instead of the
// library's range reduction and selects (weak integrals of a cubic cell at
// intOrd 32: 2.25 -> 2.11 ms).
__device__ __forceinline__ void sincos_pi(double x, double* sn, double* cs) {
  if (fabs(x) <= 0.25) {
    const double y = x * PI, t = y * y;
    double s = -1.0 / 1307674368000.0, c = 1.0 / 20922789888000.0;
    s = fma(s, t, 1.0 / 6227020800.0);
    c = fma(c, t, -1.0 / 87178291200.0);
    s = fma(s, t, -1.0 / 39916800.0);
    c = fma(c, t, 1.0 / 479001600.0);
    s = fma(s, t, 1.0 / 362880.0);
    c = fma(c, t, -1.0 / 3628800.0);
    s = fma(s, t, -1.0 / 5040.0);
    c = fma(c, t, 1.0 / 40320.0);
    s = fma(s, t, 1.0 / 120.0);
    c = fma(c, t, -1.0 / 720.0);
    s = fma(s, t, -1.0 / 6.0);
    c = fma(c, t, 1.0 / 24.0);
    c = fma(c, t, -0.5);
    *sn = fma(s * t, y, y);
    *cs = fma(c, t, 1.0);
    return;
  }
  const double2 r = sincos_pi_any(x);
  *sn = r.x;
  *cs = r.y;
}
template <bool RF>
__device__ __forceinline__ Z ego_line(double r2, bool sng, Z f, RealF rq) {
  if constexpr (RF) {
    if (!sng) {
      double i = rsqrt(r2);
      double sn, cs;
      sincos_pi(2.0 * (r2 * i) * rq.f, &sn, &cs);
      i *= rq.s;
      return Z{i * cs, i * sn};
    }
    if (r2 > 1e-14) {
      const double i = rsqrt(r2);
      double sn, cs;
      sincos_pi((r2 * i) * rq.f, &sn, &cs);
      const double g = 2.0 * sn * (i * rq.s);
      return Z{-g * sn, g * cs};
    }
    return Z{-0.5 * PI * sqrt(r2), 0.5 / rq.f};  // the limit (scl_ego_n)
  } else {
    const double d = sqrt(r2);
    return sng ? scl_ego_n(d, f) : scl_ego(d, f);
  }
}

// aS (src/glaIntSup.jl:313-332).  Both points lie on one triangle, subTri
// (src/glaIntSup.jl:365-379) is linear and the variable runs over u = th t, so
// the distance is th t |w| with w fixed by the angle and the sub-triangle
// (s_dir): the kernel's 1 / d cancels the weight u.
__device__ inline double s_dir(const Aff& a, double s1, double c1, int dir) {
  double de, dx;
  if (dir == 1) {
    de = -c1;
    dx = s1;
  } else if (dir == 2) {
    de = 0.5 * (c1 - s1 * S3);
    dx = 0.5 * (-c1 * S3 - s1);
  } else {
    de = 0.5 * (c1 + s1 * S3);
    dx = 0.5 * (c1 * S3 - s1);
  }
  double q = 0;
  for (int d = 0; d < 3; ++d) {
    const double v = a.e[d] * de + a.x[d] * dx;
    q += v * v;
  }
  return sqrt(q);
}
template <bool RF>
__device__ Z a_s(double wl, double th, const Consts& q, RealF rq) {
  Z acc{0, 0};
  for (int n = 0; n < q.ord; ++n) {
    const double u = thf(0.0, th, q.x[n]), d = u * wl;
    if constexpr (RF) {
      if (d > 1e-7) {
        double sn, cs;
        sincos_pi(d * rq.f, &sn, &cs);
        const double g = 2.0 * q.w[n] * sn;
        acc.x -= g * sn;
        acc.y += g * cs;
        continue;
      }
      acc = zadd(acc, zsc(Z{-0.5 * PI * d, 0.5 / rq.f}, q.w[n] * (d / rq.s)));  // the limit (scl_ego_n)
    } else {
      acc = zadd(acc, zsc(scl_ego_n(d, q.f), q.w[n] * u));
    }
  }
  return zsc(acc, RF ? 0.5 * th * rq.s / wl : 0.5 * th);
}
__device__ inline void psi_lim_s(int idf, double& a, double& b) {
  if (idf == 1 || idf == 5 || idf == 6) {
    a = 0.0;
    b = PI / 3.0;
  } else if (idf == 2 || idf == 7) {
    a = PI / 3.0;
    b = 2.0 * PI / 3.0;
  } else {
    a = 2.0 * PI / 3.0;
    b = PI;
  }
}
__device__ inline void eta_lim_s(int idf, double th, double& a, double& b) {
  if (idf == 1 || idf == 2) {
    a = 0.0;
    b = 1.0;
  } else if (idf == 3) {
    a = (S3 - tan(PI - th)) / (S3 + tan(PI - th));
    b = 1.0;
  } else if (idf == 4) {
    a = 0.0;
    b = (S3 - tan(PI - th)) / (S3 + tan(PI - th));
  } else if (idf == 5) {
    a = (tan(th) - S3) / (S3 + tan(th));
    b = 0.0;
  } else if (idf == 6) {
    a = -1.0;
    b = (tan(th) - S3) / (S3 + tan(th));
  } else {
    a = -1.0;
    b = 0.0;
  }
}
// nS (src/glaIntSup.jl:201-237): the n-th term (weight included) and its factor
template <bool RF>
__device__ inline Z n_s_term(int idf, double s1, double c1, double wl, double thB, int n, const Consts& q, RealF rq) {
  double L;
  if (idf == 1 || idf == 5) {
    L = (1.0 - thB) / c1;
  } else if (idf == 2 || idf == 3) {
    L = S3 * (1.0 - thB) / s1;
  } else if (idf == 6 || idf == 7) {
    L = S3 * (1.0 + thB) / s1;
  } else {
    L = -(1.0 + thB) / c1;
  }
  return zsc(a_s<RF>(wl, thf(0.0, L, q.x[n]), q, rq), 0.5 * L * q.w[n]);
}

// spxE! / aE / intNE (src/glaIntSup.jl:283-348,395-411): a pair's two
// triangles and the angles of the current point of the outer sums
struct EdgeGeo {
  const double (*v)[3];  // shared: C1 - C2, De1 + De2, Dx1, De2 c1, Dx2 s1
  double sB, cB, tB, s1, c1;
};
template <bool RF>
__device__ __forceinline__ Z a_e(const EdgeGeo& t, double lam, double eta, double sg, const Consts& q, RealF rq) {
  // sg 1: points (eta, z sB), (z cB c1 - eta, z cB s1); -1: the same with both
  // first coordinates negated
  double A[3], B[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    A[d] = t.v[0][d] + sg * eta * t.v[1][d];
    B[d] = t.v[2][d] * t.sB - t.cB * (sg * t.v[3][d] + t.v[4][d]);
  }
  Z acc{0, 0};
#pragma unroll 1
  for (int n = 0; n < q.ord; ++n) {
    const double z = thf(0.0, lam, q.x[n]);
    const double x = A[0] + B[0] * z, y = A[1] + B[1] * z, w = A[2] + B[2] * z;
    acc = zadd(acc, zsc(ego_line<RF>(x * x + y * y + w * w, true, q.f, rq), q.w[n] * z * z));
  }
  return zsc(acc, 0.5 * lam);
}
// both orientations (idf 1 and -1) of the n-th term share eta and lam
template <bool RF>
__device__ Z int_ne(int n, int idf1, double gam, const EdgeGeo& t, const Consts& q, RealF rq) {
  double eta, lam;
  if (idf1 == 1) {
    eta = thf(0.0, gam, q.x[n]);
    lam = S3 * (1 + eta) / (t.cB * (t.s1 + S3 * t.c1));
  } else if (idf1 == 2) {
    eta = thf(gam, 1.0, q.x[n]);
    lam = S3 * (1.0 - fabs(eta)) / t.sB;
  } else if (idf1 == 3) {
    eta = thf(gam, 1.0, q.x[n]);
    lam = S3 * (1.0 - fabs(eta)) / (t.cB * (t.s1 - S3 * t.c1));
  } else if (idf1 == 4) {
    eta = thf(0.0, 1.0, q.x[n]);
    lam = S3 * (1.0 - fabs(eta)) / (t.cB * (t.s1 - S3 * t.c1));
  } else {
    eta = thf(0.0, 1.0, q.x[n]);
    lam = S3 * (1.0 - eta) / t.sB;
  }
  Z v{0, 0};
#pragma unroll 1
  for (int h = 0; h < 2; ++h) v = zadd(v, a_e<RF>(t, lam, eta, h ? -1.0 : 1.0, q, rq));
  return v;
}
// n-th term of nE(idf1, 1, ...) + nE(idf1, -1, ...) (src/glaIntSup.jl:239-281),
// weight included
template <bool RF>
__device__ Z n_e_term(int idf1, int n, const EdgeGeo& t, const Consts& q, RealF rq) {
  // (idf1 1, 2: parts 1 and 2 at gam; 3: parts 1 and 3; 4, 5: one part)
  const bool two = idf1 <= 3;
  double gam = 1.0;
  if (idf1 <= 2) {
    const double k = t.s1 + S3 * t.c1;
    gam = (k - t.tB) / (k + t.tB);
  } else if (idf1 == 3) {
    gam = S3 * t.c1 / t.s1;
  }
  Z v{0, 0};
#pragma unroll 1
  for (int h = 0; h < (two ? 2 : 1); ++h) {
    const int part = !two ? (idf1 == 4 ? 4 : 5) : h == 0 ? 1 : idf1 == 3 ? 3 : 2;
    const double w = !two ? 0.5 : h == 0 ? 0.5 * gam : 0.5 - 0.5 * gam;
    v = zadd(v, zsc(int_ne<RF>(n, part, gam, t, q, rq), w));
  }
  return zsc(v, q.w[n]);
}
__device__ inline void psi_lim_e(int idf, double& a, double& b) {
  if (idf == 1) {
    a = 0.0;
    b = PI / 3.0;
  } else if (idf == 2 || idf == 3) {
    a = PI / 3.0;
    b = PI / 2.0;
  } else if (idf == 4 || idf == 6) {
    a = PI / 2.0;
    b = PI;
  } else {
    a = 0.0;
    b = PI / 2.0;
  }
}
__device__ inline void eta_lim_e(int idf, double th, double& a, double& b) {
  double s, c;
  sincos(th, &s, &c);
  if (idf == 1) {
    a = 0.0;
    b = atan(s + S3 * c);
  } else if (idf == 2) {
    a = atan(s - S3 * c);
    b = atan(s + S3 * c);
  } else if (idf == 3 || idf == 4) {
    a = 0.0;
    b = atan(s - S3 * c);
  } else if (idf == 5) {
    a = atan(s + S3 * c);
    b = 0.5 * PI;
  } else {
    a = atan(s - S3 * c);
    b = 0.5 * PI;
  }
}
// One weak item: a triangle pair and its integral type.
enum { W_S = 0, W_E = 1, W_VS = 2, W_VR = 3 };
struct WItem {
  int type;
  Tri6 t;
};

__device__ inline Z block_sum(Z v, Z* sh) {
  for (int o = 16; o > 0; o >>= 1) {
    v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
  }
  const int wid = threadIdx.x / 32, lane = threadIdx.x % 32, nw = blockDim.x / 32;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  Z s{0, 0};
  if (threadIdx.x == 0)
    for (int k = 0; k < nw; ++k) s = zadd(s, sh[k]);  // fixed order
  return s;
}

// One block per (item, outer index of its sum) of the items of one kind (0:
// self, 1: edge, 2: vertex), item0 .. item0 + nitems - 1 with `outer` blocks
// each; partial[item][outer].
//
// Bound by FP64 arithmetic (the pipe at 55 to 63% of its peak) and the latency of
// its chains at 16 warps or fewer per SM: 906 M kernel values for three directions
// at intOrd 32, a third of that where the sides are equal.  All items of a kind in one
// launch: an item alone has 32 (vertex) to 768 blocks, and one after the other
// they left most SMs idle.  A kernel per kind, with the pair's geometry in
// shared memory, holds 76 to 128 registers (one kernel for all: 152, one block
// per SM, 2.11 ms).  Cubic cell at intOrd 32: 108 launches of 49.7 ms in all,
// now 0.31 (self) + 0.78 (edge) + 0.25 ms (vertex).
template <int KIND, bool RF>
__global__ void __launch_bounds__(256, 2) k_weak(const WItem* __restrict__ items, int item0, int n_outer, int stride,
                                                 const Consts* __restrict__ qp, Z* __restrict__ partial) {
  __shared__ Consts q;
  __shared__ Z sh[8];
  __shared__ Tri6 t;
  __shared__ double geo[5][3];
  __shared__ int type;
  const int item = item0 + (int)blockIdx.x / n_outer, outer = (int)blockIdx.x % n_outer;
  for (int i = threadIdx.x; i < (int)(sizeof(Consts) / sizeof(double)); i += blockDim.x)
    reinterpret_cast<double*>(&q)[i] = reinterpret_cast<const double*>(qp)[i];
  if (threadIdx.x == 0) {
    t = items[item].t;
    type = items[item].type;
  }
  __syncthreads();
  const int n = q.ord;
  const RealF rq{q.f.x, 1.0 / (4.0 * PI * q.f.x * q.f.x)};
  Z acc{0, 0};
  double scale = 1.0;
  if constexpr (KIND == 0) {
    // outer = (k*8 + idf-1)*3 + dir-1 ; inner (it, nn)
    const int dir = outer % 3 + 1, idf = (outer / 3) % 8 + 1, k = outer / 24;
    double pa, pb, ea, eb;
    psi_lim_s(idf, pa, pb);
    const double th = thf(pa, pb, q.x[k]);
    eta_lim_s(idf, th, ea, eb);
    double s1, c1;
    sincos(th, &s1, &c1);
    const double wl = s_dir(tri_aff(t.r), s1, c1, dir);
    for (int p = threadIdx.x; p < n * n; p += blockDim.x) {
      const int it = p / n, nn = p % n;
      const double thB = thf(ea, eb, q.x[it]);
      acc = zadd(acc, zsc(n_s_term<RF>(idf, s1, c1, wl, thB, nn, q, rq), q.w[it]));
    }
    scale = 0.25 * q.w[k] * (pb - pa) * (eb - ea) * s1;
  } else if constexpr (KIND == 1) {
    const int idf = outer % 6 + 1, k = outer / 6;
    double pa, pb, ea, eb;
    psi_lim_e(idf, pa, pb);
    const double thB = thf(pa, pb, q.x[k]);
    eta_lim_e(idf, thB, ea, eb);
    EdgeGeo g;
    sincos(thB, &g.s1, &g.c1);  // the outer angle is the inner sums' th1
    if (threadIdx.x == 0) {
      const Aff a = tri_aff(t.r), b = tri_aff(t.r + 3);
      for (int d = 0; d < 3; ++d) {
        geo[0][d] = a.c[d] - b.c[d];
        geo[1][d] = a.e[d] + b.e[d];
        geo[2][d] = a.x[d];
        geo[3][d] = b.e[d] * g.c1;
        geo[4][d] = b.x[d] * g.s1;
      }
    }
    __syncthreads();
    g.v = geo;
    for (int p = threadIdx.x; p < n * n; p += blockDim.x) {
      const int it = p / n, nn = p % n;
      const double thA = thf(ea, eb, q.x[it]);
      sincos(thA, &g.sB, &g.cB);
      g.tB = g.sB / g.cB;
      acc = zadd(acc, zsc(n_e_term<RF>(idf, nn, g, q, rq), q.w[it] * g.cB));
    }
    scale = 0.25 * q.w[k] * (pb - pa) * (eb - ea);
  } else {
    const bool sng = type == W_VS;
    const int i3 = outer;
    // spxV! (src/glaIntSup.jl): points (tx c3 cA - 1, tx c3 sA) and (tx s3 cB
    // - 1, tx s3 sB) of the two triangles
    if (threadIdx.x == 0) {
      const Aff a = tri_aff(t.r), b = tri_aff(t.r + 3);
      for (int d = 0; d < 3; ++d) {
        geo[0][d] = t.r[0][d] - t.r[3][d];
        geo[1][d] = a.e[d];
        geo[2][d] = a.x[d];
        geo[3][d] = b.e[d];
        geo[4][d] = b.x[d];
      }
    }
    __syncthreads();
    for (int p = threadIdx.x; p < n * n; p += blockDim.x) {
      const int i2 = p / n, i1 = p % n;
      double sA, cA, sB, cB;
      sincos(thf(0.0, PI / 3.0, q.x[i1]), &sA, &cA);
      sincos(thf(0.0, PI / 3.0, q.x[i2]), &sB, &cB);
      const double LA = 2.0 * S3 / (sA + S3 * cA);
      const double LB = 2.0 * S3 / (sB + S3 * cB);
      const double at = atan(LB / LA);
      Z v[2];
      double s3[2], c3[2];
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        const double ang = h ? thf(at, PI / 2.0, q.x[i3]) : thf(0.0, at, q.x[i3]);
        double sn, cs;
        sincos(ang, &sn, &cs);
        const double len = h ? LB / sn : LA / cs;
        double B[3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
          B[d] = (geo[1][d] * cA + geo[2][d] * sA) * cs - (geo[3][d] * cB + geo[4][d] * sB) * sn;
        Z s{0, 0};
#pragma unroll 1
        for (int a = 0; a < n; ++a) {
          const double tx = thf(0.0, len, q.x[a]);
          const double x = geo[0][0] + B[0] * tx, y = geo[0][1] + B[1] * tx, w = geo[0][2] + B[2] * tx;
          s = zadd(s, zsc(ego_line<RF>(x * x + y * y + w * w, sng, q.f, rq), q.w[a] * (tx * tx * tx)));
        }
        v[h] = s;
        s3[h] = sn;
        c3[h] = cs;
      }
      const Z term = zadd(zsc(zsub(zsc(v[0], LA * s3[0]), zsc(v[1], LB * c3[1])), at), zsc(v[1], 0.5 * PI * LB * c3[1]));
      acc = zadd(acc, zsc(term, q.w[i1] * q.w[i2] * q.w[i3]));
    }
  }
  const Z s = block_sum(acc, sh);
  if (threadIdx.x == 0) partial[(size_t)item * stride + outer] = zsc(s, scale);
}

__device__ inline double cross_norm(const double a[3], const double b[3], const double c[3]) {
  const double u[3] = {b[0] - a[0], b[1] - a[1], b[2] - a[2]};
  const double v[3] = {c[0] - a[0], c[1] - a[1], c[2] - a[2]};
  const double x = u[1] * v[2] - u[2] * v[1], y = u[2] * v[0] - u[0] * v[2], z = u[0] * v[1] - u[1] * v[0];
  return sqrt(x * x + y * y + z * z);
}

// per item: fixed-order sum of its partials (one warp) times the Jacobian
// factor
__global__ void __launch_bounds__(32) k_weak_reduce(const WItem* __restrict__ items, int ord,
                                                    const Z* __restrict__ partial, int stride, Z* __restrict__ out) {
  const int i = blockIdx.x, ty = items[i].type, nout = ty == W_S ? 24 * ord : ty == W_E ? 6 * ord : ord;
  Z s{0, 0};
  for (int k = threadIdx.x; k < nout; k += 32) s = zadd(s, partial[(size_t)i * stride + k]);
  for (int o = 16; o > 0; o >>= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
  }
  if (threadIdx.x != 0) return;
  const Tri6& t = items[i].t;
  double jac;
  if (items[i].type == W_S) {
    const double u[3] = {t.r[0][0] - t.r[1][0], t.r[0][1] - t.r[1][1], t.r[0][2] - t.r[1][2]};
    const double v[3] = {t.r[2][0] - t.r[0][0], t.r[2][1] - t.r[0][1], t.r[2][2] - t.r[0][2]};
    const double x = u[1] * v[2] - u[2] * v[1], y = u[2] * v[0] - u[0] * v[2], z = u[0] * v[1] - u[1] * v[0];
    jac = (x * x + y * y + z * z) / 12.0;
  } else {
    jac = cross_norm(t.r[0], t.r[1], t.r[2]) * cross_norm(t.r[3], t.r[4], t.r[5]) / 12.0;
    if (items[i].type != W_E) jac *= PI * PI / 144.0;
  }
  out[i] = zsc(s, jac);
}

// closed-form static parts (src/glaInt.jl:410-488)
__device__ Z r_srf_slf(double la, double lb, Z f) {
  const double s1 = sqrt(la * la + lb * lb), s4 = sqrt(la * la + 4 * lb * lb);
  const double t =
      8 * la * la * la + 8 * lb * lb * lb - 8 * la * la * s1 - 8 * lb * lb * s1 -
      3 * la * la * lb *
          (2 * log(la) + 2 * log(la + lb - s1) + log(s1 - lb) - 5 * log(lb + s1) - 2 * log(lb - la + s1) -
           2 * log(la + 2 * lb - s4) + log(s4 - 2 * lb) + 2 * log(la - 2 * lb + s4) + log(2 * lb + s4) +
           2 * log(2 * lb - la + s4) - 2 * log(la + 2 * lb + s4)) +
      6 * la * lb * lb *
          (log(64.0) + 4 * log(lb) + 2 * log(s1 - la) + 3 * log(la + s1) - 3 * log(s4 - la) -
           3 * log(sqrt(la * la * la * la + 5 * la * la * lb * lb + 4 * lb * lb * lb * lb) + la * (s1 - la - s4)));
  return zsc(zdiv(Z{1.0, 0.0}, zsc(zmul(f, f), 48.0 * PI)), t);
}
__device__ Z r_srf_edg_crn(double la, double lb, double lc, Z f) {
  const double sab = sqrt(la * la + lb * lb + lc * lc), sbc = sqrt(lb * lb + lc * lc);
  const double t =
      8 * lb * lc * sbc - 8 * lb * lc * sab - 12 * la * la * la * atan(1.0 / (la * lc / (la * la + lb * lb - lb * sab))) +
      12 * la * la * la * atan(la / lc) - 12 * la * lc * lc * atan(la * lb / (lc * sab)) -
      12 * la * lb * lb * atan(la * lc / (lb * sab)) - 16 * la * la * la * atan(lb * lc / (la * sab)) +
      6 * lc * lc * lc * atanh(lb / sbc) - 6 * lc * (la * la + lc * lc) * atanh(lb / sab) -
      15 * la * la * lc * log(la * la + lc * lc) - lc * lc * lc * log(la * la + lc * lc) +
      2 * lc * lc * lc * log(lc / (lb + sbc)) + 6 * la * la * lc * log(sab - lb) + 24 * la * la * lc * log(sab + lb) +
      2 * lc * lc * lc * log(sab + lb) +
      6 * la * lb *
          (-2 * la * log(la * la + lb * lb) - lc * log((lb * lb + lc * lc) * (sab - la)) + 3 * lc * log(la + sab) +
           la * log(sab - lc) + 3 * la * log(sab + lc)) +
      2 * lb * lb * lb * (log((sab - lc) / (lc + sab)) + log(1 + (2 * lc * (lc + sbc)) / (lb * lb)));
  return zsc(zdiv(Z{1.0, 0.0}, zsc(zmul(f, f), 48.0 * PI)), t);
}
__device__ Z r_srf_edg_flt(double la, double lb, Z f) {
  const double s1 = sqrt(la * la + lb * lb), s4 = sqrt(la * la + 4 * lb * lb);
  const double p1 = -la * la * la + 2 * lb * lb * (3 * lb + s1 - 2 * s4) + la * la * (2 * s1 - s4);
  const double p2 =
      la * lb *
      (lb * (-62 * log(2.0) - 5 * log(-la + s1) + 4 * log(8 * lb * lb * (-la + s1)) - 33 * log(la + s1) +
             17 * log(-la + s4) - 24 * log(lb * (-la + s4)) + 57 * log(la + s4)) +
       4 * la *
           (-8 * asinh(lb / la) + 6 * asinh(2 * lb / la) + 6 * atanh(lb / s1) + 12 * log(la) - 13 * log(-lb + s1) +
            log((-lb + s1) / la) + log(la / (lb + s1)) - 7 * log(lb + s1) - 2 * log((lb + s1) / la) -
            3 * log(-(((lb + s1) * (2 * lb - s4)) / (la * la))) - 3 * log((-lb + s1) / (-2 * lb + s4)) +
            11 * log(-2 * lb + s4) - 3 * log((lb + s1) / (2 * lb + s4)) + log(2 * lb + s4) +
            9 * log((2 * lb + s4) / (lb + s1)) - 2 * log(la * la + 2 * lb * (lb - s1))));
  return zadd(zsc(zdiv(Z{1.0, 0.0}, zsc(zmul(f, f), 12.0 * PI)), p1), Z{p2 / (64.0 * PI), 0.0});
}

// wS[3], wE[9], wV[6] from the item sums (layout fixed by weak_items; uid[k]
// is the distinct item that item k equals) and the closed forms, scaled by
// inv = 1/prod(scl) (src/glaInt.jl:75-262, glaGen.jl:115-121).  One warp:
// lane k < 15 evaluates closed form k.
__global__ void __launch_bounds__(32) k_weak_combine(const Z* __restrict__ sums, const int* __restrict__ uid,
                                                     const double* __restrict__ scl, double inv, Z f,
                                                     Z* __restrict__ w /* 18 scaled */,
                                                     Z* __restrict__ wraw /* 18 unscaled */) {
  __shared__ Z cf[15];
  const double l[3] = {scl[0], scl[1], scl[2]};
  {
    // operands (axes) of the self (3), flat-edge (6) and corner (6) forms
    const signed char op[15][3] = {{1, 2, 0}, {0, 2, 0}, {0, 1, 0}, {2, 1, 0}, {1, 2, 0}, {0, 2, 0}, {2, 0, 0}, {1, 0, 0},
                                   {0, 1, 0}, {2, 1, 0}, {1, 2, 0}, {0, 2, 1}, {2, 1, 0}, {1, 2, 0}, {0, 2, 1}};
    const int k = threadIdx.x < 15 ? threadIdx.x : 14;
    double a[3];
    for (int d = 0; d < 3; ++d) a[d] = op[k][d] == 0 ? l[0] : op[k][d] == 1 ? l[1] : l[2];
    Z v;
    if (k < 3)
      v = r_srf_slf(a[0], a[1], f);
    else if (k < 9)
      v = r_srf_edg_flt(a[0], a[1], f);
    else
      v = r_srf_edg_crn(a[0], a[1], a[2], f);
    if (threadIdx.x < 15) cf[k] = v;
  }
  __syncwarp();
  if (threadIdx.x != 0) return;
  auto it = [&](int k) { return sums[uid[k]]; };
  auto sum4 = [&](int k) { return zadd(zadd(zadd(it(k), it(k + 1)), it(k + 2)), it(k + 3)); };
  // items: per dir d (0: dir 3, 1: dir 2, 2: dir 1) -> S block 8 items, E block 16, V block 12
  auto sdir = [&](int b) { return zsc(zadd(sum4(b * 36), sum4(b * 36 + 4)), 0.5); };  // wekSDir
  auto edir = [&](int b, int k) { return sum4(b * 36 + 8 + 4 * k); };                   // wekEDir value k
  auto vdir = [&](int b, int k) { return sum4(b * 36 + 24 + 4 * k); };                  // wekVDir value k
  Z r[18];
  for (int b = 0; b < 3; ++b) r[b] = zadd(sdir(b), cf[b]);
  const Z xyA = zadd(edir(0, 1), cf[9]), xzA = zadd(edir(0, 3), cf[10]);
  const Z yzA = zadd(edir(1, 1), cf[11]), xyB = zadd(edir(1, 3), cf[12]);
  const Z xzB = zadd(edir(2, 1), cf[13]), yzB = zadd(edir(2, 3), cf[14]);
  r[3] = zadd(edir(0, 0), cf[3]);  // xx along y
  r[4] = zadd(edir(0, 2), cf[4]);  // xx along z
  r[5] = zadd(edir(1, 2), cf[6]);  // yy along x
  r[6] = zadd(edir(1, 0), cf[5]);  // yy along z
  r[7] = zadd(edir(2, 0), cf[7]);  // zz along x
  r[8] = zadd(edir(2, 2), cf[8]);  // zz along y
  r[9] = zsc(zadd(xyA, xyB), 0.5);
  r[10] = zsc(zadd(xzA, xzB), 0.5);
  r[11] = zsc(zadd(yzA, yzB), 0.5);
  r[12] = vdir(0, 0);
  r[13] = vdir(1, 0);
  r[14] = vdir(2, 0);
  r[15] = zsc(zadd(vdir(0, 1), vdir(1, 2)), 0.5);
  r[16] = zsc(zadd(vdir(0, 2), vdir(2, 1)), 0.5);
  r[17] = zsc(zadd(vdir(1, 1), vdir(2, 2)), 0.5);
  for (int k = 0; k < 18; ++k) {
    wraw[k] = r[k];
    w[k] = zsc(r[k], inv);
  }
}

// ------------------------------------------------------- face-pair cubature
// Faces yzL yzU xzL xzU xyL xyU (cubFac, src/glaInt.jl:296-311); vertex 0,
// and the two edge vectors (v1 - v0, v3 - v0) used by cubVecAltAdp.
struct Faces {
  double o[6][3], a[6][3], b[6][3];
};
struct PairGeo {
  Faces tf, sf;
  double scale[36];  // srfScl (src/glaInt.jl:271-294)
  Z f;
};

// the 24 face pairs (0-based fp = 6*ft + fs) that feed the six stored
// components (xx, yy, zz, xy, xz, yz) of srfSum! (src/glaGen.jl:531-555)
#define GILA_PAIRS {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 14, 15, 16, 17, 20, 21, 22, 23, 28, 29, 34, 35}
__constant__ int c_pairs[24] = GILA_PAIRS;
__device__ constexpr int kPairs[24] = GILA_PAIRS;

// A pair's integrand at u in [0,1]^4: the vector between the two faces' points
// is o + u0 a0 + u1 a1 + u2 a2 + u3 a3 (source edges negated), the separation
// of the cells included.
struct PairLine {
  double o[3], a[4][3];
};
__device__ inline PairLine pair_line(const PairGeo& G, int fp, const double sep[3]) {
  const int ft = fp / 6, fs = fp % 6;
  PairLine l;
  for (int d = 0; d < 3; ++d) {
    l.o[d] = (G.tf.o[ft][d] - G.sf.o[fs][d]) + sep[d];
    l.a[0][d] = -G.sf.a[fs][d];
    l.a[1][d] = -G.sf.b[fs][d];
    l.a[2][d] = G.tf.a[ft][d];
    l.a[3][d] = G.tf.b[ft][d];
  }
  return l;
}
// sclEgo at a squared distance
template <bool RF>
__device__ __forceinline__ Z ego_at(double r2, Z f, RealF rq) {
  if constexpr (RF) return ego_line<true>(r2, false, f, rq);
  return scl_ego(sqrt(r2), f);
}

constexpr double GL2 = 0.35856858280031809199064515390793749545;  // sqrt(9/70)
constexpr double GL4 = 0.94868329805051379959966806332981556011;  // sqrt(9/10)
constexpr double GL5 = 0.68824720161168529772162873429362352512;  // sqrt(9/19)

// The 57-point Genz-Malik rule: points 0 (centre), 1 + 4 i + k (axis i; -l2,
// +l2, -l4, +l4), 17 .. 40 (two axes at +-l4), 41 .. 56 (all at +-l5), as
// offsets in units of the half-widths, and the degree-7 and -5 weights.
constexpr int kGm = 57;
__device__ inline void gm_point(int p, double off[4]) {
  off[0] = off[1] = off[2] = off[3] = 0.0;
  if (p == 0) return;
  if (p <= 16) {
    const int q = p - 1, i = q / 4, k = q % 4;
    const double v = (k < 2 ? GL2 : GL4) * ((k & 1) ? 1.0 : -1.0);
    for (int d = 0; d < 4; ++d)
      if (d == i) off[d] = v;
    return;
  }
  if (p <= 40) {
    const int q = p - 17, pr = q / 4;
    const int pi = pr < 3 ? 0 : pr < 5 ? 1 : 2, pk = pr < 3 ? pr + 1 : pr < 5 ? pr - 1 : 3;
    for (int d = 0; d < 4; ++d) {
      if (d == pi) off[d] = GL4 * ((q & 1) ? 1.0 : -1.0);
      if (d == pk) off[d] = GL4 * ((q & 2) ? 1.0 : -1.0);
    }
    return;
  }
  const int m = p - 41;
  for (int i = 0; i < 4; ++i) off[i] = GL5 * (((m >> i) & 1) ? 1.0 : -1.0);
}
// weights of the five classes of points (0: centre, 1: l2, 2: l4, 3: two
// axes, 4: all axes) for four dimensions
__device__ constexpr double kW7[5] = {(12824.0 - 9120.0 * 4 + 400.0 * 16) / 19683.0, 980.0 / 6561.0,
                                      (1820.0 - 400.0 * 4) / 19683.0, 200.0 / 19683.0, 6859.0 / 19683.0 / 16.0};
__device__ constexpr double kW5[5] = {(729.0 - 950.0 * 4 + 50.0 * 16) / 729.0, 245.0 / 486.0,
                                      (265.0 - 100.0 * 4) / 1458.0, 25.0 / 729.0, 0.0};
__device__ inline int gm_class(int p) { return p == 0 ? 0 : p <= 16 ? ((p - 1) % 4 < 2 ? 1 : 2) : p <= 40 ? 3 : 4; }

__device__ __forceinline__ bool cub_done(const double te[2], const double tv[2]) {
  for (int j = 0; j < 2; ++j)
    if (te[j] > CUB_ABSTOL && te[j] > fabs(tv[j]) * CUB_RELTOL) return false;
  return true;
}

// A region of the adaptive cubature and the axis to split; its key, the larger
// error, is kept in an array of its own, which the search for the largest runs
// over.
struct Region {
  double c[4], h[4], val[2], err[2];
  int split;
};
__device__ inline double region_key(const Region& r) { return r.err[0] > r.err[1] ? r.err[0] : r.err[1]; }

__device__ inline double warp_add(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One lane's share of the rule on a half-warp: four points, the l2 / l4
// points 1 .. 16 first, then 17 .. 56 and the centre.
struct GmLane {
  double off[4][4], w7[4], w5[4];
};
__device__ inline void gm_lane(int li, GmLane& g) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = 16 * q + li, p = k < 56 ? k + 1 : 0, c = gm_class(p);
    const bool on = k <= 56;
    gm_point(p, g.off[q]);
    g.w7[q] = on ? (c == 0 ? kW7[0] : c == 1 ? kW7[1] : c == 2 ? kW7[2] : c == 3 ? kW7[3] : kW7[4]) : 0.0;
    g.w5[q] = on ? (c == 0 ? kW5[0] : c == 1 ? kW5[1] : c == 2 ? kW5[2] : c == 3 ? kW5[3] : kW5[4]) : 0.0;
  }
}
__device__ __forceinline__ double half_add(double v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Genz-Malik rule on two regions by one warp, one per half-warp (Q: this
// half's, c and h set); every lane ends with its half's val, err and split.
template <bool RF>
__device__ __forceinline__ void gm_eval(const PairLine& L, Z f, RealF rq, const GmLane& g, Region& Q) {
  Z fv[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    double r2 = 0;
    double u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = Q.c[i] + g.off[q][i] * Q.h[i];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double v = L.o[d] + (u[0] * L.a[0][d] + u[1] * L.a[1][d]) + (u[2] * L.a[2][d] + u[3] * L.a[3][d]);
      r2 += v * v;
    }
    fv[q] = ego_at<RF>(r2, f, rq);
  }
  const double vol = (2.0 * Q.h[0]) * (2.0 * Q.h[1]) * ((2.0 * Q.h[2]) * (2.0 * Q.h[3]));
  const double ratio = (GL2 * GL2) / (GL4 * GL4);
  double dd = 0;
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    double s7 = 0, s5 = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double a = j ? fv[q].y : fv[q].x;
      s7 = g.w7[q] != 0.0 ? fma(g.w7[q], a, s7) : s7;  // the idle share's value may be infinite
      s5 = g.w5[q] != 0.0 ? fma(g.w5[q], a, s5) : s5;
    }
    s7 = half_add(s7);
    s5 = half_add(s5);
    Q.val[j] = vol * s7;
    Q.err[j] = fabs(vol * s5 - vol * s7);
    // fourth difference of axis i on lane 4 i (points -l2, +l2, -l4, +l4)
    const double a = j ? fv[0].y : fv[0].x, z = j ? fv[3].y : fv[3].x;
    const double f0 = __shfl_sync(0xffffffffu, z, 8, 16);
    const double fb = __shfl_down_sync(0xffffffffu, a, 1), fc = __shfl_down_sync(0xffffffffu, a, 2),
                 fd = __shfl_down_sync(0xffffffffu, a, 3);
    dd += fabs(a + fb - 2 * f0 - ratio * (fc + fd - 2 * f0));
  }
  int sd = 0;
  double md = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double d = __shfl_sync(0xffffffffu, dd, 4 * i, 16);
    if (d > md) {
      md = d;
      sd = i;
    }
  }
  Q.split = sd;
}

// hcubature(2, f, 0, 1; reltol, abstol, INDIVIDUAL) with the warp, its regions
// in H and their keys in K (capacity cap): 1 done (out set on every lane), 0 the
// capacity is exceeded.  The region of the largest error is split; the search
// over the keys is a warp reduction (ties: the older region).
template <bool RF>
__device__ int cubature(const PairLine& L, Z f, RealF rq, const GmLane& g, Region* H, double* K, int cap,
                        double out[2]) {
  const int lane = threadIdx.x & 31;
  const bool up = lane >= 16;  // the half that takes the upper child
  Region R;
#pragma unroll
  for (int i = 0; i < 4; ++i) R.c[i] = R.h[i] = 0.5;
  gm_eval<RF>(L, f, rq, g, R);
  double tv[2] = {R.val[0], R.val[1]}, te[2] = {R.err[0], R.err[1]};
  if (cub_done(te, tv)) {
    out[0] = tv[0];
    out[1] = tv[1];
    return 1;
  }
  if (lane == 0) {
    H[0] = R;
    K[0] = region_key(R);
  }
  __syncwarp();
  int n = 1;
  for (;;) {
    if (n + 1 > cap) return 0;
    double bk = -1.0;
    int bi = 0x7fffffff;
    for (int i = lane; i < n; i += 32) {
      const double k = K[i];
      if (k > bk) {
        bk = k;
        bi = i;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double k = __shfl_xor_sync(0xffffffffu, bk, o);
      const int i = __shfl_xor_sync(0xffffffffu, bi, o);
      if (k > bk || (k == bk && i < bi)) {
        bk = k;
        bi = i;
      }
    }
    if (bi >= n) bi = 0;  // every key NaN
    R = H[bi];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      tv[j] -= R.val[j];
      te[j] -= R.err[j];
    }
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      const double h = d == R.split ? R.h[d] * 0.5 : R.h[d];
      R.c[d] = d == R.split ? (up ? R.c[d] + h : R.c[d] - h) : R.c[d];
      R.h[d] = h;
    }
    gm_eval<RF>(L, f, rq, g, R);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      tv[j] += R.val[j] + __shfl_xor_sync(0xffffffffu, R.val[j], 16);
      te[j] += R.err[j] + __shfl_xor_sync(0xffffffffu, R.err[j], 16);
    }
    __syncwarp();
    if ((lane & 15) == 0) {
      const int at = up ? n : bi;
      H[at] = R;
      K[at] = region_key(R);
    }
    ++n;
    __syncwarp();
    if (cub_done(te, tv)) break;
  }
  double s0 = 0, s1 = 0;
  for (int i = lane; i < n; i += 32) {
    s0 += H[i].val[0];
    s1 += H[i].val[1];
  }
  out[0] = warp_add(s0);
  out[1] = warp_add(s1);
  __syncwarp();
  return 1;
}

// srfSum! restricted to the six stored components, accumulated in the
// reference's order; s = the 36 srfMat values (unused entries zero)
__device__ inline void srf_sum6(const Z* s_, Z out[6]) {
  const Z* s = s_ - 1;  // 1-based like srfMat
  // xx = s15 - s16 - s21 + s22 + s29 - s30 - s35 + s36
  out[0] = zadd(zsub(zsub(zadd(zadd(zsub(zsub(s[15], s[16]), s[21]), s[22]), s[29]), s[30]), s[35]), s[36]);
  // yy = s1 - s2 - s7 + s8 + s29 - s30 - s35 + s36
  out[1] = zadd(zsub(zsub(zadd(zadd(zsub(zsub(s[1], s[2]), s[7]), s[8]), s[29]), s[30]), s[35]), s[36]);
  // zz = s1 - s2 - s7 + s8 + s15 - s16 - s21 + s22
  out[2] = zadd(zsub(zsub(zadd(zadd(zsub(zsub(s[1], s[2]), s[7]), s[8]), s[15]), s[16]), s[21]), s[22]);
  // xy = -s3 + s4 + s9 - s10
  out[3] = zsub(zadd(zadd(Z{-s[3].x, -s[3].y}, s[4]), s[9]), s[10]);
  // xz = -s5 + s6 + s11 - s12
  out[4] = zsub(zadd(zadd(Z{-s[5].x, -s[5].y}, s[6]), s[11]), s[12]);
  // yz = -s17 + s18 + s23 - s24
  out[5] = zsub(zadd(zadd(Z{-s[17].x, -s[17].y}, s[18]), s[23]), s[24]);
}

// Far offsets of a chunk of items [item0, item0 + n):
//   mode 0 (self):  offset (ix,iy,iz) of the Toeplitz field, skipped when all
//                   indices <= 1 (near); sep = index * pitch;
//   mode 1 (ext):   circulant index; split indices zero; touching offsets are
//                   left to the contact kernel; sep from the grdSel tables.
// Three steps: k_far_first evaluates the rule once on the whole domain of
// every face pair (nearly all pairs of separated cells converge there) and
// lists the others; k_adapt refines the listed ones; k_far_sum combines the
// records of the items that had any.
struct FarParams {
  int mode;
  int n[3];                 // extents of the output field
  const double* sep[3];     // per-axis separation tables
  int split[3];             // ext: 0-based split index (trg cel), self: -1
  double touch[3];          // ext contact threshold per axis (cntTol + (sT+sS)/2), or -1
  Z* out;                   // [6][n2][n1][n0]
};
// a face pair to refine: its 24 values' record and place in it
struct Unit {
  int rec, pair;
};
// an item with listed pairs: the output element (near and far offsets of one
// field) and its separation
struct Rec {
  int64_t o;
  double sep[3];
};
// Work lists of one build: counters [0] records, [1] units, [2] next unit of
// k_adapt's first pass, [3] deferred units, [4] next deferred unit, [5], [6]
// the same for the last pass.
struct Lists {
  Rec* rec;
  Z* val;      // [rec][24] scaled pair values
  Unit* unit;
  Unit* ovf[2];
  int* cnt;
};

// Items one block takes at a time.  A thread runs the 57 points of one
// (item, pair) by itself -- no reductions, and the pairs of a warp differ only
// in the table column and the separation they read.  The FP64 pipe is at 46% of
// its peak at a quarter of the warps; the warp-per-offset form before it spent
// its time in the serial sums and the global-memory heap of its one active lane
// (32^3 cells: 9.0 ms, now 0.26 ms and 0.13 ms of k_adapt).
constexpr int kFarItems = 32;
template <bool RF>
__global__ void __launch_bounds__(256) k_far_first(const FarParams p, const PairGeo* __restrict__ gp, int64_t item0,
                                                   int64_t nitems, const Lists L) {
  __shared__ double D[3][kGm][24];  // face-to-face vectors of the points at separation 0
  __shared__ Z srf[kFarItems][24];
  __shared__ double sepi[kFarItems][3];
  __shared__ double scale[24];
  __shared__ int rec[kFarItems], state[kFarItems];  // 0 evaluate, 1 nothing to do
  __shared__ unsigned open[kFarItems];              // pairs that need refining
  for (int q = threadIdx.x; q < kGm * 24; q += blockDim.x) {
    const int pt = q / 24, k = q % 24;
    double off[4];
    gm_point(pt, off);
    const double zero[3] = {0, 0, 0};
    const PairLine l = pair_line(*gp, c_pairs[k], zero);
    for (int d = 0; d < 3; ++d) {
      double v = l.o[d];
      for (int i = 0; i < 4; ++i) v += (0.5 + off[i] * 0.5) * l.a[i][d];
      D[d][pt][k] = v;
    }
  }
  if (threadIdx.x < 24) scale[threadIdx.x] = gp->scale[c_pairs[threadIdx.x]];
  const Z f = gp->f;
  const RealF rq{f.x, 1.0 / (4.0 * PI * f.x * f.x)};
  const int64_t plane = (int64_t)p.n[0] * p.n[1], vol = plane * p.n[2];
  for (int64_t b0 = (int64_t)blockIdx.x * kFarItems; b0 < nitems; b0 += (int64_t)gridDim.x * kFarItems) {
    __syncthreads();
    if (threadIdx.x < kFarItems) {
      const int64_t item = item0 + b0 + threadIdx.x;
      int st = 1;
      if (b0 + threadIdx.x < nitems) {
        const int id[3] = {(int)(item % p.n[0]), (int)((item / p.n[0]) % p.n[1]), (int)(item / plane)};
        bool skip = false, zero = false;
        double sep[3];
        for (int d = 0; d < 3; ++d) sepi[threadIdx.x][d] = sep[d] = p.sep[d][id[d]];
        if (p.mode == 0) {
          skip = !(id[0] > 1 || id[1] > 1 || id[2] > 1);
        } else {
          for (int d = 0; d < 3; ++d) zero |= id[d] == p.split[d];
          if (!zero && p.touch[0] > 0) {
            bool t = true;
            for (int d = 0; d < 3; ++d) t &= fabs(sep[d]) < p.touch[d];
            skip = t;
          }
        }
        if (!skip && zero)
          for (int c = 0; c < 6; ++c) p.out[c * vol + item] = Z{0, 0};
        st = skip || zero;
      }
      state[threadIdx.x] = st;
      open[threadIdx.x] = 0;
    }
    __syncthreads();
    for (int u = threadIdx.x; u < kFarItems * 24; u += blockDim.x) {
      const int it = u / 24, k = u % 24;
      if (state[it]) continue;
      const double sx = sepi[it][0], sy = sepi[it][1], sz = sepi[it][2];
      auto at = [&](int pt) -> Z {
        const double x = D[0][pt][k] + sx, y = D[1][pt][k] + sy, z = D[2][pt][k] + sz;
        return ego_at<RF>(x * x + y * y + z * z, f, rq);
      };
      const Z s0 = at(0);
      Z s1{0, 0}, s2{0, 0}, s3{0, 0}, s4{0, 0};
#pragma unroll 1
      for (int i = 0; i < 4; ++i) {
        s1 = zadd(s1, zadd(at(1 + 4 * i), at(2 + 4 * i)));
        s2 = zadd(s2, zadd(at(3 + 4 * i), at(4 + 4 * i)));
      }
#pragma unroll 2
      for (int pt = 17; pt <= 40; ++pt) s3 = zadd(s3, at(pt));
#pragma unroll 2
      for (int pt = 41; pt < kGm; ++pt) s4 = zadd(s4, at(pt));
      auto sum = [&](const double* w) -> Z {
        return Z{w[0] * s0.x + w[1] * s1.x + w[2] * s2.x + w[3] * s3.x + w[4] * s4.x,
                 w[0] * s0.y + w[1] * s1.y + w[2] * s2.y + w[3] * s3.y + w[4] * s4.y};
      };
      const Z v7 = sum(kW7), v5 = sum(kW5);
      const double tv[2] = {v7.x, v7.y}, te[2] = {fabs(v5.x - v7.x), fabs(v5.y - v7.y)};
      srf[it][k] = zsc(v7, scale[k]);
      if (!cub_done(te, tv)) atomicOr(&open[it], 1u << k);
    }
    __syncthreads();
    if (threadIdx.x < kFarItems && !state[threadIdx.x]) {
      const int it = threadIdx.x;
      const int64_t o = item0 + b0 + it;
      if (open[it]) {
        const int r = atomicAdd(L.cnt, 1);
        rec[it] = r;
        L.rec[r] = Rec{o, {sepi[it][0], sepi[it][1], sepi[it][2]}};
        int u = atomicAdd(L.cnt + 1, __popc(open[it]));
        for (int k = 0; k < 24; ++k)
          if (open[it] >> k & 1) L.unit[u++] = Unit{r, k};
      } else {
        Z s[36], c6[6];
        for (int k = 0; k < 36; ++k) s[k] = Z{0, 0};
        for (int k = 0; k < 24; ++k) s[kPairs[k]] = srf[it][k];
        srf_sum6(s, c6);
        for (int c = 0; c < 6; ++c) p.out[c * vol + o] = c6[c];
      }
    }
    __syncthreads();
    for (int u = threadIdx.x; u < kFarItems * 24; u += blockDim.x) {
      const int it = u / 24, k = u % 24;
      if (!state[it] && open[it] && !(open[it] >> k & 1)) L.val[(int64_t)rec[it] * 24 + k] = srf[it][k];
    }
  }
}

// The listed face pairs, one warp each, over a work counter.  pass 0: regions
// in shared memory (kCap0 each, four warps a block); a pair that needs more
// goes to the next list.  pass 1: that list, kCap1 regions in shared memory,
// one warp a block; pass 2: kCap2 in global memory, past which the build
// fails.  A pair is a chain of dependent rule evaluations, so its latency
// counts (near pairs of a cubic cell: 0.81 ms with pass 1's regions in global
// memory and the two child regions one after the other, 0.53 ms with a
// half-warp each; 15.3 ms with all 36 pairs of an offset on one warp).  Cubic
// cells of 1/28 to 1/36 stay below 400 regions; flat and long ones reach pass
// 2 (cells 1/32 x 1/32 x 1/96: 31 pairs, up to 13,763 regions), whose eight
// warps take a few rounds: build at 16^3 614 -> 74 ms, 1/32 x 1/32 x 1/64 at
// 32^3 229 -> 14.5 ms, 1/16 x 1/128 x 1/128 at 16^3 419 -> 47 ms (all 36 pairs
// of an offset in turn, with a heap, before).
constexpr int kCap0 = 48, kCap1 = 512, kCap2 = 16384;
constexpr int kRegBytes = sizeof(Region) + sizeof(double);
template <bool RF>
__global__ void k_adapt(const PairGeo* __restrict__ gp, const Lists L, int pass, unsigned char* heap, int cap,
                        int* errflag) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  unsigned char* const own = heap ? heap + (size_t)(blockIdx.x * nw + wid) * cap * kRegBytes
                                  : smem_raw + (size_t)wid * cap * kRegBytes;
  Region* const H = reinterpret_cast<Region*>(own);
  double* const K = reinterpret_cast<double*>(H + cap);
  const Unit* const list = pass == 0 ? L.unit : L.ovf[pass - 1];
  const int n = L.cnt[1 + 2 * pass];
  const Z f = gp->f;
  const RealF rq{f.x, 1.0 / (4.0 * PI * f.x * f.x)};
  GmLane g;
  gm_lane(lane & 15, g);
  for (;;) {
    int k = 0;
    if (lane == 0) k = atomicAdd(L.cnt + 2 + 2 * pass, 1);
    k = __shfl_sync(0xffffffffu, k, 0);
    if (k >= n) break;
    const Unit u = list[k];
    const int fp = c_pairs[u.pair];
    const PairLine pl = pair_line(*gp, fp, L.rec[u.rec].sep);
    double v[2];
    const int ok = cubature<RF>(pl, f, rq, g, H, K, cap, v);
    if (lane == 0) {
      if (ok)
        L.val[(int64_t)u.rec * 24 + u.pair] = zsc(Z{v[0], v[1]}, gp->scale[fp]);
      else if (pass < 2)
        L.ovf[pass][atomicAdd(L.cnt + 3 + 2 * pass, 1)] = u;
      else
        atomicOr(errflag, 1);
    }
    __syncwarp();
  }
}

// the six components of every record
__global__ void k_far_sum(const FarParams p, const Lists L) {
  const int n = L.cnt[0];
  const int64_t vol = (int64_t)p.n[0] * p.n[1] * p.n[2];
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
    Z s[36], c6[6];
    for (int k = 0; k < 36; ++k) s[k] = Z{0, 0};
    for (int k = 0; k < 24; ++k) s[kPairs[k]] = L.val[(int64_t)r * 24 + k];
    srf_sum6(s, c6);
    for (int c = 0; c < 6; ++c) p.out[c * vol + L.rec[r].o] = c6[c];
  }
}

// Near offsets of a self operator (egoFunSng!, src/glaGen.jl:350-528): offsets
// (px, py, pz) in {0,1}^3 within the volume, one block each; the corrected
// pairs from the weak values, the others listed for k_adapt.  Pairs that feed
// none of the six components are not evaluated.
__constant__ signed char c_sng_cor[8][6][6];
__constant__ signed char c_sng_mask[8][6][6];

struct NearParams {
  int n[3];
  int cases[8];  // egoFunSng! case per offset (x fastest), -1 = every pair by cubature
  const double* sep[3];
  const Z* weak;  // 18 scaled weak values
};

__global__ void __launch_bounds__(32) k_near_list(const NearParams p, const Lists L) {
  __shared__ int rec;
  const int b = blockIdx.x;
  const int px = b & 1, py = (b >> 1) & 1, pz = (b >> 2) & 1;
  if (px >= p.n[0] || py >= p.n[1] || pz >= p.n[2]) return;
  if (threadIdx.x == 0) {
    rec = atomicAdd(L.cnt, 1);
    L.rec[rec] = Rec{((int64_t)pz * p.n[1] + py) * p.n[0] + px, {p.sep[0][px], p.sep[1][py], p.sep[2][pz]}};
  }
  __syncwarp();
  const int k = threadIdx.x, cs = p.cases[b];
  if (k >= 24) return;
  const int a = c_pairs[k] / 6, c = c_pairs[k] % 6;
  if (cs >= 0 && c_sng_mask[cs][a][c]) {
    const int code = c_sng_cor[cs][a][c];
    L.val[(int64_t)rec * 24 + k] = code == 0   ? Z{0, 0}
                                   : code < 10 ? p.weak[code - 1]
                                   : code < 20 ? p.weak[3 + code - 11]
                                               : p.weak[12 + code - 21];
  } else {
    L.unit[atomicAdd(L.cnt + 1, 1)] = Unit{rec, k};
  }
}

// identity (src/glaGen.jl:128-130) and egoToeCrc! (src/glaGen.jl:143-163):
// toe [6][N] -> circulant crc [6][2N]; off-diagonal signs flip on mirrored axes
__global__ void k_embed(const Z* __restrict__ toe, int nx, int ny, int nz, Z idsub, Z* __restrict__ crc) {
  const int64_t Px = 2 * nx, Py = 2 * ny, Pz = 2 * nz, vol = Px * Py * Pz, tv = (int64_t)nx * ny * nz;
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < vol; o += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(o % Px), y = (int)((o / Px) % Py), z = (int)(o / (Px * Py));
    const bool zero = x == nx || y == ny || z == nz;
    const int sx = x < nx ? x : 2 * nx - x, sy = y < ny ? y : 2 * ny - y, sz = z < nz ? z : 2 * nz - z;
    const double fx = x < nx ? 1.0 : -1.0, fy = y < ny ? 1.0 : -1.0, fz = z < nz ? 1.0 : -1.0;
    const int64_t ti = ((int64_t)sz * ny + sy) * nx + sx;
    // components xx, yy, zz, xy, xz, yz
    const double sg[6] = {1.0, 1.0, 1.0, fx * fy, fx * fz, fy * fz};
    for (int c = 0; c < 6; ++c) {
      Z v = zero ? Z{0, 0} : zsc(toe[c * tv + ti], sg[c]);
      if (!zero && ti == 0 && c < 3) v = zsub(v, idsub);
      crc[c * vol + o] = v;
    }
  }
}

// egoCntOut! (src/glaGen.jl:250-306) for the touching offsets of an external
// circulant, from the contact self circulant ccnt [6][2*cc] of the contact
// volume (genCntVol, src/glaGen.jl:308-318)
struct CntParams {
  int n[3];       // circulant extents
  int split[3];
  const double* sep[3];
  double touch[3];
  double cscl[3];  // contact cell size
  int sspan[3], tspan[3];
  int cc[3];       // contact volume cells
  const Z* ccnt;
  Z* out;
};
__global__ void k_contact(const CntParams p) {
  const int64_t vol = (int64_t)p.n[0] * p.n[1] * p.n[2];
  const int64_t Pc[3] = {2LL * p.cc[0], 2LL * p.cc[1], 2LL * p.cc[2]};
  const int64_t cvol = Pc[0] * Pc[1] * Pc[2];
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < vol; o += (int64_t)gridDim.x * blockDim.x) {
    const int id[3] = {(int)(o % p.n[0]), (int)((o / p.n[0]) % p.n[1]), (int)(o / ((int64_t)p.n[0] * p.n[1]))};
    bool split = false, touch = true;
    double sep[3];
    for (int d = 0; d < 3; ++d) {
      split |= id[d] == p.split[d];
      sep[d] = p.sep[d][id[d]];
      touch &= fabs(sep[d]) < p.touch[d];
    }
    if (split || !touch) continue;
    int64_t sL[3], sU[3], tL[3], tU[3];
    for (int d = 0; d < 3; ++d) {
      const double span = sep[d] / p.cscl[d];
      sL[d] = 1;
      sU[d] = p.sspan[d];
      tL[d] = (int64_t)nearbyint(span + p.sspan[d] / 2.0 - p.tspan[d] / 2.0) + 1;
      tU[d] = (int64_t)nearbyint(span + p.sspan[d] / 2.0 + p.tspan[d] / 2.0);
      if (tL[d] < 1) {
        const int64_t sh = (tL[d] < 0 ? -tL[d] : tL[d]) + 1;
        sL[d] += sh;
        sU[d] += sh;
        tU[d] += sh;
        tL[d] += sh;
      }
    }
    Z acc[6] = {};
    for (int64_t a = sL[2]; a <= sU[2]; ++a)
      for (int64_t b = sL[1]; b <= sU[1]; ++b)
        for (int64_t c = sL[0]; c <= sU[0]; ++c)
          for (int64_t aa = tL[2]; aa <= tU[2]; ++aa)
            for (int64_t bb = tL[1]; bb <= tU[1]; ++bb)
              for (int64_t cc = tL[0]; cc <= tU[0]; ++cc) {
                const int64_t t3[3] = {cc, bb, aa}, s3[3] = {c, b, a};
                int64_t ci[3];
                bool inb = true;
                for (int d = 0; d < 3; ++d) {
                  const int64_t v = t3[d] - s3[d];
                  ci[d] = v + (v < 0 ? 2LL * p.cc[d] : 0);
                  inb = inb && ci[d] >= 0 && ci[d] < Pc[d];
                }
                if (!inb) continue;
                const int64_t q = (ci[2] * Pc[1] + ci[1]) * Pc[0] + ci[0];
                for (int k = 0; k < 6; ++k) acc[k] = zadd(acc[k], p.ccnt[k * cvol + q]);
              }
    const double tot = (double)((tU[2] - tL[2] + 1) * (tU[1] - tL[1] + 1) * (tU[0] - tL[0] + 1));
    for (int k = 0; k < 6; ++k) p.out[k * vol + o] = Z{acc[k].x / tot, acc[k].y / tot};
  }
}

// ----------------------------------------------- FP64 3-D FFT of the circulant
// In-place forward FFT of `lines` lines of length P along one axis: element
// stride es, lines in tiles of TX contiguous (es > 1) or rows (es == 1).
__global__ void __launch_bounds__(512) k_fft_axis(double2* __restrict__ data, const AxisPlan* __restrict__ pl, int P,
                                                   const double2* __restrict__ tw, int64_t es, int64_t group_stride,
                                                   int TX, int64_t nlines_in_group, FDiv md) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* sm = reinterpret_cast<double2*>(smem_raw);
  // block -> (group g, tile t): lines l = t*TX + u, u < TX, of group g.  Line
  // l holds element i at base[l + i*es] (es > 1: lines contiguous) or at
  // base[l*P + i] (es == 1: rows).  Shared memory is [i][u].
  const int64_t ntiles = (nlines_in_group + TX - 1) / TX;
  const int64_t g = blockIdx.x / ntiles, t = blockIdx.x % ntiles;
  const int64_t l0 = t * TX;
  const int tmax = (int)((nlines_in_group - l0) < TX ? (nlines_in_group - l0) : TX);
  double2* base = data + g * group_stride;
  for (int q = threadIdx.x; q < TX * P; q += blockDim.x) {
    int i, u;
    if (es == 1) {  // coalesced along the row
      u = q / P;
      i = q - u * P;
    } else {
      i = (int)md.div((uint32_t)q);
      u = q - i * TX;
    }
    if (u < tmax) sm[i * TX + u] = es == 1 ? base[(l0 + u) * P + i] : base[l0 + u + (int64_t)i * es];
  }
  __syncthreads();
  auto lds = [=](int u, int i) -> double2 { return sm[i * TX + u]; };
  auto sts = [=](int u, int i, double2 v) { sm[i * TX + u] = v; };
  fft_run<double2, 4, false, true, true>(pl, TX, md, tw, lds, lds, sts, sts, true, true);
  for (int q = threadIdx.x; q < TX * P; q += blockDim.x) {
    int i, u;
    if (es == 1) {
      u = q / P;
      i = q - u * P;
    } else {
      i = (int)md.div((uint32_t)q);
      u = q - i * TX;
    }
    if (u < tmax) {
      const double2 v = sm[i * TX + u];
      if (es == 1)
        base[(l0 + u) * P + i] = v;
      else
        base[l0 + u + (int64_t)i * es] = v;
    }
  }
}

// parity-branch extraction + symmetric truncation + cast (src/glaMemSup.jl:138-156)
template <typename C>
__global__ void k_extract(const Z* __restrict__ crc, int Px, int Py, int Pz, int tx, int ty, int tz,
                          C* __restrict__ ker, int* __restrict__ nanflag) {
  const int64_t vol = (int64_t)Px * Py * Pz;
  const int64_t n = (int64_t)8 * tz * ty * tx * 6;
  for (int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; o < n; o += (int64_t)gridDim.x * blockDim.x) {
    int64_t q = o;  // o = ker_index(eo, iz, iy, c, ix, ...) = ((((py,pz) tz + iz) ty + iy) 6 + c) tx + ix) 2 + px
    const int px = (int)(q & 1);
    q >>= 1;
    const int ix = (int)(q % tx);
    q /= tx;
    const int c = (int)(q % 6);
    q /= 6;
    const int iy = (int)(q % ty);
    q /= ty;
    const int iz = (int)(q % tz);
    const int e = (int)(q / tz);
    const int py = (e >> 1) & 1, pz = e & 1;
    // the reference broadcasts a one-element branch slice over two entries
    const int hx = Px / 2 > 1 ? Px / 2 : 1, hy = Py / 2 > 1 ? Py / 2 : 1, hz = Pz / 2 > 1 ? Pz / 2 : 1;
    const int fx = 2 * (ix < hx ? ix : hx - 1) + px, fy = 2 * (iy < hy ? iy : hy - 1) + py,
              fz = 2 * (iz < hz ? iz : hz - 1) + pz;
    const Z v = crc[c * vol + ((int64_t)fz * Py + fy) * Px + fx];
    if (!isfinite(v.x) || !isfinite(v.y)) atomicOr(nanflag, 1);
    C r;
    r.x = (decltype(r.x))v.x;
    r.y = (decltype(r.y))v.y;
    ker[o] = r;
  }
}

}  // namespace kb
}  // namespace gila

// ======================================================================= host
namespace gila {
namespace kb {

// small rational helpers on top of Rat (exact grid arithmetic, converted to
// FP64 only at the end, as the reference's Rational -> Float64)
static Rat R(int64_t n, int64_t d = 1) { return rat(n, d); }
static Rat radd(Rat a, Rat b) { return rat(a.n * b.d + b.n * a.d, a.d * b.d); }
static Rat rsub(Rat a, Rat b) { return rat(a.n * b.d - b.n * a.d, a.d * b.d); }
static Rat rmul(Rat a, Rat b) { return rat(a.n * b.n, a.d * b.d); }
static Rat rdv(Rat a, Rat b) { return rat(a.n * b.d, a.d * b.n); }
static bool rlt(Rat a, Rat b) { return (__int128)a.n * b.d < (__int128)b.n * a.d; }
static bool rle(Rat a, Rat b) { return (__int128)a.n * b.d <= (__int128)b.n * a.d; }
static double rd(Rat a) { return (double)a.n / (double)a.d; }

struct HVol {  // GlaVol with start / stop of the grid (src/glaMem.jl:136-148)
  int64_t cel[3];
  Rat scl[3], org[3], grd[3], start[3], stop[3];
};
static HVol hvol(const Vol& v) {
  HVol h;
  for (int k = 0; k < 3; ++k) {
    h.cel[k] = v.cel[k];
    h.scl[k] = v.scl[k];
    h.org[k] = v.org[k];
    h.grd[k] = v.grd[k];
    const Rat half = R((v.cel[k] / 2) * 2 - (v.cel[k] % 2 == 0 ? 1 : 0), 2);
    const Rat brd = rmul(v.grd[k], half);
    h.start[k] = rsub(v.org[k], brd);
    h.stop[k] = radd(v.org[k], brd);
  }
  return h;
}

// Gauss-Legendre nodes (ascending) and weights by Newton iteration on P_n
static void gauss_legendre(int n, double* x, double* w) {
  for (int i = 0; i < n; ++i) {
    double z = cos(PI * (i + 0.75) / (n + 0.5)), dp = 0;
    for (int it = 0; it < 100; ++it) {
      double p0 = 1.0, p1 = 0.0;
      for (int k = 1; k <= n; ++k) {
        const double p2 = p1;
        p1 = p0;
        p0 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p2) / k;
      }
      dp = n * (z * p0 - p1) / (z * z - 1.0);
      const double dz = p0 / dp;
      z -= dz;
      if (fabs(dz) < 1e-16) break;
    }
    double p0 = 1.0, p1 = 0.0;
    for (int k = 1; k <= n; ++k) {
      const double p2 = p1;
      p1 = p0;
      p0 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p2) / k;
    }
    dp = n * (z * p0 - p1) / (z * z - 1.0);
    x[n - 1 - i] = z;
    w[n - 1 - i] = 2.0 / ((1.0 - z * z) * dp * dp);
  }
}

// faces of a cuboid (cubFac, src/glaInt.jl:296-311) as origin + two edges
static void faces(const Rat scl[3], Faces& F) {
  static const int sg[6][4][3] = {
      {{-1, -1, -1}, {-1, 1, -1}, {-1, 1, 1}, {-1, -1, 1}}, {{1, -1, -1}, {1, -1, 1}, {1, 1, 1}, {1, 1, -1}},
      {{-1, -1, -1}, {-1, -1, 1}, {1, -1, 1}, {1, -1, -1}}, {{-1, 1, -1}, {1, 1, -1}, {1, 1, 1}, {-1, 1, 1}},
      {{-1, -1, -1}, {1, -1, -1}, {1, 1, -1}, {-1, 1, -1}}, {{-1, -1, 1}, {-1, 1, 1}, {1, 1, 1}, {1, -1, 1}}};
  for (int f = 0; f < 6; ++f)
    for (int d = 0; d < 3; ++d) {
      double v[4];
      for (int k = 0; k < 4; ++k) v[k] = rd(R(sg[f][k][d] * scl[d].n, 2 * scl[d].d));
      F.o[f][d] = v[0];
      F.a[f][d] = v[1] - v[0];
      F.b[f][d] = v[3] - v[0];
    }
}
// srfScl (src/glaInt.jl:271-294)
static void srf_scales(const Rat sT[3], const Rat sS[3], double out[36]) {
  for (int a = 0; a < 6; ++a) {
    const Rat src = a < 2 ? rmul(sS[1], sS[2]) : a < 4 ? rmul(sS[0], sS[2]) : rmul(sS[0], sS[1]);
    for (int b = 0; b < 6; ++b) out[a * 6 + b] = rd(rdv(src, b < 2 ? sT[0] : b < 4 ? sT[1] : sT[2]));
  }
}

// The weak-integral items of wekS / wekE / wekV in the order k_weak_combine
// expects: per direction (3, 2, 1): 8 wekSDir items, 16 wekEDir, 12 wekVDir.
static std::vector<WItem> weak_items(const double scl[3]) {
  std::vector<WItem> v;
  for (int b = 0; b < 3; ++b) {
    const int dir = 3 - b;
    double gx, gy, gz;
    if (dir == 1) {
      gx = scl[0];
      gy = scl[1];
      gz = scl[2];
    } else if (dir == 2) {
      gx = scl[2];
      gy = scl[0];
      gz = scl[1];
    } else {
      gx = scl[1];
      gy = scl[2];
      gz = scl[0];
    }
    double P[19][3];
    int k = 1;
    for (int zz = 0; zz < 2; ++zz)
      for (int yy = 0; yy < 3; ++yy)
        for (int xx = 0; xx < 3; ++xx, ++k) {
          P[k][0] = xx * gx;
          P[k][1] = yy * gy;
          P[k][2] = zz * gz;
        }
    auto add = [&](int type, int a, int bb, int c, int d, int e, int f) {
      WItem it;
      it.type = type;
      const int id[6] = {a, bb, c, d, e, f};
      for (int q = 0; q < 6; ++q)
        for (int r = 0; r < 3; ++r) it.t.r[q][r] = P[id[q]][r];
      v.push_back(it);
    };
    // wekSDir (src/glaInt.jl:88-114)
    add(W_S, 1, 2, 5, 1, 2, 5);
    add(W_S, 1, 5, 4, 1, 5, 4);
    add(W_E, 1, 2, 5, 1, 5, 4);
    add(W_E, 1, 5, 4, 1, 2, 5);
    add(W_S, 4, 1, 2, 4, 1, 2);
    add(W_S, 4, 2, 5, 4, 2, 5);
    add(W_E, 4, 1, 2, 4, 2, 5);
    add(W_E, 4, 2, 5, 4, 1, 2);
    // wekEDir (src/glaInt.jl:165-206)
    add(W_E, 1, 2, 5, 2, 3, 5);
    add(W_VS, 1, 2, 5, 3, 6, 5);
    add(W_VS, 1, 5, 4, 2, 3, 5);
    add(W_VS, 1, 5, 4, 3, 6, 5);
    add(W_E, 1, 2, 5, 2, 11, 5);
    add(W_VS, 1, 2, 5, 11, 14, 5);
    add(W_VS, 1, 5, 4, 2, 11, 5);
    add(W_VS, 1, 5, 4, 11, 14, 5);
    add(W_VS, 1, 2, 5, 4, 5, 7);
    add(W_VS, 1, 2, 5, 5, 8, 7);
    add(W_E, 1, 5, 4, 4, 5, 7);
    add(W_VS, 1, 5, 4, 5, 8, 7);
    add(W_VS, 1, 2, 5, 4, 5, 13);
    add(W_VS, 1, 2, 5, 5, 14, 13);
    add(W_E, 1, 5, 4, 4, 5, 13);
    add(W_VS, 1, 5, 4, 5, 14, 13);
    // wekVDir (src/glaInt.jl:236-262)
    add(W_VR, 1, 2, 5, 5, 6, 9);
    add(W_VR, 1, 2, 5, 5, 9, 8);
    add(W_VR, 1, 5, 4, 5, 6, 9);
    add(W_VR, 1, 5, 4, 5, 9, 8);
    add(W_VR, 1, 2, 5, 5, 17, 14);
    add(W_VR, 1, 2, 5, 5, 8, 17);
    add(W_VR, 1, 5, 4, 5, 17, 14);
    add(W_VR, 1, 5, 4, 5, 8, 17);
    add(W_VR, 1, 2, 5, 5, 15, 14);
    add(W_VR, 1, 2, 5, 5, 6, 15);
    add(W_VR, 1, 5, 4, 5, 15, 14);
    add(W_VR, 1, 5, 4, 5, 6, 15);
  }
  return v;
}

// egoFunSng! tables (src/glaGen.jl:370-509): 0 none, 1..3 wS, 11..19 wE, 21..26 wV
static const signed char SNG_COR[8][6][6] = {
    {{1, 0, 17, 17, 18, 18}, {0, 1, 17, 17, 18, 18}, {17, 17, 2, 0, 19, 19},
     {17, 17, 0, 2, 19, 19}, {18, 18, 19, 19, 3, 0}, {18, 18, 19, 19, 0, 3}},
    {{0, 1, 17, 17, 18, 18}, {0, 0, 0, 0, 0, 0}, {0, 17, 13, 0, 26, 26},
     {0, 17, 0, 13, 26, 26}, {0, 18, 26, 26, 15, 0}, {0, 18, 26, 26, 0, 15}},
    {{0, 12, 24, 24, 0, 18}, {0, 0, 0, 0, 0, 0}, {0, 24, 22, 0, 0, 26},
     {0, 24, 0, 22, 0, 26}, {0, 18, 26, 26, 0, 15}, {0, 0, 0, 0, 0, 0}},
    {{12, 0, 24, 24, 0, 18}, {0, 12, 24, 24, 0, 18}, {24, 24, 14, 0, 0, 19},
     {24, 24, 0, 14, 0, 19}, {18, 18, 19, 19, 0, 3}, {0, 0, 0, 0, 0, 0}},
    {{11, 0, 0, 17, 25, 25}, {0, 11, 0, 17, 25, 25}, {17, 17, 0, 2, 19, 19},
     {0, 0, 0, 0, 0, 0}, {25, 25, 0, 19, 16, 0}, {25, 25, 0, 19, 0, 16}},
    {{0, 11, 0, 17, 25, 25}, {0, 0, 0, 0, 0, 0}, {0, 17, 0, 13, 26, 26},
     {0, 0, 0, 0, 0, 0}, {0, 25, 0, 26, 23, 0}, {0, 25, 0, 26, 0, 23}},
    {{21, 0, 0, 24, 0, 25}, {0, 21, 0, 24, 0, 25}, {24, 24, 0, 14, 0, 19},
     {0, 0, 0, 0, 0, 0}, {25, 25, 0, 19, 0, 16}, {0, 0, 0, 0, 0, 0}},
    {{0, 21, 0, 24, 0, 25}, {0, 0, 0, 0, 0, 0}, {0, 24, 0, 22, 0, 26},
     {0, 0, 0, 0, 0, 0}, {0, 25, 0, 26, 0, 23}, {0, 0, 0, 0, 0, 0}}};
static const signed char SNG_MASK[8][6][6] = {
    {{1, 0, 1, 1, 1, 1}, {0, 1, 1, 1, 1, 1}, {1, 1, 1, 0, 1, 1}, {1, 1, 0, 1, 1, 1}, {1, 1, 1, 1, 1, 0}, {1, 1, 1, 1, 0, 1}},
    {{0, 1, 1, 1, 1, 1}, {0, 0, 0, 0, 0, 0}, {0, 1, 1, 0, 1, 1}, {0, 1, 0, 1, 1, 1}, {0, 1, 1, 1, 1, 0}, {0, 1, 1, 1, 0, 1}},
    {{0, 1, 1, 1, 0, 1}, {0, 0, 0, 0, 0, 0}, {0, 1, 1, 0, 0, 1}, {0, 1, 0, 1, 0, 1}, {0, 1, 1, 1, 0, 1}, {0, 0, 0, 0, 0, 0}},
    {{1, 0, 1, 1, 0, 1}, {0, 1, 1, 1, 0, 1}, {1, 1, 1, 0, 0, 1}, {1, 1, 0, 1, 0, 1}, {1, 1, 1, 1, 0, 1}, {0, 0, 0, 0, 0, 0}},
    {{1, 0, 0, 1, 1, 1}, {0, 1, 0, 1, 1, 1}, {1, 1, 0, 1, 1, 1}, {0, 0, 0, 0, 0, 0}, {1, 1, 0, 1, 1, 0}, {1, 1, 0, 1, 0, 1}},
    {{0, 1, 0, 1, 1, 1}, {0, 0, 0, 0, 0, 0}, {0, 1, 0, 1, 1, 1}, {0, 0, 0, 0, 0, 0}, {0, 1, 0, 1, 1, 0}, {0, 1, 0, 1, 0, 1}},
    {{1, 0, 0, 1, 0, 1}, {0, 1, 0, 1, 0, 1}, {1, 1, 0, 1, 0, 1}, {0, 0, 0, 0, 0, 0}, {1, 1, 0, 1, 0, 1}, {0, 0, 0, 0, 0, 0}},
    {{0, 1, 0, 1, 0, 1}, {0, 0, 0, 0, 0, 0}, {0, 1, 0, 1, 0, 1}, {0, 0, 0, 0, 0, 0}, {0, 1, 0, 1, 0, 1}, {0, 0, 0, 0, 0, 0}}};

// egoFunSng! case of near offset (px, py, pz) in 1-based {1,2}^3, or -1
static int sng_case(int px, int py, int pz, const HVol& v) {
  const bool tx = !rlt(v.scl[0], v.grd[0]), ty = !rlt(v.scl[1], v.grd[1]), tz = !rlt(v.scl[2], v.grd[2]);
  if (px == 1 && py == 1 && pz == 1) return 0;
  if (px == 2 && py == 1 && pz == 1 && tx) return 1;
  if (px == 2 && py == 1 && pz == 2 && tx && tz) return 2;
  if (px == 1 && py == 1 && pz == 2 && tz) return 3;
  if (px == 1 && py == 2 && pz == 1 && ty) return 4;
  if (px == 2 && py == 2 && pz == 1 && tx && ty) return 5;
  if (px == 1 && py == 2 && pz == 2 && ty && tz) return 6;
  if (px == 2 && py == 2 && pz == 2 && tx && ty && tz) return 7;
  return -1;
}

// RAII for build scratch
struct DBuf {
  void* p = nullptr;
  ~DBuf() { cudaFree(p); }
};
#define KB_TRY(expr)                                              \
  do {                                                            \
    cudaError_t e__ = (expr);                                     \
    if (e__ != cudaSuccess) return ::gila::cuda_fail(e__, #expr); \
  } while (0)

// Scratch of one build: parts of a few large blocks.  Every device allocation
// above a megabyte costs 0.35 ms and its release 0.3 ms, and the build's dozen
// buffers took longer than its kernels (32^3 self operator: 6 of 9.6 ms).
struct Build {
  Ctx* ctx;
  cudaStream_t st;
  Z f;
  int ord;
  Consts* q_d = nullptr;  // in a block
  size_t block_bytes = size_t(32) << 20;  // of the next block, at least
  std::vector<DBuf*> keep;
  size_t off = 0, cap = 0;  // of the last block
  ~Build() {
    for (auto* b : keep) delete b;
  }
  struct Mark {
    size_t blocks, off, cap;
  };
  Mark mark() const { return Mark{keep.size(), off, cap}; }
  // gives back what was allocated after the mark (the stream is synchronised
  // first: kernels in flight may still use it)
  void release_to(const Mark& m) {
    cudaStreamSynchronize(st);
    while (keep.size() > m.blocks) {
      delete keep.back();
      keep.pop_back();
    }
    off = m.off;
    cap = m.cap;
  }
  template <typename T>
  gila_status alloc(T** out, size_t n) {
    const size_t bytes = (n * sizeof(T) + 16 + 255) / 256 * 256;
    if (off + bytes > cap) {
      DBuf* b = new DBuf;
      keep.push_back(b);
      off = cap = 0;
      const size_t want = std::max(bytes, block_bytes);
      KB_TRY(dev_malloc(&b->p, want));
      cap = want;
    }
    *out = reinterpret_cast<T*>(static_cast<unsigned char*>(keep.back()->p) + off);
    off += bytes;
    return GILA_OK;
  }
};

// the fast kernel values' condition (ego_line)
static bool real_freq(Z f) { return f.y == 0.0 && f.x != 0.0; }

// weak values (18, scaled by 1/prod(scl)) for a cell of size scl; the
// unscaled values go to raw_out when given
static gila_status weak_values(Build& B, const Rat sclr[3], Z* w_d, Z* raw_out = nullptr) {
  const double scl[3] = {rd(sclr[0]), rd(sclr[1]), rd(sclr[2])};
  const std::vector<WItem> all = weak_items(scl);
  const int ord = B.ord;
  // items that repeat another's type and vertices (cells with equal sides)
  // are evaluated once; grouped by kind
  std::vector<WItem> items;
  std::vector<int> uid(all.size());
  int first[4] = {0, 0, 0, 0};
  for (int kind = 0; kind < 3; ++kind) {
    for (size_t i = 0; i < all.size(); ++i) {
      const int t = all[i].type;
      if ((t == W_S ? 0 : t == W_E ? 1 : 2) != kind) continue;
      size_t k = 0;
      while (k < items.size() && (items[k].type != t || memcmp(&items[k].t, &all[i].t, sizeof(Tri6)) != 0)) ++k;
      uid[i] = (int)k;
      if (k == items.size()) items.push_back(all[i]);
    }
    first[kind + 1] = (int)items.size();
  }
  const int n = (int)items.size();
  WItem* it_d;
  gila_status s;
  if ((s = B.alloc(&it_d, items.size())) != GILA_OK) return s;
  KB_TRY(cudaMemcpyAsync(it_d, items.data(), items.size() * sizeof(WItem), cudaMemcpyHostToDevice, B.st));
  const int max_outer = 24 * ord;
  Z *part_d, *sums_d, *raw_d;
  int* uid_d;
  if ((s = B.alloc(&part_d, (size_t)n * max_outer)) != GILA_OK) return s;
  if ((s = B.alloc(&sums_d, n)) != GILA_OK) return s;
  if (raw_out)
    raw_d = raw_out;
  else if ((s = B.alloc(&raw_d, 18)) != GILA_OK)
    return s;
  if ((s = B.alloc(&uid_d, uid.size())) != GILA_OK) return s;
  KB_TRY(cudaMemcpyAsync(uid_d, uid.data(), uid.size() * sizeof(int), cudaMemcpyHostToDevice, B.st));
  auto weak = [&](auto kern, int kind, int outer) {
    const int m = first[kind + 1] - first[kind];
    kern<<<m * outer, 256, 0, B.st>>>(it_d, first[kind], outer, max_outer, B.q_d, part_d);
    return cudaGetLastError();
  };
  if (real_freq(B.f)) {
    KB_TRY(weak(k_weak<2, true>, 2, ord));
    KB_TRY(weak(k_weak<1, true>, 1, 6 * ord));
    KB_TRY(weak(k_weak<0, true>, 0, 24 * ord));
  } else {
    KB_TRY(weak(k_weak<2, false>, 2, ord));
    KB_TRY(weak(k_weak<1, false>, 1, 6 * ord));
    KB_TRY(weak(k_weak<0, false>, 0, 24 * ord));
  }
  k_weak_reduce<<<n, 32, 0, B.st>>>(it_d, ord, part_d, max_outer, sums_d);
  KB_TRY(cudaGetLastError());
  double* scl_d;
  if ((s = B.alloc(&scl_d, 3)) != GILA_OK) return s;
  KB_TRY(cudaMemcpyAsync(scl_d, scl, sizeof(scl), cudaMemcpyHostToDevice, B.st));
  const double inv = rd(rdv(R(1), rmul(rmul(sclr[0], sclr[1]), sclr[2])));
  k_weak_combine<<<1, 32, 0, B.st>>>(sums_d, uid_d, scl_d, inv, B.f, w_d, raw_d);
  KB_TRY(cudaGetLastError());
  return GILA_OK;
}

// The cubature's work lists, for chunks of at most kFarChunk items, and the
// last pass's regions.
constexpr int kFarChunk = 1 << 15, kWarps2 = 8;
struct Cub {
  Lists L;
  unsigned char* heap;
  const PairGeo* g;
  int* err;
};
static size_t cub_items(int64_t nitems) {
  return (size_t)std::min<int64_t>(std::max<int64_t>(nitems, 1), kFarChunk) + 8;
}
static size_t cub_bytes(int64_t nitems) {
  return cub_items(nitems) * (sizeof(Rec) + 24 * sizeof(Z) + 3 * 24 * sizeof(Unit)) +
         (size_t)kWarps2 * kCap2 * kRegBytes + 8 * 512;
}
static gila_status cub_alloc(Build& B, int64_t nitems, const PairGeo* g_d, int* err_d, Cub* q) {
  gila_status s;
  const size_t n = cub_items(nitems);
  q->g = g_d;
  q->err = err_d;
  if ((s = B.alloc(&q->L.rec, n)) != GILA_OK) return s;
  if ((s = B.alloc(&q->L.val, n * 24)) != GILA_OK) return s;
  for (Unit** u : {&q->L.unit, &q->L.ovf[0], &q->L.ovf[1]})
    if ((s = B.alloc(u, n * 24)) != GILA_OK) return s;
  if ((s = B.alloc(&q->L.cnt, 8)) != GILA_OK) return s;
  return B.alloc(&q->heap, (size_t)kWarps2 * kCap2 * kRegBytes);
}
static gila_status cub_reset(Build& B, Cub& q) {
  KB_TRY(cudaMemsetAsync(q.L.cnt, 0, 8 * sizeof(int), B.st));
  return GILA_OK;
}
// refines the listed pairs and writes the records' components
static gila_status cub_finish(Build& B, Cub& q, const FarParams& fp) {
  auto adapt = [&](int pass, int blocks, int threads, unsigned char* heap, int cap) -> cudaError_t {
    const void* fn = real_freq(B.f) ? (const void*)k_adapt<true> : (const void*)k_adapt<false>;
    const size_t sm = heap ? 0 : (size_t)threads / 32 * cap * kRegBytes;
    if (sm > 48 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      if (e != cudaSuccess) return e;
    }
    if (real_freq(B.f))
      k_adapt<true><<<blocks, threads, sm, B.st>>>(q.g, q.L, pass, heap, cap, q.err);
    else
      k_adapt<false><<<blocks, threads, sm, B.st>>>(q.g, q.L, pass, heap, cap, q.err);
    return cudaGetLastError();
  };
  KB_TRY(adapt(0, 592, 128, nullptr, kCap0));
  KB_TRY(adapt(1, 592, 32, nullptr, kCap1));
  KB_TRY(adapt(2, kWarps2 / 4, 128, q.heap, kCap2));
  k_far_sum<<<148, 128, 0, B.st>>>(fp, q.L);
  KB_TRY(cudaGetLastError());
  return GILA_OK;
}
// the far items of a field; units already listed (near offsets) are refined
// with the first chunk
static gila_status run_far(Build& B, Cub& q, const FarParams& fp, int64_t nitems) {
  gila_status s;
  for (int64_t i0 = 0; i0 < nitems; i0 += kFarChunk) {
    const int64_t n = std::min<int64_t>(kFarChunk, nitems - i0);
    const int64_t blocks = std::min<int64_t>(2 * 148, (n + kFarItems - 1) / kFarItems);
    if (i0 > 0 && (s = cub_reset(B, q)) != GILA_OK) return s;
    if (real_freq(B.f))
      k_far_first<true><<<(unsigned)blocks, 256, 0, B.st>>>(fp, q.g, i0, n, q.L);
    else
      k_far_first<false><<<(unsigned)blocks, 256, 0, B.st>>>(fp, q.g, i0, n, q.L);
    KB_TRY(cudaGetLastError());
    if ((s = cub_finish(B, q, fp)) != GILA_OK) return s;
  }
  return GILA_OK;
}

// Self circulant crc [6][2N] of a volume (genEgoSlf!, src/glaGen.jl:38-53)
static gila_status self_circulant(Build& B, const HVol& v, Z* crc_d, int* err_d) {
  gila_status s;
  const int64_t nx = v.cel[0], ny = v.cel[1], nz = v.cel[2], V = nx * ny * nz;
  Z *toe_d, *w_d;
  if ((s = B.alloc(&toe_d, 6 * V)) != GILA_OK) return s;
  if ((s = B.alloc(&w_d, 18)) != GILA_OK) return s;
  if ((s = weak_values(B, v.scl, w_d)) != GILA_OK) return s;
  PairGeo G;
  faces(v.scl, G.tf);
  faces(v.scl, G.sf);
  srf_scales(v.scl, v.scl, G.scale);
  G.f = B.f;
  PairGeo* g_d;
  if ((s = B.alloc(&g_d, 1)) != GILA_OK) return s;
  KB_TRY(cudaMemcpyAsync(g_d, &G, sizeof(G), cudaMemcpyHostToDevice, B.st));
  double* sep_d[3];
  for (int d = 0; d < 3; ++d) {
    std::vector<double> sp(v.cel[d]);
    for (int64_t i = 0; i < v.cel[d]; ++i) sp[i] = rd(rmul(R(i), v.grd[d]));
    if ((s = B.alloc(&sep_d[d], sp.size())) != GILA_OK) return s;
    KB_TRY(cudaMemcpyAsync(sep_d[d], sp.data(), sp.size() * sizeof(double), cudaMemcpyHostToDevice, B.st));
  }
  FarParams fp{};
  fp.mode = 0;
  for (int d = 0; d < 3; ++d) {
    fp.n[d] = (int)v.cel[d];
    fp.sep[d] = sep_d[d];
    fp.split[d] = -1;
    fp.touch[d] = -1;
  }
  fp.out = toe_d;
  Cub cub;
  if ((s = cub_alloc(B, V, g_d, err_d, &cub)) != GILA_OK) return s;
  if ((s = cub_reset(B, cub)) != GILA_OK) return s;
  // near offsets
  NearParams np;
  for (int d = 0; d < 3; ++d) {
    np.n[d] = (int)v.cel[d];
    np.sep[d] = sep_d[d];
  }
  for (int b = 0; b < 8; ++b) np.cases[b] = sng_case((b & 1) + 1, ((b >> 1) & 1) + 1, ((b >> 2) & 1) + 1, v);
  np.weak = w_d;
  k_near_list<<<8, 32, 0, B.st>>>(np, cub.L);
  KB_TRY(cudaGetLastError());
  // far offsets
  if ((s = run_far(B, cub, fp, V)) != GILA_OK) return s;
  // identity + circulant embedding
  const Z id = zdiv(Z{1.0, 0.0}, zmul(B.f, B.f));
  k_embed<<<1184, 256, 0, B.st>>>(toe_d, (int)nx, (int)ny, (int)nz, id, crc_d);
  KB_TRY(cudaGetLastError());
  return GILA_OK;
}

// lengths with compile-time x and y passes
static bool pass_length(int P) { return !ct_tiles(16, P, false).empty() || mx_ops<double2>(P); }

// FP64 forward 3-D FFT of the 6-component circulant, in place
static gila_status fft3(Build& B, Z* crc_d, const int P[3]) {
  gila_status s;
  const int64_t vol = (int64_t)P[0] * P[1] * P[2];
  for (int ax = 0; ax < 3; ++ax) {
    AxisPlan pl;
    if ((s = plan_axis(P[ax], &pl)) != GILA_OK) return s;
    if (pass_length(P[ax])) {
      // the matvec's x and y passes on whole lines, in place: rows, or kx
      // tiles of 6 Pz planes (y), or of 6 planes with a row of Px Py (z)
      const void* tw;
      if ((s = twiddle_table(B.ctx, P[ax], GILA_C128, &tw)) != GILA_OK) return s;
      double2* const c = reinterpret_cast<double2*>(crc_d);
      DevOp<double2> d{};
      Geom g{};
      const int k = ax == 0 ? 0 : 1;
      d.plan[k] = pl;
      d.tw[k] = static_cast<const double2*>(tw);
      g.sc[k] = g.tc[k] = g.P[k] = P[ax];
      Launch L{};
      L.y_tx = 8;
      if (ax == 0) {
        KB_TRY(launch_xfwd<double2>(g, d, L, c, c, 6 * vol / P[0], B.st));
      } else {
        g.P[0] = ax == 1 ? P[0] : P[0] * P[1];
        g.sc[2] = ax == 1 ? P[2] : 1;
        KB_TRY(launch_y<double2>(g, d, L, false, c, c, 0, ax == 1 ? 6LL * P[2] : 6, 0, 0, B.st));
      }
      continue;
    }
    AxisPlan* pl_d;
    if ((s = B.alloc(&pl_d, 1)) != GILA_OK) return s;
    KB_TRY(cudaMemcpyAsync(pl_d, &pl, sizeof(pl), cudaMemcpyHostToDevice, B.st));
    const void* tw;
    if ((s = twiddle_table(B.ctx, P[ax], GILA_C128, &tw)) != GILA_OK) return s;
    int TX = 2048 / P[ax];
    if (TX > 8) TX = 8;
    if (TX < 1) TX = 1;
    int T = ((TX * P[ax] + 3) / 4 + 31) / 32 * 32;
    while (T > 512 && TX > 1) {
      TX /= 2;
      T = ((TX * P[ax] + 3) / 4 + 31) / 32 * 32;
    }
    if (T > 512) return fail(GILA_ERR_ARG, "circulant axis too long for the kernel build FFT");
    int64_t es, gstride, lines, groups;
    if (ax == 0) {  // rows
      es = 1;
      lines = 6 * vol / P[0];
      groups = 1;
      gstride = 0;
    } else if (ax == 1) {
      es = P[0];
      lines = P[0];
      groups = 6LL * P[2];
      gstride = (int64_t)P[0] * P[1];
    } else {
      es = (int64_t)P[0] * P[1];
      lines = (int64_t)P[0] * P[1];
      groups = 6;
      gstride = vol;
    }
    const size_t sm = (size_t)TX * P[ax] * sizeof(double2);
    if (sm > 48 * 1024) KB_TRY(cudaFuncSetAttribute(k_fft_axis, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    const int64_t blocks = groups * ((lines + TX - 1) / TX);
    k_fft_axis<<<(unsigned)blocks, T, sm, B.st>>>(reinterpret_cast<double2*>(crc_d), pl_d, P[ax],
                                                  static_cast<const double2*>(tw), es, gstride, TX, lines,
                                                  make_fdiv((uint32_t)TX));
    KB_TRY(cudaGetLastError());
  }
  return GILA_OK;
}

}  // namespace kb

namespace kb {

// The external circulant of one target / source volume pair
// (genEgoCrcExt!, src/glaGen.jl:55-100) into crc_d [6][P...].
static gila_status ext_circulant(Build& B, const HVol& t, const HVol& sv, const int P[3], Z* crc_d, int* err_d) {
  gila_status s;
  const int64_t vol = (int64_t)P[0] * P[1] * P[2];
  Rat sl[3], su[3], tl[3], tu[3];
  bool c1 = true, c2 = true;
  int ovr = 0;
  for (int d = 0; d < 3; ++d) {
    const Rat hs = rdv(sv.scl[d], R(2)), ht = rdv(t.scl[d], R(2));
    sl[d] = rsub(sv.start[d], hs);
    su[d] = radd(sv.stop[d], hs);
    tl[d] = rsub(t.start[d], ht);
    tu[d] = radd(t.stop[d], ht);
    c1 = c1 && rle(sl[d], tl[d]) && rle(tl[d], su[d]);
    c2 = c2 && rle(sl[d], tu[d]) && rle(tu[d], su[d]);
    ovr += (rlt(sl[d], tl[d]) && rlt(tl[d], su[d])) + (rlt(sl[d], tu[d]) && rlt(tu[d], su[d]));
  }
  const bool contact = c1 || c2;
  if (contact && ovr > 0) return fail(GILA_ERR_OVERLAP, "Source and target volumes are overlapping.");
  // grdSel tables over sepGrd(trg, src, 0) / sepGrd(trg, src, 1)
  double* sep_d[3];
  for (int d = 0; d < 3; ++d) {
    Rat tstr = rsub(t.start[d], sv.start[d]), tstp = rsub(t.stop[d], sv.start[d]), tstep = t.grd[d];
    if (rlt(tstp, tstr)) tstep = rmul(tstep, R(-1));
    Rat sstr = rsub(t.start[d], sv.stop[d]), sstp = rsub(t.start[d], sv.start[d]), sstep = sv.grd[d];
    if (rlt(sstp, sstr)) sstep = rmul(sstep, R(-1));
    std::vector<double> sp(P[d], 0.0);
    for (int64_t ind = 1; ind <= P[d]; ++ind) {
      if (ind <= t.cel[d]) {
        sp[ind - 1] = rd(radd(tstr, rmul(R(ind - 1), tstep)));
      } else if (ind > t.cel[d] + 1) {
        sp[ind - 1] = rd(radd(sstr, rmul(R(ind - 2 - t.cel[d]), sstep)));
      }
    }
    if ((s = B.alloc(&sep_d[d], sp.size())) != GILA_OK) return s;
    KB_TRY(cudaMemcpyAsync(sep_d[d], sp.data(), sp.size() * sizeof(double), cudaMemcpyHostToDevice, B.st));
  }
  PairGeo G;
  faces(t.scl, G.tf);
  faces(sv.scl, G.sf);
  srf_scales(t.scl, sv.scl, G.scale);
  G.f = B.f;
  PairGeo* g_d;
  if ((s = B.alloc(&g_d, 1)) != GILA_OK) return s;
  KB_TRY(cudaMemcpyAsync(g_d, &G, sizeof(G), cudaMemcpyHostToDevice, B.st));
  FarParams fp{};
  fp.mode = 1;
  for (int d = 0; d < 3; ++d) {
    fp.n[d] = P[d];
    fp.sep[d] = sep_d[d];
    fp.split[d] = (int)t.cel[d];
    fp.touch[d] = contact ? CNT_TOL + (rd(t.scl[d]) + rd(sv.scl[d])) / 2.0 : -1.0;
  }
  fp.out = crc_d;
  Cub cub;
  if ((s = cub_alloc(B, vol, g_d, err_d, &cub)) != GILA_OK) return s;
  if ((s = cub_reset(B, cub)) != GILA_OK) return s;
  if ((s = run_far(B, cub, fp, vol)) != GILA_OK) return s;
  if (contact) {
    // genCntVol (src/glaGen.jl:308-318) and its self circulant
    int64_t cel[3];
    Rat cs[3];
    for (int d = 0; d < 3; ++d) {
      cs[d] = rlt(t.scl[d], sv.scl[d]) ? t.scl[d] : sv.scl[d];
      const Rat a = rdv(t.scl[d], cs[d]), b = rdv(sv.scl[d], cs[d]);
      cel[d] = a.n / a.d + b.n / b.d;
    }
    Vol cv0;
    for (int d = 0; d < 3; ++d) {
      cv0.cel[d] = cel[d];
      cv0.scl[d] = cs[d];
      cv0.org[d] = R(0);
      cv0.grd[d] = cs[d];
    }
    const HVol cv = hvol(cv0);
    Z* ccnt;
    if ((s = B.alloc(&ccnt, 6 * 8 * cel[0] * cel[1] * cel[2])) != GILA_OK) return s;
    if ((s = self_circulant(B, cv, ccnt, err_d)) != GILA_OK) return s;
    CntParams cp;
    for (int d = 0; d < 3; ++d) {
      cp.n[d] = P[d];
      cp.split[d] = (int)t.cel[d];
      cp.sep[d] = sep_d[d];
      cp.touch[d] = fp.touch[d];
      cp.cscl[d] = rd(cs[d]);
      const Rat ss = rdv(sv.scl[d], cs[d]), ts = rdv(t.scl[d], cs[d]);
      cp.sspan[d] = (int)(ss.n / ss.d);
      cp.tspan[d] = (int)(ts.n / ts.d);
      cp.cc[d] = (int)cel[d];
    }
    cp.ccnt = ccnt;
    cp.out = crc_d;
    k_contact<<<64, 128, 0, B.st>>>(cp);
    KB_TRY(cudaGetLastError());
  }
  return GILA_OK;
}

// Partition `tp` (x fastest) of a volume whose cells sit on a grid `div`
// times coarser than the pair's common grid (src/glaMemSup.jl:60-87): centre
// (off - (div - 1) / 2) * scl + org, cell scale scl, grid step div * scl,
// par_cel cells per axis.
static HVol partition_vol(const Vol& v, const int div[3], const int par_cel[3], const int off[3]) {
  Vol p;
  for (int d = 0; d < 3; ++d) {
    p.cel[d] = par_cel[d];
    p.scl[d] = v.scl[d];
    p.org[d] = radd(rmul(rsub(R(off[d]), R(div[d] - 1, 2)), v.scl[d]), v.org[d]);
    p.grd[d] = rmul(R(div[d]), v.scl[d]);
  }
  return hvol(p);
}

}  // namespace kb

// Build the operator's Fourier kernel on the GPU (GlaOprMem with
// egoFur == nothing).  Volume pairs of different cell scales are built per
// target partition (src/glaMemSup.jl:60-88), each partition's circulant
// transformed and extracted into its slice of the kernel.  Source
// partitions (a source grid finer than the target) are refused: egoOpr!
// cannot apply such an operator (src/glaAct.jl:37-49).
gila_status build_kernel(Core& c) {
  using namespace kb;
  if (c.parS != 1)
    return fail(GILA_ERR_ARG, "the GPU kernel build does not handle source partitions (a source grid finer than "
                              "the target), which egoOpr! cannot apply; pass egoFur instead");
  Build B;
  B.ctx = c.ctx;
  B.st = c.stream;
  B.f = Z{c.opt.frq_re, c.opt.frq_im};
  B.ord = c.opt.int_ord > 0 ? c.opt.int_ord : 32;
  if (B.ord > kMaxOrd) return fail(GILA_ERR_ARG, "intOrd above 64 is not supported");
  gila_status s;
  {
    // one block for the circulant, the field and the work lists
    const int64_t pv = (int64_t)c.geom.P[0] * c.geom.P[1] * c.geom.P[2], items = c.self ? pv / 8 : pv;
    B.block_bytes = (size_t)(6 * pv * (int64_t)sizeof(Z) + (c.self ? 6 * items * (int64_t)sizeof(Z) : 0)) +
                    cub_bytes(items) + (size_t(4) << 20);
  }
  {
    Consts q;
    q.ord = B.ord;
    gauss_legendre(B.ord, q.x, q.w);
    q.f = B.f;
    if ((s = B.alloc(&B.q_d, 1)) != GILA_OK) return s;
    KB_TRY(cudaMemcpyAsync(B.q_d, &q, sizeof(q), cudaMemcpyHostToDevice, B.st));
    B.block_bytes = size_t(32) << 20;  // of any further block
  }
  KB_TRY(cudaMemcpyToSymbolAsync(c_sng_cor, SNG_COR, sizeof(SNG_COR), 0, cudaMemcpyHostToDevice, B.st));
  KB_TRY(cudaMemcpyToSymbolAsync(c_sng_mask, SNG_MASK, sizeof(SNG_MASK), 0, cudaMemcpyHostToDevice, B.st));
  int* err_d;
  if ((s = B.alloc(&err_d, 2)) != GILA_OK) return s;
  KB_TRY(cudaMemsetAsync(err_d, 0, 2 * sizeof(int), B.st));
  const HVol t = hvol(c.trg), sv = hvol(c.src);
  const int P[3] = {c.geom.P[0], c.geom.P[1], c.geom.P[2]};
  const int64_t vol = (int64_t)P[0] * P[1] * P[2];
  Z* crc_d;
  if ((s = B.alloc(&crc_d, 6 * vol)) != GILA_OK) return s;
  const Geom& g = c.geom;
  const int parT = g.parT;
  const size_t cs = csize(c.dtype);
  const size_t per = (size_t)g.tru[0] * g.tru[1] * g.tru[2] * 6 * 8;  // elements per target partition
  KB_TRY(dev_malloc(&c.ker, per * parT * cs));
  c.ker_bytes = per * parT * cs;
  const Build::Mark mark = B.mark();
  for (int tp = 0; tp < parT; ++tp) {
    if (c.self) {
      if ((s = self_circulant(B, t, crc_d, err_d)) != GILA_OK) return s;
    } else {
      KB_TRY(cudaMemsetAsync(crc_d, 0, (size_t)6 * vol * sizeof(Z), B.st));
      const HVol tv = parT == 1 ? t : partition_vol(c.trg, c.mix.tdiv, c.mix.tc, g.toff[tp]);
      if ((s = ext_circulant(B, tv, sv, P, crc_d, err_d)) != GILA_OK) return s;
    }
    if ((s = fft3(B, crc_d, P)) != GILA_OK) return s;
    // extract into partition tp of the operator's kernel layout
    if (c.dtype == GILA_C128)
      k_extract<double2><<<1184, 256, 0, B.st>>>(crc_d, P[0], P[1], P[2], g.tru[0], g.tru[1], g.tru[2],
                                                static_cast<double2*>(c.ker) + per * tp, err_d + 1);
    else
      k_extract<float2><<<1184, 256, 0, B.st>>>(crc_d, P[0], P[1], P[2], g.tru[0], g.tru[1], g.tru[2],
                                               static_cast<float2*>(c.ker) + per * tp, err_d + 1);
    KB_TRY(cudaGetLastError());
    if (tp + 1 < parT) B.release_to(mark);  // this partition's cubature scratch
  }
  int flags[2];
  KB_TRY(cudaMemcpyAsync(flags, err_d, sizeof(flags), cudaMemcpyDeviceToHost, B.st));
  KB_TRY(cudaStreamSynchronize(B.st));
  if (flags[0]) return fail(GILA_ERR_INTERNAL, "kernel build: cubature region capacity exceeded");
  if (flags[1]) return fail(GILA_ERR_NAN, "Fourier information contains non-numeric values.");
  return GILA_OK;
}

// wekS / wekE / wekV (src/glaInt.jl:75-262) for one cell scale at
// Gauss-Legendre order `ord`, unscaled, evaluated on the GPU by the same
// kernels the operator build uses (out: 18 complex values as re/im pairs,
// wS[3], wE[9], wV[6]).
gila_status weak_integrals(Ctx* ctx, const Rat scl[3], kb::Z f, int ord, double out[36]) {
  using namespace kb;
  if (ord < 1 || ord > kMaxOrd) return fail(GILA_ERR_ARG, "intOrd must be in 1..64");
  for (int d = 0; d < 3; ++d)
    if (scl[d].n <= 0 || scl[d].d <= 0) return fail(GILA_ERR_ARG, "cell scales must be positive");
  cudaStream_t st = nullptr;
  KB_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  gila_status s = GILA_OK;
  {
    Build B;
    B.ctx = ctx;
    B.st = st;
    B.f = f;
    B.ord = ord;
    B.block_bytes = size_t(4) << 20;
    Consts q;
    q.ord = ord;
    gauss_legendre(ord, q.x, q.w);
    q.f = f;
    Z* w_d = nullptr;
    Z raw[18];
    if ((s = B.alloc(&B.q_d, 1)) == GILA_OK) {
      cudaError_t e = cudaMemcpyAsync(B.q_d, &q, sizeof(q), cudaMemcpyHostToDevice, st);
      if (e != cudaSuccess) s = cuda_fail(e, "cudaMemcpyAsync(weak consts)");
    }
    if (s == GILA_OK) s = B.alloc(&w_d, 36);
    if (s == GILA_OK) s = weak_values(B, scl, w_d, w_d + 18);
    if (s == GILA_OK) {
      cudaError_t e = cudaMemcpyAsync(raw, w_d + 18, sizeof(raw), cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) s = cuda_fail(e, "weak integrals");
    }
    cudaStreamSynchronize(st);
    if (s == GILA_OK)
      for (int k = 0; k < 18; ++k) {
        out[2 * k] = raw[k].x;
        out[2 * k + 1] = raw[k].y;
      }
  }
  cudaStreamDestroy(st);
  return s;
}

}  // namespace gila

extern "C" gila_status gila_weak_integrals(gila_ctx* ctx, const int64_t scl_num[3], const int64_t scl_den[3],
                                           double frq_re, double frq_im, int32_t int_ord, double out[36]) {
  using namespace gila;
  if (!ctx || !scl_num || !scl_den || !out) return fail(GILA_ERR_ARG, "null argument");
  GILA_CUDA_TRY(cudaSetDevice(ctx->impl->device));
  Rat scl[3];
  for (int d = 0; d < 3; ++d) {
    if (scl_den[d] == 0) return fail(GILA_ERR_ARG, "zero denominator in a cell scale");
    scl[d] = rat(scl_num[d], scl_den[d]);
  }
  return weak_integrals(ctx->impl, scl, kb::Z{frq_re, frq_im}, int_ord, out);
}
