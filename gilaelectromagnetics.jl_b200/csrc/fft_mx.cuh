// fft_mx.cuh -- building blocks of the mixed-radix passes (matvec_mx.cuh):
// 16-byte shared-memory elements, register butterflies of radix 2 .. 16 and
// the compile-time choice of the radices of a length.
//
// One element type serves both precisions: a ComplexF64 value, or the
// ComplexF32 values of two adjacent lines (a line pair), so every shared- or
// global-memory access of a pass moves 16 bytes per thread and the passes are
// written once.
#pragma once
#include "fft.cuh"

namespace gila {

#define GILA_HD __host__ __device__ __forceinline__

// -------------------------------------------------------------- elements
// two lines' ComplexF32 values at one position
struct alignas(16) F2x2 {
  float2 a, b;
};

template <typename C> struct MxElem;
template <> struct MxElem<double2> { using V = double2; };
template <> struct MxElem<float2> { using V = F2x2; };
template <typename V> struct MxOf;  // table / scalar types of an element
template <> struct MxOf<double2> { using W = double2; using T = double; };
template <> struct MxOf<F2x2> { using W = float2; using T = float; };

GILA_HD double2 vadd(double2 a, double2 b) { return double2{a.x + b.x, a.y + b.y}; }
GILA_HD double2 vsub(double2 a, double2 b) { return double2{a.x - b.x, a.y - b.y}; }
GILA_HD double2 vscale(double2 a, double s) { return double2{a.x * s, a.y * s}; }
GILA_HD double2 vmul(double2 a, double2 w) { return double2{fma(a.x, w.x, -a.y * w.y), fma(a.x, w.y, a.y * w.x)}; }
// c + s a
GILA_HD double2 vfma(double2 a, double s, double2 c) { return double2{fma(a.x, s, c.x), fma(a.y, s, c.y)}; }
// multiply by -i (forward) or +i (inverse)
template <bool INV> GILA_HD double2 vmi(double2 a) { return INV ? double2{-a.y, a.x} : double2{a.y, -a.x}; }
template <typename V> GILA_HD V vzero();
template <> GILA_HD double2 vzero<double2>() { return double2{0.0, 0.0}; }

GILA_HD float2 fadd2(float2 a, float2 b) { return float2{a.x + b.x, a.y + b.y}; }
GILA_HD float2 fsub2(float2 a, float2 b) { return float2{a.x - b.x, a.y - b.y}; }
GILA_HD float2 fmul2(float2 a, float2 w) { return float2{fmaf(a.x, w.x, -a.y * w.y), fmaf(a.x, w.y, a.y * w.x)}; }
GILA_HD F2x2 vadd(F2x2 a, F2x2 b) { return F2x2{fadd2(a.a, b.a), fadd2(a.b, b.b)}; }
GILA_HD F2x2 vsub(F2x2 a, F2x2 b) { return F2x2{fsub2(a.a, b.a), fsub2(a.b, b.b)}; }
GILA_HD F2x2 vscale(F2x2 a, float s) {
  return F2x2{float2{a.a.x * s, a.a.y * s}, float2{a.b.x * s, a.b.y * s}};
}
GILA_HD F2x2 vmul(F2x2 a, float2 w) { return F2x2{fmul2(a.a, w), fmul2(a.b, w)}; }
GILA_HD F2x2 vfma(F2x2 a, float s, F2x2 c) {
  return F2x2{float2{fmaf(a.a.x, s, c.a.x), fmaf(a.a.y, s, c.a.y)}, float2{fmaf(a.b.x, s, c.b.x), fmaf(a.b.y, s, c.b.y)}};
}
template <bool INV> GILA_HD F2x2 vmi(F2x2 a) {
  return INV ? F2x2{float2{-a.a.y, a.a.x}, float2{-a.b.y, a.b.x}} : F2x2{float2{a.a.y, -a.a.x}, float2{a.b.y, -a.b.x}};
}
template <> GILA_HD F2x2 vzero<F2x2>() { return F2x2{float2{0.f, 0.f}, float2{0.f, 0.f}}; }

// times exp(-+ i phi) given cos phi, sin phi (minus forward, plus inverse)
template <bool INV, typename V> GILA_HD V vrot(V a, double c, double s) {
  using T = typename MxOf<V>::T;
  return vfma(vmi<INV>(a), (T)s, vscale(a, (T)c));
}

// ------------------------------------------------------------ butterflies
// In-place R-point DFT, natural order in and out: v[k] <- sum_r v[r]
// exp(-+ 2 pi i r k / R).  Composite radices whose factors are coprime run
// the prime-factor map (Good 1958): no twiddles between the factors.
template <int R, bool INV> struct Dft;

constexpr int mx_inv_mod(int a, int m) {  // a^-1 mod m
  for (int x = 1; x < m; ++x)
    if (a * x % m == 1) return x;
  return 1;
}

// A first: where it is 2 or 4 its inputs are N / A apart, so on a zero-padded
// line its additions are of exact zeros (B first rounds once more there).
template <int A, int B, bool INV> struct DftPfa {  // R = A * B, coprime
  template <typename V> GILA_HD static void run(V* v) {
    constexpr int N = A * B;
    constexpr int ca = B * mx_inv_mod(B % A, A) % N, cb = A * mx_inv_mod(A % B, B) % N;
    V t[N];
#pragma unroll
    for (int j = 0; j < B; ++j) {
      V u[A];
#pragma unroll
      for (int i = 0; i < A; ++i) u[i] = v[(B * i + A * j) % N];
      Dft<A, INV>::run(u);
#pragma unroll
      for (int i = 0; i < A; ++i) t[i * B + j] = u[i];
    }
#pragma unroll
    for (int i = 0; i < A; ++i) {
      V u[B];
#pragma unroll
      for (int j = 0; j < B; ++j) u[j] = t[i * B + j];
      Dft<B, INV>::run(u);
#pragma unroll
      for (int j = 0; j < B; ++j) v[(ca * i + cb * j) % N] = u[j];
    }
  }
};

template <bool INV> struct Dft<1, INV> {
  template <typename V> GILA_HD static void run(V*) {}
};
template <bool INV> struct Dft<2, INV> {
  template <typename V> GILA_HD static void run(V* v) {
    const V a = v[0], b = v[1];
    v[0] = vadd(a, b);
    v[1] = vsub(a, b);
  }
};
template <bool INV> struct Dft<3, INV> {
  template <typename V> GILA_HD static void run(V* v) {
    using T = typename MxOf<V>::T;
    const T s = (T)0.86602540378443864676372317075293618347;
    const V t = vadd(v[1], v[2]);
    const V m = vfma(t, (T)-0.5, v[0]);
    const V u = vmi<INV>(vsub(v[1], v[2]));
    v[0] = vadd(v[0], t);
    v[1] = vfma(u, s, m);
    v[2] = vfma(u, -s, m);
  }
};
template <bool INV> struct Dft<4, INV> {
  template <typename V> GILA_HD static void run(V* v) {
    const V t0 = vadd(v[0], v[2]), t1 = vsub(v[0], v[2]);
    const V t2 = vadd(v[1], v[3]), t3 = vmi<INV>(vsub(v[1], v[3]));
    v[0] = vadd(t0, t2);
    v[2] = vsub(t0, t2);
    v[1] = vadd(t1, t3);
    v[3] = vsub(t1, t3);
  }
};
template <bool INV> struct Dft<5, INV> {
  template <typename V> GILA_HD static void run(V* v) {
    using T = typename MxOf<V>::T;
    const T c1 = (T)0.30901699437494742410229341718281905886, c2 = (T)-0.80901699437494742410229341718281905886;
    const T s1 = (T)0.95105651629515357211643933337938214340, s2 = (T)0.58778525229247312916870595463907276860;
    const V a1 = vadd(v[1], v[4]), b1 = vmi<INV>(vsub(v[1], v[4]));
    const V a2 = vadd(v[2], v[3]), b2 = vmi<INV>(vsub(v[2], v[3]));
    const V x0 = v[0];
    const V p1 = vfma(a2, c2, vfma(a1, c1, x0)), p2 = vfma(a2, c1, vfma(a1, c2, x0));
    const V q1 = vfma(b2, s2, vscale(b1, s1)), q2 = vfma(b2, -s1, vscale(b1, s2));
    v[0] = vadd(x0, vadd(a1, a2));
    v[1] = vadd(p1, q1);
    v[4] = vsub(p1, q1);
    v[2] = vadd(p2, q2);
    v[3] = vsub(p2, q2);
  }
};
template <bool INV> struct Dft<7, INV> {
  template <typename V> GILA_HD static void run(V* v) {
    using T = typename MxOf<V>::T;
    const T c1 = (T)0.62348980185873353052500488400423981063, c2 = (T)-0.22252093395631440428890256449679475947,
            c3 = (T)-0.90096886790241912623610231950744505117;
    const T s1 = (T)0.78183148246802980870844452667405775023, s2 = (T)0.97492791218182360701813168299393121723,
            s3 = (T)0.43388373911755812047576833284835875461;
    const V a1 = vadd(v[1], v[6]), b1 = vmi<INV>(vsub(v[1], v[6]));
    const V a2 = vadd(v[2], v[5]), b2 = vmi<INV>(vsub(v[2], v[5]));
    const V a3 = vadd(v[3], v[4]), b3 = vmi<INV>(vsub(v[3], v[4]));
    const V x0 = v[0];
    const V p1 = vfma(a3, c3, vfma(a2, c2, vfma(a1, c1, x0)));
    const V p2 = vfma(a3, c1, vfma(a2, c3, vfma(a1, c2, x0)));
    const V p3 = vfma(a3, c2, vfma(a2, c1, vfma(a1, c3, x0)));
    const V q1 = vfma(b3, s3, vfma(b2, s2, vscale(b1, s1)));
    const V q2 = vfma(b3, -s1, vfma(b2, -s3, vscale(b1, s2)));
    const V q3 = vfma(b3, s2, vfma(b2, -s1, vscale(b1, s3)));
    v[0] = vadd(x0, vadd(a1, vadd(a2, a3)));
    v[1] = vadd(p1, q1);
    v[6] = vsub(p1, q1);
    v[2] = vadd(p2, q2);
    v[5] = vsub(p2, q2);
    v[3] = vadd(p3, q3);
    v[4] = vsub(p3, q3);
  }
};
template <bool INV> struct Dft<8, INV> {
  template <typename V> GILA_HD static void run(V* v) {
    using T = typename MxOf<V>::T;
    const T h = (T)0.70710678118654752440084436210484903928;
    V e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    Dft<4, INV>::run(e);
    Dft<4, INV>::run(o);
    o[1] = vadd(o[1], vmi<INV>(o[1]));
    o[2] = vmi<INV>(o[2]);
    o[3] = vsub(vmi<INV>(o[3]), o[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[k] = k % 2 ? vfma(o[k], h, e[k]) : vadd(e[k], o[k]);
      v[k + 4] = k % 2 ? vfma(o[k], -h, e[k]) : vsub(e[k], o[k]);
    }
  }
};
template <bool INV> struct Dft<9, INV> {
  template <typename V> GILA_HD static void run(V* v) {
    const double c1 = 0.76604444311897803520239265055541667394, s1 = 0.64278760968653932632264340990726343291;
    const double c2 = 0.17364817766693034885171662676931479600, s2 = 0.98480775301220805936674302458952301367;
    const double c4 = -0.93969262078590838405410927732473146994, s4 = 0.34202014332566873304409961468225958076;
    V y[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
      for (int j = 0; j < 3; ++j) y[i][j] = v[i + 3 * j];
      Dft<3, INV>::run(y[i]);
    }
    y[1][1] = vrot<INV>(y[1][1], c1, s1);
    y[1][2] = vrot<INV>(y[1][2], c2, s2);
    y[2][1] = vrot<INV>(y[2][1], c2, s2);
    y[2][2] = vrot<INV>(y[2][2], c4, s4);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      V u[3] = {y[0][j], y[1][j], y[2][j]};
      Dft<3, INV>::run(u);
#pragma unroll
      for (int i = 0; i < 3; ++i) v[j + 3 * i] = u[i];
    }
  }
};
template <bool INV> struct Dft<16, INV> {
  template <typename V> GILA_HD static void run(V* v) {
    const double c1 = 0.92387953251128675612818318939678828682, s1 = 0.38268343236508977172845998403039886676;
    const double h = 0.70710678118654752440084436210484903928;
    V y[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) y[i][j] = v[i + 4 * j];
      Dft<4, INV>::run(y[i]);
    }
    y[1][1] = vrot<INV>(y[1][1], c1, s1);
    y[1][2] = vrot<INV>(y[1][2], h, h);
    y[1][3] = vrot<INV>(y[1][3], s1, c1);
    y[2][1] = vrot<INV>(y[2][1], h, h);
    y[2][2] = vmi<INV>(y[2][2]);
    y[2][3] = vrot<INV>(y[2][3], -h, h);
    y[3][1] = vrot<INV>(y[3][1], s1, c1);
    y[3][2] = vrot<INV>(y[3][2], -h, h);
    y[3][3] = vrot<INV>(y[3][3], -c1, -s1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      V u[4] = {y[0][j], y[1][j], y[2][j], y[3][j]};
      Dft<4, INV>::run(u);
#pragma unroll
      for (int i = 0; i < 4; ++i) v[j + 4 * i] = u[i];
    }
  }
};
template <bool INV> struct Dft<6, INV> : DftPfa<2, 3, INV> {};
template <bool INV> struct Dft<10, INV> : DftPfa<2, 5, INV> {};
template <bool INV> struct Dft<12, INV> : DftPfa<4, 3, INV> {};
template <bool INV> struct Dft<14, INV> : DftPfa<2, 7, INV> {};
template <bool INV> struct Dft<15, INV> : DftPfa<3, 5, INV> {};

// --------------------------------------------------------------- schedule
// Radices of a length-P transform (product P) and the threads that share one
// line.  A stage of radix r has P / r butterflies; a thread runs
// ceil(P / r / tpb) of them, so it is idle for part of a stage whose count
// tpb does not divide.  The schedule with the least total of these thread
// slots, plus a fixed cost for each stage's barriers and shared-memory round
// trip, is taken.
constexpr int kMxMaxStages = 5;
struct MxSched {
  int n = 0;
  int r[kMxMaxStages] = {};
  int tpb = 0;  // threads per line
};
constexpr bool mx_radix_ok(int r) { return (r >= 2 && r <= 10) || r == 12 || r == 14 || r == 15 || r == 16; }

struct MxSearch {
  int P, rmax, last_max, stage_cost;
  MxSched best{};
  long best_cost = -1;
  int cur[kMxMaxStages] = {};

  // cost in units of 1/1000 line passes
  constexpr long cost(int n, int tpb) const {
    long c = 0;
    for (int s = 0; s < n; ++s) {
      const int r = cur[s], tasks = P / r, k = (tasks + tpb - 1) / tpb;
      if (k * r > rmax + rmax / 4) return -1;  // values held by a thread
      c += 1000L * k * r * tpb / P + stage_cost;
    }
    return c;
  }
  constexpr void walk(int n, int rest, int prev) {
    if (rest == 1) {
      if (n == 0 || cur[n - 1] > last_max) return;
      for (int s = 0; s < n; ++s) {
        const int tpb = P / cur[s];
        const long c = cost(n, tpb);
        if (c >= 0 && (best_cost < 0 || c < best_cost)) {
          best_cost = c;
          best = MxSched{};
          best.n = n;
          for (int q = 0; q < n; ++q) best.r[q] = cur[q];
          best.tpb = tpb;
        }
      }
      return;
    }
    if (n == kMxMaxStages) return;
    for (int r = prev < rmax ? prev : rmax; r >= 2; --r)  // radices fall from stage to stage
      if (mx_radix_ok(r) && rest % r == 0) {
        cur[n] = r;
        walk(n + 1, rest / r, r);
      }
  }
};
// last_max: bound on the last radix (the z pass holds three components of
// it); a length below 4 keeps one stage
constexpr MxSched mx_search(int P, int rmax, int last_max, int stage_cost) {
  MxSearch m{P, rmax, last_max, stage_cost};
  m.walk(0, P, P);
  return m.best;
}

// MXK_XY: x and y passes; MXK_Z: fused z pass, whose last radix three
// components share a thread's registers
enum { MXK_XY = 0, MXK_Z = 1 };
// Radices up to 10 to length 100, where larger ones gain at some lengths (z 72 at
// 80x80 F64 62.6 -> 54.0 us, 84 76.6 -> 68.4) and lose at others and at small
// volumes (x and y 80 at 40x40x64 34.6 -> 45.3 us, F32 27.5 -> 39.5); up to 16
// above, where 10 loses (z 112 at 80x80 F64 90 -> 133 us, 140 119 -> 165; x and y
// 120 at 60x60x64 48.5 -> 58.5 us).
constexpr MxSched mx_sched(int P, int kind) {
  return mx_search(P, P <= 100 ? 10 : 16, kind == MXK_Z ? 4 : 16, 400);
}
template <int P, int KIND> struct MxPlan {
  static constexpr MxSched s = mx_sched(P, KIND);
};
// radix and span of stage S, in reversed order for the z pass's inverse
constexpr int mx_sr(const MxSched& s, bool rev, int S) { return rev ? s.r[s.n - 1 - S] : s.r[S]; }
constexpr int mx_sspan(const MxSched& s, bool rev, int S) {
  int ns = 1;
  for (int k = 0; k < S; ++k) ns *= mx_sr(s, rev, k);
  return ns;
}
template <int P, int KIND, bool REV> constexpr int mx_r(int S) { return mx_sr(MxPlan<P, KIND>::s, REV, S); }
template <int P, int KIND, bool REV> constexpr int mx_span(int S) { return mx_sspan(MxPlan<P, KIND>::s, REV, S); }

// Twiddle tables of a length, behind the P entries w^m of its table: for each
// stage after the first of the x / y plan, of the z plan and of the reversed z
// plan the factors w^(q jm P / (NS R)) as [q - 1][jm], so that neighbouring
// threads (neighbouring jm) load neighbouring entries.  From the plain table
// they load entries q P / (NS R) apart, a cache line each: in the x passes the
// twiddles then take more of the load pipe than the data.
constexpr int mx_tw_stages(const MxSched& s, bool rev, int S) {  // entries of stages 1 .. S - 1
  int n = 0;
  for (int k = 1; k < S; ++k) n += (mx_sr(s, rev, k) - 1) * mx_sspan(s, rev, k);
  return n;
}
constexpr int mx_tw_base(int P, int kind, bool rev) {
  int b = P;
  if (kind == MXK_Z) b += mx_tw_stages(mx_sched(P, MXK_XY), false, mx_sched(P, MXK_XY).n);
  if (kind == MXK_Z && rev) b += mx_tw_stages(mx_sched(P, MXK_Z), false, mx_sched(P, MXK_Z).n);
  return b;
}
constexpr int mx_tw_len(int P) {
  return mx_tw_base(P, MXK_Z, true) + mx_tw_stages(mx_sched(P, MXK_Z), true, mx_sched(P, MXK_Z).n);
}
template <int P, int KIND, bool REV, int S> struct MxTw {
  static constexpr int off = mx_tw_base(P, KIND, REV) + mx_tw_stages(MxPlan<P, KIND>::s, REV, S);
};
// exponents of the entries P .. mx_tw_len(P) - 1 (host)
template <typename F>
inline void mx_tw_fill(int P, const F& put) {
  int at = P;
  for (int t = 0; t < 3; ++t) {
    const MxSched s = mx_sched(P, t == 0 ? MXK_XY : MXK_Z);
    const bool rev = t == 2;
    for (int k = 1; k < s.n; ++k) {
      const int R = mx_sr(s, rev, k), NS = mx_sspan(s, rev, k), st = P / (NS * R);
      for (int q = 1; q < R; ++q)
        for (int jm = 0; jm < NS; ++jm) put(at++, (int)((long)q * jm * st % P));
    }
  }
}

// Shared-memory line of a plan: element i sits at i + i / R0 where the first
// radix R0 is even, at i where it is odd, so that the first stage's stores (R0
// apart) start on different banks; its length in elements.
template <int P, int KIND> GILA_HD int mx_pad(int i) {
  constexpr int r0 = MxPlan<P, KIND>::s.r[0];
  return r0 % 2 == 0 ? i + (int)((unsigned)i / (unsigned)r0) : i;
}
template <int P, int KIND> constexpr int mx_line_len() {
  constexpr int r0 = MxPlan<P, KIND>::s.r[0];
  return r0 % 2 == 0 ? P + P / r0 : P;
}
// ----------------------------------------------------------------- stages
// Twiddles q = 1 .. R-1 of a stage of span NS from its table (at jm), all
// loaded.  In FP64, three of four as products of the others are faster (one
// product at 80x80x40 0.110 against 0.122 ms, 80x80x50 0.140 / 0.147, 80x80x120
// 0.351 / 0.380) but carry the products' roundings: relative error of a product
// at 54x42x36 5.6e-16 against 4.8e-16, at 100x84x60 4.7e-16 against 4.3e-16
// (runtime-planned kernels: 5.0e-16 and 4.5e-16).
template <bool INV, typename W> GILA_HD W mx_tw(const W* __restrict__ tw, int m) {
#ifdef __CUDA_ARCH__
  W w = __ldg(tw + m);
#else
  W w = tw[m];
#endif
  if constexpr (INV) w.y = -w.y;
  return w;
}
template <int R, int NS, bool INV, typename W> GILA_HD void mx_twiddles(const W* __restrict__ tw, W* w) {
#pragma unroll
  for (int q = 1; q < R; ++q) w[q] = mx_tw<INV>(tw, (q - 1) * NS);
}

// Stage S of a line shared by TPB threads (this thread: j0 of them).  ld(k, i)
// reads input i, st(i, v) writes output i of the line (Stockham order: inputs
// j + r P/R, outputs (j - j mod NS) R + j mod NS + r NS).  All loads of the
// thread come first, then sync(), then the butterflies and stores.
template <typename V, int P, int KIND, int S, int TPB, bool INV, bool REV, class Ld, class St, class Sync>
__device__ __forceinline__ void mx_stage(int j0, const typename MxOf<V>::W* __restrict__ tw, const Ld& ld,
                                         const St& st, const Sync& sync) {
  constexpr int R = mx_r<P, KIND, REV>(S), NS = mx_span<P, KIND, REV>(S), TPL = P / R;
  constexpr int K = (TPL + TPB - 1) / TPB;
  using W = typename MxOf<V>::W;
  V v[K][R];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int j = j0 + k * TPB;
    if (TPL % TPB == 0 || j < TPL) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[k][r] = ld(j + r * TPL);
    }
  }
  sync();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int j = j0 + k * TPB;
    if (TPL % TPB == 0 || j < TPL) {
      const int jm = NS == 1 ? 0 : (NS == TPL ? j : j % NS);
      if constexpr (NS > 1) {
        W w[R];
        mx_twiddles<R, NS, INV>(tw + MxTw<P, KIND, REV, S>::off + jm, w);
#pragma unroll
        for (int r = 1; r < R; ++r) v[k][r] = vmul(v[k][r], w[r]);
      }
      Dft<R, INV>::run(v[k]);
      const int base = (j - jm) * R + jm;
#pragma unroll
      for (int r = 0; r < R; ++r) st(base + r * NS, v[k][r]);
    }
  }
}

}  // namespace gila
