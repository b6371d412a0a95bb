// matvec_mx_impl.cuh -- kernels of the five matvec passes for mixed-radix
// lengths (2^a 3^b 5^c 7^d), instantiated per length by matvec_mx_*.cu.
//
// Against the runtime-planned kernels (fft.cuh) that these lengths ran on:
// index arithmetic, radices and spans are constants, a stage's radix goes up
// to 10 at lengths to 100 and to 16 above (two or three shared-memory round
// trips a line instead of three to five), the first stage is fed from global
// memory and the last one writes it, ComplexF32 moves line pairs, and the z pass
// multiplies in registers between its last forward and first inverse butterfly
// and runs its three components on separate threads.  One product as a timed
// call, runtime-planned -> these: 16^3 F64 66 -> 35 us (25 us of it host), 50x40x30
// F64 157 -> 53 us, 100x84x60 F64 1.114 -> 0.240 ms (2.0 TB/s of the algorithmic
// bytes), 180x140x90 F32 3.63 -> 0.585 ms (1.9 TB/s).
#pragma once
#include "fft_mx.cuh"
#include "matvec_mx.cuh"

namespace gila {

// ------------------------------------------------------- element access
__device__ __forceinline__ double2 mx_ldg(const double2* p) { return *p; }
__device__ __forceinline__ F2x2 mx_ldg(const F2x2* p) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  return F2x2{float2{q.x, q.y}, float2{q.z, q.w}};
}
__device__ __forceinline__ double2 mx_ldcs(const double2* p) { return __ldcs(p); }
__device__ __forceinline__ F2x2 mx_ldcs(const F2x2* p) {
  const float4 q = __ldcs(reinterpret_cast<const float4*>(p));
  return F2x2{float2{q.x, q.y}, float2{q.z, q.w}};
}
__device__ __forceinline__ void mx_st(double2* p, double2 v) { *p = v; }
__device__ __forceinline__ void mx_st(F2x2* p, F2x2 v) {
  *reinterpret_cast<float4*>(p) = make_float4(v.a.x, v.a.y, v.b.x, v.b.y);
}

constexpr int mx_up32(int a) { return (a + 31) / 32 * 32; }
// resident blocks a kernel of T threads is compiled for at `regs` registers
constexpr int mx_blocks(int T, int regs) {
  const int b = 65536 / (mx_up32(T) * regs);
  return b < 1 ? 1 : (b > 16 ? 16 : b);
}
constexpr int kMxRegs = 96;  // y pass
// z pass, by length and last radix RL (a thread of the fused stage holds three
// components of RL values and a frequency's kernel values):
// - up to 100, RL 4 (28, 32, 36, 40): 128.  At 84 and 104 these spill 390 and
//   230 bytes in F64, 480 and 290 in F32: 80x80x20 F64 41.8 and 37.9 us, 29.7 at
//   128, F32 29.3 and 25.2, 22.9; 80x80x14 F64 33.7 and 29.9, 25.6; at 168 within
//   4% of 128 either way.
// - up to 100, RL 2 or 3: 84, two blocks more per SM than 104: 80x80x30 F64 49.3
//   against 55.4 us, 80x80x50 73.7 / 86.2, 80x80x24 41.5 / 47.8 (54 the exception,
//   59.6 / 55.5).
// - above 100: 104.  84 there: 80x80x56 F64 89 -> 100 us, 80x80x80 136 -> 186,
//   80x80x140 (RL 4) 293 -> 399; 108, 168 and 200 are faster at 84 (168: 192 ->
//   149), 126 and 252 in F64 not (116 -> 125).
// (350, 486 and 490 run 648 to 840 threads a block, which the register file
// holds at 72 to 80 a thread whatever is asked for.)
template <int P> constexpr int mx_z_regs() {
  constexpr int RL = mx_r<P, MXK_Z, false>(MxPlan<P, MXK_Z>::s.n - 1);
  return P > 100 ? 104 : RL == 4 ? 128 : 84;
}
// the next frequency's kernel values in flight while one is multiplied: F64
// above 100 (180x140x90: 613 -> 598 us); elsewhere the registers count for more
// (F32 180x140x90 345 -> 326 us without)
constexpr bool mx_z_ahead(int cs, int P) { return cs == 16 && P > 100; }

// stages [S, NST - 1) in place in shared memory
template <typename V, int P, int KIND, int S, int TPB, bool INV, class Ld, class St>
__device__ __forceinline__ void mx_middle(int j0, const typename MxOf<V>::W* __restrict__ tw, const Ld& ld,
                                          const St& st) {
  if constexpr (S < MxPlan<P, KIND>::s.n - 1) {
    mx_stage<V, P, KIND, S, TPB, INV, false>(j0, tw, ld, st, [] { __syncthreads(); });
    __syncthreads();
    mx_middle<V, P, KIND, S + 1, TPB, INV>(j0, tw, ld, st);
  }
}

// a whole line: first stage from gld, last to gst, shared memory in between
template <typename V, int P, int KIND, int TPB, bool INV, class Gld, class Gst, class Ld, class St>
__device__ __forceinline__ void mx_line(int j0, const typename MxOf<V>::W* __restrict__ tw, const Gld& gld,
                                        const Gst& gst, const Ld& ld, const St& st) {
  constexpr int N = MxPlan<P, KIND>::s.n;
  auto none = [] {};
  if constexpr (N == 1) {
    mx_stage<V, P, KIND, 0, TPB, INV, false>(j0, tw, gld, gst, none);
  } else {
    mx_stage<V, P, KIND, 0, TPB, INV, false>(j0, tw, gld, st, none);
    __syncthreads();
    mx_middle<V, P, KIND, 1, TPB, INV>(j0, tw, ld, st);
    mx_stage<V, P, KIND, N - 1, TPB, INV, false>(j0, tw, ld, gst, none);
  }
}

// -------------------------------------------------------------------- x
// A thread group of TPB threads per row (ComplexF32: per row pair), any
// number of groups per block; a row is one padded shared-memory line.
template <typename C, int P>
__global__ void __launch_bounds__(256) k_xfwd_mx(const XfParams<C> p) {
  using V = typename MxElem<C>::V;
  constexpr int TPB = MxPlan<P, MXK_XY>::s.tpb, LS = mx_line_len<P, MXK_XY>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pass_begin();
  const int l = (int)threadIdx.x / TPB, j0 = (int)threadIdx.x % TPB;
  V* const sm = reinterpret_cast<V*>(smem_raw) + l * LS;
  const int nin = p.nin;
  const int64_t u = (int64_t)blockIdx.x * p.M + l;
  auto ld = [=](int i) -> V { return mx_ldg(sm + mx_pad<P, MXK_XY>(i)); };
  auto st = [=](int i, V v) { mx_st(sm + mx_pad<P, MXK_XY>(i), v); };
  if constexpr (sizeof(C) == 16) {
    const bool ok = u < p.rows;
    const C* const src = p.in + u * nin;
    C* const dst = p.A + u * P;
    mx_line<V, P, MXK_XY, TPB, false>(
        j0, p.tw, [=](int i) -> V { return ok && i < nin ? src[i] : vzero<V>(); },
        [=](int i, V v) {
          if (ok) dst[i] = v;
        },
        ld, st);
  } else {
    const bool ok0 = 2 * u < p.rows, ok1 = 2 * u + 1 < p.rows;
    const C* const src = p.in + 2 * u * nin;
    C* const dst = p.A + 2 * u * P;
    mx_line<V, P, MXK_XY, TPB, false>(
        j0, p.tw,
        [=](int i) -> V {
          const C z = float2{0.f, 0.f};
          return F2x2{ok0 && i < nin ? src[i] : z, ok1 && i < nin ? src[nin + i] : z};
        },
        [=](int i, V v) {
          if (ok0) dst[i] = v.a;
          if (ok1) dst[P + i] = v.b;
        },
        ld, st);
  }
}

// SCAT: target partitions interleaved into the full target volume (its index
// arithmetic in the common form cost 20% of the pass)
template <typename C, int P, bool SCAT>
__global__ void __launch_bounds__(256) k_xinv_mx(const __grid_constant__ XiParams<C> p, const int axpby) {
  using V = typename MxElem<C>::V;
  constexpr int TPB = MxPlan<P, MXK_XY>::s.tpb, LS = mx_line_len<P, MXK_XY>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pass_begin();
  const int l = (int)threadIdx.x / TPB, j0 = (int)threadIdx.x % TPB;
  V* const sm = reinterpret_cast<V*>(smem_raw) + l * LS;
  const int nout = p.nout, ls = p.ls;
  const int64_t u = (int64_t)blockIdx.x * p.M + l;
  C* const out = p.out;
  const C alpha = p.alpha, beta = p.beta;
  const C *const ls_in = p.ls_in, *const ls_chi = p.ls_chi;
  const int64_t ls_chi_rs = p.ls_chi_rs, rows = p.rows, g_off = p.g_off;
  const FDiv rows_rhs = p.rows_rhs, rows_zy = p.rows_zy;
  const XiParams<C>* const pp = &p;
  auto put = [=](int64_t g, int i, C v) {
    if (g >= rows || i >= nout) return;
    const int64_t gg = g + g_off;
    int64_t o = gg * nout + i;
    if constexpr (SCAT) {
      // gg = ((rhs*parT + t)*3 + c)*tz + z)*ty + y (mrgPrtDev!)
      int64_t q = gg;
      const int y = (int)(q % pp->ty);
      q /= pp->ty;
      const int z = (int)(q % pp->tz);
      q /= pp->tz;
      const int c = (int)(q % 3);
      q /= 3;
      const int t = (int)(q % pp->parT);
      const int64_t rhs = q / pp->parT;
      const int64_t X = (int64_t)i * pp->tdiv[0] + pp->toff[t][0], Y = (int64_t)y * pp->tdiv[1] + pp->toff[t][1],
                    Zz = (int64_t)z * pp->tdiv[2] + pp->toff[t][2];
      o = (((rhs * 3 + c) * pp->full[2] + Zz) * pp->full[1] + Y) * pp->full[0] + X;
    }
    if (axpby)
      out[o] = cadd(cmul(alpha, v), cmul(beta, out[o]));
    else if (ls)
      out[o] = ls_value(ls_in, ls_chi, ls_chi_rs, rows_rhs, rows_zy, nout, gg, i, o, v);
    else
      out[o] = v;
  };
  auto ld = [=](int i) -> V { return mx_ldg(sm + mx_pad<P, MXK_XY>(i)); };
  auto st = [=](int i, V v) { mx_st(sm + mx_pad<P, MXK_XY>(i), v); };
  if constexpr (sizeof(C) == 16) {
    const bool ok = u < rows;
    const C* const src = p.A + u * P;
    mx_line<V, P, MXK_XY, TPB, true>(
        j0, p.tw, [=](int i) -> V { return ok ? src[i] : vzero<V>(); }, [=](int i, V v) { put(u, i, v); }, ld, st);
  } else {
    const bool ok0 = 2 * u < rows, ok1 = 2 * u + 1 < rows;
    const C* const src = p.A + 2 * u * P;
    mx_line<V, P, MXK_XY, TPB, true>(
        j0, p.tw,
        [=](int i) -> V {
          const C z = float2{0.f, 0.f};
          return F2x2{ok0 ? src[i] : z, ok1 ? src[P + i] : z};
        },
        [=](int i, V v) {
          put(2 * u, i, v.a);
          put(2 * u + 1, i, v.b);
        },
        ld, st);
  }
}

// -------------------------------------------------------------------- y
// A unit is a tile of 8 elements along kx (128 bytes) of one plane; small
// lengths put several units in a block.
constexpr int kMxTX = 8;
template <int P> constexpr int mx_y_units() {
  const int t = kMxTX * MxPlan<P, MXK_XY>::s.tpb;
  return t >= 96 ? 1 : 96 / t;
}
template <int P> constexpr int mx_y_threads() { return mx_y_units<P>() * kMxTX * MxPlan<P, MXK_XY>::s.tpb; }

template <typename C, int P, bool INV>
__global__ void __launch_bounds__(mx_y_threads<P>(), mx_blocks(mx_y_threads<P>(), kMxRegs))
    k_y_mx(const YParams<C> p, const uint32_t units) {
  using V = typename MxElem<C>::V;
  constexpr int TX = kMxTX, CW = 16 / sizeof(C), TPB = MxPlan<P, MXK_XY>::s.tpb, NU = mx_y_units<P>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pass_begin();
  const int t = (int)threadIdx.x % TX, q = (int)threadIdx.x / TX, j0 = q % TPB, un = q / TPB;
  V* const sm = reinterpret_cast<V*>(smem_raw) + un * (P * TX) + t;
  const int Px = p.Px, nin = p.nin, nout = p.nout;
  uint32_t u = blockIdx.x * (uint32_t)NU + un;
  const bool live = NU == 1 || u < units;
  if (!live) u = 0;
  const uint32_t ut = u / (uint32_t)p.nt;
  const int tl = (int)(u - ut * p.nt);  // tile of the kx set: low range, then high range
  const int tile = tl < p.nlo ? p.lo0 + tl : p.hi0 + (tl - p.nlo);
  const uint32_t slice = (uint32_t)p.q0 + ut;  // ch*nz + z (below 2^31, checked at the launch)
  const int64_t rc = slice / (uint32_t)p.nz;
  const int z = (int)(slice - (uint32_t)rc * p.nz);
  const int kx = (tile * TX + t) * CW;
  const bool ok = live && kx < Px;  // Px is even: a line pair is whole
  const C* const src = p.src + ((rc * p.src_z + z) - p.src_sub) * p.src_rows * (int64_t)Px + kx;
  C* const dst = p.dst + ((rc * p.dst_z + z) - p.dst_sub) * p.dst_rows * (int64_t)Px + kx;
  mx_line<V, P, MXK_XY, TPB, INV>(
      j0, p.tw,
      [=](int i) -> V {
        return ok && i < nin ? mx_ldg(reinterpret_cast<const V*>(src + (int64_t)i * Px)) : vzero<V>();
      },
      [=](int i, V v) {
        if (ok && i < nout) mx_st(reinterpret_cast<V*>(dst + (int64_t)i * Px), v);
      },
      [=](int i) -> V { return mx_ldg(sm + i * TX); }, [=](int i, V v) { mx_st(sm + i * TX, v); });
}

// -------------------------------------------------------------------- z
// kx elements per tile: 128-byte rows while three components' lines leave
// room for two blocks or more per SM, else half of that
template <int P> constexpr int mx_z_tx() { return P <= 192 ? 8 : 4; }
// z lines of a tile in shared memory: rows of TX elements, at tiles of 4 padded
// like an x line (two rows share a quarter-warp's banks)
template <int P> GILA_HD int mx_z_row(int i) { return mx_z_tx<P>() == 8 ? i : mx_pad<P, MXK_Z>(i); }
template <int P> constexpr int mx_z_rows() { return mx_z_tx<P>() == 8 ? P : mx_line_len<P, MXK_Z>(); }
template <int P> constexpr int mx_z_threads() { return 3 * mx_z_tx<P>() * MxPlan<P, MXK_Z>::s.tpb; }

// the 3x3 products of one frequency of an element's column(s)
template <typename C> struct MxKer;
template <> struct MxKer<double2> {
  double2 g[6];
  int rz;
};
template <> struct MxKer<float2> {
  float2 a[6], b[6];
  int rz;
};
// an element's columns on the x axis of the stored kernel
struct MxCol {
  int px, ix, rx, pxb, ixb, rxb, adj;
};

template <typename C, int P>
__global__ void __launch_bounds__(mx_z_threads<P>(), mx_blocks(mx_z_threads<P>(), mx_z_regs<P>()))
    k_z_mx(const ZParams<C> p) {
  using V = typename MxElem<C>::V;
  using W = C;
  using T = typename MxOf<V>::T;
  using Plan = MxPlan<P, MXK_Z>;
  constexpr int TX = mx_z_tx<P>(), CW = 16 / sizeof(C), TPB = Plan::s.tpb, N = Plan::s.n;
  constexpr int RL = mx_r<P, MXK_Z, false>(N - 1), TPL = P / RL, NJ = 3 * TPB, KF = (TPL + NJ - 1) / NJ;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  pass_begin();
  const int t = (int)threadIdx.x % TX, q = (int)threadIdx.x / TX, c = q / TPB, j0 = q % TPB;
  V* const smt = reinterpret_cast<V*>(smem_raw) + t;  // [c][z][t]
  constexpr int ZR = mx_z_rows<P>();
  V* const smc = smt + c * (ZR * TX);
  const int nrhs = p.nrhs, Px = p.Px, Py = p.Py, nin = p.nin, nout = p.nout;
  const int rhs = blockIdx.x % nrhs;
  const int rest = blockIdx.x / nrhs;
  const int tseq = p.ts0 + rest % p.nts;  // [ts0, ts0 + nts) of the mirror tile order
  const int yseq = rest / p.nts;
  const int kx = (tile_seq(tseq, p.ntiles) * TX + t) * CW;
  const int ky = mirror_seq(yseq, Py);
  const bool ok = kx < Px;
  const int64_t plane = (int64_t)Py * Px;
  C* const Bb = p.B + (int64_t)rhs * 3 * p.zb * plane + (int64_t)ky * Px + kx;
  const W* const tw = p.tw;
  auto ld = [=](int i) -> V { return mx_ldg(smc + mx_z_row<P>(i) * TX); };
  auto st = [=](int i, V v) { mx_st(smc + mx_z_row<P>(i) * TX, v); };
  auto sync = [] { __syncthreads(); };
  auto none = [] {};
  {
    const C* const src = Bb + (int64_t)c * nin * plane;
    auto gld = [=](int i) -> V {
      return ok && i < nin ? mx_ldcs(reinterpret_cast<const V*>(src + (int64_t)i * plane)) : vzero<V>();
    };
    if constexpr (N > 1) {
      mx_stage<V, P, MXK_Z, 0, TPB, false, false>(j0, tw, gld, st, none);
    } else {  // one stage: the fused one
#pragma unroll
      for (int i = 0; i < P; ++i) st(i, gld(i));
    }
  }
  int py, iy, ry;
  ax_map(p.ax[1], ky + p.ky0, py, iy, ry);
  const int tx = p.tx, ty = p.ty, tz = p.tz;
  const T s = (T)p.scale;
  MxCol col{};
  if (ok) {
    ax_map(p.ax[0], kx, col.px, col.ix, col.rx);
    if constexpr (CW == 2) {
      ax_map(p.ax[0], kx + 1, col.pxb, col.ixb, col.rxb);
      // the even and odd x parity of one unmirrored stored index are
      // adjacent (one 16-byte load per component), mirrored ones are not
      col.adj = col.ix == col.ixb;
    }
  }
  auto kload = [&](int f) -> MxKer<C> {
    MxKer<C> k;
    int pz, iz;
    ax_map(p.ax[2], f, pz, iz, k.rz);
    const C* const ga = ker_at(p.ker, 4 * col.px + 2 * py + pz, iz, iy, col.ix, tx, ty, tz);
    if constexpr (CW == 1) {
#pragma unroll
      for (int e = 0; e < 6; ++e) k.g[e] = ker_ld(ga, e, tx);
    } else if (col.adj) {
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(ga + 2 * e * tx));
        k.a[e] = make_float2(v.x, v.y);
        k.b[e] = make_float2(v.z, v.w);
      }
    } else {
      const C* const gb = ker_at(p.ker, 4 * col.pxb + 2 * py + pz, iz, iy, col.ixb, tx, ty, tz);
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        k.a[e] = ker_ld(ga, e, tx);
        k.b[e] = ker_ld(gb, e, tx);
      }
    }
    return k;
  };
  __syncthreads();
  if constexpr (N > 2) {
    mx_stage<V, P, MXK_Z, 1, TPB, false, false>(j0, tw, ld, st, sync);
    __syncthreads();
  }
  if constexpr (N > 3) {
    mx_stage<V, P, MXK_Z, 2, TPB, false, false>(j0, tw, ld, st, sync);
    __syncthreads();
  }
  if constexpr (N > 4) {
    mx_stage<V, P, MXK_Z, 3, TPB, false, false>(j0, tw, ld, st, sync);
    __syncthreads();
  }
  // last forward stage, multiply and first inverse stage on the same
  // registers: task j holds frequencies j + r P/RL of all three components,
  // and its inverse outputs j RL + r go back to the slots it read
#pragma unroll 1
  for (int k = 0; k < KF; ++k) {
    const int j = q + k * NJ;
    if (j >= TPL || !ok) break;
    constexpr bool AHEAD = mx_z_ahead(sizeof(C), P);
    MxKer<C> g;
    if constexpr (AHEAD) g = kload(j);
    V v[3][RL];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int r = 0; r < RL; ++r) v[d][r] = mx_ldg(smt + (d * ZR + mx_z_row<P>(j + r * TPL)) * TX);
    {
      W w[RL];
      if constexpr (N > 1) mx_twiddles<RL, TPL, false>(tw + MxTw<P, MXK_Z, false, N - 1>::off + j, w);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        if constexpr (N > 1) {
#pragma unroll
          for (int r = 1; r < RL; ++r) v[d][r] = vmul(v[d][r], w[r]);
        }
        Dft<RL, false>::run(v[d]);
      }
    }
#pragma unroll
    for (int r = 0; r < RL; ++r) {
      MxKer<C> gn;
      if constexpr (AHEAD) {
        if (r + 1 < RL) gn = kload(j + (r + 1) * TPL);
      } else {
        g = kload(j + r * TPL);
      }
      if constexpr (CW == 1) {
        zmul3f(v[0][r], v[1][r], v[2][r], g.g, col.rx, ry, g.rz, s);
      } else {
        zmul3f(v[0][r].a, v[1][r].a, v[2][r].a, g.a, col.rx, ry, g.rz, s);
        zmul3f(v[0][r].b, v[1][r].b, v[2][r].b, g.b, col.rxb, ry, g.rz, s);
      }
      if constexpr (AHEAD) {
        if (r + 1 < RL) g = gn;
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      Dft<RL, true>::run(v[d]);
#pragma unroll
      for (int r = 0; r < RL; ++r) mx_st(smt + (d * ZR + mx_z_row<P>(j + r * TPL)) * TX, v[d][r]);
    }
  }
  __syncthreads();
  // inverse stages in reversed order; the first reads through the fused
  // stage's permutation (input i in slot i / RL + (i % RL) P / RL)
  C* const dst = Bb + (int64_t)c * nout * plane;
  auto ldp = [=](int i) -> V { return mx_ldg(smc + mx_z_row<P>((i / RL) + (i % RL) * TPL) * TX); };
  auto gst = [=](int i, V v) {
    if (ok && i < nout) mx_st(reinterpret_cast<V*>(dst + (int64_t)i * plane), v);
  };
  if constexpr (N == 1) {
#pragma unroll
    for (int i = 0; i < P; ++i) gst(i, ldp(i));
  } else if constexpr (N == 2) {
    mx_stage<V, P, MXK_Z, 1, TPB, true, true>(j0, tw, ldp, gst, none);
  } else {
    mx_stage<V, P, MXK_Z, 1, TPB, true, true>(j0, tw, ldp, st, sync);
    __syncthreads();
    if constexpr (N > 3) {
      mx_stage<V, P, MXK_Z, 2, TPB, true, true>(j0, tw, ld, st, sync);
      __syncthreads();
    }
    if constexpr (N > 4) {
      mx_stage<V, P, MXK_Z, 3, TPB, true, true>(j0, tw, ld, st, sync);
      __syncthreads();
    }
    mx_stage<V, P, MXK_Z, N - 1, TPB, true, true>(j0, tw, ld, gst, none);
  }
}

// ------------------------------------------------------------- launchers
static inline cudaError_t mx_smem(const void* fn, size_t bytes) {
  if (bytes > 48 * 1024) return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  return cudaSuccess;
}

// rows (row pairs) per block of an x pass: about 192 threads, fewer where
// the blocks would not fill the SMs twice
constexpr int mx_x_most(int tpb) { return 192 / tpb < 1 ? 1 : 192 / tpb; }
static inline int mx_x_rows(int tpb, int64_t units) {
  int m = mx_x_most(tpb);
  while (m > 1 && m * tpb > 32 && (units + m - 1) / m < 2 * 148) m = (m + 1) / 2;
  return m;
}

template <typename C, int P>
struct MxLaunch {
  static constexpr int CW = 16 / (int)sizeof(C), LS = mx_line_len<P, MXK_XY>();
  static constexpr int XTPB = MxPlan<P, MXK_XY>::s.tpb;

  static cudaError_t xfwd(const XfParams<C>& p0, cudaStream_t st) {
    XfParams<C> p = p0;
    const int64_t units = (p.rows + CW - 1) / CW;
    p.M = mx_x_rows(XTPB, units);
    const size_t sm = (size_t)p.M * LS * 16;
    cudaError_t e = mx_smem((const void*)k_xfwd_mx<C, P>, sm);
    if (e != cudaSuccess) return e;
    return launch_pass(k_xfwd_mx<C, P>, (unsigned)((units + p.M - 1) / p.M), p.M * XTPB, sm, st, p);
  }
  static cudaError_t xinv(const XiParams<C>& p0, bool axpby, cudaStream_t st) {
    XiParams<C> p = p0;
    const int64_t units = (p.rows + CW - 1) / CW;
    p.M = mx_x_rows(XTPB, units);
    const size_t sm = (size_t)p.M * LS * 16;
    const unsigned blocks = (unsigned)((units + p.M - 1) / p.M);
    cudaError_t e = mx_smem(p.part_scatter ? (const void*)k_xinv_mx<C, P, true> : (const void*)k_xinv_mx<C, P, false>, sm);
    if (e != cudaSuccess) return e;
    return p.part_scatter ? launch_pass(k_xinv_mx<C, P, true>, blocks, p.M * XTPB, sm, st, p, axpby ? 1 : 0)
                          : launch_pass(k_xinv_mx<C, P, false>, blocks, p.M * XTPB, sm, st, p, axpby ? 1 : 0);
  }
  template <bool INV>
  static cudaError_t y_one(const YParams<C>& p, int64_t units, cudaStream_t st) {
    constexpr int NU = mx_y_units<P>();
    if (units + NU > INT32_MAX || p.q0 + units / p.nt > INT32_MAX) return cudaErrorInvalidValue;
    const size_t sm = (size_t)NU * P * kMxTX * 16;
    cudaError_t e = mx_smem((const void*)k_y_mx<C, P, INV>, sm);
    if (e != cudaSuccess) return e;
    return launch_pass(k_y_mx<C, P, INV>, (unsigned)((units + NU - 1) / NU), mx_y_threads<P>(), sm, st, p,
                       (uint32_t)units);
  }
  static cudaError_t y(const YParams<C>& p, bool inv, int64_t units, cudaStream_t st) {
    return inv ? y_one<true>(p, units, st) : y_one<false>(p, units, st);
  }
  static cudaError_t z(const ZParams<C>& p, int64_t blocks, cudaStream_t st) {
    const size_t sm = (size_t)3 * mx_z_rows<P>() * mx_z_tx<P>() * 16;
    cudaError_t e = mx_smem((const void*)k_z_mx<C, P>, sm);
    if (e != cudaSuccess) return e;
    return launch_pass(k_z_mx<C, P>, (unsigned)blocks, mx_z_threads<P>(), sm, st, p);
  }
  // launches that the dispatch can reach: at 96, 192 and 384 the x and y
  // passes, at 64 the ComplexF32 z pass; every pass elsewhere
  static constexpr bool XY = P != 64, Z = P == 64 ? sizeof(C) == 8 : !(P == 96 || P == 192 || P == 384);
  static constexpr auto xfwd_fn() -> decltype(&xfwd) {
    if constexpr (XY) return &xfwd;
    return nullptr;
  }
  static constexpr auto xinv_fn() -> decltype(&xinv) {
    if constexpr (XY) return &xinv;
    return nullptr;
  }
  static constexpr auto y_fn() -> decltype(&y) {
    if constexpr (XY) return &y;
    return nullptr;
  }
  static constexpr auto z_fn() -> decltype(&z) {
    if constexpr (Z) return &z;
    return nullptr;
  }
  static constexpr MxOps<C> ops{P, kMxTX * CW, mx_z_tx<P>() * CW, xfwd_fn(), xinv_fn(), y_fn(), z_fn()};
};

template <typename C, int... P>
static const MxOps<C>* mx_find(int n) {
  static constexpr const MxOps<C>* t[] = {&MxLaunch<C, P>::ops...};
  for (const MxOps<C>* o : t)
    if (o->P == n) return o;
  return nullptr;
}
// one translation unit's share of the lengths
#define GILA_MX_PART(K, ...)                                                                                  \
  template <> const MxOps<double2>* mx_part<double2, K>(int n) { return mx_find<double2, __VA_ARGS__>(n); } \
  template <> const MxOps<float2>* mx_part<float2, K>(int n) { return mx_find<float2, __VA_ARGS__>(n); }

}  // namespace gila
