// matvec_mx.cuh -- the mixed-radix passes: launch table by transform length.
//
// Every even length 2^a 3^b 5^c 7^d from 4 to 512 that fft_ct.cuh does not
// specialise has compile-time kernels here (matvec_mx_impl.cuh), 96, 192 and 384
// the x and y ones, 64 the ComplexF32 z one; longer lengths and the z pass of
// target partitions keep the runtime-planned kernels.
#pragma once
#include "passes.cuh"

namespace gila {

// Launches of one length's kernels; `units` counts the rows (x), kx tiles
// times planes (y) or blocks (z) of the launch.
template <typename C>
struct MxOps {
  int P;
  int y_tx, z_tx;  // kx columns per tile of the y and z passes
  // null where the tuned kernels are the faster: x and y at 64, z at 96, 192,
  // 384 and in ComplexF64 at 64
  cudaError_t (*xfwd)(const XfParams<C>&, cudaStream_t);
  cudaError_t (*xinv)(const XiParams<C>&, bool axpby, cudaStream_t);
  cudaError_t (*y)(const YParams<C>&, bool inv, int64_t units, cudaStream_t);
  cudaError_t (*z)(const ZParams<C>&, int64_t blocks, cudaStream_t);
};

// the length's launches, or nullptr where it has none; the lengths are spread
// over kMxParts translation units, which compile in parallel
constexpr int kMxParts = 8;
template <typename C, int PART>
const MxOps<C>* mx_part(int P);
constexpr int kMxMaxLen = 512;
template <typename C>
inline const MxOps<C>* mx_ops(int P) {
  struct Table {
    const MxOps<C>* t[kMxMaxLen + 1];
    Table() {
      for (int n = 0; n <= kMxMaxLen; ++n) {
        const MxOps<C>* const o[kMxParts] = {mx_part<C, 0>(n), mx_part<C, 1>(n), mx_part<C, 2>(n), mx_part<C, 3>(n),
                                             mx_part<C, 4>(n), mx_part<C, 5>(n), mx_part<C, 6>(n), mx_part<C, 7>(n)};
        t[n] = nullptr;
        for (const MxOps<C>* q : o)
          if (q) t[n] = q;
      }
    }
  };
  static const Table tab;
  return P >= 0 && P <= kMxMaxLen ? tab.t[P] : nullptr;
}

}  // namespace gila
