// FP64 tensor-core (DMMA) tile engine of the persistent FP64 kernels: tile shapes, the TMA
// operand stages, the multiply of one k-block and the fragment-to-element map.
#pragma once
#include <cstdint>

#include "f64_dmma.cuh"
#include "tc_ptx.cuh"

namespace sp2b {

// A BT x BT tile of A^T B by NW consumer warps (WM x WN), each owning a TM x TN block of
// m8n8k4 fragments; one more warp loads.  Operand tiles are rows of the symmetric inputs,
// As[k][m] = A[k0+k][i0+m] and Bs[k][n] = B[k0+k][j0+n], in k-blocks of 16.  Sixteen warps
// (edges 64 and 128) put four on each scheduler of an SM that holds one CTA: an m8n8k4
// issues every 16 cycles and returns after 32, and four warps also cover each other's waits
// and fragment loads.  (Two CTAs of eight warps did not: the scheduler favours one, which
// then waits at the step's end while the other runs alone, 17 % of the time at n = 2000.)
//
// A k-block of an operand is one TMA box: the matrix seen as [ld/16][rows][16 doubles], box
// 16 doubles x 16 rows x BT/16 column groups, 128-byte swizzle.  The eight columns of a
// fragment are taken in pairs, 0 1, 8 9, 2 3, 10 11 of a group of sixteen (the odd fragment
// 4 5, 12 13, 6 7, 14 15): under that swizzle the sixteen 8-byte words that a half-warp
// loads (four k rows, four columns) then lie in distinct banks, and k stays ascending.
// Full / empty mbarriers instead of a block barrier per k-block let the warps drift:
// with __syncthreads they waited there a fifth of the time.
template <int BT>
struct F64Tile {
  static constexpr int BK = 16;
  static constexpr int WM = BT == 32 ? 2 : 4, WN = 4, NW = WM * WN, NT = NW * 32;
  static constexpr int ST = BT == 128 ? 6 : 8;
  static constexpr int TM = BT / WM, TN = BT / WN, MI = TM / 8, NI = TN / 8;
  static constexpr bool EARLY_E = BT == 32;   // registers for the epilogue's operand
  static constexpr int OPERAND = BT * BK * 8, STAGE = 2 * OPERAND;   // bytes
  static constexpr size_t SMEM = (size_t)ST * STAGE + 1024;

  // Column (of the group of sixteen) of index j in an even fragment.
  static __device__ __forceinline__ int perm(int j) {
    return 2 * ((j >> 2) + 4 * ((j >> 1) & 1)) + (j & 1);
  }
  // This lane's byte offsets inside an operand's k-block.
  struct Frag {
    uint32_t off[2];   // k step parity
    __device__ __forceinline__ void init(int lane) {
      const int m = perm(lane >> 2);
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int r = 4 * p + (lane & 3);   // k row modulo 8
        off[p] = (uint32_t)(r * 128 + (((m >> 1) ^ r) << 4) + (m & 1) * 8);
      }
    }
    // address in the operand at `base` of fragment c8 (a multiple of eight columns), k step s
    __device__ __forceinline__ uint32_t at(uint32_t base, int c8, int s) const {
      return (base + (c8 >> 1) * (BK * 128) + (s >> 1) * 1024 + off[s & 1]) ^
             (uint32_t)((c8 & 1) << 5);
    }
  };
  static __device__ __forceinline__ double lds(uint32_t a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
  }

  // One k-block from the operands at abase / bbase (this warp's first fragments am8, bn8);
  // below edge 128 (registers) the next k step's fragments load while the current multiply.
  static __device__ __forceinline__ void mma(uint32_t abase, uint32_t bbase, int am8, int bn8,
                                             const Frag& f, double (&acc)[MI][NI][2]) {
    constexpr int NB = BT == 128 ? 1 : 2;
    double a[NB][MI], b[NB][NI];
    auto fetch = [&](int s, double (&av)[MI], double (&bv)[NI]) {
#pragma unroll
      for (int mi = 0; mi < MI; ++mi) av[mi] = lds(f.at(abase, am8 + mi, s));
#pragma unroll
      for (int ni = 0; ni < NI; ++ni) bv[ni] = lds(f.at(bbase, bn8 + ni, s));
    };
    if (NB == 2) fetch(0, a[0], b[0]);
#pragma unroll
    for (int s = 0; s < BK / 4; ++s) {
      if (NB == 1) fetch(s, a[0], b[0]);
      else if (s + 1 < BK / 4) fetch(s + 1, a[(s + 1) % NB], b[(s + 1) % NB]);
#pragma unroll
      for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < NI; ++ni) dmma884(acc[mi][ni], a[s % NB][mi], b[s % NB][ni]);
    }
  }

  // Row and first column (of two adjacent ones) of this consumer thread's fragment (mi, ni)
  // in the tile.
  static __device__ __forceinline__ int place(int c8, int j) {
    return (c8 >> 1) * 16 + (c8 & 1) * 4 + perm(j);
  }
  static __device__ __forceinline__ int row(int mi) {
    return place((int)(threadIdx.x >> 5) / WN * MI + mi, (int)(threadIdx.x & 31) >> 2);
  }
  static __device__ __forceinline__ int col(int ni) {
    return place((int)(threadIdx.x >> 5) % WN * NI + ni, 2 * (int)(threadIdx.x & 3));
  }
};

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* tm) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tm)) : "memory");
}
// Adds one to a counter after everything this thread has done or seen (gpu scope).
__device__ __forceinline__ void add_release(unsigned* word) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(word) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* tm, uint32_t mbar,
                                            int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(mbar), "r"(x), "r"(y), "r"(z)
      : "memory");
}

// Tensor map of a rows x ld FP64 array (ld a multiple of 16) for F64Tile<bt> boxes.
static inline bool make_tmap_f64(CUtensorMap* tm, const double* base, long long rows, long long ld,
                                 int bt) {
  auto fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {16, (cuuint64_t)rows, (cuuint64_t)(ld / 16)};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 8, 128};
  cuuint32_t box[3] = {16, 16, (cuuint32_t)(bt / 16)};
  cuuint32_t es[3] = {1, 1, 1};
  return fn(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double*>(base), dims, strides, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace sp2b
