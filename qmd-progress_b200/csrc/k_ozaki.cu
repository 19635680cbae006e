// Exact symmetric products on the INT8 tensor cores (tcgen05 kind::i8) for the FP64
// McWeeny refinement that ends a split-precision solve.
//
// The iterate X (symmetric, near-idempotent) is rounded to the integer matrix
// M = rint(2^S X) and held as its residues modulo nine pairwise-coprime moduli m_t <= 256
// (signed 8-bit planes R_t).  Each plane product P_t = R_t R_t is exact in the 32-bit
// accumulators (|r| <= 128, K <= 65536) and is reduced mod m_t in the epilogue.  The
// Chinese remainder theorem, in Garner's mixed-radix form evaluated by Horner's rule in
// FP64, then rebuilds (M M)_ij exactly whenever |(M M)_ij| < prod(m_t)/2.  By
// Cauchy-Schwarz |(M M)_ij| <= max_i ||M_i||^2, so S is chosen from the largest row norm of
// X.  X^2 = 2^-2S M M carries only the rounding of X to the 2^-S grid (S ~ 35 for a
// density matrix), far below the 1e-10 target of the FP64 path, at 9 INT8 products in
// place of one FP64 product.  This is the residue-number-system form of the Ozaki scheme
// (Ozaki, Uchino and Imamura, "Ozaki Scheme II: A GEMM-oriented emulation of
// floating-point matrix multiplication using an integer modular technique", 2025).
#include <algorithm>
#include <atomic>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "reduce.cuh"
#include "tc_ptx.cuh"
#include "work_lists.h"

namespace sp2b {
namespace oz {

constexpr int T = 9;  // number of moduli
// Moduli in Garner order; the even modulus 256 is last, so the sign of a residue vector
// (whether Y >= prod/2) is the top bit of the last mixed-radix digit.
__host__ __device__ constexpr int mod(int t) {
  return t == 0 ? 255 : t == 1 ? 253 : t == 2 ? 251 : t == 3 ? 247 : t == 4 ? 241
       : t == 5 ? 239 : t == 6 ? 233 : t == 7 ? 229 : 256;
}
// a^-1 mod m (gcd(a, m) = 1), extended Euclid.
__host__ __device__ constexpr int inv_mod(int a, int m) {
  int t = 0, nt = 1, r = m, nr = a % m;
  while (nr != 0) {
    const int q = r / nr;
    int tmp = t - q * nt;
    t = nt;
    nt = tmp;
    tmp = r - q * nr;
    r = nr;
    nr = tmp;
  }
  return t < 0 ? t + m : t;
}
__host__ __device__ constexpr int pow2_mod(int e, int m) {
  int v = 1 % m;
  for (int i = 0; i < e; ++i) v = (v * 2) % m;
  return v;
}
// prod(m_t) / 2 = 2^70.41; the CRT is exact for |Y| below it.
__host__ __device__ inline double half_prod() {
  double p = 0.5;
  for (int t = 0; t < T; ++t) p *= (double)mod(t);
  return p;
}

// Tile edges of the INT8 product: 128 rows x 256 columns, K in 128-byte blocks.
constexpr int BM = 128, BN = 256, BK = 128, UK = 32, ST = 4;
constexpr int A_BYTES = BM * BK, B_BYTES = BN * BK;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int SMEM_BYTES = ST * STAGE_BYTES + 1024;
constexpr int NWARP = 10, NTHR = NWARP * 32, EPI_WARPS = 8;
constexpr int TMEM_COLS = 2 * BN;
}  // namespace oz

// Scale state shared by the kernels of one refinement: the largest squared row norm
// (as the bits of a non-negative double, for atomicMax) and the chosen exponent S.
struct OzScale {
  unsigned long long r2max_bits;
  int S;      // -1: no valid scale (non-finite input)
  int kept;   // exact steps: the planes of X_k were formed with this S by the step before
};

// SP2-step context of the launches that compute one step's X^2 (the exact INT8 mode):
// they do nothing once the loop has finished or when this step's rule says stop, which
// the step's last launch (k_oz_crt_step) would decide from the same record.
__device__ __forceinline__ bool oz_skip(const OzStepCtl& c) {
  if (!c.active) return false;
  if (*(volatile const int*)&c.sout->done) return true;
  const SP2Rec r = c.rec[c.k];
  if (r.done) return true;
  return sp2_decide(c.ctl, r, c.k, c.pp_in).branch == BR_STOP;
}

template <typename T>
struct OzSplit;
template <>
struct OzSplit<__half> {
  static constexpr double kInv = 1.0 / 2048.0, kScale = 2048.0;
  __device__ static double d(__half h) { return (double)__half2float(h); }
  __device__ static __half from_d(double v) { return __double2half(v); }
};
template <>
struct OzSplit<__nv_bfloat16> {
  static constexpr double kInv = 1.0 / 256.0, kScale = 256.0;
  __device__ static double d(__nv_bfloat16 h) { return (double)__bfloat162float(h); }
  __device__ static __nv_bfloat16 from_d(double v) { return __double2bfloat16(v); }
};

// ---------------------------------------------------------------------------------
// 1. Largest squared row norm of X = hi + 2^-s lo (one warp per row).
// ---------------------------------------------------------------------------------
template <typename T>
__global__ void k_oz_rownorm(const T* __restrict__ hi, const T* __restrict__ lo, int np,
                             OzScale* sc) {
  using SP = OzSplit<T>;
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  double best = 0.0;
  for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < np; row += gridDim.x * wpb) {
    const T* h = hi + (size_t)row * np;
    const T* l = lo + (size_t)row * np;
    double s = 0.0;
    for (int c = lane * 8; c < np; c += 256) {
      alignas(16) T hv[8], lv[8];
      *reinterpret_cast<uint4*>(hv) = *reinterpret_cast<const uint4*>(h + c);
      *reinterpret_cast<uint4*>(lv) = *reinterpret_cast<const uint4*>(l + c);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const double x = fma(SP::kInv, SP::d(lv[q]), SP::d(hv[q]));
        s = fma(x, x, s);
      }
    }
    s = warp_sum(s);
    // NaN propagates as a maximum: its bit pattern is above every finite value
    if (!(s <= best)) best = s;
  }
  if (lane == 0) {
    unsigned long long b = (unsigned long long)__double_as_longlong(best);
    if (best != best) b = 0x7ff8000000000000ull;
    atomicMax(&sc->r2max_bits, b);
  }
}

// The same for an FP64 iterate (exact INT8 mode).
__global__ void k_oz_rownorm_f64(const double* __restrict__ x, int np, OzScale* sc,
                                 const OzStepCtl c) {
  if (oz_skip(c)) return;
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  double best = 0.0;
  for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < np; row += gridDim.x * wpb) {
    const double2* xr = reinterpret_cast<const double2*>(x + (size_t)row * np);
    double s = 0.0;
    for (int c = lane; c < np / 2; c += 32) {
      const double2 v = xr[c];
      s = fma(v.x, v.x, s);
      s = fma(v.y, v.y, s);
    }
    s = warp_sum(s);
    if (!(s <= best)) best = s;
  }
  if (lane == 0) {
    unsigned long long b = (unsigned long long)__double_as_longlong(best);
    if (best != best) b = 0x7ff8000000000000ull;
    atomicMax(&sc->r2max_bits, b);
  }
}

// S: the largest exponent with (2^S sqrt(r2max) + sqrt(np)/2)^2 < prod/2, which bounds
// every |(M M)_ij| (row norms of M are at most 2^S ||x_i|| + sqrt(np)/2).
__device__ __forceinline__ int oz_choose_scale(double r2, int np) {
  int S = -1;
  if (r2 == r2 && r2 < 1e300) {
    const double lim = sqrt(oz::half_prod()) * (1.0 - 1e-12);
    const double r = sqrt(r2);
    const double e = 0.5 * sqrt((double)np);
    S = 200;
    if (r > 0.0) {
      S = (int)floor(log2((lim - e) / r));
      if (S > 200) S = 200;
      while (S > -1 && ldexp(r, S) + e >= lim) --S;
    }
  }
  return S;
}
__global__ void k_oz_scale(OzScale* sc, int np) {
  sc->S = oz_choose_scale(__longlong_as_double((long long)sc->r2max_bits), np);
}

// ---------------------------------------------------------------------------------
// 2. Residue planes: R_t = rint(2^S X) mod m_t in the symmetric range (signed 8-bit).
//    Plane t is np x np at res + t * np * np.
// ---------------------------------------------------------------------------------
// M = rint(x 2^S), |M| < sqrt(prod/2) < 2^36, as the low mantissa bits of x 2^S + 1.5 2^52 (one
// FMA rounds to nearest even, like rint): no FP64 conversion or floor instruction.  It is
// split as M = mh 2^21 + ml (0 <= ml < 2^21, |mh| < 2^15), both exact in FP32.
struct OzInt {
  float mh, ml;
  uint32_t low;   // M mod 2^32
};
__device__ __forceinline__ OzInt oz_round(double x, double scale) {
  const double t = fma(x, scale, 0x1.8p52);
  const uint32_t lo = (uint32_t)__double2loint(t);
  const int hi = __double2hiint(t) - 0x43380000;
  const int mh = (int)__funnelshift_l(lo, (uint32_t)hi, 11);
  OzInt r;
  r.mh = __int_as_float(0x4b400000 + mh) - 0x1.8p23f;
  r.ml = __int_as_float(0x4b000000 | (int)(lo & 0x1fffffu)) - 0x1p23f;
  r.low = lo;
  return r;
}
// A residue of M modulo m, any representative in [-128, 127] (the products only need
// r = M mod m).  v = mh c + ml, c = 2^21 mod m in the symmetric range, is an integer below
// 2^23 in magnitude, exact in FP32; q = v / m to the nearest integer (the FMA rounds
// v inv + 1.5 2^23 once, so q errs only within 0.001 of a tie, where either neighbour's
// residue is below 128 in magnitude), and r = v - q m is exact.  The result is the low byte
// of r + 1.5 2^23: five full-rate FP32 instructions and no conversion.
template <int t>
__device__ __forceinline__ uint32_t oz_residue(const OzInt& M) {
  constexpr int m = oz::mod(t);
  if constexpr (m == 256) {
    return M.low;
  } else {
    constexpr int c0 = oz::pow2_mod(21, m);
    constexpr float c = (float)(c0 > m / 2 ? c0 - m : c0), inv = 1.0f / (float)m;
    const float v = fmaf(M.mh, c, M.ml);
    const float q = fmaf(v, inv, 0x1.8p23f) - 0x1.8p23f;
    return (uint32_t)__float_as_int(fmaf(-q, (float)m, v) + 0x1.8p23f);
  }
}
__device__ __forceinline__ uint32_t low_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// Eight consecutive elements of every plane from plane offset off.
template <int t>
__device__ __forceinline__ void oz_store_planes(int8_t* res, size_t plane, size_t off,
                                                const OzInt (&M)[8]) {
  if constexpr (t < oz::T) {
    uint2 v;
    v.x = low_bytes(oz_residue<t>(M[0]), oz_residue<t>(M[1]), oz_residue<t>(M[2]), oz_residue<t>(M[3]));
    v.y = low_bytes(oz_residue<t>(M[4]), oz_residue<t>(M[5]), oz_residue<t>(M[6]), oz_residue<t>(M[7]));
    *reinterpret_cast<uint2*>(res + (size_t)t * plane + off) = v;
    oz_store_planes<t + 1>(res, plane, off, M);
  }
}

// Four consecutive elements x of every plane, rounded to the grid 1 / scale.
template <int t>
__device__ __forceinline__ void oz_store_word(int8_t* res, size_t plane, size_t off,
                                              const OzInt (&M)[4]) {
  if constexpr (t < oz::T) {
    *reinterpret_cast<uint32_t*>(res + (size_t)t * plane + off) =
        low_bytes(oz_residue<t>(M[0]), oz_residue<t>(M[1]), oz_residue<t>(M[2]), oz_residue<t>(M[3]));
    oz_store_word<t + 1>(res, plane, off, M);
  }
}
__device__ __forceinline__ void oz_store_planes4(int8_t* res, size_t plane, size_t off,
                                                 const double (&x)[4], double scale) {
  OzInt M[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) M[j] = oz_round(x[j], scale);
  oz_store_word<0>(res, plane, off, M);
}

// Bound by HBM and FP32 issue (8 moduli x 5.75 instructions an element).
template <typename T>
__global__ void k_oz_residues(const T* __restrict__ hi, const T* __restrict__ lo, int np,
                              const OzScale* __restrict__ sc, int8_t* __restrict__ res) {
  using SP = OzSplit<T>;
  const int S = sc->S;
  const double scale = S < 0 ? 0.0 : ldexp(1.0, S);   // no valid scale: planes of zeros
  const size_t plane = (size_t)np * np;
  const size_t groups = plane / 8;
  for (size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x; g < groups;
       g += (size_t)gridDim.x * blockDim.x) {
    const size_t off = g * 8;
    alignas(16) T hv[8], lv[8];
    *reinterpret_cast<uint4*>(hv) = *reinterpret_cast<const uint4*>(hi + off);
    *reinterpret_cast<uint4*>(lv) = *reinterpret_cast<const uint4*>(lo + off);
    OzInt M[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const double x = fma(SP::kInv, SP::d(lv[q]), SP::d(hv[q]));
      M[q] = oz_round(S < 0 ? 0.0 : x, scale);
    }
    oz_store_planes<0>(res, plane, off, M);
  }
}

// (No __restrict__ on what the launch before writes here and in k_oz_crt_step: this launch
// begins before that one ends, and a read-only load may be moved ahead of the wait.)
__global__ void k_oz_residues_f64(const double* x, int np, const OzScale* sc, int8_t* res,
                                  const OzStepCtl c, int formed) {
  // (the three launches of a step are chained: each waits for the one before here)
  grid_launch_dependents();
  grid_wait();
  if (formed && sc->kept) return;   // the step before formed these planes
  if (oz_skip(c)) return;
  const int S = sc->S;
  const double scale = S < 0 ? 0.0 : ldexp(1.0, S);
  const size_t plane = (size_t)np * np;
  const size_t groups = plane / 8;
  for (size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x; g < groups;
       g += (size_t)gridDim.x * blockDim.x) {
    const size_t off = g * 8;
    const double2* src = reinterpret_cast<const double2*>(x + off);
    OzInt M[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double2 v = src[q];
      M[2 * q] = oz_round(S < 0 ? 0.0 : v.x, scale);
      M[2 * q + 1] = oz_round(S < 0 ? 0.0 : v.y, scale);
    }
    oz_store_planes<0>(res, plane, off, M);
  }
}

// ---------------------------------------------------------------------------------
// 3. Persistent INT8 product of every plane with itself, upper 128 x 256 tiles (and the
//    128 x 128 ones left over, oz_work_list),
//    epilogue P mod m_t -> uint8 plane Q_t.
//    warp 0: TMA producer; warp 1: TMEM owner + MMA issuer; warps 2..9: epilogue.
// ---------------------------------------------------------------------------------
struct OzGemmArgs {
  int np;
  int nwork;              // entries of the work list
  const int4* work;       // {plane, 128-row block, first 128-column block, 128-column blocks}
  uint8_t* q;             // T planes np x np
  int* err;
  OzStepCtl ctl;
};

__global__ void __launch_bounds__(oz::NTHR, 1)
    k_oz_gemm(const __grid_constant__ CUtensorMap tm, const OzGemmArgs p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[oz::ST];
  __shared__ __align__(8) uint64_t bar_empty[oz::ST];
  __shared__ __align__(8) uint64_t bar_tfull[2];
  __shared__ __align__(8) uint64_t bar_tempty[2];
  __shared__ __align__(8) uint64_t bar_final;
  __shared__ uint32_t tmem_holder;
  __shared__ volatile int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  // up to grid_wait() nothing of the launch before is touched
  grid_launch_dependents();
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < oz::ST; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&bar_tfull[a]), 1);
      mbar_init(smem_u32(&bar_tempty[a]), oz::EPI_WARPS);
    }
    mbar_init(smem_u32(&bar_final), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(smem_u32(&tmem_holder), oz::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_wait();
  const uint32_t tmem = tmem_holder;
  const int np = p.np;
  const int nwork = oz_skip(p.ctl) ? 0 : p.nwork;   // the same answer in every CTA
  const int KB = np / oz::BK;

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- TMA producer ----------------
      int issued_phase[oz::ST];
      for (int s = 0; s < oz::ST; ++s) issued_phase[s] = -1;
      bool ok = true;
      uint32_t g = 0;
      for (int w = blockIdx.x; w < nwork && ok; w += gridDim.x) {
        const int4 wk = p.work[w];
        if (wk.w == 0) break;   // this CTA's list has ended
        const int ra = wk.x * np + wk.y * oz::BM, rb = wk.x * np + wk.z * oz::BM;
        const bool wide = wk.w == 2;
        for (int kb = 0; kb < KB; ++kb, ++g) {
          const int s = g % oz::ST;
          const uint32_t u = g / oz::ST;
          if (g >= (uint32_t)oz::ST && !mbar_wait(smem_u32(&bar_empty[s]), (u - 1) & 1, &s_abort)) {
            ok = false;
            break;
          }
          const uint32_t fb = smem_u32(&bar_full[s]);
          const uint32_t st = sbase + s * oz::STAGE_BYTES;
          mbar_expect_tx(fb, wide ? oz::STAGE_BYTES : oz::STAGE_BYTES - oz::BM * oz::BK);
          tma_load_2d(st, &tm, fb, kb * oz::BK, ra);
          tma_load_2d(st + oz::A_BYTES, &tm, fb, kb * oz::BK, rb);
          if (wide)
            tma_load_2d(st + oz::A_BYTES + oz::BM * oz::BK, &tm, fb, kb * oz::BK, rb + oz::BM);
          issued_phase[s] = u & 1;
        }
      }
      if (!ok) {  // abort: wait (bounded) for this CTA's copies still in flight
        for (int s = 0; s < oz::ST; ++s)
          if (issued_phase[s] >= 0)
            for (uint32_t i = 0; i < kSpinLimit; ++i)
              if (mbar_try(smem_u32(&bar_full[s]), issued_phase[s])) break;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      // ---------------- MMA issuer ----------------
      constexpr uint32_t idesc2 = make_idesc_s8(oz::BM, oz::BN);
      constexpr uint32_t idesc1 = make_idesc_s8(oz::BM, oz::BN / 2);
      bool ok = true;
      uint32_t g = 0, tl = 0;
      for (int w = blockIdx.x; w < nwork && ok; w += gridDim.x, ++tl) {
        const int blocks = p.work[w].w;
        if (blocks == 0) break;
        const uint32_t idesc = blocks == 2 ? idesc2 : idesc1;
        const int a = tl & 1;
        const uint32_t v = tl >> 1;
        if (tl >= 2 && !mbar_wait(smem_u32(&bar_tempty[a]), (v - 1) & 1, &s_abort)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t acc = tmem + a * oz::BN;
        for (int kb = 0; kb < KB; ++kb, ++g) {
          const int s = g % oz::ST;
          if (!mbar_wait(smem_u32(&bar_full[s]), (g / oz::ST) & 1, &s_abort)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t st = sbase + s * oz::STAGE_BYTES;
          const uint64_t da = sw128_desc(st);
          const uint64_t db = sw128_desc(st + oz::A_BYTES);
#pragma unroll
          for (int kk = 0; kk < oz::BK / oz::UK; ++kk) {
            const uint64_t off = (uint64_t)((kk * oz::UK) >> 4);  // 32 bytes along K
            umma_i8(acc, da + off, db + off, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
          }
          umma_commit(smem_u32(&bar_empty[s]));
        }
        if (!ok) break;
        umma_commit(smem_u32(&bar_tfull[a]));
      }
      umma_commit(smem_u32(&bar_final));
      for (uint32_t i = 0; i < kSpinLimit; ++i)
        if (mbar_try(smem_u32(&bar_final), 0)) break;
      if (!ok) s_abort = 1;
    }
    __syncwarp();
  } else {
    // ---------------- epilogue (8 warps: lane quarter q, 128-column half) ----------------
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    uint32_t tl = 0;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x, ++tl) {
      const int4 wk = p.work[w];
      if (wk.w == 0) break;
      const int t = wk.x;
      const int a = tl & 1;
      if (!mbar_wait_idle(smem_u32(&bar_tfull[a]), (tl >> 1) & 1, &s_abort)) break;
      tc_fence_after();
      // P mod m: u = P + off (off a multiple of m, u < 2^32), floor(u / m) by a 64-bit
      // reciprocal (exact for u < 2^32 since 2^-32 < 1/m).
      const uint32_t m = (uint32_t)oz::mod(t);
      const unsigned long long magic = ~0ull / m + 1ull;
      const uint32_t off = m * ((1u << 30) / m + 1u);
      const int r = wk.y * oz::BM + q * 32 + lane;
      uint8_t* qrow = p.q + (size_t)t * np * np + (size_t)r * np;
#pragma unroll 1
      for (int cc = 0; cc < 2 * wk.w; ++cc) {
        const int cl = half * 64 * wk.w + cc * 32;
        uint32_t v[32];
        tmem_ld32(tmem + lane_base + a * oz::BN + cl, v);
        tmem_wait_ld();
        const int c0 = wk.z * oz::BM + cl;
        {
          alignas(16) uint8_t out[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const uint32_t u = (uint32_t)((int)v[j]) + off;
            const uint32_t d = (uint32_t)__umul64hi((unsigned long long)u, magic);
            out[j] = (uint8_t)(u - d * m);
          }
          reinterpret_cast<uint4*>(qrow + c0)[0] = reinterpret_cast<const uint4*>(out)[0];
          reinterpret_cast<uint4*>(qrow + c0)[1] = reinterpret_cast<const uint4*>(out)[1];
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_tempty[a]));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, oz::TMEM_COLS);
  if (s_abort && threadIdx.x == 0 && p.err) atomicExch(p.err, 1);
}

// ---------------------------------------------------------------------------------
// 4. CRT: X^2 (FP64) and 4 (X^2 - X) re-split to hi/lo, both triangles, from the residues
//    of the upper tiles.  One CTA per upper 32 x 32 block pair; the mirror goes through
//    shared memory so both halves are stored row-contiguous.
// ---------------------------------------------------------------------------------
// Chinese remaindering in FP64: with W_t the integer that is 1 modulo m_t and 0 modulo the
// others, Y = sum_t q_t W_t - n P, P = prod(m_t) < 2^71.4, n the nearest integer to the sum
// over P.  W_t and P are cut at 2^31 into two integers below 2^40.5 and 2^31, so that both
// partial sums (9 terms, q_t < 256) and both n multiples stay below 2^53: every operation
// but the last, which joins the two parts, is exact, and Y is the correctly rounded double.
// 30 FP64 instructions, against the chain of 16-, 32- and 64-bit modular reductions of a
// pairwise tree.
namespace ozc {
typedef unsigned __int128 u128;
__host__ __device__ constexpr u128 prod() {
  u128 p = 1;
  for (int t = 0; t < oz::T; ++t) p *= (u128)oz::mod(t);
  return p;
}
__host__ __device__ constexpr u128 weight(int t) {
  const u128 r = prod() / (u128)oz::mod(t);
  return r * (u128)oz::inv_mod((int)(r % (u128)oz::mod(t)), oz::mod(t));
}
__host__ __device__ constexpr double upper(u128 v) { return (double)(uint64_t)(v >> 31); }
__host__ __device__ constexpr double lower(u128 v) { return (double)(uint64_t)(v & 0x7fffffffu); }
}  // namespace ozc

template <int t>
__device__ __forceinline__ void crt_sums(const uint32_t (&q)[oz::T], double& s1, double& s2) {
  if constexpr (t < oz::T) {
    constexpr double w1 = ozc::upper(ozc::weight(t)), w2 = ozc::lower(ozc::weight(t));
    const double d = __hiloint2double(0x43300000, (int)q[t]) - 0x1p52;   // q_t
    s1 = fma(d, w1, s1);
    s2 = fma(d, w2, s2);
    crt_sums<t + 1>(q, s1, s2);
  }
}
// Residues (q_t in [0, m_t)) -> the symmetric integer Y, |Y| < prod/2 (1 - 1e-12).
__device__ __forceinline__ double crt_value(const uint32_t (&q)[oz::T]) {
  constexpr double p1 = ozc::upper(ozc::prod()), p2 = ozc::lower(ozc::prod());
  constexpr double p = p1 * 0x1p31 + p2, half = 0.5 * p;
  double s1 = 0.0, s2 = 0.0;
  crt_sums<0>(q, s1, s2);
  const double n = fma(s1, 0x1p31 / p, 0x1.8p52) - 0x1.8p52;
  double d1 = fma(-n, p1, s1), d2 = fma(-n, p2, s2);
  double y = fma(d1, 0x1p31, d2);
  // n left out the lower sums (2^-29 of a unit): one unit off near a tie
  if (fabs(y) > half) {
    const double sgn = y > 0.0 ? 1.0 : -1.0;
    d1 = fma(-sgn, p1, d1);
    d2 = fma(-sgn, p2, d2);
    y = fma(d1, 0x1p31, d2);
  }
  return y;
}
// Four consecutive elements of every plane, as the squares' values.
__device__ __forceinline__ void crt_load4(const uint8_t* q, size_t plane, size_t e,
                                          double down, double (&x2)[4]) {
  uint32_t w[oz::T];
#pragma unroll
  for (int t = 0; t < oz::T; ++t) w[t] = *reinterpret_cast<const uint32_t*>(q + (size_t)t * plane + e);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint32_t v[oz::T];
#pragma unroll
    for (int t = 0; t < oz::T; ++t) v[t] = (w[t] >> (8 * j)) & 255u;
    x2[j] = crt_value(v) * down;
  }
}

template <typename T>
__global__ void __launch_bounds__(256)
    k_oz_crt(const uint8_t* __restrict__ q, const T* __restrict__ xhi, const T* __restrict__ xlo,
             int np, const OzScale* __restrict__ sc, double* __restrict__ x2out,
             T* __restrict__ rhi, T* __restrict__ rlo) {
  using SP = OzSplit<T>;
  __shared__ double s_x2[32][33];
  __shared__ T s_rh[32][34], s_rl[32][34];
  int ib, jb;
  upper_tile(blockIdx.x, ib, jb);
  const int row = threadIdx.x >> 3, c4 = (threadIdx.x & 7) * 4;   // a thread's four columns
  const int S = sc->S;
  const double down = S < 0 ? __longlong_as_double(0x7ff8000000000000ll) : ldexp(1.0, -2 * S);
  const size_t plane = (size_t)np * np;
  struct alignas(8) T4 { T v[4]; };
  {
    const size_t e = (size_t)(ib * 32 + row) * np + jb * 32 + c4;
    double x2[4];
    crt_load4(q, plane, e, down, x2);
    const T4 xh = *reinterpret_cast<const T4*>(xhi + e), xl = *reinterpret_cast<const T4*>(xlo + e);
    T4 h, l;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double x = fma(SP::kInv, SP::d(xl.v[j]), SP::d(xh.v[j]));
      const double r4 = 4.0 * (x2[j] - x);
      h.v[j] = SP::from_d(r4);
      l.v[j] = SP::from_d((r4 - SP::d(h.v[j])) * SP::kScale);
      s_x2[row][c4 + j] = x2[j];
      s_rh[row][c4 + j] = h.v[j];
      s_rl[row][c4 + j] = l.v[j];
    }
    double2* o = reinterpret_cast<double2*>(x2out + e);
    o[0] = make_double2(x2[0], x2[1]);
    o[1] = make_double2(x2[2], x2[3]);
    *reinterpret_cast<T4*>(rhi + e) = h;
    *reinterpret_cast<T4*>(rlo + e) = l;
  }
  if (ib == jb) return;  // diagonal blocks hold both triangles (the product is symmetric)
  __syncthreads();
  const size_t e = (size_t)(jb * 32 + row) * np + ib * 32 + c4;
  T4 h, l;
  double2* o = reinterpret_cast<double2*>(x2out + e);
  o[0] = make_double2(s_x2[c4][row], s_x2[c4 + 1][row]);
  o[1] = make_double2(s_x2[c4 + 2][row], s_x2[c4 + 3][row]);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    h.v[j] = s_rh[c4 + j][row];
    l.v[j] = s_rl[c4 + j][row];
  }
  *reinterpret_cast<T4*>(rhi + e) = h;
  *reinterpret_cast<T4*>(rlo + e) = l;
}

// ---------------------------------------------------------------------------------
// 5. Exact INT8 mode: the step's last launch.  X_k^2 from the residues, the branch of
//    step k from its record (control_prologue), X_{k+1} = a X_k^2 + b X_k in FP64 over
//    both triangles, and the step's sums {||X_{k+1}||^2, Tr X_{k+1}, ||X_k - X_k^2||^2,
//    Tr X_k^2} through the last-CTA finalisation, like the other step kernels.  It also
//    leaves the residue planes of X_{k+1} with step k's scale, while the values are in
//    registers: the scale changes two or three times in a solve, and only then does
//    k_oz_residues_f64 form them again (planes by a pass over X cost 27 us a step at
//    n = 2744).  The row norms that the scale needs are integer sums on the way; the last
//    CTA takes their maximum (stored per block and summed by a launch of its own: 6 us a step
//    more).  50 us at n = 2744, where the bytes take 30 at the measured copy rate.  One
//    resident wave of CTAs walks the upper 32 x 32 block pairs (diagonal blocks hold both
//    triangles, whose squares are equal bit for bit: the integer products are symmetric).
// ---------------------------------------------------------------------------------
// ||row||^2 shares in units of 2^-44, rounded up: integer sums do not depend on their order,
// and the scale's bound only needs the norm from above (at most np/32 units too much, 1e-10).
// np/32 <= 2048 shares below 2^8 stay below 2^63.  Larger shares (32 elements of a diverging
// iterate; with X in [0, 1] a whole row has at most 1) enter as their largest, which NaN
// exceeds as a bit pattern; the bound then takes it for every share of the row.
__device__ __forceinline__ void oz_add_row(unsigned long long* rsum, int row, int np, double share) {
  if (share < 256.0) atomicAdd(rsum + row, __double2ull_ru(share * 0x1p44));
  else
    atomicMax(rsum + np, share == share ? (unsigned long long)__double_as_longlong(share)
                                        : 0x7ff8000000000000ull);
}

__global__ void __launch_bounds__(256)
    k_oz_crt_step(const uint8_t* q, const OzScale* sc, const StepArgs p, OzScale* next,
                  unsigned long long* rsum, int8_t* res) {
  __shared__ double s_v[32][33];
  __shared__ double red[32 * 4];
  __shared__ int s_flag;
  grid_launch_dependents();
  grid_wait();
  const int br = control_prologue(p);
  if (br < 0) return;
  const double a = br == BR_X2 ? 1.0 : -1.0, b = br == BR_X2 ? 0.0 : 2.0;
  const int np = p.np;
  const double* X = (const double*)p.E;
  double* Xo = (double*)p.out;
  const int S = sc->S;
  const double down = S < 0 ? __longlong_as_double(0x7ff8000000000000ll) : ldexp(1.0, -2 * S);
  const double up = S < 0 ? 0.0 : ldexp(1.0, S);
  const size_t plane = (size_t)np * np;
  const int row = threadIdx.x >> 3, c4 = (threadIdx.x & 7) * 4;   // a thread's four columns
  const long long nb = np / 32, nblk = nb * (nb + 1) / 2;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (long long bid = blockIdx.x; bid < nblk; bid += gridDim.x) {
    int ib, jb;
    upper_tile((int)bid, ib, jb);
    const double w = ib == jb ? 1.0 : 2.0;
    const int i = ib * 32 + row;
    const size_t e = (size_t)i * np + jb * 32 + c4;
    double x2[4], nx[4];
    crt_load4(q, plane, e, down, x2);
    const double2 xa = *reinterpret_cast<const double2*>(X + e);
    const double2 xb = *reinterpret_cast<const double2*>(X + e + 2);
    const double x[4] = {xa.x, xa.y, xb.x, xb.y};
    double rs = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      nx[j] = fma(a, x2[j], b * x[j]);
      const double d = x[j] - x2[j];
      rs = fma(nx[j], nx[j], rs);
      s[2] = fma(w * d, d, s[2]);
      if (i == jb * 32 + c4 + j) {
        s[1] += nx[j];
        s[3] += x2[j];
      }
      s_v[row][c4 + j] = nx[j];
    }
    s[0] = fma(w, rs, s[0]);
    double2* o = reinterpret_cast<double2*>(Xo + e);
    o[0] = make_double2(nx[0], nx[1]);
    o[1] = make_double2(nx[2], nx[3]);
    oz_store_planes4(res, plane, e, nx, up);
    // this block's share of ||row i of X_{k+1}||^2 (the next step's scale)
    rs += __shfl_xor_sync(0xffffffffu, rs, 1);
    rs += __shfl_xor_sync(0xffffffffu, rs, 2);
    rs += __shfl_xor_sync(0xffffffffu, rs, 4);
    if (c4 == 0) oz_add_row(rsum, i, np, rs);
    if (ib != jb) {
      __syncthreads();
      const int r = jb * 32 + row;
      double v[4];
      double cs = 0.0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j] = s_v[c4 + j][row];
        cs = fma(v[j], v[j], cs);
      }
      double2* m = reinterpret_cast<double2*>(Xo + (size_t)r * np + ib * 32 + c4);
      m[0] = make_double2(v[0], v[1]);
      m[1] = make_double2(v[2], v[3]);
      oz_store_planes4(res, plane, (size_t)r * np + ib * 32 + c4, v, up);
      cs += __shfl_xor_sync(0xffffffffu, cs, 1);
      cs += __shfl_xor_sync(0xffffffffu, cs, 2);
      cs += __shfl_xor_sync(0xffffffffu, cs, 4);
      if (c4 == 0) oz_add_row(rsum, r, np, cs);
    }
    __syncthreads();
  }
  __threadfence();
  publish_and_finalize(p, s, red, &s_flag);
  if (!s_flag) return;
  // the last CTA: the scale of X_{k+1} from its row norms, which it clears for the next step
  unsigned long long best = 0;
  for (int r = threadIdx.x; r < np; r += blockDim.x) {
    const unsigned long long v = atomicExch(rsum + r, 0ull);
    best = v > best ? v : best;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, best, o);
    best = v > best ? v : best;
  }
  __shared__ unsigned long long s_best[8];
  if ((threadIdx.x & 31) == 0) s_best[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 0; w < 8; ++w) best = s_best[w] > best ? s_best[w] : best;
  const unsigned long long large = atomicExch(rsum + np, 0ull);
  double r2 = (double)best * 0x1p-44;
  if (large) r2 += (np / 32) * __longlong_as_double((long long)large);
  const int Sn = oz_choose_scale(r2, np);
  next->r2max_bits = (unsigned long long)__double_as_longlong(r2);
  next->kept = Sn == S;
  next->S = Sn;
}

// ---------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------
int oz_nmod() { return oz::T; }

size_t oz_scale_bytes() { return sizeof(OzScale); }

static int oz_sms() {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
    v = 148;
  return v;
}

int oz_work_list(int np, std::vector<int4>& out) {
  return oz_work_items(np / oz::BM, oz::T, oz_sms(), out);
}

cudaError_t launch_oz_planes(const __half* xhi, const __half* xlo, int np, int bf16,
                             void* scale, int8_t* res, cudaStream_t st) {
  if (np % oz::BM != 0 || np > 65536) return cudaErrorInvalidValue;
  OzScale* sc = (OzScale*)scale;
  cudaError_t e = cudaMemsetAsync(sc, 0, sizeof(OzScale), st);
  if (e != cudaSuccess) return e;
  const int rgrid = std::min((np + 7) / 8, 148 * 8);
  if (bf16)
    k_oz_rownorm<__nv_bfloat16><<<rgrid, 256, 0, st>>>((const __nv_bfloat16*)xhi,
                                                       (const __nv_bfloat16*)xlo, np, sc);
  else
    k_oz_rownorm<__half><<<rgrid, 256, 0, st>>>(xhi, xlo, np, sc);
  k_oz_scale<<<1, 1, 0, st>>>(sc, np);
  const size_t groups = (size_t)np * np / 8;
  const int g = (int)std::min<size_t>((groups + 255) / 256, 148 * 16);
  if (bf16)
    k_oz_residues<__nv_bfloat16><<<g, 256, 0, st>>>((const __nv_bfloat16*)xhi,
                                                    (const __nv_bfloat16*)xlo, np, sc, res);
  else
    k_oz_residues<__half><<<g, 256, 0, st>>>(xhi, xlo, np, sc, res);
  note_launch(3);
  return cudaGetLastError();
}

cudaError_t launch_oz_gemm(const int8_t* res, int np, uint8_t* qout, const int4* work,
                           int nwork, int grid, int* err, cudaStream_t st, const OzStepCtl* ctl) {
  if (np % oz::BM != 0 || np > 65536 || nwork <= 0) return cudaErrorInvalidValue;
  CUtensorMap tm;
  if (!make_tmap_box(&tm, res, (long long)oz::T * np, np, np, TMAP_U8, oz::BM))
    return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(k_oz_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       oz::SMEM_BYTES);
  if (e != cudaSuccess) return e;
  OzGemmArgs a;
  a.np = np;
  a.nwork = nwork;
  a.work = work;
  a.q = qout;
  a.err = err;
  if (ctl) a.ctl = *ctl;
  else memset(&a.ctl, 0, sizeof(a.ctl));
  return launch_chained(k_oz_gemm, grid, oz::NTHR, oz::SMEM_BYTES, st, tm, a);
}

cudaError_t launch_oz_crt(const uint8_t* q, const __half* xhi, const __half* xlo, int np,
                          int bf16, const void* scale, double* x2, __half* rhi, __half* rlo,
                          cudaStream_t st) {
  const int nb = np / 32;
  const unsigned nblk = (unsigned)((long long)nb * (nb + 1) / 2);
  const OzScale* sc = (const OzScale*)scale;
  if (bf16)
    k_oz_crt<__nv_bfloat16><<<nblk, 256, 0, st>>>(q, (const __nv_bfloat16*)xhi,
                                                  (const __nv_bfloat16*)xlo, np, sc, x2,
                                                  (__nv_bfloat16*)rhi, (__nv_bfloat16*)rlo);
  else
    k_oz_crt<__half><<<nblk, 256, 0, st>>>(q, xhi, xlo, np, sc, x2, rhi, rlo);
  note_launch();
  return cudaGetLastError();
}

// First step: the scale and the planes from x (and rsum cleared).  Later steps: the planes
// that launch_oz_crt_step left, formed again if it found another scale for this x.
cudaError_t launch_oz_planes_f64(const double* x, int np, void* scale, unsigned long long* rsum,
                                 bool first, int8_t* res, const OzStepCtl* ctl, cudaStream_t st) {
  if (np % oz::BM != 0 || np > 65536) return cudaErrorInvalidValue;
  OzScale* sc = (OzScale*)scale;
  if (first) {
    cudaError_t e = cudaMemsetAsync(sc, 0, sizeof(OzScale), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(rsum, 0, oz_rsum_words(np) * sizeof(*rsum), st);
    if (e != cudaSuccess) return e;
    k_oz_rownorm_f64<<<std::min((np + 7) / 8, 148 * 8), 256, 0, st>>>(x, np, sc, *ctl);
    k_oz_scale<<<1, 1, 0, st>>>(sc, np);
    note_launch(2);
  }
  const size_t groups = (size_t)np * np / 8;
  // one wave: most launches only find the planes formed (9 us each with two waves of CTAs
  // that read the record first; this and the chained launches: 8.99 -> 8.73 ms for the 60
  // steps of n = 2744)
  const int g = (int)std::min<size_t>((groups + 255) / 256, (size_t)oz_sms() * 4);
  return launch_chained(k_oz_residues_f64, g, 256, 0, st, x, np, (const OzScale*)sc, res, *ctl, (int)!first);
}

size_t oz_rsum_words(int np) { return (size_t)np + 1; }

cudaError_t launch_oz_crt_step(const uint8_t* q, void* scale, const StepArgs& a,
                               unsigned long long* rsum, int8_t* res, cudaStream_t st) {
  if (a.np % 128 != 0) return cudaErrorInvalidValue;
  const long long nb = a.np / 32;
  // one resident wave: every CTA walks its share of the blocks (more CTAs than fit end in a
  // second wave that is mostly empty)
  static std::atomic<int> resident{0};
  int per_sm = resident.load(std::memory_order_relaxed);
  if (per_sm == 0) {
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_oz_crt_step, 256, 0);
    if (e != cudaSuccess) return e;
    per_sm = std::min(std::max(per_sm, 1), 8);   // the partial sums have room for eight
    resident.store(per_sm, std::memory_order_relaxed);
  }
  const int grid = (int)std::min<long long>(nb * (nb + 1) / 2, (long long)oz_sms() * per_sm);
  return launch_chained(k_oz_crt_step, grid, 256, 0, st, q, (const OzScale*)scale, a, (OzScale*)scale,
                        rsum, res);
}

// Scale exponent and largest squared row norm (diagnostics / checks): queued into pinned
// memory of oz_scale_bytes(), read after the caller's wait.
cudaError_t oz_copy_scale(const void* scale, void* pinned, cudaStream_t st) {
  return cudaMemcpyAsync(pinned, scale, sizeof(OzScale), cudaMemcpyDeviceToHost, st);
}
void oz_scale_values(const void* pinned, int* S, double* r2max) {
  OzScale h;
  memcpy(&h, pinned, sizeof(h));
  *S = h.S;
  memcpy(r2max, &h.r2max_bits, sizeof(double));
}

}  // namespace sp2b
