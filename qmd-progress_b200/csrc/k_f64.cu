// FP64 kernels: Gershgorin bounds, normalisation, and the symmetric-tile DMMA product
// with the fused SP2 epilogue.  This is the parity form of the SP2 step (1e-10).
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "f64_dmma.cuh"
#include "reduce.cuh"
#include "sp2b_tune.h"

namespace sp2b {

// ------------------------------------------------------------------------------------
// Gershgorin bounds (bml_gershgorin as used by prg_normalize, src/prg_normalize_mod.F90:41)
// H is column-major: H(i, j) = h[i + j*ld]; thread i walks row i, so a warp reads 32
// consecutive doubles of one column per step (coalesced).
// ------------------------------------------------------------------------------------
__global__ void k_gersh_partial(const double* __restrict__ h, int n, int ld, int ncol,
                                double* __restrict__ rowsum) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int j0 = blockIdx.y * ncol;
  const int j1 = min(n, j0 + ncol);
  double s = 0.0;
  for (int j = j0; j < j1; ++j)
    if (j != i) s += fabs(h[i + (size_t)j * ld]);
  rowsum[(size_t)blockIdx.y * n + i] = s;
}

// Row totals, per-block min/max of (h_ii - r_i, h_ii + r_i), and in the last block to
// arrive the min/max over the blocks in block order; a NaN or overflow anywhere makes
// both bounds NaN.
__device__ __forceinline__ double nan_min(double a, double b) {
  return (a != a || b != b) ? __longlong_as_double(0x7ff8000000000000ll) : fmin(a, b);
}
__device__ __forceinline__ double nan_max(double a, double b) {
  return (a != a || b != b) ? __longlong_as_double(0x7ff8000000000000ll) : fmax(a, b);
}
// 32 rows per block, eight warps a row's partials (a thread per row adding up to 592 of them
// in turn was latency-bound: 14 us at n = 1000).
__global__ void __launch_bounds__(256)
    k_gersh_final(const double* __restrict__ h, int n, int ld, int nsplit,
                  const double* __restrict__ rowsum, double* partials, unsigned* counter,
                  double* __restrict__ bounds) {
  __shared__ double s_r[8][33];
  __shared__ double smin[256], smax[256];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  double r = 0.0;
  if (i < n)
#pragma unroll 4
    for (int s = warp; s < nsplit; s += 8) r += rowsum[(size_t)s * n + i];
  s_r[warp][lane] = r;
  __syncthreads();
  double mn = 1e308, mx = -1e308;
  if (warp == 0) {
    if (i < n) {
      r = 0.0;
      for (int w = 0; w < 8; ++w) r += s_r[w][lane];
      const double d = h[i + (size_t)i * ld];
      if (!(r == r) || !(d == d) || fabs(r) > 1e300 || fabs(d) > 1e300) {
        mn = mx = __longlong_as_double(0x7ff8000000000000ll);
      } else {
        mn = d - r;
        mx = d + r;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      mn = nan_min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = nan_max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
  }
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = mn;
    partials[2 * blockIdx.x + 1] = mx;
    __threadfence();
    s_last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  mn = 1e308;
  mx = -1e308;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
    mn = nan_min(mn, __ldcg(partials + 2 * b));
    mx = nan_max(mx, __ldcg(partials + 2 * b + 1));
  }
  smin[threadIdx.x] = mn;
  smax[threadIdx.x] = mx;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      smin[threadIdx.x] = nan_min(smin[threadIdx.x], smin[threadIdx.x + o]);
      smax[threadIdx.x] = nan_max(smax[threadIdx.x], smax[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    bounds[0] = smin[0];
    bounds[1] = smax[0];
    *counter = 0u;
  }
}

// Delta_0 = alpha H1 (alpha = -1/(e_max - e_min)) into the zero-padded np x np buffer
// (src/prg_response_mod.F90:700: bml_scale(alpha, rsp_bml)).
__global__ void k_resp_init(const double* __restrict__ h1, int n, int ld, int np,
                            const double* __restrict__ bounds, double* __restrict__ d) {
  const double alpha = -1.0 / (bounds[1] - bounds[0]);
  const uint32_t gpr = (uint32_t)np / 8, ngroups = gpr * (uint32_t)np;
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += gridDim.x * blockDim.x) {
    const int r = (int)(g / gpr), c0 = (int)(g - (uint32_t)r * gpr) * 8;
    double v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int c = c0 + e;
      // h1 == nullptr: the identity (dX0/dmu of the SP2-Fermi normalisation)
      v[e] = (r < n && c < n) ? alpha * (h1 ? h1[(size_t)r * ld + c] : (r == c ? 1.0 : 0.0)) : 0.0;
    }
    double2* dst = reinterpret_cast<double2*>(d + (size_t)r * np + c0);
#pragma unroll
    for (int e = 0; e < 4; ++e) dst[e] = make_double2(v[2 * e], v[2 * e + 1]);
  }
}

cudaError_t launch_resp_init(const double* h1, int n, int ld, int np, const double* bounds,
                             double* d, cudaStream_t st) {
  const size_t groups = (size_t)np * np / 8;
  const int g = (int)std::min<size_t>((groups + 255) / 256, 148 * 8);
  k_resp_init<<<g, 256, 0, st>>>(h1, n, ld, np, bounds, d);
  note_launch();
  return cudaGetLastError();
}

// Lower triangle of a symmetric n x n matrix (row pitch ld) from its upper triangle, by
// 32 x 32 blocks through shared memory (the host-pointer entries copy only the upper
// triangle across PCIe).  One CTA per block pair (ib <= jb).
__global__ void __launch_bounds__(256) k_mirror_lower(double* __restrict__ a, int n, int ld) {
  __shared__ double t[32][33];
  int ib, jb;
  upper_tile(blockIdx.x, ib, jb);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = ib * 32 + ty + 8 * k, c = jb * 32 + tx;
    t[ty + 8 * k][tx] = (r < n && c < n) ? a[(size_t)r * ld + c] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = jb * 32 + ty + 8 * k, c = ib * 32 + tx;   // (r, c) = mirror of (c, r)
    if (r < n && c < n && r > c) a[(size_t)r * ld + c] = t[tx][ty + 8 * k];
  }
}

cudaError_t launch_mirror_lower(double* a, int n, int ld, cudaStream_t st) {
  const long long nb = (n + 31) / 32;
  k_mirror_lower<<<(unsigned)(nb * (nb + 1) / 2), 256, 0, st>>>(a, n, ld);
  note_launch();
  return cudaGetLastError();
}

int gersh_nsplit(int n) {
  const int rows_blocks = (n + 255) / 256;
  int ns = (4 * 148 + rows_blocks - 1) / rows_blocks;
  if (ns > n) ns = n;
  if (ns < 1) ns = 1;
  return ns;
}

cudaError_t launch_gersh(const double* h, int n, int ld, double* rowsum, int nsplit,
                         double* bounds, double* partials, unsigned* counter, cudaStream_t st) {
  const int ncol = (n + nsplit - 1) / nsplit;
  dim3 grid((n + 255) / 256, nsplit);
  k_gersh_partial<<<grid, 256, 0, st>>>(h, n, ld, ncol, rowsum);
  note_launch();
  k_gersh_final<<<(n + 31) / 32, 256, 0, st>>>(h, n, ld, nsplit, rowsum, partials, counter,
                                                  bounds);
  note_launch();
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Normalisation X0 = alpha H + beta I, alpha = -1/(emax-emin), beta = emax/(emax-emin)
// (src/prg_normalize_mod.F90:27, in the alpha/beta form of src/prg_response_mod.F90:700)
// into the zero-padded np x np buffer, with Tr X0 and ||X0||_F^2 for the first SP2 step.
// ------------------------------------------------------------------------------------
__global__ void k_normalize_f64(const double* __restrict__ h, int n, int ld, int np,
                                const double* __restrict__ bounds, double* __restrict__ x,
                                double* partials, unsigned* counter, SP2Rec* rec0,
                                double* norm_out) {
  __shared__ double red[32 * 4];
  __shared__ int s_last;
  const double emin = bounds[0], emax = bounds[1];
  const double mm = emax - emin;
  const double alpha = -1.0 / mm, beta = emax / mm;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  // groups of 8 consecutive elements of one row (np is a multiple of 128)
  const uint32_t gpr = (uint32_t)np / 8, ngroups = gpr * (uint32_t)np;
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += gridDim.x * blockDim.x) {
    const int r = (int)(g / gpr), c0 = (int)(g - (uint32_t)r * gpr) * 8;
    double v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int c = c0 + e;
      v[e] = (r < n && c < n) ? alpha * h[(size_t)r * ld + c] + (r == c ? beta : 0.0) : 0.0;
      s[0] += v[e] * v[e];
      if (r == c) s[1] += v[e];
    }
    double2* dst = reinterpret_cast<double2*>(x + (size_t)r * np + c0);
#pragma unroll
    for (int e = 0; e < 4; ++e) dst[e] = make_double2(v[2 * e], v[2 * e + 1]);
  }
  block_sum<4>(s, red);
  if (threadIdx.x == 0) {
    partials[4 * blockIdx.x] = s[0];
    partials[4 * blockIdx.x + 1] = s[1];
    __threadfence();
    s_last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double t[4] = {0.0, 0.0, 0.0, 0.0};
  for (int j = threadIdx.x; j < (int)gridDim.x; j += blockDim.x) {
    t[0] += __ldcg(partials + 4 * j);
    t[1] += __ldcg(partials + 4 * j + 1);
  }
  block_sum<4>(t, red);
  if (threadIdx.x == 0) {
    *counter = 0u;
    SP2Rec r0;
    memset(&r0, 0, sizeof(r0));
    r0.trx = t[1];
    r0.trx_data = t[1];
    r0.fro2 = t[0];
    r0.last_branch = -1;
    if (!(t[0] == t[0]) || !(mm > 0.0)) {
      r0.status = SP2B_BAD_INPUT;
      r0.done = 1;
    }
    *rec0 = r0;
    norm_out[0] = emin;
    norm_out[1] = emax;
    norm_out[2] = t[1];
    norm_out[3] = t[0];
  }
}

static int norm_grid(int np) {
  const size_t total = (size_t)np * np / 8;   // groups of eight elements
  size_t g = (total + 255) / 256;
  if (g > 148 * 8) g = 148 * 8;
  return (int)g;
}

static int elem_grid(int np) {
  const size_t g = ((size_t)np * np + 255) / 256;
  return (int)std::min<size_t>(g, 148 * 8);
}

cudaError_t launch_normalize_f64(const double* h, int n, int ld, int np, const double* bounds,
                                 double* x, double* partials, unsigned* counter, SP2Rec* rec0,
                                 double* norm_out, cudaStream_t st) {
  k_normalize_f64<<<norm_grid(np), 256, 0, st>>>(h, n, ld, np, bounds, x, partials, counter,
                                                 rec0, norm_out);
  note_launch();
  return cudaGetLastError();
}

__global__ void k_copy_in(const double* __restrict__ src, int n, int ld, int np,
                          double* __restrict__ x) {
  const size_t total = (size_t)np * np;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(idx / np), c = (int)(idx % np);
    x[idx] = (r < n && c < n) ? src[(size_t)r * ld + c] : 0.0;
  }
}

cudaError_t launch_copy_in(const double* src, int n, int ld, int np, double* x,
                           cudaStream_t st) {
  k_copy_in<<<elem_grid(np), 256, 0, st>>>(src, n, ld, np, x);
  note_launch();
  return cudaGetLastError();
}

__global__ void k_finish_f64(const double* __restrict__ x, int np, int n, double scale,
                             double* __restrict__ rho, int ld) {
  const size_t total = (size_t)n * n;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(idx / n), c = (int)(idx % n);
    rho[(size_t)r * ld + c] = scale * x[(size_t)r * np + c];
  }
}

cudaError_t launch_finish_f64(const double* x, int np, int n, double scale, double* rho,
                              int ld, cudaStream_t st) {
  k_finish_f64<<<elem_grid(np), 256, 0, st>>>(x, np, n, scale, rho, ld);
  note_launch();
  return cudaGetLastError();
}

__global__ void k_finish_solve_f64(const double* __restrict__ x0, const double* __restrict__ x1,
                                   const SolveOut* __restrict__ sout, const int* __restrict__ err,
                                   const double* __restrict__ norm, int np, int n,
                                   double* __restrict__ rho, int ld) {
  // (each test is false for a NaN; an infinite norm fails the last)
  if (!sout->done || *err || !(norm[1] - norm[0] > 0.0) || !(norm[3] <= 1e300)) return;
  const double* __restrict__ x = (sout->nupd & 1) ? x1 : x0;
  const size_t total = (size_t)n * n;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(idx / n), c = (int)(idx % n);
    rho[(size_t)r * ld + c] = 2.0 * x[(size_t)r * np + c];
  }
}

cudaError_t launch_finish_solve_f64(const double* x0, const double* x1, const SolveOut* sout,
                                    const int* err, const double* norm, int np, int n, double* rho,
                                    int ld, cudaStream_t st) {
  k_finish_solve_f64<<<elem_grid(np), 256, 0, st>>>(x0, x1, sout, err, norm, np, n, rho, ld);
  note_launch();
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------
// Symmetric-tile FP64 product with the SP2 epilogue.
// One CTA per upper tile (bi <= bj) of BT x BT; WM x WN warps, each owning a
// (BT/WM) x (BT/WN) block of m8n8k4 DMMA fragments.  Operand tiles are rows of the
// symmetric inputs: As[k][m] = A[k0+k][i0+m], Bs[k][n] = B[k0+k][j0+n], staged by a
// 3-deep cp.async pipeline with rows padded to BT+4 doubles (conflict-free fragment loads).
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

template <int BT, int WM, int WN>
struct F64Cfg {
  static constexpr int BK = 16;
  static constexpr int NW = WM * WN;
  static constexpr int NT = NW * 32;
  static constexpr int LDS = BT + 4;
  static constexpr int ST = 3;
  static constexpr int TM = BT / WM, TN = BT / WN;
  static constexpr int MI = TM / 8, NI = TN / 8;
  static constexpr size_t SMEM = (size_t)ST * 2 * BK * LDS * sizeof(double);
};

template <int BT, int WM, int WN>
__global__ void __launch_bounds__(WM* WN * 32, 1) k_sym_gemm_f64(const StepArgs p) {
  using C = F64Cfg<BT, WM, WN>;
  extern __shared__ __align__(16) double sm[];
  __shared__ double red[32 * 4];
  __shared__ int s_flag;

  double alpha = p.alpha, beta = p.beta;
  if (p.control) {
    const int br = control_prologue(p);
    if (br < 0) return;
    if (br == BR_X2) { alpha = 1.0; beta = 0.0; }
    else { alpha = -1.0; beta = 2.0; }
  }
  int bi, bj;
  upper_tile(blockIdx.x, bi, bj);
  const int i0 = bi * BT, j0 = bj * BT;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int wm = warp / WN, wn = warp % WN;
  const int ld = p.ld;
  const double* __restrict__ A = (const double*)p.A;
  const double* __restrict__ B = (const double*)p.B;

  double acc[C::MI][C::NI][2];
#pragma unroll
  for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
    for (int ni = 0; ni < C::NI; ++ni) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;

  const int KB = p.np / C::BK;
  auto load = [&](int stage, int kb) {
    double* As = sm + stage * 2 * C::BK * C::LDS;
    double* Bs = As + C::BK * C::LDS;
    const int k0 = kb * C::BK;
    for (int c = tid; c < C::BK * BT / 2; c += C::NT) {
      const int row = c / (BT / 2), col = (c % (BT / 2)) * 2;
      cp_async16(As + row * C::LDS + col, A + (size_t)(k0 + row) * ld + i0 + col);
      cp_async16(Bs + row * C::LDS + col, B + (size_t)(k0 + row) * ld + j0 + col);
    }
  };
#pragma unroll
  for (int s = 0; s < C::ST - 1; ++s) {
    if (s < KB) load(s, s);
    cp_async_commit();
  }
  for (int kb = 0; kb < KB; ++kb) {
    cp_async_wait<C::ST - 2>();
    __syncthreads();
    {
      const int nk = kb + C::ST - 1;
      if (nk < KB) load(nk % C::ST, nk);
      cp_async_commit();
    }
    const double* As = sm + (kb % C::ST) * 2 * C::BK * C::LDS;
    const double* Bs = As + C::BK * C::LDS;
#pragma unroll
    for (int kk = 0; kk < C::BK; kk += 4) {
      double a[C::MI], b[C::NI];
#pragma unroll
      for (int mi = 0; mi < C::MI; ++mi) a[mi] = As[(kk + t4) * C::LDS + wm * C::TM + mi * 8 + g];
#pragma unroll
      for (int ni = 0; ni < C::NI; ++ni) b[ni] = Bs[(kk + t4) * C::LDS + wn * C::TN + ni * 8 + g];
#pragma unroll
      for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < C::NI; ++ni) dmma884(acc[mi][ni], a[mi], b[ni]);
    }
  }
  cp_async_wait<0>();

  // ---- epilogue: out = alpha*acc + beta*E, mirrored store, FP64 sums ----
  const bool diag = (bi == bj);
  const double* __restrict__ E = (const double*)p.E;
  double* __restrict__ out = (double*)p.out;
  double s[4] = {0.0, 0.0, 0.0, 0.0};  // ||out||^2, Tr out, ||E-acc||^2 (core rows), Tr acc
#pragma unroll
  for (int mi = 0; mi < C::MI; ++mi) {
#pragma unroll
    for (int ni = 0; ni < C::NI; ++ni) {
      const int r = i0 + wm * C::TM + mi * 8 + g;
      const int c = j0 + wn * C::TN + ni * 8 + 2 * t4;
      const double2 e = *reinterpret_cast<const double2*>(E + (size_t)r * ld + c);
      const double a0 = acc[mi][ni][0], a1 = acc[mi][ni][1];
      const double v0 = alpha * a0 + beta * e.x;
      const double v1 = alpha * a1 + beta * e.y;
      const int w0 = sym_weight(diag, r, c), w1 = sym_weight(diag, r, c + 1);
      const double d0 = e.x - a0, d1 = e.y - a1;
      s[0] += w0 * v0 * v0 + w1 * v1 * v1;
      s[2] += core_weight(w0, r, c, p.core) * d0 * d0 + core_weight(w1, r, c + 1, p.core) * d1 * d1;
      if (r == c) { s[1] += v0; s[3] += a0; }
      if (r == c + 1) { s[1] += v1; s[3] += a1; }
      if (out) {
        if (!diag) {
          *reinterpret_cast<double2*>(out + (size_t)r * ld + c) = make_double2(v0, v1);
          out[(size_t)c * ld + r] = v0;
          out[(size_t)(c + 1) * ld + r] = v1;
        } else {
          if (w0) { out[(size_t)r * ld + c] = v0; out[(size_t)c * ld + r] = v0; }
          if (w1) { out[(size_t)r * ld + c + 1] = v1; out[(size_t)(c + 1) * ld + r] = v1; }
        }
      }
    }
  }
  publish_and_finalize(p, s, red, &s_flag);
}

// Tile edge of a single dense FP64 product of padded size np: the measured choice for this
// device and size (tune_f64_tile) when one was made, else 128 once its tiles fill the SMs
// twice, else 64.
int f64_tile(int np) {
  int c = 0;
  if (tune_lookup(f64_tune_key(np), &c) && (c == 64 || c == 128)) return c;
  const int t128 = np / 128;
  return (t128 * (t128 + 1) / 2 >= 2 * 148) ? 128 : 64;
}

std::string f64_tune_key(int np) {
  return "f64-step/sm" + std::to_string(device_sms()) + "/np" + std::to_string(np);
}

int f64_ntiles(int np) {
  const int t = np / f64_tile(np);
  return t * (t + 1) / 2;
}

static cudaError_t launch_f64_bt(const StepArgs& a, int bt, int ntiles, cudaStream_t st) {
  if (bt == 128) {
    using C = F64Cfg<128, 2, 4>;
    auto kern = k_sym_gemm_f64<128, 2, 4>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    kern<<<ntiles, C::NT, C::SMEM, st>>>(a);
  } else {
    using C = F64Cfg<64, 2, 2>;
    auto kern = k_sym_gemm_f64<64, 2, 2>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    kern<<<ntiles, C::NT, C::SMEM, st>>>(a);
  }
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_sym_gemm_f64(const StepArgs& a0, cudaStream_t st) {
  StepArgs a = a0;
  if (a.ld == 0) a.ld = a.np;
  const int bt = f64_tile(a.np);
  const int t = a.np / bt;
  a.ntiles = t * (t + 1) / 2;   // the partial sums the last CTA reduces: one per launched tile
  return launch_f64_bt(a, bt, a.ntiles, st);
}

// Measures the edges 128 and 64 of a single product at np (x_in -> x_out, the same k order
// per element in both, so the choice changes no result) and records the faster one for
// f64_tile.  partials must hold 4 doubles per 64-edge tile.
int tune_f64_tile(int np, const double* x_in, double* x_out, double* partials, unsigned* counter,
                  double* sums_out, cudaStream_t st) {
  int c = 0;
  const std::string key = f64_tune_key(np);
  if (!tune_enabled() || tune_lookup(key, &c)) return SP2B_OK;
  const int edges[2] = {128, 64};
  StepArgs q;
  memset(&q, 0, sizeof(q));
  q.np = np;
  q.ld = np;
  q.A = q.B = q.E = x_in;
  q.out = x_out;
  q.alpha = 1.0;
  q.partials = partials;
  q.counter = counter;
  q.sums_out = sums_out;
  // timed on zeros (the buffer may not hold data yet; DMMA time does not depend on values)
  if (cudaMemsetAsync(const_cast<double*>(x_in), 0, (size_t)np * np * sizeof(double), st) !=
      cudaSuccess)
    return SP2B_CUDA_ERROR;
  std::vector<float> ms;
  int best = 0;
  const int rc = tune_measure(2, 2, st, [&](int cand) -> int {
    const int t = np / edges[cand];
    return cudaMemsetAsync(counter, 0, 4 * sizeof(unsigned), st) == cudaSuccess &&
                   launch_f64_bt(q, edges[cand], t * (t + 1) / 2, st) == cudaSuccess
               ? SP2B_OK
               : SP2B_CUDA_ERROR;
  }, &ms, &best);
  if (rc == SP2B_OK) tune_store(key, edges[best], ms);
  return rc;
}

}  // namespace sp2b
