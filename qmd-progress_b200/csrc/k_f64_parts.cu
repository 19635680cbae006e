// The FP64 sub-graph loop as one persistent cooperative launch: every SP2 step of every
// part, in any number of parts (the whole batch, or the few parts that a reduced-precision
// solve flags for FP64).
#include <algorithm>
#include <cstring>

#include "f64_tile.cuh"
#include "kernels_subgraph.cuh"
#include "reduce.cuh"

namespace sp2b {

namespace {

struct F64PartsMaps {
  CUtensorMap x[2];   // the packed ping-pong buffers
};

}  // namespace

// An item is one BT x BT upper tile of one part at one step, numbered step by step in tile
// list order.  The loader warp draws the next item from a counter (so a CTA that got cheap
// tiles takes more of them), waits until its part has finished the step before (a count of
// the part's finished tiles, bounded wait) and streams the operands; items of lower number
// are all finished or held by a running CTA, so the waits end.  No barrier joins the parts:
// small ones run ahead while large ones still multiply.  The item of each operand stage
// travels with it (s_item; -1 ends the consumers).
//
// Tiles and k-blocks stop at the part's size (edge and 16), not at the 128-padded one, and
// every element sums k in ascending order whatever the edge: results do not depend on it.
// A consumer's own wait ends unless a copy never arrives: the loader issues every k-block of an
// item that it announces, and the end mark last, whatever ended it.
// Residual sums go out per tile and warp and are added in a fixed order afterwards.
//
// Bound by the DMMA pipe, and for a few parts by the chain of one step: operand latency,
// n/4 dependent fragments, epilogue, part count.  Per-step launches over padded tiles
// (with a block barrier per k-block and whole-grid steps) took 60 us a step for the 32 parts
// of a 16^3 lattice.
template <int BT>
__global__ void __launch_bounds__(F64Tile<BT>::NT + 32, BT == 32 ? 2 : 1)
    k_f64_parts(const __grid_constant__ F64PartsMaps maps, const __grid_constant__ F64PartsArgs p) {
  using C = F64Tile<BT>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[C::ST], bar_empty[C::ST];
  __shared__ int s_item[C::ST];
  __shared__ volatile int s_abort;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < C::ST; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), C::NW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int nitems = p.ntiles * p.nsteps;

  if (warp == C::NW) {
    // ---------------- loader ----------------
    if (lane == 0) {
      prefetch_tmap(&maps.x[0]);
      prefetch_tmap(&maps.x[1]);
      uint32_t g = 0;
      bool ok = true;
      while (ok) {
        const int item = (int)atomicAdd(p.ticket, 1u);
        if (item >= nitems) break;
        const int k = item / p.ntiles, t = item - k * p.ntiles;
        const int4 tl = p.tiles[t];
        if (k > 0) {
          const int part = p.tpart[t];
          const unsigned need = (unsigned)p.pnt[part] * (unsigned)k;
          ok = false;
          for (uint32_t it = 0; it < p.polls; ++it) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p.done + part) : "memory");
            if (v >= need) { ok = true; break; }
            if ((it & 63) == 63 && *(volatile const int*)p.err) break;
          }
          if (!ok) {
            // The call reports SP2B_TIMEOUT.  The consumers learn of it in the order of the
            // items, by the end mark: all warps finish what was loaded and leave together (one
            // that left by itself would keep the others at the barrier of its tile).
            atomicExch(p.err, 1);
            ok = true;
            break;
          }
          fence_proxy_async_global();   // the other CTAs' results, then the TMA reads
        }
        const CUtensorMap* mx = &maps.x[k & 1];
        const int bi = tl.y >> 16, bj = tl.y & 0xffff;
        for (int kk = 0; kk < tl.z; kk += C::BK, ++g) {
          const int st = g % C::ST;
          if (g >= (uint32_t)C::ST &&
              !mbar_wait(smem_u32(&bar_empty[st]), (g / C::ST - 1) & 1, &s_abort)) {
            ok = false;
            break;
          }
          const uint32_t fb = smem_u32(&bar_full[st]), dst = sbase + st * C::STAGE;
          s_item[st] = item;
          mbar_expect_tx(fb, bi == bj ? C::OPERAND : C::STAGE);   // diagonal: A and B are the same
          tma_load_3d(dst, mx, fb, 0, tl.x + kk, bi * (BT / 16));
          if (bi != bj) tma_load_3d(dst + C::OPERAND, mx, fb, 0, tl.x + kk, bj * (BT / 16));
        }
      }
      if (ok) {
        // the end mark, in the next free stage
        const int st = g % C::ST;
        if (g < (uint32_t)C::ST ||
            mbar_wait(smem_u32(&bar_empty[st]), (g / C::ST - 1) & 1, &s_abort)) {
          s_item[st] = -1;
          mbar_arrive(smem_u32(&bar_full[st]));
        }
        // every stage consumed: no consumer gave up (asked here and not by the consumers: code
        // behind their loop makes the compiler reconverge inside it, 6 % at 16^3)
        for (uint32_t u = g > (uint32_t)C::ST ? g - C::ST : 0; u < g; ++u)
          if (!mbar_wait(smem_u32(&bar_empty[u % C::ST]), (u / C::ST) & 1, &s_abort)) {
            atomicExch(p.err, 1);
            break;
          }
      } else {
        // no stage came free: the consumers gave up too (s_abort); no copy stays in flight
        atomicExch(p.err, 1);
        for (uint32_t u = g > (uint32_t)C::ST ? g - C::ST : 0; u < g; ++u)
          for (uint32_t i = 0; i < kSpinLimit; ++i)
            if (mbar_try(smem_u32(&bar_full[u % C::ST]), (u / C::ST) & 1)) break;
      }
    }
    return;
  }

  // ---------------- consumers ----------------
  const int am8 = warp / C::WN * C::MI, bn8 = warp % C::WN * C::NI;
  const int ld = p.ld;
  typename C::Frag frag;
  frag.init(lane);
  uint32_t g = 0;
  for (;;) {
    if (!mbar_wait_idle(smem_u32(&bar_full[g % C::ST]), (g / C::ST) & 1, &s_abort)) break;
    const int item = *(volatile int*)&s_item[g % C::ST];
    if (item < 0) break;
    const int k = item / p.ntiles, t = item - k * p.ntiles;
    const int4 tl = p.tiles[t];
    const int bi = tl.y >> 16, bj = tl.y & 0xffff, core = tl.w;
    const bool diag = bi == bj;
    const uint32_t boff = diag ? 0 : C::OPERAND;
    double acc[C::MI][C::NI][2];
#pragma unroll
    for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
      for (int ni = 0; ni < C::NI; ++ni) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
    const size_t base = (size_t)tl.x * ld;
    const double* E = ((k & 1) ? p.x[1] : p.x[0]) + base;
    // E of the tile: read ahead of the products where the registers allow
    double2 ev[C::EARLY_E ? C::MI : 1][C::EARLY_E ? C::NI : 1];
    if (C::EARLY_E) {
#pragma unroll
      for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < C::NI; ++ni)
          ev[mi][ni] = __ldcg(reinterpret_cast<const double2*>(
              E + (size_t)(bi * BT + C::row(mi)) * ld + bj * BT + C::col(ni)));
    }
    bool ok = true;
    for (int kk = 0; kk < tl.z; kk += C::BK, ++g) {
      const int st = g % C::ST;
      ok = mbar_wait(smem_u32(&bar_full[st]), (g / C::ST) & 1, &s_abort);
      if (!ok) break;
      const uint32_t a = sbase + st * C::STAGE;
      C::mma(a, a + boff, am8, bn8, frag, acc);
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bar_empty[st]));
    }
    if (!ok) break;
    // out = alpha acc + beta E, mirrored store, the residual over the part's core rows
    const bool sq = p.pp[k] != 0;
    const double alpha = sq ? 1.0 : -1.0, beta = sq ? 0.0 : 2.0;
    double* out = ((k & 1) ? p.x[0] : p.x[1]) + base;
    double res = 0.0;
#pragma unroll
    for (int mi = 0; mi < C::MI; ++mi) {
#pragma unroll
      for (int ni = 0; ni < C::NI; ++ni) {
        const int r = bi * BT + C::row(mi), c = bj * BT + C::col(ni);
        const double2 e = C::EARLY_E
                              ? ev[C::EARLY_E ? mi : 0][C::EARLY_E ? ni : 0]
                              : __ldcg(reinterpret_cast<const double2*>(E + (size_t)r * ld + c));
        const double a0 = acc[mi][ni][0], a1 = acc[mi][ni][1];
        const double v0 = alpha * a0 + beta * e.x;
        const double v1 = alpha * a1 + beta * e.y;
        const double d0 = e.x - a0, d1 = e.y - a1;
        const int w0 = sym_weight(diag, r, c), w1 = sym_weight(diag, r, c + 1);
        res += core_weight(w0, r, c, core) * d0 * d0 + core_weight(w1, r, c + 1, core) * d1 * d1;
        if (!diag) {
          *reinterpret_cast<double2*>(out + (size_t)r * ld + c) = make_double2(v0, v1);
          out[(size_t)c * ld + r] = v0;
          out[(size_t)(c + 1) * ld + r] = v1;
        } else {
          if (r <= c) { out[(size_t)r * ld + c] = v0; out[(size_t)c * ld + r] = v0; }
          if (r <= c + 1) { out[(size_t)r * ld + c + 1] = v1; out[(size_t)(c + 1) * ld + r] = v1; }
        }
      }
    }
    fence_proxy_async_global();   // these stores, then the other CTAs' TMA reads
    // (the barrier and the release order the whole block's stores)
    asm volatile("bar.sync 1, %0;" ::"n"(C::NT) : "memory");
    if (tid == 0) add_release(p.done + p.tpart[t]);
    if (p.partials) {
      res = warp_sum(res);
      if (lane == 0) p.partials[(size_t)item * C::NW + warp] = res;
    }
  }
}

// vv[k] = the residual sums of step k, one block per step, in a fixed order.
__global__ void __launch_bounds__(256)
    k_f64_parts_sums(const double* __restrict__ partials, int per_step, double* __restrict__ vv) {
  __shared__ double red[32];
  const double* q = partials + (size_t)blockIdx.x * per_step;
  double s[1] = {0.0};
  for (int j = threadIdx.x; j < per_step; j += blockDim.x) s[0] += q[j];
  block_sum<1>(s, red);
  if (threadIdx.x == 0) vv[blockIdx.x] = s[0];
}

template <int BT>
static cudaError_t launch_parts(const F64PartsArgs& a, long long rows, cudaStream_t st) {
  using C = F64Tile<BT>;
  F64PartsMaps m;
  for (int i = 0; i < 2; ++i)
    if (!make_tmap_f64(&m.x[i], a.x[i], rows, a.ld, BT)) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(k_f64_parts<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)C::SMEM);
  if (e != cudaSuccess) return e;
  void* args[] = {(void*)&m, (void*)&a};
  e = launch_cooperative(st, [&](int sms) {
    const int grid = std::min(a.ntiles, sms * (BT == 32 ? 2 : 1));
    return cudaLaunchCooperativeKernel((const void*)k_f64_parts<BT>, dim3(grid), dim3(C::NT + 32),
                                       args, C::SMEM, st);
  });
  note_launch();
  return e;
}

size_t f64_parts_partials(int ntiles, int nsteps, int bt) {
  return (size_t)ntiles * nsteps * (bt == 32 ? F64Tile<32>::NW : F64Tile<64>::NW);
}

cudaError_t launch_f64_parts(const F64PartsArgs& a0, int bt, long long rows, double* vv,
                             cudaStream_t st) {
  F64PartsArgs a = a0;
  if (a.polls == 0) a.polls = kSpinLimit;
  if (a.ntiles <= 0 || a.nsteps <= 0) return cudaSuccess;
  // item numbers are 32-bit
  if ((long long)a.ntiles * a.nsteps > 0x7fffffffLL - 4096) return cudaErrorInvalidValue;
  cudaError_t e = bt == 32 ? launch_parts<32>(a, rows, st) : launch_parts<64>(a, rows, st);
  if (e != cudaSuccess || !a.partials) return e;
  const int per = a.ntiles * (bt == 32 ? F64Tile<32>::NW : F64Tile<64>::NW);
  k_f64_parts_sums<<<a.nsteps, 256, 0, st>>>(a.partials, per, vv);
  note_launch();
  return cudaGetLastError();
}

// One part of one tile, two steps.  With two tiles to wait for after the first step, the
// second step's wait runs out after `polls` polls; with one, the launch ends without error.
cudaError_t launch_f64_parts_selftest(double* x0, double* x1, void* scratch, int bt, int tiles_awaited,
                                      uint32_t polls, int* err, cudaStream_t st) {
  constexpr int ld = 128;
  struct Lists {
    int4 tile;
    int tpart, pnt, pp[2];
    unsigned done, ticket;
  } h;
  memset(&h, 0, sizeof(h));
  h.tile = make_int4(0, 0, 32, 32);
  h.pnt = tiles_awaited;
  cudaError_t e = cudaMemsetAsync(x0, 0, (size_t)ld * ld * sizeof(double), st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(scratch, &h, sizeof(h), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  Lists* d = static_cast<Lists*>(scratch);
  F64PartsArgs a;
  memset(&a, 0, sizeof(a));
  a.x[0] = x0;
  a.x[1] = x1;
  a.tiles = &d->tile;
  a.tpart = &d->tpart;
  a.pnt = &d->pnt;
  a.pp = d->pp;
  a.done = &d->done;
  a.ticket = &d->ticket;
  a.err = err;
  a.ntiles = 1;
  a.nsteps = 2;
  a.ld = ld;
  a.polls = polls;
  e = launch_f64_parts(a, bt, ld, nullptr, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);   // (h leaves scope)
  return e;
}

}  // namespace sp2b
