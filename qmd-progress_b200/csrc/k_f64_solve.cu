// The dense FP64 SP2 recursion as one persistent cooperative launch: every step's
// symmetric product, the branch update, the sums and the branch decision, and for the
// forward-mode response the anticommutator {X, Delta} beside X^2.
#include <algorithm>
#include <cstring>

#include "f64_tile.cuh"
#include "reduce.cuh"
#include "work_lists.h"

namespace sp2b {

namespace {

// Set in the barrier counter by a CTA that gave up, before it arrives: the others learn of it
// from the word they poll (counts stay below it: CTAs x steps of a launch).
constexpr unsigned kGaveUp = 0x80000000u;

// Waits (at most `limit` polls) until *word >= target; false when the wait ran out or another
// CTA gave up.
__device__ __forceinline__ bool spin_until(const unsigned* word, unsigned target, const int* err,
                                           uint32_t limit) {
  for (uint32_t it = 0; it < limit; ++it) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
    if (v >= target) return !(v & kGaveUp);
    if ((it & 63) == 63 && *(volatile const int*)err) return false;
  }
  return false;
}

constexpr int kSums = kF64Sums;

// Barrier of the consumer warps.
template <int NT>
__device__ __forceinline__ void consumer_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
}

struct F64SolveMaps {
  CUtensorMap x[2], d[2];
};

}  // namespace

// Bound by the DMMA pipe (37 TFLOP/s measured with registers only) and for small orders by the
// chain of one step: its k-blocks, ~4 us per tile epilogue, ~3 us of barrier and decision.  One
// launch per step would add ~10 us of launch, record reads and a last CTA's sums to each,
// padded 128-blocks, idle SMs in the last wave of tiles and, for the response, {X, Delta} as
// two products with a stored middle.  Whole calls on B200, that form -> this one: n = 100 365
// -> 112 us, n = 1000 985 -> 604 us, n = 3500 22.0 -> 18.3 ms (0.88 of the DMMA rate over the
// call), response n = 777 2.40 -> 0.85 ms.
//
// One CTA walks its share of each step's units (F64Split), then all CTAs meet at a grid
// barrier (a counter, bounded wait) and every CTA sums the partials in CTA order and takes
// the same branch decision, so no launch, no host poll and no last-CTA pass lies between
// steps.  A CTA's segments run: the open head of its last tile first (its workspace slot is
// then long full when the owner asks for it), its whole tiles, and last the tile whose head
// other CTAs hold.  The last warp loads (its pipeline runs across segments), the others multiply.
template <int BT>
__global__ void __launch_bounds__(F64Tile<BT>::NT + 32, 1)
    k_f64_solve(const __grid_constant__ F64SolveMaps maps, const __grid_constant__ F64SolveArgs p) {
  using C = F64Tile<BT>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[C::ST], bar_empty[C::ST];
  __shared__ double s_red[kSums][C::NW + 1], s_tot[kSums];
  __shared__ SP2Decision s_dec;
  __shared__ double s_fro2;          // ||X_k||_F^2
  __shared__ int s_run;              // 0: the loop has ended
  __shared__ int s_piece[kMaxPieces], s_npiece;
  __shared__ volatile int s_abort;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int G = (int)gridDim.x, cta = (int)blockIdx.x;
  const bool resp = p.d[0] != nullptr;
  F64Split sp;
  sp.kb = p.kb;
  sp.ntiles = p.ntiles;
  sp.snap = p.snap;
  sp.G = G;
  sp.total = (long long)p.ntiles * p.kb * (resp ? 3 : 1);
  const long long u0 = sp.bound(cta), u1 = sp.bound(cta + 1);
  int ja, oa, jb, ob;
  sp.locate(u0, ja, oa);
  sp.locate(u1, jb, ob);
  const bool open = u1 > u0 && ob > 0;                     // the range ends inside tile jb
  const int nseg = u1 > u0 ? (open ? 1 : 0) + (jb - ja) : 0;
  // segment i: job and its unit range
  auto segment = [&](int i, int& job, int& k0, int& k1) {
    if (open && i == 0) {
      job = jb;
      k0 = ja == jb ? oa : 0;
      k1 = ob;
      return;
    }
    const int q = i - (open ? 1 : 0);   // 0 .. jb - ja - 1: ja + 1, ..., jb - 1, then ja
    job = q + 1 < jb - ja ? ja + 1 + q : ja;
    k0 = job == ja ? oa : 0;
    k1 = sp.len(job);
  };
  const int ld = p.ld;

  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < C::ST; ++s) {
      mbar_init(smem_u32(&bar_full[s]), 1);
      mbar_init(smem_u32(&bar_empty[s]), C::NW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // the CTAs that hold the head of this CTA's first tile, nearest first
    s_npiece = 0;
    if (nseg > (open ? 1 : 0) && oa > 0)
      for (int c = cta - 1; c >= 0 && s_npiece < kMaxPieces; --c) {
        const long long hi = sp.bound(c + 1);
        if (hi <= u0 - oa) break;
        if (sp.bound(c) < hi) s_piece[s_npiece++] = c;
      }
    const SP2Rec r = p.rec[p.k0];
    s_run = 1;
    if (p.k0 > 0 && *(volatile const int*)&p.sout->done) {
      s_run = 0;   // an earlier launch of this solve ended the loop
    } else if (r.done) {
      // reached at k = 0 when normalisation flagged the input
      s_run = 0;
      if (cta == 0) {
        p.rec[p.k0 + 1] = r;
        p.sout->nupd = p.k0;
        p.sout->iter = r.iter;
        p.sout->status = r.status;
        p.sout->done = 1;
      }
    } else {
      s_dec = sp2_decide(p.ctl, r, p.k0, p.pp_in);
      s_fro2 = r.fro2;
    }
  }
  __syncthreads();
  if (warp == C::NW && lane < 4) prefetch_tmap(lane < 2 ? &maps.x[lane] : &maps.d[lane - 2]);
  typename C::Frag frag;
  frag.init(lane);
  uint32_t g = 0;   // units loaded (loader) or consumed so far, over all steps
  for (int k = p.k0; k < p.k1; ++k) {
    if (!s_run) return;
    if (s_dec.branch == BR_STOP) {
      if (cta == 0 && tid == 0) {
        SP2Rec nx = s_dec.next;
        nx.done = 1;
        nx.last_branch = BR_STOP;
        p.rec[k + 1] = nx;
        p.sout->nupd = k;
        p.sout->iter = nx.iter;
        p.sout->status = nx.status;
        p.sout->done = 1;
      }
      return;
    }
    const bool sq = s_dec.branch == BR_X2;
    const double alpha = sq ? 1.0 : -1.0, beta = sq ? 0.0 : 2.0;
    double s[kSums] = {0.0, 0.0, 0.0, 0.0, 0.0};

    if (warp == C::NW) {
      // ---------------- producer ----------------
      if (lane == 0) {
        fence_proxy_async_global();   // the other CTAs' X_k, then the TMA reads
        const CUtensorMap* mx = &maps.x[k & 1];
        const CUtensorMap* md = &maps.d[k & 1];
        bool ok = true;
        for (int seg = 0; seg < nseg && ok; ++seg) {
          int job, k0, k1, bi, bj;
          segment(seg, job, k0, k1);
          const bool isx = job < p.ntiles;
          upper_tile(isx ? job : job - p.ntiles, bi, bj);
          const bool one = isx && bi == bj;   // a diagonal tile of X^2: A and B are the same
          for (int kk = k0; kk < k1; ++kk, ++g) {
            const int st = g % C::ST;
            if (g >= (uint32_t)C::ST &&
                !mbar_wait(smem_u32(&bar_empty[st]), (g / C::ST - 1) & 1, &s_abort)) {
              ok = false;   // no copy into a stage that may still be read
              break;
            }
            const uint32_t fb = smem_u32(&bar_full[st]), dst = sbase + st * C::STAGE;
            const bool second = kk >= p.kb;   // Delta X after X Delta
            const int row = (second ? kk - p.kb : kk) * C::BK;
            mbar_expect_tx(fb, one ? C::OPERAND : C::STAGE);
            tma_load_3d(dst, second ? md : mx, fb, 0, row, bi * (BT / 16));
            if (!one)
              tma_load_3d(dst + C::OPERAND, isx || second ? mx : md, fb, 0, row, bj * (BT / 16));
          }
        }
      }
      __syncwarp();
    } else {
      // ---------------- consumers ----------------
      double2* stash = reinterpret_cast<double2*>(smem_raw + (sbase - smem_u32(smem_raw)) +
                                                  C::ST * C::STAGE) + tid;   // this thread's
      const int am8 = warp / C::WN * C::MI, bn8 = warp % C::WN * C::NI;
      for (int seg = 0; seg < nseg; ++seg) {
        int job, k0, k1, bi, bj;
        segment(seg, job, k0, k1);
        const bool isx = job < p.ntiles;
        upper_tile(isx ? job : job - p.ntiles, bi, bj);
        const bool diag = bi == bj;
        const uint32_t boff = isx && diag ? 0 : C::OPERAND;
        double acc[C::MI][C::NI][2];
#pragma unroll
        for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
          for (int ni = 0; ni < C::NI; ++ni) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
        // E of the tile: read ahead of the products where the registers allow
        const double* E = isx ? p.x[k & 1] : p.d[k & 1];
        double2 ev[C::EARLY_E ? C::MI : 1][C::EARLY_E ? C::NI : 1];
        if (C::EARLY_E) {
#pragma unroll
          for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
            for (int ni = 0; ni < C::NI; ++ni)
              ev[mi][ni] = __ldcg(reinterpret_cast<const double2*>(
                  E + (size_t)(bi * BT + C::row(mi)) * ld + bj * BT + C::col(ni)));
        }
        // X Delta and Delta X are summed apart (one chain of 2 n terms has more rounding
        // error than two of n): the first waits in shared memory
        const bool both = !isx && k0 < p.kb && k1 > p.kb;
        for (int kk = k0; kk < k1; ++kk, ++g) {
          const int st = g % C::ST;
          if (both && kk == p.kb) {
#pragma unroll
            for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
              for (int ni = 0; ni < C::NI; ++ni) {
                stash[(mi * C::NI + ni) * C::NT] = make_double2(acc[mi][ni][0], acc[mi][ni][1]);
                acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
              }
          }
          // A wait that ran out leaves s_abort set and the step void, but every lane goes on: the
          // multiply needs the whole warp, and lanes give up each for itself.
          mbar_wait(smem_u32(&bar_full[st]), (g / C::ST) & 1, &s_abort);
          const uint32_t a = sbase + st * C::STAGE;
          C::mma(a, a + boff, am8, bn8, frag, acc);
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bar_empty[st]));
        }
        if (both) {
#pragma unroll
          for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
            for (int ni = 0; ni < C::NI; ++ni) {
              const double2 v = stash[(mi * C::NI + ni) * C::NT];
              acc[mi][ni][0] += v.x;
              acc[mi][ni][1] += v.y;
            }
        }
        if (open && seg == 0) {
          // the head (or a middle piece) of a tile another CTA finishes
          double2* w = reinterpret_cast<double2*>(p.ws) + (size_t)cta * (BT * BT / 2) + tid;
#pragma unroll
          for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
            for (int ni = 0; ni < C::NI; ++ni)
              w[(mi * C::NI + ni) * C::NT] = make_double2(acc[mi][ni][0], acc[mi][ni][1]);
          consumer_sync<C::NT>();
          if (tid == 0)
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p.flags + cta),
                         "r"((unsigned)(k + 1 - p.k0))
                         : "memory");
          continue;
        }
        if (k0 > 0) {
          // add the pieces other CTAs hold
          for (int q = 0; q < s_npiece; ++q) {
            const int c = s_piece[q];
            if (tid == 0 && !s_abort &&
                !spin_until(p.flags + c, (unsigned)(k + 1 - p.k0), p.err,
                            p.test_wait == 1 ? 0u : kSpinLimit))
              s_abort = 1;
            consumer_sync<C::NT>();
            const double2* w = reinterpret_cast<const double2*>(p.ws) + (size_t)c * (BT * BT / 2) + tid;
#pragma unroll
            for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
              for (int ni = 0; ni < C::NI; ++ni) {
                const double2 v = __ldcg(w + (mi * C::NI + ni) * C::NT);
                acc[mi][ni][0] += v.x;
                acc[mi][ni][1] += v.y;
              }
          }
        }
        // out = alpha acc + beta E, mirrored store, FP64 sums (of X, and Tr Delta')
        double* out = isx ? p.x[(k + 1) & 1] : p.d[(k + 1) & 1];
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
            if (isx) {
              const double d0 = e.x - a0, d1 = e.y - a1;
              if (!diag && p.core <= 0) {
                s[0] += 2.0 * (v0 * v0 + v1 * v1);
                s[2] += 2.0 * (d0 * d0 + d1 * d1);
              } else {
                const int w0 = sym_weight(diag, r, c), w1 = sym_weight(diag, r, c + 1);
                s[0] += w0 * v0 * v0 + w1 * v1 * v1;
                s[2] += core_weight(w0, r, c, p.core) * d0 * d0 +
                        core_weight(w1, r, c + 1, p.core) * d1 * d1;
                if (r == c) { s[1] += v0; s[3] += a0; }
                if (r == c + 1) { s[1] += v1; s[3] += a1; }
              }
            } else {
              if (r == c) s[4] += v0;
              if (r == c + 1) s[4] += v1;
            }
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
      }
      fence_proxy_async_global();   // these stores, then the other CTAs' TMA reads
    }

    // ---- grid barrier, the step's sums and the next decision ----
#pragma unroll
    for (int q = 0; q < kSums; ++q) s[q] = warp_sum(s[q]);
    if (lane == 0)
      for (int q = 0; q < kSums; ++q) s_red[q][warp] = s[q];
    __syncthreads();
    double* part = p.partials + (size_t)(k & 1) * G * kSums;
    if (warp == 0) {
#pragma unroll
      for (int q = 0; q < kSums; ++q) s[q] = warp_sum(lane < C::NW ? s_red[q][lane] : 0.0);
    }
    if (tid == 0) {
      // (the barrier above and this release order the whole block's stores)
      for (int q = 0; q < kSums; ++q) part[(size_t)q * G + cta] = s[q];
      // A wait that ran out is on record before this CTA arrives, so that no CTA passes the
      // barrier on its account and publishes the step as good.
      if (s_abort) {
        atomicExch(p.err, 1);
        atomicOr(p.bar, kGaveUp);
      }
      add_release(p.bar);
      if (!s_abort && !spin_until(p.bar, (unsigned)G * (unsigned)(k + 1 - p.k0), p.err,
                                  p.test_wait == 2 ? 0u : kSpinLimit))
        s_abort = 1;
      if (s_abort) {
        // the call reports SP2B_TIMEOUT (it reads the error word); the other CTAs leave at
        // this barrier or at their next wait
        atomicExch(p.err, 1);
        atomicOr(p.bar, kGaveUp);
        p.sout->status = SP2B_TIMEOUT;
        __threadfence();
        p.sout->done = 1;
      }
    }
    __syncthreads();
    if (s_abort) {
      // leave no copy of this CTA in flight: wait (bounded) for the last ones issued
      if (warp == C::NW && lane == 0)
        for (uint32_t u = g > (uint32_t)C::ST ? g - C::ST : 0; u < g; ++u)
          for (uint32_t i = 0; i < kSpinLimit; ++i)
            if (mbar_try(smem_u32(&bar_full[u % C::ST]), (u / C::ST) & 1)) break;
      return;
    }
    // warp q sums total q over the CTAs, in CTA order per lane
    if (warp < kSums) {
      double v = 0.0;
      for (int j = lane; j < G; j += 32) v += __ldcg(part + (size_t)warp * G + j);
      v = warp_sum(v);
      if (lane == 0) s_tot[warp] = v;
    }
    __syncthreads();
    if (tid == 0) {
      const double* t = s_tot;
      SP2Rec nx = s_dec.next;
      nx.fro2 = t[0];
      nx.trx_data = t[1];
      nx.trp = t[3];
      nx.pbias = s_fro2 - t[3];
      nx.last_branch = s_dec.branch;
      if (!(t[0] == t[0]) || !(t[1] == t[1]) || !(t[2] == t[2]) || t[0] > 1e300) {
        nx.status = SP2B_BAD_INPUT;
        nx.done = 1;
      }
      if (cta == 0) {
        if (p.pp_out) p.pp_out[k] = s_dec.branch;
        if (p.vv_out) {
          if (p.vv_accumulate) p.vv_out[k] += t[2];
          else p.vv_out[k] = sqrt(t[2]);
        }
        if (p.trd_out) *p.trd_out = t[4];
        p.rec[k + 1] = nx;
        p.sout->nupd = k + 1;
        p.sout->iter = nx.iter;
        p.sout->status = nx.status;
        if (nx.done) p.sout->done = 1;
      }
      if (nx.done) {
        s_run = 0;
      } else {
        s_dec = sp2_decide(p.ctl, nx, k + 1, p.pp_in);
        s_fro2 = nx.fro2;
      }
    }
    __syncthreads();
  }
}

namespace {

template <int BT>
cudaError_t launch_solve(const F64SolveArgs& a, int grid, cudaStream_t st) {
  using C = F64Tile<BT>;
  F64SolveMaps m;
  for (int i = 0; i < 2; ++i)
    if (!make_tmap_f64(&m.x[i], a.x[i], a.ld, a.ld, BT) ||
        !make_tmap_f64(&m.d[i], a.d[i] ? a.d[i] : a.x[i], a.ld, a.ld, BT))
      return cudaErrorInvalidValue;
  // the response keeps one tile of sums beside the stages
  const size_t smem = C::SMEM + (a.d[0] ? BT * BT * sizeof(double) : 0);
  const cudaError_t e = cudaFuncSetAttribute(k_f64_solve<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
  if (e != cudaSuccess) return e;
  void* args[] = {(void*)&m, (void*)&a};
  return cudaLaunchCooperativeKernel((const void*)k_f64_solve<BT>, dim3(grid), dim3(C::NT + 32), args,
                                     smem, st);
}

}  // namespace

int f64_solve_chunk(int n, bool resp) { return f64_steps_per_launch(n, resp); }

size_t f64_solve_ws_doubles(int n, bool resp) { return f64_solve_doubles(n, resp, device_sms()); }

cudaError_t launch_f64_solve(const F64SolveArgs& a0, int n, int np, double* work, size_t cap,
                             cudaStream_t st) {
  F64SolveArgs a = a0;
  const bool resp = a.d[0] != nullptr;
  const cudaError_t le = launch_cooperative(st, [&](int sms) {
    const F64Plan pl = f64_plan(n, f64_edge(n, resp), resp, sms);
    if (!work || f64_plan_doubles(pl) > cap) return cudaErrorInvalidValue;
    a.ld = np;
    a.kb = (n + 15) / 16;
    a.ntiles = pl.tiles * (pl.tiles + 1) / 2;
    a.snap = pl.snap;
    a.ws = work;
    a.partials = work + (size_t)pl.grid * pl.bt * pl.bt;
    a.flags = reinterpret_cast<unsigned*>(a.partials + 2 * (size_t)pl.grid * kSums);
    a.bar = a.flags + pl.grid;
    cudaError_t e = cudaMemsetAsync(a.flags, 0, (pl.grid + 1) * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    if (pl.bt == 32) return launch_solve<32>(a, pl.grid, st);
    if (pl.bt == 64) return launch_solve<64>(a, pl.grid, st);
    return launch_solve<128>(a, pl.grid, st);
  });
  note_launch();
  return le == cudaSuccess ? cudaGetLastError() : le;
}

}  // namespace sp2b
