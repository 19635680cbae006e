// Per-device library context and the dense-solve job description.
#pragma once
#include <algorithm>
#include <mutex>
#include <vector>

#include "kernels.cuh"

namespace sp2b {

struct Ctx {
  bool init = false;
  int dev = -1;
  cudaStream_t stream = nullptr;
  std::mutex mu;
  // FP64 square buffers (np x np): ping-pong iterates [0, 1]; the FP64-DMMA McWeeny
  // product [2]; the forward-mode response's Delta ping-pong [2, 3] and host staging [4]
  double* x64[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  size_t x64_cap[5] = {0, 0, 0, 0, 0};
  // FP64 solve: pieces of cut tiles, partial sums, flags
  double* f64w = nullptr;
  size_t f64w_cap = 0;
  // split-precision iterates (hi/lo ping-pong)
  __half* hi[2] = {nullptr, nullptr};
  __half* lo[2] = {nullptr, nullptr};
  size_t hi_cap[2] = {0, 0}, lo_cap[2] = {0, 0};
  // host-pointer staging of H / rho (n x n)
  double* hin = nullptr;
  size_t hin_cap = 0;
  // reductions and control
  double* partials = nullptr;
  size_t partials_cap = 0;
  unsigned* counter = nullptr;
  SP2Rec* rec = nullptr;
  size_t rec_cap = 0;
  int* pp_dev = nullptr;
  size_t pp_cap = 0;
  double* vv_dev = nullptr;
  size_t vv_cap = 0;
  double* rowsum = nullptr;
  size_t rowsum_cap = 0;
  // one small device block and its pinned mirror: scratch scalars, then what a solve reads
  // back in one copy: the normalisation's {min, max, trace, ||X0||^2}, the outcome, the
  // reduction counters and the error word
  double* small = nullptr;
  double* h_small = nullptr;
  double* norm_out = nullptr;   // small + kNorm
  SolveOut* sout = nullptr;     // behind norm_out
  SolveOut* h_sout = nullptr;
  int* err = nullptr;
  const int* h_err = nullptr;
  // doubles read back: 4, sizeof(SolveOut) / 8, four counters, the error word
  static constexpr int kNorm = 48, kBack = 4 + 3 + 2 + 1;
  cudaEvent_t poll = nullptr;   // the outcome copy of a poll
  char* pin = nullptr;          // pinned: pp, vv and the refinement's scale of a solve
  size_t pin_cap = 0;
  // INT8 refinement: residue planes, reduced product planes, work list, scale state
  int8_t* oz_res = nullptr;
  uint8_t* oz_q = nullptr;
  size_t oz_cap = 0;
  int4* oz_work = nullptr;
  int oz_work_np = 0, oz_nwork = 0, oz_grid = 0;
  void* oz_scale = nullptr;
  unsigned long long* oz_rsum = nullptr;   // exact steps: row norm sums of the iterate
  size_t oz_rsum_cap = 0;
  int oz_last_S = 0;            // scale exponent of the last INT8 refinement
  double oz_last_r2max = 0.0;   // its largest squared row norm
  int last_launches = 0;            // SP2 step launches of the last dense solve
  std::vector<cudaEvent_t> ev;      // step timing events (pairs)
  std::vector<cudaEvent_t> ev_ref;  // INT8 refinement phase boundaries

  // zeroes the outcome, the counters and the error word
  cudaError_t clear_control(cudaStream_t st) {
    return cudaMemsetAsync(sout, 0, (char*)(err + 1) - (char*)sout, st);
  }
  // norm_out, the outcome and the error word into the pinned mirror
  cudaError_t read_back(cudaStream_t st) {
    return cudaMemcpyAsync(h_small + kNorm, norm_out, kBack * sizeof(double),
                           cudaMemcpyDeviceToHost, st);
  }
  cudaError_t ensure_pin(size_t bytes);
  cudaError_t ensure_f64(int np, int nbuf);
  cudaError_t ensure_f64_solve(int n, bool resp);
  cudaError_t ensure_split(int np);
  cudaError_t ensure_common(size_t nin, int np, int maxlaunch, int n);
  cudaError_t ensure_oz(int np, cudaStream_t st);
};

static_assert(sizeof(SolveOut) == 24, "the outcome follows norm_out in one read-back");

Ctx* get_ctx(int* status);

struct DenseJob {
  const double* h;
  double* rho;
  int n;
  int prec;
  bool dev_ptrs;
  cudaStream_t stream;
  bool inplace;        // H read from rho (the *_inplace routines)
  bool given_bounds;   // use mineval/maxeval instead of Gershgorin
  double mineval, maxeval;
  SP2Ctl ctl;
  const int* pp_in;
  int* pp_out;
  double* vv_out;
  int vv_accumulate;
  int core;
  int* icount_out;
  int* iters_out;
  double* bounds_out;
  int mcweeny;
  int mcweeny_products;  // SP2B_MCW_INT8 or SP2B_MCW_FP64
  int exact_switch;      // mixed: steps after which a still-running loop restarts exact
  const double* h1;      // forward-mode response: perturbation H1 (nullptr: plain solve)
  double* rsp;           // ... and its output, the response rho1 = 2 Delta
  int test_wait;         // self-test of an FP64 solve's bounded waits (F64SolveArgs)
};

int dense_solve(const DenseJob& j);

}  // namespace sp2b
