// Launch interfaces shared by the sp2b translation units.
#pragma once
#include <string>
#include <vector>

#include "sp2b_common.cuh"

namespace sp2b {

// Counts kernel launches issued by the library (diagnostics / bench).
void note_launch(int k = 1);
long long launch_count();
void set_launch_count(long long v);

// A launch that may start before the launch ahead of it in the stream has completed
// (programmatic dependent launch): the kernel waits for it (grid_wait) before it reads or
// writes anything of another launch.
template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kern)(P...), int grid, int threads, int smem,
                                  cudaStream_t st, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  note_launch();
  return e;
}

// Outcome of a dense solve, written by the device.
struct SolveOut {
  int done;     // loop finished
  int nupd;     // number of X updates applied (final X lives in buffer nupd & 1)
  int status;   // SP2B_* code
  int iter;     // Fortran iteration count ("icount")
  double err;   // ALGO_MIXED: Tr X - Tr P of the last update (its stop reason)
};

// Arguments of one symmetric-tile product launch (FP64 or split precision).
//   acc(m, n) = sum_k A[k][m] * B[k][n]   (A, B stored np x np, symmetric)
//   out       = alpha * acc + beta * E     (upper tiles computed, mirrored on store)
// In control mode (ctl/rec set) alpha/beta come from the SP2 branch rule.
struct StepArgs {
  const void* A;
  const void* B;
  const void* A_lo;     // split mode: lo halves of the operands
  const void* B_lo;
  const void* E;        // elementwise operand (FP64; or hi/lo pair in split mode)
  void* out;            // nullptr: sums only
  const void* E_lo;     // split mode: lo half of E
  void* out_lo;         // split mode: lo half of out
  int np;               // padded dimension of a dense solve
  int ld;               // row pitch of A/B/E/out (dense: np; batched parts: max padded size)
  int ntiles;
  // Batched parts (tiles != nullptr): CTA b works on tile tiles[b] =
  //   {x: first packed row of its part, y: (bi << 16) | bj, z: padded part size, w: core rows}
  const int4* tiles;
  double alpha, beta;
  int core;             // > 0: residual sums over the first `core` rows only
  // SP2 control (control = 1)
  int control;
  SP2Ctl ctl;
  SP2Rec* rec;
  int k;
  const int* pp_in;
  int* pp_out;
  double* vv_out;
  int vv_accumulate;    // 1: vv_out[k] += res (submatrix); 0: vv_out[k] = sqrt(res)
  SolveOut* sout;
  // reductions
  double* partials;     // [ntiles][4]
  unsigned* counter;
  double* sums_out;     // non-control: the 4 totals {||out||^2, Tr out, ||E-acc||^2, Tr acc}
  int* err;             // device error word (timeouts)
  int n_out, ld_out;    // McWeeny combine: the n_out x n_out density and its row pitch
};

// FP64 path ---------------------------------------------------------------------------
int f64_tile(int np);  // tile edge of a single product of this size (64 or 128)
std::string f64_tune_key(int np);
int tune_f64_tile(int np, const double* x_in, double* x_out, double* partials, unsigned* counter,
                  double* sums_out, cudaStream_t st);
int device_sms();       // SM count of the current device
int stream_sms(cudaStream_t st);   // SMs that launches on st may use (fewer in a green context)

// A cooperative launch whose grid run(sms) sizes for so many SMs: those of the stream, and
// fewer while the driver refuses the grid as too large to be resident (a share of the SMs that
// the stream does not show).
template <typename F>
inline cudaError_t launch_cooperative(cudaStream_t st, F&& run) {
  for (int sms = stream_sms(st);; sms = (sms + 1) / 2) {
    const cudaError_t e = run(sms);
    if (e != cudaErrorCooperativeLaunchTooLarge || sms <= 1) return e;
    (void)cudaGetLastError();
  }
}
int f64_ntiles(int np);
cudaError_t launch_gersh(const double* h, int n, int ld, double* rowsum, int nsplit,
                         double* bounds, double* partials, unsigned* counter, cudaStream_t st);
int gersh_nsplit(int n);
cudaError_t launch_normalize_f64(const double* h, int n, int ld, int np, const double* bounds,
                                 double* x, double* partials, unsigned* counter, SP2Rec* rec0,
                                 double* norm_out, cudaStream_t st);
cudaError_t launch_sym_gemm_f64(const StepArgs& a, cudaStream_t st);

// SP2 steps [k0, k1) of a dense solve in one cooperative launch (k_f64_solve.cu); fewer
// when the loop ends first.  With d[0] != nullptr each step also forms the response
// Delta' = a {X, Delta} + b Delta, (a, b) the step's branch.
struct F64SolveArgs {
  double* x[2];         // ping-pong iterates, np x np; x[k0 & 1] holds X_k0
  double* d[2];         // ping-pong Delta, or null
  int k0, k1;
  int core;             // > 0: residual sums over the first `core` rows only
  SP2Ctl ctl;
  SP2Rec* rec;
  const int* pp_in;
  int* pp_out;
  double* vv_out;
  int vv_accumulate;
  double* trd_out;      // Tr Delta' of the last step taken (may be null)
  SolveOut* sout;
  int* err;
  int test_wait;        // self-test: 1 the waits for pieces run out, 2 the grid barrier's
  // set by launch_f64_solve
  int ld, kb, ntiles, snap;
  double* ws;           // one BT x BT piece per CTA
  double* partials;
  unsigned* flags;      // per CTA: its piece of step k is complete (k + 1 - k0)
  unsigned* bar;        // grid barrier counter
};
// Workspace of an order-n solve: with a response also of solves of that order without one.
size_t f64_solve_ws_doubles(int n, bool resp);
int f64_solve_chunk(int n, bool resp);
// cudaErrorInvalidValue when the launch would not fit the `cap` doubles at `work`.
cudaError_t launch_f64_solve(const F64SolveArgs& a, int n, int np, double* work, size_t cap,
                             cudaStream_t st);

cudaError_t launch_finish_f64(const double* x, int np, int n, double scale, double* rho,
                              int ld, cudaStream_t st);
// rho = 2 X of the iterate that a finished solve left in x[nupd & 1], chosen on the device;
// nothing when the solve has not ended, a wait in it ran out (*err) or its normalisation
// (norm: bounds, trace, ||X0||_F^2) was not finite.
cudaError_t launch_finish_solve_f64(const double* x0, const double* x1, const SolveOut* sout,
                                    const int* err, const double* norm, int np, int n, double* rho,
                                    int ld, cudaStream_t st);
cudaError_t launch_copy_in(const double* src, int n, int ld, int np, double* x,
                           cudaStream_t st);
cudaError_t launch_mirror_lower(double* a, int n, int ld, cudaStream_t st);
cudaError_t launch_resp_init(const double* h1, int n, int ld, int np, const double* bounds,
                             double* d, cudaStream_t st);

// Split-precision (tcgen05) path ------------------------------------------------------
int tc_ntiles(int np);
cudaError_t launch_normalize_split(const double* h, int n, int ld, int np,
                                   const double* bounds, __half* hi, __half* lo, int bf16,
                                   double* partials, unsigned* counter, SP2Rec* rec0,
                                   double* norm_out, cudaStream_t st);
cudaError_t launch_sym_gemm_tc(const StepArgs& a, int bf16, cudaStream_t st);
// {G, X} = G X + X G of symmetric split matrices (A = G, B = X) on the upper tiles in one
// pass over the concatenated K range; out = alpha {G, X} + beta E.  FP16 split only;
// cudaErrorNotSupported unless np is at most 1280 or a multiple of 256.
cudaError_t launch_anti_tc(const StepArgs& a, cudaStream_t st);
// batched parts: A/B tensors are rows x ld packed buffers
cudaError_t launch_sym_gemm_tc_batched(const StepArgs& a, long long rows, int bf16,
                                       cudaStream_t st);
cudaError_t launch_split_to_f64(const __half* hi, const __half* lo, int np, int bf16,
                                double* x, cudaStream_t st);
cudaError_t launch_wait_selftest(uint32_t limit, int* err, cudaStream_t st);
cudaError_t launch_f32_rows_to_split(const float* a, int m, int n, int mp, int np, __half* hi,
                                     __half* lo, cudaStream_t st);
cudaError_t launch_tc_panel(const __half* ahi, const __half* alo, int mp, const __half* bhi,
                            const __half* blo, int np, float* c, int m, int n, cudaStream_t st,
                            int* err);
cudaError_t launch_f32_to_split(const float* a, int n, int np, __half* hi, __half* lo,
                                cudaStream_t st);
cudaError_t launch_mcweeny_tc(const __half* xhi, const __half* xlo, const __half* rhi,
                              const __half* rlo, const double* x2, int np, int bf16, double* d,
                              int n, int ldd, double* partials, unsigned* counter,
                              double* sums_out, int* err, cudaStream_t st);

// INT8 (Ozaki residue) refinement products -------------------------------------------
int oz_nmod();
size_t oz_scale_bytes();
int oz_work_list(int np, std::vector<int4>& out);   // returns the grid it is dealt to
cudaError_t launch_oz_planes(const __half* xhi, const __half* xlo, int np, int bf16,
                             void* scale, int8_t* res, cudaStream_t st);
// SP2-step context of the launches that compute one step's X^2 in the exact INT8 mode.
struct OzStepCtl {
  const SolveOut* sout;
  const SP2Rec* rec;
  const int* pp_in;
  SP2Ctl ctl;
  int k;
  int active;   // 0: not part of an SP2 step (the McWeeny refinement)
};
cudaError_t launch_oz_gemm(const int8_t* res, int np, uint8_t* qout, const int4* work,
                           int nwork, int grid, int* err, cudaStream_t st,
                           const OzStepCtl* ctl = nullptr);
cudaError_t launch_oz_planes_f64(const double* x, int np, void* scale, unsigned long long* rsum,
                                 bool first, int8_t* res, const OzStepCtl* ctl, cudaStream_t st);
size_t oz_rsum_words(int np);   // row norm sums of the iterate a step writes
cudaError_t launch_oz_crt_step(const uint8_t* q, void* scale, const StepArgs& a,
                               unsigned long long* rsum, int8_t* res, cudaStream_t st);
cudaError_t launch_oz_crt(const uint8_t* q, const __half* xhi, const __half* xlo, int np,
                          int bf16, const void* scale, double* x2, __half* rhi, __half* rlo,
                          cudaStream_t st);
cudaError_t oz_copy_scale(const void* scale, void* pinned, cudaStream_t st);
void oz_scale_values(const void* pinned, int* S, double* r2max);
cudaError_t launch_tc_plain(const __half* ahi, const __half* alo, const __half* bhi,
                            const __half* blo, int np, float* c, int n, cudaStream_t st,
                            int* err);

}  // namespace sp2b
