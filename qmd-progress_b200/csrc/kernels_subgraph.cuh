// Launch interfaces of the graph-partitioned SP2 path.
#pragma once
#include "kernels.cuh"

namespace sp2b {

// One core+halo part inside the packed buffers.
struct PartDesc {
  long long row0;   // first packed row
  long long hoff;   // offset of its node list in the halo / sorted arrays
  long long coff;   // offset of its ncore x n block in the packed core-row output
  int n;            // core+halo size (lsize)
  int np;           // n padded to 128
  int ncore;        // core size (llsize)
  int pad_;
};

cudaError_t launch_extract_csr(const long long* rp, const int* col, const double* val,
                               const PartDesc* parts, int nparts, const int* halo,
                               const int* skey, const int* sval, int ld, double* xs,
                               cudaStream_t st);
cudaError_t launch_norm_parts(double* xs, const int* row_part, const PartDesc* parts,
                              long long rows, int ld, double emin, double emax, int prec,
                              void* hi, void* lo, cudaStream_t st);
cudaError_t launch_scatter_parts(const double* x64, const void* hi, const void* lo, int prec,
                                 const PartDesc* parts, int nparts, const int* halo, int ld,
                                 double* core_out, double* dense, long long n, cudaStream_t st);

// CSR extraction and normalisation with the global bounds in one pass (ld <= kFusedLd):
// split precisions into the packed hi/lo buffers, FP64 into xs.
// Up to 2048 eight rows and the node list of a part fit in shared memory (147 KB there, one CTA
// an SM, sized by the largest part).  A call without steps, the two-pass form (clear, extract,
// normalise) -> this: 16 parts of 2000 0.80 -> 0.31 ms, 60 of them 1.60 -> 0.89, 250 of 400 and
// one of 1900 1.36 -> 0.52, 100 of 600 0.39 -> 0.19 (FP64; split and INT8 alike).
constexpr int kFusedLd = 2048;
cudaError_t launch_extract_split(const long long* rp, const int* col, const double* val,
                                 const PartDesc* parts, int nparts, const int* halo,
                                 const int* skey, const int* sval, int ld, double emin,
                                 double emax, int prec, void* hi, void* lo, double* xs,
                                 cudaStream_t st);

// Sum over each part's core rows of (X - X^2)_ii from the split iterate (hi, lo), as
// kPartIdemGroups partial sums per part (out[part * kPartIdemGroups + g]).
constexpr int kPartIdemGroups = 16;
cudaError_t launch_part_idem(const void* hi, const void* lo, int prec, const PartDesc* parts,
                             int nparts, int ld, double* out, cudaStream_t st);

cudaError_t launch_place_core(const long long* hptr, const int* halo, const int* lls,
                              const long long* off, int nparts, const double* src, double* rho,
                              long long n, cudaStream_t st);

// The FP64 batch in one persistent launch (k_f64_parts.cu): tiles {row0, bi << 16 | bj,
// K extent (a multiple of 16), core} of edge bt over each part's upper blocks.
struct F64PartsArgs {
  double* x[2];         // packed ping-pong buffers; x[0] holds X_0
  const int4* tiles;
  const int* tpart;     // part of each tile
  const int* pnt;       // tiles of each part
  const int* pp;        // branch of each step: 0 = 2X - X^2, else X^2
  unsigned* done;       // per part, finished tiles over all steps (zero at launch)
  unsigned* ticket;     // next item (zero at launch)
  double* partials;     // residual sums, f64_parts_partials() doubles (null: not formed)
  int* err;
  int ntiles, nsteps, ld;
  uint32_t polls;       // bound of a tile's wait for its part (0: kSpinLimit)
};
size_t f64_parts_partials(int ntiles, int nsteps, int bt);
cudaError_t launch_f64_parts(const F64PartsArgs& a, int bt, long long rows, double* vv,
                             cudaStream_t st);
// Self-test of its bounded waits on 128 x 128 buffers and 64 bytes of scratch.
cudaError_t launch_f64_parts_selftest(double* x0, double* x1, void* scratch, int bt, int tiles_awaited,
                                      uint32_t polls, int* err, cudaStream_t st);

// Batched INT8 digit-split form (exact INT8 precision of the sub-graph loop): the
// iterate as four signed 8-bit planes of M = rint(2^31 (X - I/2)) in each packed buffer
// (plane s at base + s rows ld).  Tiles {row0, bi << 16 | bj64, K extent, core} of
// 128 x 64 over the upper band of each part's block.  All steps run in one persistent
// launch; vv[k] += the core-row ||X_k - X_k^2||_F^2 of step k.
struct I8StepsArgs {
  const int4* tiles;
  const int* tpart;     // part of each tile
  const int* pnt;       // tiles of each part
  const int* pp;        // branch of each step: 0 = 2X - X^2, else X^2
  unsigned* done;       // per part, finished tiles over all steps (zero at launch)
  double* partials;     // step sums per (step, CTA, epilogue warp): i8_steps_partials (zero)
  int* err;
  int ntiles, nsteps, rows;
};
size_t i8_steps_partials(int nsteps);   // doubles
cudaError_t launch_i8_steps(const I8StepsArgs& a, const void* buf0, const void* buf1, int ld,
                            double* vv, cudaStream_t st);
cudaError_t launch_extract_digits(const long long* rp, const int* col, const double* val,
                                  const PartDesc* parts, int nparts, const int* halo,
                                  const int* skey, const int* sval, int ld, long long rows,
                                  double emin, double emax, int8_t* dig, cudaStream_t st);
cudaError_t launch_norm_digits(const double* xs, const int* row_part, const PartDesc* parts,
                               long long rows, int ld, double emin, double emax, int8_t* dig,
                               cudaStream_t st);
cudaError_t launch_scatter_digits(const int8_t* dig, long long rows, const PartDesc* parts,
                                  int nparts, const int* halo, int ld, double* core_out,
                                  double* dense, long long n, double* idem, cudaStream_t st);

// One warp of the fused extractions: row r of part P as FP64 entries of H in buf[0, np)
// (zero where the CSR row has none or its column is outside the part).  keys / vals: the
// part's sorted node list and local positions, in shared memory (a binary search there
// costs nine shared-memory reads instead of nine dependent trips to L2).
__device__ __forceinline__ void extract_row(const long long* __restrict__ rp,
                                            const int* __restrict__ col,
                                            const double* __restrict__ val, const PartDesc& P,
                                            int node, int lane, const int* keys, const int* vals,
                                            double* buf) {
  for (int c = lane * 2; c < P.np; c += 64) *reinterpret_cast<double2*>(buf + c) = make_double2(0.0, 0.0);
  __syncwarp();
  if (node >= 0)
    for (long long e = rp[node] + lane; e < rp[node + 1]; e += 32) {
      const int u = col[e];
      int a = 0, b = P.n - 1;
      while (a <= b) {
        const int mid = (a + b) >> 1;
        const int key = keys[mid];
        if (key == u) {
          buf[vals[mid]] = val[e];
          break;
        }
        if (key < u) a = mid + 1;
        else b = mid - 1;
      }
    }
  __syncwarp();
}
constexpr size_t extract_smem(int ld) { return (size_t)ld * (8 * sizeof(double) + 2 * sizeof(int)); }

}  // namespace sp2b
