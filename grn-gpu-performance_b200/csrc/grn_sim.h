// grn_sim.h -- launch interface between the host evaluator and the
// simulation kernels (grn_sim_kernel.cu).  Internal to the library.
#ifndef GRN_SIM_H_
#define GRN_SIM_H_

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <cmath>

#include "grn_packed.h"

namespace grn {

// Everything a simulation launch reads or writes.  Pointers are device
// pointers.
struct SimArgs {
  const uint4 *packed;       // model records (grn_packed.h)
  const int32_t *offsets;    // [n_models] first word of each record
  int32_t n_models;
  int32_t n_exp;             // experiments
  int32_t n_in;              // input morphogens (initial channels)
  int32_t n_target;          // target morphogens
  int32_t W, H;              // grid width (x) and height (y)
  int32_t Wg;                // float4 groups per row = ceil(W / 4)
  uint32_t inv_wg;           // inverse(Wg) (unused when Wg is 1)
  int32_t wg_shift;          // inverse_shift(Wg)
  uint32_t inv_w;            // ceil(2^32 / W): a cell's row by multiplication, or 0
                             // where that is not exact
  int32_t row_floats, row_bytes;      // one padded state row
  int32_t row_pad;                    // floats after every two rows (strip_pad or 0)
  int32_t plane_floats, plane_bytes;  // one state plane (of a CTA's band)
  int32_t gmax;              // genes a global state slot (or a streaming
                             // stage) holds
  int32_t n_steps;           // max Euler steps per experiment
  int32_t fitness_kind;      // grn_fitness_kind
  int32_t planes;            // shared-memory state planes per block (even)
  int32_t fast_ok;           // experiments allow the fast path (non-negative
                             // finite initial state, minConc >= 0)
  float dt;
  float min_conc;
  double min_conc_change;
  float change_bound;        // the largest float <= min_conc_change: a step's
                             // change (a float) exceeds both or neither
  double dist_threshold;
  const float *initial;      // [n_exp][n_in][H][W]
  const float *target;       // [n_exp][n_target][H][W]
  const double *max_error;   // [caller index]
  double *raw_error;         // [caller index] out
  int32_t *steps;            // [caller index] out, may be null
  int32_t *work_counter;     // zeroed before the launch
  int32_t *error_flag;       // set non-zero on an internal error
  float *gstate;             // global state slots, one per block (or null)
  int64_t slot_floats;       // floats per global state slot
  float *state_out;          // optional final states
                             // [caller index][n_exp][state_planes][H][W]
  int32_t state_planes;
  int32_t trace_every;       // steps between trace frames (frame 0: initial)
  float *trace_out;          // optional trace frames [caller index][n_exp]
                             // [trace_frames][state_planes][H][W]
  int32_t trace_frames;
  int32_t band_rows;         // streaming schedule: rows per staged band
  int32_t test_hooks;        // kHook* bits (tests of the error paths)
};

// Test hooks (grn_set_test_hooks): make a bounded wait run out on purpose.
constexpr int32_t kHookWithholdBandCopy = 1;  // streaming: band 1's copy is never issued
constexpr int32_t kHookWithholdChunkCount = 8;  // steps without a block barrier: no wait for
                                                // chunk 0 (of a cluster's first CTA) ends

// One compiled kernel variant.
struct KernelVariant {
  int max_threads;  // most threads per block
  bool loop;    // warps walk the grid's strips (any grid size); else a warp
                // owns one chunk of 32 strips (strip_chunks)
  bool ragged;  // compiled for W not a multiple of 4
  bool cluster; // cluster-split: a cluster of CTAs per model, one band of
                // rows each
  bool trace;   // writes trace frames (SimArgs::trace_out)
  int stream;   // 0; 1 streaming schedule (SimArgs::band_rows); 2 streaming
                // with two Euler steps per pass (temporal blocking)
};

// Launch plan chosen by the host.
struct LaunchPlan {
  KernelVariant v;
  int schedule;          // grn_schedule actually used
  int threads;           // threads per block (whole warps)
  int gmax;              // genes per global state slot or streaming stage
  int blocks;            // persistent grid size
  int planes;            // state planes in shared memory (even; may be 0)
  size_t smem_bytes;     // dynamic shared memory
  int blocks_per_sm;
  int64_t slot_floats;   // floats of one block's global state slot (0: none)
  int cluster;           // CTAs per cluster (1: one CTA per model)
  int band_rows;         // streaming schedule: rows per staged band (else 0)
  int row_pad;           // floats after every two rows of a plane: strip_pad or 0
};

#ifdef __CUDACC__
#define GRN_HOST_DEVICE __host__ __device__
#else
#define GRN_HOST_DEVICE
#endif

// Floats of one padded state row: W rounded up to float4 groups, plus one
// zero group when W is a multiple of 4, so that every row ends in at least
// one zero cell (the right border of its last cell and the left border of
// the next row's first cell).
GRN_HOST_DEVICE inline int row_floats(int W) {
  return 4 * ((W + 3) / 4) + (W % 4 == 0 ? 4 : 0);
}

// Rows of a strip, the cells one thread computes: 4 columns x 2 rows.
// Measured on 64 x 64 (2368 models x 400 steps, G cell-updates/s): 1 row
// 169, 2 rows 189, 4 rows 179 (a 4-row strip needs 120 registers: half the
// warps).
constexpr int kStripRows = 2;
// Rows a plane holds for `rows` rows of the grid: whole strips, so that a
// thread may read past the last row.
GRN_HOST_DEVICE inline int strip_rows(int rows) {
  return (rows + kStripRows - 1) / kStripRows * kStripRows;
}

// Floats to add after a strip's rows so that shared memory serves a warp's
// 128-bit accesses without bank conflicts.  Such an access goes through in
// four parts of 8 lanes; where a part crosses from one row of strips to the
// next, its lanes hit distinct banks only if the two rows of strips lie
// 4 * (groups per row) floats apart modulo the 32 banks.  Rows of a multiple
// of 8 groups are never crossed.
// Measured without and with the padding (ms): 51 x 37, 600 models with two
// experiments 4.22 -> 3.96; 57 x 32, 1964 x 489 15.3 -> 14.8; 46 x 37, 1531
// x 86 6.55 -> 6.30; 73 x 168 on clusters 5.9 -> 5.75; grids bound elsewhere
// (48 x 48 with 9-16 genes, 42 x 74) within 1%.  Where it would move a gene to
// global memory (100 x 100 on 2 CTAs: 5 genes on chip, 4 with it) planes stay
// unpadded.
GRN_HOST_DEVICE inline int strip_pad(int W) {
  const int Wg = (W + 3) / 4;
  return Wg % 8 == 0 ? 0 : (4 * Wg - kStripRows * row_floats(W)) & 31;
}

// Floats before row r of a plane (row 0 is the zero row above the grid).
GRN_HOST_DEVICE inline int64_t row_offset(int r, int row_floats, int pad) {
  return (int64_t)r * row_floats + (int64_t)((r + kStripRows - 1) / kStripRows) * pad;
}

// Floats of one state plane of a W x H grid: padded rows plus a zero row
// above and below (see the kernel's Geom).  With a cluster of C CTAs per
// model a CTA's plane holds a band of ceil(H / C) rows.
inline int64_t plane_floats(int W, int H, int cluster, int pad) {
  const int rows = strip_rows((H + cluster - 1) / cluster);
  return row_offset(rows + 1, row_floats(W), pad) + row_floats(W);
}

// Chunks of 32 strips of `rows` rows of a W-wide grid: a warp's unit of
// work.
inline int strip_chunks(int W, int rows) {
  return ((strip_rows(rows) / kStripRows) * ((W + 3) / 4) + 31) / 32;
}

// Division by a number d that is the same for a whole launch (Granlund and
// Montgomery, "Division by invariant integers using multiplication", 1994):
// with 2^k < d <= 2^(k+1) and inv = ceil(2^(32+k) / d), which fits 32 bits,
// (i * inv) >> (32 + k) is floor(i / d) for every 0 <= i < 2^31: it exceeds
// i / d by i * e / (d * 2^(32+k)) with e < d <= 2^(k+1), i.e. by less than
// 1 / d.
inline int inverse_shift(int d) {
  int k = 0;
  while (((int64_t)2 << k) < d) ++k;
  return k;
}
inline uint32_t inverse(int d) {
  const uint64_t p = (uint64_t)1 << (32 + inverse_shift(d));
  return d > 1 ? (uint32_t)((p + d - 1) / d) : 0u;
}
// Row of group i in rows of Wg float4 groups.
GRN_HOST_DEVICE inline int group_row(int i, int Wg, uint32_t inv_wg, int wg_shift) {
  return Wg == 1 ? i : (int)((uint32_t)(((uint64_t)(uint32_t)i * inv_wg) >> 32) >> wg_shift);
}

// Whether counts of finished work, which grow by at most one per warp of a block
// and step, stay below 2^31 over n_steps.  (Comparing them modulo 2^32 instead
// takes an instruction more per poll: 64 x 64, 592 models x 500 steps 5.74 ->
// 5.77 ms.)
GRN_HOST_DEVICE inline bool counts_fit(int n_steps) { return n_steps <= 0x7fffffff / 32; }

// SimArgs::change_bound.
inline float float_below(double x) {
  const float f = (float)x;
  return (double)f > x ? std::nextafter(f, -HUGE_VALF) : f;
}

// The launch geometry of a W x H grid split over `cluster` CTAs per model.
inline void set_geometry(SimArgs *a, int W, int H, int cluster, int pad) {
  a->W = W;
  a->H = H;
  a->Wg = (W + 3) / 4;
  a->inv_wg = inverse(a->Wg);
  a->wg_shift = inverse_shift(a->Wg);
  const uint32_t w_inv = W > 1 ? (uint32_t)((((uint64_t)1 << 32) + W - 1) / W) : 0u;
  a->inv_w = (int64_t)W * H * W < (int64_t)1 << 32 ? w_inv : 0u;
  a->row_floats = row_floats(W);
  a->row_bytes = 4 * a->row_floats;
  a->row_pad = pad;
  a->plane_floats = (int32_t)plane_floats(W, H, cluster, pad);
  a->plane_bytes = 4 * a->plane_floats;
}

// Bytes of shared memory a block needs besides the state planes.
size_t sim_fixed_smem_bytes();

// Number of compiled variants and their descriptions.
int sim_variant_count();
KernelVariant sim_variant(int i);

// Occupancy of a variant with blocks of `threads` and `smem_bytes` dynamic shared memory: resident
// blocks per SM (0 if it does not fit).  Sets the function's max dynamic
// shared memory attribute as a side effect.
cudaError_t sim_occupancy(const KernelVariant &v, int threads, size_t smem_bytes,
                          int *blocks_per_sm);

// Cluster-split variant: resident clusters of `cluster` CTAs on the device
// (0 if it does not fit).
cudaError_t sim_cluster_occupancy(const KernelVariant &v, int threads, size_t smem_bytes,
                                  int cluster, int *clusters);

// Launches a variant; the caller has zeroed args.work_counter on `stream`.
cudaError_t sim_launch(const LaunchPlan &plan, const SimArgs &args,
                       cudaStream_t stream);

}  // namespace grn

#endif  // GRN_SIM_H_
