// grn_sim_kernel.cu -- persistent batched GRN simulation + fitness kernels
// for sm_100a.
//
// Replaces the reference's simulateModelKernel
// (Src/GPUSimulator/modelsimulatordevice.cu:154-251), which runs one model
// per launch on one 1024-thread CTA with FP64 state in global memory and a
// function-pointer op interpreter.  Here:
//   - one persistent grid evaluates a whole batch; each CTA pulls the next
//     model from an atomic work counter (the host orders models by cost,
//     longest first);
//   - a model's state lives in shared memory for all Euler steps (planar
//     [gene][y][x] FP32, rows padded to float4 groups), double buffered;
//     genes that do not fit use the same code on double-buffered
//     global-memory slots, and grids too large for shared memory stream bands
//     of rows through it (or split across a cluster);
//   - one block (or cluster) barrier per step where the step's maximum may end
//     the simulation or warps walk their items; owned chunks otherwise wait for
//     the counts of the chunks next to their own (see "steps without a block
//     barrier");
//   - the work of a step is cut into warp items: 32 strips of 4 columns x 2
//     rows, for one gene or all of them (see "the step" below).  A thread
//     loads its own strip's rows once for both rows' neighbour sums; left and
//     right neighbours come from the neighbouring lanes, and from 32-bit loads
//     next to the group where no lane holds them (every padded row ends in zero
//     cells, so a row's borders read 0 without tests);
//   - regulation is evaluated in exponent form (grn_packed.h): per link lg2
//     of the regulator's cells, one FMA + min/max, and per regulated gene
//     ex2 + rcp, on the MUFU pipe;
//   - the step's max |rate| (early-exit test) is a warp max on the float
//     bits plus one shared-memory pass; fitness sums are FP64.
// Semantics follow the reference CPU simulator
// (Src/Simulator/modelsimulator.cpp:205-280), not the reference GPU kernel:
// every cell is updated (the GPU kernel drops W*H mod 1024 cells,
// modelsimulatordevice.cu:44-47) and a zero rate keeps the current value
// (the GPU kernel's double buffer keeps a two-steps-old one, :178).

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/grn_gpu.h"
#include "grn_packed.h"
#include "grn_sim.h"

// GRN_BOUNDS_CHECK=1 builds the bounds-checked library
// (lib/libgrn_b200_checked.so): every state access is checked (see chk).
#ifndef GRN_BOUNDS_CHECK
#define GRN_BOUNDS_CHECK 0
#endif

namespace grn {
namespace {

namespace cg = cooperative_groups;

constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxCluster = 16;

// ---- MUFU instructions (PTX ISA: lg2/ex2/rcp .approx.ftz.f32) ----------
__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ---- paired FP32 arithmetic (PTX ISA: add/mul/fma .rn.f32x2, sm_100+) ---
// Two lanes per instruction, each rounded exactly like its scalar
// counterpart, so results are bit-identical to fmaf / + / *.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{.reg .b64 ra, rb, rc, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("{.reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 lo2(const float4 &v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 &v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float2 f2(float v) { return make_float2(v, v); }

// ---- bulk copies and mbarriers (PTX ISA; streaming schedule) -----------
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}
// One bulk copy global -> this CTA's shared memory, completing on `bar`.
// Both addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes,
                                         uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Waits for the phase with `parity` to complete, giving up after about one
// second (a bulk copy of a band takes microseconds): false on a time-out,
// which the caller reports through the error flag instead of hanging.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  for (uint32_t i = 0; i < (1u << 30); ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (global_ns() - t0 > 1000000000ull) return false;
  }
  return false;
}
// Orders this thread's generic-proxy accesses before later async-proxy
// (bulk copy) accesses of the same memory.
__device__ __forceinline__ void fence_proxy_async_global() {
  asm volatile("fence.proxy.async.global;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_shared() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Shared-memory copy of one model record.
struct ModelSmem {
  PackedHeader hdr;
  PackedGene genes[GRN_MAX_GENES];
  PackedLink links[GRN_MAX_LINKS];
};
constexpr int kModelWords = sizeof(ModelSmem) / 16;
static_assert(sizeof(ModelSmem) % 16 == 0, "model smem is whole words");

// The program in the form the step reads, built in shared memory when a
// model is loaded.  Coefficients are stored as pairs, so that one load gives
// the register pairs of the paired FP32 instructions.
struct GeneSmem {
  float4 ld;     // lim, lim, -deg, -deg
  float2 dif;    // dif, dif
  int ctl;       // GeneCtl fields
  int pad;
};
struct LinkSmem {
  float4 ab;     // a, a, b, b
  int slot;      // regulator, or kConstSlot (exact only)
  int pad[3];
};
struct ProgSmem {
  GeneSmem gene[GRN_MAX_GENES];      // in the order the splits take them
  LinkSmem link[GRN_MAX_LINKS + 1];  // the slot after the last is read ahead
  int start[33];  // walked items: each warp's first (chunk * 16 + gene entry)
  int pad[3];
};
static_assert(sizeof(GeneSmem) == 32 && sizeof(LinkSmem) == 32, "program words");

// GeneSmem::ctl: bits 0-3 the gene, 4 diffuses, 5-12 its first link, 13-20
// its OR links, 21-28 its links in all (OR first).
__host__ __device__ constexpr int gene_ctl(int p, bool diffuses, int link, int n_or, int n) {
  return p | (diffuses ? 16 : 0) | (link << 5) | (n_or << 13) | (n << 21);
}
static_assert(GRN_MAX_GENES <= 16 && GRN_MAX_LINKS < 256, "GeneCtl fields");

// A value that is the same in every lane, as one the compiler knows to be:
// branches on it need no divergence handling.
__device__ __forceinline__ int uniform(int x) { return __shfl_sync(kFull, x, 0); }

// Fixed shared-memory layout in front of the state planes.
constexpr size_t kProgOffset = sizeof(ModelSmem);
constexpr size_t kRedOffset = kProgOffset + sizeof(ProgSmem);  // float [2][32]
constexpr size_t kDredOffset = kRedOffset + 2 * 32 * 4;  // double [32]
constexpr size_t kWorkOffset = kDredOffset + 32 * 8;     // int [2]
// Cluster exchange slots: step maxima float [2][kMaxCluster][32] (by step
// parity, CTA and warp; the fitness sums' lanes between the steps) and the
// fitness sum double.
constexpr size_t kCmaxOffset = kWorkOffset + 16;
constexpr size_t kCsumOffset = kCmaxOffset + 2 * kMaxCluster * 32 * 4;
// Two mbarriers of the streaming schedule's copy stages, then its copy
// time-out flag (int).
constexpr size_t kMbarOffset = (kCsumOffset + 8 + 15) & ~size_t(15);
constexpr size_t kStreamFailOffset = kMbarOffset + 16;
// Steps without a block barrier (StepSync): finished work per chunk (int [32]),
// the halo counts (int [2]) and the last vote with a rate (int).
constexpr int kMaxDone = 32;
constexpr int kDoneInts = kMaxDone + 3;
constexpr size_t kDoneOffset = kStreamFailOffset + 16;
// Bounds-checked build only: the regions that state accesses are checked
// against (CheckRegions).
constexpr size_t kCheckOffset = (kDoneOffset + kDoneInts * 4 + 15) & ~size_t(15);
constexpr size_t kCheckBytes = GRN_BOUNDS_CHECK ? 64 : 0;
constexpr size_t kStateOffset = (kCheckOffset + kCheckBytes + 127) & ~size_t(127);

__device__ __forceinline__ float4 f4(float v) { return make_float4(v, v, v, v); }

// ---- bounds-checked build ----------------------------------------------
//
// With GRN_BOUNDS_CHECK every state access goes through chk: the N floats
// at p must lie inside the block's shared-memory state area (from the state
// offset to the end of the dynamic shared memory) or the launch's global
// state slots, and a float4 access must be 16-byte aligned.  An access that
// is not is redirected to a scratch float4 (nothing outside the buffers is
// touched) and sets the error flag to 3, which the host reports as
// GRN_ERR_KERNEL.  Without it chk is the identity.  This stands in for a
// memory checker: the GPU tests run every schedule through the checked
// library on small grids.
struct CheckRegions {
  const float *sm_lo, *sm_hi;  // shared-memory state area
  const float *gl_lo, *gl_hi;  // global state slots of the whole launch
  int32_t *flag;
  float4 scratch;              // target of redirected accesses
};
static_assert(sizeof(CheckRegions) <= 64, "check regions fit their slot");

extern __shared__ __align__(128) unsigned char grn_dyn_smem[];

__device__ __forceinline__ bool check_span(const float *p, long n) {
  const CheckRegions &c = *reinterpret_cast<const CheckRegions *>(grn_dyn_smem + kCheckOffset);
  return (p >= c.sm_lo && p + n <= c.sm_hi) || (c.gl_lo && p >= c.gl_lo && p + n <= c.gl_hi);
}

__device__ __forceinline__ void check_failed() {
  CheckRegions &c = *reinterpret_cast<CheckRegions *>(grn_dyn_smem + kCheckOffset);
  atomicCAS(c.flag, 0, 3);
}

template <int N>
__device__ __forceinline__ float *chk(const float *p) {
#if GRN_BOUNDS_CHECK
  const bool aligned = N < 4 || (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
  if (!aligned || !check_span(p, N)) {
    check_failed();
    CheckRegions &c = *reinterpret_cast<CheckRegions *>(grn_dyn_smem + kCheckOffset);
    return reinterpret_cast<float *>(&c.scratch);
  }
#endif
  return const_cast<float *>(p);
}

// A bulk copy's source and destination spans (floats); false (and the flag)
// if either leaves its buffer, in which case the copy is not issued.
__device__ __forceinline__ bool chk_copy(const float *dst, const float *src, long n) {
#if GRN_BOUNDS_CHECK
  if (!check_span(dst, n) || !check_span(src, n)) {
    check_failed();
    return false;
  }
#endif
  (void)dst;
  (void)src;
  (void)n;
  return true;
}

// ---- regulation ------------------------------------------------------
//
// A gene's regulation is 1 / (1 + 2^V), V combined in exponent space over
// its links (grn_packed.h).  Two combine modes:
//   fast   min / max (fminf / fmaxf).  Identical to the reference whenever
//          no link term is NaN, which holds for models with finite K > 0,
//          finite Hill coefficients and 0 < K^n <= 1e300 on bounded
//          non-negative states (flag kFlagFast, which the host also clears
//          for a step size that could leave the state unbounded, and the
//          context's fast_ok for the initial states).
//   exact  the reference's comparison order (simopor.cpp:20-22,
//          simopand.cpp:20-22 with MathAlgo::max/min): a NaN term on
//          either side yields the new term; a NaN start makes the first
//          link's term the initial value ("first used link writes
//          ratios[p]", modelsimulator.cpp:156-192).

// Reference OR (Hill max) in exponent space: keep the running v only if it
// is strictly smaller.
__device__ __forceinline__ float comb_or(float run, float t) { return (run < t) ? run : t; }
// Reference AND (Hill min) in exponent space.
__device__ __forceinline__ float comb_and(float run, float t) { return (run > t) ? run : t; }

template <bool B>
struct Bool {
  static constexpr bool value = B;
};
using True = Bool<true>;
using False = Bool<false>;

// Hides how a value was computed, so that it stays in a register instead of
// being computed again at each use (the register-poor variants do that).
__device__ __forceinline__ int opaque(int x) {
  asm volatile("" : "+r"(x));
  return x;
}

enum CombMode { kOrFast, kAndFast, kOrExact, kAndExact };

template <int MODE>
__device__ __forceinline__ float comb(float run, float t) {
  if constexpr (MODE == kOrFast) return fminf(run, t);
  else if constexpr (MODE == kAndFast) return fmaxf(run, t);
  else if constexpr (MODE == kOrExact) return comb_or(run, t);
  else return comb_and(run, t);
}

__device__ __forceinline__ int gene_cost(const PackedGene &g) {
  return gene_work(g.n_or + g.n_and);
}

// Builds the program of the model in M (all threads; a barrier follows).
// Owned chunks: `splits` is the number of warps that share a chunk's genes,
// which are dealt to them in snake order of their cost, so that the splits'
// loads differ by little.
// Walked chunks (splits 0): the genes keep their order, and the items
// (chunk, gene), chunk by chunk, are cut into one range per warp of nearly
// equal cost, so that a warp changes its strips at most once per G items.
// Measured on 100 x 100 (G cell-updates/s): 142; warps taking whole chunks
// in turn, 1, 2 or 4 warps to a chunk, 127.
__device__ __forceinline__ void build_program(const ModelSmem &M, ProgSmem &P, int splits,
                                              int chunks, int n_warps, int tid) {
  const int G = M.hdr.n_genes;
  for (int l = tid; l < M.hdr.n_links; l += blockDim.x) {
    const PackedLink lk = M.links[l];
    P.link[l].ab = make_float4(lk.a, lk.a, lk.b, lk.b);
    P.link[l].slot = lk.slot;
  }
  if (tid == 0) P.link[M.hdr.n_links].slot = 0;
  if (splits == 0 && tid <= n_warps) {
    int total = 0;
    for (int q = 0; q < G; ++q) total += gene_cost(M.genes[q]);
    // The first item whose middle lies at or past tid / n_warps of the cost.
    const int64_t goal2 = 2 * (int64_t)total * chunks * tid;
    int64_t chunk = goal2 / (2 * (int64_t)total * n_warps);
    int64_t at = chunk * total;
    int k = 0;
    while (k < G) {
      const int c = gene_cost(M.genes[k]);
      if ((2 * at + c) * n_warps >= goal2) break;
      at += c;
      ++k;
    }
    if (k == G) {
      k = 0;
      ++chunk;
    }
    P.start[tid] = (int)chunk * 16 + k;
  }
  if (tid >= G) return;
  const PackedGene g = M.genes[tid];
  int place = tid;
  if (splits > 0) {
    // Rank by cost (then index), then the snake deal: round r of the splits
    // runs backwards in odd full rounds.
    const int cost = gene_cost(g);
    int rank = 0;
    for (int q = 0; q < G; ++q) {
      const int cq = gene_cost(M.genes[q]);
      rank += (cq > cost || (cq == cost && q < tid)) ? 1 : 0;
    }
    const int round = rank / splits, pos = rank - round * splits;
    const bool back = (round & 1) && (round + 1) * splits <= G;
    place = round * splits + (back ? splits - 1 - pos : pos);
  }
  GeneSmem &o = P.gene[place];
  o.ld = make_float4(g.lim, g.lim, -g.deg, -g.deg);
  o.dif = f2(g.dif);
  o.ctl = gene_ctl(tid, g.dif > 0.0f, g.link_begin, g.n_or, g.n_or + g.n_and);
}

// ---- geometry ----------------------------------------------------------
//
// A state plane holds the W x H grid as rows of RS = row_floats(W) floats
// (whole float4 groups, ending in at least one zero cell) plus one zero row
// above and one below, and rows for whole strips (strip_rows; the
// no-allocation entry's planes have none, and their over-reads land in what
// follows): PS = plane_floats, row y at row_offset(y + 1): `pad` zero floats follow the
// row above the grid and then every two rows, i.e. every row of strips
// (strip_pad; 0 where streamed).  The zero rows make the up/down neighbours of
// the first and last rows read +0.0, which leaves the reference's neighbour
// sum unchanged.  Steps write data groups only; when W is not a multiple of 4
// the cells past W of a row's last group are written as 0, otherwise a zero
// group ends the row: either way the cell after a row's last cell, and the cell
// before the next row's first, read 0.
//
// A cluster-split launch gives each CTA of a cluster a band of rows
// [y0, y0 + H) of the Hg-row grid, held the same way: one halo row above and
// one below (the neighbouring bands' edge rows, pushed into them after every
// step, or zero at the grid border).
struct Geom {
  int W, H, Wg, RS, PS, Q;  // Q: strips of the band
  int pad;                  // floats after every two rows (0: streamed bands)
  int RSb, PSb, SSb;        // RS, PS and a row of strips (R * RS + pad) in bytes
  bool edges;               // chunks do not hold whole rows of groups
  int y0, Hg;               // first grid row of the band, grid height
  uint32_t inv_wg;          // q / Wg by multiplication (group_row)
  int wg_shift;
};

// Strips of R rows x 4 columns in H rows of Wg groups.
template <int R>
__device__ __forceinline__ int strip_count(int H, int Wg) {
  return ((H + R - 1) / R) * Wg;
}

// The 4 x R cells a thread computes: columns 4gx .. 4gx + 3 of rows y ..
// y + R - 1.  A strip index past the end is clamped onto the last strip: its
// values are computed (they are that strip's own) and not stored.  Rows past
// the grid's last (a plane holds whole strips) are computed from whatever
// the plane holds there, and neither stored nor part of the max.
template <int R>
struct Strip {
  int base;            // byte offset of the first row's group in a plane
  int rows;            // rows that exist (1 .. R)
  bool valid;          // false: nothing is stored
  bool el, er;         // the left / right neighbour group is not the
                       // neighbouring lane's
  bool m1, m2, m3;     // cells 1..3 of the group exist (cell 0 always does)
  bool first, last;    // holds the band's first row / its last one, and a
                       // neighbouring CTA has that row as a halo row
  float2 nt[R][2];     // -(existing neighbours) of each cell, as pairs
};

template <int R>
__device__ __forceinline__ Strip<R> strip_at(int q, const Geom &g) {
  Strip<R> s;
  s.valid = q < g.Q;
  const int qc = s.valid ? q : g.Q - 1;
  const int ys = group_row(qc, g.Wg, g.inv_wg, g.wg_shift);
  const int gx = qc - ys * g.Wg, y = R * ys, x0 = 4 * gx;
  s.rows = min(R, g.H - y);
  s.el = gx == 0 || (q & 31) == 0;
  s.er = gx == g.Wg - 1 || (q & 31) == 31;
  s.base = (ys + 1) * g.SSb - (R - 1) * g.RSb + 4 * x0;
  s.first = s.valid && y == 0 && g.y0 > 0;
  s.last = s.valid && y + R >= g.H && g.y0 + g.H < g.Hg;
  const int yg = y + g.y0;
  const float hx = (x0 > 0 ? 1.0f : 0.0f) + (x0 + 1 < g.W ? 1.0f : 0.0f);
  const float hy = 1.0f + (x0 + 2 < g.W ? 1.0f : 0.0f);
  const float hz = 1.0f + (x0 + 3 < g.W ? 1.0f : 0.0f);
  const float hw = 1.0f + (x0 + 4 < g.W ? 1.0f : 0.0f);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const float tv = (i > 0 || yg > 0 ? 1.0f : 0.0f) + (yg + i + 1 < g.Hg ? 1.0f : 0.0f);
    s.nt[i][0] = make_float2(-(tv + hx), -(tv + hy));
    s.nt[i][1] = make_float2(-(tv + hz), -(tv + hw));
  }
  s.m1 = x0 + 1 < g.W;
  s.m2 = x0 + 2 < g.W;
  s.m3 = x0 + 3 < g.W;
  return s;
}

__device__ __forceinline__ int cell_offset(const Geom &g, int y, int x) {
  return (int)row_offset(y + 1, g.RS, g.pad) + x;
}

// ---- the step ------------------------------------------------------------
//
// Work is cut into warp items: one gene of a chunk of 32 strips.  A warp owns
// a chunk and its part of the genes, or walks a range of (chunk, gene) items
// (build_program).  A thread evaluates one gene after the other for its 8 cells; the
// regulators' values are read again, and their lg2 taken again, for every
// link that reads them.  That is more MUFU work than holding every gene's
// lg2 in registers (one lg2 per link instead of one per gene), but it needs
// no register array: no per-gene-count instantiations, no dispatch from a
// link to a register index (which cost more instructions than the links'
// arithmetic), a link is a plain loop iteration, and half the registers
// give twice the warps.  Bound by the MUFU and shared-memory pipes together
// (each 55-60% busy, issue 60%).  Measured against the register array, same
// bits (ms): 64 x 64, 4096 models x 2000 steps 203.0 -> 175.2; 100 x 100,
// 2048 x 500 86.2 -> 77.5; 48 x 48 with 9-16 genes, 600 x 300 18.5 -> 7.5;
// 256 x 256 with 8 genes, 592 x 100 66.7 -> 57.0; one 32 x 32 model x 500
// 0.53 -> 0.35.

// How a model's step is evaluated: kFast and kClamp the fast combine (see
// regulation) and the simplified update, with minConc 0 and above it; kConst
// that update and the reference's comparison order in the combine, for fast
// models with constant link terms, under any minConc; kExact the reference's
// comparisons throughout.  48 x 40, 600 models x 300 steps with minConc 0.01:
// kExact 2.33 ms, kClamp 1.96.  kClamp and kConst have one form (some
// planes may be in the global slot) and step with a barrier: compiled into
// the barrier-free loop as well kClamp gave 1.88, but cost kFast there 1% (64 x
// 64) to 3% (32 x 32).  Models with constant terms (ms, kExact -> kConst): 64 x
// 64, 592 x 500 8.74 -> 7.62; 100 x 100, 296 x 300 8.61 -> 7.35; 32 x 32, 64 x
// 500 0.73 -> 0.61.  Constant terms taken in the fast combine, for the genes that
// have them, gave 6.05, 5.80 and 0.48, but cost all other models 1% to 3%.
enum Path { kFast, kClamp, kConst, kExact };

template <int P>
struct PathTag {
  static constexpr int value = P;
};

// The new value n of a cell with rate r under minConc: a zero rate keeps the
// value (n) whatever it is.
__device__ __forceinline__ float clamped(float n, float r, float min_conc) {
  return n < min_conc && r != 0.0f ? 0.0f : n;
}

// Euler update of one cell (modelsimulator.cpp:224-275), the exact path:
//   r = lim*h - deg*c (+ dif*(s - tot*c) for diffusing genes)
// with the reference's guard on the diffusion term, "a zero rate keeps the
// value", the minConc clamp and a NaN-ignoring max.
__device__ __forceinline__ float update_cell(float c, float h, float lim, float ndeg, float dif,
                                             bool diffuses, float s, float ntot, float dt,
                                             float min_conc, float &mx) {
  float r = fmaf(ndeg, c, lim * h);
  if (diffuses && (s > 0.0f || (ntot < 0.0f && c > 0.0f))) r = fmaf(dif, fmaf(ntot, c, s), r);
  float nc = c;
  if (r != 0.0f) {  // NaN counts as non-zero, like the reference's `if (ratio)`
    nc = fmaf(dt, r, c);
    nc = (nc < min_conc) ? 0.0f : nc;
    const float ar = fabsf(r);
    mx = (ar > mx) ? ar : mx;  // a NaN rate never raises the max
  }
  return nc;
}

// State accesses of the step: byte offsets from the shared-memory state area
// (a constant address, so that an offset is all a load needs), or unsigned
// ones from a global pointer that is the same for the whole block (a uniform
// base and a 32-bit offset; a slot is smaller than 4 GB).
template <int N, bool GL>
__device__ __forceinline__ const float *state_at(const char *gl, int off) {
  return chk<N>(reinterpret_cast<const float *>(
      GL ? gl + (uint32_t)off
         : reinterpret_cast<const char *>(grn_dyn_smem) + kStateOffset + off));
}
template <bool GL>
__device__ __forceinline__ float4 load4(const char *gl, int off) {
  return *reinterpret_cast<const float4 *>(state_at<4, GL>(gl, off));
}

// Planes a step reads and writes.  Plane k of the current state is at shared
// offset sm + k * PSb for k < n_sm, else at gl + k * PSb; its next state at
// sm_out + k * PSb, or (a staged band) at gl_out + k * out_stride.
struct Planes {
  int sm, sm_out;
  const char *gl;
  char *gl_out;
  int out_stride;
  int n_sm;
};

// Where a band's edge rows also go: the halo rows of the neighbouring CTAs'
// planes, up_rows bytes further down (down_rows bytes further up) than the
// row's own place, in their shared memory (cluster addresses of their state
// areas) or their global slots (slot_bytes before and after this CTA's).
struct Halo {
  uint32_t up, down;
  int up_rows, down_rows;
  int64_t slot_bytes;
};

__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  return a;
}

template <bool GL>
__device__ __forceinline__ void halo_store(uint32_t remote, char *gl, int off, const float4 &v) {
  if constexpr (GL) {
    *reinterpret_cast<float4 *>(chk<4>(reinterpret_cast<float *>(gl + off))) = v;
  } else {
    (void)state_at<4, false>(nullptr, off);  // the same offset in this CTA, checked
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(remote + off),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
  }
}

// The terms a*lg2(x) + b of one link for the strip's cells.
template <int R, bool SPILL>
__device__ __forceinline__ void link_terms(float4 (&t)[R], const float4 &ab, int slot,
                                           const Planes &pl, const Strip<R> &st,
                                           const Geom &g) {
  float4 x[R];
  if (SPILL && slot >= pl.n_sm) {
    const int o = slot * g.PSb + st.base;
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = load4<true>(pl.gl, o + i * g.RSb);
  } else {
    const int o = slot * g.PSb + (pl.sm + st.base);
#pragma unroll
    for (int i = 0; i < R; ++i) x[i] = load4<false>(nullptr, o + i * g.RSb);
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const float2 t01 = fma2(lo2(ab), make_float2(lg2_approx(x[i].x), lg2_approx(x[i].y)), hi2(ab));
    const float2 t23 = fma2(lo2(ab), make_float2(lg2_approx(x[i].z), lg2_approx(x[i].w)), hi2(ab));
    t[i] = make_float4(t01.x, t01.y, t23.x, t23.y);
  }
}

template <int MODE, int R>
__device__ __forceinline__ void comb_strip(float4 (&v)[R], const float4 (&t)[R]) {
#pragma unroll
  for (int i = 0; i < R; ++i) {
    v[i].x = comb<MODE>(v[i].x, t[i].x);
    v[i].y = comb<MODE>(v[i].y, t[i].y);
    v[i].z = comb<MODE>(v[i].z, t[i].z);
    v[i].w = comb<MODE>(v[i].w, t[i].w);
  }
}

// Regulation 1 / (1 + 2^v) of four cells.
__device__ __forceinline__ float4 hill4(const float4 &v) {
  const float2 e01 = add2(f2(1.0f), make_float2(ex2_approx(v.x), ex2_approx(v.y)));
  const float2 e23 = add2(f2(1.0f), make_float2(ex2_approx(v.z), ex2_approx(v.w)));
  return make_float4(rcp_approx(e01.x), rcp_approx(e01.y), rcp_approx(e23.x), rcp_approx(e23.y));
}

// Regulation of one gene (its ctl word) for the strip: the first link's
// terms start the running exponents, OR links take the min, AND links the
// max.  ORDERED: the reference's comparison order, where a Hill coefficient
// of 0 (kConstSlot) gives the constant term 0; models on the other paths have
// no such link.
template <int R, bool ORDERED, bool SPILL>
__device__ __forceinline__ void regulation(const ProgSmem &P, int ctl, const Planes &pl,
                                           const Strip<R> &st, const Geom &g, float4 (&h)[R]) {
  const int n = ctl >> 21;
  if (n == 0) {  // OpZero
#pragma unroll
    for (int i = 0; i < R; ++i) h[i] = f4(0.0f);
    return;
  }
  const LinkSmem *L = P.link + ((ctl >> 5) & 255);
  const int n_or = (ctl >> 13) & 255;
  float4 v[R], t[R];
  if constexpr (ORDERED) {
#pragma unroll
    for (int i = 0; i < R; ++i) v[i] = f4(__int_as_float(0x7fc00000));
#pragma unroll 1
    for (int l = 0; l < n; ++l) {
      const int slot = L[l].slot;
      if (slot == kConstSlot) {
#pragma unroll
        for (int i = 0; i < R; ++i) t[i] = f4(0.0f);
      } else {
        link_terms<R, SPILL>(t, L[l].ab, slot, pl, st, g);
      }
      if (l < n_or) comb_strip<kOrExact, R>(v, t);
      else comb_strip<kAndExact, R>(v, t);
    }
  } else {
    link_terms<R, SPILL>(v, L->ab, L->slot, pl, st, g);
    ++L;
    int slot = L->slot;  // read one link ahead
    int left = n_or - 1;
#pragma unroll 1
    for (; left > 0; --left) {
      const float4 ab = L->ab;
      const int s = slot;
      ++L;
      slot = L->slot;
      link_terms<R, SPILL>(t, ab, s, pl, st, g);
      comb_strip<kOrFast, R>(v, t);
    }
    left = n - max(n_or, 1);
#pragma unroll 1
    for (; left > 0; --left) {
      const float4 ab = L->ab;
      const int s = slot;
      ++L;
      slot = L->slot;
      link_terms<R, SPILL>(t, ab, s, pl, st, g);
      comb_strip<kAndFast, R>(v, t);
    }
  }
#pragma unroll
  for (int i = 0; i < R; ++i) h[i] = hill4(v[i]);
}

// New values of one gene for the strip, from its current plane (at src_gl,
// or shared offset src) to its next one (dst_gl, dst).  `mx` takes the
// max |rate| of the strip's real cells.
// Fast paths (a non-negative finite state, host-checked): the reference's
// diffusion guard only ever skips adding dif*0, a zero rate gives c + dt*0 =
// c, and with minConc 0 the clamp is a max with 0, so these simplify without
// changing any result.
template <int R, int PATH, bool RAGGED, bool DIFFUSES, bool SG, bool DG, bool CL>
__device__ __forceinline__ void update_strip(const GeneSmem &gn, const float4 (&h)[R],
                                             const char *src_gl, int src, char *dst_gl, int dst,
                                             const Strip<R> &st, const Geom &g,
                                             const Halo &halo, float dt, float min_conc,
                                             float &mx) {
  const float4 ld = gn.ld;
  const float2 dif = DIFFUSES ? gn.dif : f2(0.0f);
  const int o = src + st.base;
  // Rows -1 .. R of the strip's group (row i at c[i + 1]).
  float4 c[R + 2];
  float lft[R], rgt[R];
#pragma unroll
  for (int i = 0; i < R; ++i) c[i + 1] = load4<SG>(src_gl, o + i * g.RSb);
  if constexpr (DIFFUSES) {
    c[0] = load4<SG>(src_gl, o + (R - 1) * g.RSb - g.SSb);
    c[R + 1] = load4<SG>(src_gl, o + g.SSb);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float l = __shfl_up_sync(kFull, c[i + 1].w, 1);
      const float r = __shfl_down_sync(kFull, c[i + 1].x, 1);
      lft[i] = st.el ? 0.0f : l;
      rgt[i] = st.er ? 0.0f : r;
    }
    if (g.edges) {
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (st.el) lft[i] = *state_at<1, SG>(src_gl, o + i * g.RSb - 4);
        if (st.er) rgt[i] = *state_at<1, SG>(src_gl, o + i * g.RSb + 16);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const float4 ci = c[i + 1];
    float2 s01 = f2(0.0f), s23 = f2(0.0f);
    if constexpr (DIFFUSES) {
      // Reference order: x-1, x+1, y-1, y+1.
      s01 = make_float2(lft[i] + ci.y, ci.x + ci.z);
      s23 = make_float2(ci.y + ci.w, ci.z + rgt[i]);
      s01 = add2(add2(s01, lo2(c[i])), lo2(c[i + 2]));
      s23 = add2(add2(s23, hi2(c[i])), hi2(c[i + 2]));
    }
    float4 nv;
    float m, m1, m2, m3;
    if constexpr (PATH != kExact) {
      float2 r01 = fma2(hi2(ld), lo2(ci), mul2(lo2(ld), lo2(h[i])));
      float2 r23 = fma2(hi2(ld), hi2(ci), mul2(lo2(ld), hi2(h[i])));
      if constexpr (DIFFUSES) {
        r01 = fma2(dif, fma2(st.nt[i][0], lo2(ci), s01), r01);
        r23 = fma2(dif, fma2(st.nt[i][1], hi2(ci), s23), r23);
      }
      const float2 n01 = fma2(f2(dt), r01, lo2(ci));
      const float2 n23 = fma2(f2(dt), r23, hi2(ci));
      if constexpr (PATH != kFast)
        nv = make_float4(clamped(n01.x, r01.x, min_conc), clamped(n01.y, r01.y, min_conc),
                         clamped(n23.x, r23.x, min_conc), clamped(n23.y, r23.y, min_conc));
      else
        nv = make_float4(fmaxf(n01.x, 0.0f), fmaxf(n01.y, 0.0f), fmaxf(n23.x, 0.0f),
                         fmaxf(n23.y, 0.0f));
      m = fabsf(r01.x);
      m1 = fabsf(r01.y);
      m2 = fabsf(r23.x);
      m3 = fabsf(r23.y);
    } else {
      m = m1 = m2 = m3 = 0.0f;
      nv.x = update_cell(ci.x, h[i].x, ld.x, ld.z, dif.x, DIFFUSES, s01.x, st.nt[i][0].x, dt,
                         min_conc, m);
      nv.y = update_cell(ci.y, h[i].y, ld.x, ld.z, dif.x, DIFFUSES, s01.y, st.nt[i][0].y, dt,
                         min_conc, m1);
      nv.z = update_cell(ci.z, h[i].z, ld.x, ld.z, dif.x, DIFFUSES, s23.x, st.nt[i][1].x, dt,
                         min_conc, m2);
      nv.w = update_cell(ci.w, h[i].w, ld.x, ld.z, dif.x, DIFFUSES, s23.y, st.nt[i][1].y, dt,
                         min_conc, m3);
    }
    if constexpr (RAGGED) {
      // Cells past W are padding: kept at 0, never part of the max.
      if (!st.m1) { nv.y = 0.0f; m1 = 0.0f; }
      if (!st.m2) { nv.z = 0.0f; m2 = 0.0f; }
      if (!st.m3) { nv.w = 0.0f; m3 = 0.0f; }
    }
    const int row = dst + st.base + i * g.RSb;
    if (st.valid && (i == 0 || i < st.rows)) {
      mx = fmaxf(fmaxf(mx, m), fmaxf(fmaxf(m1, m2), m3));
      *reinterpret_cast<float4 *>(const_cast<float *>(state_at<4, DG>(dst_gl, row))) = nv;
    }
    if constexpr (CL) {
      if (i == 0 && st.first)
        halo_store<DG>(halo.up, dst_gl - halo.slot_bytes, row + halo.up_rows, nv);
      if (i == st.rows - 1 && st.last)
        halo_store<DG>(halo.down, dst_gl + halo.slot_bytes, row - halo.down_rows, nv);
    }
  }
}

// One gene (entry k of the program) for the strip.  SPILL: genes n_sm and on
// live in the global slot.  BAND: the source planes are a staged band in
// shared memory, the destination is global.
template <int R, int PATH, bool RAGGED, bool SPILL, bool BAND, bool CL>
__device__ __forceinline__ void gene_step(const ProgSmem &P, int k, const Planes &pl,
                                          const Strip<R> &st, const Geom &g, const Halo &halo,
                                          float dt, float min_conc, float &mx) {
  const GeneSmem &gn = P.gene[k];
  const int ctl = uniform(gn.ctl);
  const int p = ctl & 15;
  float4 h[R];
  regulation<R, PATH == kExact || PATH == kConst, SPILL>(P, ctl, pl, st, g, h);
  const auto update = [&](auto diffuses) {
    constexpr bool D = decltype(diffuses)::value;
    const int o = p * g.PSb;
    if (SPILL && p >= pl.n_sm)
      update_strip<R, PATH, RAGGED, D, true, true, CL>(gn, h, pl.gl, o, pl.gl_out, o, st, g, halo,
                                                        dt, min_conc, mx);
    else
      update_strip<R, PATH, RAGGED, D, false, BAND, CL>(
          gn, h, nullptr, pl.sm + o, pl.gl_out, BAND ? p * pl.out_stride : pl.sm_out + o, st, g,
          halo, dt, min_conc, mx);
  };
  if (ctl & 16) update(True{});
  else update(False{});
}

// Block-wide max of a non-negative, non-NaN float (bit order == value
// order): each warp publishes its max, a barrier follows, and any thread
// can read the block's.  `parity` alternates two buffers so that one barrier
// per step suffices.
__device__ __forceinline__ void publish_max(float v, float *red, int parity, int lane, int warp) {
  const unsigned bits = __reduce_max_sync(kFull, __float_as_uint(v));
  if (lane == 0) red[parity * 32 + warp] = __uint_as_float(bits);
}
__device__ __forceinline__ float published_max(const float *red, int parity, int lane,
                                               int n_warps) {
  // One warp value per lane, then a warp max (redux) in every warp.
  const unsigned mine = lane < n_warps ? __float_as_uint(red[parity * 32 + lane]) : 0u;
  return __uint_as_float(__reduce_max_sync(kFull, mine));
}
__device__ __forceinline__ float block_max(float v, float *red, int parity, int lane, int warp,
                                           int n_warps) {
  publish_max(v, red, parity, lane, warp);
  __syncthreads();
  return published_max(red, parity, lane, n_warps);
}

// The experiment's fitness sum over the grid's cells (simstate.cpp:135-158)
// in FP64.  Cell i belongs to lane i % 32 of virtual warp (i / 32) %
// kSumWarps, whatever the block size, a virtual lane adds its cells in order,
// and the virtual warps' sums are added in order, so every schedule, block and
// cluster size gives the same bits.
constexpr int kSumWarps = 16;
constexpr int kSumLanes = kSumWarps * 32;
static_assert(kSumLanes * 8 <= 2 * kMaxCluster * 32 * 4 && kCmaxOffset % 8 == 0, "lane sums fit");

// A virtual lane's sum v continued over the cells first .. end - 1.
template <typename F>
__device__ __forceinline__ double lane_sum(double v, int slot, int first, int end, F term) {
  const int d = (slot - first) & (kSumLanes - 1);
  for (int i = first + d; i < end; i += kSumLanes) v = term(i, v);
  return v;
}

// The virtual lanes' sums of virtual warp vw into dred[vw].
__device__ __forceinline__ void warp_sum(double v, double *dred, int vw, int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
  if (lane == 0) dred[vw] = v;
}

// The whole sum, in every thread of the block (after a barrier).
__device__ __forceinline__ double total_sum(const double *dred) {
  double s = 0.0;
#pragma unroll
  for (int w = 0; w < kSumWarps; ++w) s += dred[w];
  return s;
}

// ---- steps without a block barrier ----------------------------------------
//
// A chunk's step s needs, of the step before, only the chunks within one row
// above and below it (and those chunks' own earlier reads, which the same
// counts cover, before it overwrites the older buffer).  So where no step's
// maximum has to be known before the next step, a warp waits for its
// neighbours' counts instead of a block barrier, and warps drift apart by up
// to a step per chunk: their loads, MUFU bursts and waits overlap.
// Measured with the barrier and without (G cell-updates/s): 64 x 64 198 and
// 219.  Testing every step's maximum one step late, so that models with an
// early-exit threshold could run the same way, took more than the barrier
// (202; 51 x 37 with early exit 100 -> 94), so those keep it.
//
// A cluster's CTAs step the same way: a warp that has stored edge rows into a
// neighbouring CTA's halo adds to that CTA's halo count, and a warp whose
// chunk reads a halo row also waits for it, so no cluster barrier is passed
// until the experiment ends (100 x 100 on 2 CTAs per model: 136 -> 152 G
// cell-updates/s; one such model on 8 CTAs 1.23 -> 1.08 ms for 500 steps).
struct StepSync {
  int *done;           // [chunk] gene parts finished since the experiment began
  volatile int *fail;  // a wait ran out
  const int *wait;     // the count this lane waits for: a chunk's, or the halo
                       // count of the CTA above (lane 30) or below (lane 31)
  int per_step;        // what it grows by in a step
  bool first, last;    // the chunk holds the band's first / last row: the warp
                       // waits for the halo count there (cluster scope) and adds
                       // to the neighbouring CTA's, whose address it takes from
                       // the halo's (in registers of their own they cost 1%)
};

// Waits until this lane's count has reached `steps` steps, in every lane;
// false, and *fail set, after 2^24 polls (0.5 to 1 s measured; a step takes
// microseconds) or once another warp has given up.  Every decision to leave is
// a vote: lanes that read *fail at different moments must not part ways at the
// vote of the next poll.
constexpr uint32_t kMaxPolls = 1u << 24;
template <bool CL>
__device__ __forceinline__ bool wait_counts(const StepSync &y, int steps) {
  const uint32_t a = smem_addr(y.wait);
  const int target = y.per_step * steps;  // counts_fit
  for (uint32_t i = 0; i < kMaxPolls; ++i) {
    int v;
    if (CL && (y.first || y.last))
      asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    else
      asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    if (__all_sync(kFull, v >= target)) {
      __syncwarp();
      return true;
    }
    if ((i & 1023u) == 1023u && __any_sync(kFull, *y.fail)) return false;
  }
  *y.fail = 1;
  return false;
}

// Chunk c's step reads cells of the chunks c - reach .. c + reach.
__device__ __forceinline__ int chunk_reach(const Geom &g) { return (g.Wg + 31) / 32; }

// The warp's part of a step on chunk c is finished.
template <bool CL>
__device__ __forceinline__ void finish_chunk(const StepSync &y, const Halo &halo, int c, int lane) {
  __syncwarp();
  if (lane == 0) {
    asm volatile("red.release.cta.shared::cta.add.u32 [%0], 1;" ::"r"(smem_addr(y.done + c))
                 : "memory");
    if constexpr (CL) {
      // A neighbour's halo counts, by way of the address of its state area.
      constexpr int counts = (int)(kDoneOffset + kMaxDone * 4) - (int)kStateOffset;
      if (y.first)
        asm volatile("red.release.cluster.shared::cluster.add.u32 [%0], 1;" ::"r"(
                         halo.up + counts + 4)
                     : "memory");
      if (y.last)
        asm volatile("red.release.cluster.shared::cluster.add.u32 [%0], 1;" ::"r"(
                         halo.down + counts)
                     : "memory");
    }
  }
}

// Whether a model is at rest is looked at every kVoteSteps steps.  A warp whose
// part has a rate in step s, such a step, raises *alive to s (in every CTA of a
// cluster).  *alive below s - lag at step s then means that no part of the grid
// had a rate in step s - lag, and that none has had one since: warps are never
// further apart than the chunks between them (each is at most a step ahead of
// its neighbours), fewer than lag, so every warp has been through step s - lag,
// and its word is here by way of the counts.  For the same reason all warps
// come to the same answer at the same step.  A model that comes to rest runs
// lag + kVoteSteps steps more at most.  4 models of 64 x 64 that rest
// after 150 steps, asked for 400,000: 1524 -> 0.8 ms.  Models that never rest
// pay a word per warp and vote: 64 x 64, 4096 x 500 39.11 -> 39.13 ms; 32 x 32,
// 64 x 500 0.440 -> 0.435 (a block barrier every 64 steps instead: 39.85 and
// 0.434).
constexpr int kVoteSteps = 64;
template <bool CL>
__device__ __forceinline__ bool at_rest(int *alive, int s, bool rate, int C, int lane) {
  constexpr int lag = CL ? kMaxCluster * kMaxDone + kVoteSteps : kVoteSteps;
  static_assert(kMaxDone <= kVoteSteps && lag % kVoteSteps == 0, "lag covers all chunks");
  if (rate) {
    if constexpr (CL) {
      if (lane < C)
        asm volatile("red.relaxed.cluster.shared::cluster.max.s32 [%0], %1;" ::"r"(
                         cluster_addr(smem_addr(alive), lane)),
                     "r"(s)
                     : "memory");
    } else if (lane == 0) {
      asm volatile("red.relaxed.cta.shared::cta.max.s32 [%0], %1;" ::"r"(smem_addr(alive)), "r"(s)
                   : "memory");
    }
  }
  const int seen = *reinterpret_cast<volatile int *>(alive);
  return !__any_sync(kFull, seen >= s - lag);
}

// Where a model's state lives during one step: genes p < n_sm are double
// buffered in shared-memory planes p and p + n_sm; the others in the
// block's global slot, planes p and p + gmax.  `par` selects the buffer
// holding the current values.
struct StatePtrs {
  float *sm;   // shared-memory planes
  float *gl;   // global-memory slot
  int n_sm;    // genes held in shared memory
  int gmax;    // genes a global slot holds
};

__device__ __forceinline__ float *plane_of(const StatePtrs &sp, const Geom &g, int p, int par) {
  return p < sp.n_sm ? sp.sm + (p + (par ? sp.n_sm : 0)) * g.PS
                     : sp.gl + (p + (par ? sp.gmax : 0)) * g.PS;
}

// The planes of a step from buffer `par` to the other one.
__device__ __forceinline__ Planes planes_of(const StatePtrs &sp, const Geom &g, int par) {
  const int half = sp.n_sm * g.PSb;
  const size_t gl_half = (size_t)sp.gmax * g.PSb;
  char *gl = reinterpret_cast<char *>(sp.gl);
  return Planes{opaque(par ? half : 0),   opaque(par ? 0 : half), gl + (par ? gl_half : 0),
                gl + (par ? 0 : gl_half), 0,                      sp.n_sm};
}

// Genes first, first + splits, .. of the program for one strip.
template <int R, int PATH, bool RAGGED, bool SPILL, bool CL>
__device__ __forceinline__ void strip_step(const ProgSmem &P, const Planes &pl, int G,
                                           const Geom &g, const Strip<R> &st, const Halo &halo,
                                           int first, int splits, float dt, float min_conc,
                                           float &mx) {
#pragma unroll 1
  for (int k = first; k < G; k += splits)
    gene_step<R, PATH, RAGGED, SPILL, false, CL>(P, k, pl, st, g, halo, dt, min_conc, mx);
}

// A warp's range of walked items, of the first `chunks` chunks.
template <int R, int PATH, bool RAGGED, bool SPILL, bool BAND, bool CL>
__device__ __forceinline__ void walk_step(const ProgSmem &P, const Planes &pl, int G,
                                          const Geom &g, const Halo &halo, int chunks, int warp,
                                          int lane, float dt, float min_conc, float &mx) {
  const int end = uniform(P.start[warp + 1]);
  int at = uniform(P.start[warp]);
#pragma unroll 1
  while (at < end && (at >> 4) < chunks) {
    const int chunk = at >> 4;
    const Strip<R> st = strip_at<R>(chunk * 32 + lane, g);
    const int stop = (end >> 4) == chunk ? end & 15 : G;
#pragma unroll 1
    for (int k = at & 15; k < stop; ++k)
      gene_step<R, PATH, RAGGED, SPILL, BAND, CL>(P, k, pl, st, g, halo, dt, min_conc, mx);
    at = (chunk + 1) << 4;
  }
}

// One step of the warp's work by the model's class: all planes in shared
// memory or some in the global slot; the other paths always take the general
// form.  SYNC (owned chunks): between the waits of step s and its counts;
// false if a wait ran out.
template <int R, bool LOOP, bool RAGGED, bool CL, bool SYNC>
__device__ __forceinline__ bool block_step(int path, const ProgSmem &P, const StatePtrs &sp,
                                           int G, const Geom &g, const Strip<R> &st,
                                           const Halo &halo, int own, int first, int splits,
                                           int chunks, int warp, int lane, int par, float dt,
                                           float min_conc, float &mx, const StepSync &sync,
                                           int s) {
  const Planes pl = planes_of(sp, g, par);
  if constexpr (SYNC) {
    if (s > 1 && !wait_counts<CL>(sync, s - 1)) return false;
  }
  const auto run = [&](auto e, auto spill) {
    constexpr int E = decltype(e)::value;
    constexpr bool S = decltype(spill)::value;
    if constexpr (LOOP)
      walk_step<R, E, RAGGED, S, false, CL>(P, pl, G, g, halo, chunks, warp, lane, dt, min_conc,
                                            mx);
    else
      strip_step<R, E, RAGGED, S, CL>(P, pl, G, g, st, halo, first, splits, dt, min_conc, mx);
  };
  if (path == kExact) run(PathTag<kExact>{}, True{});
  else if (path == kClamp) run(PathTag<kClamp>{}, True{});
  else if (path == kConst) run(PathTag<kConst>{}, True{});
  else if (sp.n_sm < G) run(PathTag<kFast>{}, True{});
  else run(PathTag<kFast>{}, False{});
  if constexpr (SYNC) finish_chunk<CL>(sync, halo, own, lane);
  return true;
}

// ---- streaming schedule -------------------------------------------------
//
// For grids whose planes do not fit shared memory: every plane lives in the
// block's global slot and each step walks the grid in bands of R rows.  A
// band's rows plus one halo row above and below, of every gene, arrive in a
// shared-memory stage by bulk copies (the TMA engine's cp.async.bulk, one
// per gene, completing on the stage's mbarrier) while the previous band is
// computed from the other stage; new values go straight to the global slot.
// The step's arithmetic is the other schedules' (regulation and
// update_strip), so states are bit-identical.

// New values of all genes of one band from its stage planes (of gb.PS
// floats), written to the global next-state planes: the warps walk the
// band's items.  `out` addresses the band's cells as a plane does: cell (x,
// local row y) of gene p at out + p * gps + (y + 1) * RS + x.
template <int R, bool RAGGED>
__device__ __forceinline__ void band_step(int path, const ProgSmem &P, const float *stage,
                                          int G, const Geom &gb, float *out, size_t gps,
                                          float dt, float min_conc, float &mx) {
  const int warp = uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const Planes pl{(int)(reinterpret_cast<const unsigned char *>(stage) - grn_dyn_smem) -
                      (int)kStateOffset,
                  0, nullptr, reinterpret_cast<char *>(out), (int)(gps * sizeof(float)), G};
  const int chunks = (gb.Q + 31) / 32;
  const auto run = [&](auto e) {
    walk_step<R, decltype(e)::value, RAGGED, false, true, false>(
        P, pl, G, gb, Halo{}, chunks, warp, lane, dt, min_conc, mx);
  };
  if (path == kFast) run(PathTag<kFast>{});
  else if (path == kClamp) run(PathTag<kClamp>{});
  else if (path == kConst) run(PathTag<kConst>{});
  else run(PathTag<kExact>{});
}

// One Euler step of the streaming schedule.  Stages alternate by band.  The
// warps pass no block barrier between bands: a warp goes on to the next band
// once that band's copy has arrived, and the last warp to finish band b
// issues the copy of band b + 2 into its stage.  Bound by issue slots and the
// MUFU pipe (each about half busy) and by the waits for them, so warps help:
// 256 x 256, 8 genes, 592 models x 100 steps, kernel ms with 16 warps and a
// barrier per band 54.3, 20 warps 53.0; without the barrier 16 warps 54.6, 18
// warps 54.7, 20 warps 50.5.  24 warps (72 registers, bands of 6 rows) took
// 1.30x as long in a 50-step sample.
// mphase holds each stage's
// next wait parity across steps; `counts` are the stages' finished warps (0
// between steps) and the copies issued for each in this step.
// Returns false (the same in every thread) if a copy did not complete in
// time; the copies still in flight have then been waited for (bounded).
// A warp whose wait runs out raises *fail and leaves, as do the others at
// their next wait; the barrier at the end makes the decision block-wide.
// *fail is 0 on entry and is never cleared: the kernel returns after a
// failure.
template <bool RAGGED>
__device__ bool stream_step(const SimArgs &A, const ProgSmem &P, const StatePtrs &sp,
                            const Geom &g, int G, int par, int path,
                            float dt, float min_conc, float &mx, uint64_t *bars,
                            uint32_t &mphase, int *counts, volatile int *fail, int R) {
  const int nb = (g.H + R - 1) / R;
  const int SPS = (R + 2) * g.RS;
  float *stage0 = sp.sm;
  const size_t gps = (size_t)g.PS;
  const float *gl_cur = sp.gl + (par ? sp.gmax : 0) * gps;
  float *gl_nxt = sp.gl + (par ? 0 : sp.gmax) * gps;
  volatile int *issued = counts + 2;
  auto issue = [&](int b) {
    float *st = stage0 + (b & 1) * sp.gmax * SPS;
    const int rows = min(R + 2, g.H + 2 - b * R);  // plane rows b*R .. b*R + rows - 1
    const uint32_t bytes = (uint32_t)rows * g.RS * 4u;
    issued[b & 1] = b / 2 + 1;
    fence_proxy_async_shared();
    mbar_expect_tx(bars + (b & 1), bytes * (uint32_t)G);
    for (int p = 0; p < G; ++p) {
      float *dst = st + p * SPS;
      const float *src = gl_cur + p * gps + (size_t)b * R * g.RS;
      if (chk_copy(dst, src, (long)rows * g.RS)) bulk_g2s(dst, src, bytes, bars + (b & 1));
    }
  };
  // Test hook: withhold band 1's copy, so that its wait runs out.
  const bool withhold = A.test_hooks & kHookWithholdBandCopy;
  if (threadIdx.x == 0) {
    issued[1] = 0;
    issue(0);
    if (nb > 1 && !withhold) issue(1);
  }
  const uint32_t mphase0 = mphase;
  for (int b = 0; b < nb; ++b) {
    const int s = b & 1;
    const bool arrived = mbar_wait(bars + s, (mphase >> s) & 1u);
    if (!arrived) *fail = 1;
    if (!__all_sync(kFull, arrived && !*fail)) break;
    mphase ^= 1u << s;
    Geom gb = g;
    gb.y0 = b * R;
    gb.H = min(R, g.H - b * R);
    gb.PS = SPS;
    gb.PSb = 4 * SPS;
    gb.Q = strip_count<kStripRows>(gb.H, g.Wg);
    band_step<kStripRows, RAGGED>(path, P, stage0 + s * sp.gmax * SPS, G, gb,
                          gl_nxt + (size_t)gb.y0 * g.RS, gps, dt, min_conc, mx);
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
      // Releases this warp's reads of the stage; the last one acquires all.
      int n;
      asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;"
                   : "=r"(n)
                   : "r"(smem_addr(counts + s))
                   : "memory");
      if (n == (int)(blockDim.x >> 5) - 1) {
        counts[s] = 0;
        if (b + 2 < nb) issue(b + 2);
      }
    }
    __syncwarp();
  }
  fence_proxy_async_global();  // this step's writes before the next step's copies
  __syncthreads();             // *fail is the same for every thread
  if (*fail) {
    // Bounded second waits for the copies that may still be in flight.
    for (int s = 0; s < 2; ++s)
      if (issued[s] > 0) mbar_wait(bars + s, ((mphase0 >> s) ^ (issued[s] - 1)) & 1u);
    return false;
  }
  return true;
}

// ---- temporal blocking: two Euler steps per pass over the state --------
//
// The streaming schedule reads and writes every plane once per step.  This
// variant (kernel ST == 2) advances the state two steps per pass.  A band
// of R output rows (grid rows [bR, bR + R)) needs the current state of
// grid rows [bR - 2, bR + R + 2): plane rows [bR - 1, bR + R + 3), clipped
// to the plane, arrive in one shared-memory stage by bulk copies.  Step one
// computes grid rows [bR - 1, bR + R] (clipped to the grid) from the stage
// into an intermediate buffer of R + 2 rows -- the band and one halo row on
// either side, which the neighbouring bands compute as well; step two
// computes the band from the intermediate and writes it to the global
// next-state planes.  The copy of band b + 1 is issued once step one of band
// b has read the stage, so it overlaps step two.  Both steps run
// band_step, the one-step schedules' arithmetic, so states are
// bit-identical to them.  Shared memory: G * (R + 4) stage rows and
// G * (R + 2) intermediate rows (R = A.band_rows); the same space holds the
// one-step schedule's two stages of R + 2 rows, which the kernel uses
// for a single step (an odd last step, or a first step after which the
// simulation stops).
//
// mx1 / mx2 receive the threads' max |rate| of the first / second step.
// Returns false (the same in every thread) if a copy did not complete in
// time, after a bounded wait for the copy still in flight.
template <bool RAGGED>
__device__ bool stream_step2(const SimArgs &A, const ProgSmem &P, const StatePtrs &sp,
                             const Geom &g, int G, int par, int path,
                             float dt, float min_conc, float &mx1, float &mx2, uint64_t *bars,
                             uint32_t &mphase, volatile int *fail) {
  const int R = A.band_rows;
  const int nb = (g.H + R - 1) / R;
  const int SPS = (R + 4) * g.RS;   // stage plane stride: plane rows bR-1 .. bR+R+2
  const int IPS = (R + 2) * g.RS;   // intermediate plane stride: grid rows bR-1 .. bR+R
  float *stage = sp.sm;
  float *inter = sp.sm + (size_t)sp.gmax * SPS;
  const size_t gps = (size_t)g.PS;
  const float *gl_cur = sp.gl + (par ? sp.gmax : 0) * gps;
  float *gl_nxt = sp.gl + (par ? 0 : sp.gmax) * gps;
  auto issue = [&](int b) {
    const int p0 = max(b * R - 1, 0);               // first plane row copied
    const int p1 = min(b * R + R + 3, g.H + 2);     // one past the last
    const int off = p0 - (b * R - 1);               // its stage row (1 for band 0)
    const uint32_t bytes = (uint32_t)(p1 - p0) * g.RS * 4u;
    fence_proxy_async_shared();
    mbar_expect_tx(bars, bytes * (uint32_t)G);
    for (int p = 0; p < G; ++p) {
      float *dst = stage + p * SPS + off * g.RS;
      const float *src = gl_cur + p * gps + (size_t)p0 * g.RS;
      if (chk_copy(dst, src, (long)(p1 - p0) * g.RS)) bulk_g2s(dst, src, bytes, bars);
    }
  };
  if (threadIdx.x == 0) issue(0);
  for (int b = 0; b < nb; ++b) {
    const uint32_t parity = mphase & 1u;
    if (!mbar_wait(bars, parity)) *fail = 1;
    mphase ^= 1u;
    // Step one: grid rows [y1, y1 + h1) into the intermediate.
    const int y1 = max(b * R - 1, 0);
    const int h1 = min(b * R + R, g.H - 1) - y1 + 1;
    Geom g1 = g;
    g1.y0 = y1;
    g1.H = h1;
    g1.PS = SPS;
    g1.PSb = 4 * SPS;
    g1.Q = strip_count<kStripRows>(h1, g.Wg);
    // Stage row of grid row y is y - bR + 2; g1's row 0 is grid row y1 - 1.
    const float *st1 = stage + (y1 - b * R + 1) * g.RS;
    float *out1 = inter + (y1 - b * R) * g.RS;  // cell rows land at y - (bR - 1)
    band_step<kStripRows, RAGGED>(path, P, st1, G, g1, out1, (size_t)IPS, dt, min_conc, mx1);
    // Intermediate rows outside the grid are the planes' zero rows.
    const int zlo = (b == 0) ? 0 : -1;                            // grid row -1
    const int zhi = (b * R + R >= g.H) ? g.H - (b * R - 1) : -1;  // grid row H
    for (int i = threadIdx.x; i < 2 * G * g.RS; i += blockDim.x) {
      const int z = i / (G * g.RS), r = i - z * G * g.RS;
      const int row = z == 0 ? zlo : zhi;
      if (row < 0) continue;
      const int p = r / g.RS, x = r - p * g.RS;
      *chk<1>(inter + p * IPS + row * g.RS + x) = 0.0f;
    }
    __syncthreads();  // the stage is free; the intermediate is complete
    if (*fail) {
      mbar_wait(bars, parity);  // bounded second wait for the copy still in flight
      return false;
    }
    if (threadIdx.x == 0 && b + 1 < nb) issue(b + 1);
    // Step two: the band's rows from the intermediate.
    Geom g2 = g;
    g2.y0 = b * R;
    g2.H = min(R, g.H - b * R);
    g2.PS = IPS;
    g2.PSb = 4 * IPS;
    g2.Q = strip_count<kStripRows>(g2.H, g.Wg);
    band_step<kStripRows, RAGGED>(path, P, inter, G, g2, gl_nxt + (size_t)g2.y0 * g.RS, gps, dt,
                          min_conc, mx2);
    __syncthreads();  // the intermediate is free again
  }
  fence_proxy_async_global();  // this pass's writes before the next pass's copies
  return true;
}

// Sets n floats (whole float4 words) to 0, all threads of the block.
__device__ __forceinline__ void zero_floats(float *p, int n) {
  for (int i = threadIdx.x; i < n / 4; i += blockDim.x)
    *reinterpret_cast<float4 *>(chk<4>(p + 4 * (size_t)i)) = f4(0.0f);
}

// Copies the first min(G, A.state_planes) genes' current values of the
// block's rows into dst ([plane][H][W], unpadded).
__device__ __forceinline__ void write_planes(const SimArgs &A, const StatePtrs &sp, const Geom &g,
                                          int G, int par, float *dst) {
  const int planes_out = min(G, A.state_planes);
  for (int i = threadIdx.x; i < planes_out * g.W * g.H; i += blockDim.x) {
    const int kk = i / (g.W * g.H), r = i - kk * g.W * g.H;
    const int y = r / g.W, x = r - y * g.W;
    dst[((size_t)kk * g.Hg + g.y0 + y) * g.W + x] =
        *chk<1>(plane_of(sp, g, kk, par) + cell_offset(g, y, x));
  }
}

// Max of a non-negative, non-NaN float over the cluster's CTAs with one
// cluster barrier: every warp stores its max into slot [rank][warp] of every
// CTA's array.  The barrier also orders the step's halo rows.
__device__ __forceinline__ float cluster_max(float v, float *slots, int rank, int C, int lane,
                                             int warp, int n_warps) {
  const unsigned bits = __reduce_max_sync(kFull, __float_as_uint(v));
  if (lane < C) {
    const uint32_t a = cluster_addr(smem_addr(slots + rank * 32 + warp), lane);
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(bits) : "memory");
  }
  cg::this_cluster().sync();
  unsigned mine = 0u;
  if (lane < n_warps)
    for (int r = 0; r < C; ++r) mine = max(mine, __float_as_uint(slots[r * 32 + lane]));
  return __uint_as_float(__reduce_max_sync(kFull, mine));
}

// The simulation kernel.  A.threads threads per block (whole warps).
//   NTMAX   most threads per block (the register budget: 65536 / NTMAX)
//   LOOP    false: one chunk of strips per warp, geometry computed once per
//           launch; warp w owns chunk w % chunks and takes its part of the
//           genes, w / chunks of (warps / chunks) parts.  true: the warps walk
//           (chunk, gene part) items, any grid size
//   RAGGED  W is not a multiple of 4
//   TRACE   writes trace frames (trace_out) during the step loop; only the
//           variants compiled for it carry that code
//   ST      streaming schedule: planes in the global slot, bands of
//           A.band_rows rows staged through shared memory by bulk copies
//   CL      cluster-split: a cluster of C CTAs (launch attribute) simulates
//           one model at a time, CTA r owning rows [r*Hb, r*Hb + Hb) with
//           Hb = ceil(H / C).  Every CTA of a cluster takes the same branches
//           and passes the same cluster barriers: the model index, the step
//           max and the fitness sum are shared values, identical bits in
//           every CTA.
template <int NTMAX, bool LOOP, bool RAGGED, bool CL, bool TRACE, int ST>
__global__ void __launch_bounds__(NTMAX, 1) sim_kernel(const SimArgs A) {
  extern __shared__ __align__(128) unsigned char smem[];
  ModelSmem &M = *reinterpret_cast<ModelSmem *>(smem);
  ProgSmem &P = *reinterpret_cast<ProgSmem *>(smem + kProgOffset);
  float *s_red = reinterpret_cast<float *>(smem + kRedOffset);
  double *s_dred = reinterpret_cast<double *>(smem + kDredOffset);
  int *s_work = reinterpret_cast<int *>(smem + kWorkOffset);
  float *s_cmax = reinterpret_cast<float *>(smem + kCmaxOffset);
  double *s_csum = reinterpret_cast<double *>(smem + kCsumOffset);

  // Owned chunks step without a block barrier where they can (walked ones lose
  // by it: 100 x 100 147 G cell-updates/s with the barrier, 138 without).
  constexpr bool FREE = !LOOP && !TRACE && ST == 0;
  const int NT = blockDim.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = uniform(tid >> 5), n_warps = NT >> 5;
  int rank = 0, C = 1;
  if constexpr (CL) {
    rank = (int)cg::this_cluster().block_rank();
    C = (int)cg::this_cluster().num_blocks();
  }
  const int Hb = (A.H + C - 1) / C;  // band rows (the last band may be shorter)
  Geom g;
  g.W = A.W;
  g.Hg = A.H;
  g.y0 = rank * Hb;
  g.H = min(A.H - g.y0, Hb);
  g.Wg = A.Wg;
  g.RS = A.row_floats;
  g.PS = A.plane_floats;
  g.RSb = A.row_bytes;
  g.pad = A.row_pad;
  g.SSb = kStripRows * g.RSb + 4 * g.pad;
  g.edges = 32 % g.Wg != 0;
  g.PSb = A.plane_bytes;
  g.Q = strip_count<kStripRows>(g.H, A.Wg);
  g.inv_wg = A.inv_wg;
  g.wg_shift = A.wg_shift;
  const float dt = A.dt, min_conc = A.min_conc;
  uint4 *Mw = reinterpret_cast<uint4 *>(smem);

  StatePtrs sp;
  sp.sm = reinterpret_cast<float *>(smem + kStateOffset);
  sp.gl = A.gstate ? A.gstate + (size_t)blockIdx.x * (size_t)A.slot_floats : nullptr;
  sp.gmax = A.gmax;

#if GRN_BOUNDS_CHECK
  if (tid == 0) {
    CheckRegions &cr = *reinterpret_cast<CheckRegions *>(smem + kCheckOffset);
    uint32_t dyn = 0;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
    cr.sm_lo = sp.sm;
    cr.sm_hi = reinterpret_cast<const float *>(smem + dyn);
    cr.gl_lo = A.gstate;
    // Planes without a row past an odd height's zero row (the no-allocation
    // entry's): the last slot's last strip reads one row further.
    const bool over = C == 1 && (A.H & 1) && A.plane_floats == (A.H + 2) * A.row_floats;
    cr.gl_hi = A.gstate ? A.gstate + (size_t)gridDim.x * (size_t)A.slot_floats +
                              (over ? A.row_floats : 0)
                        : nullptr;
    cr.flag = A.error_flag;
  }
  __syncthreads();
#endif

  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kMbarOffset);
  volatile int *s_stream_fail = reinterpret_cast<volatile int *>(smem + kStreamFailOffset);
  uint32_t mphase = 0;  // streaming: next wait parity of each stage
  int *s_done = reinterpret_cast<int *>(smem + kDoneOffset);
  volatile int *s_fail = s_stream_fail;
  if (tid == 0) *s_fail = 0;  // barriers follow before its first use
  if constexpr (ST) {
    if (tid == 0) {
      mbar_init(bars, 1);
      mbar_init(bars + 1, 1);
      mbar_init_fence();
    }
    __syncthreads();
  }

  Halo halo{};
  if constexpr (CL) {
    const uint32_t state = smem_addr(smem + kStateOffset);
    if (rank > 0) halo.up = cluster_addr(state, rank - 1);
    if (rank < C - 1) halo.down = cluster_addr(state, rank + 1);
    // The first row (plane row 1) to plane row Hb + 1, the last one (Hb) to 0.
    halo.up_rows = 4 * (int)(row_offset(Hb + 1, g.RS, g.pad) - row_offset(1, g.RS, g.pad));
    halo.down_rows = 4 * (int)row_offset(Hb, g.RS, g.pad);
    halo.slot_bytes = A.slot_floats * (int64_t)sizeof(float);
  }

  // Chunks of a full band: the same in every CTA of a cluster.
  // (Streaming: of a full band; of a two-step pass's first step, whose last
  // chunks the second step does not have.)
  const int rows = ST ? min(Hb, A.band_rows + (ST == 2 ? 2 : 0)) : Hb;
  const int chunks = (strip_count<kStripRows>(rows, g.Wg) + 31) / 32;
  // Fixed items: geometry once per launch.
  Strip<kStripRows> fixed;
  int fixed_part = 0;
  const int splits = LOOP ? 0 : max(1, n_warps / chunks);
  const int own = warp % chunks;
  if constexpr (!LOOP) {
    fixed = strip_at<kStripRows>(own * 32 + lane, g);
    fixed_part = warp / chunks;
    if (fixed_part >= splits) fixed_part = GRN_MAX_GENES;  // no work
  }

  StepSync sync{s_done, s_fail, s_done, 0, false, false};
  bool free_steps = false;  // the counts' lanes are enough for this grid
  if constexpr (FREE) {
    const int reach = chunk_reach(g);
    free_steps = min(chunks, 2 * reach + 1) <= (CL ? 30 : 32) && chunks <= kMaxDone &&
                 counts_fit(A.n_steps);
    sync.wait = s_done + min(max(own - reach, 0) + lane, min(own + reach, chunks - 1));
    sync.per_step = splits;
    if constexpr (CL) {
      // Chunks with a band's first row of strips, and with a full band's last.
      const int Q = strip_count<kStripRows>(Hb, g.Wg);
      const int n_first = (g.Wg + 31) / 32, n_last = (Q - 1) / 32 - (Q - g.Wg) / 32 + 1;
      const bool first = rank > 0 && own < n_first;
      const bool last = rank < C - 1 && own >= (Q - g.Wg) / 32 && own <= (Q - 1) / 32;
      if (first && lane == 30) {
        sync.wait = s_done + kMaxDone;
        sync.per_step = n_last * splits;
      }
      if (last && lane == 31) {
        sync.wait = s_done + kMaxDone + 1;
        sync.per_step = n_first * splits;
      }
      sync.first = first;
      sync.last = last;
    }
  }

  for (int iter = 0;; ++iter) {
    int m;
    if constexpr (CL) {
      // Rank 0 hands the next model to every CTA of the cluster.  Two slots
      // by iteration parity: a CTA may still be reading this iteration's
      // slot when rank 0 (past the next cluster barrier at the earliest)
      // writes the following one.
      int *slot = s_work + (iter & 1);
      if (rank == 0 && tid == 0) {
        const int v = atomicAdd(A.work_counter, 1);
        for (int r = 0; r < C; ++r) *cg::this_cluster().map_shared_rank(slot, r) = v;
      }
      cg::this_cluster().sync();
      m = *slot;
    } else {
      if (tid == 0) *s_work = atomicAdd(A.work_counter, 1);
      __syncthreads();
      m = *s_work;
    }
    if (m >= A.n_models) break;
    const uint4 *rec = A.packed + A.offsets[m];
    {
      const uint4 w0 = rec[0];
      const int G0 = (int)(short)(w0.y & 0xffff);
      const int L0 = (int)(short)(w0.y >> 16);
      // Counts outside the format's limits: copy the header alone (the model
      // is rejected below) rather than read past the record.
      const bool sane = G0 >= 0 && G0 <= GRN_MAX_GENES && L0 >= 0 && L0 <= GRN_MAX_LINKS;
      const int words = sane ? 1 + G0 + L0 : 1;
      // Header and genes keep their word; links move to ModelSmem::links.
      for (int w = tid; w < words; w += NT) {
        const int dst = (w <= G0) ? w : w - 1 - G0 + 1 + GRN_MAX_GENES;
        if (dst < kModelWords) Mw[dst] = rec[w];
      }
    }
    __syncthreads();
    const int G = M.hdr.n_genes;
    const int orig = M.hdr.orig_index;
    sp.n_sm = min(G, A.planes / 2);
    const bool exact = !(A.fast_ok && (M.hdr.flags & kFlagFast) &&
                         G <= GRN_MAX_GENES);
    const int path = exact                            ? kExact
                     : M.hdr.flags & kFlagConstantTerm ? kConst
                     : min_conc > 0.0f                ? kClamp
                                                      : kFast;
    const bool bad = G < 1 || G > GRN_MAX_GENES || M.hdr.n_links < 0 ||
                     M.hdr.n_links > GRN_MAX_LINKS || (sp.n_sm < G && sp.gl == nullptr) ||
                     ((sp.n_sm < G || ST) && G > A.gmax) || (!LOOP && chunks > n_warps) ||
                     (ST && (A.band_rows < 1 || sp.gl == nullptr || A.planes != 0));
    if (bad) {
      if (tid == 0 && rank == 0) {
        atomicExch(A.error_flag, 1);
        A.raw_error[orig] = __longlong_as_double(0x7ff8000000000000ll);
        if (A.steps) A.steps[orig] = 0;
      }
      if constexpr (CL) cg::this_cluster().sync();
      else __syncthreads();
      continue;
    }

    build_program(M, P, splits, chunks, n_warps, tid);
    __syncthreads();

    double error = 0.0, change_sum = 0.0;
    int steps_total = 0;
    const double max_err = A.max_error[orig];

    for (int e = 0; e < A.n_exp && error <= max_err; ++e) {
      // Initial state: every plane of both buffers 0, then buffer 0 of the
      // input morphogens from the experiment (simstate.cpp:64-90); the other
      // buffer's cells are all written by the first step.  A band's halo rows
      // start as the neighbouring grid rows.
      const float *init = A.initial + (size_t)e * A.n_in * A.W * A.H;
      for (int i = tid; i < kDoneInts; i += NT) s_done[i] = 0;
      if constexpr (FREE) {
        // Test hook: chunk 0's count starts so far back that no wait for it ends.
        if ((A.test_hooks & kHookWithholdChunkCount) && rank == 0 && tid == 0)
          s_done[0] = -(1 << 30);
      }
      zero_floats(sp.sm, 2 * sp.n_sm * g.PS);
      if (sp.n_sm < G) {
        zero_floats(sp.gl + (size_t)sp.n_sm * g.PS, (G - sp.n_sm) * g.PS);
        zero_floats(sp.gl + (size_t)(sp.gmax + sp.n_sm) * g.PS, (G - sp.n_sm) * g.PS);
      }
      __syncthreads();
      for (int kk = 0; kk < min(A.n_in, G); ++kk) {
        float *pl = plane_of(sp, g, kk, 0);
        for (int i = tid; i < (g.H + 2) * g.Wg; i += NT) {
          const int rr = group_row(i, g.Wg, g.inv_wg, g.wg_shift);
          const int x0 = 4 * (i - rr * g.Wg), y = g.y0 - 1 + rr;  // grid row
          if (y < 0 || y >= g.Hg) continue;
          const float *src = init + ((size_t)kk * g.Hg + y) * g.W + x0;
          float *dst = chk<4>(pl + cell_offset(g, rr - 1, x0));
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (x0 + j < g.W) dst[j] = src[j];
        }
      }
      if constexpr (ST == 2) {
        // The two-step pass's intermediate buffer: its rows' trailing zero
        // cells are never written by a step, so they start at 0 here (the
        // one-step pass's stage copies that may land there carry the
        // planes' zero cells in the same columns).
        float *inter = sp.sm + (size_t)sp.gmax * (A.band_rows + 4) * g.RS;
        for (int i = tid; i < sp.gmax * (A.band_rows + 2) * g.RS; i += NT)
          *chk<1>(inter + i) = 0.0f;
      }
      if constexpr (ST) fence_proxy_async_global();  // before the first bulk copies
      if constexpr (CL) cg::this_cluster().sync();
      else __syncthreads();

      // Trace frames: the state after every trace_every-th step, frame 0
      // the initial state.  A frame reads the current buffer while the
      // next step writes the other one.
      float *trace = nullptr;
      if constexpr (TRACE) {
        trace = A.trace_out + ((size_t)orig * A.n_exp + e) * A.trace_frames * A.state_planes *
                                  g.W * g.Hg;
        write_planes(A, sp, g, G, 0, trace);
      }

      float change = 1.0f;
      int step = 0;
      int par = 0;  // buffer holding the current values
      if constexpr (FREE) {
        // Fast models that stop early only on a change of exactly 0: every
        // rate is then 0 and the state stays as it is, so the steps after it
        // change nothing, and the last step with a rate tells when it was.  They
        // are not run to the end (at_rest).
        if (path == kFast && A.change_bound <= 0.0f && A.n_steps > 0 && free_steps) {
          float mx = 0.0f;
          int last = 0;  // steps up to the warp's last one with a rate
          // Steps s .. end, and whether to go on after them.
          const auto steps_to = [&](int s, int end) {
            for (; s <= end; ++s) {
              mx = 0.0f;
              if (!block_step<kStripRows, LOOP, RAGGED, CL, true>(
                      kFast, P, sp, G, g, fixed, halo, own, fixed_part, splits, chunks, warp, lane,
                      (s - 1) & 1, dt, min_conc, mx, sync, s)) {
                last = 0x7fffffff;
                return false;
              }
              if (__any_sync(kFull, mx > 0.0f)) last = s;
            }
            return !(A.change_bound == 0.0f && end < A.n_steps &&
                     at_rest<CL>(s_done + kMaxDone + 2, end, last == end, C, lane));
          };
          if constexpr (CL) {
            // The same as below.  With the test for a part inside the loop the
            // cluster kernel comes out 3% faster (100 x 100, 592 x 300: 10.74 ->
            // 10.43 ms), the others 1% slower (64 x 64, 592 x 500: 5.77 -> 5.84).
            for (int s = 0; s < A.n_steps;) {
              const int end = min(A.n_steps - s, kVoteSteps) + s;
              if (!(fixed_part < splits && steps_to(s + 1, end))) break;
              s = end;
            }
          } else if (fixed_part < splits) {
            bool go = true;
            for (int s = 1; go && s <= A.n_steps; s += kVoteSteps)
              go = steps_to(s, s + min(A.n_steps - s, kVoteSteps - 1));
          }
          step = A.n_steps;
          par = step & 1;
          if constexpr (CL) {
            change = cluster_max(mx, s_cmax, rank, C, lane, warp, n_warps);
            last = __float_as_int(cluster_max(__int_as_float(last), s_cmax + kMaxCluster * 32, rank,
                                              C, lane, warp, n_warps));
          } else {
            change = block_max(mx, s_red, 0, lane, warp, n_warps);
            last = __float_as_int(block_max(__int_as_float(last), s_red, 1, lane, warp, n_warps));
          }
          if (last == 0x7fffffff) {
            if (tid == 0) {
              atomicExch(A.error_flag, 4);
              A.raw_error[orig] = __longlong_as_double(0x7ff8000000000000ll);
            }
            return;  // every thread of the block (the cluster): a shared value
          }
          if (A.change_bound == 0.0f && last < step) {
            step = last + 1;
            change = 0.0f;
          }
        }
      }
      while (step < A.n_steps && change > A.change_bound) {
        float mx = 0.0f;
        int adv = 1;  // Euler steps this iteration advanced
        if constexpr (ST) {
          // ST == 2: two steps per pass while two remain.  If the first
          // step's change already ends the simulation, that step is run alone
          // again (the one-step pass, in the same shared memory), so the
          // state is the one after exactly one step.
          bool ok = true, single = true;
          if (ST == 2 && step + 2 <= A.n_steps) {
            float mx2 = 0.0f;
            ok = stream_step2<RAGGED>(A, P, sp, g, G, par, path, dt, min_conc, mx, mx2,
                                          bars, mphase, s_stream_fail);
            if (ok) {
              const float b1 = block_max(mx, s_red, par ^ 1, lane, warp, n_warps);
              single = !(b1 > A.change_bound);
              mx = single ? 0.0f : mx2;
              adv = single ? 1 : 2;
            }
          }
          if (ok && single)
            ok = stream_step<RAGGED>(A, P, sp, g, G, par, path, dt, min_conc, mx, bars,
                                         mphase, s_done, s_stream_fail, A.band_rows);
          if (!ok) {
            if (tid == 0) {
              atomicExch(A.error_flag, 2);
              A.raw_error[orig] = __longlong_as_double(0x7ff8000000000000ll);
            }
            return;  // every thread of the block: the decision is block-uniform
          }
        } else {
          block_step<kStripRows, LOOP, RAGGED, CL, false>(path, P, sp, G, g, fixed, halo, own,
                                                          fixed_part, splits, chunks, warp, lane,
                                                          par, dt, min_conc, mx, StepSync{}, 0);
        }
        if constexpr (CL)  // also orders the halo rows stored by this step
          change = cluster_max(mx, s_cmax + par * kMaxCluster * 32, rank, C, lane, warp, n_warps);
        else
          change = block_max(mx, s_red, par, lane, warp, n_warps);
        par ^= 1;
        step += adv;
        if constexpr (TRACE) {
          if (step % A.trace_every == 0 && step / A.trace_every < A.trace_frames)
            write_planes(A, sp, g, G, par,
                         trace + (size_t)(step / A.trace_every) * A.state_planes * g.W * g.Hg);
        }
      }
      steps_total += step;
      change_sum += (double)change;
      if (A.state_out)  // final state of this experiment, unpadded [gene][y][x]
        write_planes(A, sp, g, G, par,
                               A.state_out + ((size_t)orig * A.n_exp + e) * A.state_planes *
                                                 g.W * g.Hg);

      // Fitness of the experiment (simstate.cpp:135-158), FP64 sums.
      const float *tgt = A.target + (size_t)e * A.n_target * A.W * A.H;
      const int cell0 = g.y0 * g.W;  // the band's first cell
      const auto term = [&](int cell, double acc) {
        const int i = cell - cell0;
        const int y = A.inv_w ? (int)__umulhi((uint32_t)i, A.inv_w) : i / g.W, x = i - y * g.W;
        for (int kk = 0; kk < A.n_target; ++kk) {
          const double a = *chk<1>(plane_of(sp, g, A.n_in + kk, par) + cell_offset(g, y, x));
          const double b = tgt[((size_t)kk * g.Hg + g.y0 + y) * g.W + x];
          if (A.fitness_kind == GRN_FITNESS_MSE) {
            acc += (a - b) * (a - b);
          } else {
            const double sub = fabs(a - b) - A.dist_threshold;
            if (sub > 0) acc += log(1.0 + sub);
          }
        }
        return acc;
      };
      const int cell1 = cell0 + g.H * g.W;
      double dist = 0.0;
      if constexpr (CL) {
        // The virtual lanes' sums go from band to band (in the slots of the
        // step maxima, which nobody reads now), so that they add the cells in
        // the order of one CTA.
        double *s_acc = reinterpret_cast<double *>(s_cmax);
        for (int r = 0; r < C; ++r) {
          cg::this_cluster().sync();
          if (rank != r) continue;
          for (int vw = warp; vw < kSumWarps; vw += n_warps) {
            const int slot = vw * 32 + lane;
            const double v = lane_sum(r > 0 ? s_acc[slot] : 0.0, slot, cell0, cell1, term);
            if (r < C - 1) *cg::this_cluster().map_shared_rank(s_acc + slot, r + 1) = v;
            else warp_sum(v, s_dred, vw, lane);
          }
          if (r == C - 1) {
            __syncthreads();
            if (tid < C) *cg::this_cluster().map_shared_rank(s_csum, tid) = total_sum(s_dred);
          }
        }
        cg::this_cluster().sync();
        dist = s_csum[0];
      } else {
        for (int vw = warp; vw < kSumWarps; vw += n_warps)
          warp_sum(lane_sum(0.0, vw * 32 + lane, cell0, cell1, term), s_dred, vw, lane);
        __syncthreads();
        dist = total_sum(s_dred);
      }
      if (A.fitness_kind == GRN_FITNESS_MSE)
        dist /= (double)g.W * g.Hg * A.n_target;
      else
        dist /= (double)(g.W * g.Hg);
      // Non-convergence penalty on the running change sum
      // (evaluatormorphogens.cpp:62-65).
      if (change_sum > A.min_conc_change) dist += change_sum - A.min_conc_change;
      error += dist / A.n_exp;
    }
    if (tid == 0 && rank == 0) {
      A.raw_error[orig] = error;
      if (A.steps) A.steps[orig] = steps_total;
    }
    __syncthreads();
  }
}

// ---- variant table -----------------------------------------------------

typedef void (*KernelFn)(const SimArgs);

struct VariantEntry {
  KernelVariant v;
  KernelFn fn;
};

#define GRN_VARIANT(NT, LOOP, CL, TR, ST)                                     \
  {{NT, LOOP, false, CL, TR, ST}, &sim_kernel<NT, LOOP, false, CL, TR, ST>}, \
  {{NT, LOOP, true, CL, TR, ST}, &sim_kernel<NT, LOOP, true, CL, TR, ST>}

const VariantEntry kVariants[] = {
    GRN_VARIANT(512, false, false, false, 0), GRN_VARIANT(512, true, false, false, 0),
    GRN_VARIANT(1024, false, false, false, 0), GRN_VARIANT(1024, true, false, false, 0),
    // cluster-split
    GRN_VARIANT(1024, false, true, false, 0), GRN_VARIANT(1024, true, true, false, 0),
    // trace frames (one model at a time: any grid, any gene count)
    GRN_VARIANT(512, true, false, true, 0),
    // streaming (bands staged by bulk copies)
    GRN_VARIANT(640, true, false, false, 1),
    // streaming with temporal blocking: two Euler steps per pass
    GRN_VARIANT(640, true, false, false, 2),
};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);

const VariantEntry *find_variant(const KernelVariant &v) {
  for (int i = 0; i < kNumVariants; ++i) {
    const KernelVariant &k = kVariants[i].v;
    if (k.max_threads == v.max_threads && k.loop == v.loop && k.ragged == v.ragged &&
        k.cluster == v.cluster && k.trace == v.trace && k.stream == v.stream)
      return &kVariants[i];
  }
  return nullptr;
}

}  // namespace

size_t sim_fixed_smem_bytes() { return kStateOffset; }

int sim_variant_count() { return kNumVariants; }

KernelVariant sim_variant(int i) { return kVariants[i].v; }

cudaError_t sim_occupancy(const KernelVariant &v, int threads, size_t smem_bytes,
                          int *blocks_per_sm) {
  const VariantEntry *e = find_variant(v);
  if (!e) return cudaErrorInvalidValue;
  cudaError_t err =
      cudaFuncSetAttribute(e->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes);
  if (err != cudaSuccess) {
    *blocks_per_sm = 0;
    cudaGetLastError();
    return cudaSuccess;
  }
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, e->fn, threads,
                                                       smem_bytes);
}

cudaError_t sim_cluster_occupancy(const KernelVariant &v, int threads, size_t smem_bytes,
                                  int cluster, int *clusters) {
  *clusters = 0;
  const VariantEntry *e = find_variant(v);
  if (!e || !v.cluster || cluster < 2 || cluster > kMaxCluster) return cudaErrorInvalidValue;
  if (cudaFuncSetAttribute(e->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes) !=
          cudaSuccess ||
      cudaFuncSetAttribute(e->fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
          cudaSuccess) {
    cudaGetLastError();
    return cudaSuccess;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem_bytes;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(clusters, e->fn, &cfg) != cudaSuccess) {
    *clusters = 0;
    cudaGetLastError();
  }
  return cudaSuccess;
}

cudaError_t sim_launch(const LaunchPlan &plan, const SimArgs &args, cudaStream_t stream) {
  const VariantEntry *e = find_variant(plan.v);
  if (!e) return cudaErrorInvalidValue;
  if (plan.v.cluster != (plan.cluster > 1) || plan.threads < 32 || plan.threads % 32 != 0 ||
      plan.threads > plan.v.max_threads)
    return cudaErrorInvalidValue;
  cudaError_t err = cudaFuncSetAttribute(e->fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)plan.smem_bytes);
  if (err != cudaSuccess) return err;
  if (plan.cluster > 1) {
    // Whole clusters only, each band non-empty.
    const int hb = (args.H + plan.cluster - 1) / plan.cluster;
    if (plan.cluster > kMaxCluster || plan.blocks % plan.cluster != 0 ||
        (plan.cluster - 1) * hb >= args.H)
      return cudaErrorInvalidValue;
    err = cudaFuncSetAttribute(e->fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (err != cudaSuccess) return err;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(plan.blocks, 1, 1);
    cfg.blockDim = dim3(plan.threads, 1, 1);
    cfg.dynamicSmemBytes = plan.smem_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = plan.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, e->fn, args);
  }
  e->fn<<<plan.blocks, plan.threads, plan.smem_bytes, stream>>>(args);
  return cudaGetLastError();
}

}  // namespace grn
