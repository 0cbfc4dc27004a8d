// rak_lpa.cuh -- the persistent label-propagation kernel (all iterations in one cooperative
// launch) for νMG-LPA (S >= 2 Misra-Gries slots) and νBM-LPA (S == 1).
//
// Reference path replaced: rakLowmemLoopCuU (inc/rakLowmemCuda.hxx:469-490) and the move kernels
// it launches every iteration -- rakLowmemMgMoveIterationGroupCukU (:269-317),
// rakLowmemMgMoveIterationBlockCukU (:362-419), rakLowmemBmMoveIterationThreadCukU (:138-161),
// rakLowmemBmMoveIterationBlockCukU (:198-229) -- plus the per-iteration changed-count reset
// (fillValueCuW, :477) and blocking read-back (:486). Here the changed count, the traversed-edge
// count and the convergence test stay on the device; iterations are separated by a bounded grid
// barrier instead of kernel launches and host round trips.
//
// Work is a list of items over the plan's regions (rak_internal.hpp), heaviest first; warps take
// the next item from a per-iteration counter, so the load balances dynamically. Sketches live in
// registers, one per lane.
#pragma once
#include <map>
#include <mutex>
#include <utility>

#include "rak_device.cuh"
#include "rak_internal.hpp"

// Edges per stage of the scan pipeline, and the resident blocks per SM the register
// budget is sized for. Four blocks (64 registers; the asynchronous instantiations spill a few
// hundred bytes) against three (80 registers), measured on B200 on renumbered resident graphs, one
// box, runs alternated: R-MAT s27 100.5-100.7 vs 102.3-102.4 ms at lower clocks, s24 ef32 weighted
// 30.2 vs 31.4 ms, 2D lattice 2^25 9.0 vs 9.8 ms (on the graphs as given, earlier, four blocks were
// 1-5% slower): the loads in flight of the extra warps pay for the spills.
#ifndef RAK_SCAN_BATCH
#define RAK_SCAN_BATCH 2
#endif
#ifndef RAK_MIN_BLOCKS
#define RAK_MIN_BLOCKS 4
#endif

namespace rak {

struct Counters {
  unsigned long long edges;
  unsigned long long moved_edges;
  unsigned int changed;
  unsigned int processed;
};

// How an asynchronous iteration treats the frontier (LpaArgs::dense_moved_edges). all: every
// vertex is processed, whatever its flag (the previous iteration marked no neighbours); nomark:
// moved vertices mark no neighbours (the next iteration processes every vertex). Both false in
// the other modes and in batches: the reference's pruning, flags marked by every move.
// How a synchronous iteration's active set is found (LpaArgs::pull). pull_in: the flags read hold the
// vertices that moved in the previous iteration, and a vertex is active if a neighbour's is set;
// pull_out: this iteration's moves set the mover's own flag for that, and mark no neighbours.
struct Phase {
  bool all;
  bool nomark;
  bool pull_in;
  bool pull_out;
};

template <class O>
struct G_ {
  const O *off;
  const uint32_t *tgt;
  const float *wt;
};

// Edge-stream loads (targets, weights): non-coherent loads. RAK_STREAM_HINT=1 gives them an L2
// evict-first cache policy (an operand of the load instruction, not a setting of the GPU), meant to
// leave L2 capacity to the label gathers; measured on B200 it was 2-3% slower (R-MAT scale 27: 116
// vs 119 G edges/s; scale 24 weighted: 126 vs 128), so it is off.
#ifndef RAK_STREAM_HINT
#define RAK_STREAM_HINT 0
#endif
__device__ __forceinline__ uint64_t l2_stream_policy() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
// RAK_L1_HINTS=1: edge-stream loads allocate in L1 as evict-first and label gathers as evict-last,
// so the streamed edge lines leave L1 before the labels that neighbours share.
#ifndef RAK_L1_HINTS
#define RAK_L1_HINTS 0
#endif
__device__ __forceinline__ uint32_t ld_edge(const uint32_t *p) {
#if RAK_L1_HINTS
  uint32_t v;
  asm("ld.global.nc.L1::evict_first.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
#elif RAK_STREAM_HINT
  uint32_t v;
  asm("ld.global.nc.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(l2_stream_policy()));
  return v;
#else
  return __ldg(p);
#endif
}
__device__ __forceinline__ float ld_weight(const float *p) {
#if RAK_L1_HINTS
  float v;
  asm("ld.global.nc.L1::evict_first.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
#elif RAK_STREAM_HINT
  float v;
  asm("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(l2_stream_policy()));
  return v;
#else
  return __ldg(p);
#endif
}

// Label gathers (neighbour labels, which change during the launch: plain coherent loads).
// RAK_LABEL_HINT=1 gives them an L2 evict-last cache policy (an operand of the load instruction):
// when the label array is larger than L2, the lines of frequently read labels then outlast the
// streamed edge lines; RAK_LABEL_HINT=2 reads them from L2 only (not cached in L1).
#ifndef RAK_LABEL_HINT
#define RAK_LABEL_HINT 0
#endif
__device__ __forceinline__ uint64_t l2_keep_policy() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint32_t ld_label(const uint32_t *p) {
#if RAK_L1_HINTS && RAK_LABEL_HINT == 1
  uint32_t v;
  asm volatile("ld.global.L1::evict_last.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(l2_keep_policy()) : "memory");
  return v;
#elif RAK_L1_HINTS
  uint32_t v;
  asm volatile("ld.global.L1::evict_last.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
#elif RAK_LABEL_HINT == 1
  uint32_t v;
  asm volatile("ld.global.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(l2_keep_policy()) : "memory");
  return v;
#elif RAK_LABEL_HINT == 2
  return __ldcg(p);
#else
  return *p;
#endif
}

template <bool UNIT>
__device__ __forceinline__ float edge_w(const float *wt, int64_t e) {
  if constexpr (UNIT) return 1.0f;
  else return ld_weight(wt + e);
}

// Sequential accumulation (acc) of edges e, e+st, ... < ee of u (self-loops skipped), in edge order.
// Software-pipelined in three stages of two edges: while one stage's labels are accumulated, the next
// stage's labels and the targets (and weights) of the one after are on their way. Positions past the
// end are given the target u itself, which the self-loop rule skips. Labels are read with plain loads:
// they change during the launch. Two stages of four edges, whose labels were waited for -> this, with the
// whole-number sketch below, asynchronous runs measured on B200: R-MAT scale 24 ef 16 11.3 -> 10.5 ms, scale 22
// 3.37 -> 3.15 ms, scale 22 ef 32 weighted 9.7 -> 9.2 ms.
template <bool UNIT, class ACC>
__device__ __forceinline__ void scan_edges(ACC &&acc, uint32_t u, int64_t e, int64_t ee, int st, const uint32_t *tgt,
                                           const float *wt, const uint32_t *vin, uint32_t base) {
  constexpr int B = RAK_SCAN_BATCH;
  // edges of this lane: a chain is at most hub_min / 32, hub_chunk / 32 or lane_max edges, so an int holds
  // it, and 32-bit counts keep the 64-bit address arithmetic to one add per stage
  int left = int((ee - e + st - 1) >> (31 - __clz(st)));   // st: a power of two
  const uint32_t *tp = tgt + e;
  const float *wp = UNIT ? nullptr : wt + e;
  uint32_t t[B], t1[B], c[B];
  float w[B], w1[B];
#pragma unroll
  for (int j = 0; j < B; ++j) {
    t[j] = j < left ? base + ld_edge(tp + j * st) : u;
    w[j] = j < left ? edge_w<UNIT>(wp, j * st) : 0.0f;
    t1[j] = B + j < left ? base + ld_edge(tp + (B + j) * st) : u;
    w1[j] = B + j < left ? edge_w<UNIT>(wp, (B + j) * st) : 0.0f;
  }
#pragma unroll
  for (int j = 0; j < B; ++j) c[j] = ld_label(vin + t[j]);
  tp += 2 * B * st;
  if constexpr (!UNIT) wp += 2 * B * st;
  for (; left > 0; left -= B) {
    uint32_t c1[B], t2[B];
    float w2[B];
#pragma unroll
    for (int j = 0; j < B; ++j) c1[j] = ld_label(vin + t1[j]);
#pragma unroll
    for (int j = 0; j < B; ++j) {
      t2[j] = 2 * B + j < left ? base + ld_edge(tp + j * st) : u;
      w2[j] = 2 * B + j < left ? edge_w<UNIT>(wp, j * st) : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < B; ++j)
      if (t[j] != u) acc(c[j], w[j]);
#pragma unroll
    for (int j = 0; j < B; ++j) { t[j] = t1[j]; c[j] = c1[j]; w[j] = w1[j]; t1[j] = t2[j]; w1[j] = w2[j]; }
    tp += B * st;
    if constexpr (!UNIT) wp += B * st;
  }
}

// Unit weights under the CPU rules accumulate in whole numbers (UnitSketch) where a sketch, clear at
// the start, sees at most 2^24 edges: about half the instructions of the float form on a miss.
template <int S, bool UNIT, int RULE>
__host__ __device__ constexpr bool unit_sketch() { return UNIT && S > 1 && RULE == RULE_CPU; }

// ORDER: the sketch goes straight to the argmax, with no merge in between (one lane per vertex).
template <int S, bool UNIT, int RULE, bool ORDER = false>
__device__ __forceinline__ void scan_range(Sketch<S> &sk, uint32_t u, int64_t e, int64_t ee, int st,
                                           const uint32_t *tgt, const float *wt, const uint32_t *vin,
                                           uint32_t base) {
  if constexpr (unit_sketch<S, UNIT, RULE>()) {
    if (ee - e <= (int64_t(st) << 24)) {
      UnitSketch<S> us;
      unit_clear(us);
      scan_edges<UNIT>([&](uint32_t c, float) { unit_acc(us, c); }, u, e, ee, st, tgt, wt, vin, base);
      unit_to_sketch<S, ORDER>(us, sk);
      return;
    }
  }
  scan_edges<UNIT>([&](uint32_t c, float w) { sk_acc<S, RULE>(sk, c, w); }, u, e, ee, st, tgt, wt, vin, base);
}

// Neighbour marking reads a neighbour's flag before storing it when the launch asks for it
// (LpaArgs::mark_test, mark_test_for). The read goes through L1: most neighbours of a moved vertex
// are flagged already, and a flag line that L1 holds answers without a request to L2. In the
// synchronous modes the flags being set are only set during an iteration (and L1 is invalidated
// by the grid barrier's acquire), so a read can at worst miss a fresh mark and store it again. In
// the asynchronous mode a line L1 holds can also show a flag that another SM has cleared since
// (its vertex was processed); that neighbour is then not marked again for this move -- the same
// kind of lost update as the mode's unordered plain stores, measured with no change of modularity
// (R-MAT scale 24 and 27). RAK_MARK_FORCE=1/2 forces the test on/off (measurements).
#ifndef RAK_MARK_FORCE
#define RAK_MARK_FORCE 0
#endif
__device__ __forceinline__ uint32_t ld_flag_test(const uint8_t *p) { return *p; }

// ---- one lane per vertex: the edge list read in 16-byte vectors -------------------------------
//
// A lane that scans its own vertex of degree RAK_VEC_MIN_DEG or more reads 4 targets (and 4
// weights) per load instead of one: a warp issues a quarter of the edge-stream loads. Requires
// targets (and weights) at 16-byte aligned addresses (checked per launch, lane_vec_ok). Vector v covers edges 4v .. 4v+3; edges outside [e, ee) are masked with the
// target u itself, which the self-loop rule skips, so the lane accumulates exactly edges e .. ee-1
// in order, as scan_range with stride 1 does. Whole-vector loads stay inside [4*floor(e/4), ee);
// the last vector of a range whose end is not a multiple of 4 is read edge by edge.
template <bool UNIT>
__device__ __forceinline__ void load_vec4(int64_t v, int64_t ee, const uint32_t *tgt, const float *wt, uint4 &t4,
                                          float4 &w4) {
  const int64_t x0 = v << 2;
  if (x0 + 4 <= ee) {
#if RAK_L1_HINTS
    asm("ld.global.nc.L1::evict_first.v4.u32 {%0, %1, %2, %3}, [%4];"
        : "=r"(t4.x), "=r"(t4.y), "=r"(t4.z), "=r"(t4.w) : "l"(tgt + x0));
    if constexpr (!UNIT)
      asm("ld.global.nc.L1::evict_first.v4.f32 {%0, %1, %2, %3}, [%4];"
          : "=f"(w4.x), "=f"(w4.y), "=f"(w4.z), "=f"(w4.w) : "l"(wt + x0));
#else
    t4 = __ldg(reinterpret_cast<const uint4 *>(tgt) + v);
    if constexpr (!UNIT) w4 = __ldg(reinterpret_cast<const float4 *>(wt) + v);
#endif
  } else {
    t4.x = x0 < ee ? ld_edge(tgt + x0) : 0u;
    t4.y = x0 + 1 < ee ? ld_edge(tgt + x0 + 1) : 0u;
    t4.z = x0 + 2 < ee ? ld_edge(tgt + x0 + 2) : 0u;
    t4.w = 0u;   // x0 + 3 >= ee here
    if constexpr (!UNIT) {
      w4.x = x0 < ee ? ld_weight(wt + x0) : 0.0f;
      w4.y = x0 + 1 < ee ? ld_weight(wt + x0 + 1) : 0.0f;
      w4.z = x0 + 2 < ee ? ld_weight(wt + x0 + 2) : 0.0f;
      w4.w = 0.0f;
    }
  }
}

// Vector loads pay only on longer lists: a list's first and last vector carry masked positions,
// and the short lists of sparse graphs are mostly such vectors. Measured on B200 (vectors from
// degree 32 / always / never): 2D lattice 2^25 (degree ~4) 9.73 / 12.05 / 9.73 ms; R-MAT scale 25
// ef 4 8.22 / 8.51 / 8.10 ms; R-MAT scale 27 ef 16 128.0 / 128.5 / 130.2 ms; R-MAT scale 24 ef 32
// weighted 32.5 / 32.6 / 33.1 ms.
#ifndef RAK_VEC_MIN_DEG
#define RAK_VEC_MIN_DEG 32
#endif
__device__ __forceinline__ bool lane_vec_ok(const uint32_t *tgt, const float *wt) {
  return ((reinterpret_cast<uintptr_t>(tgt) | (wt ? reinterpret_cast<uintptr_t>(wt) : 0)) & 15u) == 0;
}

template <bool UNIT, class ACC>
__device__ __forceinline__ void scan_vectors(ACC &&acc, uint32_t u, int64_t e, int64_t ee, const uint32_t *tgt,
                                             const float *wt, const uint32_t *vin, uint32_t base) {
  if (e >= ee) return;
  int64_t v = e >> 2;
  const int64_t vend = (ee + 3) >> 2;
  uint4 t4;
  float4 w4 = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
  load_vec4<UNIT>(v, ee, tgt, wt, t4, w4);
  for (; v < vend; ++v) {
    const int64_t x0 = v << 2;
    uint32_t t[4] = {t4.x, t4.y, t4.z, t4.w};
    float w[4] = {w4.x, w4.y, w4.z, w4.w};
    uint32_t c[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t x = x0 + j;
      t[j] = x >= e && x < ee ? base + t[j] : u;
      c[j] = t[j] != u ? ld_label(vin + t[j]) : NONE;
    }
    if (v + 1 < vend) load_vec4<UNIT>(v + 1, ee, tgt, wt, t4, w4);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (t[j] != u) acc(c[j], UNIT ? 1.0f : w[j]);
  }
}

template <int S, bool UNIT, int RULE>
__device__ __forceinline__ void scan_lane(Sketch<S> &sk, uint32_t u, int64_t e, int64_t ee, const uint32_t *tgt,
                                          const float *wt, const uint32_t *vin, uint32_t base) {
  if constexpr (unit_sketch<S, UNIT, RULE>()) {
    UnitSketch<S> us;
    unit_clear(us);
    scan_vectors<UNIT>([&](uint32_t c, float) { unit_acc(us, c); }, u, e, ee, tgt, wt, vin, base);
    unit_to_sketch<S, true>(us, sk);
  } else {
    scan_vectors<UNIT>([&](uint32_t c, float w) { sk_acc<S, RULE>(sk, c, w); }, u, e, ee, tgt, wt, vin, base);
  }
}

// Neighbour marking of a moved vertex scanned by one lane (mark_range with stride 1), from 16-byte
// vectors of targets, two vectors in flight; TEST as in mark_range.
template <bool TEST>
__device__ __forceinline__ void mark_lane(uint32_t u, int64_t e, int64_t ee, const uint32_t *tgt, uint8_t *fout,
                                          uint32_t base) {
  if (e >= ee) return;
  const int64_t vend = (ee + 3) >> 2;
  float4 unused;
  for (int64_t v = e >> 2; v < vend; v += 2) {
    uint4 a4, b4 = make_uint4(0, 0, 0, 0);
    load_vec4<true>(v, ee, tgt, nullptr, a4, unused);
    if (v + 1 < vend) load_vec4<true>(v + 1, ee, tgt, nullptr, b4, unused);
    uint32_t t[8] = {a4.x, a4.y, a4.z, a4.w, b4.x, b4.y, b4.z, b4.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int64_t x = (v << 2) + j;
      t[j] = x >= e && x < ee ? base + t[j] : u;
    }
    uint32_t f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = t[j] == u ? 1u : (TEST ? ld_flag_test(fout + t[j]) : 0u);
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (!f[j]) fout[t[j]] = 1;
  }
}

// Exact weights of the sketch keys in edge order (inc/rakLowmem.hxx:154-162), one lane.
template <int S, bool UNIT>
__device__ __forceinline__ void rescan_range(Sketch<S> &sk, uint32_t u, int64_t e, int64_t ee,
                                             const uint32_t *tgt, const float *wt, const uint32_t *vin,
                                             uint32_t base) {
#pragma unroll
  for (int i = 0; i < S; ++i) sk.w[i] = 0.0f;
  for (; e < ee; ++e) {
    const uint32_t v = base + ld_edge(tgt + e);
    if (v == u) continue;
    const uint32_t c = ld_label(vin + v);
    const float w = edge_w<UNIT>(wt, e);
#pragma unroll
    for (int i = 0; i < S; ++i)
      if (sk.k[i] == c) sk.w[i] = __fadd_rn(sk.w[i], w);
  }
}


// Marks neighbours e, e+st, ... < ee of a moved vertex u as affected (inc/rakCuda.hxx:95-103),
// except u itself (the reference CPU loop clears u after marking, inc/rakLowmem.hxx:203,209).
// Pipelined in batches of eight: the next batch's targets load while this batch is stored.
// test: store a flag only if it reads as clear (ld_flag_test). A random byte store costs the L2 a
// partial write, and most neighbours of a moved vertex are flagged already on large graphs; on
// small or sparse ones the read only lengthens the marking (mark_test_for chooses per launch).
template <bool TEST>
__device__ __forceinline__ void mark_range(uint32_t u, int64_t e, int64_t ee, int st, const uint32_t *tgt,
                                           uint8_t *fout, uint32_t base) {
  constexpr int MB = 8;
  uint32_t v[MB];
#pragma unroll
  for (int j = 0; j < MB; ++j) {
    const int64_t x = e + int64_t(j) * st;
    v[j] = x < ee ? base + ld_edge(tgt + x) : u;
  }
  while (e < ee) {
    uint32_t f[MB];
#pragma unroll
    for (int j = 0; j < MB; ++j) f[j] = v[j] == u ? 1u : (TEST ? ld_flag_test(fout + v[j]) : 0u);
    const int64_t en = e + int64_t(MB) * st;
    uint32_t v2[MB];
#pragma unroll
    for (int j = 0; j < MB; ++j) {
      const int64_t x = en + int64_t(j) * st;
      v2[j] = x < ee ? base + ld_edge(tgt + x) : u;
    }
#pragma unroll
    for (int j = 0; j < MB; ++j)
      if (!f[j]) fout[v[j]] = 1;
#pragma unroll
    for (int j = 0; j < MB; ++j) v[j] = v2[j];
    e = en;
  }
}


template <int S>
__device__ __forceinline__ bool mark_tested(const LpaArgs &a) {
  return RAK_MARK_FORCE == 1 || (RAK_MARK_FORCE == 0 && a.mark_test != 0);
}
template <int S>
__device__ __forceinline__ void mark_item(const LpaArgs &a, uint32_t u, int64_t e, int64_t ee, int st,
                                          const uint32_t *tgt, uint8_t *fout, uint32_t base) {
  if (mark_tested<S>(a)) mark_range<true>(u, e, ee, st, tgt, fout, base);
  else mark_range<false>(u, e, ee, st, tgt, fout, base);
}

// ---- edge tiles staged in shared memory by the bulk-copy engine (TMA) -------------------------
//
// Vertices scanned by a whole warp -- lane groups of 32 (region 1) and split-vertex chunks
// (region 0) -- read one contiguous edge range. With LpaArgs::stage the range is copied tile by
// tile into shared memory with 1-D bulk copies (cp.async.bulk, completion counted in bytes on an
// mbarrier), one tile ahead of the lanes, and the lanes read their edges there instead of loading
// them from global memory. Lane s still accumulates edges eb+s, eb+s+32, ... in that order, so the
// sketches are bit-identical to scan_range's. Bulk copies need 16-byte aligned addresses and sizes:
// the few edges before the range's first aligned address and after its last one are read from
// global memory directly, so no copy reads outside [eb, ee). The source is always this GPU's own
// memory; no copy uses a multicast form.
#ifndef RAK_STAGE
#define RAK_STAGE 1
#endif
constexpr int LPA_WARPS = 8;      // warps per block (256 threads)
constexpr int STG_TILE = 256;     // edges per tile (8 per lane): 16 KB of tiles per block (32 KB weighted)
constexpr int STG_STAGES = 2;     // tiles per warp: one in use, one in flight

// Dynamic shared memory of an lpa_run block that stages tiles: per warp STG_STAGES tiles of
// targets (and of weights, for weighted graphs), then one mbarrier per tile buffer.
__host__ __device__ constexpr size_t stage_bytes(bool unit) {
  return size_t(LPA_WARPS) * STG_STAGES * STG_TILE * 4 * (unit ? 1 : 2) + size_t(LPA_WARPS) * STG_STAGES * 8;
}

struct StageCtx {
  uint32_t *t;     // this warp's target buffers (STG_STAGES x STG_TILE)
  float *w;        // this warp's weight buffers (weighted graphs)
  uint32_t bar;    // shared-memory address of this warp's first mbarrier
  uint32_t phase;  // per buffer, the parity of the next completion to wait for (warp-uniform)
  bool on;         // staging in use for this launch
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_arrive(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// 1-D bulk copy global -> this CTA's shared memory, completing `bytes` on the mbarrier.
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// Waits for the completion of `parity` on an mbarrier, for at most timeout_ns of wall time. On
// expiry it records RAK_ERR_TIMEOUT and the launch's abort flag, as the grid barrier does (the
// launch then ends at its next barrier), and returns false: the caller reads that tile's edges
// from global memory instead.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, RunState *rs, long long timeout_ns) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (!mbar_try(bar, parity)) {
    if ((long long)(global_ns() - t0) > timeout_ns) {
      atomicCAS(&rs->error, 0u, 5u);
      atomicExch(&rs->abort, 1u);
      return false;
    }
  }
  return true;
}

// Lane 0 starts the copy of tile k of [cs, ce) into buffer k % STG_STAGES (all lanes call this).
template <bool UNIT>
__device__ __forceinline__ void stage_issue(const StageCtx &sc, int k, int64_t cs, int64_t ce, const uint32_t *tgt,
                                            const float *wt) {
  const int buf = k % STG_STAGES;
  const int64_t tb = cs + int64_t(k) * STG_TILE;
  const int64_t te = tb + STG_TILE < ce ? tb + STG_TILE : ce;
  const uint32_t bytes = te > tb ? uint32_t(te - tb) * 4u : 0u;
  const uint32_t bar = sc.bar + 8u * uint32_t(buf);
  fence_proxy_async_smem();  // this buffer's earlier reads come before the copy that refills it
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    mbar_expect_arrive(bar, bytes * (UNIT ? 1u : 2u));
    if (bytes) {
      bulk_g2s(smem_u32(sc.t + buf * STG_TILE), tgt + tb, bytes, bar);
      if constexpr (!UNIT) bulk_g2s(smem_u32(sc.w + buf * STG_TILE), wt + tb, bytes, bar);
    }
  }
}

// Staged form of scan_range(sk, u, eb + lane, ee, 32, ...) for a range scanned by the whole warp.
// Every lane calls it with the same range (eb == ee: nothing to scan).
template <int S, bool UNIT, int RULE>
__device__ __forceinline__ void staged_scan(Sketch<S> &sk, StageCtx &sc, uint32_t u, int64_t eb, int64_t ee,
                                            const uint32_t *tgt, const float *wt, const uint32_t *vin, uint32_t base,
                                            RunState *rs, long long timeout_ns) {
  constexpr int B = 4;
  const int lane = threadIdx.x & 31;
  // Copies cover [cs, ce): cs the first edge at a 16-byte aligned address at or after eb, ce the
  // last such boundary at or before ee. Tile k copies [cs + k*STG_TILE, min(cs + (k+1)*STG_TILE, ce));
  // the lanes take edges before cs in tile 0 and after ce in the last tile from global memory.
  int64_t cs = eb + int64_t(((16u - (uint32_t(reinterpret_cast<uintptr_t>(tgt + eb)) & 15u)) & 15u) >> 2);
  if (cs > ee) cs = ee;
  const int64_t ce = cs + ((ee - cs) & ~int64_t(3));
  int nt = ee > eb ? int((ee - cs + STG_TILE - 1) / STG_TILE) : 0;
  if (ee > eb && nt < 1) nt = 1;
  for (int k = 0; k < STG_STAGES && k < nt; ++k) stage_issue<UNIT>(sc, k, cs, ce, tgt, wt);
  int rel = int(eb - cs) + lane;   // the lane's next edge, relative to the current tile's first edge
  for (int k = 0; k < nt; ++k) {
    const int buf = k % STG_STAGES;
    const bool ok = mbar_wait(sc.bar + 8u * uint32_t(buf), (sc.phase >> buf) & 1u, rs, timeout_ns);
    sc.phase ^= 1u << buf;
    const int64_t tb = cs + int64_t(k) * STG_TILE;
    const uint32_t *bt = sc.t + buf * STG_TILE;
    const float *bw = sc.w + buf * STG_TILE;
    const bool whole = ok && k > 0 && tb + STG_TILE <= ce;   // every edge of the tile is in shared memory
    if (whole) {
#pragma unroll
      for (int b0 = 0; b0 < STG_TILE / 32; b0 += B) {
        uint32_t t[B], c[B];
        float w[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
          const int x = rel + (b0 + j) * 32;
          t[j] = base + bt[x];
          w[j] = UNIT ? 1.0f : bw[x];
        }
#pragma unroll
        for (int j = 0; j < B; ++j) c[j] = ld_label(vin + t[j]);
#pragma unroll
        for (int j = 0; j < B; ++j)
          if (t[j] != u) sk_acc<S, RULE>(sk, c[j], w[j]);
      }
      rel += STG_TILE;
    } else {
      // the first or last tile (or a tile whose copy gave up): edges outside the copy from global
      const int hi = k + 1 >= nt ? int(ee - tb) : STG_TILE;
      const int se = ok ? (tb + STG_TILE < ce ? STG_TILE : int(ce - tb)) : 0;
      // the lane consumes only its edges below hi, so that it enters the next tile at an offset
      // in [0, 32): the whole-tile path reads offsets up to that offset + STG_TILE - 32
      while (rel < hi) {
        const int left = (hi - rel + 31) >> 5;
        const int take = left < B ? left : B;
        uint32_t t[B], c[B];
        float w[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
          const int x = rel + j * 32;
          t[j] = u;
          w[j] = 0.0f;
          if (j < take) {
            const bool in = x >= 0 && x < se;
            t[j] = base + (in ? bt[x] : ld_edge(tgt + (tb + x)));
            if constexpr (UNIT) w[j] = 1.0f;
            else w[j] = in ? bw[x] : ld_weight(wt + (tb + x));
          }
        }
#pragma unroll
        for (int j = 0; j < B; ++j) c[j] = ld_label(vin + t[j]);
#pragma unroll
        for (int j = 0; j < B; ++j)
          if (t[j] != u) sk_acc<S, RULE>(sk, c[j], w[j]);
        rel += take * 32;
      }
    }
    rel -= STG_TILE;
    __syncwarp();
    if (k + STG_STAGES < nt) stage_issue<UNIT>(sc, k + STG_STAGES, cs, ce, tgt, wt);
  }
}

// Exact edge-order scan of u by the G lanes of one aligned group: lanes load G edges at a time,
// then every lane applies them in order from shuffles, so all lanes hold the same sketch as a
// single sequential scan would build (and, with rescan, the same exact weights).
template <int S, bool UNIT>
__device__ __forceinline__ void exact_group_scan(Sketch<S> &sk, uint32_t u, int64_t eb, int64_t ee, int G,
                                                 int g, int s, bool rescan, const uint32_t *tgt,
                                                 const float *wt, const uint32_t *vin, uint32_t base) {
  const unsigned gmask = G == 32 ? FULL : (((1u << G) - 1u) << (g * G));
  for (int pass = 0; pass < (rescan ? 2 : 1); ++pass) {
    if (pass == 1) {
#pragma unroll
      for (int i = 0; i < S; ++i) sk.w[i] = 0.0f;
    }
    for (int64_t e0 = eb; e0 < ee; e0 += G) {
      const int64_t e = e0 + s;
      uint32_t c = NONE;
      float w = 0.0f;
      int ok = 0;
      if (e < ee) {
        const uint32_t v = base + ld_edge(tgt + e);
        w = edge_w<UNIT>(wt, e);
        c = ld_label(vin + v);
        ok = v != u;
      }
      const int cnt = int(ee - e0 < G ? ee - e0 : G);
      for (int t = 0; t < cnt; ++t) {
        const uint32_t ct = __shfl_sync(gmask, c, g * G + t);
        const float wt_ = __shfl_sync(gmask, w, g * G + t);
        const int okt = __shfl_sync(gmask, ok, g * G + t);
        if (!okt) continue;
        if (pass == 0) {
          sk_acc(sk, ct, wt_);
        } else {
#pragma unroll
          for (int i = 0; i < S; ++i)
            if (sk.k[i] == ct) sk.w[i] = __fadd_rn(sk.w[i], wt_);
        }
      }
    }
  }
}

// The same sequential scan of one vertex by a whole warp, 32 edges at a time, for long lists. Lane i < S holds
// slot i: its key, its weight and which of the 32 edges hit it (a vote per slot). Edges up to the first miss are
// applied at once, each slot's by its lane: unit weights by counting, others by adding in order. Then the misses
// that follow each other without a hit: with free slots, as many as there are take them together, the first the
// last free one and so on, if their labels differ (a label that repeats would hit what the first one inserted;
// one match at the start tells) and their weights are not zero; with none, unit weights drop by as many misses as
// the smallest weight bears. With rescan a second pass does the same with the final keys. exact_group_scan
// instead takes every edge through every lane's copy of the sketch, about 430 cycles an edge for both passes, and
// the longest list is the iteration. Measured on B200, exact synchronous runs, before -> misses one at a time ->
// this: R-MAT scale 16 ef 16 22.8 -> 10.5 -> 5.8 ms, weighted 55 -> 35 -> 22 ms, scale 18 147 -> 82 -> 36 ms (the
// last two with marking instead of pulling before).
template <int S, bool UNIT>
__device__ __forceinline__ void exact_warp_scan(Sketch<S> &sk, uint32_t u, int64_t eb, int64_t ee, bool rescan,
                                                const uint32_t *tgt, const float *wt, const uint32_t *vin,
                                                uint32_t base) {
  const int lane = threadIdx.x & 31;
  const unsigned before = (1u << lane) - 1u;   // the lanes before this one
  uint32_t k = NONE, num = 0u, low = 0u;       // slot `lane`; unit weights: it weighs num - low
  float w = 0.0f;
  for (int pass = 0; pass < (rescan ? 2 : 1); ++pass) {
    if (pass == 1) { num = low = 0u; w = 0.0f; }
    uint32_t t = eb + lane < ee ? base + ld_edge(tgt + eb + lane) : u;
    float x = !UNIT && eb + lane < ee ? ld_weight(wt + eb + lane) : 0.0f;
    uint32_t c = t != u ? ld_label(vin + t) : NONE;
    for (int64_t e = eb; e < ee; e += 32) {
      // the next 32 edges and their labels are on their way while these are applied
      const int64_t y = e + 32 + lane;
      const uint32_t t2 = y < ee ? base + ld_edge(tgt + y) : u;
      const float x2 = !UNIT && y < ee ? ld_weight(wt + y) : 0.0f;
      const uint32_t c2 = t2 != u ? ld_label(vin + t2) : NONE;
      const bool ok = t != u;   // self-loops and positions past the end take no part
      const unsigned valid = __ballot_sync(FULL, ok);
      unsigned own = 0u, hits = 0u;   // edges that hit slot `lane`; any slot
#pragma unroll
      for (int i = 0; i < S; ++i) {
        const uint32_t ki = __shfl_sync(FULL, k, i);
        const unsigned m = __ballot_sync(FULL, ok && c == ki);
        hits |= m;
        if (lane == i) own = m;
      }
      unsigned left = FULL;   // edges not applied yet
      unsigned miss = pass == 0 ? valid & ~hits : 0u;
      unsigned peers = 0u, light = 0u;   // edges of the same label; edges of weight 0
      if (miss) {
        peers = __match_any_sync(FULL, c) & valid;
        if constexpr (!UNIT) light = __ballot_sync(FULL, x == 0.0f);
      }
      for (;;) {
        const unsigned now = left & (miss ? (miss & (0u - miss)) - 1u : FULL);
        if constexpr (UNIT) {
          num += unsigned(__popc(own & now));
        } else {
          unsigned mine = own & now;
          const int most = __reduce_max_sync(FULL, __popc(mine));
          for (int n = 0; n < most; ++n) {
            const float xw = __shfl_sync(FULL, x, mine ? __ffs(int(mine)) - 1 : 0);
            if (mine) w = __fadd_rn(w, xw);
            mine &= mine - 1u;
          }
        }
        if (!miss) break;
        const int p = __ffs(int(miss)) - 1;
        const unsigned open = __ballot_sync(FULL, lane < S && (UNIT ? num == low : w == 0.0f));
        int done = 1;   // misses settled now: edges p .. p + done - 1
        if (open) {
          // misses from p on whose label has not come up since p
          const unsigned again = __ballot_sync(FULL, ((peers & before) >> p) != 0u);
          const unsigned run = (miss & ~again) >> p;
          const int len = run == FULL ? 32 : __ffs(int(~run)) - 1, room = __popc(open);
          done = len < room ? len : room;
          if (!UNIT && ((light >> p) & ((done == 32 ? 0u : 1u << done) - 1u)) != 0u) done = 1;
          const int j = __popc(open & ~before & ~(1u << lane));   // free slots after this one
          const int from = p + (j < done ? j : 0);
          const uint32_t cn = __shfl_sync(FULL, c, from);
          const unsigned next = __shfl_sync(FULL, peers, from);
          const float xn = UNIT ? 1.0f : __shfl_sync(FULL, x, from);
          if (((open >> lane) & 1u) && j < done) {
            k = cn;
            num = low + 1u;
            w = xn;
            own = next & ~((2u << from) - 1u);
          }
          hits = __reduce_or_sync(FULL, own);
        } else if constexpr (UNIT) {
          const unsigned run = miss >> p;
          const unsigned len = run == FULL ? 32u : unsigned(__ffs(int(~run)) - 1);
          const unsigned bears = __reduce_min_sync(FULL, lane < S ? num - low : 32u);
          done = int(len < bears ? len : bears);
          low += unsigned(done);
        } else {
          const float xp = __shfl_sync(FULL, x, p);
          w = fmaxf(__fsub_rn(w, xp), 0.0f);
        }
        left = p + done > 31 ? 0u : FULL << (p + done);
        miss = valid & ~hits & left;
      }
      t = t2; x = x2; c = c2;
    }
  }
#pragma unroll
  for (int i = 0; i < S; ++i) {
    sk.k[i] = __shfl_sync(FULL, k, i);
    sk.w[i] = __shfl_sync(FULL, UNIT ? float(num - low) : w, i);
  }
}
// Whether a list is scanned that way: Misra-Gries, and short enough for whole-number unit weights.
template <int S, bool UNIT>
__device__ __forceinline__ bool exact_by_warp(int64_t edges) { return S > 1 && (!UNIT || edges <= (int64_t(1) << 24)); }

// Batches: a vertex's graph, whether that graph has converged, and its first vertex (the offset
// of the graph's local target ids). Single graphs: never finished, offset 0.
template <bool BATCH>
__device__ __forceinline__ bool graph_of(const LpaArgs &a, uint32_t u, uint32_t &gi, uint32_t &base) {
  if constexpr (BATCH) {
    gi = __ldg(a.gid + u);
    base = uint32_t(__ldg(a.vbase + gi));
    return a.gdone[gi] != 0;
  } else {
    gi = 0;
    base = 0;
    return false;
  }
}

template <bool BATCH>
__device__ __forceinline__ void count_move(const LpaArgs &a, uint32_t gi, int it) {
  if constexpr (BATCH) atomicAdd(a.gchanged + int64_t(it & 1) * a.ngraphs + gi, 1ull);
}

// The same with one add for the lanes of the warp that come here together from the same graph: the counters of
// a batch's graphs lie side by side in a few sectors of L2, which takes their adds one after the other. Measured
// on B200, an add per moved vertex -> this: 256 graphs of 8.4 M vertices, synchronous split, 37.5 -> 23.6 ms.
template <bool BATCH>
__device__ __forceinline__ void count_moves(const LpaArgs &a, uint32_t gi, int it) {
  if constexpr (BATCH) {
    const unsigned here = __activemask(), peers = __match_any_sync(here, gi);
    if ((threadIdx.x & 31) == unsigned(__ffs(int(peers)) - 1))
      atomicAdd(a.gchanged + int64_t(it & 1) * a.ngraphs + gi, (unsigned long long)__popc(peers));
  }
}

// CPU rule: w > 0 && c != d (inc/rakLowmem.hxx:203). GPU rule: the best weight is non-zero for
// Misra-Gries (inc/rakLowmemCuda.hxx:306), any candidate for Boyer-Moore (:152). Both: on pickless
// iterations no move to a larger label (:309, :153).
template <int S, int RULE, bool BITS = false>
__device__ __forceinline__ bool move_rule(float w, uint32_t c, uint32_t d, bool pickless) {
  const bool weight_ok = RULE == RULE_GPU ? (S == 1 || w != 0.0f) : heavier<BITS>(w, 0.0f);
  return weight_ok && c != d && !(pickless && c > d);
}

// Argmax of a vertex's sketch under the launch's tie rule: hashed ties on iterations
// l < a.tie_until (Misra-Gries, CPU rules), else the rule set's own. u_local: the vertex's id within
// its graph, so a graph breaks its ties the same way alone and in a batch.
template <int S, int RULE, bool BITS = false>
__device__ __forceinline__ void choose(const LpaArgs &a, const Sketch<S> &sk, uint32_t u_local, int it, uint32_t &c,
                                       float &w) {
  if constexpr (S > 1 && RULE != RULE_GPU) {
    const int l = a.start_iter + it;
    if (l < a.tie_until) {
      sk_choose_hashed<S, BITS>(sk, u_local, uint32_t(l), c, w);
      return;
    }
  }
  sk_choose<S, RULE, BITS>(sk, c, w);
}

// ---- the active set of a synchronous iteration, pulled ------------------------------------------
//
// On a symmetric graph a vertex has been marked exactly if one of its neighbours moved. Marking stores
// a flag for every edge of every moved vertex -- and B200's L2 takes one store per 32-byte sector in
// about 22 cycles, so the flags of a few popular vertices serialise: random flag stores measured 123
// G/s over 2^20 flags, 44 over 2^16, 11 over 2^12, against 289 G/s for label gathers. When most vertices
// move, looking for one neighbour that moved ends at the first or second edge instead. The kernel
// chooses per iteration (lpa_run), on graphs whose symmetry the launch has checked (k_symmetry);
// results are the same either way. Measured on B200 (synchronous split runs, marked -> pulled):
// R-MAT scale 24 ef 16 77.6 -> 50.7 ms, scale 22 20.8 -> 12.5 ms, scale 20 ef 32 weighted 32.6 -> 13.8 ms, scale
// 16 2.4 -> 1.6 ms, SBM 1 M vertices 4.1 -> 2.7 ms.

// Whether a neighbour of u among edges [e, ee) moved; one lane, four edges in flight.
__device__ __forceinline__ bool lane_pull(uint32_t u, int64_t e, int64_t ee, const uint32_t *tgt, const uint8_t *fin,
                                          uint32_t base) {
  constexpr int B = 4;
  for (; e < ee; e += B) {
    uint32_t t[B], any = 0;
#pragma unroll
    for (int j = 0; j < B; ++j) t[j] = e + j < ee ? base + ld_edge(tgt + e + j) : u;
#pragma unroll
    for (int j = 0; j < B; ++j) any |= t[j] != u ? uint32_t(fin[t[j]]) : 0u;
    if (any) return true;
  }
  return false;
}

// The same by the aligned groups of G lanes, each for its own vertex (want: the group looks at all);
// every lane of the warp calls it, and a group's lanes get the same answer. One edge a lane first, which
// mostly finds one; then PULL_BATCH at a time: a list without a moved neighbour is read to its end, and with
// one edge in flight a lane 60000 edges took a warp 0.7 ms.
constexpr int PULL_BATCH = 8;
__device__ __forceinline__ bool group_pull(bool want, uint32_t u, int64_t eb, int64_t ee, int s, int G, int grp,
                                           const uint32_t *tgt, const uint8_t *fin, uint32_t base) {
  const unsigned gm = G == 32 ? FULL : ((1u << G) - 1u) << (grp * G);
  int64_t e = eb + s;
  uint32_t any = 0u;
  if (want && e < ee) {
    const uint32_t t = base + ld_edge(tgt + e);
    any = t != u ? uint32_t(fin[t]) : 0u;
  }
  bool found = (__ballot_sync(FULL, any != 0u) & gm) != 0;
  e += G;
  while (__ballot_sync(FULL, want && !found && e < ee)) {
    if (want && !found && e < ee) {
      uint32_t t[PULL_BATCH];
#pragma unroll
      for (int j = 0; j < PULL_BATCH; ++j) t[j] = e + j * G < ee ? base + ld_edge(tgt + e + j * G) : u;
#pragma unroll
      for (int j = 0; j < PULL_BATCH; ++j) any |= t[j] != u ? uint32_t(fin[t[j]]) : 0u;
    }
    const unsigned hits = __ballot_sync(FULL, any != 0u);   // by every lane, outside any condition
    found = found || (hits & gm) != 0;
    e += int64_t(PULL_BATCH) * G;
  }
  return found;
}

// ---- work items: open (what to scan), close (choose, move) --------------------------------------

// Region 6: one lane per vertex. Items are collected into a per-warp queue of active vertices
// (inactive ones are settled at once), and the queue is processed 32 vertices at a time so every
// lane has work; region 6 is sorted by degree, so a batch holds vertices of similar degree.
template <class O, bool BATCH>
__device__ __forceinline__ bool lane_active(const LpaArgs &a, const G_<O> &g, uint32_t u, const uint8_t *fin, Phase ph) {
  uint32_t gi, base;
  if (graph_of<BATCH>(a, u, gi, base)) return false;
  if (ph.pull_in) return lane_pull(u, int64_t(__ldg(g.off + u)), int64_t(__ldg(g.off + u + 1)), g.tgt, fin, base);
  return ph.all || fin[u] != 0;
}

template <int MODE, class O, bool BATCH>
__device__ __forceinline__ int lane_collect(const LpaArgs &a, const Regions &rg, const G_<O> &g, int64_t local,
                                            const uint32_t *vin, uint32_t *vout, const uint8_t *fin, uint8_t *fout,
                                            uint32_t *q, int qn, Phase ph) {
  const int lane = threadIdx.x & 31;
  const int64_t idx = local * 32 + lane;
  bool act = false;
  uint32_t u = 0;
  if (idx < rg.vcount[REG_LANE]) {
    u = __ldg(a.order + rg.vbegin[REG_LANE] + idx);
    act = lane_active<O, BATCH>(a, g, u, fin, ph);
    if constexpr (MODE != MODE_ASYNC)
      if (!act) {
        vout[u] = vin[u];
        if (ph.pull_out) fout[u] = 0;
      }
  }
  const unsigned m = __ballot_sync(FULL, act);
  if (act) q[qn + __popc(m & ((1u << lane) - 1u))] = u;
  __syncwarp();
  return qn + __popc(m);
}

// The choice and move of an active vertex scanned by one lane; true if it moved.
template <int S, int MODE, bool UNIT, bool BATCH, int RULE>
__device__ __forceinline__ bool lane_close(const LpaArgs &a, const Sketch<S> &sk, uint32_t u, uint32_t d, uint32_t gi,
                                           uint32_t base, int64_t deg, int it, bool pickless, uint32_t *vout, uint8_t *fin,
                                           uint8_t *fout, Counters &cnt, Phase ph) {
  uint32_t c;
  float w;
  constexpr bool BITS = unit_sketch<S, UNIT, RULE>();   // weights as unit_to_sketch<S, true> leaves them
  choose<S, RULE, BITS>(a, sk, u - base, it, c, w);
  const bool moved = move_rule<S, RULE, BITS>(w, c, d, pickless);
  cnt.processed += 1;
  cnt.edges += (unsigned long long)deg;
  if constexpr (MODE == MODE_ASYNC) {
    fin[u] = 0;
    if (moved) vout[u] = c;
  } else {
    vout[u] = moved ? c : d;
    if (ph.pull_out) fout[u] = moved ? 1 : 0;
  }
  if (moved) {
    cnt.changed += 1;
    cnt.moved_edges += (unsigned long long)deg;
    count_moves<BATCH>(a, gi, it);
  }
  return moved;
}

template <int S, int MODE, class O, bool UNIT, bool BATCH, int RULE>
__device__ __forceinline__ void lane_batch(const LpaArgs &a, const G_<O> &g, const uint32_t *q, int count,
                                           int it, bool pickless, const uint32_t *vin, uint32_t *vout,
                                           uint8_t *fin, uint8_t *fout, Counters &cnt, Phase ph) {
  const int lane = threadIdx.x & 31;
  if (lane >= count) return;
  const uint32_t u = q[lane];
  const uint32_t d = vin[u];
  uint32_t gi, base;
  graph_of<BATCH>(a, u, gi, base);
  const int64_t eb = int64_t(__ldg(g.off + u)), ee = int64_t(__ldg(g.off + u + 1));
  Sketch<S> sk;
  sk_clear<S, RULE>(sk, d);
  const bool vec = lane_vec_ok(g.tgt, g.wt) && ee - eb >= RAK_VEC_MIN_DEG;
  if (vec) scan_lane<S, UNIT, RULE>(sk, u, eb, ee, g.tgt, g.wt, vin, base);
  else scan_range<S, UNIT, RULE, true>(sk, u, eb, ee, 1, g.tgt, g.wt, vin, base);
  if constexpr (MODE == MODE_SYNC && S > 1)
    if (a.rescan) rescan_range<S, UNIT>(sk, u, eb, ee, g.tgt, g.wt, vin, base);
  if (!lane_close<S, MODE, UNIT, BATCH, RULE>(a, sk, u, d, gi, base, ee - eb, it, pickless, vout, fin, fout, cnt, ph)) return;
  if (ph.nomark || ph.pull_out) return;
  if (!vec) mark_item<S>(a, u, eb, ee, 1, g.tgt, fout, base);
  else if (mark_tested<S>(a)) mark_lane<true>(u, eb, ee, g.tgt, fout, base);
  else mark_lane<false>(u, eb, ee, g.tgt, fout, base);
}

// Regions 1..5: aligned groups of G lanes per vertex. A lane's view of its group's vertex.
struct GroupVertex {
  uint32_t u, d, gi, base;
  int64_t eb, ee;
  bool valid, active;
};

// Notes a long list of region 1 that an iteration left out of its active set (LONG_IDLE, for pulls_next): the
// lane that calls it speaks for its vertex u.
template <class O>
__device__ __forceinline__ void note_idle(const LpaArgs &a, const G_<O> &g, uint32_t u, int it) {
  const int64_t deg = int64_t(__ldg(g.off + u + 1)) - int64_t(__ldg(g.off + u));
  if (deg > a.m / 512) atomicOr(a.stats + STATS_STRIDE * it + STAT_MOVED_EDGES, LONG_IDLE);
}

template <int MODE, class O, bool BATCH>
__device__ __forceinline__ GroupVertex group_open(const LpaArgs &a, const Regions &rg, const G_<O> &g, int r,
                                                  int64_t local, int it, const uint32_t *vin, const uint8_t *fin,
                                                  Phase ph) {
  const int G = region_group(r);
  const int lane = threadIdx.x & 31, grp = lane / G, s = lane & (G - 1);
  const int64_t idx = local * (32 / G) + grp;
  GroupVertex v{0, 0, 0, 0, 0, 0, idx < rg.vcount[r], false};
  bool running = false;
  if (v.valid) {
    v.u = __ldg(a.order + rg.vbegin[r] + idx);
    v.d = vin[v.u];
    running = !graph_of<BATCH>(a, v.u, v.gi, v.base);
    v.active = running && (ph.pull_in || ph.all || fin[v.u] != 0);
    if (v.active) { v.eb = int64_t(__ldg(g.off + v.u)); v.ee = int64_t(__ldg(g.off + v.u + 1)); }
  }
  if (ph.pull_in)
    v.active = G == 1 ? v.active && lane_pull(v.u, v.eb, v.ee, g.tgt, fin, v.base)
                      : group_pull(v.active, v.u, v.eb, v.ee, s, G, grp, g.tgt, fin, v.base);
  if constexpr (MODE != MODE_ASYNC)
    if (G == 32 && s == 0 && a.pull != 0 && running && !v.active) note_idle(a, g, v.u, it);
  return v;
}
// Merges the group's sketches, chooses and moves; true on every lane of the group if it moved.
template <int S, int MODE, bool BATCH, int RULE>
__device__ __forceinline__ bool group_close(const LpaArgs &a, Sketch<S> &sk, const GroupVertex &v, int r, int it,
                                            bool pickless, uint32_t *vout, uint8_t *fin, uint8_t *fout, Counters &cnt,
                                            Phase ph) {
  const int G = region_group(r);
  const int lane = threadIdx.x & 31, grp = lane / G, s = lane & (G - 1);
  if constexpr (MODE != MODE_SYNC) sk_tree<S, RULE>(sk, G);
  uint32_t c;
  float w;
  choose<S, RULE>(a, sk, v.u - v.base, it, c, w);
  bool moved = v.active && move_rule<S, RULE>(w, c, v.d, pickless);
  moved = __shfl_sync(FULL, moved, grp * G);
  if (s == 0 && v.valid) {
    if (v.active) { cnt.processed += 1; cnt.edges += (unsigned long long)(v.ee - v.eb); }
    if constexpr (MODE == MODE_ASYNC) {
      if (v.active) fin[v.u] = 0;
      if (moved) vout[v.u] = c;
    } else {
      vout[v.u] = moved ? c : v.d;
      if (ph.pull_out) fout[v.u] = moved ? 1 : 0;
    }
    if (moved) { cnt.changed += 1; cnt.moved_edges += (unsigned long long)(v.ee - v.eb); count_moves<BATCH>(a, v.gi, it); }
  }
  return moved;
}

template <int S, int MODE, class O, bool UNIT, bool BATCH, int RULE>
__device__ __forceinline__ void group_item(const LpaArgs &a, const Regions &rg, const G_<O> &g, int r, int64_t local,
                                           int it, bool pickless, const uint32_t *vin, uint32_t *vout,
                                           uint8_t *fin, uint8_t *fout, Counters &cnt, StageCtx &sc, Phase ph) {
  const int G = region_group(r);
  const int lane = threadIdx.x & 31, grp = lane / G, s = lane & (G - 1);
  const GroupVertex v = group_open<MODE, O, BATCH>(a, rg, g, r, local, it, vin, fin, ph);
  Sketch<S> sk;
  sk_clear<S, RULE>(sk, v.d);
  if constexpr (MODE == MODE_SYNC) {
    // groups of 8 lanes or more (lists above 4 * lane_max edges, 1024 by default): their lists one after the other
    // by the whole warp; smaller groups side by side (lists one after the other from 2 lanes on: R-MAT scale 12 without
    // rescan 2.0 -> 3.5 ms). With a small lane_max the same line pays: lane_max 8, lists of 33 edges or more, edge by
    // edge -> this, degree 34 1.80 -> 1.47 ms, degree 64 4.85 -> 2.46 ms, R-MAT scale 14 6.6 -> 1.57 ms
    if (S > 1 && G >= 8) {
      for (int o = 0; o < 32; o += G) {
        if (__shfl_sync(FULL, int(v.active), o) == 0) continue;
        const uint32_t u = __shfl_sync(FULL, v.u, o), base = __shfl_sync(FULL, v.base, o);
        const int64_t eb = __shfl_sync(FULL, v.eb, o), ee = __shfl_sync(FULL, v.ee, o);
        Sketch<S> whole;
        if (exact_by_warp<S, UNIT>(ee - eb)) {
          exact_warp_scan<S, UNIT>(whole, u, eb, ee, a.rescan != 0, g.tgt, g.wt, vin, base);
          if (grp * G == o) sk = whole;
        } else if (grp * G == o) {
          exact_group_scan<S, UNIT>(sk, u, eb, ee, G, grp, s, a.rescan != 0, g.tgt, g.wt, vin, base);
        }
      }
    } else if (v.active) {
      exact_group_scan<S, UNIT>(sk, v.u, v.eb, v.ee, G, grp, s, S > 1 && a.rescan, g.tgt, g.wt, vin, v.base);
    }
  } else {
    if (sc.on && G == 32)   // one vertex per warp: the warp's range is uniform
      staged_scan<S, UNIT, RULE>(sk, sc, v.u, v.active ? v.eb : 0, v.active ? v.ee : 0, g.tgt, g.wt, vin, v.base,
                                 static_cast<RunState *>(a.rs), a.timeout_ns);
    else if (v.active)
      scan_range<S, UNIT, RULE>(sk, v.u, v.eb + s, v.ee, G, g.tgt, g.wt, vin, v.base);
  }
  const bool moved = group_close<S, MODE, BATCH, RULE>(a, sk, v, r, it, pickless, vout, fin, fout, cnt, ph);
  if (moved && !ph.nomark && !ph.pull_out) mark_item<S>(a, v.u, v.eb + s, v.ee, G, g.tgt, fout, v.base);
}

// Region 0: one chunk of a split vertex per item. In the synchronous exact mode chunk 0's warp
// scans the whole vertex in edge order and the other chunks do nothing. Otherwise each chunk's
// warp builds a partial sketch (lane-strided, tree-merged), stores it, and the last chunk to
// arrive merges all partial sketches in a fixed order and makes the move; its neighbours are
// marked in a second phase after the iteration's barrier.
struct HubChunk {
  uint32_t h, u, gi, base;
  int64_t first, nch, j;   // the vertex's first chunk and chunks, this one's index among them
  int64_t eb, ee, cb, ce;  // edges of the vertex and of the chunk
  bool active;
};

// Which split vertices have a neighbour that moved, before iteration `next` pulls: every chunk's warp looks
// through its own edges, unless a chunk of the vertex has found one, and hub_claim (which only asynchronous
// launches use otherwise) takes the iteration's number. Each edge is looked at once at most, by as many warps as
// there are chunks; a search of the whole list by every chunk's warp instead made a settled vertex of a million
// edges beside moving ones cost 12 ms an iteration (R-MAT graphs, whose first edges find a mover: the same). The
// caller's barrier comes before and after. Inlined: as a function of its own it cost batches 4%.
template <class O, bool BATCH>
__device__ __forceinline__ void hub_pull(const LpaArgs &a, const Regions &rg, const uint8_t *movers, int next) {
  const G_<O> g{static_cast<const O *>(a.off), a.tgt, a.wt};
  const int lane = threadIdx.x & 31;
  const int64_t gw = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  for (int64_t i = gw; i < a.nchunks; i += nw) {
    const uint32_t h = __ldg(a.chunk_hub + i);
    unsigned int known = 0u;
    if (lane == 0) known = *(volatile unsigned int *)(a.hub_claim + h);
    if (__shfl_sync(FULL, known, 0) == unsigned(next + 1)) continue;
    const uint32_t u = __ldg(a.order + rg.vbegin[REG_HUB] + h);
    uint32_t gi, base;
    // a batch may be settling its graphs meanwhile: one lane's reading holds for the warp, and either will do
    if (__shfl_sync(FULL, int(graph_of<BATCH>(a, u, gi, base)), 0)) continue;
    const int64_t eb = int64_t(__ldg(g.off + u)), ee = int64_t(__ldg(g.off + u + 1));
    const int64_t cb = eb + (i - __ldg(a.hub_first + h)) * a.hub_chunk;
    const int64_t ce = cb + a.hub_chunk < ee ? cb + a.hub_chunk : ee;
    const bool found = group_pull(true, u, cb, ce, lane, 32, 0, g.tgt, movers, base);
    if (found && lane == 0) *(volatile unsigned int *)(a.hub_claim + h) = unsigned(next + 1);
  }
}

template <int MODE, class O, bool BATCH>
__device__ __forceinline__ HubChunk hub_open(const LpaArgs &a, const Regions &rg, const G_<O> &g, int64_t local, int it,
                                             uint8_t *fin, Phase ph) {
  const int lane = threadIdx.x & 31;
  HubChunk k;
  k.h = __ldg(a.chunk_hub + local);
  k.first = __ldg(a.hub_first + k.h);
  k.nch = __ldg(a.hub_first + k.h + 1) - k.first;
  k.j = local - k.first;
  k.u = __ldg(a.order + rg.vbegin[REG_HUB] + k.h);
  k.eb = int64_t(__ldg(g.off + k.u));
  k.ee = int64_t(__ldg(g.off + k.u + 1));
  k.cb = k.eb + k.j * a.hub_chunk;
  k.ce = k.cb + a.hub_chunk < k.ee ? k.cb + a.hub_chunk : k.ee;
  const bool gfin = graph_of<BATCH>(a, k.u, k.gi, k.base);  // stable within an iteration
  if (gfin) {
    k.active = false;
  } else if (MODE != MODE_ASYNC) {
    k.active = ph.pull_in ? __ldcg(a.hub_claim + k.h) == unsigned(it + 1) : fin[k.u] != 0;   // hub_pull
  } else {
    // All chunks of u agree on whether u is processed this iteration: the first chunk to get
    // here decides from u's flag (and clears it); the others read the decision.
    unsigned int dec = 0;
    if (lane == 0) {
      const unsigned int tag = unsigned(it + 1);
      unsigned int cur = *(volatile unsigned int *)(a.hub_claim + k.h);
      if ((cur >> 1) != tag) {
        const unsigned int want = (tag << 1) | (ph.all || *(volatile uint8_t *)(fin + k.u) ? 1u : 0u);
        const unsigned int prev = atomicCAS(a.hub_claim + k.h, cur, want);
        if (prev == cur) {
          cur = want;
          if (want & 1u) fin[k.u] = 0;
        } else {
          cur = prev;
        }
      }
      dec = cur & 1u;
    }
    k.active = __shfl_sync(FULL, dec, 0) != 0;
  }
  return k;
}
// sk: the warp's lanes' sketches of the chunk (d0: what a clear sketch starts from).
template <int S, int MODE, bool BATCH, int RULE>
__device__ __forceinline__ void hub_close(const LpaArgs &a, Sketch<S> &sk, const HubChunk &k, uint32_t d0, int64_t local,
                                          int it, bool pickless, const uint32_t *vin, uint32_t *vout, uint8_t *fout,
                                          Counters &cnt, Phase ph) {
  const int lane = threadIdx.x & 31;
  sk_tree<S, RULE>(sk, 32);
  unsigned int last = 0;
  if (lane == 0) {
    if (k.active) {
      cnt.edges += (unsigned long long)(k.ce - k.cb);
#pragma unroll
      for (int i = 0; i < S; ++i) {
        a.sk_keys[local * S + i] = sk.k[i];
        a.sk_wts[local * S + i] = sk.w[i];
      }
    }
    __threadfence();
    last = atomicAdd(a.hub_arrive + k.h, 1u) == unsigned(k.nch - 1);
  }
  last = __shfl_sync(FULL, last, 0);
  if (!last) return;
  __threadfence();
  if (lane == 0) a.hub_arrive[k.h] = 0;
  const uint32_t d = vin[k.u];
  if (!k.active) {
    if (MODE != MODE_ASYNC && lane == 0) {
      vout[k.u] = d;
      if (ph.pull_out) fout[k.u] = 0;
    }
    return;
  }
  Sketch<S> acc;
  sk_clear<S, RULE>(acc, d0);
  for (int64_t jj = lane; jj < k.nch; jj += 32) {
    uint32_t bk[S];
    float bw[S];
#pragma unroll
    for (int i = 0; i < S; ++i) {
      bk[i] = __ldcg(a.sk_keys + (k.first + jj) * S + i);
      bw[i] = __ldcg(a.sk_wts + (k.first + jj) * S + i);
    }
    sk_merge<S, RULE>(acc, bk, bw);
  }
  sk_tree<S, RULE>(acc, 32);
  if (lane == 0) {
    uint32_t c;
    float w;
    choose<S, RULE>(a, acc, k.u - k.base, it, c, w);
    const bool moved = move_rule<S, RULE>(w, c, d, pickless);
    cnt.processed += 1;
    if constexpr (MODE == MODE_ASYNC) {
      if (moved) vout[k.u] = c;
    } else {
      vout[k.u] = moved ? c : d;
      if (ph.pull_out) fout[k.u] = moved ? 1 : 0;
    }
    if (moved) {
      cnt.changed += 1;
      cnt.moved_edges += (unsigned long long)(k.ee - k.eb);
      count_moves<BATCH>(a, k.gi, it);
      a.hub_moved[k.h] = it;
      atomicAdd(a.stats + STATS_STRIDE * it + STAT_HUBS_MOVED, 1ull);
    }
  }
}

template <int S, int MODE, class O, bool UNIT, bool BATCH, int RULE>
__device__ __forceinline__ void hub_item(const LpaArgs &a, const Regions &rg, const G_<O> &g, int64_t local, int it, bool pickless,
                                         const uint32_t *vin, uint32_t *vout, uint8_t *fin, uint8_t *fout,
                                         Counters &cnt, StageCtx &sc, Phase ph) {
  const int lane = threadIdx.x & 31;
  if constexpr (MODE == MODE_SYNC) {
    if (local != __ldg(a.hub_first + __ldg(a.chunk_hub + local))) return;
    const HubChunk k = hub_open<MODE, O, BATCH>(a, rg, g, local, it, fin, ph);
    const uint32_t d = vin[k.u];
    Sketch<S> sk;
    sk_clear<S, RULE>(sk, d);
    if (k.active) {   // the same on every lane
      if (exact_by_warp<S, UNIT>(k.ee - k.eb))
        exact_warp_scan<S, UNIT>(sk, k.u, k.eb, k.ee, a.rescan != 0, g.tgt, g.wt, vin, k.base);
      else
        exact_group_scan<S, UNIT>(sk, k.u, k.eb, k.ee, 32, 0, lane, S > 1 && a.rescan, g.tgt, g.wt, vin, k.base);
    }
    uint32_t c;
    float w;
    choose<S, RULE>(a, sk, k.u - k.base, it, c, w);
    const bool moved = k.active && move_rule<S, RULE>(w, c, d, pickless);
    if (lane == 0) {
      vout[k.u] = moved ? c : d;
      if (ph.pull_out) fout[k.u] = moved ? 1 : 0;
      if (k.active) { cnt.processed += 1; cnt.edges += (unsigned long long)(k.ee - k.eb); }
      if (moved) { cnt.changed += 1; cnt.moved_edges += (unsigned long long)(k.ee - k.eb); count_moves<BATCH>(a, k.gi, it); }
    }
    if (moved && !ph.pull_out) mark_item<S>(a, k.u, k.eb + lane, k.ee, 32, g.tgt, fout, k.base);
    return;
  } else {
    const HubChunk k = hub_open<MODE, O, BATCH>(a, rg, g, local, it, fin, ph);
    // Boyer-Moore under the GPU rules starts every partial vote from u's label
    const uint32_t d0 = (S == 1 && RULE == RULE_GPU) ? vin[k.u] : NONE;
    Sketch<S> sk;
    sk_clear<S, RULE>(sk, d0);
    if (sc.on)   // active is the same on every lane
      staged_scan<S, UNIT, RULE>(sk, sc, k.u, k.active ? k.cb : 0, k.active ? k.ce : 0, g.tgt, g.wt, vin, k.base,
                                 static_cast<RunState *>(a.rs), a.timeout_ns);
    else if (k.active)
      scan_range<S, UNIT, RULE>(sk, k.u, k.cb + lane, k.ce, 32, g.tgt, g.wt, vin, k.base);
    hub_close<S, MODE, BATCH, RULE>(a, sk, k, d0, local, it, pickless, vin, vout, fout, cnt, ph);
  }
}

// ---- wide items: 32 sketches scanned by a whole block, a thread for every slot -------------------
//
// A warp item scans 32 edge sequences (chains), one per lane. A chain cannot be split -- each edge meets
// the sketch the ones before it left -- so its warp's pace bounds the iteration: about 1000 cycles a step
// on a busy SM (measured; 2048 steps for a degree of 65536), and on graphs of a few million edges that is
// most of the iteration (R-MAT scale 20: 1.0 of 1.03 ms; the edges alone take 0.1 ms). Here the block's 256
// threads take the same 32 chains, S threads a chain and one slot each: a step is a shuffle, a compare and
// two votes instead of a pass over S slots, the S threads load S edges of the chain at once, and the next
// edges' labels are gathered meanwhile. The sketches go through shared memory to the block's first warp,
// which merges, chooses and moves exactly as for a warp item; marking is spread over the block. Bit for
// bit the same sketches. It costs more instructions per edge, so only chains too long for the graph are
// scanned this way (Regions::wide_len). Measured on B200, split runs, without -> with: R-MAT scale 12 ef 16
// 0.42 -> 0.31 ms, scale 16 1.5 -> 1.03 ms, scale 18 2.7 -> 2.3 ms, scale 20 10.9 -> 6.5 ms, scale 20 ef 32
// weighted 13.7 -> 9.6 ms.
template <int S>
struct WideShared {
  long long item;
  int64_t eb[32], ee[32];   // chain: edges eb, eb + st, ... < ee of vertex u
  uint32_t u[32], base[32];
  int st;
  unsigned live, moved;     // chains to scan; chains whose vertex moved
  uint32_t k[32 * S];
  float w[32 * S];
};
template <int S, int MODE>
__host__ __device__ constexpr bool has_wide() { return MODE == MODE_SPLIT && S > 1; }

// A function of its own: what the first warp of wide_items holds meanwhile is put away once a call, not spilled
// inside the loop (R-MAT scale 20 6.1 -> 5.7 ms, scale 20 ef 32 weighted 9.73 -> 9.49 ms, a small run without allocation
// 0.58 -> 0.56 ms).
template <int S, bool UNIT>
__device__ __noinline__ void scan_slots(WideShared<S> &ws, const uint32_t *tgt, const float *wt, const uint32_t *vin) {
  const int slot = threadIdx.x & (S - 1), shift = threadIdx.x & 31 & ~(S - 1), st = ws.st;
  const unsigned gm = ((1u << S) - 1u) << shift;   // the chain's S threads in a vote
  const int lane = threadIdx.x & 31;
  for (int c = threadIdx.x / S; c < 32; c += 256 / S) {   // the same trip count on every lane of a warp
    const uint32_t u = ws.u[c], base = ws.base[c];
    const int64_t e = ws.eb[c];
    const int len = (ws.live >> c) & 1u ? int((ws.ee[c] - e + st - 1) / st) : 0;
    const int most = __reduce_max_sync(FULL, len);
    const uint32_t *tp = tgt + e + int64_t(slot) * st;
    const float *wp = UNIT ? nullptr : wt + e + int64_t(slot) * st;
    const int64_t hop = int64_t(S) * st;
    uint32_t k = NONE, num = 0u, low = 0u;   // unit weights: the weight is num - low, low shared by the chain
    float w = 0.0f;
    // this thread's edge of the current S steps (its label gathered), and of the next S
    uint32_t t0 = slot < len ? base + ld_edge(tp) : u, t1 = S + slot < len ? base + ld_edge(tp + hop) : u;
    float w0 = slot < len ? edge_w<UNIT>(wp, 0) : 0.0f, w1 = S + slot < len ? edge_w<UNIT>(wp, hop) : 0.0f;
    uint32_t c0 = t0 != u ? ld_label(vin + t0) : NONE;
    for (int done = 0; done < most; done += S) {
      const uint32_t c1 = t1 != u ? ld_label(vin + t1) : NONE;
      const bool far = done + 2 * S + slot < len;
      const uint32_t t2 = far ? base + ld_edge(tp + 2 * hop) : u;
      const float w2 = far ? edge_w<UNIT>(wp, 2 * hop) : 0.0f;
      const unsigned has = __ballot_sync(FULL, t0 != u) >> shift;   // self-loops and ends take no step
#pragma unroll
      for (int i = 0; i < S; ++i) {
        const uint32_t cc = __shfl_sync(FULL, c0, i, S);
        const float x = UNIT ? 1.0f : __shfl_sync(FULL, w0, i, S);
        const bool on = (has >> i) & 1u;
        const bool hit = on && k == cc;
        // votes by every lane, outside any condition (both votes side by side measured 10-15% slower)
        const unsigned hits = __ballot_sync(FULL, hit) & gm;
        const bool miss = on && hits == 0u;
        const unsigned open = __ballot_sync(FULL, miss && (UNIT ? num == low : w == 0.0f)) & gm;
        // the last free slot: the highest of the chain's votes. A step waits for the one before it, so each
        // instruction from vote to key counts (with a search for the bit instead: R-MAT of 200 k vertices 2.02 -> 1.81 ms,
        // 1.5 M 4.89 -> 4.54 ms, scale 20 ef 32 weighted 9.49 -> 9.41 ms)
        const bool take = open >> lane == 1u;
        if constexpr (UNIT) {
          if (hit) num += 1u;
          if (take) { k = cc; num = low + 1u; }
          if (miss && open == 0u) low += 1u;
        } else {
          if (hit) w = __fadd_rn(w, x);
          if (take) { k = cc; w = x; }
          if (miss && open == 0u) w = fmaxf(__fsub_rn(w, x), 0.0f);
        }
      }
      t0 = t1; c0 = c1; w0 = w1; t1 = t2; w1 = w2;
      tp += hop;
      if constexpr (!UNIT) wp += hop;
    }
    ws.k[c * S + slot] = k;
    ws.w[c * S + slot] = UNIT ? float(num - low) : w;
  }
}

// Whether item `local` of region 0 or 1 is a wide one where only their longest are (!Regions::wide_all).
template <class O>
__device__ __forceinline__ bool long_item(const LpaArgs &a, const Regions &rg, const G_<O> &g, int r, int64_t local) {
  int64_t edges = a.hub_chunk;
  if (r != REG_HUB) {
    const uint32_t u = __ldg(a.order + rg.vbegin[r] + local);
    edges = int64_t(__ldg(g.off + u + 1)) - int64_t(__ldg(g.off + u));
  }
  return edges > 32 * int64_t(rg.wide_len);
}

// The iteration's wide items, taken by whole blocks from a counter of their own. A function of its own,
// not inlined: its registers would crowd the warp items' loops (inlined: lattice 2047x2049 1.16 -> 1.36 ms).
template <int S, int MODE, class O, bool UNIT, bool BATCH>
__device__ __noinline__ Counters wide_items(const LpaArgs &a, const Regions &rg, int it, bool pickless,
                                            const uint32_t *vin, uint32_t *vout, uint8_t *fin, uint8_t *fout, Phase ph,
                                            WideShared<S> &ws) {
  const G_<O> g{static_cast<const O *>(a.off), a.tgt, a.wt};
  const int lane = threadIdx.x & 31;
  Counters cnt{0, 0, 0, 0};
  for (int64_t taken = 0; taken <= rg.wide_items; ++taken) {
    __syncthreads();   // ws of the item before is no longer read
    if (threadIdx.x == 0) ws.item = (long long)atomicAdd(a.stats + STATS_STRIDE * it + STAT_WIDE, 1ull);
    __syncthreads();
    const int64_t item = ws.item;
    if (item >= rg.wide_items) break;
    int r = 0;
    while (r < REG_LANE && item >= rg.ibegin[r + 1]) ++r;
    const int64_t local = item - rg.ibegin[r];   // region 6: a batch of 32 vertices
    if (!rg.wide_all && !long_item(a, rg, g, r, local)) continue;
    GroupVertex v;
    HubChunk k;
    if (threadIdx.x < 32) {
      const int G = region_group(r), s = lane & (G - 1);
      if (r == REG_HUB) {
        k = hub_open<MODE, O, BATCH>(a, rg, g, local, it, fin, ph);
        ws.u[lane] = k.u; ws.base[lane] = k.base; ws.eb[lane] = k.cb + lane; ws.ee[lane] = k.ce;
      } else {
        v = group_open<MODE, O, BATCH>(a, rg, g, r, local, it, vin, fin, ph);
        ws.u[lane] = v.u; ws.base[lane] = v.base; ws.eb[lane] = v.eb + s; ws.ee[lane] = v.ee;
      }
      const unsigned live = __ballot_sync(FULL, r == REG_HUB ? k.active : v.active);
      if (lane == 0) { ws.st = G; ws.live = live; ws.moved = 0u; }
    }
    __syncthreads();
    if (ws.live) scan_slots<S, UNIT>(ws, g.tgt, g.wt, vin);
    __syncthreads();
    if (threadIdx.x < 32) {
      Sketch<S> sk;
      sk_clear<S>(sk);
      if ((ws.live >> lane) & 1u) {
#pragma unroll
        for (int i = 0; i < S; ++i) { sk.k[i] = ws.k[lane * S + i]; sk.w[i] = ws.w[lane * S + i]; }
      }
      if (r == REG_HUB) {
        hub_close<S, MODE, BATCH, RULE_CPU>(a, sk, k, NONE, local, it, pickless, vin, vout, fout, cnt, ph);
      } else {
        const unsigned moved = __ballot_sync(FULL, group_close<S, MODE, BATCH, RULE_CPU>(a, sk, v, r, it, pickless, vout, fin, fout, cnt, ph));
        if (lane == 0) ws.moved = moved;
      }
    }
    if (ph.nomark || ph.pull_out || r == REG_HUB) continue;
    __syncthreads();
    const int c = threadIdx.x >> 3;   // eight threads mark a chain's edges
    if ((ws.moved >> c) & 1u)
      mark_item<S>(a, ws.u[c], ws.eb[c] + int64_t(threadIdx.x & 7) * ws.st, ws.ee[c], 8 * ws.st, g.tgt, fout, ws.base[c]);
  }
  return cnt;
}

// Whether iteration it + 1 records its movers for the one after it: when the vertices that moved in
// iteration it hold a quarter of the edges or more (the first iteration always does, pull_for), and no
// list of region 1 that one warp would read to its end in vain is so long as to outlast the iteration: L
// edges take L / 256 round trips of about half a microsecond, a balanced iteration m / 250 G/s, so L up to
// m / 512. (Split vertices are searched by all their chunks' warps, hub_pull; the lists of smaller groups
// are 16 * lane_max edges at most: the same rule for them made 4096 settled edges 0.73 -> 0.44 ms over 30
// iterations, and the exact mode's kernel 2% slower.) Measured on B200, 30 iterations of a settled vertex of
// 60000 edges beside vertices that move in pairs: never pulled 1.22 ms, pulled whatever the list 19.6 ms,
// this 1.22 ms. Every block reads the same counter after the barrier, so all agree; the choice changes what
// the flags hold, not the result.
__device__ __forceinline__ bool pulls_next(const LpaArgs &a, int it, bool can_pull) {
  return can_pull && it + 2 < a.iters &&   // negative: LONG_IDLE
         (long long)__ldcg(a.stats + STATS_STRIDE * it + STAT_MOVED_EDGES) >= (a.m + 3) / 4;
}

// WIDE: the launch has wide items. Launches without any take a kernel that does not hold their code and
// shared memory (one kernel for both: R-MAT scale 24 ef 16 split 50.7 -> 52.4 ms, lattice 2047x2049 1.16 -> 1.24
// ms). Asynchronous runs take this kernel only where their result does not show its pace (rak_lpa_async.cuh).
// RULE: the rule set of the work items. Only split runs know both, each with a kernel of its own: the exact mode
// follows the CPU rules, and wide items and asynchronous runs that come here do.
template <int S, int MODE, class O, bool UNIT, bool BATCH, bool WIDE, int RULE>
__global__ void __launch_bounds__(256, RAK_MIN_BLOCKS) lpa_run(const __grid_constant__ LpaArgs a) {
  const G_<O> g{static_cast<const O *>(a.off), a.tgt, a.wt};
  RunState *rs = static_cast<RunState *>(a.rs);
  const int lane = threadIdx.x & 31;
  const int64_t gw = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  __shared__ unsigned long long blk[4];
  __shared__ Regions rg;  // copied once: indexed by region at run time
  __shared__ uint32_t lq[8][64];  // per-warp queue of active one-lane vertices
  __shared__ WideShared<WIDE ? S : 1> ws;
  if (threadIdx.x == 0) rg = a.rg;
  // staged edge tiles (not in the exact synchronous mode, which shuffles edges in order instead)
  StageCtx sc{};
  if constexpr (MODE != MODE_SYNC && RAK_STAGE) {
    extern __shared__ __align__(128) unsigned char lpa_dsm[];
    const int w = threadIdx.x >> 5;
    constexpr size_t tbytes = size_t(LPA_WARPS) * STG_STAGES * STG_TILE * 4;
    sc.t = reinterpret_cast<uint32_t *>(lpa_dsm) + size_t(w) * STG_STAGES * STG_TILE;
    sc.w = UNIT ? nullptr : reinterpret_cast<float *>(lpa_dsm + tbytes) + size_t(w) * STG_STAGES * STG_TILE;
    sc.bar = smem_u32(lpa_dsm + tbytes * (UNIT ? 1 : 2)) + 8u * uint32_t(w * STG_STAGES);
    sc.phase = 0;
    // the tiles and their mbarriers exist only in launches given the dynamic shared memory for them
    // (lpa_dynamic_smem); the launch's actual size is checked before any of it is touched
    uint32_t dyn_bytes;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn_bytes));
    const bool have = a.stage && dyn_bytes >= stage_bytes(UNIT);
    // targets and weights must share their 16-byte alignment (one copy range serves both)
    sc.on = have && (UNIT || ((reinterpret_cast<uintptr_t>(a.tgt) ^ reinterpret_cast<uintptr_t>(a.wt)) & 15u) == 0);
    if (have) {
      if (lane < STG_STAGES) mbar_init(sc.bar + 8u * uint32_t(lane), 1);
      fence_mbar_init();
      __syncwarp();
    }
  }
  unsigned int epoch = 0;
  // Dense iterations (asynchronous single-graph runs with LpaArgs::dense_moved_edges > 0): when
  // the vertices that moved in the previous iteration hold at least that many edges, this
  // iteration's moves mark no neighbours and the next iteration processes every vertex. Such a
  // frontier would hold nearly every vertex anyway, and the marking it saves is a re-read of each
  // moved vertex's edges plus a random flag access per edge. Decided from the previous iteration's
  // counter, which every block reads after the barrier, so all blocks agree.
  Phase ph{false, false, false, false};
  const bool can_pull = MODE != MODE_ASYNC && a.pull != 0 && __ldcg(&rs->asym) == 0ull && __ldcg(&rs->oneway) == 0u;
  bool next_out = false;   // whether the next iteration records its movers (Phase::pull_out)
  for (int it = 0; it < a.iters; ++it) {
    if (threadIdx.x < 4) blk[threadIdx.x] = 0;
    if constexpr (MODE == MODE_ASYNC && !BATCH) {
      ph.all = ph.nomark;
      ph.nomark = a.dense_moved_edges > 0 && it > 0 &&
                  __ldcg(a.stats + STATS_STRIDE * (it - 1) + STAT_MOVED_EDGES) >= a.dense_moved_edges;
      if (blockIdx.x == 0 && threadIdx.x == 0)
        a.stats[STATS_STRIDE * it + STAT_PHASE] = (ph.all ? 2ull : 0ull) | (ph.nomark ? 1ull : 0ull);
    }
    if constexpr (MODE != MODE_ASYNC) {
      ph.pull_in = ph.pull_out;
      ph.pull_out = it == 0 ? can_pull : next_out;
    }
    __syncthreads();
    const int l = a.start_iter + it;
    const bool pickless = a.pickless_step > 0 && l % a.pickless_step == 0;
    const bool odd = MODE != MODE_ASYNC && (it & 1);
    const uint32_t *vin = odd ? a.vcom1 : a.vcom0;
    uint32_t *vout = MODE == MODE_ASYNC ? a.vcom0 : (odd ? a.vcom0 : a.vcom1);
    uint8_t *fin = odd ? a.aff1 : a.aff0;
    uint8_t *fout = MODE == MODE_ASYNC ? a.aff0 : (odd ? a.aff0 : a.aff1);
    Counters cnt{0, 0, 0, 0};
    const int64_t total = rg.ibegin[NREG];
    unsigned long long *work = a.stats + STATS_STRIDE * it + STAT_WORK;
    uint32_t *q = lq[threadIdx.x >> 5];
    int qn = 0;
    int64_t item0 = 0;     // the first warp item: after the wide ones where these are all of the first
    bool skip_long = false;
    if constexpr (WIDE) {
      cnt = wide_items<S, MODE, O, UNIT, BATCH>(a, rg, it, pickless, vin, vout, fin, fout, ph, ws);
      if (rg.wide_all) item0 = rg.ibegin[REG_LANE] + rg.wide_lanes / rg.lane_item;
      else skip_long = true;
    }
    for (;;) {
      unsigned long long got = 0;
      if (lane == 0) got = atomicAdd(work, 1ull);
      const int64_t item = item0 + int64_t(__shfl_sync(FULL, got, 0));
      if (item >= total) break;
      int r = 0;
      while (item >= rg.ibegin[r + 1]) ++r;
      const int64_t local = item - rg.ibegin[r];
      if (WIDE && skip_long && r <= 1 && long_item(a, rg, g, r, local)) continue;
      if (r == REG_LANE) {
        for (int64_t sb = 0; sb < rg.lane_item; ++sb) {
          const int64_t sub = local * rg.lane_item + sb;
          if (sub * 32 >= rg.vcount[REG_LANE]) break;
          qn = lane_collect<MODE, O, BATCH>(a, rg, g, sub, vin, vout, fin, fout, q, qn, ph);
          if (qn >= 32) {
            lane_batch<S, MODE, O, UNIT, BATCH, RULE>(a, g, q, 32, it, pickless, vin, vout, fin, fout, cnt, ph);
            __syncwarp();
            if (lane < qn - 32) q[lane] = q[32 + lane];
            __syncwarp();
            qn -= 32;
          }
        }
      } else if (r == REG_HUB) {
        hub_item<S, MODE, O, UNIT, BATCH, RULE>(a, rg, g, local, it, pickless, vin, vout, fin, fout, cnt, sc, ph);
      } else {
        group_item<S, MODE, O, UNIT, BATCH, RULE>(a, rg, g, r, local, it, pickless, vin, vout, fin, fout, cnt, sc, ph);
      }
    }
    if (qn > 0) lane_batch<S, MODE, O, UNIT, BATCH, RULE>(a, g, q, qn, it, pickless, vin, vout, fin, fout, cnt, ph);
    __syncwarp();
    const unsigned long long ch = warp_sum((unsigned long long)cnt.changed);
    const unsigned long long ed = warp_sum(cnt.edges);
    const unsigned long long pr = warp_sum((unsigned long long)cnt.processed);
    const unsigned long long me = warp_sum(cnt.moved_edges);
    if (lane == 0) {
      if (ch) atomicAdd(&blk[0], ch);
      if (ed) atomicAdd(&blk[1], ed);
      if (pr) atomicAdd(&blk[2], pr);
      if (me) atomicAdd(&blk[3], me);
    }
    __syncthreads();
    if (threadIdx.x < 4 && blk[threadIdx.x]) {
      const int slot = threadIdx.x == 3 ? STAT_MOVED_EDGES : int(threadIdx.x);
      atomicAdd(a.stats + STATS_STRIDE * it + slot, blk[threadIdx.x]);
    }
    if (!grid_barrier(rs, ++epoch, a.timeout_ns)) return;
    const unsigned long long changed = __ldcg(a.stats + STATS_STRIDE * it + STAT_CHANGED);
    const bool test = !pickless || a.check_on_pickless;
    // Batches finish when no graph is still running (decided in the per-graph phase below).
    const bool done = !BATCH && (it + 1 >= a.iters || (test && double(changed) / double(a.n) <= a.tolerance));
    // The synchronous split mode completes the next flags even on the last iteration, so a
    // single step returns them whole.
    if (MODE != MODE_SYNC && !ph.nomark && !ph.pull_out && (!done || MODE == MODE_SPLIT) && a.nchunks > 0 &&
        __ldcg(a.stats + STATS_STRIDE * it + STAT_HUBS_MOVED) > 0) {
      // Second phase: neighbours of split vertices that moved this iteration.
      for (int64_t i = gw; i < a.nchunks; i += nw) {
        const uint32_t h = __ldg(a.chunk_hub + i);
        if (__ldcg(a.hub_moved + h) != it) continue;
        const uint32_t u = __ldg(a.order + rg.vbegin[REG_HUB] + h);
        const int64_t eb = int64_t(__ldg(g.off + u)), ee = int64_t(__ldg(g.off + u + 1));
        const int64_t j = i - __ldg(a.hub_first + h);
        const int64_t cb = eb + j * a.hub_chunk, ce = cb + a.hub_chunk < ee ? cb + a.hub_chunk : ee;
        uint32_t gi, base;
        graph_of<BATCH>(a, u, gi, base);
        mark_range<true>(u, cb + lane, ce, 32, g.tgt, fout, base);
      }
    }
    if constexpr (BATCH) {
      // Per-graph convergence, each graph by one thread: the rule of the single-graph loop applied
      // to the graph's own changed count and vertex count; also clears the graph's counter for the
      // iteration after next.
      const int64_t tid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, nt = int64_t(gridDim.x) * blockDim.x;
      unsigned int run = 0;
      for (int64_t gi = tid; gi < a.ngraphs; gi += nt) {
        if (a.gdone[gi]) continue;
        const int64_t ng = a.vbase[gi + 1] - a.vbase[gi];
        const unsigned long long c = __ldcg(a.gchanged + int64_t(it & 1) * a.ngraphs + gi);
        if (ng == 0 || it + 1 >= a.iters || (test && double(c) / double(ng) <= a.tolerance)) {
          a.gdone[gi] = 1;
          a.giters[gi] = it + 1;
        } else {
          ++run;
        }
        a.gchanged[int64_t((it + 1) & 1) * a.ngraphs + gi] = 0ull;
      }
      run = warp_sum(run);
      if (lane == 0 && run) atomicAdd(a.running + it, run);
      if constexpr (MODE != MODE_ASYNC) {
        next_out = pulls_next(a, it, can_pull);
        if (ph.pull_out && a.nchunks > 0) hub_pull<O, BATCH>(a, rg, fout, it + 1);
        uint4 *f4 = reinterpret_cast<uint4 *>(fin);
        const int64_t n16 = a.n >> 4;
        for (int64_t i = tid; i < n16; i += nt) f4[i] = make_uint4(0, 0, 0, 0);
        for (int64_t i = (n16 << 4) + tid; i < a.n; i += nt) fin[i] = 0;
      }
      if (!grid_barrier(rs, ++epoch, a.timeout_ns)) return;
      if (__ldcg(a.running + it) == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) rs->iterations = unsigned(it + 1);
        return;
      }
      continue;
    }
    if (done) {
      if (blockIdx.x == 0 && threadIdx.x == 0) rs->iterations = unsigned(it + 1);
      return;
    }
    if constexpr (MODE != MODE_ASYNC) {
      next_out = pulls_next(a, it, can_pull);
      // Every vertex with an edge writes its flag in an iteration that records movers: nothing to clear,
      // and nothing after the barrier above to wait for unless this one marked split vertices' neighbours or
      // the next one needs to know which of them have a moved neighbour.
      const bool clear = !(next_out && ph.pull_out);
      if (ph.pull_out && a.nchunks > 0) hub_pull<O, BATCH>(a, rg, fout, it + 1);
      else if (!clear) continue;
      // The flags just read become next iteration's output: clear them.
      if (clear) {
        const int64_t tid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, nt = int64_t(gridDim.x) * blockDim.x;
        uint4 *f4 = reinterpret_cast<uint4 *>(fin);
        const int64_t n16 = a.n >> 4;
        for (int64_t i = tid; i < n16; i += nt) f4[i] = make_uint4(0, 0, 0, 0);
        for (int64_t i = (n16 << 4) + tid; i < a.n; i += nt) fin[i] = 0;
      }
      if (!grid_barrier(rs, ++epoch, a.timeout_ns)) return;
    }
  }
}

// Dynamic shared memory of an lpa_run launch: the staged edge tiles, when the launch stages edges.
// Without staging the launch takes none, which leaves the SM's L1 cache its full size for the
// label gathers (shared memory and L1 share the SM's 256 KB).
inline size_t lpa_dynamic_smem(int mode, bool unit, bool stage) {
  return (mode != MODE_SYNC && RAK_STAGE && stage) ? stage_bytes(unit) : 0;
}

// The kernel instantiation for a launch and its resident blocks per SM, cached per (function,
// device). The first query of an instantiation loads its module (CUDA loads modules lazily, which
// can take a millisecond), so runs resolve before their timed region (prepare_lpa).
template <int S>
cudaError_t resolve_lpa_slots(int mode, bool off64, bool unit, bool batch, bool stage, int alt, const void **fn_out,
                              int *per_sm_out) {
  const void *fn = nullptr;
#define RAK_PICK(M, O, U, B)                                                          \
  if (mode == M && off64 == (sizeof(O) == 8) && unit == U && batch == B) {           \
    if constexpr (M == MODE_ASYNC) {                                                  \
      fn = async_kernel<S>(off64, unit, batch);                                        \
      if constexpr (S > 1 && !B) {                                                    \
        if (alt) fn = reinterpret_cast<const void *>(&lpa_run<S, M, O, U, B, false, RULE_CPU>); \
      }                                                                               \
    } else {                                                                          \
      fn = reinterpret_cast<const void *>(&lpa_run<S, M, O, U, B, false, RULE_CPU>);  \
      if constexpr (M == MODE_SPLIT) {                                                \
        if (alt == ALT_GPU_RULE) fn = reinterpret_cast<const void *>(&lpa_run<S, M, O, U, B, false, RULE_GPU>); \
      }                                                                               \
      if constexpr (has_wide<S, M>()) {                                               \
        if (alt == ALT_FAST) fn = reinterpret_cast<const void *>(&lpa_run<S, M, O, U, B, true, RULE_CPU>); \
      }                                                                               \
    }                                                                                 \
  }
#define RAK_PICK_MODE(M)                                                             \
  RAK_PICK(M, int32_t, false, false) RAK_PICK(M, int32_t, true, false)                \
  RAK_PICK(M, int64_t, false, false) RAK_PICK(M, int64_t, true, false)                \
  RAK_PICK(M, int64_t, false, true) RAK_PICK(M, int64_t, true, true)
  RAK_PICK_MODE(MODE_ASYNC) RAK_PICK_MODE(MODE_SYNC) RAK_PICK_MODE(MODE_SPLIT)
#undef RAK_PICK_MODE
#undef RAK_PICK
  if (!fn) return cudaErrorInvalidValue;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, int> cache;   // (kernel, device * 2 + stage)
  {
    std::lock_guard<std::mutex> lk(mu);
    const auto it = cache.find({fn, dev * 2 + (stage ? 1 : 0)});
    if (it != cache.end()) {
      *fn_out = fn;
      *per_sm_out = it->second;
      return cudaSuccess;
    }
  }
  int per_sm = 0;
  const size_t dyn = lpa_dynamic_smem(mode, unit, stage);
  if (dyn > 0 && (e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(dyn))) != cudaSuccess)
    return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 256, dyn)) != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  std::lock_guard<std::mutex> lk(mu);
  cache[{fn, dev * 2 + (stage ? 1 : 0)}] = per_sm;
  *fn_out = fn;
  *per_sm_out = per_sm;
  return cudaSuccess;
}

template <int S>
cudaError_t launch_lpa_slots(const LpaArgs &a, int mode, bool off64, bool batch, cudaStream_t st, int *grid_out) {
  const void *fn = nullptr;
  int per_sm = 0, dev = 0, sms = 0;
  cudaError_t e = resolve_lpa_slots<S>(mode, off64, a.wt == nullptr, batch, a.stage != 0, a.alt, &fn, &per_sm);
  if (e != cudaSuccess) return e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  const int64_t warps_needed = a.rg.ibegin[NREG] > 0 ? a.rg.ibegin[NREG] : 1;
  int64_t grid = int64_t(per_sm) * sms;
  int64_t want = (warps_needed + 7) / 8;
  if (mode == MODE_SPLIT && a.alt == ALT_FAST && a.rg.wide_items > want) want = a.rg.wide_items;   // a block each
  if (want < grid) grid = want;
  if (a.grid_cap > 0 && grid > a.grid_cap) grid = a.grid_cap;
  if (grid < 1) grid = 1;
  if (grid_out) *grid_out = int(grid);
  // Cooperative attribute through cudaLaunchKernelEx: co-residency is guaranteed (the grid
  // barrier relies on it) and the launch can be captured into a CUDA graph.
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = lpa_dynamic_smem(mode, a.wt == nullptr, a.stage != 0);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void *args[] = {const_cast<LpaArgs *>(&a)};
  return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace rak
