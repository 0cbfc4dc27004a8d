// rak_lpa_async.cuh -- the persistent kernel of asynchronous runs whose result shows the kernel's pace.
//
// Asynchronous runs read labels that other warps change meanwhile, so the pace of the scan is part of their
// result: on lattices, planted partitions and with Boyer-Moore, kernels with the same reads and the same
// rules at another pace ended at another modularity, by several times what runs of one kernel differ by --
// even where only the order of instructions had changed (eight lattices of 2047x2049: 0.6592 +- 0.0002
// against 0.6569 to 0.6604; SBM of 300 k vertices 0.1043 +- 0.0001 against 0.1032 to 0.1051). These runs keep
// their first kernel, with its scan, accumulate and barrier. Runs with 8 slots on large skewed graphs (async_fast,
// with the measurements) take the faster lpa_run (rak_lpa.cuh): there the pace does not show.
//
// Work items, phases and rules as described in rak_lpa.cuh. Compiled in units of its own, and none of the library's
// with a split compilation (--split-compile), which orders the instructions differently: here it shows in the
// result as above.
#pragma once
#include "rak_lpa.cuh"

namespace rak {

// Sequential sketch of edges e, e+st, ... < ee of u (self-loops skipped), in edge order, in batches of four:
// the next batch's targets and weights are loaded while the current batch's labels are gathered and
// accumulated.
template <int S, bool UNIT, int RULE>
__device__ __forceinline__ void async_scan_range(Sketch<S> &sk, uint32_t u, int64_t e, int64_t ee, int st,
                                           const uint32_t *tgt, const float *wt, const uint32_t *vin,
                                           uint32_t base) {
  constexpr int B = 4;
  uint32_t t[B];
  float w[B];
#pragma unroll
  for (int j = 0; j < B; ++j) {
    const int64_t x = e + int64_t(j) * st;
    t[j] = x < ee ? base + ld_edge(tgt + x) : u;
    w[j] = x < ee ? edge_w<UNIT>(wt, x) : 0.0f;
  }
  while (e < ee) {
    uint32_t c[B];
#pragma unroll
    for (int j = 0; j < B; ++j) c[j] = ld_label(vin + t[j]);
    const int64_t en = e + int64_t(B) * st;
    uint32_t t2[B];
    float w2[B];
#pragma unroll
    for (int j = 0; j < B; ++j) {
      const int64_t x = en + int64_t(j) * st;
      t2[j] = x < ee ? base + ld_edge(tgt + x) : u;
      w2[j] = x < ee ? edge_w<UNIT>(wt, x) : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < B; ++j)
      if (t[j] != u) sk_acc<S, RULE>(sk, c[j], w[j]);
#pragma unroll
    for (int j = 0; j < B; ++j) { t[j] = t2[j]; w[j] = w2[j]; }
    e = en;
  }
}

template <int S, bool UNIT, int RULE>
__device__ __forceinline__ void async_scan_lane(Sketch<S> &sk, uint32_t u, int64_t e, int64_t ee, const uint32_t *tgt,
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
      if (t[j] != u) sk_acc<S, RULE>(sk, c[j], UNIT ? 1.0f : w[j]);
  }
}

// Region 6: one lane per vertex. Items are collected into a per-warp queue of active vertices
// (inactive ones are settled at once), and the queue is processed 32 vertices at a time so every
// lane has work; region 6 is sorted by degree, so a batch holds vertices of similar degree.
template <int S, class O, bool UNIT, bool BATCH>
__device__ __forceinline__ int async_lane_collect(const LpaArgs &a, const Regions &rg, int64_t local, const uint32_t *vin,
                                            uint32_t *vout, const uint8_t *fin, uint32_t *q, int qn, Phase ph) {
  const int lane = threadIdx.x & 31;
  const int64_t idx = local * 32 + lane;
  bool act = false;
  uint32_t u = 0;
  if (idx < rg.vcount[REG_LANE]) {
    u = __ldg(a.order + rg.vbegin[REG_LANE] + idx);
    uint32_t gi, base;
    act = (ph.all || fin[u] != 0) && !graph_of<BATCH>(a, u, gi, base);
  }
  const unsigned m = __ballot_sync(FULL, act);
  if (act) q[qn + __popc(m & ((1u << lane) - 1u))] = u;
  __syncwarp();
  return qn + __popc(m);
}

template <int S, class O, bool UNIT, bool BATCH, int RULE>
__device__ __forceinline__ void async_lane_batch(const LpaArgs &a, const G_<O> &g, const uint32_t *q, int count,
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
  if (vec) async_scan_lane<S, UNIT, RULE>(sk, u, eb, ee, g.tgt, g.wt, vin, base);
  else async_scan_range<S, UNIT, RULE>(sk, u, eb, ee, 1, g.tgt, g.wt, vin, base);
  uint32_t c;
  float w;
  choose<S, RULE>(a, sk, u - base, it, c, w);
  const bool moved = move_rule<S, RULE>(w, c, d, pickless);
  cnt.processed += 1;
  cnt.edges += (unsigned long long)(ee - eb);
  fin[u] = 0;
  if (moved) vout[u] = c;
  if (moved) {
    cnt.changed += 1;
    cnt.moved_edges += (unsigned long long)(ee - eb);
    count_move<BATCH>(a, gi, it);
    if (ph.nomark) return;
    if (!vec) mark_item<S>(a, u, eb, ee, 1, g.tgt, fout, base);
    else if (mark_tested<S>(a)) mark_lane<true>(u, eb, ee, g.tgt, fout, base);
    else mark_lane<false>(u, eb, ee, g.tgt, fout, base);
  }
}

// Regions 1..5: aligned groups of G lanes per vertex.
template <int S, class O, bool UNIT, bool BATCH, int RULE>
__device__ __forceinline__ void async_group_item(const LpaArgs &a, const Regions &rg, const G_<O> &g, int r, int64_t local,
                                           int it, bool pickless, const uint32_t *vin, uint32_t *vout,
                                           uint8_t *fin, uint8_t *fout, Counters &cnt, StageCtx &sc, Phase ph) {
  const int G = region_group(r);
  const int lane = threadIdx.x & 31, grp = lane / G, s = lane & (G - 1);
  const int64_t idx = local * (32 / G) + grp;
  const bool valid = idx < rg.vcount[r];
  uint32_t u = 0, d = 0, gi = 0, base = 0;
  int64_t eb = 0, ee = 0;
  bool active = false;
  if (valid) {
    u = __ldg(a.order + rg.vbegin[r] + idx);
    d = vin[u];
    active = (ph.all || fin[u] != 0) && !graph_of<BATCH>(a, u, gi, base);
    if (active) { eb = int64_t(__ldg(g.off + u)); ee = int64_t(__ldg(g.off + u + 1)); }
  }
  Sketch<S> sk;
  sk_clear<S, RULE>(sk, d);
  if (sc.on && G == 32)   // one vertex per warp: the warp's range is uniform
    staged_scan<S, UNIT, RULE>(sk, sc, u, active ? eb : 0, active ? ee : 0, g.tgt, g.wt, vin, base,
                               static_cast<RunState *>(a.rs), a.timeout_ns);
  else if (active)
    async_scan_range<S, UNIT, RULE>(sk, u, eb + s, ee, G, g.tgt, g.wt, vin, base);
  sk_tree<S, RULE>(sk, G);
  uint32_t c;
  float w;
  choose<S, RULE>(a, sk, u - base, it, c, w);
  bool moved = active && move_rule<S, RULE>(w, c, d, pickless);
  moved = __shfl_sync(FULL, moved, grp * G);
  if (s == 0 && valid) {
    if (active) { cnt.processed += 1; cnt.edges += (unsigned long long)(ee - eb); }
    if (active) fin[u] = 0;
    if (moved) vout[u] = c;
    if (moved) { cnt.changed += 1; cnt.moved_edges += (unsigned long long)(ee - eb); count_move<BATCH>(a, gi, it); }
  }
  if (moved && !ph.nomark) mark_item<S>(a, u, eb + s, ee, G, g.tgt, fout, base);
}

// Region 0: one chunk of a split vertex per item. Each chunk's warp builds a partial sketch
// (lane-strided, tree-merged), stores it, and the last chunk to arrive merges all partial sketches
// in a fixed order and makes the move; its neighbours are marked in a second phase after the
// iteration's barrier.
template <int S, class O, bool UNIT, bool BATCH, int RULE>
__device__ __forceinline__ void async_hub_item(const LpaArgs &a, const Regions &rg, const G_<O> &g, int64_t local, int it, bool pickless,
                                         const uint32_t *vin, uint32_t *vout, uint8_t *fin, uint8_t *fout,
                                         Counters &cnt, StageCtx &sc, Phase ph) {
  const int lane = threadIdx.x & 31;
  const uint32_t h = __ldg(a.chunk_hub + local);
  const int64_t first = __ldg(a.hub_first + h), nch = __ldg(a.hub_first + h + 1) - first, j = local - first;
  const uint32_t u = __ldg(a.order + rg.vbegin[REG_HUB] + h);
  const int64_t eb = int64_t(__ldg(g.off + u)), ee = int64_t(__ldg(g.off + u + 1));
  uint32_t gi, base;
  const bool gfin = graph_of<BATCH>(a, u, gi, base);  // stable within an iteration
  bool active;
  if (gfin) {
    active = false;
  } else {
    // All chunks of u agree on whether u is processed this iteration: the first chunk to get
    // here decides from u's flag (and clears it); the others read the decision.
    unsigned int dec = 0;
    if (lane == 0) {
      const unsigned int tag = unsigned(it + 1);
      unsigned int cur = *(volatile unsigned int *)(a.hub_claim + h);
      if ((cur >> 1) != tag) {
        const unsigned int want = (tag << 1) | (ph.all || *(volatile uint8_t *)(fin + u) ? 1u : 0u);
        const unsigned int prev = atomicCAS(a.hub_claim + h, cur, want);
        if (prev == cur) {
          cur = want;
          if (want & 1u) fin[u] = 0;
        } else {
          cur = prev;
        }
      }
      dec = cur & 1u;
    }
    active = __shfl_sync(FULL, dec, 0) != 0;
  }
  // Boyer-Moore under the GPU rules starts every partial vote from u's label
  const uint32_t d0 = (S == 1 && RULE == RULE_GPU) ? vin[u] : NONE;
  Sketch<S> sk;
  sk_clear<S, RULE>(sk, d0);
  const int64_t cb = eb + j * a.hub_chunk, ce = cb + a.hub_chunk < ee ? cb + a.hub_chunk : ee;
  if (sc.on)   // active is the same on every lane
    staged_scan<S, UNIT, RULE>(sk, sc, u, active ? cb : 0, active ? ce : 0, g.tgt, g.wt, vin, base,
                               static_cast<RunState *>(a.rs), a.timeout_ns);
  else if (active)
    async_scan_range<S, UNIT, RULE>(sk, u, cb + lane, ce, 32, g.tgt, g.wt, vin, base);
  sk_tree<S, RULE>(sk, 32);
  unsigned int last = 0;
  if (lane == 0) {
    if (active) {
      cnt.edges += (unsigned long long)(ce - cb);
#pragma unroll
      for (int i = 0; i < S; ++i) {
        a.sk_keys[local * S + i] = sk.k[i];
        a.sk_wts[local * S + i] = sk.w[i];
      }
    }
    __threadfence();
    last = atomicAdd(a.hub_arrive + h, 1u) == unsigned(nch - 1);
  }
  last = __shfl_sync(FULL, last, 0);
  if (!last) return;
  __threadfence();
  if (lane == 0) a.hub_arrive[h] = 0;
  const uint32_t d = vin[u];
  if (!active) return;
  Sketch<S> acc;
  sk_clear<S, RULE>(acc, d0);
  for (int64_t jj = lane; jj < nch; jj += 32) {
    uint32_t bk[S];
    float bw[S];
#pragma unroll
    for (int i = 0; i < S; ++i) {
      bk[i] = __ldcg(a.sk_keys + (first + jj) * S + i);
      bw[i] = __ldcg(a.sk_wts + (first + jj) * S + i);
    }
    sk_merge<S, RULE>(acc, bk, bw);
  }
  sk_tree<S, RULE>(acc, 32);
  if (lane == 0) {
    uint32_t c;
    float w;
    choose<S, RULE>(a, acc, u - base, it, c, w);
    const bool moved = move_rule<S, RULE>(w, c, d, pickless);
    cnt.processed += 1;
    if (moved) vout[u] = c;
    if (moved) {
      cnt.changed += 1;
      cnt.moved_edges += (unsigned long long)(ee - eb);
      count_move<BATCH>(a, gi, it);
      a.hub_moved[h] = it;
      atomicAdd(a.stats + STATS_STRIDE * it + STAT_HUBS_MOVED, 1ull);
    }
  }
}

#define RAK_ASYNC_BY_RULE(F, ARGS)                                   \
  do {                                                              \
    if (a.gpu_rule) F<S, O, UNIT, BATCH, RULE_GPU> ARGS;             \
    else F<S, O, UNIT, BATCH, RULE_CPU_ASYNC> ARGS;                  \
  } while (0)

template <int S, class O, bool UNIT, bool BATCH>
__global__ void __launch_bounds__(256, RAK_MIN_BLOCKS) lpa_run_async(const LpaArgs a) {
  const G_<O> g{static_cast<const O *>(a.off), a.tgt, a.wt};
  RunState *rs = static_cast<RunState *>(a.rs);
  const int lane = threadIdx.x & 31;
  const int64_t gw = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = (int64_t(gridDim.x) * blockDim.x) >> 5;
  __shared__ unsigned long long blk[4];
  __shared__ Regions rg;  // copied once: indexed by region at run time
  __shared__ uint32_t lq[8][64];  // per-warp queue of active one-lane vertices
  if (threadIdx.x == 0) rg = a.rg;
  // staged edge tiles (not in the exact synchronous mode, which shuffles edges in order instead)
  StageCtx sc{};
  if constexpr (RAK_STAGE) {
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
  for (int it = 0; it < a.iters; ++it) {
    if (threadIdx.x < 4) blk[threadIdx.x] = 0;
    if constexpr (!BATCH) {
      ph.all = ph.nomark;
      ph.nomark = a.dense_moved_edges > 0 && it > 0 &&
                  __ldcg(a.stats + STATS_STRIDE * (it - 1) + STAT_MOVED_EDGES) >= a.dense_moved_edges;
      if (blockIdx.x == 0 && threadIdx.x == 0)
        a.stats[STATS_STRIDE * it + STAT_PHASE] = (ph.all ? 2ull : 0ull) | (ph.nomark ? 1ull : 0ull);
    }
    __syncthreads();
    const int l = a.start_iter + it;
    const bool pickless = a.pickless_step > 0 && l % a.pickless_step == 0;
    const uint32_t *vin = a.vcom0;
    uint32_t *vout = a.vcom0;
    uint8_t *fin = a.aff0, *fout = a.aff0;
    Counters cnt{0, 0, 0, 0};
    const int64_t total = rg.ibegin[NREG];
    unsigned long long *work = a.stats + STATS_STRIDE * it + STAT_WORK;
    uint32_t *q = lq[threadIdx.x >> 5];
    int qn = 0;
    for (;;) {
      unsigned long long got = 0;
      if (lane == 0) got = atomicAdd(work, 1ull);
      const int64_t item = int64_t(__shfl_sync(FULL, got, 0));
      if (item >= total) break;
      int r = 0;
      while (item >= rg.ibegin[r + 1]) ++r;
      const int64_t local = item - rg.ibegin[r];
      if (r == REG_LANE) {
        for (int64_t sb = 0; sb < rg.lane_item; ++sb) {
          const int64_t sub = local * rg.lane_item + sb;
          if (sub * 32 >= rg.vcount[REG_LANE]) break;
          qn = async_lane_collect<S, O, UNIT, BATCH>(a, rg, sub, vin, vout, fin, q, qn, ph);
          if (qn >= 32) {
            RAK_ASYNC_BY_RULE(async_lane_batch, (a, g, q, 32, it, pickless, vin, vout, fin, fout, cnt, ph));
            __syncwarp();
            if (lane < qn - 32) q[lane] = q[32 + lane];
            __syncwarp();
            qn -= 32;
          }
        }
      } else if (r == REG_HUB) {
        RAK_ASYNC_BY_RULE(async_hub_item, (a, rg, g, local, it, pickless, vin, vout, fin, fout, cnt, sc, ph));
      } else {
        RAK_ASYNC_BY_RULE(async_group_item, (a, rg, g, r, local, it, pickless, vin, vout, fin, fout, cnt, sc, ph));
      }
    }
    if (qn > 0) RAK_ASYNC_BY_RULE(async_lane_batch, (a, g, q, qn, it, pickless, vin, vout, fin, fout, cnt, ph));
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
    if (!grid_barrier_count(rs, ++epoch, a.timeout_ns)) return;
    const unsigned long long changed = __ldcg(a.stats + STATS_STRIDE * it + STAT_CHANGED);
    const bool test = !pickless || a.check_on_pickless;
    // Batches finish when no graph is still running (decided in the per-graph phase below).
    const bool done = !BATCH && (it + 1 >= a.iters || (test && double(changed) / double(a.n) <= a.tolerance));
    if (!ph.nomark && !done && a.nchunks > 0 &&
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
      if (!grid_barrier_count(rs, ++epoch, a.timeout_ns)) return;
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
  }
}
#undef RAK_ASYNC_BY_RULE

template <int S>
const void *async_kernel(bool off64, bool unit, bool batch) {
  if (batch) return unit ? reinterpret_cast<const void *>(&lpa_run_async<S, int64_t, true, true>)
                         : reinterpret_cast<const void *>(&lpa_run_async<S, int64_t, false, true>);
  if (off64) return unit ? reinterpret_cast<const void *>(&lpa_run_async<S, int64_t, true, false>)
                         : reinterpret_cast<const void *>(&lpa_run_async<S, int64_t, false, false>);
  return unit ? reinterpret_cast<const void *>(&lpa_run_async<S, int32_t, true, false>)
              : reinterpret_cast<const void *>(&lpa_run_async<S, int32_t, false, false>);
}

}  // namespace rak
