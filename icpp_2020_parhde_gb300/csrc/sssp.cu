// sssp.cu -- exact weighted shortest paths for WParHDE, one persistent cooperative launch per source.
//
// Replaces gapbs DeltaStep (gapbs/sssp.cc:53-140) as called from WParHDE (WParHDE.cpp:116 through
// DrawingBase.cpp:116).  The reference runs delta-stepping with thread-local bins of width delta and
// CAS-min relaxations; this kernel keeps the same bucketing idea in a GPU shape (near-far):
//   near set  : vertices whose tentative distance is below the current band limit T, processed in
//               rounds; every round relaxes all out-edges of the near frontier, edge-balanced exactly
//               like the top-down BFS step (owner found by binary search over the frontier's
//               start-edge prefix array), with atomicMin on the distance;
//   far pile  : improved vertices at or beyond T; when the near frontier empties, T jumps to the band
//               holding the smallest far distance and the pile is split into the new near frontier and
//               what stays far.
// On graphs whose longest row has at most SG_MAX_ROW neighbours the rounds are not edge-balanced: a lane group per
// frontier vertex reads its row at once (sssp_group_kernel), which spares the owner search.
// Both lists are de-duplicated with per-vertex stamps.  Shortest-path distances are unique, so the
// result is bit-exact against the reference whatever the band width or relaxation order.
#include <algorithm>
#include <cstdlib>

#include "ctx.h"

namespace {

constexpr int SS_THREADS = 1024;
constexpr int32_t SSSP_INF = 0x7fffffff / 2;  // kDistInf, gapbs/sssp.cc:50

struct SsArgs {
  const int64_t *off;
  const uint32_t *adj;
  const int32_t *w;
  int64_t n;
  const int64_t *src;
  int32_t *dist;  // [n], SSSP_INF initially
  int32_t delta;
  int lmax;                         // block-local relaxation rounds per grid round
  uint32_t *qv0, *qv1, *qe0, *qe1;  // near frontier (vertex, start-edge prefix)
  uint32_t *qo0, *qo1;              // near frontier: the vertex's first adjacency index
  uint32_t *far0, *far1;            // far pile
  int32_t *stamp_near, *stamp_far;  // [n], -1 initially
  ull *ctr;                         // [4] near ring
  unsigned *farctr;                 // [2]
  ull *minfar;                      // [2], alternating by phase
  ull *edges;  // [0] += adjacency entries read, [1] += rounds; may be null
  GridSync *gs;
  int *err;
  uint64_t timeout_ns;
};

constexpr int SS_LQ = SS_THREADS;  // block-local queue capacity (one entry per thread for its prefix scan)

// The block-local queue: vertices a block improved below the band limit, relaxed again by the same block
// before the grid barrier.
struct LocalQ {
  uint32_t v[2][SS_LQ], deg[2][SS_LQ], first[2][SS_LQ], off[2][SS_LQ];  // first: exclusive prefix of deg
  uint32_t cnt[2];  // entries claimed (may exceed SS_LQ: the excess went to the grid queue)
  uint32_t total;   // edges of the buffer being relaxed
  uint32_t warp_sum[32];
};

// One edge u -> v (index j).  Returns the flags of what the improvement asks for: near (below the band
// limit T) or far; atomicMin has already lowered dist[v].  ov/dv: v's adjacency start and out-degree.
__device__ __forceinline__ void relax_edge(const SsArgs &a, uint32_t u, int64_t j, int64_t T, uint32_t &v, bool &near,
                                           bool &far, uint32_t &ov, uint32_t &dv) {
  v = __ldg(a.adj + j);
  const int32_t du = __ldcg(a.dist + u);
  const int32_t nd = du + __ldg(a.w + j);
  if (nd < __ldcg(a.dist + v)) {
    const int64_t ov0 = __ldg(a.off + v), ov1 = __ldg(a.off + v + 1);  // in flight with the atomic
    const int32_t old = atomicMin(a.dist + v, nd);
    if (nd < old) {
      near = nd < T;
      far = !near;
      ov = (uint32_t)ov0;
      dv = (uint32_t)(ov1 - ov0);
    }
  }
}

// Offers near improvements to local buffer b (warp-aggregated slot claims in shared memory); those that do
// not fit fall back to the grid queue, de-duplicated by the round's stamp.  Far improvements are
// de-duplicated by the phase's stamp.  On return to_near / to_far are the grid-queue and far-pile flags.
__device__ __forceinline__ void place(const SsArgs &a, LocalQ &lq, int b, bool local_ok, uint32_t v, uint32_t dv,
                                      uint32_t ov, int32_t it, int32_t phase, bool &to_near, bool &to_far) {
  const int lane = threadIdx.x & 31;
  bool want = local_ok && to_near;
  const unsigned m = __ballot_sync(PHDE_FULL_MASK, want);
  if (m) {
    const int leader = __ffs(m) - 1;
    uint32_t wb = 0;
    if (lane == leader) wb = atomicAdd(&lq.cnt[b], (uint32_t)__popc(m));
    wb = __shfl_sync(PHDE_FULL_MASK, wb, leader);
    if (want) {
      const uint32_t slot = wb + __popc(m & ((1u << lane) - 1u));
      if (slot < SS_LQ) {
        lq.v[b][slot] = v;
        lq.deg[b][slot] = dv;
        lq.off[b][slot] = ov;
        to_near = false;  // handled locally
      }
    }
  }
  if (to_near) to_near = atomicExch(a.stamp_near + v, it + 1) != it + 1;
  if (to_far) to_far = atomicExch(a.stamp_far + v, phase) != phase;
}

template <int MINB>
__global__ void __launch_bounds__(SS_THREADS, MINB) sssp_nearfar_kernel(SsArgs a) {
  __shared__ Push2Scratch psc;
  __shared__ uint32_t s_win[SS_THREADS / 32][32];
  __shared__ ull red[32];
  extern __shared__ __align__(16) unsigned char ss_dyn[];  // the LocalQ, present only when a.lmax > 0
  LocalQ &lq = *reinterpret_cast<LocalQ *>(ss_dyn);
  const int tid = threadIdx.x;
  const int64_t gstride = (int64_t)gridDim.x * blockDim.x;
  const int64_t gbase = (int64_t)blockIdx.x * blockDim.x;
  const int64_t src = *a.src;
  if (blockIdx.x == 0 && tid == 0) {
    a.dist[src] = 0;
    a.qv0[0] = (uint32_t)src;
    a.qe0[0] = 0;
    a.qo0[0] = (uint32_t)a.off[src];
    a.stamp_near[src] = 0;
  }
  ull edges_local = 0;
  uint32_t f_cnt = 1, f_edges = (uint32_t)(a.off[src + 1] - a.off[src]);
  unsigned far_cnt = 0;
  int64_t T = a.delta;
  int32_t it = 0, phase = 0;
  uint32_t step = 0;
  if (!grid_sync(a.gs, a.err, a.timeout_ns)) return;

  while (true) {
    // ---- relaxation rounds over the near frontier ----
    while (f_cnt > 0) {
      const uint32_t *qin_v = (step & 1) ? a.qv1 : a.qv0;
      const uint32_t *qin_e = (step & 1) ? a.qe1 : a.qe0;
      const uint32_t *qin_o = (step & 1) ? a.qo1 : a.qo0;
      uint32_t *qout_v = (step & 1) ? a.qv0 : a.qv1;
      uint32_t *qout_e = (step & 1) ? a.qe0 : a.qe1;
      uint32_t *qout_o = (step & 1) ? a.qo0 : a.qo1;
      ull *octr = a.ctr + (step & 3);
      uint32_t *far_in = (phase & 1) ? a.far1 : a.far0;
      unsigned *fctr = a.farctr + (phase & 1);
      if (blockIdx.x == 0 && tid == 0) a.ctr[(step + 1) & 3] = 0ull;
      const int64_t E = f_edges;
      const bool local_on = a.lmax > 0;
      if (local_on) {
        if (tid == 0) lq.cnt[0] = lq.cnt[1] = 0;
        __syncthreads();
      }
      for (int64_t base = gbase; base < E; base += gstride) {
        const int64_t e = base + tid, e0w = base + (tid & ~31);
        bool to_near = false, to_far = false;
        uint32_t v = 0, dv = 0, ov = 0;
        if (e0w < E) {  // warp-uniform
          uint32_t es;
          const uint32_t s = warp_owner_slots(qin_e, f_cnt, (uint32_t)e0w, s_win[tid >> 5], es);
          if (e < E) {
            const uint32_t u = qin_v[s];
            const int64_t j = (int64_t)qin_o[s] + (e - (int64_t)es);  // qin_o[s] = off[u], loaded with u
            edges_local++;
            relax_edge(a, u, j, T, v, to_near, to_far, ov, dv);
          }
        }
        place(a, lq, 0, local_on, v, dv, ov, it, phase, to_near, to_far);
        block_push2(to_near, v, dv, qout_v, qout_e, octr, to_far, far_in, fctr, &psc, qout_o, ov);
      }
      // ---- block-local rounds: relax what this block improved, without a grid barrier; the last local
      // round (and any overflow of the local queue) sends its improvements to the grid queue ----
      int cur = 0;
      for (int li = 0; li < a.lmax; li++) {
        __syncthreads();  // the buffer's entries are written
        const uint32_t cnt = min(lq.cnt[cur], (uint32_t)SS_LQ);
        if (cnt == 0) break;
        {  // exclusive prefix of the out-degrees, one entry per thread
          const int lane = tid & 31, w = tid >> 5;
          const uint32_t d = (uint32_t)tid < cnt ? lq.deg[cur][tid] : 0u;
          uint32_t x = d;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(PHDE_FULL_MASK, x, o);
            if (lane >= o) x += y;
          }
          if (lane == 31) lq.warp_sum[w] = x;
          __syncthreads();
          if (w == 0) {
            const uint32_t ws_ = lane < (int)(blockDim.x >> 5) ? lq.warp_sum[lane] : 0u;
            uint32_t y = ws_;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const uint32_t z = __shfl_up_sync(PHDE_FULL_MASK, y, o);
              if (lane >= o) y += z;
            }
            lq.warp_sum[lane] = y - ws_;
            if (lane == 31) lq.total = y;
          }
          __syncthreads();
          if ((uint32_t)tid < cnt) lq.first[cur][tid] = lq.warp_sum[w] + x - d;
          if (tid == 0) lq.cnt[cur ^ 1] = 0;
          __syncthreads();
        }
        const uint32_t total = lq.total;
        for (uint32_t eb = 0; eb < total; eb += blockDim.x) {
          const uint32_t e = eb + tid;
          bool to_near = false, to_far = false;
          uint32_t v = 0, dv = 0, ov = 0;
          if (e < total) {
            uint32_t lo = 0, hi = cnt;  // the entry owning local edge e
            while (hi - lo > 1) {
              const uint32_t mid = (lo + hi) >> 1;
              if (lq.first[cur][mid] <= e)
                lo = mid;
              else
                hi = mid;
            }
            const uint32_t u = lq.v[cur][lo];
            const int64_t j = (int64_t)lq.off[cur][lo] + (e - lq.first[cur][lo]);
            edges_local++;
            relax_edge(a, u, j, T, v, to_near, to_far, ov, dv);
          }
          place(a, lq, cur ^ 1, li + 1 < a.lmax, v, dv, ov, it, phase, to_near, to_far);
          block_push2(to_near, v, dv, qout_v, qout_e, octr, to_far, far_in, fctr, &psc, qout_o, ov);
        }
        cur ^= 1;
      }
      ull out;
      if (!grid_sync_read(a.gs, a.err, a.timeout_ns, octr, &out)) return;
      f_cnt = (uint32_t)(out >> 32);
      f_edges = (uint32_t)(out & 0xffffffffull);
      it++;
      step++;
    }
    // ---- near frontier empty: move to the band of the closest far vertex ----
    far_cnt = block_read(a.farctr + (phase & 1));
    if (far_cnt == 0) break;
    const uint32_t *far_in = (phase & 1) ? a.far1 : a.far0;
    uint32_t *far_out = (phase & 1) ? a.far0 : a.far1;
    unsigned *fout_ctr = a.farctr + ((phase + 1) & 1);
    ull *mslot = a.minfar + (phase & 1);
    ull mloc = ~0ull;
    for (int64_t i = gbase + tid; i < far_cnt; i += gstride) {
      const int32_t d = __ldcg(a.dist + far_in[i]);
      if (d >= T) mloc = (ull)d < mloc ? (ull)d : mloc;
    }
    const ull bm = block_max_u64(~mloc, red);  // block minimum through the complement
    if (tid == 0 && bm != 0ull) atomicMin(mslot, ~bm);
    if (blockIdx.x == 0 && tid == 0) {
      *fout_ctr = 0u;
      a.minfar[(phase + 1) & 1] = ~0ull;
    }
    ull mf;
    if (!grid_sync_read(a.gs, a.err, a.timeout_ns, mslot, &mf)) return;
    const int64_t T_old = T;
    if (mf != ~0ull) T = ((int64_t)mf / a.delta + 1) * (int64_t)a.delta;
    // split the pile: this is a step of its own, writing the next round's input queue
    uint32_t *qout_v = (step & 1) ? a.qv0 : a.qv1;
    uint32_t *qout_e = (step & 1) ? a.qe0 : a.qe1;
    uint32_t *qout_o = (step & 1) ? a.qo0 : a.qo1;
    ull *octr = a.ctr + (step & 3);
    if (blockIdx.x == 0 && tid == 0) a.ctr[(step + 1) & 3] = 0ull;
    for (int64_t base = gbase; base < (int64_t)far_cnt; base += gstride) {
      const int64_t i = base + tid;
      bool to_near = false, keep = false;
      uint32_t v = 0, dv = 0, ov = 0;
      if (i < far_cnt) {
        v = far_in[i];
        const int32_t d = __ldcg(a.dist + v);
        if (d >= T_old && d < T) {
          if (atomicExch(a.stamp_near + v, it + 1) != it + 1) {
            to_near = true;
            ov = (uint32_t)a.off[v];
            dv = (uint32_t)(a.off[v + 1] - ov);
          }
        } else if (d >= T) {
          keep = atomicExch(a.stamp_far + v, phase + 1) != phase + 1;
        }
      }
      block_push2(to_near, v, dv, qout_v, qout_e, octr, keep, far_out, fout_ctr, &psc, qout_o, ov);
    }
    ull out;
    if (!grid_sync_read(a.gs, a.err, a.timeout_ns, octr, &out)) return;
    f_cnt = (uint32_t)(out >> 32);
    f_edges = (uint32_t)(out & 0xffffffffull);
    it++;
    step++;
    phase++;
    if (f_cnt == 0 && __ldcg(a.farctr + (phase & 1)) == 0) break;
  }
  ull etot = block_sum(edges_local, red);
  if (tid == 0 && a.edges) atomicAdd(a.edges, etot);
  if (blockIdx.x == 0 && tid == 0 && a.edges) atomicAdd(a.edges + 1, (ull)it);  // rounds (relaxation + split)
}

// ---- graphs of bounded degree (grids, meshes, geometric graphs): a lane group per frontier vertex ----
// A round is a chain of dependent memory trips ended by a grid barrier, whatever it relaxes; the edge-balanced
// kernel above spends about a third of its trips finding the owner of every edge.  Where no row is longer than
// SG_MAX_ROW, G lanes take one frontier entry (vertex, row start and length in one 16-byte word) and R edges each:
// entry -> adjacency, weight and the vertex's distance -> the neighbours' distances -> the
// updates -> push.  The update is a reduction (no value returned) with the duplicate stamp's exchange beside it
// instead of after it: a thread that found the neighbour's distance larger pushes when its stamp is the round's
// first, whether its own minimum was the one that stayed -- some thread lowered the distance in this round, and
// every thread that did so takes the stamp.  Bands, far pile and results as in sssp_nearfar_kernel.
// Measured, 20 passes: 256^3 grid 238 -> 180 ms (12.4 -> 9.4 us a round), 65 x 61 x 70 grid 24.8 -> 20.4 ms (6.8 ->
// 5.6 us a round; 4.7 us of a round is the chain itself, measured with a band that leaves 7k edges a round).
// Shapes (G, R), passes of a layout with k = 10: rows up to 16, 300k vertices (16, 1) 94 ms, (8, 2) 101; rows up to 32,
// 300k vertices (16, 2) 42, (32, 1) 44, (8, 4) 54; 2M vertices in 3-D 33, 40 and 36.  Fewer lanes with more edges each
// lose on grids too: 256^3 (8, 1) 233, (4, 2) 255, (2, 4) 319 ms a layout.
constexpr int SG_MAX_ROW = 32;

struct PushRScratch {
  uint32_t warp_tot[32];
  uint32_t base_near, base_far;
};

// Appends each thread's flagged entries: near ones (16-byte entries) and far ones (vertices).  Called by every
// thread of the block.
template <int R>
__device__ __forceinline__ void block_push_r(unsigned nearm, unsigned farm, const uint32_t (&v)[R],
                                             const uint32_t (&ov)[R], const uint32_t (&dv)[R], uint4 *q, unsigned *qctr,
                                             uint32_t *far, unsigned *fctr, PushRScratch *sc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t mine = (uint32_t)__popc(nearm) | ((uint32_t)__popc(farm) << 16);  // at most 4 * 1024 of each
  uint32_t x = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(PHDE_FULL_MASK, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sc->warp_tot[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const uint32_t w = lane < nw ? sc->warp_tot[lane] : 0u;
    uint32_t incl = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(PHDE_FULL_MASK, incl, o);
      if (lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(PHDE_FULL_MASK, incl, 31);
    sc->warp_tot[lane] = incl - w;
    if (lane == 0) sc->base_near = total & 0xffffu ? atomicAdd(qctr, total & 0xffffu) : 0u;
    if (lane == 1) sc->base_far = total >> 16 ? atomicAdd(fctr, total >> 16) : 0u;
  }
  __syncthreads();
  const uint32_t before = sc->warp_tot[warp] + x - mine;
  uint32_t an = sc->base_near + (before & 0xffffu), af = sc->base_far + (before >> 16);
#pragma unroll
  for (int r = 0; r < R; r++) {
    if ((nearm >> r) & 1u) q[an++] = make_uint4(v[r], ov[r], dv[r], 0u);
    if ((farm >> r) & 1u) far[af++] = v[r];
  }
}

template <int G, int R, int MINB>
__global__ void __launch_bounds__(SS_THREADS, MINB) sssp_group_kernel(SsArgs a) {
  __shared__ PushRScratch psc;
  __shared__ ull red[32];
  const int tid = threadIdx.x, gl = tid & (G - 1);
  const int64_t gstride = (int64_t)gridDim.x * blockDim.x;
  const int64_t gbase = (int64_t)blockIdx.x * blockDim.x;
  const int64_t src = *a.src;
  uint4 *q0 = (uint4 *)a.qv0, *q1 = (uint4 *)a.qv1;
  unsigned *ctr = (unsigned *)a.ctr;
  if (blockIdx.x == 0 && tid == 0) {
    a.dist[src] = 0;
    q0[0] = make_uint4((uint32_t)src, (uint32_t)a.off[src], (uint32_t)(a.off[src + 1] - a.off[src]), 0u);
    a.stamp_near[src] = 0;
  }
  ull edges_local = 0;
  uint32_t f_cnt = 1;
  int64_t T = a.delta;
  int32_t it = 0, phase = 0;
  uint32_t step = 0;
  if (!grid_sync(a.gs, a.err, a.timeout_ns)) return;
  while (true) {
    while (f_cnt > 0) {
      const uint4 *qin = (step & 1) ? q1 : q0;
      uint4 *qout = (step & 1) ? q0 : q1;
      unsigned *octr = ctr + (step & 3);
      uint32_t *far_in = (phase & 1) ? a.far1 : a.far0;
      unsigned *fctr = a.farctr + (phase & 1);
      if (blockIdx.x == 0 && tid == 0) ctr[(step + 1) & 3] = 0u;
      const int64_t lanes = (int64_t)f_cnt * G;
      for (int64_t base = gbase; base < lanes; base += gstride) {
        uint32_t v[R], ov[R], dv[R];
        unsigned nearm = 0, farm = 0;
        if (base + tid < lanes) {
          const uint4 en = __ldcg(qin + (base + tid) / G);
          const int32_t du = __ldcg(a.dist + en.x);
          int32_t nd[R], old[R];
#pragma unroll
          for (int r = 0; r < R; r++) {
            const uint32_t e = gl + r * G;
            const bool has = e < en.z;
            v[r] = has ? __ldg(a.adj + en.y + e) : en.x;  // the vertex itself: never an improvement
            nd[r] = has ? __ldg(a.w + en.y + e) : 0;
            if (has) edges_local++;
          }
#pragma unroll
          for (int r = 0; r < R; r++) old[r] = __ldcg(a.dist + v[r]);
#pragma unroll
          for (int r = 0; r < R; r++) {
            nd[r] += du;
            if (nd[r] >= old[r]) continue;
            atomicMin(a.dist + v[r], nd[r]);
            const bool near = nd[r] < T;
            const int32_t mark = near ? it + 1 : phase;
            const int64_t o0 = __ldg(a.off + v[r]), o1 = __ldg(a.off + v[r] + 1);
            if (atomicExch((near ? a.stamp_near : a.stamp_far) + v[r], mark) != mark) {
              if (near)
                nearm |= 1u << r;
              else
                farm |= 1u << r;
            }
            ov[r] = (uint32_t)o0;
            dv[r] = (uint32_t)(o1 - o0);
          }
        }
        if (__syncthreads_or(nearm | farm)) block_push_r<R>(nearm, farm, v, ov, dv, qout, octr, far_in, fctr, &psc);
      }
      if (!grid_sync_read(a.gs, a.err, a.timeout_ns, octr, &f_cnt)) return;
      it++;
      step++;
    }
    // ---- near frontier empty: move to the band of the closest far vertex (as in sssp_nearfar_kernel) ----
    const unsigned far_cnt = block_read(a.farctr + (phase & 1));
    if (far_cnt == 0) break;
    const uint32_t *far_in = (phase & 1) ? a.far1 : a.far0;
    uint32_t *far_out = (phase & 1) ? a.far0 : a.far1;
    unsigned *fout_ctr = a.farctr + ((phase + 1) & 1);
    ull *mslot = a.minfar + (phase & 1);
    ull mloc = ~0ull;
    for (int64_t i = gbase + tid; i < far_cnt; i += gstride) {
      const int32_t d = __ldcg(a.dist + __ldcg(far_in + i));
      if (d >= T) mloc = (ull)d < mloc ? (ull)d : mloc;
    }
    const ull bm = block_max_u64(~mloc, red);
    if (tid == 0 && bm != 0ull) atomicMin(mslot, ~bm);
    if (blockIdx.x == 0 && tid == 0) {
      *fout_ctr = 0u;
      a.minfar[(phase + 1) & 1] = ~0ull;
    }
    ull mf;
    if (!grid_sync_read(a.gs, a.err, a.timeout_ns, mslot, &mf)) return;
    const int64_t T_old = T;
    if (mf != ~0ull) T = ((int64_t)mf / a.delta + 1) * (int64_t)a.delta;
    uint4 *qout = (step & 1) ? q0 : q1;
    unsigned *octr = ctr + (step & 3);
    if (blockIdx.x == 0 && tid == 0) ctr[(step + 1) & 3] = 0u;
    for (int64_t base = gbase; base < (int64_t)far_cnt; base += gstride) {
      const int64_t i = base + tid;
      uint32_t v[1] = {0}, ov[1] = {0}, dv[1] = {0};
      unsigned nearm = 0, keepm = 0;
      if (i < far_cnt) {
        v[0] = __ldcg(far_in + i);
        const int32_t d = __ldcg(a.dist + v[0]);
        if (d >= T_old && d < T) {
          if (atomicExch(a.stamp_near + v[0], it + 1) != it + 1) {
            nearm = 1;
            ov[0] = (uint32_t)a.off[v[0]];
            dv[0] = (uint32_t)(a.off[v[0] + 1] - ov[0]);
          }
        } else if (d >= T) {
          keepm = atomicExch(a.stamp_far + v[0], phase + 1) != phase + 1;
        }
      }
      block_push_r<1>(nearm, keepm, v, ov, dv, qout, octr, far_out, fout_ctr, &psc);
      __syncthreads();
    }
    if (!grid_sync_read(a.gs, a.err, a.timeout_ns, octr, &f_cnt)) return;
    it++;
    step++;
    phase++;
    if (f_cnt == 0 && __ldcg(a.farctr + (phase & 1)) == 0) break;
  }
  const ull etot = block_sum(edges_local, red);
  if (tid == 0 && a.edges) atomicAdd(a.edges, etot);
  if (blockIdx.x == 0 && tid == 0 && a.edges) atomicAdd(a.edges + 1, (ull)it);
}

// Fold one finished distance column into the Kcenters state (WParHDE.cpp:117-136).
__global__ void fold_kernel(const int32_t *col, int64_t n, int32_t *min_d, ull *key_out, ull *ssq_out, int *err) {
  __shared__ ull red[32];
  ull kbest = 0, ssq = 0;
  int bad = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v0 < n; v0 += 4 * stride) {
    int32_t d[4], m[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {  // four rows' loads in flight: 16.8M rows 104 -> 35 us
      const int64_t v = v0 + t * stride;
      d[t] = v < n ? col[v] : 0;
      m[t] = v < n ? min_d[v] : 0;
    }
#pragma unroll
    for (int t = 0; t < 4; t++) {
      const int64_t v = v0 + t * stride;
      if (v >= n) continue;
      if (d[t] >= SSSP_INF || d[t] < 0) {
        bad = 1;
        continue;
      }
      ssq += (ull)d[t] * (ull)d[t];
      if (d[t] < m[t]) min_d[v] = m[t] = d[t];
      const ull key = ((ull)(uint32_t)m[t] << 32) | (ull)(0xffffffffu - (uint32_t)v);
      kbest = key > kbest ? key : kbest;
    }
  }
  if (__syncthreads_or(bad)) {
    if (threadIdx.x == 0) atomicCAS(err, 0, PHDE_ERR_DISCONNECTED);
    return;
  }
  ssq = block_sum(ssq, red);
  kbest = block_max_u64(kbest, red);
  if (threadIdx.x == 0) {
    atomicAdd(ssq_out, ssq);
    atomicMax(key_out, kbest);
  }
}

// Choose the next source (one block): raw argmax, duplicate fix-up against the history of raw argmaxes
// (WParHDE.cpp:137-153), append the raw argmax to the history.
__global__ void select_kernel(const ull *key_in, const int32_t *min_d, int64_t n, int pass, int check_fix,
                              int64_t *hist, int64_t *next_src) {
  __shared__ ull red[32];
  const ull key = *key_in;
  const int64_t raw = (int64_t)(0xffffffffu - (uint32_t)(key & 0xffffffffull));
  const int32_t maxval = (int32_t)(key >> 32);
  int hit = 0;
  for (int i = threadIdx.x; i < pass; i += blockDim.x) hit |= (hist[i] == raw);
  hit = __syncthreads_or(hit);
  int64_t next = raw;
  if (check_fix && hit) {
    ull best = 0;
    for (int64_t v = threadIdx.x; v < n; v += blockDim.x) {
      if (min_d[v] != maxval) continue;
      bool inh = false;
      for (int i = 0; i < pass && !inh; i++) inh = hist[i] == v;
      if (!inh) best = (ull)v + 1 > best ? (ull)v + 1 : best;
    }
    best = block_max_u64(best, red);
    if (best) next = (int64_t)best - 1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    hist[pass] = raw;
    *next_src = next;
  }
}

}  // namespace

int phde_fill_i32(phde_ctx *ctx, int32_t *p, int64_t n, int32_t v);

namespace {
// sum of the (non-negative) edge weights, for the band width
__global__ void weight_sum_kernel(const int32_t *w, int64_t nnz, ull *sum) {
  ull s = 0;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz; e += (int64_t)gridDim.x * blockDim.x)
    s += (ull)(w[e] > 0 ? w[e] : 0);
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0 && s) atomicAdd(sum, s);
}
}  // namespace

int phde_run_sssp(phde_ctx *ctx, const int64_t *d_src, int32_t *d_col, int32_t delta, unsigned long long *d_edges) {
  const int64_t n = ctx->n;
  if (ctx->nnz >= (int64_t)0xffffffffll || n >= (int64_t)0xffffffffll)
    return phde_fail(ctx, PHDE_ERR_INVALID, "graphs with 2^32 or more vertices or adjacency entries are not supported");
  if (!ctx->d_w) return phde_fail(ctx, PHDE_ERR_WEIGHTS, "SSSP needs edge weights");
  // The band width changes the work, never the distances (they are unique).  The reference's width
  // (10000, WParHDE.cpp:104) is far above typical weights, which makes the search nearly Bellman-Ford: on
  // a 256^3 grid with weights in [1, 255] a band of 8 mean weights is three times faster (on a 64^3 grid,
  // where every round is short, the wide band is as fast or faster).  So graphs of 2^20 vertices or more
  // use min(delta, max(64, 8 * mean weight)); PHDE_SSSP_DELTA sets the band outright.
  if (const char *e = getenv("PHDE_SSSP_DELTA")) {
    delta = atoi(e);
  } else if (n >= (int64_t)1 << 20) {
    if (ctx->w_mean_epoch != ctx->graph_epoch) {
      ull *wsum = (ull *)phde_buf(ctx, "ss.wsum", sizeof(ull));
      if (!wsum) return PHDE_ERR_OOM;
      PHDE_CK(ctx, cudaMemsetAsync(wsum, 0, sizeof(ull), ctx->stream));
      const int g = (int)std::max<int64_t>(1, std::min<int64_t>((ctx->nnz + 255) / 256, (int64_t)ctx->nsm * 8));
      weight_sum_kernel<<<g, 256, 0, ctx->stream>>>(ctx->d_w, ctx->nnz, wsum);
      PHDE_LAUNCHED(ctx);
      ull h = 0;
      PHDE_CK(ctx, cudaMemcpyAsync(&h, wsum, sizeof(ull), cudaMemcpyDeviceToHost, ctx->stream));
      PHDE_CK(ctx, cudaStreamSynchronize(ctx->stream));
      ctx->w_mean = ctx->nnz > 0 ? (double)h / (double)ctx->nnz : 1.0;
      ctx->w_mean_epoch = ctx->graph_epoch;
    }
    const double band = std::max(64.0, 8.0 * ctx->w_mean);
    if (band < (double)delta) delta = (int32_t)band;
  }
  if (delta < 1) delta = 1;
  const char *le = getenv("PHDE_SSSP_LOCAL");
  const int lmax = le ? std::max(0, atoi(le)) : 0;
  const bool group = lmax == 0 && ctx->max_degree_epoch == ctx->graph_epoch && ctx->max_degree <= SG_MAX_ROW;
  uint32_t *qv0, *qv1, *qe0 = nullptr, *qe1 = nullptr, *qo0 = nullptr, *qo1 = nullptr;
  if (group) {
    qv0 = (uint32_t *)phde_buf(ctx, "ss.q0", sizeof(uint4) * n);
    qv1 = (uint32_t *)phde_buf(ctx, "ss.q1", sizeof(uint4) * n);
    if (!qv0 || !qv1) return PHDE_ERR_OOM;
  } else {
    qv0 = (uint32_t *)phde_buf(ctx, "q.v0", sizeof(uint32_t) * n);
    qv1 = (uint32_t *)phde_buf(ctx, "q.v1", sizeof(uint32_t) * n);
    qe0 = (uint32_t *)phde_buf(ctx, "q.e0", sizeof(uint32_t) * n);
    qe1 = (uint32_t *)phde_buf(ctx, "q.e1", sizeof(uint32_t) * n);
    qo0 = (uint32_t *)phde_buf(ctx, "ss.qo0", sizeof(uint32_t) * n);
    qo1 = (uint32_t *)phde_buf(ctx, "ss.qo1", sizeof(uint32_t) * n);
    if (!qv0 || !qv1 || !qe0 || !qe1 || !qo0 || !qo1) return PHDE_ERR_OOM;
  }
  uint32_t *far0 = (uint32_t *)phde_buf(ctx, "ss.far0", sizeof(uint32_t) * n);
  uint32_t *far1 = (uint32_t *)phde_buf(ctx, "ss.far1", sizeof(uint32_t) * n);
  int32_t *stn = (int32_t *)phde_buf(ctx, "ss.stamp_near", sizeof(int32_t) * n);
  int32_t *stf = (int32_t *)phde_buf(ctx, "ss.stamp_far", sizeof(int32_t) * n);
  ull *ctr = (ull *)phde_buf(ctx, "q.ctr", sizeof(ull) * 4);
  unsigned *farctr = (unsigned *)phde_buf(ctx, "ss.farctr", sizeof(unsigned) * 2);
  ull *minfar = (ull *)phde_buf(ctx, "ss.minfar", sizeof(ull) * 2);
  if (!far0 || !far1 || !stn || !stf || !ctr || !farctr || !minfar) return PHDE_ERR_OOM;
  int rc;
  if ((rc = phde_fill_i32(ctx, d_col, n, SSSP_INF))) return rc;
  PHDE_CK(ctx, cudaMemsetAsync(stn, 0xff, sizeof(int32_t) * n, ctx->stream));
  PHDE_CK(ctx, cudaMemsetAsync(stf, 0xff, sizeof(int32_t) * n, ctx->stream));
  PHDE_CK(ctx, cudaMemsetAsync(ctr, 0, sizeof(ull) * 4, ctx->stream));
  PHDE_CK(ctx, cudaMemsetAsync(farctr, 0, sizeof(unsigned) * 2, ctx->stream));
  PHDE_CK(ctx, cudaMemsetAsync(minfar, 0xff, sizeof(ull) * 2, ctx->stream));
  if ((rc = phde_reset_sync(ctx))) return rc;
  // Resident CTAs per SM: one (with the registers it wants) on small graphs, whose rounds are short, two (registers
  // capped at 32) on larger ones; PHDE_SSSP_CTAS=1 or 2 picks outright.  Lane groups change over at 2^18 vertices, where
  // grids cross (four passes with one and two, ms: 52^3 2.85 and 3.13, 58^3 3.48 and 3.51, 63^3 4.22 and 4.17, 72^3 5.23
  // and 4.89; a 600 x 600 mesh 20.5 and 20.8, longer rows cross lower: 200k vertices in 2-D 17.8 and 17.1, in 3-D 7.6 and
  // 5.7), the edge-balanced kernel at 2^20 (64^3 grid: 1.5 ms per pass with one against 2.1; 256^3: 14.3 with two against
  // 16.1).
  const char *ce = getenv("PHDE_SSSP_CTAS");
  const int want = ce ? (atoi(ce) == 1 ? 1 : 2) : (n < ((int64_t)1 << (group ? 18 : 20)) ? 1 : 2);
  const void *kfn = want == 1 ? (const void *)sssp_nearfar_kernel<1> : (const void *)sssp_nearfar_kernel<2>;
  if (group) {  // (lanes, edges per lane) by the longest row
    const int shape = ctx->max_degree <= 8 ? 0 : ctx->max_degree <= 16 ? 1 : 2;
    static const void *const kernels[3][2] = {
        {(const void *)sssp_group_kernel<8, 1, 1>, (const void *)sssp_group_kernel<8, 1, 2>},
        {(const void *)sssp_group_kernel<16, 1, 1>, (const void *)sssp_group_kernel<16, 1, 2>},
        {(const void *)sssp_group_kernel<16, 2, 1>, (const void *)sssp_group_kernel<16, 2, 2>}};
    kfn = kernels[shape][want - 1];
  }
  // block-local rounds per grid round (PHDE_SSSP_LOCAL, none by default): each block keeps relaxing the
  // vertices it improved below the band limit (up to SS_LQ of them) this many times before the grid
  // barrier.  On a 256^3 grid four local rounds took 10-12.5 ms per pass on some runs and 43-50 ms on
  // others (same inputs, band 1024; band 512 stayed near 13 ms), against 14.6 ms without: the blocks that
  // run ahead inside the band relax with distances other blocks later lower, and how much of that is
  // wasted depends on timing.  Off until that is bounded.
  const size_t dyn = lmax > 0 ? sizeof(LocalQ) : 0;  // the queue's shared memory, below the 48 KB default
  int per_sm = 0;
  PHDE_CK(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, SS_THREADS, dyn));
  if (per_sm < 1) return phde_fail(ctx, PHDE_ERR_CUDA, "sssp kernel cannot be resident");
  per_sm = std::min(per_sm, want);
  SsArgs a;
  a.off = ctx->d_off;
  a.adj = ctx->d_adj;
  a.w = ctx->d_w;
  a.n = n;
  a.src = d_src;
  a.dist = d_col;
  a.delta = delta;
  a.lmax = lmax;
  a.qv0 = qv0;
  a.qv1 = qv1;
  a.qe0 = qe0;
  a.qe1 = qe1;
  a.qo0 = qo0;
  a.qo1 = qo1;
  a.far0 = far0;
  a.far1 = far1;
  a.stamp_near = stn;
  a.stamp_far = stf;
  a.ctr = ctr;
  a.farctr = farctr;
  a.minfar = minfar;
  a.edges = d_edges;
  a.gs = ctx->d_sync;
  a.err = ctx->d_err;
  a.timeout_ns = ctx->timeout_ns;
  void *args[] = {&a};
  cudaEventRecord(ctx->kev[0], ctx->stream);
  PHDE_CK(ctx, cudaLaunchCooperativeKernel(kfn, dim3(ctx->nsm * per_sm),
                                           dim3(SS_THREADS), args, dyn, ctx->stream));
  PHDE_LAUNCHED(ctx);
  cudaEventRecord(ctx->kev[1], ctx->stream);
  ctx->kev_pending = true;
  return PHDE_OK;
}

int phde_run_select(phde_ctx *ctx, const int32_t *d_col, int32_t *d_min, int pass, int check_fix, int64_t *d_hist,
                    int64_t *d_next_src, unsigned long long *d_sumsq) {
  ull *key = (ull *)phde_buf(ctx, "sel.key", sizeof(ull));
  if (!key) return PHDE_ERR_OOM;
  PHDE_CK(ctx, cudaMemsetAsync(key, 0, sizeof(ull), ctx->stream));
  int blocks = (int)std::min<int64_t>((ctx->n + 511) / 512, (int64_t)ctx->nsm * 4);
  fold_kernel<<<std::max(blocks, 1), 512, 0, ctx->stream>>>(d_col, ctx->n, d_min, key, d_sumsq, ctx->d_err);
  PHDE_LAUNCHED(ctx);
  select_kernel<<<1, 1024, 0, ctx->stream>>>(key, d_min, ctx->n, pass, check_fix, d_hist, d_next_src);
  PHDE_LAUNCHED(ctx);
  return PHDE_OK;
}
