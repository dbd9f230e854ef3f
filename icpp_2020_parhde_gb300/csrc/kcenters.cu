// kcenters.cu -- Kcenters pivot distances: P breadth-first searches in ONE persistent cooperative launch.
//
// Replaces the serial Kcenters loop of variants/ParHDE.cpp:118-157 (and DrawingBase.cpp:119-172), whose
// every pass calls gapbs DOBFS (gapbs/bfs.cc:144-185) and then an OpenMP min/argmax reduction.  Each pass
// here is a level-synchronous direction-optimising BFS over the device CSR, followed by the Kcenters
// selection folded into one sweep; grid barriers (bounded waits) separate the levels, so the 3k
// dependent passes cost no host round trip.
//
// Per level, with frontier F_L (vertices at hop distance L):
//   top-down  : edge-balanced -- thread e takes the e-th out-edge of F_L, finds its owner vertex over the
//               frontier's start-edge prefix array (a warp's 32 owners by one 32-ary search, 3-4 dependent
//               loads where a binary search per thread took 15; 8 passes on the 8M-vertex 3-D geometric
//               graph 45 -> 36 ms), and claims the neighbour with a CAS on its distance entry (-1 -> L+1);
//   bottom-up : every unvisited vertex scans its neighbours for one in the frontier and stops at the
//               first; the frontier is a bitmap (one bit per vertex) that every block copies into
//               shared memory at the start of the level when it fits (80 KB for 646k vertices), so the
//               membership test is a shared-memory hit;
//   both append the new frontier with block-aggregated 64-bit atomics that keep (slot, edge prefix)
//   together, so the next top-down step is load balanced even around hub vertices.
// The top-down / bottom-up switch has the reference's form (bfs.cc:159-183): go bottom-up when the
// frontier's out-edges exceed edges_to_check / alpha, stay there while the frontier grows or exceeds
// n / beta, beta = 18 as there, alpha = 6 instead of 15: on the GPU a bottom-up level scans every
// unvisited vertex, and at the frontier sizes between the two rules (R-MAT 22: 8.7 M out-edges) the
// top-down level is the faster one (130-235 us against 300-320 us).  Hop distances are unique, so the
// result is bit-exact whatever the direction schedule.
//
// Selection (ParHDE.cpp:127-155): min_d[v] = min(min_d[v], d_p[v]); the next source is the vertex of
// largest min_d, lowest index first (a 64-bit atomicMax on (min_d << 32) | ~v); if that vertex is in
// the history, the duplicate fix-up takes the highest-index vertex with the same min_d that is not.
//
// Three kernels share that rule and give the same bits.  kcenters_bfs_kernel is the grid-wide one above.
// kcenters_cluster_kernel runs the passes of a sparse graph of up to 3 << 20 vertices in one cluster's shared memory:
// its levels are a few hundred vertices, so the grid barrier was most of their time.  kcenters_block_kernel gives
// every graph of a large batch its own CTA.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "ctx.h"

namespace {

constexpr int KC_THREADS = 1024;
constexpr int KC_HISTORY = 4096;  // passes whose history is kept in shared memory, at most
// Shared memory with the frontier bitmap in it, at most: the copy of a larger bitmap costs a bottom-up level what its
// reads gain (216 KB against 116, 12 passes: R-MAT 21 1.61 against 1.69 ms, 1.6M-vertex 3-D geometric graph 15.33 against
// 15.20, 1200 x 1200 mesh 74.9 against 72.1; none against 116: R-MAT 20, 30 passes, 3.07 against 3.00).
constexpr size_t KC_SMEM = 116 * 1024;

struct KcArgs {
  const int64_t *off;
  const uint32_t *adj;
  int64_t n, nnz;
  int32_t *D;  // n * P, column-major, pre-filled with -1
  int P;
  int variant;  // 0: ParHDE history (raw argmax), 1: fixed sources, 2: DrawingBase history (used source)
  int require_all;  // an unreached vertex is an error (always for the Kcenters variants)
  const int64_t *fixed_src;
  int64_t *sources;
  int32_t *min_d;   // [n], INT32_MAX initially
  ull *sumsq;       // [P]
  ull *keys;        // [P]
  ull *fixkey;      // [P]
  uint32_t *qv0, *qv1, *qe0, *qe1;  // frontier: vertex, start-edge prefix
  uint32_t *qo0, *qo1;              // and its first adjacency index
  uint32_t *bm[3];  // frontier bitmaps, W words each, rotating with the global step (zero initially)
  int64_t W;        // words per bitmap
  int smem_bm;      // copy the frontier bitmap into shared memory for bottom-up levels
  int cap;          // entries of the block's list of new vertices: a multiple of KC_THREADS, at least two of them
  uint32_t *hist;   // [grid x P] selection histories of the blocks when they are not in shared memory
  ull *ctr;         // [4] ring of (count << 32 | edges)
  ull *edges;       // [1] adjacency entries read
  ull *trace;       // optional timeline: per level {globaltimer, pass<<40 | level<<32 | in_bu, frontier count, edges}
  int trace_cap;    // entries of 4 words
  GridSync *gs;
  int *err;
  uint64_t timeout_ns;
  int alpha, beta;
  // batched layouts: the graph is the disjoint union of B graphs (vertex ranges vbase[b]..vbase[b+1]);
  // every pass runs one BFS per graph, all from the same launch, and the selection is per graph.  Then
  // sources, keys and sumsq are indexed [p * B + b], and gid[v] is v's graph.
  int B;
  const int64_t *vbase;
  const int32_t *gid;
  ull *qinit;       // [1] level-0 queue counter of the pass (count << 32 | edges)
  const int64_t *resume;  // where kcenters_cluster_kernel stopped (KlArgs::resume; null: it did not run)
};

// Per-graph fold of a batched pass: the max of `key` and the sum of `ssq` over the lanes of one graph
// (a warp covers consecutive vertices, so almost always one graph), one atomic per graph per warp.
__device__ __forceinline__ void batch_fold(ull *keys, ull *sumsq, int g, ull key, ull ssq, bool valid) {
  const int lane = threadIdx.x & 31;
  const int g0 = __shfl_sync(PHDE_FULL_MASK, g, 0);
  if (__all_sync(PHDE_FULL_MASK, valid && g == g0)) {
    const ull km = warp_max_u64(key);
    const ull ss = warp_sum(ssq);
    if (lane == 0) {
      atomicMax(keys + g0, km);
      if (ss) atomicAdd(sumsq + g0, ss);
    }
  } else if (valid) {
    atomicMax(keys + g, key);
    if (ssq) atomicAdd(sumsq + g, ssq);
  }
}

// The vertices a block finds in a level wait in a shared-memory list (warp-aggregated appends) and go to the grid's
// queue a block-width at a time: a push is two block barriers and a round trip to the queue's counter, 2700-3200
// clocks, and one per iteration also kept the iterations' memory trips from overlapping.
// A level that is one iteration of the grid pushes straight away, its rows' offsets read beside the claim: the list
// would only add three barriers and a trip (R-MAT 14 and 17, mixed layouts: 2.05 and 2.59 ms with it, 2.02 and 2.42
// without).
struct KcList {
  uint32_t *v;
  unsigned *n;
  __device__ __forceinline__ void add(bool flag, uint32_t x) const {
    const unsigned bal = __ballot_sync(PHDE_FULL_MASK, flag);
    if (!bal) return;
    const int lane = threadIdx.x & 31;
    unsigned at = 0;
    if (lane == 0) at = atomicAdd(n, (unsigned)__popc(bal));
    at = __shfl_sync(PHDE_FULL_MASK, at, 0) + __popc(bal & ((1u << lane) - 1u));
    if (flag) v[at] = x;
  }
  // every thread of the block; the list is empty after it
  __device__ __forceinline__ void flush(const int64_t *off, uint32_t *qv, uint32_t *qe, uint32_t *qo, ull *ctr,
                                        PushScratch *sc) const {
    __syncthreads();
    const unsigned c = *(volatile unsigned *)n;
    if (c == 0) return;
    for (unsigned i0 = 0; i0 < c; i0 += blockDim.x) {
      const bool has = i0 + threadIdx.x < c;
      uint32_t x = 0, o = 0, d = 0;
      if (has) {
        x = v[i0 + threadIdx.x];
        const int64_t o0 = __ldg(off + x);
        o = (uint32_t)o0;
        d = (uint32_t)(__ldg(off + x + 1) - o0);
      }
      block_push(has, x, d, qv, qe, ctr, sc, qo, o);
    }
    __syncthreads();
    if (threadIdx.x == 0) *n = 0u;
    __syncthreads();
  }
};

__global__ void __launch_bounds__(KC_THREADS) kcenters_bfs_kernel(KcArgs a) {
  __shared__ PushScratch psc;
  __shared__ unsigned s_listed;
  __shared__ uint32_t s_win[KC_THREADS / 32][32];
  __shared__ ull red[32];
  extern __shared__ __align__(16) uint32_t kc_smem[];  // the selection history, the list, the bitmap
  // every block keeps the same history: [P] in shared memory, or for very many passes each block's own in global memory
  uint32_t *s_hist = a.hist ? a.hist + (int64_t)blockIdx.x * a.P : kc_smem;
  const KcList list{kc_smem + (a.hist ? 0 : (a.P + 3) & ~3), &s_listed};
  uint32_t *s_bm = list.v + a.cap;
  const int full = a.cap / KC_THREADS - 1;  // iterations between looks at the list
  if (threadIdx.x == 0) s_listed = 0u;  // barriers of the first pass's start come before its use
  const int64_t n = a.n;
  const int tid = threadIdx.x;
  const int64_t gstride = (int64_t)gridDim.x * blockDim.x;
  const int64_t gbase = (int64_t)blockIdx.x * blockDim.x;
  int64_t src = a.variant == 1 ? a.fixed_src[0] : 0;
  uint32_t step = 0;
  ull edges_local = 0;
  int p0 = 0;
  if (a.resume) {  // go on where the cluster stopped: the same history, from the passes' keys or sources
    p0 = (int)a.resume[0];
    if (p0 >= a.P) return;
    src = a.resume[1];
    for (int i = tid; i < p0; i += blockDim.x)
      s_hist[i] = a.variant == 2 ? (uint32_t)a.sources[i] : 0xffffffffu - (uint32_t)(a.keys[i] & 0xffffffffull);
    __syncthreads();
  }

  for (int p = p0; p < a.P; p++) {
    int32_t *Dp = a.D + (int64_t)p * n;
    int64_t s_off = 0;
    uint32_t sdeg = 0;
    uint32_t f_cnt = 1, f_edges = 0;
    int64_t edges_to_check = a.nnz;
    int32_t L = 0;
    if (a.resume && p == (int)a.resume[0] && a.resume[2] > 0) {
      // a pass that the cluster began: its last level, read back from the column, is the frontier (step is 0).  Where it
      // stopped is read here again: kept in registers across the passes, it cost every level (1 % of a batch's union).
      const int32_t level0 = (int32_t)a.resume[2];
      L = level0;
      edges_to_check -= a.resume[3];
      const bool once = n <= gstride;
      int since = 0;
      for (int64_t base = gbase; base < n; base += gstride) {
        const int64_t v = base + tid;
        const bool f = v < n && Dp[v] == level0;
        const uint32_t bal = __ballot_sync(PHDE_FULL_MASK, f);
        const int64_t v0 = v - (tid & 31);
        if ((tid & 31) == 0 && v0 < n) a.bm[0][v0 >> 5] = bal;
        if (once) {
          uint32_t ov = 0, dv = 0;
          if (f) {
            ov = (uint32_t)__ldg(a.off + v);
            dv = (uint32_t)__ldg(a.off + v + 1) - ov;
          }
          block_push(f, (uint32_t)v, dv, a.qv0, a.qe0, a.qinit, &psc, a.qo0, ov);
          break;
        }
        list.add(f, (uint32_t)v);
        if (++since == full) {
          since = 0;
          __syncthreads();
          if (__syncthreads_or(s_listed > KC_THREADS)) list.flush(a.off, a.qv0, a.qe0, a.qo0, a.qinit, &psc);
        }
      }
      if (!once) list.flush(a.off, a.qv0, a.qe0, a.qo0, a.qinit, &psc);
      ull q;
      if (!grid_sync_read(a.gs, a.err, a.timeout_ns, a.qinit, &q)) return;
      f_cnt = (uint32_t)(q >> 32);
      f_edges = (uint32_t)(q & 0xffffffffull);
    } else if (a.B == 0) {
      if (tid == 0) {
        Dp[src] = 0;
        // the level-0 frontier bitmap holds only the source (the previous pass left it empty)
        atomicOr(a.bm[step % 3] + (src >> 5), 1u << (src & 31));
        if (blockIdx.x == 0) a.sources[p] = src;
      }
      __syncthreads();
      s_off = a.off[src];
      sdeg = (uint32_t)(a.off[src + 1] - s_off);
      f_edges = sdeg;
    } else {
      // batched: block 0 queues every graph's source (vertex 0 of the graph, then the previous pass's
      // farthest vertex) as the level-0 frontier, in graph order
      if (blockIdx.x == 0) {
        if (tid == 0) *a.qinit = 0ull;
        __syncthreads();
        uint32_t *q0v = (step & 1) ? a.qv1 : a.qv0;
        uint32_t *q0e = (step & 1) ? a.qe1 : a.qe0;
        uint32_t *q0o = (step & 1) ? a.qo1 : a.qo0;
        for (int b0 = 0; b0 < a.B; b0 += blockDim.x) {
          const int b = b0 + tid;
          uint32_t v = 0, dv = 0, ov = 0;
          if (b < a.B) {
            v = p == 0 ? (uint32_t)a.vbase[b]
                       : 0xffffffffu - (uint32_t)(__ldcg(a.keys + (int64_t)(p - 1) * a.B + b) & 0xffffffffull);
            ov = (uint32_t)a.off[v];
            dv = (uint32_t)(a.off[v + 1] - a.off[v]);
            Dp[v] = 0;
            atomicOr(a.bm[step % 3] + (v >> 5), 1u << (v & 31));
            a.sources[(int64_t)p * a.B + b] = v;
          }
          block_push(b < a.B, v, dv, q0v, q0e, a.qinit, &psc, q0o, ov);
        }
      }
      ull q;
      if (!grid_sync_read(a.gs, a.err, a.timeout_ns, a.qinit, &q)) return;
      f_cnt = (uint32_t)(q >> 32);
      f_edges = (uint32_t)(q & 0xffffffffull);
    }
    int64_t scout = f_edges;
    bool in_bu = false;
    int64_t awake = 0, old_awake = 0;

    while (f_cnt > 0) {
      if (!in_bu) {
        if (scout > edges_to_check / a.alpha) {
          in_bu = true;
          awake = f_cnt;
        } else {
          edges_to_check -= scout;
        }
      }
      if (in_bu) old_awake = awake;
      const uint32_t *qin_v = (step & 1) ? a.qv1 : a.qv0;
      const uint32_t *qin_e = (step & 1) ? a.qe1 : a.qe0;
      uint32_t *qout_v = (step & 1) ? a.qv0 : a.qv1;
      uint32_t *qout_e = (step & 1) ? a.qe0 : a.qe1;
      const uint32_t *qin_o = (step & 1) ? a.qo1 : a.qo0;
      uint32_t *qout_o = (step & 1) ? a.qo0 : a.qo1;
      ull *octr = a.ctr + (step & 3);
      if (blockIdx.x == 0 && tid == 0) a.ctr[(step + 2) & 3] = 0ull;
      const uint32_t *bm_cur = a.bm[step % 3];
      uint32_t *bm_next = a.bm[(step + 1) % 3];
      {  // the bitmap of the previous level becomes the next level's (empty) output
        uint32_t *bm_clr = a.bm[(step + 2) % 3];
        for (int64_t w = gbase + tid; w < a.W; w += gstride) bm_clr[w] = 0u;
      }

      if (!in_bu) {
        const int64_t E = f_edges;
        const bool once = E <= gstride;
        int since = 0;
        for (int64_t base = gbase; base < E; base += gstride) {
          const int64_t e = base + tid, e0w = base + (tid & ~31);
          bool claimed = false;
          uint32_t v = 0, ov = 0, dv = 0;
          if (e0w < E) {  // warp-uniform
            int64_t j = s_off + e;
            if (L != 0 || a.B != 0) {
              uint32_t es;
              const uint32_t s = warp_owner_slots(qin_e, f_cnt, (uint32_t)e0w, s_win[tid >> 5], es);
              if (e < E) j = (int64_t)qin_o[s] + (e - (int64_t)es);
            }
            if (e < E) {
              v = __ldg(a.adj + j);
              edges_local++;
              if (Dp[v] == -1) {
                if (once) {  // in flight with the CAS
                  ov = (uint32_t)__ldg(a.off + v);
                  dv = (uint32_t)__ldg(a.off + v + 1) - ov;
                }
                if (atomicCAS(Dp + v, -1, L + 1) == -1) {
                  claimed = true;
                  atomicOr(bm_next + (v >> 5), 1u << (v & 31));
                }
              }
            }
            if (!once) list.add(claimed, v);
          }
          if (once) {
            block_push(claimed, v, dv, qout_v, qout_e, octr, &psc, qout_o, ov);
            break;
          }
          if (++since == full) {  // as many more as the list holds for sure
            since = 0;
            __syncthreads();
            if (__syncthreads_or(s_listed > KC_THREADS)) list.flush(a.off, qout_v, qout_e, qout_o, octr, &psc);
          }
        }
        if (!once) list.flush(a.off, qout_v, qout_e, qout_o, octr, &psc);
      } else {
        const bool once = n <= gstride;
        if (a.smem_bm) {
          // 16 bytes per copy, all of a thread's in flight (word by word: 11k clocks for R-MAT 20's 80 KB)
          for (int64_t w = 4 * (int64_t)tid; w < a.W; w += 4 * (int64_t)blockDim.x) cp_async16(s_bm + w, bm_cur + w);
          cp_async_commit();
          cp_async_wait<0>();
          __syncthreads();
        }
        const uint32_t *front = a.smem_bm ? s_bm : bm_cur;
        int since = 0;
        for (int64_t base = gbase; base < n; base += gstride) {
          const int64_t v = base + tid;
          bool found = false;
          uint32_t ov = 0, dv = 0;
          if (v < n && Dp[v] == -1) {
            const int64_t j0 = a.off[v], j1 = a.off[v + 1];
            // four neighbours per round (their adjacency entries, then their bitmap words, all in flight): a
            // vertex far from the frontier tests every neighbour, one dependent L2 round trip each otherwise
            for (int64_t j = j0; j < j1 && !found; j += 4) {
              uint32_t u[4], word[4];
#pragma unroll
              for (int q = 0; q < 4; q++) u[q] = j + q < j1 ? __ldg(a.adj + j + q) : 0u;
#pragma unroll
              for (int q = 0; q < 4; q++)
                word[q] = j + q < j1 ? (a.smem_bm ? front[u[q] >> 5] : __ldcg(front + (u[q] >> 5))) : 0u;
#pragma unroll
              for (int q = 0; q < 4; q++) {
                if (found || j + q >= j1) continue;
                edges_local++;  // counted up to the first frontier neighbour, as a one-at-a-time scan would
                found = (word[q] >> (u[q] & 31)) & 1u;
              }
            }
            if (found) {
              Dp[v] = L + 1;
              ov = (uint32_t)j0;
              dv = (uint32_t)(j1 - j0);
            }
          }
          // one bitmap word per warp: the warp covers 32 consecutive, 32-aligned vertices
          const uint32_t bal = __ballot_sync(PHDE_FULL_MASK, found);
          const int64_t v0 = v - (tid & 31);
          if ((tid & 31) == 0 && v0 < n) bm_next[v0 >> 5] = bal;
          if (once) {
            block_push(found, (uint32_t)v, dv, qout_v, qout_e, octr, &psc, qout_o, ov);
            break;
          }
          list.add(found, (uint32_t)v);
          if (++since == full) {
            since = 0;
            __syncthreads();
            if (__syncthreads_or(s_listed > KC_THREADS)) list.flush(a.off, qout_v, qout_e, qout_o, octr, &psc);
          }
        }
        if (!once) list.flush(a.off, qout_v, qout_e, qout_o, octr, &psc);
      }
      ull out;
      if (!grid_sync_read(a.gs, a.err, a.timeout_ns, octr, &out)) return;
      f_cnt = (uint32_t)(out >> 32);
      f_edges = (uint32_t)(out & 0xffffffffull);
      if (a.trace && blockIdx.x == 0 && tid == 0 && step < (uint32_t)a.trace_cap) {
        ull *tr = a.trace + 4 * (size_t)step;
        tr[0] = global_timer_ns();
        tr[1] = ((ull)p << 40) | ((ull)(uint32_t)L << 32) | (in_bu ? 1ull : 0ull);
        tr[2] = f_cnt;
        tr[3] = f_edges;
      }
      if (in_bu) {
        awake = f_cnt;
        if (!(awake >= old_awake || awake > n / a.beta)) {
          in_bu = false;
          scout = 1;
        }
      } else {
        scout = f_edges;
      }
      L++;
      step++;
    }

    // ---- fold the finished column: min distance, farthest vertex, sum of squares ----
    ull kbest = 0, ssq = 0;
    int bad = 0;
    if (a.B > 0) {  // batched: per-graph keys and sums; the grid-stride loop keeps warps together
      for (int64_t base = gbase; base < n; base += gstride) {
        const int64_t v = base + tid;
        ull key = 0, sq = 0;
        int g = -1;
        const bool valid = v < n;
        if (valid) {
          const int32_t d = Dp[v];
          g = a.gid[v];
          if (d < 0) {
            bad = 1;
          } else {
            sq = (ull)d * (ull)d;
            int32_t m = a.min_d[v];
            if (d < m) {
              m = d;
              a.min_d[v] = m;
            }
            key = ((ull)(uint32_t)m << 32) | (ull)(0xffffffffu - (uint32_t)v);
          }
        }
        batch_fold(a.keys + (int64_t)p * a.B, a.sumsq + (int64_t)p * a.B, g, key, sq, valid);
      }
      if (__syncthreads_or(bad)) {
        if (tid == 0) atomicCAS(a.err, 0, PHDE_ERR_DISCONNECTED);
        return;
      }
      if (p + 1 == a.P) break;
      if (!grid_sync(a.gs, a.err, a.timeout_ns)) return;
      continue;
    }
    for (int64_t v = gbase + tid; v < n; v += gstride) {
      const int32_t d = Dp[v];
      if (d < 0) {
        bad = 1;
        continue;
      }
      ssq += (ull)d * (ull)d;
      if (a.variant != 1) {
        int32_t m = a.min_d[v];
        if (d < m) {
          m = d;
          a.min_d[v] = m;
        }
        const ull key = ((ull)(uint32_t)m << 32) | (ull)(0xffffffffu - (uint32_t)v);
        kbest = key > kbest ? key : kbest;
      }
    }
    if ((a.variant != 1 || a.require_all) && __syncthreads_or(bad)) {
      if (tid == 0) atomicCAS(a.err, 0, PHDE_ERR_DISCONNECTED);
      return;
    }
    ssq = block_sum(ssq, red);
    if (tid == 0) atomicAdd(a.sumsq + p, ssq);
    if (a.variant != 1) {
      kbest = block_max_u64(kbest, red);
      if (tid == 0) atomicMax(a.keys + p, kbest);
    }
    if (p + 1 == a.P) break;
    ull key;
    if (!grid_sync_read(a.gs, a.err, a.timeout_ns, a.keys + p, &key)) return;

    if (a.variant == 1) {
      src = a.fixed_src[p + 1];
      continue;
    }
    const uint32_t raw = 0xffffffffu - (uint32_t)(key & 0xffffffffull);
    const int32_t maxval = (int32_t)(key >> 32);
    int hit = 0;
    for (int i = tid; i < p; i += blockDim.x) hit |= (s_hist[i] == raw);
    hit = __syncthreads_or(hit);
    int64_t next = raw;
    if (p >= 1 && hit) {
      // duplicate fix-up (ParHDE.cpp:144-154 at one thread): highest-index vertex with the same
      // minimum distance that is not in the history
      for (int64_t v = gbase + tid; v < n; v += gstride) {
        if (a.min_d[v] != maxval) continue;
        bool inh = false;
        for (int i = 0; i < p && !inh; i++) inh = (s_hist[i] == (uint32_t)v);
        if (!inh) atomicMax(a.fixkey + p, (ull)v + 1ull);
      }
      ull fk;
      if (!grid_sync_read(a.gs, a.err, a.timeout_ns, a.fixkey + p, &fk)) return;
      if (fk) next = (int64_t)(fk - 1ull);
    }
    __syncthreads();
    if (tid == 0) s_hist[p] = a.variant == 2 ? (uint32_t)src : raw;
    __syncthreads();
    src = next;
  }
  ull etot = block_sum(edges_local, red);
  if (tid == 0 && a.edges) atomicAdd(a.edges, etot);
}

// ---------------------------------------------------------------------------------------------
// Batched Kcenters with one CTA per graph (batches of small graphs).  A grid-wide level barrier costs
// more than a small graph's whole level, and every grid-wide level waits for the deepest graph of the
// batch; here each CTA takes whole graphs from a work list (largest first) and runs their 3k passes with
// block barriers only.  Per pass: a level-synchronous top-down BFS from the pass's source, then the Kcenters
// fold over the graph's vertices (min distance, farthest vertex with the lowest index on ties -- the key
// (min_d << 32) | ~v --, exact sum of squares).
// What bounds a level is its chain of dependent accesses (frontier entry -> offsets -> adjacency -> claim ->
// append), so everything but the CSR stays on the SM: the visited set is a bitmap in shared memory (claims are
// shared-memory ORs), the frontier lists are in shared memory up to qcap entries and spill to the graph's slice
// of the union's queues, distances are written once and never read back inside a level.  2^k lanes share a
// frontier vertex, as many as leave the whole frontier in one round of the CTA.
// Measured, 512 geometric graphs of 1k-200k vertices, 30 passes: 150 -> 49 ms (claims by a global compare-and-swap
// per edge and queues in global memory before); the largest graph alone is 44 ms of it, 2.7 us a level: a round of
// claims and appends by 32 warps about 1000 clocks, two DRAM trips (152 graphs at once do not fit L2) as much again.
// Tried: 32-byte row records of 16-bit index differences in place of offsets and adjacency, 2-10 % slower (the
// extra slots cost more instructions than the saved access).
// Same outputs as the batched variant of kcenters_bfs_kernel: D columns over the union, sources, keys and
// sums indexed [p * B + b].
struct KbArgs {
  const int64_t *off;
  const uint32_t *adj;
  int64_t N;
  int32_t *D;
  int P, B;
  const int64_t *vbase;
  const int32_t *order;  // graphs, largest first
  unsigned *next;        // work-list counter (zeroed)
  int64_t *sources;
  int32_t *min_d;
  ull *sumsq;
  uint32_t *q0, *q1;     // [N] each: frontier vertices beyond qcap
  uint32_t *vis;         // visited bitmaps in global memory when the largest graph's does not fit on the SM:
  int64_t vis_stride;    // vis_stride words per CTA
  int vis_words;         // shared memory: visited words, then two lists of qcap entries
  uint32_t qcap;
  ull *edges;
  int *err;
};

constexpr int KB_THREADS = 1024;

constexpr uint32_t KB_ROUND = 16;  // neighbours of a row per round: one round covers most rows of a geometric graph
constexpr uint32_t KB_ROW = 256;  // neighbours of a row taken by its lane group; the rest by the whole warp

extern __shared__ __align__(16) uint32_t kb_smem[];  // [vis_words] visited, then the two frontier lists

struct KbLevel {
  const uint32_t *gq_in;  // frontier: entry i in kb_smem[s_in + i] below qcap, else in gq_in
  uint32_t *gq_out;
  uint32_t *vis;          // visited bitmap when it is in global memory
  uint32_t s_in, s_out;
  unsigned *c;  // entries appended
  int32_t *Dp;  // the graph's rows of the pass's column
  const int64_t *off;  // the graph's rows
  const uint32_t *adj;
  uint32_t vb, cnt, qcap, src;
  int32_t d;
};

// Shared-memory OR unless `skip`: a predicated instruction, no branch, so that several are in flight at once.
// Returns the word before (all ones where skipped).
__device__ __forceinline__ uint32_t shared_or_unless(uint32_t addr, uint32_t bits, uint32_t skip) {
  uint32_t old;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %3, 0;\n\tmov.u32 %0, 0xffffffff;\n\t"
      "@p atom.shared.or.b32 %0, [%1], %2;\n\t}"
      : "=&r"(old)
      : "r"(addr), "r"(bits), "r"(skip)
      : "memory");
  return old;
}

// Claim the warp's neighbours v[t] (graph-local; a visited vertex where a lane has none) and append the new ones.
template <bool SV, int NB>
__device__ __forceinline__ void kb_claim(const KbLevel &l, const uint32_t (&v)[NB]) {
  const uint32_t *vis = SV ? kb_smem : l.vis;
  const uint32_t vis_s = (uint32_t)__cvta_generic_to_shared(kb_smem);
  const int lane = threadIdx.x & 31;
  uint32_t word[NB], seen = 1;
#pragma unroll
  for (int t = 0; t < NB; t++) word[t] = *(const volatile uint32_t *)(vis + (v[t] >> 5));
#pragma unroll
  for (int t = 0; t < NB; t++) {
    word[t] = __funnelshift_r(word[t], 0u, v[t]);  // shifted to the vertex's bit, here and below
    seen &= word[t];
  }
  if (__all_sync(PHDE_FULL_MASK, seen)) return;
#pragma unroll
  for (int t = 0; t < NB; t++) {  // every OR issued before any of their results is used
    if (SV)
      word[t] = shared_or_unless(vis_s + (v[t] >> 5) * 4u, 1u << (v[t] & 31), word[t] & 1u);
    else
      word[t] = word[t] & 1u ? 0xffffffffu : atomicOr(l.vis + (v[t] >> 5), 1u << (v[t] & 31));
  }
  unsigned bal[NB], total = 0;
#pragma unroll
  for (int t = 0; t < NB; t++) {
    word[t] = __funnelshift_r(word[t], 0xffffffffu, v[t]);
    bal[t] = __ballot_sync(PHDE_FULL_MASK, !(word[t] & 1u));
    total += __popc(bal[t]);
  }
  if (!total) return;
  unsigned base = 0;
  if (lane == 0) base = atomicAdd(l.c, total);
  base = __shfl_sync(PHDE_FULL_MASK, base, 0);
  const unsigned below = (1u << lane) - 1u;
#pragma unroll
  for (int t = 0; t < NB; t++) {
    if (!(word[t] & 1u)) {
      const unsigned slot = base + __popc(bal[t] & below);
      if (slot < l.qcap)
        kb_smem[l.s_out + slot] = v[t];
      else
        l.gq_out[slot] = v[t];
      l.Dp[v[t]] = l.d;
    }
    base += __popc(bal[t]);
  }
}

// One level with G lanes per frontier vertex: up to KB_ROW of its neighbours by the lane group, 16 per round, then
// the rest of long rows one row at a time by the whole warp.
template <bool SV, int G>
__device__ __forceinline__ void kb_level(const KbLevel &l) {
  constexpr int NB = KB_ROUND / G;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  const uint32_t step = blockDim.x / G;
  for (uint32_t i0 = (threadIdx.x & ~31u) / G; i0 < l.cnt; i0 += step) {
    const uint32_t i = i0 + lane / G;
    uint32_t u = l.src, deg = 0;
    int64_t e0 = 0;
    if (i < l.cnt) {
      u = i < l.qcap ? kb_smem[l.s_in + i] : l.gq_in[i];
      const int64_t *o = l.off + u;
      e0 = __ldg(o);
      deg = (uint32_t)(__ldg(o + 1) - e0);
    }
    const uint32_t *row = l.adj + e0;
    const uint32_t own = min(deg, KB_ROW);
    const uint32_t most = __reduce_max_sync(PHDE_FULL_MASK, own);
    for (uint32_t r = 0; r < most; r += KB_ROUND) {
      uint32_t v[NB];
#pragma unroll
      for (int t = 0; t < NB; t++) {
        const uint32_t e = r + t * G + gl;
        v[t] = e < own ? __ldg(row + e) - l.vb : u;
      }
      kb_claim<SV, NB>(l, v);
    }
    for (unsigned big = __ballot_sync(PHDE_FULL_MASK, gl == 0 && deg > KB_ROW); big; big &= big - 1) {
      const int from = __ffs(big) - 1;
      const uint32_t *brow = l.adj + __shfl_sync(PHDE_FULL_MASK, e0, from);
      const uint32_t bd = __shfl_sync(PHDE_FULL_MASK, deg, from);
      for (uint32_t r = KB_ROW; r < bd; r += 128) {
        uint32_t v[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
          const uint32_t e = r + t * 32 + lane;
          v[t] = e < bd ? __ldg(brow + e) - l.vb : u;
        }
        kb_claim<SV, 4>(l, v);
      }
    }
  }
}

template <bool SV>
__global__ void __launch_bounds__(KB_THREADS) kcenters_block_kernel(KbArgs a) {
  __shared__ int s_graph;
  // level L appends through s_c[L % 3]; after the level every thread reads it, and
  // thread 0 clears s_c[(L + 2) % 3] -- last read before this level's final barrier, next used two levels on
  __shared__ unsigned s_c[3];
  __shared__ ull red[32];
  __shared__ int64_t s_src;
  const int tid = threadIdx.x;
  KbLevel l;
  uint32_t *vis = SV ? kb_smem : a.vis + (int64_t)blockIdx.x * a.vis_stride;
  l.vis = vis;
  l.qcap = a.qcap;
  l.adj = a.adj;
  ull edges_local = 0;
  for (;;) {
    if (tid == 0) s_graph = (int)atomicAdd(a.next, 1u);
    __syncthreads();
    const int gi = s_graph;
    __syncthreads();
    if (gi >= a.B) break;
    const int b = a.order[gi];
    const int64_t vb = a.vbase[b], nb = a.vbase[b + 1] - vb;
    const int words = (int)((nb + 31) >> 5);
    l.vb = (uint32_t)vb;
    l.off = a.off + vb;
    uint32_t src = 0;  // Kcenters starts at the graph's vertex 0
    for (int p = 0; p < a.P; p++) {
      for (int w = tid; w < words; w += blockDim.x) vis[w] = 0u;
      __syncthreads();
      l.Dp = a.D + (int64_t)p * a.N + vb;
      l.s_in = (uint32_t)a.vis_words;
      l.s_out = (uint32_t)a.vis_words + a.qcap;
      l.gq_in = a.q0 + vb;
      l.gq_out = a.q1 + vb;
      l.cnt = 1;
      l.d = 0;
      l.src = src;
      edges_local += a.off[vb + nb] - a.off[vb];  // a connected graph's pass reads every row once
      if (tid == 0) {
        vis[src >> 5] = 1u << (src & 31);
        l.Dp[src] = 0;
        kb_smem[a.vis_words] = src;
        s_c[0] = 0u;
        s_c[1] = 0u;
      }
      int64_t reached = 1;
      int ring = 0;
      __syncthreads();
      while (l.cnt > 0) {
        l.c = s_c + ring;
        l.d++;
        if (l.cnt * 8 <= blockDim.x)
          kb_level<SV, 8>(l);
        else if (l.cnt * 4 <= blockDim.x)
          kb_level<SV, 4>(l);
        else
          kb_level<SV, 2>(l);
        __syncthreads();
        l.cnt = *(volatile unsigned *)l.c;
        reached += l.cnt;
        if (tid == 0) s_c[ring == 0 ? 2 : ring - 1] = 0u;
        ring = ring == 2 ? 0 : ring + 1;
        const uint32_t s = l.s_in;
        l.s_in = l.s_out;
        l.s_out = s;
        uint32_t *g = (uint32_t *)l.gq_in;
        l.gq_in = l.gq_out;
        l.gq_out = g;
      }
      if (reached < nb) {
        if (tid == 0) atomicCAS(a.err, 0, PHDE_ERR_DISCONNECTED);
        break;
      }
      // fold: min distance, farthest vertex (lowest index on ties), exact sum of squares
      ull kbest = 0, ssq = 0;
      int32_t *mind = a.min_d + vb;
      for (int64_t v0 = tid; v0 < nb; v0 += 8 * (int64_t)blockDim.x) {
        int32_t d[8], m[8];
#pragma unroll
        for (int t = 0; t < 8; t++) {
          const int64_t v = v0 + t * (int64_t)blockDim.x;
          d[t] = v < nb ? __ldcg(l.Dp + v) : 0;
          m[t] = v < nb ? __ldcg(mind + v) : -1;
        }
#pragma unroll
        for (int t = 0; t < 8; t++) {
          const int64_t v = v0 + t * (int64_t)blockDim.x;
          if (v >= nb) continue;
          ssq += (ull)d[t] * (ull)d[t];
          if (d[t] < m[t]) mind[v] = m[t] = d[t];
          const ull key = ((ull)(uint32_t)m[t] << 32) | (ull)(0xffffffffu - (uint32_t)(vb + v));
          kbest = key > kbest ? key : kbest;
        }
      }
      ssq = block_sum(ssq, red);
      kbest = block_max_u64(kbest, red);
      if (tid == 0) {
        a.sumsq[(int64_t)p * a.B + b] = ssq;
        a.sources[(int64_t)p * a.B + b] = vb + src;
        s_src = (int64_t)(0xffffffffu - (uint32_t)(kbest & 0xffffffffull)) - vb;
      }
      __syncthreads();
      src = (uint32_t)s_src;
    }
    __syncthreads();
  }
  if (tid == 0 && a.edges) atomicAdd(a.edges, edges_local);
}

// ---------------------------------------------------------------------------------------------
// Kcenters on one thread-block cluster, for graphs whose levels are narrow (meshes, geometric graphs: hundreds of
// levels of a few hundred vertices).  There a level of kcenters_bfs_kernel is a chain of latencies -- the grid
// barrier, the frontier queue, offsets, adjacency, claim and append, each through L2 -- of about 4-5 us whatever
// it finds.  Here the search state lives in the shared memory of the cluster's CTAs: 32-vertex words are dealt to
// the CTAs in turn, the owner of a word keeps its visited word, two next-frontier words (the levels alternate) and
// its rows' starts; a level is
//   expand   the CTA's frontier vertices (a list in shared memory) send one remote OR per neighbour to the owner's
//            next-frontier word -- no value returned, so nothing waits for it --;
//   barrier  of the cluster (hardware, ~0.25 us), which also orders the ORs;
//   scan     the owner takes next & ~visited of its words: new vertices, their distances and its next list.
// Only the adjacency is read from L2.  Every CTA posts its frontier's size to all others before the barrier, so all
// see the same total: 0 ends the pass, more than `limit` (a wide level: the whole grid is faster) leaves the
// kernel, and kcenters_bfs_kernel, launched after it, goes on from that level: it reads the level's vertices back from
// the distance column.
// Sources, history and duplicate fix-up as in kcenters_bfs_kernel; distances are unique, so the results are equal.
// Measured (16 CTAs of 512 threads): a level was 3100 clocks on the 125 x 125 mesh (expand 840, barrier with the ORs in
// flight 1240, scan 990) and 4000 on a 150k-vertex 2-D geometric graph before the words were dealt to the scanning
// warps in turn and the listed rows prefetched (4 % less); whole layouts 21.4 -> 6.4 ms and 139 -> 40.6 ms.
// 8 CTAs: 7.7 and 54 ms; 256 threads: 7.2 and 50 ms; 1024 threads: 5 and 2 % slower.
struct KlArgs {
  const int64_t *off;
  const uint32_t *adj;
  int64_t n;
  int32_t *D;
  int P, variant, require_all;
  const int64_t *fixed_src;
  int64_t *sources;
  int32_t *min_d;
  ull *sumsq, *keys, *edges;
  int *err;
  // [5]: passes finished; of the next one its source, the level it stopped at (0: not begun) and the edges of the
  // levels before that; 0, the counter of the queue that kcenters_bfs_kernel makes of that level
  int64_t *resume;
  int words;         // words owned by a CTA
  int rows;          // row starts in shared memory
  uint32_t limit;
};

constexpr int KL_THREADS = 512;
constexpr int KL_MAX_CLUSTER = 16;
constexpr uint32_t KL_LIST = 4096;   // frontier entries of a CTA; the limit of a level's total as well
constexpr uint32_t KL_ROW = 512;     // longer rows are taken by the whole CTA

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The shared-memory address of CTA `rank`'s copy of a local address.
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void remote_or(uint32_t addr, uint32_t v) {
  asm volatile("red.relaxed.cluster.shared::cluster.or.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void remote_st32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void remote_st64(uint32_t addr, ull v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

struct KlLevel {
  const int64_t *off;
  const uint32_t *adj;
  const uint32_t *rs;    // row starts, 33 per word (null: from off)
  const uint2 *list;     // the CTA's frontier: row start and length
  uint32_t next;         // shared address of the level's next-frontier words
  uint32_t cnt, rank, cmask, clog, pitch;
};

// Place of the CTA's word w in its bitmaps: the words of scanning warp w % KL_WARPS side by side, so that neighbouring
// words, which a wave fills together, go to different warps.
constexpr int KL_WARPS = KL_THREADS / 32;
__device__ __forceinline__ uint32_t kl_place(uint32_t w, uint32_t pitch) {
  return (w % KL_WARPS) * pitch + w / KL_WARPS;
}

__device__ __forceinline__ uint32_t kl_vertex(const KlLevel &l, uint32_t x) {
  return (((x >> 5) << l.clog | l.rank) << 5) | (x & 31);
}
__device__ __forceinline__ void kl_send(const KlLevel &l, uint32_t v) {
  const uint32_t w = v >> 5;
  remote_or(map_rank(l.next + (kl_place(w >> l.clog, l.pitch) << 2), w & l.cmask), 1u << (v & 31));
}
__device__ __forceinline__ uint2 kl_row(const KlLevel &l, uint32_t x) {
  if (l.rs) {
    const uint32_t *r = l.rs + (x >> 5) * 33 + (x & 31);
    return make_uint2(r[0], r[1] - r[0]);
  }
  const int64_t *o = l.off + kl_vertex(l, x);
  const int64_t e0 = __ldg(o);
  return make_uint2((uint32_t)e0, (uint32_t)(__ldg(o + 1) - e0));
}

// Rows of at most KL_ROW neighbours with G lanes per frontier vertex, 16 neighbours per group and round.
template <int G>
__device__ __forceinline__ void kl_expand(const KlLevel &l, uint32_t &edges) {
  constexpr int NB = 16 / G;
  const uint32_t gl = threadIdx.x & (G - 1);
  for (uint32_t i = threadIdx.x / G; i < l.cnt; i += KL_THREADS / G) {
    const uint2 x = l.list[i];
    const uint32_t deg = x.y;
    if (deg > KL_ROW) continue;
    if (gl == 0) edges += deg;
    const uint32_t *row = l.adj + x.x;
    for (uint32_t r = gl; r < deg; r += 16) {
      uint32_t v[NB];
#pragma unroll
      for (int t = 0; t < NB; t++) v[t] = r + t * G < deg ? __ldg(row + r + t * G) : 0xffffffffu;
#pragma unroll
      for (int t = 0; t < NB; t++)
        if (v[t] != 0xffffffffu) kl_send(l, v[t]);
    }
  }
}

// The cluster's maximum of every CTA's `mine` (thread 0's value counts); `slots` is a shared array of ranks.
__device__ __forceinline__ ull cluster_max(ull mine, ull *slots, uint32_t rank, uint32_t C) {
  if (threadIdx.x < C)
    remote_st64(map_rank((uint32_t)__cvta_generic_to_shared(slots + rank), threadIdx.x), mine);
  cluster_barrier();
  ull m = 0;
  for (uint32_t r = 0; r < C; r++) m = slots[r] > m ? slots[r] : m;
  return m;
}

__global__ void __launch_bounds__(KL_THREADS, 1) kcenters_cluster_kernel(KlArgs a) {
  extern __shared__ __align__(16) uint32_t kl_smem[];  // list, visited, next[2], (row starts), history
  __shared__ uint32_t s_counts[2][KL_MAX_CLUSTER];
  __shared__ ull s_keys[KL_MAX_CLUSTER], s_sums[KL_MAX_CLUSTER], s_fix[KL_MAX_CLUSTER];
  // of the two levels in turn: vertices listed, and whether a listed row is longer than KL_ROW
  __shared__ uint32_t s_cnt[2], s_long[2];
  __shared__ ull red[32];
  const uint32_t tid = threadIdx.x, rank = cluster_rank(), C = cluster_size();
  const int words = a.words, warp = tid >> 5, lane = tid & 31;
  const int pitch = words / KL_WARPS;  // words of a warp (words is a multiple of KL_WARPS)
  uint32_t *vis = kl_smem + 2 * KL_LIST, *next = vis + words;
  uint32_t *rs = vis + 3 * words;
  uint2 *list = (uint2 *)kl_smem;
  uint32_t *hist = rs + (a.rows ? 33 * words : 0);
  KlLevel l;
  l.off = a.off;
  l.adj = a.adj;
  l.rs = a.rows ? rs : nullptr;
  l.list = list;
  l.rank = rank;
  l.cmask = C - 1;
  l.clog = 31 - __clz((int)C);
  l.pitch = (uint32_t)pitch;
  if (a.rows)
    for (int i = tid; i < 33 * words; i += KL_THREADS) {
      const int64_t v = ((((int64_t)(i / 33) << l.clog) | rank) << 5) + i % 33;
      rs[i] = (uint32_t)a.off[v < a.n ? v : a.n];
    }
  const uint32_t next_s = (uint32_t)__cvta_generic_to_shared(next);
  uint32_t edges = 0;
  ull edges_all = 0;
  int64_t src = a.variant == 1 ? a.fixed_src[0] : 0;
  if (tid == 0 && rank == 0) a.resume[3] = a.resume[4] = 0;
  for (int p = 0; p < a.P; p++) {
    int32_t *Dp = a.D + (int64_t)p * a.n;
    for (int w = tid; w < 3 * words; w += KL_THREADS) vis[w] = 0u;
    const bool mine = (((uint32_t)(src >> 5)) & l.cmask) == rank;
    const uint32_t sx = (uint32_t)(((src >> 5) >> l.clog) << 5 | (src & 31));
    if (tid == 0) s_long[1] = mine;
    __syncthreads();
    if (tid == 0 && mine) {
      vis[kl_place(sx >> 5, l.pitch)] = 1u << (sx & 31);
      list[0] = kl_row(l, sx);
      Dp[src] = 0;
    }
    if (tid == 0 && rank == 0) a.sources[p] = src;
    cluster_barrier();  // every CTA's words are clear
    l.cnt = mine ? 1u : 0u;
    uint32_t L = 0;
    bool wide = false;
    for (;;) {
      const uint32_t par = L & 1;
      l.next = next_s + par * 4u * words;
      // ---- expand ----
      if (tid == 0) {  // for the scan after the barrier; what the last scan left is in the other place
        s_cnt[par] = 0u;
        s_long[par] = 0u;
      }
      if (tid >= KL_THREADS - 32) {  // the last warp posts the count: it has no rows to expand in a narrow level
        const uint32_t r = tid - (KL_THREADS - 32);
        if (r < C) remote_st32(map_rank((uint32_t)__cvta_generic_to_shared(&s_counts[par][rank]), r), l.cnt);
      }
      if (l.cnt <= KL_LIST) {
        if (l.cnt * 16 <= KL_THREADS)
          kl_expand<16>(l, edges);
        else if (l.cnt * 8 <= KL_THREADS)
          kl_expand<8>(l, edges);
        else
          kl_expand<4>(l, edges);
        if (s_long[par ^ 1]) {  // rows above KL_ROW, one at a time (set by the scan that listed them, or for the source)
          for (uint32_t i = 0; i < l.cnt; i++) {
            const uint2 x = list[i];
            if (x.y <= KL_ROW) continue;
            if (tid == 0) edges += x.y;
            for (uint32_t e = tid; e < x.y; e += KL_THREADS) kl_send(l, __ldg(a.adj + x.x + e));
          }
        }
      }
      cluster_barrier();
      const uint32_t total = __reduce_add_sync(PHDE_FULL_MASK, lane < (int)C ? s_counts[par][lane] : 0u);
      if (total == 0) break;
      if (total > a.limit) {
        wide = true;
        break;
      }
      // ---- scan: level L + 1 ----
      L++;
      // the new vertices of each word are listed by a warp together (a lane per bit): a wave that runs along the
      // numbering fills whole words, and one thread per word took 2000-2700 clocks a level
      uint32_t *nx = next + par * words;
      for (int i0 = 0; i0 < pitch; i0 += 32) {
        const int at0 = warp * pitch + i0 + lane;
        uint32_t nw = 0, slot = 0;
        if (i0 + lane < pitch) {
          nw = nx[at0];
          if (nw) {
            nx[at0] = 0u;
            const uint32_t seen = vis[at0];
            nw &= ~seen;
            vis[at0] = seen | nw;
            if (nw) slot = atomicAdd(&s_cnt[par], (uint32_t)__popc(nw));
          }
        }
        bool longrow = false;
        for (unsigned some = __ballot_sync(PHDE_FULL_MASK, nw != 0u); some; some &= some - 1) {
          const int j = __ffs(some) - 1;
          const uint32_t bits = __shfl_sync(PHDE_FULL_MASK, nw, j);
          const uint32_t at = __shfl_sync(PHDE_FULL_MASK, slot, j) + __popc(bits & ((1u << lane) - 1u));
          if (!((bits >> lane) & 1u)) continue;
          const uint32_t y = (((uint32_t)(i0 + j) * KL_WARPS + warp) << 5) | lane;
          Dp[kl_vertex(l, y)] = (int32_t)L;
          if (at >= KL_LIST) continue;
          const uint2 row = kl_row(l, y);
          list[at] = row;
          longrow |= row.y > KL_ROW;
          // read after the block's barrier; an empty row may start past the array (a directed graph's last vertices): a
          // select, as a branch here is 2 % of a geometric graph's passes
          asm volatile("prefetch.global.L1 [%0];" ::"l"(a.adj + (row.y ? row.x : 0u)));
        }
        if (longrow) s_long[par] = 1u;
      }
      __syncthreads();
      l.cnt = *(volatile uint32_t *)&s_cnt[par];
    }
    edges_all += edges;
    if (wide) {  // leave the rest of the pass to the whole grid, which expands level L again
      ull e = edges;  // summed modulo 2^64: without the rows of level L, which a CTA expanded where its list held them
      if (l.cnt <= KL_LIST)
        for (uint32_t i = tid; i < l.cnt; i += KL_THREADS) {
          e -= list[i].y;
          edges_all -= list[i].y;
        }
      e = block_sum(e, red);
      if (tid == 0) atomicAdd((ull *)a.resume + 3, e);
      if (tid == 0 && rank == 0) {
        a.resume[0] = p;
        a.resume[1] = src;
        a.resume[2] = L;
      }
      break;
    }
    edges = 0;
    // ---- fold the CTA's vertices: min distance, farthest vertex, sum of squares ----
    ull kbest = 0, ssq = 0;
    int bad = 0;
    for (int i0 = tid; i0 < 32 * words; i0 += 4 * KL_THREADS) {
      int32_t d[4], m[4];
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const int i = i0 + t * KL_THREADS;
        const int64_t v = ((((int64_t)(i >> 5) << l.clog) | rank) << 5) | (i & 31);
        const bool ok = i < 32 * words && v < a.n;
        const bool seen = ok && ((vis[kl_place(i >> 5, l.pitch)] >> (i & 31)) & 1u);
        if (ok && !seen) {
          bad = 1;
          Dp[v] = -1;
        }
        d[t] = seen ? __ldcg(Dp + v) : -1;
        m[t] = seen && a.variant != 1 ? __ldcg(a.min_d + v) : 0;
      }
#pragma unroll
      for (int t = 0; t < 4; t++) {
        if (d[t] < 0) continue;
        const int i = i0 + t * KL_THREADS;
        const int64_t v = ((((int64_t)(i >> 5) << l.clog) | rank) << 5) | (i & 31);
        ssq += (ull)d[t] * (ull)d[t];
        if (a.variant == 1) continue;
        if (d[t] < m[t]) a.min_d[v] = m[t] = d[t];
        const ull key = ((ull)(uint32_t)m[t] << 32) | (ull)(0xffffffffu - (uint32_t)v);
        kbest = key > kbest ? key : kbest;
      }
    }
    bad = __syncthreads_or(bad);
    ssq = block_sum(ssq, red);
    kbest = block_max_u64(kbest, red);
    if (bad && (a.variant != 1 || a.require_all)) kbest = ~0ull;  // no key has every bit set
    if (tid < C) remote_st64(map_rank((uint32_t)__cvta_generic_to_shared(s_sums + rank), tid), ssq);
    const ull key = cluster_max(kbest, s_keys, rank, C);
    if (key == ~0ull) {
      if (tid == 0) atomicCAS(a.err, 0, PHDE_ERR_DISCONNECTED);
      if (tid == 0 && rank == 0) a.resume[0] = a.P;
      break;
    }
    if (tid == 0 && rank == 0) {
      ull s = 0;
      for (uint32_t r = 0; r < C; r++) s += s_sums[r];
      a.sumsq[p] = s;
      a.keys[p] = key;
      a.resume[0] = p + 1;
      a.resume[2] = 0;
    }
    if (p + 1 == a.P) break;
    if (a.variant == 1) {
      src = a.fixed_src[p + 1];
      continue;
    }
    const uint32_t raw = 0xffffffffu - (uint32_t)(key & 0xffffffffull);
    const int32_t maxval = (int32_t)(key >> 32);
    int hit = 0;
    for (int i = tid; i < p; i += KL_THREADS) hit |= hist[i] == raw;
    hit = __syncthreads_or(hit);
    int64_t nsrc = raw;
    if (hit) {  // the highest-index vertex with the same minimum distance that is not in the history
      ull best = 0;
      for (int i = tid; i < 32 * words; i += KL_THREADS) {
        const int64_t v = ((((int64_t)(i >> 5) << l.clog) | rank) << 5) | (i & 31);
        if (v >= a.n || a.min_d[v] != maxval) continue;
        bool inh = false;
        for (int q = 0; q < p && !inh; q++) inh = hist[q] == (uint32_t)v;
        if (!inh) best = (ull)v + 1ull;
      }
      best = block_max_u64(best, red);
      best = cluster_max(best, s_fix, rank, C);
      if (best) nsrc = (int64_t)(best - 1ull);
    }
    __syncthreads();
    if (tid == 0) hist[p] = a.variant == 2 ? (uint32_t)src : raw;
    src = nsrc;
  }
  cluster_barrier();  // no CTA leaves while another may still write to its shared memory
  edges_all = block_sum(edges_all, red);
  if (tid == 0 && a.edges) atomicAdd(a.edges, edges_all);
}

__global__ void fill_i32_kernel(int32_t *p, int64_t n, int32_t v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) p[i] = v;
}

}  // namespace

int phde_fill_i32(phde_ctx *ctx, int32_t *p, int64_t n, int32_t v) {
  int blocks = (int)std::min<int64_t>((n + 255) / 256, (int64_t)ctx->nsm * 8);
  if (blocks < 1) blocks = 1;
  fill_i32_kernel<<<blocks, 256, 0, ctx->stream>>>(p, n, v);
  PHDE_LAUNCHED(ctx);
  return PHDE_OK;
}

// The passes on one cluster first, where the graph may have narrow levels and its bitmaps fit the cluster's shared
// memory; g.resume tells the whole-grid kernel what is left.  Average degree above KL_DEGREE: scale-free graphs,
// whose second or third level is most of the graph.  More than KL_VERTICES: every level scans the CTAs' words, whose
// number grows with the graph, and the grid alone is as fast from 4 million on (four passes, grid alone against cluster:
// meshes of 1.0, 2.0, 2.9, 4.0 and 5.8 million vertices 25.8 / 15.0, 37.4 / 27.7, 47.9 / 41.2, 56.9 / 55.5 and
// 69.7 / 84.9 ms; one source in the middle of the 4-million mesh 12.4 / 13.7, of 3 million in 2-D 9.7 / 9.6).
// The width at which a pass moves to the grid is the list's size: smaller ones were never faster up to a million vertices
// (12 passes at 1024, 2048, 3072 and 4096: 60k in 3-D 3.73, 3.71, 2.58, 2.58 ms; 60^3 grid 9.97, 9.95, 8.98, 5.55).
constexpr int64_t KL_DEGREE = 24;
constexpr int64_t KL_VERTICES = (int64_t)3 << 20;

static int run_cluster_passes(phde_ctx *ctx, KcArgs &g) {
  if (g.nnz > KL_DEGREE * g.n || g.n > KL_VERTICES) return PHDE_OK;
  const auto kernel = kcenters_cluster_kernel;
  int C = KL_MAX_CLUSTER;
  KlArgs a;
  size_t smem = 0;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  cfg.blockDim = dim3(KL_THREADS);
  cfg.stream = ctx->stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  PHDE_CK(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  for (;; C /= 2) {  // 16 CTAs, or 8 where the device cannot place 16
    if (C < 8) return PHDE_OK;
    a.words = (int)((g.W + C * KL_WARPS - 1) / (C * KL_WARPS)) * KL_WARPS;
    const size_t fixed = sizeof(uint2) * KL_LIST + sizeof(uint32_t) * (size_t)((g.P + 3) & ~3);
    const size_t room = 224 * 1024;
    a.rows = fixed + sizeof(uint32_t) * 36 * (size_t)a.words <= room;
    smem = fixed + sizeof(uint32_t) * (a.rows ? 36 : 3) * (size_t)a.words;
    if (smem > room) return PHDE_OK;
    if (int arc = phde_allow_smem(ctx, (const void *)kernel)) return arc;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(C);
    cfg.dynamicSmemBytes = smem;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) == cudaSuccess && fit >= 1) break;
    cudaGetLastError();
  }
  int64_t *res = (int64_t *)phde_buf(ctx, "kl.resume", sizeof(int64_t) * 5);
  if (!res) return PHDE_ERR_OOM;
  a.off = g.off;
  a.adj = g.adj;
  a.n = g.n;
  a.D = g.D;
  a.P = g.P;
  a.variant = g.variant;
  a.require_all = g.require_all;
  a.fixed_src = g.fixed_src;
  a.sources = g.sources;
  a.min_d = g.min_d;
  a.sumsq = g.sumsq;
  a.keys = g.keys;
  a.edges = g.edges;
  a.err = g.err;
  a.resume = res;
  a.limit = KL_LIST;
  PHDE_CK(ctx, cudaLaunchKernelEx(&cfg, kernel, a));
  PHDE_LAUNCHED(ctx);
  g.resume = res;
  g.qinit = (ull *)(res + 4);
  return PHDE_OK;
}

int phde_run_bfs_passes(phde_ctx *ctx, int P, int variant, const int64_t *d_fixed_src, int32_t *d_D,
                        int64_t *d_sources, unsigned long long *d_sumsq, unsigned long long *d_edges, int require_all) {
  const int64_t n = ctx->n;
  if (ctx->nnz >= (int64_t)0xffffffffll || n >= (int64_t)0xffffffffll)
    return phde_fail(ctx, PHDE_ERR_INVALID, "graphs with 2^32 or more vertices or adjacency entries are not supported");
  // variant 3: batched ParHDE Kcenters over the uploaded batch (per-graph sources, keys and sums)
  const int B = variant == 3 ? ctx->batch_B : 0;
  if (variant == 3 && B < 1) return phde_fail(ctx, PHDE_ERR_INVALID, "no batch uploaded");
  const int64_t PB = (int64_t)P * (B ? B : 1);
  int32_t *min_d = (int32_t *)phde_buf(ctx, "kc.min_d", sizeof(int32_t) * n);
  ull *keys = (ull *)phde_buf(ctx, "kc.keys", sizeof(ull) * PB);
  ull *fixkey = (ull *)phde_buf(ctx, "kc.fixkey", sizeof(ull) * P);
  ull *qinit = (ull *)phde_buf(ctx, "kc.qinit", sizeof(ull));
  uint32_t *qv0 = (uint32_t *)phde_buf(ctx, "q.v0", sizeof(uint32_t) * n);
  uint32_t *qv1 = (uint32_t *)phde_buf(ctx, "q.v1", sizeof(uint32_t) * n);
  uint32_t *qe0 = (uint32_t *)phde_buf(ctx, "q.e0", sizeof(uint32_t) * n);
  uint32_t *qe1 = (uint32_t *)phde_buf(ctx, "q.e1", sizeof(uint32_t) * n);
  uint32_t *qo0 = (uint32_t *)phde_buf(ctx, "kc.qo0", sizeof(uint32_t) * n);
  uint32_t *qo1 = (uint32_t *)phde_buf(ctx, "kc.qo1", sizeof(uint32_t) * n);
  ull *ctr = (ull *)phde_buf(ctx, "q.ctr", sizeof(ull) * 4);
  const int64_t W = ((n + 31) / 32 + 3) & ~(int64_t)3;  // whole 16-byte pieces
  uint32_t *bms = (uint32_t *)phde_buf(ctx, "kc.bitmaps", sizeof(uint32_t) * 3 * W);
  if (!bms) return PHDE_ERR_OOM;
  PHDE_CK(ctx, cudaMemsetAsync(bms, 0, sizeof(uint32_t) * 3 * W, ctx->stream));
  if (!min_d || !keys || !fixkey || !qinit || !qv0 || !qv1 || !qe0 || !qe1 || !qo0 || !qo1 || !ctr) return PHDE_ERR_OOM;

  PHDE_CK(ctx, cudaMemsetAsync(d_D, 0xff, sizeof(int32_t) * (size_t)n * (size_t)P, ctx->stream));
  PHDE_CK(ctx, cudaMemsetAsync(keys, 0, sizeof(ull) * PB, ctx->stream));
  PHDE_CK(ctx, cudaMemsetAsync(fixkey, 0, sizeof(ull) * P, ctx->stream));
  PHDE_CK(ctx, cudaMemsetAsync(ctr, 0, sizeof(ull) * 4, ctx->stream));
  PHDE_CK(ctx, cudaMemsetAsync(d_sumsq, 0, sizeof(ull) * PB, ctx->stream));
  int rc = phde_fill_i32(ctx, min_d, n, 0x7fffffff);
  if (rc) return rc;
  if ((rc = phde_reset_sync(ctx))) return rc;

  int per_sm = 0;
  // shared memory: the selection history, the list of new vertices, then the frontier bitmap up to KC_SMEM; one block per
  // SM (its registers are the SM's)
  const int cap = 4 * KC_THREADS;
  uint32_t *hist = nullptr;
  if (P > KC_HISTORY) {
    hist = (uint32_t *)phde_buf(ctx, "kc.hist", sizeof(uint32_t) * (size_t)P * ctx->nsm);
    if (!hist) return PHDE_ERR_OOM;
  }
  const size_t fixed = sizeof(uint32_t) * (size_t)((hist ? 0 : (P + 3) & ~3) + cap);
  const size_t bm_bytes = sizeof(uint32_t) * (size_t)W;
  const int smem_bm = fixed + bm_bytes <= KC_SMEM;
  const size_t smem = fixed + (smem_bm ? bm_bytes : 0);
  if (int arc = phde_allow_smem(ctx, (const void *)kcenters_bfs_kernel)) return arc;
  PHDE_CK(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kcenters_bfs_kernel, KC_THREADS, smem));
  if (per_sm < 1) return phde_fail(ctx, PHDE_ERR_CUDA, "kcenters kernel cannot be resident");
  KcArgs a;
  a.off = ctx->d_off;
  a.adj = ctx->d_adj;
  a.n = n;
  a.nnz = ctx->nnz;
  a.D = d_D;
  a.P = P;
  a.variant = variant == 3 ? 0 : variant;
  a.B = B;
  a.vbase = ctx->d_vbase;
  a.gid = ctx->d_gid;
  a.qinit = qinit;
  a.require_all = require_all || variant != 1;
  a.fixed_src = d_fixed_src;
  a.sources = d_sources;
  a.min_d = min_d;
  a.sumsq = d_sumsq;
  a.keys = keys;
  a.fixkey = fixkey;
  a.qv0 = qv0;
  a.qv1 = qv1;
  a.qe0 = qe0;
  a.qe1 = qe1;
  a.qo0 = qo0;
  a.qo1 = qo1;
  a.ctr = ctr;
  a.bm[0] = bms;
  a.bm[1] = bms + W;
  a.bm[2] = bms + 2 * W;
  a.W = W;
  a.smem_bm = smem_bm;
  a.cap = cap;
  a.hist = hist;
  a.edges = d_edges;
  // PHDE_BFS_TRACE=<file>: write the per-level timeline of this launch as CSV after it completes
  const char *trace_file = getenv("PHDE_BFS_TRACE");
  const int trace_cap = 1 << 16;
  a.trace = nullptr;
  a.trace_cap = 0;
  if (trace_file) {
    a.trace = (ull *)phde_buf(ctx, "kc.trace", sizeof(ull) * 4 * trace_cap);
    if (a.trace) {
      PHDE_CK(ctx, cudaMemsetAsync(a.trace, 0, sizeof(ull) * 4 * trace_cap, ctx->stream));
      a.trace_cap = trace_cap;
    }
  }
  a.gs = ctx->d_sync;
  a.err = ctx->d_err;
  a.timeout_ns = ctx->timeout_ns;
  a.alpha = 6;
  a.beta = 18;
  void *args[] = {&a};
  cudaEventRecord(ctx->kev[0], ctx->stream);
  a.resume = nullptr;
  // a traced call keeps every pass in the kernel that writes the timeline
  if (B == 0 && !a.trace && (rc = run_cluster_passes(ctx, a))) return rc;
  PHDE_CK(ctx, cudaLaunchCooperativeKernel((const void *)kcenters_bfs_kernel, dim3(ctx->nsm), dim3(KC_THREADS), args,
                                           smem, ctx->stream));
  PHDE_LAUNCHED(ctx);
  cudaEventRecord(ctx->kev[1], ctx->stream);
  ctx->kev_pending = true;
  if (a.trace) {
    std::vector<ull> h((size_t)4 * trace_cap);
    PHDE_CK(ctx, cudaMemcpyAsync(h.data(), a.trace, sizeof(ull) * 4 * trace_cap, cudaMemcpyDeviceToHost, ctx->stream));
    PHDE_CK(ctx, cudaStreamSynchronize(ctx->stream));
    if (FILE *f = fopen(trace_file, "w")) {
      fprintf(f, "step,t_ns,pass,level,bottom_up,frontier,frontier_edges\n");
      for (int i = 0; i < trace_cap && h[4 * i]; i++)
        fprintf(f, "%d,%llu,%llu,%llu,%llu,%llu,%llu\n", i, h[4 * i], h[4 * i + 1] >> 40, (h[4 * i + 1] >> 32) & 0xff,
                h[4 * i + 1] & 1, h[4 * i + 2], h[4 * i + 3]);
      fclose(f);
    }
  }
  return PHDE_OK;
}

// Batched Kcenters, one CTA per graph (see kcenters_block_kernel).  d_order lists the graphs largest first.
int phde_run_bfs_batched_blocks(phde_ctx *ctx, int P, const int32_t *d_order, int32_t *d_D, int64_t *d_sources,
                                unsigned long long *d_sumsq, unsigned long long *d_edges) {
  const int64_t N = ctx->n;
  const int B = ctx->batch_B;
  int32_t *min_d = (int32_t *)phde_buf(ctx, "kc.min_d", sizeof(int32_t) * N);
  uint32_t *q0 = (uint32_t *)phde_buf(ctx, "q.v0", sizeof(uint32_t) * N);
  uint32_t *q1 = (uint32_t *)phde_buf(ctx, "q.v1", sizeof(uint32_t) * N);
  unsigned *next = (unsigned *)phde_buf(ctx, "kb.next", sizeof(unsigned));
  if (!min_d || !q0 || !q1 || !next) return PHDE_ERR_OOM;
  PHDE_CK(ctx, cudaMemsetAsync(next, 0, sizeof(unsigned), ctx->stream));
  int rc = phde_fill_i32(ctx, min_d, N, 0x7fffffff);
  if (rc) return rc;
  // the context's error word: what an earlier call left there, or a new context's memory, is not this call's
  if ((rc = phde_reset_sync(ctx))) return rc;
  KbArgs a;
  a.off = ctx->d_off;
  a.adj = ctx->d_adj;
  a.N = N;
  a.D = d_D;
  a.P = P;
  a.B = B;
  a.vbase = ctx->d_vbase;
  a.order = d_order;
  a.next = next;
  a.sources = d_sources;
  a.min_d = min_d;
  a.sumsq = d_sumsq;
  a.q0 = q0;
  a.q1 = q1;
  a.edges = d_edges;
  a.err = ctx->d_err;
  // shared memory: the visited bitmap of the largest graph and two frontier lists; a bitmap that leaves no room
  // for the lists moves to global memory.  One CTA of 1024 threads per SM: the largest graph's passes are the
  // critical path, and a second CTA on its SM slows them (512 RGGs, 1k-200k vertices: 83.6 ms a layout with one,
  // 106.6 ms with two of 512 threads, 100.1 ms with one of 512).
  int64_t nmax = 0;
  for (int b = 0; b < B; b++) nmax = std::max(nmax, ctx->batch_vbase[b + 1] - ctx->batch_vbase[b]);
  const int64_t words = (nmax + 31) / 32;
  int64_t room = (int64_t)(227 * 1024) - 1024 - 4 * words;
  a.vis = nullptr;
  a.vis_words = (int)words;
  if (room < 8 * 1024) {
    room = 64 * 1024;
    a.vis_words = 0;
  }
  const int grid = std::min(B, ctx->nsm);
  if (a.vis_words == 0) {
    a.vis = (uint32_t *)phde_buf(ctx, "kb.vis", sizeof(uint32_t) * (size_t)words * grid);
    if (!a.vis) return PHDE_ERR_OOM;
  }
  a.vis_stride = words;
  a.qcap = (uint32_t)std::min<int64_t>(room / 8, 4096);
  const size_t smem = sizeof(uint32_t) * ((size_t)a.vis_words + 2 * (size_t)a.qcap);
  const auto kernel = a.vis ? kcenters_block_kernel<false> : kcenters_block_kernel<true>;
  if (int arc = phde_allow_smem(ctx, (const void *)kernel)) return arc;
  kernel<<<grid, KB_THREADS, smem, ctx->stream>>>(a);
  PHDE_LAUNCHED(ctx);
  return PHDE_OK;
}
