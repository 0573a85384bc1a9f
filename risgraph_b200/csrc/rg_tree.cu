// Dependency-tree kernels: the B200 form of Graph::build_tree,
// update_tree_add / do_update_tree_add, update_tree_del / do_update_tree_del,
// need_update_tree_* and update_label (core/graph.hpp:873-1887).
//
// Frontiers are device queues of u32 vertex ids deduplicated per level by a
// stamp word per vertex (the reference's ActiveSet keeps duplicates,
// core/actset.hpp:114-147; duplicates only repeat work).  One level of push
// relaxation is one launch of k_push (+ k_push_hub for split hub lists):
//   * each warp takes 32 frontier vertices, scans their degrees with shuffles
//     and walks the concatenated edge slots 32 at a time, so consecutive lanes
//     read consecutive slots (coalesced 8-byte {nbr,w} loads) whatever the
//     degree mix;
//   * lists longer than HUB slots are cut into CHUNK-slot tasks that any warp
//     of the hub kernel picks up (CTA-per-hub balance without a scan);
//   * a relaxation reads the 16-byte label of the target from L2, and only when
//     update_func improves it does a 128-bit CAS of {value, parent|weight}
//     (update_label, core/graph.hpp:1799-1826); successes are appended to the
//     next frontier with one warp-aggregated atomic.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include <cooperative_groups.h>
#include <cub/block/block_reduce.cuh>
#include <cub/block/block_scan.cuh>
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "rg_internal.cuh"
#include "rg_storage_dev.cuh"

namespace rg {

namespace {

constexpr int TPB = 256;
constexpr uint32_t HUB = 64;     // longer lists of a small frontier are split into
constexpr uint32_t CHUNK = 64;   // CHUNK-slot tasks so no warp walks a long list alone

template <bool W>
struct PoolT;
template <>
struct PoolT<true> {
  using E = uint2;
  static __device__ __forceinline__ uint32_t nbr(E e) { return e.x; }
  static __device__ __forceinline__ uint32_t wt(E e) { return e.y; }
};
template <>
struct PoolT<false> {
  using E = uint32_t;
  static __device__ __forceinline__ uint32_t nbr(E e) { return e; }
  static __device__ __forceinline__ uint32_t wt(E) { return 0u; }
};

__device__ __forceinline__ uint32_t seg_len(const DevDir &d, uint32_t v) {
  uint32_t l = d.len[v], c = d.cap[v];
  return l < c ? l : c;
}

// update_label (core/graph.hpp:1799-1826): CAS {value, parent} while the new
// value still improves the current one.
template <int A>
__device__ __forceinline__ bool relax(const DevGraph &g, uint32_t u, uint64_t su, uint32_t v, uint32_t w) {
  const uint64_t nv = Hook<A>::combine(su, w);
  if (!Hook<A>::better(nv, ld_v32(g.val32, v))) return false;
  ulonglong2 cur = ld_lab(&g.lab[v]);
  while (Hook<A>::better(nv, cur.x)) {
    ulonglong2 want = make_ulonglong2(nv, pack_parent(u, w));
    ulonglong2 old = cas128(&g.lab[v], cur, want);
    if (old.x == cur.x && old.y == cur.y) {
      mirror_improve<A>(g.val32, v, nv);
      return true;
    }
    cur = old;
  }
  return false;
}

// relax without the 4-byte value filter: the label itself is the first load,
// so that an improving edge costs two round trips (load, CAS) instead of
// three.  For latency-bound single-CTA levels, where the filter saves no
// bandwidth worth having.
template <int A>
__device__ __forceinline__ bool relax_lab(const DevGraph &g, uint32_t u, uint64_t su, uint32_t v, uint32_t w) {
  const uint64_t nv = Hook<A>::combine(su, w);
  ulonglong2 cur = ld_lab(&g.lab[v]);
  while (Hook<A>::better(nv, cur.x)) {
    ulonglong2 want = make_ulonglong2(nv, pack_parent(u, w));
    ulonglong2 old = cas128(&g.lab[v], cur, want);
    if (old.x == cur.x && old.y == cur.y) {
      mirror_improve<A>(g.val32, v, nv);
      return true;
    }
    cur = old;
  }
  return false;
}

__device__ __forceinline__ void warp_add_result(unsigned long long local, unsigned long long *dst) {
  for (int o = 16; o; o >>= 1) local += __shfl_down_sync(FULL, local, o);
  if (lane_id() == 0 && local) atomicAdd(dst, local);
}

// Serial work without a bound of its own that matters (a walk up a deep tree, a
// warp's search of a vertex's whole list) beats every BEAT_STEPS steps, which
// tells the CTAs that wait at the grid engine's barrier that it goes on.
constexpr uint32_t BEAT_STEPS = 256;
__device__ __forceinline__ void beat(const DevGraph &g) { atomicAdd(&g.ctl[C_BEAT], 1ull); }

// Record v in the modified list (trace_modified graphs); the epoch is read
// from the control block so cached graphs follow rg_clear_modified.
__device__ __forceinline__ void mark_modified(const DevGraph &g, bool pred, uint32_t v, uint32_t /*on*/) {
  const uint32_t mst = (uint32_t)g.ctl[C_MODEPOCH];
  bool app = pred && atomicExch(&g.modstamp[v], mst) != mst;
  warp_append(app, v, g.modq, &g.ctl[C_MODN], FULL);
}

// One push level over a frontier list (stream_edges / stream_edges_sparse
// push lambdas, core/graph.hpp:910-935, :1017-1042, :1083-1104).
template <int A, bool W>
__global__ void __launch_bounds__(TPB) k_push(DevGraph g, const uint32_t *fin, const unsigned long long *fin_n,
                                              uint32_t *fout, unsigned long long *fout_n, uint64_t *hubq,
                                              unsigned long long *hub_n, uint32_t mst) {
  if (g.ctl[C_MODE] != M_SPARSE) return;
  const uint32_t st = (uint32_t)g.ctl[C_STAMP];
  using P = PoolT<W>;
  const typename P::E *pool = reinterpret_cast<const typename P::E *>(g.out.pool);
  const uint64_t n = *fin_n;
  const int lane = lane_id();
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long local = 0, scanned = 0;
  // vertices per warp: as few as the frontier allows (at most 32), so that a
  // frontier smaller than 32 x the grid's warps still spreads over every warp
  // instead of leaving a few warps to walk 32 lists each
  const uint64_t per = (n + nwarps - 1) / nwarps;
  const uint32_t vpw = per >= 32 ? 32u : (per ? (uint32_t)per : 1u);
  for (uint64_t base = warp * vpw; base < n; base += nwarps * vpw) {
    uint64_t i = base + lane;
    uint32_t u = 0, len = 0;
    uint64_t off = 0, su = 0;
    uint32_t hub_c = 0;            // tasks of this lane's hub list
    unsigned long long hub_k = 0;  // where they go in the task queue
    if (lane < vpw && i < n) {
      u = fin[i];
      len = seg_len(g.out, u);
      off = g.out.off[u];
      su = ld_v32(g.val32, u);
      if (len > HUB) {
        hub_c = (len + CHUNK - 1) / CHUNK;
        hub_k = atomicAdd(hub_n, (unsigned long long)hub_c);
        len = 0;
      }
    }
    // the whole warp writes each hub's task list (a hub of 100K slots has 1,563
    // tasks: one lane writing them alone took longer than the rest of the level)
    for (unsigned hm = __ballot_sync(FULL, hub_c != 0); hm; hm &= hm - 1) {
      const int src = __ffs(hm) - 1;
      const uint32_t hu = __shfl_sync(FULL, u, src), hc = __shfl_sync(FULL, hub_c, src);
      const unsigned long long hk = __shfl_sync(FULL, hub_k, src);
      for (uint32_t c = lane; c < hc; c += 32) hubq[hk + c] = (uint64_t)hu | ((uint64_t)c << 32);
    }
    uint32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t t = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += t;
    }
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    if (lane == 0) scanned += total;
    for (uint32_t kb = 0; kb < total; kb += 32) {
      const uint32_t k = kb + lane;
      const bool valid = k < total;
      int owner = 0;
#pragma unroll
      for (int step = 16; step; step >>= 1) {
        uint32_t t = __shfl_sync(FULL, incl, owner + step - 1);
        if (t <= k) owner += step;
      }
      const uint32_t ou = __shfl_sync(FULL, u, owner);
      const uint64_t ooff = __shfl_sync(FULL, off, owner);
      const uint64_t osu = __shfl_sync(FULL, su, owner);
      const uint32_t ostart = __shfl_sync(FULL, incl - len, owner);
      bool upd = false;
      uint32_t v = 0;
      if (valid) {
        typename P::E e = pool[ooff + (k - ostart)];
        uint32_t nb = P::nbr(e);
        if (!(nb & DEAD)) {
          v = nb;
          upd = relax<A>(g,ou, osu, v, P::wt(e));
        }
      }
      local += upd;
      bool app = upd && atomicExch(&g.stamp[v], st) != st;
      warp_append(app, v, fout, fout_n, FULL);
      if (mst) mark_modified(g, upd, v, mst);
    }
  }
  if (lane == 0 && scanned) atomicAdd(&g.ctl[C_EDGES], scanned);
  warp_add_result(local, &g.ctl[C_RESULT]);
}

// Hub chunks: CHUNK consecutive slots of one long list per warp iteration.
template <int A, bool W>
__global__ void __launch_bounds__(TPB) k_push_hub(DevGraph g, const uint64_t *hubq, const unsigned long long *hub_n,
                                                  uint32_t *fout, unsigned long long *fout_n, uint32_t mst) {
  if (g.ctl[C_MODE] != M_SPARSE) return;
  const uint32_t st = (uint32_t)g.ctl[C_STAMP];
  using P = PoolT<W>;
  const typename P::E *pool = reinterpret_cast<const typename P::E *>(g.out.pool);
  const uint64_t n = *hub_n;
  const int lane = lane_id();
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long local = 0, scanned = 0;
  for (uint64_t t = warp; t < n; t += nwarps) {
    const uint64_t task = hubq[t];
    const uint32_t u = (uint32_t)task, c = (uint32_t)(task >> 32);
    const uint32_t len = seg_len(g.out, u);
    const uint64_t off = g.out.off[u];
    const uint64_t su = ld_v32(g.val32, u);
    const uint32_t start = c * CHUNK, end = min(len, start + CHUNK);
    if (lane == 0 && end > start) scanned += end - start;
    for (uint32_t kb = start; kb < end; kb += 32) {
      const uint32_t k = kb + lane;
      bool upd = false;
      uint32_t v = 0;
      if (k < end) {
        typename P::E e = pool[off + k];
        uint32_t nb = P::nbr(e);
        if (!(nb & DEAD)) {
          v = nb;
          upd = relax<A>(g,u, su, v, P::wt(e));
        }
      }
      local += upd;
      bool app = upd && atomicExch(&g.stamp[v], st) != st;
      warp_append(app, v, fout, fout_n, FULL);
      if (mst) mark_modified(g, upd, v, mst);
    }
  }
  if (lane == 0 && scanned) atomicAdd(&g.ctl[C_EDGES], scanned);
  warp_add_result(local, &g.ctl[C_RESULT]);
}

// Relaxation of N independent candidate edges held by one thread (u[k] -> v[k]
// with weight w[k], source value su[k]), in two steps.
// relax_filter reads the 32-bit value mirror of every target and keeps the
// candidates whose update_func value improves it; it returns whether any lane
// of the warp kept one, so a warp whose candidates all fail (the common case
// in late levels) skips the commit entirely.
template <int A, int N>
__device__ __forceinline__ bool relax_filter(const DevGraph &g, bool (&on)[N], const uint32_t (&v)[N],
                                             const uint32_t (&w)[N], const uint64_t (&su)[N]) {
  uint64_t dv[N];
#pragma unroll
  for (int k = 0; k < N; k++) dv[k] = on[k] ? ld_v32(g.val32, v[k]) : 0;
  bool any = false;
#pragma unroll
  for (int k = 0; k < N; k++) {
    on[k] = on[k] && Hook<A>::better(Hook<A>::combine(su[k], w[k]), dv[k]);
    any |= on[k];
  }
  return __any_sync(FULL, any);
}

// relax_commit (all lanes of the warp): issues every CAS of the kept
// candidates before any result is used, then the stamp exchanges, then one
// warp-wide append for every new frontier entry of the warp, so the success
// path costs three round trips per N edges instead of three per edge.
template <int A, int N>
__device__ __forceinline__ void relax_commit(const DevGraph &g, const bool (&on)[N], const uint32_t (&u)[N],
                                             const uint32_t (&v)[N], const uint32_t (&w)[N],
                                             const uint64_t (&su)[N], uint32_t st, uint32_t *fout,
                                             unsigned long long *fout_n, unsigned long long &local, uint32_t mst) {
  bool pend[N], upd[N];
  ulonglong2 want[N], old[N], cur[N];
#pragma unroll
  for (int k = 0; k < N; k++) {
    pend[k] = on[k];
    want[k] = make_ulonglong2(Hook<A>::combine(su[k], w[k]), pack_parent(u[k], w[k]));
    upd[k] = false;
  }
#pragma unroll
  for (int k = 0; k < N; k++) cur[k] = pend[k] ? ld_lab(&g.lab[v[k]]) : make_ulonglong2(0, 0);
#pragma unroll
  for (int k = 0; k < N; k++) pend[k] = pend[k] && Hook<A>::better(want[k].x, cur[k].x);
#pragma unroll
  for (int k = 0; k < N; k++)
    if (pend[k]) old[k] = cas128(&g.lab[v[k]], cur[k], want[k]);
#pragma unroll
  for (int k = 0; k < N; k++) {
    if (!pend[k]) continue;
    if (old[k].x == cur[k].x && old[k].y == cur[k].y) {
      upd[k] = true;
      continue;
    }
    cur[k] = old[k];
    while (Hook<A>::better(want[k].x, cur[k].x)) {  // lost a race: retry while still better
      ulonglong2 o = cas128(&g.lab[v[k]], cur[k], want[k]);
      if (o.x == cur[k].x && o.y == cur[k].y) {
        upd[k] = true;
        break;
      }
      cur[k] = o;
    }
  }
  uint32_t ex[N];
#pragma unroll
  for (int k = 0; k < N; k++)
    if (upd[k]) {
      mirror_improve<A>(g.val32, v[k], want[k].x);
      ex[k] = atomicExch(&g.stamp[v[k]], st);
    }
  uint32_t cnt = 0;
#pragma unroll
  for (int k = 0; k < N; k++) {
    local += upd[k];
    cnt += (upd[k] && ex[k] != st);
  }
  // one atomic per warp for all new entries
  uint32_t incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(FULL, incl, o);
    if (lane_id() >= o) incl += t;
  }
  const uint32_t total = __shfl_sync(FULL, incl, 31);
  if (total) {
    unsigned long long base = 0;
    if (lane_id() == 31) base = atomicAdd(fout_n, (unsigned long long)total);
    base = __shfl_sync(FULL, base, 31) + (incl - cnt);
#pragma unroll
    for (int k = 0; k < N; k++)
      if (upd[k] && ex[k] != st) fout[base++] = v[k];
  }
  if (mst) {
#pragma unroll
    for (int k = 0; k < N; k++) mark_modified(g, upd[k], v[k], mst);
  }
}

template <int A, int N>
__device__ __forceinline__ void relax_batch(const DevGraph &g, const bool (&on)[N], const uint32_t (&u)[N],
                                            const uint32_t (&v)[N], const uint32_t (&w)[N],
                                            const uint64_t (&su)[N], uint32_t st, uint32_t *fout,
                                            unsigned long long *fout_n, unsigned long long &local, uint32_t mst) {
  bool keep[N];
#pragma unroll
  for (int k = 0; k < N; k++) keep[k] = on[k];
  if (relax_filter<A, N>(g, keep, v, w, su)) relax_commit<A, N>(g, keep, u, v, w, su, st, fout, fout_n, local, mst);
}

// ---- edge-balanced push for large frontiers -------------------------------
// The frontier's degrees are prefix-summed (P), the concatenated edge range
// [0, P[n]) is cut into LB_TILE-edge tiles, and each CTA takes whole tiles:
// the frontier entries a tile touches are staged in shared memory, and each
// thread relaxes LB_ITEMS edges strided by the block size (coalesced pool
// reads).  The edge loads of a thread are all issued before the label loads,
// and those before any CAS, so each thread keeps LB_ITEMS independent memory
// round trips in flight instead of one.
constexpr int LB_TPB = 256;
constexpr int LB_ITEMS = 4;
constexpr uint32_t LB_TILE = LB_TPB * LB_ITEMS;
constexpr uint32_t LB_CAP = 1025;  // staged entries per tile (sparser tiles search P in global memory)

// Exclusive prefix of the frontier's degrees into P[0..n] (P[n] = total),
// with n read on the device: every block owns one contiguous range; pass 1
// sums the ranges, pass 2 scans the range sums in one block, pass 3 scans
// each range with its offset.
constexpr int SC_BLOCKS = 512;
constexpr int SC_TPB = 256;

__device__ __forceinline__ void scan_range(uint64_t n1, int b, uint64_t &lo, uint64_t &hi) {
  const uint64_t per = (n1 + SC_BLOCKS - 1) / SC_BLOCKS;
  lo = min(n1, (uint64_t)b * per);
  hi = min(n1, lo + per);
}

__global__ void __launch_bounds__(SC_TPB) k_scan_sums(DevGraph g, const uint32_t *fin,
                                                      const unsigned long long *fin_n, uint64_t *deg,
                                                      uint64_t *sums) {
  using BR = cub::BlockReduce<uint64_t, SC_TPB>;
  __shared__ typename BR::TempStorage tmp;
  const uint64_t n = *fin_n;
  uint64_t lo, hi;
  scan_range(n + 1, blockIdx.x, lo, hi);
  uint64_t s = 0;
  for (uint64_t i = lo + threadIdx.x; i < hi; i += SC_TPB) {
    const uint64_t d = i < n ? seg_len(g.out, fin[i]) : 0;
    deg[i] = d;
    s += d;
  }
  s = BR(tmp).Sum(s);
  if (threadIdx.x == 0) sums[blockIdx.x] = s;
}

__global__ void __launch_bounds__(SC_BLOCKS) k_scan_top(uint64_t *sums) {
  using BS = cub::BlockScan<uint64_t, SC_BLOCKS>;
  __shared__ typename BS::TempStorage tmp;
  uint64_t v = sums[threadIdx.x];
  BS(tmp).ExclusiveSum(v, v);
  sums[threadIdx.x] = v;
}

__global__ void __launch_bounds__(SC_TPB) k_scan_final(const unsigned long long *fin_n, const uint64_t *deg,
                                                       const uint64_t *sums, uint64_t *P) {
  using BS = cub::BlockScan<uint64_t, SC_TPB>;
  __shared__ typename BS::TempStorage tmp;
  __shared__ uint64_t carry;
  const uint64_t n = *fin_n;
  uint64_t lo, hi;
  scan_range(n + 1, blockIdx.x, lo, hi);
  if (threadIdx.x == 0) carry = sums[blockIdx.x];
  __syncthreads();
  for (uint64_t base = lo; base < hi; base += SC_TPB) {
    const uint64_t i = base + threadIdx.x;
    uint64_t d = i < hi ? deg[i] : 0, x, total;
    BS(tmp).ExclusiveSum(d, x, total);
    if (i < hi) P[i] = carry + x;
    __syncthreads();
    if (threadIdx.x == 0) carry += total;
    __syncthreads();
  }
}

// tile_lo[t] = last frontier index whose edge range starts at or before t*LB_TILE.
__global__ void k_partition(const uint64_t *P, const unsigned long long *fin_n, uint32_t *tile_lo) {
  const uint64_t n = *fin_n;
  const uint64_t T = P[n];
  const uint64_t ntiles = (T + LB_TILE - 1) / LB_TILE;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t <= ntiles; t += stride) {
    uint64_t x = t < ntiles ? t * LB_TILE : T;
    uint64_t lo = 0, hi = n;  // largest i in [0, n] with P[i] <= x
    while (lo < hi) {
      uint64_t mid = (lo + hi + 1) >> 1;
      if (__ldg(&P[mid]) <= x) lo = mid;
      else hi = mid - 1;
    }
    tile_lo[t] = (uint32_t)(lo < n ? lo : (n ? n - 1 : 0));
  }
}

template <int A, bool W>
__global__ void __launch_bounds__(LB_TPB, 3) k_push_lbs(DevGraph g, const uint32_t *fin,
                                                     const unsigned long long *fin_n, const uint64_t *P,
                                                     const uint32_t *tile_lo, uint32_t *fout,
                                                     unsigned long long *fout_n, uint32_t mst) {
  const uint64_t n = *fin_n;
  const uint32_t st = (uint32_t)g.ctl[C_STAMP];
  using P_ = PoolT<W>;
  const typename P_::E *pool = reinterpret_cast<const typename P_::E *>(g.out.pool);
  __shared__ uint32_t s_rel[LB_CAP];
  __shared__ uint32_t s_u[LB_CAP];
  __shared__ uint64_t s_base[LB_CAP];
  __shared__ uint64_t s_su[LB_CAP];
  const uint64_t T = P[n];
  const uint64_t ntiles = (T + LB_TILE - 1) / LB_TILE;
  unsigned long long local = 0;
  for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const uint64_t t0 = t * LB_TILE;
    const uint64_t t1 = min(t0 + LB_TILE, T);
    const uint32_t lo = tile_lo[t];
    const uint32_t hi = tile_lo[t + 1];
    const uint32_t m = hi - lo + 1;
    const bool staged = m <= LB_CAP;
    if (staged) {
      for (uint32_t j = threadIdx.x; j < m; j += LB_TPB) {
        uint64_t pj = P[lo + j];
        uint32_t u = fin[lo + j];
        s_rel[j] = pj <= t0 ? 0u : (uint32_t)(pj - t0);
        s_u[j] = u;
        s_base[j] = g.out.off[u] - pj;
        s_su[j] = ld_v32(g.val32, u);
      }
    }
    __syncthreads();
    uint64_t slot[LB_ITEMS], su[LB_ITEMS];
    uint32_t uu[LB_ITEMS];
#pragma unroll
    for (int k = 0; k < LB_ITEMS; k++) {
      const uint64_t e = t0 + (uint64_t)k * LB_TPB + threadIdx.x;
      slot[k] = ~0ull;
      if (e < t1) {
        uint32_t j;
        if (staged) {
          const uint32_t er = (uint32_t)(e - t0);
          uint32_t a = 0, b = m - 1;  // largest j with s_rel[j] <= er
          while (a < b) {
            uint32_t mid = (a + b + 1) >> 1;
            if (s_rel[mid] <= er) a = mid;
            else b = mid - 1;
          }
          j = a;
          slot[k] = s_base[j] + e;
          uu[k] = s_u[j];
          su[k] = s_su[j];
        } else {
          uint64_t a = lo, b = hi;  // many empty entries: search P directly
          while (a < b) {
            uint64_t mid = (a + b + 1) >> 1;
            if (P[mid] <= e) a = mid;
            else b = mid - 1;
          }
          uint32_t u = fin[a];
          slot[k] = g.out.off[u] + (e - P[a]);
          uu[k] = u;
          su[k] = ld_v32(g.val32, u);
        }
      }
    }
    bool on[LB_ITEMS];
    uint32_t vv[LB_ITEMS], ww[LB_ITEMS];
#pragma unroll
    for (int k = 0; k < LB_ITEMS; k++) {
      on[k] = false;
      vv[k] = 0;
      ww[k] = 0;
      if (slot[k] != ~0ull) {
        typename P_::E ent = __ldg(&pool[slot[k]]);
        vv[k] = P_::nbr(ent);
        ww[k] = P_::wt(ent);
        on[k] = !(vv[k] & DEAD);
      } else {
        uu[k] = 0;
        su[k] = 0;
      }
    }
    relax_batch<A, LB_ITEMS>(g, on, uu, vv, ww, su, st, fout, fout_n, local, mst);
    __syncthreads();
  }
  warp_add_result(local, &g.ctl[C_RESULT]);
  if (threadIdx.x == 0 && blockIdx.x == 0) atomicAdd(&g.ctl[C_EDGES], T);
}

// ---- edge-centric push for dense levels -----------------------------------
// When the frontier holds a large share of the vertices (the reference switches
// to its dense mode at the same point, core/graph.hpp:334), streaming the whole
// out-pool beats locating every frontier segment: slot i belongs to owner[i]
// and is relaxed when its owner is active in this level (act[owner] == id).
// Reads of owner[] and of the pool are fully coalesced; there is no staging,
// search or barrier, and each thread keeps DN_ITEMS slots in flight.
constexpr int DN_TPB = 256;
constexpr int DN_ITEMS = 4;

__global__ void k_mark_active(DevGraph g, const uint32_t *fin, const unsigned long long *fin_n, uint32_t *act) {
  if (g.ctl[C_MODE] != M_DENSE_PUSH) return;
  const uint32_t id = (uint32_t)g.ctl[C_ACT];
  const uint64_t n = *fin_n;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += stride) act[fin[i]] = id;
}

template <int A, bool W>
__global__ void __launch_bounds__(DN_TPB, 3) k_push_dense(DevGraph g, const uint32_t *act, uint32_t *fout,
                                                       unsigned long long *fout_n, uint32_t mst) {
  if (g.ctl[C_MODE] != M_DENSE_PUSH) return;
  const uint32_t act_id = (uint32_t)g.ctl[C_ACT];
  const uint32_t st = (uint32_t)g.ctl[C_STAMP];
  using P_ = PoolT<W>;
  const typename P_::E *pool = reinterpret_cast<const typename P_::E *>(g.out.pool);
  const uint64_t top = *g.out.pool_top;
  const uint64_t slots = top < g.out.pool_cap ? top : g.out.pool_cap;
  const uint64_t tile = (uint64_t)DN_TPB * DN_ITEMS;
  unsigned long long local = 0, scanned = 0;
  for (uint64_t base = blockIdx.x * tile; base < slots; base += (uint64_t)gridDim.x * tile) {
    uint32_t o[DN_ITEMS];
#pragma unroll
    for (int k = 0; k < DN_ITEMS; k++) {
      const uint64_t i = base + (uint64_t)k * DN_TPB + threadIdx.x;
      o[k] = i < slots ? __ldg(&g.out.owner[i]) : NONE;
    }
    bool a[DN_ITEMS], any = false;
#pragma unroll
    for (int k = 0; k < DN_ITEMS; k++) {
      a[k] = o[k] != NONE && __ldg(&act[o[k]]) == act_id;
      any |= a[k];
    }
    if (!__any_sync(FULL, any)) continue;  // no active owner in the warp's slots
    uint32_t vv[DN_ITEMS], ww[DN_ITEMS];
    uint64_t su[DN_ITEMS];
#pragma unroll
    for (int k = 0; k < DN_ITEMS; k++) {
      vv[k] = 0;
      ww[k] = 0;
      su[k] = 0;
      if (a[k]) {
        typename P_::E ent = __ldg(&pool[base + (uint64_t)k * DN_TPB + threadIdx.x]);
        su[k] = ld_v32(g.val32, o[k]);
        vv[k] = P_::nbr(ent);
        ww[k] = P_::wt(ent);
        a[k] = !(vv[k] & DEAD);
        scanned++;
      }
    }
    relax_batch<A, DN_ITEMS>(g, a, o, vv, ww, su, st, fout, fout_n, local, mst);
  }
  warp_add_result(local, &g.ctl[C_RESULT]);
  warp_add_result(scanned, &g.ctl[C_EDGES]);
}

// ---- dense pull over in-edges ----------------------------------------------
// The reference's dense mode (stream_edges dense lambda, core/graph.hpp:936-976):
// every vertex takes the best update_func value over its in-edges.  For full
// builds the live in-edges are copied once per adjacency version into a sliced
// ELLPACK layout (SELL-32): rows sorted by length, 32 consecutive rows per
// slice, a slice stored column-major so that lane l of a warp reads row l and
// the 32 lanes of a warp read 32 consecutive entries.  A row is a vertex's
// in-list, or for a hub (in-list longer than PULL_HUB) one of the equal pieces
// its list is cut into, so every row holds at most PULL_HUB entries, a lane's
// chain of dependent loads is short (pieces of 576 took 60 us a level on a graph
// of 150K vertices, most of it one chain), and the
// warps stay balanced.  A pull level is one warp per slice with no search and
// no atomics on labels: a vertex row is written only by its own lane; a piece
// leaves its best in a side array and k_pull_hub_fix combines the pieces of
// each hub.
constexpr int PS_TPB = 256;
// Split pull levels (RG_OPT_PULL_SPLIT): a level first pulls the hubs' pieces
// and combines them (pull_hub_fix), then every other row, which reads the hubs'
// values of this level, where one pass reads them stale from L1 for most of the
// level: values move along hub paths faster and fewer levels pull.  Without the
// split all rows go first and the pieces are combined at the end.
// Entries of a row that a lane reads at a time.
constexpr int PULL_DEPTH = 8;
constexpr int PULL_CTAS = 4;  // resident CTAs per SM that the pull kernel's registers allow

template <bool W>
struct SellE;
template <>
struct SellE<true> {
  using E = uint2;
  static __device__ __forceinline__ E none() { return make_uint2(NONE, 0u); }
  static __device__ __forceinline__ E make(uint32_t u, uint32_t w) { return make_uint2(u, w); }
  static __device__ __forceinline__ uint32_t nbr(E e) { return e.x; }
  static __device__ __forceinline__ uint32_t wt(E e) { return e.y; }
};
template <>
struct SellE<false> {
  using E = uint32_t;
  static __device__ __forceinline__ E none() { return NONE; }
  static __device__ __forceinline__ E make(uint32_t u, uint32_t) { return u; }
  static __device__ __forceinline__ uint32_t nbr(E e) { return e; }
  static __device__ __forceinline__ uint32_t wt(E) { return 0u; }
};

// Pieces of a hub of in-list length len: equal lengths of at most PULL_PIECE.
__device__ __forceinline__ uint32_t hub_pieces(uint32_t len) { return (len + PULL_PIECE - 1) / PULL_PIECE; }
// Entries of a row of key k.
__host__ __device__ __forceinline__ uint32_t sell_width(uint32_t k) { return k > PULL_HUB ? k - PULL_HUB : k; }

// The copy is laid out in three passes over the vertices' list lengths: count
// the rows of each key (k_sell_count), turn the counts into row and slice
// positions (k_sell_plan, one block), and put each row in its place
// (k_sell_rows).  There are few keys, so a histogram in shared memory
// replaces a sort of all vertices, and the host waits once, for the plan, to
// size the arrays.  (RMAT-20, 16M weighted edges: the whole preparation takes
// 0.25 ms; 8.0 ms with a radix sort, five host synchronisations, temporary
// allocations and one thread copying each row.)
__global__ void __launch_bounds__(1024) k_sell_count(DevGraph g, uint32_t *hub_v, uint64_t *hub_pc, SellPlan *plan) {
  __shared__ uint32_t s_n[SELL_KEYS];
  for (int b = threadIdx.x; b < SELL_KEYS; b += blockDim.x) s_n[b] = 0;
  __syncthreads();
  const uint64_t V = g.V;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += stride) {
    const uint32_t d = seg_len(g.in, (uint32_t)v);
    if (d > PULL_HUB) {
      const uint32_t np = hub_pieces(d), base = d / np, extra = d % np;
      const unsigned long long h = atomicAdd(&plan->hubs, 1ull);
      hub_v[h] = (uint32_t)v;
      hub_pc[h] = atomicAdd(&plan->pieces, (unsigned long long)np) | ((uint64_t)np << 32);
      atomicAdd(&s_n[PULL_HUB + base], np - extra);
      if (extra) atomicAdd(&s_n[PULL_HUB + base + 1], extra);
    } else if (d) {
      atomicAdd(&s_n[d], 1u);
    }
  }
  __syncthreads();
  for (int b = threadIdx.x; b < SELL_KEYS; b += blockDim.x)
    if (s_n[b]) atomicAdd(&plan->count[b], s_n[b]);
}

// Rows of key k take the positions after all larger keys, the first vertex row
// after a gap to the next slice; slices are 32 consecutive rows, as wide as
// their first.
constexpr int SP_TPB = 1024;
static_assert(SELL_KEYS <= SP_TPB + 1, "one thread per key");
__global__ void __launch_bounds__(SP_TPB) k_sell_plan(SellPlan *plan) {
  using Scan = cub::BlockScan<uint64_t, SP_TPB>;
  __shared__ typename Scan::TempStorage tmp;
  const int t = threadIdx.x, k = SELL_KEYS - 1 - t;  // largest first
  const uint64_t n = k >= 1 ? plan->count[k] : 0;
  const uint64_t P = plan->pieces, gap = (32 - P % 32) % 32;
  uint64_t row, rows;
  Scan(tmp).ExclusiveSum(n, row, rows);
  if (k <= (int)PULL_HUB) row += gap;
  const uint64_t s0 = (row + 31) / 32, s1 = (row + n + 31) / 32;
  __syncthreads();
  uint64_t base, total;
  Scan(tmp).ExclusiveSum(k >= 1 ? 32 * (uint64_t)sell_width(k) * (s1 - s0) : 0, base, total);
  if (k >= 1) {
    plan->cursor[k] = (uint32_t)row;
    plan->slice[k] = (uint32_t)s0;
    plan->base[k] = base;
  }
  if (t == 0) {
    plan->rows = rows + gap;
    plan->slices = (rows + gap + 31) / 32;
    plan->total = total;
    plan->slice[0] = (uint32_t)((rows + gap + 31) / 32);
  }
}

// Row ids (a vertex, or |V| + a piece of a hub) in their places, the piece
// table, and the slice offsets.  A block reserves the places of its rows of
// one length together, which keeps rows of near vertices near each other.
constexpr int SR_TPB = 512, SR_ITEMS = 8;

__global__ void __launch_bounds__(SR_TPB) k_sell_rows(DevGraph g, const uint32_t *hub_v, unsigned long long *hub_pc,
                                                      SellPlan *plan, uint32_t *row_id, uint32_t *piece_v,
                                                      uint32_t *piece_start, uint32_t *piece_len, uint32_t *piece_hub,
                                                      uint64_t *off) {
  __shared__ uint32_t s_n[PULL_HUB + 1], s_at[PULL_HUB + 1];
  const uint64_t V = g.V;
  constexpr uint64_t TILE = SR_TPB * SR_ITEMS;
  for (uint64_t b0 = blockIdx.x * TILE; b0 < V; b0 += gridDim.x * TILE) {
    for (int b = threadIdx.x; b <= (int)PULL_HUB; b += SR_TPB) s_n[b] = 0;
    __syncthreads();
    uint32_t d[SR_ITEMS], at[SR_ITEMS];
#pragma unroll
    for (int k = 0; k < SR_ITEMS; k++) {
      const uint64_t v = b0 + (uint64_t)k * SR_TPB + threadIdx.x;
      d[k] = v < V ? seg_len(g.in, (uint32_t)v) : 0u;
      if (d[k] > PULL_HUB) d[k] = 0;
    }
#pragma unroll
    for (int k = 0; k < SR_ITEMS; k++) at[k] = d[k] ? atomicAdd(&s_n[d[k]], 1u) : 0u;
    __syncthreads();
    for (int b = threadIdx.x; b <= (int)PULL_HUB; b += SR_TPB)
      s_at[b] = s_n[b] ? atomicAdd(&plan->cursor[b], s_n[b]) : 0u;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SR_ITEMS; k++)
      if (d[k]) row_id[s_at[d[k]] + at[k]] = (uint32_t)(b0 + (uint64_t)k * SR_TPB + threadIdx.x);
    __syncthreads();
  }
  // one warp per hub writes its pieces, and clears its best
  const int lane = lane_id();
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const uint64_t nh = plan->hubs;
  for (uint64_t h = warp; h < nh; h += nwarps) {
    const uint32_t v = hub_v[h];
    const uint32_t dv = seg_len(g.in, v);
    const uint64_t pc = hub_pc[h];
    const uint32_t p0 = (uint32_t)pc, np = (uint32_t)(pc >> 32), base = dv / np, extra = dv % np;
    uint32_t a1 = 0, a0 = 0;  // the first `extra` pieces are one longer
    if (lane == 0) {
      if (extra) a1 = atomicAdd(&plan->cursor[PULL_HUB + base + 1], extra);
      a0 = atomicAdd(&plan->cursor[PULL_HUB + base], np - extra);
    }
    a1 = __shfl_sync(FULL, a1, 0);
    a0 = __shfl_sync(FULL, a0, 0);
    for (uint32_t k = lane; k < np; k += 32) {
      piece_v[p0 + k] = v;
      piece_start[p0 + k] = k * base + min(k, extra);
      piece_len[p0 + k] = base + (k < extra ? 1u : 0u);
      piece_hub[p0 + k] = (uint32_t)h;
      row_id[k < extra ? a1 + k : a0 + (k - extra)] = (uint32_t)(V + p0 + k);
    }
    __syncwarp();
    if (lane == 0) hub_pc[h] = ~0ull;
  }
  if (blockIdx.x == 0 && threadIdx.x < 32) {  // the gap before the vertex rows
    const uint64_t P = plan->pieces;
    if (P % 32 && threadIdx.x >= P % 32) row_id[P - P % 32 + threadIdx.x] = NONE;
  }
  const uint64_t ns = plan->slices;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t s = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; s <= ns; s += stride) {
    int lo = 1, hi = SELL_KEYS - 1;  // the smallest key k with slice[k] <= s
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      if (plan->slice[mid] <= s) hi = mid;
      else lo = mid + 1;
    }
    off[s] = s < ns ? plan->base[lo] + (s - plan->slice[lo]) * 32 * sell_width(lo) : plan->total;
  }
}

// Weight classes of the entry order: 0 to 127 exactly, then sixteen to each
// power of two (device weights and ids are below 2^31, so there are 512).  w_floor /
// w_ceil: the smallest / largest weight of w's class.
constexpr int W_CLASSES = 512;
__device__ __forceinline__ uint32_t w_class(uint32_t w) {
  if (w < 128) return w;
  const uint32_t e = 31 - __clz(w);
  return (128 + 16 * (e - 7) + ((w >> (e - 4)) & 15)) & (W_CLASSES - 1);
}
__device__ __forceinline__ uint32_t w_floor(uint32_t w) {
  return w < 128 ? w : w & ~((1u << (27 - __clz(w))) - 1u);
}
__device__ __forceinline__ uint32_t w_ceil(uint32_t w) {
  return w < 128 ? w : w | ((1u << (27 - __clz(w))) - 1u);
}

// Where row r's entries come from.
struct RowSrc {
  uint64_t from;
  uint32_t n;
};
__device__ __forceinline__ RowSrc sell_row_src(const DevGraph &g, const uint32_t *row_id, uint64_t r, uint64_t rows,
                                               const uint32_t *piece_v, const uint32_t *piece_start,
                                               const uint32_t *piece_len) {
  RowSrc s = {0, 0};
  const uint32_t id = r < rows ? row_id[r] : NONE;
  if (id != NONE) {
    if (id < g.V) {
      s.from = g.in.off[id];
      s.n = seg_len(g.in, id);
    } else {
      const uint32_t p = id - g.V;
      s.from = g.in.off[piece_v[p]] + piece_start[p];
      s.n = piece_len[p];
    }
  }
  return s;
}

// Copy the live in-entries of each row of slices [s_lo, s_hi) into its column;
// pad with NONE.  One thread per row, in the order of the pool: for narrow
// rows.
template <bool W>
__global__ void k_sell_fill(DevGraph g, const uint32_t *row_id, uint64_t rows, uint64_t s_lo, uint64_t s_hi,
                            const uint64_t *off, const uint32_t *piece_v, const uint32_t *piece_start,
                            const uint32_t *piece_len, typename SellE<W>::E *ent) {
  using P_ = PoolT<W>;
  using S_ = SellE<W>;
  const typename P_::E *pool = reinterpret_cast<const typename P_::E *>(g.in.pool);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t r = s_lo * 32 + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < s_hi * 32; r += stride) {
    const uint64_t s = r >> 5, lane = r & 31;
    const uint64_t o0 = off[s];
    const uint32_t width = (uint32_t)((off[s + 1] - o0) >> 5);
    typename S_::E *col = ent + o0 + lane;
    const RowSrc src = sell_row_src(g, row_id, r, rows, piece_v, piece_start, piece_len);
    uint32_t j = 0;
    for (uint32_t k0 = 0; k0 < src.n; k0 += 8) {
      typename P_::E e[8];
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (k0 + k < src.n) e[k] = pool[src.from + k0 + k];
#pragma unroll
      for (int k = 0; k < 8; k++)
        if (k0 + k < src.n && !(P_::nbr(e[k]) & DEAD)) col[(uint64_t)j++ * 32] = S_::make(P_::nbr(e[k]), P_::wt(e[k]));
    }
    for (; j < width; j++) col[(uint64_t)j * 32] = S_::none();
  }
}

// The same for rows of more than 8 entries, each row's live entries by class of
// their weight, lightest first, or without weights of their source's id, lowest
// first, so that a pull can stop inside the row.
// One CTA per slice and one warp per row: a lane keeps its K entries in
// registers (one round trip to the pool), the row's class counts and the
// sorted slice are in shared memory, and the slice leaves it column-major in
// coalesced stores.  A row of the tile is padded to an odd number of entries,
// so that a column of 32 rows touches every bank pair once.
constexpr int SF_TPB = 1024;
constexpr size_t sell_fill_smem(int K, size_t entry) { return 32 * (32 * (size_t)K + 1) * entry + 32 * W_CLASSES * 2; }

template <bool W, int K>
__global__ void __launch_bounds__(SF_TPB) k_sell_fill_sorted(DevGraph g, const uint32_t *row_id, uint64_t rows,
                                                             uint64_t s_lo, uint64_t s_hi, const uint64_t *off,
                                                             const uint32_t *piece_v, const uint32_t *piece_start,
                                                             const uint32_t *piece_len, typename SellE<W>::E *ent) {
  using P_ = PoolT<W>;
  using S_ = SellE<W>;
  using E = typename S_::E;
  extern __shared__ __align__(16) unsigned char s_fill[];
  E *s_tile = reinterpret_cast<E *>(s_fill);  // [32 rows][32 K + 1], then [32 rows][W_CLASSES] u16 in pairs
  constexpr int RS = 32 * K + 1;
  const int lane = lane_id(), row = threadIdx.x >> 5;
  uint32_t *cnt = reinterpret_cast<uint32_t *>(s_tile + 32 * RS) + row * (W_CLASSES / 2);  // two classes per word
  constexpr int CW = W_CLASSES / 64;  // words of classes per lane
  const E *pool = reinterpret_cast<const E *>(g.in.pool);
  auto key = [](const E &e) { return w_class(W ? P_::wt(e) : P_::nbr(e)); };
  for (uint64_t s = s_lo + blockIdx.x; s < s_hi; s += gridDim.x) {
    const uint64_t o0 = off[s];
    const uint32_t width = (uint32_t)((off[s + 1] - o0) >> 5);
    const RowSrc src = sell_row_src(g, row_id, s * 32 + row, rows, piece_v, piece_start, piece_len);
    E e[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t i = 32 * k + lane;
      e[k] = i < src.n ? pool[src.from + i] : S_::none();
    }
#pragma unroll
    for (int k = 0; k < CW; k++) cnt[32 * k + lane] = 0;
    __syncwarp();
    uint32_t at[K];  // rank within the class
#pragma unroll
    for (int k = 0; k < K; k++) {
      at[k] = 0;
      if (!(P_::nbr(e[k]) & DEAD)) {  // (NONE has the bit too)
        const uint32_t c = key(e[k]);
        at[k] = (atomicAdd(&cnt[c >> 1], 1u << (16 * (c & 1))) >> (16 * (c & 1))) & 0xFFFFu;
      }
    }
    __syncwarp();
    // exclusive prefix over the classes, each lane the words CW l .. CW l + CW - 1
    uint32_t c2[CW], sum = 0;
#pragma unroll
    for (int k = 0; k < CW; k++) {
      c2[k] = cnt[CW * lane + k];
      sum += (c2[k] & 0xFFFFu) + (c2[k] >> 16);
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    const uint32_t live = __shfl_sync(FULL, incl, 31);
    uint32_t run = incl - sum;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < CW; k++) {
      const uint32_t a = run, b = run + (c2[k] & 0xFFFFu);
      cnt[CW * lane + k] = a | (b << 16);
      run = b + (c2[k] >> 16);
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (!(P_::nbr(e[k]) & DEAD)) {
        const uint32_t c = key(e[k]);
        s_tile[row * RS + ((cnt[c >> 1] >> (16 * (c & 1))) & 0xFFFFu) + at[k]] = e[k];
      }
    }
    for (uint32_t j = live + lane; j < width; j += 32) s_tile[row * RS + j] = S_::none();
    __syncthreads();
    for (uint32_t j = row; j < width; j += 32) ent[o0 + (uint64_t)j * 32 + lane] = s_tile[lane * RS + j];
    __syncthreads();
  }
}

// Values in 32 bits (every hook's fit): update_func's value and its order.
template <int A>
__device__ __forceinline__ uint32_t combine32(uint32_t s, uint32_t w) {
  return (uint32_t)Hook<A>::combine(s, w);
}
template <int A>
__device__ __forceinline__ bool better32(uint32_t a, uint32_t b) {
  return A == RG_SSWP ? a > b : a < b;
}

// What a pull may leave out.  No vertex in the level's frontier has a value
// better than the level's bound m (the best value that the level before
// committed, or the best possible one), and neither has any vertex that changes
// in this level; a source that is in neither set was relaxed over all its edges
// after its last change.  So an in-edge of weight w can only improve v if
// combine(m, w) does, and since rows are in order of weight (lightest first;
// SSWP reads them from the other end), the first weight class that cannot
// improve v ends its row.  With weights of 1 to 255 that leaves a few entries
// of each list: a hub of value 5 reads the entries lighter than 5.  The values
// after the level are those of the full pull.
// (RMAT-22 SSSP, four pull levels: 0.17, 0.13, 0.11 and 0.09 ms and 0.7 E
// entries read in all; over every entry 0.31 to 0.34 ms each and 4.0 E.)
template <int A>
__device__ __forceinline__ bool pull_open(uint32_t m, uint32_t w, uint32_t best) {
  return better32<A>(combine32<A>(m, w), best);
}
// the remaining entries of a row after one of weight w
template <int A>
__device__ __forceinline__ bool pull_more(uint32_t m, uint32_t w, uint32_t best) {
  return pull_open<A>(m, A == RG_SSWP ? w_ceil(w) : w_floor(w), best);
}

// One row's pull: the value it improves (its vertex's, or for a piece its
// hub's), the best candidate so far and where that came from.
struct PullRow {
  uint32_t best, bsrc, bw;
  bool has;
};

template <int A, bool W>
__device__ __forceinline__ void pull_take(const typename SellE<W>::E &e, uint32_t sv, bool on, PullRow &p) {
  using S_ = SellE<W>;
  const uint32_t c = combine32<A>(sv, S_::wt(e));
  if (on && better32<A>(c, p.best)) {
    p.has = true;
    p.best = c;
    p.bsrc = S_::nbr(e);
    p.bw = S_::wt(e);
  }
}

// A warp's new frontier entries, collected in shared memory: a full buffer goes
// to the queue with one atomic on its counter, and at the end the CTA's buffers
// go together.  (One atomic for every slice with a change, and one for every
// warp on each of the counts, took most of a level on graphs of 10^5 vertices:
// same-address atomics are served one after the other.)
constexpr uint32_t PQ_CAP = 128;
struct PullQueue {
  uint32_t *buf;  // this warp's PQ_CAP entries
  uint32_t n;     // entries held (the same in every lane)
};

__device__ __forceinline__ void pull_flush(PullQueue &q, uint32_t *fout, unsigned long long *fout_n) {
  const uint32_t lane = (uint32_t)lane_id();
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(fout_n, (unsigned long long)q.n);
  base = __shfl_sync(FULL, base, 0);
  __syncwarp();
  for (uint32_t i = lane; i < q.n; i += 32) fout[base + i] = q.buf[i];
  __syncwarp();
  q.n = 0;
}

// Append by every lane with pred set.
__device__ __forceinline__ void pull_append(PullQueue &q, bool pred, uint32_t v, uint32_t *fout,
                                            unsigned long long *fout_n) {
  const unsigned b = __ballot_sync(FULL, pred);
  if (b) {
    if (pred) q.buf[q.n + __popc(b & ((1u << lane_id()) - 1))] = v;
    q.n += __popc(b);
    if (q.n > PQ_CAP - 32) pull_flush(q, fout, fout_n);
  }
}

// Work counts of a CTA, summed in shared memory.
struct BlockCounts {
  unsigned long long updates, scanned;
};
__device__ __forceinline__ void block_count(BlockCounts *bc, unsigned long long updates, unsigned long long scanned) {
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    updates += __shfl_down_sync(FULL, updates, o);
    scanned += __shfl_down_sync(FULL, scanned, o);
  }
  if (lane_id() == 0) {
    if (updates) atomicAdd(&bc->updates, updates);
    if (scanned) atomicAdd(&bc->scanned, scanned);
  }
}

// End of a pass (all threads of the CTA): what the warps' buffers still hold
// goes to the queue with one atomic per CTA.
__device__ __forceinline__ void pull_drain(PullQueue &q, uint32_t *fout, unsigned long long *fout_n) {
  __shared__ unsigned long long s_at[32];
  const unsigned w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (lane == 0) s_at[w] = q.n;
  __syncthreads();
  if (w == 0) {
    const uint32_t n = lane < nw ? (uint32_t)s_at[lane] : 0u;
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULL, incl, o);
      if (lane >= (unsigned)o) incl += y;
    }
    unsigned long long base = 0;
    if (lane == 31 && incl) base = atomicAdd(fout_n, (unsigned long long)incl);
    base = __shfl_sync(FULL, base, 31);
    if (lane < nw) s_at[lane] = base + incl - n;
  }
  __syncthreads();
  for (uint32_t i = lane; i < q.n; i += 32) fout[s_at[w] + i] = q.buf[i];
  __syncthreads();
  q.n = 0;
}

// Commit of one pulled row (all lanes of the warp call it): a vertex has a
// single writer, so its label needs no atomic; a piece that improves its hub
// leaves its best for pull_hub_fix, and its number with its hub if no other
// piece has a better value.  fb: the best value committed by this thread.
struct PullHubs {
  const uint32_t *piece_v, *piece_hub, *hub_v;
  ulonglong2 *piece_best;        // {value, parent | w << 32}
  unsigned long long *hub_best;  // {order of the value, piece}; all ones: none
};
// Values as words that a minimum orders best first.
template <int A>
__device__ __forceinline__ uint64_t hub_order(uint32_t v) {
  return (uint64_t)(A == RG_SSWP ? ~v : v) << 32;
}

template <int A>
__device__ __forceinline__ void pull_row_done(const DevGraph &g, bool active, uint32_t id, const PullRow &p,
                                              const PullHubs &hubs, PullQueue &q, uint32_t *fout,
                                              unsigned long long *fout_n, uint32_t mst, uint32_t &local, uint32_t &fb) {
  const bool upd = active && id < g.V && p.has;
  if (upd) {
    g.lab[id] = make_ulonglong2(p.best, pack_parent(p.bsrc, p.bw));
    g.val32[id] = p.best;
    if (better32<A>(p.best, fb)) fb = p.best;
  } else if (active && p.has) {
    const uint32_t pi = id - g.V;
    hubs.piece_best[pi] = make_ulonglong2(p.best, pack_parent(p.bsrc, p.bw));
    atomicMin(&hubs.hub_best[hubs.piece_hub[pi]], (unsigned long long)(hub_order<A>(p.best) | pi));
  }
  local += upd;
  pull_append(q, upd, id, fout, fout_n);
  if (mst) mark_modified(g, upd, id, mst);
}

// The best value committed by the CTA, into the bound of the next frontier (all
// threads of the CTA).
template <int A>
__device__ __forceinline__ void pull_bound_out(uint32_t fb, unsigned long long *bout) {
  __shared__ uint32_t s_b[32];
  const unsigned w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const uint32_t b = A == RG_SSWP ? __reduce_max_sync(FULL, fb) : __reduce_min_sync(FULL, fb);
  if (lane == 0) s_b[w] = b;
  __syncthreads();
  if (w == 0) {
    const uint32_t x = s_b[lane < nw ? lane : 0];
    const uint32_t y = A == RG_SSWP ? __reduce_max_sync(FULL, x) : __reduce_min_sync(FULL, x);
    if (lane == 0) {
      if (A == RG_SSWP) atomicMax(bout, (unsigned long long)y);
      else atomicMin(bout, (unsigned long long)y);
    }
  }
  __syncthreads();
}
template <int A>
__device__ __forceinline__ uint32_t pull_worst() {
  return A == RG_SSWP ? 0u : 0xFFFFFFFFu;
}

// Source values through L1: the values of popular sources stay there.  A value
// cached before its owner improved in this level is only older, and that owner
// is in the next frontier anyway.
__device__ __forceinline__ uint32_t pull_src_val(const DevGraph &g, uint32_t u) { return __ldca(&g.val32[u]); }

// Slices are sorted by width (the length of their longest row).  A warp takes
// one slice and reads its rows PULL_DEPTH entries at a time; slices at most 4,
// 2 and 1 entries wide are taken G = 2, 4 and 8 at a time, so that every lane
// still keeps eight entries in flight per round trip.  (Sixteen took 112
// registers a thread and left a quarter of the warps resident.)
template <int A, bool W, int G>
__device__ __forceinline__ void pull_narrow(const DevGraph &g, const typename SellE<W>::E *ent, const uint64_t *off,
                                            const uint32_t *row_id, uint32_t rows, uint32_t s0, uint32_t hi, uint32_t m,
                                            PullQueue &q, uint32_t *fout, unsigned long long *fout_n, uint32_t mst,
                                            uint32_t &local, uint32_t &fb) {
  using S_ = SellE<W>;
  constexpr int NP = PULL_DEPTH / G;
  const int lane = lane_id();
  typename S_::E e[PULL_DEPTH];
  uint32_t id[G];
#pragma unroll
  for (int gi = 0; gi < G; gi++) {
    const uint32_t s = s0 + gi;
    const uint64_t o = s < hi ? off[s] : 0;
    const uint32_t w = s < hi ? (uint32_t)((off[s + 1] - o) >> 5) : 0u;
    id[gi] = s < hi && s * 32 + lane < rows ? row_id[s * 32 + lane] : NONE;
#pragma unroll
    for (int k = 0; k < NP; k++) e[gi * NP + k] = k < w ? __ldcs(&ent[o + (uint64_t)k * 32 + lane]) : S_::none();
  }
  uint32_t cur[G];
#pragma unroll
  for (int gi = 0; gi < G; gi++) cur[gi] = id[gi] != NONE ? __ldcg(&g.val32[id[gi]]) : 0u;
  uint32_t sv[PULL_DEPTH];
  bool on[PULL_DEPTH];
#pragma unroll
  for (int k = 0; k < PULL_DEPTH; k++) {
    on[k] = S_::nbr(e[k]) != NONE && pull_open<A>(m, S_::wt(e[k]), cur[k / NP]);
    sv[k] = on[k] ? pull_src_val(g, S_::nbr(e[k])) : 0u;
  }
#pragma unroll
  for (int gi = 0; gi < G; gi++) {
    PullRow p = {cur[gi], 0u, 0u, false};
#pragma unroll
    for (int k = 0; k < NP; k++) pull_take<A, W>(e[gi * NP + k], sv[gi * NP + k], on[gi * NP + k], p);
    // (a row this narrow is a vertex)
    pull_row_done<A>(g, id[gi] != NONE, id[gi], p, PullHubs{}, q, fout, fout_n, mst, local, fb);
  }
}

// What one launch of a pull level covers: the slices of the hubs and their
// pieces (PART_HUBS), every slice after them (PART_REST), all slices
// (PART_ALL), none (PART_NONE), or the wide slices [s_lo, s_hi), and with
// `rest` the narrow ones too (PART_RANGE, grouped pull levels).  The bounds of
// the named parts come from the plan in device memory, so that the cached loop
// graph outlives the copy it was captured for.
enum PullPart : int { PART_HUBS, PART_REST, PART_ALL, PART_NONE, PART_RANGE };

// (q_buf: this warp's PQ_CAP words of shared memory)
template <int A, bool W>
__device__ __forceinline__ void pull_part(const DevGraph &g, const typename SellE<W>::E *ent, const uint64_t *off,
                                          const uint32_t *row_id, const PullHubs &hubs, const SellPlan *plan,
                                          int part, uint32_t s_lo, uint32_t s_hi, int rest, uint32_t m,
                                          unsigned long long *bout, uint32_t *q_buf, uint32_t *fout,
                                          unsigned long long *fout_n, uint32_t mst, BlockCounts *bc, bool first,
                                          uint32_t warp, uint32_t nwarps) {
  using S_ = SellE<W>;
  constexpr bool rev = A == RG_SSWP;  // heaviest entries first
  constexpr bool by_w = W && (A == RG_SSSP || A == RG_SSWP);
  constexpr bool by_id = !W && A == RG_WCC;
  constexpr int N = PULL_DEPTH;
  const uint32_t rows = (uint32_t)plan->rows, c4 = plan->slice[4];
  if (part != PART_RANGE) {
    const uint32_t mid = plan->slice[PULL_HUB];
    s_lo = part == PART_REST ? mid : 0;
    s_hi = part == PART_HUBS ? mid : c4;
    rest = part != PART_HUBS;
  }
  // the warps' work items: the wide slices one by one, then the narrow ones
  // in groups of 2, 4 and 8, so that on a small graph, where each warp has one
  // item, the classes run side by side
  const uint32_t c2 = plan->slice[2], c1 = plan->slice[1], slices = (uint32_t)plan->slices;
  const uint32_t n1 = s_hi - s_lo, n2 = rest ? (c2 - c4 + 1) / 2 : 0, n4 = rest ? (c1 - c2 + 3) / 4 : 0,
                 n8 = rest ? (slices - c1 + 7) / 8 : 0;
  const int lane = lane_id();
  PullQueue q = {q_buf, 0u};
  uint32_t fb = pull_worst<A>();
  uint32_t local = 0, chunks = 0;
  unsigned long long scanned = 0;
  for (uint32_t i = warp; i < n1 + n2 + n4 + n8; i += nwarps) {
    if (i >= n1) {
      const uint32_t x = i - n1;
      if (x < n2)
        pull_narrow<A, W, 2>(g, ent, off, row_id, rows, c4 + 2 * x, c2, m, q, fout, fout_n, mst, local, fb);
      else if (x < n2 + n4)
        pull_narrow<A, W, 4>(g, ent, off, row_id, rows, c2 + 4 * (x - n2), c1, m, q, fout, fout_n, mst, local, fb);
      else
        pull_narrow<A, W, 8>(g, ent, off, row_id, rows, c1 + 8 * (x - n2 - n4), slices, m, q, fout, fout_n, mst, local,
                             fb);
      continue;
    }
    const uint32_t s = s_lo + i, r = s * 32 + lane;
    const uint32_t id = r < rows ? row_id[r] : NONE;
    const bool active = id != NONE;
    const uint64_t o0 = off[s];
    const uint32_t width = (uint32_t)((off[s + 1] - o0) >> 5);
    const typename S_::E *col = ent + o0 + lane;
    auto load = [&](typename S_::E(&x)[N], uint32_t j, bool on) {
#pragma unroll
      for (int k = 0; k < N; k++)
        x[k] = on && j + k < width ? __ldcs(&col[(rev ? width - 1 - (j + k) : j + k) * 32]) : S_::none();
    };
    typename S_::E e[N];
    load(e, 0, true);  // (the first entries travel with the row's value)
    PullRow p = {0u, 0u, 0u, false};
    if (active) p.best = __ldcg(&g.val32[id < g.V ? id : hubs.piece_v[id - g.V]]);
    bool live = active && pull_open<A>(m, A == RG_SSWP ? 0xFFFFFFFFu : 0u, p.best);
    // takes the entries held and says whether the row goes on
    auto take = [&](uint32_t next) -> bool {
      uint32_t sv[N];
      bool on[N];
#pragma unroll
      for (int k = 0; k < N; k++) {
        on[k] = live && S_::nbr(e[k]) != NONE && pull_open<A>(m, S_::wt(e[k]), p.best);
        sv[k] = on[k] ? pull_src_val(g, S_::nbr(e[k])) : 0u;
      }
#pragma unroll
      for (int k = 0; k < N; k++) pull_take<A, W>(e[k], sv[k], on[k], p);
      chunks += live;
      if (next >= width) return false;
      if constexpr (by_w) {
        // padding ends a row read forwards and comes first in one read backwards
        if (S_::nbr(e[N - 1]) == NONE) live = live && rev;
        else live = live && pull_more<A>(m, S_::wt(e[N - 1]), p.best);
      } else {
        live = live && pull_open<A>(m, 0u, p.best);
        // WCC's first level starts with every label its vertex's id, and the
        // rows are in order of ids: the sources still to come start above the
        // best (those that changed in this level are in the next frontier)
        if (by_id && first)
          live = live && S_::nbr(e[N - 1]) != NONE && better32<A>(w_floor(S_::nbr(e[N - 1])), p.best);
      }
      return __any_sync(FULL, live);
    };
    if (take(N)) {
      // past its first entries a row is likely to go on: the next ones are on
      // their way while these are taken
      load(e, N, live);
      for (uint32_t j = 2 * N;; j += N) {
        typename S_::E ne[N];
        load(ne, j, live);
        if (!take(j)) break;
#pragma unroll
        for (int k = 0; k < N; k++) e[k] = ne[k];
      }
    }
    pull_row_done<A>(g, active, id, p, hubs, q, fout, fout_n, mst, local, fb);
  }
  scanned += (unsigned long long)chunks * N;
  if (rest && blockIdx.x == 0 && threadIdx.x == 0) scanned += off[slices] - off[c4];
  pull_drain(q, fout, fout_n);
  pull_bound_out<A>(fb, bout);
  block_count(bc, local, scanned);
}

// A CTA's counts into the control block (all threads of the CTA).
__device__ __forceinline__ void counts_out(const DevGraph &g, BlockCounts *bc) {
  __syncthreads();
  if (threadIdx.x == 0) {
    if (bc->updates) atomicAdd(&g.ctl[C_RESULT], bc->updates);
    if (bc->scanned) atomicAdd(&g.ctl[C_EDGES], bc->scanned);
  }
}

template <int A, bool W>
__global__ void __launch_bounds__(PS_TPB, PULL_CTAS)
    k_pull_sell(DevGraph g, const typename SellE<W>::E *ent, const uint64_t *off, const uint32_t *row_id, PullHubs hubs,
                const SellPlan *plan, int part, uint32_t s_lo, uint32_t s_hi, int rest, const unsigned long long *bin,
                unsigned long long *bout, uint32_t *fout, unsigned long long *fout_n, uint32_t mst) {
  if (g.ctl[C_MODE] != M_PULL || part == PART_NONE) return;
  __shared__ uint32_t s_q[PS_TPB / 32][PQ_CAP];
  __shared__ BlockCounts s_bc;
  if (threadIdx.x == 0) s_bc = BlockCounts{0, 0};
  __syncthreads();
  pull_part<A, W>(g, ent, off, row_id, hubs, plan, part, s_lo, s_hi, rest, (uint32_t)*bin, bout, s_q[threadIdx.x >> 5],
                  fout, fout_n, mst, &s_bc, g.ctl[C_DEPTH] == 0, (blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                  (gridDim.x * blockDim.x) >> 5);
  counts_out(g, &s_bc);
}

// The best piece of each hub, one lane per hub, one write (pieces only compete
// when they improve their hub).
template <int A>
__device__ __forceinline__ void pull_hub_fix(const DevGraph &g, const PullHubs &hubs, const SellPlan *plan,
                                             unsigned long long *bout, uint32_t *fout, unsigned long long *fout_n,
                                             uint32_t mst, unsigned long long &local, uint64_t gtid,
                                             uint64_t gthreads) {
  const uint64_t nh = plan->hubs;
  uint32_t fb = pull_worst<A>();
  for (uint64_t h0 = gtid - lane_id(); h0 < nh; h0 += gthreads) {
    const uint64_t h = h0 + lane_id();
    const unsigned long long b = h < nh ? __ldcg(&hubs.hub_best[h]) : ~0ull;
    const bool upd = b != ~0ull;
    uint32_t v = 0;
    if (upd) {
      v = hubs.hub_v[h];
      const ulonglong2 lab = __ldcg(&hubs.piece_best[(uint32_t)b]);
      hubs.hub_best[h] = ~0ull;
      g.lab[v] = lab;
      g.val32[v] = (uint32_t)lab.x;
      if (better32<A>((uint32_t)lab.x, fb)) fb = (uint32_t)lab.x;
    }
    local += upd;
    warp_append(upd, v, fout, fout_n, FULL);
    if (mst) mark_modified(g, upd, v, mst);
  }
  pull_bound_out<A>(fb, bout);
}

template <int A>
__global__ void __launch_bounds__(256) k_pull_hub_fix(DevGraph g, PullHubs hubs, const SellPlan *plan,
                                                      unsigned long long *bout, uint32_t *fout,
                                                      unsigned long long *fout_n, uint32_t mst) {
  if (g.ctl[C_MODE] != M_PULL) return;
  unsigned long long local = 0;
  pull_hub_fix<A>(g, hubs, plan, bout, fout, fout_n, mst, local, blockIdx.x * (uint64_t)blockDim.x + threadIdx.x,
                  (uint64_t)gridDim.x * blockDim.x);
  warp_add_result(local, &g.ctl[C_RESULT]);
}

// Bottom-up BFS level for full builds (the reference's dense pull,
// core/graph.hpp:936-976, specialised to BFS): every unreached vertex scans
// its in-edges and takes the first in-neighbour at depth d as its parent,
// stopping there.  Used when the frontier is large; each vertex is written
// only by its own thread, so no atomics on labels.
// Most vertices find a parent in the first few entries: each thread reads up to
// BU_ALONE of its own list, four at a time (the search is a chain of dependent
// loads), and the warp then searches what is left of each longer list together.
constexpr uint32_t BU_ALONE = 8;
template <bool W>
__device__ __forceinline__ void bottom_up(const DevGraph &g, uint64_t d, uint32_t *fout, unsigned long long *fout_n,
                                          uint64_t gtid, uint64_t gthreads, uint32_t *q_buf, BlockCounts *bc) {
  PullQueue q = {q_buf, 0u};
  unsigned long long local = 0, scanned = 0;
  using P_ = PoolT<W>;
  const typename P_::E *pool = reinterpret_cast<const typename P_::E *>(g.in.pool);
  const uint64_t V = g.V;
  const int lane = lane_id();
  // (a stale value only hides a parent found this level)
  auto is_parent = [&](uint32_t u) { return !(u & DEAD) && __ldca(&g.val32[u]) == (uint32_t)d; };
  for (uint64_t v0 = gtid - lane; v0 < V; v0 += gthreads) {
    const uint64_t v = v0 + lane;
    uint32_t parent = NONE, pw = 0, len = 0;
    uint64_t off = 0;
    if (v < V && ld_v32(g.val32, (uint32_t)v) == BFS_MAXL) {
      len = seg_len(g.in, (uint32_t)v);
      off = g.in.off[v];
      for (uint32_t k = 0; k < len && k < BU_ALONE && parent == NONE; k += 4) {
        typename P_::E e[4];
        bool ok[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
          if (k + i < len) e[i] = pool[off + k + i];
#pragma unroll
        for (int i = 0; i < 4; i++) ok[i] = k + i < len && is_parent(P_::nbr(e[i]));
        scanned += min(4u, len - k);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          if (parent == NONE && ok[i]) {
            parent = P_::nbr(e[i]);
            pw = P_::wt(e[i]);
          }
        }
      }
    }
    for (unsigned rest = __ballot_sync(FULL, parent == NONE && len > BU_ALONE); rest; rest &= rest - 1) {
      const int l = __ffs(rest) - 1;
      const uint32_t n = __shfl_sync(FULL, len, l);
      const uint64_t o = __shfl_sync(FULL, off, l);
      for (uint32_t k = BU_ALONE; k < n; k += 64) {
        typename P_::E e[2];
        bool ok[2];
#pragma unroll
        for (int i = 0; i < 2; i++)
          if (k + 32 * i + lane < n) e[i] = pool[o + k + 32 * i + lane];
#pragma unroll
        for (int i = 0; i < 2; i++) ok[i] = k + 32 * i + lane < n && is_parent(P_::nbr(e[i]));
        if (lane == l) scanned += min(64u, n - k);
        if ((k - BU_ALONE) / 64 % BEAT_STEPS == BEAT_STEPS - 1 && lane == 0) beat(g);
        const unsigned hit = __ballot_sync(FULL, ok[0] || ok[1]);
        if (hit) {
          const int h = __ffs(hit) - 1;
          const uint32_t hp = __shfl_sync(FULL, ok[0] ? P_::nbr(e[0]) : P_::nbr(e[1]), h);
          const uint32_t hw = __shfl_sync(FULL, ok[0] ? P_::wt(e[0]) : P_::wt(e[1]), h);
          if (lane == l) {
            parent = hp;
            pw = hw;
          }
          break;
        }
      }
    }
    const bool found = parent != NONE;
    if (found) {
      g.lab[v] = make_ulonglong2(d + 1, pack_parent(parent, pw));
      g.val32[v] = (uint32_t)(d + 1);
    }
    local += found;
    pull_append(q, found, (uint32_t)v, fout, fout_n);
  }
  pull_drain(q, fout, fout_n);
  block_count(bc, local, scanned);
}

template <bool W>
__global__ void __launch_bounds__(TPB) k_bfs_bottom_up(DevGraph g, uint32_t *fout, unsigned long long *fout_n) {
  if (g.ctl[C_MODE] != M_BOTTOM_UP) return;
  __shared__ uint32_t s_q[TPB / 32][PQ_CAP];
  __shared__ BlockCounts s_bc;
  if (threadIdx.x == 0) s_bc = BlockCounts{0, 0};
  __syncthreads();
  bottom_up<W>(g, g.ctl[C_DEPTH], fout, fout_n, blockIdx.x * (uint64_t)blockDim.x + threadIdx.x,
               (uint64_t)gridDim.x * blockDim.x, s_q[threadIdx.x >> 5], &s_bc);
  counts_out(g, &s_bc);
}

// ---- small frontiers: several levels in one CTA -----------------------------
// Incremental repairs and the tail of a build run many levels whose frontier
// is a handful of vertices; one launch per level would cost more than the
// work.  k_push_tiny takes a frontier of at most TINY_N vertices and
// TINY_EDGES out-slots and keeps relaxing level after level inside one CTA
// (CTA barriers between levels), until the frontier empties or outgrows those
// limits; the frontier it leaves is in the level's output queue, as after any
// other level kernel.  Each slot is found by a binary search of the frontier's
// degree prefix in shared memory.
constexpr uint32_t TINY_N = 1024;
constexpr uint64_t TINY_EDGES = 1ull << 20;
constexpr int TINY_TPB = 1024;

//
// tiny_levels is that loop as a device function for a CTA of TINY_TPB threads:
// it leaves the frontier in q_final (one of q_in, q_out) with its count in
// *n_final.  first_begun: k_level_begin did the first level's bookkeeping (the
// level counter, stamp, depth and trace); otherwise the loop does it for every
// level, the first included.
template <int A, bool W>
__device__ __forceinline__ void tiny_levels(const DevGraph &g, uint32_t *q_in, unsigned long long *n_in,
                                            uint32_t *q_out, unsigned long long *n_out, uint32_t *q_final,
                                            unsigned long long *n_final, uint64_t max_levels, uint64_t max_edges,
                                            uint32_t mst, bool first_begun) {
  using P_ = PoolT<W>;
  using Scan = cub::BlockScan<uint32_t, TINY_TPB>;
  __shared__ typename Scan::TempStorage scan_tmp;
  __shared__ uint32_t s_pref[TINY_N + 1];
  __shared__ uint32_t s_v[TINY_N];
  __shared__ uint64_t s_off[TINY_N];
  __shared__ uint32_t s_su[TINY_N];
  __shared__ int s_go;
  const typename P_::E *pool = reinterpret_cast<const typename P_::E *>(g.out.pool);
  unsigned long long *c = g.ctl;
  const unsigned tid = threadIdx.x;
  uint32_t *cur = q_in, *nxt = q_out;
  unsigned long long *cur_n = n_in, *nxt_n = n_out;
  unsigned long long local = 0, scanned = 0;
  for (bool first = true;; first = false) {
    const uint64_t n = *cur_n;
    // stage the frontier and its degree prefix
    uint32_t d = 0;
    if (n <= TINY_N && tid < n) {
      const uint32_t u = cur[tid];
      s_v[tid] = u;
      s_off[tid] = g.out.off[u];
      s_su[tid] = (uint32_t)ld_v32(g.val32, u);
      d = seg_len(g.out, u);
    }
    uint32_t excl, total;
    Scan(scan_tmp).ExclusiveSum(d, excl, total);
    if (tid < TINY_N) s_pref[tid] = excl;
    if (tid == 0) {
      s_pref[TINY_N] = total;
      bool go = n > 0 && n <= TINY_N && total <= max_edges;
      if ((!first || !first_begun) && go) {
        // a new level: the bookkeeping k_level_begin does for the first one
        const uint64_t lvl = c[C_LEVEL];
        go = lvl < max_levels;
        if (go) {
          c[C_STAMP] += 1;
          c[C_DEPTH] = lvl;
          if (lvl < TRACE_CAP) {
            g.trace[lvl] = n;
            g.trace[TRACE_CAP + lvl] = global_ns();
          }
          c[C_LEVEL] = lvl + 1;
          *nxt_n = 0;
        }
      }
      s_go = go;
    }
    __syncthreads();
    if (!s_go) break;
    const uint32_t st = (uint32_t)c[C_STAMP];
    for (uint32_t base = 0; base < total; base += TINY_TPB) {
      const uint32_t e = base + tid;
      bool upd = false;
      uint32_t v = 0;
      if (e < total) {
        uint32_t lo = 0, hi = (uint32_t)n - 1;
        while (lo < hi) {
          const uint32_t mid = (lo + hi + 1) >> 1;
          if (s_pref[mid] <= e) lo = mid;
          else hi = mid - 1;
        }
        const typename P_::E ent = pool[s_off[lo] + (e - s_pref[lo])];
        v = P_::nbr(ent);
        scanned++;
        if (!(v & DEAD)) upd = relax_lab<A>(g, s_v[lo], s_su[lo], v, P_::wt(ent));
      }
      local += upd;
      const bool app = upd && atomicExch(&g.stamp[v], st) != st;
      warp_append(app, v, nxt, nxt_n, FULL);
      if (mst) mark_modified(g, upd, v, mst);
    }
    __syncthreads();  // the next level reads the queue this one wrote
    uint32_t *t = cur;
    cur = nxt;
    nxt = t;
    unsigned long long *tn = cur_n;
    cur_n = nxt_n;
    nxt_n = tn;
  }
  if (cur != q_final) {
    const uint64_t n = *cur_n;
    for (uint64_t i = tid; i < n; i += TINY_TPB) q_final[i] = cur[i];
    __syncthreads();
    if (tid == 0) *n_final = n;
  }
  __syncthreads();
  warp_add_result(local, &c[C_RESULT]);
  warp_add_result(scanned, &c[C_EDGES]);
}

// The frontier is left in the output queue of the level the launch stands for.
template <int A, bool W>
__global__ void __launch_bounds__(TINY_TPB) k_push_tiny(DevGraph g, uint32_t *q_in, unsigned long long *n_in,
                                                        uint32_t *q_out, unsigned long long *n_out,
                                                        uint64_t max_levels, uint64_t max_edges, uint32_t mst) {
  if (g.ctl[C_MODE] != M_TINY) return;
  tiny_levels<A, W>(g, q_in, n_in, q_out, n_out, q_out, n_out, max_levels, max_edges, mst, true);
}

// ---- cluster levels ------------------------------------------------------------
// (Levels of the host-stepped loop, and of the graph-driven one on a GPU that
// launches no cooperative grid; the grid engine runs the others.)
// A frontier too large for one CTA but at most CL_TPB vertices per CTA of a
// thread-block cluster (16 CTAs where the GPU schedules a cluster that size,
// else 8; one per SM) runs in k_push_cluster: successive levels inside one
// launch, separated by the hardware cluster barrier (barrier.cluster, with
// release/acquire ordering of the global queue and labels) instead of kernel
// boundaries and a conditional node per level, which cost 25-40 us per
// mid-size level in the graph-driven loop.  Each CTA stages CL_TPB frontier
// vertices (offset, value, degree prefix) in its shared memory; the level's
// out-slots are spread evenly over every thread of the cluster, and a thread
// finds the vertex of its slot in the owning CTA's shared memory through
// distributed shared memory.  Every decision that ends the loop is made from
// values that all CTAs read alike (the frontier size after a barrier, the
// CTAs' slot totals in global memory), so that every CTA passes the same
// barriers.  The loop ends when the frontier empties or outgrows the cluster
// (more than CL_TPB vertices per CTA or max_edges slots), leaving the frontier
// in the level's output queue like tiny_levels.
constexpr int CL_TPB = 1024;
constexpr int CL_MAX_CTAS = 16;
constexpr uint64_t CL_EDGES = 1ull << 20;  // largest slot limit of a cluster level

template <int A, bool W>
__global__ void __launch_bounds__(CL_TPB, 1)
    k_push_cluster(DevGraph g, uint32_t *q_in, unsigned long long *n_in, uint32_t *q_out, unsigned long long *n_out,
                   unsigned long long *tot, uint64_t max_levels, uint64_t max_edges, uint32_t mst) {
  namespace cgr = cooperative_groups;
  if (g.ctl[C_MODE] != M_CLUSTER) return;  // the same in every CTA
  cgr::cluster_group cluster = cgr::this_cluster();
  using P_ = PoolT<W>;
  using Scan = cub::BlockScan<uint32_t, CL_TPB>;
  __shared__ typename Scan::TempStorage scan_tmp;
  __shared__ uint32_t s_pref[CL_TPB + 1];
  __shared__ uint32_t s_v[CL_TPB];
  __shared__ uint64_t s_off[CL_TPB];
  __shared__ uint32_t s_su[CL_TPB];
  __shared__ uint64_t s_base[CL_MAX_CTAS + 1];
  const typename P_::E *pool = reinterpret_cast<const typename P_::E *>(g.out.pool);
  unsigned long long *c = g.ctl;
  const unsigned tid = threadIdx.x;
  const unsigned nc = cluster.num_blocks(), r = cluster.block_rank();
  const uint64_t cap = (uint64_t)nc * CL_TPB;  // frontier vertices the cluster stages
  uint32_t *cur = q_in, *nxt = q_out;
  unsigned long long *cur_n = n_in, *nxt_n = n_out;
  unsigned long long local = 0, scanned = 0;
  uint64_t n = 0;
  for (bool first = true;; first = false) {
    // values every CTA reads alike: written before the last barrier (or the launch)
    n = __ldcg(cur_n);
    const unsigned long long st0 = __ldcg(&c[C_STAMP]), lvl = __ldcg(&c[C_LEVEL]);
    const bool book = !first;  // k_level_begin did the first level's bookkeeping
    const uint64_t i = (uint64_t)r * CL_TPB + tid;
    uint32_t d = 0;
    if (n <= cap && i < n) {
      const uint32_t u = __ldcg(&cur[i]);
      s_v[tid] = u;
      s_off[tid] = g.out.off[u];
      s_su[tid] = (uint32_t)ld_v32(g.val32, u);
      d = seg_len(g.out, u);
    }
    uint32_t excl, total;
    Scan(scan_tmp).ExclusiveSum(d, excl, total);
    s_pref[tid] = excl;
    if (tid == 0) {
      s_pref[CL_TPB] = total;
      tot[r] = total;
      // the output count: the input of the level before this one, read by every CTA
      // before the last barrier
      if (r == 0 && book) *nxt_n = 0;
    }
    cluster.sync();  // A: totals and stage visible, output count cleared
    if (tid < 32) {
      // the CTAs' slot totals, loaded together and scanned in one warp
      const uint64_t t = tid < nc ? __ldcg(&tot[tid]) : 0;
      uint64_t incl = t;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(FULL, incl, o);
        if (tid >= (unsigned)o) incl += y;
      }
      if (tid <= nc) s_base[tid] = incl - t;  // entry nc: the level's slots
    }
    __syncthreads();
    const uint64_t S = s_base[nc];
    const bool go = n > 0 && n <= cap && (first || (S <= max_edges && lvl < max_levels));
    if (!go) break;  // the same in every CTA
    if (book && r == 0 && tid == 0) {
      c[C_STAMP] = st0 + 1;
      c[C_DEPTH] = lvl;
      if (lvl < TRACE_CAP) {
        g.trace[lvl] = n;
        g.trace[TRACE_CAP + lvl] = global_ns();
      }
      c[C_LEVEL] = lvl + 1;
    }
    const uint32_t st = (uint32_t)(book ? st0 + 1 : st0);
    for (uint64_t base = 0; base < S; base += cap) {
      const uint64_t e = base + i;
      bool upd = false;
      uint32_t v = 0;
      if (e < S) {
        unsigned k = 0;  // the CTA that staged slot e: largest k with s_base[k] <= e
        while (k + 1 < nc && s_base[k + 1] <= e) k++;
        const uint32_t el = (uint32_t)(e - s_base[k]);
        const uint32_t *rp = cluster.map_shared_rank(s_pref, k);
        const uint64_t left = n - (uint64_t)k * CL_TPB;
        const uint64_t nk = left < CL_TPB ? left : CL_TPB;
        uint32_t lo = 0, hi = (uint32_t)nk - 1;  // largest j with rp[j] <= el
        while (lo < hi) {
          const uint32_t mid = (lo + hi + 1) >> 1;
          if (rp[mid] <= el) lo = mid;
          else hi = mid - 1;
        }
        const uint64_t off = *cluster.map_shared_rank(&s_off[lo], k);
        const uint32_t u = *cluster.map_shared_rank(&s_v[lo], k);
        const uint32_t su = *cluster.map_shared_rank(&s_su[lo], k);
        const typename P_::E ent = __ldg(&pool[off + (el - rp[lo])]);
        v = P_::nbr(ent);
        scanned++;
        if (!(v & DEAD)) upd = relax_lab<A>(g, u, su, v, P_::wt(ent));
      }
      local += upd;
      const bool app = upd && atomicExch(&g.stamp[v], st) != st;
      warp_append(app, v, nxt, nxt_n, FULL);
      if (mst) mark_modified(g, upd, v, mst);
    }
    cluster.sync();  // B: this level's queue and labels visible; nobody reads a peer's stage any more
    uint32_t *t = cur;
    cur = nxt;
    nxt = t;
    unsigned long long *tn = cur_n;
    cur_n = nxt_n;
    nxt_n = tn;
  }
  // the frontier that ended the loop goes to the launch's output queue
  if (cur != q_out) {
    for (uint64_t k = (uint64_t)r * CL_TPB + tid; k < n; k += cap) q_out[k] = __ldcg(&cur[k]);
    if (r == 0 && tid == 0) *n_out = n;
  }
  warp_add_result(local, &c[C_RESULT]);
  warp_add_result(scanned, &c[C_EDGES]);
}

// ---- device-driven level loop ------------------------------------------------
// A tree call runs k_prologue, its seed kernel, then a CUDA graph whose WHILE
// node repeats a pair of levels (queue 0 -> 1, then 1 -> 0).  Each level
// starts with k_level_begin, which reads the frontier size and picks the level
// mode and stamp on the device; every level kernel returns at once unless the
// mode is its own; k_loop_cond stops the loop when the frontier is empty.  No
// host round trip happens between levels (the reference's driver decides
// between levels on the host, core/graph.hpp:898-983, :1013-1111).

// (all of it but the frontier stamp)
__device__ __forceinline__ void prologue_words(unsigned long long *c, unsigned long long inv_tag) {
  c[C_INVTAG] = inv_tag;
  c[C_INVITER] = 0;
  c[C_OVER] = 0;
  c[C_QN0] = 0;
  c[C_QN1] = 0;
  c[C_HUBN] = 0;
  c[C_RESULT] = 0;
  c[C_TREEN] = 0;
  c[C_RECOMPUTE] = 0;
  c[C_LEVEL] = 0;
  c[C_EDGES] = 0;
  c[C_MODE] = M_EMPTY;
  c[C_KLAUNCH] = 0;
  c[C_ELEFT] = 0;
  c[C_HVR] = 0;
  c[C_HVE] = 0;
  c[C_HVP] = 0;
}

// stamp: the control block's C_STAMP when the caller read it already.
__device__ __forceinline__ void prologue_ctl(unsigned long long *c, unsigned long long inv_tag,
                                             const unsigned long long *stamp = nullptr) {
  prologue_words(c, inv_tag);
  c[C_STAMP] = (stamp ? *stamp : c[C_STAMP]) + 1;
}

__global__ void k_prologue(DevGraph g, unsigned long long inv_tag) { prologue_ctl(g.ctl, inv_tag); }

// Kernels a level of each mode launches (k_level_begin not included).
__host__ __device__ __forceinline__ int mode_launches(unsigned long long mode) {
  switch (mode) {
    case M_SPARSE: return 2;
    case M_PULL: return 3;
    case M_DENSE_PUSH: return 2;
    case M_BOTTOM_UP: return 1;
    case M_LBS: return 5;
    case M_TINY: return 1;
    case M_CLUSTER: return 1;
  }
  return 0;
}

struct LevelCfg {
  uint64_t dense_div;
  uint64_t lbs_min;
  uint64_t bu_div;    // BFS builds go bottom-up once frontier * bu_div >= |V|
  uint64_t pull_div;  // builds pull once frontier * pull_div >= |V|
  uint64_t pull_split;  // pull levels run in two launches
  uint64_t tiny_edges;
  uint64_t max_levels;  // level bound baked into the loop graphs
  uint64_t pull_groups;  // launches of a split pull level
  uint64_t cl_edges;     // out-slot limit of a cluster level (0: no cluster levels)
  uint64_t cl_v;         // frontier vertices a cluster stages (its CTAs x CL_TPB)
  int allow_pull;
  int bottom_up;
  uint32_t bnd_best, bnd_worst;  // the best and the worst value of the hook's order
};

// Picks the level mode from the frontier size (the reference's push/pull rule
// at core/graph.hpp:334 and its vertex/edge-centric rule at :595-612 play the
// same role); inside a graph it also selects the SWITCH case to run.
// Threads of k_level_begin (they sum small frontiers' degrees).  256, not
// 1024: the kernel starts every level, and in served mode the epochs of other
// instances occupy the SMs, where a 1024-thread CTA waits longer for room.
constexpr int LVB_TPB = 256;
// A frontier that both a tiny level and a cluster level could take goes to the
// cluster when it has more out-slots than this: one CTA walks them
// 1024 at a time, the cluster 16,384 at a time.
constexpr uint64_t CL_TINY_PREF = 4096;

__global__ void __launch_bounds__(LVB_TPB) k_level_begin(DevGraph g, const uint32_t *fin,
                                                         const unsigned long long *fin_n, unsigned long long *fout_n,
                                                         LevelCfg cfg, int use_switch, cudaGraphConditionalHandle sw) {
  using BR = cub::BlockReduce<unsigned long long, LVB_TPB>;
  __shared__ typename BR::TempStorage br_tmp;
  const uint64_t n0 = *fin_n;
  unsigned long long d = 0;
  if ((cfg.tiny_edges && n0 && n0 <= TINY_N) || (cfg.cl_edges && n0 && n0 <= cfg.cl_v)) {
    // eight frontier entries per thread in flight (a frontier of up to 16K vertices)
    for (uint64_t i0 = threadIdx.x; i0 < n0; i0 += 8 * LVB_TPB) {
      uint32_t u[8];
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const uint64_t i = i0 + (uint64_t)k * LVB_TPB;
        u[k] = i < n0 ? fin[i] : NONE;
      }
#pragma unroll
      for (int k = 0; k < 8; k++) d += u[k] != NONE ? seg_len(g.out, u[k]) : 0u;
    }
  }
  // a tree reduction: 1024 threads adding into one shared word contend for it
  const unsigned long long s_edges = BR(br_tmp).Sum(d);  // valid in thread 0
  if (threadIdx.x != 0) return;
  const bool tiny = cfg.tiny_edges && n0 && n0 <= TINY_N && s_edges <= cfg.tiny_edges;
  const bool clus = cfg.cl_edges && n0 && n0 <= cfg.cl_v && s_edges <= cfg.cl_edges;
  unsigned long long *c = g.ctl;
  const uint64_t n = n0;
  const uint64_t lvl = c[C_LEVEL];
  *fout_n = 0;
  c[C_ELEFT] = 0;
  c[C_HUBN] = 0;
  c[C_STAMP] += 1;
  c[C_DEPTH] = lvl;
  const bool dense = n * cfg.dense_div >= g.V;
  unsigned long long mode = M_SPARSE;
  if (n == 0) mode = M_EMPTY;
  // (a pull level commits values deeper than the level, which a bottom-up level,
  // looking for parents of one depth, would miss: none follows a pull)
  else if (cfg.bottom_up && !(lvl && c[C_PULLED]) && n * cfg.bu_div >= g.V) mode = M_BOTTOM_UP;
  // pull once the frontier passes |V| / pull_div, and keep pulling until it
  // falls below 4x that (the frontier's first large levels are hub-heavy, its
  // last ones are not: the direction switch of Beamer et al., by vertex count)
  else if (cfg.allow_pull && n * (c[C_MODE] == M_PULL ? (cfg.pull_div + 3) / 4 : cfg.pull_div) >= g.V) mode = M_PULL;
  else if (tiny && !(clus && s_edges > CL_TINY_PREF)) mode = M_TINY;
  else if (clus) mode = M_CLUSTER;
  else if (dense) mode = M_DENSE_PUSH;
  else if (n >= cfg.lbs_min) mode = M_LBS;
  if (mode == M_DENSE_PUSH) c[C_ACT] += 1;
  if (lvl == 0 || mode == M_PULL) c[C_PULLED] = mode == M_PULL;
  c[C_MODE] = mode;
  // bounds on the frontiers' values: pull levels collect theirs, others give none
  const int half = fin_n == &c[C_QN0] ? 0 : 1;
  if (lvl == 0) c[C_BND0 + half] = cfg.bnd_best;
  c[C_BND0 + (half ^ 1)] = mode == M_PULL ? cfg.bnd_worst : cfg.bnd_best;
  if (use_switch) c[C_KLAUNCH] += 1 + mode_launches(mode) + (mode == M_PULL ? cfg.pull_groups - 2 : 0);
  if (n) {
    if (lvl < TRACE_CAP) {
      g.trace[lvl] = n;
      g.trace[TRACE_CAP + lvl] = global_ns();  // the level's start on the device clock
    }
    c[C_LEVEL] = lvl + 1;
  }
  if (use_switch) cudaGraphSetConditional(sw, (unsigned)mode);
}

__global__ void k_loop_cond(DevGraph g, const unsigned long long *n_after, uint64_t max_levels,
                            cudaGraphConditionalHandle handle) {
  const uint64_t n = *n_after;
  const uint64_t lvl = g.ctl[C_LEVEL];
  g.ctl[C_KLAUNCH] += 1;
  // the end of the levels so far (the next level's start overwrites it)
  if (lvl < TRACE_CAP) g.trace[TRACE_CAP + lvl] = global_ns();
  if (n && lvl >= max_levels) atomicCAS(&g.ctl[C_ERR], 0ull, (unsigned long long)RG_ETIMEOUT);
  cudaGraphSetConditional(handle, (n && lvl < max_levels) ? 1u : 0u);
}

// Deletion repair loop control (do_update_tree_del, core/graph.hpp:1250-1418):
// one invalidation level per k_inv_begin; the full-recompute fallback
// (:1252) stops the loop and turns the rest of the repair into no-ops.
__global__ void k_inv_begin(DevGraph g, const unsigned long long *fin_n, unsigned long long *fout_n, uint64_t big) {
  unsigned long long *c = g.ctl;
  const uint64_t n = *fin_n;
  *fout_n = 0;
  c[C_HVR] = 0;
  c[C_HVE] = 0;
  c[C_KLAUNCH] += 5;  // this kernel, k_rescue, k_rescue_heavy, k_expand, k_expand_heavy
  if (n == 0 || c[C_RECOMPUTE]) return;
  const uint64_t it = c[C_INVITER];
  if (it <= 10 && c[C_TREEN] + n > big) c[C_RECOMPUTE] = 1;
  c[C_INVITER] = it + 1;
}

// in_graph = 0: launched by the host (profile mode); the condition goes to
// C_HOSTCOND instead of the WHILE node's handle.
__global__ void k_inv_cond(DevGraph g, const unsigned long long *n_after, uint64_t max_iter,
                           cudaGraphConditionalHandle handle, int in_graph) {
  unsigned long long *c = g.ctl;
  const uint64_t n = *n_after;
  c[C_KLAUNCH] += 1;
  const unsigned go = (n && !c[C_RECOMPUTE] && c[C_INVITER] < max_iter) ? 1u : 0u;
  if (in_graph) cudaGraphSetConditional(handle, go);
  else c[C_HOSTCOND] = go;
}

__global__ void k_copy_frontier(DevGraph g, const uint32_t *src, const unsigned long long *src_n, uint32_t *dst,
                                unsigned long long *dst_n) {
  if (blockIdx.x == 0 && threadIdx.x == 0) g.ctl[C_KLAUNCH] += 4;  // k_reset, k_pull, k_pull_heavy, this kernel
  if (g.ctl[C_RECOMPUTE]) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *dst_n = 0;
    return;
  }
  const uint64_t n = *src_n;
  if (blockIdx.x == 0 && threadIdx.x == 0) *dst_n = n;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += stride) dst[i] = src[i];
}

// build_tree init (core/graph.hpp:886-896): every label to init_label_func,
// parent to empty; the active set is the root, or every vertex (WCC).
template <int A>
__device__ __forceinline__ void init_labels(const DevGraph &g, uint64_t root, uint32_t *fout, uint64_t gtid,
                                            uint64_t stride) {
  for (uint64_t v = gtid; v < g.V; v += stride) {
    g.lab[v] = make_ulonglong2(Hook<A>::init(v, root), pack_parent(NONE, 0));
    g.val32[v] = (uint32_t)Hook<A>::init(v, root);
    if (Hook<A>::all_active) fout[v] = (uint32_t)v;
    else if (v == root) fout[0] = (uint32_t)v;
  }
}

template <int A>
__global__ void k_init(DevGraph g, uint64_t root, uint32_t *fout) {
  init_labels<A>(g, root, fout, blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, (uint64_t)gridDim.x * blockDim.x);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    g.ctl[C_QN0] = Hook<A>::all_active ? g.V : 1;
    g.ctl[C_ROOT] = root;
  }
}

// Seed relaxations of update_tree_add (single :1140-1153, batch :1180-1214):
// relax each inserted edge, both orientations when undirected.
template <int A>
__device__ __forceinline__ unsigned long long seed_add(const DevGraph &g, const uint32_t *os, const uint32_t *od,
                                                       const uint32_t *ow, const uint32_t *cand, uint64_t n,
                                                       int directed, uint32_t *fout, unsigned long long *fout_n,
                                                       uint32_t mst, uint64_t warp, uint64_t nwarps) {
  const uint32_t st = (uint32_t)g.ctl[C_STAMP];
  unsigned long long local = 0;
  for (uint64_t base = warp * 32; base < n; base += nwarps * 32) {
    uint64_t i = base + lane_id();
    for (int dir = 0; dir < (directed ? 1 : 2); dir++) {
      bool upd = false;
      uint32_t v = 0;
      if (i < n) {
        uint64_t e = cand ? cand[i] : i;
        uint64_t op = directed ? e : 2 * e + dir;
        uint32_t u = os[op];
        v = od[op];
        upd = relax<A>(g, u, ld_v32(g.val32, u), v, ow[op]);
      }
      local += upd;
      bool app = upd && atomicExch(&g.stamp[v], st) != st;
      warp_append(app, v, fout, fout_n, FULL);
      if (mst) mark_modified(g, upd, v, mst);
    }
  }
  return local;
}

template <int A>
__global__ void k_seed_add(DevGraph g, const uint32_t *os, const uint32_t *od, const uint32_t *ow, const uint32_t *cand,
                           const unsigned long long *cand_n, uint64_t n_all, int directed, uint32_t *fout,
                           unsigned long long *fout_n, uint32_t mst) {
  const uint64_t n = cand ? *cand_n : n_all;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long local = seed_add<A>(g, os, od, ow, cand, n, directed, fout, fout_n, mst, warp, nwarps);
  warp_add_result(local, &g.ctl[C_RESULT]);
}

// Seeds of update_tree_del (single :1640-1649, batch :1680-1714): a deleted
// edge that is dst's parent edge invalidates dst.
__device__ __forceinline__ void seed_del(const DevGraph &g, const uint32_t *os, const uint32_t *od, const uint32_t *ow,
                                         const uint32_t *cand, uint64_t n, int directed, uint32_t *fout,
                                         unsigned long long *fout_n, uint64_t warp, uint64_t nwarps) {
  const uint32_t tag_inv = (uint32_t)g.ctl[C_INVTAG];
  for (uint64_t base = warp * 32; base < n; base += nwarps * 32) {
    uint64_t i = base + lane_id();
    for (int dir = 0; dir < (directed ? 1 : 2); dir++) {
      bool app = false;
      uint32_t v = 0;
      if (i < n) {
        uint64_t e = cand ? cand[i] : i;
        uint64_t op = directed ? e : 2 * e + dir;
        uint32_t u = os[op];
        v = od[op];
        if (ld_meta(&g.lab[v]) == pack_parent(u, ow[op])) app = atomicExch(&g.inv[v], tag_inv) != tag_inv;
      }
      warp_append(app, v, fout, fout_n, FULL);
    }
  }
}

__global__ void k_seed_del(DevGraph g, const uint32_t *os, const uint32_t *od, const uint32_t *ow, const uint32_t *cand,
                           const unsigned long long *cand_n, uint64_t n_all, int directed, uint32_t *fout,
                           unsigned long long *fout_n) {
  const uint64_t n = cand ? *cand_n : n_all;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  seed_del(g, os, od, ow, cand, n, directed, fout, fout_n, warp, nwarps);
}

// has_parents (core/graph.hpp:1889-1907): does x's parent chain reach a root
// without meeting a vertex invalidated (or rescued) by this repair?  The chain
// guard (0.1 |V| steps) requests a full recompute, as the reference does.
//
// A chain found clear stays clear for the rest of the repair: tags only go to
// the tree descendants of vertices tagged before (the seeds are tagged first),
// and only tagged vertices change parent, so an untagged chain never gains a
// tag.  The walk therefore stops at a vertex marked clear earlier in this
// repair (chk == the repair's tag), and a clear walk marks the first vertices
// of its chain, so that walks from their descendants end there.
//
// The three words of a step are loaded together, so that a step costs one
// round trip to memory rather than three.
//
// On a deep tree the walks of one lane can take many seconds: every BEAT_STEPS
// steps a walk beats, and ends if the repair has already asked for a recompute
// (which makes its answer void).
__device__ __forceinline__ bool has_parents(const DevGraph &g, uint32_t x0, uint32_t tag_inv, uint64_t limit) {
  uint64_t num = 0;
  uint32_t x = x0;
  for (;;) {
    const uint32_t ck = ld_u32(&g.chk[x]);
    const uint32_t t = ld_u32(&g.inv[x]);
    const uint32_t p = (uint32_t)ld_meta(&g.lab[x]);
    if (ck == tag_inv) break;
    if (t == tag_inv || t == tag_inv + 1) return true;
    if (p == NONE) break;
    x = p;
    if (++num > limit) {
      atomicExch(&g.ctl[C_RECOMPUTE], 1ull);
      return true;
    }
    if (num % BEAT_STEPS == 0) {
      if (__ldcg(&g.ctl[C_RECOMPUTE])) return true;
      beat(g);
    }
  }
  x = x0;
  for (int k = 0; k < 16 && x != NONE && ld_u32(&g.chk[x]) != tag_inv; k++) {
    g.chk[x] = tag_inv;
    x = (uint32_t)ld_meta(&g.lab[x]);
  }
  return false;
}

// Rescue (core/graph.hpp:1323-1361): an invalidated dst keeps its value when an
// in-neighbour satisfies equal_func and has a clean parent chain; the parent
// moves to that in-edge.  One warp per frontier vertex.
// Heavy vertices: a warp per vertex would scan an RMAT hub's 10^5 edges 32 at
// a time.  The warp-per-vertex passes of the deletion repair (rescue, expand,
// the pull over the reset set) queue the vertices whose list is longer than
// HEAVY_DEG instead, and a second kernel spreads each queued vertex's list over
// every warp of the grid.  Without a queue (the one-CTA repair, which hands
// heavy vertices over to the grid-wide one) or when it is full, the warp scans
// the whole list itself.
constexpr uint32_t HEAVY_DEG = 2048;

__device__ __forceinline__ bool queue_heavy(uint32_t *hv, unsigned long long *hv_n, uint64_t hv_cap, uint32_t v,
                                            int lane) {
  unsigned long long k = 0;
  if (lane == 0) k = atomicAdd(hv_n, 1ull);
  k = __shfl_sync(FULL, k, 0);
  if (k < hv_cap) {
    if (lane == 0) hv[k] = v;
    return true;
  }
  return false;
}

// Rescue of one invalidated vertex d (value sd) by a warp, over slots [lo, len)
// of its in-list at off; returns whether d is rescued.
template <int A, bool W>
__device__ __forceinline__ bool rescue_one(const DevGraph &g, uint32_t d, uint64_t sd, uint32_t lo, uint32_t len,
                                           uint64_t off, uint32_t tag_inv, uint64_t limit) {
  using P = PoolT<W>;
  const typename P::E *pool = reinterpret_cast<const typename P::E *>(g.in.pool);
  const int lane = lane_id();
  for (uint32_t kb = lo; kb < len; kb += 32) {
    const uint32_t k = kb + lane;
    bool ok = false;
    uint32_t src = 0, w = 0;
    if (k < len) {
      typename P::E e = pool[off + k];
      src = P::nbr(e);
      w = P::wt(e);
      if (!(src & DEAD) && Hook<A>::combine(ld_v32(g.val32, src), w) == sd) ok = !has_parents(g, src, tag_inv, limit);
    }
    const unsigned b = __ballot_sync(FULL, ok);
    if (b) {  // the first candidate, unless another warp was first
      if (lane == __ffs(b) - 1 && atomicCAS(&g.inv[d], tag_inv, tag_inv + 1) == tag_inv)
        reinterpret_cast<unsigned long long *>(&g.lab[d])[1] = pack_parent(src, w);
      return true;
    }
    if (__shfl_sync(FULL, ld_u32(&g.inv[d]), 0) != tag_inv) return true;
  }
  return false;
}

// Long lists in the grid engine: a warp scans the first TASK_SLOTS slots of a
// list of more than TASK_DEG and queues the rest as tasks of TASK_SLOTS, which
// every warp of the grid takes after the next barrier.  (With whole lists of up
// to HEAVY_DEG to a warp, each pass of a batch of 100,000 deletions waited 70 us
// for its longest list.)
constexpr uint32_t TASK_DEG = 256, TASK_SLOTS = 128;
struct RepQueue {
  uint32_t *hv = nullptr;  // vertices left for a pass of their own ...
  unsigned long long *n = nullptr;
  uint64_t cap = 0;
  uint64_t *task = nullptr;  // ... or tasks (vertex | chunk << 32), with n their count
};
__device__ __forceinline__ void queue_tasks(const RepQueue &q, uint32_t v, uint32_t len, int lane) {
  const uint32_t nt = (len - 1) / TASK_SLOTS;  // chunks 1 .. nt
  unsigned long long at = 0;
  if (lane == 0) at = atomicAdd(q.n, (unsigned long long)nt);
  at = __shfl_sync(FULL, at, 0);
  for (uint32_t c = lane; c < nt; c += 32) q.task[at + c] = (uint64_t)v | ((uint64_t)(c + 1) << 32);
}

// The passes of the deletion repair over more vertices than there are warps
// take four vertices to a warp, eight lanes each: most lists are a few entries,
// and a pass is chains of dependent loads, not bandwidth.  (One vertex to a
// warp, the rescue of 517 vertices in the one-CTA repair took 16 rounds, 125 us; a
// batch of 1,000 undirected updates with it 310 us, now 205.)
// Lists longer than REP_LONG get the whole warp, one after the other.
constexpr uint32_t REP_GS = 8, REP_NG = 32 / REP_GS, REP_LONG = 64;

// Whether this group's vertex went to the heavy queue.
__device__ __forceinline__ bool queue_heavy_group(bool want, uint32_t *hv, unsigned long long *hv_n, uint64_t hv_cap,
                                                  uint32_t v) {
  bool in = false;
  if (want && lane_id() % REP_GS == 0) {
    const unsigned long long k = atomicAdd(hv_n, 1ull);
    in = k < hv_cap;
    if (in) hv[k] = v;
  }
  return __shfl_sync(FULL, in, lane_id() & ~(REP_GS - 1));
}

template <int A, bool W>
__device__ __forceinline__ void rescue_warps(const DevGraph &g, const uint32_t *fin, uint64_t n, uint64_t limit,
                                             uint64_t warp, uint64_t nwarps, const RepQueue &rq = RepQueue{}) {
  const uint32_t tag_inv = (uint32_t)g.ctl[C_INVTAG];
  using P = PoolT<W>;
  const typename P::E *pool = reinterpret_cast<const typename P::E *>(g.in.pool);
  const int lane = lane_id();
  uint32_t *const hv = rq.hv;
  unsigned long long *const hv_n = rq.n;
  const uint64_t hv_cap = rq.cap;
  auto one = [&](uint32_t d, uint64_t sd, uint32_t len, uint64_t off) {
    const bool cut = rq.task && len > TASK_DEG;
    const bool done = rescue_one<A, W>(g, d, sd, 0, cut ? TASK_SLOTS : len, off, tag_inv, limit);
    if (cut && !done) queue_tasks(rq, d, len, lane);
  };
  if (n <= nwarps) {
    for (uint64_t idx = warp; idx < n; idx += nwarps) {
      const uint32_t d = fin[idx];
      // (the vertex's words in one round trip)
      const uint32_t td = ld_u32(&g.inv[d]);
      const uint64_t sd = ld_v32(g.val32, d);
      const uint32_t len = seg_len(g.in, d);
      const uint64_t off = g.in.off[d];
      if (td != tag_inv) continue;
      if (hv && len > HEAVY_DEG && queue_heavy(hv, hv_n, hv_cap, d, lane)) continue;
      one(d, sd, len, off);
    }
    return;
  }
  const uint32_t sub = lane % REP_GS, gsh = lane & ~(REP_GS - 1);
  for (uint64_t base = warp * REP_NG; base < n; base += nwarps * REP_NG) {
    const uint64_t idx = base + lane / REP_GS;
    uint32_t d = 0, len = 0;
    uint64_t sd = 0, off = 0;
    bool act = false;
    if (idx < n) {
      d = fin[idx];
      const uint32_t td = ld_u32(&g.inv[d]);
      sd = ld_v32(g.val32, d);
      len = seg_len(g.in, d);
      off = g.in.off[d];
      act = td == tag_inv;
    }
    if (hv) {
      const bool queued = queue_heavy_group(act && len > HEAVY_DEG, hv, hv_n, hv_cap, d);
      act = act && !queued;
    }
    const unsigned lng = __ballot_sync(FULL, act && len > REP_LONG && sub == 0);
    bool open = act && len <= REP_LONG;
    for (uint32_t kb = 0; __any_sync(FULL, open && kb < len); kb += REP_GS) {
      const uint32_t k = kb + sub;
      bool ok = false;
      uint32_t src = 0, w = 0;
      if (open && k < len) {
        typename P::E e = pool[off + k];
        src = P::nbr(e);
        w = P::wt(e);
        if (!(src & DEAD) && Hook<A>::combine(ld_v32(g.val32, src), w) == sd)
          ok = !has_parents(g, src, tag_inv, limit);
      }
      const unsigned gb = (__ballot_sync(FULL, ok) >> gsh) & ((1u << REP_GS) - 1);
      if (gb) {  // the group's first candidate
        if (sub == (uint32_t)__ffs(gb) - 1 && atomicCAS(&g.inv[d], tag_inv, tag_inv + 1) == tag_inv)
          reinterpret_cast<unsigned long long *>(&g.lab[d])[1] = pack_parent(src, w);
        open = false;
      }
    }
    for (unsigned m = lng; m; m &= m - 1) {
      const int l = __ffs(m) - 1;
      const uint32_t d1 = __shfl_sync(FULL, d, l), len1 = __shfl_sync(FULL, len, l);
      const uint64_t sd1 = __shfl_sync(FULL, sd, l), off1 = __shfl_sync(FULL, off, l);
      one(d1, sd1, len1, off1);
    }
  }
}

template <int A, bool W>
__global__ void __launch_bounds__(TPB) k_rescue(DevGraph g, const uint32_t *fin, const unsigned long long *fin_n,
                                                uint64_t limit) {
  if (g.ctl[C_RECOMPUTE]) return;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  rescue_warps<A, W>(g, fin, *fin_n, limit, warp, nwarps, RepQueue{g.heavy, &g.ctl[C_HVR], g.heavy_cap});
}

// Rescue of the queued heavy vertices: for each in turn, every warp scans a
// 32-entry stride of its in-list; the first valid candidate wins the CAS.
template <int A, bool W>
__device__ __forceinline__ void rescue_heavy_warps(const DevGraph &g, uint64_t queued, uint64_t limit, uint64_t warp,
                                                   uint64_t nwarps) {
  const uint32_t tag_inv = (uint32_t)g.ctl[C_INVTAG];
  using P = PoolT<W>;
  const typename P::E *pool = reinterpret_cast<const typename P::E *>(g.in.pool);
  const int lane = lane_id();
  const uint64_t nh = min(queued, g.heavy_cap);
  for (uint64_t h = 0; h < nh; h++) {
    const uint32_t d = g.heavy[h];
    const uint64_t sd = ld_v32(g.val32, d);
    const uint32_t len = seg_len(g.in, d);
    const uint64_t off = g.in.off[d];
    for (uint64_t kb = warp * 32; kb < len; kb += nwarps * 32) {
      if (__shfl_sync(FULL, ld_u32(&g.inv[d]), 0) != tag_inv) break;  // rescued by another warp
      const uint64_t k = kb + lane;
      bool ok = false;
      uint32_t src = 0, w = 0;
      if (k < len) {
        typename P::E e = pool[off + k];
        src = P::nbr(e);
        w = P::wt(e);
        if (!(src & DEAD) && Hook<A>::combine(ld_v32(g.val32, src), w) == sd) ok = !has_parents(g, src, tag_inv, limit);
      }
      unsigned b = __ballot_sync(FULL, ok);
      if (b) {
        const int l = __ffs(b) - 1;
        if (lane == l && atomicCAS(&g.inv[d], tag_inv, tag_inv + 1) == tag_inv)
          reinterpret_cast<unsigned long long *>(&g.lab[d])[1] = pack_parent(src, w);
        break;
      }
    }
  }
}

template <int A, bool W>
__global__ void __launch_bounds__(TPB) k_rescue_heavy(DevGraph g, uint64_t limit) {
  if (g.ctl[C_RECOMPUTE]) return;
  rescue_heavy_warps<A, W>(g, g.ctl[C_HVR], limit, (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5,
                           ((uint64_t)gridDim.x * blockDim.x) >> 5);
}

// Collect and expand (core/graph.hpp:1363-1417): a still-invalid vertex joins
// the reset set; its tree children (parent == (u,w)) are invalidated next.
// The tree children of u among N slots a lane holds, invalidated and appended
// (all lanes of the warp).
template <bool W, int N>
__device__ __forceinline__ void expand_slots(const DevGraph &g, uint32_t u, uint64_t off, uint32_t k0, uint32_t step,
                                             uint32_t len, uint32_t tag_inv, uint32_t *fout,
                                             unsigned long long *fout_n) {
  using P = PoolT<W>;
  const typename P::E *pool = reinterpret_cast<const typename P::E *>(g.out.pool);
  typename P::E e[N];
  uint64_t meta[N];
  uint32_t t[N];
#pragma unroll
  for (int i = 0; i < N; i++)
    if (k0 + i * step < len) e[i] = pool[off + k0 + i * step];
#pragma unroll
  for (int i = 0; i < N; i++) {
    const bool on = k0 + i * step < len && !(P::nbr(e[i]) & DEAD);
    meta[i] = on ? ld_meta(&g.lab[P::nbr(e[i])]) : ~0ull;
    t[i] = on ? ld_u32(&g.inv[P::nbr(e[i])]) : tag_inv;
  }
#pragma unroll
  for (int i = 0; i < N; i++) {
    bool app = false;
    uint32_t v = 0;
    if (t[i] != tag_inv && t[i] != tag_inv + 1 && meta[i] == pack_parent(u, P::wt(e[i]))) {
      v = P::nbr(e[i]);
      app = atomicCAS(&g.inv[v], t[i], tag_inv) == t[i];
    }
    warp_append(app, v, fout, fout_n, FULL);
  }
}

template <int A, bool W>
__device__ __forceinline__ void expand_warps(const DevGraph &g, const uint32_t *fin, uint64_t n, uint32_t *tree,
                                             uint32_t *fout, unsigned long long *fout_n, uint64_t warp,
                                             uint64_t nwarps, const RepQueue &rq = RepQueue{}) {
  const uint32_t tag_inv = (uint32_t)g.ctl[C_INVTAG];
  const int lane = lane_id();
  uint32_t *const hv = rq.hv;
  unsigned long long *const hv_n = rq.n;
  const uint64_t hv_cap = rq.cap;
  auto one = [&](uint32_t u, uint32_t len, uint64_t off) {
    const bool cut = rq.task && len > TASK_DEG;
    if (cut) queue_tasks(rq, u, len, lane);
    const uint32_t end = cut ? TASK_SLOTS : len;
    uint32_t kb = 0;
    for (; kb + 32 < end; kb += 128) expand_slots<W, 4>(g, u, off, kb + lane, 32, end, tag_inv, fout, fout_n);
    if (kb < end) expand_slots<W, 1>(g, u, off, kb + lane, 32, end, tag_inv, fout, fout_n);
  };
  if (n <= nwarps) {
    for (uint64_t idx = warp; idx < n; idx += nwarps) {
      const uint32_t u = fin[idx];
      // (the vertex's words in one round trip; its slot in the reset set is
      // taken here and written after the scan, off the critical path)
      const uint32_t tu = ld_u32(&g.inv[u]);
      const uint32_t len = seg_len(g.out, u);
      const uint64_t off = g.out.off[u];
      if (tu != tag_inv) continue;
      unsigned long long slot = 0;
      if (lane == 0) slot = atomicAdd(&g.ctl[C_TREEN], 1ull);
      if (!(hv && len > HEAVY_DEG && queue_heavy(hv, hv_n, hv_cap, u, lane))) one(u, len, off);
      if (lane == 0) tree[slot] = u;
    }
    return;
  }
  const uint32_t sub = lane % REP_GS;
  for (uint64_t base = warp * REP_NG; base < n; base += nwarps * REP_NG) {
    const uint64_t idx = base + lane / REP_GS;
    uint32_t u = 0, len = 0;
    uint64_t off = 0;
    bool act = false;
    if (idx < n) {
      u = fin[idx];
      const uint32_t tu = ld_u32(&g.inv[u]);
      len = seg_len(g.out, u);
      off = g.out.off[u];
      act = tu == tag_inv;
    }
    if (!__any_sync(FULL, act)) continue;
    warp_append(act && sub == 0, u, tree, &g.ctl[C_TREEN], FULL);
    if (hv) {
      const bool queued = queue_heavy_group(act && len > HEAVY_DEG, hv, hv_n, hv_cap, u);
      act = act && !queued;
    }
    const unsigned lng = __ballot_sync(FULL, act && len > REP_LONG && sub == 0);
    const uint32_t end = act && len <= REP_LONG ? len : 0u;
    for (uint32_t kb = 0; __any_sync(FULL, kb < end); kb += 2 * REP_GS)
      expand_slots<W, 2>(g, u, off, kb + sub, REP_GS, end, tag_inv, fout, fout_n);
    for (unsigned m = lng; m; m &= m - 1) {
      const int l = __ffs(m) - 1;
      const uint32_t u1 = __shfl_sync(FULL, u, l), len1 = __shfl_sync(FULL, len, l);
      const uint64_t off1 = __shfl_sync(FULL, off, l);
      one(u1, len1, off1);
    }
  }
}

// Expansion of the queued heavy vertices: their tree children, found by every
// warp over a stride of the out-list.
template <int A, bool W>
__device__ __forceinline__ void expand_heavy_warps(const DevGraph &g, uint64_t queued, uint32_t *fout,
                                                   unsigned long long *fout_n, uint64_t warp, uint64_t nwarps) {
  const uint32_t tag_inv = (uint32_t)g.ctl[C_INVTAG];
  using P = PoolT<W>;
  const typename P::E *pool = reinterpret_cast<const typename P::E *>(g.out.pool);
  const int lane = lane_id();
  const uint32_t *hv = g.heavy + g.heavy_cap;
  const uint64_t nh = min(queued, g.heavy_cap);
  for (uint64_t h = 0; h < nh; h++) {
    const uint32_t u = hv[h];
    const uint32_t len = seg_len(g.out, u);
    const uint64_t off = g.out.off[u];
    for (uint64_t kb = warp * 32; kb < len; kb += nwarps * 32) {
      const uint64_t k = kb + lane;
      bool app = false;
      uint32_t v = 0;
      if (k < len) {
        typename P::E e = pool[off + k];
        v = P::nbr(e);
        if (!(v & DEAD) && ld_meta(&g.lab[v]) == pack_parent(u, P::wt(e))) {
          uint32_t t = ld_u32(&g.inv[v]);
          if (t != tag_inv && t != tag_inv + 1) app = atomicCAS(&g.inv[v], t, tag_inv) == t;
        }
      }
      warp_append(app, v, fout, fout_n, FULL);
    }
  }
}

template <int A, bool W>
__global__ void __launch_bounds__(TPB) k_expand_heavy(DevGraph g, uint32_t *fout, unsigned long long *fout_n) {
  if (g.ctl[C_RECOMPUTE]) return;
  expand_heavy_warps<A, W>(g, g.ctl[C_HVE], fout, fout_n, (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5,
                           ((uint64_t)gridDim.x * blockDim.x) >> 5);
}

template <int A, bool W>
__global__ void __launch_bounds__(TPB) k_expand(DevGraph g, const uint32_t *fin, const unsigned long long *fin_n,
                                                uint32_t *tree, uint32_t *fout, unsigned long long *fout_n) {
  if (g.ctl[C_RECOMPUTE]) return;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  expand_warps<A, W>(g, fin, *fin_n, tree, fout, fout_n, warp, nwarps,
                     RepQueue{g.heavy + g.heavy_cap, &g.ctl[C_HVE], g.heavy_cap});
}

// Reset the invalid set to init (core/graph.hpp:1420-1430).
template <int A>
__device__ __forceinline__ void reset_warps(const DevGraph &g, const uint32_t *tree, uint64_t n, uint32_t mst,
                                            uint64_t warp, uint64_t nwarps) {
  const uint64_t root = g.ctl[C_ROOT];
  for (uint64_t base = warp * 32; base < n; base += nwarps * 32) {
    uint64_t i = base + lane_id();
    uint32_t u = 0;
    if (i < n) {
      u = tree[i];
      g.lab[u] = make_ulonglong2(Hook<A>::init(u, root), pack_parent(NONE, 0));
      g.val32[u] = (uint32_t)Hook<A>::init(u, root);
    }
    if (mst) mark_modified(g, i < n, u, mst);
  }
}

template <int A>
__global__ void k_reset(DevGraph g, const uint32_t *tree, const unsigned long long *tree_n, uint32_t mst) {
  if (g.ctl[C_RECOMPUTE]) return;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  reset_warps<A>(g, tree, *tree_n, mst, warp, nwarps);
}

// One transposed pull over the reset set (core/graph.hpp:1433-1511): each
// vertex takes its best in-neighbour by update_func.
struct PullBest {
  uint64_t best, su;
  uint32_t src, w;
};

// The best of the N slots a lane holds and of p.
template <int A, bool W, int N>
__device__ __forceinline__ void pull_slots(const DevGraph &g, uint64_t off, uint32_t k0, uint32_t step, uint32_t len,
                                           PullBest &p) {
  using P = PoolT<W>;
  const typename P::E *pool = reinterpret_cast<const typename P::E *>(g.in.pool);
  typename P::E e[N];
  uint64_t su[N];
#pragma unroll
  for (int i = 0; i < N; i++)
    if (k0 + i * step < len) e[i] = pool[off + k0 + i * step];
#pragma unroll
  for (int i = 0; i < N; i++) {
    const bool on = k0 + i * step < len && !(P::nbr(e[i]) & DEAD);
    su[i] = on ? ld_v32(g.val32, P::nbr(e[i])) : ~0ull;
  }
#pragma unroll
  for (int i = 0; i < N; i++) {
    if (su[i] == ~0ull) continue;
    const uint64_t nv = Hook<A>::combine(su[i], P::wt(e[i]));
    if (Hook<A>::better(nv, p.best)) p = PullBest{nv, su[i], P::nbr(e[i]), P::wt(e[i])};
  }
}

// The best over the `width` lanes of each group, in its first lane; relaxes the
// vertex with it there (all lanes of the warp).
template <int A>
__device__ __forceinline__ bool pull_reduce(const DevGraph &g, PullBest p, uint32_t d, bool act, int width,
                                            uint32_t mst) {
  for (int o = width / 2; o; o >>= 1) {
    const uint64_t ob = __shfl_down_sync(FULL, p.best, o), osu = __shfl_down_sync(FULL, p.su, o);
    const uint32_t os = __shfl_down_sync(FULL, p.src, o), ow = __shfl_down_sync(FULL, p.w, o);
    if (os != NONE && (p.src == NONE || Hook<A>::better(ob, p.best))) p = PullBest{ob, osu, os, ow};
  }
  const bool upd = act && lane_id() % width == 0 && p.src != NONE && relax<A>(g, p.src, p.su, d, p.w);
  __syncwarp();
  if (mst) mark_modified(g, upd, d, mst);
  return upd;
}

template <int A, bool W>
__device__ __forceinline__ unsigned long long pull_warps(const DevGraph &g, const uint32_t *fin, uint64_t n,
                                                         uint32_t mst, uint64_t warp, uint64_t nwarps,
                                                         const RepQueue &rq = RepQueue{}) {
  const int lane = lane_id();
  unsigned long long local = 0;
  uint32_t *const hv = rq.hv;
  unsigned long long *const hv_n = rq.n;
  const uint64_t hv_cap = rq.cap;
  auto one = [&](uint32_t d, uint32_t len, uint64_t off) {
    const bool cut = rq.task && len > TASK_DEG;
    if (cut) queue_tasks(rq, d, len, lane);
    const uint32_t end = cut ? TASK_SLOTS : len;
    PullBest p = {ld_v32(g.val32, d), 0, NONE, 0};
    uint32_t kb = 0;
    for (; kb + 32 < end; kb += 128) pull_slots<A, W, 4>(g, off, kb + lane, 32, end, p);
    if (kb < end) pull_slots<A, W, 1>(g, off, kb + lane, 32, end, p);
    local += pull_reduce<A>(g, p, d, true, 32, mst);
  };
  if (n <= nwarps) {
    for (uint64_t idx = warp; idx < n; idx += nwarps) {
      const uint32_t d = fin[idx];
      const uint32_t len = seg_len(g.in, d);
      const uint64_t off = g.in.off[d];
      if (hv && len > HEAVY_DEG && queue_heavy(hv, hv_n, hv_cap, d, lane)) continue;
      one(d, len, off);
    }
    return local;
  }
  const uint32_t sub = lane % REP_GS;
  for (uint64_t base = warp * REP_NG; base < n; base += nwarps * REP_NG) {
    const uint64_t idx = base + lane / REP_GS;
    uint32_t d = 0, len = 0;
    uint64_t off = 0;
    bool act = idx < n;
    PullBest p = {0, 0, NONE, 0};
    if (act) {
      d = fin[idx];
      len = seg_len(g.in, d);
      off = g.in.off[d];
      p.best = ld_v32(g.val32, d);
    }
    if (hv) {
      const bool queued = queue_heavy_group(act && len > HEAVY_DEG, hv, hv_n, hv_cap, d);
      act = act && !queued;
    }
    const unsigned lng = __ballot_sync(FULL, act && len > REP_LONG && sub == 0);
    const uint32_t end = act && len <= REP_LONG ? len : 0u;
    for (uint32_t kb = 0; __any_sync(FULL, kb < end); kb += 2 * REP_GS)
      pull_slots<A, W, 2>(g, off, kb + sub, REP_GS, end, p);
    local += pull_reduce<A>(g, p, d, act && end, REP_GS, mst);
    for (unsigned m = lng; m; m &= m - 1) {
      const int l = __ffs(m) - 1;
      const uint32_t d1 = __shfl_sync(FULL, d, l), len1 = __shfl_sync(FULL, len, l);
      const uint64_t off1 = __shfl_sync(FULL, off, l);
      one(d1, len1, off1);
    }
  }
  return local;
}

template <int A, bool W>
__global__ void __launch_bounds__(TPB) k_pull(DevGraph g, const uint32_t *fin, const unsigned long long *fin_n,
                                              uint32_t mst) {
  if (g.ctl[C_RECOMPUTE]) return;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long local =
      pull_warps<A, W>(g, fin, *fin_n, mst, warp, nwarps,
                       RepQueue{g.heavy + 2 * g.heavy_cap, &g.ctl[C_HVP], g.heavy_cap});
  warp_add_result(local, &g.ctl[C_RESULT]);
}

// The pull of the queued heavy reset vertices: every warp takes the best of a
// stride of the in-list and relaxes the vertex with it (the CAS keeps the best).
template <int A, bool W>
__device__ __forceinline__ unsigned long long pull_heavy_warps(const DevGraph &g, uint32_t mst, uint64_t warp,
                                                               uint64_t nwarps) {
  using P = PoolT<W>;
  const typename P::E *pool = reinterpret_cast<const typename P::E *>(g.in.pool);
  const int lane = lane_id();
  const uint32_t *hv = g.heavy + 2 * g.heavy_cap;
  const uint64_t nh = min(__ldcg(&g.ctl[C_HVP]), (unsigned long long)g.heavy_cap);
  unsigned long long local = 0;
  for (uint64_t h = 0; h < nh; h++) {
    const uint32_t d = hv[h];
    const uint32_t len = seg_len(g.in, d);
    const uint64_t off = g.in.off[d];
    if (warp * 32 >= len) continue;
    uint64_t best = ld_v32(g.val32, d), bsu = 0;
    uint32_t bsrc = NONE, bw = 0;
    for (uint64_t k = warp * 32 + lane; k < len; k += nwarps * 32) {
      typename P::E e = pool[off + k];
      uint32_t s = P::nbr(e);
      if (s & DEAD) continue;
      uint64_t su = ld_v32(g.val32, s);
      uint64_t nv = Hook<A>::combine(su, P::wt(e));
      if (Hook<A>::better(nv, best)) { best = nv; bsrc = s; bw = P::wt(e); bsu = su; }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      uint64_t ob = __shfl_down_sync(FULL, best, o);
      uint64_t osu = __shfl_down_sync(FULL, bsu, o);
      uint32_t os = __shfl_down_sync(FULL, bsrc, o);
      uint32_t ow = __shfl_down_sync(FULL, bw, o);
      if (os != NONE && (bsrc == NONE || Hook<A>::better(ob, best))) { best = ob; bsu = osu; bsrc = os; bw = ow; }
    }
    bool upd = false;
    if (lane == 0 && bsrc != NONE) upd = relax<A>(g, bsrc, bsu, d, bw);
    local += upd;
    if (mst) mark_modified(g, __shfl_sync(FULL, upd, 0) && lane == 0, d, mst);
  }
  return local;
}

template <int A, bool W>
__global__ void __launch_bounds__(TPB) k_pull_heavy(DevGraph g, uint32_t mst) {
  if (g.ctl[C_RECOMPUTE]) return;
  const unsigned long long local =
      pull_heavy_warps<A, W>(g, mst, (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5,
                             ((uint64_t)gridDim.x * blockDim.x) >> 5);
  warp_add_result(local, &g.ctl[C_RESULT]);
}

// Small deletion repairs in one CTA: the invalidation levels (rescue, expand),
// the reset and the pull with CTA barriers in place of launches, then the
// reset set copied to queue 0 for the push loop.  When a level's frontier or
// the reset set outgrows one CTA it hands over to the multi-CTA repair (the
// IF node it opens), with the frontier left in queue 0 where that repair
// starts.
constexpr int DT_TPB = 1024;
constexpr uint64_t DEL_TINY_N = 1024, DEL_TINY_TREE = 8192;

// del_tiny_levels is that repair as a device function for a CTA of DT_TPB
// threads; it returns true when it hands over.
template <int A, bool W>
__device__ __forceinline__ bool del_tiny_levels(const DevGraph &g, uint32_t *q0, uint32_t *q1, uint32_t *tree,
                                                uint64_t limit, uint64_t big, uint64_t max_iter, uint32_t mst) {
  __shared__ int s_go, s_rec;  // decisions by thread 0: every thread takes the same branch
  unsigned long long *c = g.ctl;
  const unsigned tid = threadIdx.x;
  const uint64_t warp = tid >> 5, nwarps = DT_TPB / 32;
  uint32_t *cur = q0, *nxt = q1;
  unsigned long long *cur_n = &c[C_QN0], *nxt_n = &c[C_QN1];
  for (;;) {
    // a heavy vertex (a list longer than HEAVY_DEG) in this level's frontier,
    // or in the reset set once the levels are done, goes to the grid-wide repair
    int heavy = 0;
    {
      const uint64_t n0 = *cur_n;
      if (n0 && n0 <= DEL_TINY_N) {
        for (uint64_t i = tid; i < n0; i += DT_TPB)
          heavy |= seg_len(g.in, cur[i]) > HEAVY_DEG || seg_len(g.out, cur[i]) > HEAVY_DEG;
      } else if (n0 == 0) {
        const uint64_t tn = c[C_TREEN];
        if (tn <= DEL_TINY_TREE)
          for (uint64_t i = tid; i < tn; i += DT_TPB) heavy |= seg_len(g.in, tree[i]) > HEAVY_DEG;
      }
    }
    heavy = __syncthreads_or(heavy);
    if (tid == 0) {
      const uint64_t n = *cur_n, tree_n = c[C_TREEN];
      bool rec = c[C_RECOMPUTE] != 0;
      int go = 1;  // 1: run this level; 0: invalidation done; 2: hand over
      if (n == 0 || rec) {
        go = 0;
      } else if (n > DEL_TINY_N || heavy) {
        go = 2;
      } else {
        const uint64_t it = c[C_INVITER];
        if (it >= max_iter) {
          go = 0;
        } else if (it <= 10 && tree_n + n > big) {  // core/graph.hpp:1252
          c[C_RECOMPUTE] = 1;
          rec = true;
          go = 0;
        } else {
          c[C_INVITER] = it + 1;
          *nxt_n = 0;
        }
      }
      if (go == 0 && (tree_n > DEL_TINY_TREE || heavy) && !rec) go = 2;
      s_go = go;
      s_rec = rec;
    }
    __syncthreads();
    if (s_go != 1) break;
    const uint64_t n = *cur_n;
    rescue_warps<A, W>(g, cur, n, limit, warp, nwarps);
    __syncthreads();
    expand_warps<A, W>(g, cur, n, tree, nxt, nxt_n, warp, nwarps);
    __syncthreads();
    uint32_t *t = cur;
    cur = nxt;
    nxt = t;
    unsigned long long *tn = cur_n;
    cur_n = nxt_n;
    nxt_n = tn;
  }
  if (s_go == 2) {
    // the multi-CTA repair continues from queue 0
    if (cur != q0) {
      const uint64_t n = *cur_n;
      for (uint64_t i = tid; i < n; i += DT_TPB) q0[i] = cur[i];
      __syncthreads();
      if (tid == 0) c[C_QN0] = n;
    }
    __syncthreads();
    return true;
  }
  unsigned long long local = 0;
  const bool recompute = s_rec != 0;
  if (!recompute) {
    const uint64_t tn = c[C_TREEN];
    reset_warps<A>(g, tree, tn, mst, warp, nwarps);
    __syncthreads();
    local = pull_warps<A, W>(g, tree, tn, mst, warp, nwarps);
    __syncthreads();
    for (uint64_t i = tid; i < tn; i += DT_TPB) q0[i] = tree[i];
    __syncthreads();
    if (tid == 0) c[C_QN0] = tn;
  } else if (tid == 0) {
    c[C_QN0] = 0;
  }
  warp_add_result(local, &c[C_RESULT]);
  __syncthreads();
  return false;
}

// in_graph = 0: launched by the host (profile mode); the hand-over decision
// goes to C_HOSTCOND instead of the IF node's handle.
template <int A, bool W>
__global__ void __launch_bounds__(DT_TPB) k_del_tiny(DevGraph g, uint32_t *q0, uint32_t *q1, uint32_t *tree,
                                                     uint64_t limit, uint64_t big, uint64_t max_iter, uint32_t mst,
                                                     cudaGraphConditionalHandle standard, int in_graph) {
  const bool over = del_tiny_levels<A, W>(g, q0, q1, tree, limit, big, max_iter, mst);
  if (threadIdx.x == 0) {
    g.ctl[C_KLAUNCH] += 1;
    if (in_graph) cudaGraphSetConditional(standard, over ? 1u : 0u);
    else g.ctl[C_HOSTCOND] = over ? 1 : 0;
  }
}

// The hand-over decision of the fused apply kernel's deletion repair, for the
// IF node of the grid-wide repair (a kernel sets the handle of a conditional
// node in its own graph).
__global__ void k_handover(DevGraph g, cudaGraphConditionalHandle standard) {
  g.ctl[C_KLAUNCH] += 1;
  cudaGraphSetConditional(standard, g.ctl[C_OVER] ? 1u : 0u);
}

// Fused small-batch apply: one CTA runs the storage steps of a batch of at
// most SMALL_EDGES edges (unpack from the mapped staging buffer, lookup/create,
// growth, new-slot write, multiplicity count, candidates) and the seeding of
// the tree repair, with CTA barriers where the multi-kernel path has kernel
// boundaries.  A small repair then runs in the same CTA: the one-CTA deletion
// repair (del_tiny_levels) for a delete batch, and push levels while the
// frontier stays small (tiny_levels).  The kernel ends by writing the control
// block to the host's mapped copy; C_LEFT there tells the host what is left
// for the graphs it launches next (the level loop; the grid-wide deletion
// repair when the one-CTA repair handed over, C_OVER).  A safe update (the
// common case, need_update_tree_* false) and most unsafe single updates cost
// this one kernel and no conditional node: a conditional node costs about
// 10 us even when its condition is false.  A storage error (edge
// index or pool full) stops before the count step, leaving the op arrays for
// the host's compaction and replay, exactly like the multi-kernel path.
constexpr int FS_TPB = 1024;
static_assert(FS_TPB == TINY_TPB && FS_TPB == DT_TPB, "the fused kernel runs the one-CTA repairs");

// What the fused kernel's in-place repair needs besides queue 0.
struct FusedRepair {
  uint32_t *q1, *tree;
  uint64_t limit;       // has_parents chain guard
  uint64_t big;         // invalidated-set size that asks for a full recompute
  uint64_t max_iter;    // invalidation levels
  uint64_t max_levels;  // level bound of the push loop
  uint64_t tiny_edges;  // out-slot limit of an in-place push level (0: none in place)
};

// The control block to the host's mapped copy, by the whole CTA after its
// last update (the host reads it once the stream has synchronised, and the
// kernel's end makes its writes visible).  One warp and 256 bytes: two words more
// cost 0.7 us of a 20 us call.
__device__ __forceinline__ void ctl_to_host(const DevGraph &g, unsigned long long *ctl_host) {
  __syncthreads();
  if (threadIdx.x < C_HOST) ctl_host[threadIdx.x] = g.ctl[threadIdx.x];
}

// A batch's header as the fused kernels read it.
struct StagedBatch {
  uint64_t n, pairs, want, inv_tag;
  unsigned long long stamp;  // C_STAMP at the kernel's start (used by its first batch)
};

// A batch of at most INLINE_EDGES edges travels inside the kernel's parameters
// (the launch carries it to the SM), so the kernel reads no staging buffer
// across the bus: single updates and the served path's small epochs skip the
// one PCIe round trip (about 6 us) that staging from mapped memory costs.
// words[] holds the batch as the caller gave it: rg_edge records (3 words per
// edge) or (src, dst) pairs (2 words).
constexpr unsigned INLINE_EDGES = INLINE_MAX_EDGES;
struct InlineBatch {
  uint64_t n, pairs, want, inv_tag;
  uint64_t words[3 * INLINE_EDGES];
};

// The batch crosses the bus in 16-byte loads into device scratch: the first
// APPLY_SPEC chunks in the same round trip as the header (thread hdr_t reads
// the header, threads chunk_t .. chunk_t + APPLY_SPEC - 1 the chunks), the
// rest in apply_batch once the header gives the size.  The host wrote both
// before the launch; they are read past any cache.
constexpr unsigned APPLY_SPEC = 256;

__device__ __forceinline__ void stage_batch(const DevGraph &g, const ApplyHdr *hdr, const char *data, uint4 *scratch,
                                            StagedBatch &sb, unsigned hdr_t, unsigned chunk_t) {
  const unsigned tid = threadIdx.x;
  const uint4 *raw = reinterpret_cast<const uint4 *>(data);
  if (tid >= chunk_t && tid < chunk_t + APPLY_SPEC) scratch[tid - chunk_t] = __ldcv(&raw[tid - chunk_t]);
  if (tid == hdr_t) {
    sb.stamp = g.ctl[C_STAMP];
    sb.n = __ldcv(&hdr->n);
    sb.pairs = __ldcv(&hdr->pairs);
    sb.want = __ldcv(&hdr->want_old);
    sb.inv_tag = __ldcv(&hdr->inv_tag);
  }
}

// The in-place repair of a batch whose seeds are in queue 0, by all threads of
// the CTA after a barrier: returns 1 when work is left for the launches after
// the kernel (C_OVER set when the deletion repair handed over), else 0.
template <int A, bool W>
__device__ __forceinline__ int batch_repair(const DevGraph &g, const FusedRepair &fr, int add, uint32_t *q0,
                                            uint32_t mst, unsigned long long *tr) {
  unsigned long long *c = g.ctl;
  bool over = false;
  if (c[C_QN0] && !c[C_ERR]) {
    if (!add) over = del_tiny_levels<A, W>(g, q0, fr.q1, fr.tree, fr.limit, fr.big, fr.max_iter, mst);
    if (tr && threadIdx.x == 0) tr[RG_PH_DELREPAIR] = global_ns();
    if (!over && fr.tiny_edges && c[C_QN0])
      tiny_levels<A, W>(g, q0, &c[C_QN0], fr.q1, &c[C_QN1], q0, &c[C_QN0], fr.max_levels, fr.tiny_edges, mst, false);
  }
  const bool left = over || (c[C_QN0] && !c[C_ERR]);
  __syncthreads();  // every thread has read the counts before the next batch resets them
  if (threadIdx.x == 0) {
    c[C_OVER] = over ? 1 : 0;
    c[C_QN1] = 0;  // (the engine's first output count)
  }
  return left ? 1 : 0;
}

// One staged batch through the storage steps, the seeding and the in-place
// repair, by all threads of the CTA after a barrier.  Returns 0 when nothing
// is left, 1 when the repair left work for the graph nodes after the kernel
// (C_OVER set when the deletion repair handed over), 2 after a storage error
// or when it skipped the batch.  inl: the batch's words in the kernel's
// parameters (an inline batch), or null when they were staged into scratch.
template <int A, bool W>
__device__ __forceinline__ int apply_batch(const DevGraph &g, const sdev::OpView &ops, const StagedBatch &sb,
                                           const char *data, uint64_t *old_host, uint32_t *cand, int add, int directed,
                                           uint32_t *q0, uint32_t mst, int second, const FusedRepair &fr,
                                           uint4 *scratch, const uint64_t *inl = nullptr) {
  __shared__ int s_skip;
  __shared__ unsigned long long s_rec_top;  // (no other CTA creates records meanwhile)
  unsigned long long *c = g.ctl;
  const unsigned tid = threadIdx.x;
  // phase trace (RG_OPT_PHASE_TRACE): thread 0 stamps the device clock
  unsigned long long *tr = g.ptrace ? g.ptrace + 16 * second : nullptr;
  auto stamp = [&](int k) {
    if (tr && tid == 0) tr[k] = global_ns();
  };
  if (tid == 0) {
    // the second batch of a submission does nothing after an error in the first,
    // or before the levels that the engine left of the first one's repair
    s_skip = second && (c[C_ERR] != 0 || c[C_ELEFT] != 0);
    if (!s_skip) {
      s_rec_top = *g.rec_top;
      const unsigned long long kl = c[C_KLAUNCH];
      prologue_ctl(c, sb.inv_tag, second ? nullptr : &sb.stamp);
      if (second) c[C_KLAUNCH] = kl;  // the count covers the whole submission
      c[C_CANDN] = 0;
      c[C_GROWN_OUT] = 0;
      c[C_GROWN_IN] = 0;
    }
  }
  __syncthreads();
  if (s_skip) return 2;
  if (tr && tid == 0) tr[15] = 1;
  stamp(RG_PH_BEGIN);
  const uint64_t n = sb.n < SMALL_EDGES ? sb.n : SMALL_EDGES;
  const uint64_t nops = directed ? n : 2 * n;
  const int weighted = W ? 1 : 0;
  const uint64_t chunks = (n * (sb.pairs ? 16 : sizeof(rg_edge)) + 15) / 16;
  if (!inl && chunks > APPLY_SPEC) {
    const uint4 *raw = reinterpret_cast<const uint4 *>(data);
    for (uint64_t k = APPLY_SPEC + tid; k < chunks; k += FS_TPB) scratch[k] = __ldcv(&raw[k]);
    __syncthreads();
  }
  // staged words are read past L1 (this CTA wrote them); inline ones are parameters
  const uint64_t *words = inl ? inl : reinterpret_cast<const uint64_t *>(scratch);
  auto word = [&](uint64_t k) -> uint64_t { return inl ? inl[k] : __ldcg(&words[k]); };
  if (sb.pairs) {
    for (uint64_t i = tid; i < n; i += FS_TPB) {
      uint64_t s64 = word(2 * i), d64 = word(2 * i + 1);
      uint32_t w = weighted ? (uint32_t)(splitmix64((s64 << 32) | d64) % 255 + 1) : 0u;
      sdev::put_ops(ops, i, (uint32_t)s64, (uint32_t)d64, w, directed);
    }
  } else {
    for (uint64_t i = tid; i < n; i += FS_TPB) {
      uint64_t s64 = word(3 * i), d64 = word(3 * i + 1), w64 = word(3 * i + 2);
      sdev::put_ops(ops, i, (uint32_t)s64, (uint32_t)d64, weighted ? (uint32_t)w64 : 0u, directed);
    }
  }
  __syncthreads();
  stamp(RG_PH_UNPACK);
  if (add) {
    for (uint64_t j = tid; j < nops; j += FS_TPB) sdev::lookup_op<4>(g, ops, j, 1, &s_rec_top);
  } else {
    for (uint64_t j = tid; j < nops; j += FS_TPB) sdev::lookup_op<1>(g, ops, j, 0, &s_rec_top);
  }
  __syncthreads();
  if (add && tid == 0) *g.rec_top = s_rec_top;
  stamp(RG_PH_LOOKUP);
  if (add) {
    // each warp grows its own vertices (a vertex is in a grow list once); the
    // copies of long lists (a hub's) are left to the whole CTA below
    constexpr unsigned BIG = 16;
    __shared__ sdev::GrowClaim s_big[BIG];
    __shared__ int s_big_in[BIG];
    __shared__ unsigned s_nbig;
    if (tid == 0) s_nbig = 0;
    __syncthreads();
    const unsigned gw = tid >> 5, gl = tid & 31;
    for (int in = 0; in < (g.symmetric ? 1 : 2); in++) {
      const DevDir &dir = in ? g.in : g.out;
      const unsigned long long nv = c[in ? C_GROWN_IN : C_GROWN_OUT];
      for (unsigned long long k = gw; k < nv; k += FS_TPB / 32) {
        const uint32_t v = dir.grow[k];
        // a slot may be free (taken below, or the warp copies after all);
        // lane 0's view keeps the choice uniform across the warp
        const bool more = __shfl_sync(FULL, s_nbig < BIG ? 1 : 0, 0) != 0;
        sdev::GrowClaim cl;
        if (sdev::grow_vertex_warp<W>(dir, c, v, gl, more, &cl)) {
          unsigned slot = 0;
          if (gl == 0) slot = atomicAdd(&s_nbig, 1u);
          slot = __shfl_sync(FULL, slot, 0);
          if (slot < BIG) {
            if (gl == 0) {
              s_big[slot] = cl;
              s_big_in[slot] = in;
            }
          } else {
            sdev::grow_copy<W>(dir, cl, gl, 32);
            __syncwarp();
            if (gl == 0) sdev::grow_publish(dir, cl);
          }
        }
      }
    }
    __syncthreads();
    const unsigned nbig = s_nbig < BIG ? s_nbig : BIG;
    for (unsigned b = 0; b < nbig; b++) sdev::grow_copy<W>(s_big_in[b] ? g.in : g.out, s_big[b], tid, FS_TPB);
    __syncthreads();
    if (tid < nbig) sdev::grow_publish(s_big_in[tid] ? g.in : g.out, s_big[tid]);
  }
  __syncthreads();
  stamp(RG_PH_GROW);
  if (c[C_ERR]) return 2;
  if (add) {
    for (uint64_t j = tid; j < nops; j += FS_TPB) sdev::write_new_op<W>(g, ops, j);
    __syncthreads();
    stamp(RG_PH_WRITE);
  }
  for (uint64_t j = tid; j < nops; j += FS_TPB) sdev::count_op<W>(g, ops, j, add);
  __syncthreads();
  stamp(RG_PH_COUNT);
  for (uint64_t i = tid; i < n; i += FS_TPB) sdev::edge_old(ops, i, directed, add, 1, sb.want ? old_host : nullptr, cand, c);
  __syncthreads();
  stamp(RG_PH_OLD);
  const uint64_t ncand = c[C_CANDN];
  const uint64_t warp = tid >> 5, nwarps = FS_TPB / 32;
  if (add) {
    unsigned long long local = seed_add<A>(g, ops.src, ops.dst, ops.w, cand, ncand, directed, q0, &c[C_QN0], mst, warp, nwarps);
    warp_add_result(local, &c[C_RESULT]);
  } else {
    seed_del(g, ops.src, ops.dst, ops.w, cand, ncand, directed, q0, &c[C_QN0], warp, nwarps);
  }
  __syncthreads();
  stamp(RG_PH_SEED);
  const int left = batch_repair<A, W>(g, fr, add, q0, mst, tr);
  stamp(RG_PH_END);
  return left;
}

// ---- inline batches without a complication -----------------------------------
// An inline batch (at most INLINE_EDGES edges) usually meets none of the cases
// that the phases of apply_batch exist for: no list has to grow, no two edges of
// the submission are the same, each key is found or its slot is free within the
// first FAST_PROBES index slots (at the index's usual load of 0.45 two leave a
// quarter of the keys open, six 2 in a hundred).  fast_inline then has one lane per directed op (warp 0
// the inserts, warp 1 the deletes) load everything the op can need in one round
// trip: the index slots, the ends and offsets of both lists, the value of the
// source and the label of the destination; a second trip loads the records of
// edges that exist.  The rest is stores and atomics that nothing waits for.
// apply_batch takes the same update through eight phases with barriers and one
// or two dependent trips each, 5 to 8 us a batch (RMAT-20 SSSP, an insert and a
// delete per call: 33 us a call through the phases, 22 with this).  Anything
// else is decided before the first store, and the submission goes to apply_batch
// untouched.
constexpr int FAST_PROBES = 6;
struct FastShared {
  uint32_t s[32], d[32], w[32];  // the inserts' ops
  uint32_t n_ins;
  unsigned fall[2], improve, seeds;
};
enum FastResult : int { FAST_NO = -1, FAST_INS_SEEDS = 1, FAST_DEL_DONE = 2, FAST_DEL_SEEDS = 4 };

// old_host: where the per-edge old counts of a single batch go, or null.
// Returns FAST_NO (nothing done), or what was done: the insert batch's storage
// and seeds (FAST_INS_SEEDS when queue 0 holds some; the delete batch is then
// still to do), the delete batch's (FAST_DEL_DONE, FAST_DEL_SEEDS).
template <int A, bool W>
__device__ __forceinline__ int fast_inline(const DevGraph &g, const InlineBatch *ins, const InlineBatch *del,
                                           int directed, uint64_t *old_host, uint32_t *q0, uint32_t mst) {
  using E = typename std::conditional<W, uint2, uint32_t>::type;
  __shared__ FastShared fs;
  unsigned long long *c = g.ctl;
  const unsigned tid = threadIdx.x, lane = tid & 31, lt = (1u << lane) - 1;
  const bool is_ins = tid < 32 && ins, is_del = tid >= 32 && tid < 64 && del;
  const InlineBatch *ib = is_ins ? ins : del;
  bool on = false, fall = false, better_now = false;
  uint32_t s = 0, d = 0, w = 0;
  uint64_t n = 0;
  if (is_ins || is_del) {
    n = ib->n < INLINE_EDGES ? ib->n : INLINE_EDGES;
    const uint64_t nops = directed ? n : 2 * n;
    on = lane < nops;
    if (is_ins && lane == 0) fs.n_ins = (uint32_t)nops;
    if (on) {
      const uint64_t i = directed ? lane : lane >> 1;
      const uint64_t a = ib->words[(ib->pairs ? 2 : 3) * i], b = ib->words[(ib->pairs ? 2 : 3) * i + 1];
      if (W) w = ib->pairs ? (uint32_t)(splitmix64((a << 32) | b) % 255 + 1) : (uint32_t)ib->words[3 * i + 2];
      const bool flip = !directed && (lane & 1);
      s = (uint32_t)(flip ? b : a);
      d = (uint32_t)(flip ? a : b);
      fall = !directed && s == d;  // (a self-loop is one op of multiplicity 2)
    }
    if (is_ins) {
      fs.s[lane] = s;
      fs.d[lane] = d;
      fs.w[lane] = w;
    }
  }
  // 1. everything the ops can need, in one round trip
  const ulonglong2 none = make_ulonglong2(~0ull, ~0ull);
  const ulonglong2 key = make_ulonglong2((uint64_t)s | ((uint64_t)d << 32), (uint64_t)w);
  const uint64_t h0 = on ? sdev::ht_hash(s, d, w) & g.ht_mask : 0;
  ulonglong2 e[FAST_PROBES], lab = none;
  uint32_t len_o = 0, cap_o = 0, len_i = 0, cap_i = 0, val = 0;
  uint64_t off_o = 0, off_i = 0;
  unsigned long long top = 0;
  if (on) {
#pragma unroll
    for (int k = 0; k < FAST_PROBES; k++) e[k] = __ldcg(&g.ht[(h0 + k) & g.ht_mask]);
    off_o = g.out.off[s];
    cap_o = g.out.cap[s];
    if (!g.symmetric) {
      off_i = g.in.off[d];
      cap_i = g.in.cap[d];
    }
    lab = ld_lab(&g.lab[d]);
    if (is_ins) {
      len_o = __ldcg(&g.out.len[s]);
      if (!g.symmetric) len_i = __ldcg(&g.in.len[d]);
      val = (uint32_t)ld_v32(g.val32, s);
      top = __ldcg(g.rec_top);
    }
  }
  // 2. found, free, or past the last probe
  uint32_t rid = UNSET;
  bool create = false, open = on;
  uint64_t slot = h0;
#pragma unroll
  for (int k = 0; k < FAST_PROBES; k++) {
    if (open && e[k].x == key.x && (uint32_t)e[k].y == w) {
      rid = (uint32_t)(e[k].y >> 32);
      open = false;
    } else if (open && (uint32_t)e[k].x == NONE) {
      slot = (h0 + k) & g.ht_mask;
      create = is_ins;
      open = false;
    }
  }
  fall = fall || open;
  uint32_t pos_o = 0, pos_i = 0, made = 0;
  if (is_ins || is_del) {
    // two ops on one record, or claiming one slot
    const unsigned long long id = rid != UNSET ? rid : create ? (1ull << 40) | slot : (1ull << 50) | lane;
    const bool twice = __popc(__match_any_sync(FULL, id)) > 1;  // (by every lane, whatever it has found)
    fall = fall || twice;
  }
  if (is_ins) {
    const unsigned cm = __ballot_sync(FULL, create);
    made = __popc(cm);
    const unsigned ms = __match_any_sync(FULL, create ? (unsigned long long)s : (1ull << 40) | lane);
    const unsigned md = __match_any_sync(FULL, create ? (unsigned long long)d : (1ull << 40) | lane);
    if (create) {
      rid = (uint32_t)top + __popc(cm & lt);
      pos_o = len_o + __popc(ms & lt);
      pos_i = len_i + __popc(md & lt);
      fall = fall || top + made > g.rec_cap || pos_o >= cap_o || (!g.symmetric && pos_i >= cap_i);
    }
    better_now = on && Hook<A>::better(Hook<A>::combine(val, w), lab.x);
    const unsigned f = __ballot_sync(FULL, fall), im = __ballot_sync(FULL, better_now);
    if (lane == 0) {
      fs.fall[0] = f;
      fs.improve = im;
    }
  }
  __syncthreads();
  if (is_del) {
    for (uint32_t k = 0; ins && k < fs.n_ins; k++)  // an edge that this submission also inserts
      fall = fall || (on && fs.s[k] == s && fs.d[k] == d && fs.w[k] == w);
    const unsigned f = __ballot_sync(FULL, fall);
    if (lane == 0) fs.fall[1] = f;
  }
  if (tid == 64) {  // (a warp of its own)
    fs.seeds = 0;
    prologue_ctl(c, del ? del->inv_tag : 0ull);
    c[C_STAMP] += ins && del ? 1 : 0;  // as two batches count
    c[C_CANDN] = 0;
  }
  __syncthreads();
  if ((ins && fs.fall[0]) || (del && fs.fall[1])) return FAST_NO;
  const bool seeds_ins = ins && fs.improve != 0;
  // 3. storage; the delete batch waits for an insert that changes labels
  const bool go = is_ins || (is_del && !seeds_ins);
  uint32_t old = 0, ro = pos_o, ri = pos_i;
  if (go && on && rid != UNSET && !create) {
    old = __ldcg(&g.rec_num[rid]);
    ro = __ldcg(&g.rec_out[rid]);
    ri = __ldcg(&g.rec_in[rid]);
  }
  bool seed = false;
  if (go && on && rid != UNSET && (is_ins || old)) {
    E *po = reinterpret_cast<E *>(g.out.pool) + off_o, *pi = reinterpret_cast<E *>(g.in.pool) + off_i;
    auto put = [](E *p, uint32_t x, uint32_t wt) {
      if constexpr (W) *p = make_uint2(x, wt);
      else *p = x;
    };
    const unsigned long long delta = is_ins ? 1ull : ~0ull;
    if (create) {
      g.ht[slot] = make_ulonglong2(key.x, key.y | ((uint64_t)rid << 32));
      g.rec_out[rid] = ro;
      g.rec_in[rid] = g.symmetric ? UNSET : ri;
      g.out.owner[off_o + ro] = s;
      atomicAdd(&g.out.len[s], 1u);
      if (!g.symmetric) {
        g.in.owner[off_i + ri] = d;
        atomicAdd(&g.in.len[d], 1u);
      }
    }
    g.rec_num[rid] = old + (uint32_t)delta;
    atomicAdd(&g.out.deg[s], delta);
    if (!g.symmetric) atomicAdd(&g.in.deg[d], delta);
    if (old == (is_ins ? 0u : 1u)) {  // 0 -> 1 or 1 -> 0
      const uint32_t dead = is_ins ? 0u : DEAD;
      if (ro < cap_o) put(po + ro, d | dead, w);
      if (!g.symmetric && ri < cap_i) put(pi + ri, s | dead, w);
    }
  }
  if (is_ins && made && lane == 0) *g.rec_top = top + made;
  if (go) {
    // The count that comes back and makes the edge a candidate, as in edge_old:
    // an undirected edge's is that of the orientation with the lower source
    // (they differ where directed updates came before).
    const uint32_t ways = __shfl_sync(FULL, old, directed ? lane : (lane & ~1u) + (((lane & 1) != 0) == (s < d)));
    if (on && old_host) {
      if (directed) old_host[lane] = ways;
      else if (!(lane & 1)) old_host[lane >> 1] = ways;
    }
    seed = on && (is_ins ? ways == 0 && better_now : ways == 1 && lab.y == pack_parent(s, w));
  }
  // 4. seeds
  if (is_ins && seeds_ins) {
    const uint32_t st = (uint32_t)c[C_STAMP];
    const bool upd = seed && relax<A>(g, s, ld_v32(g.val32, s), d, w);
    const bool app = upd && atomicExch(&g.stamp[d], st) != st;
    warp_append(app, d, q0, &c[C_QN0], FULL);
    if (mst) mark_modified(g, upd, d, mst);
    warp_add_result(upd, &c[C_RESULT]);
    if (__any_sync(FULL, app) && lane == 0) fs.seeds = 1;
  } else if (is_del && !seeds_ins) {
    const uint32_t tag = (uint32_t)del->inv_tag;
    const bool app = seed && atomicExch(&g.inv[d], tag) != tag;
    warp_append(app, d, q0, &c[C_QN0], FULL);
    if (__any_sync(FULL, app) && lane == 0) fs.seeds = 1;
  }
  __syncthreads();
  if (seeds_ins) return FAST_INS_SEEDS;
  return (del ? FAST_DEL_DONE : 0) | (fs.seeds ? FAST_DEL_SEEDS : 0);
}

// The repair after fast_inline, as a call (its code is in the kernel once more
// in apply_batch), with the kernel's parameters in shared memory: a reference
// into parameter space would be read through L1.
struct FusedShared {
  DevGraph g;
  FusedRepair fr;
};
template <int A, bool W>
__device__ __noinline__ int fast_repair(const FusedShared &f, int add, uint32_t *q0, uint32_t mst) {
  return batch_repair<A, W>(f.g, f.fr, add, q0, mst, nullptr);
}

template <int A, bool W>
__global__ void __launch_bounds__(FS_TPB)
    k_apply_small(const __grid_constant__ DevGraph g, const __grid_constant__ sdev::OpView ops, const ApplyHdr *hdr,
                  const char *data, uint64_t *old_host, uint32_t *cand, int add, int directed, uint32_t *q0,
                  uint32_t mst, int second, const __grid_constant__ FusedRepair fr, uint4 *scratch,
                  unsigned long long *ctl_host) {
  __shared__ StagedBatch sb;
  if (g.ptrace && threadIdx.x == 0) {
    g.ptrace[32 + 2 * second] = global_ns();
    g.ptrace[16 * second + 15] = 0;
    if (!second) g.ptrace[31] = 0;  // a single batch: no delete batch ran
  }
  stage_batch(g, hdr, data, scratch, sb, 0, 32);
  __syncthreads();
  if (g.ptrace && threadIdx.x == 0) g.ptrace[33 + 2 * second] = global_ns();
  const int r = apply_batch<A, W>(g, ops, sb, data, old_host, cand, add, directed, q0, mst, second, fr, scratch);
  if (threadIdx.x == 0) g.ctl[C_LEFT] = r == 1 ? (add ? 1 : 2) : 0;
  ctl_to_host(g, ctl_host);
}

// An insert batch and then a delete batch in one kernel (both staged in one
// round trip): the delete batch runs here too when the insert batch's repair
// finished in place.  C_LEFT tells the host what is left: 1 the insert
// batch's level loop and then the whole delete batch, 2 the delete batch's
// repair.
template <int A, bool W>
__global__ void __launch_bounds__(FS_TPB)
    k_apply_mixed(const __grid_constant__ DevGraph g, const __grid_constant__ sdev::OpView ops, const ApplyHdr *hdr1,
                  const char *data1, const ApplyHdr *hdr2, const char *data2, uint32_t *cand, int directed,
                  uint32_t *q0, uint32_t mst, const __grid_constant__ FusedRepair fr, uint4 *scratch1, uint4 *scratch2,
                  unsigned long long *ctl_host) {
  __shared__ StagedBatch sb1, sb2;
  if (g.ptrace && threadIdx.x == 0) {
    g.ptrace[32] = g.ptrace[34] = global_ns();
    g.ptrace[15] = g.ptrace[31] = 0;
  }
  stage_batch(g, hdr1, data1, scratch1, sb1, 0, 32);
  stage_batch(g, hdr2, data2, scratch2, sb2, 32 + APPLY_SPEC, 64 + APPLY_SPEC);
  __syncthreads();
  if (g.ptrace && threadIdx.x == 0) g.ptrace[33] = g.ptrace[35] = global_ns();
  int r = apply_batch<A, W>(g, ops, sb1, data1, nullptr, cand, 1, directed, q0, mst, 0, fr, scratch1);
  unsigned long long lf = r == 1 ? 1 : 0;
  if (r == 0) {
    __syncthreads();
    r = apply_batch<A, W>(g, ops, sb2, data2, nullptr, cand, 0, directed, q0, mst, 1, fr, scratch2);
    lf = r == 1 ? 2 : 0;
  }
  if (threadIdx.x == 0) g.ctl[C_LEFT] = lf;
  ctl_to_host(g, ctl_host);
}

// The header of an inline batch (its size clamped to what the parameters hold).
__device__ __forceinline__ void inline_header(const DevGraph &g, const InlineBatch &ib, StagedBatch &sb) {
  if (threadIdx.x == 0) {
    sb.stamp = g.ctl[C_STAMP];
    sb.n = ib.n < INLINE_EDGES ? ib.n : INLINE_EDGES;
    sb.pairs = ib.pairs;
    sb.want = ib.want;
    sb.inv_tag = ib.inv_tag;
  }
}

// k_apply_small for an inline batch (launched directly, not from a graph).
// (With the phase trace on, batches take the phases that it stamps.)
template <int A, bool W>
__global__ void __launch_bounds__(FS_TPB)
    k_apply_small_inl(const __grid_constant__ DevGraph g, const __grid_constant__ sdev::OpView ops,
                      const __grid_constant__ InlineBatch ib, uint64_t *old_host, uint32_t *cand, int add, int directed,
                      uint32_t *q0, uint32_t mst, const __grid_constant__ FusedRepair fr,
                      unsigned long long *ctl_host) {
  __shared__ StagedBatch sb;
  __shared__ FusedShared f;
  if (threadIdx.x == 96) {  // (a thread off the critical path)
    f.g = g;
    f.fr = fr;
  }
  inline_header(g, ib, sb);
  __syncthreads();
  int r = g.ptrace ? FAST_NO
                   : fast_inline<A, W>(g, add ? &ib : nullptr, add ? nullptr : &ib, directed,
                                       ib.want ? old_host : nullptr, q0, mst);
  if (r == FAST_NO) {
    if (g.ptrace && threadIdx.x == 0) {
      g.ptrace[32] = g.ptrace[33] = global_ns();
      g.ptrace[15] = 0;
      g.ptrace[31] = 0;
    }
    r = apply_batch<A, W>(g, ops, sb, nullptr, old_host, cand, add, directed, q0, mst, 0, fr, nullptr, ib.words);
  } else {
    r = r & (FAST_INS_SEEDS | FAST_DEL_SEEDS) ? fast_repair<A, W>(f, add, q0, mst) : 0;
  }
  if (threadIdx.x == 0) g.ctl[C_LEFT] = r == 1 ? (add ? 1 : 2) : 0;
  ctl_to_host(g, ctl_host);
}

// k_apply_mixed for two inline batches.  When the insert batch leaves work,
// the host continues exactly as after k_apply_mixed: the delete batch is in
// the staging buffer too (the host wrote it there before the launch).
template <int A, bool W>
__global__ void __launch_bounds__(FS_TPB)
    k_apply_mixed_inl(const __grid_constant__ DevGraph g, const __grid_constant__ sdev::OpView ops,
                      const __grid_constant__ InlineBatch ib1, const __grid_constant__ InlineBatch ib2, uint32_t *cand,
                      int directed, uint32_t *q0, uint32_t mst, const __grid_constant__ FusedRepair fr,
                      unsigned long long *ctl_host) {
  __shared__ StagedBatch sb1, sb2;
  __shared__ FusedShared f;
  if (threadIdx.x == 96) {  // (a thread off the critical path)
    f.g = g;
    f.fr = fr;
  }
  inline_header(g, ib1, sb1);
  inline_header(g, ib2, sb2);
  __syncthreads();
  const int fast = g.ptrace ? FAST_NO : fast_inline<A, W>(g, &ib1, &ib2, directed, nullptr, q0, mst);
  int r = 0;  // the insert batch
  if (fast == FAST_NO) {
    if (g.ptrace && threadIdx.x == 0) {
      g.ptrace[32] = g.ptrace[33] = g.ptrace[34] = g.ptrace[35] = global_ns();
      g.ptrace[15] = g.ptrace[31] = 0;
    }
    r = apply_batch<A, W>(g, ops, sb1, nullptr, nullptr, cand, 1, directed, q0, mst, 0, fr, nullptr, ib1.words);
  } else if (fast & FAST_INS_SEEDS) {
    r = fast_repair<A, W>(f, 1, q0, mst);
  }
  unsigned long long lf = r == 1 ? 1 : 0;
  if (r == 0) {
    __syncthreads();
    if (fast == FAST_NO || !(fast & FAST_DEL_DONE))
      r = apply_batch<A, W>(g, ops, sb2, nullptr, nullptr, cand, 0, directed, q0, mst, 1, fr, nullptr, ib2.words);
    else if (fast & FAST_DEL_SEEDS)
      r = fast_repair<A, W>(f, 0, q0, mst);
    lf = r == 1 ? 2 : 0;
  }
  if (threadIdx.x == 0) g.ctl[C_LEFT] = lf;
  ctl_to_host(g, ctl_host);
}

// ---- the grid engine: levels and deletion repairs in one persistent launch ------
// One CTA per SM (or per two, see ENG_HALF_EDGES), launched cooperatively, runs every level of a build or of a
// repair, with a grid barrier where the graph-driven loop has kernel
// boundaries, a level-begin kernel and a conditional node.  That loop spends
// 15 to 25 us of a level on launches and conditions; a barrier is about 1.5 us.
// Each CTA picks the level's mode from the same counters by the same rules, so
// no decision has to be sent around:
//   * a bottom-up or a pull level, as in the graph-driven loop;
//   * a frontier of at most ENG_STAGE vertices is staged (offset, value, degree
//     prefix) in every CTA's shared memory; with few out-slots CTA 0 runs
//     successive levels alone (tiny_levels), else the slots are spread over
//     all CTAs;
//   * a larger frontier is prefix-summed piecewise, one contiguous piece per
//     CTA, and after a barrier each CTA takes an equal share of the level's
//     slots and stages the vertices that own them.
// Queue counters rotate over three words (in, out, cleared for the next level),
// so that clearing one needs no barrier of its own.  Served graphs keep the
// graph-driven loop: the engine waits until every SM has room, which other
// instances' epochs delay.
constexpr int ENG_TPB = 1024;
constexpr uint32_t ENG_STAGE = 2048;
constexpr int ENG_MAX_CTAS = 256;
constexpr uint32_t ENG_TINY = 1024;          // out-slots that CTA 0 relaxes alone (4096 took 20 us a level, the grid 9)
// a build's push level pulls instead when its out-slots are at least 1 / 12 of the copy's
// entries (RMAT-22 SSWP: the push of 97K vertices took 241 us, a pull level 75).  Builds, us, at
// 1/1, 1/6, 1/12 and 1/24: SSWP RMAT-22 1010, 833, 797, 800; RMAT-20 693, 678, 707, 752; RMAT-18
// 422, 435, 441, 443; SSSP RMAT-20 440, 440, 426, 426; the same at RMAT-18 and 22
constexpr uint64_t ENG_PULL_DIV = 12;
// A push level of Graph::push_slots out-slots (8M) is left, with all that follow, to the graph-driven
// loop (ELEFT_PUSH), whose edge-balanced and dense pushes keep more edges in flight per SM and win there.
// An edge that joins the root to an RMAT-20 graph, us a call, left and not left: SSSP 1165, 1850; BFS
// 525, 596; WCC 688, 832 (RMAT-18, 4M edges, never left: 754, 290, 366; left from 2M on: 695, 331, 390).
// With the line at 4M, putting 300,000 tree edges of RMAT-20 SSSP back took 1438 instead of 1250.  The
// first level of a deletion repair stays unless it is dense: few slots of a reset set with hubs in it
// improve anything, and the engine reads them as fast (such batches of 10,000 deletes lost 70 us each).
constexpr uint64_t ENG_TINY_LEVELS = 2048;   // levels it runs before the others look in again
constexpr int ENG_ITEMS = 2;                 // slots a thread relaxes at a time
// Repairs of batches up to this size take half the SMs, so that those of two
// graphs driven from two threads run side by side (4,000 inserts and deletes on
// each of two RMAT-20 graphs, one call of each: 1,050 us on all SMs, 720 on half,
// 834 for the graph-driven loop; one graph alone 707 and 676).  Larger ones take
// all: deleting 30,000 tree edges of RMAT-20 SSSP 879 us against 935 on half,
// 300,000 2,350 against 2,900; 3,000 the same, 470.  A repair on half that comes to a
// frontier or a reset set of more than Graph::half_vertices (32,768), or to a push of 32
// times as many out-slots, goes on in a second launch, on all (deleting 3,000 edges of an
// RMAT-20 graph, the one that joins it to the root among them, us so, on half alone and on
// all alone: SSSP 2090, 2520, 1970; BFS 1600, 1940, 1675; WCC 2750, 3540, 2760).
constexpr uint64_t ENG_HALF_EDGES = 16384;
static_assert(ENG_TPB == TINY_TPB, "CTA 0 runs the one-CTA levels");
static_assert(TASK_SLOTS >= CHUNK && TASK_DEG >= 2 * TASK_SLOTS, "the hub task queue holds the tasks");

struct EngineArgs {
  // sliced in-edge copy (pull levels)
  const void *ent;
  const uint64_t *off;
  const uint32_t *row_id;
  PullHubs hubs;
  const SellPlan *plan;
  // queues and scratch
  uint32_t *q[2], *tree;
  uint64_t *task;               // tasks of long lists (deletion repairs)
  uint64_t *P;                  // frontier degree prefix, per CTA piece
  unsigned long long *tot;      // slots of each CTA's piece
  unsigned long long *bar;      // barrier words, third queue counter, bounds
  unsigned long long *ctl_host;
  uint64_t root;                // builds
  uint64_t limit, big, max_iter;  // deletion repairs
  LevelCfg cfg;
  uint32_t mst;
  uint32_t polls;               // before a wait gives up
  uint64_t push_slots;          // out-slots of a push level that is left to the loop
  uint64_t half_vertices, half_slots;  // vertices and out-slots at which a launch on half the SMs leaves off
  int build;                    // initialise the labels first
  int del;                      // repair deletions from the invalidated frontier in queue 0 first
};

struct GridBar {
  unsigned long long *w;
  unsigned gen;  // thread 0's
  uint32_t polls;
};

// All CTAs of the grid; false when the wait gave up (the caller returns).  A
// CTA that gives up has arrived, so the others may run the phase after this
// barrier, but none gets past the next one: what that phase lacks is not read.
// It gives up after b.polls polls without a beat from the work that it waits for.
// quiet: giving up is no error (the last barrier, for all CTAs but the one that
// still has work after it).
// A CTA may leave a barrier long before another one has looked at what it
// decides on next, so a word that every CTA reads after a barrier is written
// again only past the barrier after that: counters and flags of successive
// levels alternate between words.
__device__ __forceinline__ bool grid_sync(const DevGraph &g, GridBar &b, bool quiet = false) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned *count = reinterpret_cast<unsigned *>(b.w + EB_COUNT), *gen = reinterpret_cast<unsigned *>(b.w + EB_GEN);
    int ok = 1;
    __threadfence();
    if (atomicAdd(count, 1u) == gridDim.x - 1) {
      atomicExch(count, 0u);
      __threadfence();
      atomicExch(gen, b.gen + 1);
    } else {
      unsigned x, spins = 0;
      unsigned long long beats = 0;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(x) : "l"(gen) : "memory");
        if (x != b.gen) break;
        if (++spins < b.polls) continue;
        const unsigned long long now = __ldcg(&g.ctl[C_BEAT]);
        if (now == beats) break;
        beats = now;
        spins = 0;
      }
      if (x == b.gen) {
        if (!quiet) atomicCAS(&g.ctl[C_ERR], 0ull, (unsigned long long)RG_ETIMEOUT);
        ok = 0;
      }
    }
    __threadfence();
    b.gen++;
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

struct EngStage {
  uint64_t pref[ENG_STAGE + 1];  // first level slot of each staged vertex
  uint64_t base[ENG_STAGE];      // pool slot minus level slot
  uint32_t u[ENG_STAGE], su[ENG_STAGE];
  uint64_t tot[ENG_MAX_CTAS + 1];
};
struct EngShared {
  EngStage p;
  uint32_t q[ENG_TPB / 32][PQ_CAP];
  BlockCounts bc;
  // why the level loop ended early and with how many vertices (thread 0's; in
  // registers they cost BFS builds 3 %)
  unsigned long long left;
  uint64_t left_n;
  // the kernel's parameters: the level kinds are calls and take them by
  // reference, and a reference into parameter space is read through L1, which
  // every barrier empties
  DevGraph g;
  EngineArgs a;
};

// Relax level slots [e0, e1) over the staged vertices (pref ascending; the
// slots of vertex j start at pref[j]).  All threads of the CTA.
template <int A, bool W>
__device__ __noinline__ void eng_relax(const DevGraph &g, EngShared &sh, uint32_t m, uint64_t e0, uint64_t e1,
                                       uint32_t st, uint32_t *fout, unsigned long long *fout_n, uint32_t mst) {
  unsigned long long local = 0;
  using P_ = PoolT<W>;
  const typename P_::E *pool = reinterpret_cast<const typename P_::E *>(g.out.pool);
  for (uint64_t b = e0; b < e1; b += ENG_TPB * ENG_ITEMS) {
    bool on[ENG_ITEMS];
    uint32_t uu[ENG_ITEMS], vv[ENG_ITEMS], ww[ENG_ITEMS];
    uint64_t su[ENG_ITEMS];
#pragma unroll
    for (int k = 0; k < ENG_ITEMS; k++) {
      const uint64_t e = b + (uint64_t)k * ENG_TPB + threadIdx.x;
      on[k] = e < e1;
      uu[k] = vv[k] = ww[k] = 0;
      su[k] = 0;
      if (on[k]) {
        uint32_t lo = 0, hi = m - 1;  // the last vertex that starts at or before e
        while (lo < hi) {
          const uint32_t mid = (lo + hi + 1) >> 1;
          if (sh.p.pref[mid] <= e) lo = mid;
          else hi = mid - 1;
        }
        const typename P_::E ent = pool[sh.p.base[lo] + e];
        uu[k] = sh.p.u[lo];
        su[k] = sh.p.su[lo];
        vv[k] = P_::nbr(ent);
        ww[k] = P_::wt(ent);
        on[k] = !(vv[k] & DEAD);
      }
    }
    relax_batch<A, ENG_ITEMS>(g, on, uu, vv, ww, su, st, fout, fout_n, local, mst);
  }
  block_count(&sh.bc, local, 0);
}

// CTA r's share of S level slots.
__device__ __forceinline__ void eng_share(uint64_t S, uint64_t &e0, uint64_t &e1) {
  uint64_t per = (S + gridDim.x - 1) / gridDim.x;
  if (per < 256) per = 256;
  per = (per + 31) & ~31ull;
  e0 = min(S, per * blockIdx.x);
  e1 = min(S, e0 + per);
}

// Deletion repair over the whole grid (do_update_tree_del,
// core/graph.hpp:1250-1511): the phases of k_rescue, k_expand, k_reset and
// k_pull, each followed by the tasks of the long lists it met.
// Leaves the reset set in queue 0 with its count in ctl[C_QN0], or leaves off
// with the frontier of n vertices there.
enum DelResult : int { DEL_GAVE_UP, DEL_DONE, DEL_LEFT };
// A frontier of queue 1 into queue 0, which holds the one before it (all CTAs).
__device__ __noinline__ void eng_to_q0(const EngineArgs &a, uint64_t n) {
  for (uint64_t i = blockIdx.x * (uint64_t)ENG_TPB + threadIdx.x; i < n; i += (uint64_t)gridDim.x * ENG_TPB)
    a.q[0][i] = a.q[1][i];
}
template <int A, bool W>
__device__ __noinline__ DelResult eng_del(const DevGraph &g, const EngineArgs &a, GridBar &bar, uint64_t &n_left) {
  unsigned long long *c = g.ctl;
  unsigned long long *hvr = a.bar + EB_HVR, *hve = a.bar + EB_HVE;  // two words each, by turns
  auto cnt = [&](uint64_t k) { return k % 3 == 2 ? a.bar + EB_QN2 : &c[C_QN0 + k % 3]; };
  const uint64_t warp = (blockIdx.x * (uint64_t)ENG_TPB + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * ENG_TPB) >> 5;
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  bool recompute = false;
  // the invalidation levels that the one-CTA repair ran before it handed over
  // (every CTA reads them here: the word is written again at the end)
  const uint64_t done = __ldcg(&c[C_INVITER]);
  uint64_t it = 0;
  for (; done + it < a.max_iter; it++) {
    const uint32_t *fin = a.q[it & 1];
    uint32_t *fout = a.q[(it & 1) ^ 1];
    const uint64_t n = __ldcg(cnt(it));
    if (n == 0) break;
    if (done + it <= 10 && __ldcg(&c[C_TREEN]) + n > a.big) {  // core/graph.hpp:1252
      recompute = true;
      break;
    }
    if (n > a.half_vertices) {
      if (it & 1) eng_to_q0(a, n);
      if (lead) c[C_INVITER] = done + it;
      n_left = n;
      return DEL_LEFT;
    }
    if (lead) *cnt(it + 2) = 0;
    RepQueue rq;
    rq.task = a.task;
    rq.n = &hvr[it & 1];
    rescue_warps<A, W>(g, fin, n, a.limit, warp, nwarps, rq);
    if (!grid_sync(g, bar)) return DEL_GAVE_UP;
    const uint64_t nr = __ldcg(rq.n);
    if (nr) {
      const uint32_t tag_inv = (uint32_t)c[C_INVTAG];
      for (uint64_t t = warp; t < nr; t += nwarps) {
        const uint64_t x = a.task[t];
        const uint32_t d = (uint32_t)x, k0 = (uint32_t)(x >> 32) * TASK_SLOTS;
        const uint32_t td = ld_u32(&g.inv[d]);
        const uint64_t sd = ld_v32(g.val32, d);
        const uint32_t len = seg_len(g.in, d);
        const uint64_t off = g.in.off[d];
        if (__shfl_sync(FULL, td, 0) != tag_inv) continue;  // rescued by another task
        rescue_one<A, W>(g, d, sd, k0, min(len, k0 + TASK_SLOTS), off, tag_inv, a.limit);
      }
      if (!grid_sync(g, bar)) return DEL_GAVE_UP;
    }
    if (__ldcg(&c[C_RECOMPUTE])) {  // a chain ran past the guard (nothing sets it before the next level's rescue)
      recompute = true;
      break;
    }
    if (lead) hvr[(it + 1) & 1] = hve[(it + 1) & 1] = 0;
    rq.n = &hve[it & 1];
    expand_warps<A, W>(g, fin, n, a.tree, fout, cnt(it + 1), warp, nwarps, rq);
    if (!grid_sync(g, bar)) return DEL_GAVE_UP;
    const uint64_t ne = __ldcg(rq.n);
    if (ne) {
      const uint32_t tag_inv = (uint32_t)c[C_INVTAG];
      for (uint64_t t = warp; t < ne; t += nwarps) {
        const uint64_t x = a.task[t];
        const uint32_t u = (uint32_t)x, k0 = (uint32_t)(x >> 32) * TASK_SLOTS;
        const uint32_t len = seg_len(g.out, u);
        expand_slots<W, 4>(g, u, g.out.off[u], k0 + lane_id(), 32, min(len, k0 + TASK_SLOTS), tag_inv, fout,
                           cnt(it + 1));
      }
      if (!grid_sync(g, bar)) return DEL_GAVE_UP;
    }
  }
  const uint64_t tn = __ldcg(&c[C_TREEN]);
  if (!grid_sync(g, bar)) return DEL_GAVE_UP;  // (every CTA has read the last counts)
  if (tn > a.half_vertices && !recompute) {
    if (lead) c[C_INVITER] = done + it;
    n_left = 0;  // (nothing is left to invalidate)
    return DEL_LEFT;
  }
  if (lead) {
    c[C_QN0] = recompute ? 0 : tn;
    c[C_QN1] = 0;
    c[C_INVITER] = done + it;
    if (recompute) c[C_RECOMPUTE] = 1;
  }
  if (recompute) return grid_sync(g, bar) ? DEL_DONE : DEL_GAVE_UP;
  // reset the invalid set; it is also the frontier of the push levels
  reset_warps<A>(g, a.tree, tn, a.mst, warp, nwarps);
  for (uint64_t i = blockIdx.x * (uint64_t)ENG_TPB + threadIdx.x; i < tn; i += (uint64_t)gridDim.x * ENG_TPB)
    a.q[0][i] = a.tree[i];
  if (!grid_sync(g, bar)) return DEL_GAVE_UP;
  RepQueue rq;
  rq.task = a.task;
  rq.n = &c[C_HVP];
  unsigned long long local = pull_warps<A, W>(g, a.tree, tn, a.mst, warp, nwarps, rq);
  if (!grid_sync(g, bar)) return DEL_GAVE_UP;
  const uint64_t np = __ldcg(rq.n);
  if (np) {
    for (uint64_t t = warp; t < np; t += nwarps) {
      const uint64_t x = a.task[t];
      const uint32_t d = (uint32_t)x, k0 = (uint32_t)(x >> 32) * TASK_SLOTS;
      const uint32_t len = seg_len(g.in, d);
      PullBest p = {ld_v32(g.val32, d), 0, NONE, 0};
      pull_slots<A, W, 4>(g, g.in.off[d], k0 + lane_id(), 32, min(len, k0 + TASK_SLOTS), p);
      local += pull_reduce<A>(g, p, d, true, 32, a.mst);
    }
    if (!grid_sync(g, bar)) return DEL_GAVE_UP;
  }
  warp_add_result(local, &c[C_RESULT]);
  return DEL_DONE;
}

// The levels end here, with n vertices in queue k & 1 (all CTAs): the launch after
// this one starts with queue 0.
__device__ __noinline__ void eng_leave(const EngineArgs &a, EngShared &sh, unsigned long long what, uint32_t k,
                                       uint64_t n) {
  if (k & 1) eng_to_q0(a, n);
  if (threadIdx.x == 0) {
    sh.left = what;
    sh.left_n = n;
  }
}

// What the next launch needs: this level begins anew there.
__device__ __noinline__ void eng_left_words(const DevGraph &g, const EngineArgs &a, const EngShared &sh, uint64_t lvl,
                                            unsigned pulled) {
  unsigned long long *c = g.ctl;
  c[C_QN0] = sh.left_n;
  c[C_LEVEL] = lvl;
  c[C_MODE] = M_EMPTY;
  c[C_BND0] = a.cfg.bnd_best;
  c[C_PULLED] = pulled != 0;
  c[C_ELEFT] = sh.left;
}

// The level kinds as calls: each gets the registers of a thread for itself
// (inlined into one function they spilled over a kilobyte per thread).
template <int A, bool W>
__device__ __noinline__ void eng_pull(const DevGraph &g, const EngineArgs &a, EngShared &sh, int what, uint32_t m,
                                      bool first, unsigned long long *bout, uint32_t *fout, unsigned long long *fout_n) {
  pull_part<A, W>(g, reinterpret_cast<const typename SellE<W>::E *>(a.ent), a.off, a.row_id, a.hubs, a.plan, what, 0,
                  0, 0, m, bout, sh.q[threadIdx.x >> 5], fout, fout_n, a.mst, &sh.bc, first,
                  (blockIdx.x * ENG_TPB + threadIdx.x) >> 5, (gridDim.x * ENG_TPB) >> 5);
}

template <int A>
__device__ __noinline__ void eng_hub_fix(const DevGraph &g, const EngineArgs &a, EngShared &sh,
                                         unsigned long long *bout, uint32_t *fout, unsigned long long *fout_n) {
  unsigned long long local = 0;
  pull_hub_fix<A>(g, a.hubs, a.plan, bout, fout, fout_n, a.mst, local, blockIdx.x * (uint64_t)ENG_TPB + threadIdx.x,
                  (uint64_t)gridDim.x * ENG_TPB);
  block_count(&sh.bc, local, 0);
}

template <bool W>
__device__ __noinline__ void eng_bottom_up(const DevGraph &g, EngShared &sh, uint64_t d, uint32_t *fout,
                                           unsigned long long *fout_n) {
  bottom_up<W>(g, d, fout, fout_n, blockIdx.x * (uint64_t)ENG_TPB + threadIdx.x, (uint64_t)gridDim.x * ENG_TPB,
               sh.q[threadIdx.x >> 5], &sh.bc);
}

template <int A, bool W>
__device__ __noinline__ void eng_tiny(const DevGraph &g, const EngineArgs &a, uint32_t *q_in, unsigned long long *n_in,
                                      uint32_t *q_out, unsigned long long *n_out, uint64_t max_levels) {
  tiny_levels<A, W>(g, q_in, n_in, q_out, n_out, q_out, n_out, max_levels,
                    min((uint64_t)ENG_TINY, (uint64_t)a.cfg.tiny_edges), a.mst, true);
}

using EngScan = cub::BlockScan<uint64_t, ENG_TPB>;

// Stages a frontier of at most ENG_STAGE vertices (two a thread) and returns its
// out-slots.
__device__ __noinline__ uint64_t eng_stage(const DevGraph &g, EngShared &sh, EngScan::TempStorage &tmp,
                                           const uint32_t *fin, uint32_t n) {
  static_assert(ENG_STAGE == 2 * ENG_TPB, "two vertices per thread");
  const unsigned i = 2 * threadIdx.x;
  uint64_t d[2] = {0, 0}, excl, S;
  uint32_t u[2];
#pragma unroll
  for (int k = 0; k < 2; k++)
    if (i + k < n) u[k] = fin[i + k];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    if (i + k < n) {
      d[k] = seg_len(g.out, u[k]);
      sh.p.u[i + k] = u[k];
      sh.p.base[i + k] = g.out.off[u[k]];
      sh.p.su[i + k] = (uint32_t)ld_v32(g.val32, u[k]);
    }
  }
  EngScan(tmp).ExclusiveSum(d[0] + d[1], excl, S);
#pragma unroll
  for (int k = 0; k < 2; k++) {
    if (i + k < n) {
      sh.p.pref[i + k] = excl;
      sh.p.base[i + k] -= excl;
    }
    excl += d[k];
  }
  __syncthreads();
  return S;
}

// The degree prefix of this CTA's contiguous piece of a large frontier.
__device__ __noinline__ void eng_prefix(const DevGraph &g, const EngineArgs &a, EngScan::TempStorage &tmp,
                                        const uint32_t *fin, uint32_t n, uint32_t per) {
  const uint32_t i0 = min(n, per * blockIdx.x), i1 = min(n, i0 + per);
  uint64_t carry = 0;
  for (uint32_t b = i0; b < i1; b += ENG_TPB) {
    const uint32_t i = b + threadIdx.x;
    uint64_t d = i < i1 ? seg_len(g.out, fin[i]) : 0, x, total;
    EngScan(tmp).ExclusiveSum(d, x, total);
    if (i < i1) a.P[i] = carry + x;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) a.tot[blockIdx.x] = carry;
}

// Where every piece starts; returns the level's slots, and the first vertex of
// this CTA's share [e0, e1) of them: its piece, then 32 probes at a time.
__device__ __noinline__ uint64_t eng_first(const EngineArgs &a, EngShared &sh, EngScan::TempStorage &tmp, uint32_t n,
                                           uint32_t per, uint64_t &e0, uint64_t &e1, uint32_t &first) {
  __shared__ uint32_t s_first;
  const unsigned tid = threadIdx.x, G = gridDim.x;
  uint64_t t = tid < G ? __ldcg(&a.tot[tid]) : 0, x, S;
  EngScan(tmp).ExclusiveSum(t, x, S);
  if (tid < G) sh.p.tot[tid] = x;
  __syncthreads();
  eng_share(S, e0, e1);
  if (tid < 32 && e0 < e1) {
    uint32_t lo = 0, hi = G - 1;  // the last piece that starts at or before e0
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (sh.p.tot[mid] <= e0) lo = mid;
      else hi = mid - 1;
    }
    const uint64_t want = e0 - sh.p.tot[lo];
    uint32_t at = min(n, per * lo), len = min(n, at + per) - at;
    while (len > 1) {
      const uint32_t step = (len + 31) / 32, i = tid * step;
      const bool le = i < len && __ldcg(&a.P[at + i]) <= want;
      const uint32_t last = 31 - __clz(__ballot_sync(FULL, le));  // (lane 0 always passes)
      at += last * step;
      len = min(step, len - last * step);
    }
    if (tid == 0) s_first = at;
  }
  __syncthreads();
  first = s_first;
  return S;
}

// Stages up to ENG_STAGE vertices from i on; returns their number.
__device__ __noinline__ uint32_t eng_stage_from(const DevGraph &g, const EngineArgs &a, EngShared &sh,
                                                const uint32_t *fin, uint32_t n, uint32_t per, uint32_t i, uint64_t S) {
  const uint32_t m = min(ENG_STAGE, n - i);
  for (uint32_t j = threadIdx.x; j <= m; j += ENG_TPB) {
    const uint32_t ij = i + j;
    const uint64_t pj = ij < n ? sh.p.tot[ij / per] + __ldcg(&a.P[ij]) : S;
    sh.p.pref[j] = pj;  // (entry m: where the next vertex starts)
    if (j < m) {
      const uint32_t u = fin[ij];
      sh.p.u[j] = u;
      sh.p.base[j] = g.out.off[u] - pj;
      sh.p.su[j] = (uint32_t)ld_v32(g.val32, u);
    }
  }
  __syncthreads();
  return m;
}

template <int A, bool W>
__global__ void __launch_bounds__(ENG_TPB, 1) k_engine(const __grid_constant__ DevGraph g_arg,
                                                       const __grid_constant__ EngineArgs a_arg) {
  __shared__ EngScan::TempStorage scan_tmp;
  extern __shared__ __align__(16) unsigned char eng_smem[];
  EngShared &sh = *reinterpret_cast<EngShared *>(eng_smem);
  if (threadIdx.x == 0) {
    sh.g = g_arg;
    sh.a = a_arg;
    sh.bc = BlockCounts{0, 0};
    sh.left = ELEFT_NONE;
  }
  __syncthreads();
  const DevGraph &g = sh.g;
  const EngineArgs &a = sh.a;
  unsigned long long *c = g.ctl;
  unsigned long long *bnd = a.bar + EB_BND;
  auto cnt = [&](uint32_t k) { return k % 3 == 2 ? a.bar + EB_QN2 : &c[C_QN0 + k % 3]; };
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  GridBar bar = {a.bar, 0u, a.polls};
  if (threadIdx.x == 0) bar.gen = *reinterpret_cast<volatile unsigned *>(a.bar + EB_GEN);
  // what the launch before left, read before anything below may change it
  uint32_t st = (uint32_t)__ldcg(&c[C_STAMP]);
  uint64_t lvl = a.build ? 0 : __ldcg(&c[C_LEVEL]);
  if (lead) a.bar[EB_QN2] = a.bar[EB_HVR] = a.bar[EB_HVE] = c[C_ELEFT] = 0;
  if (a.build) {
    init_labels<A>(g, a.root, a.q[0], blockIdx.x * (uint64_t)ENG_TPB + threadIdx.x, (uint64_t)gridDim.x * ENG_TPB);
    if (lead) {
      prologue_words(c, 0ull);
      c[C_QN0] = Hook<A>::all_active ? g.V : 1;
      c[C_ROOT] = a.root;
      bnd[1] = a.cfg.bnd_worst;  // (the first level's output bound; only builds pull)
    }
  }
  if (!grid_sync(g, bar)) return;
  bool levels = true;
  if (a.del) {
    uint64_t n = 0;
    const DelResult r = eng_del<A, W>(g, a, bar, n);
    if (r == DEL_GAVE_UP) return;
    levels = r == DEL_DONE;
    if (!levels) eng_leave(a, sh, ELEFT_REPAIR, 0, n);
  }
  unsigned pulled = 0;  // 1: the level before, 2: any level before (one register: two cost 1% of a build)
  for (uint32_t k = 0; levels; k++) {
    const uint32_t *fin = a.q[k & 1];
    uint32_t *fout = a.q[(k & 1) ^ 1];
    unsigned long long *fout_n = cnt(k + 1);
    const uint64_t n = __ldcg(cnt(k));
    if (n == 0) break;
    if (lvl >= a.cfg.max_levels) {
      if (lead) atomicCAS(&c[C_ERR], 0ull, (unsigned long long)RG_ETIMEOUT);
      break;
    }
    if (n > a.half_vertices) {
      eng_leave(a, sh, ELEFT_LEVELS, k, n);
      break;
    }
    st++;
    if (lead) {
      *cnt(k + 2) = 0;
      bnd[(k + 2) % 3] = a.cfg.bnd_worst;
      c[C_STAMP] = st;
      c[C_DEPTH] = lvl;
      if (lvl < TRACE_CAP) {
        g.trace[lvl] = n;
        g.trace[TRACE_CAP + lvl] = global_ns();
      }
      c[C_LEVEL] = lvl + 1;
    }
    // the mode rules of k_level_begin, and a pull in place of a push that
    // would relax a large part of the graph
    const bool bu = a.cfg.bottom_up && !pulled && n * a.cfg.bu_div >= g.V;
    bool pull = !bu && a.cfg.allow_pull && n * (pulled & 1 ? (a.cfg.pull_div + 3) / 4 : a.cfg.pull_div) >= g.V;
    if (bu) {
      eng_bottom_up<W>(g, sh, lvl, fout, fout_n);
    } else if (!pull && n <= ENG_STAGE) {
      const uint64_t S = eng_stage(g, sh, scan_tmp, fin, (uint32_t)n);
      if (n <= TINY_N && S <= a.cfg.tiny_edges && S <= ENG_TINY) {
        if (!grid_sync(g, bar)) return;  // (every CTA has read the counts that CTA 0 now uses by turns)
        unsigned long long *at = a.bar + EB_LVL + 2 * (k & 1);  // where CTA 0 got to
        if (blockIdx.x == 0) {
          eng_tiny<A, W>(g, a, a.q[k & 1], cnt(k), fout, fout_n,
                         min((uint64_t)a.cfg.max_levels, lvl + ENG_TINY_LEVELS));
          if (threadIdx.x == 0) {
            at[0] = c[C_LEVEL];
            at[1] = c[C_STAMP];
          }
        }
        if (!grid_sync(g, bar)) return;
        lvl = __ldcg(&at[0]);
        st = (uint32_t)__ldcg(&at[1]);
        pulled &= 2;
        continue;
      }
      uint64_t e0, e1;
      eng_share(S, e0, e1);
      eng_relax<A, W>(g, sh, (uint32_t)n, e0, e1, st, fout, fout_n, a.mst);
      if (lead) atomicAdd(&sh.bc.scanned, (unsigned long long)S);
    } else if (!pull) {
      const uint32_t per = (uint32_t)((n + gridDim.x - 1) / gridDim.x);
      eng_prefix(g, a, scan_tmp, fin, (uint32_t)n, per);
      if (!grid_sync(g, bar)) return;
      uint64_t e0, e1;
      uint32_t i;
      const uint64_t S = eng_first(a, sh, scan_tmp, (uint32_t)n, per, e0, e1, i);
      pull = a.cfg.allow_pull && S * ENG_PULL_DIV >= a.plan->total;
      if (!pull && S >= a.push_slots && !(a.del && k == 0 && n * 20 < g.V)) {
        eng_leave(a, sh, ELEFT_PUSH, k, n);
        break;
      }
      if (S >= a.half_slots) {
        eng_leave(a, sh, ELEFT_LEVELS, k, n);
        break;
      }
      for (uint64_t e = e0; e < e1 && !pull;) {
        const uint32_t m = eng_stage_from(g, a, sh, fin, (uint32_t)n, per, i, S);
        const uint64_t end = min(e1, sh.p.pref[m]);
        eng_relax<A, W>(g, sh, m, e, end, st, fout, fout_n, a.mst);
        __syncthreads();
        e = end;
        i += m;
      }
      if (lead && !pull) atomicAdd(&sh.bc.scanned, (unsigned long long)S);
    }
    if (pull) {
      const uint32_t m = pulled & 1 ? (uint32_t)__ldcg(&bnd[k % 3]) : a.cfg.bnd_best;
      unsigned long long *bout = &bnd[(k + 1) % 3];
      eng_pull<A, W>(g, a, sh, a.cfg.pull_split ? PART_HUBS : PART_ALL, m, lvl == 0, bout, fout, fout_n);
      if (!grid_sync(g, bar)) return;
      eng_hub_fix<A>(g, a, sh, bout, fout, fout_n);
      if (a.cfg.pull_split) {
        if (!grid_sync(g, bar)) return;
        eng_pull<A, W>(g, a, sh, PART_REST, m, lvl == 0, bout, fout, fout_n);
      }
    }
    pulled = pull ? 3 : pulled & 2;
    lvl++;
    if (!grid_sync(g, bar)) return;
  }
  counts_out(g, &sh.bc);
  if (!grid_sync(g, bar, blockIdx.x != 0)) return;  // (every CTA has read the last queue counts)
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) {
      c[C_QN0] = 0;
      c[C_QN1] = 0;
      if (sh.left) eng_left_words(g, a, sh, lvl, pulled);
      if (lvl < TRACE_CAP) g.trace[TRACE_CAP + lvl] = global_ns();
    }
    ctl_to_host(g, a.ctl_host);
  }
}

// need_update_tree_add (core/graph.hpp:987-1000) / need_update_tree_del
// (:1220-1233) per edge.
template <int A>
__global__ void k_classify(DevGraph g, const uint32_t *os, const uint32_t *od, const uint32_t *ow, uint64_t n,
                           int directed, const uint8_t *is_del, uint8_t *unsafe) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    bool del = is_del && is_del[i];
    bool r = false;
    for (int dir = 0; dir < (directed ? 1 : 2); dir++) {
      uint64_t op = directed ? i : 2 * i + dir;
      uint32_t u = os[op], v = od[op], w = ow[op];
      if (del) r = r || ld_meta(&g.lab[v]) == pack_parent(u, w);
      else r = r || Hook<A>::better(Hook<A>::combine(ld_v32(g.val32, u), w), ld_val(&g.lab[v]));
    }
    unsafe[i] = r;
  }
}

__global__ void k_unpack_labels(DevGraph g, uint64_t *val, uint64_t *par, uint64_t *pw) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < g.V; v += stride) {
    ulonglong2 l = g.lab[v];
    if (val) val[v] = l.x;
    uint32_t p = (uint32_t)l.y;
    if (par) par[v] = p == NONE ? (uint64_t)g.V : (uint64_t)p;
    if (pw) pw[v] = p == NONE ? 0 : (l.y >> 32);
  }
}

__global__ void k_checksum(DevGraph g) {
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  unsigned long long h = 0;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < g.V; v += stride)
    h += splitmix64(g.lab[v].x ^ (v * 0x9E3779B97F4A7C15ull));
  for (int o = 16; o; o >>= 1) h += __shfl_down_sync(FULL, h, o);
  if (lane_id() == 0) atomicAdd(&g.ctl[C_CHECKSUM], h);
}

// ---------------------------------------------------------------- host side

int grid_warps(const Graph &g, uint64_t warps) {
  uint64_t b = (warps * 32 + TPB - 1) / TPB;
  uint64_t cap = (uint64_t)g.num_sms * 16;
  if (b > cap) b = cap;
  return (int)(b ? b : 1);
}

uint32_t mod_stamp(Graph &g) { return g.trace ? 1u : 0u; }

// Wait for the call's work and take the control block, which the last kernel
// may have written to the host's copy itself.
int read_ctl(Graph &g) {
  if (g.ctl_on_host) return sync_ctl(g);
  RG_CUDA(cudaMemcpyAsync(g.h_ctl, g.d.ctl, sizeof(unsigned long long) * C_COUNT, cudaMemcpyDeviceToHost, g.stream));
  RG_CUDA(cudaStreamSynchronize(g.stream));
  return RG_OK;
}

// Stamps and dense-level activity ids count up on the device, one per level.
// A call runs at most max_levels levels, so clearing the arrays whenever the
// last observed counter is within that margin of 2^32 keeps them unique.
int guard_counters(Graph &g) {
  const uint64_t margin = 8 * (uint64_t)g.V + (1ull << 16);
  if (g.h_ctl[C_STAMP] + margin >= 0xFFFFFFFFull) {
    RG_CUDA(cudaMemsetAsync(g.d.stamp, 0, (size_t)g.V * 4 + 4, g.stream));
    RG_CUDA(cudaMemsetAsync(&g.d.ctl[C_STAMP], 0, 8, g.stream));
    g.h_ctl[C_STAMP] = 0;
  }
  if (g.h_ctl[C_ACT] + margin >= 0xFFFFFFFFull) {
    RG_CUDA(cudaMemsetAsync(g.act, 0, (size_t)g.V * 4 + 4, g.stream));
    RG_CUDA(cudaMemsetAsync(&g.d.ctl[C_ACT], 0, 8, g.stream));
    g.h_ctl[C_ACT] = 0;
  }
  return RG_OK;
}

template <bool W, int K>
int sell_fill_sorted(Graph &g, uint64_t s_lo, uint64_t s_hi, const uint32_t *pv, const uint32_t *pst,
                     const uint32_t *pln) {
  if (s_lo >= s_hi) return RG_OK;
  using E = typename SellE<W>::E;
  const size_t smem = sell_fill_smem(K, sizeof(E));
  RG_CUDA(cudaFuncSetAttribute(k_sell_fill_sorted<W, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  count_launch(g);
  const uint64_t blocks = std::min<uint64_t>(s_hi - s_lo, (uint64_t)g.num_sms * 8);
  k_sell_fill_sorted<W, K><<<(unsigned)blocks, SF_TPB, smem, g.stream>>>(g.d, g.sell_row, g.sell_plan_host->rows, s_lo, s_hi,
                                                                      g.sell_off, pv, pst, pln,
                                                                      reinterpret_cast<E *>(g.sell_ent));
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

// Sliced-ELL copy of the in-edges for dense pull levels, rebuilt only after
// the adjacency changed (three passes over the list lengths, one host
// synchronisation for the sizes, one copy of the entries per version).
template <bool W>
int prepare_pull_w(Graph &g) {
  const uint64_t V = g.V;
  auto grow = [&](void **p, uint64_t &cap, uint64_t want, size_t esz) -> int {
    if (want <= cap && *p) return RG_OK;
    if (*p) {
      cudaFree(*p);
      g.bytes -= cap * esz;
    }
    *p = nullptr;
    cap = 0;
    g.sell_epoch++;  // cached loop graphs hold the old address
    const uint64_t c = want + want / 8 + 64;
    if (cudaMalloc(p, c * esz) != cudaSuccess) {
      cudaGetLastError();
      set_error("device allocation failed: pull preparation");
      return RG_ENOMEM_HBM;
    }
    cap = c;
    g.bytes += c * esz;
    return RG_OK;
  };
  int rc = RG_OK;
  // the hub arrays are sized for every vertex once, so their addresses stay
  // fixed for the cached level-loop graph
  if ((rc = grow((void **)&g.sell_hub, g.sell_hub_cap, V + 1, 4))) return rc;
  if (!g.sell_hub_best) {
    if (cudaMalloc(&g.sell_hub_best, g.sell_hub_cap * 8) != cudaSuccess) {
      cudaGetLastError();
      set_error("device allocation failed: pull preparation");
      return RG_ENOMEM_HBM;
    }
    g.bytes += g.sell_hub_cap * 8;
  }
  RG_CUDA(cudaMemsetAsync(g.sell_plan, 0, sizeof(SellPlan), g.stream));
  count_launch(g, 2);
  k_sell_count<<<g.num_sms * 2, 1024, 0, g.stream>>>(g.d, g.sell_hub, reinterpret_cast<uint64_t *>(g.sell_hub_best),
                                                      g.sell_plan);
  k_sell_plan<<<1, SP_TPB, 0, g.stream>>>(g.sell_plan);
  RG_CUDA(cudaMemcpyAsync(g.sell_plan_host, g.sell_plan, sizeof(SellPlan), cudaMemcpyDeviceToHost, g.stream));
  RG_CUDA(cudaStreamSynchronize(g.stream));
  const SellPlan &plan = *g.sell_plan_host;
  const uint64_t P = plan.pieces;
  if ((rc = grow((void **)&g.sell_piece, g.sell_piece_cap, 4 * (P + 1), 4))) return rc;
  if ((rc = grow((void **)&g.sell_piece_best, g.sell_best_cap, P + 1, 16))) return rc;
  if ((rc = grow((void **)&g.sell_row, g.sell_row_cap, V + P + 32, 4))) return rc;
  if ((rc = grow((void **)&g.sell_off, g.sell_off_cap, plan.slices + 1, 8))) return rc;
  if ((rc = grow(&g.sell_ent, g.sell_cap, plan.total, W ? 8 : 4))) return rc;
  // (the parts of the piece table lie by its capacity: the cached loop graphs hold their addresses)
  const uint64_t pcap = g.sell_piece_cap / 4;
  uint32_t *pv = g.sell_piece, *pst = pv + pcap, *pln = pst + pcap;
  count_launch(g);
  k_sell_rows<<<g.num_sms * 4, SR_TPB, 0, g.stream>>>(g.d, g.sell_hub, g.sell_hub_best, g.sell_plan, g.sell_row, pv, pst,
                                                      pln, pln + pcap, g.sell_off);
  RG_CUDA(cudaGetLastError());
  // the rows that a pull reads in parts, in order; K = ceil(width / 32)
  constexpr int KP = ((int)PULL_PIECE + 31) / 32, KV = ((int)PULL_HUB + 31) / 32;
  static_assert(KV > 8 && PULL_HUB > 256, "K of the fills below");
  const uint32_t *sl = plan.slice;
  if ((rc = sell_fill_sorted<W, KP>(g, 0, sl[PULL_HUB], pv, pst, pln))) return rc;
  if ((rc = sell_fill_sorted<W, KV>(g, sl[PULL_HUB], sl[256], pv, pst, pln))) return rc;
  if ((rc = sell_fill_sorted<W, 8>(g, sl[256], sl[128], pv, pst, pln))) return rc;
  if ((rc = sell_fill_sorted<W, 4>(g, sl[128], sl[64], pv, pst, pln))) return rc;
  if ((rc = sell_fill_sorted<W, 2>(g, sl[64], sl[32], pv, pst, pln))) return rc;
  if ((rc = sell_fill_sorted<W, 1>(g, sl[32], sl[8], pv, pst, pln))) return rc;
  const uint64_t plain_lo = sl[8];
  if (plain_lo < plan.slices) {
    count_launch(g);
    k_sell_fill<W><<<g.num_sms * 16, TPB, 0, g.stream>>>(g.d, g.sell_row, plan.rows, plain_lo, plan.slices,
                                                         g.sell_off, pv, pst, pln,
                                                         reinterpret_cast<typename SellE<W>::E *>(g.sell_ent));
    RG_CUDA(cudaGetLastError());
  }
  g.pull_version = g.adj_version;
  return RG_OK;
}

// Dense build levels pull (sliced ELL) for SSSP / SSWP / WCC by default; BFS
// builds use their bottom-up levels.  RG_OPT_DENSE_PULL 0 / 1 force push / pull.
bool pull_on(const Graph &g, int A) { return g.dense_pull == 1 || (g.dense_pull == 2 && A != RG_BFS); }

// Two-launch pull levels: RG_OPT_PULL_SPLIT 1 always, 0 never, 2 (default) for SSSP and WCC.
bool pull_split_on(const Graph &g, int A) {
  return g.pull_split == 1 || (g.pull_split == 2 && (A == RG_SSSP || A == RG_WCC));
}

int prepare_pull(Graph &g) {
  if (g.pull_version == g.adj_version) return RG_OK;
  return g.weighted ? prepare_pull_w<true>(g) : prepare_pull_w<false>(g);
}

PullHubs pull_hubs(const Graph &g) {
  return PullHubs{g.sell_piece, g.sell_piece + 3 * (g.sell_piece_cap / 4), g.sell_hub, g.sell_piece_best, g.sell_hub_best};
}

// First entry of slice s (or the entries in all).
uint64_t sell_offset(const Graph &g, uint64_t s) {
  const SellPlan &p = *g.sell_plan_host;
  if (s >= p.slices) return p.total;
  int lo = 1, hi = SELL_KEYS - 1;  // the smallest key k with slice[k] <= s
  while (lo < hi) {
    const int mid = (lo + hi) / 2;
    if (p.slice[mid] <= s) hi = mid;
    else lo = mid + 1;
  }
  return p.base[lo] + (s - p.slice[lo]) * 32 * sell_width(lo);
}

// Slice bounds of the launches that follow the hub launch of a split pull
// level: [mid, b1), [b1, b2), ..., [b_k, c4), the narrow slices with the last
// launch; groups - 1 launches holding about equal shares of the entries of
// slices [mid, end).
std::vector<uint64_t> pull_group_bounds(const Graph &g, uint64_t mid, uint64_t c4, uint64_t groups) {
  std::vector<uint64_t> b{mid};
  const uint64_t k = groups > 2 ? groups - 1 : 1;
  if (k > 1 && mid <= c4) {
    const uint64_t e0 = sell_offset(g, mid), e1 = g.sell_plan_host->total;
    for (uint64_t i = 1; i < k; i++) {
      const uint64_t target = e0 + (e1 - e0) * i / k;
      uint64_t lo = mid, hi = c4;  // first slice at or past the target
      while (lo < hi) {
        const uint64_t m = (lo + hi) / 2;
        if (sell_offset(g, m) < target) lo = m + 1;
        else hi = m;
      }
      const uint64_t s = std::min(std::max(lo, b.back()), c4);
      if (s > b.back() && s < c4) b.push_back(s);
    }
  }
  b.push_back(c4);
  return b;
}

uint64_t max_levels_of(const Graph &g) { return g.max_levels ? g.max_levels : 4 * (uint64_t)g.V + 1024; }

// Kernels of one level mode for one half-level (queue half -> queue half^1).
template <int A, bool W>
int enqueue_mode(Graph &g, cudaStream_t s, int half, unsigned long long mode) {
  const uint32_t *fin = g.q[half];
  unsigned long long *fin_n = &g.d.ctl[C_QN0 + half];
  uint32_t *fout = g.q[half ^ 1];
  unsigned long long *fout_n = &g.d.ctl[C_QN0 + (half ^ 1)];
  unsigned long long *hub_n = &g.d.ctl[C_HUBN];
  const uint32_t mst = mod_stamp(g);
  switch (mode) {
    case M_SPARSE:
      k_push<A, W><<<g.num_sms * 16, TPB, 0, s>>>(g.d, fin, fin_n, fout, fout_n, g.hubq, hub_n, mst);
      k_push_hub<A, W><<<g.num_sms * 8, TPB, 0, s>>>(g.d, g.hubq, hub_n, fout, fout_n, mst);
      break;
    case M_PULL: {
      const auto *ent = reinterpret_cast<const typename SellE<W>::E *>(g.sell_ent);
      const bool split = pull_split_on(g, A);
      const unsigned long long *bin = &g.d.ctl[C_BND0 + half];
      unsigned long long *bout = &g.d.ctl[C_BND0 + (half ^ 1)];
      auto pull = [&](int part, uint32_t lo, uint32_t hi, int rest) {
        k_pull_sell<A, W><<<g.num_sms * 8, PS_TPB, 0, s>>>(g.d, ent, g.sell_off, g.sell_row, pull_hubs(g), g.sell_plan,
                                                           part, lo, hi, rest, bin, bout, fout, fout_n, mst);
      };
      pull(split ? PART_HUBS : PART_ALL, 0, 0, 0);
      k_pull_hub_fix<A><<<g.num_sms * 2, 256, 0, s>>>(g.d, pull_hubs(g), g.sell_plan, bout, fout, fout_n, mst);
      if (!split || g.pull_groups <= 2) {
        pull(split ? PART_REST : PART_NONE, 0, 0, 0);
      } else {
        // the other rows, in widest-first groups of equal entries: each group
        // reads the values the groups before it set in this level
        const std::vector<uint64_t> b = pull_group_bounds(g, g.sell_plan_host->slice[PULL_HUB],
                                                          g.sell_plan_host->slice[4], g.pull_groups);
        for (size_t i = 0; i + 1 < b.size(); i++) pull(PART_RANGE, (uint32_t)b[i], (uint32_t)b[i + 1], i + 2 == b.size() ? 1 : 0);
      }
      break;
    }
    case M_DENSE_PUSH:
      k_mark_active<<<g.num_sms * 8, TPB, 0, s>>>(g.d, fin, fin_n, g.act);
      k_push_dense<A, W><<<g.num_sms * 3, DN_TPB, 0, s>>>(g.d, g.act, fout, fout_n, mst);
      break;
    case M_TINY:
      k_push_tiny<A, W><<<1, TINY_TPB, 0, s>>>(g.d, g.q[half], fin_n, g.q[half ^ 1], fout_n, max_levels_of(g),
                                               std::min<uint64_t>(g.tiny_edges, TINY_EDGES), mst);
      break;
    case M_BOTTOM_UP:
      k_bfs_bottom_up<W><<<g.num_sms * 8, TPB, 0, s>>>(g.d, fout, fout_n);
      break;
    case M_CLUSTER: {
      if (!g.cl_ctas) break;  // never selected then
      cudaLaunchConfig_t lc = {};
      lc.gridDim = dim3((unsigned)g.cl_ctas);
      lc.blockDim = dim3(CL_TPB);
      lc.stream = s;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = (unsigned)g.cl_ctas;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      lc.attrs = at;
      lc.numAttrs = 1;
      uint32_t *qi = g.q[half], *qo = g.q[half ^ 1];
      if (cudaLaunchKernelEx(&lc, k_push_cluster<A, W>, g.d, qi, fin_n, qo, fout_n,
                             reinterpret_cast<unsigned long long *>(g.lb_sums), max_levels_of(g),
                             std::min<uint64_t>(g.cluster_edges, CL_EDGES), mst) != cudaSuccess)
        return RG_ECUDA;
      break;
    }
    case M_LBS:
      k_scan_sums<<<SC_BLOCKS, SC_TPB, 0, s>>>(g.d, fin, fin_n, g.scratch64, g.lb_sums);
      k_scan_top<<<1, SC_BLOCKS, 0, s>>>(g.lb_sums);
      k_scan_final<<<SC_BLOCKS, SC_TPB, 0, s>>>(fin_n, g.scratch64, g.lb_sums, g.lb_P);
      k_partition<<<g.num_sms * 4, TPB, 0, s>>>(g.lb_P, fin_n, g.lb_tile);
      k_push_lbs<A, W><<<g.num_sms * 3, LB_TPB, 0, s>>>(g.d, fin, fin_n, g.lb_P, g.lb_tile, fout, fout_n, mst);
      break;
    default:
      break;
  }
  return cudaGetLastError() == cudaSuccess ? RG_OK : RG_ECUDA;
}

// Hash of every level-mode knob: cached graphs bake them into kernel arguments.
uint64_t cfg_key(const LevelCfg &c) {
  uint64_t h = splitmix64(c.dense_div);
  h = splitmix64(h ^ c.lbs_min);
  h = splitmix64(h ^ c.bu_div);
  h = splitmix64(h ^ c.pull_div);
  h = splitmix64(h ^ c.pull_split);
  h = splitmix64(h ^ c.tiny_edges);
  h = splitmix64(h ^ c.max_levels);
  h = splitmix64(h ^ c.pull_groups);
  h = splitmix64(h ^ c.cl_edges);
  h = splitmix64(h ^ c.cl_v);
  return splitmix64(h ^ ((uint64_t)c.allow_pull << 1) ^ (uint64_t)c.bottom_up);
}

LevelCfg level_cfg(const Graph &g, int A, bool build_variant) {
  LevelCfg cfg;
  cfg.dense_div = g.dense_div;
  cfg.lbs_min = g.lbs_min;
  cfg.allow_pull = (build_variant && pull_on(g, A)) ? 1 : 0;
  cfg.bottom_up = (A == RG_BFS && build_variant && g.bfs_bottom_up) ? 1 : 0;
  cfg.bu_div = g.bu_div;
  cfg.pull_div = g.pull_div;
  cfg.pull_split = pull_split_on(g, A) ? 1 : 0;
  cfg.tiny_edges = g.tiny_edges < TINY_EDGES ? g.tiny_edges : TINY_EDGES;
  cfg.max_levels = max_levels_of(g);
  cfg.pull_groups = cfg.pull_split ? std::max<uint64_t>(2, g.pull_groups) : 2;
  cfg.cl_edges = g.cl_ctas ? std::min<uint64_t>(g.cluster_edges, CL_EDGES) : 0;
  cfg.cl_v = (uint64_t)g.cl_ctas * CL_TPB;
  cfg.bnd_best = A == RG_SSWP ? 0xFFFFFFFFu : 0u;
  cfg.bnd_worst = ~cfg.bnd_best;
  return cfg;
}

uint64_t recompute_threshold(const Graph &g) {
  return std::max<uint64_t>((uint64_t)(0.05 * (double)g.V), g.recompute_min);
}

// The level loop as a node of a CUDA graph:
//   WHILE (frontier non-empty) {
//     k_level_begin(q0 -> q1) ; SWITCH(mode) { sparse | pull | dense push | bottom-up | edge-balanced }
//     k_level_begin(q1 -> q0) ; SWITCH(mode) { ... }
//     k_loop_cond
//   }
// added to `graph` after `deps`.
template <int A, bool W>
int add_level_loop(Graph &g, cudaGraph_t graph, const cudaGraphNode_t *deps, size_t ndeps, const LevelCfg &cfg,
                   cudaGraphNode_t *out) {
  if (!g.cap_stream) RG_CUDA(cudaStreamCreateWithFlags(&g.cap_stream, cudaStreamNonBlocking));
  int rc = RG_OK;
  cudaError_t e = cudaSuccess;
  do {
    cudaGraphConditionalHandle wh;
    if ((e = cudaGraphConditionalHandleCreate(&wh, graph, 1, cudaGraphCondAssignDefault)) != cudaSuccess) break;
    cudaGraphNodeParams wp = {};
    wp.type = cudaGraphNodeTypeConditional;
    wp.conditional.handle = wh;
    wp.conditional.type = cudaGraphCondTypeWhile;
    wp.conditional.size = 1;
    if ((e = cudaGraphAddNode(out, graph, deps, ndeps, &wp)) != cudaSuccess) break;
    cudaGraph_t body = wp.conditional.phGraph_out[0];
    cudaGraphNode_t prev = nullptr;
    for (int half = 0; half < 2 && e == cudaSuccess && !rc; half++) {
      cudaGraphConditionalHandle sw;
      if ((e = cudaGraphConditionalHandleCreate(&sw, body, 0, 0)) != cudaSuccess) break;
      const uint32_t *fin = g.q[half];
      const unsigned long long *fin_n = &g.d.ctl[C_QN0 + half];
      unsigned long long *fout_n = &g.d.ctl[C_QN0 + (half ^ 1)];
      int use_switch = 1;
      LevelCfg c = cfg;
      void *args[] = {(void *)&g.d, (void *)&fin, (void *)&fin_n, (void *)&fout_n, (void *)&c, (void *)&use_switch,
                      (void *)&sw};
      cudaKernelNodeParams kp = {};
      kp.func = (void *)k_level_begin;
      kp.gridDim = dim3(1);
      kp.blockDim = dim3(LVB_TPB);
      kp.kernelParams = args;
      cudaGraphNode_t kn;
      if ((e = cudaGraphAddKernelNode(&kn, body, prev ? &prev : nullptr, prev ? 1 : 0, &kp)) != cudaSuccess) break;
      cudaGraphNodeParams sp = {};
      sp.type = cudaGraphNodeTypeConditional;
      sp.conditional.handle = sw;
      sp.conditional.type = cudaGraphCondTypeSwitch;
      sp.conditional.size = M_COUNT;
      cudaGraphNode_t sn;
      if ((e = cudaGraphAddNode(&sn, body, &kn, 1, &sp)) != cudaSuccess) break;
      for (unsigned long long m = 1; m < M_COUNT && e == cudaSuccess && !rc; m++) {
        if (m == M_PULL && !cfg.allow_pull) continue;
        if (m == M_BOTTOM_UP && !cfg.bottom_up) continue;
        if (m == M_CLUSTER && !cfg.cl_edges) continue;
        cudaGraph_t cg = sp.conditional.phGraph_out[m];
        if ((e = cudaStreamBeginCaptureToGraph(g.cap_stream, cg, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed)) !=
            cudaSuccess)
          break;
        rc = enqueue_mode<A, W>(g, g.cap_stream, half, m);
        e = cudaStreamEndCapture(g.cap_stream, &cg);
      }
      prev = sn;
    }
    if (e != cudaSuccess || rc) break;
    const unsigned long long *n_after = &g.d.ctl[C_QN0];
    uint64_t maxl = max_levels_of(g);
    void *cargs[] = {(void *)&g.d, (void *)&n_after, (void *)&maxl, (void *)&wh};
    cudaKernelNodeParams cp = {};
    cp.func = (void *)k_loop_cond;
    cp.gridDim = dim3(1);
    cp.blockDim = dim3(1);
    cp.kernelParams = cargs;
    cudaGraphNode_t cn;
    e = cudaGraphAddKernelNode(&cn, body, &prev, 1, &cp);
  } while (0);
  if (e != cudaSuccess) return cuda_fail(e, "building the level-loop graph");
  return rc;
}

// Deletion repair as nodes of a CUDA graph (do_update_tree_del,
// core/graph.hpp:1235-1612):
//   k_del_tiny (small repairs in one CTA) -> IF (it handed over) {
//     WHILE (invalidated frontier non-empty and no recompute) {
//       k_inv_begin ; k_rescue ; k_expand     (queue 0 -> 1)
//       k_inv_begin ; k_rescue ; k_expand     (queue 1 -> 0)
//       k_inv_cond }
//     k_reset ; k_pull ; k_copy_frontier (reset set -> queue 0 for the push loop) }
// *out is the IF node.  With `fused` (the fused apply kernel ran the one-CTA
// repair and left its hand-over decision in C_OVER) the first node is
// k_handover instead of k_del_tiny.
template <int A, bool W>
int add_del_repair(Graph &g, cudaGraph_t graph, const cudaGraphNode_t *deps, size_t ndeps, cudaGraphNode_t *out,
                   bool fused = false) {
  if (!g.cap_stream) RG_CUDA(cudaStreamCreateWithFlags(&g.cap_stream, cudaStreamNonBlocking));
  const uint64_t big = recompute_threshold(g);
  const uint64_t limit = (uint64_t)((double)g.V * 0.1);  // has_parents guard, core/graph.hpp:1900
  uint32_t mst = mod_stamp(g);
  const int gridw = g.num_sms * 16;
  cudaError_t e = cudaSuccess;
  do {
    cudaGraphConditionalHandle th;
    if ((e = cudaGraphConditionalHandleCreate(&th, graph, 1, cudaGraphCondAssignDefault)) != cudaSuccess) break;
    uint32_t *q0 = g.q[0], *q1 = g.q[1], *tr = g.tree;
    uint64_t max_iter = (uint64_t)g.V + 2;
    int in_graph = 1;
    void *ta[] = {(void *)&g.d, (void *)&q0, (void *)&q1, (void *)&tr, (void *)&limit, (void *)&big,
                  (void *)&max_iter, (void *)&mst, (void *)&th, (void *)&in_graph};
    void *hoa[] = {(void *)&g.d, (void *)&th};
    cudaKernelNodeParams tp = {};
    tp.func = fused ? (void *)k_handover : (void *)k_del_tiny<A, W>;
    tp.gridDim = dim3(1);
    tp.blockDim = dim3(fused ? 1 : DT_TPB);
    tp.kernelParams = fused ? hoa : ta;
    cudaGraphNode_t tn;
    if ((e = cudaGraphAddKernelNode(&tn, graph, deps, ndeps, &tp)) != cudaSuccess) break;
    cudaGraphNodeParams ip = {};
    ip.type = cudaGraphNodeTypeConditional;
    ip.conditional.handle = th;
    ip.conditional.type = cudaGraphCondTypeIf;
    ip.conditional.size = 1;
    if ((e = cudaGraphAddNode(out, graph, &tn, 1, &ip)) != cudaSuccess) break;
    graph = ip.conditional.phGraph_out[0];  // the multi-CTA repair below goes into the IF body
    deps = nullptr;
    ndeps = 0;
    cudaGraphConditionalHandle wh;
    if ((e = cudaGraphConditionalHandleCreate(&wh, graph, 1, cudaGraphCondAssignDefault)) != cudaSuccess) break;
    cudaGraphNodeParams wp = {};
    wp.type = cudaGraphNodeTypeConditional;
    wp.conditional.handle = wh;
    wp.conditional.type = cudaGraphCondTypeWhile;
    wp.conditional.size = 1;
    cudaGraphNode_t wnode;
    if ((e = cudaGraphAddNode(&wnode, graph, deps, ndeps, &wp)) != cudaSuccess) break;
    cudaGraph_t body = wp.conditional.phGraph_out[0];
    if ((e = cudaStreamBeginCaptureToGraph(g.cap_stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed)) !=
        cudaSuccess)
      break;
    for (int half = 0; half < 2; half++) {
      unsigned long long *fin_n = &g.d.ctl[C_QN0 + half], *fout_n = &g.d.ctl[C_QN0 + (half ^ 1)];
      k_inv_begin<<<1, 1, 0, g.cap_stream>>>(g.d, fin_n, fout_n, big);
      k_rescue<A, W><<<gridw, TPB, 0, g.cap_stream>>>(g.d, g.q[half], fin_n, limit);
      k_rescue_heavy<A, W><<<gridw, TPB, 0, g.cap_stream>>>(g.d, limit);
      k_expand<A, W><<<gridw, TPB, 0, g.cap_stream>>>(g.d, g.q[half], fin_n, g.tree, g.q[half ^ 1], fout_n);
      k_expand_heavy<A, W><<<gridw, TPB, 0, g.cap_stream>>>(g.d, g.q[half ^ 1], fout_n);
    }
    k_inv_cond<<<1, 1, 0, g.cap_stream>>>(g.d, &g.d.ctl[C_QN0], (uint64_t)g.V + 2, wh, 1);
    if ((e = cudaStreamEndCapture(g.cap_stream, &body)) != cudaSuccess) break;
    // k_reset -> k_pull -> k_copy_frontier after the loop
    unsigned long long *tree_n = &g.d.ctl[C_TREEN], *q0_n = &g.d.ctl[C_QN0];
    const uint32_t *tree = g.tree;
    void *ra[] = {(void *)&g.d, (void *)&tree, (void *)&tree_n, (void *)&mst};
    void *ca[] = {(void *)&g.d, (void *)&tree, (void *)&tree_n, (void *)&q0, (void *)&q0_n};
    cudaKernelNodeParams kp = {};
    kp.gridDim = dim3(gridw);
    kp.blockDim = dim3(TPB);
    kp.func = (void *)k_reset<A>;
    kp.kernelParams = ra;
    cudaGraphNode_t n1, n2;
    if ((e = cudaGraphAddKernelNode(&n1, graph, &wnode, 1, &kp)) != cudaSuccess) break;
    kp.func = (void *)k_pull<A, W>;
    if ((e = cudaGraphAddKernelNode(&n2, graph, &n1, 1, &kp)) != cudaSuccess) break;
    void *ha[] = {(void *)&g.d, (void *)&mst};
    kp.func = (void *)k_pull_heavy<A, W>;
    kp.kernelParams = ha;
    cudaGraphNode_t n2h;
    if ((e = cudaGraphAddKernelNode(&n2h, graph, &n2, 1, &kp)) != cudaSuccess) break;
    kp.func = (void *)k_copy_frontier;
    kp.gridDim = dim3(g.num_sms * 4);
    kp.kernelParams = ca;
    cudaGraphNode_t n3;
    e = cudaGraphAddKernelNode(&n3, graph, &n2h, 1, &kp);
  } while (0);
  if (e != cudaSuccess) return cuda_fail(e, "building the deletion-repair graph");
  return RG_OK;
}

// Cached standalone level loop per (algorithm, weighting, variant), rebuilt
// when the pool is relocated by a compaction or an option changes.
template <int A, bool W>
int loop_exec(Graph &g, bool build_variant, cudaGraphExec_t *out) {
  const LevelCfg cfg = level_cfg(g, A, build_variant);
  LoopGraph &slot = g.loops[(A * 2 + (W ? 1 : 0)) * 2 + (build_variant ? 1 : 0)];
  // (the launches of grouped pull levels hold slice bounds of the current copy)
  const uint64_t key = cfg_key(cfg) ^ splitmix64(g.layout_version) ^ splitmix64(build_variant ? g.sell_epoch + 5 : 0) ^
                       splitmix64(build_variant && cfg.pull_groups > 2 ? g.pull_version + 23 : 0);
  if (slot.exec && slot.key == key) {
    *out = slot.exec;
    return RG_OK;
  }
  if (slot.exec) {
    cudaGraphExecDestroy(slot.exec);
    slot.exec = nullptr;
  }
  cudaGraph_t graph;
  RG_CUDA(cudaGraphCreate(&graph, 0));
  cudaGraphNode_t node;
  int rc = add_level_loop<A, W>(g, graph, nullptr, 0, cfg, &node);
  if (!rc) {
    cudaError_t e = cudaGraphInstantiate(&slot.exec, graph, 0);
    if (e != cudaSuccess) {
      slot.exec = nullptr;
      rc = cuda_fail(e, "instantiating the level-loop graph");
    }
  }
  cudaGraphDestroy(graph);
  if (rc) return rc;
  slot.key = key;
  *out = slot.exec;
  return RG_OK;
}

// Push levels to a fixpoint from the frontier in queue 0 (do_update_tree_add,
// core/graph.hpp:1013-1111; build_tree :898-983).  Enqueues one graph launch;
// with profiling on, the host runs the same kernels level by level (syncing)
// so each level can be timed.
template <int A, bool W>
int push_levels(Graph &g, bool build_variant) {
  if (build_variant && pull_on(g, A)) {
    int rc = prepare_pull(g);
    if (rc) return rc;
  }
  if (!g.profiling) {
    cudaGraphExec_t exec;
    int rc = loop_exec<A, W>(g, build_variant, &exec);
    if (rc) return rc;
    RG_CUDA(cudaGraphLaunch(exec, g.stream));
    return RG_OK;
  }
  const LevelCfg cfg = level_cfg(g, A, build_variant);
  int rc = read_ctl(g);
  if (rc) return rc;
  for (int half = 0; g.h_ctl[C_QN0 + half]; half ^= 1) {
    if (g.h_ctl[C_LEVEL] >= max_levels_of(g)) {
      set_error("push levels did not converge");
      return RG_ETIMEOUT;
    }
    RG_CUDA(cudaEventRecord(g.pev[0], g.stream));
    count_launch(g);
    k_level_begin<<<1, LVB_TPB, 0, g.stream>>>(g.d, g.q[half], &g.d.ctl[C_QN0 + half], &g.d.ctl[C_QN0 + (half ^ 1)],
                                                cfg, 0, cudaGraphConditionalHandle{});
    if ((rc = read_ctl(g))) return rc;
    const unsigned long long mode = g.h_ctl[C_MODE];
    count_launch(g, mode_launches(mode));
    if ((rc = enqueue_mode<A, W>(g, g.stream, half, mode))) return rc;
    RG_CUDA(cudaEventRecord(g.pev[1], g.stream));
    if ((rc = read_ctl(g))) return rc;
    float ms = 0.f;
    RG_CUDA(cudaEventElapsedTime(&ms, g.pev[0], g.pev[1]));
    g.prof_ms += ms;
    g.prof_launches += 1;
    g.st_level_ms.push_back(ms);
  }
  return RG_OK;
}


// Cached standalone deletion repair (the push loop follows as its own graph).
template <int A, bool W>
int del_exec(Graph &g, bool fused, cudaGraphExec_t *out) {
  LoopGraph &slot = g.dels[(A * 2 + (W ? 1 : 0)) * 2 + (fused ? 1 : 0)];
  const uint64_t key = (g.layout_version << 40) ^ recompute_threshold(g);
  if (slot.exec && slot.key == key) {
    *out = slot.exec;
    return RG_OK;
  }
  if (slot.exec) {
    cudaGraphExecDestroy(slot.exec);
    slot.exec = nullptr;
  }
  cudaGraph_t graph;
  RG_CUDA(cudaGraphCreate(&graph, 0));
  cudaGraphNode_t last;
  int rc = add_del_repair<A, W>(g, graph, nullptr, 0, &last, fused);
  if (!rc) {
    cudaError_t e = cudaGraphInstantiate(&slot.exec, graph, 0);
    if (e != cudaSuccess) {
      slot.exec = nullptr;
      rc = cuda_fail(e, "instantiating the deletion-repair graph");
    }
  }
  cudaGraphDestroy(graph);
  if (rc) return rc;
  slot.key = key;
  *out = slot.exec;
  return RG_OK;
}

// The deletion repair of add_del_repair launched kernel by kernel from the
// host (profile mode): the same kernels in the same order, with the IF and
// WHILE decisions read back through C_HOSTCOND, so that every kernel is a
// plain launch a profiler lists.
template <int A, bool W>
int del_repair_stepped(Graph &g) {
  const uint64_t big = recompute_threshold(g);
  const uint64_t limit = (uint64_t)((double)g.V * 0.1);  // has_parents guard, core/graph.hpp:1900
  const uint32_t mst = mod_stamp(g);
  const int gridw = g.num_sms * 16;
  const uint64_t max_iter = (uint64_t)g.V + 2;
  count_launch(g);
  k_del_tiny<A, W><<<1, DT_TPB, 0, g.stream>>>(g.d, g.q[0], g.q[1], g.tree, limit, big, max_iter, mst,
                                               cudaGraphConditionalHandle{}, 0);
  RG_CUDA(cudaGetLastError());
  int rc = read_ctl(g);
  if (rc) return rc;
  if (!g.h_ctl[C_HOSTCOND]) return RG_OK;
  for (uint64_t it = 0;; it++) {
    if (it > max_iter) {
      set_error("deletion repair did not converge");
      return RG_ETIMEOUT;
    }
    for (int half = 0; half < 2; half++) {
      unsigned long long *fin_n = &g.d.ctl[C_QN0 + half], *fout_n = &g.d.ctl[C_QN0 + (half ^ 1)];
      count_launch(g, 5);
      k_inv_begin<<<1, 1, 0, g.stream>>>(g.d, fin_n, fout_n, big);
      k_rescue<A, W><<<gridw, TPB, 0, g.stream>>>(g.d, g.q[half], fin_n, limit);
      k_rescue_heavy<A, W><<<gridw, TPB, 0, g.stream>>>(g.d, limit);
      k_expand<A, W><<<gridw, TPB, 0, g.stream>>>(g.d, g.q[half], fin_n, g.tree, g.q[half ^ 1], fout_n);
      k_expand_heavy<A, W><<<gridw, TPB, 0, g.stream>>>(g.d, g.q[half ^ 1], fout_n);
    }
    count_launch(g);
    k_inv_cond<<<1, 1, 0, g.stream>>>(g.d, &g.d.ctl[C_QN0], max_iter, cudaGraphConditionalHandle{}, 0);
    RG_CUDA(cudaGetLastError());
    if ((rc = read_ctl(g))) return rc;
    if (!g.h_ctl[C_HOSTCOND]) break;
  }
  count_launch(g, 4);
  k_reset<A><<<gridw, TPB, 0, g.stream>>>(g.d, g.tree, &g.d.ctl[C_TREEN], mst);
  k_pull<A, W><<<gridw, TPB, 0, g.stream>>>(g.d, g.tree, &g.d.ctl[C_TREEN], mst);
  k_pull_heavy<A, W><<<gridw, TPB, 0, g.stream>>>(g.d, mst);
  k_copy_frontier<<<g.num_sms * 4, TPB, 0, g.stream>>>(g.d, g.tree, &g.d.ctl[C_TREEN], g.q[0], &g.d.ctl[C_QN0]);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

// The engine runs every tree call but those of served graphs (which run without
// cluster levels, RG_OPT_CLUSTER_EDGES 0) and host-stepped ones.
bool engine_on(const Graph &g) { return g.eng_ctas && g.cluster_edges && !g.profiling; }

// One engine launch (see k_engine): build from scratch, or the levels of a
// repair whose frontier is in queue 0, after the deletion repair when `del`.
// It ends with the control block in the host's copy.
// n_edges: the edges of the repair's batch; ~0 for one that one CTA has run already
// and that outgrew it (an edge that joins the root to an RMAT-18 graph: 750 us on all
// SMs, 783 begun on half).
template <int A, bool W>
int engine_launch(Graph &g, bool build, bool del, uint64_t root, uint64_t n_edges) {
  EngineArgs a = {};
  a.cfg = level_cfg(g, A, build);
  if (a.cfg.allow_pull) {
    int rc = prepare_pull(g);
    if (rc) return rc;
    a.ent = g.sell_ent;
    a.off = g.sell_off;
    a.row_id = g.sell_row;
    a.hubs = pull_hubs(g);
    a.plan = g.sell_plan;
  }
  a.q[0] = g.q[0];
  a.q[1] = g.q[1];
  a.tree = g.tree;
  a.task = g.hubq;  // (at least a task for every CHUNK slots of a pool)
  a.P = g.lb_P;
  a.tot = reinterpret_cast<unsigned long long *>(g.lb_sums);
  a.bar = g.eng_bar;
  a.ctl_host = g.h_ctl_dev;
  a.root = root;
  a.limit = (uint64_t)((double)g.V * 0.1);  // has_parents guard, core/graph.hpp:1900
  a.big = recompute_threshold(g);
  a.max_iter = (uint64_t)g.V + 2;
  a.mst = mod_stamp(g);
  a.polls = g.wait_polls;
  const int ctas = !build && n_edges <= ENG_HALF_EDGES ? (g.eng_ctas + 1) / 2 : g.eng_ctas;
  a.push_slots = g.push_slots;
  a.half_vertices = ctas < g.eng_ctas ? g.half_vertices : ~0ull;
  a.half_slots = ctas < g.eng_ctas ? 32 * g.half_vertices : ~0ull;
  a.build = build ? 1 : 0;
  a.del = del ? 1 : 0;
  g.h_ctl[C_KLAUNCH] = CTL_PENDING;
  count_launch(g);
  void *args[] = {(void *)&g.d, (void *)&a};
  RG_CUDA(cudaLaunchCooperativeKernel((const void *)k_engine<A, W>, dim3((unsigned)ctas), dim3(ENG_TPB), args,
                                      sizeof(EngShared), g.stream));
  g.ctl_on_host = true;
  return RG_OK;
}

// The levels that the engine left, to their end.
template <int A, bool W>
int engine_left(Graph &g, bool build) {
  while (g.h_ctl[C_ELEFT] && !g.h_ctl[C_ERR]) {
    int rc = RG_OK;
    if (g.h_ctl[C_ELEFT] == ELEFT_PUSH) {
      cudaGraphExec_t exec;
      if ((rc = loop_exec<A, W>(g, build, &exec))) return rc;
      RG_CUDA(cudaGraphLaunch(exec, g.stream));
    } else {
      rc = engine_launch<A, W>(g, build, g.h_ctl[C_ELEFT] == ELEFT_REPAIR, 0, ~0ull);
    }
    if (rc || (rc = read_ctl(g))) return rc;
  }
  return RG_OK;
}

template <int A, bool W>
int build_enqueue(Graph &g, uint64_t root) {
  int rc = guard_counters(g);
  if (rc) return rc;
  if (engine_on(g)) return engine_launch<A, W>(g, true, false, root, 0);
  count_launch(g, 2);
  k_prologue<<<1, 1, 0, g.stream>>>(g.d, 0ull);
  k_init<A><<<g.num_sms * 16, TPB, 0, g.stream>>>(g.d, root, g.q[0]);
  RG_CUDA(cudaGetLastError());
  return push_levels<A, W>(g, true);
}

template <int A, bool W>
int add_enqueue(Graph &g, uint64_t n_edges, int directed, bool from_cands) {
  int rc = guard_counters(g);
  if (rc) return rc;
  count_launch(g, 2);
  k_prologue<<<1, 1, 0, g.stream>>>(g.d, 0ull);
  k_seed_add<A><<<grid_warps(g, (n_edges + 31) / 32), TPB, 0, g.stream>>>(
      g.d, op_src(g), op_dst(g), op_w(g), from_cands ? op_cand(g) : nullptr, &g.d.ctl[C_CANDN], n_edges, directed,
      g.q[0], &g.d.ctl[C_QN0], mod_stamp(g));
  RG_CUDA(cudaGetLastError());
  if (engine_on(g)) return engine_launch<A, W>(g, false, false, 0, n_edges);
  return push_levels<A, W>(g, false);
}

template <int A, bool W>
int del_enqueue(Graph &g, uint64_t n_edges, int directed, bool from_cands) {
  int rc = guard_counters(g);
  if (rc) return rc;
  if (++g.inv_epoch >= 0x7FFFFFFFu) {
    RG_CUDA(cudaMemsetAsync(g.d.inv, 0, (size_t)g.V * 4, g.stream));
    RG_CUDA(cudaMemsetAsync(g.d.chk, 0, (size_t)g.V * 4, g.stream));
    g.inv_epoch = 1;
  }
  const unsigned long long tag = 2ull * g.inv_epoch;  // tag: invalidated; tag+1: rescued
  count_launch(g, 2);
  k_prologue<<<1, 1, 0, g.stream>>>(g.d, tag);
  k_seed_del<<<grid_warps(g, (n_edges + 31) / 32), TPB, 0, g.stream>>>(
      g.d, op_src(g), op_dst(g), op_w(g), from_cands ? op_cand(g) : nullptr, &g.d.ctl[C_CANDN], n_edges, directed,
      g.q[0], &g.d.ctl[C_QN0]);
  RG_CUDA(cudaGetLastError());
  if (engine_on(g)) return engine_launch<A, W>(g, false, true, 0, n_edges);
  if (g.profiling) {
    rc = del_repair_stepped<A, W>(g);
  } else {
    cudaGraphExec_t exec;
    if ((rc = del_exec<A, W>(g, false, &exec))) return rc;
    RG_CUDA(cudaGraphLaunch(exec, g.stream));
  }
  if (rc) return rc;
  return push_levels<A, W>(g, false);
}

// After the stream has been synchronised and h_ctl read: errors, statistics
// and the full-recompute fallback of a deletion repair.
template <int A, bool W>
int after_sync(Graph &g, int what) {
  if (g.h_ctl[C_ERR]) {
    int code = (int)g.h_ctl[C_ERR];
    set_error(code == RG_ETIMEOUT ? "push levels did not converge" : "device error in tree update");
    if (code == RG_ETIMEOUT) engine_reset(g);
    cudaMemsetAsync(&g.d.ctl[C_ERR], 0, 8, g.stream);
    return code;
  }
  if (g.h_ctl[C_ELEFT]) {
    const int rc = engine_left<A, W>(g, what == 0);
    return rc ? rc : after_sync<A, W>(g, what);
  }
  g.launches += g.h_ctl[C_KLAUNCH];  // kernels run inside graphs, counted on the device
  g.st_levels = g.h_ctl[C_LEVEL];
  if (what == 2) {
    g.st_invalidated = g.h_ctl[C_TREEN];
    if (g.h_ctl[C_RECOMPUTE]) {
      g.st_recomputes++;
      RG_CUDA(cudaMemsetAsync(g.d.inv, 0, (size_t)g.V * 4, g.stream));
      RG_CUDA(cudaMemsetAsync(g.d.chk, 0, (size_t)g.V * 4, g.stream));
      g.inv_epoch = 0;
      int rc = build_enqueue<A, W>(g, g.root);
      if (!rc) rc = read_ctl(g);
      if (!rc) rc = after_sync<A, W>(g, 0);
      return rc;
    }
  }
  return RG_OK;
}

template <int A, bool W>
int run_what(Graph &g, int what, uint64_t a, int directed, bool from_cands, int phase) {
  if (phase == 1) return after_sync<A, W>(g, what);
  if (what == 0) return build_enqueue<A, W>(g, a);
  if (what == 1) return add_enqueue<A, W>(g, a, directed, from_cands);
  return del_enqueue<A, W>(g, a, directed, from_cands);
}

template <int A>
int dispatch_w(Graph &g, int what, uint64_t a, int directed, bool from_cands, int phase) {
  if (g.weighted) return run_what<A, true>(g, what, a, directed, from_cands, phase);
  return run_what<A, false>(g, what, a, directed, from_cands, phase);
}

// phase 0: enqueue the call's device work; phase 1: finish it after a sync.
int dispatch(Graph &g, int algo, int what, uint64_t a, int directed, bool from_cands, int phase) {
  switch (algo) {
    case RG_BFS: return dispatch_w<RG_BFS>(g, what, a, directed, from_cands, phase);
    case RG_SSSP: return dispatch_w<RG_SSSP>(g, what, a, directed, from_cands, phase);
    case RG_SSWP: return dispatch_w<RG_SSWP>(g, what, a, directed, from_cands, phase);
    case RG_WCC: return dispatch_w<RG_WCC>(g, what, a, directed, from_cands, phase);
  }
  set_error("unknown algorithm");
  return RG_EINVAL;
}

}  // namespace

// CTAs of the cluster-level kernel: 16 where this GPU schedules a cluster of
// sixteen 1024-thread CTAs, else the portable 8; 0 (cluster levels off) when
// neither can run.
template <int A, bool W>
void cluster_allow(cudaError_t &e) {
  cudaError_t x = cudaFuncSetAttribute(k_push_cluster<A, W>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (x != cudaSuccess) e = x;
}

static void cluster_setup(Graph &g) {
  cudaError_t e = cudaSuccess;
  cluster_allow<RG_BFS, false>(e);
  cluster_allow<RG_BFS, true>(e);
  cluster_allow<RG_SSSP, false>(e);
  cluster_allow<RG_SSSP, true>(e);
  cluster_allow<RG_SSWP, false>(e);
  cluster_allow<RG_SSWP, true>(e);
  cluster_allow<RG_WCC, false>(e);
  cluster_allow<RG_WCC, true>(e);
  g.cl_ctas = 0;
  for (int n : {CL_MAX_CTAS, 8}) {
    if (e != cudaSuccess && n > 8) continue;  // without the attribute only the portable size
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)n);
    lc.blockDim = dim3(CL_TPB);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)n;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, k_push_cluster<RG_SSSP, true>, &lc) == cudaSuccess && clusters > 0) {
      g.cl_ctas = n;
      break;
    }
  }
  cudaGetLastError();
}

template <int A, bool W>
static bool engine_fits(const Graph &g) {
  int n = 0;
  return cudaFuncSetAttribute(k_engine<A, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(EngShared)) ==
             cudaSuccess &&
         cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_engine<A, W>, ENG_TPB, sizeof(EngShared)) == cudaSuccess &&
         n > 0;
}

// CTAs of the engine: one per SM where the GPU launches cooperatively.
static void engine_setup(Graph &g) {
  int coop = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, g.device);
  const bool fits = coop && engine_fits<RG_BFS, false>(g) && engine_fits<RG_BFS, true>(g) &&
                    engine_fits<RG_SSSP, false>(g) && engine_fits<RG_SSSP, true>(g) &&
                    engine_fits<RG_SSWP, false>(g) && engine_fits<RG_SSWP, true>(g) &&
                    engine_fits<RG_WCC, false>(g) && engine_fits<RG_WCC, true>(g);
  g.eng_ctas = fits ? std::min(g.num_sms, ENG_MAX_CTAS) : 0;
  cudaGetLastError();
}

void engine_reset(Graph &g) {
  // a barrier left half counted, stamps past the one in the control block, hubs'
  // best pieces that no pull_hub_fix took
  cudaMemsetAsync(g.eng_bar, 0, EB_WORDS * 8, g.stream);
  cudaMemsetAsync(g.d.stamp, 0, g.V * 4 + 4, g.stream);
  if (g.sell_hub_best) cudaMemsetAsync(g.sell_hub_best, 0xff, g.sell_hub_cap * 8, g.stream);
}

int tree_alloc(Graph &g) {
  uint64_t V = g.V;
  cluster_setup(g);
  engine_setup(g);
  auto alloc = [&](void **p, size_t bytes, const char *what) -> int {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {
      cudaGetLastError();
      set_error(std::string("device allocation failed: ") + what);
      return RG_ENOMEM_HBM;
    }
    g.bytes += bytes;
    return RG_OK;
  };
  int rc;
  if ((rc = alloc((void **)&g.d.lab, V * 16 + 16, "labels"))) return rc;
  if ((rc = alloc((void **)&g.d.val32, V * 4 + 4, "label value mirror"))) return rc;
  RG_CUDA(cudaMemset(g.d.val32, 0, V * 4 + 4));
  if ((rc = alloc((void **)&g.d.stamp, V * 4 + 4, "frontier stamps"))) return rc;
  if ((rc = alloc((void **)&g.d.inv, V * 4 + 4, "invalidation tags"))) return rc;
  if ((rc = alloc((void **)&g.d.chk, V * 4 + 4, "clear-chain marks"))) return rc;
  // at most (edge slots / HEAVY_DEG) vertices have a longer list
  g.d.heavy_cap = std::max(g.d.out.pool_cap, g.d.in.pool_cap) / HEAVY_DEG + 1024;
  if ((rc = alloc((void **)&g.d.heavy, 3 * g.d.heavy_cap * 4, "heavy-vertex lists"))) return rc;
  if ((rc = alloc((void **)&g.d.modstamp, V * 4 + 4, "modified stamps"))) return rc;
  if ((rc = alloc((void **)&g.d.modq, V * 4 + 4, "modified list"))) return rc;
  if ((rc = alloc((void **)&g.q[0], V * 4 + 4, "frontier"))) return rc;
  if ((rc = alloc((void **)&g.q[1], V * 4 + 4, "frontier"))) return rc;
  if ((rc = alloc((void **)&g.tree, V * 4 + 4, "reset set"))) return rc;
  if ((rc = alloc((void **)&g.scratch64, V * 8 + 8, "scratch"))) return rc;
  g.hubq_cap = g.d.out.pool_cap / CHUNK + V / HUB + 1024;
  if ((rc = alloc((void **)&g.hubq, g.hubq_cap * 8, "hub tasks"))) return rc;
  if ((rc = alloc((void **)&g.lb_P, V * 8 + 16, "frontier degree prefix"))) return rc;
  if ((rc = alloc((void **)&g.act, V * 4 + 4, "dense-level activity"))) return rc;
  if ((rc = alloc((void **)&g.lb_sums, SC_BLOCKS * 8, "scan block sums"))) return rc;
  if ((rc = alloc((void **)&g.eng_bar, EB_WORDS * 8, "engine barrier"))) return rc;
  RG_CUDA(cudaMemset(g.eng_bar, 0, EB_WORDS * 8));
  if ((rc = alloc((void **)&g.sell_plan, sizeof(SellPlan), "pull plan"))) return rc;
  RG_CUDA(cudaHostAlloc(&g.sell_plan_host, sizeof(SellPlan), cudaHostAllocDefault));
  RG_CUDA(cudaMemset(g.act, 0, V * 4 + 4));
  if ((rc = alloc((void **)&g.lb_tile, (g.d.out.pool_cap / LB_TILE + 4) * 4, "tile partition"))) return rc;
  g.cub_tmp_bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, g.cub_tmp_bytes, g.scratch64, g.lb_P, V + 1);
  if ((rc = alloc(&g.cub_tmp, g.cub_tmp_bytes + 256, "scan scratch"))) return rc;
  if ((rc = alloc((void **)&g.d.ctl, sizeof(unsigned long long) * C_COUNT, "control block"))) return rc;
  RG_CUDA(cudaMemset(g.d.ctl, 0, sizeof(unsigned long long) * C_COUNT));
  {
    unsigned long long one = 1;
    RG_CUDA(cudaMemcpy(&g.d.ctl[C_MODEPOCH], &one, 8, cudaMemcpyHostToDevice));
  }
  // frontier sizes, then the levels' start stamps (one more: the end of the last)
  if ((rc = alloc((void **)&g.d.trace, (2 * TRACE_CAP + 1) * 8, "level trace"))) return rc;
  if ((rc = alloc((void **)&g.ptrace_buf, RG_PHASE_SLOTS * 8, "phase trace"))) return rc;
  RG_CUDA(cudaMemset(g.ptrace_buf, 0, RG_PHASE_SLOTS * 8));
  g.d.ptrace = g.phase_trace ? g.ptrace_buf : nullptr;
  RG_CUDA(cudaMemset(g.d.stamp, 0, V * 4 + 4));
  RG_CUDA(cudaMemset(g.d.inv, 0, V * 4 + 4));
  RG_CUDA(cudaMemset(g.d.chk, 0, V * 4 + 4));
  RG_CUDA(cudaMemset(g.d.modstamp, 0, V * 4 + 4));
  // labels start as "no parent", value 0 until build_tree (alloc_vertex_tree_array, :255-262)
  RG_CUDA(cudaMemset(g.d.lab, 0, V * 16 + 16));
  return RG_OK;
}

static void reset_stats(Graph &g) {
  g.st_levels = g.st_invalidated = g.st_recomputes = 0;
  g.st_level_ms.clear();
}

int tree_enqueue(Graph &g, int what, uint64_t n_edges, int directed, bool from_cands) {
  reset_stats(g);
  return dispatch(g, g.algo, what, n_edges, directed, from_cands, 0);
}

int tree_after_sync(Graph &g, int what, uint64_t *total) {
  int rc = dispatch(g, g.algo, what, 0, 1, false, 1);
  if (rc) return rc;
  if (total) *total = g.h_ctl[C_RESULT];
  return RG_OK;
}

int tree_build(Graph &g, int algo, uint64_t root, uint64_t *total) {
  reset_stats(g);
  g.algo = algo;
  g.root = root;
  int rc = dispatch(g, algo, 0, root, 1, false, 0);
  if (!rc) rc = read_ctl(g);
  if (!rc) rc = tree_after_sync(g, 0, total);
  return rc;
}

int tree_add(Graph &g, uint64_t n_edges, int directed, bool from_cands, uint64_t *total) {
  int rc = tree_enqueue(g, 1, n_edges, directed, from_cands);
  if (!rc) rc = read_ctl(g);
  if (!rc) rc = tree_after_sync(g, 1, total);
  return rc;
}

int tree_del(Graph &g, uint64_t n_edges, int directed, bool from_cands, uint64_t *total) {
  int rc = tree_enqueue(g, 2, n_edges, directed, from_cands);
  if (!rc) rc = read_ctl(g);
  if (!rc) rc = tree_after_sync(g, 2, total);
  return rc;
}

FusedRepair fused_repair(const Graph &g, const LevelCfg &cfg) {
  FusedRepair fr = {};
  fr.q1 = g.q[1];
  fr.tree = g.tree;
  fr.limit = (uint64_t)((double)g.V * 0.1);  // has_parents guard, core/graph.hpp:1900
  fr.big = recompute_threshold(g);
  fr.max_iter = (uint64_t)g.V + 2;
  fr.max_levels = cfg.max_levels;
  fr.tiny_edges = cfg.tiny_edges;
  return fr;
}

// The fused kernel for one batch as a graph node after `deps`: k_apply_small
// with the header at hdr_off of the staging buffer (second: the delete batch
// of an insert+delete submission, whose edges start at apply_data2_off()).
template <int A, bool W>
int add_apply_kernel(Graph &g, cudaGraph_t graph, const cudaGraphNode_t *deps, size_t ndeps, bool add, int directed,
                     uint64_t hdr_off, int second, const LevelCfg &cfg, cudaGraphNode_t *out) {
  sdev::OpView ops = sdev::op_view(g);
  char *base = reinterpret_cast<char *>(g.stage_host_dev);
  const ApplyHdr *hdr = reinterpret_cast<const ApplyHdr *>(base + hdr_off);
  const char *data = base + APPLY_DATA_OFF + (second ? apply_data2_off() : 0);
  uint64_t *old_host = reinterpret_cast<uint64_t *>(base + apply_old_off());
  uint4 *scratch = reinterpret_cast<uint4 *>(g.stage_dev);
  uint32_t *cand = op_cand(g);
  int a_add = add ? 1 : 0, a_dir = directed ? 1 : 0, a_second = second;
  uint32_t *q0 = g.q[0];
  uint32_t mst = mod_stamp(g);
  FusedRepair fr = fused_repair(g, cfg);
  unsigned long long *ctl_host = g.h_ctl_dev;
  void *args[] = {(void *)&g.d,    (void *)&ops, (void *)&hdr, (void *)&data,   (void *)&old_host,
                  (void *)&cand,   (void *)&a_add, (void *)&a_dir, (void *)&q0, (void *)&mst,
                  (void *)&a_second, (void *)&fr, (void *)&scratch, (void *)&ctl_host};
  cudaKernelNodeParams kp = {};
  kp.func = (void *)k_apply_small<A, W>;
  kp.gridDim = dim3(1);
  kp.blockDim = dim3(FS_TPB);
  kp.kernelParams = args;
  cudaError_t e = cudaGraphAddKernelNode(out, graph, deps, ndeps, &kp);
  return e == cudaSuccess ? RG_OK : cuda_fail(e, "building the fused apply graph");
}

uint64_t apply_key(const Graph &g, const LevelCfg &cfg) {
  return splitmix64(g.layout_version) ^ splitmix64((uint64_t)(uintptr_t)g.ops ^ (g.ops_cap << 1)) ^
         splitmix64((uint64_t)(uintptr_t)g.d.ptrace + 17) ^ splitmix64((uint64_t)(uintptr_t)g.h_ctl_dev + 19) ^
         splitmix64((uint64_t)(uintptr_t)g.stage_host_dev + 7) ^ splitmix64((uint64_t)(uintptr_t)g.stage_dev + 13) ^
         cfg_key(cfg) ^ splitmix64(recompute_threshold(g) + 11);
}

// A cached graph: `build` adds its nodes; rebuilt when `key` changes.
template <typename F>
int cached_graph(LoopGraph &slot, uint64_t key, F build, const char *what, cudaGraphExec_t *out) {
  if (slot.exec && slot.key == key) {
    *out = slot.exec;
    return RG_OK;
  }
  if (slot.exec) {
    cudaGraphExecDestroy(slot.exec);
    slot.exec = nullptr;
  }
  cudaGraph_t graph;
  RG_CUDA(cudaGraphCreate(&graph, 0));
  int rc = build(graph);
  if (!rc) {
    cudaError_t e = cudaGraphInstantiate(&slot.exec, graph, 0);
    if (e != cudaSuccess) {
      slot.exec = nullptr;
      rc = cuda_fail(e, what);
    }
  }
  cudaGraphDestroy(graph);
  if (rc) return rc;
  slot.key = key;
  *out = slot.exec;
  return RG_OK;
}

// Insert batch then delete batch: one node, k_apply_mixed (both batches, and
// their repairs while they stay small).
template <int A, bool W>
int mixed_exec(Graph &g, int directed, cudaGraphExec_t *out) {
  const LevelCfg cfg = level_cfg(g, A, false);
  auto build = [&](cudaGraph_t graph) -> int {
    sdev::OpView ops = sdev::op_view(g);
    char *base = reinterpret_cast<char *>(g.stage_host_dev);
    const ApplyHdr *hdr1 = reinterpret_cast<const ApplyHdr *>(base);
    const ApplyHdr *hdr2 = reinterpret_cast<const ApplyHdr *>(base + APPLY_HDR2);
    const char *data1 = base + APPLY_DATA_OFF, *data2 = base + APPLY_DATA_OFF + apply_data2_off();
    uint4 *scr1 = reinterpret_cast<uint4 *>(g.stage_dev);
    uint4 *scr2 = reinterpret_cast<uint4 *>(reinterpret_cast<char *>(g.stage_dev) + apply_data2_off());
    uint32_t *cand = op_cand(g), *q0 = g.q[0];
    int a_dir = directed ? 1 : 0;
    uint32_t mst = mod_stamp(g);
    FusedRepair fr = fused_repair(g, cfg);
    unsigned long long *ctl_host = g.h_ctl_dev;
    void *args[] = {(void *)&g.d,  (void *)&ops,   (void *)&hdr1, (void *)&data1, (void *)&hdr2,
                    (void *)&data2, (void *)&cand, (void *)&a_dir, (void *)&q0,   (void *)&mst,
                    (void *)&fr,   (void *)&scr1,  (void *)&scr2, (void *)&ctl_host};
    cudaKernelNodeParams kp = {};
    kp.func = (void *)k_apply_mixed<A, W>;
    kp.gridDim = dim3(1);
    kp.blockDim = dim3(FS_TPB);
    kp.kernelParams = args;
    cudaGraphNode_t kn;
    cudaError_t e = cudaGraphAddKernelNode(&kn, graph, nullptr, 0, &kp);
    return e == cudaSuccess ? RG_OK : cuda_fail(e, "building the fused insert+delete graph");
  };
  return cached_graph(g.mixes[(A * 2 + (W ? 1 : 0)) * 2 + (directed ? 1 : 0)], apply_key(g, cfg), build,
                      "instantiating the fused insert+delete graph", out);
}

// After k_apply_mixed left the insert batch's level loop: that loop, then the
// delete batch in its own fused kernel (k_apply_small, second batch).
template <int A, bool W>
int rest_exec(Graph &g, int directed, cudaGraphExec_t *out) {
  const LevelCfg cfg = level_cfg(g, A, false);
  auto build = [&](cudaGraph_t graph) -> int {
    cudaGraphNode_t loop, kn;
    int rc = add_level_loop<A, W>(g, graph, nullptr, 0, cfg, &loop);
    if (!rc) rc = add_apply_kernel<A, W>(g, graph, &loop, 1, false, directed, APPLY_HDR2, 1, cfg, &kn);
    return rc;
  };
  return cached_graph(g.rests[(A * 2 + (W ? 1 : 0)) * 2 + (directed ? 1 : 0)], apply_key(g, cfg), build,
                      "instantiating the insert loop + delete batch graph", out);
}

// One batch: one node, k_apply_small.  Its parameters hold the op, staging and
// pool addresses, so it is rebuilt when any of them moves.
template <int A, bool W>
int apply_exec(Graph &g, bool add, int directed, cudaGraphExec_t *out) {
  const LevelCfg cfg = level_cfg(g, A, false);
  auto build = [&](cudaGraph_t graph) -> int {
    cudaGraphNode_t kn;
    return add_apply_kernel<A, W>(g, graph, nullptr, 0, add, directed, 0, 0, cfg, &kn);
  };
  return cached_graph(g.applies[((A * 2 + (W ? 1 : 0)) * 2 + (add ? 1 : 0)) * 2 + (directed ? 1 : 0)],
                      apply_key(g, cfg), build, "instantiating the fused apply graph", out);
}

// What a fused kernel left (C_LEFT in the host's copy of the control block):
// 1 the insert batch's level loop; 2 the delete batch's repair, that is the
// grid-wide deletion repair when the one-CTA repair handed over (k_handover
// reads C_OVER) and then the level loop.  Ends with the control block read
// back.
template <int A, bool W>
int finish_left(Graph &g, unsigned long long left) {
  int rc = RG_OK;
  if (engine_on(g)) {
    rc = engine_launch<A, W>(g, false, left == 2 && g.h_ctl[C_OVER], 0, ~0ull);
    return rc ? rc : read_ctl(g);
  }
  if (left == 2) {
    cudaGraphExec_t de;
    if ((rc = del_exec<A, W>(g, true, &de))) return rc;
    RG_CUDA(cudaGraphLaunch(de, g.stream));
  }
  cudaGraphExec_t le;
  if ((rc = loop_exec<A, W>(g, false, &le))) return rc;
  RG_CUDA(cudaGraphLaunch(le, g.stream));
  return read_ctl(g);
}

// The delete batch of an insert+delete submission in its own kernel, from the
// staging buffer.
template <int A, bool W>
int launch_apply_second(Graph &g, int directed) {
  const LevelCfg cfg = level_cfg(g, A, false);
  char *base = reinterpret_cast<char *>(g.stage_host_dev);
  k_apply_small<A, W><<<1, FS_TPB, 0, g.stream>>>(
      g.d, sdev::op_view(g), reinterpret_cast<const ApplyHdr *>(base + APPLY_HDR2),
      base + APPLY_DATA_OFF + apply_data2_off(), reinterpret_cast<uint64_t *>(base + apply_old_off()), op_cand(g), 0,
      directed ? 1 : 0, g.q[0], mod_stamp(g), 1, fused_repair(g, cfg), reinterpret_cast<uint4 *>(g.stage_dev),
      g.h_ctl_dev);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

// An inline batch from the caller's edges (n <= INLINE_EDGES).
InlineBatch inline_batch(const void *src, uint64_t n, bool pairs, bool want, uint64_t inv_tag) {
  InlineBatch ib;
  ib.n = n;
  ib.pairs = pairs ? 1 : 0;
  ib.want = want ? 1 : 0;
  ib.inv_tag = inv_tag;
  std::memset(ib.words, 0, sizeof(ib.words));
  std::memcpy(ib.words, src, n * (pairs ? 16 : sizeof(rg_edge)));
  return ib;
}

// One batch of at most INLINE_EDGES edges: k_apply_small_inl, launched
// directly with the batch in its parameters.
template <int A, bool W>
int launch_apply_inline(Graph &g, const InlineBatch &ib, bool add, int directed) {
  const LevelCfg cfg = level_cfg(g, A, false);
  uint64_t *old_host = reinterpret_cast<uint64_t *>(reinterpret_cast<char *>(g.stage_host_dev) + apply_old_off());
  k_apply_small_inl<A, W><<<1, FS_TPB, 0, g.stream>>>(g.d, sdev::op_view(g), ib, old_host, op_cand(g), add ? 1 : 0,
                                                      directed ? 1 : 0, g.q[0], mod_stamp(g), fused_repair(g, cfg),
                                                      g.h_ctl_dev);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

// An insert batch and a delete batch of at most INLINE_EDGES edges each:
// k_apply_mixed_inl.
template <int A, bool W>
int launch_mixed_inline(Graph &g, const InlineBatch &ib1, const InlineBatch &ib2, int directed) {
  const LevelCfg cfg = level_cfg(g, A, false);
  k_apply_mixed_inl<A, W><<<1, FS_TPB, 0, g.stream>>>(g.d, sdev::op_view(g), ib1, ib2, op_cand(g), directed ? 1 : 0,
                                                      g.q[0], mod_stamp(g), fused_repair(g, cfg), g.h_ctl_dev);
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

template <int A, bool W>
int apply_small_t(Graph &g, const rg_edge *edges, const uint64_t *pairs, uint64_t n, int directed, bool add,
                  uint64_t *old_num) {
  int rc = storage_reserve(g, 3 * SMALL_EDGES);  // op arrays and staging sized once for the small path
  if (rc) return rc;
  char *st = reinterpret_cast<char *>(g.stage_host);
  ApplyHdr *h = reinterpret_cast<ApplyHdr *>(st);
  std::memcpy(st + APPLY_DATA_OFF, pairs ? (const void *)pairs : (const void *)edges,
              n * (pairs ? 16 : sizeof(rg_edge)));
  h->n = n;
  h->pairs = pairs ? 1 : 0;
  h->want_old = old_num ? 1 : 0;
  h->inv_tag = 0;
  h->data_off = 0;
  g.adj_version++;
  if ((rc = guard_counters(g))) return rc;
  if (!add) {
    if (++g.inv_epoch >= 0x7FFFFFFFu) {
      RG_CUDA(cudaMemsetAsync(g.d.inv, 0, (size_t)g.V * 4, g.stream));
      RG_CUDA(cudaMemsetAsync(g.d.chk, 0, (size_t)g.V * 4, g.stream));
      g.inv_epoch = 1;
    }
    h->inv_tag = 2ull * g.inv_epoch;  // tag: invalidated; tag+1: rescued
  }
  reset_stats(g);
  count_launch(g);
  if (n <= g.inline_max) {
    const InlineBatch ib = inline_batch(pairs ? (const void *)pairs : (const void *)edges, n, pairs != nullptr,
                                        old_num != nullptr, h->inv_tag);
    if ((rc = launch_apply_inline<A, W>(g, ib, add, directed))) return rc;
  } else {
    cudaGraphExec_t exec;
    if ((rc = apply_exec<A, W>(g, add, directed, &exec))) return rc;
    RG_CUDA(cudaGraphLaunch(exec, g.stream));
  }
  RG_CUDA(cudaStreamSynchronize(g.stream));
  const int what = add ? 1 : 2;
  bool replayed = false;
  if (add && g.h_ctl[C_ERR] == RG_ENOSPACE && g.h_ctl[C_AUX] == 1) {
    // growth ran out of pool: compact, then replay from the growth step
    const uint64_t nops = directed ? n : 2 * n;
    rc = storage_recover(g);
    if (!rc) rc = storage_replay(g, n, nops, directed, true);
    if (!rc) rc = dispatch(g, A, what, n, directed, true, 0);
    if (!rc && old_num) rc = storage_copy_old(g, n);
    if (!rc) rc = sync_ctl(g);
    if (rc) return rc;
    replayed = true;
  }
  if ((rc = storage_error(g))) return rc;
  if (!replayed && g.h_ctl[C_LEFT] && (rc = finish_left<A, W>(g, g.h_ctl[C_LEFT]))) return rc;
  if ((rc = after_sync<A, W>(g, what))) return rc;
  if (old_num) std::memcpy(old_num, replayed ? (const void *)storage_old_host(g) : (const void *)(st + apply_old_off()),
                           n * 8);
  return RG_OK;
}

template <int A, bool W>
int apply_add_del_t(Graph &g, const rg_edge *adds, uint64_t n_add, const rg_edge *dels, uint64_t n_del,
                    int directed) {
  int rc = storage_reserve(g, 3 * SMALL_EDGES);
  if (rc) return rc;
  char *st = reinterpret_cast<char *>(g.stage_host);
  ApplyHdr *h1 = reinterpret_cast<ApplyHdr *>(st), *h2 = reinterpret_cast<ApplyHdr *>(st + APPLY_HDR2);
  std::memcpy(st + APPLY_DATA_OFF, adds, n_add * sizeof(rg_edge));
  std::memcpy(st + APPLY_DATA_OFF + apply_data2_off(), dels, n_del * sizeof(rg_edge));
  *h1 = ApplyHdr{n_add, 0, 0, 0, 0};
  *h2 = ApplyHdr{n_del, 0, 0, 0, apply_data2_off()};
  g.adj_version++;
  if ((rc = guard_counters(g))) return rc;
  if (++g.inv_epoch >= 0x7FFFFFFFu) {
    RG_CUDA(cudaMemsetAsync(g.d.inv, 0, (size_t)g.V * 4, g.stream));
    RG_CUDA(cudaMemsetAsync(g.d.chk, 0, (size_t)g.V * 4, g.stream));
    g.inv_epoch = 1;
  }
  h2->inv_tag = 2ull * g.inv_epoch;
  reset_stats(g);
  count_launch(g);
  if (n_add <= g.inline_max && n_del <= g.inline_max) {
    // both batches in the parameters; the staging buffer keeps them too for
    // the graphs that run when the insert batch leaves work
    const InlineBatch ib1 = inline_batch(adds, n_add, false, false, 0);
    const InlineBatch ib2 = inline_batch(dels, n_del, false, false, h2->inv_tag);
    if ((rc = launch_mixed_inline<A, W>(g, ib1, ib2, directed))) return rc;
  } else {
    cudaGraphExec_t exec;
    if ((rc = mixed_exec<A, W>(g, directed, &exec))) return rc;
    RG_CUDA(cudaGraphLaunch(exec, g.stream));
  }
  RG_CUDA(cudaStreamSynchronize(g.stream));
  if (g.h_ctl[C_ERR] == RG_ENOSPACE && g.h_ctl[C_AUX] == 1) {
    // the insert phase ran out of pool during growth (the delete phase did not
    // run): compact, replay the inserts, then apply the deletes on their own
    const uint64_t nops = directed ? n_add : 2 * n_add;
    rc = storage_recover(g);
    if (!rc) rc = storage_replay(g, n_add, nops, directed, true);
    if (!rc) rc = dispatch(g, A, 1, n_add, directed, true, 0);
    if (!rc) rc = sync_ctl(g);
    if (!rc) rc = storage_error(g);
    if (!rc) rc = after_sync<A, W>(g, 1);
    if (rc) return rc;
    return n_del ? apply_small_t<A, W>(g, dels, nullptr, n_del, directed, false, nullptr) : RG_OK;
  }
  if ((rc = storage_error(g))) return rc;
  unsigned long long left = g.h_ctl[C_LEFT];
  if (left == 1) {
    // the insert batch's level loop, then the delete batch in its own kernel
    count_launch(g);
    if (engine_on(g)) {
      if ((rc = engine_launch<A, W>(g, false, false, 0, ~0ull))) return rc;
      g.ctl_on_host = false;  // (the kernel after it writes the host's copy last)
      if ((rc = launch_apply_second<A, W>(g, directed))) return rc;
      RG_CUDA(cudaStreamSynchronize(g.stream));
      if (g.h_ctl[C_ELEFT] && !g.h_ctl[C_ERR]) {
        // the engine left levels of the insert batch: the delete batch waited
        if ((rc = engine_left<A, W>(g, false))) return rc;
        if ((rc = storage_error(g))) return rc;
        count_launch(g);
        if ((rc = launch_apply_second<A, W>(g, directed))) return rc;
      }
    } else {
      cudaGraphExec_t re;
      if ((rc = rest_exec<A, W>(g, directed, &re))) return rc;
      RG_CUDA(cudaGraphLaunch(re, g.stream));
    }
    RG_CUDA(cudaStreamSynchronize(g.stream));
    if ((rc = storage_error(g))) return rc;
    left = g.h_ctl[C_LEFT];
  }
  if (left == 2 && (rc = finish_left<A, W>(g, 2))) return rc;
  return after_sync<A, W>(g, 2);
}

int apply_add_del_small(Graph &g, const rg_edge *adds, uint64_t n_add, const rg_edge *dels, uint64_t n_del,
                        int directed) {
  const bool W = g.weighted != 0;
  switch (g.algo) {
    case RG_BFS: return W ? apply_add_del_t<RG_BFS, true>(g, adds, n_add, dels, n_del, directed)
                          : apply_add_del_t<RG_BFS, false>(g, adds, n_add, dels, n_del, directed);
    case RG_SSSP: return W ? apply_add_del_t<RG_SSSP, true>(g, adds, n_add, dels, n_del, directed)
                           : apply_add_del_t<RG_SSSP, false>(g, adds, n_add, dels, n_del, directed);
    case RG_SSWP: return W ? apply_add_del_t<RG_SSWP, true>(g, adds, n_add, dels, n_del, directed)
                           : apply_add_del_t<RG_SSWP, false>(g, adds, n_add, dels, n_del, directed);
    case RG_WCC: return W ? apply_add_del_t<RG_WCC, true>(g, adds, n_add, dels, n_del, directed)
                          : apply_add_del_t<RG_WCC, false>(g, adds, n_add, dels, n_del, directed);
  }
  set_error("labels were not built (call rg_build_tree first)");
  return RG_ESTATE;
}

int apply_small(Graph &g, const rg_edge *edges, const uint64_t *pairs, uint64_t n, int directed, bool add,
                uint64_t *old_num) {
  const bool W = g.weighted != 0;
  switch (g.algo) {
    case RG_BFS: return W ? apply_small_t<RG_BFS, true>(g, edges, pairs, n, directed, add, old_num)
                          : apply_small_t<RG_BFS, false>(g, edges, pairs, n, directed, add, old_num);
    case RG_SSSP: return W ? apply_small_t<RG_SSSP, true>(g, edges, pairs, n, directed, add, old_num)
                           : apply_small_t<RG_SSSP, false>(g, edges, pairs, n, directed, add, old_num);
    case RG_SSWP: return W ? apply_small_t<RG_SSWP, true>(g, edges, pairs, n, directed, add, old_num)
                           : apply_small_t<RG_SSWP, false>(g, edges, pairs, n, directed, add, old_num);
    case RG_WCC: return W ? apply_small_t<RG_WCC, true>(g, edges, pairs, n, directed, add, old_num)
                          : apply_small_t<RG_WCC, false>(g, edges, pairs, n, directed, add, old_num);
  }
  set_error("labels were not built (call rg_build_tree first)");
  return RG_ESTATE;
}

int tree_classify(Graph &g, uint64_t n, int directed, const uint8_t *is_del_dev, uint8_t *unsafe_dev) {
  int grid = grid_warps(g, (n + 31) / 32);
  count_launch(g);
  switch (g.algo) {
    case RG_BFS: k_classify<RG_BFS><<<grid, TPB, 0, g.stream>>>(g.d, op_src(g), op_dst(g), op_w(g), n, directed, is_del_dev, unsafe_dev); break;
    case RG_SSSP: k_classify<RG_SSSP><<<grid, TPB, 0, g.stream>>>(g.d, op_src(g), op_dst(g), op_w(g), n, directed, is_del_dev, unsafe_dev); break;
    case RG_SSWP: k_classify<RG_SSWP><<<grid, TPB, 0, g.stream>>>(g.d, op_src(g), op_dst(g), op_w(g), n, directed, is_del_dev, unsafe_dev); break;
    default: k_classify<RG_WCC><<<grid, TPB, 0, g.stream>>>(g.d, op_src(g), op_dst(g), op_w(g), n, directed, is_del_dev, unsafe_dev); break;
  }
  RG_CUDA(cudaGetLastError());
  return RG_OK;
}

int tree_labels(Graph &g, uint64_t *val, uint64_t *par, uint64_t *pw) {
  uint64_t *outs[3] = {val, par, pw};
  for (int k = 0; k < 3; k++) {
    if (!outs[k]) continue;
    count_launch(g);
    k_unpack_labels<<<g.num_sms * 8, TPB, 0, g.stream>>>(g.d, k == 0 ? g.scratch64 : nullptr,
                                                          k == 1 ? g.scratch64 : nullptr, k == 2 ? g.scratch64 : nullptr);
    RG_CUDA(cudaGetLastError());
    RG_CUDA(cudaMemcpyAsync(outs[k], g.scratch64, g.V * 8, cudaMemcpyDeviceToHost, g.stream));
  }
  RG_CUDA(cudaStreamSynchronize(g.stream));
  return RG_OK;
}

int tree_checksum(Graph &g, uint64_t *sum) {
  RG_CUDA(cudaMemsetAsync(&g.d.ctl[C_CHECKSUM], 0, 8, g.stream));
  count_launch(g);
  k_checksum<<<g.num_sms * 8, TPB, 0, g.stream>>>(g.d);
  RG_CUDA(cudaGetLastError());
  int rc = read_ctl(g);
  if (rc) return rc;
  *sum = g.h_ctl[C_CHECKSUM];
  return RG_OK;
}

}  // namespace rg
