// Object engine kernels (see engine.hpp). A "group" — one CTA, or a cluster of 4 or 8 CTAs
// for a large object — runs one object's chain as floods of synchronised rounds. A round's frontier
// is a queue of (voxel, value) pairs in the shared memory of the group's CTAs, each CTA taking an
// even share of the whole; a warp takes a frontier voxel, its lanes the 26 neighbours, so that the
// neighbour offsets and step weights are registers and pushes are aggregated by ballot. A pair is
// stale when the voxel's value has moved on since it was queued, so a queue needs no membership
// flags; what does not fit the queue spills to the object's list in HBM, kept unique by a flag.
// The group's counters live in the shared memory of its first CTA (distributed shared memory for a
// cluster, updated with 32-bit atomics only); 64-bit reductions (nearest rail, nearest deferred
// voxel, argmax) keep one copy per CTA, updated with CTA-local atomics and combined across the group
// at barriers. State other threads update with atomics (distances, keys, flags, lists) is always
// read through L2; state that is only written between floods, behind a group barrier (PDRF during a
// railroad flood), is read through L1, where a voxel's 26 neighbours find it again.
#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "common.cuh"
#include "engine.hpp"
#include "runtime.hpp"

namespace bk {
namespace {

namespace cg = cooperative_groups;

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr unsigned long long kMinFarNone = 0x7f8000007f800000ull;
// Invalidation keys (M bits << 32 | source + 1): 0 marks a dead voxel, below every offer. A voxel on
// the waiting list holds its best offer with this bit (a distance's sign bit), which puts it above
// every claim; BK_UNCLAIMED, above every offer, is a voxel at rest.
constexpr unsigned long long kWaits = 1ull << 63;

struct Shared {
  // the object (written by the group's first CTA, copied by the others)
  int obj, begin, count, status;
  int a0, sx, sy, sz;
  // unsigned divisions by sx * sy and sx as multiplications (FastDiv)
  unsigned mxy, mx;
  int pxy, px;
  // group counters (used in the first CTA's copy)
  int spilled[3];  // spilled frontier voxels, a ring like qn
  int far_n[2];    // the two deferred lists' lengths
  int n_touch, n_redo, len;
  unsigned long long rounds;
  // per-CTA copies, combined with Group::min_over / max_over
  int qn[3];  // this CTA's queue, a ring: current = qn[r % 3], next = qn[(r + 1) % 3]
  unsigned long long rb, minfar[2], best;
  unsigned lowest[2], pos;
  // each CTA's own result of a band end
  int flag;
  float T;
  // this CTA's copy of the object's neighbour offsets and step weights
  int off[26];
  float w[26];
  // trace: the object's root, its soma radius (< 0: none) and the loop's step (0 the soma's ball,
  // 1 the parents' field, 2 paths)
  double soma_radius;
  int root, step;
  float rscale, rconst;  // invalidation: reach = rscale * DBF[source] + rconst
  int skipped;           // manual targets from which no rail was reachable (empty paths)
};

__device__ __forceinline__ float inf() { return __uint_as_float(BK_INF_BITS); }

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void unravel3(int i, int sx, int sy, int &x, int &y, int &z) {
  const int sxy = sx * sy;
  z = i / sxy;
  const int r = i - z * sxy;
  y = r / sx;
  x = r - y * sx;
}

// n / d for 0 <= n < 2^31 as n * m >> p with p = 31 + ceil(log2 d) and m = ceil(2^p / d): m exceeds
// 2^p / d by less than 1, so the product exceeds n 2^p / d by less than 2^31 <= 2^p / d.
__device__ __forceinline__ void fast_div(unsigned d, unsigned &m, int &p) {
  p = 31 + (d > 1 ? 32 - __clz(int(d - 1)) : 0);
  m = unsigned(((1ull << p) + d - 1) / d);
}
__device__ __forceinline__ int divided(int n, unsigned m, int p) {
  return int((static_cast<unsigned long long>(unsigned(n)) * m) >> p);
}
// The coordinates of the object's arena-local flat index i.
__device__ __forceinline__ void coordinates(const Shared &sh, int i, int &x, int &y, int &z) {
  z = divided(i, sh.mxy, sh.pxy);
  const int r = i - z * (sh.sx * sh.sy);
  y = divided(r, sh.mx, sh.px);
  x = r - y * sh.sx;
}

// A group of C CTAs working on one object. For C == 1 it is the CTA.
template <int C>
struct Group {
  __device__ static int rank() {
    if constexpr (C == 1) return 0;
    else return int(cg::this_cluster().block_rank());
  }
  __device__ static void sync() {
    if constexpr (C == 1) __syncthreads();
    else cg::this_cluster().sync();
  }
  __device__ static Shared *leader(Shared *own) {
    if constexpr (C == 1) return own;
    else return cg::this_cluster().map_shared_rank(own, 0);
  }
  __device__ static int tid() { return rank() * int(blockDim.x) + int(threadIdx.x); }
  // Least / greatest of the group's copies of a per-CTA field (plain loads; call between barriers).
  __device__ static unsigned long long min_over(unsigned long long *own) {
    if constexpr (C == 1) return *(volatile unsigned long long *)own;
    else {
      unsigned long long r = ~0ull;
      for (int q = 0; q < C; ++q) {
        const unsigned long long v = *(volatile unsigned long long *)cg::this_cluster().map_shared_rank(own, q);
        r = v < r ? v : r;
      }
      return r;
    }
  }
  __device__ static unsigned min_over(unsigned *own) {
    if constexpr (C == 1) return *(volatile unsigned *)own;
    else {
      unsigned r = ~0u;
      for (int q = 0; q < C; ++q) {
        const unsigned v = *(volatile unsigned *)cg::this_cluster().map_shared_rank(own, q);
        r = v < r ? v : r;
      }
      return r;
    }
  }
  __device__ static unsigned long long max_over(unsigned long long *own) {
    if constexpr (C == 1) return *(volatile unsigned long long *)own;
    else {
      unsigned long long r = 0;
      for (int q = 0; q < C; ++q) {
        const unsigned long long v = *(volatile unsigned long long *)cg::this_cluster().map_shared_rank(own, q);
        r = v > r ? v : r;
      }
      return r;
    }
  }
  __device__ static int threads() { return C * int(blockDim.x); }
  __device__ static bool first() { return rank() == 0 && threadIdx.x == 0; }
};

template <class T>
__device__ __forceinline__ T vload(const T *p) { return *(const volatile T *)p; }

// A loop bound, lowered to the test cap when one is set.
__device__ __forceinline__ long long capped(const EngineArgs &a, long long bound) {
  return a.round_limit > 0 && a.round_limit < bound ? a.round_limit : bound;
}

// The queues' (dynamic) shared memory. Floods: two buffers of (voxel, distance bits) pairs. Invalidation:
// two buffers of (voxel, key) pairs and the round's staged records.
// One CTA is resident per SM, so the queues take what leaves L1 its half: 28 KB, which spilled a tenth of the
// large objects' frontiers to HBM, cost 4 % of the 512^3 dense trace (28.5 -> 27.4 ms) and of an arbor's (37.7 ->
// 36.1).
// Those of a CTA of W threads, which shares its SM with kEngineThreads / W - 1 others.
template <int W> constexpr int kQueueBytes = 96 * W;
template <int W> constexpr int kFloodQueue = kQueueBytes<W> / 16;         // pairs per buffer
template <int W> constexpr int kInvalQueue = kQueueBytes<W> / 56 / 2 * 2;  // pairs per buffer, and records
// Frontier voxels a warp has in flight: their loads overlap. Three and four spill registers (512^3 dense trace
// 27.4, 28.4, 29.9 ms with 2, 3 and 4).
constexpr int kPipe = 2;

__device__ __forceinline__ unsigned char *queue_bytes() {
  extern __shared__ __align__(16) unsigned char dynamic_queue[];
  return dynamic_queue;
}

// This CTA's even share [lo, hi) of the entries that the group's CTAs hold in their queues, taken in
// rank order (pre: before lane q's CTA). Every warp computes it; every CTA reads the same counts.
struct Share {
  int lo, hi, total, pre;
};

template <int C>
__device__ __forceinline__ Share share_of(Shared &sh, int slot, int cap) {
  Share s;
  if constexpr (C == 1) {
    s.lo = 0;
    s.hi = s.total = min(vload(&sh.qn[slot]), cap);
    s.pre = 0;
  } else {
    const int lane = threadIdx.x & 31;
    const int n = lane < C ? min(vload(cg::this_cluster().map_shared_rank(&sh.qn[slot], lane)), cap) : 0;
    int sum = n;
#pragma unroll
    for (int off = 1; off < C; off <<= 1) {
      const int o = __shfl_up_sync(kFull, sum, off);
      if (lane >= off) sum += o;
    }
    s.total = __shfl_sync(kFull, sum, C - 1);
    s.pre = sum - n;
    const int r = Group<C>::rank();
    s.lo = s.total * r / C;
    s.hi = s.total * (r + 1) / C;
  }
  return s;
}

// The CTA whose queue holds entry i of the group's, and the entry's place there (i may differ
// between lanes; every lane calls).
template <int C>
__device__ __forceinline__ void locate(const Share &s, int i, int &rank, int &at) {
  rank = 0;
  at = i;
  if constexpr (C > 1) {
#pragma unroll
    for (int q = 1; q < C; ++q) {
      const int p = __shfl_sync(kFull, s.pre, q);
      if (p <= i) { rank = q; at = i - p; }
    }
  }
}

// p of the group's first CTA r's copy.
template <int C, class T>
__device__ __forceinline__ T *of_rank(T *p, int r) {
  if constexpr (C == 1) return p;
  else return cg::this_cluster().map_shared_rank(p, r);
}

__device__ __forceinline__ unsigned below(int lane) { return (1u << lane) - 1u; }

// Appends v of the lanes with p to a list whose length is *count (every lane of the warp calls).
__device__ __forceinline__ void append(bool p, int v, int *list, int *count) {
  const unsigned b = __ballot_sync(kFull, p);
  if (!b) return;
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == 0) base = atomicAdd(count, __popc(b));
  base = __shfl_sync(kFull, base, 0);
  if (p) list[base + __popc(b & below(lane))] = v;
}

// Places in one list for what the lanes of a warp push out of kPipe voxels' neighbourhoods: the pushes'
// ballots, and the list's next place (reserve), handed out voxel by voxel.
struct Places {
  unsigned ballot[kPipe];
  int next;
  __device__ int total() const {
    int n = 0;
#pragma unroll
    for (int j = 0; j < kPipe; ++j) n += __popc(ballot[j]);
    return n;
  }
  __device__ int take(int j) {  // this lane's place for voxel j, if it pushes there
    const int at = next + __popc(ballot[j] & below(threadIdx.x & 31));
    next += __popc(ballot[j]);
    return at;
  }
};

// One counter atomic per list, the three at once, since each is a round trip (to the group's first CTA
// for the lists).
__device__ __forceinline__ void reserve(Places &queued, Places &touched, Places &far, int *queue_n, int *touched_n,
                                        int *far_n) {
  const int lane = threadIdx.x & 31;
  const int nq = queued.total(), nt = touched.total(), nf = far.total();
  const int n = lane == 0 ? nq : lane == 1 ? nt : lane == 2 ? nf : 0;
  int base = 0;
  if (n) base = atomicAdd(lane == 0 ? queue_n : lane == 1 ? touched_n : far_n, n);
  queued.next = __shfl_sync(kFull, base, 0);
  touched.next = __shfl_sync(kFull, base, 1);
  far.next = __shfl_sync(kFull, base, 2);
}

// A place in this CTA's next queue for each lane with p (at or past the queue's end: spill).
__device__ __forceinline__ int queue_place(Shared &sh, bool p, unsigned b, int slot) {
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == 0) base = atomicAdd(&sh.qn[slot], __popc(b));
  base = __shfl_sync(kFull, base, 0);
  return base + __popc(b & below(lane));
}

// A voxel that found no place in a queue goes to the round's spill list unless `bit` says it is there.
__device__ __forceinline__ void spill(const EngineArgs &a, int v, unsigned bit, int *list, int *count) {
  if (!(atomicOr(a.flags + v, bit) & bit)) list[atomicAdd(count, 1)] = v;
}
// The flag of the spill list that round r reads: two, so that round r clears its own while it sets
// the other for the round after.
__device__ __forceinline__ unsigned spill_bit(int r) { return (r & 1) ? kSpillOdd : kSpillEven; }

// Queues (v, d) of the lanes with p for round r + 1 of a flood.
template <int W>
__device__ __forceinline__ void queue_flood(const EngineArgs &a, Shared &sh, Shared *L, bool p, int v, unsigned d, int r,
                                            int *spill_list) {
  const unsigned b = __ballot_sync(kFull, p);
  if (!b) return;
  const int slot = (r + 1) % 3;
  const int at = queue_place(sh, p, b, slot);
  if (!p) return;
  if (at < kFloodQueue<W>) reinterpret_cast<uint2 *>(queue_bytes())[((r + 1) & 1) * kFloodQueue<W> + at] = make_uint2(unsigned(v), d);
  else spill(a, v, spill_bit(r + 1), spill_list, &L->spilled[slot]);
}

// Pulls the next object for this group; false when its queue is empty. The group's first CTA
// pops and publishes; every CTA copies the object into its own shared memory.
template <int C>
__device__ bool next_object(const EngineArgs &a, Shared &sh, Shared *L, bool big) {
  using G = Group<C>;
  if (G::first()) {
    const int j = atomicAdd(a.queue + (big ? 0 : 1), 1);
    const int limit = big ? a.nbig : a.nobj - a.nbig;
    L->obj = j < limit ? a.schedule[big ? j : a.nbig + j] : -1;
    if (L->obj >= 0) {
      const int o = L->obj;
      L->begin = a.obj_begin[o];
      L->count = a.obj_count[o];
      L->status = a.status[o];  // kOk unless an earlier pass gave up on the object
      const int r = a.obj_arena[o];
      L->a0 = a.arena_offset[r];
      L->sx = a.arena_dims[3 * r];
      L->sy = a.arena_dims[3 * r + 1];
      L->sz = a.arena_dims[3 * r + 2];
    }
  }
  G::sync();
  if (threadIdx.x == 0) {
    sh.obj = vload(&L->obj);
    if (sh.obj >= 0) {
      sh.begin = vload(&L->begin); sh.count = vload(&L->count);
      sh.a0 = vload(&L->a0); sh.sx = vload(&L->sx); sh.sy = vload(&L->sy); sh.sz = vload(&L->sz);
      fast_div(unsigned(sh.sx) * unsigned(sh.sy), sh.mxy, sh.pxy);
      fast_div(unsigned(sh.sx), sh.mx, sh.px);
    }
  }
  __syncthreads();
  if (sh.obj >= 0 && threadIdx.x < 26) {
    const int k = threadIdx.x;
    sh.off[k] = c_dx[k] + sh.sx * (c_dy[k] + sh.sy * c_dz[k]);
    sh.w[k] = a.w[k];
  }
  // every CTA has its copy before the first CTA moves on (or exits, ending its shared memory)
  G::sync();
  return sh.obj >= 0;
}

// ---------------------------------------------------------------------------------------------
// Geometric flood from `source` over the object's voxels into `d` (+inf at rest on them):
// Bellman-Ford rounds, fl(d[u] + w[k]). The fixed point is the least float32 path sum, which any
// schedule reaches. Returns false when the round bound is hit.
// The free-space seed of a soma's DAF (sssp_kernels.cuh:14-35): the 26-connected distance from
// the root through empty space, for voxels within `radius` (float32 physical distance) of it;
// -1 beyond. One rounding per operation, in the reference's order.
__device__ float freespace_seed(const EngineArgs &a, int x, int y, int z, int rx, int ry, int rz, float radius) {
  const float wx = a.wx, wy = a.wy, wz = a.wz;
  const float rdx = __fmul_rn(wx, float(x - rx)), rdy = __fmul_rn(wy, float(y - ry)), rdz = __fmul_rn(wz, float(z - rz));
  const float r2 = __fadd_rn(__fadd_rn(__fmul_rn(rdx, rdx), __fmul_rn(rdy, rdy)), __fmul_rn(rdz, rdz));
  if (r2 > __fmul_rn(radius, radius)) return -1.0f;
  const float dx = fabsf(float(x - rx)), dy = fabsf(float(y - ry)), dz = fabsf(float(z - rz));
  const float dxyz = fminf(fminf(dx, dy), dz);
  const float dxy = fminf(dx, dy), dyz = fminf(dy, dz), dxz = fminf(dx, dz);
  const float wxx = __fmul_rn(wx, wx), wyy = __fmul_rn(wy, wy), wzz = __fmul_rn(wz, wz);
  float v = __fmul_rn(dxyz, sqrtf(__fadd_rn(__fadd_rn(wxx, wyy), wzz)));
  v = __fadd_rn(v, __fmul_rn(wx, __fsub_rn(dx, dxyz)));
  v = __fadd_rn(v, __fmul_rn(wy, __fsub_rn(dy, dxyz)));
  v = __fadd_rn(v, __fmul_rn(wz, __fsub_rn(dz, dxyz)));
  v = __fadd_rn(v, __fmul_rn(__fsub_rn(dxy, dxyz), __fsub_rn(__fsub_rn(sqrtf(__fadd_rn(wxx, wyy)), wx), wy)));
  v = __fadd_rn(v, __fmul_rn(__fsub_rn(dxz, dxyz), __fsub_rn(__fsub_rn(sqrtf(__fadd_rn(wxx, wzz)), wx), wz)));
  v = __fadd_rn(v, __fmul_rn(__fsub_rn(dyz, dxyz), __fsub_rn(__fsub_rn(sqrtf(__fadd_rn(wyy, wzz)), wy), wz)));
  return v;
}

// seed_radius > 0 (a soma's DAF): every object voxel within it of `source` starts at its
// free-space seed, and the rounds relax from all of them.
// A round waits for two dependent L2 round trips (the neighbours' distances, then the atomic
// minimum of those that improve) and one group barrier. A queued pair whose voxel has a smaller
// distance by now is skipped: that distance has been queued too.
// A lone CTA's flood goes by bands: distances past the band's end T only enter the far list, at their first
// touch; when the band has converged the list's voxels become the frontier, each with the least of the offers it
// got meanwhile. Without bands a voxel was queued 2.2 to 2.9 times; a lone CTA is bound by the voxels it takes
// (512^3 dense prepare 11.8 -> 9.3 ms), a cluster by its rounds, of which bands make more (256^3 dense 2.3 -> 3.4).
// The band is the largest step wide, so the next band holds the whole list: a distance is at most T plus one
// step. A soma's seeds lie anywhere: its flood has one band.
template <int C, int W>
__device__ bool flood_geometric(const EngineArgs &a, Shared &sh, Shared *L, float *d, int source, int *A, int *B,
                                int *FA, int *FB, float seed_radius = 0.0f) {
  using G = Group<C>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  if (threadIdx.x == 0) { sh.qn[0] = 0; sh.qn[1] = 0; sh.qn[2] = 0; }
  if (G::first()) {
    L->spilled[0] = 0; L->spilled[1] = 0; L->spilled[2] = 0;
    L->far_n[0] = 0; L->far_n[1] = 0;
  }
  G::sync();
  uint2 *queue = reinterpret_cast<uint2 *>(queue_bytes());
  int r = -1;  // the seeds are queued for round 0
  if (seed_radius > 0.0f) {
    int rx, ry, rz;
    unravel3(source - sh.a0, sh.sx, sh.sy, rx, ry, rz);
    for (int i0 = G::tid() - lane; i0 < sh.count; i0 += G::threads()) {
      const int i = i0 + lane;
      float s = -1.0f;
      int v = 0;
      if (i < sh.count) {
        v = a.vox[sh.begin + i];
        int x, y, z;
        unravel3(v - sh.a0, sh.sx, sh.sy, x, y, z);
        s = freespace_seed(a, x, y, z, rx, ry, rz, seed_radius);
        if (s >= 0.0f) d[v] = s;
      }
      queue_flood<W>(a, sh, L, s >= 0.0f, v, __float_as_uint(s), r, A);
    }
  } else if (G::first()) {
    d[source] = 0.0f;
    queue[0] = make_uint2(unsigned(source), 0u);
    sh.qn[0] = 1;
  }
  G::sync();
  const bool neighbour = lane < 26;
  const int off = neighbour ? sh.off[lane] : 0;
  const float w = neighbour ? sh.w[lane] : 0.0f;
  const long long bound = capped(a, 8LL * sh.count + 256);
  const float width = C > 1 || seed_radius > 0.0f ? inf() : a.w[25];
  float T = width;
  int p = 0;  // the far list in use
  for (r = 0;; ++r) {
    const Share s = share_of<C>(sh, r % 3, kFloodQueue<W>);
    const int spilled = vload(&L->spilled[r % 3]);
    if (s.total + spilled == 0) {
      const int nf = vload(&L->far_n[p]);
      if (nf == 0) break;
      if (r >= bound) return false;
      // the far list becomes round r + 1's frontier (round r's counters may still be read by a CTA that
      // finds them empty)
      if (threadIdx.x == 0) sh.qn[(r + 2) % 3] = 0;
      if (G::first()) L->spilled[(r + 2) % 3] = 0;
      const int *far = p ? FB : FA;
      for (int i0 = G::tid() - lane; i0 < nf; i0 += G::threads()) {
        const int i = i0 + lane;
        const int v = i < nf ? __ldcg(far + i) : 0;
        const float dv = i < nf ? __ldcg(d + v) : 0.0f;
        queue_flood<W>(a, sh, L, i < nf && dv > T, v, __float_as_uint(dv), r, (r & 1) ? A : B);
      }
      T = __fadd_rn(T, width);
      G::sync();
      if (G::first()) L->far_n[p] = 0;
      p ^= 1;
      continue;
    }
    if (r >= bound) return false;
    if (threadIdx.x == 0) sh.qn[(r + 2) % 3] = 0;
    if (G::first()) L->spilled[(r + 2) % 3] = 0;
    int *cur = (r & 1) ? B : A, *nxt = (r & 1) ? A : B;
    auto relax = [&](const uint2 (&e)[kPipe]) {
      unsigned m[kPipe];
      float du[kPipe], dv[kPipe], old[kPipe], cand[kPipe];
#pragma unroll
      for (int j = 0; j < kPipe; ++j) {
        const int u = int(e[j].x), v = u + off;
        m[j] = a.mask[u];
        du[j] = __ldcg(d + u);
        dv[j] = neighbour && unsigned(v) < a.n ? __ldcg(d + v) : 0.0f;
      }
#pragma unroll
      for (int j = 0; j < kPipe; ++j) {
        const float x = __uint_as_float(e[j].y);
        cand[j] = __fadd_rn(x, w);
        const bool want = neighbour && ((m[j] >> lane) & 1u) && du[j] >= x && cand[j] < dv[j];
        old[j] = want ? atomic_min_pos(d + int(e[j].x) + off, cand[j]) : -1.0f;
      }
      Places near, later;
#pragma unroll
      for (int j = 0; j < kPipe; ++j) {
        const bool improved = old[j] > cand[j];
        near.ballot[j] = __ballot_sync(kFull, improved && cand[j] <= T);
        later.ballot[j] = __ballot_sync(kFull, improved && cand[j] > T && old[j] == inf());
      }
      const int nn = near.total(), nl = later.total();
      if (!(nn + nl)) return;
      const int slot = (r + 1) % 3, n = lane == 0 ? nn : lane == 1 ? nl : 0;
      int next = 0;
      if (n) next = atomicAdd(lane == 0 ? &sh.qn[slot] : &L->far_n[p], n);
      near.next = __shfl_sync(kFull, next, 0);
      later.next = __shfl_sync(kFull, next, 1);
      int *far = p ? FB : FA;
#pragma unroll
      for (int j = 0; j < kPipe; ++j) {
        const int v = int(e[j].x) + off;
        const int q = near.take(j);
        if ((near.ballot[j] >> lane) & 1u) {
          if (q < kFloodQueue<W>) queue[((r + 1) & 1) * kFloodQueue<W> + q] = make_uint2(unsigned(v), __float_as_uint(cand[j]));
          else spill(a, v, spill_bit(r + 1), nxt, &L->spilled[slot]);
        }
        const int f = later.take(j);
        if ((later.ballot[j] >> lane) & 1u) far[f] = v;
      }
    };
    for (int i = s.lo + warp * kPipe; i < s.hi; i += warps * kPipe) {
      uint2 e[kPipe];
#pragma unroll
      for (int j = 0; j < kPipe; ++j) {
        int q, at;
        locate<C>(s, min(i + j, s.hi - 1), q, at);
        e[j] = of_rank<C>(queue, q)[(r & 1) * kFloodQueue<W> + at];
        if (i + j >= s.hi) e[j].y = BK_INF_BITS;  // past the share: relaxes nothing
      }
      relax(e);
    }
    for (int i = (G::tid() >> 5) * kPipe; i < spilled; i += (G::threads() >> 5) * kPipe) {
      uint2 e[kPipe];
#pragma unroll
      for (int j = 0; j < kPipe; ++j) {
        const int u = __ldcg(cur + min(i + j, spilled - 1));
        if (lane == 0 && i + j < spilled) atomicAnd(a.flags + u, ~spill_bit(r));
        e[j] = make_uint2(unsigned(u), i + j < spilled ? __float_as_uint(__ldcg(d + u)) : BK_INF_BITS);
      }
      relax(e);
    }
    G::sync();
  }
  return true;
}

// Largest finite value of `f` over the object's voxels, ties -> lowest flat index: the packed key
// (value bits << 32 | ~flat), 0 when nothing is finite.
template <int C>
__device__ unsigned long long object_argmax(const EngineArgs &a, Shared &sh, Shared *L, const float *f) {
  using G = Group<C>;
  if (threadIdx.x == 0) sh.best = 0;
  G::sync();
  unsigned long long best = 0;
  for (int i = G::tid(); i < sh.count; i += G::threads()) {
    const int v = a.vox[sh.begin + i];
    const float x = __ldcg(f + v);
    if (x < inf()) {
      const unsigned long long k = (static_cast<unsigned long long>(__float_as_uint(x)) << 32) | (0xFFFFFFFFu - unsigned(v));
      best = k > best ? k : best;
    }
  }
  const unsigned hi = __reduce_max_sync(kFull, unsigned(best >> 32));
  const unsigned lo = __reduce_max_sync(kFull, unsigned(best >> 32) == hi ? unsigned(best) : 0u);
  if ((threadIdx.x & 31) == 0) atomicMax(&sh.best, (static_cast<unsigned long long>(hi) << 32) | lo);
  G::sync();
  const unsigned long long r = G::max_over(&sh.best);
  G::sync();
  return r;
}

template <int C, int W>
__device__ void prepare_loop(const EngineArgs &a, bool big) {
  using G = Group<C>;
  __shared__ Shared sh;
  Shared *L = G::leader(&sh);
  while (next_object<C>(a, sh, L, big)) {
    const int o = sh.obj;
    int *A = a.lists + sh.begin, *B = A + a.F, *FA = B + a.F, *FB = FA + a.F;
    int root = a.border_root[o];
    bool ok = true;
    if (root < 0) {
      // the farthest voxel (geometric distance) from the object's first voxel
      ok = flood_geometric<C, W>(a, sh, L, a.daf, a.vox[sh.begin], A, B, FA, FB);
      if (ok) {
        const unsigned long long k = object_argmax<C>(a, sh, L, a.daf);
        root = int(0xFFFFFFFFu - unsigned(k));
        for (int i = G::tid(); i < sh.count; i += G::threads()) a.daf[a.vox[sh.begin + i]] = inf();
        G::sync();
      }
    }
    if (ok) ok = flood_geometric<C, W>(a, sh, L, a.daf, root, A, B, FA, FB, a.free_radius[o]);
    if (!ok) {
      if (G::first()) a.status[o] = kBudget;
      G::sync();
      continue;
    }
    const unsigned long long k = object_argmax<C>(a, sh, L, a.daf);
    const float farthest = __uint_as_float(unsigned(k >> 32));
    const int target = int(0xFFFFFFFFu - unsigned(k));
    // PDRF of the object's voxels (the reference's pdrf_lab, batched_regular.inc:93-108):
    // (1 - dbf * M)^(2^squarings) * scale + daf * inv, one rounding per operation.
    const float M = a.M[o];
    const bool with_daf = farthest != 0.0f;
    const float inv = with_daf ? __double2float_rn(__ddiv_rn(1.0, (double)farthest)) : 0.0f;
    for (int i = G::tid(); i < sh.count; i += G::threads()) {
      const int v = a.vox[sh.begin + i];
      a.pdrf[v] = pdrf_value(a.dbf[v], with_daf ? __ldcg(a.daf + v) : 0.0f, M, inv, a.pdrf_scale, a.squarings,
                             a.exponent);
    }
    G::sync();
    if (G::first()) {
      if (a.fix_branching) a.pdrf[root] = 0.0f;  // the root is the first rail
      a.root[o] = root;
      a.target[o] = target;
      a.max_daf[o] = farthest;
    }
    G::sync();
  }
}

// Every CTA belongs to a cluster. The clusters first take the large objects, one each, then every
// CTA takes small objects on its own: large objects start first (they set the kernel's length),
// and no CTA idles while any object is left.
// (C == 1: a launch without large objects.)
template <int C, int W>
__global__ void __launch_bounds__(W, kEngineThreads / W) prepare_kernel(const __grid_constant__ EngineArgs a) {
  if constexpr (C > 1) prepare_loop<C, W>(a, true);
  prepare_loop<1, W>(a, false);
}

// ---------------------------------------------------------------------------------------------
// Railroad flood from target t over the object's voxels: entering v costs pdrf[v] (vw_step), rails
// (pdrf == 0) absorb. Near-far bands: the near band [.., T] is relaxed to convergence, bounded by
// the best rail found so far; the next band starts at the nearest deferred voxel. Returns the
// nearest rail as (distance bits << 32 | flat), BK_UNCLAIMED when no rail is reachable, and sets
// L->status on a bound. The result is schedule-independent: every voxel at distance <= D (the
// nearest rail's) is exact when the flood stops.
// The far list holds the voxels first reached beyond T (at their first touch, so once each); one
// whose distance is at most the T before has since been queued as near.
template <int C, int W>
__device__ unsigned long long railroad(const EngineArgs &a, Shared &sh, Shared *L, int t, int *A, int *B, int *FA,
                                       int *FB, int *touched) {
  using G = Group<C>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  uint2 *queue = reinterpret_cast<uint2 *>(queue_bytes());
  const bool rails = a.fix_branching != 0;
  // without fix_branching there are no rails: a full SSSP from t (the parents' field)
  const float ft = __ldcg(a.pdrf + t);
  const bool on_rail = rails && ft == 0.0f;
  if (threadIdx.x == 0) {
    sh.rb = BK_UNCLAIMED;
    sh.minfar[0] = kMinFarNone; sh.minfar[1] = kMinFarNone;
    sh.qn[0] = 0; sh.qn[1] = 0; sh.qn[2] = 0;
    sh.T = fmaxf(__fmul_rn(a.rail_band, ft), 1e-30f);
  }
  if (G::first()) {
    L->n_touch = 1;
    touched[0] = t;
    L->spilled[0] = 0; L->spilled[1] = 0; L->spilled[2] = 0;
    L->far_n[0] = 0; L->far_n[1] = 0;
    a.dist[t] = 0.0f;
    if (!on_rail) {
      queue[0] = make_uint2(unsigned(t), 0u);
      sh.qn[0] = 1;
    }
  }
  G::sync();
  if (on_rail) return static_cast<unsigned long long>(unsigned(t));
  const bool neighbour = lane < 26;
  const int off = neighbour ? sh.off[lane] : 0;
  int p = 0;  // the far list in use
  // The bound counts rounds, which bounds the bands too: after an empty band the nearest deferred offer is the
  // nearest waiting voxel's own distance, so that voxel is inside the next band.
  const long long bound = capped(a, 16LL * sh.count + 256);
  long long work = 0;
  int r = 0;
  for (int band = 0;; ++band) {
    int *far = p ? FB : FA, *keep = p ? FA : FB;
    const float T = vload(&sh.T);
    unsigned long long *minfar = &sh.minfar[band & 1];
    // the nearest deferred voxel: the lanes' least (distance, penalty)
    auto defer = [&](bool is, float dist, float penalty) {
      const unsigned mine = is ? __float_as_uint(dist) : BK_INF_BITS;
      const unsigned least = __reduce_min_sync(kFull, mine);
      if (least < unsigned(vload(minfar) >> 32) && is && mine == least)
        atomicMin(minfar, (static_cast<unsigned long long>(mine) << 32) | __float_as_uint(penalty));
    };
    for (const int first_round = r;; ++r) {
      const Share s = share_of<C>(sh, r % 3, kFloodQueue<W>);
      const int spilled = vload(&L->spilled[r % 3]);
      if (s.total + spilled == 0) {
        // A band may be empty: the offer that named it can have been improved into the band before it. The
        // barrier that every round ends with then stands here, between this band's reading of sh.T and the
        // clearing of the last band's list, before it, and the next band's end and list, after it.
        if (r == first_round) G::sync();
        break;
      }
      if (++work > bound) {
        if (G::first()) L->status = kBudget;
        G::sync();
        return BK_UNCLAIMED;
      }
      if (threadIdx.x == 0) sh.qn[(r + 2) % 3] = 0;
      if (G::first()) { L->spilled[(r + 2) % 3] = 0; L->rounds += 1; }
      int *cur = (r & 1) ? B : A, *nxt = (r & 1) ? A : B;
      auto relax = [&](const uint2 (&e)[kPipe]) {
        unsigned m[kPipe];
        float du[kPipe], dv[kPipe], fv[kPipe], old[kPipe], cand[kPipe];
#pragma unroll
        for (int j = 0; j < kPipe; ++j) {
          const int u = int(e[j].x), v = u + off;
          m[j] = a.mask[u];
          du[j] = __ldcg(a.dist + u);
          const bool in = neighbour && unsigned(v) < a.n;
          fv[j] = in ? a.pdrf[v] : 0.0f;
          dv[j] = in ? __ldcg(a.dist + v) : 0.0f;
        }
        // beyond the nearest rail found so far nothing matters: its distance only falls
        const float nearest = __uint_as_float(min(unsigned(vload(&sh.rb) >> 32), BK_INF_BITS));
#pragma unroll
        for (int j = 0; j < kPipe; ++j) {
          const float x = __uint_as_float(e[j].y);
          cand[j] = vw_step(x, fv[j]);
          const bool want = neighbour && ((m[j] >> lane) & 1u) && du[j] >= x && cand[j] < dv[j] && cand[j] <= nearest;
          old[j] = want ? atomic_min_pos(a.dist + int(e[j].x) + off, cand[j]) : -1.0f;
        }
        Places near, first, later;
        unsigned beyond = 0;  // by voxel, this lane's
        bool any = false;
#pragma unroll
        for (int j = 0; j < kPipe; ++j) {
          const bool improved = old[j] > cand[j], rail = rails && fv[j] == 0.0f, fresh = improved && old[j] == inf();
          const bool far = improved && !rail && cand[j] > T;
          near.ballot[j] = __ballot_sync(kFull, improved && !rail && !far);
          first.ballot[j] = __ballot_sync(kFull, fresh);
          later.ballot[j] = __ballot_sync(kFull, far && fresh);
          beyond |= far ? 1u << j : 0u;
          any |= improved;
          if (improved && rail)
            atomicMin(&sh.rb, (static_cast<unsigned long long>(__float_as_uint(cand[j])) << 32) | unsigned(int(e[j].x) + off));
        }
        if (!__any_sync(kFull, any)) return;
        const int slot = (r + 1) % 3;
        reserve(near, first, later, &sh.qn[slot], &L->n_touch, &L->far_n[p]);
        const bool defers = __any_sync(kFull, beyond);
#pragma unroll
        for (int j = 0; j < kPipe; ++j) {
          const int v = int(e[j].x) + off;
          const int q = near.take(j);
          if ((near.ballot[j] >> lane) & 1u) {
            if (q < kFloodQueue<W>) queue[((r + 1) & 1) * kFloodQueue<W> + q] = make_uint2(unsigned(v), __float_as_uint(cand[j]));
            else spill(a, v, spill_bit(r + 1), nxt, &L->spilled[slot]);
          }
          const int w = first.take(j);
          if ((first.ballot[j] >> lane) & 1u) touched[w] = v;
          const int f = later.take(j);
          if ((later.ballot[j] >> lane) & 1u) far[f] = v;
        }
        if (defers) {  // the lane's nearest of its voxels, then the warp's
          float d = inf(), f = 0.0f;
#pragma unroll
          for (int j = 0; j < kPipe; ++j)
            if (((beyond >> j) & 1u) && (cand[j] < d || (cand[j] == d && fv[j] < f))) { d = cand[j]; f = fv[j]; }
          defer(beyond != 0, d, f);
        }
      };
      for (int i = s.lo + warp * kPipe; i < s.hi; i += warps * kPipe) {
        uint2 e[kPipe];
#pragma unroll
        for (int j = 0; j < kPipe; ++j) {
          int q, at;
          locate<C>(s, min(i + j, s.hi - 1), q, at);
          e[j] = of_rank<C>(queue, q)[(r & 1) * kFloodQueue<W> + at];
          if (i + j >= s.hi) e[j].y = BK_INF_BITS;  // past the share: relaxes nothing
        }
        relax(e);
      }
      for (int i = (G::tid() >> 5) * kPipe; i < spilled; i += (G::threads() >> 5) * kPipe) {
        uint2 e[kPipe];
#pragma unroll
        for (int j = 0; j < kPipe; ++j) {
          const int u = __ldcg(cur + min(i + j, spilled - 1));
          if (lane == 0 && i + j < spilled) atomicAnd(a.flags + u, ~spill_bit(r));
          e[j] = make_uint2(unsigned(u), i + j < spilled ? __float_as_uint(__ldcg(a.dist + u)) : BK_INF_BITS);
        }
        relax(e);
      }
      G::sync();
    }
    // Band end. Each CTA combines the group's copies by itself (they rest since the round's
    // barrier; the next band's minima go to the other copy): the nearest rail is final once it lies
    // inside the band or nothing deferred is as near.
    if (warp == 0) {
      unsigned long long rb = lane < C ? vload(of_rank<C>(&sh.rb, lane < C ? lane : 0)) : BK_UNCLAIMED;
      unsigned long long mf = lane < C ? vload(of_rank<C>(minfar, lane < C ? lane : 0)) : kMinFarNone;
#pragma unroll
      for (int o = 1; o < C; o <<= 1) {
        const unsigned long long x = __shfl_xor_sync(kFull, rb, o), y = __shfl_xor_sync(kFull, mf, o);
        rb = x < rb ? x : rb;
        mf = y < mf ? y : mf;
      }
      if (lane == 0) {
        const float D = __uint_as_float(unsigned(rb >> 32)), d = __uint_as_float(unsigned(mf >> 32));
        int flag = 0;
        if (rb != BK_UNCLAIMED && (D <= T || mf == kMinFarNone || d > D)) flag = 1;
        else if (mf == kMinFarNone) flag = 2;
        else {
          float w = __fmul_rn(a.rail_band, __uint_as_float(unsigned(mf)));
          const float lo = __fmul_rn(5e-4f, d);
          if (!(w > lo)) w = lo;
          sh.T = __fadd_rn(d, w);
        }
        sh.flag = flag;
        sh.rb = rb;
        sh.minfar[(band + 1) & 1] = kMinFarNone;
        sh.qn[(r + 2) % 3] = 0;
      }
    }
    if (G::first()) L->spilled[(r + 2) % 3] = 0;
    __syncthreads();
    const int flag = vload(&sh.flag);
    if (flag) {
      const unsigned long long rb = vload(&sh.rb);
      G::sync();
      return flag == 1 ? rb : BK_UNCLAIMED;
    }
    // the deferred voxels inside the new band become round r + 1's frontier (round r's counters may
    // still be read by a CTA that finds them empty)
    int *nxt = (r & 1) ? A : B;
    const int nf = vload(&L->far_n[p]);
    const float Tn = vload(&sh.T);
    minfar = &sh.minfar[(band + 1) & 1];
    for (int i0 = G::tid() - lane; i0 < nf; i0 += G::threads()) {
      const int i = i0 + lane;
      int w = 0;
      float dw = 0.0f, fw = 0.0f;
      if (i < nf) {
        w = __ldcg(far + i);
        dw = __ldcg(a.dist + w);
        fw = a.pdrf[w];
      }
      const bool waits = i < nf && dw > T;
      queue_flood<W>(a, sh, L, waits && dw <= Tn, w, __float_as_uint(dw), r, nxt);
      append(waits && dw > Tn, w, keep, &L->far_n[p ^ 1]);
      defer(waits && dw > Tn, dw, fw);
    }
    G::sync();
    if (G::first()) L->far_n[p] = 0;
    p ^= 1;
    ++r;
  }
}

// One warp walks from the nearest rail back to the target: the step goes to the neighbour of least
// distance (non-rail, lowest neighbour index among ties); at the first step the rail end is
// re-picked as the last road voxel's first rail in dijkstra3d order (lockstep_regular.inc:61-155).
// Writes the path target-first to out and returns its length (-1: no room).
__device__ int backtrace(const EngineArgs &a, const Shared &sh, unsigned long long rb, int t, int *out, long long room) {
  const int lane = threadIdx.x & 31;
  const int off = lane < 26 ? sh.off[lane] : 0;
  int cur = int(unsigned(rb));
  int len = 0;
  const long long bound = 2LL * sh.count + 2;
  for (long long step = 0; step < bound; ++step) {
    int kb = -1;
    if (cur != t) {
      const uint32_t m = a.mask[cur];
      unsigned db = BK_INF_BITS;
      const int u = cur + off;
      if (lane < 26 && unsigned(u) < a.n) {  // read beside the mask, not after it
        const float f = a.pdrf[u];
        const unsigned du = __float_as_uint(__ldcg(a.dist + u));
        if (((m >> lane) & 1u) && f != 0.0f) db = du;
      }
      const unsigned mb = __reduce_min_sync(kFull, db);
      if (mb < BK_INF_BITS) kb = int(__reduce_min_sync(kFull, db == mb ? unsigned(lane) : 64u));
    }
    if (step == 0 && kb >= 0) {
      const int u = cur + sh.off[kb];
      const uint32_t mu = a.mask[u];
      unsigned key = 64;
      if (lane < 26 && ((mu >> lane) & 1u) && a.pdrf[u + sh.off[lane]] == 0.0f) key = unsigned(c_d3rank[lane]);
      const unsigned r = __reduce_min_sync(kFull, key);
      if (r < 26) {
        const int ks = c_d3inv[r];
        cur = u + sh.off[ks];
        kb = c_opp[ks];
      }
    }
    if (len >= room) return -1;
    if (lane == 0) out[len] = cur;
    ++len;
    if (kb < 0) break;
    cur += sh.off[kb];
  }
  __syncwarp();
  for (int i = lane; i < len / 2; i += 32) {
    const int x = out[i];
    out[i] = out[len - 1 - i];
    out[len - 1 - i] = x;
  }
  __syncwarp();
  return len;
}

// Without fix_branching: one warp walks from target t to the root through the parents' field (the
// object's SSSP distances from the root): each step goes to the neighbour of least distance,
// lowest neighbour index among ties (vw_assign_parents, sssp_kernels.cuh:89-110). Writes the path
// target-first to out and returns its length (-1: no room). The walk stops at the first voxel of
// an earlier path (kOnPath): the parents' field is a tree, so from there it would repeat that
// path's tail, whose vertices and edges the skeleton already holds and whose voxels are already
// dead (no invalidation source); the stored paths then total at most the object's voxels plus
// one per path.
__device__ int parent_walk(const EngineArgs &a, const Shared &sh, int t, int root, int *out, long long room) {
  const int lane = threadIdx.x & 31;
  int cur = t;
  int len = 0;
  const long long bound = 2LL * sh.count + 2;
  for (long long step = 0; step < bound; ++step) {
    if (len >= room) return -1;
    if (lane == 0) out[len] = cur;
    ++len;
    if (cur == root || (__ldcg(a.flags + cur) & kOnPath) || !(__ldcg(a.dist + cur) < inf())) break;
    const uint32_t m = a.mask[cur];
    unsigned db = BK_INF_BITS;
    if (lane < 26 && ((m >> lane) & 1u)) db = __float_as_uint(__ldcg(a.dist + cur + sh.off[lane]));
    const unsigned mb = __reduce_min_sync(kFull, db);
    if (!(mb < BK_INF_BITS)) break;
    cur += sh.off[__reduce_min_sync(kFull, db == mb ? unsigned(lane) : 64u)];
  }
  __syncwarp();
  return len;
}

// Soma trimming of a stored path (trace.cu:222-236), one warp, in place. A vertex is far when its
// float64 physical distance from the root exceeds the soma radius. With fix_branching (a
// target-first railroad path) the first vertex stays, then every far vertex, then the root when
// the rail end is not far. Without it (a target-first walk that stopped at w, the root or a vertex
// of an earlier trimmed path) the far vertices before w stay, then w: the reference's root-first
// path [root, far vertices] joins the earlier paths exactly there (its far vertices beyond w are
// those paths' own). Returns the new length (-1: no room).
__device__ int soma_trim(const EngineArgs &a, const Shared &sh, int *path, int len, int root, double radius, bool rails,
                         long long room) {
  const int lane = threadIdx.x & 31;
  int rx, ry, rz;
  unravel3(root - sh.a0, sh.sx, sh.sy, rx, ry, rz);
  auto far = [&](int v) {
    int x, y, z;
    unravel3(v - sh.a0, sh.sx, sh.sy, x, y, z);
    const double dx = __dmul_rn(double(a.wx), double(x - rx)), dy = __dmul_rn(double(a.wy), double(y - ry)),
                 dz = __dmul_rn(double(a.wz), double(z - rz));
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz))) > radius;
  };
  const int last = path[len - 1];
  const bool last_far = far(last);
  // the kept range: [1, len) with the first vertex kept as it is (rails), or [0, len - 1) with the
  // stop vertex appended (no rails)
  const int begin = rails ? 1 : 0, end = rails ? len : len - 1;
  int k = rails ? 1 : 0;
  for (int base = begin; base < end; base += 32) {
    const int i = base + lane;
    const int v = i < end ? path[i] : 0;
    const bool keep = i < end && far(v);
    const unsigned ballot = __ballot_sync(kFull, keep);
    __syncwarp();
    if (keep) path[k + __popc(ballot & ((1u << lane) - 1u))] = v;
    k += __popc(ballot);
    __syncwarp();
  }
  if (rails && !last_far) {
    if (k >= room) return -1;
    if (lane == 0) path[k] = root;
    ++k;
  } else if (!rails) {
    if (lane == 0) path[k] = last;
    ++k;
  }
  __syncwarp();
  return k;
}

__device__ __forceinline__ float distance_to(const EngineArgs &a, int x, int y, int z, int qx, int qy, int qz) {
  const float dx = __fmul_rn(a.wx, float(x - qx)), dy = __fmul_rn(a.wy, float(y - qy)), dz = __fmul_rn(a.wz, float(z - qz));
  return sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
}
__device__ __forceinline__ float reach(const EngineArgs &a, int s, float scale, float constant) {
  return __fadd_rn(__fmul_rn(scale, a.dbf[s]), constant);
}
__device__ __forceinline__ int band_of(unsigned mbits, float delta, int kmin) {
  const float m = __uint_as_float(mbits);
  int k = int(__fdiv_rn(m, delta));
  while (__fmul_rn(float(k + 1), delta) <= m) ++k;
  while (k > 0 && __fmul_rn(float(k), delta) > m) --k;
  return k < kmin ? kmin : k;
}

// The re-claimed voxels of a band that are listed: a sixteenth of the object's voxels. With more, looking at every waiting
// voxel is the shorter way. (0.3 % on the 512^3 dense workload; up to 11 % in porous objects at spacings 40 times apart.)
__device__ __forceinline__ int redo_room(const Shared &sh) { return sh.count >> 4; }

// Claim-order invalidation of one path (invalidation_kernels.cuh:105-297; lockstep_coop.inc:530-845):
// alive path vertices become sources (bottleneck M = 0); a claimed voxel u holding (M, s) offers
// an alive neighbour v the source s when |aniso (v - s)| < scale DBF[s] + const, with
// M' = max(M, |v - s|). Inside the band [k delta, (k+1) delta) offers claim at once, keeping the
// least (M bits, source); rounds are synchronous (offers come from the keys of the round
// boundary). Offers beyond the band wait; at the boundary the best offer that each waiting voxel has
// from its claimed neighbours counts: the smallest names the next band, those inside it are claimed.
// Claimed voxels die. Returns false when a loop bound is hit.
//
// A waiting voxel's best offer is kept where offers are made (an atomic minimum on its key), not
// gathered at the boundary: a voxel's key is final once its band has converged (every later offer
// is at least the next band's), so an offer made from a voxel's final key stays right. A voxel whose
// key improves again after its claim may have made offers from the earlier key: it is listed, and
// at the boundary its waiting neighbours take their best offer from their claimed neighbours anew.
// On the 512^3 dense workload 0.3 % of the claims are listed; gathering at every boundary instead
// read 2.3 waiting voxels' neighbourhoods per foreground voxel and was 43 % of the trace's object time
// (24 us a boundary).
// A round has two steps with a group barrier between them. Step A takes the queued pairs whose key
// is still the voxel's (the round boundary's keys) and stages per voxel what its offers share: mask,
// key, position relative to the source and the source's reach. Step B makes the offers, a warp per
// voxel: one L2 read per neighbour decides it (dead, holding a better key or offer, or out of reach:
// done), an atomic follows only where the key changes.
template <int C, int W>
__device__ bool invalidate(const EngineArgs &a, Shared &sh, Shared *L, const int *path, int npath, int *A, int *B,
                           int *FA, int *FB, int *touched, int *redo, unsigned long long *wide) {
  using G = Group<C>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  int4 *stage_id = reinterpret_cast<int4 *>(queue_bytes());           // voxel, mask, source + 1, M bits
  float4 *stage_at = reinterpret_cast<float4 *>(stage_id + kInvalQueue<W>);  // position - source's, reach
  unsigned long long *queue_key = reinterpret_cast<unsigned long long *>(stage_at + kInvalQueue<W>);
  int *queue_vox = reinterpret_cast<int *>(queue_key + 2 * kInvalQueue<W>);
  if (threadIdx.x == 0) {
    sh.qn[0] = 0; sh.qn[1] = 0; sh.qn[2] = 0;
    sh.lowest[0] = BK_INF_BITS; sh.lowest[1] = BK_INF_BITS;
  }
  if (G::first()) {
    L->spilled[0] = 0; L->spilled[1] = 0; L->spilled[2] = 0;
    L->far_n[0] = 0; L->far_n[1] = 0;
    L->n_touch = 0;
    L->n_redo = 0;
  }
  G::sync();
  // queues the claimed voxels v (keys k) of the lanes with p in queue slot `slot`, buffer `buffer`
  auto queue = [&](bool p, int v, unsigned long long k, int slot, int buffer, int *spill_list) {
    const unsigned b = __ballot_sync(kFull, p);
    if (!b) return;
    const int at = queue_place(sh, p, b, slot);
    if (!p) return;
    if (at < kInvalQueue<W>) {
      queue_vox[buffer * kInvalQueue<W> + at] = v;
      queue_key[buffer * kInvalQueue<W> + at] = k;
    } else spill(a, v, kFront, spill_list, &L->spilled[slot]);
  };
  for (int i0 = G::tid() - lane; i0 < npath; i0 += G::threads()) {
    const int i = i0 + lane;
    const int v = i < npath ? __ldcg(path + i) : 0;
    const unsigned long long k = unsigned(v) + 1u;
    bool claimed = false;
    if (i < npath && __ldcg(a.key + v) != 0) claimed = atomicMin(a.key + v, k) == BK_UNCLAIMED;
    queue(claimed, v, k, 0, 0, A);
    append(claimed, v, touched, &L->n_touch);
  }
  G::sync();
  auto stage = [&](int i, int u, int m, unsigned long long k) {
    const int source = int(unsigned(k)) - 1;
    const float rs = reach(a, source, sh.rscale, sh.rconst);
    int x, y, z, qx, qy, qz;
    coordinates(sh, u - sh.a0, x, y, z);
    coordinates(sh, source - sh.a0, qx, qy, qz);
    stage_id[i] = make_int4(u, m, source + 1, int(k >> 32));
    stage_at[i] = make_float4(float(x - qx), float(y - qy), float(z - qz), rs);
  };
  auto list_redo = [&](int v) {
    const int at = atomicAdd(&L->n_redo, 1);
    if (at < redo_room(sh)) redo[at] = v;
  };
  const bool neighbour = lane < 26;
  const int off = neighbour ? sh.off[lane] : 0;
  const float ox = neighbour ? float(c_dx[lane]) : 0.0f, oy = neighbour ? float(c_dy[lane]) : 0.0f,
              oz = neighbour ? float(c_dz[lane]) : 0.0f;
  int p = 0;  // the waiting list in use
  const long long bound = capped(a, 64LL * sh.count + 1024);
  long long work = 0;
  int band = 0, r = 0;
  for (int boundary = 0;; ++boundary) {
    int *far = p ? FB : FA, *keep = p ? FA : FB;
    unsigned hi = __float_as_uint(__fmul_rn(float(band + 1), a.delta));
    for (;; ++r) {
      const Share s = share_of<C>(sh, r % 3, kInvalQueue<W>);
      const int spilled = vload(&L->spilled[r % 3]);
      if (s.total + spilled == 0) break;
      if (++work > bound) return false;
      if (threadIdx.x == 0) sh.qn[(r + 2) % 3] = 0;
      if (G::first()) { L->spilled[(r + 2) % 3] = 0; L->rounds += 1ull << 32; }
      int *cur = (r & 1) ? B : A, *nxt = (r & 1) ? A : B;
      // step A: a thread per queued pair
      for (int i0 = s.lo + warp * 32; i0 < s.hi; i0 += warps * 32) {
        const int i = i0 + lane;
        int q, at;
        locate<C>(s, min(i, s.hi - 1), q, at);
        if (i < s.hi) {
          const int u = of_rank<C>(queue_vox, q)[(r & 1) * kInvalQueue<W> + at];
          const unsigned long long k = of_rank<C>(queue_key, q)[(r & 1) * kInvalQueue<W> + at];
          const unsigned m = a.mask[u];
          const bool current = __ldcg(a.key + u) == k;
          stage(i - s.lo, u, current ? int(m) : 0, k);
        }
      }
      for (int i = G::tid(); i < spilled; i += G::threads()) {
        const int u = __ldcg(cur + i);
        wide[i] = __ldcg(a.key + u);
        atomicAnd(a.flags + u, ~kFront);
      }
      G::sync();
      // step B: a warp per voxel; the spilled voxels come after the queued ones, staged by this CTA
      int staged = s.hi - s.lo;
      for (int base = G::rank() * kInvalQueue<W>;;) {
        for (int i = warp * kPipe; i < staged; i += warps * kPipe) {
          unsigned long long kv[kPipe], old[kPipe];
          unsigned hb[kPipe];  // the offers' upper words
#pragma unroll
          for (int j = 0; j < kPipe; ++j) {
            const int2 e = *reinterpret_cast<const int2 *>(stage_id + min(i + j, staged - 1));
            const bool is = neighbour && i + j < staged && ((unsigned(e.y) >> lane) & 1u);
            kv[j] = is ? __ldcg(a.key + e.x + off) : 0ull;
          }
#pragma unroll
          for (int j = 0; j < kPipe; ++j) {
            const int4 e = stage_id[min(i + j, staged - 1)];
            const float4 at = stage_at[min(i + j, staged - 1)];
            const float dx = __fmul_rn(a.wx, at.x + ox), dy = __fmul_rn(a.wy, at.y + oy), dz = __fmul_rn(a.wz, at.z + oz);
            const float d = sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
            const unsigned mb = max(__float_as_uint(d), unsigned(e.w));
            hb[j] = mb < hi ? mb : mb | 0x80000000u;
            const unsigned long long cand = (static_cast<unsigned long long>(hb[j]) << 32) | unsigned(e.z);
            old[j] = 0;
            if (d < at.w && cand < kv[j]) old[j] = atomicMin(a.key + e.x + off, cand);
          }
          Places claimed, first, waits;
          unsigned any = 0;
#pragma unroll
          for (int j = 0; j < kPipe; ++j) {
            const int4 e = stage_id[min(i + j, staged - 1)];
            const unsigned long long cand = (static_cast<unsigned long long>(hb[j]) << 32) | unsigned(e.z);
            const bool claims = old[j] > cand && cand < kWaits;
            claimed.ballot[j] = __ballot_sync(kFull, claims);
            first.ballot[j] = __ballot_sync(kFull, claims && old[j] >= kWaits);
            waits.ballot[j] = __ballot_sync(kFull, cand >= kWaits && old[j] == BK_UNCLAIMED);
            any |= claimed.ballot[j] | waits.ballot[j];
            if (claims && old[j] < kWaits) list_redo(e.x + off);
          }
          if (!any) continue;
          const int slot = (r + 1) % 3, buffer = ((r + 1) & 1) * kInvalQueue<W>;
          reserve(claimed, first, waits, &sh.qn[slot], &L->n_touch, &L->far_n[p]);
#pragma unroll
          for (int j = 0; j < kPipe; ++j) {
            const int4 e = stage_id[min(i + j, staged - 1)];
            const int v = e.x + off;
            const int q = claimed.take(j);
            if ((claimed.ballot[j] >> lane) & 1u) {
              if (q < kInvalQueue<W>) {
                queue_vox[buffer + q] = v;
                queue_key[buffer + q] = (static_cast<unsigned long long>(hb[j]) << 32) | unsigned(e.z);
              } else spill(a, v, kFront, nxt, &L->spilled[slot]);
            }
            const int w = first.take(j);
            if ((first.ballot[j] >> lane) & 1u) touched[w] = v;
            const int f = waits.take(j);
            if ((waits.ballot[j] >> lane) & 1u) far[f] = v;
          }
        }
        if (base >= spilled) break;
        __syncthreads();  // the records are free
        staged = min(kInvalQueue<W>, spilled - base);
        for (int i = threadIdx.x; i < staged; i += blockDim.x) {
          const int u = __ldcg(cur + base + i);
          const unsigned long long k = __ldcg(wide + base + i);
          stage(i, u, int(a.mask[u]), k);
        }
        base += C * kInvalQueue<W>;
        __syncthreads();
      }
      G::sync();
    }
    const int nf = vload(&L->far_n[p]);
    if (nf == 0) break;
    if (++work > bound) return false;
    // band boundary: the neighbours of the listed voxels first, a warp per listed voxel and then per
    // waiting neighbour of it (the neighbours' keys, then their sources' reach)
    const int nr = vload(&L->n_redo);
    if (nr > 0) {
      const bool all = nr > redo_room(sh);  // more than the list holds: every waiting voxel
      const int m = all ? nf : nr;
      for (int i = G::tid() >> 5; i < m; i += G::threads() >> 5) {
        const int u = __ldcg((all ? far : redo) + i);
        unsigned again = 0;
        if (!all) {
          const unsigned long long kc = neighbour && ((a.mask[u] >> lane) & 1u) ? __ldcg(a.key + u + off) : 0ull;
          again = __ballot_sync(kFull, kc >= kWaits && kc != BK_UNCLAIMED);
        } else again = __ldcg(a.key + u) >= kWaits ? 1u << 26 : 0u;
        for (; again; again &= again - 1) {
          const int k = __ffs(again) - 1;
          const int c = all ? u : u + sh.off[k];
          unsigned long long ku = neighbour && ((a.mask[c] >> lane) & 1u) ? __ldcg(a.key + c + off) : 0ull;
          if (ku >= kWaits) ku = 0;
          unsigned mb = ~0u, from = ~0u;
          if (ku) {
            const int source = int(unsigned(ku)) - 1;
            int x, y, z, qx, qy, qz;
            coordinates(sh, c - sh.a0, x, y, z);
            coordinates(sh, source - sh.a0, qx, qy, qz);
            const float d = distance_to(a, x, y, z, qx, qy, qz);
            if (d < reach(a, source, sh.rscale, sh.rconst)) {
              mb = max(__float_as_uint(d), unsigned(ku >> 32)) | 0x80000000u;
              from = unsigned(ku);
            }
          }
          const unsigned least = __reduce_min_sync(kFull, mb);
          from = __reduce_min_sync(kFull, mb == least ? from : ~0u);
          // no offer left: all ones, and the voxel leaves the list below
          if (lane == 0) a.key[c] = (static_cast<unsigned long long>(least) << 32) | from;
        }
      }
      G::sync();
      if (G::first()) L->n_redo = 0;
    }
    // the smallest offer names the next band. The first strip's voxels stay in registers.
    unsigned lowest = BK_INF_BITS;
    int c0 = 0;
    unsigned long long k0 = 0;
    for (int i0 = G::tid() - lane; i0 < nf; i0 += G::threads()) {
      const int i = i0 + lane;
      int c = 0;
      unsigned long long k = 0;
      if (i < nf) {
        c = __ldcg(far + i);
        k = __ldcg(a.key + c);
      }
      if (k >= kWaits && k != BK_UNCLAIMED) lowest = min(lowest, unsigned(k >> 32) & 0x7FFFFFFFu);
      if (i < G::threads()) { c0 = c; k0 = k; }
    }
    lowest = __reduce_min_sync(kFull, lowest);
    if (lane == 0 && lowest != BK_INF_BITS) atomicMin(&sh.lowest[boundary & 1], lowest);
    G::sync();
    lowest = __reduce_min_sync(kFull, lane < C ? vload(of_rank<C>(&sh.lowest[boundary & 1], lane < C ? lane : 0)) : BK_INF_BITS);
    if (threadIdx.x == 0) sh.lowest[(boundary + 1) & 1] = BK_INF_BITS;
    if (lowest != BK_INF_BITS) band = band_of(lowest, a.delta, band + 1);
    hi = __float_as_uint(__fmul_rn(float(band + 1), a.delta));
    // offers inside it claim, the rest wait on
    int *cur = (r & 1) ? B : A;
    for (int i0 = G::tid() - lane; i0 < nf; i0 += G::threads()) {
      const int i = i0 + lane;
      int c = c0;
      unsigned long long k = k0;
      if (i >= G::threads()) {
        c = i < nf ? __ldcg(far + i) : 0;
        k = i < nf ? __ldcg(a.key + c) : 0;
      }
      const bool waits = k >= kWaits && k != BK_UNCLAIMED;
      k &= ~kWaits;
      const bool claims = waits && unsigned(k >> 32) < hi;
      if (claims) a.key[c] = k;
      queue(claims, c, k, r % 3, r & 1, cur);
      append(claims, c, touched, &L->n_touch);
      append(waits && !claims, c, keep, &L->far_n[p ^ 1]);
    }
    G::sync();
    if (G::first()) L->far_n[p] = 0;
    p ^= 1;
  }
  // the claimed voxels die
  const int nt = vload(&L->n_touch);
  for (int i = G::tid(); i < nt; i += G::threads()) a.key[__ldcg(touched + i)] = 0;
  G::sync();
  return true;
}

// A function of its own: inlined into a kernel of lone CTAs the same loop took 33.1 ms of the 512^3 dense
// trace and 23.3 as a call, on the same 148 CTAs (64 registers either way).
template <int C, int W>
__device__ __noinline__ void trace_loop(const EngineArgs &a, bool big) {
  using G = Group<C>;
  __shared__ Shared sh;
  __shared__ unsigned long long s_work[4];
  __shared__ unsigned long long s_prof[6];  // start, last lap, time in the four phases
  Shared *L = G::leader(&sh);
  if (threadIdx.x < 4) s_work[threadIdx.x] = 0;
  while (next_object<C>(a, sh, L, big)) {
    const int o = sh.obj;
    if (vload(&L->status) != kOk) {  // preparation failed; its status stands
      G::sync();
      continue;
    }
    int *L0 = a.lists + sh.begin, *L1 = L0 + a.F, *L2 = L1 + a.F, *L3 = L2 + a.F, *L4 = L3 + a.F, *L5 = L4 + a.F;
    unsigned long long *wide = a.wide + sh.begin;
    int *store = a.store + a.store_begin[o];
    const long long store_cap = a.store_cap[o];
    int *rec_start = a.rec_start + a.rec_begin[o], *rec_len = a.rec_len + a.rec_begin[o];
    const long long rec_cap = a.rec_cap[o];
    const int mcount = a.manual_count[o];
    const int *manual = a.manual + a.manual_begin[o];
    const int acount = a.after_count[o];
    const int *after = a.after + a.after_begin[o];
    int after_used = 0;
    const int *order = a.order + sh.begin;
    const long long maxp = a.max_paths[o];
    long long paths = 0, used = 0;
    int cursor = 0;
    int status = kOk;
    // per-object phase timers, kept in shared memory by the first thread (registers are scarce)
    if (G::first()) {
      L->rounds = 0;
      s_prof[0] = s_prof[1] = now_ns();
      s_prof[2] = s_prof[3] = s_prof[4] = s_prof[5] = 0;
    }
    auto lap = [&](int phase) {
      if (G::first()) { const unsigned long long t = now_ns(); s_prof[2 + phase] += t - s_prof[1]; s_prof[1] = t; }
    };
    // The loop's steps, each with one flood: first the soma's ball (a soma: an invalidation from the
    // root with the soma's reach, trace.cu:199), then the parents' field (without fix_branching:
    // the object's SSSP from the root, kept until the object is done), then the paths. Every flood
    // function has this one call site, which keeps the kernel's registers for the paths' loop.
    if (threadIdx.x == 0) {
      sh.root = a.root[o];
      sh.soma_radius = a.soma_radius[o];
      sh.step = sh.soma_radius >= 0.0 ? 0 : (a.fix_branching ? 2 : 1);
      sh.skipped = 0;
    }
    __syncthreads();
    while (status == kOk) {
      const int step = sh.step;  // 0: the soma's ball, 1: the parents' field, 2: paths
      int t = -1, len = 1;
      bool ordered = false;  // t is the first alive voxel of the DAF order
      if (step == 2) {
        const long long taken = paths + sh.skipped;  // targets taken so far, empty paths included
        if (taken >= maxp) break;
        // the next target: manual targets first, then the first alive voxel of the order, then the
        // targets after (trace.cu:209-212)
        if (taken < mcount) {
          t = manual[taken];
          if (t < 0) t = a.target[o];  // the object's own target (the DAF argmax)
        } else {
          for (;;) {
            if (threadIdx.x == 0) sh.pos = INT32_MAX;
            G::sync();
            const int pos = cursor + G::tid();
            if (pos < sh.count && __ldcg(a.key + order[pos]) != 0) atomicMin(&sh.pos, unsigned(pos));
            G::sync();
            const int found = int(G::min_over(&sh.pos));
            G::sync();
            if (found != INT32_MAX) { cursor = found; t = order[found]; ordered = true; break; }
            cursor += G::threads();
            if (cursor >= sh.count) { cursor = sh.count; break; }
          }
          if (t < 0 && after_used < acount) t = after[after_used++];
          if (t < 0) break;
        }
        lap(0);
      }
      if (step == 0) {
        if (G::first()) store[used] = sh.root;  // the ball's one source (the slot is reused)
        G::sync();
      } else if (step == 1 || a.fix_branching) {
        const unsigned long long rb = railroad<C, W>(a, sh, L, step == 1 ? sh.root : t, L0, L1, L2, L3, L4);
        lap(1);
        if (vload(&L->status) != kOk) { status = vload(&L->status); break; }
        const int nt = vload(&L->n_touch);
        if (step == 1) {  // the parents' field stays
          if (G::first()) { s_work[0] += nt; s_work[1] += nt; }
          if (threadIdx.x == 0) sh.step = 2;  // every CTA of the group moves on (each has its own copy)
          G::sync();
          continue;
        }
        if (rb == BK_UNCLAIMED) {
          // No rail is reachable from t: an infinite penalty walls it off (a cavity the avocado
          // stage painted without refreshing the field). A target of the DAF order would be picked
          // again and again, so the object ends here (trace.cu:218-224); a manual target leaves an
          // empty path. Either way the flood's state goes back to rest first.
          for (int i = G::tid(); i < nt; i += G::threads()) a.dist[__ldcg(L4 + i)] = inf();
          if (G::first()) s_work[1] += nt;
          if (threadIdx.x == 0 && !ordered) sh.skipped += 1;  // every CTA keeps its own copy
          G::sync();
          if (ordered) break;
          continue;
        }
        // walk (one warp of the first CTA), then reset the flood's state over the voxels it touched
        if (G::rank() == 0 && threadIdx.x < 32) {
          const int n = backtrace(a, sh, rb, t, store + used, store_cap - used);
          if (threadIdx.x == 0) L->len = n;
        }
        G::sync();
        const float D = __uint_as_float(unsigned(rb >> 32));
        unsigned settled = 0;
        for (int i = G::tid(); i < nt; i += G::threads()) {
          const int v = __ldcg(L4 + i);
          settled += __ldcg(a.dist + v) <= D;
          a.dist[v] = inf();
        }
        settled = __reduce_add_sync(kFull, settled);
        if ((threadIdx.x & 31) == 0) atomicAdd(&s_work[0], (unsigned long long)settled);
        if (G::first()) s_work[1] += nt;
        G::sync();
        lap(2);
      } else {  // the walk to the root through the parents' field
        if (G::rank() == 0 && threadIdx.x < 32) {
          const int n = parent_walk(a, sh, t, sh.root, store + used, store_cap - used);
          if (threadIdx.x == 0) L->len = n;
        }
        G::sync();
        lap(2);
      }
      if (step == 2) {
        len = vload(&L->len);
        if (sh.soma_radius >= 0.0 && len > 0) {
          if (G::rank() == 0 && threadIdx.x < 32) {
            const int n = soma_trim(a, sh, store + used, len, sh.root, sh.soma_radius, a.fix_branching != 0,
                                    store_cap - used);
            if (threadIdx.x == 0) L->len = n;
          }
          G::sync();
          len = vload(&L->len);
        }
        if (len < 0) { status = kStoreFull; break; }
        if (paths >= rec_cap) { status = kRecordsFull; break; }
      }
      const bool ball = step == 0;
      if (threadIdx.x == 0) {  // the reach of the invalidation's sources (the soma's for its ball)
        sh.rscale = ball ? a.soma_scale : a.scale;
        sh.rconst = ball ? a.soma_constant : a.constant;
      }
      __syncthreads();
      if (!invalidate<C, W>(a, sh, L, store + used, len, L0, L1, L2, L3, L4, L5, wide)) {
        status = kBudget;
        break;
      }
      if (ball) {
        if (G::first()) s_work[2] += vload(&L->n_touch);
        if (threadIdx.x == 0) sh.step = a.fix_branching ? 2 : 1;  // every CTA of the group moves on
        G::sync();
        continue;
      }
      if (G::first()) { s_work[2] += vload(&L->n_touch); s_work[3] += 1; }
      lap(3);
      if (a.fix_branching)
        for (int i = G::tid(); i < len; i += G::threads()) a.pdrf[__ldcg(store + used + i)] = 0.0f;
      else
        for (int i = G::tid(); i < len; i += G::threads()) atomicOr(a.flags + __ldcg(store + used + i), kOnPath);
      if (G::first()) { rec_start[paths] = int(used); rec_len[paths] = len; }
      G::sync();
      used += len;
      ++paths;
    }
    if (!a.fix_branching) {  // the parents' field and the path marks go back to rest
      for (int i = G::tid(); i < sh.count; i += G::threads()) a.dist[a.vox[sh.begin + i]] = inf();
      for (long long i = G::tid(); i < used; i += G::threads()) atomicAnd(a.flags + __ldcg(store + i), ~kOnPath);
      G::sync();
    }
    if (G::first()) {
      a.status[o] = status;
      a.npaths[o] = int(paths);
      a.nstore[o] = int(used);
      unsigned long long *pr = a.profile + 8LL * o;
      pr[0] = s_prof[0]; pr[1] = now_ns();
      for (int q = 0; q < 4; ++q) pr[2 + q] = s_prof[2 + q];
      pr[6] = L->rounds & 0xFFFFFFFFull; pr[7] = L->rounds >> 32;
    }
    G::sync();
  }
  if (threadIdx.x < 4 && s_work[threadIdx.x]) atomicAdd(a.work + threadIdx.x, s_work[threadIdx.x]);
}

// The first a.lone_first clusters start on the small objects (each CTA alone, largest first) and
// then join the large ones; the others take the large objects first. So the longest lone-CTA
// objects run beside the clusters' objects from the start instead of after them. (C == 1: a launch
// without large objects.)
template <int C, int W>
__global__ void __launch_bounds__(W, kEngineThreads / W) trace_kernel(const __grid_constant__ EngineArgs a) {
  if constexpr (C == 1) trace_loop<1, W>(a, false);
  else if (int(blockIdx.x) / C < a.lone_first) {
    trace_loop<1, W>(a, false);
    trace_loop<C, W>(a, true);
  } else {
    trace_loop<C, W>(a, true);
    trace_loop<1, W>(a, false);
  }
}

// A kernel, its CTAs' number in a cluster and threads.
struct Variant {
  const void *kernel;
  int ctas, threads;
  int queue_bytes() const { return kQueueBytes<1> * threads; }
};

cudaLaunchConfig_t cluster_config(int clusters, const Variant &k, cudaStream_t stream, cudaLaunchAttribute *attr) {
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(unsigned(clusters * k.ctas));
  config.blockDim = dim3(unsigned(k.threads));
  config.dynamicSmemBytes = size_t(k.queue_bytes());
  config.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(k.ctas);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  config.attrs = attr;
  config.numAttrs = 1;
  return config;
}

// Resident clusters of a kernel on the current device (queried once per device and kernel: the
// query costs far more than a launch).
int resident_clusters(const Variant &k, cudaStream_t stream) {
  static std::mutex lock;
  static std::map<std::pair<int, const void *>, int> known;
  int device = 0;
  BK_CUDA(cudaGetDevice(&device));
  std::lock_guard<std::mutex> guard(lock);
  auto it = known.find({device, k.kernel});
  if (it != known.end()) return it->second;
  // once per device and kernel, before its first launch
  BK_CUDA(cudaFuncSetAttribute(k.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, k.queue_bytes()));
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t probe = cluster_config(1, k, stream, attr);
  int cap = 1;
  BK_CUDA(cudaOccupancyMaxActiveClusters(&cap, k.kernel, &probe));
  known[{device, k.kernel}] = cap;
  return cap;
}

// As many clusters as are resident at once (no more than the work needs).
void launch(const Variant &k, const EngineArgs &a, int nbig, cudaStream_t stream, int lone_percent = 0) {
  EngineArgs args = a;
  args.nbig = nbig;
  void *kargs[] = {&args};
  cudaLaunchAttribute attr[1];
  const int cap = std::max(1, resident_clusters(k, stream) * std::min(100, std::max(1, a.grid_percent)) / 100);
  const long long need = nbig + (a.nobj - nbig + k.ctas - 1) / k.ctas;
  const int clusters = int(std::max(1LL, std::min<long long>(cap, need)));
  args.lone_first = nbig > 0 && nbig < a.nobj ? clusters * lone_percent / 100 : 0;
  cudaLaunchConfig_t config = cluster_config(clusters, k, stream, attr);
  BK_CUDA(cudaLaunchKernelExC(&config, k.kernel, kargs));
}

// The tiny objects in a launch of their own after the others'.
int launch_all(const Variant &k, const Variant &tiny, const EngineArgs &a, int nbig, cudaStream_t stream,
               int lone_percent = 0) {
  EngineArgs part = a;
  part.nobj = a.nobj - a.ntiny;
  if (part.nobj > 0) launch(k, part, nbig, stream, lone_percent);
  if (a.ntiny == 0) return 1;
  const int rest = part.nobj;
  part.nobj = a.ntiny;
  part.schedule = a.schedule + rest;
  part.queue = a.queue + 1;
  launch(tiny, part, 0, stream);
  return rest > 0 ? 2 : 1;
}

}  // namespace

// The engine's resident CTAs on the current device.
static long long resident_ctas() {
  static std::mutex lock;
  static std::map<int, long long> known;
  int device = 0;
  BK_CUDA(cudaGetDevice(&device));
  std::lock_guard<std::mutex> guard(lock);
  auto it = known.find(device);
  if (it == known.end()) {
    int sms = 1, per_sm = 1;
    BK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    BK_CUDA(cudaFuncSetAttribute(trace_kernel<kClusterCtas, kEngineThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kQueueBytes<kEngineThreads>));
    BK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, trace_kernel<kClusterCtas, kEngineThreads>,
                                                          kEngineThreads, kQueueBytes<kEngineThreads>));
    it = known.emplace(device, std::max(1LL, (long long)sms * per_sm)).first;
  }
  return it->second;
}

long long voxel_share(long long foreground) { return foreground / resident_ctas(); }

long long trace_cluster_voxels(long long foreground) {
  return std::max(kTraceClusterFloor, voxel_share(foreground) * 3 / 2);
}

long long prepare_cluster_voxels(long long foreground) {
  const long long share = voxel_share(foreground);
  return std::max(kPrepareClusterFloor, share >= kPrepareWholeShare ? share : share / 2);
}

int cluster_ctas(long long largest, long long foreground) {
  return largest * kWideClusterShare >= foreground ? kWideClusterCtas : kClusterCtas;
}

// The kernel for nbig large objects. Without any, CTAs are launched alone: clusters of 4 fit only 132 of the 148
// SMs, since an SM short of a whole cluster in its part of the chip stays idle.
static Variant prepare_variant(int nbig, int ctas) {
  if (nbig == 0) return {(const void *)prepare_kernel<1, kEngineThreads>, 1, kEngineThreads};
  if (ctas == kWideClusterCtas)
    return {(const void *)prepare_kernel<kWideClusterCtas, kEngineThreads>, kWideClusterCtas, kEngineThreads};
  return {(const void *)prepare_kernel<kClusterCtas, kEngineThreads>, kClusterCtas, kEngineThreads};
}
static Variant trace_variant(int nbig, int ctas) {
  if (nbig == 0) return {(const void *)trace_kernel<1, kEngineThreads>, 1, kEngineThreads};
  if (ctas == kWideClusterCtas)
    return {(const void *)trace_kernel<kWideClusterCtas, kEngineThreads>, kWideClusterCtas, kEngineThreads};
  return {(const void *)trace_kernel<kClusterCtas, kEngineThreads>, kClusterCtas, kEngineThreads};
}
static Variant tiny_prepare() { return {(const void *)prepare_kernel<1, kTinyThreads>, 1, kTinyThreads}; }
static Variant tiny_trace() { return {(const void *)trace_kernel<1, kTinyThreads>, 1, kTinyThreads}; }

int launch_prepare(const EngineArgs &a, int nbig, int ctas, cudaStream_t stream) {
  return launch_all(prepare_variant(nbig, ctas), tiny_prepare(), a, nbig, stream);
}

void prepare_engine_launches(int ntiny, int nbig_prepare, int prepare_ctas, int nbig_trace, int trace_ctas,
                             cudaStream_t stream) {
  resident_clusters(prepare_variant(nbig_prepare, prepare_ctas), stream);
  resident_clusters(trace_variant(nbig_trace, trace_ctas), stream);
  if (ntiny == 0) return;
  resident_clusters(tiny_prepare(), stream);
  resident_clusters(tiny_trace(), stream);
}

int launch_trace(const EngineArgs &a, int nbig, int ctas, int lone_percent, cudaStream_t stream) {
  return launch_all(trace_variant(nbig, ctas), tiny_trace(), a, nbig, stream, lone_percent);
}

}  // namespace bk
