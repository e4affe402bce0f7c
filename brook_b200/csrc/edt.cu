// Multi-label anisotropic EDT on sm_100a, three separable passes with the reference's arithmetic
// (edt_kernels.cuh:15-144 of giorgioangel/brook):
//   x: distance to the walls of each run of equal ids, from a float32 table of accumulated
//      spacings (one rounding per step); one warp per x-line, coalesced, with run starts and ends
//      found by warp max/min scans and the starts staged in shared memory;
//   y, z: per run the least of height + squared spacing * squared steps, in float32 by scans over lines in
//      shared memory where that gives the reference's float64 lower envelope of parabolas bit for bit
//      (scan_is_exact), else by that envelope, one thread per line, lines x-consecutive across a warp
//      (coalesced), envelope stacks interleaved across lines; stored as float32;
//   the last pass takes the square root (background: 0).
// The reference compiles the envelope with FMA contraction; its two product-plus-height sums are
// written as explicit fused operations here, everything else rounds per operation (--fmad=false).
#include <algorithm>
#include <climits>
#include <cmath>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "kernels.hpp"

namespace bk {
namespace {

constexpr int kWarpsX = 4;
// The x pass's dynamic shared memory (kWarpsX line starts per CTA) is at most this.
constexpr size_t kEdtXMaxSmem = 200 * 1024;

// bb (here and in the envelope passes): walls beyond the line's ends, bit 0 before the first voxel,
// bit 1 after the last (a black border sets both).
template <class L>
__global__ void edt_x(const L *__restrict__ ids, float *__restrict__ D, Dims d, const float *__restrict__ acc, int bb,
                      int finish) {
  using Id = std::conditional_t<sizeof(L) == 8, unsigned long long, uint32_t>;  // what a shuffle carries
  extern __shared__ int s_start[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long line = (long long)blockIdx.x * kWarpsX + warp;
  if (line >= (long long)d.sy * d.sz) return;
  const int sx = d.sx;
  int *start = s_start + warp * sx;
  const long long base = line * sx;
  int carry_start = 0;
  Id carry_label = 0;
  for (int c0 = 0; c0 < sx; c0 += 32) {
    const int p = c0 + lane;
    const bool in = p < sx;
    const Id lab = in ? Id(ids[base + p]) : Id(0);
    Id prev = __shfl_up_sync(0xFFFFFFFFu, lab, 1);
    if (lane == 0) prev = carry_label;
    int st = (in && (p == 0 || lab != prev)) ? p : -1;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_up_sync(0xFFFFFFFFu, st, off);
      if (lane >= off) st = max(st, o);
    }
    st = max(st, carry_start);
    if (in) start[p] = st;
    carry_start = __shfl_sync(0xFFFFFFFFu, st, 31);
    carry_label = __shfl_sync(0xFFFFFFFFu, lab, 31);
  }
  __syncwarp();
  int carry_end = sx - 1;
  Id carry_next = 0;
  for (int c0 = ((sx - 1) / 32) * 32; c0 >= 0; c0 -= 32) {
    const int p = c0 + lane;
    const bool in = p < sx;
    const Id lab = in ? Id(ids[base + p]) : Id(0);
    Id next = __shfl_down_sync(0xFFFFFFFFu, lab, 1);
    if (lane == 31) next = carry_next;
    int en = (in && (p == sx - 1 || lab != next)) ? p : INT_MAX;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_down_sync(0xFFFFFFFFu, en, off);
      if (lane + off < 32) en = min(en, o);
    }
    en = min(en, carry_end);
    if (in) {
      const int c = start[p];
      float best = __uint_as_float(BK_INF_BITS);
      if (c > 0 || (bb & 1)) { const float dd = acc[p - c + 1]; const float v = __fmul_rn(dd, dd); if (v < best) best = v; }
      if (en < sx - 1 || (bb & 2)) { const float dd = acc[en + 1 - p]; const float v = __fmul_rn(dd, dd); if (v < best) best = v; }
      if (finish) best = lab == 0 ? 0.0f : sqrtf(best);
      D[base + p] = best;
    }
    carry_end = __shfl_sync(0xFFFFFFFFu, en, 0);
    carry_next = __shfl_sync(0xFFFFFFFFu, lab, 0);
  }
}

// Lets every edt_x launch of this device use up to kEdtXMaxSmem of dynamic shared memory. The
// limit is a process-wide attribute of the kernel: set per call to the call's own need, it races
// with other threads' launches of other extents (a launch above the limit another thread just
// set fails), so it is raised once per device to the bound every launch is checked against.
void allow_edt_x_smem() {
  static std::mutex lock;
  static bool raised[256] = {};
  int device = 0;
  BK_CUDA(cudaGetDevice(&device));
  if (device < 0 || device >= 256) throw std::invalid_argument("device index out of range");
  std::lock_guard<std::mutex> guard(lock);
  if (raised[device]) return;
  for (const void *kernel : {(const void *)edt_x<uint8_t>, (const void *)edt_x<uint16_t>, (const void *)edt_x<uint32_t>,
                             (const void *)edt_x<uint64_t>})
    BK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEdtXMaxSmem));
  raised[device] = true;
}

// One line of the y or z pass: n voxels from `base` with `stride`. Stacks V/H/Z are interleaved:
// entry k of this thread's stack is at [k * pitch]. One streaming sweep: ids and heights are read
// four voxels ahead of use (independent loads, so their latency overlaps the envelope work), a run
// ends where the id changes, and the top of the stack is kept in registers, so that only a pop
// reads the stack back from memory. The envelope is the reference's per run: parabolas are
// placed in order with the same float64 operations, and the fill walks the stack forward.
__device__ void envelope_line(const uint32_t *__restrict__ ids, float *__restrict__ D, long long base, long long stride,
                              int n, float w, int bb, int *V, float *H, double *Z, long long pitch, int finish) {
  const double w2 = (double)__fmul_rn(w, w);
  const float kInf = __uint_as_float(BK_INF_BITS);
  int c = 0;        // first voxel of the current run
  uint32_t L = 0;   // its id
  int k = -1;       // stack top (-1: empty)
  int vt = 0;       // the top entry, also in memory
  float ht = 0.0f;
  double zt = 0.0;
  auto push = [&](int at, int v, float h, double z) {
    V[(long long)at * pitch] = v; H[(long long)at * pitch] = h; Z[(long long)at * pitch] = z;
    vt = v; ht = h; zt = z;
  };
  // the parabola of height ph at p joins the lower envelope
  auto place = [&](int p, double ph) {
    while (k >= 0) {
      const double num = __dsub_rn(__fma_rn(__dmul_rn(w2, (double)p), (double)p, ph),
                                   __fma_rn(__dmul_rn(w2, (double)vt), (double)vt, (double)ht));
      const double sv = __ddiv_rn(num, __dmul_rn(__dmul_rn(2.0, w2), __dsub_rn((double)p, (double)vt)));
      if (sv <= zt) {
        if (--k >= 0) {
          vt = V[(long long)k * pitch]; ht = H[(long long)k * pitch]; zt = Z[(long long)k * pitch];
        }
      } else {
        ++k;
        push(k, p, (float)ph, sv);
        return;
      }
    }
    k = 0;
    push(0, p, (float)ph, -1e300);
  };
  // the run [c, e] ends; rightw: a wall follows it
  auto finish_run = [&](int e, bool rightw) {
    if (L == 0) {
      if (finish)
        for (int q = c; q <= e; ++q) D[base + (long long)q * stride] = 0.0f;
      return;
    }
    if (rightw) place(e + 1, 0.0);
    if (k < 0) {
      for (int q = c; q <= e; ++q) D[base + (long long)q * stride] = kInf;
      return;
    }
    // entry kk serves the voxels q up to Z[kk + 1] (the last entry: the rest); the next entry is
    // read while this one's voxels are written
    int q = c;
    int vk = V[0];
    float hk = H[0];
    double zn = k > 0 ? Z[pitch] : 0.0;
    for (int kk = 0; q <= e; ++kk) {
      int vn = 0;
      float hn = 0.0f;
      double znn = 0.0;
      if (kk < k) {
        vn = V[(long long)(kk + 1) * pitch];
        hn = H[(long long)(kk + 1) * pitch];
        if (kk + 1 < k) znn = Z[(long long)(kk + 2) * pitch];
      }
      for (; q <= e && (kk == k || !(zn < (double)q)); ++q) {
        const double dq = __dsub_rn((double)q, (double)vk);
        float v = __double2float_rn(__fma_rn(__dmul_rn(w2, dq), dq, (double)hk));
        if (finish) v = sqrtf(v);
        D[base + (long long)q * stride] = v;
      }
      vk = vn; hk = hn; zn = znn;
    }
  };
  auto step = [&](int p, uint32_t lab, float hf) {
    if (p == 0 || lab != L) {
      if (p > 0) finish_run(p - 1, true);
      c = p;
      L = lab;
      k = -1;
      if (L != 0 && (c > 0 || (bb & 1))) { k = 0; push(0, c - 1, 0.0f, -1e300); }
    }
    if (L != 0 && hf < kInf) place(p, (double)hf);
  };
  auto id_at = [&](int p) { return p < n ? ids[base + (long long)p * stride] : 0u; };
  auto d_at = [&](int p) { return p < n ? D[base + (long long)p * stride] : 0.0f; };
  uint32_t a0 = id_at(0), a1 = id_at(1), a2 = id_at(2), a3 = id_at(3);
  float f0 = d_at(0), f1 = d_at(1), f2 = d_at(2), f3 = d_at(3);
  for (int p = 0; p < n; p += 4) {
    const uint32_t b0 = id_at(p + 4), b1 = id_at(p + 5), b2 = id_at(p + 6), b3 = id_at(p + 7);
    const float g0 = d_at(p + 4), g1 = d_at(p + 5), g2 = d_at(p + 6), g3 = d_at(p + 7);
    step(p, a0, f0);
    if (p + 1 < n) step(p + 1, a1, f1);
    if (p + 2 < n) step(p + 2, a2, f2);
    if (p + 3 < n) step(p + 3, a3, f3);
    a0 = b0; a1 = b1; a2 = b2; a3 = b3;
    f0 = g0; f1 = g1; f2 = g2; f3 = g3;
  }
  finish_run(n - 1, (bb & 2) != 0);
}

// Line `line` of the y (axis 1) or z (axis 2) pass of a (sx, sy, sz) volume at `offset`.
__device__ __forceinline__ bool line_of(long long line, long long offset, Dims d, int axis, long long &base,
                                        long long &stride, int &n) {
  const long long x = line % d.sx, rest = line / d.sx;
  if (axis == 1) {
    if (rest >= d.sz) return false;
    base = offset + x + (long long)d.sx * d.sy * rest; stride = d.sx; n = d.sy;
  } else {
    if (rest >= d.sy) return false;
    base = offset + x + (long long)d.sx * rest; stride = (long long)d.sx * d.sy; n = d.sz;
  }
  return true;
}

__global__ void edt_envelope(const uint32_t *__restrict__ ids, float *__restrict__ D, Dims d, int axis, float w, int bb,
                             long long line0, long long nbatch, int *__restrict__ Vs, float *__restrict__ Hs,
                             double *__restrict__ Zs, int finish) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= nbatch) return;
  long long base, stride;
  int n;
  if (!line_of(line0 + tid, 0, d, axis, base, stride, n)) return;
  envelope_line(ids, D, base, stride, n, w, bb, Vs + tid, Hs + tid, Zs + tid, nbatch, finish);
}

// The y pass of a stack of 2D images in groups of `per_group` slices, each group with its own
// spacing w[group] (the border targets' face stack: one group per axis pair).
struct GroupSpacing {
  float w[3];
};
__global__ void edt_envelope_groups(const uint32_t *__restrict__ ids, float *__restrict__ D, Dims d, GroupSpacing gs,
                                    int per_group, int bb, long long line0, long long nbatch, int *__restrict__ Vs,
                                    float *__restrict__ Hs, double *__restrict__ Zs) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= nbatch) return;
  long long base, stride;
  int n;
  const long long line = line0 + tid;
  if (!line_of(line, 0, d, 1, base, stride, n)) return;
  const int group = int((line / d.sx) / per_group);
  envelope_line(ids, D, base, stride, n, gs.w[group], bb, Vs + tid, Hs + tid, Zs + tid, nbatch, 1);
}

// The y or z pass of several volumes of one flat index space in one launch: volume v's lines are
// [line_begin[v], line_begin[v + 1]) of the launch's line space.
struct EnvelopeVolume {
  long long offset, line_begin;
  int sx, sy, sz, bb;
};

__global__ void edt_envelope_volumes(const uint32_t *__restrict__ ids, float *__restrict__ D,
                                     const EnvelopeVolume *__restrict__ vols, int nvol, int axis, float w,
                                     long long line0, long long nbatch, int *__restrict__ Vs, float *__restrict__ Hs,
                                     double *__restrict__ Zs, int finish) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= nbatch) return;
  const long long line = line0 + tid;
  int lo = 0, hi = nvol - 1;  // the last volume whose first line is <= line
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (vols[mid].line_begin <= line) lo = mid; else hi = mid - 1;
  }
  const EnvelopeVolume v = vols[lo];
  long long base, stride;
  int n;
  if (!line_of(line - v.line_begin, v.offset, Dims{v.sx, v.sy, v.sz}, axis, base, stride, n)) return;
  envelope_line(ids, D, base, stride, n, w, v.bb, Vs + tid, Hs + tid, Zs + tid, nbatch, finish);
}

// ---------------------------------------------------------------------------------------------
// The y and z passes by bounded scans: a voxel's distance is the least of h(p) + w2 (q - p)^2 over its
// run and of w2 j^2 to the run's walls, looked for outwards from q until w2 j^2 alone is no better.
// Every value is one fused multiply-add in float32 (w2, j^2 and h are float32 values), that is the
// exact sum rounded once, and rounding keeps the order, so the least rounded value is the rounded
// least value. The envelope's float64 values are those sums too wherever scan_is_exact holds: its
// numerators and products are then exact, and an intersection that is not a whole voxel lies farther
// from it than the division rounds, so that each voxel is served by a parabola that is least there.
//
// A CTA holds 32 x-adjacent whole lines in shared memory (4 bytes a voxel: the height, whose sign bit
// says that a run starts here; background: all ones), so the pass reads ids and heights once, writes once
// and keeps no stacks in memory (the envelope's: 16 bytes a voxel written and read back). A lane owns
// a column, so the banks never conflict. The scan is bound by its two shared loads a step; its length is
// the distance found, a few voxels in segmentations. Past kNearSteps it goes by blocks of 32 voxels,
// skipping those whose least height cannot improve (0 where a run starts in the block, but for the line's first):
// solid volumes cost n / 32 steps instead of n. A voxel farther from the walls seen so far than the near steps
// passes over its own block by the same rule, without near steps: with near steps always, thick boxes took longer
// than with the envelope (a 384^3 box's EDT at (1, 1, 1): envelope 4.9 ms, near steps always 6.8, now 3.0; the three
// passes of a 512^3 volume without a wall 22.2 -> 4.3, of 512 cells in 320^3 1.45 -> 1.49).
constexpr int kScanCols = 32, kScanBlock = 32, kNearSteps = 24;
constexpr unsigned kScanBackground = 0xFFFFFFFFu, kScanStart = 0x80000000u;
constexpr size_t kScanMaxSmem = 220 * 1024;

// A volume's tiles are [tile_begin, next tile_begin) of the launch's; bb as in the envelope passes.
struct ScanVolume {
  long long offset;
  int tile_begin, sx, sy, sz, bb;
  float w;
};
constexpr int kScanInline = 4;  // volumes described by the launch's parameters; more: by a table in memory
struct ScanVolumes {
  ScanVolume few[kScanInline];
  const ScanVolume *many;
  int count;
};

__host__ __device__ inline int scan_blocks(int n) { return (n + kScanBlock - 1) / kScanBlock; }
inline size_t scan_smem(int n) { return size_t(n + scan_blocks(n)) * kScanCols * sizeof(float); }

template <class L>
__global__ void __launch_bounds__(512) edt_scan(const L *__restrict__ ids, float *__restrict__ D,
                                                const __grid_constant__ ScanVolumes vols, int axis, int finish) {
  extern __shared__ unsigned s_line[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const ScanVolume *table = vols.many ? vols.many : vols.few;
  int lo = 0, hi = vols.count - 1;  // the last volume whose first tile is at or before this one
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (table[mid].tile_begin <= int(blockIdx.x)) lo = mid; else hi = mid - 1;
  }
  const ScanVolume v = table[lo];
  const int across = (v.sx + kScanCols - 1) / kScanCols, tile = int(blockIdx.x) - v.tile_begin;
  const int x = (tile % across) * kScanCols + lane;
  const long long rest = tile / across;  // z (y pass) or y (z pass)
  const int n = axis == 1 ? v.sy : v.sz;
  const long long stride = axis == 1 ? v.sx : (long long)v.sx * v.sy;
  const long long base = v.offset + x + (axis == 1 ? (long long)v.sx * v.sy : (long long)v.sx) * rest;
  const bool in = x < v.sx;
  const int blocks = scan_blocks(n);
  unsigned *column = s_line + lane;
  float *least = reinterpret_cast<float *>(s_line + n * kScanCols) + lane;  // per block of the column
  // a warp loads whole blocks of 32 rows, so that a row's previous id is in a register
  for (int b = warp; b < blocks; b += warps) {
    const int p0 = b * kScanBlock, p1 = min(n, p0 + kScanBlock);
    L before = in ? ids[base + max(p0 - 1, 0) * stride] : L(0);
    float m = __uint_as_float(BK_INF_BITS);
#pragma unroll 8
    for (int p = p0; p < p1; ++p) {
      const L id = in ? ids[base + p * stride] : L(0);
      const float h = in ? D[base + p * stride] : 0.0f;
      const bool turn = id != before, start = p == 0 || turn;
      before = id;
      m = fminf(m, turn ? 0.0f : h);
      column[p * kScanCols] = id == 0 ? kScanBackground : (__float_as_uint(h) | (start ? kScanStart : 0u));
    }
    least[b * kScanCols] = m;
  }
  __syncthreads();
  if (!in) return;
  const float w2 = __fmul_rn(v.w, v.w), distant = __fmul_rn(w2, float(kNearSteps * kNearSteps));
  for (int q = warp; q < n; q += warps) {
    const unsigned own = column[q * kScanCols];
    if (own == kScanBackground) {
      if (finish) D[base + q * stride] = 0.0f;
      continue;
    }
    float best = __uint_as_float(own & ~kScanStart);
    // the low side goes on while the run started below the voxels seen, the high side until a start
    bool low = true, high = true;
    unsigned seen = own;
    int below = 1, above = 0;  // each side's next step
    if (best > distant) {
      const int b = q / kScanBlock;
      if (__fadd_rn(w2, least[b * kScanCols]) >= best) {
        below = q - b * kScanBlock + 1;
        seen = b == 0 ? kScanStart : 0u;
        above = (b + 1) * kScanBlock <= n ? (b + 1) * kScanBlock - q : 1;
      }
    }
    // (above is 0 unless the voxel's own block is passed over)
    if (!above) for (int j = 1;; ++j) {
      below = above = j;
      if (j > kNearSteps || !(low || high)) break;
      const float jj = float(j * j), c = __fmul_rn(w2, jj);
      if (c >= best) { low = high = false; break; }
      if (low) {
        const int p = q - j;
        if (seen & kScanStart) {
          if (p >= 0 || (v.bb & 1)) best = fminf(best, c);
          low = false;
        } else {
          seen = column[p * kScanCols];
          best = fminf(best, __fmaf_rn(w2, jj, __uint_as_float(seen & ~kScanStart)));
        }
      }
      if (high) {
        const int p = q + j;
        const unsigned s = p < n ? column[p * kScanCols] : kScanStart;
        if (s & kScanStart) {
          if (p < n || (v.bb & 2)) best = fminf(best, c);
          high = false;
        } else best = fminf(best, __fmaf_rn(w2, jj, __uint_as_float(s)));
      }
    }
    if (low)
      for (int i = below;; ++i) {
        const int p = q - i;
        const float ii = float(i * i), c = __fmul_rn(w2, ii);
        if (c >= best) break;
        if (seen & kScanStart) {
          if (p >= 0 || (v.bb & 1)) best = c;
          break;
        }
        if ((p & (kScanBlock - 1)) == kScanBlock - 1 &&
            __fmaf_rn(w2, ii, least[p / kScanBlock * kScanCols]) >= best) {
          i += kScanBlock - 1;  // no start in the block but the line's: the run goes on below it
          seen = p == kScanBlock - 1 ? kScanStart : 0u;
          continue;
        }
        seen = column[p * kScanCols];
        best = fminf(best, __fmaf_rn(w2, ii, __uint_as_float(seen & ~kScanStart)));
      }
    if (high)
      for (int i = above;; ++i) {
        const int p = q + i;
        const float ii = float(i * i), c = __fmul_rn(w2, ii);
        if (c >= best) break;
        if (p + kScanBlock <= n && (p & (kScanBlock - 1)) == 0 &&
            __fmaf_rn(w2, ii, least[p / kScanBlock * kScanCols]) >= best) {
          i += kScanBlock - 1;
          continue;
        }
        const unsigned s = p < n ? column[p * kScanCols] : kScanStart;
        if (s & kScanStart) {
          if (p < n || (v.bb & 2)) best = c;
          break;
        }
        best = fminf(best, __fmaf_rn(w2, ii, __uint_as_float(s)));
      }
    D[base + q * stride] = finish ? sqrtf(best) : best;
  }
}

// Whether the scans give the envelope's values for spacings w and extents n (entries `axes` of each).
// Every height and w2 is 0 or a float32 of at least the least squared spacing, so a whole multiple of
// that square's last place g; sums stay below V. Numerators and products of the envelope are exact in 53
// bits below V / g = 2^52, and an intersection lies on a whole voxel or at least g / (2 w2 n) from it,
// which a division rounding at 2^-53 n resolves below 8 w2 n^2 / g = 2^53. (512 voxels an axis: spacings up to
// 11 to 16 times apart, by the least one's digits; 1024: up to 5.6 to 8.)
bool scan_is_exact(const float *w, const int *n, int axes) {
  double total = 0, last = INFINITY;
  for (int a = 0; a < axes; ++a) {
    const float w2 = w[a] * w[a];
    if (!(w2 > 1e-30f) || !(w2 < 1e30f)) return false;
    total += double(w2) * (double(n[a]) + 1) * (double(n[a]) + 1) * 1.01;  // 1.01: the x pass's accumulated spacings
    last = std::min(last, std::ldexp(1.0, std::ilogb(w2) - 23));
  }
  return 16.0 * total < last * 9007199254740992.0;
}

// The line must fit a CTA's shared memory (1706 voxels); longer ones take the envelope.
bool scan_fits(int n) { return scan_smem(n) <= kScanMaxSmem; }

void allow_edt_scan_smem() {
  static std::mutex lock;
  static bool raised[256] = {};
  int device = 0;
  BK_CUDA(cudaGetDevice(&device));
  if (device < 0 || device >= 256) throw std::invalid_argument("device index out of range");
  std::lock_guard<std::mutex> guard(lock);
  if (raised[device]) return;
  for (const void *kernel : {(const void *)edt_scan<uint8_t>, (const void *)edt_scan<uint16_t>,
                             (const void *)edt_scan<uint32_t>, (const void *)edt_scan<uint64_t>})
    BK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScanMaxSmem));
  raised[device] = true;
}

// Sets the volumes' tile_begin for a y (axis 1) or z (axis 2) pass; returns the launch's tiles.
long long number_tiles(std::vector<ScanVolume> &vols, int axis, int &longest) {
  long long tiles = 0;
  longest = 1;
  for (auto &v : vols) {
    v.tile_begin = int(std::min<long long>(tiles, INT_MAX));
    tiles += (long long)((v.sx + kScanCols - 1) / kScanCols) * (axis == 1 ? v.sz : v.sy);
    longest = std::max(longest, axis == 1 ? v.sy : v.sz);
  }
  if (tiles > INT_MAX) throw std::invalid_argument("volume too large for the EDT scans");
  return tiles;
}

template <class L>
void launch_edt_scan(cudaStream_t s, const L *ids, float *D, std::vector<ScanVolume> &vols,
                     const ScanVolume *many, long long tiles, int longest, int axis, int finish) {
  ScanVolumes args{};
  args.count = int(vols.size());
  args.many = many;
  if (!many) std::copy(vols.begin(), vols.end(), args.few);
  allow_edt_scan_smem();
  // 16 warps hide the loads of long lines; short ones have too few rows for them
  edt_scan<<<unsigned(tiles), longest > 128 ? 512 : 256, scan_smem(longest), s>>>(ids, D, args, axis, finish);
  BK_CUDA(cudaGetLastError());
}

template <class L>
void edt_scan_pass(Context &ctx, const L *ids, float *D, std::vector<ScanVolume> vols, int axis, bool finish) {
  int longest = 1;
  const long long tiles = number_tiles(vols, axis, longest);
  if (!tiles) return;
  Buffer<ScanVolume> table;
  if (vols.size() > size_t(kScanInline)) table = to_device(ctx, vols);
  launch_edt_scan(ctx.stream(), ids, D, vols, table.data(), tiles, longest, axis, finish ? 1 : 0);
  ++ctx.launches;
}

}  // namespace

void edt(Context &ctx, const uint32_t *ids, VolumeDims vd, const float aniso[3], bool black_border, int dims,
         float *D) {
  const Dims d{vd.sx, vd.sy, vd.sz};
  const long long n = vd.n();
  if (!n) return;
  for (int a = 0; a < 3; ++a)
    if (!(aniso[a] > 0) || !std::isfinite(aniso[a])) throw std::invalid_argument("anisotropy must be finite and positive");
  if (dims < 2 && (vd.sy != 1 || vd.sz != 1)) throw std::invalid_argument("1D EDT of a volume");
  cudaStream_t s = ctx.stream();
  // x pass
  std::vector<float> acc(vd.sx + 2, 0.0f);
  for (size_t k = 1; k < acc.size(); ++k) acc[k] = acc[k - 1] + aniso[0];
  Buffer<float> dacc = to_device(ctx, acc);
  const size_t smem = size_t(kWarpsX) * vd.sx * sizeof(int);
  if (smem > kEdtXMaxSmem) throw std::invalid_argument("x extent too large for the EDT x pass");
  allow_edt_x_smem();
  const long long xlines = (long long)vd.sy * vd.sz;
  const bool only_x = dims == 1 || (vd.sy == 1 && vd.sz == 1 && dims == 1);
  edt_x<<<(unsigned)((xlines + kWarpsX - 1) / kWarpsX), kWarpsX * 32, smem, s>>>(ids, D, d, dacc.data(),
                                                                                black_border ? 3 : 0, only_x ? 1 : 0); ++ctx.launches;
  BK_CUDA(cudaGetLastError());
  const int extent[3] = {vd.sx, vd.sy, vd.sz};
  const bool scans = scan_is_exact(aniso, extent, 3);
  for (int axis = 1; axis < dims; ++axis) {
    const int len = extent[axis];
    if (scans && scan_fits(len)) {
      edt_scan_pass(ctx, ids, D, {{0, 0, d.sx, d.sy, d.sz, black_border ? 3 : 0, aniso[axis]}}, axis, axis == dims - 1);
      continue;
    }
    const long long lines = axis == 1 ? (long long)vd.sx * vd.sz : (long long)vd.sx * vd.sy;
    const long long budget = 4LL << 30;  // bytes of envelope stacks per batch
    long long batch = std::max(1LL, std::min(lines, budget / (16LL * (len + 3))));
    Buffer<int> V(ctx, batch * (len + 3));
    Buffer<float> H(ctx, batch * (len + 3));
    Buffer<double> Z(ctx, batch * (len + 3));
    const int last = axis == dims - 1;
    for (long long l0 = 0; l0 < lines; l0 += batch) {
      const long long nb = std::min(batch, lines - l0);
      edt_envelope<<<blocks_for(nb, 128), 128, 0, s>>>(ids, D, d, axis, aniso[axis], black_border ? 3 : 0, l0, nb,
                                                      V.data(), H.data(), Z.data(), last); ++ctx.launches;
      BK_CUDA(cudaGetLastError());
    }
  }
}

namespace {

template <class L>
void edt_of_labels(Context &ctx, const L *labels, Dims d, const float aniso[3], int bb, float *D) {
  std::vector<float> acc(d.sx + 2, 0.0f);
  for (size_t k = 1; k < acc.size(); ++k) acc[k] = acc[k - 1] + aniso[0];
  Buffer<float> dacc = to_device(ctx, acc);
  allow_edt_x_smem();
  const long long xlines = (long long)d.sy * d.sz;
  edt_x<<<(unsigned)((xlines + kWarpsX - 1) / kWarpsX), kWarpsX * 32, size_t(kWarpsX) * d.sx * sizeof(int),
          ctx.stream()>>>(labels, D, d, dacc.data(), bb, 0);
  ++ctx.launches;
  BK_CUDA(cudaGetLastError());
  for (int axis = 1; axis <= 2; ++axis)
    edt_scan_pass(ctx, labels, D, {{0, 0, d.sx, d.sy, d.sz, bb, aniso[axis]}}, axis, axis == 2);
}

}  // namespace

bool edt_labels(Context &ctx, const void *labels, int dtype, VolumeDims vd, const float aniso[3], bool black_border,
                float *D) {
  const int extent[3] = {vd.sx, vd.sy, vd.sz};
  if (!scan_fits(vd.sy) || !scan_fits(vd.sz) || size_t(kWarpsX) * vd.sx * sizeof(int) > kEdtXMaxSmem) return false;
  for (int a = 0; a < 3; ++a)
    if (!(aniso[a] > 0) || !std::isfinite(aniso[a])) return false;
  if (!scan_is_exact(aniso, extent, 3)) return false;
  const Dims d{vd.sx, vd.sy, vd.sz};
  const int bb = black_border ? 3 : 0;
  switch (label_bytes(dtype)) {
    case 1: edt_of_labels(ctx, static_cast<const uint8_t *>(labels), d, aniso, bb, D); break;
    case 2: edt_of_labels(ctx, static_cast<const uint16_t *>(labels), d, aniso, bb, D); break;
    case 4: edt_of_labels(ctx, static_cast<const uint32_t *>(labels), d, aniso, bb, D); break;
    default: edt_of_labels(ctx, static_cast<const uint64_t *>(labels), d, aniso, bb, D); break;
  }
  return true;
}

void edt_xy_squared(Context &ctx, const uint32_t *ids, VolumeDims vd, const float aniso[3], bool black_border, float *D) {
  const Dims d{vd.sx, vd.sy, vd.sz};
  if (!vd.n()) return;
  cudaStream_t s = ctx.stream();
  std::vector<float> acc(vd.sx + 2, 0.0f);
  for (size_t k = 1; k < acc.size(); ++k) acc[k] = acc[k - 1] + aniso[0];
  Buffer<float> dacc = to_device(ctx, acc);
  const size_t smem = size_t(kWarpsX) * vd.sx * sizeof(int);
  if (smem > kEdtXMaxSmem) throw std::invalid_argument("x extent too large for the EDT x pass");
  allow_edt_x_smem();
  const long long xlines = (long long)vd.sy * vd.sz;
  edt_x<<<(unsigned)((xlines + kWarpsX - 1) / kWarpsX), kWarpsX * 32, smem, s>>>(ids, D, d, dacc.data(),
                                                                                black_border ? 3 : 0, 0);
  ++ctx.launches;
  BK_CUDA(cudaGetLastError());
  const long long lines = (long long)vd.sx * vd.sz;
  const long long batch = std::max(1LL, std::min(lines, (4LL << 30) / (16LL * (vd.sy + 3))));
  Buffer<int> V(ctx, batch * (vd.sy + 3));
  Buffer<float> H(ctx, batch * (vd.sy + 3));
  Buffer<double> Z(ctx, batch * (vd.sy + 3));
  for (long long l0 = 0; l0 < lines; l0 += batch) {
    const long long nb = std::min(batch, lines - l0);
    edt_envelope<<<blocks_for(nb, 128), 128, 0, s>>>(ids, D, d, 1, aniso[1], black_border ? 3 : 0, l0, nb, V.data(),
                                                    H.data(), Z.data(), 0);
    ++ctx.launches;
    BK_CUDA(cudaGetLastError());
  }
}

void edt_z_finish(Context &ctx, const uint32_t *ids, VolumeDims vd, float wz, bool black_border, float *D) {
  const Dims d{vd.sx, vd.sy, vd.sz};
  if (!vd.n()) return;
  cudaStream_t s = ctx.stream();
  const long long lines = (long long)vd.sx * vd.sy;
  const long long batch = std::max(1LL, std::min(lines, (4LL << 30) / (16LL * (vd.sz + 3))));
  Buffer<int> V(ctx, batch * (vd.sz + 3));
  Buffer<float> H(ctx, batch * (vd.sz + 3));
  Buffer<double> Z(ctx, batch * (vd.sz + 3));
  for (long long l0 = 0; l0 < lines; l0 += batch) {
    const long long nb = std::min(batch, lines - l0);
    edt_envelope<<<blocks_for(nb, 128), 128, 0, s>>>(ids, D, d, 2, wz, black_border ? 3 : 0, l0, nb, V.data(),
                                                    H.data(), Z.data(), 1);
    ++ctx.launches;
    BK_CUDA(cudaGetLastError());
  }
}

void edt_planes(Context &ctx, const uint32_t *ids, int W, int H, int groups, int per_group, const float wx[3],
                const float wy[3], float *D) {
  if (groups < 1 || groups > 3 || per_group < 1) throw std::invalid_argument("planar EDT groups out of range");
  const long long slice = (long long)W * H, S = (long long)groups * per_group;
  if (!slice) return;
  cudaStream_t s = ctx.stream();
  const size_t smem = size_t(kWarpsX) * W * sizeof(int);
  if (smem > kEdtXMaxSmem) throw std::invalid_argument("x extent too large for the EDT x pass");
  allow_edt_x_smem();
  // x passes, one per group (its spacing table)
  for (int g = 0; g < groups; ++g) {
    std::vector<float> acc(W + 2, 0.0f);
    for (size_t k = 1; k < acc.size(); ++k) acc[k] = acc[k - 1] + wx[g];
    Buffer<float> dacc = to_device(ctx, acc);
    const long long lines = (long long)H * per_group;
    edt_x<<<(unsigned)((lines + kWarpsX - 1) / kWarpsX), kWarpsX * 32, smem, s>>>(
        ids + slice * per_group * g, D + slice * per_group * g, Dims{W, H, per_group}, dacc.data(), 3, 0);
    ++ctx.launches;
  }
  BK_CUDA(cudaGetLastError());
  // the y pass of every group in one launch
  bool scans = scan_fits(H);
  std::vector<ScanVolume> stacks;
  for (int g = 0; g < groups; ++g) {
    const float spacing[2] = {wx[g], wy[g]};
    const int extent[2] = {W, H};
    scans = scans && scan_is_exact(spacing, extent, 2);
    stacks.push_back({slice * per_group * g, 0, W, H, per_group, 3, wy[g]});
  }
  if (scans) {
    edt_scan_pass(ctx, ids, D, std::move(stacks), 1, true);
    return;
  }
  const long long lines = (long long)W * S;
  const long long budget = 4LL << 30;
  const long long batch = std::max(1LL, std::min(lines, budget / (16LL * (H + 3))));
  Buffer<int> V(ctx, batch * (H + 3));
  Buffer<float> Hb(ctx, batch * (H + 3));
  Buffer<double> Z(ctx, batch * (H + 3));
  GroupSpacing gs{{wy[0], groups > 1 ? wy[1] : 0.0f, groups > 2 ? wy[2] : 0.0f}};
  for (long long l0 = 0; l0 < lines; l0 += batch) {
    const long long nb = std::min(batch, lines - l0);
    edt_envelope_groups<<<blocks_for(nb, 128), 128, 0, s>>>(ids, D, Dims{W, H, int(S)}, gs, per_group, 3, l0, nb,
                                                            V.data(), Hb.data(), Z.data());
    ++ctx.launches;
    BK_CUDA(cudaGetLastError());
  }
}

// The walls of a volume's lines along `axis`: bit 0 the low end, bit 1 the high end.
static int walls(const EdtVolume &v, int axis) {
  if (v.faces < 0) return v.black_border ? 3 : 0;
  return (v.faces >> (2 * axis)) & 3;
}

void edt_volumes(Context &ctx, const uint32_t *ids, const std::vector<EdtVolume> &vols, const float aniso[3], float *D) {
  if (vols.empty()) return;
  for (int a = 0; a < 3; ++a)
    if (!(aniso[a] > 0) || !std::isfinite(aniso[a])) throw std::invalid_argument("anisotropy must be finite and positive");
  cudaStream_t s = ctx.stream();
  int maxx = 1;
  for (const auto &v : vols) maxx = std::max(maxx, v.d.sx);
  // x pass, volume by volume (a warp per line fills the GPU on its own), one spacing table
  std::vector<float> acc(maxx + 2, 0.0f);
  for (size_t k = 1; k < acc.size(); ++k) acc[k] = acc[k - 1] + aniso[0];
  Buffer<float> dacc = to_device(ctx, acc);
  const size_t smem = size_t(kWarpsX) * maxx * sizeof(int);
  if (smem > kEdtXMaxSmem) throw std::invalid_argument("x extent too large for the EDT x pass");
  allow_edt_x_smem();
  for (const auto &v : vols) {
    if (!v.d.n()) continue;
    const long long xlines = (long long)v.d.sy * v.d.sz;
    edt_x<<<(unsigned)((xlines + kWarpsX - 1) / kWarpsX), kWarpsX * 32, smem, s>>>(
        ids + v.offset, D + v.offset, Dims{v.d.sx, v.d.sy, v.d.sz}, dacc.data(), walls(v, 0), 0);
    ++ctx.launches;
  }
  BK_CUDA(cudaGetLastError());
  // y and z passes: every volume's lines in one launch (a thread per line)
  for (int axis = 1; axis <= 2; ++axis) {
    bool scans = true;
    std::vector<ScanVolume> tiled;
    for (const auto &v : vols) {
      if (!v.d.n()) continue;
      const int extent[3] = {v.d.sx, v.d.sy, v.d.sz};
      scans = scans && scan_fits(extent[axis]) && scan_is_exact(aniso, extent, 3);
      tiled.push_back({v.offset, 0, v.d.sx, v.d.sy, v.d.sz, walls(v, axis), aniso[axis]});
    }
    if (scans) {
      edt_scan_pass(ctx, ids, D, std::move(tiled), axis, axis == 2);
      continue;
    }
    std::vector<EnvelopeVolume> table;
    long long lines = 0;
    int len = 1;
    for (const auto &v : vols) {
      if (!v.d.n()) continue;
      table.push_back({v.offset, lines, v.d.sx, v.d.sy, v.d.sz, walls(v, axis)});
      lines += axis == 1 ? (long long)v.d.sx * v.d.sz : (long long)v.d.sx * v.d.sy;
      len = std::max(len, axis == 1 ? v.d.sy : v.d.sz);
    }
    if (!lines) continue;
    Buffer<EnvelopeVolume> dtable = to_device(ctx, table);
    const long long budget = 4LL << 30;  // bytes of envelope stacks per launch
    const long long batch = std::max(1LL, std::min(lines, budget / (16LL * (len + 3))));
    Buffer<int> V(ctx, batch * (len + 3));
    Buffer<float> H(ctx, batch * (len + 3));
    Buffer<double> Z(ctx, batch * (len + 3));
    for (long long l0 = 0; l0 < lines; l0 += batch) {
      const long long nb = std::min(batch, lines - l0);
      edt_envelope_volumes<<<blocks_for(nb, 128), 128, 0, s>>>(ids, D, dtable.data(), int(table.size()), axis,
                                                              aniso[axis], l0, nb, V.data(), H.data(), Z.data(),
                                                              axis == 2 ? 1 : 0);
      ++ctx.launches;
      BK_CUDA(cudaGetLastError());
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The EDT with a fixed device scratch, for callers that cannot allocate device memory: code that
// runs inside another framework's memory budget (a caching allocator or a pre-reserved pool that
// owns the device's free memory), code on a path where an allocation would synchronise the device
// or fail under memory pressure at the worst moment, and embedded callers that keep a fixed
// device-memory footprint. The envelope stacks and the spacing table live in one file-scope
// device array of kFixedScratchBytes (32 MiB) that every GPU loading this library holds until the
// process exits; nothing is allocated per call.
namespace {

constexpr size_t kFixedScratchBytes = size_t(32) << 20;
static __device__ __align__(256) unsigned char g_edt_scratch[kFixedScratchBytes];

// acc[k] = the spacing added k times in float32, one rounding per step (the host loop of edt()).
__global__ void spacing_table(float *acc, int n, float w) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  float a = 0.0f;
  acc[0] = a;
  for (int k = 1; k < n; ++k) {
    a = __fadd_rn(a, w);
    acc[k] = a;
  }
}

std::mutex g_scratch_mutex;
void *g_scratch_address[256];

// The device address of g_edt_scratch on the current device. Host code cannot use the array's
// name as a device address (it is a host-side stand-in), so the address is looked up once per
// device, with that device current, and cached.
void *fixed_scratch() {
  int device = 0;
  BK_CUDA(cudaGetDevice(&device));
  if (device < 0 || device >= 256) throw std::invalid_argument("device index out of range");
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (!g_scratch_address[device]) {
    void *p = nullptr;
    const cudaError_t status = cudaGetSymbolAddress(&p, g_edt_scratch);
    if (status != cudaSuccess) {
      cudaGetLastError();
      throw CudaError(status, "cudaGetSymbolAddress(EDT scratch)");
    }
    g_scratch_address[device] = p;
  }
  return g_scratch_address[device];
}

}  // namespace

size_t edt_fixed_scratch_bytes() { return kFixedScratchBytes; }

// The EDT of uint32 labels (Fortran order) into D on `stream`, using only the fixed scratch. The
// result equals edt() on the labels' component ids (runs of equal labels along a line are runs of
// one component). Nothing in the scratch must start at zero: the spacing table is rewritten by
// every call and every stack entry is written before it is read. Calls that overlap on the GPU
// (two streams, two threads) share the scratch and race.
void edt_fixed_scratch(const uint32_t *labels, VolumeDims vd, const float aniso[3], bool black_border, float *D,
                       cudaStream_t s) {
  const Dims d{vd.sx, vd.sy, vd.sz};
  const long long n = vd.n();
  if (n <= 0) return;
  for (int a = 0; a < 3; ++a)
    if (!(aniso[a] > 0) || !std::isfinite(aniso[a])) throw std::invalid_argument("anisotropy must be finite and positive");
  const size_t smem = size_t(kWarpsX) * vd.sx * sizeof(int);
  const size_t table = (size_t(vd.sx + 2) * sizeof(float) + 255) / 256 * 256;
  const size_t line = 16 * size_t(std::max(vd.sy, vd.sz) + 3);
  if (smem > kEdtXMaxSmem || table + line > kFixedScratchBytes)
    throw std::invalid_argument("volume too large for the EDT's fixed 32 MiB scratch (x extent at most 12800 and "
                                "16 * (max(y, z) extent + 3) + 4 * (x extent + 2) bytes within it)");
  unsigned char *base = static_cast<unsigned char *>(fixed_scratch());
  float *acc = reinterpret_cast<float *>(base);
  spacing_table<<<1, 1, 0, s>>>(acc, vd.sx + 2, aniso[0]);
  BK_CUDA(cudaGetLastError());
  allow_edt_x_smem();
  const long long xlines = (long long)vd.sy * vd.sz;
  edt_x<<<(unsigned)((xlines + kWarpsX - 1) / kWarpsX), kWarpsX * 32, smem, s>>>(labels, D, d, acc,
                                                                                black_border ? 3 : 0, 0);
  BK_CUDA(cudaGetLastError());
  const int extent[3] = {vd.sx, vd.sy, vd.sz};
  const bool scans = scan_is_exact(aniso, extent, 3);
  for (int axis = 1; axis < 3; ++axis) {
    const int len = extent[axis];
    if (scans && scan_fits(len)) {
      std::vector<ScanVolume> volume{{0, 0, d.sx, d.sy, d.sz, black_border ? 3 : 0, aniso[axis]}};
      int longest = 1;
      const long long tiles = number_tiles(volume, axis, longest);
      launch_edt_scan(s, labels, D, volume, nullptr, tiles, longest, axis, axis == 2);
      continue;
    }
    const long long lines = axis == 1 ? (long long)vd.sx * vd.sz : (long long)vd.sx * vd.sy;
    const long long room = (long long)((kFixedScratchBytes - table) / (16 * size_t(len + 3)));
    const long long batch = std::max(1LL, std::min(lines, room));
    // stacks of one batch: Z (8 bytes per entry, 256-aligned after the table), then V, then H
    double *Z = reinterpret_cast<double *>(base + table);
    int *V = reinterpret_cast<int *>(Z + batch * (len + 3));
    float *H = reinterpret_cast<float *>(V + batch * (len + 3));
    for (long long l0 = 0; l0 < lines; l0 += batch) {
      const long long nb = std::min(batch, lines - l0);
      edt_envelope<<<blocks_for(nb, 128), 128, 0, s>>>(labels, D, d, axis, aniso[axis], black_border ? 3 : 0, l0, nb,
                                                      V, H, Z, axis == 2);
      BK_CUDA(cudaGetLastError());
    }
  }
}

}  // namespace bk
