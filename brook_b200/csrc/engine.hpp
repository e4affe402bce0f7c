// The object engine: persistent kernels in which one CTA owns one object at a time (objects are
// pulled from a queue, largest first) and runs that object's whole sequential chain inside the
// CTA, so that every round of a flood costs a block barrier instead of a grid barrier:
//   prepare: root search flood + argmax, DAF flood + argmax, the object's PDRF, its root rail;
//   trace:   target, railroad flood, warp backtrace with the dijkstra3d join, claim-order
//            invalidation, rails, repeated until the object has no alive voxel left.
// Objects never read or write another object's voxels (every step is gated by the same-id
// neighbour mask), so concurrent CTAs need no synchronisation with one another.
#pragma once
#include <cstdint>

namespace bk {

// Threads per CTA: one CTA per SM at 64 registers (the trace's loop spills some 70 words of state). A frontier
// voxel is a warp's work, so an object's rounds are as fast as its warps are many, and a lone CTA's
// barrier costs a fraction of a cluster's. On the 512^3 dense workload (trace ms, every object on one
// CTA) 256 threads 57.7, 512 35.7, 1024 29.7.
constexpr int kEngineThreads = 1024;

// Per-voxel flag bits (uint32 per voxel, 0 at rest).
constexpr unsigned kSpillEven = 1u;    // floods: on the spill list of an even round
constexpr unsigned kSpillOdd = 2u;     // floods: on the spill list of an odd round
constexpr unsigned kFront = 4u;        // invalidation: on the next round's spill list
constexpr unsigned kOnPath = 16u;      // without fix_branching: on a stored path of the object

enum EngineStatus : int {
  kOk = 0,
  kBudget = 1,        // a loop bound was reached (never expected; guards against hangs)
  kNoRail = 2,        // no rail reachable from a target
  kStoreFull = 3,     // path store region exhausted (cannot happen on a valid field)
  kRecordsFull = 4,
};

struct EngineArgs {
  // Arenas: volumes laid end to end in one flat index space (one arena per volume of a batch).
  // Arena r starts at arena_offset[r] and has shape arena_dims[3r .. 3r+2]; a voxel's neighbours
  // never leave its arena (the neighbour mask says so).
  const int *arena_offset, *arena_dims;
  const int *obj_arena;  // per object
  const uint32_t *mask;  // same-id neighbour mask per voxel
  const float *dbf;
  float *pdrf;           // penalty; rails are 0
  float *dist;           // railroad distances, +inf at rest
  float *daf;            // DAF, +inf before prepare
  uint32_t *flags;       // 0 at rest
  unsigned long long *key;  // invalidation keys: all ones for a living voxel at rest, 0 for a dead one
  unsigned n;               // voxels of the flat space

  int nobj;
  const int *obj_begin;  // offset of the object's voxels in vox and in the list pool
  const int *obj_count;
  const int *vox;        // voxels of every object, ascending flat index
  const int *schedule;   // processing order (object indices): large objects first, then the rest
  int nbig;              // schedule[0, nbig) run on clusters (set by launch_prepare / launch_trace)
  int lone_first;        // trace: clusters [0, lone_first) take the small objects first
  int ntiny;             // the schedule's last ntiny objects take a launch of small CTAs after the others'
  int *queue;            // three work counters (large, small, tiny), 0 at launch
  int *status;           // per object
  int *lists;            // 6 lists of F ints: list w of object o at lists + w * F + obj_begin[o]
  unsigned long long *wide;  // F entries: object o at wide + obj_begin[o] (a spilled frontier's keys)
  long long F;

  // prepare
  const int *border_root;  // per object: flat index, or -1 (search)
  const float *M;          // per object: float(1 / dbf_max^1.01)
  float pdrf_scale;
  int squarings;           // the exponent is 2^squarings; -1: any other exponent (powf)
  float exponent;
  // fix_branching: each path runs to the nearest rail (the root, then every earlier path). Without
  // it, one SSSP from the root over the PDRF is kept for the object's whole trace and each path
  // walks from its target to the root (trace.cu:151-160, batched_regular.inc:113-152).
  int fix_branching;
  // somata (trace.cu:98-131): per object the free-space radius of its DAF seed (the DBF maximum;
  // 0: none) and the soma radius its paths are trimmed to (< 0: not a soma); the soma's own ball is
  // invalidated first with soma_scale / soma_constant as the reach
  const float *free_radius;
  const double *soma_radius;
  float soma_scale, soma_constant;
  float w[26];             // geometric step weights
  int *root, *target;
  float *max_daf;

  // trace
  const int *order;            // target order of every object at obj_begin
  const int *manual_begin, *manual_count, *manual;  // manual targets in pop order
  const int *after_begin, *after_count, *after;     // targets once no voxel is alive, in pop order
  const long long *max_paths;
  int *store;                  // path vertices, target first
  const long long *store_begin, *store_cap;
  int *rec_start, *rec_len;    // per path: offset in the object's store region, length
  const long long *rec_begin, *rec_cap;
  int *npaths, *nstore;
  // work counters (added over all objects): [0] voxels a railroad settled (distance <= its rail's),
  // [1] voxels a railroad touched, [2] voxels invalidated, [3] paths
  unsigned long long *work;
  // per object (8 entries, nanoseconds of %globaltimer): start, end, time in target search,
  // railroad, backtrace, invalidation; railroad rounds; invalidation rounds
  unsigned long long *profile;
  float wx, wy, wz, scale, constant, delta;
  // A lower cap on the round bounds of every flood (0: none). The bounds guard against a loop
  // that does not end; the cap lets a test make one run out and check that the call fails with
  // kBudget and leaves the device usable.
  long long round_limit;
  // The railroad's band past the nearest deferred voxel: its distance plus rail_band times its
  // penalty (at least 5e-4 of the distance). Any band gives the same distances; wider bands take
  // fewer band ends and more re-relaxations.
  float rail_band;
  // The share (percent) of the device's resident clusters the persistent launches take: below 100
  // they leave CTA slots free for another stream's kernels (a second batch's preamble).
  int grid_percent;
};

// Objects with at least prepare_cluster_voxels voxels (preparation) or trace_cluster_voxels (tracing)
// run on a cluster of CTAs that share the object's frontiers through distributed shared memory;
// smaller objects on one CTA each. A cluster's round pays for its barrier and for remote counters and
// queues, so it spends more CTA-time on an object than a lone CTA, which pays only where the
// object's own chain would outlast an even share of the work over all CTAs. Clusters have
// kClusterCtas CTAs, or kWideClusterCtas when the largest object holds at least 1/kWideClusterShare of
// the foreground (its chain is then the kernel's length whatever else runs beside it).
constexpr int kClusterCtas = 4;
constexpr int kWideClusterCtas = 8;
constexpr long long kWideClusterShare = 16;
int cluster_ctas(long long largest, long long foreground);
// Tracing: one and a half shares of the foreground voxels per resident CTA, at least kTraceClusterFloor.
// Measured (trace ms by the objects' least voxels for a cluster): 512^3 dense (share 190 k) 64 from 30 k, 45 from
// 60 k, 23.3 without; 16 volumes in a batch (56 k) 17.8 from 30 k, 10.4 from 56 k, 8.2 from 80 k, 7.9 from 160 k;
// 256^3 dense (24 k) 11.7 from 33 k and from 80 k, 13.7 from 160 k; 128^3 tubes (3 k; objects up to 61 k) 8.9 from
// 33 k, 9.5 from 80 k; a 48^3 request (objects of 16-31 k) 3.1 at each.
constexpr long long kTraceClusterFloor = 32768;
long long trace_cluster_voxels(long long foreground);
// Preparation, whose floods have frontiers ten times as wide: the share from kPrepareWholeShare on, below it
// half the share, at least kPrepareClusterFloor. Measured (prepare ms by the objects' least voxels for a cluster: half
// the share, the share, one and a half, none): dense volumes with shares of 19 k 2.05, 2.15, 2.16, 3.53; 24 k 2.42, 2.68,
// 2.72, 3.16; 34 k 3.50, 3.41, 2.96, 5.24; 43 k 4.18, 3.83, 3.43, 4.22; 55 k 4.79, 3.90, 3.87, 4.82; 89 k 6.97, 5.05, 5.48,
// 5.80; 129 k 8.47, 6.37, 5.68, 5.68; batches with 40 k 3.66, 2.76, 2.29, 2.07; 62 k 4.92, 3.49, 2.88, 2.91. Half and whole
// shares cross at about 30 k; one and a half were better than the whole by more than 2 % in 15 of 24 workloads from
// 34 k on, and worse in 2 (by 4 and 9 %).
constexpr long long kPrepareClusterFloor = 4096, kPrepareWholeShare = 32768;
long long prepare_cluster_voxels(long long foreground);
// An even share of the foreground voxels over the device's resident CTAs.
long long voxel_share(long long foreground);

// Tiny objects, below kTinyVoxels, take small CTAs, four to an SM, when a call has at least kTinyObjects of them and
// they hold half of its foreground: their chains are a few dozen rounds of barriers and L2 round trips, and a CTA that
// fills an SM serves one object at a time. They are launched after the others, in whose shadow fewer of them cost
// nothing (a batch of 32 volumes, 1795 objects, more than 1024 of them tiny: 20.1 in one launch, 22.2 in two). Measured
// (prepare + trace ms, on large CTAs, on small ones of 256 threads, of 128): 32768 cubes of 6^3 26.5, 8.7, 6.1; 15625 of
// 8^3 19.5, 7.9, 6.5; 4096 of 13^3 11.7, 6.7, 6.4; 2744 of 16^3 13.2, 9.4, 10.2; 1331 of 20^3 10.3, 9.1, 11.1; 2048 of
// 6^3 1.5, 0.6, 0.4.
constexpr int kTinyThreads = 256;
constexpr int kTinyVoxels = 4096, kTinyObjects = 1024;

// One pass of the engine: clusters take schedule[0, nbig) (large objects, largest first), then
// every CTA takes schedule[nbig, nobj - ntiny) alone, then small CTAs the rest. The queue's counters must be zero.
// Returns the launches made.
int launch_prepare(const EngineArgs &a, int nbig, int cluster_ctas, cudaStream_t stream);
// lone_percent: the share of clusters (percent) whose CTAs take small objects first.
int launch_trace(const EngineArgs &a, int nbig, int cluster_ctas, int lone_percent, cudaStream_t stream);
constexpr int kLoneFirstPercent = 10;
// The railroad band's width in penalties of the nearest deferred voxel (EngineArgs::rail_band).
// Measured (trace ms at 0.1, 0.25, 0.5, 0.75, 1, 2, 4): 512^3 dense 30.0, 25.7, 25.5, 26.8, 28.1, 34.7, 55.4; 256^3 dense
// 24.1, 18.3, 17.0, 16.9, 16.8, 17.9, 19.8; one arbor 64.4, 46.1, 40.0, 38.3, 38.3, 38.2, 42.1; a 48^3 request 8.8, 6.1, 5.5,
// 5.4, 5.3, 5.1, 5.4; a batch of 16 10.1, 8.5, 8.0, 8.1, 11.5, 10.7, 19.5. Narrower bands take more band ends, wider
// ones more re-relaxations.
constexpr float kRailBand = 0.5f;
// The device queries the launches above make (resident clusters per kernel), done ahead so that
// a stream capture of the launches holds launches only.
void prepare_engine_launches(int ntiny, int nbig_prepare, int prepare_cluster_ctas, int nbig_trace,
                             int trace_cluster_ctas, cudaStream_t stream);

}  // namespace bk
