// Projector kernels on transaxial tracks (column.cuh): forward projection,
// backprojection and the fused OSEM sub-iteration, and the images in z
// columns that they read and write.
//
// Blocks of 128 threads: with 256 the serial part of a track's construction
// holds twice the warps (clinical forward projection 10.96 against 10.4 ms).
// The projections run at 48 registers, the backprojection at 64: the gathers'
// latency wants the warps (10.0 against 10.4 ms), the atomics do not (12.1
// against 11.9).  48 registers cost 92 to 356 bytes of spills a thread, at the
// edges of the walks: local accesses are 1.7 % of the instructions.
#include "column.cuh"

#include <algorithm>
#include <cmath>

namespace fir
{
namespace
{
// One of a thread's two LORs: its ends in z and its bin.
struct ColumnLor
{
  bool valid;
  int pair;  // ring pair
  int bin;
  double z1, z2;
};

// The first track of the launch's block number `block`.
__device__ __forceinline__ int first_track(const ColumnPlan& p, int block) { return block / p.blocks * p.per_block; }

// The part of the launch that a warp's group (the block's warps that serve
// its track) traces: ring pairs [begin, end) of one track.
struct ColumnShare
{
  int group, warp;  // track within the block (the last one for warps past it), warp within the group
  int sv, tang;
  int begin, end;
};

__device__ __forceinline__ ColumnShare column_share(const Sino& s, const ColumnPlan& p, int block, int first)
{
  const int warp = threadIdx.x >> 5;
  ColumnShare c;
  c.group = warp / p.warps;
  c.warp = warp - c.group * p.warps;
  const bool any = c.group < p.per_block && first + c.group < p.tracks;
  c.group = min(c.group, p.per_block - 1);
  const int vt = first + c.group;
  c.sv = vt / s.n_tang;
  c.tang = vt - c.sv * s.n_tang;
  c.begin = block % p.blocks * p.share;
  c.end = any ? min(c.begin + p.share, p.pairs) : c.begin;
  return c;
}

// Ring pair r of a track: its segment and plane.  The pairs are those of the
// enumeration's segments in order; with p.interleave the planes of segments
// 2k and 2k + 1 alternate, whose LORs lie half a ring spacing apart, so that
// a warp's lanes share more of a column's sectors.
__device__ __forceinline__ void ring_pair(const Sino& s, const ColumnPlan& p, int r, int& seg, int& axial)
{
  // the enumeration of a segment starts at tracks * its first ring pair
  const int key = r * p.tracks;
  int lo = 0, hi = s.n_segments;
  while (hi - lo > 1)
  {
    const int mid = (lo + hi) >> 1;
    if (s.enum_base[mid] <= key)
      lo = mid;
    else
      hi = mid;
  }
  seg = lo;
  axial = (key - s.enum_base[lo]) / p.tracks;
  const int even = lo & ~1;
  if (p.interleave && even + 1 < s.n_segments)
  {
    const int i = axial + (lo != even ? s.n_axial[even] : 0);
    const int both = 2 * min(s.n_axial[even], s.n_axial[even + 1]);
    // (the longer segment's last planes follow)
    seg = i < both ? even + (i & 1) : (s.n_axial[even] > s.n_axial[even + 1] ? even : even + 1);
    axial = i < both ? i >> 1 : i - (both >> 1);
  }
}

__device__ __forceinline__ int column_bin(const Sino& s, const ColumnShare& c, int subset, int seg, int axial)
{
  return s.seg_base[seg] + ((c.sv * s.n_subsets + subset) * s.n_axial[seg] + axial) * s.n_tang + c.tang;
}

__device__ __forceinline__ ColumnLor column_lor(const Sino& s, const Tables& t, const ColumnPlan& p,
                                                const ColumnShare& c, int subset, bool valid, int r)
{
  ColumnLor l{};
  l.valid = valid;
  if (valid)
  {
    int seg, axial, a1, a2;
    l.pair = r;
    ring_pair(s, p, r, seg, axial);
    crystal_axial(s, seg - s.seg_offset, axial, a1, a2);
    l.z1 = __ldg(t.z + a1);
    l.z2 = __ldg(t.z + a2);
    l.bin = column_bin(s, c, subset, seg, axial);
  }
  return l;
}

// The LORs of a block that cannot use their track, in shared memory: they are
// traced at the end, 32 to a warp, where a few of each warp's lanes would
// hold up the others for a whole walk.
struct Leftover
{
  int* count;
  unsigned* lors;  // their places (block_place)
};

__device__ __forceinline__ Leftover leftover(unsigned char* smem, const ColumnPlan& p)
{
  int* count = reinterpret_cast<int*>(smem + p.per_block * track_bytes(p.cap));
  return Leftover{count, reinterpret_cast<unsigned*>(count + 4)};
}

// The lane's two LORs of the warp's 64.
__device__ __forceinline__ void column_lors(const Sino& s, const Tables& t, const ColumnPlan& p,
                                            const ColumnShare& c, int subset, ColumnLor lor[2])
{
#pragma unroll
  for (int k = 0; k < 2; ++k)
  {
    const int r = c.begin + c.warp * 64 + 32 * k + (int)(threadIdx.x & 31);
    lor[k] = column_lor(s, t, p, c, subset, r < c.end, r);
  }
}

// Where bins that are 0 are skipped and less than a share of them is left, the
// launch leaves those to the queue, one LOR per thread of its own kernel: a
// block would build its tracks for a few LORs, most of its warps' lanes idle.
// (Decided block by block, the two kernels of a launch are each too short to fill
// the GPU: 58 % of a span-3 subset, 281 us against 245 and 239.)  Listing and the
// launch that finds nothing to do cost about 10 us.  Above the share
// * the fused kernel traces all LORs as without skipping, those of zero bins
//   idle.  Sub-iterations at 20, 40, 60 % non-zero bins, queue; packed as below;
//   idle at any share: clinical 0.65, 0.97, 1.34 ms; 0.92, 1.03, 1.52; 1.43; 24 rings
//   355, 521, 702 us; 506, 556, 871; 770; 64 rings 2.2, 3.2, 4.5 ms; 3.0, 3.5, 5.2; 6.0.
// * the backprojection, which gains twice as much on tracks, packs the other
//   ring pairs of a block's tracks: at 12, 20, 50 %, queue; packed; idle: clinical
//   335, 448, 928 us; 352, 386, 580; 750; 24 rings 203, 264, 531; 235, 244, 323; 390; 64
//   rings 1.05, 1.47, 3.2 ms; 1.28, 1.37, 2.1; 3.1.
constexpr int kQueuePercent = 65, kQueuePercentBackward = 16;

// A packing block has twice the ring pairs, as half of the bins are often 0.  A
// batch, which has no queue, packs too (12 problems of 1e5 counts: 11.1 ms; with
// the zero bins' lanes idle 13.2).
constexpr int kPackedTurn = 128;

// counts and pairs are in shared memory.
struct PackedPairs
{
  int* counts;            // of each warp
  unsigned short* pairs;  // of each group, counted from the block's first
};

__device__ __forceinline__ PackedPairs packed_pairs(unsigned char* smem, const ColumnPlan& p)
{
  const Leftover l = leftover(smem, p);
  int* counts = reinterpret_cast<int*>(l.lors + p.per_block * p.share);
  return PackedPairs{counts, reinterpret_cast<unsigned short*>(counts + 8)};
}

// Packs them; returns the number of the group's.  Every thread of the block
// calls this.
__device__ __forceinline__ int pack_nonzero(const Sino& s, const ColumnPlan& p, const ColumnShare& c, int subset,
                                            const float* __restrict__ sino, const PackedPairs& q)
{
  const int lane = threadIdx.x & 31;
  unsigned mask[kPackedTurn / 32];
  int n = 0;
#pragma unroll
  for (int k = 0; k < kPackedTurn / 32; ++k)
  {
    const int i = c.warp * kPackedTurn + 32 * k + lane;
    int seg, axial;
    bool on = false;
    if (c.begin + i < c.end)
    {
      ring_pair(s, p, c.begin + i, seg, axial);
      on = __ldg(sino + column_bin(s, c, subset, seg, axial)) != 0.0f;
    }
    mask[k] = __ballot_sync(0xffffffffu, on);
    n += __popc(mask[k]);
  }
  if (lane == 0)
  {
    q.counts[threadIdx.x >> 5] = n;
  }
  __syncthreads();
  int all = 0, at = c.group * p.share;
  for (int w = 0; w < p.warps && c.end > c.begin; ++w)
  {
    const int m = q.counts[c.group * p.warps + w];
    all += m;
    at += w < c.warp ? m : 0;
  }
#pragma unroll
  for (int k = 0; k < kPackedTurn / 32; ++k)
  {
    if (mask[k] >> lane & 1)
    {
      q.pairs[at + __popc(mask[k] & ((1u << lane) - 1))] = (unsigned short)(c.warp * kPackedTurn + 32 * k + lane);
    }
    at += __popc(mask[k]);
  }
  __syncthreads();
  return all;
}

// Calls trace(lor) for the LORs that the warp's group has packed, 64 at a time,
// two per lane.  Every thread of the block calls this.
template<class Trace>
__device__ __forceinline__ void packed_each(const Sino& s, const Tables& t, const ColumnPlan& p,
                                            const ColumnShare& c, int subset, const float* __restrict__ sino,
                                            unsigned char* smem, Trace&& trace)
{
  const PackedPairs q = packed_pairs(smem, p);
  const int n = pack_nonzero(s, p, c, subset, sino, q);
  for (int i0 = c.warp * 64; i0 < n; i0 += p.warps * 64)
  {
    ColumnLor lor[2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
    {
      const int i = i0 + 32 * k + (int)(threadIdx.x & 31);
      lor[k] = column_lor(s, t, p, c, subset, i < n, i < n ? c.begin + q.pairs[c.group * p.share + i] : 0);
    }
    trace(lor);
  }
}

// Whether the launch that skips zero bins leaves the others to the queue.
__device__ __forceinline__ bool queued(const LorQueue& q) { return q.list != nullptr && __ldg(q.count) < q.room; }

// The general walk in z columns, for the LORs that cannot use their track.
// Not inlined: few lanes take it, and its registers are not the kernel's.
// ok is false for a lane that hit the step bound.
struct GeneralLine
{
  float line;
  int ok;
};

__device__ __noinline__ GeneralLine general_line(const Grid& g, const TrackHead& h, double z1, double z2,
                                           const double* __restrict__ img, int* check)
{
  const double e[6] = {h.x1, h.y1, z1, h.x2, h.y2, z2};
  Walk w{};
  const bool go = siddon_setup<true>(g, e, w);
  float line = 0.0f;
  const bool ok = siddon_walk<true>(g, w, go, [&](bool, int c, double len) {
    line = accumulate(line, len, __ldg(img + (unsigned)c));
  });
  if (!ok)
  {
    flag(check, kCheckWalkGuard);
  }
  return GeneralLine{line, ok ? 1 : 0};
}

__device__ __noinline__ void general_scatter(const Grid& g, const TrackHead& h, double z1, double z2, double value,
                                             float* acc, int* check)
{
  const double e[6] = {h.x1, h.y1, z1, h.x2, h.y2, z2};
  Walk w{};
  const bool go = siddon_setup<true>(g, e, w);
  __builtin_assume(__isGlobal(acc));
  const bool ok = siddon_walk<true>(g, w, go, [&](bool, int c, double len) {
    atomicAdd(acc + c, __double2float_rn(dmul(len, value)));
  });
  if (!ok)
  {
    flag(check, kCheckWalkGuard);
  }
}

// Sets up a lane's two LORs, those that are on; go says which of them use the
// track.  Those that need the general walk are left over.
__device__ __forceinline__ void column_setup(const Grid& g, const ColumnPlan& p, const Track& tr,
                                             const ColumnShare& c, const ColumnLor lor[2], const bool on[2],
                                             const Leftover& left, ColumnLane w[2], bool go[2])
{
#pragma unroll
  for (int k = 0; k < 2; ++k)
  {
    const int kind = on[k] && lor[k].valid && tr.head->crosses
                       ? lane_setup(g, *tr.head, lor[k].z1, lor[k].z2, w[k])
                       : kLorNone;
    go[k] = kind == kLorColumn;
    if (kind == kLorGeneral)
    {
      left.lors[atomicAdd(left.count, 1)] = block_place(p, BlockLor{c.group, lor[k].pair - c.begin});
    }
  }
}

// Calls trace(lor, track) for the leftover LORs of block number `block`.  Every
// thread of the block calls this.
template<class Trace>
__device__ __forceinline__ void column_leftover(const Sino& s, const Tables& t, const ColumnPlan& p, int subset,
                                                int block, int first, unsigned char* smem, const Leftover& left,
                                                Trace&& trace)
{
  __syncthreads();
  for (int i = threadIdx.x; i < *left.count; i += blockDim.x)
  {
    const BlockLor l = block_lor(p, left.lors[i]);
    ColumnShare c;
    c.group = l.group;
    const int vt = first + c.group;
    c.sv = vt / s.n_tang;
    c.tang = vt - c.sv * s.n_tang;
    trace(column_lor(s, t, p, c, subset, true, block % p.blocks * p.share + l.offset),
          track_at(smem, p.cap, c.group));
  }
}

// Line integrals of the image in z columns (VolData.cc:357-371).
__device__ __forceinline__ void column_lines(const Track& tr, const bool go[2], const ColumnLane w[2],
                                             const double* __restrict__ img, float line[2])
{
  LineSum sum[2] = {};
  column_walk(
    tr, w, go, [&](unsigned& at, ColumnState* st) { column_run_line(at, st, img, sum); },
    [&](int k, int c, double len) {
      sum[k].line = accumulate(sum[k].line, sum[k].len, sum[k].value);
      sum[k].len = len;
      sum[k].value = __ldg(img + (unsigned)c);
    });
#pragma unroll
  for (int k = 0; k < 2; ++k)
  {
    line[k] = go[k] ? accumulate(sum[k].line, sum[k].len, sum[k].value) : 0.0f;
  }
}

// acc += value along each LOR (VolData.cc:373-385).
__device__ __forceinline__ void column_scatter(const Track& tr, const bool go[2], const ColumnLane w[2],
                                               const double value[2], float* acc)
{
  __builtin_assume(__isGlobal(acc));
  const bool all = __all_sync(0xffffffffu, go[0] && go[1]);
  column_walk(
    tr, w, go, [&](unsigned& at, ColumnState* st) { column_run_scatter(at, st, acc, value, go, all); },
    [&](int k, int c, double len) { atomicAdd(acc + (unsigned)c, __double2float_rn(dmul(len, value[k]))); });
}

// exp evaluated in double and rounded once: the correctly rounded float
// exponential that FIR's std::exp(float) returns (ProjData.cc:531).
template<FwdEpilogue EP>
__device__ __forceinline__ float epilogue(float line)
{
  if (EP == FwdEpilogue::Exp)
  {
    return (double)line > kEps ? __double2float_rn(exp((double)line)) : 1.0f;
  }
  return line;
}

// projections::forward (projections.cc:15-92), optionally with
// ProjData::exponential (ProjData.cc:514-539).
template<FwdEpilogue EP>
__global__ void __launch_bounds__(256, 5) k_column_forward(const __grid_constant__ Grid g,
                                                           const __grid_constant__ Sino s, Tables t, ColumnPlan p,
                                                           const double* __restrict__ img, float* __restrict__ sino,
                                                           int* check)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int first = first_track(p, (int)blockIdx.x);
  const Leftover left = leftover(smem, p);
  build_tracks(g, s, t, p, s.subset, first, smem, left.count);
  const ColumnShare c = column_share(s, p, (int)blockIdx.x, first);
  const Track tr = track_at(smem, p.cap, c.group);
  ColumnLor lor[2];
  column_lors(s, t, p, c, s.subset, lor);
  ColumnLane w[2] = {};
  bool go[2];
  float line[2];
  const bool on[2] = {true, true};
  column_setup(g, p, tr, c, lor, on, left, w, go);
  column_lines(tr, go, w, img, line);
#pragma unroll
  for (int k = 0; k < 2; ++k)
  {
    if (lor[k].valid)
    {
      sino[lor[k].bin] = epilogue<EP>(line[k]);
    }
  }
  column_leftover(s, t, p, s.subset, (int)blockIdx.x, first, smem, left, [&](const ColumnLor& l, const Track& own) {
    sino[l.bin] = epilogue<EP>(general_line(g, *own.head, l.z1, l.z2, img, check).line);
  });
}

__device__ __forceinline__ float* accumulator_of(const Grid& g, const TrackHead& h, float* acc)
{
  return acc + (h.crosses ? (size_t)h.acc * g.nxy * g.nz : 0);
}

// The sum of the accumulators' elements k (n each).
__device__ __forceinline__ float accumulated(const float* __restrict__ acc, size_t n, size_t k)
{
  static_assert(kColumnAccumulators == 4, "");
  return __fadd_rn(__fadd_rn(acc[k], acc[2 * n + k]), __fadd_rn(acc[n + k], acc[3 * n + k]));
}

// projections::backward (projections.cc:94-184) into the accumulators in z
// columns; sino == nullptr is the all-ones sinogram (projections.cc:186-197).
template<bool kSkip>
__global__ void __launch_bounds__(256, 4) k_column_backward(const __grid_constant__ Grid g,
                                                            const __grid_constant__ Sino s, Tables t, ColumnPlan p,
                                                            const float* __restrict__ sino, float* acc,
                                                            LorQueue queue, int* check)
{
  extern __shared__ __align__(16) unsigned char smem[];
  const int first = first_track(p, (int)blockIdx.x);
  const ColumnShare c = column_share(s, p, (int)blockIdx.x, first);
  if (kSkip && queued(queue))
  {
    return;
  }
  const Leftover left = leftover(smem, p);
  build_tracks(g, s, t, p, s.subset, first, smem, left.count);
  const Track tr = track_at(smem, p.cap, c.group);
  auto trace = [&](const ColumnLor lor[2]) {
    ColumnLane w[2] = {};
    bool go[2];
    double value[2];
    const bool on[2] = {true, true};
#pragma unroll
    for (int k = 0; k < 2; ++k)
    {
      value[k] = lor[k].valid && sino != nullptr ? (double)__ldg(sino + lor[k].bin) : 1.0;
    }
    column_setup(g, p, tr, c, lor, on, left, w, go);
    column_scatter(tr, go, w, value, accumulator_of(g, *tr.head, acc));
  };
  if constexpr (kSkip)
  {
    packed_each(s, t, p, c, s.subset, sino, smem, trace);
  }
  else
  {
    ColumnLor lor[2];
    column_lors(s, t, p, c, s.subset, lor);
    trace(lor);
  }
  column_leftover(s, t, p, s.subset, (int)blockIdx.x, first, smem, left, [&](const ColumnLor& l, const Track& own) {
    const double v = sino != nullptr ? (double)__ldg(sino + l.bin) : 1.0;
    general_scatter(g, *own.head, l.z1, l.z2, v, accumulator_of(g, *own.head, acc), check);
  });
}

// measured / estimated of one bin (reconAlgos.cc:119-150, see osem_lor_body);
// false where nothing is backprojected.
template<bool kWeighted>
__device__ __forceinline__ bool osem_ratio(float line, int bin, const float* __restrict__ sino,
                                           const float* __restrict__ mult, const float* __restrict__ bias, double& q)
{
  const float m = kWeighted ? __ldg(mult + bin) : 1.0f;
  if (kWeighted)
  {
    line = __fmul_rn(line, m);
  }
  if (bias != nullptr)
  {
    line = __fadd_rn(line, __ldg(bias + bin));
  }
  q = 0.0;
  if (!((double)line > kEps))
  {
    return false;
  }
  const float r = __fdiv_rn(__ldg(sino + bin), line);
  q = (double)(kWeighted ? __fmul_rn(r, m) : r);
  return true;
}

// What becomes of bins that are 0.
enum class ZeroBins
{
  Trace,  // not skipped
  Queue,  // their lanes idle, or (see kQueuePercent) the others queued
  Pack    // the others packed
};

// The LORs of block number `block` of one OSEM sub-iteration
// (reconAlgos.cc:119-158, see osem_lor_body): image and accumulators in z
// columns.
template<bool kWeighted, ZeroBins kZero>
__device__ __forceinline__ void column_osem(const Grid& g, const Sino& s, const Tables& t, const ColumnPlan& p,
                                            int subset, int block, const double* __restrict__ img,
                                            const float* __restrict__ sino, const float* __restrict__ mult,
                                            const float* __restrict__ bias, float* acc, const LorQueue& queue,
                                            int* check, unsigned char* smem)
{
  const int first = first_track(p, block);
  const ColumnShare c = column_share(s, p, block, first);
  if (kZero == ZeroBins::Queue && queued(queue))
  {
    return;
  }
  const Leftover left = leftover(smem, p);
  build_tracks(g, s, t, p, subset, first, smem, left.count);
  const Track tr = track_at(smem, p.cap, c.group);
  auto trace = [&](const ColumnLor lor[2], const bool on[2]) {
    ColumnLane w[2] = {};
    bool go[2];
    float line[2];
    column_setup(g, p, tr, c, lor, on, left, w, go);
    column_lines(tr, go, w, img, line);
    double value[2] = {0.0, 0.0};
#pragma unroll
    for (int k = 0; k < 2; ++k)
    {
      go[k] = go[k] && osem_ratio<kWeighted>(line[k], lor[k].bin, sino, mult, bias, value[k]);
    }
    column_scatter(tr, go, w, value, accumulator_of(g, *tr.head, acc));
  };
  bool on[2] = {true, true};
  if constexpr (kZero == ZeroBins::Pack)
  {
    packed_each(s, t, p, c, subset, sino, smem, [&](const ColumnLor lor[2]) { trace(lor, on); });
  }
  else
  {
    ColumnLor lor[2];
    column_lors(s, t, p, c, subset, lor);
#pragma unroll
    for (int k = 0; k < 2; ++k)
    {
      on[k] = kZero == ZeroBins::Trace || (lor[k].valid && __ldg(sino + lor[k].bin) != 0.0f);
    }
    trace(lor, on);
  }
  column_leftover(s, t, p, subset, block, first, smem, left, [&](const ColumnLor& l, const Track& own) {
    const GeneralLine gl = general_line(g, *own.head, l.z1, l.z2, img, check);
    double q;
    if (osem_ratio<kWeighted>(gl.line, l.bin, sino, mult, bias, q) && gl.ok)
    {
      general_scatter(g, *own.head, l.z1, l.z2, q, accumulator_of(g, *own.head, acc), check);
    }
  });
}

template<bool kWeighted, ZeroBins kZero>
__global__ void __launch_bounds__(256, 5) k_column_osem(const __grid_constant__ Grid g,
                                                        const __grid_constant__ Sino s, Tables t, ColumnPlan p,
                                                        const double* __restrict__ img,
                                                        const float* __restrict__ sino,
                                                        const float* __restrict__ mult,
                                                        const float* __restrict__ bias, float* acc,
                                                        LorQueue queue, int* check)
{
  extern __shared__ __align__(16) unsigned char smem[];
  column_osem<kWeighted, kZero>(g, s, t, p, s.subset, (int)blockIdx.x, img, sino, mult, bias, acc, queue, check, smem);
}

// The queue: the enumerated indices of the subset's non-zero bins, as far as
// there is room, and their number.  A block takes a tile of 32 ring pairs x 32
// tangential bins: its warps read along the latter, eight pairs each, and it
// appends track by track, since the LORs of a track run through the same columns.
constexpr int kListPairs = 8, kListWarps = 4;

__global__ void __launch_bounds__(32 * kListWarps) k_list_nonzero(const __grid_constant__ Sino s, ColumnPlan p,
                                                                  const float* __restrict__ sino, LorQueue q)
{
  constexpr unsigned kAll = 0xffffffffu;
  __shared__ int counts[kListWarps][32];
  __shared__ int place;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int across = (s.n_tang + 31) / 32;
  const int tiles = across * ((p.pairs + kListWarps * kListPairs - 1) / (kListWarps * kListPairs));
  const int sv = (int)blockIdx.x / tiles, tile = (int)blockIdx.x - sv * tiles;
  const int tang = tile % across * 32 + lane;
  const int first = (tile / across * kListWarps + warp) * kListPairs;
  int seg, axial;
  ring_pair(s, p, min(first + (lane & (kListPairs - 1)), p.pairs - 1), seg, axial);
  const int bin = s.seg_base[seg] + ((sv * s.n_subsets + s.subset) * s.n_axial[seg] + axial) * s.n_tang;
  const int key = s.enum_base[seg] + (sv * s.n_axial[seg] + axial) * s.n_tang;
  float y[kListPairs];
#pragma unroll
  for (int k = 0; k < kListPairs; ++k)
  {
    const int row = __shfl_sync(kAll, bin, k);
    y[k] = tang < s.n_tang && first + k < p.pairs ? __ldg(sino + row + tang) : 0.0f;
  }
  int n = 0;
#pragma unroll
  for (int k = 0; k < kListPairs; ++k)
  {
    n += y[k] != 0.0f ? 1 : 0;
  }
  counts[warp][lane] = n;
  __syncthreads();
  int own = 0, before = 0;  // entries of the lane's track, and of the warps before this one
#pragma unroll
  for (int w = 0; w < kListWarps; ++w)
  {
    own += counts[w][lane];
    before += w < warp ? counts[w][lane] : 0;
  }
  int end = own;
#pragma unroll
  for (int d = 1; d < 32; d *= 2)
  {
    const int below = __shfl_up_sync(kAll, end, d);
    end += lane >= d ? below : 0;
  }
  if (threadIdx.x == 31)
  {
    place = end > 0 ? atomicAdd(q.count, end) : 0;
  }
  __syncthreads();
  int at = place + end - own + before;
#pragma unroll
  for (int k = 0; k < kListPairs; ++k)
  {
    const int index = __shfl_sync(kAll, key, k) + tang;
    if (y[k] != 0.0f)
    {
      if (at < q.room)
      {
        q.list[at] = index;
      }
      ++at;
    }
  }
}

// The queued LORs (s.list), one per thread, on the same images.  The LORs of a
// track lie side by side in the queue and run through the same columns.
template<bool kWeighted>
__global__ void __launch_bounds__(128, 8) k_queue_osem(const __grid_constant__ Grid g, const __grid_constant__ Sino s,
                                                       Tables t, const double* __restrict__ img,
                                                       const float* __restrict__ sino, const float* __restrict__ mult,
                                                       const float* __restrict__ bias, float* acc, int views,
                                                       LorQueue queue, int* check)
{
  if (!queued(queue))
  {
    return;
  }
  osem_lor_body<kWeighted, double, true>(g, s, s.subset, t, img, img, sino, mult, bias, acc, acc, true,
                                         blockIdx.x * blockDim.x + threadIdx.x, check, -1, views);
}

__global__ void __launch_bounds__(128, 8) k_queue_backward(const __grid_constant__ Grid g,
                                                           const __grid_constant__ Sino s, Tables t,
                                                           const float* __restrict__ sino, float* acc, int views,
                                                           LorQueue queue, int* check)
{
  if (!queued(queue))
  {
    return;
  }
  bool valid = false;
  const int i = enum_index(s, blockIdx.x * blockDim.x + threadIdx.x, valid);
  Walk w{};
  bool go = false;
  double value = 0.0;
  float* to = acc;
  if (valid)
  {
    const Lor l = decode_bin(s, i);
    double e[6];
    lor_ends(s, t, l, e);
    go = siddon_setup<true>(g, e, w);
    value = (double)__ldg(sino + l.bin);
    to += (size_t)column_accumulator(fabs(dsub(e[3], e[0])) > fabs(dsub(e[4], e[1])), l.view / s.n_subsets, views) *
          g.nxy * g.nz;
  }
  const bool ok = siddon_walk<true>(
    g, w, go, [&](bool, int c, double len) { atomicAdd(to + c, __double2float_rn(dmul(len, value))); });
  if (!ok)
  {
    flag(check, kCheckWalkGuard);
  }
}

// The same for the items of a batch (batch.cu), whose work units are the
// blocks of their problems' plans.
template<ZeroBins kZero>
__global__ void __launch_bounds__(kBatchColumnBlock, 10)
  k_batch_column_osem(const BatchProblem* __restrict__ P, const BatchItem* __restrict__ items, int n_items, int* check)
{
  extern __shared__ __align__(16) unsigned char smem[];
  int lo = 0, hi = n_items;
  while (hi - lo > 1)
  {
    const int mid = (lo + hi) >> 1;
    if (__ldg(&items[mid].unit_begin) <= (int)blockIdx.x)
      lo = mid;
    else
      hi = mid;
  }
  const BatchProblem& pb = P[__ldg(&items[lo].problem)];
  column_osem<false, kZero>(pb.g, pb.s, pb.t, pb.plan, __ldg(&items[lo].subset),
                            (int)blockIdx.x - __ldg(&items[lo].unit_begin), pb.wide, pb.sino, nullptr, pb.bias, pb.bp,
                            LorQueue{}, check, smem);
}

// Images between [z][y][x] and z columns, through 32 x 32 tiles of
// (column, slice) in shared memory.  np = nx * ny.
constexpr int kTile = 32, kTileRows = 8;

dim3 column_tiles(int np, int nz)
{
  return dim3((unsigned)((np + kTile - 1) / kTile), (unsigned)((nz + kTile - 1) / kTile));
}

// out = the double copy of in in z columns; the accumulators at acc (or null)
// and the queue's count behind them = 0.
__global__ void __launch_bounds__(kTile * kTileRows) k_to_columns(int np, int nz, const float* __restrict__ in,
                                                                  double* __restrict__ out, float* __restrict__ acc)
{
  __shared__ float tile[kTile][kTile + 1];
  const int p0 = blockIdx.x * kTile, z0 = blockIdx.y * kTile;
  if (acc != nullptr && blockIdx.x + blockIdx.y + threadIdx.x + threadIdx.y == 0)
  {
    *queue_count(acc, (size_t)np * nz) = 0;
  }
  for (int j = threadIdx.y; j < kTile; j += kTileRows)
  {
    const int p = p0 + threadIdx.x, z = z0 + j;
    if (p < np && z < nz)
    {
      tile[j][threadIdx.x] = in[(size_t)z * np + p];
    }
  }
  __syncthreads();
  for (int j = threadIdx.y; j < kTile; j += kTileRows)
  {
    const int z = z0 + threadIdx.x, p = p0 + j;
    if (p < np && z < nz)
    {
      const size_t k = (size_t)p * nz + z;
      out[k] = (double)tile[threadIdx.x][j];
      if (acc != nullptr)
      {
#pragma unroll
        for (int a = 0; a < kColumnAccumulators; ++a)
        {
          acc[(size_t)a * np * nz + k] = 0.0f;
        }
      }
    }
  }
}

// out = the sum of the accumulators at acc in [z][y][x].
__global__ void __launch_bounds__(kTile * kTileRows) k_from_columns(int np, int nz, const float* __restrict__ acc,
                                                                    float* __restrict__ out)
{
  __shared__ float tile[kTile][kTile + 1];
  const int p0 = blockIdx.x * kTile, z0 = blockIdx.y * kTile;
  for (int j = threadIdx.y; j < kTile; j += kTileRows)
  {
    const int z = z0 + threadIdx.x, p = p0 + j;
    if (p < np && z < nz)
    {
      tile[j][threadIdx.x] = accumulated(acc, (size_t)np * nz, (size_t)p * nz + z);
    }
  }
  __syncthreads();
  for (int j = threadIdx.y; j < kTile; j += kTileRows)
  {
    const int p = p0 + threadIdx.x, z = z0 + j;
    if (p < np && z < nz)
    {
      out[(size_t)z * np + p] = tile[threadIdx.x][j];
    }
  }
}

// k_em_update with the backprojection in z columns.
__global__ void __launch_bounds__(kTile * kTileRows) k_em_update_columns(int np, int nz, const float* img, float* out,
                                                                         const float* __restrict__ acc,
                                                                         const float* __restrict__ sens)
{
  __shared__ float tile[kTile][kTile + 1];
  const int p0 = blockIdx.x * kTile, z0 = blockIdx.y * kTile;
  for (int j = threadIdx.y; j < kTile; j += kTileRows)
  {
    const int z = z0 + threadIdx.x, p = p0 + j;
    if (p < np && z < nz)
    {
      tile[j][threadIdx.x] = accumulated(acc, (size_t)np * nz, (size_t)p * nz + z);
    }
  }
  __syncthreads();
  for (int j = threadIdx.y; j < kTile; j += kTileRows)
  {
    const int p = p0 + threadIdx.x, z = z0 + j;
    if (p < np && z < nz)
    {
      const size_t k = (size_t)z * np + p;
      const float b = tile[threadIdx.x][j];
      const float sv = __ldg(sens + k);
      const float q = ((double)b > kEps && (double)sv > kEps) ? __fdiv_rn(b, sv) : 0.0f;
      const float v = img[k];
      out[k] = ((double)v > kEps && (double)q > kEps) ? __fmul_rn(v, q) : 0.0f;
    }
  }
}

// Allows a kernel shared memory above 48 KB.  The limit belongs to the kernel,
// which all contexts and threads share, so that it is always the same one: a
// call that set its own need would take away a larger one that another thread
// has just asked for.  False (and an error for cudaGetLastError) if it fails.
template<typename K>
bool ask_shared(K kernel, size_t bytes)
{
  return bytes <= 48 * 1024 || cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (int)kColumnSharedLimit) == cudaSuccess;
}
}  // namespace

size_t column_smem(const ColumnPlan& p)
{
  const size_t packed = 8 * sizeof(int) + (size_t)p.per_block * p.share * sizeof(unsigned short);
  return (size_t)p.per_block * (track_bytes(p.cap) + p.share * sizeof(unsigned)) + 4 * sizeof(int) +
         (p.skip != 0 && p.turn == kPackedTurn ? packed : 0);
}

int column_blocks(const ColumnPlan& p) { return (p.tracks + p.per_block - 1) / p.per_block * p.blocks; }

ColumnPlan column_plan(const Grid& g, const Sino& s, const double* z, int block, bool skip, bool pack, bool fixed)
{
  ColumnPlan p{};
  for (int k = 0; k < s.n_segments; ++k)
  {
    p.pairs += s.n_axial[k];
  }
  p.tracks = p.pairs > 0 ? s.n_enum / p.pairs : 0;
  p.cap = g.nx + g.ny;
  p.skip = skip ? 1 : 0;
  // neighbouring LORs of a segment lie one ring apart in z, or with a span half
  // a ring
  const double apart = s.n_rings > 1 ? std::fabs(z[2] - z[0]) * (s.span > 1 ? 0.5 : 1.0) : 0.0;
  p.interleave = apart >= 1.6 * g.ext[2] ? 1 : 0;
  p.turn = skip && pack ? kPackedTurn : 64;
  const int warps = std::max((p.pairs + p.turn - 1) / p.turn, 1);
  // a track's warps in equal blocks of nearly the wanted size: the count
  // that leaves the fewest warps idle
  const int want = block / 32;
  int best = want, idle = 1 << 30;
  for (int w : {want, want + 1, want - 1, want + 2})
  {
    if (w >= 1 && w <= 8 && (w == want || !fixed))
    {
      const int off = warps >= w ? (warps + w - 1) / w * w - warps : (w % warps);
      // (compared as a share of all warps)
      if ((long long)off * 64 / std::max(warps, w) < idle)
      {
        idle = (int)((long long)off * 64 / std::max(warps, w));
        best = w;
      }
    }
  }
  p.block = best * 32;
  p.blocks = std::max((warps + best - 1) / best, 1);
  p.warps = p.blocks > 1 ? best : warps;
  p.share = p.blocks > 1 ? best * p.turn : std::max(p.pairs, 1);
  p.per_block = best / p.warps;
  return p;
}

// Where the tracks of view and tang run through the volume (track_setup, as a
// fraction of the LOR); false where they miss it.
static bool track_span(const Grid& g, const Sino& s, const double* xy, int view, int tang, double span[2])
{
  int c[2];
  crystal_ang(s, view, tang, c[0], c[1]);
  span[0] = 0.0;
  span[1] = 1.0;
  for (int d = 0; d < 2; ++d)
  {
    const double p1 = xy[2 * c[0] + d], df = xy[2 * c[1] + d] - p1;
    if (std::fabs(df) <= kEps)
    {
      if (p1 < g.low[d] || p1 > g.high[d])
      {
        return false;
      }
      continue;
    }
    const double a = (g.low[d] - p1) / df, b = (g.high[d] - p1) / df;
    span[0] = std::max(span[0], std::min(a, b));
    span[1] = std::min(span[1], std::max(a, b));
  }
  return span[0] < span[1];
}

// lane_setup's choice for a LOR between z1 and z2 on such a track, up to its
// rounding.
static LorKind lor_kind(const Grid& g, const double span[2], double z1, double z2)
{
  const double lo = g.low[2], hi = g.high[2];
  const double diff = z2 - z1, df = std::fabs(diff) > kEps ? diff : kEps;
  const bool moves = std::fabs(diff) > kEps, up = diff > kEps;
  const double in = moves ? ((up ? lo : hi) - z1) / df : 0.0, out = moves ? ((up ? hi : lo) - z1) / df : 1.0;
  if ((!moves && (z1 < lo || z1 > hi)) || std::max(in, span[0]) >= std::min(out, span[1]))
  {
    return kLorNone;
  }
  const double dz = std::fabs(g.ext[2] / df);
  const double at = std::trunc((z1 + df * span[0] - lo) / g.ext[2]);
  const double ind = std::min(std::max(at, 0.0), g.nz - 1.0);
  const double next = (moves ? (lo + g.ext[2] * ind - z1) / df : 1.0) + (up ? dz : 0.0);
  const double leaves = next + (up ? g.nz - 1 - ind : ind) * dz;
  return in <= span[0] && out >= span[1] && dz > 4.0 * kEps && leaves > span[1] + 4.0 * kEps ? kLorColumn
                                                                                           : kLorGeneral;
}

double column_general(const Grid& g, const Sino& s, const HostTables& t)
{
  const double *xy = t.xy, *z = t.z;
  long long pairs = 0;
  for (int k = 0; k < s.n_segments; ++k)
  {
    pairs += s.n_axial[k];
  }
  const double bottom = std::min(z[0], z[2 * s.n_rings - 2]), top = std::max(z[0], z[2 * s.n_rings - 2]);
  // (the traversal's slices may be thinner than the voxels and end below the
  // volume's top)
  const double end = std::min(g.low[2] + g.nz * g.ext[2], g.high[2]), margin = 1e-4 * (top - bottom);
  if (bottom > g.low[2] + margin && top < end - margin)
  {
    // z clips nothing.  The direct LORs of the lowest slice take the general
    // walk where they end at a crystal within the volume.
    int inside = 0;
    for (int c = 0; c < s.n_cpr; ++c)
    {
      const double x = xy[2 * c], y = xy[2 * c + 1];
      inside += x >= g.low[0] && x <= g.high[0] && y >= g.low[1] && y <= g.high[1] ? 1 : 0;
    }
    int direct = 0;
    for (int axial = 0; inside > 0 && axial < s.n_axial[s.seg_offset]; ++axial)
    {
      int a1, a2;
      crystal_axial(s, 0, axial, a1, a2);
      direct += z[a1] < g.low[2] + g.ext[2] ? 1 : 0;
    }
    return (double)inside / s.n_cpr * direct / pairs;
  }
  // sampled: 8 views x 5 tangential bins, 32 or a few more segments where there
  // are more (the calls' host time: 127 segments 0.11 ms, sampled 0.03).  In a
  // segment they are the first or the last planes, so it is read from both ends.
  const int step = std::max(s.n_segments / 32, 1);
  long long general = 0, meeting = 0;
  for (int i = 0; i < 40; ++i)
  {
    double span[2];
    if (!track_span(g, s, xy, i / 5 * s.n_views / 8, (2 * (i % 5) + 1) * s.n_tang / 10 - s.tang_offset, span))
    {
      continue;
    }
    for (int k = (s.n_segments - 1) % step / 2; k < s.n_segments; k += step)
    {
      meeting += s.n_axial[k];
      auto kind = [&](int axial) {
        int a1, a2;
        crystal_axial(s, k - s.seg_offset, axial, a1, a2);
        return lor_kind(g, span, z[a1], z[a2]);
      };
      int first = 0, last = s.n_axial[k];
      for (LorKind q; first < last && (q = kind(first)) != kLorColumn; ++first)
      {
        (q == kLorGeneral ? general : meeting) += q == kLorGeneral ? 1 : -1;
      }
      for (LorKind q; last > first && (q = kind(last - 1)) != kLorColumn; --last)
      {
        (q == kLorGeneral ? general : meeting) += q == kLorGeneral ? 1 : -1;
      }
    }
  }
  return meeting > 0 ? (double)general / meeting : 0.0;
}

// Mean number of z crossings that stop a warp's turn per crossing of its
// track: the LORs of a segment cross together where their planes lie whole
// voxels apart, so a segment counts once per distinct offset.
double column_stops(const Grid& g, const Sino& s, const ColumnPlan& p, const HostTables& t)
{
  const double* z = t.z;
  const double diameter = 2.0 * std::hypot(t.xy[0], t.xy[1]);
  const double apart = s.n_rings > 1 ? std::fabs(z[2] - z[0]) * (s.span > 1 ? 0.5 : 1.0) / g.ext[2] : 0.0;
  int offsets = 1;
  while (offsets < 64 && std::fabs(offsets * apart - std::round(offsets * apart)) > 1e-3)
  {
    ++offsets;
  }
  // a line's mean step between transaxial crossings, and z's rise in it
  const double step = 0.7853981633974483 * 0.5 * (g.ext[0] + g.ext[1]) / (diameter * g.ext[2]);
  double sum = 0.0;
  for (int k = 0; k < s.n_segments; ++k)
  {
    int a1, a2;
    crystal_axial(s, k - s.seg_offset, s.n_axial[k] / 2, a1, a2);
    sum += std::fabs(z[a2] - z[a1]) * step * std::min(offsets, s.n_axial[k]);
  }
  return sum / ((p.pairs + 63) / 64);
}

// Warps of the launch that have work.
long long column_warps(const ColumnPlan& p) { return (long long)p.tracks * ((p.pairs + p.turn - 1) / p.turn); }

// Tracks need about six warps per scheduler (kColumnWarps) to hide the loops'
// latency (a turn waits for its entry and test): the LOR-by-LOR kernels, with
// twice the warps, are faster below that (measured 0.63x to 0.98x below 3000
// warps, 1.3x and more above 8000).
//
// They also need ring pairs to fill a warp's 64 slots, and a z crossing that stops
// a turn costs as much as the turn.  The backprojection, bound by its atomics,
// gains all the same (1.2x to 1.6x with 25 pairs, 1.06x to 2.6x at 3 to 11 stops).
// Projection and fused kernel, 600 geometries, tracks against LOR by LOR by the
// share of slots filled:
//   full (16, 32, 40, 64 rings): projection 1.3x to 1.6x at one stop, 1.1x to 1.3x
//   at 2.2, 0.9x to 1.05x at 3 to 10; fused kernel 1.3x to 1.8x, 1.04x to 1.45x,
//   1.0x to 1.5x
//   0.75 (12 rings): projection 1.06x at 0.8, 0.99x at 1.5, 0.92x at 2.7; fused
//   kernel 1.25x, 1.09x, 0.95x
//   0.63 (9 rings): projection 1.15x at 0.3, 1.0x at 0.8, 0.92x at 1.3; fused
//   kernel 1.24x, 1.15x, 1.05x
// A track of one warp shares its block with others, whose walks differ in
// length: 8 rings (full) 1.03x and 1.16x at 0.8 stops, 10 (0.78) 1.11x and 1.24x;
// 7 rings (0.77) 0.96x and 1.03x, 6 (0.56) 0.85x and 0.9x.
// The lines below are where these cross 1.
//
// A block with a LOR that z clips takes a whole walk longer, with most of its
// warps idle, so the gain goes with the share of such LORs, and sooner where the
// launch has few waves to fill the gaps.  Tracks against LOR by LOR:
//   fused kernel, 25000 warps and more: 24 rings 1.73x unclipped, 1.31x at 1.7 %,
//   1.06x at 5.8 %; 32 rings 1.15x at 1.5 %, 1.05x at 5 %, 0.99x at 8.7 %, 40 rings
//   1.11x at 7.4 %; 24 rings 0.98x at 22 %
//   12000 to 25000: 17 rings 1.57x, 1.04x at 1.7 %; span 3 1.38x, 1.10x at 0.2 %,
//   1.0x at 1.5 %, 0.95x at 2.7 %
//   fewer: 24 rings 1.38x, 0.97x at 1.7 %; 8 rings 1.15x, 0.88x at 0.13 %
//   projection (all views): 1.04x at 8.7 %, 1.0x at 8.2 % (span 3), 1.0x at 22 %;
//   with 64 pairs, whose blocks hold four tracks, 0.96x at 0.13 %, 0.5x at 12 %
//   backprojection: 1.15x to 1.4x at 20 %, even at 45 % with 36 pairs.
// Beyond 2.2 stops too little is gained to pay for clipped LORs (64 rings, fused
// kernel: 1.05x at 2.3 stops unclipped, 0.94x at 1 %; 1.2x and 0.92x at 3.7).
bool columns_pay(const Grid& g, const Sino& s, const ColumnPlan& p, const HostTables& t, TrackUse use)
{
  const bool back = use == TrackUse::Backward;
  if (g.exact_only || p.pairs < 30 || column_smem(p) > kColumnSharedLimit ||
      (long long)g.nxy * g.nz >= 1LL << 29)
  {
    return false;
  }
  if ((g.nz + kTile - 1) / kTile > 65535)
  {
    return false;  // beyond the tile grid of the z-column copies
  }
  const long long warps = use == TrackUse::Batch ? 12000 : column_warps(p);
  double most = 0.2;
  if (!back)
  {
    const double fill = p.pairs / (64.0 * ((p.pairs + 63) / 64)) * (p.pairs <= 64 ? 0.78 : 1.0);
    const double stops = column_stops(g, s, p, t);
    if (stops > (use == TrackUse::Forward ? 6.3 * (fill - 0.55) : 9.0 * (fill - 0.5)))
    {
      return false;
    }
    most = p.pairs <= 64 || warps < 12000 || stops > 2.2 ? 3e-4 : (warps < 25000 ? 0.012 : 0.08);
  }
  return column_general(g, s, t) <= most;
}

void launch_to_columns(const Grid& g, const float* in, double* out, float* acc, const LaunchCfg& cfg)
{
  k_to_columns<<<column_tiles(g.nxy, g.nz), dim3(kTile, kTileRows), 0, cfg.stream>>>(g.nxy, g.nz, in, out, acc);
}

void launch_from_columns(const Grid& g, const float* acc, float* out, const LaunchCfg& cfg)
{
  k_from_columns<<<column_tiles(g.nxy, g.nz), dim3(kTile, kTileRows), 0, cfg.stream>>>(g.nxy, g.nz, acc, out);
}

void launch_em_update_columns(const Grid& g, const float* img, float* out, const float* acc, const float* sens,
                              const LaunchCfg& cfg)
{
  k_em_update_columns<<<column_tiles(g.nxy, g.nz), dim3(kTile, kTileRows), 0, cfg.stream>>>(g.nxy, g.nz, img, out, acc,
                                                                                            sens);
}

void launch_column_forward(const Grid& g, const Sino& s, const Tables& t, const ColumnPlan& p, const double* img,
                           float* sino, FwdEpilogue ep, const LaunchCfg& cfg)
{
  if (p.tracks == 0)
  {
    return;
  }
  const size_t bytes = column_smem(p);
  auto* kernel = ep == FwdEpilogue::Exp ? k_column_forward<FwdEpilogue::Exp> : k_column_forward<FwdEpilogue::None>;
  if (!ask_shared(kernel, bytes))
  {
    return;
  }
  kernel<<<(unsigned)column_blocks(p), p.block, bytes, cfg.stream>>>(g, s, t, p, img, sino, cfg.check);
}

void launch_column_backward(const Grid& g, const Sino& s, const Tables& t, const ColumnPlan& p, const float* sino,
                            float* acc, const LorQueue& queue, const LaunchCfg& cfg)
{
  if (p.tracks == 0)
  {
    return;
  }
  const size_t bytes = column_smem(p);
  auto* kernel = p.skip ? k_column_backward<true> : k_column_backward<false>;
  if (!ask_shared(kernel, bytes))
  {
    return;
  }
  kernel<<<(unsigned)column_blocks(p), p.block, bytes, cfg.stream>>>(g, s, t, p, sino, acc, queue, cfg.check);
}

int queue_room(const Sino& s, TrackUse use)
{
  return (int)((long long)s.n_enum * (use == TrackUse::Backward ? kQueuePercentBackward : kQueuePercent) / 100) + 1;
}

void launch_list_nonzero(const Sino& s, const ColumnPlan& p, const float* sino, const LorQueue& queue,
                         const LaunchCfg& cfg)
{
  constexpr int deep = kListWarps * kListPairs;
  const int tiles = (s.n_tang + 31) / 32 * ((p.pairs + deep - 1) / deep);
  k_list_nonzero<<<(unsigned)(tiles * (p.tracks / s.n_tang)), 32 * kListWarps, 0, cfg.stream>>>(s, p, sino, queue);
}

// s with the queue as its enumeration.
static Sino queue_of(const Sino& s, const LorQueue& queue)
{
  Sino q = s;
  q.list = queue.list;
  q.list_n = queue.count;
  return q;
}

void launch_queue_backward(const Grid& g, const Sino& s, const Tables& t, const ColumnPlan& p, const float* sino,
                           float* acc, const LorQueue& queue, const LaunchCfg& cfg)
{
  k_queue_backward<<<(unsigned)(queue.room + 127) / 128, 128, 0, cfg.stream>>>(g, queue_of(s, queue), t, sino, acc,
                                                                                 p.tracks / s.n_tang, queue, cfg.check);
}

void launch_queue_osem(const Grid& g, const Sino& s, const Tables& t, const ColumnPlan& p, const double* img,
                       const float* sino, const float* mult, const float* bias, float* acc, const LorQueue& queue,
                       const LaunchCfg& cfg)
{
  auto* kernel = mult != nullptr ? k_queue_osem<true> : k_queue_osem<false>;
  kernel<<<(unsigned)(queue.room + 127) / 128, 128, 0, cfg.stream>>>(g, queue_of(s, queue), t, img, sino, mult, bias,
                                                                       acc, p.tracks / s.n_tang, queue, cfg.check);
}

void launch_batch_column_osem(const BatchProblem* P, const BatchItem* items, int n_items, int n_blocks, size_t bytes,
                              bool skip, int* check, cudaStream_t stream)
{
  if (n_blocks <= 0)
  {
    return;
  }
  auto* kernel = skip ? k_batch_column_osem<ZeroBins::Pack> : k_batch_column_osem<ZeroBins::Trace>;
  if (!ask_shared(kernel, bytes))
  {
    return;
  }
  kernel<<<(unsigned)n_blocks, kBatchColumnBlock, bytes, stream>>>(P, items, n_items, check);
}

void launch_column_osem(const Grid& g, const Sino& s, const Tables& t, const ColumnPlan& p, const double* img,
                        const float* sino, const float* mult, const float* bias, float* acc, const LorQueue& queue,
                        const LaunchCfg& cfg)
{
  if (p.tracks == 0)
  {
    return;
  }
  const size_t bytes = column_smem(p);
  // (a plan that packs is a batch's, which has no multiplicative factors)
  auto* kernel =
    mult != nullptr
      ? (p.skip != 0 ? k_column_osem<true, ZeroBins::Queue> : k_column_osem<true, ZeroBins::Trace>)
      : (p.skip == 0 ? k_column_osem<false, ZeroBins::Trace>
                     : (p.turn == kPackedTurn ? k_column_osem<false, ZeroBins::Pack>
                                              : k_column_osem<false, ZeroBins::Queue>));
  if (!ask_shared(kernel, bytes))
  {
    return;
  }
  kernel<<<(unsigned)column_blocks(p), p.block, bytes, cfg.stream>>>(g, s, t, p, img, sino, mult, bias, acc, queue,
                                                                     cfg.check);
}
}  // namespace fir
