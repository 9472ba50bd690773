// Traversal of the lines of response that share a transaxial track.
//
// All LORs with the same view and tangential bin join the same two crystals
// of a ring; they differ in their end slices only.  FIR's traversal advances
// each dimension by a running sum of its own (Siddon.cc:379-392), so the x
// and y crossings of all of them are the same doubles, whatever z does: one
// sorted list of crossings (a track) serves up to n_rings^2 LORs.  A block
// builds the tracks of its LORs in shared memory, and a warp then leads 64 of
// them along the list, two per lane: per step a LOR needs its length, its
// gather or atomic, and one test for the whole warp, where the general walk
// orders three sequences, tests three ties and advances three sums.
//
// The LORs of a warp run through the same columns of voxels at different z,
// so the images are kept in z columns ([y][x][z]): a warp's gather or atomic
// touches two to four lines.
//
// The result is FIR's bit for bit.  A step of FIR's loop takes the smallest
// next alpha m and advances every dimension whose alpha is within EPS of m.
// * A dimension advances at most once per step, and its steps are longer than
//   4 EPS (checked), so the crossings taken by a step are a prefix of the
//   sorted list's remainder: its first entry, perhaps the second.
// * Where z's next alpha is further than EPS from the list's next entry and
//   that entry further than EPS from the one after it, the step takes either
//   z alone or the entry alone.
// * Otherwise, and at the entries that end the walk (alphaMax, or a crossing
//   that leaves the volume), the LOR takes FIR's step as written
//   (column_walk).  Entries at which every LOR must do so hold a NaN in place
//   of their alpha, so that one comparison finds them and the ties with z.
// A LOR may use the track when x and y decide its entry and exit (z clips
// nothing and leaves the volume after alphaMax).  Others take the general
// walk, 32 to a warp, at the end of their block.
//
// Bound by instruction issue (74 % of the slots in the projection, 68 % in the
// fused kernel; 22 instructions per LOR and step with the gather, 20 with the
// atomic, against 45 of the general walk), the backprojection by its atomics'
// sectors (L1 78 %, L2 63 %, issue 57 %).  Clinical scanner (32 rings x 512 crystals,
// 3.28e7 LORs, 200x200x64 voxels): forward projection 16.15 -> 9.5 ms,
// backprojection of 16 subsets 23.0 -> 12.0 ms, OSEM sub-iteration 2.08 ->
// 1.28 ms.
#pragma once

#include "lor_body.cuh"

namespace fir
{
// One crossing of a track: its alpha and the first voxel of the column that
// the path leaves there, as byte offsets into float and double images.  At a
// crossing that ends the walk, or that the next one follows within EPS, a
// LOR must take FIR's step as written: its entry holds a NaN whose low word
// is the column, and its alpha in the other half.
struct __align__(16) Crossing
{
  double alpha;
  unsigned float_bytes, double_bytes;
};

struct TrackHead
{
  double amin, amax;  // alphaMin and alphaMax of x and y
  double s2;          // dx^2 + dy^2
  double x1, y1, x2, y2;
  double a[2], da[2];
  int left[2], step[2];
  int col;     // first column
  int exit;    // index of the first crossing that leaves the volume
  int crosses; // 0: no LOR of the track crosses the volume
  int acc;     // number of the track's accumulator
  int shared;  // 1: the LORs may use the list
};

__device__ __forceinline__ unsigned shared_address(const void* p)
{
  return (unsigned)__cvta_generic_to_shared(p);
}

constexpr int kExactHigh = 0x7ff80000;

// A crossing whichever way its entry is written.
struct PlainCrossing
{
  double alpha;
  int col;
};

__device__ __forceinline__ PlainCrossing plain_crossing(const Crossing& c)
{
  const int4 v = *reinterpret_cast<const int4*>(&c);
  return v.y == kExactHigh ? PlainCrossing{__hiloint2double(v.w, v.z), v.x}
                           : PlainCrossing{__hiloint2double(v.y, v.x), v.z >> 2};
}

// The accumulator of a track in view number sv of the subset's views.
__device__ __forceinline__ int column_accumulator(bool along_x, int sv, int views)
{
  return (along_x ? 1 : 0) + (2 * sv >= views ? 2 : 0);
}

// x and y parts of siddon_setup for one track.
__device__ __forceinline__ void track_setup(const Grid& g, TrackHead& h)
{
  const double e1[2] = {h.x1, h.y1}, e2[2] = {h.x2, h.y2};
  double diff[2], smin[2], smax[2], snext[2];
  int dir[2];
  h.crosses = 0;
  h.shared = 0;
  h.exit = 0x7fffffff;
#pragma unroll
  for (int d = 0; d < 2; ++d)
  {
    const double c1 = e1[d], lo = g.low[d], hi = g.high[d];
    double df = dsub(e2[d], c1);
    if (fabs(df) > kEps)
    {
      const double rdf = __drcp_rn(df);
      dir[d] = df > 0 ? 1 : -1;
      smin[d] = ddiv_r(dsub(df > 0 ? lo : hi, c1), df, rdf);
      smax[d] = ddiv_r(dsub(df > 0 ? hi : lo, c1), df, rdf);
      snext[d] = 0.0;
    }
    else
    {
      if (c1 < lo || c1 > hi)
      {
        return;
      }
      df = kEps;
      dir[d] = -1;
      smin[d] = 0.0;
      smax[d] = 1.0;
      snext[d] = 1.0;
    }
    diff[d] = df;
  }
  double t = smin[1] > 0.0 ? smin[1] : 0.0;
  h.amin = smin[0] > t ? smin[0] : t;
  t = smax[1] < 1.0 ? smax[1] : 1.0;
  h.amax = smax[0] < t ? smax[0] : t;
  if (h.amin >= h.amax)
  {
    return;
  }
  h.crosses = 1;
  const int n[2] = {g.nx, g.ny};
  const int stride[2] = {g.nz, g.nx * g.nz};
  h.s2 = dadd(dmul(diff[0], diff[0]), dmul(diff[1], diff[1]));
  h.col = 0;
  bool ok = !g.exact_only;
#pragma unroll
  for (int d = 0; d < 2; ++d)
  {
    const double rdiff = __drcp_rn(diff[d]);
    h.da[d] = fabs(ddiv_r(g.ext[d], diff[d], rdiff));
    int ind = __double2int_rz(ddiv_r(dsub(dadd(e1[d], dmul(diff[d], h.amin)), g.low[d]), g.ext[d], g.rext[d]));
    ind = ind < n[d] - 1 ? ind : n[d] - 1;
    ind = ind > 0 ? ind : 0;
    double al = snext[d];
    if (al < 1.0)
    {
      al = ddiv_r(dsub(dadd(g.low[d], dmul(g.ext[d], (double)ind)), e1[d]), diff[d], rdiff);
    }
    if (dir[d] > 0)
    {
      al = dadd(al, h.da[d]);
    }
    h.a[d] = al;
    h.left[d] = dir[d] > 0 ? n[d] - 1 - ind : ind;
    h.step[d] = dir[d] * stride[d];
    h.col += ind * stride[d];
    ok = ok && al > -1.0 && h.da[d] > 4.0 * kEps;
  }
  h.shared = ok ? 1 : 0;
}

// Number of the m ascending values v that lie below x (or_equal: at or below).
__device__ __forceinline__ int count_below(const double* v, int m, double x, bool or_equal)
{
  int lo = 0, hi = m;
  while (lo < hi)
  {
    const int mid = (lo + hi) >> 1;
    if (or_equal ? v[mid] <= x : v[mid] < x)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// A track in shared memory: its crossings in ascending order, closed by one
// at infinity.
struct Track
{
  TrackHead* head;
  Crossing* crossings;  // cap + 1
  double* seq;          // cap: while it is built, the x sequence at 0 and the y sequence at nx
};

__host__ __device__ constexpr size_t track_bytes(int cap)
{
  return (sizeof(TrackHead) + 15) / 16 * 16 + (size_t)(cap + 1) * sizeof(Crossing) +
         (size_t)((cap + 1) / 2) * 2 * sizeof(double);
}

__device__ __forceinline__ Track track_at(unsigned char* smem, int cap, int k)
{
  unsigned char* p = smem + (size_t)k * track_bytes(cap);
  Track t;
  t.head = reinterpret_cast<TrackHead*>(p);
  t.crossings = reinterpret_cast<Crossing*>(p + (sizeof(TrackHead) + 15) / 16 * 16);
  t.seq = reinterpret_cast<double*>(t.crossings + cap + 1);
  return t;
}

// Builds the block's tracks, the first of them number `first`.  Every thread
// of the block calls this.  Sets *left to 0 too.
//
// The running sums are serial, so two threads per track make them while the
// others wait; the rest is a rank computation per crossing.
__device__ __forceinline__ void build_tracks(const Grid& g, const Sino& s, const Tables& t, const ColumnPlan& p,
                                             int subset, int first, unsigned char* smem, int* left)
{
  const int tid = threadIdx.x;
  if (tid == 0)
  {
    *left = 0;
  }
  for (int k = tid; k < p.per_block; k += blockDim.x)
  {
    TrackHead& h = *track_at(smem, p.cap, k).head;
    h.crosses = 0;
    h.shared = 0;
    if (first + k < p.tracks)
    {
      const int sv = (first + k) / s.n_tang;
      const int tang = first + k - sv * s.n_tang - s.tang_offset;
      int c1, c2;
      crystal_ang(s, sv * s.n_subsets + subset, tang, c1, c2);
      const double2 p1 = __ldg(t.xy + c1), p2 = __ldg(t.xy + c2);
      h.x1 = p1.x;
      h.y1 = p1.y;
      h.x2 = p2.x;
      h.y2 = p2.y;
      h.acc = column_accumulator(fabs(dsub(p2.x, p1.x)) > fabs(dsub(p2.y, p1.y)), sv, p.tracks / s.n_tang);
      track_setup(g, h);
    }
  }
  __syncthreads();
  for (int k = tid; k < 2 * p.per_block; k += blockDim.x)
  {
    const Track tr = track_at(smem, p.cap, k >> 1);
    const TrackHead& h = *tr.head;
    const int d = k & 1;
    if (h.shared)
    {
      double* q = tr.seq + (d ? g.nx : 0);
      double a = h.a[d];
      const double da = h.da[d];
      const int n = h.left[d];
      for (int j = 0; j <= n; ++j)
      {
        q[j] = a;
        a = dadd(a, da);
      }
      if (d == 0)
      {
        *reinterpret_cast<int4*>(tr.crossings + h.left[0] + h.left[1] + 2) = make_int4(0, kExactHigh, 0, 0x7ff00000);
      }
    }
  }
  __syncthreads();
  for (int k = tid; k < p.per_block * p.cap; k += blockDim.x)
  {
    const int v = p.per_block == 1 ? 0 : k / p.cap;
    const int q = k - v * p.cap;
    const Track tr = track_at(smem, p.cap, v);
    TrackHead& h = *tr.head;
    const int d = q < g.nx ? 0 : 1;
    const int i = d ? q - g.nx : q;
    if (!h.shared || i > h.left[d])
    {
      continue;
    }
    const double* other = tr.seq + (d ? 0 : g.nx);
    const int last = h.left[d ^ 1];
    const double a = tr.seq[q];
    // equal alphas: x first
    const int before = count_below(other, last + 1, a, d == 1);
    const int rank = i + before;
    // the next crossing within EPS can only be the other dimension's
    const bool exact = i == h.left[d] || !(a < h.amax) || (before <= last && dsub(other[before], a) < kEps);
    const int col = h.col + (d ? before : i) * h.step[0] + (d ? i : before) * h.step[1];
    const int lo = __double2loint(a), hi = __double2hiint(a);
    *reinterpret_cast<int4*>(tr.crossings + rank) =
      exact ? make_int4(col, kExactHigh, lo, hi) : make_int4(lo, hi, 4 * col, 8 * col);
    if (i == h.left[d])
    {
      atomicMin(&h.exit, rank);
    }
  }
  __syncthreads();
}

// A lane's walk along its track.
struct ColumnLane
{
  double az, dz;   // alpha of the next z crossing, and between two
  double d12;
  int z, sz;       // slice, its change per crossing
};

enum LorKind : int
{
  kLorNone,     // misses the volume
  kLorColumn,   // uses the track
  kLorGeneral   // takes the general walk
};

// The z part of siddon_setup for a LOR of track h between slices at z1, z2.
__device__ __forceinline__ int lane_setup(const Grid& g, const TrackHead& h, double z1, double z2, ColumnLane& w)
{
  const double lo = g.low[2], hi = g.high[2];
  double df = dsub(z2, z1), smin = 0.0, smax = 1.0, al = 1.0;
  const bool moves = fabs(df) > kEps;
  bool up = false;
  if (moves)
  {
    const double rdf = __drcp_rn(df);
    up = df > 0;
    smin = ddiv_r(dsub(up ? lo : hi, z1), df, rdf);
    smax = ddiv_r(dsub(up ? hi : lo, z1), df, rdf);
  }
  else
  {
    if (z1 < lo || z1 > hi)
    {
      return kLorNone;
    }
    df = kEps;
  }
  if ((smin > h.amin ? smin : h.amin) >= (smax < h.amax ? smax : h.amax))
  {
    return kLorNone;
  }
  if (!h.shared || !(smin <= h.amin && smax >= h.amax))
  {
    return kLorGeneral;
  }
  const double rdiff = __drcp_rn(df);
  w.dz = fabs(ddiv_r(g.ext[2], df, rdiff));
  w.d12 = __dsqrt_rn(dadd(h.s2, dmul(df, df)));
  int ind = __double2int_rz(ddiv_r(dsub(dadd(z1, dmul(df, h.amin)), lo), g.ext[2], g.rext[2]));
  ind = ind < g.nz - 1 ? ind : g.nz - 1;
  ind = ind > 0 ? ind : 0;
  if (moves)
  {
    al = ddiv_r(dsub(dadd(lo, dmul(g.ext[2], (double)ind)), z1), df, rdiff);
  }
  if (up)
  {
    al = dadd(al, w.dz);
  }
  w.az = al;
  w.z = ind;
  w.sz = up ? 1 : -1;
  const int left = up ? g.nz - 1 - ind : ind;
  // z leaves the volume after the walk's end (the closed form is within a
  // few ulps of the running sum)
  const double leaves = dadd(al, dmul((double)left, w.dz));
  return w.dz > 4.0 * kEps && leaves > dadd(h.amax, 4.0 * kEps) ? kLorColumn : kLorGeneral;
}

// The state of one of a lane's LORs between steps.
struct ColumnState
{
  int z, sz;        // slice, its change per z crossing
  double az, prev;  // alpha of the next z crossing, and of the last step
  double dz, d12;
};

// |d| with a high word below this one's, as the bits of a float: z and the
// crossing may tie (1.00001e-5, just above EPS).
__device__ __forceinline__ float column_near() { return __int_as_float(__double2hiint(1.00001e-5) + 1); }

// The loops below run a warp's steps up to the first in which some LOR must
// take FIR's step as written; nearly all steps are theirs.  They are in PTX
// because the compiler mixes parts of the exact step into them otherwise.
//
// A lane has two LORs, and all LORs of the warp are at one crossing.  A turn
// takes d = (the smaller az) - alpha, whose high word as the bits of a float
// tells d < 0 (z comes first), a small |d| and the NaN of an entry at once.
// Where there is none of these, every LOR steps to the crossing.  Where z
// comes first for some, those alone take their step, and the turn is tried
// again: the others wait, so that a turn's gathers or atomics fall into one
// column.  A column's sectors are what they cost (an atomic about 1.4 cycles
// of an SM per sector); with every lane at its own crossing there were twice
// as many.  Two LORs per lane share the entry, the test and the loop, and
// hide each other's latency.
//
// A turn loads and tests the next entry while it makes its own step, so that
// neither waits for the other; the alphas of the last, this and the next
// crossing rotate through a0, a1 and a2.  The last alpha is all LORs' after a
// turn; before the first one, and after a step of z, p0 and p1 are theirs.
// ptr is the address of the LOR's voxel in column 0; S the column's field of
// the entry scaled by the voxel's size.
#define FIR_COLUMN_BEGIN                                                                                             \
  "{\n"                                                                                                              \
  ".reg .pred zf0, zf1, stop, any;\n"                                                                                       \
  ".reg .b32 at, z0, z1, c0, c1, c2, dl, dh0, dh1;\n"                                                                \
  ".reg .f32 f, g, near, line0, line1;\n"                                                                            \
  ".reg .f64 azm, az0, az1, dz0, dz1, p0, p1, u0, u1, a0, a1, a2, d, t, t1, x;\n"                                    \
  ".reg .f64 len0, len1, value0, value1, wide0, wide1, d120, d121;\n"                                                \
  ".reg .b64 ptr0, ptr1, sz0, sz1, adr0, adr1, off;\n"                                                               \
  "mov.b32 at, %0;\n"                                                                                                \
  "mov.b64 ptr0, %1;\n"                                                                                              \
  "mov.b64 ptr1, %2;\n"                                                                                              \
  "mov.f64 az0, %3;\n"                                                                                               \
  "mov.f64 az1, %4;\n"                                                                                               \
  "mov.f64 p0, %5;\n"                                                                                                \
  "mov.f64 p1, %6;\n"
#define FIR_COLUMN_TEST(A)                                                                                           \
  "sub.rn.f64 d, azm, " A ";\n"                                                                                      \
  "mov.b64 {dl, dh0}, d;\n"                                                                                          \
  "mov.b32 f, dh0;\n"                                                                                                \
  "setp.ltu.f32 stop, f, near;\n"                                                                                    \
  "vote.sync.any.pred stop, stop, 0xffffffff;\n"
#define FIR_COLUMN_ADDRESS(K, C)                                                                                     \
  "cvt.u64.u32 off, " C ";\n"                                                                                        \
  "add.s64 adr" K ", ptr" K ", off;\n"
// The entry after this one into alpha A and column C, and its test.
#define FIR_COLUMN_NEXT(S, A, C)                                                                                     \
  "ld.shared.f64 " A ", [at+16];\n"                                                                                  \
  "ld.shared.u32 " C ", [at+16+" S "];\n" FIR_COLUMN_TEST(A)
// One step of all LORs from alpha FROM to alpha TO through column C.
#define FIR_COLUMN_TURN(S, FROM, TO, C, NEXT, NEXT_C, EXIT, STEP)                                                    \
  FIR_COLUMN_NEXT(S, NEXT, NEXT_C)                                                                                   \
  "sub.rn.f64 t, " TO ", " FROM ";\n" FIR_COLUMN_ADDRESS("0", C) FIR_COLUMN_ADDRESS("1", C) STEP("t", "t")           \
  "add.s32 at, at, 16;\n"                                                                                            \
  "@stop bra.uni " EXIT ";\n"
// z's step of LOR K in the lanes where z comes first.
#define FIR_COLUMN_Z(K, SKIP, Z_STEP)                                                                                \
  "@!zf" K " bra " SKIP ";\n"                                                                                        \
  "sub.rn.f64 t, az" K ", p" K ";\n" FIR_COLUMN_ADDRESS(K, "c0") Z_STEP(K)                                           \
  "mov.f64 p" K ", az" K ";\n"                                                                                       \
  "add.rn.f64 az" K ", az" K ", dz" K ";\n"                                                                          \
  "add.s64 ptr" K ", ptr" K ", sz" K ";\n" SKIP ":\n"
#define FIR_COLUMN_MIN                                                                                               \
  "setp.lt.f64 any, az1, az0;\n"                                                                                     \
  "selp.f64 azm, az1, az0, any;\n"
#define FIR_COLUMN_LOOP(S, STEP, Z_STEP)                                                                             \
  FIR_COLUMN_MIN                                                                                                     \
  "ld.shared.f64 a0, [at];\n"                                                                                        \
  "ld.shared.u32 c0, [at+" S "];\n" FIR_COLUMN_TEST("a0")                                                            \
  "@stop bra.uni Z;\n"                                                                                               \
  "START:\n" FIR_COLUMN_NEXT(S, "a1", "c1")                                                                          \
  "sub.rn.f64 t, a0, p0;\n"                                                                                          \
  "sub.rn.f64 t1, a0, p1;\n" FIR_COLUMN_ADDRESS("0", "c0") FIR_COLUMN_ADDRESS("1", "c0") STEP("t", "t1")             \
  "add.s32 at, at, 16;\n"                                                                                            \
  "@stop bra.uni STOP0;\n"                                                                                           \
  "LOOP:\n" FIR_COLUMN_TURN(S, "a0", "a1", "c1", "a2", "c2", "STOP1", STEP)                                          \
  FIR_COLUMN_TURN(S, "a1", "a2", "c2", "a0", "c0", "STOP2", STEP)                                                    \
  FIR_COLUMN_TURN(S, "a2", "a0", "c0", "a1", "c1", "STOP0", STEP)                                                    \
  "bra.uni LOOP;\n"                                                                                                  \
  "STOP0:\n"                                                                                                         \
  "mov.f64 p0, a0;\n"                                                                                                \
  "mov.f64 p1, a0;\n"                                                                                                \
  "mov.f64 a0, a1;\n"                                                                                                \
  "mov.b32 c0, c1;\n"                                                                                                \
  "bra.uni Z;\n"                                                                                                     \
  "STOP1:\n"                                                                                                         \
  "mov.f64 p0, a1;\n"                                                                                                \
  "mov.f64 p1, a1;\n"                                                                                                \
  "mov.f64 a0, a2;\n"                                                                                                \
  "mov.b32 c0, c2;\n"                                                                                                \
  "bra.uni Z;\n"                                                                                                     \
  "STOP2:\n"                                                                                                         \
  "mov.f64 p0, a2;\n"                                                                                                \
  "mov.f64 p1, a2;\n"                                                                                                \
  "Z:\n"                                                                                                             \
  "sub.rn.f64 d, az0, a0;\n"                                                                                         \
  "mov.b64 {dl, dh0}, d;\n"                                                                                          \
  "sub.rn.f64 d, az1, a0;\n"                                                                                         \
  "mov.b64 {dl, dh1}, d;\n"                                                                                          \
  "mov.b32 f, dh0;\n"                                                                                                \
  "mov.b32 g, dh1;\n"                                                                                                \
  "abs.f32 f, f;\n"                                                                                                  \
  "abs.f32 g, g;\n"                                                                                                  \
  "min.f32 f, f, g;\n"                                                                                               \
  "setp.ltu.f32 stop, f, near;\n"                                                                                    \
  "vote.sync.any.pred stop, stop, 0xffffffff;\n"                                                                     \
  "@stop bra.uni OUT;\n"                                                                                             \
  "setp.lt.s32 zf0, dh0, 0;\n"                                                                                       \
  "setp.lt.s32 zf1, dh1, 0;\n" FIR_COLUMN_Z("0", "SKIP0", Z_STEP) FIR_COLUMN_Z("1", "SKIP1", Z_STEP)                 \
  FIR_COLUMN_MIN FIR_COLUMN_TEST("a0")                                                                               \
  "@stop bra.uni Z;\n"                                                                                               \
  "bra.uni START;\n"                                                                                                 \
  "OUT:\n"                                                                                                           \
  "mov.b32 %0, at;\n"                                                                                                \
  "mov.b64 %1, ptr0;\n"                                                                                              \
  "mov.b64 %2, ptr1;\n"                                                                                              \
  "mov.f64 %3, az0;\n"                                                                                               \
  "mov.f64 %4, az1;\n"                                                                                               \
  "mov.f64 %5, p0;\n"                                                                                                \
  "mov.f64 %6, p1;\n"

// A projection so far, without its last term, len * value: each gather is
// issued one step before its term is added.
struct LineSum
{
  float line;
  double len, value;
};

#define FIR_COLUMN_TERM(K)                                                                                           \
  "mul.rn.f64 u" K ", len" K ", value" K ";\n"                                                                       \
  "cvt.f64.f32 wide" K ", line" K ";\n"                                                                              \
  "add.rn.f64 wide" K ", wide" K ", u" K ";\n"
#define FIR_COLUMN_LINE_OF(K, T)                                                                                     \
  FIR_COLUMN_TERM(K)                                                                                                 \
  "ld.global.nc.f64 value" K ", [adr" K "];\n"                                                                       \
  "cvt.rn.f32.f64 line" K ", wide" K ";\n"                                                                           \
  "mul.rn.f64 len" K ", " T ", d12" K ";\n"
#define FIR_COLUMN_LINE(T0, T1) FIR_COLUMN_LINE_OF("0", T0) FIR_COLUMN_LINE_OF("1", T1)
#define FIR_COLUMN_Z_LINE(K) FIR_COLUMN_LINE_OF(K, "t")

__device__ __forceinline__ void column_run_line(unsigned& at, ColumnState w[2], const double* __restrict__ img,
                                                LineSum s[2])
{
  const double* p[2] = {img + w[0].z, img + w[1].z};
  asm volatile(FIR_COLUMN_BEGIN
               "mov.f32 line0, %7;\n"
               "mov.f32 line1, %8;\n"
               "mov.f64 len0, %9;\n"
               "mov.f64 len1, %10;\n"
               "mov.f64 value0, %11;\n"
               "mov.f64 value1, %12;\n"
               "cvt.s64.s32 sz0, %13;\n"
               "cvt.s64.s32 sz1, %14;\n"
               "mov.f64 dz0, %15;\n"
               "mov.f64 dz1, %16;\n"
               "mov.f64 d120, %17;\n"
               "mov.f64 d121, %18;\n"
               "mov.f32 near, %19;\n" FIR_COLUMN_LOOP("12", FIR_COLUMN_LINE, FIR_COLUMN_Z_LINE)
               "mov.f32 %7, line0;\n"
               "mov.f32 %8, line1;\n"
               "mov.f64 %9, len0;\n"
               "mov.f64 %10, len1;\n"
               "mov.f64 %11, value0;\n"
               "mov.f64 %12, value1;\n"
               "}\n"
               : "+r"(at), "+l"(p[0]), "+l"(p[1]), "+d"(w[0].az), "+d"(w[1].az), "+d"(w[0].prev), "+d"(w[1].prev),
                 "+f"(s[0].line), "+f"(s[1].line), "+d"(s[0].len), "+d"(s[1].len), "+d"(s[0].value),
                 "+d"(s[1].value)
               : "r"(w[0].sz * (int)sizeof(double)), "r"(w[1].sz * (int)sizeof(double)), "d"(w[0].dz), "d"(w[1].dz),
                 "d"(w[0].d12), "d"(w[1].d12), "f"(column_near()));
  w[0].z = (int)(p[0] - img);
  w[1].z = (int)(p[1] - img);
}

#define FIR_COLUMN_VALUE(K, T)                                                                                       \
  "mul.rn.f64 u" K ", " T ", d12" K ";\n"                                                                            \
  "mul.rn.f64 u" K ", u" K ", value" K ";\n"                                                                         \
  "cvt.rn.f32.f64 line" K ", u" K ";\n"
#define FIR_COLUMN_ADD(T0, T1)                                                                                       \
  FIR_COLUMN_VALUE("0", T0)                                                                                          \
  FIR_COLUMN_VALUE("1", T1)                                                                                          \
  "red.global.add.f32 [adr0], line0;\n"                                                                              \
  "red.global.add.f32 [adr1], line1;\n"
#define FIR_COLUMN_ADD_LIVE(T0, T1)                                                                                  \
  FIR_COLUMN_VALUE("0", T0)                                                                                          \
  FIR_COLUMN_VALUE("1", T1)                                                                                          \
  "@live0 red.global.add.f32 [adr0], line0;\n"                                                                       \
  "@live1 red.global.add.f32 [adr1], line1;\n"
#define FIR_COLUMN_Z_ADD(K)                                                                                          \
  FIR_COLUMN_VALUE(K, "t")                                                                                           \
  "red.global.add.f32 [adr" K "], line" K ";\n"
#define FIR_COLUMN_SCATTER(STEP)                                                                                     \
  asm volatile(FIR_COLUMN_BEGIN                                                                                      \
               ".reg .pred live0, live1;\n"                                                                          \
               "cvt.s64.s32 sz0, %7;\n"                                                                              \
               "cvt.s64.s32 sz1, %8;\n"                                                                              \
               "mov.f64 dz0, %9;\n"                                                                                  \
               "mov.f64 dz1, %10;\n"                                                                                 \
               "mov.f64 d120, %11;\n"                                                                                \
               "mov.f64 d121, %12;\n"                                                                                \
               "mov.f32 near, %13;\n"                                                                                \
               "mov.f64 value0, %14;\n"                                                                              \
               "mov.f64 value1, %15;\n"                                                                              \
               "setp.ne.s32 live0, %16, 0;\n"                                                                        \
               "setp.ne.s32 live1, %17, 0;\n" FIR_COLUMN_LOOP("8", STEP, FIR_COLUMN_Z_ADD)                           \
               "}\n"                                                                                                 \
               : "+r"(at), "+l"(p[0]), "+l"(p[1]), "+d"(w[0].az), "+d"(w[1].az), "+d"(w[0].prev), "+d"(w[1].prev)    \
               : "r"(w[0].sz * (int)sizeof(float)), "r"(w[1].sz * (int)sizeof(float)), "d"(w[0].dz), "d"(w[1].dz),   \
                 "d"(w[0].d12), "d"(w[1].d12), "f"(column_near()), "d"(value[0]), "d"(value[1]), "r"((int)live[0]),  \
                 "r"((int)live[1])                                                                                   \
               : "memory")

// all: every LOR of the warp is live (a guarded atomic costs a branch).
__device__ __forceinline__ void column_run_scatter(unsigned& at, ColumnState w[2], float* acc, const double value[2],
                                                   const bool live[2], bool all)
{
  float* p[2] = {acc + w[0].z, acc + w[1].z};
  if (all)
  {
    FIR_COLUMN_SCATTER(FIR_COLUMN_ADD);
  }
  else
  {
    FIR_COLUMN_SCATTER(FIR_COLUMN_ADD_LIVE);
  }
  w[0].z = (int)(p[0] - acc);
  w[1].z = (int)(p[1] - acc);
}

// Walks the LORs of a warp along their track.  run(at, state) runs steps up
// to the first in which some LOR must take FIR's step as written; those are
// made here, through emit(k, voxel, length) for a lane's LOR k.  Every lane of
// the warp calls this; go is false for LORs without work, for which run may
// emit anything.
template<class Run, class Emit>
__device__ __forceinline__ void column_walk(const Track& t, const ColumnLane l[2], const bool go[2], Run&& run,
                                            Emit&& emit)
{
  constexpr unsigned kAll = 0xffffffffu;
  if (!__any_sync(kAll, go[0] || go[1]))
  {
    return;
  }
  const TrackHead& h = *t.head;
  const float near_bits = column_near();
  const unsigned base = shared_address(t.crossings);
  ColumnState w[2];
  bool live[2];
  unsigned at[2];
#pragma unroll
  for (int k = 0; k < 2; ++k)
  {
    live[k] = go[k];
    // a LOR without work meets no z crossing
    w[k] = go[k] ? ColumnState{l[k].z, l[k].sz, l[k].az, h.amin, l[k].dz, l[k].d12}
                 : ColumnState{0, 0, 1e300, 0.0, 0.0, 0.0};
  }
  unsigned from = base;
  while (true)
  {
    run(from, w);
    // The LORs that end or may tie here take exact steps past this crossing,
    // then those short of the foremost follow, so that all are at one crossing
    // again.  None goes further: at the crossing that ends the walk all end,
    // and run makes no turn for LORs that have.
    unsigned to = from;
    at[0] = at[1] = from;
    while (true)
    {
#pragma unroll
      for (int k = 0; k < 2; ++k)
      {
        while (live[k] && at[k] <= to)
        {
          const Crossing* c = t.crossings + (int)(at[k] - base) / (int)sizeof(Crossing);
          if (at[k] == to &&
              (to != from || fabsf(__int_as_float(__double2hiint(dsub(w[k].az, c->alpha)))) >= near_bits))
          {
            break;
          }
          // FIR's step as written
          const PlainCrossing c0 = plain_crossing(c[0]), c1 = plain_crossing(c[1]);
          const double m = min_of(c0.alpha, w[k].az);
          const bool more = m < h.amax;
          const double next = more ? m : h.amax;
          emit(k, c0.col + w[k].z, dmul(dsub(next, w[k].prev), w[k].d12));
          const int taken = dsub(c0.alpha, next) < kEps ? (dsub(c1.alpha, next) < kEps ? 2 : 1) : 0;
          at[k] += (unsigned)(taken * (int)sizeof(Crossing));
          if (!more || (int)(at[k] - base) > h.exit * (int)sizeof(Crossing))
          {
            live[k] = false;
            break;
          }
          if (dsub(w[k].az, next) < kEps)
          {
            w[k].az = dadd(w[k].az, w[k].dz);
            w[k].z += w[k].sz;
          }
          w[k].prev = next;
        }
      }
      __syncwarp();
      const unsigned mine = max(live[0] ? at[0] : 0u, live[1] ? at[1] : 0u);
      to = __reduce_max_sync(kAll, mine);
      if (to == 0u)
      {
        return;
      }
      if (__all_sync(kAll, (!live[0] || at[0] == to) && (!live[1] || at[1] == to)))
      {
        from = to;
        break;
      }
    }
  }
}
}  // namespace fir
