// Brick kernels for 3-D quadratic and cubic sampling in brick-major order.
//
// pp_brick_order sorts the sampling points by the brick (PP_BRICK_X x
// PP_BRICK_Y x PP_BRICK_Z source voxels) of their floor voxel.  A brick's
// points then touch only the brick's source window: the brick plus the
// support halo [-1, +2] of quadratic and cubic stencils, 7 x 7 x 9 voxels.
//
// pp_brick_scatter_kernel (push, count, and the image gradient of the pull's
// backward pass).  The reference scatters every tap with a global atomic add
// (nitorch/_C/src/impl/bounds_common.h:185-191, from the tap loop of
// pushpull_common.cpp:1232-1240): 64 * C float reductions per point.  Here a
// warp owns one brick and a shared accumulator window:
//   1. the window starts at zero;
//   2. points are read 32 at a time, one per lane (coordinates, the
//      out-of-bound test, B-spline weights), into shared records;
//   3. the warp walks the recorded points one at a time, lane (i, j, kk)
//      taking taps (i, j, kk) and (i, j, kk + 2) of a 4x4x4 support (27 lanes
//      the taps of a 3x3x3 support), runs of points of one support summed
//      first where there are many: plain shared read-modify-writes (the
//      lanes touch distinct voxels and the window belongs to this warp
//      alone, so no atomics);
//   4. the window is added to the output with one vector reduction per
//      touched window voxel (boundary index and sign applied there), ~14x
//      fewer global reductions than one per tap.
// Float shared-memory atomics are no alternative: on B200 they sustain
// ~0.7 T adds/s on scatter-like patterns, below the ~1-1.5 T of global
// reductions.  Bound by shared-memory wavefronts (76 % of the pipe) and
// issue (60 %).
//
// pp_brick_gather_kernel (pull, spatial gradient, push backward) and
// pp_brick_pullbwd_kernel (the grid gradient of the pull's backward pass).
// A CTA takes a group of 2 x 2 x 2 bricks, 8 x 8 x 12 voxels: its threads
// stage the group's source window in shared memory (boundary condition
// applied per window voxel: value times sign), then each thread takes points
// and gathers their taps from the window at compile-time offsets.  The
// group's window holds 2.4 voxels per voxel of the group; that of one brick,
// staged by a CTA of 128 threads, 4.6: staging was a third of the
// instructions.  Bounds are evaluated once per axis and window node, into
// tables: evaluated per voxel, inlined in an unrolled loop, they overflowed
// the instruction cache (5 of 12 stalls per issue) and took as many
// instructions as the taps.
//
// Measured on 3 x 192^3, cubic, rough deformation (std 4 over 2 voxels), one
// brick per CTA (push backward: the per-point kernel) before and this form
// after: pull 0.654 -> 0.405 ms, push backward 1.111 -> 0.555 ms, pull
// backward (was one kernel for both gradients) 1.755 -> 0.572 + 0.603 ms, push
// 0.731 -> 0.603 ms.  160 x 192 x 160, one channel: pull 0.322 -> 0.158 ms,
// grid gradient 0.583 -> 0.236 ms.  The gathers are latency-bound (scattered
// reads and writes by sample index, three or four CTAs per SM).
//
// Points whose support leaves the window (sampling outside the volume with
// extrapolation, or just below a volume edge) run the per-point body
// pp_point with global memory, after the others: a warp that met any looks
// through its samples again and collects them to full warps.  (Run where they
// are met, one or two lanes at a time in most warps of the edge bricks, they
// took a third of the kernel.)  Points outside the field of view write zeros.
//
// Window layout: voxel (x, y, z) of the window at (x * PX + y * PY + z) * CP
// floats, CP channel slots per voxel (1, 2 or 4).  In the scatter, with
// lane = kk + 2j + 8i and PY = 10, PX = 72 (voxels), the 32 lanes of a step
// fall in distinct banks for 4-, 8- and 16-byte voxels alike; the gather's
// pitches are chosen for its own access pattern (GatherWin).
#pragma once
#include "pp_kernels.cuh"
#include "../../include/nitorch_b200.h"

namespace ppk {

constexpr int BRK_X = PP_BRICK_X, BRK_Y = PP_BRICK_Y, BRK_Z = PP_BRICK_Z;

// Parameters: the general ones, the field-of-view bounds, and, where all
// per-sample tensors are laid out by the sample's index, their step per
// sample (`lin`), which saves taking the index apart.
struct BrickArgs {
  PPArgs p;
  float lo, hi[3];
  int per_item;             // samples of a batch item
  int chunk, nchunk;        // samples per chunk, chunks (see brick_chunk)
  int lin;                  // out_l, trgt_l, gg_l hold
  int out_l, trgt_l, gg_l;  // elements per sample
};

// Source window of one brick for the taps [floor(x) - 1, floor(x) + 2] of
// floor(x) in [o, o + B).
struct BrickWin {
  static constexpr int LO = 1;
  static constexpr int EX = BRK_X + 3, EY = BRK_Y + 3, EZ = BRK_Z + 3;
  static constexpr int PY = 10, PX = 72;
  static constexpr int NV = EX * PX;       // storage voxels
  static constexpr int NE = EX * EY * EZ;  // window voxels
  static_assert(PY >= EZ && PX >= EY * PY, "window pitches too small");
};

// Per-point scatter record in shared memory (floats, 16-byte aligned rows,
// five to a row of banks: a warp's records fall in distinct banks):
//   [0, 4) x tap weights   [4, 8) y tap weights
//   [8, 12) z tap weights (cubic: in the order 0, 2, 1, 3)   [12, 16) target values
//   [16] window offset of the lowest node ([15] where three channels or
//   fewer leave it free: one shared read less per point)
constexpr int BRK_REC = 20;

constexpr int BRK_SCATTER_WARPS = 4;  // warps (bricks) per scatter CTA

template <int CP> struct BrickScatterSmem {
  static constexpr int PER_WARP = BrickWin::NV * CP + 32 * BRK_REC;  // floats
  static constexpr size_t bytes = size_t(PER_WARP) * 4 * BRK_SCATTER_WARPS;
};

// Window of a gather CTA: a group of 2 x 2 x 2 bricks.  Pitches for
// thread-per-point reads: eight consecutive points (one phase of a 16-byte
// shared load) are mostly a brick's run along z, 6 voxels, and the start of
// the next column's; with PY = 6 and PX = 0 (mod 8) voxels those fall in
// distinct 16-byte bank groups.
constexpr int GRP = 2;  // bricks per axis
constexpr int BRK_GATHER_THREADS = 256;
struct GatherWin {
  static constexpr int EX = GRP * BRK_X + 3, EY = GRP * BRK_Y + 3, EZ = GRP * BRK_Z + 3;
  static constexpr int PY = 22, PX = 248;
  static constexpr int NV = EX * PX, NE = EX * EY * EZ;
  static_assert(PY >= EZ && PX >= EY * PY, "window pitches too small");
};
template <int CP> struct BrickGatherSmem {
  static constexpr size_t bytes = size_t(GatherWin::NV) * CP * 4;
};
// Resident CTAs of 256 threads the gathers are built for (register caps of 64
// and 80: a few dozen bytes spill, and the resident warps are worth more;
// 3 x 192^3 pull 0.462 -> 0.419 ms, push backward 0.725 -> 0.657 ms at one CTA
// more than without spills).
template <int MODE, int CB> struct GatherBlocks {
  static constexpr int value = MODE == K_PULL ? 4 : MODE == K_PUSHGRAD ? 3 : (CB == 1 ? 4 : 3);
};

template <int CP> __device__ __forceinline__ void vload(const float* p, float (&v)[CP]) {
  if constexpr (CP == 4) { const float4 q = *reinterpret_cast<const float4*>(p); v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w; }
  else if constexpr (CP == 2) { const float2 q = *reinterpret_cast<const float2*>(p); v[0] = q.x; v[1] = q.y; }
  else v[0] = *p;
}
template <int CP> __device__ __forceinline__ void vstore(float* p, const float (&v)[CP]) {
  if constexpr (CP == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else if constexpr (CP == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  else *p = v[0];
}

// acc[p .. p + CP) += w * t
template <int CP> __device__ __forceinline__ void vaxpy(float* p, float w, const float (&t)[CP]) {
  float v[CP];
  vload<CP>(p, v);
#pragma unroll
  for (int c = 0; c < CP; ++c) v[c] = fmaf(w, t[c], v[c]);
  vstore<CP>(p, v);
}

// Accumulator windows of the scatters, by voxel: CP = 1, 2, 4 channel slots
// interleaved per voxel; CP = 3 three channel planes BrickWin::NV floats
// apart (no padding slot: a quarter less shared-memory traffic per tap).
template <int CP> __device__ __forceinline__ void win_axpy(float* acc, int vox, float w, const float (&t)[CP]) {
  if constexpr (CP == 3) {
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[c * BrickWin::NV + vox] = fmaf(w, t[c], acc[c * BrickWin::NV + vox]);
  } else {
    vaxpy<CP>(acc + vox * CP, w, t);
  }
}
template <int CP> __device__ __forceinline__ void win_get(const float* acc, int vox, float (&v)[CP]) {
  if constexpr (CP == 3) {
#pragma unroll
    for (int c = 0; c < 3; ++c) v[c] = acc[c * BrickWin::NV + vox];
  } else {
    vload<CP>(acc + vox * CP, v);
  }
}

// Origin (absolute voxel of window voxel 0) of brick b's window, its batch
// item, and whether the window lies inside the volume on every axis.
struct BrickPos {
  int n, ox, oy, oz;
  bool interior;
};
__device__ __forceinline__ BrickPos brick_pos(const PPArgs& a, int b) {
  using W = BrickWin;
  const int nx = static_cast<int>(a.nbrick[0]), ny = static_cast<int>(a.nbrick[1]), nz = static_cast<int>(a.nbrick[2]);
  BrickPos q;
  int r = b;
  const int bz = r % nz; r /= nz;
  const int by = r % ny; r /= ny;
  const int bx = r % nx;
  q.n = r / nx;
  q.ox = bx * BRK_X - W::LO;
  q.oy = by * BRK_Y - W::LO;
  q.oz = bz * BRK_Z - W::LO;
  q.interior = q.ox >= 0 && q.oy >= 0 && q.oz >= 0 && q.ox + W::EX <= a.src_size[0] &&
               q.oy + W::EY <= a.src_size[1] && q.oz + W::EZ <= a.src_size[2];
  return q;
}

// Dense bricks.  One CTA or warp for a brick of far more samples than its
// share (a grid that samples few voxels of its source, a small source, points
// outside the volume collected in its edge bricks) would outlast the others by
// far.  So the samples in brick order are also cut into chunks of b.chunk, and
// bricks (scatter) or columns of a group's bricks (gathers) of that many
// samples or more are left to one CTA or warp per chunk: the last b.nchunk of
// the launch, of which those whose chunk does not begin in a dense brick have
// nothing to do.  (At the launch's start they delay the others, and leave the
// groups of small sources unevenly on the SMs: 64^3, 66 -> 90 us.)  A chunk's work ends where the next begins or its bricks end,
// and starts with their first sample where no chunk begins before it.
// Chunks are longer than what bricks hold of grids up to twice as dense as
// their source, whose windows are then staged or added once.
// 160^3 samples of one channel, cubic, without chunks / with them: of 20^3
// voxels, pull 1020 / 68 us, push 2990 / 188, pull backward 4540 / 280, spatial
// gradient 1380 / 89 (per point 250); of twice the volume, mirrored at its
// edges, gradient 49.6 / 0.94 ms (per point 0.66); dense grids as without.
__device__ __forceinline__ float4 brick_sample(const PPArgs& a, int p);

// Brick that holds the sample at position p of the brick order: the one that
// its coordinates name, or by bisection (a grid written since it was ordered).
__device__ __forceinline__ int brick_of(const BrickArgs& b, int p) {
  const PPArgs& a = b.p;
  const float4 r = brick_sample(a, p);
  const float x[3] = {r.x, r.y, r.z};
  const int nbricks = static_cast<int>(a.N * a.nbrick[0] * a.nbrick[1] * a.nbrick[2]);
  int q = __float_as_int(r.w) / b.per_item;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int f = x[d] >= 0.f ? static_cast<int>(fminf(x[d], static_cast<float>(a.src_size[d] - 1))) : 0;
    q = q * static_cast<int>(a.nbrick[d]) + f / (d == 0 ? BRK_X : d == 1 ? BRK_Y : BRK_Z);
  }
  q = min(max(q, 0), nbricks - 1);
  if (__ldg(a.brick_start + q) <= p && p < __ldg(a.brick_start + q + 1)) return q;
  int lo = 0, hi = nbricks;  // brick_start[lo] <= p < brick_start[hi]
  while (hi - lo > 1) {
    const int m = (lo + hi) >> 1;
    if (__ldg(a.brick_start + m) <= p) lo = m;
    else hi = m;
  }
  return lo;
}

// Samples [s0, s1) that chunk c is to work on, of those [s0, s1) of the bricks
// that its first sample lies in: empty if they are not dense.
__device__ __forceinline__ void brick_chunk(const BrickArgs& b, int c, int& s0, int& s1) {
  const int p = c * b.chunk;
  const bool dense = s1 - s0 >= b.chunk;
  if (p - b.chunk >= s0) s0 = p;
  s1 = dense ? (s1 - p > b.chunk ? p + b.chunk : s1) : s0;
}

// Window voxel e (x slowest, z fastest) -> window coordinates.
template <int EY, int EZ>
__device__ __forceinline__ void win_coords(int e, int& wx, int& wy, int& wz) {
  wx = e / (EY * EZ);
  const int rem = e - wx * (EY * EZ);
  wy = rem / EZ;
  wz = rem - wy * EZ;
}

// Add the accumulator window of brick bp to the output: one vector reduction
// per touched window voxel, boundary index and sign applied, by one warp.
// `tab`: 96 words of the warp's shared memory for the per-axis offsets and
// signs (a bound evaluated per voxel and axis costs more than the rest).
template <int CP>
__device__ __forceinline__ void flush_window(const PPArgs& a, const BrickPos& bp, const float* acc, float* tab, int lane) {
  using W = BrickWin;
  static_assert(W::EX <= 8 && W::EY <= 8 && W::EZ <= 16, "window tables");
  float* out_n = static_cast<float*>(a.out) + static_cast<int64_t>(bp.n) * a.out_sN;
  const bool vec = (a.flags & F_VEC) != 0;
  int* at = reinterpret_cast<int*>(tab);  // x at 0, y at 8, z at 16; signs 32 further
  {
    const int d = lane < 8 ? 0 : lane < 16 ? 1 : 2, k = lane < 16 ? lane & 7 : lane - 16;
    const int m = static_cast<int>(a.src_size[d]), i = (d == 0 ? bp.ox : d == 1 ? bp.oy : bp.oz) + k;
    const bool in = i >= 0 && i < m;
    const int sg = in ? 1 : bound_sign<int>(a.bound[d], i, m);
    const int ix = in ? i : sg ? bound_index<int>(a.bound[d], i, m) : 0;
    at[lane] = ix * static_cast<int>(a.out_s[d]);
    tab[32 + lane] = static_cast<float>(sg);
  }
  __syncwarp();
#pragma unroll 2
  for (int e = lane; e < W::NE; e += 32) {
    int wx, wy, wz;
    win_coords<W::EY, W::EZ>(e, wx, wy, wz);
    float v[CP];
    win_get<CP>(acc, wx * W::PX + wy * W::PY + wz, v);
    bool any = false;
#pragma unroll
    for (int c = 0; c < CP; ++c) any = any || v[c] != 0.f;
    if (!any) continue;
    const int off = at[wx] + at[8 + wy] + at[16 + wz];
    if (!bp.interior) {
      const float sg = tab[32 + wx] * tab[40 + wy] * tab[48 + wz];
      if (sg == 0.f) continue;
#pragma unroll
      for (int c = 0; c < CP; ++c) v[c] *= sg;
    }
    if constexpr (CP == 3) {
      if (vec) {  // the interleaved accumulator has four slots for three channels
        const float v4[4] = {v[0], v[1], v[2], 0.f};
        red_vec<4>(out_n + off, v4);
        continue;
      }
    } else if constexpr (CP >= 2) {
      if (vec) {
        red_vec<CP>(out_n + off, v);
        continue;
      }
    }
#pragma unroll
    for (int c = 0; c < CP; ++c)
      if (v[c] != 0.f) atomicAdd(out_n + c * a.out_sC + off, v[c]);
  }
}

// Sample p (in brick order): coordinates and index, from its record or
// through perm and the grid.
__device__ __forceinline__ float4 brick_sample(const PPArgs& a, int p) {
  if (a.brec) return __ldg(a.brec + p);
  const int v = __ldg(a.perm + p);
  int r = v;
  const int s2 = r % static_cast<int>(a.trgt_size[2]); r /= static_cast<int>(a.trgt_size[2]);
  const int s1 = r % static_cast<int>(a.trgt_size[1]); r /= static_cast<int>(a.trgt_size[1]);
  const int s0 = r % static_cast<int>(a.trgt_size[0]);
  const int n = r / static_cast<int>(a.trgt_size[0]);
  const float* gp = static_cast<const float*>(a.grid) + static_cast<int64_t>(n) * a.grid_sN + s0 * a.grid_s[0] +
                    s1 * a.grid_s[1] + s2 * a.grid_s[2];
  return make_float4(__ldg(gp), __ldg(gp + a.grid_sD), __ldg(gp + 2 * a.grid_sD), __int_as_float(v));
}

// Grid position of sample index v (batch item 0 .. N - 1 in n).
__device__ __forceinline__ void sample_sub(const PPArgs& a, int v, int (&sub)[3], int& n) {
  sub[2] = v % static_cast<int>(a.trgt_size[2]); v /= static_cast<int>(a.trgt_size[2]);
  sub[1] = v % static_cast<int>(a.trgt_size[1]); v /= static_cast<int>(a.trgt_size[1]);
  sub[0] = v % static_cast<int>(a.trgt_size[0]);
  n = v / static_cast<int>(a.trgt_size[0]);
}

// The per-point body for a sample whose support leaves the window.
template <int ORD, int CB, class S, int MODE>
__device__ __noinline__ void brick_fallback(const PPArgs& a, int v) {
  int sub[3], n;
  sample_sub(a, v, sub, n);
  pp_point<3, ORD, CB, S, MODE, int>(a, sub, n);
}

// A warp's list of sample indices in shared memory (64 slots): `add` collects
// the lanes that have one, and tells when 32 are there to `take`.
struct MissList {
  int* buf;
  int have;
  __device__ explicit MissList(int* slots) : buf(slots), have(0) {}
  __device__ __forceinline__ bool add(bool on, int v, int lane) {
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (on) buf[have + __popc(m & ((1u << lane) - 1u))] = v;
    have += __popc(m);
    __syncwarp();
    return have >= 32;
  }
  __device__ __forceinline__ int take(int lane) {
    have -= 32;
    const int v = buf[have + lane];
    __syncwarp();
    return v;
  }
  __device__ __forceinline__ bool rest(int lane) const { return lane < have; }
};

// Axis by axis: lowest support node minus the window's origin (fits: the taps
// lie in a window of extent E) and the offset of the sample in its support.
template <int ORD>
__device__ __forceinline__ bool brick_axis(float x, int o, int E, int& rel, float& f) {
  x = fminf(fmaxf(x, -1073741824.f), 1073741824.f);  // NaN -> -2^30
  const float fl = floorf(x);
  const float r = x - fl;
  rel = static_cast<int>(fl) - 1 - o;
  f = r;
  if (ORD == 2) {  // floor(x - 1/2) (r is exact where it decides, near 1/2)
    if (r >= 0.5f) rel += 1;
    f = r < 0.5f ? r + 0.5f : r - 0.5f;
  }
  return rel >= 0 && rel <= E - (ORD + 1);
}

// Offsets (elements, inside the batch item) of a sample in its tensors.
struct SampleAt {
  int64_t out, trgt, gg;
};
__device__ __forceinline__ SampleAt sample_at(const BrickArgs& b, int v, int n) {
  const int r = v - n * b.per_item;
  if (b.lin) return {static_cast<int64_t>(r) * b.out_l, static_cast<int64_t>(r) * b.trgt_l, static_cast<int64_t>(r) * b.gg_l};
  int sub[3], m;
  sample_sub(b.p, v, sub, m);
  SampleAt q;
  q.out = sub[0] * b.p.out_s[0] + sub[1] * b.p.out_s[1] + sub[2] * b.p.out_s[2];
  q.trgt = sub[0] * b.p.trgt_s[0] + sub[1] * b.p.trgt_s[1] + sub[2] * b.p.trgt_s[2];
  q.gg = sub[0] * b.p.gg_s[0] + sub[1] * b.p.gg_s[1] + sub[2] * b.p.gg_s[2];
  return q;
}

// ===========================================================================
// Scatter: one warp per brick (see the file comment).  CB: channel block of
// the per-point fallback body (= C for C <= 4); CP: window layout (1, 2, 4
// slots, 3: planes).
// ===========================================================================
// The warp walks `cnt` recorded points one at a time.  Cubic: lane (i, j, kk)
// has taps (i, j, kk) and (i, j, kk + 2) of the 4x4x4 support; quadratic: 27
// lanes one tap each of the 3x3x3 support.  RUNS: points of the same support,
// which follow one another in brick order, are summed in registers and added
// to the window at the end of their run (`ends`: bit q set where point q ends
// one); else every point is added at once.
template <int ORD, int CP, bool RUNS>
__device__ __forceinline__ void scatter_walk(float* acc, const float* rec, int cnt, unsigned ends, int lane) {
  using W = BrickWin;
  const int ti = ORD == 3 ? lane >> 3 : lane / 9, tj = ORD == 3 ? (lane >> 1) & 3 : lane / 3 % 3;
  const int tk = ORD == 3 ? lane & 1 : lane % 3;
  const int loff = ti * W::PX + tj * W::PY + tk;
  float s[2][CP] = {};
  for (int q = 0; q < cnt; ++q, rec += BRK_REC) {
    const float4 tq = *reinterpret_cast<const float4*>(rec + 12);
    const float tt[4] = {tq.x, tq.y, tq.z, tq.w};
    float t[CP];
#pragma unroll
    for (int c = 0; c < CP; ++c) t[c] = tt[c];
    const int vox0 = __float_as_int(CP < 4 ? tq.w : rec[16]) + loff;
    const float wxy = rec[ti] * rec[4 + tj];
    const float2 zp = ORD == 3 ? *reinterpret_cast<const float2*>(rec + 8 + 2 * tk)  // (wz_k, wz_k+2)
                               : make_float2(rec[8 + tk], 0.f);
    const float w0 = wxy * zp.x, w1 = wxy * zp.y;
    const bool on = ORD == 3 || lane < 27;
    if constexpr (RUNS) {
#pragma unroll
      for (int c = 0; c < CP; ++c) {
        s[0][c] = fmaf(w0, t[c], s[0][c]);
        if (ORD == 3) s[1][c] = fmaf(w1, t[c], s[1][c]);
      }
      if (ends >> q & 1) {
        if (on) win_axpy<CP>(acc, vox0, 1.f, s[0]);
        if (ORD == 3) win_axpy<CP>(acc, vox0 + 2, 1.f, s[1]);
#pragma unroll
        for (int c = 0; c < CP; ++c) s[0][c] = s[1][c] = 0.f;
        __syncwarp();
      }
    } else {
      if (on) win_axpy<CP>(acc, vox0, w0, t);
      if (ORD == 3) win_axpy<CP>(acc, vox0 + 2, w1, t);
      __syncwarp();
    }
  }
}

// Sums runs first where a warp's points have enough of them: at one run per
// point the walk with runs takes up to 7 % longer (smooth deformations), at
// 0.63 runs per point (independent uniform positions) 9 % less: 3 x 192^3,
// rough, 0.652 -> 0.600 ms.  It also rounds less often.
template <int ORD, int CP>
__device__ __forceinline__ void scatter_recorded(float* acc, const float* rec, int cnt, int lane) {
  const int at = lane < cnt ? __float_as_int(rec[lane * BRK_REC + (CP < 4 ? 15 : 16)]) : -1;
  const int next = __shfl_down_sync(0xffffffffu, at, 1);
  const unsigned ends = __ballot_sync(0xffffffffu, lane < cnt && (lane + 1 >= cnt || next != at));
  if (__popc(ends) * 8 <= cnt * 7) scatter_walk<ORD, CP, true>(acc, rec, cnt, ends, lane);
  else scatter_walk<ORD, CP, false>(acc, rec, cnt, ends, lane);
}

// Six CTAs per SM (at most 85 registers): the shared-memory budget of
// 3-channel windows holds six.
template <int MODE, int ORD, int CB, int CP, class S>
__global__ void __launch_bounds__(32 * BRK_SCATTER_WARPS, 6) pp_brick_scatter_kernel(const __grid_constant__ BrickArgs b) {
  using W = BrickWin;
  using SM = BrickScatterSmem<CP>;
  static_assert(MODE == K_PUSH || MODE == K_COUNT, "scatter modes");
  extern __shared__ float4 brick_smem4[];
  const PPArgs& a = b.p;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float* acc = reinterpret_cast<float*>(brick_smem4) + wid * SM::PER_WARP;
  float* rec = acc + W::NV * CP;

  int brick = static_cast<int>(blockIdx.x) * BRK_SCATTER_WARPS + wid;
  const int chunk = brick - static_cast<int>(a.N * a.nbrick[0] * a.nbrick[1] * a.nbrick[2]);
  if (chunk >= b.nchunk) return;  // whole warp
  if (chunk >= 0) brick = brick_of(b, chunk * b.chunk);
  int p0 = __ldg(a.brick_start + brick), p1 = __ldg(a.brick_start + brick + 1);
  if (chunk >= 0) brick_chunk(b, chunk, p0, p1);
  else if (p1 - p0 >= b.chunk) return;  // its chunks' work
  if (p0 >= p1) return;
  const BrickPos bp = brick_pos(a, brick);

  {
    float4* a4 = reinterpret_cast<float4*>(acc);
    for (int e = lane; e < W::NV * CP / 4; e += 32) a4[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncwarp();

  const S* tn = MODE == K_COUNT ? nullptr : static_cast<const S*>(a.trgt) + bp.n * a.trgt_sN;
  bool missed = false;  // this lane met a sample that contributes but does not fit
  // sample p: do its taps lie in the window?
  auto fit = [&](int p, int& v, int (&rel)[3], float (&f)[3]) {
    const float4 r = brick_sample(a, p);
    v = __float_as_int(r.w);
    const bool inb = r.x >= b.lo && r.x < b.hi[0] && r.y >= b.lo && r.y < b.hi[1] && r.z >= b.lo && r.z < b.hi[2];
    if (!inb && !(a.extrapolate & 1)) return false;
    bool ok = brick_axis<ORD>(r.x, bp.ox, W::EX, rel[0], f[0]);
    ok = brick_axis<ORD>(r.y, bp.oy, W::EY, rel[1], f[1]) && ok;
    ok = brick_axis<ORD>(r.z, bp.oz, W::EZ, rel[2], f[2]) && ok;
    missed = missed || !ok;
    return ok;
  };
  for (int c0 = p0; c0 < p1; c0 += 32) {
    const int p = c0 + lane;
    int rel[3], v = 0;
    float f[3];
    const bool mine = p < p1 && fit(p, v, rel, f);
    const unsigned todo = __ballot_sync(0xffffffffu, mine);
    if (mine) {
      float w[3][4];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        float wd[ORD + 1], g[ORD + 1];
        spline_weights<ORD, false>(f[d], wd, g);
#pragma unroll
        for (int k = 0; k < 4; ++k) w[d][k] = k <= ORD ? wd[k <= ORD ? k : 0] : 0.f;
      }
      float t[4] = {1.f, 0.f, 0.f, 0.f};
      if (MODE != K_COUNT) {
        const S* tp = tn + sample_at(b, v, bp.n).trgt;
#pragma unroll
        for (int c = 0; c < CB; ++c) t[c] = ldg_acc(tp + c * a.trgt_sC);
      }
      const float off = __int_as_float(rel[0] * W::PX + rel[1] * W::PY + rel[2]);
      if (CP < 4) t[3] = off;
      float* rr = rec + __popc(todo & ((1u << lane) - 1u)) * BRK_REC;
      *reinterpret_cast<float4*>(rr + 0) = make_float4(w[0][0], w[0][1], w[0][2], w[0][3]);
      *reinterpret_cast<float4*>(rr + 4) = make_float4(w[1][0], w[1][1], w[1][2], w[1][3]);
      *reinterpret_cast<float4*>(rr + 8) =
          ORD == 3 ? make_float4(w[2][0], w[2][2], w[2][1], w[2][3]) : make_float4(w[2][0], w[2][1], w[2][2], 0.f);
      *reinterpret_cast<float4*>(rr + 12) = make_float4(t[0], t[1], t[2], t[3]);
      if (CP == 4) rr[16] = off;
    }
    __syncwarp();
    scatter_recorded<ORD, CP>(acc, rec, __popc(todo), lane);
  }

  flush_window<CP>(a, bp, acc, rec, lane);
  __syncwarp();

  if (__any_sync(0xffffffffu, missed)) {
    // the samples that did not fit, collected to full warps: global reductions
    MissList list(reinterpret_cast<int*>(rec));
    for (int c0 = p0; c0 < p1; c0 += 32) {
      int rel[3], v = 0;
      float f[3];
      missed = false;
      if (c0 + lane < p1) fit(c0 + lane, v, rel, f);
      if (list.add(missed, v, lane)) brick_fallback<ORD, CB, S, MODE>(a, list.take(lane));
    }
    if (list.rest(lane)) brick_fallback<ORD, CB, S, MODE>(a, list.buf[lane]);
  }
}

// ===========================================================================
// Gathers: one CTA per group of bricks, a point per thread.  Modes:
//   K_PULL      out[c] = sum w src[c]
//   K_SGRAD     out[c, d] = sum dw_d src[c]; with F_A also aux[c] = sum w src[c]
//   K_PULLGRAD  push backward: out[c] = sum w src[c] (F_A), gg_d = sum_c t[c] sum dw_d src[c]
//   K_PUSHGRAD  pull backward's grid gradient: gg_d = sum_c t[c] sum dw_d src[c]
// ===========================================================================
template <int MODE, int ORD, int CB, int CP, class S>
__device__ __forceinline__ void brick_gather(const BrickArgs& b) {
  using G = GatherWin;
  constexpr int NT = ORD + 1;
  constexpr bool VAL = MODE != K_PUSHGRAD;   // values of the interpolant
  constexpr bool DOT = MODE == K_PULLGRAD || MODE == K_PUSHGRAD;  // gradient of <t, interpolant>
  constexpr bool GR = MODE != K_PULL;
  extern __shared__ float4 brick_smem4[];
  __shared__ int first[4], upto[4];  // per brick column of the group: its first sample, samples up to its end
  __shared__ int miss[BRK_GATHER_THREADS / 32][64];
  __shared__ int at_t[3][16];    // per axis of the window: node offset under the bound condition
  __shared__ float sgn_t[3][16];  // ... and sign (0: no node)
  float* img = reinterpret_cast<float*>(brick_smem4);
  const PPArgs& a = b.p;
  const int nx = static_cast<int>(a.nbrick[0]), ny = static_cast<int>(a.nbrick[1]), nz = static_cast<int>(a.nbrick[2]);
  const int gx = (nx + GRP - 1) / GRP, gy = (ny + GRP - 1) / GRP, gz = (nz + GRP - 1) / GRP;
  const int chunk = static_cast<int>(blockIdx.x) - static_cast<int>(a.N) * gx * gy * gz;
  int bx, by, bz, n, s0 = 0, s1 = 0;  // s0, s1: a chunk's samples, or those of a column (threads 0 - 3)
  if (chunk >= 0) {
    int r = brick_of(b, chunk * b.chunk);
    bz = r % nz & -GRP;
    const int q = r - r % nz + bz;
    s0 = __ldg(a.brick_start + q);
    s1 = __ldg(a.brick_start + q + min(GRP, nz - bz));
    brick_chunk(b, chunk, s0, s1);
    if (s0 >= s1) return;  // whole CTA
    if (threadIdx.x) s0 = s1 = 0;
    r /= nz;
    by = r % ny; r /= ny;
    bx = r % nx;
    n = r / nx;
  } else {
    int r = static_cast<int>(blockIdx.x);
    bz = r % gz * GRP; r /= gz;
    by = r % gy * GRP; r /= gy;
    bx = r % gx * GRP;
    n = r / gx;
    const int x = bx + static_cast<int>(threadIdx.x >> 1 & 1u), y = by + static_cast<int>(threadIdx.x & 1);
    if (threadIdx.x < 4 && x < nx && y < ny) {
      const int q = ((n * nx + x) * ny + y) * nz + bz;
      s0 = __ldg(a.brick_start + q);
      s1 = __ldg(a.brick_start + q + min(GRP, nz - bz));
      if (s1 - s0 >= b.chunk) s1 = s0;  // its chunks' work
    }
  }
  if (threadIdx.x < 4) {
    first[threadIdx.x] = s0;
    int inc = s1 - s0;
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      const int u = __shfl_up_sync(0xfu, inc, o);
      if (static_cast<int>(threadIdx.x) >= o) inc += u;
    }
    upto[threadIdx.x] = inc;
  }
  bx &= -GRP;
  by &= -GRP;
  const int ox = bx * BRK_X - 1, oy = by * BRK_Y - 1, oz = bz * BRK_Z - 1;
  if (threadIdx.x >= 32 && threadIdx.x < 32 + 48) {
    static_assert(G::EX <= 16 && G::EY <= 16 && G::EZ <= 16, "window tables");
    const int d = (static_cast<int>(threadIdx.x) - 32) >> 4, k = (static_cast<int>(threadIdx.x) - 32) & 15;
    const int m = static_cast<int>(a.src_size[d]), i = (d == 0 ? ox : d == 1 ? oy : oz) + k;
    const int sg = i >= 0 && i < m ? 1 : bound_sign<int>(a.bound[d], i, m);
    const int ix = i >= 0 && i < m ? i : sg ? bound_index<int>(a.bound[d], i, m) : 0;
    at_t[d][k] = ix * static_cast<int>(a.src_s[d]);
    sgn_t[d][k] = static_cast<float>(sg);
  }
  __syncthreads();
  const int total = upto[3];
  if (total == 0) return;  // whole CTA
  const bool interior = ox >= 0 && oy >= 0 && oz >= 0 && ox + G::EX <= a.src_size[0] && oy + G::EY <= a.src_size[1] &&
                        oz + G::EZ <= a.src_size[2];

  // ---- the window ----------------------------------------------------------
  {
    const S* sn = static_cast<const S*>(a.src) + n * a.src_sN;
    constexpr int NIT = (G::NE + BRK_GATHER_THREADS - 1) / BRK_GATHER_THREADS;
    constexpr int HALF = (NIT + 1) / 2;  // loads in flight: half of a thread's voxels at a time
#pragma unroll
    for (int h = 0; h < NIT; h += HALF) {
      float v[HALF][CP];
      int dst[HALF];
#pragma unroll
      for (int k = 0; k < HALF; ++k) {
        const int e = static_cast<int>(threadIdx.x) + (h + k) * BRK_GATHER_THREADS;
#pragma unroll
        for (int c = 0; c < CP; ++c) v[k][c] = 0.f;
        dst[k] = -1;
        if (h + k < NIT && e < G::NE) {
          int wx, wy, wz;
          win_coords<G::EY, G::EZ>(e, wx, wy, wz);
          dst[k] = (wx * G::PX + wy * G::PY + wz) * CP;
          const S* p = sn + (at_t[0][wx] + at_t[1][wy] + at_t[2][wz]);
          const float sg = interior ? 1.f : sgn_t[0][wx] * sgn_t[1][wy] * sgn_t[2][wz];
          if (sg != 0.f) {
#pragma unroll
            for (int c = 0; c < CB; ++c) v[k][c] = ldg_acc(p + c * a.src_sC);
            if (!interior) {
#pragma unroll
              for (int c = 0; c < CB; ++c) v[k][c] *= sg;
            }
          }
        }
      }
#pragma unroll
      for (int k = 0; k < HALF; ++k)
        if (dst[k] >= 0) vstore<CP>(img + dst[k], v[k]);
    }
  }
  __syncthreads();

  // ---- the points ----------------------------------------------------------
  const bool do_a = (a.flags & F_A) != 0, do_grad = (a.flags & F_GRAD) != 0;
  const int u0 = upto[0], u1 = upto[1], u2 = upto[2];
  // sample i of the group
  auto sample = [&](int i) {
    const int col = (i >= u0) + (i >= u1) + (i >= u2);
    return brick_sample(a, first[col] + i - (col ? upto[col - 1] : 0));
  };
  auto inside = [&](const float4& r) {
    return r.x >= b.lo && r.x < b.hi[0] && r.y >= b.lo && r.y < b.hi[1] && r.z >= b.lo && r.z < b.hi[2];
  };
  bool missed = false;  // this thread met a sample to compute that does not fit
  float4 next = make_float4(0.f, 0.f, 0.f, 0.f);  // the next sample, read one ahead
  if (static_cast<int>(threadIdx.x) < total) next = sample(static_cast<int>(threadIdx.x));
  for (int i = static_cast<int>(threadIdx.x); i < total; i += BRK_GATHER_THREADS) {
    const float4 rec = next;
    if (i + BRK_GATHER_THREADS < total) next = sample(i + BRK_GATHER_THREADS);
    const int v = __float_as_int(rec.w);
    const bool on = inside(rec) || (a.extrapolate & 1);
    int rx, ry, rz;
    float fx, fy, fz;
    bool fits = brick_axis<ORD>(rec.x, ox, G::EX, rx, fx);
    fits = brick_axis<ORD>(rec.y, oy, G::EY, ry, fy) && fits;
    fits = brick_axis<ORD>(rec.z, oz, G::EZ, rz, fz) && fits;
    if (on && !fits) {
      missed = true;
      continue;
    }
    const SampleAt at = sample_at(b, v, n);
    // target values: read before the taps, used after them
    float t[CB];
#pragma unroll
    for (int c = 0; c < CB; ++c) t[c] = 0.f;
    if (DOT && do_grad && on) {
      const S* tp = static_cast<const S*>(a.trgt) + n * a.trgt_sN + at.trgt;
#pragma unroll
      for (int c = 0; c < CB; ++c) t[c] = ldg_acc(tp + c * a.trgt_sC);
    }
    // separable partial sums per channel, x innermost
    float val[CB], sx[CB], sy[CB], sz[CB];
#pragma unroll
    for (int c = 0; c < CB; ++c) val[c] = sx[c] = sy[c] = sz[c] = 0.f;
    if (on) {  // (points outside the field of view: zeros)
      float wx[NT], wy[NT], wz[NT], dx[NT], dy[NT], dz[NT];
      spline_weights<ORD, GR>(fx, wx, dx);
      spline_weights<ORD, GR>(fy, wy, dy);
      spline_weights<ORD, GR>(fz, wz, dz);
      const float* ib = img + (rx * G::PX + ry * G::PY + rz) * CP;
#pragma unroll
      for (int k = 0; k < NT; ++k) {
        float yv[CB], yx[CB], yy[CB];
#pragma unroll
        for (int c = 0; c < CB; ++c) yv[c] = yx[c] = yy[c] = 0.f;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          float xv[CB], xd[CB];
#pragma unroll
          for (int q = 0; q < NT; ++q) {
            float iv[CP];
            vload<CP>(ib + (q * G::PX + j * G::PY + k) * CP, iv);
#pragma unroll
            for (int c = 0; c < CB; ++c) {
              xv[c] = q == 0 ? wx[0] * iv[c] : fmaf(wx[q], iv[c], xv[c]);
              if (GR) xd[c] = q == 0 ? dx[0] * iv[c] : fmaf(dx[q], iv[c], xd[c]);
            }
          }
#pragma unroll
          for (int c = 0; c < CB; ++c) {
            yv[c] = fmaf(wy[j], xv[c], yv[c]);
            if (GR) {
              yx[c] = fmaf(wy[j], xd[c], yx[c]);
              yy[c] = fmaf(dy[j], xv[c], yy[c]);
            }
          }
        }
#pragma unroll
        for (int c = 0; c < CB; ++c) {
          if (VAL) val[c] = fmaf(wz[k], yv[c], val[c]);
          if (GR) {
            sx[c] = fmaf(wz[k], yx[c], sx[c]);
            sy[c] = fmaf(wz[k], yy[c], sy[c]);
            sz[c] = fmaf(dz[k], yv[c], sz[c]);
          }
        }
      }
    }
    S* op = static_cast<S*>(a.out) + n * a.out_sN + at.out;
#pragma unroll
    for (int c = 0; c < CB; ++c) {
      if (MODE == K_PULL || (MODE == K_PULLGRAD && do_a)) op[c * a.out_sC] = from_acc<S>(val[c]);
      if (MODE == K_SGRAD) {
        S* oc = op + c * a.out_sC;
        oc[0] = from_acc<S>(sx[c]); oc[a.out_sK] = from_acc<S>(sy[c]); oc[2 * a.out_sK] = from_acc<S>(sz[c]);
        if (do_a) (static_cast<S*>(a.aux) + n * a.trgt_sN + at.trgt)[c * a.trgt_sC] = from_acc<S>(val[c]);
      }
    }
    if (DOT && do_grad) {
      float g0 = t[0] * sx[0], g1 = t[0] * sy[0], g2 = t[0] * sz[0];
#pragma unroll
      for (int c = 1; c < CB; ++c) {
        g0 = fmaf(t[c], sx[c], g0);
        g1 = fmaf(t[c], sy[c], g1);
        g2 = fmaf(t[c], sz[c], g2);
      }
      float* gg = static_cast<float*>(a.gg) + n * a.gg_sN + at.gg;
      gg[0] = g0; gg[a.gg_sD] = g1; gg[2 * a.gg_sD] = g2;
    }
  }
  if (__any_sync(0xffffffffu, missed)) {
    // the samples that did not fit, collected to full warps: global memory
    const int lane = static_cast<int>(threadIdx.x) & 31;
    MissList list(miss[threadIdx.x >> 5]);
    for (int i0 = static_cast<int>(threadIdx.x) - lane; i0 < total; i0 += BRK_GATHER_THREADS) {
      bool on = false;
      int v = 0;
      if (i0 + lane < total) {
        const float4 rec = sample(i0 + lane);
        int r_;
        float f_;
        bool fits = brick_axis<ORD>(rec.x, ox, G::EX, r_, f_);
        fits = brick_axis<ORD>(rec.y, oy, G::EY, r_, f_) && fits;
        fits = brick_axis<ORD>(rec.z, oz, G::EZ, r_, f_) && fits;
        on = !fits && (inside(rec) || (a.extrapolate & 1));
        v = __float_as_int(rec.w);
      }
      if (list.add(on, v, lane)) brick_fallback<ORD, CB, S, MODE>(a, list.take(lane));
    }
    if (list.rest(lane)) brick_fallback<ORD, CB, S, MODE>(a, list.buf[lane]);
  }
}

template <int MODE, int ORD, int CB, int CP, class S>
__global__ void __launch_bounds__(BRK_GATHER_THREADS, GatherBlocks<MODE, CB>::value)
    pp_brick_gather_kernel(const __grid_constant__ BrickArgs b) {
  brick_gather<MODE, ORD, CB, CP, S>(b);
}
template <int ORD, int CB, int CP, class S>
__global__ void __launch_bounds__(BRK_GATHER_THREADS, GatherBlocks<K_PUSHGRAD, CB>::value)
    pp_brick_pullbwd_kernel(const __grid_constant__ BrickArgs b) {
  brick_gather<K_PUSHGRAD, ORD, CB, CP, S>(b);
}

// Dynamic shared memory above 48 KB must be opted into, once per kernel and
// device: `done` is the caller's per-instantiation record of the devices
// already set up (bit d = device d).  `carve`: percentage of the unified L1 /
// shared array that the resident CTAs' windows need.
template <class K>
inline cudaError_t brick_smem_optin(K kernel, size_t bytes, std::atomic<unsigned long long>& done,
                                    int carve = cudaSharedmemCarveoutMaxShared) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (done.load(std::memory_order_relaxed) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, carve);
  if (e == cudaSuccess) done.fetch_or(bit);
  return e;
}

// Chunks of a power of two samples, `least` or more, up to `most` chunks.
inline void set_chunks(BrickArgs& b, int64_t most, int64_t least) {
  int64_t chunk = least;
  while (chunk * most < b.p.nvox) chunk *= 2;
  b.chunk = static_cast<int>(chunk);
  b.nchunk = static_cast<int>((b.p.nvox + chunk - 1) / chunk);
}

template <int MODE, int ORD, int CB, class S>
inline cudaError_t launch_brick_scatter(BrickArgs b, cudaStream_t st) {
  constexpr int CP = CB;  // 3: channel planes
  constexpr size_t bytes = BrickScatterSmem<CP>::bytes;
  const PPArgs& a = b.p;
  set_chunks(b, 148 * 6 * BRK_SCATTER_WARPS, 1024);  // up to one per resident warp
  const int64_t grid =
      (b.nchunk + a.N * a.nbrick[0] * a.nbrick[1] * a.nbrick[2] + BRK_SCATTER_WARPS - 1) / BRK_SCATTER_WARPS;
  static std::atomic<unsigned long long> optin_done{0};  // one per kernel instantiation
  cudaError_t e = brick_smem_optin(pp_brick_scatter_kernel<MODE, ORD, CB, CP, S>, bytes, optin_done);
  if (e != cudaSuccess) return e;
  note_kernel("pp_brick_scatter_kernel", MODE, ORD, CB);
  pp_brick_scatter_kernel<MODE, ORD, CB, CP, S><<<static_cast<unsigned>(grid), 32 * BRK_SCATTER_WARPS, bytes, st>>>(b);
  return cudaGetLastError();
}

template <int MODE, int ORD, int CB, class S>
inline cudaError_t launch_brick_gather(BrickArgs b, cudaStream_t st) {
  constexpr int CP = CB == 3 ? 4 : CB;
  constexpr size_t bytes = BrickGatherSmem<CP>::bytes;
  const PPArgs& a = b.p;
  set_chunks(b, 4 * 148 * GatherBlocks<MODE, CB>::value, 2048);  // up to four per resident CTA
  int64_t grid = a.N;
  for (int d = 0; d < 3; ++d) grid *= (a.nbrick[d] + GRP - 1) / GRP;
  grid += b.nchunk;
  static std::atomic<unsigned long long> optin_done{0};
  // the rest stays L1, for the samples' scattered reads and writes and the
  // points past the window (160^3, one channel, all of it as shared memory: pull
  // 143 -> 132 us, gradient 166 -> 152; mostly outside points 1.88 -> 1.14 ms)
  constexpr int carve = static_cast<int>(
      std::min<size_t>(100, (bytes + 3584) * GatherBlocks<MODE, CB>::value * 100 / (228 * 1024) + 1));
  if constexpr (MODE == K_PUSHGRAD) {
    cudaError_t e = brick_smem_optin(pp_brick_pullbwd_kernel<ORD, CB, CP, S>, bytes, optin_done, carve);
    if (e != cudaSuccess) return e;
    note_kernel("pp_brick_pullbwd_kernel", MODE, ORD, CB);
    pp_brick_pullbwd_kernel<ORD, CB, CP, S><<<static_cast<unsigned>(grid), BRK_GATHER_THREADS, bytes, st>>>(b);
  } else {
    cudaError_t e = brick_smem_optin(pp_brick_gather_kernel<MODE, ORD, CB, CP, S>, bytes, optin_done, carve);
    if (e != cudaSuccess) return e;
    note_kernel("pp_brick_gather_kernel", MODE, ORD, CB);
    pp_brick_gather_kernel<MODE, ORD, CB, CP, S><<<static_cast<unsigned>(grid), BRK_GATHER_THREADS, bytes, st>>>(b);
  }
  return cudaGetLastError();
}

// Brick kernels of one mode.  The pull's backward pass is two kernels: the
// scatter of the incoming gradient (image gradient) and the gather of the grid
// gradient.
template <int MODE, int ORD, int CB, class S>
inline cudaError_t launch_brick(const PPArgs& p, cudaStream_t st) {
  BrickArgs b;
  b.p = p;
  const float tol = (p.extrapolate & 2) ? 0.55f : 0.05f;
  b.lo = -tol;
  int64_t per = 1;
  for (int d = 0; d < 3; ++d) {
    b.hi[d] = static_cast<float>(p.src_size[d] - 1) + tol;
    per *= p.trgt_size[d];
  }
  b.per_item = static_cast<int>(per);
  // strides (s Y Z, s Z, s): s elements per sample
  auto linear = [&](const int64_t (&s)[3], int& l) {
    l = static_cast<int>(s[2]);
    return (p.trgt_size[1] == 1 || s[1] == s[2] * p.trgt_size[2]) &&
           (p.trgt_size[0] == 1 || s[0] == s[2] * p.trgt_size[2] * p.trgt_size[1]) && s[2] < (1 << 30);
  };
  constexpr bool scatters = MODE == K_PUSH || MODE == K_COUNT || MODE == K_PUSHGRAD;
  bool lin = linear(p.trgt_s, b.trgt_l) && linear(p.gg_s, b.gg_l);  // (unused tensors have strides 0)
  b.out_l = 0;
  if (!scatters) lin = linear(p.out_s, b.out_l) && lin;
  b.lin = lin;
  if constexpr (MODE == K_PUSH || MODE == K_COUNT) {
    return launch_brick_scatter<MODE, ORD, CB, S>(b, st);
  } else if constexpr (MODE == K_PUSHGRAD) {
    if (p.flags & F_A) {
      BrickArgs s = b;
      s.p.flags &= ~F_GRAD;
      const cudaError_t e = launch_brick_scatter<K_PUSH, ORD, CB, S>(s, st);
      if (e != cudaSuccess || !(p.flags & F_GRAD)) return e;
    }
    b.p.flags &= ~F_A;
    return launch_brick_gather<MODE, ORD, CB, S>(b, st);
  } else {
    return launch_brick_gather<MODE, ORD, CB, S>(b, st);
  }
}

template <int ORD, class S, int MODE>
inline cudaError_t launch_brick_cb(const PPArgs& a, cudaStream_t st) {
  if constexpr (MODE != K_COUNT) {
    switch (static_cast<int>(a.C)) {
      case 2: return launch_brick<MODE, ORD, 2, S>(a, st);
      case 3: return launch_brick<MODE, ORD, 3, S>(a, st);
      case 4: return launch_brick<MODE, ORD, 4, S>(a, st);
      default: break;
    }
  }
  return launch_brick<MODE, ORD, 1, S>(a, st);
}

}  // namespace ppk
