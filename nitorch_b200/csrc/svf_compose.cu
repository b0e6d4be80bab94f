// One scaling-and-squaring step of a 3-D float32 displacement field at
// linear order: out = u + pull(u, id + u).
//
// nitorch's exp (nitorch/spatial/_svf.py:85-94, _pull_vel :323-362)
// materialises id + u and pulls every component at it, linear, dft by
// default.  The general pull kernel (flags F_IDGRID | F_ADDSELF) does the
// same for any order and dimension; this kernel is its 3-D linear float32
// case: a thread per voxel reads the voxel's three components once (they
// are the sampling offset and the added identity term), then the eight
// corners of the cell, the separable partial sums x innermost as the
// general kernel forms them.  A corner's boundary index and sign are only
// computed on axes where the cell leaves the volume; 32-bit offsets.
// Points outside the field of view without extrapolation keep the identity
// term alone, as there.
#include <cstdint>

#include "../../include/nitorch_b200.h"
#include "pp_capi_internal.cuh"
#include "pp_kernels.cuh"

namespace {

// Points of both kernels: a CTA is a tile of 8 x 32 voxels (y, z), of other
// proportions where an axis is short, a thread its (y, z) on `run` consecutive
// planes, so that a voxel's coordinates cost no division.  Planes are numbered
// n * X + x over the batch.
constexpr int SVF_THREADS = 256;

struct PlaneRun {
  int o, end, n, x;  // plane, end of the run, batch item, x
  __device__ __forceinline__ PlaneRun(int block, int run, int outer, int X) {
    o = block * run;
    end = min(o + run, outer);
    n = o / X;
    x = o - n * X;
  }
  __device__ __forceinline__ bool step(int X) {  // whether the next plane starts a batch item
    ++o;
    if (++x < X) return false;
    x = 0;
    ++n;
    return true;
  }
};

struct ComposeArgs {
  int32_t size[3], bound[3];
  int32_t extrapolate, outer, run, tzs;  // 1 << tzs: the tile along z
  float lo, hi[3];     // field of view: [lo, hi)
  int64_t fN, oN;      // batch strides
  int32_t fs[3], fC;   // field strides (elements): spatial, component
  int32_t os[3], oC;   // output strides
  const float* u;
  float* out;
};

// UV4 / OV4: the field / the output is the first three slots of a four-slot
// buffer (strides (., 4YZ, 4Z, 4, 1), 16-byte aligned): one 16-byte access
// per voxel or corner instead of three.
template <bool UV4>
__device__ __forceinline__ void load3(const float* p, int fC, float (&v)[3]) {
  if constexpr (UV4) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = q.x; v[1] = q.y; v[2] = q.z;
  } else {
    v[0] = __ldg(p); v[1] = __ldg(p + fC); v[2] = __ldg(p + 2 * fC);
  }
}

template <bool UV4, bool OV4>
__global__ void __launch_bounds__(SVF_THREADS, UV4 ? 4 : 5) svf_compose_lin3(const __grid_constant__ ComposeArgs A) {
  const int z = (static_cast<int>(blockIdx.x) << A.tzs) + (static_cast<int>(threadIdx.x) & ((1 << A.tzs) - 1));
  const int y = (static_cast<int>(blockIdx.y) << (8 - A.tzs)) + (static_cast<int>(threadIdx.x) >> A.tzs);
  if (z >= A.size[2] || y >= A.size[1]) return;
  PlaneRun P(static_cast<int>(blockIdx.z), A.run, A.outer, A.size[0]);
  auto at_u = [&](const PlaneRun& q) { return A.u + q.n * A.fN + (q.x * A.fs[0] + y * A.fs[1] + z * A.fs[2]); };
  float next[3];  // the next plane's voxel, read one ahead
  load3<UV4>(at_u(P), A.fC, next);
  while (P.o < P.end) {
    const int sub[3] = {P.x, y, z};
    const float* un = A.u + P.n * A.fN;
    float* o = A.out + P.n * A.oN + (P.x * A.os[0] + y * A.os[1] + z * A.os[2]);
    const float self[3] = {next[0], next[1], next[2]};
    float x[3];
    P.step(A.size[0]);
    if (P.o < P.end) load3<UV4>(at_u(P), A.fC, next);
#pragma unroll
    for (int d = 0; d < 3; ++d) x[d] = static_cast<float>(sub[d]) + self[d];
    bool inb = true;
    if (!(A.extrapolate & 1)) {
#pragma unroll
      for (int d = 0; d < 3; ++d) inb = inb && x[d] >= A.lo && x[d] < A.hi[d];
    }
    float res[3];
    if (!inb) {  // outside the field of view: the identity term alone
#pragma unroll
      for (int d = 0; d < 3; ++d) res[d] = self[d];
    } else {
      // per axis: the two nodes' offsets and weights (boundary sign folded in)
      int off[3][2];
      float w[3][2];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float xc = fminf(fmaxf(x[d], -1073741824.f), 1073741824.f);
        const float f = floorf(xc);
        const int i0 = static_cast<int>(f);
        const float t = xc - f;
        const int nn = A.size[d];
        const int bd = A.bound[d];
        w[d][0] = 1.f - t;
        w[d][1] = t;
        if (i0 >= 0 && i0 + 1 < nn) {
          off[d][0] = i0 * A.fs[d];
          off[d][1] = off[d][0] + A.fs[d];
        } else if (bd != ppk::BND_DST1 && bd != ppk::BND_DST2 && bd != ppk::BND_ZERO) {
          // bounds that map every node to one of the volume (signs cost the
          // edge warps as much again)
          off[d][0] = ppk::bound_index<int>(bd, i0, nn) * A.fs[d];
          off[d][1] = ppk::bound_index<int>(bd, i0 + 1, nn) * A.fs[d];
        } else {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const int s = ppk::bound_sign<int>(bd, i0 + k, nn);
            const int idx = s ? ppk::bound_index<int>(bd, i0 + k, nn) : 0;
            off[d][k] = idx * A.fs[d];
            w[d][k] *= static_cast<float>(s);
          }
        }
      }
      // separable partial sums, x innermost, the three components together
      float acc[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        float accy[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int oyz = off[1][j] + off[2][k];
          float c0[3], c1[3];
          load3<UV4>(un + off[0][0] + oyz, A.fC, c0);
          load3<UV4>(un + off[0][1] + oyz, A.fC, c1);
#pragma unroll
          for (int c = 0; c < 3; ++c) accy[c] = fmaf(w[1][j], fmaf(w[0][1], c1[c], w[0][0] * c0[c]), accy[c]);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] = fmaf(w[2][k], accy[c], acc[c]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) res[c] = acc[c] + self[c];
    }
    if constexpr (OV4) {
      *reinterpret_cast<float4*>(o) = make_float4(res[0], res[1], res[2], 0.f);
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) o[c * A.oC] = res[c];
    }
  }
}

// Its adjoint with respect to u, for g = d loss / d out: the push of g
// through the cell's eight corners, the grid gradient sum_c g_c grad(u_c),
// and the identity term g, into a four-slot channel-interleaved float
// accumulator (acc[v * 4 + c]) by vector reductions (red.global.add.v4.f32).
// Nine reductions of 16 bytes per voxel, unmerged, bind on their sectors
// through L2, so corners that neighbours share are summed in registers first:
//   * along x, a thread keeps the four upper-x corners of its cell; at the
//     next plane, a smooth field's cell is the one above, and they join its
//     four lower-x corners.  Otherwise they are reduced as they are;
//   * along z, a lane's upper-z corners are the next lane's lower-z corners
//     when that lane's cell is the next along z (whichever row of the tile it
//     has): handed over by shuffles;
//   * the voxel's own term (g and the grid gradient) joins the corner of its
//     cell that is the voxel itself, when there is one.
// A smooth field then takes about two reductions per voxel.  Cells are
// compared by their unbounded node indices: equal nodes have equal addresses
// under every bound.  Cells past the volume's edge stay on the merged path
// under bounds without signs: with a path of their own, run for a lane or two
// in every warp at the edge, they took a third of the kernel.
// 160 x 192 x 160: 0.169 -> 0.113 ms per composition (the kernel before merged
// along z only and took its coordinates from 64-bit divisions), forward 0.080
// -> 0.064 ms.  Bound by issue (65 % active, ~515 instructions per voxel and
// warp); the reductions are at 44 % of L2.
struct ComposeBwdArgs {
  int32_t size[3], bound[3];
  int32_t extrapolate, outer, run, tzs;  // 1 << tzs: the tile along z
  float lo, hi[3];
  int64_t fN, gN, aN;
  int32_t fs[3], fC;   // field strides
  int32_t gs[3], gC;   // gradient strides
  int32_t as[3];       // accumulator strides (floats): Y*Z*4, Z*4, 4
  const float* u;
  const float* g;
  float* acc;
};

__device__ __forceinline__ void red3(float* p, const float (&v)[3]) {
  const float q[4] = {v[0], v[1], v[2], 0.f};
  ppk::red_vec<4>(p, q);
}

template <bool UV4, bool GV4>
__global__ void __launch_bounds__(SVF_THREADS, 3) svf_compose_backward_lin3(const __grid_constant__ ComposeBwdArgs A) {
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int z = (static_cast<int>(blockIdx.x) << A.tzs) + (static_cast<int>(threadIdx.x) & ((1 << A.tzs) - 1));
  const int y = (static_cast<int>(blockIdx.y) << (8 - A.tzs)) + (static_cast<int>(threadIdx.x) >> A.tzs);
  const bool in_tile = z < A.size[2] && y < A.size[1];
  if (!__any_sync(0xffffffffu, in_tile)) return;  // whole warp
  // the upper-x corners of the last cell: values, accumulator offset of the
  // first and steps to the others, and the cell they are the lower-x corners of
  float up[2][2][3];
  int up_at = 0, up_dy = 0, up_dz = 0, up_cell[3] = {0, 0, 0};
  bool pending = false;
  PlaneRun P(static_cast<int>(blockIdx.z), A.run, A.outer, A.size[0]);
  float* acc = A.acc + P.n * A.aN;
  auto flush = [&]() {
    float* p = acc + up_at;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int k = 0; k < 2; ++k) red3(p + ((j ? up_dy : 0) + (k ? up_dz : 0)), up[j][k]);
    pending = false;
  };
  float nu[3] = {0.f, 0.f, 0.f}, ng[3] = {0.f, 0.f, 0.f};  // the next plane's field and gradient, read one ahead
  auto fetch = [&]() {
    if (!in_tile) return;
    load3<UV4>(A.u + P.n * A.fN + (P.x * A.fs[0] + y * A.fs[1] + z * A.fs[2]), A.fC, nu);
    load3<GV4>(A.g + P.n * A.gN + (P.x * A.gs[0] + y * A.gs[1] + z * A.gs[2]), A.gC, ng);
  };
  fetch();
  while (P.o < P.end) {
    const float* un = A.u + P.n * A.fN;
    const int px = P.x;
    const float gv[3] = {ng[0], ng[1], ng[2]};
    const float x[3] = {static_cast<float>(px) + nu[0], static_cast<float>(y) + nu[1], static_cast<float>(z) + nu[2]};
    const bool last = P.step(A.size[0]);
    if (P.o < P.end) fetch();
    bool active = in_tile;
    if (!(A.extrapolate & 1)) {
#pragma unroll
      for (int d = 0; d < 3; ++d) active = active && x[d] >= A.lo && x[d] < A.hi[d];
    }
    // the cell and the offset in it
    int cell[3];
    float t[3];
    int idx[3], dn[3];  // lower node's index, steps to the upper node
    bool inside = active;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float xc = fminf(fmaxf(x[d], -1073741824.f), 1073741824.f);
      const float f = floorf(xc);
      cell[d] = static_cast<int>(f);
      t[d] = xc - f;
      idx[d] = cell[d];
      dn[d] = 1;
      if (cell[d] < 0 || cell[d] + 1 >= A.size[d]) {
        // past the edge: bounds that map every node to one of the volume
        // stay on this path
        const int bd = A.bound[d];
        if (bd == ppk::BND_DST1 || bd == ppk::BND_DST2 || bd == ppk::BND_ZERO) {
          inside = false;
        } else {
          idx[d] = ppk::bound_index<int>(bd, cell[d], A.size[d]);
          dn[d] = ppk::bound_index<int>(bd, cell[d] + 1, A.size[d]) - idx[d];
        }
      }
    }
    float self[3] = {gv[0], gv[1], gv[2]};  // the voxel's own term
    const float w[3][2] = {{1.f - t[0], t[0]}, {1.f - t[1], t[1]}, {1.f - t[2], t[2]}};
    bool own = false;  // ... joins a corner of its cell
    const int sx = px - cell[0], sy = y - cell[1], sz = z - cell[2];
    if (inside) {
      // grid gradient: og_d = sum over corners of (derivative along d of the
      // corner weight) * <g, u(corner)>
      const float* uc = un + (idx[0] * A.fs[0] + idx[1] * A.fs[1] + idx[2] * A.fs[2]);
      const int fx = dn[0] * A.fs[0], fy = dn[1] * A.fs[1], fz = dn[2] * A.fs[2];
      float yv[2], yx[2], yy[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        float sv[2], sd[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float c0[3], c1[3];
          const float* p = uc + ((j ? fy : 0) + (k ? fz : 0));
          load3<UV4>(p, A.fC, c0);
          load3<UV4>(p + fx, A.fC, c1);
          const float d0 = fmaf(gv[2], c0[2], fmaf(gv[1], c0[1], gv[0] * c0[0]));
          const float d1 = fmaf(gv[2], c1[2], fmaf(gv[1], c1[1], gv[0] * c1[0]));
          sv[j] = fmaf(w[0][1], d1, w[0][0] * d0);
          sd[j] = d1 - d0;
        }
        yv[k] = fmaf(w[1][1], sv[1], w[1][0] * sv[0]);
        yx[k] = fmaf(w[1][1], sd[1], w[1][0] * sd[0]);
        yy[k] = sv[1] - sv[0];
      }
      self[0] += fmaf(w[2][1], yx[1], w[2][0] * yx[0]);
      self[1] += fmaf(w[2][1], yy[1], w[2][0] * yy[0]);
      self[2] += yv[1] - yv[0];
      own = ((sx | sy | sz) & ~1) == 0;
    } else if (active) {
      // bounds with signs or missing nodes: per node, every corner by itself
      int fo[3][2], ao[3][2];
      float ws[3][2], dw[3][2];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int nn = A.size[d];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int s = ppk::bound_sign<int>(A.bound[d], cell[d] + k, nn);
          const int idx = s ? ppk::bound_index<int>(A.bound[d], cell[d] + k, nn) : 0;
          fo[d][k] = idx * A.fs[d];
          ao[d][k] = s ? idx * A.as[d] : -1;
          ws[d][k] = static_cast<float>(s) * w[d][k];
          dw[d][k] = static_cast<float>(s) * (k ? 1.f : -1.f);
        }
      }
      float og[3] = {0.f, 0.f, 0.f};
#pragma unroll 1
      for (int k = 0; k < 2; ++k) {
        const int fz = k ? fo[2][1] : fo[2][0], az = k ? ao[2][1] : ao[2][0];
        const float wz = k ? ws[2][1] : ws[2][0], dz = k ? dw[2][1] : dw[2][0];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float sx_ = 0.f, dx_ = 0.f;
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            if ((ao[0][q] | ao[1][j] | az) < 0) continue;  // a corner without a node: no tap
            float cu[3];
            load3<UV4>(un + fo[0][q] + fo[1][j] + fz, A.fC, cu);
            const float dot = gv[0] * cu[0] + gv[1] * cu[1] + gv[2] * cu[2];
            sx_ = fmaf(ws[0][q], dot, sx_);
            dx_ = fmaf(dw[0][q], dot, dx_);
            const float wt = ws[0][q] * ws[1][j] * wz;
            const float v[3] = {wt * gv[0], wt * gv[1], wt * gv[2]};
            red3(acc + (ao[0][q] + ao[1][j] + az), v);
          }
          og[0] = fmaf(ws[1][j] * wz, dx_, og[0]);
          og[1] = fmaf(dw[1][j] * wz, sx_, og[1]);
          og[2] = fmaf(ws[1][j] * dz, sx_, og[2]);
        }
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) self[d] += og[d];
    }
    if (in_tile && !own) red3(acc + (px * A.as[0] + y * A.as[1] + z * A.as[2]), self);

    const bool joins = pending && inside && up_cell[0] == cell[0] && up_cell[1] == cell[1] && up_cell[2] == cell[2];
    if (pending && !joins) flush();
    // upper-z corners go to the next lane when they are its lower-z corners
    const int cx = __shfl_down_sync(0xffffffffu, cell[0], 1), cy = __shfl_down_sync(0xffffffffu, cell[1], 1),
              cz = __shfl_down_sync(0xffffffffu, cell[2], 1);
    const unsigned ins = __ballot_sync(0xffffffffu, inside);
    const bool gives = lane < 31 && inside && ((ins >> lane) & 2u) && cx == cell[0] && cy == cell[1] && cz == cell[2] + 1;
    const unsigned given = __ballot_sync(0xffffffffu, gives);
    const bool takes = lane > 0 && ((given >> (lane - 1)) & 1u);
    const int at = idx[0] * A.as[0] + idx[1] * A.as[1] + idx[2] * 4, dy = dn[1] * A.as[1], dz = dn[2] * 4;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      // lower-x corners: this cell's, the pending ones, the own term
      float lo[2][3];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float wyz = w[1][j] * w[2][k], w0 = w[0][0] * wyz, w1 = w[0][1] * wyz;
        const bool me = own && sy == j && sz == k, me0 = me && sx == 0, me1 = me && sx == 1;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          lo[k][c] = w0 * gv[c];
          if (joins) lo[k][c] += up[j][k][c];
          if (me0) lo[k][c] += self[c];
          up[j][k][c] = w1 * gv[c];
          if (me1) up[j][k][c] += self[c];
        }
      }
      if (given) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float v = __shfl_up_sync(0xffffffffu, lo[1][c], 1);
          if (takes) lo[0][c] += v;
        }
      }
      float* p = acc + (at + (j ? dy : 0));
      if (inside) red3(p, lo[0]);
      if (inside && !gives) red3(p + dz, lo[1]);
    }
    pending = inside;
    up_cell[0] = cell[0] + 1;
    up_cell[1] = cell[1];
    up_cell[2] = cell[2];
    up_at = at + dn[0] * A.as[0];
    up_dy = dy;
    up_dz = dz;
    if (last) {  // the next plane is another batch item's: its own accumulator
      if (pending) flush();
      acc = A.acc + P.n * A.aN;
    }
  }
  if (pending) flush();
}

template <class Args> void set_fov(Args& A) {
  const float tol = (A.extrapolate & 2) ? 0.55f : 0.05f;
  A.lo = -tol;
  for (int d = 0; d < 3; ++d) A.hi[d] = static_cast<float>(A.size[d] - 1) + tol;
}

// The tile's extent along z, as a power of two: 32, or what covers the plane
// with at least an eighth fewer threads (160 x 192 x 8 voxels: forward
// 16.2 -> 6.2 us, backward 29.5 -> 14.1 us; 160 x 192 x 40: 25 -> 16, 55 -> 39 us).  Then
// planes per thread, up to `most`: the number whose CTAs fill the resident
// ones' waves best (long runs share more, and pay the start of a run less
// often: `start` planes' worth); 0 where the grid does not fit a launch.
int plane_run(const int32_t (&size)[3], int64_t outer, int resident, int most, double start, dim3& grid, int32_t& tzs) {
  int64_t least = 0;
  for (int s : {5, 4, 3, 2, 1, 0, 6, 7, 8}) {
    const int64_t tz = 1 << s, ty = SVF_THREADS >> s;
    const int64_t cover = (size[2] + tz - 1) / tz * tz * ((size[1] + ty - 1) / ty * ty);
    if (s == 5 || cover * 8 < least * 7) { least = cover; tzs = s; }
  }
  const int64_t tz = 1 << tzs, ty = SVF_THREADS >> tzs;
  const int64_t gz = (size[2] + tz - 1) / tz, gy = (size[1] + ty - 1) / ty;
  const int64_t slots = int64_t(148) * resident;
  int64_t run = 1;
  double best = 0.;
  for (int64_t r = 1; r <= most && r <= outer; ++r) {
    const int64_t ctas = gz * gy * ((outer + r - 1) / r), waves = (ctas + slots - 1) / slots;
    const double cost = static_cast<double>(waves) * (r + start);
    if (r == 1 || cost < best) { best = cost; run = r; }
  }
  if ((outer + run - 1) / run > 65535) run = (outer + 65534) / 65535;
  if (gy > 65535 || outer >= (int64_t(1) << 31) - run) return 0;
  grid = dim3(static_cast<unsigned>(gz), static_cast<unsigned>(gy), static_cast<unsigned>((outer + run - 1) / run));
  return static_cast<int>(run);
}

bool fits_int(int64_t v) { return v < (int64_t(1) << 31) - 1; }

// The first three slots of a 16-byte aligned four-slot (N, X, Y, Z, 4) buffer.
bool padded4(const pp_tensor* t) {
  if (t->ndim != 5 || t->sizes[4] != 3 || reinterpret_cast<uintptr_t>(t->data) % 16 != 0) return false;
  const int64_t want[5] = {t->strides[0], t->sizes[2] * t->sizes[3] * 4, t->sizes[3] * 4, 4, 1};
  if (t->strides[0] % 4 != 0) return false;
  for (int i = 1; i < 5; ++i)
    if (t->sizes[i] > 1 && t->strides[i] != want[i]) return false;
  return true;
}

}  // namespace

namespace ppc {

// The 3-D linear float32 self-composition above, or PP_ERR_UNSUPPORTED when
// the call is not that case (the caller then runs the general kernel).
int svf_compose_linear3(const pp_tensor* disp, const pp_tensor* out, const int32_t bound[3], int32_t extrapolate,
                        cudaStream_t st) {
  if (disp->ndim != 5 || disp->sizes[4] != 3 || disp->dtype != PP_FLOAT32 || out->dtype != PP_FLOAT32)
    return PP_ERR_UNSUPPORTED;
  const int64_t per_item_f = max_offset(disp, 1), per_item_o = max_offset(out, 1);
  if (!fits_int(per_item_f + 1) || !fits_int(per_item_o + 1)) return PP_ERR_UNSUPPORTED;
  for (int d = 1; d < 4; ++d)
    if (!fits_int(disp->sizes[d])) return PP_ERR_UNSUPPORTED;
  ComposeArgs A;
  for (int d = 0; d < 3; ++d) {
    A.size[d] = static_cast<int32_t>(disp->sizes[1 + d]);
    A.bound[d] = bound[d];
    A.fs[d] = static_cast<int32_t>(disp->strides[1 + d]);
    A.os[d] = static_cast<int32_t>(out->strides[1 + d]);
  }
  A.fC = static_cast<int32_t>(disp->strides[4]);
  A.oC = static_cast<int32_t>(out->strides[4]);
  A.fN = disp->strides[0];
  A.oN = out->strides[0];
  A.extrapolate = extrapolate;
  set_fov(A);
  A.u = static_cast<const float*>(disp->data);
  A.out = static_cast<float*>(out->data);
  if (numel(disp) == 0) return PP_OK;
  dim3 nb;
  const int64_t outer = disp->sizes[0] * disp->sizes[1];
  A.run = plane_run(A.size, outer, 4, 8, 0.5, nb, A.tzs);
  if (!A.run) return PP_ERR_UNSUPPORTED;
  A.outer = static_cast<int32_t>(outer);
  ppk::note_kernel("svf_compose_lin3", ppk::K_PULL, 1, 3);
  const bool uv4 = padded4(disp), ov4 = padded4(out);
  if (uv4 && ov4) svf_compose_lin3<true, true><<<nb, SVF_THREADS, 0, st>>>(A);
  else if (uv4) svf_compose_lin3<true, false><<<nb, SVF_THREADS, 0, st>>>(A);
  else if (ov4) svf_compose_lin3<false, true><<<nb, SVF_THREADS, 0, st>>>(A);
  else svf_compose_lin3<false, false><<<nb, SVF_THREADS, 0, st>>>(A);
  count_launch();
  return cuda_check(cudaGetLastError(), "svf compose launch");
}

// The 3-D linear float32 self-composition backward into a four-slot
// channel-interleaved accumulator (zeroed by the caller, V * 4 floats per
// batch item, the last axis fastest), or PP_ERR_UNSUPPORTED (nothing
// launched) for any other field.
int svf_compose_backward_linear3(const pp_tensor* grad, const pp_tensor* disp, float* acc, const int32_t bound[3],
                                 int32_t extrapolate, cudaStream_t st) {
  if (disp->ndim != 5 || disp->sizes[4] != 3 || disp->dtype != PP_FLOAT32 || grad->dtype != PP_FLOAT32)
    return PP_ERR_UNSUPPORTED;
  const int64_t V = disp->sizes[1] * disp->sizes[2] * disp->sizes[3];
  if (!fits_int(max_offset(disp, 1) + 1) || !fits_int(max_offset(grad, 1) + 1) || !fits_int(V * 4))
    return PP_ERR_UNSUPPORTED;
  ComposeBwdArgs A;
  for (int d = 0; d < 3; ++d) {
    A.size[d] = static_cast<int32_t>(disp->sizes[1 + d]);
    A.bound[d] = bound[d];
    A.fs[d] = static_cast<int32_t>(disp->strides[1 + d]);
    A.gs[d] = static_cast<int32_t>(grad->strides[1 + d]);
  }
  A.as[2] = 4;
  A.as[1] = static_cast<int32_t>(disp->sizes[3] * 4);
  A.as[0] = static_cast<int32_t>(disp->sizes[2] * disp->sizes[3] * 4);
  A.fC = static_cast<int32_t>(disp->strides[4]);
  A.gC = static_cast<int32_t>(grad->strides[4]);
  A.fN = disp->strides[0];
  A.gN = grad->strides[0];
  A.aN = V * 4;
  A.extrapolate = extrapolate;
  set_fov(A);
  A.u = static_cast<const float*>(disp->data);
  A.g = static_cast<const float*>(grad->data);
  A.acc = acc;
  if (numel(disp) == 0) return PP_OK;
  dim3 nb;
  const int64_t outer = disp->sizes[0] * disp->sizes[1];
  A.run = plane_run(A.size, outer, 3, 32, 1.0, nb, A.tzs);
  if (!A.run) return PP_ERR_UNSUPPORTED;
  A.outer = static_cast<int32_t>(outer);
  ppk::note_kernel("svf_compose_backward_lin3", ppk::K_PUSHGRAD, 1, 3);
  const bool uv4 = padded4(disp), gv4 = padded4(grad);
  if (uv4 && gv4) svf_compose_backward_lin3<true, true><<<nb, SVF_THREADS, 0, st>>>(A);
  else if (uv4) svf_compose_backward_lin3<true, false><<<nb, SVF_THREADS, 0, st>>>(A);
  else if (gv4) svf_compose_backward_lin3<false, true><<<nb, SVF_THREADS, 0, st>>>(A);
  else svf_compose_backward_lin3<false, false><<<nb, SVF_THREADS, 0, st>>>(A);
  count_launch();
  return cuda_check(cudaGetLastError(), "svf compose backward launch");
}

}  // namespace ppc
