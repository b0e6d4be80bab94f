// Direct kernels: sampling in the grid's own order for stencils of few taps
// (3-D linear, and quadratic where no brick order is given; 2-D linear,
// quadratic and cubic), float arithmetic.
//
// The per-point kernel (pp_kernel) serves every order, bound, stride width
// and flag; its index arithmetic -- 64-bit strides, per-tap offsets and
// masks, a linear index taken apart by divisions -- costs a linear sample
// several hundred instructions for 8 taps.  Here a CTA is a tile of the grid
// (32 points along the last axis by 8, narrower where that fits a short axis
// better), sizes and strides arrive as 32-bit kernel parameters, and a point
// whose support lies inside the volume takes a path without bound conditions.
//
// The points stay in the grid's order: a sample order is not worth its sort
// here.  Sorting 9.8 M points costs 0.26 ms and makes the linear pull slower
// (0.205 ms against 0.187 ms for the per-point kernel in natural order); its
// gain is for the 64-tap stencils of the brick kernels.
//
// Scatters (push, count, the image gradient of the pull's backward pass).
// Reductions to global memory cost by the 32-byte sectors that each
// instruction touches, and a point's taps along the last axis lie in one
// sector or two.  So a point's taps along the last axis are spread over two
// (linear) or four consecutive lanes before they are reduced, 16 or 8 points
// to an instruction: 35.6 M sectors for the 9.8 M points below, 44.4 M with
// one lane per point.  (Summing neighbouring lanes' shared nodes through
// shuffles first measured slower: 345 us against 318 us.)
//
// Measured on 2 x 1 x 160 x 192 x 160 float32, linear, smooth displacement
// (std 3 over 6 voxels), per-point / lane-split kernels before and these
// after: pull 205 -> 120 us, pull backward 555 -> 311 us, and the 255 us
// sort is gone; push of 256^3 627 -> 298 us; 4 x 8 x 512^2 cubic pull 178 ->
// 75 us, backward 482 -> 218 us.  What bounds them: instruction issue (58 %
// active, ~245 instructions per linear pull) and L1 latency for the gathers,
// the reductions' sectors through L1 and L2 (72 % and 57 % of peak) for the
// scatters.
#pragma once
#include "pp_kernels.cuh"

namespace ppk {

constexpr int DIR_THREADS = 256;

// Parameters of a direct kernel: element strides and sizes inside a batch
// item, axes in the order (x, y, z) with z the last axis (2-D: x of size 1).
struct DirArgs {
  const void* src;
  const void* trgt;
  const float* grid;
  void* out;
  float* gg;
  void* aux;
  int64_t src_sN, trgt_sN, grid_sN, out_sN, gg_sN, src_sC, out_sC;
  int X, Y, Z, outer;   // grid sizes; outer = batch items * X
  int n[3];             // source sizes
  int src_s[3], trgt_s[3], grid_s[3], out_s[3], gg_s[3];
  int trgt_sC, grid_sD, out_sK, gg_sD;
  int bound[3];
  float lo, hi[3];      // field of view: [lo, hi)
  float invX;
  int C, extrapolate, flags, tzs, run;
};

// Stencil of one axis: node offsets (elements) in the gathered and the
// scattered tensor, weights and derivative weights with the boundary sign
// folded in; bit k of `mask` is clear where tap k has no node (zero and dst1
// bounds), its weights and offsets are then zero.
template <int NT> struct DirAxis {
  float w[NT], g[NT];
  int os[NT], oo[NT];
  unsigned mask;
};

template <int ORD, bool NEED_G, bool NEED_OS, bool NEED_OO>
__device__ __forceinline__ void dir_axis(DirAxis<ORD + 1>& ax, int bnd, float x, int n, int ss, int so) {
  constexpr int NT = ORD + 1;
  x = fminf(fmaxf(x, -1073741824.f), 1073741824.f);  // NaN -> -2^30
  const float fl = floorf(x);
  const float r = x - fl;
  float f = r;
  int low = static_cast<int>(fl);
  if (ORD == 3) low -= 1;
  if (ORD == 2) {  // floor(x - 1/2): r is exact where it decides (r near 1/2)
    if (r < 0.5f) low -= 1;
    f = r < 0.5f ? r + 0.5f : r - 0.5f;
  }
  spline_weights<ORD, NEED_G>(f, ax.w, ax.g);
  ax.mask = (1u << NT) - 1u;
  if (low >= 0 && low + NT <= n) {
#pragma unroll
    for (int k = 0; k < NT; ++k) {
      if (NEED_OS) ax.os[k] = k == 0 ? low * ss : ax.os[k - 1] + ss;
      if (NEED_OO) ax.oo[k] = k == 0 ? low * so : ax.oo[k - 1] + so;
    }
  } else {
#pragma unroll
    for (int k = 0; k < NT; ++k) {
      const int s = bound_sign<int>(bnd, low + k, n);
      const int i = s ? bound_index<int>(bnd, low + k, n) : 0;
      if (s == 0) ax.mask &= ~(1u << k);
      ax.w[k] *= static_cast<float>(s);
      if (NEED_G) ax.g[k] *= static_cast<float>(s);
      if (NEED_OS) ax.os[k] = i * ss;
      if (NEED_OO) ax.oo[k] = i * so;
    }
  }
}

// Resident CTAs of 256 threads the register budget is set for.
template <int D, int ORD, int MODE, int CB> struct DirBlocks {
  static constexpr bool one = MODE == K_PULL || MODE == K_PUSH || MODE == K_COUNT;
  static constexpr int value = ORD > 1 ? (one ? 3 : 2) : one ? (CB == 1 ? 5 : 4) : (CB == 1 ? 4 : 3);
};

// MODE as in pp_kernel: K_PULL, K_SGRAD, K_PUSH, K_COUNT, K_PULLGRAD,
// K_PUSHGRAD; 1 << tzs points of a CTA's tile lie along the last axis.
//
// Grid gradient, sum_c t[c] sum_nodes dw src[c]: the nodes' differences first,
// each channel's by itself, its product with t after them.  DOT: the products
// of all channels first, one sum over the nodes of their dot product; fewer
// registers, but the differences then carry the rounding of the products (rms
// error of 2-D linear gradients of a smooth 4-channel image: 4.7e-7 against
// 2.2e-7; 4 x 8 x 512^2 cubic, both passes: 293 and 300 us).  Only the
// 3-D linear pull backward of two to four channels sums so, as its lane-split
// kernel (pp_lanes_pullbwd_kernel) does.
template <int D, int ORD, int CB, class S, int MODE, bool DOT>
__global__ void __launch_bounds__(DIR_THREADS, (DirBlocks<D, ORD, MODE, CB>::value))
    pp_direct_kernel(const __grid_constant__ DirArgs a) {
  constexpr int NT = ORD + 1;
  constexpr int NX = D == 3 ? NT : 1;  // taps along axes before the last two
  constexpr bool GATHER = MODE != K_PUSH && MODE != K_COUNT;
  constexpr bool SCATTER = MODE == K_PUSH || MODE == K_COUNT || MODE == K_PUSHGRAD;
  constexpr bool NEED_G = MODE == K_SGRAD || MODE == K_PULLGRAD || MODE == K_PUSHGRAD;
  const int z = (static_cast<int>(blockIdx.x) << a.tzs) + (static_cast<int>(threadIdx.x) & ((1 << a.tzs) - 1));
  const int y = (static_cast<int>(blockIdx.y) << (8 - a.tzs)) + (static_cast<int>(threadIdx.x) >> a.tzs);
  const bool in_tile = z < a.Z && y < a.Y;
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const bool do_a = (a.flags & F_A) != 0, do_grad = (a.flags & F_GRAD) != 0;

  // This thread's points: (y, z) on `run` consecutive planes of the grid
  // (2-D: one image), so that the index arithmetic is done once per run.
  int o = static_cast<int>(blockIdx.z) * a.run;
  const int end = min(o + a.run, a.outer);
  int n = o, x = 0;
  if (D == 3) {  // o = n X + x (o < 2^24: the quotient is off by one at most)
    n = static_cast<int>(static_cast<float>(o) * a.invX);
    x = o - n * a.X;
    if (x < 0) { --n; x += a.X; }
    else if (x >= a.X) { ++n; x -= a.X; }
  }
  const float* gp;   // the point's coordinates
  float* gg;         // ... grid gradient
  S* op;             // ... outputs (gathers)
  S* vp;             // ... values (K_SGRAD)
  const S* tp;       // ... target values
  const S* sn;       // gathered image of the batch item
  float* on;         // scattered image of the batch item
  auto start = [&]() {  // pointers of point (n, x, y, z)
    auto at = [&](const int (&s)[3]) { return (D == 3 ? x * s[0] : 0) + y * s[1] + z * s[2]; };
    gp = a.grid + n * a.grid_sN + at(a.grid_s);
    if (NEED_G && MODE != K_SGRAD) gg = a.gg + n * a.gg_sN + at(a.gg_s);
    if (MODE == K_PULL || MODE == K_SGRAD || MODE == K_PULLGRAD) op = static_cast<S*>(a.out) + n * a.out_sN + at(a.out_s);
    if (MODE == K_SGRAD) vp = static_cast<S*>(a.aux) + n * a.trgt_sN + at(a.trgt_s);
    if (MODE == K_PUSH || MODE == K_PULLGRAD || MODE == K_PUSHGRAD)
      tp = static_cast<const S*>(a.trgt) + n * a.trgt_sN + at(a.trgt_s);
    if (GATHER) sn = static_cast<const S*>(a.src) + n * a.src_sN;
    if (SCATTER) on = static_cast<float*>(a.out) + n * a.out_sN;
  };
  auto step = [&]() {  // on to the next plane
    if (D == 3 && ++x < a.X) {
      gp += a.grid_s[0];
      if (NEED_G && MODE != K_SGRAD) gg += a.gg_s[0];
      if (MODE == K_PULL || MODE == K_SGRAD || MODE == K_PULLGRAD) op += a.out_s[0];
      if (MODE == K_SGRAD) vp += a.trgt_s[0];
      if (MODE == K_PUSH || MODE == K_PULLGRAD || MODE == K_PUSHGRAD) tp += a.trgt_s[0];
    } else {
      x = 0;
      ++n;
      start();
    }
  };
  auto coords = [&](float (&v)[3]) {
    if (!in_tile) return;
#pragma unroll
    for (int d = 3 - D; d < 3; ++d) v[d] = __ldg(gp + (d - (3 - D)) * a.grid_sD);
  };
  start();
  float ahead[3] = {0.f, 0.f, 0.f};  // coordinates of the next point, read one point ahead
  coords(ahead);

  for (; o < end; ++o, step()) {
    float c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) c[d] = ahead[d];
    if (o + 1 < end) {
      const bool same = D == 3 && x + 1 < a.X;
      const float* gq = gp;
      if (same) gp += a.grid_s[0];
      else gp = a.grid + (n + 1) * a.grid_sN + y * a.grid_s[1] + z * a.grid_s[2];
      coords(ahead);
      gp = gq;
    }
    bool live = false;
    if (in_tile) {
      live = true;
#pragma unroll
      for (int d = 3 - D; d < 3; ++d) live = live && c[d] >= a.lo && c[d] < a.hi[d];
      live = live || (a.extrapolate & 1);
    }

    if (in_tile && !live) {  // outside the field of view: zeros
      if (MODE == K_PULL || (MODE == K_PULLGRAD && do_a))
        for (int q = 0; q < a.C; ++q) op[q * a.out_sC] = from_acc<S>(0.f);
      if (MODE == K_SGRAD) {
        for (int q = 0; q < a.C; ++q) {
#pragma unroll
          for (int d = 0; d < D; ++d) op[q * a.out_sC + d * a.out_sK] = from_acc<S>(0.f);
          if (do_a) vp[q * a.trgt_sC] = from_acc<S>(0.f);
        }
      }
      if ((MODE == K_PULLGRAD || MODE == K_PUSHGRAD) && do_grad) {
#pragma unroll
        for (int d = 0; d < D; ++d) gg[d * a.gg_sD] = 0.f;
      }
    }
    if (!SCATTER && !live) continue;

    DirAxis<NX> ax;
    DirAxis<NT> ay, az;
    if constexpr (D == 3) {
      dir_axis<ORD, NEED_G, GATHER, SCATTER>(ax, a.bound[0], c[0], a.n[0], a.src_s[0], a.out_s[0]);
    } else {
      ax.w[0] = 1.f; ax.g[0] = 0.f; ax.os[0] = ax.oo[0] = 0; ax.mask = 1u;
    }
    dir_axis<ORD, NEED_G, GATHER, SCATTER>(ay, a.bound[1], c[1], a.n[1], a.src_s[1], a.out_s[1]);
    dir_axis<ORD, NEED_G, GATHER, SCATTER>(az, a.bound[2], c[2], a.n[2], a.src_s[2], a.out_s[2]);
    const bool full = ax.mask == (1u << NX) - 1u && ay.mask == (1u << NT) - 1u && az.mask == (1u << NT) - 1u;

    float og[3] = {0.f, 0.f, 0.f};
    const int C = MODE == K_COUNT ? 1 : a.C;
    for (int c0 = 0; c0 < C; c0 += CB) {
      const int nc = C - c0 < CB ? C - c0 : CB;
      float t[CB];
#pragma unroll
      for (int q = 0; q < CB; ++q) {
        t[q] = 0.f;
        if (MODE == K_COUNT) t[q] = live ? 1.f : 0.f;
        if ((MODE == K_PUSH || MODE == K_PULLGRAD || MODE == K_PUSHGRAD) && live && (CB == 1 || q < nc))
          t[q] = (MODE == K_PUSHGRAD && (a.flags & F_NOTRGT)) ? 1.f : ldg_acc(tp + (c0 + q) * a.trgt_sC);
      }
      // ---- gather: separable sums, the first axis innermost ------------------
      if (GATHER && live && (MODE != K_PUSHGRAD || do_grad)) {
        const S* sp = sn + c0 * a.src_sC;
        constexpr int NGC = DOT ? 1 : CB;  // gradients of the dot product with t, or per channel
        float val[CB], gx[NGC], gy[NGC], gz[NGC];
#pragma unroll
        for (int q = 0; q < CB; ++q) val[q] = 0.f;
#pragma unroll
        for (int q = 0; q < NGC; ++q) gx[q] = gy[q] = gz[q] = 0.f;
        auto taps = [&](auto all) {
#pragma unroll
          for (int k = 0; k < NT; ++k) {
            float zv[CB], zw[NGC], zgx[NGC], zgy[NGC];
#pragma unroll
            for (int q = 0; q < CB; ++q) zv[q] = 0.f;
#pragma unroll
            for (int q = 0; q < NGC; ++q) zw[q] = zgx[q] = zgy[q] = 0.f;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              const int oyz = ay.os[j] + az.os[k];
              float sv[CB], sw[NGC], sd[NGC];
#pragma unroll
              for (int q = 0; q < CB; ++q) sv[q] = 0.f;
#pragma unroll
              for (int q = 0; q < NGC; ++q) sw[q] = sd[q] = 0.f;
#pragma unroll
              for (int i = 0; i < NX; ++i) {
                const S* p = sp + (ax.os[i] + oyz);
                const bool ok = decltype(all)::value || (((ax.mask >> i) & (ay.mask >> j) & (az.mask >> k)) & 1u);
                float v[CB];
#pragma unroll
                for (int q = 0; q < CB; ++q) v[q] = (ok && (CB == 1 || q < nc)) ? ldg_acc(p + q * a.src_sC) : 0.f;
                if (!DOT) {
#pragma unroll
                  for (int q = 0; q < CB; ++q) {
                    sv[q] = D == 3 ? fmaf(ax.w[i], v[q], sv[q]) : v[q];
                    if (NEED_G && D == 3) sd[q] = fmaf(ax.g[i], v[q], sd[q]);
                  }
                } else {
                  float dot = t[0] * v[0];
#pragma unroll
                  for (int q = 1; q < CB; ++q) dot = fmaf(t[q], v[q], dot);
                  sw[0] = D == 3 ? fmaf(ax.w[i], dot, sw[0]) : dot;
                  if (D == 3) sd[0] = fmaf(ax.g[i], dot, sd[0]);
                }
              }
#pragma unroll
              for (int q = 0; q < CB; ++q)
                if (!DOT) zv[q] = fmaf(ay.w[j], sv[q], zv[q]);
              if (NEED_G) {
#pragma unroll
                for (int q = 0; q < NGC; ++q) {
                  const float s0 = DOT ? sw[q] : sv[q];
                  if (DOT) zw[q] = fmaf(ay.w[j], s0, zw[q]);
                  if (D == 3) zgx[q] = fmaf(ay.w[j], sd[q], zgx[q]);
                  zgy[q] = fmaf(ay.g[j], s0, zgy[q]);
                }
              }
            }
#pragma unroll
            for (int q = 0; q < CB; ++q)
              if (MODE != K_PUSHGRAD) val[q] = fmaf(az.w[k], zv[q], val[q]);
            if (NEED_G) {
#pragma unroll
              for (int q = 0; q < NGC; ++q) {
                if (D == 3) gx[q] = fmaf(az.w[k], zgx[q], gx[q]);
                gy[q] = fmaf(az.w[k], zgy[q], gy[q]);
                gz[q] = fmaf(az.g[k], DOT ? zw[q] : zv[q], gz[q]);
              }
            }
          }
        };
        if (full) taps(std::true_type{});
        else taps(std::false_type{});
#pragma unroll
        for (int q = 0; q < CB; ++q) {
          if (CB > 1 && q >= nc) continue;
          if (MODE == K_PULL || (MODE == K_PULLGRAD && do_a)) op[(c0 + q) * a.out_sC] = from_acc<S>(val[q]);
          if (MODE == K_SGRAD) {
            S* oq = op + (c0 + q) * a.out_sC;
            if (D == 3) {
              oq[0] = from_acc<S>(gx[q]); oq[a.out_sK] = from_acc<S>(gy[q]); oq[2 * a.out_sK] = from_acc<S>(gz[q]);
            } else {
              oq[0] = from_acc<S>(gy[q]); oq[a.out_sK] = from_acc<S>(gz[q]);
            }
            if (do_a) vp[(c0 + q) * a.trgt_sC] = from_acc<S>(val[q]);
          }
        }
        if (MODE == K_PULLGRAD || MODE == K_PUSHGRAD) {
#pragma unroll
          for (int q = 0; q < NGC; ++q) {
            const float sc = DOT ? 1.f : t[q];
            og[0] = fmaf(sc, gx[q], og[0]); og[1] = fmaf(sc, gy[q], og[1]); og[2] = fmaf(sc, gz[q], og[2]);
          }
        }
      }
      // ---- scatter: LN lanes take one point's taps along the last axis --------
      if (SCATTER && (MODE != K_PUSHGRAD || do_a)) {
        constexpr int LN = NT == 2 ? 2 : 4;  // 3 taps: the fourth lane idles
        float* oc = on + c0 * a.out_sC;
        const int tap = lane & (LN - 1);
#pragma unroll
        for (int p = 0; p < LN; ++p) {
          const int from = p * (32 / LN) + lane / LN;  // the lane whose point this one serves
          float wz = 0.f;
          int oz = 0;
#pragma unroll
          for (int k = 0; k < NT; ++k) {
            const float w_ = __shfl_sync(0xffffffffu, az.w[k], from);
            const int o_ = __shfl_sync(0xffffffffu, az.oo[k], from);
            if (tap == k) { wz = w_; oz = o_; }
          }
          const unsigned m = __shfl_sync(0xffffffffu, live ? (ax.mask | ay.mask << 8 | az.mask << 16) : 0u, from);
          const bool okz = (m >> (16 + tap)) & 1u;
          float tv[CB];
#pragma unroll
          for (int q = 0; q < CB; ++q) tv[q] = __shfl_sync(0xffffffffu, t[q], from);
#pragma unroll
          for (int i = 0; i < NX; ++i) {
#pragma unroll
            for (int j = 0; j < NT; ++j) {
              const float w = __shfl_sync(0xffffffffu, D == 3 ? ax.w[i] * ay.w[j] : ay.w[j], from) * wz;
              const int off = __shfl_sync(0xffffffffu, ax.oo[i] + ay.oo[j], from) + oz;
              const bool ok = okz && ((m >> i) & (m >> (8 + j)) & 1u);
              float* oq = oc + off;
#pragma unroll
              for (int q = 0; q < CB; ++q) {
                const float v = w * tv[q];
                if (ok && (CB == 1 || q < nc) && v != 0.f) atomicAdd(oq + q * a.out_sC, v);
              }
            }
          }
        }
      }
    }
    if ((MODE == K_PULLGRAD || MODE == K_PUSHGRAD) && do_grad && live) {
#pragma unroll
      for (int d = 3 - D; d < 3; ++d) gg[(d - (3 - D)) * a.gg_sD] = og[d];
    }
  }
}

template <int D, int ORD, int CB, class S, int MODE, bool DOT = false>
inline cudaError_t launch_direct(const PPArgs& p, cudaStream_t st) {
  DirArgs a;
  a.src = p.src; a.trgt = p.trgt; a.grid = static_cast<const float*>(p.grid);
  a.out = p.out; a.gg = static_cast<float*>(p.gg); a.aux = p.aux;
  a.src_sN = p.src_sN; a.trgt_sN = p.trgt_sN; a.grid_sN = p.grid_sN; a.out_sN = p.out_sN; a.gg_sN = p.gg_sN;
  a.src_sC = p.src_sC; a.out_sC = p.out_sC;
  a.trgt_sC = static_cast<int>(p.trgt_sC); a.grid_sD = static_cast<int>(p.grid_sD);
  a.out_sK = static_cast<int>(p.out_sK); a.gg_sD = static_cast<int>(p.gg_sD);
  const float tol = (p.extrapolate & 2) ? 0.55f : 0.05f;
  a.lo = -tol;
  for (int e = 0; e < 3; ++e) {  // e: axis of the kernel, d: of the tensors
    const int d = e - (3 - D);
    const bool on = d >= 0;
    a.n[e] = on ? static_cast<int>(p.src_size[d]) : 1;
    a.hi[e] = static_cast<float>(a.n[e] - 1) + tol;
    a.bound[e] = on ? p.bound[d] : 0;
    a.src_s[e] = on ? static_cast<int>(p.src_s[d]) : 0;
    a.trgt_s[e] = on ? static_cast<int>(p.trgt_s[d]) : 0;
    a.grid_s[e] = on ? static_cast<int>(p.grid_s[d]) : 0;
    a.out_s[e] = on ? static_cast<int>(p.out_s[d]) : 0;
    a.gg_s[e] = on ? static_cast<int>(p.gg_s[d]) : 0;
  }
  a.X = D == 3 ? static_cast<int>(p.trgt_size[0]) : 1;
  a.Y = static_cast<int>(p.trgt_size[D - 2]);
  a.Z = static_cast<int>(p.trgt_size[D - 1]);
  a.outer = static_cast<int>(p.N) * a.X;
  a.invX = 1.f / static_cast<float>(a.X);
  a.C = static_cast<int>(p.C); a.extrapolate = p.extrapolate; a.flags = p.flags;
  // the tile's extent along the last axis: 32, or what covers the grid with at
  // least an eighth fewer threads (256 x 256 x 2, linear, in tiles of 8 / 2
  // along z: push 13.4 / 6.7, pull backward 19.1 / 8.7 us)
  a.tzs = 5;
  int64_t best = 0;
  for (int s : {5, 4, 3, 2, 1, 0, 6, 7, 8}) {
    const int tz = 1 << s, ty = DIR_THREADS >> s;
    const int64_t cover = static_cast<int64_t>((a.Z + tz - 1) / tz * tz) * ((a.Y + ty - 1) / ty * ty);
    if (s == 5 || cover * 8 < best * 7) { best = cover; a.tzs = s; }
  }
  const int tz = 1 << a.tzs, ty = DIR_THREADS >> a.tzs;
  const int64_t gx = (a.Z + tz - 1) / tz, gy = (a.Y + ty - 1) / ty;
  // planes per thread: as many as leave eight CTAs per SM and more (2-D
  // images and small volumes: one), up to 4; grid.z holds 65535
  int64_t run = D == 3 ? gx * gy * a.outer / (148 * 8) : 1;
  run = run < 1 ? 1 : run > 4 ? 4 : run;
  if ((a.outer + run - 1) / run > 65535) run = (a.outer + 65534) / 65535;
  a.run = static_cast<int>(run);
  const dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy), static_cast<unsigned>((a.outer + run - 1) / run));
  note_kernel("pp_direct_kernel", MODE, ORD, CB);
  pp_direct_kernel<D, ORD, CB, S, MODE, DOT><<<grid, DIR_THREADS, 0, st>>>(a);
  return cudaGetLastError();
}

// Channel block: the whole channel set up to 4, else groups of 4.
template <int D, int ORD, class S, int MODE>
inline cudaError_t launch_direct_cb(const PPArgs& a, cudaStream_t st) {
  if constexpr (MODE != K_COUNT) {
    constexpr bool DOT = D == 3 && ORD == 1 && MODE == K_PUSHGRAD;
    switch (a.C >= 4 ? 4 : static_cast<int>(a.C)) {
      case 2: return launch_direct<D, ORD, 2, S, MODE, DOT>(a, st);
      case 3: return launch_direct<D, ORD, 3, S, MODE, DOT>(a, st);
      case 4:
        if (a.C > 4) return launch_direct<D, ORD, 4, S, MODE>(a, st);
        return launch_direct<D, ORD, 4, S, MODE, DOT>(a, st);
      default: break;
    }
  }
  return launch_direct<D, ORD, 1, S, MODE>(a, st);
}

}  // namespace ppk
