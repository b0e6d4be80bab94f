// Interpolating B-spline prefilter (spline_coeff / spline_coeff_nd).
//
// Arithmetic restated from the vendored prefilter nitorch/_C/_ts/coeff.py
// (Unser-Aldroubi-Eden recursive filtering): gain (coeff.py:61-65), one
// causal and one anti-causal first-order recursion per pole (coeff.py:
// 254-281), initial / final conditions per boundary (coeff.py:69-251).
//
// B200 mapping: a tile of lines per CTA staged in shared memory (element-major:
// warps of recursing threads read one sample of 32 adjacent lines per access),
// the whole tile in flight at once, 16 bytes per access.  A line is cut into
// segments, one thread each, whose recursions warm up over the end of the
// neighbour: the poles forget within a few dozen samples.  The recursions run
// out of shared memory and the global traffic is one read and one write of the
// volume per axis; two or three CTAs share an SM, one's transfers overlapping
// the others' recursions.  The recursions run in float (double for double
// storage, whose lines stay whole); the initial / final condition sums in
// double with per-pole constants computed on the host.  Lines too long for a
// shared tile fall back to the same recursion directly on global memory.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>

#include "pp_capi_internal.cuh"

namespace {

struct LineArgs {
  const void* in;
  void* out;
  int64_t nlines;
  int64_t n;          // line length
  int64_t in_st, out_st;  // element stride along the line
  int ndo;            // number of non-filtered dims
  int64_t osz[PP_MAX_DIM];     // their sizes (last fastest)
  int64_t ist[PP_MAX_DIM];     // their input strides
  int64_t ost[PP_MAX_DIM];     // their output strides
  int kind;           // 1 dct1, 2 dct2, 3 dft
  int npoles;
  double z[3];
  double gain;
  // per-pole boundary constants, the same for every line (host-computed):
  int64_t hz[3];      // dct2: series length K; dct1: truncation m; dft: min(m, n)
  double zp[3];       // dct2: z^n; dct1: z^(n-1); dft: z^hz
  double zq[3];       // dct2: z^(2n-1-k2), k2 = max(1, 2n-1-K): the mirrored tail's first weight
  int line_major;     // 1: the filtered axis is the fastest (warps stage whole lines)
  int quad_in, quad_out;  // line_major: all lines whole, aligned groups of four samples
  int nseg;           // tile kernel: segments per line, one thread each
  int warm;           // samples of a segment's warm-up: |z|^warm < 1e-13 for every pole
};

__device__ __forceinline__ void line_base(const LineArgs& a, int64_t l, int64_t& bi, int64_t& bo) {
  bi = 0; bo = 0;
  for (int d = a.ndo - 1; d >= 0; --d) {
    const int64_t q = l / a.osz[d];
    const int64_t r = l - q * a.osz[d];
    bi += r * a.ist[d];
    bo += r * a.ost[d];
    l = q;
  }
}

// Accessors to the samples of one line.
template <class C>
struct LineRef {  // in global memory, any stride
  using value_type = C;
  using index_type = int64_t;
  C* p;
  int64_t st;
  __device__ __forceinline__ C load(int64_t i) const { return p[i * st]; }
  __device__ __forceinline__ void store(int64_t i, C x) const { p[i * st] = x; }
};

template <class C>
struct TileLine {  // one column of a shared tile, runtime pitch
  using value_type = C;
  using index_type = int;
  C* p;
  int pitch;
  __device__ __forceinline__ C load(int i) const { return p[i * pitch]; }
  __device__ __forceinline__ void store(int i, C x) const { p[i * pitch] = x; }
};

template <class C, int P>
struct TileCol {  // one column of a shared tile, compile-time pitch
  using value_type = C;
  using index_type = int;
  C* p;
  __device__ __forceinline__ C load(int i) const { return p[i * P]; }
  __device__ __forceinline__ void store(int i, C x) const { p[i * P] = x; }
};

// Initial causal coefficient (coeff.py:69-170), double accumulation.  The
// samples are read as L[k] * g (g: the filter gain on the first pole's pass,
// 1 afterwards), so the gain costs no separate sweep.
template <class R, class C = typename R::value_type>
__device__ double initial(const R& L, int64_t n, const LineArgs& a, int q, C g) {
  const double z = a.z[q];
  auto x = [&](int64_t k) { return static_cast<double>(L.load(static_cast<typename R::index_type>(k)) * g); };
  const double x0 = x(0);
  double acc = x0;
  if (a.kind == 2) {  // dct2 / replicate (coeff.py:137-170)
    const double zn = a.zp[q];
    const double zlast = zn * (1.0 + 1.0 / (z + zn * zn));
    acc += zlast * x(n - 1);
    // sum_{k=1}^{n-2} (z^k + z^(2n-1-k)) L[k]; both power series decay
    // geometrically, terms below 2^-64 of the leading one are dropped.
    const int64_t K = a.hz[q];
    const int64_t k1 = n - 2 < K ? n - 2 : K;
    double zk = z;
    for (int64_t k = 1; k <= k1; ++k, zk *= z) acc += zk * x(k);
    int64_t k2 = 2 * n - 1 - K;
    if (k2 < 1) k2 = 1;
    if (k2 <= n - 2) {
      double zq = a.zq[q];
      const double iz = 1.0 / z;
      for (int64_t k = k2; k <= n - 2; ++k, zq *= iz) acc += zq * x(k);
    }
    const double s = z / (1.0 - zn * zn);
    return acc * s + x0;
  }
  if (a.kind == 1) {  // dct1 / zero (coeff.py:94-134)
    const int64_t m = a.hz[q];
    if (m < n) {
      double zk = z;
      for (int64_t k = 1; k < m; ++k, zk *= z) acc += zk * x(k);
      return acc;
    }
    const double zn = a.zp[q];
    acc += zn * x(n - 1);
    double zk = z;
    for (int64_t k = 1; k < n - 1; ++k, zk *= z) acc += (zk + zn * zn / zk) * x(k);
    return acc * (1.0 / (1.0 - zn * zn));
  }
  // dft (coeff.py:69-91)
  const int64_t m = a.hz[q];
  double zj = z;
  for (int64_t j = 1; j < m; ++j, zj *= z) acc += zj * x(n - j);
  return acc * (1.0 / (1.0 - a.zp[q]));
}

// Final anti-causal coefficient (coeff.py:173-215).
template <class R>
__device__ double final_value(const R& L, int64_t n, const LineArgs& a, int q) {
  const double z = a.z[q];
  auto x = [&](int64_t k) { return static_cast<double>(L.load(static_cast<typename R::index_type>(k))); };
  if (a.kind == 2) return x(n - 1) * (z / (z - 1.0));
  if (a.kind == 1) return (z * x(n - 2) + x(n - 1)) * (z / (z * z - 1.0));
  const int64_t m = a.hz[q];
  double acc = z * x(n - 1);
  double zj = z * z;
  for (int64_t j = 0; j < m - 1; ++j, zj *= z) acc += zj * x(j);
  return acc * (1.0 / (a.zp[q] - 1.0));
}

// One first-order recursion over `count` samples from i on, step DIR:
//   causal       (DIR = 1):   c[i] = z c[i - 1] + g x[i]
//   anti-causal  (DIR = -1):  c[i] = z (c[i + 1] - x[i])
// `prev` enters as the coefficient before the first sample and leaves as the
// last one.  The walk goes in chunks of U samples held in registers, the next
// chunk loaded before the current one is filtered, so that the memory latency
// leaves the dependency chain.  STORE = false only advances `prev`.  The
// operations of a step are written out (diff = c[i + 1] - x[i], carried along the
// anti-causal walk): contracted as the compiler likes, a warm-up and the walk
// that it stands in for would round differently and never arrive at one value.
template <int DIR, bool STORE, class R>
__device__ __forceinline__ void walk(const R& L, typename R::index_type i, typename R::index_type count,
                                     typename R::value_type z, typename R::value_type g,
                                     typename R::value_type& prev) {
  using C = typename R::value_type;
  constexpr int U = 8;
  C diff = prev, zz = 1;  // (the first difference is from `prev` itself)
  auto step = [&](C x) {
    if (DIR > 0) {
      prev = fma(z, prev, x * g);
    } else {
      diff = fma(zz, diff, -x);
      zz = z;
      prev = z * diff;
    }
  };
  if (count >= U) {
    C x[U], y[U];
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = L.load(i + DIR * u);
    for (;;) {
      const bool more = count >= 2 * U;
      if (more) {
#pragma unroll
        for (int u = 0; u < U; ++u) y[u] = L.load(i + DIR * (U + u));
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        step(x[u]);
        if (STORE) L.store(i + DIR * u, prev);
      }
      i += DIR * U;
      count -= U;
      if (!more) break;
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = y[u];
    }
  }
  for (; count > 0; --count, i += DIR) {
    step(L.load(i));
    if (STORE) L.store(i, prev);
  }
}

// Gain (coeff.py:61-65) folded into the first causal pass, then one causal
// and one anti-causal recursion per pole (coeff.py:254-281).
template <class R>
__device__ void filter_line(const R& L, typename R::index_type n, const LineArgs& a) {
  using C = typename R::value_type;
  C g = static_cast<C>(a.gain);
  for (int q = 0; q < a.npoles; ++q) {
    const C z = static_cast<C>(a.z[q]);
    C prev = static_cast<C>(initial(L, n, a, q, g));
    L.store(0, prev);
    walk<1, true>(L, 1, n - 1, z, g, prev);
    prev = static_cast<C>(final_value(L, n, a, q));
    L.store(n - 1, prev);
    walk<-1, true>(L, n - 2, n - 1, z, g, prev);
    g = C(1);
  }
}

// Two recursions are at the same value (two NaNs are).
template <class C> __device__ __forceinline__ bool differ(C x, C y) { return !(x == y) && (x == x || y == y); }

// Segments whose recursions began elsewhere than their neighbours' ended: the
// difference runs on through the segment as d z, d z^2, ... (the recursions
// are linear).  `count` samples from i on, step DIR; `has`: a neighbour ends
// right before i; from: the segment's start.  A segment is right once those
// before it are, hence nseg - 1 rounds at most.  All threads of the CTA.
template <int DIR, class R>
__device__ __noinline__ void settle(const R& L, int i, int count, bool has, typename R::value_type z,
                                    typename R::value_type from, int nseg) {
  using C = typename R::value_type;
  for (int k = 1; k < nseg; ++k) {
    const C end = has ? L.load(i - DIR) : from;
    const bool off = differ(end, from);
    if (!__syncthreads_or(off)) return;
    if (off) {
      C d = end - from;
      for (int m = 0; m < count && d != C(0); ++m) {
        d *= z;
        L.store(i + DIR * m, L.load(i + DIR * m) + d);
      }
    }
    from = end;
    __syncthreads();
  }
}

// The same with the line cut into nseg segments, one thread of the CTA each
// (thread (line, j) calls with its j; active: the thread has a line).  A
// segment's recursion starts from a warm-up over the a.warm samples before
// it, from zero.  That is where the whole line's recursion would arrive, but
// for what |z|^warm < 1e-13 leaves of the coefficients before the warm-up:
// nothing in float between samples of like size, but everything next to an
// infinity, a NaN or a sample 1e13 times as large.  So each segment then
// compares its start with its neighbour's end, and where they differ (in the
// lines of ordinary volumes only past a stretch of exact zeros) the difference
// is carried on until all agree: the result is the whole line's.  (The checks
// cost 2-4 %: 3 x 256^3 cubic 274 -> 280 us for the three axes, 3 x 192^3
// 125 -> 128 us, one kernel serving whole and cut lines.)  The warm-ups read what the neighbour is about to overwrite,
// hence the barriers; all threads of the CTA make the call.
template <class R>
__device__ void filter_segment(const R& L, int n, const LineArgs& a, int j, bool active) {
  using C = typename R::value_type;
  const bool last = j == a.nseg - 1;
  const int s = j * n / a.nseg, e = (j + 1) * n / a.nseg, w = a.warm;
  C g = static_cast<C>(a.gain);
  for (int q = 0; q < a.npoles; ++q) {
    const C z = static_cast<C>(a.z[q]);
    C prev = 0;
    if (active) {
      if (j == 0) prev = static_cast<C>(initial(L, n, a, q, g));
      else walk<1, false>(L, s - w, w, z, g, prev);
    }
    C from = prev;
    __syncthreads();
    if (active) {
      if (j == 0) L.store(0, prev);
      walk<1, true>(L, j == 0 ? 1 : s, e - (j == 0 ? 1 : s), z, g, prev);
    }
    __syncthreads();
    for (bool right = false;;) {
      const bool off = !right && active && j > 0 && differ(L.load(s - 1), from);
      prev = 0;
      if (active) {
        if (last) prev = static_cast<C>(final_value(L, n, a, q));
        else walk<-1, false>(L, e + w - 1, w, z, g, prev);
      }
      if (!__syncthreads_or(off)) break;
      settle<1>(L, s, e - s, active && j > 0, z, from, a.nseg);  // ... and the warm-up again
      right = true;
    }
    from = prev;
    if (active) {
      if (last) L.store(n - 1, prev);
      walk<-1, true>(L, last ? n - 2 : e - 1, (last ? n - 1 : e) - s, z, g, prev);
    }
    g = C(1);
    __syncthreads();
    if (__syncthreads_or(active && !last && differ(L.load(e), from)))
      settle<-1>(L, e - 1, e - s, active && !last, z, from, a.nseg);
  }
}

// Asynchronous global -> shared copies (no register round trip).
template <int B>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  if constexpr (B == 4) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(src) : "memory");
  else if constexpr (B == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(src) : "memory");
  else asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(src) : "memory");
}

// G adjacent samples of 16-bit storage <-> G floats (one 8-byte access).
template <class S, class C>
__device__ __forceinline__ void load_group(C* dst, const S* src) {
  static_assert(sizeof(S) == 2 && sizeof(C) == 4, "16-bit storage, float arithmetic");
  const uint2 r = *reinterpret_cast<const uint2*>(src);
  const S* v = reinterpret_cast<const S*>(&r);
  *reinterpret_cast<float4*>(dst) = make_float4(ppk::to_acc(v[0]), ppk::to_acc(v[1]), ppk::to_acc(v[2]),
                                                ppk::to_acc(v[3]));
}

// Vector eligibility of the group of G adjacent lines starting at tile line
// l: all present, adjacent in memory, every sample row aligned to the group
// width in bytes.
template <class S, int G>
__device__ __forceinline__ bool group_vec(const int64_t* base, const void* ptr, int64_t st, int l, int nl) {
  constexpr int bytes = G * static_cast<int>(sizeof(S));
  if (l + G > nl) return false;
  for (int k = 1; k < G; ++k)
    if (base[l + k] != base[l] + k) return false;
  const uintptr_t p = reinterpret_cast<uintptr_t>(ptr) + static_cast<uintptr_t>(base[l]) * sizeof(S);
  return (p % bytes) == 0 && ((st * static_cast<int64_t>(sizeof(S))) % bytes) == 0;
}

// Four adjacent samples of one line, moved as one access (16 bytes of float
// storage, 8 of 16-bit storage).
template <class S>
struct alignas(4 * sizeof(S)) Quad {
  S v[4];
  using C = typename ppk::Acc<S>::type;
  using Raw = typename std::conditional<sizeof(S) == 2, uint2, uint4>::type;
  __device__ __forceinline__ void load(const S* p) { *reinterpret_cast<Raw*>(this) = *reinterpret_cast<const Raw*>(p); }
  __device__ __forceinline__ void store(S* p) const { *reinterpret_cast<Raw*>(p) = *reinterpret_cast<const Raw*>(this); }
  __device__ __forceinline__ C get(int k) const { return ppk::to_acc(v[k]); }
  __device__ __forceinline__ void set(int k, C x) { v[k] = ppk::from_acc<S>(x); }
};

// Full-tile kernel: NT lines per CTA, held element-major in shared memory
// (tile[i * P + l]), staged and stored by TILE_THREADS threads; each line is
// filtered by a.nseg of them (filter_segment).  With one thread per line the
// recursions, two dependent passes of n steps, took longer than the
// transfers: at 64 lines per CTA and four segments of 64 samples (warm-ups of
// 23) per line of 256, three CTAs per SM, the three axes of 3 x 256^3 floats
// take 279 us (375 with one thread per line and 96 lines per CTA), 187 us of it
// memory traffic at the copy rate; 3 x 192^3 127 us (150).  More registers per
// thread or a fourth CTA per SM gain nothing further.
//  * filtered axis the fastest (LM): a warp instruction covers 8 groups of
//    four consecutive samples of 4 lines (128-byte segments), through
//    registers; with an odd pitch the transposed writes (bank 4 qj + qs) fall
//    in 32 distinct banks.  Lines that are not aligned for it: 8 single
//    samples of 4 lines, 8 lines apart for the same reason.  (double: single
//    samples of adjacent lines, P = NT + 4.)
//  * otherwise each thread a group of G = 16 / sizeof(C) adjacent lines on
//    every few sample rows, moved as one 16-byte copy (8-byte load for 16-bit
//    storage) when the lines are adjacent and aligned in memory, else G
//    scalar copies; P = NT + 4 (16-byte rows).
// Strided float / double lines and single samples stage with asynchronous
// copies, the whole tile in flight at once; 16-bit storage converts through
// registers.
constexpr int TILE_THREADS = 256;

template <class C> constexpr int tile_pitch(int nt, bool line_major) { return line_major && sizeof(C) == 4 ? nt + 1 : nt + 4; }

template <class S, int NT, bool LM, bool SEG>
__global__ void __launch_bounds__(TILE_THREADS, sizeof(S) == 8 ? 2 : 3) coeff_tile_kernel(LineArgs a) {
  using C = typename ppk::Acc<S>::type;
  constexpr int G = 16 / static_cast<int>(sizeof(C));
  constexpr int P = tile_pitch<C>(NT, LM);
  constexpr int NW = TILE_THREADS / 32;
  constexpr int GPR = NT / G;                 // strided: groups per sample row
  constexpr int RS = TILE_THREADS / GPR;      // strided: rows per step (threads past RS * GPR idle)
  constexpr bool kAsync = sizeof(S) == sizeof(C);
  static_assert(NT % 32 == 0 && NT % G == 0 && RS >= 1 && NT <= TILE_THREADS, "tile shape");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* sm = reinterpret_cast<C*>(smem_raw);
  const int64_t l0 = static_cast<int64_t>(blockIdx.x) * NT;
  const int nl = static_cast<int>(a.nlines - l0 < NT ? a.nlines - l0 : NT);
  const S* in = static_cast<const S*>(a.in);
  S* out = static_cast<S*>(a.out);
  __shared__ int64_t bin[NT], bout[NT];
  for (int l = threadIdx.x; l < nl; l += TILE_THREADS) line_base(a, l0 + l, bin[l], bout[l]);
  __syncthreads();
  const int n32 = static_cast<int>(a.n);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int qs = lane >> 3, qj = lane & 7;  // line_major: line in the quad, first sample
  // line_major, single samples: the lane's line in step qd
  auto single_line = [&](int qd) { return P % 2 ? (qd >> 3) * 32 + (qd & 7) + 8 * qs : qd * 4 + qs; };
  const bool vin = sizeof(C) == 4 && a.quad_in, vout = sizeof(C) == 4 && a.quad_out;
  const int gl = threadIdx.x < RS * GPR ? (threadIdx.x % GPR) * G : NT;  // strided: group (NT: idle)
  const int r0 = threadIdx.x / GPR;                                       // strided: first row
  if constexpr (LM) {
    if (vin) {
      // 8 groups of 4 samples of 4 lines per warp instruction, 8 of them in flight
      for (int qd = warp; qd * 4 < nl; qd += NW) {
        const int l = qd * 4 + qs;
        if (l >= nl) continue;
        const S* src = in + bin[l];
        for (int i0 = 4 * qj; i0 < n32; i0 += 256) {
          Quad<S> v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (i0 + 32 * u < n32) v[u].load(src + i0 + 32 * u);
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            C* dst = sm + (i0 + 32 * u) * P + l;
            if (i0 + 32 * u < n32) {
#pragma unroll
              for (int k = 0; k < 4; ++k) dst[k * P] = v[u].get(k);
            }
          }
        }
      }
    } else {
      for (int qd = warp; qd < NT / 4; qd += NW) {
        const int l = single_line(qd);
        if (l >= nl) continue;
        const S* src = in + bin[l];
        C* dst = sm + l;
        if constexpr (kAsync) {
          for (int i = qj; i < n32; i += 8) cp_async<sizeof(C)>(dst + i * P, src + i * a.in_st);
        } else {
          for (int i = qj; i < n32; i += 8) dst[i * P] = ppk::to_acc(src[i * a.in_st]);
        }
      }
    }
  } else if (gl < nl) {
    const bool vec = group_vec<S, G>(bin, in, a.in_st, gl, nl);
    const S* src = in + bin[gl];
    for (int i = r0; i < n32; i += RS) {
      C* dst = sm + i * P + gl;
      const int64_t off = i * a.in_st;
      if (vec) {
        if constexpr (kAsync) cp_async<16>(dst, src + off);
        else load_group(dst, src + off);
      } else {
        for (int k = 0; k < G && gl + k < nl; ++k) {
          if constexpr (kAsync) cp_async<sizeof(C)>(dst + k, in + bin[gl + k] + off);
          else dst[k] = ppk::to_acc(in[bin[gl + k] + off]);
        }
      }
    }
  }
  if constexpr (kAsync) asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  const int col = threadIdx.x % NT, seg = threadIdx.x / NT;
  const bool active = seg < (SEG ? a.nseg : 1) && col < nl;
  if constexpr (SEG) {
    filter_segment(TileCol<C, P>{sm + col}, n32, a, seg, active);
  } else {
    if (active) filter_line(TileCol<C, P>{sm + col}, n32, a);
    __syncthreads();
  }
  if constexpr (LM) {
    if (vout) {
      for (int qd = warp; qd * 4 < nl; qd += NW) {
        const int l = qd * 4 + qs;
        if (l >= nl) continue;
        S* dst = out + bout[l];
        for (int i = 4 * qj; i < n32; i += 32) {
          Quad<S> v;
#pragma unroll
          for (int k = 0; k < 4; ++k) v.set(k, sm[(i + k) * P + l]);
          v.store(dst + i);
        }
      }
    } else {
      for (int qd = warp; qd < NT / 4; qd += NW) {
        const int l = single_line(qd);
        if (l >= nl) continue;
        S* dst = out + bout[l];
        const C* src = sm + l;
        for (int i = qj; i < n32; i += 8) dst[i * a.out_st] = ppk::from_acc<S>(src[i * P]);
      }
    }
  } else if (gl < nl) {
    const bool vec = group_vec<S, G>(bout, out, a.out_st, gl, nl);
    S* dst = out + bout[gl];
    for (int i = r0; i < n32; i += RS) {
      const C* src = sm + i * P + gl;
      const int64_t off = i * a.out_st;
      if (vec) {
        if constexpr (kAsync) {
          *reinterpret_cast<uint4*>(dst + off) = *reinterpret_cast<const uint4*>(src);
        } else {
          const float4 f = *reinterpret_cast<const float4*>(src);
          S v[4] = {ppk::from_acc<S>(f.x), ppk::from_acc<S>(f.y), ppk::from_acc<S>(f.z), ppk::from_acc<S>(f.w)};
          *reinterpret_cast<uint2*>(dst + off) = *reinterpret_cast<const uint2*>(v);
        }
      } else {
        for (int k = 0; k < G && gl + k < nl; ++k) out[bout[gl + k] + off] = ppk::from_acc<S>(src[k]);
      }
    }
  }
}

// Long-line kernel: LL threads, up to LL lines per CTA, one per thread, with
// a runtime pitch (fewer lines for longer lines, up to 200 KB of shared
// memory): odd when warps stage whole lines (conflict-free column writes),
// else a multiple of G = 16 / sizeof(C) for the group copies.
constexpr int LL = 64;

template <class S>
__global__ void __launch_bounds__(LL) coeff_smem_kernel(LineArgs a, int pitch, int lines) {
  using C = typename ppk::Acc<S>::type;
  constexpr int G = 16 / static_cast<int>(sizeof(C));
  constexpr int GPR = LL / G;  // groups per sample row
  constexpr int NW = LL / 32;
  constexpr bool kAsync = sizeof(S) == sizeof(C);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* sm = reinterpret_cast<C*>(smem_raw);
  const int64_t l0 = static_cast<int64_t>(blockIdx.x) * lines;
  const int nl = static_cast<int>(a.nlines - l0 < lines ? a.nlines - l0 : lines);
  const S* in = static_cast<const S*>(a.in);
  S* out = static_cast<S*>(a.out);
  __shared__ int64_t bin[LL], bout[LL];
  for (int l = threadIdx.x; l < nl; l += LL) line_base(a, l0 + l, bin[l], bout[l]);
  __syncthreads();
  const int n32 = static_cast<int>(a.n);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool gvec_ok = (pitch % G) == 0;
  const int gl = (threadIdx.x % GPR) * G, r0 = threadIdx.x / GPR;  // strided: group line, first row
  if (a.line_major) {
    for (int l = warp; l < nl; l += NW) {
      const S* src = in + bin[l];
      C* dst = sm + l;
      for (int i = lane; i < n32; i += 32) {
        if constexpr (kAsync) cp_async<sizeof(C)>(dst + i * pitch, src + i * a.in_st);
        else dst[i * pitch] = ppk::to_acc(src[i * a.in_st]);
      }
    }
  } else if (gl < nl) {
    const bool vec = gvec_ok && group_vec<S, G>(bin, in, a.in_st, gl, nl);
    const S* src = in + bin[gl];
    for (int i = r0; i < n32; i += G) {
      C* dst = sm + i * pitch + gl;
      const int64_t off = i * a.in_st;
      if (vec) {
        if constexpr (kAsync) cp_async<16>(dst, src + off);
        else load_group(dst, src + off);
      } else {
        for (int k = 0; k < G && gl + k < nl; ++k) {
          if constexpr (kAsync) cp_async<sizeof(C)>(dst + k, in + bin[gl + k] + off);
          else dst[k] = ppk::to_acc(in[bin[gl + k] + off]);
        }
      }
    }
  }
  if constexpr (kAsync) asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  if (threadIdx.x < nl) filter_line(TileLine<C>{sm + threadIdx.x, pitch}, n32, a);
  __syncthreads();
  if (a.line_major) {
    for (int l = warp; l < nl; l += NW) {
      S* dst = out + bout[l];
      const C* src = sm + l;
      for (int i = lane; i < n32; i += 32) dst[i * a.out_st] = ppk::from_acc<S>(src[i * pitch]);
    }
  } else if (gl < nl) {
    const bool vec = gvec_ok && group_vec<S, G>(bout, out, a.out_st, gl, nl);
    S* dst = out + bout[gl];
    for (int i = r0; i < n32; i += G) {
      const C* src = sm + i * pitch + gl;
      const int64_t off = i * a.out_st;
      if (vec) {
        if constexpr (kAsync) {
          *reinterpret_cast<uint4*>(dst + off) = *reinterpret_cast<const uint4*>(src);
        } else {
          const float4 f = *reinterpret_cast<const float4*>(src);
          S v[4] = {ppk::from_acc<S>(f.x), ppk::from_acc<S>(f.y), ppk::from_acc<S>(f.z), ppk::from_acc<S>(f.w)};
          *reinterpret_cast<uint2*>(dst + off) = *reinterpret_cast<const uint2*>(v);
        }
      } else {
        for (int k = 0; k < G && gl + k < nl; ++k) out[bout[gl + k] + off] = ppk::from_acc<S>(src[k]);
      }
    }
  }
}

// Global-memory fallback for lines too long for shared memory (more than
// ~50k elements): copy, then filter in place in the output.  float / double
// storage only.
template <class S>
__global__ void coeff_global_kernel(LineArgs a) {
  using C = typename ppk::Acc<S>::type;
  const int64_t l = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (l >= a.nlines) return;
  int64_t bi, bo;
  line_base(a, l, bi, bo);
  const S* in = static_cast<const S*>(a.in);
  S* out = static_cast<S*>(a.out);
  if (in != out || bi != bo || a.in_st != a.out_st)
    for (int64_t i = 0; i < a.n; ++i) out[bo + i * a.out_st] = in[bi + i * a.in_st];
  LineRef<S> L{out + bo, a.out_st};
  filter_line(L, a.n, a);
}

template <class S>
__global__ void copy_strided(const S* in, S* out, ppc::Strided si, ppc::Strided so) {
  int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (; i < si.numel; i += step) out[ppc::strided_offset(so, i)] = in[ppc::strided_offset(si, i)];
}

int poles(int order, double* z) {
  switch (order) {
    case 0: case 1: return 0;
    case 2: z[0] = sqrt(8.0) - 3.0; return 1;
    case 3: z[0] = sqrt(3.0) - 2.0; return 1;
    case 4:
      z[0] = sqrt(664.0 - sqrt(438976.0)) + sqrt(304.0) - 19.0;
      z[1] = sqrt(664.0 + sqrt(438976.0)) - sqrt(304.0) - 19.0;
      return 2;
    case 5:
      z[0] = sqrt(67.5 - sqrt(4436.25)) + sqrt(26.25) - 6.5;
      z[1] = sqrt(67.5 + sqrt(4436.25)) - sqrt(26.25) - 6.5;
      return 2;
    case 6:
      z[0] = -0.488294589303044755130118038883789062112279161239377608394;
      z[1] = -0.081679271076237512597937765737059080653379610398148178525368;
      z[2] = -0.00141415180832581775108724397655859252786416905534669851652709;
      return 3;
    case 7:
      z[0] = -0.5352804307964381655424037816816460718339231523426924148812;
      z[1] = -0.122554615192326690515272264359357343605486549427295558490763;
      z[2] = -0.0091486948096082769285930216516478534156925639545994482648003;
      return 3;
  }
  return -1;
}

template <class S>
int copy_tensor(const pp_tensor* in, const pp_tensor* out, cudaStream_t st) {
  const int64_t n = ppc::numel(in);
  if (n == 0 || in->data == out->data) return PP_OK;
  ppc::Strided si = ppc::make_strided(in), so = ppc::make_strided(out);
  copy_strided<S><<<ppc::grid_blocks(n), 256, 0, st>>>(static_cast<const S*>(in->data), static_cast<S*>(out->data), si, so);
  ppc::count_launch();
  return ppc::cuda_check(cudaGetLastError(), "copy");
}

int copy_any(const pp_tensor* in, const pp_tensor* out, cudaStream_t st) {
  switch (in->dtype) {
    case PP_FLOAT32: return copy_tensor<float>(in, out, st);
    case PP_FLOAT64: return copy_tensor<double>(in, out, st);
    case PP_BFLOAT16: return copy_tensor<__nv_bfloat16>(in, out, st);
    default: return copy_tensor<__half>(in, out, st);
  }
}

// Opts kernel K into `most` bytes of dynamic shared memory, the most that any
// of its launches takes, once per device (bit d of `done`).  Set to each
// launch's own size, the limit could drop below another thread's launch
// between that thread's setting and its launch.
template <auto K>
int allow_smem(size_t most) {
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  if (int rc = ppc::cuda_check(cudaGetDevice(&dev), "prefilter device")) return rc;
  const unsigned long long bit = 1ull << (dev & 63);
  if (done.load() & bit) return PP_OK;
  if (int rc = ppc::cuda_check(cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most)),
                               "prefilter smem attribute"))
    return rc;
  done.fetch_or(bit);
  return PP_OK;
}

constexpr size_t TILE_SMEM = 113 * 1024, LONG_SMEM = 200 * 1024;  // two tiles per SM, one set of long lines

template <class S, int NT, bool LM, bool SEG>
int launch_tile(const LineArgs& a, cudaStream_t st) {
  using C = typename ppk::Acc<S>::type;
  const size_t smem = static_cast<size_t>(a.n) * tile_pitch<C>(NT, LM) * sizeof(C);
  if (int rc = allow_smem<coeff_tile_kernel<S, NT, LM, SEG>>(TILE_SMEM)) return rc;
  const int64_t blocks = (a.nlines + NT - 1) / NT;
  coeff_tile_kernel<S, NT, LM, SEG><<<static_cast<unsigned>(blocks), TILE_THREADS, smem, st>>>(a);
  ppc::count_launch();
  return ppc::cuda_check(cudaGetLastError(), "prefilter launch");
}

template <class S, int NT, bool SEG>
int launch_tile(const LineArgs& a, cudaStream_t st) {
  return a.line_major ? launch_tile<S, NT, true, SEG>(a, st) : launch_tile<S, NT, false, SEG>(a, st);
}

template <class S>
int launch_tiles(const LineArgs& a, int NT, cudaStream_t st) {
  if constexpr (sizeof(S) < 8) {
    if (a.nseg > 1) {
      if (NT == 128) return launch_tile<S, 128, true>(a, st);
      if (NT == 64) return launch_tile<S, 64, true>(a, st);
      return launch_tile<S, 32, true>(a, st);
    }
  }
  if (NT == 128) return launch_tile<S, 128, false>(a, st);
  if (NT == 96) return launch_tile<S, 96, false>(a, st);
  if (NT == 64) return launch_tile<S, 64, false>(a, st);
  return launch_tile<S, 32, false>(a, st);
}

// Whether every line starts on, and consists of, aligned groups of four.  A
// thread keeps the groups of one line in flight: lines of fewer than 96
// samples leave too few (4 x 400 x 400 lines of 40: 137 us so, 101 us by
// asynchronous copies of single samples).
bool quads(const LineArgs& a, const void* p, int64_t st, const int64_t* os, size_t elem) {
  if (st != 1 || a.n < 96 || a.n % 4 != 0 || reinterpret_cast<uintptr_t>(p) % (4 * elem) != 0) return false;
  for (int d = 0; d < a.ndo; ++d)
    if (a.osz[d] > 1 && os[d] % 4 != 0) return false;
  return true;
}

template <class S>
int run_axis(LineArgs& a, cudaStream_t st) {
  using C = typename ppk::Acc<S>::type;
  constexpr int G = 16 / static_cast<int>(sizeof(C));
  if (a.nlines == 0) return PP_OK;
  // Full tiles: the widest NT (multiple of 32) whose tile leaves room for two
  // CTAs per SM, at most 64 lines where a line has four segments or more (all
  // threads recurse; at 96 lines there is room for two segments: 134 against
  // 92 us on 3 x 256^3, at 32 for eight: 117 us) and 128 where it has fewer
  // (4 x 400 x 400 lines of 40: 137 us at 64 lines, 94 at 128).
  {
    const int64_t fit = static_cast<int64_t>(TILE_SMEM / (static_cast<size_t>(a.n) * sizeof(C))) - 4;
    // segments, each longer than a warm-up; with fewer than four their warm-ups
    // and checks cost what they save (cubic 72^3: 20.3 us in two, 19 whole)
    int64_t most = sizeof(C) == 4 ? a.n / (a.warm + 1) : 1;
    if (most < 4) most = 1;
    // (128 lines in two segments where all are then one wave of two CTAs per SM,
    // and 64-line tiles a wave of three and a remainder: 192^3, 49 -> 42 us)
    const bool one_wave = fit >= 128 && a.nlines > 64 * 3 * 148 && a.nlines <= 128 * 2 * 148;
    const int most_nt = most > 1 && !one_wave ? 64 : 128;
    const int NT = static_cast<int>(std::min<int64_t>(most_nt, fit / 32 * 32));
    if (NT > 0) {
      a.nseg = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(TILE_THREADS / NT, most)));
      a.quad_in = quads(a, a.in, a.in_st, a.ist, sizeof(S));
      a.quad_out = quads(a, a.out, a.out_st, a.ost, sizeof(S));
      return launch_tiles<S>(a, NT, st);
    }
  }
  // longer lines: fewer per CTA, one per thread
  const int64_t fit = static_cast<int64_t>(LONG_SMEM / (static_cast<size_t>(a.n) * sizeof(C)));
  int lines = static_cast<int>(fit < LL ? fit : LL), pitch = 0;
  if (a.line_major) {
    pitch = lines | 1;
    if (static_cast<int64_t>(pitch) > fit) pitch = --lines;  // lines was even: drop one
  } else {
    if (lines >= G) lines -= lines % G;
    pitch = lines;
  }
  if (lines >= 1) {
    const size_t smem = static_cast<size_t>(a.n) * pitch * sizeof(C);
    if (int rc = allow_smem<coeff_smem_kernel<S>>(LONG_SMEM)) return rc;
    const int64_t blocks = (a.nlines + lines - 1) / lines;
    coeff_smem_kernel<S><<<static_cast<unsigned>(blocks), LL, smem, st>>>(a, pitch, lines);
    ppc::count_launch();
  } else {
    if constexpr (sizeof(S) < 4) {
      return ppc::fail(PP_ERR_UNSUPPORTED, "(): 16-bit spline_coeff lines longer than %lld elements",
                       (long long)(LONG_SMEM / sizeof(C)));
    } else {
      const int64_t blocks = (a.nlines + 127) / 128;
      coeff_global_kernel<S><<<static_cast<unsigned>(blocks), 128, 0, st>>>(a);
      ppc::count_launch();
    }
  }
  return ppc::cuda_check(cudaGetLastError(), "prefilter launch");
}

int coeff_axis(const pp_tensor* in, const pp_tensor* out, int bound, int order, int axis,
               cudaStream_t st) {
  LineArgs a;
  a.in = in->data;
  a.out = out->data;
  a.n = in->sizes[axis];
  a.in_st = in->strides[axis];
  a.out_st = out->strides[axis];
  a.npoles = poles(order, a.z);
  if (a.npoles < 0) return ppc::fail(PP_ERR_ARG, "(): unsupported interpolation order %d", order);
  if (a.npoles == 0) return copy_any(in, out, st);
  if (bound == 0 || bound == 2) a.kind = 1;
  else if (bound == 1 || bound == 3) a.kind = 2;
  else if (bound == 6) a.kind = 3;
  else return ppc::fail(PP_ERR_UNSUPPORTED, "(): spline_coeff is not implemented for bound code %d "
                        "(only zero, replicate, dct1, dct2 and dft)", bound);
  if (a.n == 1) return copy_any(in, out, st);
  a.gain = 1.0;
  a.nseg = 1;
  a.warm = 0;
  for (int q = 0; q < a.npoles; ++q) {
    const double z = a.z[q];
    a.gain *= (1.0 - z) * (1.0 - 1.0 / z);
    // truncation of the causal initial sums (coeff.py:75, :100): |z|^m < 1e-13
    const int64_t m = static_cast<int64_t>(std::ceil(-30.0 / std::log(std::fabs(z))));
    a.warm = std::max(a.warm, static_cast<int>(m));
    if (a.kind == 2) {
      const int64_t K = static_cast<int64_t>(std::ceil(-44.4 / std::log(std::fabs(z)))) + 1;
      const int64_t k2 = std::max<int64_t>(1, 2 * a.n - 1 - K);
      a.hz[q] = K;
      a.zp[q] = std::pow(z, static_cast<double>(a.n));
      a.zq[q] = std::pow(z, static_cast<double>(2 * a.n - 1 - k2));
    } else if (a.kind == 1) {
      a.hz[q] = m;
      a.zp[q] = std::pow(z, static_cast<double>(a.n - 1));
      a.zq[q] = 0.0;
    } else {
      a.hz[q] = std::min<int64_t>(m, a.n);
      a.zp[q] = std::pow(z, static_cast<double>(a.hz[q]));
      a.zq[q] = 0.0;
    }
  }
  a.ndo = 0;
  a.nlines = 1;
  int64_t min_other = INT64_MAX;
  for (int d = 0; d < in->ndim; ++d) {
    if (d == axis) continue;
    a.osz[a.ndo] = in->sizes[d];
    a.ist[a.ndo] = in->strides[d];
    a.ost[a.ndo] = out->strides[d];
    if (in->sizes[d] > 1 && in->strides[d] < min_other) min_other = in->strides[d];
    a.nlines *= in->sizes[d];
    ++a.ndo;
  }
  a.line_major = (a.in_st <= min_other) ? 1 : 0;
  switch (in->dtype) {
    case PP_FLOAT32: return run_axis<float>(a, st);
    case PP_FLOAT64: return run_axis<double>(a, st);
    case PP_BFLOAT16: return run_axis<__nv_bfloat16>(a, st);
    default: return run_axis<__half>(a, st);
  }
}

int check_coeff_io(const pp_tensor* in, const pp_tensor* out) {
  int rc = ppc::check_tensor(in, "input");
  if (rc) return rc;
  if ((rc = ppc::check_tensor(out, "output"))) return rc;
  if (in->ndim != out->ndim) return ppc::fail(PP_ERR_ARG, "(): output must have the input's shape");
  for (int d = 0; d < in->ndim; ++d)
    if (in->sizes[d] != out->sizes[d]) return ppc::fail(PP_ERR_ARG, "(): output must have the input's shape");
  if (in->dtype != out->dtype) return ppc::fail(PP_ERR_DTYPE, "(): output dtype must match input");
  return PP_OK;
}

}  // namespace

extern "C" {

int pp_spline_coeff(const pp_tensor* input, const pp_tensor* out, int32_t bound, int32_t order,
                    int32_t axis, void* stream) {
  int rc = check_coeff_io(input, out);
  if (rc) return rc;
  if (input->ndim == 0) return copy_any(input, out, static_cast<cudaStream_t>(stream));
  if (axis < 0) axis += input->ndim;
  if (axis < 0 || axis >= input->ndim) return ppc::fail(PP_ERR_ARG, "(): axis out of range");
  if (order < 0 || order > 7) return ppc::fail(PP_ERR_ARG, "(): unsupported interpolation order %d", order);
  if (ppc::numel(input) == 0) return PP_OK;
  return coeff_axis(input, out, bound, order, axis, static_cast<cudaStream_t>(stream));
}

int pp_spline_coeff_nd(const pp_tensor* input, const pp_tensor* out, int32_t nbound, const int32_t* bound,
                       int32_t norder, const int32_t* order, int32_t dim, void* stream) {
  int rc = check_coeff_io(input, out);
  if (rc) return rc;
  if (dim < 0 || dim > input->ndim) return ppc::fail(PP_ERR_ARG, "(): dim out of range");
  if (nbound < 1 || norder < 1 || !bound || !order) return ppc::fail(PP_ERR_ARG, "(): empty bound / order list");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (ppc::numel(input) == 0) return PP_OK;
  const pp_tensor* src = input;
  bool wrote = false;
  for (int d = 0; d < dim; ++d) {
    const int b = bound[d < nbound ? d : nbound - 1];
    const int o = order[d < norder ? d : norder - 1];
    if (o < 0 || o > 7) return ppc::fail(PP_ERR_ARG, "(): unsupported interpolation order %d", o);
    const int axis = input->ndim - dim + d;
    if (o <= 1) continue;  // identity along this axis
    if ((rc = coeff_axis(src, out, b, o, axis, st))) return rc;
    src = out;
    wrote = true;
  }
  if (!wrote) return copy_any(input, out, st);
  return PP_OK;
}

}  // extern "C"
