// CUDA kernels of the GB300 NCC find path (sm_103a).
//
// Numerics.  Every pyramid value is an integer sum of 4^k input pixels, held
// exactly in float.  Window moments (sum S, sum S^2) come from row prefix sums:
// int64, or uint32 modulo 2^32 where the host found that a run's sum S^2 stays
// below 2^32 (its longest run times the level's largest value squared), so that
// a difference of two entries is exact; windows whose sums and variance numerator
// are bounded as well are summed in 32 bits (TrackArgs::narrow).  Either way the
// variance numerator n*sum(S^2) - (sum S)^2 is exact and the "variance <= 0 ->
// no score" rule of the reference is decided exactly.
// The template dot product sum(w * (S - S_first)) runs in FP32 on the CUDA
// cores.  The full-resolution score and the Gauss-Newton moments accumulate
// in FP32 per thread and combine as FP32 (hi, lo) two-sum pairs; the 3x3
// normal equations are solved in FP64, an entry per lane.
//
// sm_103 issues FP64 at a small fraction of the FP32 rate, so FP64 appears
// only where the reference's decisions need it: pose lattice arithmetic (or
// an FP32 form the host proved exact), the normal-equation solve, and the
// rectangle overlap of the MaxOverlap rule.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>

#include "ncc_kernels.h"

namespace mvg {
namespace {

__device__ __forceinline__ int off_row(int32_t o) { return o >> 16; }
__device__ __forceinline__ int off_col(int32_t o) { return int(int16_t(o & 0xffff)); }

__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }

// pose coordinate of integer position r on a level: crop + step*(r + o) + off
// (src/ncc_matching/matcher.cpp:558,592,687)
__device__ __forceinline__ double lattice_pose(double crop, double step, int r, double o, double off) {
  return dadd(dadd(crop, dmul(step, dadd(double(r), o))), off);
}
__device__ __forceinline__ float lattice_pose32(float crop, float step, int r, float o, float off) {
  return __fadd_rn(__fadd_rn(crop, __fmul_rn(step, __fadd_rn(float(r), o))), off);
}

// ------------------------------------------------------------ search domain
// domain_contains (src/ncc_matching/matcher.cpp:249-251): the pixel nearest
// to the pose lies in the domain.
__device__ __forceinline__ bool domain_contains(const DomainView& d, double row, double col) {
  const double rr = floor(row + .5), cc = floor(col + .5);
  if (!(rr >= 0 && cc >= 0 && rr < d.h && cc < d.w)) return false;
  return !d.mask || d.mask[size_t(rr) * d.w + size_t(cc)] != 0;
}

// may_contain (matcher.cpp:507-534) for a reduced domain, beyond the bounding
// box that the position ranges encode: spacing 1 tests the nearest pixel; a
// coarser spacing s accepts a pose with a domain pixel within 2s rows and
// columns (a run [b, e] of row y meets |y - row| <= 2s, b <= col + 2s,
// e >= col - 2s exactly when the mask has a pixel in the integer rectangle
// [ceil(row - 2s), floor(row + 2s)] x [ceil(col - 2s), floor(col + 2s)]),
// counted from the mask's 2-D prefix counts.  The full image (mask null)
// passes.
__device__ bool may_contain(const DomainView& d, double row, double col, double spacing) {
  if (!d.mask) return true;
  if (spacing == 1) return domain_contains(d, row, col);
  const double m = 2 * spacing;
  if (row < d.rmin - m || row > d.rmax + m || col < d.cmin - m || col > d.cmax + m) return false;
  if (!d.sparse) return true;
  const int r0 = max(0, int(ceil(dsub(row, m)))), r1 = min(d.h - 1, int(floor(dadd(row, m))));
  const int c0 = max(0, int(ceil(dsub(col, m)))), c1 = min(d.w - 1, int(floor(dadd(col, m))));
  if (r0 > r1 || c0 > c1) return false;
  const size_t pitch = size_t(d.w) + 1;
  const int32_t n = d.count[size_t(r1 + 1) * pitch + c1 + 1] - d.count[size_t(r0) * pitch + c1 + 1] -
                    d.count[size_t(r1 + 1) * pitch + c0] + d.count[size_t(r0) * pitch + c0];
  return n > 0;
}

// ------------------------------------------------------- FP32 pair arithmetic
struct __align__(8) F2 {  // stored as one 8-byte word
  float hi, lo;
};
__device__ __forceinline__ F2 f2(float x) { return F2{x, 0.f}; }
__device__ __forceinline__ F2 f2_add(F2 x, F2 y) {
  const float s = __fadd_rn(x.hi, y.hi);
  const float bb = __fsub_rn(s, x.hi);
  const float e = __fadd_rn(__fadd_rn(__fsub_rn(x.hi, __fsub_rn(s, bb)), __fsub_rn(y.hi, bb)), __fadd_rn(x.lo, y.lo));
  const float h = __fadd_rn(s, e);
  return F2{h, __fsub_rn(e, __fsub_rn(h, s))};
}
__device__ __forceinline__ F2 f2_neg(F2 x) { return F2{-x.hi, -x.lo}; }
__device__ __forceinline__ F2 f2_sub(F2 x, F2 y) { return f2_add(x, f2_neg(y)); }
__device__ __forceinline__ F2 f2_mul(F2 x, F2 y) {
  const float p = __fmul_rn(x.hi, y.hi);
  float e = __fmaf_rn(x.hi, y.hi, -p);
  e = __fmaf_rn(x.hi, y.lo, e);
  e = __fmaf_rn(x.lo, y.hi, e);
  const float h = __fadd_rn(p, e);
  return F2{h, __fsub_rn(e, __fsub_rn(h, p))};
}
__device__ __forceinline__ F2 f2_div(F2 x, F2 y) {
  const float q1 = __fdiv_rn(x.hi, y.hi);
  const F2 r = f2_sub(x, f2_mul(f2(q1), y));
  const float q2 = __fdiv_rn(r.hi, y.hi);
  const float h = __fadd_rn(q1, q2);
  return F2{h, __fsub_rn(q2, __fsub_rn(h, q1))};
}
__device__ __forceinline__ float f2_val(F2 x) { return x.hi + x.lo; }
__device__ __forceinline__ double f2_dbl(F2 x) { return double(x.hi) + double(x.lo); }

// Score of one window from the FP32 template dot and exact integer moments.
// D = sum w (S - S0) relates to the reference's sum w q by a 4^k factor that
// cancels against the variance, giving score = D / sqrt(V / n) with
// V = n sum S^2 - (sum S)^2 (src/ncc_matching/matcher.cpp:97-105).
__device__ __forceinline__ float window_score(float dot, long long s1, long long s2, int n, int absolute) {
  const __int128 v = (__int128)n * s2 - (__int128)s1 * s1;
  if (v <= 0) return -INFINITY;
  const long long hi = (long long)(v >> 62);
  const float vf = hi ? __ll2float_rn(hi) * 4.611686018427387904e18f +
                            __ull2float_rn((unsigned long long)(v & ((((__int128)1) << 62) - 1)))
                      : __ll2float_rn((long long)v);
  float s = dot * rsqrtf(vf / float(n));
  s = fminf(1.f, fmaxf(-1.f, s));
  return absolute ? fabsf(s) : s;
}

// The same where the variance numerator stays below 2^62.
__device__ __forceinline__ float window_score_narrow(float dot, uint32_t s1, unsigned long long s2, int n, int absolute) {
  const long long v = (long long)(s2 * (unsigned long long)n) - (long long)((unsigned long long)s1 * s1);
  if (v <= 0) return -INFINITY;
  float s = dot * rsqrtf(__ll2float_rn(v) / float(n));
  s = fminf(1.f, fmaxf(-1.f, s));
  return absolute ? fabsf(s) : s;
}

// Window moments {sum S, sum S^2} of a patch at (r, c) from the level's row
// prefixes: runs first, first + step, ... (step > 1 splits the runs over
// threads; the caller adds the parts).
__device__ __forceinline__ void window_moments(const LevelImage& lev, int pitch, int r, int c,
                                               const int4* __restrict__ runs, int nruns, long long& s1, long long& s2,
                                               int first = 0, int step = 1) {
  s1 = 0;
  s2 = 0;
  if (lev.prefix32) {
    // four runs per step, all eight prefix loads issued before the sums
    const uint2* __restrict__ P = lev.prefix32;
    int j = first;
    for (; j + 3 * step < nruns; j += 4 * step) {
      int4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = __ldg(runs + j + u * step);
      uint2 hi[4], lo[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const size_t base = size_t(r + q[u].x) * pitch + c;
        hi[u] = P[base + q[u].z + 1];
        lo[u] = P[base + q[u].y];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        s1 += (long long)(hi[u].x - lo[u].x);
        s2 += (long long)(hi[u].y - lo[u].y);
      }
    }
    for (; j < nruns; j += step) {
      const int4 q = __ldg(runs + j);
      const size_t base = size_t(r + q.x) * pitch + c;
      const uint2 hi = P[base + q.z + 1];
      const uint2 lo = P[base + q.y];
      s1 += (long long)(hi.x - lo.x);
      s2 += (long long)(hi.y - lo.y);
    }
    return;
  }
  const longlong2* __restrict__ P = lev.prefix;
  int j = first;
  for (; j + step < nruns; j += 2 * step) {
    const int4 q0 = __ldg(runs + j), q1 = __ldg(runs + j + step);
    const size_t b0 = size_t(r + q0.x) * pitch + c, b1 = size_t(r + q1.x) * pitch + c;
    const longlong2 h0 = P[b0 + q0.z + 1], l0 = P[b0 + q0.y];
    const longlong2 h1 = P[b1 + q1.z + 1], l1 = P[b1 + q1.y];
    s1 += (h0.x - l0.x) + (h1.x - l1.x);
    s2 += (h0.y - l0.y) + (h1.y - l1.y);
  }
  for (; j < nruns; j += step) {
    const int4 q = __ldg(runs + j);
    const size_t base = size_t(r + q.x) * pitch + c;
    const longlong2 hi = P[base + q.z + 1];
    const longlong2 lo = P[base + q.y];
    s1 += hi.x - lo.x;
    s2 += hi.y - lo.y;
  }
}

// (score, order) with the first strict maximum in iteration order winning
__device__ __forceinline__ bool better(float s, int o, float bs, int bo) {
  return s > bs || (s == bs && o < bo);
}

// ------------------------------------------------------------------ pyramid
// Word (8 bits) or word pair (16 bits) of a pixel's quad.
template <int Bits> __device__ __forceinline__ uint32_t quad_at(int x, int y, int tiles) {
  constexpr int W = Bits == 8 ? 8 : 4;  // tile width; tiles are 4 high
  // ((y / 4) tiles + x / W) 4 W + (y mod 4) W + x mod W
  return uint32_t((y & ~3) * ((tiles - 1) * W) + y * W + (x & ~(W - 1)) * 3 + x);
}
template <int Bits>
__device__ __forceinline__ void quad_store(uint32_t* quads, uint32_t at, uint32_t a, uint32_t b, uint32_t c,
                                           uint32_t d) {
  if (Bits == 8)
    quads[at] = a | b << 8 | c << 16 | d << 24;
  else
    reinterpret_cast<uint2*>(quads)[at] = make_uint2(a | b << 16, c | d << 16);
}

// Level 0: the crop as float; with `quads`, also the crop's quads.
template <class T>
__global__ void pyramid0_kernel(const T* __restrict__ src, int64_t pitch, int crop_row, int crop_col, LevelImage dst,
                                uint32_t* __restrict__ quads, int quad_tiles) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y * blockDim.y + threadIdx.y;
  if (c >= dst.w || r >= dst.h) return;
  const T* row = src + (int64_t(crop_row) + r) * pitch + crop_col;
  const uint32_t v = row[c];
  dst.v[size_t(r) * dst.w + c] = float(v);
  if (quads) {
    const int c1 = c + 1 < dst.w ? c + 1 : c;
    const T* next = r + 1 < dst.h ? row + pitch : row;
    constexpr int Bits = 8 * sizeof(T);
    quad_store<Bits>(quads, quad_at<Bits>(c, r, quad_tiles), v, row[c1], next[c], next[c1]);
  }
}

// Quads of a level held as float.
template <int Bits>
__global__ void quads_kernel(const float* __restrict__ v, int w, int h, int tiles, uint32_t* __restrict__ quads) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y * blockDim.y + threadIdx.y;
  if (c >= w || r >= h) return;
  const int c1 = c + 1 < w ? c + 1 : c;
  const float* row = v + size_t(r) * w;
  const float* next = r + 1 < h ? row + w : row;
  quad_store<Bits>(quads, quad_at<Bits>(c, r, tiles), uint32_t(row[c]), uint32_t(row[c1]), uint32_t(next[c]),
                   uint32_t(next[c1]));
}

// level k+1 from level k: 2x2 sums with the reference's clamped neighbours
// (src/ncc_matching/matcher.cpp:436-453)
__global__ void pyramid_kernel(LevelImage src, LevelImage dst, int32_t* error_flag) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y * blockDim.y + threadIdx.y;
  if (c >= dst.w || r >= dst.h) return;
  const int r0 = 2 * r, r1 = min(r0 + 1, src.h - 1), c0 = 2 * c, c1 = min(c0 + 1, src.w - 1);
  const float a = src.v[size_t(r0) * src.w + c0], b = src.v[size_t(r0) * src.w + c1];
  const float d = src.v[size_t(r1) * src.w + c0], e = src.v[size_t(r1) * src.w + c1];
  const float s = ((a + b) + d) + e;
  if (s >= 16777216.f) atomicExch(error_flag, int32_t(kUnsupported));
  dst.v[size_t(r) * dst.w + c] = s;
}

// Prefixes of one row by a warp: a lane sums four consecutive columns, the
// lanes' totals are scanned, and the next 128 columns are loaded before this
// step's scan.  T: uint32 (modulo 2^32, the same stored values) or int64.
template <class T, class Pair>
__device__ __forceinline__ void prefix_row(const float* __restrict__ row, int w, Pair* out) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) out[0] = Pair{0, 0};
  auto load = [&](int base, float (&v)[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = base + 4 * lane + k < w ? row[base + 4 * lane + k] : 0.f;
  };
  float next[4];
  load(0, next);
  T c1 = 0, c2 = 0;
  for (int base = 0; base < w; base += 128) {
    T a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const T s = T(next[k]);
      a[k] = (k ? a[k - 1] : T(0)) + s;
      b[k] = (k ? b[k - 1] : T(0)) + s * s;
    }
    load(base + 128, next);
    T t1 = a[3], t2 = b[3];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T u1 = __shfl_up_sync(0xffffffffu, t1, o), u2 = __shfl_up_sync(0xffffffffu, t2, o);
      if (lane >= o) {
        t1 += u1;
        t2 += u2;
      }
    }
    const T e1 = c1 + t1 - a[3], e2 = c2 + t2 - b[3];  // before this lane's columns
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = base + 4 * lane + k;
      if (c < w) out[c + 1] = Pair{e1 + a[k], e2 + b[k]};
    }
    c1 += __shfl_sync(0xffffffffu, t1, 31);
    c2 += __shfl_sync(0xffffffffu, t2, 31);
  }
}

// Row prefix sums {sum S, sum S^2}, one warp per row, the rows of every level
// of the find in one launch (the widest level first): the levels' chains of
// row steps run side by side.  Three levels of 2048^2: 0.043 -> 0.010 ms.
__global__ void prefix_kernel(const __grid_constant__ PrefixArgs a) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, l = 0;
  while (l < a.n && warp >= a.lev[l].h) warp -= a.lev[l++].h;
  if (l >= a.n) return;
  const LevelImage& lev = a.lev[l];
  const float* row = lev.v + size_t(warp) * lev.w;
  const size_t at = size_t(warp) * (lev.w + 1);
  if (lev.prefix32)
    prefix_row<uint32_t>(row, lev.w, lev.prefix32 + at);
  else
    prefix_row<long long>(row, lev.w, lev.prefix + at);
}

// ---------------------------------------------------------------- coarse scan
// Dense score planes of the top level for the kept coarse patches
// (src/ncc_matching/matcher.cpp:542-579).  Block = 32x8 positions of one
// patch; the image tile with the patch's reach is staged in shared memory.
constexpr int kTileW = 32, kTileH = 8;

__global__ void __launch_bounds__(256) coarse_kernel(CoarseArgs a) {
  extern __shared__ float tile[];
  const int p = blockIdx.z;
  if (a.skip && a.skip[p]) return;  // plane written by the tensor-core scan
  const PatchDesc pd = a.view.patches[a.plist[p]];
  const PosRange rg = a.ranges[p];
  const int R0 = blockIdx.y * kTileH, C0 = blockIdx.x * kTileW;
  const int TW = kTileW + pd.cmax - pd.cmin, TH = kTileH + pd.rmax - pd.rmin;
  const int tid = threadIdx.y * kTileW + threadIdx.x;
  const int w = a.lev.w, h = a.lev.h;
  // tiles with no valid position only write -inf
  const bool any = R0 < rg.r1 && R0 + kTileH > rg.r0 && C0 < rg.c1 && C0 + kTileW > rg.c0;
  if (any) {
    for (int i = tid; i < TW * TH; i += 256) {
      const int gr = R0 + pd.rmin + i / TW, gc = C0 + pd.cmin + i % TW;
      tile[i] = (gr >= 0 && gc >= 0 && gr < h && gc < w) ? a.lev.v[size_t(gr) * w + gc] : 0.f;
    }
  }
  __syncthreads();
  const int r = R0 + threadIdx.y, c = C0 + threadIdx.x;
  if (r >= h || c >= w) return;
  float score = -INFINITY;
  if (any && r >= rg.r0 && r < rg.r1 && c >= rg.c0 && c < rg.c1 &&
      (!a.dom.mask || may_contain(a.dom, lattice_pose(a.crop_row, a.scale, r, pd.orow, a.phase),
                                  lattice_pose(a.crop_col, a.scale, c, pd.ocol, a.phase), a.scale))) {
    const int2* sw = a.view.sw + pd.sample_off;
    const float* base = tile + (threadIdx.y - pd.rmin) * TW + (threadIdx.x - pd.cmin);
    const int2 f0 = __ldg(sw);
    const float s0 = base[off_row(f0.x) * TW + off_col(f0.x)];
    float acc0 = 0.f, acc1 = 0.f;
    int i = 0;
    for (; i + 1 < pd.n; i += 2) {
      const int2 x = __ldg(sw + i), y = __ldg(sw + i + 1);
      acc0 = fmaf(__int_as_float(x.y), base[off_row(x.x) * TW + off_col(x.x)] - s0, acc0);
      acc1 = fmaf(__int_as_float(y.y), base[off_row(y.x) * TW + off_col(y.x)] - s0, acc1);
    }
    if (i < pd.n) {
      const int2 x = __ldg(sw + i);
      acc0 = fmaf(__int_as_float(x.y), base[off_row(x.x) * TW + off_col(x.x)] - s0, acc0);
    }
    long long s1, s2;
    window_moments(a.lev, w + 1, r, c, a.view.run4 + pd.run_off, pd.nruns, s1, s2);
    score = window_score(acc0 + acc1, s1, s2, pd.n, a.absolute);
  }
  a.planes[(size_t(p) * h + r) * w + c] = score;
}

// Pseudo-candidates of the tensor-core coarse scan: per virtual source, one
// per 5x5 block of top-level positions, centred in the block; they are
// already grouped by source, so the order is the identity and a source's
// tiles are runs of 16 consecutive candidates.
__global__ void coarse_lattice_kernel(Cand* cand, int2* rc, int nsrc, int nbr, int nbc, const int32_t* group_of_src,
                                      int32_t* order, TcTiles* tiles, QueryState* state, int slot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int nb = nbr * nbc, tps = (nb + kTcCands - 1) / kTcCands;  // tiles per source
  if (i == 0) {
    state->count[slot] = nsrc * nb;
    tiles->count = nsrc * tps;
    tiles->next = 0;
  }
  if (i < nsrc * tps) {
    const int src = i / tps, u = i % tps;
    tiles->group[i] = group_of_src[src];
    tiles->first[i] = src * nb + u * kTcCands;
    tiles->last[i] = src * nb + min(nb, (u + 1) * kTcCands);
  }
  if (i >= nsrc * nb) return;
  const int b = i % nb;
  Cand c{};
  c.patch = i / nb;
  cand[i] = c;
  order[i] = i;
  rc[i] = make_int2(5 * (b / nbc) + 2, 5 * (b % nbc) + 2);
}

// Score planes of the patches the tensor cores correlated (a patch per grid
// row): one thread per plane position (consecutive threads, consecutive
// columns: coalesced moment loads); exact moments and the score as
// coarse_kernel computes them.  A position whose dot is not positive has no
// score above a positive threshold, and only scores above it are read: it
// gets -inf, and the block packs the others, so that the moments (two prefix
// loads per run, which bound the kernel) are summed for about half of the
// positions.  2048^2, 25 patches of 16^2: 70 -> 50 us (with the plain patch 0.073
// -> 0.057 ms); full circle, 48^2: 0.25 -> 0.18 ms.
__global__ void __launch_bounds__(256) coarse_tc_score_kernel(CoarseTcArgs a) {
  __shared__ float s_dot[256];
  __shared__ unsigned char s_at[256];
  __shared__ int s_count[8];
  const int w = a.lev.w, h = a.lev.h, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j = blockIdx.y, src = a.src_of[j];
  if (src < 0) return;  // coarse_kernel's plane
  const int base = int(blockIdx.x) * 256, cells = h * w;
  float* plane = a.planes + size_t(j) * cells;
  const PatchDesc& pd = a.view.patches[a.plist[j]];
  float dot = 0.f;
  bool need = false;
  if (const int at = base + int(threadIdx.x); at < cells) {
    const int r = at / w, c = at - r * w;
    const PosRange rg = a.ranges[j];
    if (r >= rg.r0 && r < rg.r1 && c >= rg.c0 && c < rg.c1 &&
        (!a.dom.mask || may_contain(a.dom, lattice_pose(a.crop_row, a.scale, r, pd.orow, a.phase),
                                    lattice_pose(a.crop_col, a.scale, c, pd.ocol, a.phase), a.scale))) {
      const int ci = (src * a.lat_r + r / 5) * a.lat_c + c / 5;
      const int pos = (r % 5) * 5 + c % 5, k = a.k_of[j];
      // sum w (S - S0) = sum w S - S0 sum w (first sample S0)
      const int2 f0 = __ldg(a.view.sw + pd.sample_off);
      const float s0 = a.lev.v[size_t(r + off_row(f0.x)) * w + c + off_col(f0.x)];
      dot = fmaf(-s0, a.groups[a.group_of_src[src]].weff_k[k], a.dots[size_t(ci) * kTcScoreStride + k * 25 + pos]);
      need = a.absolute || !(a.threshold > 0) || dot > 0;
    }
    if (!need) plane[at] = -INFINITY;
  }
  const unsigned m = __ballot_sync(0xffffffffu, need);
  if (lane == 0) s_count[warp] = __popc(m);
  __syncthreads();
  int slot = 0, total = 0;
  for (int q = 0; q < 8; ++q) {
    if (q < warp) slot += s_count[q];
    total += s_count[q];
  }
  if (need) {
    slot += __popc(m & ((1u << lane) - 1));
    s_dot[slot] = dot;
    s_at[slot] = (unsigned char)threadIdx.x;
  }
  __syncthreads();
  if (int(threadIdx.x) >= total) return;
  const int at = base + s_at[threadIdx.x], r = at / w, c = at - r * w;
  long long s1, s2;
  window_moments(a.lev, w + 1, r, c, a.view.run4 + pd.run_off, pd.nruns, s1, s2);
  plane[at] = window_score(s_dot[threadIdx.x], s1, s2, pd.n, a.absolute);
}

// 3x3 local maxima >= 0.4*MinScore with the reference's tie rule, compacted
// into the candidate list (src/ncc_matching/matcher.cpp:581-593).
__global__ void nms_kernel(NmsArgs a) {
  const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t plane = int64_t(a.w) * a.h;
  if (idx >= plane * a.nplist) return;
  const int p = int(idx / plane);
  const int rem = int(idx % plane);
  const int r = rem / a.w, c = rem % a.w;
  const float* s = a.planes + size_t(p) * plane;
  const float v = s[rem];
  if (!(v >= a.threshold) || !isfinite(v)) return;
  for (int dr = -1; dr <= 1; ++dr)
    for (int dc = -1; dc <= 1; ++dc) {
      const int rr = r + dr, cc = c + dc;
      if (rr < 0 || cc < 0 || rr >= a.h || cc >= a.w || (!dr && !dc)) continue;
      const float o = s[rr * a.w + cc];
      if (o > v || (o == v && (dr < 0 || (!dr && dc < 0)))) return;
    }
  const int k = atomicAdd(&a.state->count[0], 1);
  if (k >= a.max_candidates) {
    atomicExch(&a.state->overflow, 1);
    return;
  }
  const int32_t pi = a.plist[p];
  const PatchDesc pd = a.view.patches[pi];
  Cand out;
  out.row = lattice_pose(a.crop_row, a.scale, r, pd.orow, a.phase);
  out.col = lattice_pose(a.crop_col, a.scale, c, pd.ocol, a.phase);
  out.angle = pd.angle;
  out.score = double(v);
  out.patch = pi;
  out.pad = 0;
  a.out[k] = out;
}

// ------------------------------------------------------------------ tracking
// For every candidate: the target level's query patches inside its angle
// window (a precomputed list per source patch), 5x5 positions each; the first
// strict maximum in (patch order, dr, dc) wins (src/ncc_matching/matcher.cpp:
// 670-757).  Lane p < 25 of a warp holds position (dr, dc) = (p / 5, p mod 5)
// of one patch at a time.
constexpr int kTrackMaxSel = 64;
constexpr int kTrackWarps = 4;          // tensor-core levels: at most this many warps per candidate
constexpr int kTrackParts = 4;          // column-strip groups of a patch (one warp each)

// Target patch of a candidate: plist entry, and the centre position on the
// target level, round((pose - crop - offset) / step - origin).
struct TrackCentre {
  float x32r, x32c;
  double xr, xc;
};
__device__ __forceinline__ TrackCentre track_centre(const TrackArgs& a, const Cand& cd) {
  TrackCentre t{};
  if (a.exact32) {
    t.x32r = __fmul_rn(__fsub_rn(__fsub_rn(float(cd.row), a.crop_row32), a.offset32), a.inv_step32);
    t.x32c = __fmul_rn(__fsub_rn(__fsub_rn(float(cd.col), a.crop_col32), a.offset32), a.inv_step32);
  } else {
    t.xr = dsub(dsub(cd.row, a.crop_row), a.offset) / a.step;
    t.xc = dsub(dsub(cd.col, a.crop_col), a.offset) / a.step;
  }
  return t;
}
__device__ __forceinline__ int track_row(const TrackArgs& a, const TrackCentre& t, const PatchDesc& pd) {
  return a.exact32 ? int(roundf(__fsub_rn(t.x32r, pd.orow32))) : int(round(dsub(t.xr, pd.orow)));
}
__device__ __forceinline__ int track_col(const TrackArgs& a, const TrackCentre& t, const PatchDesc& pd) {
  return a.exact32 ? int(roundf(__fsub_rn(t.x32c, pd.ocol32))) : int(round(dsub(t.xc, pd.ocol)));
}

__device__ __forceinline__ bool track_valid(const TrackArgs& a, const PatchDesc& pd, const PosRange& rg, int r, int c) {
  if (!(r >= rg.r0 && r < rg.r1 && c >= rg.c0 && c < rg.c1)) return false;
  return !a.dom.mask || may_contain(a.dom, lattice_pose(a.crop_row, a.step, r, pd.orow, a.offset),
                                    lattice_pose(a.crop_col, a.step, c, pd.ocol, a.offset), a.step);
}

// Window moments of lane position (dr, dc) at level position (r, c) of one
// patch; lanes of a warp share the patch.  A lane starts dr runs behind, so
// that in every step the lanes of all five dr read the same image row (the
// runs of successive rows begin and end within a few columns of one
// another): a step's 25 prefix entries lie in one or two cache lines instead
// of five.  The sums are exact integers, so their order is free.
template <int U>  // runs in flight with int64 prefixes
__device__ __forceinline__ void lane_moments(const LevelImage& lev, int pitch, int r, int c,
                                             const int4* __restrict__ runs, int nruns, int dr, long long& s1,
                                             long long& s2) {
  s1 = 0;
  s2 = 0;
  int at = nruns - dr;
  while (at < 0) at += nruns;
  if (at == nruns) at = 0;
  auto next = [&] {
    const int4 q = __ldg(runs + at);
    if (++at == nruns) at = 0;
    return q;
  };
  if (lev.prefix32) {
    const uint2* __restrict__ P = lev.prefix32;
    int j = 0;
    for (; j + 3 < nruns; j += 4) {
      int4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = next();
      uint2 hi[4], lo[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t base = uint32_t(r + q[u].x) * uint32_t(pitch) + uint32_t(c);
        hi[u] = P[base + uint32_t(q[u].z + 1)];
        lo[u] = P[base + uint32_t(q[u].y)];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        s1 += (long long)(hi[u].x - lo[u].x);
        s2 += (long long)(hi[u].y - lo[u].y);
      }
    }
    for (; j < nruns; ++j) {
      const int4 q = next();
      const uint32_t base = uint32_t(r + q.x) * uint32_t(pitch) + uint32_t(c);
      const uint2 hi = P[base + uint32_t(q.z + 1)], lo = P[base + uint32_t(q.y)];
      s1 += (long long)(hi.x - lo.x);
      s2 += (long long)(hi.y - lo.y);
    }
    return;
  }
  const longlong2* __restrict__ P = lev.prefix;
  int j = 0;
  for (; j + U - 1 < nruns; j += U) {
    longlong2 hi[U], lo[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int4 q = next();
      const uint32_t base = uint32_t(r + q.x) * uint32_t(pitch) + uint32_t(c);
      hi[u] = P[base + uint32_t(q.z + 1)];
      lo[u] = P[base + uint32_t(q.y)];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      s1 += hi[u].x - lo[u].x;
      s2 += hi[u].y - lo[u].y;
    }
  }
  for (; j < nruns; ++j) {
    const int4 q = next();
    const uint32_t base = uint32_t(r + q.x) * uint32_t(pitch) + uint32_t(c);
    const longlong2 hi = P[base + uint32_t(q.z + 1)], lo = P[base + uint32_t(q.y)];
    s1 += hi.x - lo.x;
    s2 += hi.y - lo.y;
  }
}

// The same with 32-bit sums, where the host found that sum S of a window and
// sum S^2 of any four runs stay below 2^32 (uint8 levels 1 and 2): the index
// and sum arithmetic around the loads is what bounds these levels.
__device__ __forceinline__ void lane_moments_narrow(const LevelImage& lev, int pitch, int r, int c,
                                                    const int4* __restrict__ runs, int nruns, int dr, uint32_t& s1,
                                                    unsigned long long& s2) {
  const uint2* __restrict__ P = lev.prefix32 + (size_t(r) * pitch + c);
  int at = nruns - dr;
  while (at < 0) at += nruns;
  if (at == nruns) at = 0;
  s1 = 0;
  s2 = 0;
  for (int j = 0; j < nruns; j += 4) {
    uint2 hi[4], lo[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int4 q = __ldg(runs + at);
      if (j + u < nruns) {
        if (++at == nruns) at = 0;
        const int base = q.x * pitch;
        hi[u] = P[base + q.z + 1];
        lo[u] = P[base + q.y];
      } else {
        hi[u] = lo[u] = make_uint2(0, 0);
      }
    }
    uint32_t four = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s1 += hi[u].x - lo[u].x;
      four += hi[u].y - lo[u].y;
    }
    s2 += four;
  }
}

// Totals of 25 per-lane values over a warp: lane p < 25 returns value p's.
// Each of the five steps halves the values a lane carries (31 shuffles
// instead of 125).
__device__ __forceinline__ float lane_total25(const float (&v)[25]) {
  const int lane = threadIdx.x & 31;
  float x[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float lo = v[i], hi = i + 16 < 25 ? v[i + 16 < 25 ? i + 16 : 0] : 0.f;
    const bool up = lane & 16;
    x[i] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, 16);
  }
#pragma unroll
  for (int w = 8; w > 0; w >>= 1) {
    const bool up = lane & w;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float lo = x[i], hi = x[i + w];
      x[i] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, w);
    }
  }
  return x[0];
}

// First and last run of a patch with samples in columns [x0, x1] (a warp's
// lanes test 32 runs at a time); last < 0 when there is none.
__device__ __forceinline__ int2 runs_meeting(const int4* __restrict__ runs, int nruns, int x0, int x1) {
  const int lane = threadIdx.x & 31;
  int first = INT32_MAX, last = -1;
  for (int j0 = 0; j0 < nruns; j0 += 32) {
    bool meets = false;
    if (j0 + lane < nruns) {
      const int4 q = __ldg(runs + j0 + lane);
      meets = q.y <= x1 && q.z >= x0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, meets);
    if (!m) continue;
    if (first == INT32_MAX) first = j0 + __ffs(m) - 1;
    last = j0 + 31 - __clz(m);
  }
  return make_int2(first, last);
}

// Two FP32 values in a 64-bit register pair, and acc += a * b on both.
using F32x2 = unsigned long long;
__device__ __forceinline__ F32x2 twice(float x) {
  F32x2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float2 halves(F32x2 x) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
  return r;
}
__device__ __forceinline__ void fma_both(F32x2& acc, F32x2 a, F32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// sum w (S - centre) of one patch at the 25 positions from a window in shared
// memory (values minus its centre value); lane p < 25 returns position p's.
// Position (0, 0) puts the patch's row y and column x on window row
// y + rshift and column x + cshift.  The patch is cut into strips of 16
// window columns (strip0, strip0 + step, ... are summed): four lanes own four
// columns each, and the eight groups of four lanes share the runs that meet
// the strip, so a strip costs about an eighth of its rows.  A lane walks down
// its rows with the 5 x 8 values under its four samples in registers: per
// row two 16-byte reads and four weights feed 100 multiply-adds.  The values
// sit in pairs of columns, so that 80 of them are 40 two-wide instructions
// (the kernel is bound by the instructions it issues); an even and an odd
// sample column pair the placements differently and have their own sums.
__device__ __forceinline__ float staged_dots(const float* win, int pitch, const LevelView& view, const PatchDesc& pd,
                                             int rshift, int cshift, int strip0, int step) {
  const int lane = threadIdx.x & 31, group = lane >> 2;
  const int4* __restrict__ runs = view.run4 + pd.run_off;
  const float* __restrict__ weights = view.w + pd.sample_off;
  const int xlast = (pd.cmax + cshift) & ~3;  // window columns of the last samples
  // sums by placement row: even sample columns dc (0, 1), (2, 3), 4; odd ones 0, (1, 2), (3, 4)
  F32x2 e01[5] = {}, e23[5] = {}, o12[5] = {}, o34[5] = {};
  float e4[5] = {}, o0[5] = {};
  for (int base = ((pd.cmin + cshift) & ~3) + 16 * strip0; base <= xlast; base += 16 * step) {
    const int2 span = runs_meeting(runs, pd.nruns, base - cshift, base + 15 - cshift);
    if (span.y < 0) continue;
    const int per = (span.y - span.x + 8) >> 3;  // runs per group
    const int j0 = span.x + group * per, j1 = min(span.y, j0 + per - 1);
    const int X = min(base + 4 * (lane & 3), xlast);  // past the patch: repeats its last columns, no weights
    const int x = base + 4 * (lane & 3) - cshift;     // first sample column
    const float* col = win + X;
    F32x2 v[5][4];  // window row y + i in v[(i + phase) % 5], columns in pairs
    auto load = [&](F32x2 (&r)[4], const float* at) {
      const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(at), hi = *reinterpret_cast<const ulonglong2*>(at + 4);
      r[0] = lo.x, r[1] = lo.y, r[2] = hi.x, r[3] = hi.y;
    };
    // the next run and its weights are loaded one row ahead of their use
    auto run_at = [&](int j) { return __ldg(runs + min(j, pd.nruns - 1)); };
    auto weights_of = [&](const int4& q, bool live, float (&w)[4]) {
      const int u = x - q.y;
      const unsigned len = unsigned(q.z - q.y);
      const float* wp = weights + q.w + u;
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = live && unsigned(u + e) <= len ? __ldg(wp + e) : 0.f;
    };
    int4 next = run_at(j0);
    float wn[4];
    weights_of(next, j0 <= j1, wn);
    int4 after = run_at(j0 + 1);
    int ynext = INT32_MIN;
    for (int it = 0; it < per; it += 5) {
#pragma unroll
      for (int phase = 0; phase < 5; ++phase) {
        const int j = j0 + it + phase;
        if (it + phase < per && j <= j1) {
          const float* row = col + (next.x + rshift) * pitch;
          if (next.x != ynext) {
#pragma unroll
            for (int i = 0; i < 4; ++i) load(v[(phase + i) % 5], row + i * pitch);
          }
          load(v[(phase + 4) % 5], row + 4 * pitch);
          ynext = next.x + 1;
          const float w[4] = {wn[0], wn[1], wn[2], wn[3]};
          next = after;
          weights_of(next, j + 1 <= j1, wn);
          after = run_at(j + 2);
          const F32x2 ww[4] = {twice(w[0]), twice(w[1]), twice(w[2]), twice(w[3])};
#pragma unroll
          for (int i = 0; i < 5; ++i) {
            const F32x2(&r)[4] = v[(phase + i) % 5];
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
              fma_both(e01[i], ww[e], r[e / 2]);
              fma_both(e23[i], ww[e], r[e / 2 + 1]);
              e4[i] = fmaf(w[e], halves(r[e / 2 + 2 < 4 ? e / 2 + 2 : 3]).x, e4[i]);
              o0[i] = fmaf(w[e + 1], halves(r[e / 2]).y, o0[i]);
              fma_both(o12[i], ww[e + 1], r[e / 2 + 1]);
              fma_both(o34[i], ww[e + 1], r[e / 2 + 2 < 4 ? e / 2 + 2 : 3]);
            }
          }
        }
      }
    }
  }
  float acc[25];
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const float2 a = halves(e01[i]), b = halves(e23[i]), c = halves(o12[i]), d = halves(o34[i]);
    acc[5 * i] = a.x + o0[i];
    acc[5 * i + 1] = a.y + c.x;
    acc[5 * i + 2] = b.x + c.y;
    acc[5 * i + 3] = b.y + d.x;
    acc[5 * i + 4] = e4[i] + d.y;
  }
  return lane_total25(acc);
}

// The same straight from the level, for windows that do not fit shared memory
// and for single patches: window position (0, 0) is level position (r0, c0);
// positions outside the level are clamped (they only reach placements that
// are not scored).  Strips of 32 columns, one per lane.
struct LevelWindow {
  const float* v;
  int w, h, r0, c0;
  float centre;
  __device__ __forceinline__ const float* row(int r) const { return v + size_t(min(max(r0 + r, 0), h - 1)) * w; }
  __device__ __forceinline__ int col(int c) const { return min(max(c0 + c, 0), w - 1); }
};
__device__ __forceinline__ float level_dots(const LevelWindow& win, const LevelView& view, const PatchDesc& pd,
                                            int rshift, int cshift, int strip0, int step) {
  const int lane = threadIdx.x & 31;
  const int4* __restrict__ runs = view.run4 + pd.run_off;
  const float* __restrict__ weights = view.w + pd.sample_off;
  float acc[25];
#pragma unroll
  for (int i = 0; i < 25; ++i) acc[i] = 0.f;
  for (int x0 = pd.cmin + 32 * strip0; x0 <= pd.cmax; x0 += 32 * step) {
    const int2 span = runs_meeting(runs, pd.nruns, x0, x0 + 31);
    const int x = x0 + lane, xc = min(x, pd.cmax) + cshift;
    for (int j = span.x; j <= span.y; ++j) {
      const int4 q = __ldg(runs + j);
      const float w = x >= q.y && x <= q.z ? __ldg(weights + q.w + (x - q.y)) : 0.f;
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const float* row = win.row(q.x + i + rshift);
#pragma unroll
        for (int d = 0; d < 5; ++d) acc[5 * i + d] = fmaf(w, __ldg(row + win.col(xc + d)) - win.centre, acc[5 * i + d]);
      }
    }
  }
  return lane_total25(acc);
}

// The tracked candidate from the best item (patch k, position l), or a
// candidate without a score.
__device__ void track_write(const TrackArgs& a, int i, const Cand& cd, float best, int item, const TrackCentre& t,
                            int sel0) {
  Cand out = cd;
  out.score = -INFINITY;
  if (item != INT32_MAX && best > -INFINITY) {
    const int l = item % 25;
    const int32_t pi = a.plist[a.sel_idx[sel0 + item / 25]];
    const PatchDesc pd = a.view.patches[pi];
    const int r = track_row(a, t, pd) + l / 5 - 2, c = track_col(a, t, pd) + l % 5 - 2;
    if (a.exact32) {
      out.row = double(lattice_pose32(a.crop_row32, a.step32, r, pd.orow32, a.offset32));
      out.col = double(lattice_pose32(a.crop_col32, a.step32, c, pd.ocol32, a.offset32));
    } else {
      out.row = lattice_pose(a.crop_row, a.step, r, pd.orow, a.offset);
      out.col = lattice_pose(a.crop_col, a.step, c, pd.ocol, a.offset);
    }
    out.angle = pd.angle;
    out.score = double(best);
    out.patch = pi;
  }
  a.out[i] = out;
}

// sum w (S - S0) = sum w S - S0 sum w of a patch scored on the tensor cores (first sample S0)
__device__ __forceinline__ float track_tc_dot(const TrackArgs& a, const PatchDesc& pd, int src, int i, int k, int pos,
                                              int r, int c) {
  const int2 f0 = __ldg(a.view.sw + pd.sample_off);
  const float s0 = a.lev.v[size_t(r + off_row(f0.x)) * a.lev.w + c + off_col(f0.x)];
  return fmaf(-s0, a.tc_groups[a.tc_group_of_src[src]].weff_k[k],
              a.tc_dots[size_t(i) * kTcScoreStride + k * 25 + pos]);
}

// Levels whose lists were scored on the tensor cores, all but at most two
// patches each (the unrotated patch: its origin is off the lattice): one block
// of one to four warps per candidate, each warp with its own patches; they add the exact moments,
// the score and the choice.  The few patches the tensor cores left out are
// correlated first, by the block.  Bound by the instructions around the
// prefix loads and their latency.  2048^2 u8, 128^2 template, two steps: 0.27
// -> 0.16 ms; 57,000 candidates of a 48^2 template over a full circle: 1.03 ->
// 0.56 ms.

// Dots of patch k of candidate cd, sum w (S - S0), by the whole block, to
// out[position].  Kept out of line: few candidates need it, and its registers
// would cost the loop over the moments its occupancy.
__device__ __noinline__ void plain_dots(const TrackArgs& a, const Cand& cd, int k, float (*part)[32], float* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const PatchDesc pd = a.view.patches[a.plist[a.sel_idx[a.sel_off[cd.patch] + k]]];
  const TrackCentre t = track_centre(a, cd);
  const int row = track_row(a, t, pd), col = track_col(a, t, pd);
  const int cr = min(max(row, 0), a.lev.h - 1), cc = min(max(col, 0), a.lev.w - 1);
  const LevelWindow win{a.lev.v, a.lev.w, a.lev.h, row - 2, col - 2, a.lev.v[size_t(cr) * a.lev.w + cc]};
  part[warp][lane] = level_dots(win, a.view, pd, 0, 0, warp, blockDim.x >> 5);
  __syncthreads();
  if (warp == 0) {
    float dot = 0.f;
    for (int u = 0; u < int(blockDim.x >> 5); ++u) dot += part[u][lane];
    // sum w (S - S0) = sum w (S - centre) - (S0 - centre) sum w
    const int2 f0 = __ldg(a.view.sw + pd.sample_off);
    const float s0 = __ldg(win.row(lane / 5 + off_row(f0.x)) + win.col(lane % 5 + off_col(f0.x)));
    out[lane] = fmaf(-(s0 - win.centre), pd.wsum, dot);
    if (lane == 0) atomicAdd(&a.state->track_macs, 25ull * (unsigned long long)pd.n);
  }
  __syncthreads();
}

template <bool Narrow>
__global__ void __launch_bounds__(32 * kTrackWarps, 8) track_warp_kernel(const __grid_constant__ TrackArgs a) {
  __shared__ float s_part[kTrackWarps][32], s_dot[2][32];
  __shared__ float s_best[kTrackWarps];
  __shared__ int s_item[kTrackWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int live = live_count(a.state, a.in_slot);
  const int dr = lane / 5, dc = lane - 5 * dr;
  for (int i = blockIdx.x; i < live; i += gridDim.x) {
    const Cand cd = a.in[i];
    const int src = cd.patch;
    const int sel0 = src >= 0 ? a.sel_off[src] : 0;
    const int n = src >= 0 ? min(a.sel_off[src + 1] - sel0, kTcMaxP) : 0;
    const bool tc = src >= 0 && a.tc_group_of_src[src] >= 0;
    // patches without dots
    bool plain = false;
    if (lane < n) {
      const PatchDesc& pd = a.view.patches[a.plist[a.sel_idx[sel0 + lane]]];
      plain = !tc || !pd.lattice;
    }
    const unsigned left = __ballot_sync(0xffffffffu, plain);
    int slot = 0;
    for (unsigned todo = left; todo && slot < 2; todo &= todo - 1, ++slot)
      plain_dots(a, cd, __ffs(todo) - 1, s_part, s_dot[slot]);
    const TrackCentre t = track_centre(a, cd);
    float best = -INFINITY;
    int border = INT32_MAX;
    for (int k = warp; k < n; k += nwarps) {
      const int j = a.sel_idx[sel0 + k];
      const PatchDesc pd = a.view.patches[a.plist[j]];
      const int r = track_row(a, t, pd) + dr - 2, c = track_col(a, t, pd) + dc - 2;
      if (lane >= 25 || !track_valid(a, pd, a.ranges[j], r, c)) continue;
      const float dot = left >> k & 1 ? s_dot[min(1, __popc(left & ((1u << k) - 1)))][lane]
                                      : track_tc_dot(a, pd, src, i, k, lane, r, c);
      float sc;
      if (Narrow) {
        uint32_t s1;
        unsigned long long s2;
        lane_moments_narrow(a.lev, a.lev.w + 1, r, c, a.view.run4 + pd.run_off, pd.nruns, dr, s1, s2);
        sc = window_score_narrow(dot, s1, s2, pd.n, a.absolute);
      } else {
        long long s1, s2;
        lane_moments<2>(a.lev, a.lev.w + 1, r, c, a.view.run4 + pd.run_off, pd.nruns, dr, s1, s2);
        sc = window_score(dot, s1, s2, pd.n, a.absolute);
      }
      if (better(sc, k * 25 + lane, best, border)) {
        best = sc;
        border = k * 25 + lane;
      }
    }
    __syncwarp();
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oo = __shfl_xor_sync(0xffffffffu, border, o);
      if (better(ob, oo, best, border)) {
        best = ob;
        border = oo;
      }
    }
    if (lane == 0) {
      s_best[warp] = best;
      s_item[warp] = border;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < nwarps; ++w)
        if (better(s_best[w], s_item[w], best, border)) {
          best = s_best[w];
          border = s_item[w];
        }
      track_write(a, i, cd, best, border, t, sel0);
    }
    __syncthreads();
  }
}

// Other levels: one block per candidate.  The union window of the patches
// the block correlates is staged in shared memory, centred on one of its
// pixels (exact small integers in float; zero outside the level); the warps
// take (patch, strip group) and (patch, run group) tasks, and then the items
// are scored.  Windows larger than shared memory read the level.  Bound by
// the latency of a candidate's phases with the 16 warps per SM that the
// register tiles leave (set-up and staging a quarter of them, dots and
// moments 60 %).  uint16 lists, two steps at 2048^2 with a 128^2 template
// (3.1 G multiply-adds): 1.98 -> 0.92 ms; three at 4096^2 with 256^2 (21 G):
// 40 -> 5.0 ms.
__global__ void __launch_bounds__(512) track_block_kernel(TrackArgs a) {
  extern __shared__ float smem[];
  __shared__ int s_row[kTrackMaxSel], s_col[kTrackMaxSel];
  __shared__ unsigned char s_istc[kTrackMaxSel];
  __shared__ int s_bound[4];
  __shared__ float s_wbest[16];
  __shared__ int s_word[16];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  // dots of the strip groups | moments | window
  float* s_dot = smem;
  long long* s_mom = reinterpret_cast<long long*>(smem + size_t(a.sel_max) * kTrackParts * 32);
  float* win = smem + size_t(a.sel_max) * (kTrackParts * 32 + 2 * 2 * 32);
  const int live = live_count(a.state, a.in_slot);
  for (int i = blockIdx.x; i < live; i += gridDim.x) {
    const Cand cd = a.in[i];
    const int src = cd.patch;
    const int sel0 = src >= 0 ? a.sel_off[src] : 0;
    const int n = src >= 0 ? min(a.sel_off[src + 1] - sel0, kTrackMaxSel) : 0;
    const bool tc = a.tc_dots && src >= 0 && a.tc_group_of_src[src] >= 0;
    const TrackCentre t = track_centre(a, cd);
    if (warp == 0) {
      int wr0 = INT32_MAX, wc0 = INT32_MAX, wr1 = INT32_MIN, wc1 = INT32_MIN;
      unsigned samples = 0;
      for (int k = lane; k < n; k += 32) {
        const PatchDesc pd = a.view.patches[a.plist[a.sel_idx[sel0 + k]]];
        const int row = track_row(a, t, pd), col = track_col(a, t, pd);
        s_row[k] = row;
        s_col[k] = col;
        const bool istc = tc && pd.lattice && k < kTcMaxP;
        s_istc[k] = istc;
        if (!istc) {
          samples += unsigned(pd.n);
          wr0 = min(wr0, row - 2 + pd.rmin);
          wr1 = max(wr1, row + 2 + pd.rmax);
          wc0 = min(wc0, col - 2 + pd.cmin);
          wc1 = max(wc1, col + 2 + pd.cmax);
        }
      }
      wr0 = __reduce_min_sync(0xffffffffu, wr0);
      wc0 = __reduce_min_sync(0xffffffffu, wc0);
      wr1 = __reduce_max_sync(0xffffffffu, wr1);
      wc1 = __reduce_max_sync(0xffffffffu, wc1);
      samples = __reduce_add_sync(0xffffffffu, samples);
      if (lane == 0) {
        if (samples) atomicAdd(&a.state->track_macs, 25ull * samples);
        s_bound[0] = wr0;
        s_bound[1] = wr1;
        s_bound[2] = wc0;
        s_bound[3] = wc1;
      }
    }
    __syncthreads();
    const bool any = s_bound[0] <= s_bound[1];  // the block correlates some patch
    const int wr0 = any ? s_bound[0] : 0, wc0 = any ? s_bound[2] : 0;
    const int wh = any ? s_bound[1] - wr0 + 1 : 0, ww = any ? s_bound[3] - wc0 + 1 : 0;
    const bool staged = any && wh <= a.win_rows && ww + 4 <= a.win_pitch;
    float centre = 0.f;
    if (any) {
      const int cr = min(max(wr0 + wh / 2, 0), a.lev.h - 1), cc = min(max(wc0 + ww / 2, 0), a.lev.w - 1);
      centre = a.lev.v[size_t(cr) * a.lev.w + cc];
    }
    for (int t = threadIdx.x; t < n * 32; t += blockDim.x) s_mom[t] = s_mom[a.sel_max * 32 + t] = 0;
    if (staged) {
      // a warp per row, consecutive columns, four rows in flight
      const int cols = min(ww + 4, a.win_pitch);
      for (int r0 = warp; r0 < wh; r0 += 4 * nwarps)
        for (int x = lane; x < cols; x += 32) {
          const bool in_x = wc0 + x >= 0 && wc0 + x < a.lev.w;
          float v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int r = wr0 + r0 + u * nwarps;
            v[u] = in_x && r >= 0 && r < a.lev.h ? a.lev.v[size_t(r) * a.lev.w + wc0 + x] - centre : 0.f;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (r0 + u * nwarps < wh) win[(r0 + u * nwarps) * a.win_pitch + x] = v[u];
        }
    }
    __syncthreads();
    // (patch, strip group) and (patch, run group) tasks; the moments' run
    // groups keep their loads' latency off the block's critical path
    constexpr int parts = kTrackParts;
    for (int task = warp; task < n * 2 * kTrackParts; task += nwarps) {
      const int k = task % n, part = task / n;
      const int j = a.sel_idx[sel0 + k];
      const PatchDesc pd = a.view.patches[a.plist[j]];
      if (part >= parts) {
        const int dr = lane / 5, dc = lane - 5 * dr;
        const int r = s_row[k] + dr - 2, c = s_col[k] + dc - 2;
        const int per = (pd.nruns + kTrackParts - 1) / kTrackParts, first = (part - parts) * per;
        const int count = min(per, pd.nruns - first);
        if (count > 0 && lane < 25 && track_valid(a, pd, a.ranges[j], r, c)) {
          long long s1 = 0, s2 = 0;
          lane_moments<4>(a.lev, a.lev.w + 1, r, c, a.view.run4 + pd.run_off + first, count, dr, s1, s2);
          atomicAdd(reinterpret_cast<unsigned long long*>(s_mom + k * 32 + lane), (unsigned long long)s1);
          atomicAdd(reinterpret_cast<unsigned long long*>(s_mom + (a.sel_max + k) * 32 + lane), (unsigned long long)s2);
        }
      } else if (!s_istc[k]) {
        const int rs = s_row[k] - 2 - wr0, cs = s_col[k] - 2 - wc0;
        s_dot[(k * kTrackParts + part) * 32 + lane] =
            staged ? staged_dots(win, a.win_pitch, a.view, pd, rs, cs, part, parts)
                   : level_dots(LevelWindow{a.lev.v, a.lev.w, a.lev.h, wr0, wc0, centre}, a.view, pd, rs, cs, part,
                                parts);
      }
    }
    __syncthreads();
    float best = -INFINITY;
    int border = INT32_MAX;
    for (int it = threadIdx.x; it < n * 25; it += blockDim.x) {
      const int k = it / 25, pos = it - 25 * k;
      const int j = a.sel_idx[sel0 + k];
      const PatchDesc pd = a.view.patches[a.plist[j]];
      const int r = s_row[k] + pos / 5 - 2, c = s_col[k] + pos % 5 - 2;
      if (!track_valid(a, pd, a.ranges[j], r, c)) continue;
      float dot;
      if (s_istc[k]) {
        dot = track_tc_dot(a, pd, src, i, k, pos, r, c);
      } else {
        dot = 0.f;
        for (int q = 0; q < parts; ++q) dot += s_dot[(k * kTrackParts + q) * 32 + pos];
        // sum w (S - S0) = sum w (S - centre) - (S0 - centre) sum w
        const int2 f0 = __ldg(a.view.sw + pd.sample_off);
        const float x0 = a.lev.v[size_t(r + off_row(f0.x)) * a.lev.w + c + off_col(f0.x)] - centre;
        dot = fmaf(-x0, pd.wsum, dot);
      }
      const float sc = window_score(dot, s_mom[k * 32 + pos], s_mom[(a.sel_max + k) * 32 + pos], pd.n, a.absolute);
      if (better(sc, it, best, border)) {
        best = sc;
        border = it;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oo = __shfl_xor_sync(0xffffffffu, border, o);
      if (better(ob, oo, best, border)) {
        best = ob;
        border = oo;
      }
    }
    if (lane == 0) {
      s_wbest[warp] = best;
      s_word[warp] = border;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 0; w < nwarps; ++w)
        if (better(s_wbest[w], s_word[w], best, border)) {
          best = s_wbest[w];
          border = s_word[w];
        }
      track_write(a, i, cd, best, border, t, sel0);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------ merge_identical
__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdULL;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ULL;
  x ^= x >> 33;
  return x;
}

// Snap poses outside the image to the nearest in-image pixel within 4 rows
// and columns (full-image domain; src/ncc_matching/matcher.cpp:633-643).
__device__ void snap_pose(Cand& p, double height, double width) {
  const double rr = floor(p.row + .5), cc = floor(p.col + .5);
  if (rr >= 0 && cc >= 0 && rr < height && cc < width) return;
  double best = INFINITY, nr = p.row, nc = p.col;
  const double first = fmax(0., ceil(p.row - 4));
  for (double r = first; r <= p.row + 4 && r < height; r += 1) {
    const double c = fmin(fmax(round(p.col), 0.), width - 1);
    if (fabs(c - p.col) > 4) continue;
    const double dist = hypot(r - p.row, c - p.col);
    if (dist < best) {
      best = dist;
      nr = r;
      nc = c;
    }
  }
  if (isfinite(best)) {
    p.row = nr;
    p.col = nc;
    p.patch = -1;
  } else {
    p.score = -INFINITY;
  }
}

// The same for a reduced domain: the nearest pixel of the domain's runs
// within 4 rows and columns; runs are visited in (row, begin) order and only
// a strictly nearer one replaces the best (src/ncc_matching/matcher.cpp:633-643).
__device__ void snap_pose_domain(Cand& p, const DomainView& d) {
  if (domain_contains(d, p.row, p.col)) return;
  double best = INFINITY, nr = p.row, nc = p.col;
  const int first = max(0, int(ceil(p.row - 4)));
  const double rc = round(p.col);
  for (int y = first; y < d.h && y <= p.row + 4; ++y)
    for (int k = d.row_run[y]; k < d.row_run[y + 1]; ++k) {
      const int4 run = d.runs[k];
      const double c = fmin(fmax(rc, double(run.y)), double(run.z));
      if (fabs(c - p.col) > 4) continue;
      const double dist = hypot(double(run.x) - p.row, c - p.col);
      if (dist < best) {
        best = dist;
        nr = double(run.x);
        nc = c;
      }
    }
  if (isfinite(best)) {
    p.row = nr;
    p.col = nc;
    p.patch = -1;
  } else {
    p.score = -INFINITY;
  }
}

__global__ void snap_kernel(Cand* c, const QueryState* state, int slot, double height, double width, DomainView dom) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= live_count(state, slot)) return;
  Cand p = c[i];
  if (dom.mask)
    snap_pose_domain(p, dom);
  else
    snap_pose(p, height, width);
  c[i] = p;
}

// merge_identical + threshold (src/ncc_matching/matcher.cpp:241-248,758-760):
// keep one candidate per exact (row, column, angle), drop non-finite scores
// and scores below the threshold; order is irrelevant downstream.
__global__ void dedup_kernel(DedupArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= live_count(a.state, a.in_slot)) return;
  const Cand p = a.in[i];
  if (!isfinite(p.score) || p.score < a.threshold) return;
  const unsigned long long kr = __double_as_longlong(p.row), kc = __double_as_longlong(p.col),
                           ka = __double_as_longlong(p.angle);
  const unsigned mask = unsigned(a.hash_slots - 1);
  unsigned slot = unsigned(mix64(kr ^ mix64(kc ^ mix64(ka)))) & mask;
  for (int probe = 0; probe < a.hash_slots; ++probe) {
    const int prev = atomicCAS(a.table + slot, -1, i);
    if (prev == -1) {
      const int k = atomicAdd(&a.state->count[a.out_slot], 1);
      a.out[k] = p;
      return;
    }
    const Cand q = a.in[prev];
    if ((unsigned long long)__double_as_longlong(q.row) == kr && (unsigned long long)__double_as_longlong(q.col) == kc &&
        (unsigned long long)__double_as_longlong(q.angle) == ka)
      return;
    slot = (slot + 1) & mask;
  }
}

// -------------------------------------------------- full-resolution scoring
// Block totals of K per-thread values as FP32 pairs, in s.total[k] for every
// thread.  The order of the additions is that of a shuffle tree over the
// lanes (16, 8, 4, 2, 1 apart) and one over the warps, but a lane carries
// only the values it will own: each step halves them, so 19 values cost 21
// pair additions a lane instead of 95, and the warps' partials are added by
// one warp per value instead of one warp for all.  (Pair addition is
// commutative to the bit, and adding a zero pair changes nothing.)
// The threads may be spread over the C blocks of a cluster (the warps of
// block r follow those of block r - 1): a warp writes its partials into
// every block's shared memory, so each block has the totals and goes on by
// itself, and one cluster barrier separates the passes (two buffers: a block
// may be one pass ahead of a reader).
template <int K> struct BlockTotals {
  F2 part[2][K][16];  // by value and warp
  F2 total[K];
};

template <int C> __device__ __forceinline__ int team_rank() {
  if (C == 1) return 0;
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return int(r);
}
// This thread's number among the C blocks' threads, and their count.
template <int C> __device__ __forceinline__ int team_thread() { return team_rank<C>() * int(blockDim.x) + int(threadIdx.x); }
template <int C> __device__ __forceinline__ int team_size() { return C * int(blockDim.x); }
template <int C> __device__ __forceinline__ void team_sync() {
  if (C == 1) {
    __syncthreads();
    return;
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Stores a pair at the same place of every block's shared memory.
template <int C> __device__ __forceinline__ void team_store(F2* p, F2 v) {
  static_assert(alignof(F2) == 8, "one vector store per pair");
  if (C == 1) {
    *p = v;
    return;
  }
  const uint32_t at = uint32_t(__cvta_generic_to_shared(p));
#pragma unroll
  for (int r = 0; r < C; ++r)
    asm volatile(
        "{\n .reg .b32 a;\n mapa.shared::cluster.u32 a, %0, %1;\n st.shared::cluster.v2.f32 [a], {%2, %3};\n}\n" ::"r"(
            at),
        "r"(r), "f"(v.hi), "f"(v.lo)
        : "memory");
}

template <int N> struct LaneFold {
  // x: N values of which this lane's subset holds `count`; halves them
  static __device__ __forceinline__ F2 run(const F2 (&x)[N], int bit, int& index, int& count) {
    constexpr int H = (N + 1) / 2;
    const bool up = threadIdx.x & bit;
    F2 y[H];
#pragma unroll
    for (int i = 0; i < H; ++i) {
      const F2 a = x[i], b = i + H < N ? x[i + H < N ? i + H : 0] : F2{0.f, 0.f};
      const F2 send = up ? a : b, keep = up ? b : a;
      y[i] = f2_add(keep, F2{__shfl_xor_sync(0xffffffffu, send.hi, bit), __shfl_xor_sync(0xffffffffu, send.lo, bit)});
    }
    index += up ? H : 0;
    count = up ? count - H : min(count, H);
    return LaneFold<H>::run(y, bit >> 1, index, count);
  }
};
template <> struct LaneFold<1> {
  static __device__ __forceinline__ F2 run(const F2 (&x)[1], int bit, int&, int&) {
    F2 y = x[0];
    for (; bit > 0; bit >>= 1)
      y = f2_add(y, F2{__shfl_xor_sync(0xffffffffu, y.hi, bit), __shfl_xor_sync(0xffffffffu, y.lo, bit)});
    return y;
  }
};

template <int C = 1, int K>
__device__ __forceinline__ void block_total(const float (&v)[K], BlockTotals<K>& s, int buffer = 0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  F2 x[K];
#pragma unroll
  for (int k = 0; k < K; ++k) x[k] = f2(v[k]);
  int index = 0, count = K;
  const F2 mine = LaneFold<K>::run(x, 16, index, count);
  if (count > 0) team_store<C>(&s.part[buffer][index][team_rank<C>() * nw + warp], mine);
  team_sync<C>();
  const int parts = C * nw, per = 32 / parts, sub = lane % parts;  // partials per value, values per warp
  for (int k0 = warp * per; k0 < K; k0 += nw * per) {
    const int k = k0 + lane / parts;
    F2 y = k < K ? s.part[buffer][k][sub] : F2{0.f, 0.f};
    for (int o = parts >> 1; o > 0; o >>= 1)
      y = f2_add(y, F2{__shfl_down_sync(0xffffffffu, y.hi, o), __shfl_down_sync(0xffffffffu, y.lo, o)});
    if (sub == 0 && k < K) s.total[k] = y;
  }
  __syncthreads();
}

// Pose in the frame of an integer anchor.
struct LocalPose {
  int R0, C0;        // integer anchor
  float fr, fc;      // fractional part of the pose relative to the anchor
  float ca, sa;
};

// Level-local pose of a pose in image coordinates, by lanes 0 to 2 of a warp
// (row, column, angle side by side: FP64 latencies once).  The level scale is
// a power of two, so multiplying by its inverse divides exactly.
__device__ __forceinline__ void set_local(LocalPose& l, const double* pose, double crop_row, double crop_col,
                                          double phase, double inv_scale) {
  const int lane = threadIdx.x & 31;
  if (lane < 2) {
    const double v = (pose[lane] - (lane ? crop_col : crop_row) - phase) * inv_scale;
    const double f = floor(v);
    (lane ? l.C0 : l.R0) = int(f);
    (lane ? l.fc : l.fr) = float(v - f);
  } else if (lane == 2) {
    sincosf(float(pose[2]), &l.sa, &l.ca);
  }
}

// True when every sample of the rotated original lies inside the image by a
// margin: the sample positions are affine in (dr, dc), so the corners of the
// offset box bound them (the margin covers FP32 rounding of the per-sample
// expressions).  Inside, the passes drop their per-sample bounds tests.
__device__ __forceinline__ bool samples_inside(const LocalPose& L, const OriginalView& o, float hmin, float hmax,
                                               float wmin, float wmax) {
  float y0 = INFINITY, y1 = -INFINITY, x0 = INFINITY, x1 = -INFINITY;
  const float drs[2] = {o.dr_min, o.dr_max}, dcs[2] = {o.dc_min, o.dc_max};
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float y = L.fr + (L.ca * drs[i] - L.sa * dcs[j]), x = L.fc + (L.sa * drs[i] + L.ca * dcs[j]);
      y0 = fminf(y0, y);
      y1 = fmaxf(y1, y);
      x0 = fminf(x0, x);
      x1 = fmaxf(x1, x);
    }
  const float m = 1e-2f;
  return y0 >= hmin + m && x0 >= wmin + m && y1 <= hmax - 1.f - m && x1 <= wmax - 1.f - m;
}

__device__ __forceinline__ float bilinear_at(const ImageView& img, int r, int c, float fy, float fx, int r1, int c1) {
  const float* v = img.v;
  return (1 - fy) * ((1 - fx) * __ldg(v + size_t(r) * img.w + c) + fx * __ldg(v + size_t(r) * img.w + c1)) +
         fy * ((1 - fx) * __ldg(v + size_t(r1) * img.w + c) + fx * __ldg(v + size_t(r1) * img.w + c1));
}

// Integer part (towards minus infinity) and fraction of |v| < 2^22, without
// the conversion unit: v + 1.5 * 2^23 rounded down is floor(v) + 1.5 * 2^23.
__device__ __forceinline__ int split_floor(float v, float& frac) {
  const float t = __fadd_rd(v, 12582912.f);
  frac = v - __fsub_rn(t, 12582912.f);
  return __float_as_int(t) - 0x4b400000;
}

// The four values of the bilinear cell at (x, y), which lies inside: loaded
// from the quads (integers of 8 or 16 bits) or the level (Bits 0), and put
// into floats when they are used (an integer under the exponent of 2^23).
struct Cell {
  float a, b, d, e;
};
__device__ __forceinline__ float quad_value(uint32_t q, uint32_t sel) {
  return __uint_as_float(__byte_perm(q, 0x4b000000u, sel)) - 8388608.f;
}
template <int Bits> struct RawCell;
template <> struct RawCell<8> {
  uint32_t q = 0;
  __device__ __forceinline__ void load(const ImageView& img, int x, int y) {
    q = __ldg(img.quads + quad_at<8>(x, y, img.tiles));
  }
  __device__ __forceinline__ Cell cell() const {
    return Cell{quad_value(q, 0x7440), quad_value(q, 0x7441), quad_value(q, 0x7442), quad_value(q, 0x7443)};
  }
};
template <> struct RawCell<16> {
  uint2 q = {0, 0};
  __device__ __forceinline__ void load(const ImageView& img, int x, int y) {
    q = __ldg(reinterpret_cast<const uint2*>(img.quads) + quad_at<16>(x, y, img.tiles));
  }
  __device__ __forceinline__ Cell cell() const {
    return Cell{quad_value(q.x, 0x7410), quad_value(q.x, 0x7432), quad_value(q.y, 0x7410), quad_value(q.y, 0x7432)};
  }
};
template <> struct RawCell<0> {
  Cell c = {0.f, 0.f, 0.f, 0.f};
  __device__ __forceinline__ void load(const ImageView& img, int x, int y) {
    const float* v = img.v + (size_t(y) * img.w + x);
    c = Cell{__ldg(v), __ldg(v + 1), __ldg(v + img.w), __ldg(v + img.w + 1)};
  }
  __device__ __forceinline__ Cell cell() const { return c; }
};

// The arithmetic of a sample with its fused operations spelled out, so that a
// pass rounds alike whatever the code around it.
// a b - c d and a b + c d: the first product is the fused one.
__device__ __forceinline__ float fms2(float a, float b, float c, float d) { return __fmaf_rn(a, b, -__fmul_rn(c, d)); }
__device__ __forceinline__ float fma2(float a, float b, float c, float d) { return __fmaf_rn(a, b, __fmul_rn(c, d)); }
// (1 - f) a + f b
__device__ __forceinline__ float mix(float f, float a, float b) { return fma2(__fsub_rn(1.f, f), a, f, b); }
__device__ __forceinline__ float cell_value(const Cell& v, float fy, float fx) {
  return mix(fy, mix(fx, v.a, v.b), mix(fx, v.d, v.e));
}

// FP32 score from pair totals of sum q, sum q^2, sum w q.
__device__ __forceinline__ float pair_score(F2 sum, F2 sq, F2 dot, int n, int absolute, bool* ok) {
  const F2 var = f2_sub(sq, f2_div(f2_mul(sum, sum), f2(float(n))));
  const float v = f2_val(var);
  *ok = v > 0;
  if (!*ok) return -INFINITY;
  float s = fminf(1.f, fmaxf(-1.f, f2_val(dot) / sqrtf(v)));
  return absolute ? fabsf(s) : s;
}

// Sums of the samples of a pose whose cells all lie inside: sum q, sum q^2,
// sum w q.  Six samples per step, all loads issued before the arithmetic (full
// circle 0.293 ms, 4096^2 uint16 1.12; four 0.309 and 1.48, eight with ten blocks
// per SM 0.297 and 1.11); each thread adds its samples in order first, first +
// stride, ...  The samples past the last whole step go one by one: only cells of
// real samples may be loaded, since the samples' box is what was tested and the
// model origin of a masked template may lie outside it on a coarser level.
constexpr int kScoreUnroll = 6;
constexpr int kTeamUnroll = 8;  // passes of a cluster: more registers per thread
template <int Bits> struct InsideSample {
  float w, fy, fx;
  RawCell<Bits> raw;
  __device__ __forceinline__ void load(const ImageView& img, const LocalPose& L, const float4& p) {
    const float y = __fadd_rn(L.fr, fms2(L.ca, p.x, L.sa, p.y));
    const float x = __fadd_rn(L.fc, fma2(L.ca, p.y, L.sa, p.x));
    const int iy = split_floor(y, fy), ix = split_floor(x, fx);
    w = p.z;
    raw.load(img, L.C0 + ix, L.R0 + iy);
  }
  __device__ __forceinline__ void add(float offset, float (&acc)[4]) const {
    const float q = __fsub_rn(cell_value(raw.cell(), fy, fx), offset);
    acc[0] += q;
    acc[1] = fmaf(q, q, acc[1]);
    acc[2] = fmaf(w, q, acc[2]);
  }
};
template <int Bits, int Unroll>
__device__ __forceinline__ void inside_sums(const ImageView& img, const OriginalView& orig, const LocalPose& L,
                                            float offset, int first, int stride, float (&acc)[4]) {
  int s = first;
  for (; s + (Unroll - 1) * stride < orig.n; s += Unroll * stride) {
    float4 p[Unroll];
    InsideSample<Bits> at[Unroll];
#pragma unroll
    for (int u = 0; u < Unroll; ++u) p[u] = __ldg(orig.dcw + s + u * stride);
#pragma unroll
    for (int u = 0; u < Unroll; ++u) at[u].load(img, L, p[u]);
#pragma unroll
    for (int u = 0; u < Unroll; ++u) at[u].add(offset, acc);
  }
  for (; s < orig.n; s += stride) {
    InsideSample<Bits> at;
    at.load(img, L, __ldg(orig.dcw + s));
    at.add(offset, acc);
  }
}

// continuous() of src/ncc_matching/matcher.cpp:144-156 at a level-local pose;
// every thread of the block calls it and gets the score.
template <int Bits, int C = 1>
__device__ __forceinline__ double continuous_pass(const ImageView& img, const OriginalView& orig, const LocalPose& lp,
                                                  int absolute, BlockTotals<4>& tot, int buffer = 0) {
  const LocalPose L = lp;
  const float hmax = float(img.h - 1 - L.R0), wmax = float(img.w - 1 - L.C0);
  const float hmin = float(-L.R0), wmin = float(-L.C0);
  float offset = 0.f;
  {
    const float dr = orig.dr[0], dc = orig.dc[0];
    const float y = L.fr + (L.ca * dr - L.sa * dc), x = L.fc + (L.sa * dr + L.ca * dc);
    if (y >= hmin && x >= wmin && y <= hmax && x <= wmax) {
      const float fy0 = floorf(y), fx0 = floorf(x);
      const int r = L.R0 + int(fy0), c = L.C0 + int(fx0);
      offset = bilinear_at(img, r, c, y - fy0, x - fx0, min(r + 1, img.h - 1), min(c + 1, img.w - 1));
    }
  }
  float acc[4] = {0.f, 0.f, 0.f, 0.f};  // sum q, sum q^2, sum w q, out-of-image flag
  if (samples_inside(L, orig, hmin, hmax, wmin, wmax)) {
    inside_sums<Bits, C == 1 ? kScoreUnroll : kTeamUnroll>(img, orig, L, offset, team_thread<C>(), team_size<C>(), acc);
  } else
  for (int s = team_thread<C>(); s < orig.n; s += team_size<C>()) {
    const float dr = __ldg(orig.dr + s), dc = __ldg(orig.dc + s), w = __ldg(orig.w + s);
    const float y = L.fr + (L.ca * dr - L.sa * dc), x = L.fc + (L.sa * dr + L.ca * dc);
    if (!(y >= hmin && x >= wmin && y <= hmax && x <= wmax)) {
      acc[3] = 1.f;
      continue;
    }
    const float fy0 = floorf(y), fx0 = floorf(x);
    const int r = L.R0 + int(fy0), c = L.C0 + int(fx0);
    const float q = bilinear_at(img, r, c, y - fy0, x - fx0, min(r + 1, img.h - 1), min(c + 1, img.w - 1)) - offset;
    acc[0] += q;
    acc[1] = fmaf(q, q, acc[1]);
    acc[2] = fmaf(w, q, acc[2]);
  }
  block_total<C>(acc, tot, buffer);
  bool ok = false;
  const float sc = tot.total[3].hi > 0 ? -INFINITY
                                       : pair_score(tot.total[0], tot.total[1], tot.total[2], orig.n, absolute, &ok);
  return ok ? double(sc) : -INFINITY;
}

// Full-resolution score of every candidate.  Bound by the latency of the
// gathers and the instructions around them (some 55 per 32 samples, one
// gather).  4096^2 uint16 with a 256^2 template 3.17 -> 1.12 ms, 1024x1280
// full circle with 48^2 0.52 -> 0.29 ms, 2048^2 uint8 0.172 -> 0.163 ms.
template <int Bits> __global__ void __launch_bounds__(128, 12) score_kernel(ScoreArgs a) {
  __shared__ BlockTotals<4> tot;
  __shared__ LocalPose lp;
  const int live = live_count(a.state, a.slot);
  // candidates strided over a bounded grid: a block per possible candidate
  // costs more than a short list's work when the budget is large
  for (int i = blockIdx.x; i < live; i += gridDim.x) {
    const Cand& c = a.cand[i];
    if (!isfinite(c.score)) continue;
    if (threadIdx.x < 32) set_local(lp, &c.row, a.crop_row, a.crop_col, a.phase, a.inv_scale);
    __syncthreads();
    const double score = continuous_pass<Bits>(a.img, a.orig, lp, a.absolute, tot);
    if (threadIdx.x == 0) a.cand[i].score = score;
  }
}

// ------------------------------------------------------------- NCC adjoint
// Scale degree of freedom (no counterpart in the rigid reference).  Sample i
// of the original (offsets dr, dc from the model origin, weight w) lands at
//   y = row + s (ca dr - sa dc),  x = col + s (sa dr + ca dc),
// q_i is the bilinear image value there, and
//   NCC = D / sqrt(E),  D = sum w q - (sum q / n) sum w,  E = sum q^2 - (sum q)^2 / n
// (continuous(), src/ncc_matching/matcher.cpp:121-157, with the scale).  With
// the bilinear cell gradient (gy, gx), dq/dp = gy dy/dp + gx dx/dp for p in
// (row, col, angle, scale), and
//   dNCC = dD / sqrt(E) - D dE / (2 E^1.5),
//   dD = sum w dq - (sum dq / n) sum w,  dE = 2 sum q dq - 2 (sum q)(sum dq) / n.
// Per-thread sums in FP32 (q centred by the first sample, which changes
// neither NCC nor its gradient), block totals as FP32 pairs, the final
// algebra in FP64, a parameter or matrix entry per lane of one warp.  The
// samples come straight from the caller's pixels (no float copy of the whole
// image for a few windows of it).
constexpr int kAdjointThreads = 256;

struct SimLocal {
  int R0, C0;              // integer anchor
  float fr, fc, ca, sa, sc;
  float offset;            // value at the first sample (0 outside)
};

// Pixel (r, c) of the search image as float: an integer of at most 16 bits
// under the exponent of 2^23 (the conversion unit is slower).
template <class T> __device__ __forceinline__ float pixel(const T* __restrict__ v, size_t at) {
  return __uint_as_float(0x4b000000u | uint32_t(__ldg(v + at))) - 8388608.f;
}

// Local pose of a similarity pose (warp 0).
template <class T>
__device__ __forceinline__ void set_sim(SimLocal& l, const PixelView& img, const OriginalView& orig,
                                        const double* pose) {
  const int lane = threadIdx.x;
  if (lane < 2) {
    const double p = pose[lane], f = floor(p);
    (lane ? l.C0 : l.R0) = int(f);
    (lane ? l.fc : l.fr) = float(p - f);
  } else if (lane == 2) {
    double sd, cd;
    sincos(pose[2], &sd, &cd);
    l.ca = float(cd);
    l.sa = float(sd);
  } else if (lane == 3) {
    l.sc = float(pose[3]);
  }
  __syncwarp();
  if (lane == 0) {
    const T* v = static_cast<const T*>(img.v);
    const float dr = orig.dr[0], dc = orig.dc[0];
    const float u = fms2(l.ca, dr, l.sa, dc);
    const float w = fma2(l.sa, dr, l.ca, dc);
    const float y = __fmaf_rn(l.sc, u, l.fr), x = __fmaf_rn(l.sc, w, l.fc);
    float off = 0.f;
    if (y >= float(-l.R0) && x >= float(-l.C0) && y <= float(img.h - 1 - l.R0) && x <= float(img.w - 1 - l.C0)) {
      const int iy = __float2int_rd(y), ix = __float2int_rd(x), r = l.R0 + iy, c = l.C0 + ix;
      const float fy = y - float(iy), fx = x - float(ix);
      const int r1 = min(r + 1, img.h - 1), c1 = min(c + 1, img.w - 1);
      const Cell q{pixel(v, size_t(r) * img.pitch + c), pixel(v, size_t(r) * img.pitch + c1),
                   pixel(v, size_t(r1) * img.pitch + c), pixel(v, size_t(r1) * img.pitch + c1)};
      off = cell_value(q, fy, fx);
    }
    l.offset = off;
  }
}

// One sample of a similarity pose: its value and derivatives.
struct SimSample {
  float q, g[4];
};

// Calls use(weight, inside, sample) for this thread's samples in order; four
// samples' loads are issued before their arithmetic.
template <class T, int C = 1, class Use>
__device__ __forceinline__ void sim_samples(const PixelView& img, const OriginalView& orig, const SimLocal& l, Use use) {
  constexpr int U = C == 1 ? 4 : kTeamUnroll;
  const T* __restrict__ v = static_cast<const T*>(img.v);
  const float hmin = float(-l.R0), wmin = float(-l.C0), hmax = float(img.h - 1 - l.R0), wmax = float(img.w - 1 - l.C0);
  const int stride = team_size<C>();
  for (int s0 = team_thread<C>(); s0 < orig.n; s0 += U * stride) {
    float4 p[U];
    float fy[U], fx[U], uu[U], vv[U];
    uint32_t raw[U][4];
    bool in[U];
#pragma unroll
    for (int k = 0; k < U; ++k)
      p[k] = s0 + k * stride < orig.n ? __ldg(orig.dcw + s0 + k * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < U; ++k) {
      uu[k] = fms2(l.ca, p[k].x, l.sa, p[k].y);
      vv[k] = fma2(l.sa, p[k].x, l.ca, p[k].y);
      const float y = __fmaf_rn(l.sc, uu[k], l.fr), x = __fmaf_rn(l.sc, vv[k], l.fc);
      in[k] = y >= hmin && x >= wmin && y <= hmax && x <= wmax;
      const int iy = __float2int_rd(y), ix = __float2int_rd(x), r = l.R0 + iy, c = l.C0 + ix;
      fy[k] = y - float(iy);
      fx[k] = x - float(ix);
      raw[k][0] = raw[k][1] = raw[k][2] = raw[k][3] = 0;
      if (in[k] && s0 + k * stride < orig.n) {
        const T* row = v + size_t(r) * img.pitch;
        const T* next = r + 1 < img.h ? row + img.pitch : row;
        const int c1 = min(c + 1, img.w - 1);
        raw[k][0] = __ldg(row + c);
        raw[k][1] = __ldg(row + c1);
        raw[k][2] = __ldg(next + c);
        raw[k][3] = __ldg(next + c1);
      }
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (s0 + k * stride >= orig.n) break;
      float w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = __uint_as_float(0x4b000000u | raw[k][j]) - 8388608.f;
      SimSample s;
      s.q = __fsub_rn(cell_value(Cell{w[0], w[1], w[2], w[3]}, fy[k], fx[k]), l.offset);
      const float gy = mix(fx[k], __fsub_rn(w[2], w[0]), __fsub_rn(w[3], w[1]));
      const float gx = mix(fy[k], __fsub_rn(w[1], w[0]), __fsub_rn(w[3], w[2]));
      // dy/dp, dx/dp: row (1, 0), col (0, 1), angle (-s v, s u), scale (u, v)
      s.g[0] = gy;
      s.g[1] = gx;
      s.g[2] = __fmul_rn(l.sc, fms2(gx, uu[k], gy, vv[k]));
      s.g[3] = fma2(gy, uu[k], gx, vv[k]);
      use(p[k].z, in[k], s);
    }
  }
}

__device__ __forceinline__ double pair_double(const F2& x) { return double(x.hi) + double(x.lo); }

// Bound by the latency of the gathers.  256 poses of a 128^2 template in a
// 5120^2 image: 184 -> 98 us a call, the copy of the image to float (131 MB)
// and one FP64 sincos per warp gone.
template <class T> __global__ void __launch_bounds__(kAdjointThreads) adjoint_kernel(AdjointArgs a) {
  __shared__ BlockTotals<17> tot;
  __shared__ SimLocal loc;
  const int k = blockIdx.x;
  const OriginalView orig = a.orig;
  if (threadIdx.x < 32) set_sim<T>(loc, a.img, orig, a.poses + 4 * k);
  __syncthreads();
  const SimLocal l = loc;
  // 0 sum q, 1 sum q^2, 2 sum w q, 3..6 sum dq, 7..10 sum q dq, 11..14 sum w dq, 15 sum w, 16 outside
  float acc[17];
#pragma unroll
  for (int j = 0; j < 17; ++j) acc[j] = 0.f;
  sim_samples<T>(a.img, orig, l, [&](float w, bool in, const SimSample& s) {
    acc[15] += w;
    if (!in) {
      acc[16] = 1.f;
      return;
    }
    acc[0] += s.q;
    acc[1] = fmaf(s.q, s.q, acc[1]);
    acc[2] = fmaf(w, s.q, acc[2]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc[3 + j] += s.g[j];
      acc[7 + j] = fmaf(s.q, s.g[j], acc[7 + j]);
      acc[11 + j] = fmaf(w, s.g[j], acc[11 + j]);
    }
  });
  block_total(acc, tot);
  if (threadIdx.x < 4) {
    const F2* t = tot.total;
    const int j = threadIdx.x;
    const double n = double(orig.n);
    const double sq = pair_double(t[0]), sqq = pair_double(t[1]), swq = pair_double(t[2]), sw = pair_double(t[15]);
    const double D = swq - sq / n * sw, E = sqq - sq * sq / n;
    if (t[16].hi > 0 || !(E > 0)) {
      if (j == 0) a.score[k] = -INFINITY;
      a.grad[4 * k + j] = 0;
      return;
    }
    const double rs = 1 / sqrt(E);
    double ncc = D * rs;
    const double sign = a.absolute && ncc < 0 ? -1. : 1.;
    if (j == 0) a.score[k] = sign * ncc;
    const double sdq = pair_double(t[3 + j]), sqdq = pair_double(t[7 + j]), swdq = pair_double(t[11 + j]);
    const double dD = swdq - sdq / n * sw, dE = 2 * (sqdq - sq * sdq / n);
    a.grad[4 * k + j] = sign * (dD * rs - D * dE * .5 * rs * rs * rs);
  }
}

// Similarity pass of the 4-parameter refinement: block totals of
// 0 q, 1 q^2, 2 w q, 3..6 g, 7..10 q g, 11..14 w g, 15..24 g_i g_j (i <= j),
// 25 w, 26 outside, with g = dq / d(row, col, angle, scale).
constexpr int kSimSums = 27;

template <class T, int C>
__device__ __noinline__ void sim_pass(const Refine4Args& a, SimLocal& loc, const double* pose,
                                      BlockTotals<kSimSums>& tot, int buffer) {
  if (threadIdx.x < 32) set_sim<T>(loc, a.img, a.orig, pose);
  __syncthreads();
  const SimLocal l = loc;
  float acc[kSimSums];
#pragma unroll
  for (int j = 0; j < kSimSums; ++j) acc[j] = 0.f;
  sim_samples<T, C>(a.img, a.orig, l, [&](float w, bool in, const SimSample& s) {
    acc[25] += w;
    if (!in) {
      acc[26] = 1.f;
      return;
    }
    acc[0] += s.q;
    acc[1] = fmaf(s.q, s.q, acc[1]);
    acc[2] = fmaf(w, s.q, acc[2]);
    int at = 15;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[3 + i] += s.g[i];
      acc[7 + i] = fmaf(s.q, s.g[i], acc[7 + i]);
      acc[11 + i] = fmaf(w, s.g[i], acc[11 + i]);
#pragma unroll
      for (int j = i; j < 4; ++j, ++at) acc[at] = fmaf(s.g[i], s.g[j], acc[at]);
    }
  });
  block_total<C>(acc, tot, buffer);
}

// The score alone: totals of 0 q, 1 q^2, 2 w q, 3 w, 4 outside.
template <class T, int C>
__device__ __noinline__ double sim_score(const Refine4Args& a, SimLocal& loc, const double* pose, BlockTotals<5>& tot,
                                         int buffer) {
  if (threadIdx.x < 32) set_sim<T>(loc, a.img, a.orig, pose);
  __syncthreads();
  const SimLocal l = loc;
  float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  sim_samples<T, C>(a.img, a.orig, l, [&](float w, bool in, const SimSample& s) {
    acc[3] += w;
    if (!in) {
      acc[4] = 1.f;
      return;
    }
    acc[0] += s.q;
    acc[1] = fmaf(s.q, s.q, acc[1]);
    acc[2] = fmaf(w, s.q, acc[2]);
  });
  block_total<C>(acc, tot, buffer);
  const F2* t = tot.total;
  const double n = double(a.orig.n);
  const double sq = pair_double(t[0]), sqq = pair_double(t[1]), swq = pair_double(t[2]), sw = pair_double(t[3]);
  const double E = sqq - sq * sq / n, D = swq - sq / n * sw;
  if (!(t[4].hi == 0 && E > 0)) return -INFINITY;
  const double ncc = D / sqrt(E);
  return a.absolute ? fabs(ncc) : ncc;
}

// One block per pose.  Each iteration: the normal equations of the NCC in
// the four parameters (Gauss-Newton on the centred, normalised samples, as
// the reference's refinement_step), an FP64 Gauss-Jordan solve with partial
// pivoting (a matrix entry per lane of warp 0), the step clipped to the
// limits, and up to four halvings; a step is taken only when the score
// strictly increases.  Bound by the latency of the passes.  64 poses of a
// 161^2 template in a 3000x4096 image: 2.17 -> 1.56 ms (1.79 with one block per pose).
constexpr int kRefine4Threads = 256;  // of a team of C blocks

template <class T, int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(kRefine4Threads / C)
    refine4_kernel(const __grid_constant__ Refine4Args a) {
  __shared__ BlockTotals<kSimSums> tot;
  __shared__ BlockTotals<5> tot5;
  __shared__ SimLocal loc;
  __shared__ double s_pose[4], s_try[4], s_delta[4], s_score, s_factor;
  __shared__ int s_go;
  const int k = blockIdx.x / C, tid = threadIdx.x;
  int pass = 0;
  if (tid < 4) s_pose[tid] = a.poses[4 * k + tid];
  team_sync<C>();  // every block of the cluster runs and has read the pose
  double score = -INFINITY;
  const double n = double(a.orig.n);
  for (int it = 0; it <= a.iterations; ++it) {
    __syncthreads();
    sim_pass<T, C>(a, loc, s_pose, tot, pass++ & 1);
    if (tid < 32) {
      const F2* t = tot.total;
      const double sq = pair_double(t[0]), sqq = pair_double(t[1]), swq = pair_double(t[2]), sw = pair_double(t[25]);
      const double E = sqq - sq * sq / n, D = swq - sq / n * sw;
      const bool scored = t[26].hi == 0 && E > 0;
      bool go = false;
      double value = -INFINITY;
      if (scored) {
        const double rs = 1 / sqrt(E);
        const double ncc = D * rs, sign = a.absolute && ncc < 0 ? -1. : 1.;
        value = sign * ncc;
        if (it < a.iterations) {
          // lane l < 20: entry (l / 5, l mod 5) of the equations
          const int row = tid / 5, j = tid % 5, i = min(row, 3);
          const double gi = pair_double(t[3 + i]), qi = pair_double(t[7 + i]) - sq / n * gi;
          double e;
          if (j < 4) {
            const double gj = pair_double(t[3 + j]), qj = pair_double(t[7 + j]) - sq / n * gj;
            const int lo = min(i, j), hi = max(i, j);
            const int at = 15 + lo * 4 - lo * (lo - 1) / 2 + (hi - lo);
            e = ((pair_double(t[at]) - gi * gj / n) - qi * qj / E) / E;
          } else {
            e = sign * (pair_double(t[11 + i]) - gi / n * sw) * rs - value * qi / E;
          }
          bool good = true;
          for (int c = 0; c < 4; ++c) {
            int pivot = c;
            double pv = __shfl_sync(0xffffffffu, e, c * 5 + c);
            for (int r = c + 1; r < 4; ++r) {
              const double x = __shfl_sync(0xffffffffu, e, r * 5 + c);
              if (fabs(x) > fabs(pv)) {
                pv = x;
                pivot = r;
              }
            }
            if (fabs(pv) < 1e-14) {
              good = false;
              break;
            }
            const int from = row == c ? pivot * 5 + j : row == pivot ? c * 5 + j : tid;
            e = __shfl_sync(0xffffffffu, e, from);
            const double inv = 1 / pv;
            if (row == c) e *= inv;
            const double prow = __shfl_sync(0xffffffffu, e, c * 5 + j);
            const double f = __shfl_sync(0xffffffffu, e, i * 5 + c);
            if (row != c) e -= f * prow;
          }
          if (good) {
            const double d = __shfl_sync(0xffffffffu, e, (tid & 3) * 5 + 4);
            const double limit = (tid & 3) < 2 ? a.max_shift : (tid & 3) == 2 ? a.max_angle : a.max_scale;
            double f = fmin(1., limit / fmax(1e-20, fabs(d)));
            f = fmin(f, __shfl_xor_sync(0xffffffffu, f, 1));
            f = fmin(f, __shfl_xor_sync(0xffffffffu, f, 2));
            if (tid < 4) s_delta[tid] = d;
            if (tid == 0) s_factor = f;
            go = isfinite(f) && __all_sync(0xffffffffu, isfinite(d));
          }
        }
      }
      if (tid == 0) {
        s_go = go;
        if (scored) s_score = value;
        else s_score = score;
      }
    }
    __syncthreads();
    score = s_score;
    if (!s_go) break;
    bool accepted = false;
    for (int bt = 0; bt < 4 && !accepted; ++bt) {
      if (tid < 4) s_try[tid] = s_pose[tid] + ldexp(s_factor, -bt) * s_delta[tid];
      __syncthreads();
      const double got = sim_score<T, C>(a, loc, s_try, tot5, pass++ & 1);
      if (got > score) {
        accepted = true;
        if (tid < 4) s_pose[tid] = s_try[tid];
      }
      __syncthreads();
    }
    if (!accepted) break;
    if (tid == 0) {
      const double st = s_factor;
      s_go = hypot(st * s_delta[0], st * s_delta[1]) >= 1e-4 || fabs(st * s_delta[2]) >= 1e-5 ||
             fabs(st * s_delta[3]) >= 1e-6;
    }
    __syncthreads();
    if (!s_go) {
      // converged: the score at the final pose
      score = sim_score<T, C>(a, loc, s_pose, tot5, pass++ & 1);
      break;
    }
  }
  __syncthreads();
  if (team_rank<C>() != 0) return;
  if (tid < 4) a.poses[4 * k + tid] = s_pose[tid];
  if (tid == 0) a.score[k] = score;
}

// --------------------------------------------------------------------- sort
// 64-bit keys ordering scores descending (order-preserving bit transform).
__device__ __forceinline__ unsigned long long desc_key(double s) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(s);
  const unsigned long long asc = (b >> 63) ? ~b : (b | 0x8000000000000000ULL);
  return ~asc;
}

// Candidate sort in the reference's order (score descending, then row,
// column, angle; matcher.cpp:824-827; the list index for exact duplicates):
// 256-entry segments are ranked in shared memory, then an entry's place among
// up to 64 sorted lists is its place in its own plus the entries of every
// other list before it (binary search).  One merge covers 16384 candidates,
// two 2^20, three 2^26; every launch reads the live count and returns when
// the list is already sorted.  Bound by the latency of the searches.
constexpr int kSortSeg = 256, kSortFan = 64, kSortLanes = 8;
constexpr unsigned long long kNoScoreKey = 0xfff0000000000000ULL;  // desc_key(-inf)

__device__ __forceinline__ bool sort_before(unsigned long long ka, int ia, unsigned long long kb, int ib,
                                            const Cand* __restrict__ in) {
  if (ka != kb) return ka < kb;
  if (ka >= kNoScoreKey) return ia < ib;  // without a score: the order is not read
  const Cand x = in[ia], y = in[ib];
  if (x.row != y.row) return x.row < y.row;
  if (x.col != y.col) return x.col < y.col;
  if (x.angle != y.angle) return x.angle < y.angle;
  return ia < ib;
}

__device__ RectAux make_rect(const Cand& m, const RectGeom& g);

// Candidate i at its final rank, and the selection's per-candidate state.
__device__ __forceinline__ bool sort_emit(const SortArgs& a, int rank, int i) {
  const Cand c = a.in[i];
  a.out[rank] = c;
  if (a.aux) {
    a.aux[rank] = make_rect(c, a.geom);
    a.refined_flag[rank] = 0;
    a.tested[rank] = 0;
    a.sup[rank] = 0;
  }
  return isfinite(c.score);
}

__global__ void __launch_bounds__(kSortSeg) sort_segments_kernel(SortArgs a) {
  __shared__ __align__(16) unsigned long long s_key[kSortSeg];
  const int n = live_count(a.state, a.slot);
  const int base = blockIdx.x * kSortSeg, t = threadIdx.x, i = base + t;
  if (base >= n) return;
  const unsigned long long key = i < n ? desc_key(a.in[i].score) : ~0ULL;
  s_key[t] = key;
  __syncthreads();
  const int m = min(kSortSeg, n - base);
  int rank = 0;
  bool tie = false;  // another candidate has the same score
#pragma unroll 8
  for (int k = 0; k < m; k += 2) {
    const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(s_key + k);
    rank += int(q.x < key || (q.x == key && k < t)) + int(q.y < key || (q.y == key && k + 1 < t));
    tie |= (q.x == key && k != t) || (q.y == key && k + 1 != t);
  }
  if (tie && i < n && key < kNoScoreKey)
    for (int k = 0; k < m; ++k)
      if (k != t && s_key[k] == key) rank += int(sort_before(key, base + k, key, i, a.in)) - int(k < t);
  bool finite = false;
  if (i < n) {
    if (n > kSortSeg) {
      a.keys[base + rank] = key;
      a.idx[base + rank] = i;
    } else {
      finite = sort_emit(a, rank, i);
    }
  }
  const unsigned scored = __ballot_sync(0xffffffffu, finite);
  if ((t & 31) == 0 && scored) atomicAdd(&a.state->sorted_count, __popc(scored));
}

// Merges groups of kSortFan sorted segments of `seg` entries (eight threads
// per entry share the group's segments).
__global__ void __launch_bounds__(256) sort_merge_kernel(SortArgs a, int seg, const unsigned long long* __restrict__ keys,
                                                         const int32_t* __restrict__ idx, unsigned long long* keys_out,
                                                         int32_t* idx_out) {
  const int n = live_count(a.state, a.slot);
  if (n <= seg) return;
  const int sub = threadIdx.x % kSortLanes;
  const int e = int((blockIdx.x * 256u + threadIdx.x) / kSortLanes);
  bool finite = false;
  const long long span = (long long)seg * kSortFan;
  const int group = int(e / span) * kSortFan, own = e / seg;  // first segment of the group; the entry's segment
  int rank = 0;
  if (e < n) {
    const unsigned long long key = keys[e];
    const int i = idx[e];
    for (int t = group + sub; t < group + kSortFan && (long long)t * seg < n; t += kSortLanes) {
      if (t == own) continue;
      const int first = t * seg;
      int lo = 0, hi = min(seg, n - first);
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (sort_before(keys[first + mid], idx[first + mid], key, i, a.in))
          lo = mid + 1;
        else
          hi = mid;
      }
      rank += lo;
    }
  }
#pragma unroll
  for (int o = 1; o < kSortLanes; o <<= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
  if (e < n && sub == 0) {
    rank += group * seg + (e - own * seg);
    if (n <= span) {
      finite = sort_emit(a, rank, idx[e]);
    } else {
      keys_out[rank] = keys[e];
      idx_out[rank] = idx[e];
    }
  }
  const unsigned m = __ballot_sync(0xffffffffu, finite);
  if ((threadIdx.x & 31) == 0 && m) atomicAdd(&a.state->sorted_count, __popc(m));
}

// ----------------------------------------------------------------- overlap
// Rotated rectangle of a pose: FP32 cos/sin and a conservative FP32 box for
// the cheap disjointness test.  The angle is brought near zero in FP64 (the
// search range may lie anywhere) and what its float drops goes in to first
// order, so cos and sin are within an ulp or two of the FP64 ones.  FP64 sincos
// is left to the exact overlap, which few pairs need.
__device__ RectAux make_rect(const Cand& m, const RectGeom& g) {
  RectAux r;
  const double angle = dadd(dsub(m.angle, g.angle_from), g.angle_to);
  const float hi = float(angle), lo = float(dsub(angle, double(hi)));
  float sh, ch;
  sincosf(hi, &sh, &ch);
  r.sa = __fmaf_rn(ch, lo, sh);
  r.ca = __fmaf_rn(-sh, lo, ch);
  float x0 = INFINITY, y0 = INFINITY, x1 = -INFINITY, y1 = -INFINITY;
  const double xs[2] = {g.left, g.right}, ys[2] = {g.top, g.bottom};
  for (double x : xs)
    for (double y : ys) {
      const float px = float(m.col) + r.ca * float(x) + r.sa * float(y);
      const float py = float(m.row) - r.sa * float(x) + r.ca * float(y);
      x0 = fminf(x0, px);
      x1 = fmaxf(x1, px);
      y0 = fminf(y0, py);
      y1 = fmaxf(y1, py);
    }
  const float pad = 1e-3f * (1.f + fabsf(float(m.row)) + fabsf(float(m.col)));
  r.x0 = x0 - pad;
  r.y0 = y0 - pad;
  r.x1 = x1 + pad;
  r.y1 = y1 + pad;
  return r;
}

__device__ __forceinline__ bool boxes_disjoint(const RectAux& a, const RectAux& b) {
  return a.x1 < b.x0 || b.x1 < a.x0 || a.y1 < b.y0 || b.y1 < a.y0;
}

struct Pt {
  double x, y;
};

// Intersection area of two rotated template rectangles over the template
// area (src/ncc_matching/matcher.cpp:252-277); a is the candidate, b the
// accepted match.  Corners are relative to a's centre.
__device__ double overlap_ratio(const Cand& a, const RectAux& ra, const Cand& b, const RectAux& rb, const RectGeom& g) {
  if (boxes_disjoint(ra, rb)) return 0.;
  double aca, asa, bca, bsa;
  sincos(a.angle, &asa, &aca);
  sincos(b.angle, &bsa, &bca);
  const Pt in[4] = {{g.left, g.top}, {g.right, g.top}, {g.right, g.bottom}, {g.left, g.bottom}};
  Pt clip[4], poly[16], next[16];
  for (int i = 0; i < 4; ++i) {
    clip[i].x = dadd(dadd(dsub(b.col, a.col), dmul(bca, in[i].x)), dmul(bsa, in[i].y));
    clip[i].y = dadd(dsub(dsub(b.row, a.row), dmul(bsa, in[i].x)), dmul(bca, in[i].y));
    poly[i].x = dadd(dmul(aca, in[i].x), dmul(asa, in[i].y));
    poly[i].y = dadd(-dmul(asa, in[i].x), dmul(aca, in[i].y));
  }
  int count = 4;
  for (int edge = 0; edge < 4 && count; ++edge) {
    const Pt p = clip[edge], q = clip[(edge + 1) & 3];
    int out = 0;
    for (int i = 0; i < count; ++i) {
      const Pt u = poly[i], v = poly[(i + 1) % count];
      const double du = dsub(dmul(dsub(q.x, p.x), dsub(u.y, p.y)), dmul(dsub(q.y, p.y), dsub(u.x, p.x)));
      const double dv = dsub(dmul(dsub(q.x, p.x), dsub(v.y, p.y)), dmul(dsub(q.y, p.y), dsub(v.x, p.x)));
      if (du >= 0 && out < 16) next[out++] = u;
      if ((du >= 0) != (dv >= 0) && out < 16) {
        const double t = du / dsub(du, dv);
        next[out++] = Pt{dadd(u.x, dmul(t, dsub(v.x, u.x))), dadd(u.y, dmul(t, dsub(v.y, u.y)))};
      }
    }
    for (int i = 0; i < out; ++i) poly[i] = next[i];
    count = out;
  }
  double area = 0;
  for (int i = 0; i < count; ++i)
    area = dadd(area, dsub(dmul(poly[i].x, poly[(i + 1) % count].y), dmul(poly[(i + 1) % count].x, poly[i].y)));
  return fabs(area) * .5 / g.area;
}

// The same clip in FP32 (corners relative to a's centre are small numbers):
// within 1e-3 of the true ratio, used to decide clear cases without FP64.
__device__ float overlap_ratio32(const Cand& a, const RectAux& ra, const Cand& b, const RectAux& rb, const RectGeom& g) {
  if (boxes_disjoint(ra, rb)) return 0.f;
  const float L = float(g.left), R = float(g.right), T = float(g.top), B = float(g.bottom);
  const float inx[4] = {L, R, R, L}, iny[4] = {T, T, B, B};
  const float dx = float(b.col - a.col), dy = float(b.row - a.row);
  const float bca = rb.ca, bsa = rb.sa, aca = ra.ca, asa = ra.sa;
  float cx[4], cy[4], px[16], py[16], nx[16], ny[16];
  for (int i = 0; i < 4; ++i) {
    cx[i] = dx + bca * inx[i] + bsa * iny[i];
    cy[i] = dy - bsa * inx[i] + bca * iny[i];
    px[i] = aca * inx[i] + asa * iny[i];
    py[i] = -asa * inx[i] + aca * iny[i];
  }
  int count = 4;
  for (int edge = 0; edge < 4 && count; ++edge) {
    const float p0x = cx[edge], p0y = cy[edge], qx = cx[(edge + 1) & 3], qy = cy[(edge + 1) & 3];
    int out = 0;
    for (int i = 0; i < count; ++i) {
      const int j = (i + 1) % count;
      const float du = (qx - p0x) * (py[i] - p0y) - (qy - p0y) * (px[i] - p0x);
      const float dv = (qx - p0x) * (py[j] - p0y) - (qy - p0y) * (px[j] - p0x);
      if (du >= 0 && out < 16) {
        nx[out] = px[i];
        ny[out++] = py[i];
      }
      if ((du >= 0) != (dv >= 0) && out < 16) {
        const float t = du / (du - dv);
        nx[out] = px[i] + t * (px[j] - px[i]);
        ny[out++] = py[i] + t * (py[j] - py[i]);
      }
    }
    for (int i = 0; i < out; ++i) {
      px[i] = nx[i];
      py[i] = ny[i];
    }
    count = out;
  }
  float area = 0;
  for (int i = 0; i < count; ++i) area += px[i] * py[(i + 1) % count] - px[(i + 1) % count] * py[i];
  return fabsf(area) * .5f / float(g.area);
}

// overlap(a, b) > thr, deciding in FP32 when the FP32 ratio is clearly on
// one side and in FP64 otherwise.
__device__ __forceinline__ bool overlaps(const Cand& a, const RectAux& ra, const Cand& b, const RectAux& rb,
                                         const RectGeom& g, double thr) {
  if (boxes_disjoint(ra, rb)) return 0. > thr;
  const float r32 = overlap_ratio32(a, ra, b, rb, g);
  if (double(r32) > thr + 1e-3) return true;
  if (double(r32) < thr - 1e-3) return false;
  return overlap_ratio(a, ra, b, rb, g) > thr;
}

// Greedy MaxOverlap selection over the sorted candidates
// (src/ncc_matching/matcher.cpp:1063-1076).  A window of candidates is tested
// against the accepted matches in parallel; the first unsuppressed one is
// then accepted or rejected from its refinement result.  When it has none,
// the kernel queues it and the next unsuppressed, unrefined candidates that
// do not overlap a higher-ranked queued one, and returns with need = 1.
constexpr int kSelectThreads = 1024;

__global__ void __launch_bounds__(kSelectThreads) select_kernel(SelectArgs a) {
  __shared__ int s_next, s_acc, s_first, s_hit;
  __shared__ unsigned char s_sup[kSelectThreads];
  __shared__ int s_batch[64];
  QueryState* st = a.state;
  if (st->done) return;
  const int total = st->sorted_count;
  const double thr = a.max_overlap + 1e-12;
  if (threadIdx.x == 0) {
    s_next = st->next;
    s_acc = st->accepted;
    st->need = 0;
  }
  __syncthreads();
  while (true) {
    const int base = s_next, acc = s_acc;
    if (base >= total || (a.num_matches && acc >= a.num_matches)) break;
    // suppression of the window by the accepted matches; each candidate is
    // tested only against matches accepted since its last test
    const int wcount = min(kSelectThreads, total - base);
    const int t = threadIdx.x;
    bool sup = true;
    if (t < wcount) {
      const int idx = base + t;
      sup = a.sup[idx] != 0;
      const int from = a.tested[idx];
      if (!sup && from < acc) {
        const Cand c = a.sorted[idx];
        const RectAux rc = a.aux[idx];
        for (int j = from; j < acc && !sup; ++j)
          if (overlaps(c, rc, a.accepted[j], a.accepted_aux[j], a.geom, thr)) sup = true;
        a.tested[idx] = acc;
        if (sup) a.sup[idx] = 1;
      }
    }
    s_sup[t] = sup ? 1 : 0;
    if (t == 0) s_first = INT32_MAX;
    __syncthreads();
    if (!sup) atomicMin(&s_first, t);
    __syncthreads();
    const int first = s_first;
    if (first == INT32_MAX) {
      __syncthreads();
      if (threadIdx.x == 0) s_next = base + wcount;
      __syncthreads();
      continue;
    }
    const int i = base + first;
    if (a.refined_flag[i] != 2) {
      // queue i and the next unsuppressed, unrefined candidates of the window
      // that no higher-ranked queued candidate overlaps (speculation only)
      if (threadIdx.x == 0) {
        int nb = 0;
        s_batch[nb++] = i;
        for (int k = first + 1; k < wcount && nb < a.batch_limit && nb < 64; ++k) {
          const int idx = base + k;
          if (s_sup[k] || a.refined_flag[idx] == 2) continue;
          const RectAux rk = a.aux[idx];
          bool dup = false;
          for (int q = 0; q < nb && !dup; ++q) {
            const RectAux rq = a.aux[s_batch[q]];
            // boxes overlapping by more than half of the smaller box
            const float ix = fminf(rk.x1, rq.x1) - fmaxf(rk.x0, rq.x0), iy = fminf(rk.y1, rq.y1) - fmaxf(rk.y0, rq.y0);
            if (ix > 0 && iy > 0) {
              const float ak = (rk.x1 - rk.x0) * (rk.y1 - rk.y0), aq = (rq.x1 - rq.x0) * (rq.y1 - rq.y0);
              if (ix * iy > 0.5f * fminf(ak, aq)) dup = true;
            }
          }
          if (!dup) s_batch[nb++] = idx;
        }
        for (int q = 0; q < nb; ++q) {
          a.batch[q] = s_batch[q];
          a.refined_flag[s_batch[q]] = 1;
        }
        st->batch_count = nb;
        st->need = 1;
        st->next = i;
        st->accepted = acc;
      }
      return;
    }
    const Refined r = a.refined[i];
    const bool keep = r.ok != 0;
    Cand rc;
    rc.row = r.row;
    rc.col = r.col;
    rc.angle = r.angle;
    rc.score = r.score;
    rc.patch = -1;
    rc.pad = 0;
    // re-check against the accepted matches with the refined pose
    if (threadIdx.x == 0) s_hit = 0;
    __syncthreads();
    if (keep)
      for (int j = threadIdx.x; j < acc; j += kSelectThreads)
        if (overlaps(rc, r.rect, a.accepted[j], a.accepted_aux[j], a.geom, thr)) s_hit = 1;
    __syncthreads();
    if (threadIdx.x == 0) {
      if (keep && !s_hit) {
        a.accepted[acc] = rc;
        a.accepted_aux[acc] = r.rect;
        s_acc = acc + 1;
      }
      s_next = i + 1;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    st->next = s_next;
    st->accepted = s_acc;
    // final order: score desc, row, column, angle (src/ncc_matching/matcher.cpp:1072-1075)
    const int n = s_acc;
    for (int x = 1; x < n; ++x) {
      const Cand v = a.accepted[x];
      int y = x - 1;
      while (y >= 0) {
        const Cand u = a.accepted[y];
        const bool after = u.score != v.score ? u.score < v.score
                           : u.row != v.row   ? u.row > v.row
                           : u.col != v.col   ? u.col > v.col
                                              : u.angle > v.angle;
        if (!after) break;
        a.accepted[y + 1] = u;
        --y;
      }
      a.accepted[y + 1] = v;
    }
    st->done = 1;
  }
}

// --------------------------------------------------------------- refinement
// A candidate is refined by 512 threads: one block, or a cluster of four
// blocks whose SMs share the samples and which each follow the fit.
constexpr int kRefineThreads = 512;

// State of a block's fit.  Poses are {row, column, angle}; scalar FP64 work
// is done by warp 0, a pose component per lane, and read by all threads
// after a barrier.
struct FitShared {
  LocalPose lp;        // pose of the next pass
  BlockTotals<4> tot4;
  BlockTotals<19> tot19;
  double pose[3], trial[3], seed[3], best[3];
  double delta[3], gn_delta[3], next_delta[3];
  double gscore, factor;  // score seen by the last Gauss-Newton pass (-inf if none); step factor
  int buffer;             // of the next block total
  int ok, flag;           // result of the last Gauss-Newton pass; a decision of warp 0
  F2 wbest[16];           // recovery search: {score, order} by warp
  double best_score;
};

// refinement_step of src/ncc_matching/matcher.cpp:170-240 at the pose in
// f.lp: bilinear samples with the analytic gradient, FP32 per thread, pair
// totals, normal equations in pair arithmetic and the Gauss-Jordan solve in
// FP64, a matrix entry per lane of warp 0.  Afterwards f.ok / f.gscore /
// f.gn_delta hold the result, for every thread.  Kept out of line: its code
// runs once per pass and is called from several places, and copies of it
// would miss the instruction cache.
template <int Bits, int C>
__device__ __noinline__ void gn_pass(const RefineArgs& a, FitShared& f, bool use_minimum, double minimum) {
  const ImageView& img = a.img;
  const OriginalView& orig = a.orig;
  const LocalPose L = f.lp;
  const float hmax = float(img.h - 1 - L.R0), wmax = float(img.w - 1 - L.C0);
  const float hmin = float(-L.R0), wmin = float(-L.C0);
  float offset = 0.f;
  {
    const float dr = orig.dr[0], dc = orig.dc[0];
    const float y = L.fr + (L.ca * dr - L.sa * dc), x = L.fc + (L.sa * dr + L.ca * dc);
    if (y >= hmin && x >= wmin && y < hmax && x < wmax) {
      const float fy0 = floorf(y), fx0 = floorf(x);
      const int r = L.R0 + int(fy0), c = L.C0 + int(fx0);
      offset = bilinear_at(img, r, c, y - fy0, x - fx0, r + 1, c + 1);
    }
  }
  // 0 sum q, 1 sum q^2, 2 sum wq, 3..5 gs, 6..8 qg, 9..11 wg, 12..17 gg (00,10,11,20,21,22), 18 out
  float acc[19];
#pragma unroll
  for (int k = 0; k < 19; ++k) acc[k] = 0.f;
  const bool inside = samples_inside(L, orig, hmin, hmax, wmin, wmax);
  const int stride = team_size<C>();
  // U samples per step, all loads issued before the arithmetic; each
  // thread still adds its samples in order s, s + stride, ...
  constexpr int U = C == 1 ? 4 : kTeamUnroll;
  for (int s0 = team_thread<C>(); s0 < orig.n; s0 += U * stride) {
    float4 p[U];
    float fy[U], fx[U];
    RawCell<Bits> raw[U];
    bool in[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int s = s0 + u * stride;
      in[u] = s < orig.n;
      p[u] = in[u] ? __ldg(orig.dcw + s) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float y = __fadd_rn(L.fr, fms2(L.ca, p[u].x, L.sa, p[u].y));
      const float x = __fadd_rn(L.fc, fma2(L.sa, p[u].x, L.ca, p[u].y));
      if (!inside && in[u] && !(y >= hmin && x >= wmin && y < hmax && x < wmax)) {
        acc[18] = 1.f;
        in[u] = false;
      }
      const int iy = split_floor(y, fy[u]), ix = split_floor(x, fx[u]);
      if (in[u]) raw[u].load(img, L.C0 + ix, L.R0 + iy);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!in[u]) continue;
      const Cell v = raw[u].cell();
      const float dr = p[u].x, dc = p[u].y, wt = p[u].z;
      const float q = __fsub_rn(cell_value(v, fy[u], fx[u]), offset);
      const float gy = mix(fx[u], __fsub_rn(v.d, v.a), __fsub_rn(v.e, v.b));
      const float gx = mix(fy[u], __fsub_rn(v.b, v.a), __fsub_rn(v.e, v.d));
      const float g2 = fma2(gy, fms2(-L.sa, dr, L.ca, dc), gx, fms2(L.ca, dr, L.sa, dc));
      acc[0] += q;
      acc[1] = fmaf(q, q, acc[1]);
      acc[2] = fmaf(wt, q, acc[2]);
      acc[3] += gy;
      acc[4] += gx;
      acc[5] += g2;
      acc[6] = fmaf(q, gy, acc[6]);
      acc[7] = fmaf(q, gx, acc[7]);
      acc[8] = fmaf(q, g2, acc[8]);
      acc[9] = fmaf(wt, gy, acc[9]);
      acc[10] = fmaf(wt, gx, acc[10]);
      acc[11] = fmaf(wt, g2, acc[11]);
      acc[12] = fmaf(gy, gy, acc[12]);
      acc[13] = fmaf(gx, gy, acc[13]);
      acc[14] = fmaf(gx, gx, acc[14]);
      acc[15] = fmaf(g2, gy, acc[15]);
      acc[16] = fmaf(g2, gx, acc[16]);
      acc[17] = fmaf(g2, g2, acc[17]);
    }
  }
  block_total<C>(acc, f.tot19, f.buffer);
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) f.buffer ^= 1;
    // every lane evaluates the scalar terms, lane l < axes (axes + 1) one
    // matrix or right-hand-side entry (row l / (axes + 1)), which it carries
    // through the elimination
    const F2* t = f.tot19.total;
    const int lane = threadIdx.x;
    const F2 n = f2(float(orig.n));
    const F2 sum = t[0], dot = t[2];
    const F2 energy = f2_sub(t[1], f2_div(f2_mul(sum, sum), n));
    const float ef = f2_val(energy);
    const bool scored = !(t[18].hi > 0) && ef > 0;
    const float sign = a.absolute && f2_val(dot) < 0 ? -1.f : 1.f;
    const float sq = scored ? sqrtf(ef) : 1.f;
    const float score = sign * f2_val(dot) / sq;
    const double gscore = scored ? double(fminf(1.f, fmaxf(-1.f, score))) : -INFINITY;
    const bool solve = scored && !(use_minimum && gscore <= minimum);
    const int axes = a.rotate ? 3 : 2, cols = axes + 1;
    const int i = min(lane / cols, axes - 1), j = lane % cols;
    bool good = solve;
    double e = 0;
    if (solve) {
      const F2 sn = f2_div(sum, n);
      const F2 inv_e = f2_div(f2(1.f), energy);
      const F2 gsi = t[3 + i];
      const F2 qi = f2_sub(t[6 + i], f2_mul(sn, gsi));
      if (j < axes) {
        const F2 gsj = t[3 + j];
        const F2 qj = f2_sub(t[6 + j], f2_mul(sn, gsj));
        const int hi = max(i, j), lo = min(i, j);
        const F2 gg = t[12 + hi * (hi + 1) / 2 + lo];
        const F2 m = f2_sub(f2_sub(gg, f2_div(f2_mul(gsi, gsj), n)), f2_mul(f2_mul(qi, qj), inv_e));
        e = f2_dbl(f2_mul(m, inv_e));
      } else {
        e = f2_dbl(f2_sub(f2_mul(f2(sign / sq), t[9 + i]), f2_mul(f2_mul(f2(score), qi), inv_e)));
      }
      // Gauss-Jordan with partial pivoting
      const int row = lane / cols;
      for (int c = 0; c < axes; ++c) {
        int pivot = c;
        double pv = __shfl_sync(0xffffffffu, e, c * cols + c);
        for (int r = c + 1; r < axes; ++r) {
          const double v = __shfl_sync(0xffffffffu, e, r * cols + c);
          if (fabs(v) > fabs(pv)) {
            pv = v;
            pivot = r;
          }
        }
        if (fabs(pv) < 1e-14) {
          good = false;
          break;
        }
        const int from = row == c ? pivot * cols + j : row == pivot ? c * cols + j : lane;
        e = __shfl_sync(0xffffffffu, e, from);
        const double inv = 1.0 / pv;
        if (row == c) e *= inv;
        const double prow = __shfl_sync(0xffffffffu, e, c * cols + j);
        const double g = __shfl_sync(0xffffffffu, e, min(row, axes - 1) * cols + c);
        if (row != c) e -= g * prow;
      }
    }
    const double d = __shfl_sync(0xffffffffu, e, lane < axes ? lane * cols + axes : 0);
    const double mine = good && lane < axes ? d : 0.;
    const bool finite = __all_sync(0xffffffffu, isfinite(mine));
    if (lane < 3) f.gn_delta[lane] = mine;
    if (lane == 0) {
      f.ok = good && finite;
      f.gscore = gscore;
    }
  }
  __syncthreads();
}

__device__ __forceinline__ void local_pose(const RefineArgs& a, FitShared& f, const double* pose) {
  set_local(f.lp, pose, a.crop_row, a.crop_col, a.phase, a.inv_scale);
}

// Score at the pose in f.lp, for every thread.
template <int Bits, int C> __device__ __noinline__ double score_pass(const RefineArgs& a, FitShared& f) {
  const double score = continuous_pass<Bits, C>(a.img, a.orig, f.lp, a.absolute, f.tot4, f.buffer);
  if (threadIdx.x == 0) f.buffer ^= 1;
  __syncthreads();
  return score;
}

// The step's factor from f.delta (warp 0): at most .75 rows and columns and
// one angle step.
__device__ __forceinline__ void step_factor(const RefineArgs& a, FitShared& f) {
  const int lane = threadIdx.x;
  double q = INFINITY;
  if (lane < 2 || (lane == 2 && a.rotate)) q = (lane < 2 ? .75 : a.angle_step) / fmax(1e-20, fabs(f.delta[lane]));
  const double q1 = __shfl_sync(0xffffffffu, q, 1), q2 = __shfl_sync(0xffffffffu, q, 2);
  if (lane == 0) f.factor = fmin(fmin(1., fmin(q, q1)), q2);
  __syncwarp();
}

// Trial pose number bt of the step (warp 0): half the last one's way, the
// angle clamped; f.flag tells whether it lies in the domain, f.lp is its
// local pose.  `unit`: level pixels per row and column of the step.
__device__ __forceinline__ void trial_pose(const RefineArgs& a, FitShared& f, int bt, double unit) {
  const int lane = threadIdx.x;
  const double st = f.factor * (1. / double(1 << bt));  // exact
  int pixel = 0;
  if (lane < 3) {
    const double s = lane < 2 ? dmul(unit, st) : st;
    double v = dadd(f.pose[lane], dmul(s, f.delta[lane]));
    if (lane == 2) v = fmin(fmax(v, a.angle_start), a.angle_end);
    f.trial[lane] = v;
    if (lane < 2) {
      // domain_contains: the nearest pixel lies in the image (and the mask)
      const double p = floor(v + .5);
      pixel = p >= 0 && p < double(lane ? a.dom.w : a.dom.h) ? int(p) : -1;
    }
  }
  const int r = __shfl_sync(0xffffffffu, pixel, 0), c = __shfl_sync(0xffffffffu, pixel, 1);
  const bool in = r >= 0 && c >= 0 && (!a.dom.mask || a.dom.mask[size_t(r) * a.dom.w + size_t(c)] != 0);
  if (lane == 0) f.flag = in;
  __syncwarp();
  if (in) local_pose(a, f, f.trial);
}

// fit() of src/ncc_matching/matcher.cpp:903-982 for the pose in f.pose with
// score `score` (single-model query: no memo, no background guard); returns
// the fitted pose's score.
template <int Bits, int C> __device__ __noinline__ double fit_full(const RefineArgs& a, FitShared& f, double score) {
  if (!a.subpixel) return score;
  bool cached = false;  // f.next_delta is the step at f.pose
  for (int it = 0; it < 6; ++it) {
    if (!cached) {
      if (threadIdx.x < 32) local_pose(a, f, f.pose);
      __syncthreads();
      gn_pass<Bits, C>(a, f, false, 0.);
      if (!f.ok) break;
    }
    bool accepted = false, next_valid = false;
    for (int bt = 0; bt < 4 && !accepted; ++bt) {
      __syncthreads();  // f.lp, f.flag and the last pass's results have been read
      if (threadIdx.x < 32) {
        if (bt == 0) {
          if (threadIdx.x < 3) f.delta[threadIdx.x] = cached ? f.next_delta[threadIdx.x] : f.gn_delta[threadIdx.x];
          __syncwarp();
          step_factor(a, f);
        }
        trial_pose(a, f, bt, 1.);
      }
      __syncthreads();
      if (bt == 0) cached = false;
      if (!f.flag) continue;
      double got;
      if (bt == 0 && it + 1 < 6) {
        gn_pass<Bits, C>(a, f, true, score);
        got = f.gscore;
        next_valid = f.ok;
        if (threadIdx.x < 3) f.next_delta[threadIdx.x] = f.gn_delta[threadIdx.x];
        if (!isfinite(got)) got = score_pass<Bits, C>(a, f);
      } else {
        next_valid = false;
        got = score_pass<Bits, C>(a, f);
      }
      if (got > score) {
        score = got;
        accepted = true;
        cached = next_valid;
        if (threadIdx.x < 3) f.pose[threadIdx.x] = f.trial[threadIdx.x];
      }
    }
    if (!accepted) break;
    if (threadIdx.x == 0) f.flag = hypot(f.delta[0], f.delta[1]) < 1e-4 && fabs(f.delta[2]) < 1e-5;
    __syncthreads();
    if (f.flag) break;
  }
  __syncthreads();
  return score;
}

// refine_coarse_candidate of src/ncc_matching/matcher.cpp:853-877
template <int Bits, int C> __device__ __noinline__ double fit_coarse(const RefineArgs& a, FitShared& f, double score) {
  if (!a.subpixel) return score;
  for (int it = 0; it < 6; ++it) {
    if (threadIdx.x < 32) local_pose(a, f, f.pose);
    __syncthreads();
    gn_pass<Bits, C>(a, f, false, 0.);
    if (!f.ok) break;
    bool accepted = false;
    for (int bt = 0; bt < 4 && !accepted; ++bt) {
      __syncthreads();
      if (threadIdx.x < 32) {
        if (bt == 0) {
          if (threadIdx.x < 3) f.delta[threadIdx.x] = f.gn_delta[threadIdx.x];
          __syncwarp();
          step_factor(a, f);
        }
        trial_pose(a, f, bt, a.scale);
      }
      __syncthreads();
      if (!f.flag) continue;
      const double got = score_pass<Bits, C>(a, f);
      if (got > score) {
        score = got;
        accepted = true;
        if (threadIdx.x < 3) f.pose[threadIdx.x] = f.trial[threadIdx.x];
      }
    }
    if (!accepted) break;
    __syncthreads();
  }
  __syncthreads();
  return score;
}

// Discrete level-0 search around the seed (matcher.cpp:986-1059): one warp per
// (patch, position), exact integer moments in the loop.  Leaves the first
// strict maximum over (patch order, dr, dc) in f.best and f.best_score (-inf if none).
template <int C> __device__ __noinline__ void recovery_search(const RefineArgs& a, FitShared& f) {
  const int lane = threadIdx.x & 31, warp = team_thread<C>() >> 5, nw = team_size<C>() >> 5;
  const double seed_row = f.seed[0], seed_col = f.seed[1], seed_angle = f.seed[2];
  float best = -INFINITY;
  int border = INT32_MAX;
  int k = 0;
  for (int j = 0; j < a.nplist0; ++j) {
    const PatchDesc pd = a.view0.patches[a.plist0[j]];
    if (fabs(pd.angle - seed_angle) > a.angle_step * 1.01) continue;
    const PosRange rg = a.ranges0[j];
    const int r0 = int(round(seed_row - a.crop_row - pd.orow)), c0 = int(round(seed_col - a.crop_col - pd.ocol));
    for (int pos = warp; pos < 25; pos += nw) {
      const int r = r0 + pos / 5 - 2, c = c0 + pos % 5 - 2;
      if (r < rg.r0 || r >= rg.r1 || c < rg.c0 || c >= rg.c1) continue;
      if (a.dom.mask && !domain_contains(a.dom, double((long long)a.crop_row + r) + pd.orow,
                                         double((long long)a.crop_col + c) + pd.ocol))
        continue;
      const int2* sw = a.view0.sw + pd.sample_off;
      const float* base = a.lev0.v + size_t(r) * a.lev0.w + c;
      const int2 f0 = __ldg(sw);
      const float s0 = base[off_row(f0.x) * a.lev0.w + off_col(f0.x)];
      float dot = 0.f;
      long long s1 = 0, s2 = 0;
      for (int s = lane; s < pd.n; s += 32) {
        const int2 o = __ldg(sw + s);
        const float x = base[off_row(o.x) * a.lev0.w + off_col(o.x)] - s0;
        dot = fmaf(__int_as_float(o.y), x, dot);
        const long long xi = (long long)x;
        s1 += xi;
        s2 += xi * xi;
      }
      for (int o = 16; o > 0; o >>= 1) {
        dot += __shfl_down_sync(0xffffffffu, dot, o);
        s1 += __shfl_down_sync(0xffffffffu, s1, o);
        s2 += __shfl_down_sync(0xffffffffu, s2, o);
      }
      if (lane == 0) {
        const float sc = window_score(dot, s1, s2, pd.n, a.absolute);
        const int order = k * 25 + pos;
        if (better(sc, order, best, border)) {
          best = sc;
          border = order;
        }
      }
    }
    ++k;
  }
  if (lane == 0) team_store<C>(&f.wbest[warp], F2{best, __int_as_float(border)});
  team_sync<C>();
  if (threadIdx.x == 0) {
    float bs = -INFINITY;
    int bo = INT32_MAX;
    for (int w = 0; w < nw; ++w)
      if (better(f.wbest[w].hi, __float_as_int(f.wbest[w].lo), bs, bo)) {
        bs = f.wbest[w].hi;
        bo = __float_as_int(f.wbest[w].lo);
      }
    f.best[0] = seed_row;
    f.best[1] = seed_col;
    f.best[2] = seed_angle;
    f.best_score = -INFINITY;
    if (bo != INT32_MAX && bs > -INFINITY) {
      int kk = 0;
      for (int j = 0; j < a.nplist0; ++j) {
        const PatchDesc pd = a.view0.patches[a.plist0[j]];
        if (fabs(pd.angle - seed_angle) > a.angle_step * 1.01) continue;
        if (kk == bo / 25) {
          const int r0 = int(round(seed_row - a.crop_row - pd.orow)), c0 = int(round(seed_col - a.crop_col - pd.ocol));
          f.best[0] = double((long long)a.crop_row + r0 + (bo % 25) / 5 - 2) + pd.orow;
          f.best[1] = double((long long)a.crop_col + c0 + (bo % 25) % 5 - 2) + pd.ocol;
          f.best[2] = pd.angle;
          f.best_score = double(bs);
          break;
        }
        ++kk;
      }
    }
  }
  __syncthreads();
}

// refine_candidate (src/ncc_matching/matcher.cpp:878-1061) for one queued
// candidate per block, or per cluster of C blocks (launch_refine says when).
// Bound by the latency of a chain of passes: gathers, two reductions and FP64
// algebra each.  Five 128^2 candidates (six Gauss-Newton passes and four scores
// each): 0.385 -> 0.143 ms.
template <int Bits, int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(kRefineThreads / C)
    refine_kernel(const __grid_constant__ RefineArgs a) {
  __shared__ FitShared f;
  const int b = blockIdx.x / C;
  // a queued round after the end of the selection has nothing to refine
  if (a.batch_count < 0 && a.state->done) return;
  if (b >= (a.batch_count >= 0 ? a.batch_count : a.state->batch_count)) return;
  const int i = a.batch[b], t = threadIdx.x;
  double score = a.sorted[i].score;
  if (t < 3) f.pose[t] = f.seed[t] = (&a.sorted[i].row)[t];
  if (t == 0) f.buffer = 0;
  team_sync<C>();  // every block of the cluster runs
  if (a.finest) {
    score = fit_coarse<Bits, C>(a, f, score);
  } else {
    score = fit_full<Bits, C>(a, f, score);
    if (a.subpixel && a.top > 0 && score < a.min_score) {
      recovery_search<C>(a, f);
      // the search starts from the fitted candidate: only a strictly higher
      // discrete score moves it
      const bool move = f.best_score > score && (f.best[0] != f.pose[0] || f.best[1] != f.pose[1] || f.best[2] != f.pose[2]);
      __syncthreads();
      if (move) {
        const double fitted = score;
        if (t < 3) {
          f.seed[t] = f.pose[t];  // keep the fitted candidate
          f.pose[t] = f.best[t];
        }
        if (t < 32) local_pose(a, f, f.pose);
        __syncthreads();
        score = score_pass<Bits, C>(a, f);
        score = fit_full<Bits, C>(a, f, score);
        if (!(score > fitted)) {
          score = fitted;
          if (t < 3) f.pose[t] = f.seed[t];
          __syncthreads();
        }
      }
    }
  }
  if (t == 0 && team_rank<C>() == 0) {
    Refined r;
    Cand c{};
    r.row = c.row = f.pose[0];
    r.col = c.col = f.pose[1];
    r.angle = c.angle = f.pose[2];
    r.score = score;
    r.ok = (score >= a.min_score) && domain_contains(a.dom, r.row, r.col);
    r.pad = 0;
    r.rect = make_rect(c, a.geom);
    a.refined[i] = r;
    __threadfence();
    a.refined_flag[i] = 2;
  }
}

}  // namespace

// 2-D prefix counts of a domain mask, (h + 1) x (w + 1): row prefixes (one
// thread per row), then column sums (one thread per column, coalesced).
__global__ void domain_rows_kernel(const uint8_t* mask, int w, int h, int32_t* count) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  const size_t pitch = size_t(w) + 1;
  if (y == 0)
    for (int x = 0; x <= w; ++x) count[x] = 0;
  if (y >= h) return;
  int32_t sum = 0;
  int32_t* out = count + size_t(y + 1) * pitch;
  out[0] = 0;
  const uint8_t* row = mask + size_t(y) * w;
  for (int x = 0; x < w; ++x) {
    sum += row[x] != 0;
    out[x + 1] = sum;
  }
}

__global__ void domain_cols_kernel(int w, int h, int32_t* count) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x > w) return;
  const size_t pitch = size_t(w) + 1;
  int32_t sum = 0;
  for (int y = 1; y <= h; ++y) {
    sum += count[size_t(y) * pitch + x];
    count[size_t(y) * pitch + x] = sum;
  }
}

__global__ void interleave_kernel(const int32_t* offs, const float* w, int2* sw, size_t n) {
  const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) sw[i] = make_int2(offs[i], __float_as_int(w[i]));
}

// --------------------------------------------------------------- launchers
cudaError_t launch_interleave(const int32_t* offs, const float* w, int2* sw, size_t n, cudaStream_t s) {
  if (n) interleave_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(offs, w, sw, n);
  return cudaGetLastError();
}

cudaError_t launch_domain_count(const uint8_t* mask, int w, int h, int32_t* count, cudaStream_t s) {
  domain_rows_kernel<<<(h + 127) / 128, 128, 0, s>>>(mask, w, h, count);
  domain_cols_kernel<<<(w + 1 + 255) / 256, 256, 0, s>>>(w, h, count);
  return cudaGetLastError();
}

cudaError_t reserve_dynamic_smem(const void* kernel, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, size_t> granted;
  int dev = 0;
  if (const cudaError_t e = cudaGetDevice(&dev)) return e;
  std::lock_guard<std::mutex> lock(mu);
  size_t& cur = granted[{kernel, dev}];
  if (bytes <= cur) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
  if (e == cudaSuccess) cur = bytes;
  return e;
}

cudaError_t launch_pyramid0(const void* src, int type, int64_t pitch_elems, int crop_row, int crop_col, LevelImage dst,
                            int32_t* error_flag, cudaStream_t s, uint32_t* quads, int quad_tiles) {
  (void)error_flag;
  const dim3 block(32, 8), grid((dst.w + 31) / 32, (dst.h + 7) / 8);
  if (type == 1)
    pyramid0_kernel<uint16_t><<<grid, block, 0, s>>>(static_cast<const uint16_t*>(src), pitch_elems, crop_row, crop_col,
                                                     dst, quads, quad_tiles);
  else
    pyramid0_kernel<uint8_t><<<grid, block, 0, s>>>(static_cast<const uint8_t*>(src), pitch_elems, crop_row, crop_col,
                                                    dst, quads, quad_tiles);
  return cudaGetLastError();
}

cudaError_t launch_pyramid(const LevelImage& src, LevelImage dst, int32_t* error_flag, cudaStream_t s) {
  const dim3 block(32, 8), grid((dst.w + 31) / 32, (dst.h + 7) / 8);
  pyramid_kernel<<<grid, block, 0, s>>>(src, dst, error_flag);
  return cudaGetLastError();
}

cudaError_t launch_prefix(const PrefixArgs& a, cudaStream_t s) {
  int warps = 0;
  for (int l = 0; l < a.n; ++l) warps += a.lev[l].h;
  const int threads = 256;
  if (warps > 0) prefix_kernel<<<(warps * 32 + threads - 1) / threads, threads, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_coarse(const CoarseArgs& a, int max_bh, int max_bw, cudaStream_t s, size_t smem_limit) {
  const size_t smem = size_t(kTileH + max_bh) * size_t(kTileW + max_bw) * sizeof(float);
  if (smem > smem_limit) return cudaErrorInvalidConfiguration;
  if (const cudaError_t e = reserve_dynamic_smem(reinterpret_cast<const void*>(coarse_kernel), smem)) return e;
  const dim3 block(kTileW, kTileH), grid((a.lev.w + kTileW - 1) / kTileW, (a.lev.h + kTileH - 1) / kTileH, a.nplist);
  coarse_kernel<<<grid, block, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_nms(const NmsArgs& a, cudaStream_t s) {
  const int64_t n = int64_t(a.w) * a.h * a.nplist;
  nms_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_track(const TrackArgs& a, int max_candidates, cudaStream_t s, size_t smem_limit, int sms) {
  // candidates are strided over a grid that fills the GPU a few times: the
  // list's length is only known on the device, and a block per possible
  // candidate costs more than the work when the budget is large (65536
  // blocks: about 60 us)
  if (a.warp_lists) {
    // a warp for every four patches of the longest list, against one and four
    // warps for every list: 128^2 templates at 2048^2 0.158 / 0.171 / 0.169 ms,
    // 96^2 0.129 / 0.139 / 0.138; short lists would take one warp alone (64^2
    // 0.224 / 0.197 / 0.238, 57,000 candidates of 48^2 0.56 / 0.46 / 0.75)
    const int warps = a.sel_max <= 4 ? 1 : a.sel_max <= 8 ? 2 : kTrackWarps;
    const int grid = std::min(max_candidates, 96 / warps * sms);
    if (a.narrow)
      track_warp_kernel<true><<<grid, 32 * warps, 0, s>>>(a);
    else
      track_warp_kernel<false><<<grid, 32 * warps, 0, s>>>(a);
    return cudaGetLastError();
  }
  TrackArgs b = a;
  const size_t tables = size_t(a.sel_max) * (kTrackParts * 32 + 2 * 2 * 32) * sizeof(float);
  const size_t fixed = 4 * 1024;  // static and reserved shared memory of the kernel
  size_t smem = size_t(a.win_pitch) * size_t(a.win_rows) * sizeof(float);
  if (smem + tables + fixed > smem_limit) {
    b.win_rows = b.win_pitch = 0;
    smem = 0;
  }
  smem += tables;
  if (const cudaError_t e = reserve_dynamic_smem(reinterpret_cast<const void*>(track_block_kernel), smem)) return e;
  // 128 registers a thread leave an SM 16 warps: in as many blocks as the
  // window lets in, so that their phases overlap.  One block size for all sizes,
  // 128 / 256 / 512 threads, uint16 lists at 2048^2 by the windows of their larger
  // level: 41 KB 0.40 / 0.44 / 0.56 ms, 62 KB 0.32 / 0.32 / 0.37, 86 KB 0.69 /
  // 0.57 / 0.67, 113 KB 0.15 / 0.09 / 0.07, 164 KB 1.05 / 0.73 / 0.64.  Lines
  // drawn where four and two blocks still fit instead (57 and 112 KB) gave 4 % at
  // 101 KB and took 7 % at 55 KB, where the lists were short.
  const int threads = smem > 100 * 1024 ? 512 : smem > 50 * 1024 ? 256 : 128;
  track_block_kernel<<<std::min(max_candidates, 16 * sms), threads, smem, s>>>(b);
  return cudaGetLastError();
}

cudaError_t launch_dedup(const DedupArgs& a, int max_candidates, cudaStream_t s) {
  const unsigned blocks = unsigned((max_candidates + 255) / 256);
  if (a.snap)
    snap_kernel<<<blocks, 256, 0, s>>>(const_cast<Cand*>(a.in), a.state, a.in_slot, a.height, a.width, a.dom);
  dedup_kernel<<<blocks, 256, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_adjoint(const AdjointArgs& a, cudaStream_t s) {
  if (a.n <= 0) return cudaSuccess;
  if (a.img.type == 1)
    adjoint_kernel<uint16_t><<<a.n, kAdjointThreads, 0, s>>>(a);
  else
    adjoint_kernel<uint8_t><<<a.n, kAdjointThreads, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_refine4(const Refine4Args& a, cudaStream_t s, int sms) {
  if (a.n <= 0) return cudaSuccess;
  // Four SMs share the samples of a pose where rows a multiple of 256 bytes
  // apart fall on few L1 sets, so that a rotated pose's gathers on one SM push
  // one another out: 32 poses at all angles, one block -> cluster, rows 2560
  // apart, 96^2 0.74 -> 0.80, 128^2 1.17 -> 1.04, 200^2 2.36 -> 2.00, 256^2 3.53
  // -> 2.87 ms; 4096 apart, 128^2 1.28 -> 1.04, 256^2 4.02 -> 3.07.  Upright poses
  // do not gain there (4096 apart, 128^2 0.92 -> 1.11, 256^2 3.20 -> 3.21), and
  // other row lengths lose at every angle (3000 apart, 96^2 0.62 -> 0.78, 161^2
  // 1.21 -> 1.32, 256^2 3.39 -> 3.32), as do full GPUs: from a pose per SM on the
  // cluster barriers only cost.
  const int64_t row_bytes = a.img.pitch * (a.img.type == 1 ? 2 : 1);
  const bool team = a.n < sms && a.orig.n >= 12288 && row_bytes % 256 == 0;
  const int grid = team ? 4 * a.n : a.n, threads = team ? kRefine4Threads / 4 : kRefine4Threads;
  if (a.img.type == 1)
    team ? refine4_kernel<uint16_t, 4><<<grid, threads, 0, s>>>(a) : refine4_kernel<uint16_t, 1><<<grid, threads, 0, s>>>(a);
  else
    team ? refine4_kernel<uint8_t, 4><<<grid, threads, 0, s>>>(a) : refine4_kernel<uint8_t, 1><<<grid, threads, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_score(const ScoreArgs& a, int max_candidates, cudaStream_t s, int sms) {
  const int grid = std::min(max_candidates, 48 * sms);
  switch (a.img.bits) {
    case 8: score_kernel<8><<<grid, 128, 0, s>>>(a); break;
    case 16: score_kernel<16><<<grid, 128, 0, s>>>(a); break;
    default: score_kernel<0><<<grid, 128, 0, s>>>(a); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_coarse_lattice(Cand* cand, int2* rc, int nsrc, int nbr, int nbc, const int32_t* group_of_src,
                                  int32_t* order, TcTiles* tiles, QueryState* state, int slot, cudaStream_t s) {
  const int n = std::max(1, nsrc * nbr * nbc);
  coarse_lattice_kernel<<<(n + 255) / 256, 256, 0, s>>>(cand, rc, nsrc, nbr, nbc, group_of_src, order, tiles, state,
                                                        slot);
  return cudaGetLastError();
}

cudaError_t launch_coarse_tc_score(const CoarseTcArgs& a, cudaStream_t s) {
  const unsigned cells = unsigned(a.lev.h) * unsigned(a.lev.w);
  coarse_tc_score_kernel<<<dim3((cells + 255) / 256, unsigned(a.nplist)), 256, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_quads(const float* v, int w, int h, const QuadShape& shape, uint32_t* quads, cudaStream_t s) {
  const dim3 block(32, 8), grid((w + 31) / 32, (h + 7) / 8);
  if (shape.bits == 8)
    quads_kernel<8><<<grid, block, 0, s>>>(v, w, h, shape.tiles, quads);
  else if (shape.bits == 16)
    quads_kernel<16><<<grid, block, 0, s>>>(v, w, h, shape.tiles, quads);
  else
    return cudaErrorInvalidValue;
  return cudaGetLastError();
}

cudaError_t launch_sort(const SortArgs& a, int max_candidates, cudaStream_t s) {
  sort_segments_kernel<<<(max_candidates + kSortSeg - 1) / kSortSeg, kSortSeg, 0, s>>>(a);
  const unsigned blocks = unsigned(((long long)max_candidates * kSortLanes + 255) / 256);
  int from = 0;  // lists alternate between the two halves of keys / idx
  for (long long seg = kSortSeg; seg < max_candidates; seg *= kSortFan, from ^= 1) {
    const size_t in = from ? max_candidates : 0, out = from ? 0 : max_candidates;
    sort_merge_kernel<<<blocks, 256, 0, s>>>(a, int(seg), a.keys + in, a.idx + in, a.keys + out, a.idx + out);
  }
  return cudaGetLastError();
}

int sort_launches(int max_candidates) {
  int n = 1;
  for (long long seg = kSortSeg; seg < max_candidates; seg *= kSortFan) ++n;
  return n;
}

cudaError_t launch_select(const SelectArgs& a, cudaStream_t s) {
  select_kernel<<<1, kSelectThreads, 0, s>>>(a);
  return cudaGetLastError();
}

namespace {
template <int C> void refine_launch(const RefineArgs& a, int batch_limit, cudaStream_t s) {
  const int grid = C * batch_limit, threads = kRefineThreads / C;
  switch (a.img.bits) {
    case 8: refine_kernel<8, C><<<grid, threads, 0, s>>>(a); break;
    case 16: refine_kernel<16, C><<<grid, threads, 0, s>>>(a); break;
    default: refine_kernel<0, C><<<grid, threads, 0, s>>>(a); break;
  }
}
}  // namespace

cudaError_t launch_refine(const RefineArgs& a, int batch_limit, cudaStream_t s) {
  // a large template's samples pay for the cluster's barriers.  One block ->
  // cluster, four candidates of a uint8 search: 64^2 0.080 -> 0.090 ms, 96^2
  // 0.088 -> 0.096, 104^2 0.092 -> 0.098, 112^2 0.127 -> 0.131, 128^2 0.123 ->
  // 0.115, 160^2 0.186 -> 0.164, 256^2 0.36 -> 0.28; of a uint16 one: 104^2 0.111
  // -> 0.109, 112^2 0.129 -> 0.121.  Long candidate lists cross over near 88^2.
  if (a.orig.n >= 12288)
    refine_launch<4>(a, batch_limit, s);
  else
    refine_launch<1>(a, batch_limit, s);
  return cudaGetLastError();
}

}  // namespace mvg
