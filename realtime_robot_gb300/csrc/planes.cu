// planes.cu — plane segmentation with convex-hull areas, and the plane-area
// vector of keypoints: the reference's ModelPoint::getArea /
// ScanPoint::get_Area (model_point.h:170-245, scan_point.h:117-188) and
// KeyPoint::get_Vector3D (key_point.h:87-111), which the reference runs
// through PCL's SACSegmentation, ExtractIndices and ConvexHull.
//
// One call extracts planes one after another from the points still
// unclaimed (the reference's loop, while more than 15 % remain).  What bounds
// it at the clouds' sizes (thousands to a few 100k points) is not work but
// the length of the chain: launches, host round trips, and steps that ran on
// one thread or one block.  So a round is five launches and three waits, and
// results reach the host through page-locked memory that the last block of a
// kernel writes:
//   RANSAC   192 sample slots at a time (the walk usually ends in the first):
//            each block forms the planes of the batch itself (SplitMix64 of
//            seed, round, slot draws three positions; float) and counts its
//            points within each, one ballot per warp and plane; the host
//            walks the slots in order with the adaptive stop rule (99 %
//            confidence, at most max_iterations valid samples);
//   refit    the best plane's inliers summed in FP64: partial t over positions
//            t, t + 1024, ... in order, each of the nine sums by threads of
//            its own over 36 blocks, then a pairwise tree in the last block (a
//            fixed order, the oracle's); the host solves the 3x3
//            eigenproblem (planes_host.cpp);
//   select   the refitted plane's inliers (float test), projected onto the
//            plane (float), and the extreme points along 16 directions;
//   rest     the others close up in order; inliers strictly inside the polygon
//            of the extremes (exact orientation tests) cannot be hull
//            vertices and are dropped;
//   hull     one block sorts what is left by (u, v) in shared memory and runs
//            Andrew's monotone chain (orientation in float where its error
//            bound decides, else exact); more than PL_HULL_CAP points, or
//            PL_HULL_OUT vertices, take the radix sort and one thread's chain
//            from memory; the host measures the hull's area and perimeter.
// A 20k-point chair, 5 planes: 4.38 ms before, 0.55 ms now.
// Everything that decides which points are inliers is computed exactly as
// in the CPU oracle (oracle/planes.c), so planes, inlier sets and hulls are
// bit-identical to it.
#include <math.h>
#include <string.h>

#include <vector>

#include "grid.cuh"
#include "planes_host.h"

namespace rtr {

constexpr int PL_SLOTS = 192;       // RANSAC samples scored per batch
constexpr int PL_HULL_CAP = 2048;   // points the hull kernel sorts in shared memory
constexpr int PL_HULL_OUT = 1024;   // hull vertices returned through page-locked memory
constexpr int PL_TILE = 1024;       // points per block of the ordered compaction

// What kernels tell the host, in page-locked memory.
struct PlHost {
  int valid[PL_SLOTS], count[PL_SLOTS];
  float4 coef[PL_SLOTS];
  double sums[9];
  int n_fit;
  int m_rest;     // points that remain
  int n_left;     // inliers not dropped by the polygon
  int hull;       // hull vertices (-1: too many points or vertices for the hull kernel)
  float2 uv[PL_HULL_OUT];
};
// Device words that start at zero and are reset by whoever reads them last.
struct PlDev {
  int count[PL_SLOTS];
  unsigned ticket_score, ticket_refit;
  int n_in, n_left;            // inliers projected, inliers left by the polygon
  unsigned long long ext[16];  // extreme of each direction: ordered value << 32 | position in uv
};
constexpr int PL_PARTIALS = 1024;   // strided FP64 partial sums of the refit

__device__ __forceinline__ uint64_t pl_mix(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ int pl_pick(uint64_t seed, int round, int slot, int k, int m) {
  const uint64_t key = seed ^ ((uint64_t)round << 48) ^ ((uint64_t)slot << 16) ^ (uint64_t)k;
  return (int)(pl_mix(key) % (uint64_t)m);
}

__device__ __forceinline__ bool pl_within(float4 c, float4 p, float thr) {
  const float s = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(c.x, p.x), __fmul_rn(c.y, p.y)), __fmul_rn(c.z, p.z)), c.w);
  return fabsf(s) <= thr;
}

// Position j of the list (the whole cloud when rem is NULL).
__device__ __forceinline__ int pl_at(const int* rem, int j) { return rem ? rem[j] : j; }

// one sample slot: three positions and their plane
__device__ __forceinline__ int pl_slot(const float4* __restrict__ pts, const int* __restrict__ rem, int m,
                                       uint64_t seed, int round, int gs, float4* out) {
  const int i0 = pl_pick(seed, round, gs, 0, m), i1 = pl_pick(seed, round, gs, 1, m), i2 = pl_pick(seed, round, gs, 2, m);
  int ok = i0 != i1 && i0 != i2 && i1 != i2;
  float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
  if (ok) {
    const float4 p0 = pts[rem[i0]], p1 = pts[rem[i1]], p2 = pts[rem[i2]];
    const float ax = __fsub_rn(p1.x, p0.x), ay = __fsub_rn(p1.y, p0.y), az = __fsub_rn(p1.z, p0.z);
    const float bx = __fsub_rn(p2.x, p0.x), by = __fsub_rn(p2.y, p0.y), bz = __fsub_rn(p2.z, p0.z);
    float nx = __fsub_rn(__fmul_rn(ay, bz), __fmul_rn(az, by));
    float ny = __fsub_rn(__fmul_rn(az, bx), __fmul_rn(ax, bz));
    float nz = __fsub_rn(__fmul_rn(ax, by), __fmul_rn(ay, bx));
    const float l2 = __fadd_rn(__fadd_rn(__fmul_rn(nx, nx), __fmul_rn(ny, ny)), __fmul_rn(nz, nz));
    ok = (l2 > 0.f) && (l2 < __int_as_float(0x7f800000));
    if (ok) {
      const float L = __fsqrt_rn(l2);
      nx = __fdiv_rn(nx, L);
      ny = __fdiv_rn(ny, L);
      nz = __fdiv_rn(nz, L);
      c = make_float4(nx, ny, nz,
                      -__fadd_rn(__fadd_rn(__fmul_rn(nx, p0.x), __fmul_rn(ny, p0.y)), __fmul_rn(nz, p0.z)));
    }
  }
  *out = c;
  return ok;
}

// The batch's planes and their inlier counts over the remaining points.  A
// lane keeps the counts of planes lane, lane + 32, ...; the last block hands
// everything to the host.
__global__ void __launch_bounds__(256) k_pl_score(const float4* __restrict__ pts, const int* __restrict__ rem, int m,
                                                  uint64_t seed, int round, int slot0, int n_slots, float thr,
                                                  PlDev* __restrict__ dev, PlHost* __restrict__ host) {
  __shared__ float4 sc[PL_SLOTS];
  __shared__ int sv[PL_SLOTS], cnt[PL_SLOTS];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31;
  for (int s = threadIdx.x; s < PL_SLOTS; s += blockDim.x) {
    float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
    sv[s] = s < n_slots ? pl_slot(pts, rem, m, seed, round, slot0 + s, &c) : 0;
    sc[s] = c;
    cnt[s] = 0;
  }
  __syncthreads();
  int mine[PL_SLOTS / 32];
#pragma unroll
  for (int k = 0; k < PL_SLOTS / 32; ++k) mine[k] = 0;
  for (int base = blockIdx.x * blockDim.x; base < m; base += gridDim.x * blockDim.x) {
    const int j = base + threadIdx.x;
    const bool live = j < m;
    const float4 p = live ? pts[rem[j]] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < PL_SLOTS / 32; ++k)
#pragma unroll 4
      for (int q = 0; q < 32; ++q) {
        const unsigned b = __ballot_sync(0xffffffffu, live && pl_within(sc[32 * k + q], p, thr));
        if (lane == q) mine[k] += __popc(b);
      }
  }
#pragma unroll
  for (int k = 0; k < PL_SLOTS / 32; ++k)
    if (mine[k] && sv[32 * k + lane]) atomicAdd(&cnt[32 * k + lane], mine[k]);
  __syncthreads();
  for (int s = threadIdx.x; s < PL_SLOTS; s += blockDim.x)
    if (cnt[s]) atomicAdd(&dev->count[s], cnt[s]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&dev->ticket_score, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int s = threadIdx.x; s < PL_SLOTS; s += blockDim.x) {
    host->valid[s] = sv[s];
    host->count[s] = __ldcg(&dev->count[s]);
    host->coef[s] = sc[s];
    dev->count[s] = 0;
  }
  if (threadIdx.x == 0) dev->ticket_score = 0u;
}

// FP64 sums of the inliers of plane c in the oracle's fixed order: block b has
// sum b / 4 (x, y, z, xx, xy, xz, yy, yz, zz) of partials 256 (b % 4) ..., a
// thread per partial; the last block adds the partials pairwise.
constexpr int PL_REFIT_BLOCKS = 36;
__global__ void __launch_bounds__(256) k_pl_refit(const float4* __restrict__ pts, const int* __restrict__ rem, int m,
                                                  float4 c, float thr, double* __restrict__ part,
                                                  int* __restrict__ part_n, PlDev* __restrict__ dev,
                                                  PlHost* __restrict__ host) {
  extern __shared__ double sp[];  // [PL_PARTIALS][9], the last block's
  __shared__ int sn[PL_PARTIALS];
  __shared__ int s_last;
  const int k = blockIdx.x >> 2, t = (blockIdx.x & 3) * 256 + threadIdx.x;
  double a = 0.0;
  int n = 0;
#pragma unroll 4
  for (int j = t; j < m; j += PL_PARTIALS) {
    const float4 p = pts[rem[j]];
    if (!pl_within(c, p, thr)) continue;
    const double x = p.x, y = p.y, z = p.z;
    double v = k == 0 ? x : (k == 1 ? y : z);
    if (k >= 3) v = __dmul_rn(k < 6 ? x : (k < 8 ? y : z), k == 3 ? x : ((k == 4 || k == 6) ? y : z));
    a = __dadd_rn(a, v);
    ++n;
  }
  part[k * PL_PARTIALS + t] = a;
  if (k == 0) part_n[t] = n;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&dev->ticket_refit, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int i = threadIdx.x; i < 9 * PL_PARTIALS; i += 256) sp[i] = __ldcg(part + i);
  for (int i = threadIdx.x; i < PL_PARTIALS; i += 256) sn[i] = __ldcg(part_n + i);
  __syncthreads();
  for (int width = PL_PARTIALS / 2; width >= 1; width >>= 1) {
    for (int i = threadIdx.x; i < 9 * width; i += 256) {
      const int q = i / width, e = i - q * width;
      double* P = sp + q * PL_PARTIALS;
      P[e] = __dadd_rn(P[e], P[e + width]);
    }
    for (int e = threadIdx.x; e < width; e += 256) sn[e] += sn[e + width];
    __syncthreads();
  }
  if (threadIdx.x < 9) host->sums[threadIdx.x] = sp[threadIdx.x * PL_PARTIALS];
  if (threadIdx.x == 0) {
    host->n_fit = sn[0];
    dev->ticket_refit = 0u;
  }
}

__device__ __forceinline__ bool finite3(float4 p) { return isfinite(p.x) && isfinite(p.y) && isfinite(p.z); }

// The directions of the extreme points, by angle.
__device__ __forceinline__ float pl_dir(int d, float u, float v) {
  const int q = d >> 2, r = d & 3;  // quadrant: (u, v) turned back by q quarter turns
  const float a = q == 0 ? u : (q == 1 ? v : (q == 2 ? -u : -v)), b = q == 0 ? v : (q == 1 ? -u : (q == 2 ? -v : u));
  return r == 0 ? a : (r == 1 ? __fadd_rn(__fmul_rn(2.f, a), b) : (r == 2 ? __fadd_rn(a, b) : __fadd_rn(a, __fmul_rn(2.f, b))));
}

// Whether point p of the list stays: finite (FIRST), or off the plane.
template <bool FIRST>
__device__ __forceinline__ bool pl_stays(float4 p, float4 c, float thr) {
  return FIRST ? finite3(p) : !pl_within(c, p, thr);
}

// Per tile the number of points that stay; the others (inliers) are projected
// into uv, in any order (-0 becomes +0, so that sort keys order as the float
// comparisons do), and the extremes are taken.
template <bool FIRST>
__global__ void __launch_bounds__(256) k_pl_select(const float4* __restrict__ pts, const int* __restrict__ rem, int m,
                                                   float4 c, float thr, float4 e1, float4 e2,
                                                   int* __restrict__ tile_cnt, float2* __restrict__ uv,
                                                   PlDev* __restrict__ dev) {
  __shared__ int s_stay;
  __shared__ unsigned long long s_ext[16];
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s_stay = 0;
  if (threadIdx.x < 16) s_ext[threadIdx.x] = 0ull;
  __syncthreads();
  unsigned long long best[16];
#pragma unroll
  for (int d = 0; d < 16; ++d) best[d] = 0ull;
  int stay_cnt = 0;
#pragma unroll
  for (int r = 0; r < PL_TILE / 256; ++r) {
    const int j = blockIdx.x * PL_TILE + r * 256 + threadIdx.x;
    const bool live = j < m;
    const float4 p = live ? pts[pl_at(rem, j)] : make_float4(0.f, 0.f, 0.f, 0.f);
    const bool stay = live && pl_stays<FIRST>(p, c, thr);
    stay_cnt += __popc(__ballot_sync(0xffffffffu, stay));
    if (FIRST) continue;
    const bool in = live && !stay;
    const unsigned b = __ballot_sync(0xffffffffu, in);
    if (!b) continue;
    int base = 0;
    if (lane == 0) base = atomicAdd(&dev->n_in, __popc(b));
    base = __shfl_sync(0xffffffffu, base, 0) + __popc(b & lanemask_lt());
    if (in) {
      float u = __fadd_rn(__fadd_rn(__fmul_rn(p.x, e1.x), __fmul_rn(p.y, e1.y)), __fmul_rn(p.z, e1.z));
      float v = __fadd_rn(__fadd_rn(__fmul_rn(p.x, e2.x), __fmul_rn(p.y, e2.y)), __fmul_rn(p.z, e2.z));
      u = __fadd_rn(u, 0.f);
      v = __fadd_rn(v, 0.f);
      uv[base] = make_float2(u, v);
#pragma unroll
      for (int d = 0; d < 16; ++d) {
        const unsigned long long key =
            ((unsigned long long)float_to_ordered(pl_dir(d, u, v)) << 32) | (unsigned)base;
        best[d] = key > best[d] ? key : best[d];
      }
    }
  }
  if (lane == 0 && stay_cnt) atomicAdd(&s_stay, stay_cnt);
  if (!FIRST) {
#pragma unroll
    for (int d = 0; d < 16; ++d) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long x = __shfl_xor_sync(0xffffffffu, best[d], o);
        best[d] = x > best[d] ? x : best[d];
      }
      if (lane == 0 && best[d]) atomicMax(&s_ext[d], best[d]);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) tile_cnt[blockIdx.x] = s_stay;
  if (!FIRST && threadIdx.x < 16 && s_ext[threadIdx.x]) atomicMax(&dev->ext[threadIdx.x], s_ext[threadIdx.x]);
}

__device__ __forceinline__ double pl_cross(float2 o, float2 a, float2 b) {
  const double ax = __dsub_rn((double)a.x, (double)o.x), ay = __dsub_rn((double)a.y, (double)o.y);
  const double bx = __dsub_rn((double)b.x, (double)o.x), by = __dsub_rn((double)b.y, (double)o.y);
  return __dsub_rn(__dmul_rn(ax, by), __dmul_rn(ay, bx));
}

// Whether o, a, b turn left (cross > 0): the float cross where its error bound
// decides (a few parts in 10^7 of its two products), else the exact one.  sign
// 0 stands for a cross of exactly 0 (collinear).
__device__ __forceinline__ int pl_turn(float2 o, float2 a, float2 b) {
  const float l = (a.x - o.x) * (b.y - o.y), r = (a.y - o.y) * (b.x - o.x);
  const float d = l - r, e = 1.0e-6f * (fabsf(l) + fabsf(r)) + 1.0e-30f;
  if (d > e) return 1;
  if (d < -e) return -1;
  const double x = pl_cross(o, a, b);
  return x > 0.0 ? 1 : (x < 0.0 ? -1 : 0);
}

// The points that stay close up in order (offset: the tiles before, then the
// tile's own ranks); and of the inliers those not strictly inside the polygon
// of the extreme points are appended to su, in any order.
template <bool FIRST>
__global__ void __launch_bounds__(256) k_pl_rest(const float4* __restrict__ pts, const int* __restrict__ rem, int m,
                                                 float4 c, float thr, const int* __restrict__ tile_cnt,
                                                 int* __restrict__ out, const float2* __restrict__ uv,
                                                 float2* __restrict__ su, PlDev* __restrict__ dev,
                                                 PlHost* __restrict__ host) {
  constexpr int R = PL_TILE / 256;
  __shared__ int s_cnt[R][8], s_before[8];
  __shared__ float2 E[16];
  __shared__ int s_ne;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int before = 0;
  for (int t = threadIdx.x; t < blockIdx.x; t += 256) before += tile_cnt[t];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  if (lane == 0) s_before[warp] = before;
  int id[R];
  unsigned bal[R];
  bool stay[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int j = blockIdx.x * PL_TILE + r * 256 + threadIdx.x;
    const bool live = j < m;
    id[r] = live ? pl_at(rem, j) : 0;
    stay[r] = live && pl_stays<FIRST>(pts[id[r]], c, thr);
    bal[r] = __ballot_sync(0xffffffffu, stay[r]);
    if (lane == 0) s_cnt[r][warp] = __popc(bal[r]);
  }
  if (!FIRST && warp == 0) {  // the polygon, duplicate corners left out
    const bool any = dev->n_in > 0;
    if (any && lane < 16) E[lane] = uv[(unsigned)(dev->ext[lane] & 0xffffffffull)];
    __syncwarp();
    if (lane == 0) {
      int ne = 0;
      for (int d = 0; any && d < 16; ++d) {
        const float2 p = E[d];
        if (ne == 0 || p.x != E[ne - 1].x || p.y != E[ne - 1].y) E[ne++] = p;
      }
      while (ne > 1 && E[ne - 1].x == E[0].x && E[ne - 1].y == E[0].y) --ne;
      s_ne = ne;
    }
  }
  __syncthreads();
  int off = 0, total = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) off += s_before[w];
  int at = off;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    int o = at;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      o += w < warp ? s_cnt[r][w] : 0;
      at += s_cnt[r][w];
    }
    if (stay[r]) out[o + __popc(bal[r] & lanemask_lt())] = id[r];
  }
  total = at;
  if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1) host->m_rest = total;
  if (FIRST) return;
  const int n = dev->n_in, ne = s_ne;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ((n + 31) & ~31); i += gridDim.x * blockDim.x) {
    const float2 p = i < n ? uv[i] : make_float2(0.f, 0.f);
    bool inside = ne >= 3;
    for (int e = 0; e < ne && inside; ++e) inside = pl_turn(E[e], E[e + 1 < ne ? e + 1 : 0], p) > 0;
    const bool keep = i < n && !inside;
    const unsigned b = __ballot_sync(0xffffffffu, keep);
    if (!b) continue;
    int base = 0;
    if (lane == 0) base = atomicAdd(&dev->n_left, __popc(b));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (keep) su[base + __popc(b & lanemask_lt())] = p;
  }
}

// Half of Andrew's monotone chain (one thread): the left-turning chain over
// at(0), ..., at(n - 1) into H; returns its length.  The last two vertices are
// held in registers.  H may be where at reads from: the chain is never longer
// than what has been read.
template <typename F, typename G>
__device__ __forceinline__ int pl_half(int n, F at, G put_get) {
  int h = 0;
  float2 p1 = make_float2(0.f, 0.f), p2 = p1;  // H[h - 1], H[h - 2]
  for (int i = 0; i < n; ++i) {
    const float2 p = at(i);
    while (h >= 2 && pl_turn(p2, p1, p) <= 0) {
      --h;
      p1 = p2;
      if (h >= 2) p2 = *put_get(h - 2);
    }
    *put_get(h) = p;
    ++h;
    p2 = p1;
    p1 = p;
  }
  return h;
}
// The hull from its halves, the lower one from left to right and the upper
// one from right to left: each but its last point (the other's first).  A
// single point is its own hull.
__device__ __forceinline__ int pl_join(int lower, int upper) {
  const int h = lower + upper - 1;
  return h > 1 ? h - 1 : h;
}

// Hull of at most PL_HULL_CAP points: a bitonic sort by (u, v) in shared
// memory; then 32 lanes each reduce a run of the points to its own half chain
// (a point off the hull of its run is off the hull), and one thread chains
// what is left; warp 0 does the lower half and warp 1 the upper.  One thread
// chaining all of a few hundred points took 53 us, this 22 us.  Resets the
// round's device words.
__global__ void __launch_bounds__(512) k_pl_hull(const float2* __restrict__ su, PlDev* __restrict__ dev,
                                                 PlHost* __restrict__ host) {
  __shared__ unsigned long long key[PL_HULL_CAP];
  __shared__ float2 s_half[2][PL_HULL_CAP];
  __shared__ int s_h[2];
  const int n = dev->n_left, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();  // everyone has it: it is reset below
  if (threadIdx.x < 16) dev->ext[threadIdx.x] = 0ull;
  if (threadIdx.x == 0) {
    dev->n_in = dev->n_left = 0;
    host->n_left = n;
    if (n > PL_HULL_CAP) host->hull = -1;
  }
  if (n > PL_HULL_CAP) return;
  int P = 32;
  while (P < n) P <<= 1;
  for (int i = threadIdx.x; i < P; i += blockDim.x)
    key[i] = i < n ? ((unsigned long long)float_to_ordered(su[i].x) << 32) | float_to_ordered(su[i].y) : ~0ull;
  __syncthreads();
  for (int k = 2; k <= P; k <<= 1)
    for (int jj = k >> 1; jj > 0; jj >>= 1) {
      for (int t = threadIdx.x; t < (P >> 1); t += blockDim.x) {
        const int i = ((t & ~(jj - 1)) << 1) | (t & (jj - 1)), l = i | jj;
        const unsigned long long x = key[i], y = key[l];
        if ((x > y) == ((i & k) == 0)) {
          key[i] = y;
          key[l] = x;
        }
      }
      __syncthreads();
    }
  if (warp < 2) {
    float2* half = s_half[warp];
    const int run = (n + 31) / 32, b = min(n, lane * run), len = min(n - b, run);
    auto at = [&](int i) {  // the upper half goes from right to left
      const unsigned long long x = key[warp == 0 ? i : n - 1 - i];
      return make_float2(ordered_to_float((unsigned)(x >> 32)), ordered_to_float((unsigned)x));
    };
    const int h = pl_half(len, [&](int i) { return at(b + i); }, [&](int i) { return half + b + i; });
    __syncwarp();  // every lane's run is written: the others read it below (shuffles order no memory)
    // close the runs up (a lane writes at or before its own run, after every
    // lane before it has read)
    int to = h;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, to, o);
      if (lane >= o) to += t;
    }
    const int total = __shfl_sync(0xffffffffu, to, 31);
    to -= h;
    for (int l = 0; l < 32; ++l) {
      const int lh = __shfl_sync(0xffffffffu, h, l), lb = min(n, l * run), lt = __shfl_sync(0xffffffffu, to, l);
      for (int i0 = 0; i0 < lh; i0 += 32) {
        const float2 v = half[lb + min(i0 + lane, lh - 1)];
        __syncwarp();
        if (i0 + lane < lh) half[lt + i0 + lane] = v;
        __syncwarp();
      }
    }
    if (lane == 0) s_h[warp] = pl_half(total, [&](int i) { return half[i]; }, [&](int i) { return half + i; });
  }
  __syncthreads();
  const int lower = s_h[0], h = n > 0 ? pl_join(lower, s_h[1]) : 0;
  for (int i = threadIdx.x; i < min(h, PL_HULL_OUT); i += blockDim.x)
    host->uv[i] = i < lower ? s_half[0][i] : s_half[1][i - lower + 1];
  if (threadIdx.x == 0) host->hull = h > PL_HULL_OUT ? -1 : h;
}

// radix keys of a larger set: the points' v, then (second pass) their u in
// that order
__global__ void k_pl_keys_v(const float2* __restrict__ su, int n, uint32_t* __restrict__ k) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) k[i] = float_to_ordered(su[i].y);
}
__global__ void k_pl_keys_u(const float2* __restrict__ su, const uint32_t* __restrict__ order, int n,
                            uint32_t* __restrict__ k) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    k[i] = float_to_ordered(su[order[i]].x);
}
__global__ void k_pl_chain(const float2* __restrict__ su, const uint32_t* __restrict__ order, int n,
                           float2* __restrict__ H, PlHost* __restrict__ host) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int lower = pl_half(n, [&](int i) { return su[order[i]]; }, [&](int i) { return H + i; });
  float2* U = H + lower - 1;  // starts at the lower half's last point, the same
  const int upper = pl_half(n, [&](int i) { return su[order[n - 1 - i]]; }, [&](int i) { return U + i; });
  host->hull = pl_join(lower, upper);
}

// get_Vector3D for each keypoint over the kept surfaces, in list order
__global__ void k_vector3d(const float4* __restrict__ keys, int nk, const rtr_surface* __restrict__ s, int ns,
                           double* __restrict__ v3) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nk; k += gridDim.x * blockDim.x) {
    const float4 p = keys[k];
    double v[3] = {0.16, 0.16, 0.16};
    int vertical = 0, horizontal = 0;
    for (int i = 0; i < ns; ++i) {
      if (!s[i].kept) continue;
      const float* c = s[i].coeffs;
      const double d =
          (double)__fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(c[0], c[0]), __fmul_rn(c[1], c[1])), __fmul_rn(c[2], c[2])));
      const float e = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(c[0], p.x), __fmul_rn(c[1], p.y)), __fmul_rn(c[2], p.z)),
                                c[3]);
      const double dist = __ddiv_rn((double)fabsf(e), d);
      if (s[i].is_vertical == 0 && horizontal == 0 && dist <= 0.05) {
        v[0] = s[i].area;
        ++horizontal;
      } else if (s[i].is_vertical == 1 && vertical <= 1 && dist <= 0.02) {
        v[1 + vertical] = s[i].area;
        ++vertical;
      }
    }
    if (v[1] < v[2]) {
      const double t = v[2];
      v[2] = v[1];
      v[1] = t;
    }
    v3[3 * (size_t)k] = v[0];
    v3[3 * (size_t)k + 1] = v[1];
    v3[3 * (size_t)k + 2] = v[2];
  }
}

static int pl_blocks(int n) {
  int b = (n + 255) / 256;
  if (b > 152 * 8) b = 152 * 8;
  return b < 1 ? 1 : b;
}

// Tiles of the ordered compaction of m points.
static int pl_tiles(int m) { return m > 0 ? (m + PL_TILE - 1) / PL_TILE : 1; }

}  // namespace rtr

using namespace rtr;

extern "C" {

void rtr_plane_default_params(rtr_plane_params* p) {
  if (!p) return;
  memset(p, 0, sizeof(*p));
  p->max_iterations = 150;
  p->distance = 0.005f;
  p->remain_frac = 0.15;
  p->min_area = 0.16;
  p->seed = 0;
}

rtr_status rtr_plane_segment(rtr_context* ctx, const float* d_pts, int n, const rtr_plane_params* prm,
                             rtr_surface* h_surfaces, int max_surfaces, int* h_n_surfaces, rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && prm && n >= 0 && h_n_surfaces && max_surfaces >= 0 && (max_surfaces == 0 || h_surfaces),
                "rtr_plane_segment: bad arguments");
  RTR_CHECK_ARG(prm->max_iterations >= 1 && prm->max_iterations <= 100000 && prm->distance > 0.f &&
                    prm->remain_frac >= 0.0 && prm->remain_frac < 1.0,
                "rtr_plane_segment: parameter out of range");
  RTR_CHECK_ARG(n == 0 || d_pts, "rtr_plane_segment: NULL points");
  *h_n_surfaces = 0;
  if (n == 0) return RTR_OK;
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  // page-locked words that the kernels write, kept by the context
  if (!ctx->plane_host && cudaMallocHost(&ctx->plane_host, sizeof(PlHost)) != cudaSuccess) {
    (void)cudaGetLastError();
    ctx->plane_host = nullptr;
    return fail(RTR_ERR_OOM, "rtr_plane_segment: page-locked words");
  }
  PlHost* const host = static_cast<PlHost*>(ctx->plane_host);
  ScratchPlan plan;
  const size_t o_dev = plan.add<PlDev>(1), o_tile = plan.add<int>(pl_tiles(n));
  const size_t o_rem = plan.add<int>(n), o_rem2 = plan.add<int>(n);
  const size_t o_part = plan.add<double>(9 * PL_PARTIALS), o_pn = plan.add<int>(PL_PARTIALS);
  const size_t o_uv = plan.add<float2>(n), o_su = plan.add<float2>(n), o_hull = plan.add<float2>(2 * (size_t)n + 4);
  const size_t o_k0 = plan.add<uint32_t>(n), o_v0 = plan.add<uint32_t>(n), o_k1 = plan.add<uint32_t>(n),
               o_v1 = plan.add<uint32_t>(n), o_hist = plan.add<uint32_t>(radix_hist_entries(n));
  Scratch s;
  RTR_TRY(ensure_scratch(ctx, plan.bytes, st, &s));
  char* B = s.base;
  PlDev* dev = reinterpret_cast<PlDev*>(B + o_dev);
  int* tile_cnt = reinterpret_cast<int*>(B + o_tile);
  int* rem = reinterpret_cast<int*>(B + o_rem);
  int* rem2 = reinterpret_cast<int*>(B + o_rem2);
  double* part = reinterpret_cast<double*>(B + o_part);
  int* part_n = reinterpret_cast<int*>(B + o_pn);
  float2* uv = reinterpret_cast<float2*>(B + o_uv);
  float2* su = reinterpret_cast<float2*>(B + o_su);
  float2* hull = reinterpret_cast<float2*>(B + o_hull);
  uint32_t* k0 = reinterpret_cast<uint32_t*>(B + o_k0);
  uint32_t* v0 = reinterpret_cast<uint32_t*>(B + o_v0);
  uint32_t* k1 = reinterpret_cast<uint32_t*>(B + o_k1);
  uint32_t* v1 = reinterpret_cast<uint32_t*>(B + o_v1);
  uint32_t* hist = reinterpret_cast<uint32_t*>(B + o_hist);
  const float4* pts = reinterpret_cast<const float4*>(d_pts);
  ProfScope ps(ctx, st, "plane_segment");
  // the refit's partial sums take 72 KB of shared memory (set per call: the
  // attribute belongs to the current device)
  RTR_CUDA(cudaFuncSetAttribute(k_pl_refit, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(PL_PARTIALS * 9 * sizeof(double))));
  RTR_CUDA(cudaMemsetAsync(dev, 0, sizeof(PlDev), st));

  // the finite points, in index order
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  k_pl_select<true><<<pl_tiles(n), 256, 0, st>>>(pts, nullptr, n, zero4, 0.f, zero4, zero4, tile_cnt, nullptr, dev);
  k_pl_rest<true><<<pl_tiles(n), 256, 0, st>>>(pts, nullptr, n, zero4, 0.f, tile_cnt, rem, nullptr, nullptr, dev, host);
  RTR_LAUNCHED(2);
  RTR_CUDA(cudaGetLastError());
  RTR_CUDA(cudaStreamSynchronize(st));
  int m = host->m_rest;
  const int nr_points = m;
  const int max_slots = 11 * prm->max_iterations;
  int np = 0;
  for (int round = 0; (double)m > prm->remain_frac * (double)nr_points && m >= 3; ++round) {
    // RANSAC, batch by batch until the walk ends
    PlaneWalk w;
    float4 bc = zero4;
    for (int base = 0; base < max_slots && !w.done; base += PL_SLOTS) {
      const int ns = max_slots - base < PL_SLOTS ? max_slots - base : PL_SLOTS;
      k_pl_score<<<pl_blocks(m), 256, 0, st>>>(pts, rem, m, prm->seed, round, base, ns, prm->distance, dev, host);
      RTR_LAUNCHED(1);
      RTR_CUDA(cudaGetLastError());
      RTR_CUDA(cudaStreamSynchronize(st));
      w.slot = 0;
      w.base = base;
      const int prev_best = w.best;
      plane_ransac_walk(host->valid, host->count, ns, m, prm->max_iterations, &w);
      if (w.best != prev_best && w.best >= base) bc = host->coef[w.best - base];
    }
    if (w.best < 0) break;
    // least-squares refit over the best sample's inliers
    k_pl_refit<<<PL_REFIT_BLOCKS, 256, PL_PARTIALS * 9 * sizeof(double), st>>>(pts, rem, m, bc, prm->distance, part,
                                                                             part_n, dev, host);
    RTR_LAUNCHED(1);
    RTR_CUDA(cudaGetLastError());
    RTR_CUDA(cudaStreamSynchronize(st));
    float c_in[4] = {bc.x, bc.y, bc.z, bc.w}, c[4];
    int flat = 1;
    plane_refit(host->sums, host->n_fit, c_in, c, &flat);
    const float4 cf = make_float4(c[0], c[1], c[2], c[3]);
    float e1[3], e2[3];
    plane_basis(c, e1, e2);
    // the refitted plane's inliers, what remains, the hull
    k_pl_select<false><<<pl_tiles(m), 256, 0, st>>>(pts, rem, m, cf, prm->distance, make_float4(e1[0], e1[1], e1[2], 0.f),
                                                    make_float4(e2[0], e2[1], e2[2], 0.f), tile_cnt, uv, dev);
    k_pl_rest<false><<<pl_tiles(m), 256, 0, st>>>(pts, rem, m, cf, prm->distance, tile_cnt, rem2, uv, su, dev, host);
    k_pl_hull<<<1, 512, 0, st>>>(su, dev, host);
    RTR_LAUNCHED(3);
    RTR_CUDA(cudaGetLastError());
    RTR_CUDA(cudaStreamSynchronize(st));
    const int nk = host->m_rest, ni = m - nk;
    if (ni == 0) break;
    std::vector<float2> far_uv;
    if (host->hull < 0) {  // too many points, or vertices, for the hull kernel
      const int nl = host->n_left;
      k_pl_keys_v<<<pl_blocks(nl), 256, 0, st>>>(su, nl, k0);
      uint32_t *ks, *vs;
      RTR_TRY(radix_sort_pairs(ctx, k0, v0, k1, v1, hist, nl, nl, nullptr, 32, true, st, &ks, &vs));
      // second, stable pass by u over the first pass's order
      uint32_t* ka = ks == k0 ? k1 : k0;
      uint32_t* va = vs == v0 ? v1 : v0;
      k_pl_keys_u<<<pl_blocks(nl), 256, 0, st>>>(su, vs, nl, ka);
      RTR_CUDA(cudaMemcpyAsync(va, vs, sizeof(uint32_t) * (size_t)nl, cudaMemcpyDeviceToDevice, st));
      uint32_t *ks2, *vs2;
      RTR_TRY(radix_sort_pairs(ctx, ka, va, ka == k0 ? k1 : k0, va == v0 ? v1 : v0, hist, nl, nl, nullptr, 32, false,
                               st, &ks2, &vs2));
      k_pl_chain<<<1, 32, 0, st>>>(su, vs2, nl, hull, host);
      RTR_LAUNCHED(3);
      RTR_CUDA(cudaGetLastError());
      RTR_CUDA(cudaStreamSynchronize(st));
      far_uv.resize((size_t)host->hull);
      RTR_CUDA(cudaMemcpyAsync(far_uv.data(), hull, sizeof(float2) * far_uv.size(), cudaMemcpyDeviceToHost, st));
      RTR_CUDA(cudaStreamSynchronize(st));
    }
    const int nh = host->hull;
    double area = 0.0, perim = 0.0;
    hull_measure(reinterpret_cast<const float*>(far_uv.empty() ? host->uv : far_uv.data()), nh, &area, &perim);
    if (np < max_surfaces) {
      rtr_surface& S = h_surfaces[np];
      memset(&S, 0, sizeof(S));
      S.area = area;
      S.perimeter = perim;
      memcpy(S.coeffs, c, sizeof(c));
      S.n_inliers = ni;
      S.hull_vertices = nh;
      S.flat = flat;
      S.is_vertical = plane_class(c);
      S.kept = S.is_vertical >= 0 && area >= prm->min_area;
    }
    ++np;
    int* t = rem;
    rem = rem2;
    rem2 = t;
    m = nk;
  }
  *h_n_surfaces = np < max_surfaces ? np : max_surfaces;
  if (np > max_surfaces)
    return fail(RTR_ERR_CAPACITY, "rtr_plane_segment: %d planes extracted, room for %d", np, max_surfaces);
  return RTR_OK;
}

rtr_status rtr_vector3d(rtr_context* ctx, const float* d_keys, int n_keys, const rtr_surface* h_surfaces,
                        int n_surfaces, double* d_v3, rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && n_keys >= 0 && n_surfaces >= 0 && (n_surfaces == 0 || h_surfaces),
                "rtr_vector3d: bad arguments");
  if (n_keys == 0) return RTR_OK;
  RTR_CHECK_ARG(d_keys && d_v3, "rtr_vector3d: NULL keypoints or output");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  ScratchPlan plan;
  const size_t o_s = plan.add<rtr_surface>(n_surfaces > 0 ? n_surfaces : 1);
  Scratch s;
  RTR_TRY(ensure_scratch(ctx, plan.bytes, st, &s));
  rtr_surface* d_s = reinterpret_cast<rtr_surface*>(s.base + o_s);
  if (n_surfaces > 0)
    RTR_CUDA(cudaMemcpyAsync(d_s, h_surfaces, sizeof(rtr_surface) * (size_t)n_surfaces, cudaMemcpyHostToDevice, st));
  k_vector3d<<<pl_blocks(n_keys), 256, 0, st>>>(reinterpret_cast<const float4*>(d_keys), n_keys, d_s, n_surfaces,
                                                d_v3);
  RTR_LAUNCHED(1);
  RTR_CUDA(cudaGetLastError());
  // the host array may be reused once the call returns
  RTR_CUDA(cudaStreamSynchronize(st));
  return RTR_OK;
}

}  // extern "C"
