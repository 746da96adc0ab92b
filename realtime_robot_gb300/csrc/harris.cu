// harris.cu — the reference's keypoint detector: pcl::HarrisKeypoint3D as
// ModelPoint::getKeypoint / ScanPoint::getKeypoint use it (model_point.h:
// 127-136, scan_point.h:85-94: radius 0.05, threshold 0.01, non-maximum
// suppression, refinement at its default).  The operator is the 3-D Harris
// response on surface normals (Sipiran & Bustos 2011):
//   normal   smallest eigenvector of the neighbours' FP32 covariance;
//   M        mean of n n^T over the neighbours' normals;
//   R        det(M) - k tr(M)^2 + k, k = 0.04 (for unit normals tr(M) = 1
//            and R = det(M): 0 on faces and edges, up to 1/27 at a corner
//            of three faces, the scale the reference's 0.01 threshold fits);
//   keypoint R > threshold and no neighbour's R larger;
//   refine   the least-squares intersection of the tangent planes near the
//            keypoint (FP64), up to 10 steps.
// Neighbours are every point within the radius, the point included; every
// sum runs over them in ascending index order, so the results equal the CPU
// oracle's (oracle/harris.c) bit for bit.
//
// Kernels: one warp per point.  The warp walks the rows of grid cells (edge =
// radius) around the point and lists the points within the radius in
// ascending index: hits set a bit each in the warp's bitmap of the cloud,
// which is then read out in order (clouds of up to HR_BITS points; larger
// ones append the hits and sort the list).  A sum
// in that order is one chain per accumulator, so the terms of 32 neighbours
// are formed by 32 lanes, staged, and each accumulator's lane adds its own:
// the chains run side by side.  With one lane doing all of it (gather, terms
// and sums) 20,000 points took 383 us of normals, 230 of responses and 3,074
// of refinement; 158, 116 and 207 us now.  A list longer than HR_CAP sets an error
// (RTR_ERR_CAPACITY).
#include <limits.h>
#include <string.h>

#include "eig3.cuh"
#include "grid.cuh"
#include "scan.cuh"
#include "search.cuh"

namespace rtr {

constexpr int HR_WARPS = 4;
constexpr int HR_CAP = 1024;  // neighbours of one point within the radius
// Largest cloud whose bitmap is used.  The bitmap is read out whole for every
// point, so its cost follows the cloud, the sort's the neighbours (whole call,
// us, bitmap / sort; sparse: lattices of chairs, 60 neighbours; dense: one
// chair, up to 1,000): sparse 20k 345 / 365, 30k 431 / 413, 40k 589 / 467, 60k
// 852 / 564, 131k 3276 / 869; dense 20k 635 / 993, 30k 1032 / 1736, 40k 1675 /
// 2577.
constexpr int HR_BITS = 40960;

struct HrArgs {
  GridDev grid;
  const float4* pts;
  int n;
  float r, r2;
  int* err;
};

// The cells that can hold a point within r of q: those of q -+ rr on each
// axis, rr = r with a margin over the rounding of q -+ rr (the cell index is
// monotone in the coordinate).
struct HrBox {
  int x0, x1, y0, y1, z0, z1;
};
__device__ __forceinline__ HrBox hr_box(const GridView& g, float4 q, float r) {
  const float rr = __fadd_rn(__fmul_rn(r, 1.0001f), 1e-6f);
  HrBox b;
  b.x0 = min(max(q_cell(__fsub_rn(q.x, rr), g.ox, g.inv_h), 0), g.nx - 1);
  b.x1 = min(max(q_cell(__fadd_rn(q.x, rr), g.ox, g.inv_h), 0), g.nx - 1);
  b.y0 = min(max(q_cell(__fsub_rn(q.y, rr), g.oy, g.inv_h), 0), g.ny - 1);
  b.y1 = min(max(q_cell(__fadd_rn(q.y, rr), g.oy, g.inv_h), 0), g.ny - 1);
  b.z0 = min(max(q_cell(__fsub_rn(q.z, rr), g.oz, g.inv_h), 0), g.nz - 1);
  b.z1 = min(max(q_cell(__fadd_rn(q.z, rr), g.oz, g.inv_h), 0), g.nz - 1);
  return b;
}

// A warp's shared memory: the list, the staged terms of 32 neighbours (up to
// six accumulators) and the bitmap, all zero between calls.
struct HrWarp {
  int list[HR_CAP];
  float buf[6][33];
};
// words of the bitmap: an odd number per lane, so that the lanes' chunks do
// not share banks
static __host__ __device__ int hr_lane_words(int n) { return ((n + 1023) / 1024) | 1; }
static size_t hr_bits_bytes(int n) { return n <= HR_BITS ? (size_t)hr_lane_words(n) * 32 * sizeof(unsigned) : 0; }
static size_t hr_smem(int n) { return HR_WARPS * (sizeof(HrWarp) + hr_bits_bytes(n)); }
// Warp w's part; its bitmap (cleared here, once) follows.
template <bool BITS>
__device__ __forceinline__ HrWarp* hr_warp(unsigned char* smem, int n, int w, int lane, unsigned** bits) {
  const int words = BITS ? hr_lane_words(n) * 32 : 0;
  unsigned char* base = smem + (size_t)w * (sizeof(HrWarp) + (size_t)words * sizeof(unsigned));
  *bits = reinterpret_cast<unsigned*>(base + sizeof(HrWarp));
  for (int i = lane; i < words; i += 32) (*bits)[i] = 0u;
  __syncwarp();
  return reinterpret_cast<HrWarp*>(base);
}

// The points within r of q (original indices), ascending; returns the count
// (HR_CAP + 1 on overflow, with *err set).
template <bool BITS>
__device__ int hr_gather(const HrArgs& a, const GridView& g, float4 q, int* list, unsigned* bits, int lane) {
  const HrBox bb = hr_box(g, q, a.r);
  int cnt = 0;
  for (int z = bb.z0; z <= bb.z1; ++z)
    for (int y = bb.y0; y <= bb.y1; ++y) {
      const uint2 c = row_span(g, bb.x0, bb.x1, y, z);
      for (unsigned j0 = c.x; j0 < c.y; j0 += 32) {
        const unsigned j = j0 + (unsigned)lane;
        bool in = false;
        int id = 0;
        if (j < c.y) {
          const float4 p = g.pts[j];
          in = dist2_exact(q, p) <= a.r2;
          id = pt_index(p);
        }
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) {
          if (BITS) {
            atomicOr(&bits[id >> 5], 1u << (id & 31));
          } else {
            const int pos = cnt + __popc(b & lanemask_lt());
            if (pos < HR_CAP) list[pos] = id;
          }
        }
        cnt += __popc(b);
      }
    }
  __syncwarp();
  const bool over = cnt > HR_CAP;
  if (over && lane == 0) atomicOr(a.err, 1);
  if (BITS) {
    // lane l reads out its run of words, clearing them
    const int lw = hr_lane_words(a.n), w0 = lane * lw;
    int mine = 0;
    for (int i = 0; i < lw; ++i) mine += __popc(bits[w0 + i]);
    int at = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, at, o);
      if (lane >= o) at += t;
    }
    at -= mine;
    for (int i = 0; i < lw; ++i) {
      unsigned b = bits[w0 + i];
      if (!b) continue;
      bits[w0 + i] = 0u;
      while (b) {
        const int k = __ffs(b) - 1;
        b &= b - 1;
        if (at < HR_CAP) list[at] = (w0 + i) * 32 + k;
        ++at;
      }
    }
    __syncwarp();
    return over ? HR_CAP + 1 : cnt;
  }
  if (over) return HR_CAP + 1;
  // ascending index: bitonic sort over the next power of two
  int P = 1;
  while (P < cnt) P <<= 1;
  for (int i = cnt + lane; i < P; i += 32) list[i] = INT_MAX;
  __syncwarp();
  for (int k = 2; k <= P; k <<= 1)
    for (int jj = k >> 1; jj > 0; jj >>= 1) {
      for (int t = lane; t < (P >> 1); t += 32) {
        const int i = ((t & ~(jj - 1)) << 1) | (t & (jj - 1));
        const int l = i | jj;
        const int x = list[i], y = list[l];
        if ((x > y) == ((i & k) == 0)) {
          list[i] = y;
          list[l] = x;
        }
      }
      __syncwarp();
    }
  return cnt;
}

// Sums over the list in its order: terms(id, t) forms neighbour id's NS terms,
// lane v < NS ends with the sum of term v.
template <int NS, typename F>
__device__ __forceinline__ float hr_sum(const int* list, int cnt, float (&buf)[6][33], int lane, F terms) {
  float s = 0.f;
  for (int c0 = 0; c0 < cnt; c0 += 32) {
    const int m = min(32, cnt - c0);
    if (lane < m) {
      float t[NS];
      terms(list[c0 + lane], t);
#pragma unroll
      for (int v = 0; v < NS; ++v) buf[v][lane] = t[v];
    }
    __syncwarp();
    if (lane < NS) {
      if (m == 32) {
#pragma unroll
        for (int k = 0; k < 32; ++k) s = __fadd_rn(s, buf[lane][k]);
      } else {
        for (int k = 0; k < m; ++k) s = __fadd_rn(s, buf[lane][k]);
      }
    }
    __syncwarp();
  }
  return s;
}

extern __shared__ __align__(16) unsigned char hr_shared[];

template <bool BITS>
__global__ void __launch_bounds__(HR_WARPS * 32) k_hr_normals(HrArgs a, float4* __restrict__ nrm) {
  const GridView g = load_view(a.grid);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned* bits;
  HrWarp& S = *hr_warp<BITS>(hr_shared, a.n, w, lane, &bits);
  for (int i = blockIdx.x * HR_WARPS + w; i < a.n; i += gridDim.x * HR_WARPS) {
    const float4 q = a.pts[i];
    const int cnt = hr_gather<BITS>(a, g, q, S.list, bits, lane);
    float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
    if (cnt <= HR_CAP) {
      const float c = (float)cnt;
      const float sm = hr_sum<3>(S.list, cnt, S.buf, lane, [&](int id, float* t) {
        const float4 p = a.pts[id];
        t[0] = p.x;
        t[1] = p.y;
        t[2] = p.z;
      });
      const float mean = __fdiv_rn(sm, c);
      const float mx = __shfl_sync(0xffffffffu, mean, 0), my = __shfl_sync(0xffffffffu, mean, 1),
                  mz = __shfl_sync(0xffffffffu, mean, 2);
      const float C = hr_sum<6>(S.list, cnt, S.buf, lane, [&](int id, float* t) {
        const float4 p = a.pts[id];
        const float dx = __fsub_rn(p.x, mx), dy = __fsub_rn(p.y, my), dz = __fsub_rn(p.z, mz);
        t[0] = __fmul_rn(dx, dx);
        t[1] = __fmul_rn(dx, dy);
        t[2] = __fmul_rn(dx, dz);
        t[3] = __fmul_rn(dy, dy);
        t[4] = __fmul_rn(dy, dz);
        t[5] = __fmul_rn(dz, dz);
      });
      float Cv[6];
#pragma unroll
      for (int e = 0; e < 6; ++e) Cv[e] = __shfl_sync(0xffffffffu, C, e);
      const float A[9] = {Cv[0], Cv[1], Cv[2], Cv[1], Cv[3], Cv[4], Cv[2], Cv[4], Cv[5]};
      float ev[3], V[9];
      eig3_exact(A, ev, V);
      out = make_float4(V[0], V[3], V[6], 0.f);
    }
    if (lane == 0) nrm[i] = out;
  }
}

__device__ __forceinline__ float hr_det3(const float* m) {
  const float a = __fsub_rn(__fmul_rn(m[3], m[5]), __fmul_rn(m[4], m[4]));
  const float b = __fsub_rn(__fmul_rn(m[1], m[5]), __fmul_rn(m[4], m[2]));
  const float c = __fsub_rn(__fmul_rn(m[1], m[4]), __fmul_rn(m[3], m[2]));
  return __fadd_rn(__fsub_rn(__fmul_rn(m[0], a), __fmul_rn(m[1], b)), __fmul_rn(m[2], c));
}

template <bool BITS>
__global__ void __launch_bounds__(HR_WARPS * 32) k_hr_response(HrArgs a, const float4* __restrict__ nrm,
                                                                float* __restrict__ R) {
  const GridView g = load_view(a.grid);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned* bits;
  HrWarp& S = *hr_warp<BITS>(hr_shared, a.n, w, lane, &bits);
  for (int i = blockIdx.x * HR_WARPS + w; i < a.n; i += gridDim.x * HR_WARPS) {
    const int cnt = hr_gather<BITS>(a, g, a.pts[i], S.list, bits, lane);
    float r = 0.f;
    if (cnt <= HR_CAP) {
      const float sum = hr_sum<6>(S.list, cnt, S.buf, lane, [&](int id, float* t) {
        const float4 v = nrm[id];
        t[0] = __fmul_rn(v.x, v.x);
        t[1] = __fmul_rn(v.x, v.y);
        t[2] = __fmul_rn(v.x, v.z);
        t[3] = __fmul_rn(v.y, v.y);
        t[4] = __fmul_rn(v.y, v.z);
        t[5] = __fmul_rn(v.z, v.z);
      });
      const float mean = __fdiv_rn(sum, (float)cnt);
      float M[6];
#pragma unroll
      for (int e = 0; e < 6; ++e) M[e] = __shfl_sync(0xffffffffu, mean, e);
      const float tr = __fadd_rn(__fadd_rn(M[0], M[3]), M[5]);
      r = __fadd_rn(__fsub_rn(hr_det3(M), __fmul_rn(0.04f, __fmul_rn(tr, tr))), 0.04f);
    }
    if (lane == 0) R[i] = r;
  }
}

// keypoint flags: R over the threshold and (non_max) no neighbour larger
__global__ void __launch_bounds__(HR_WARPS * 32) k_hr_select(HrArgs a, const float* __restrict__ R, float thr,
                                                              int non_max, uint32_t* __restrict__ flag) {
  const GridView g = load_view(a.grid);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int i = blockIdx.x * HR_WARPS + w; i < a.n; i += gridDim.x * HR_WARPS) {
    const float ri = R[i];
    bool ok = ri > thr;
    if (ok && non_max) {
      const float4 q = a.pts[i];
      const HrBox bb = hr_box(g, q, a.r);
      for (int z = bb.z0; z <= bb.z1 && ok; ++z)
        for (int y = bb.y0; y <= bb.y1 && ok; ++y) {
            const uint2 c = row_span(g, bb.x0, bb.x1, y, z);
            bool larger = false;
            for (unsigned j = c.x + (unsigned)lane; j < c.y; j += 32) {
              const float4 p = g.pts[j];
              if (dist2_exact(q, p) <= a.r2 && ri < R[pt_index(p)]) larger = true;
            }
            ok = !__any_sync(0xffffffffu, larger);
          }
    }
    if (lane == 0) flag[i] = ok ? 1u : 0u;
  }
}

// keypoints in ascending source index
__global__ void __launch_bounds__(256) k_hr_list(const uint32_t* __restrict__ flag, const uint32_t* __restrict__ pos,
                                                 int n, int* __restrict__ list) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (flag[i]) list[pos[i]] = i;
}

// refinement and output of the keypoints, a block of HR_REFINE threads each.
// The sums are nine chains of FP64 adds, as long as the neighbourhood, which
// one warp runs; everything before them (the gather, the terms) is spread over
// the block, so that the chains are what is left of a step: 35 us of it with
// one warp doing everything, 20 us now.
constexpr int HR_REFINE = 128;
struct HrRefine {
  int list[HR_CAP];
  int cnt, warp_sum[HR_REFINE / 32];
  double buf[9][HR_CAP + 1];
};
static size_t hr_refine_smem(int n) { return sizeof(HrRefine) + hr_bits_bytes(n); }

// hr_gather by the whole block
template <bool BITS>
__device__ int hr_gather_block(const HrArgs& a, const GridView& g, float4 q, HrRefine& S, unsigned* bits) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (!BITS) {
    __syncthreads();
    if (warp == 0) {
      const int c = hr_gather<false>(a, g, q, S.list, bits, lane);
      if (lane == 0) S.cnt = c;
    }
    __syncthreads();
    return S.cnt;
  }
  const HrBox bb = hr_box(g, q, a.r);
  const int ey = bb.y1 - bb.y0 + 1, rows = ey * (bb.z1 - bb.z0 + 1);
  for (int r = warp; r < rows; r += HR_REFINE / 32) {
    const uint2 c = row_span(g, bb.x0, bb.x1, bb.y0 + r % ey, bb.z0 + r / ey);
    for (unsigned j = c.x + (unsigned)lane; j < c.y; j += 32) {
      const float4 p = g.pts[j];
      const int id = pt_index(p);
      if (dist2_exact(q, p) <= a.r2) atomicOr(&bits[id >> 5], 1u << (id & 31));
    }
  }
  __syncthreads();
  const int words = hr_lane_words(a.n) * 32, per = (words + HR_REFINE - 1) / HR_REFINE;
  const int w0 = min(words, tid * per), w1 = min(words, w0 + per);
  int mine = 0;
  for (int i = w0; i < w1; ++i) mine += __popc(bits[i]);
  int at = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, at, o);
    if (lane >= o) at += t;
  }
  if (lane == 31) S.warp_sum[warp] = at;
  __syncthreads();
  int cnt = 0;
  at -= mine;
#pragma unroll
  for (int w = 0; w < HR_REFINE / 32; ++w) {
    at += w < warp ? S.warp_sum[w] : 0;
    cnt += S.warp_sum[w];
  }
  for (int i = w0; i < w1; ++i) {
    unsigned b = bits[i];
    if (!b) continue;
    bits[i] = 0u;
    while (b) {
      const int k = __ffs(b) - 1;
      b &= b - 1;
      if (at < HR_CAP) S.list[at] = i * 32 + k;
      ++at;
    }
  }
  __syncthreads();
  if (cnt <= HR_CAP) return cnt;
  if (tid == 0) atomicOr(a.err, 1);
  return HR_CAP + 1;
}

template <bool BITS>
__global__ void __launch_bounds__(HR_REFINE) k_hr_refine(HrArgs a, const float4* __restrict__ nrm,
                                                         const float* __restrict__ R, const int* __restrict__ key_src,
                                                         const int* __restrict__ d_nk, int refine,
                                                         float4* __restrict__ keys, int* __restrict__ src) {
  const GridView g = load_view(a.grid);
  const int tid = threadIdx.x, lane = tid & 31, nk = *d_nk;
  HrRefine& S = *reinterpret_cast<HrRefine*>(hr_shared);
  unsigned* bits = reinterpret_cast<unsigned*>(hr_shared + sizeof(HrRefine));
  if (BITS)
    for (int i = tid; i < hr_lane_words(a.n) * 32; i += HR_REFINE) bits[i] = 0u;
  __shared__ double s_sum[9];
  __syncthreads();
  for (int kp = blockIdx.x; kp < nk; kp += gridDim.x) {
    const int i = key_src[kp];
    const float4 p0 = a.pts[i];
    float4 x = make_float4(p0.x, p0.y, p0.z, 0.f);
    for (int it = 0; it < (refine ? 10 : 0); ++it) {
      const int cnt = hr_gather_block<BITS>(a, g, x, S, bits);
      if (cnt > HR_CAP) break;
      // terms 0-5: n n^T, 6-8: n (n . p)
      for (int k = tid; k < cnt; k += HR_REFINE) {
        const float4 v = nrm[S.list[k]];
        const float4 p = a.pts[S.list[k]];
        const double nx = v.x, ny = v.y, nz = v.z;
        const double d = __dadd_rn(__dadd_rn(__dmul_rn(nx, (double)p.x), __dmul_rn(ny, (double)p.y)),
                                   __dmul_rn(nz, (double)p.z));
        S.buf[0][k] = __dmul_rn(nx, nx);
        S.buf[1][k] = __dmul_rn(nx, ny);
        S.buf[2][k] = __dmul_rn(nx, nz);
        S.buf[3][k] = __dmul_rn(ny, ny);
        S.buf[4][k] = __dmul_rn(ny, nz);
        S.buf[5][k] = __dmul_rn(nz, nz);
        S.buf[6][k] = __dmul_rn(nx, d);
        S.buf[7][k] = __dmul_rn(ny, d);
        S.buf[8][k] = __dmul_rn(nz, d);
      }
      __syncthreads();
      if (tid < 9) {
        double t = 0.0;
#pragma unroll 16
        for (int k = 0; k < cnt; ++k) t = __dadd_rn(t, S.buf[tid][k]);
        s_sum[tid] = t;
      }
      __syncthreads();
      double A[6], b[3];
#pragma unroll
      for (int e = 0; e < 6; ++e) A[e] = s_sum[e];
#pragma unroll
      for (int e = 0; e < 3; ++e) b[e] = s_sum[6 + e];
      int stop = 0;
      float4 y = x;
      const double c00 = __dsub_rn(__dmul_rn(A[3], A[5]), __dmul_rn(A[4], A[4]));
      const double c01 = __dsub_rn(__dmul_rn(A[2], A[4]), __dmul_rn(A[1], A[5]));
      const double c02 = __dsub_rn(__dmul_rn(A[1], A[4]), __dmul_rn(A[2], A[3]));
      const double det = __dadd_rn(__dadd_rn(__dmul_rn(A[0], c00), __dmul_rn(A[1], c01)), __dmul_rn(A[2], c02));
      const double tr = __dadd_rn(__dadd_rn(A[0], A[3]), A[5]);
      if (!(det > __dmul_rn(__dmul_rn(__dmul_rn(1e-12, tr), tr), tr))) {
        stop = 1;
      } else {
        const double c11 = __dsub_rn(__dmul_rn(A[0], A[5]), __dmul_rn(A[2], A[2]));
        const double c12 = __dsub_rn(__dmul_rn(A[1], A[2]), __dmul_rn(A[0], A[4]));
        const double c22 = __dsub_rn(__dmul_rn(A[0], A[3]), __dmul_rn(A[1], A[1]));
        // row (lane % 3) of the adjugate times b, over det, in lanes 0-2
        const int e = lane % 3;
        const double r0 = e == 0 ? c00 : (e == 1 ? c01 : c02), r1 = e == 0 ? c01 : (e == 1 ? c11 : c12),
                     r2 = e == 0 ? c02 : (e == 1 ? c12 : c22);
        const float v = (float)__ddiv_rn(__dadd_rn(__dadd_rn(__dmul_rn(r0, b[0]), __dmul_rn(r1, b[1])),
                                                   __dmul_rn(r2, b[2])), det);
        y = make_float4(__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 1),
                        __shfl_sync(0xffffffffu, v, 2), 0.f);
        if (!(dist2_exact(y, p0) <= a.r2)) {
          stop = 1;
        } else {
          const float mv = dist2_exact(y, x);
          if (mv < 1e-12f) stop = 2;  // moved, then done
        }
      }
      if (stop == 1) break;
      x = y;
      if (stop == 2) break;
    }
    if (tid == 0) {
      keys[kp] = make_float4(x.x, x.y, x.z, R[i]);
      if (src) src[kp] = i;
    }
    __syncthreads();
  }
}

static int hr_blocks(int n) {
  int b = (n + HR_WARPS - 1) / HR_WARPS;
  if (b > 152 * 16) b = 152 * 16;
  return b < 1 ? 1 : b;
}

template <bool BITS>
static rtr_status hr_run(const HrArgs& a, float4* nrm, float* R, uint32_t* flag, uint32_t* pos, uint32_t* tiles,
                         int* list, const rtr_harris_params* prm, float4* keys, int* src, int* d_count,
                         cudaStream_t st) {
  const int n = a.n, nb = hr_blocks(n);
  const size_t sm = hr_smem(n), smr = hr_refine_smem(n);
  // set per call: the attribute belongs to the current device
  RTR_CUDA(cudaFuncSetAttribute(k_hr_normals<BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  RTR_CUDA(cudaFuncSetAttribute(k_hr_response<BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  RTR_CUDA(cudaFuncSetAttribute(k_hr_refine<BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smr));
  k_hr_normals<BITS><<<nb, HR_WARPS * 32, sm, st>>>(a, nrm);
  k_hr_response<BITS><<<nb, HR_WARPS * 32, sm, st>>>(a, nrm, R);
  k_hr_select<<<nb, HR_WARPS * 32, 0, st>>>(a, R, prm->threshold, prm->non_max, flag);
  scan_exclusive(flag, pos, tiles, n + 1, n, nullptr, reinterpret_cast<uint32_t*>(d_count), st);
  int lb = (n + 255) / 256;
  if (lb > 152 * 8) lb = 152 * 8;
  k_hr_list<<<lb, 256, 0, st>>>(flag, pos, n, list);
  k_hr_refine<BITS><<<n < 152 * 8 ? n : 152 * 8, HR_REFINE, smr, st>>>(a, nrm, R, list, d_count, prm->refine, keys, src);
  RTR_LAUNCHED(5);
  RTR_CUDA(cudaGetLastError());
  return RTR_OK;
}

}  // namespace rtr

using namespace rtr;

extern "C" {

void rtr_harris_default_params(rtr_harris_params* p) {
  if (!p) return;
  memset(p, 0, sizeof(*p));
  p->radius = 0.05f;
  p->threshold = 0.01f;
  p->non_max = 1;
  p->refine = 1;
}

rtr_status rtr_harris3d(rtr_context* ctx, const float* d_pts, int n, const rtr_harris_params* prm, float* d_keys,
                        int32_t* d_src, int* d_count, rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && prm && n >= 0 && d_count, "rtr_harris3d: bad arguments");
  RTR_CHECK_ARG(prm->radius > 0.f && isfinite(prm->radius), "rtr_harris3d: radius must be positive");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  if (n == 0) {
    RTR_CUDA(cudaMemsetAsync(d_count, 0, sizeof(int), st));
    return RTR_OK;
  }
  RTR_CHECK_ARG(d_pts && d_keys, "rtr_harris3d: NULL points or output");
  const unsigned cap = default_cell_cap(n);
  ScratchPlan plan;
  grid_plan(plan, n, cap);
  const size_t o_n = plan.add<float4>(n), o_r = plan.add<float>(n), o_f = plan.add<uint32_t>(n + 1),
               o_p = plan.add<uint32_t>(n + 1), o_t = plan.add<uint32_t>(scan_tiles(n + 1)), o_e = plan.add<int>(4), o_l = plan.add<int>(n);
  Scratch s;
  RTR_TRY(ensure_scratch(ctx, plan.bytes, st, &s));
  GridBufs gb;
  if (!grid_take(s, n, cap, &gb)) return fail(RTR_ERR_CAPACITY, "rtr_harris3d: scratch carve");
  // the plan's own entries follow the grid's in the arena
  float4* nrm = reinterpret_cast<float4*>(s.base + o_n);
  float* R = reinterpret_cast<float*>(s.base + o_r);
  uint32_t* flag = reinterpret_cast<uint32_t*>(s.base + o_f);
  uint32_t* pos = reinterpret_cast<uint32_t*>(s.base + o_p);
  uint32_t* tiles = reinterpret_cast<uint32_t*>(s.base + o_t);
  int* err = reinterpret_cast<int*>(s.base + o_e);
  ProfScope ps(ctx, st, "harris3d");
  const float4* pts = reinterpret_cast<const float4*>(d_pts);
  RTR_TRY(grid_build(gb, pts, n, nullptr, prm->radius, st));
  RTR_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
  HrArgs a{grid_dev(gb), pts, n, prm->radius, prm->radius * prm->radius, err};
  int* list = reinterpret_cast<int*>(s.base + o_l);
  float4* keys = reinterpret_cast<float4*>(d_keys);
  RTR_TRY(n <= HR_BITS ? hr_run<true>(a, nrm, R, flag, pos, tiles, list, prm, keys, d_src, d_count, st)
                       : hr_run<false>(a, nrm, R, flag, pos, tiles, list, prm, keys, d_src, d_count, st));
  int h_err = 0;
  RTR_CUDA(cudaMemcpyAsync(&h_err, err, sizeof(int), cudaMemcpyDeviceToHost, st));
  RTR_CUDA(cudaStreamSynchronize(st));
  if (h_err)
    return fail(RTR_ERR_CAPACITY, "rtr_harris3d: a point has more than %d neighbours within the radius", HR_CAP);
  return RTR_OK;
}

}  // extern "C"
