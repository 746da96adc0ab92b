// refmatch.cu — the reference's own descriptor route on the GPU:
//
//   KeyPoint::getOccupiedGrid  key_point.h:112-161  -> rtr_ref_occupancy
//   KeyPoint::get_TSDF         key_point.h:251-334  -> rtr_ref_tdf
//   get_Distance               matching.h:122-222   -> rtr_ref_distance
//   the all-pairs loop + match_by_* gates
//                              RealTimeRobot.cpp:70-102, function.h:158-178
//                                                   -> rtr_ref_correspond
//   Ransac                     function.h:35-109    -> rtr_ref_ransac
//
// The reference runs each of these through PCL 1.8.0 octrees built per call
// (per keypoint, per pair and per rotation).  Here nothing is a tree: an
// octree with a defined bounding box is a cube of 2^depth leaves, so a leaf
// is its integer key, the leaves' depth-first order is the Morton order of
// the keys (x the high bit of each level), and the tree's growth when a point
// lands outside is a rule on the cube's corner and depth.  The octree rules
// restated (the same in the CPU oracle):
//   define: depth = fewest levels covering ceil((hi - lo - FLT_EPSILON)/res)
//     leaves on the widest axis (at least 2); each axis padded equally on
//     both sides to the cube edge 2^depth * res (when the pad exceeds
//     FLT_EPSILON);
//   growth: a point with p < min or p >= max on some axis adds a level: on
//     every axis where the point is not above, min -= old edge; then
//     max = min + new edge - FLT_EPSILON; repeated until the point fits;
//     points are inserted in ascending order of their cloud index;
//   key = (unsigned)((p - min) / res) in double against the final cube;
//   centre = (float)((key + 0.5) * res + min).
// All double and float arithmetic that has to agree with the oracle uses the
// _rn intrinsics, so nothing is contracted into an FMA.
//
// Kernels (one CTA per keypoint, a warp or a CTA per pair; the work is gather-
// and issue-bound, the pair kernels' inner loops run from registers and a
// 4 KB shared bitmap):
//   k_ref_occ        box search over the cloud, occupied-leaf count (Number),
//                    ordered append of the box's point indices;
//   k_ref_tdf_cells  the keypoint's occupied leaves in the +-half_tdf cube,
//                    first leaf dropped, as integer voxels -> k_tdf (tdf.cu);
//   k_ref_distance   36 yaw steps of the translated occupancy cloud, leaves
//                    deduplicated in a 32^3 bitmap around the cloud, the
//                    field read per leaf, the leaves sorted into tree order
//                    and their squared values added in float one by one
//                    (the reference's running score), pair transform: a CTA
//                    per pair, for clouds above 512 points and pairs that
//   k_ref_distance_warp leaves (a warp per pair, fixed point; its tables come
//                    from k_ref_keybox);
//   k_ref_gates / k_ref_scatter   the kept pairs in loop order;
//   k_ref_ransac / k_ref_argmax   inliers of every kept pair's transform.
#include <math.h>
#include <string.h>

#include "common.cuh"
#include "scan.cuh"

namespace rtr {

constexpr int REF_DIM = 30;
constexpr int REF_VOL = REF_DIM * REF_DIM * REF_DIM;
constexpr int REF_MAX_DEPTH = 21;
constexpr int REF_PPT = 8;        // cloud points per thread in k_ref_distance
constexpr int REF_WIN = 32;       // leaves per axis of the distance kernel's bitmap window
constexpr unsigned REFW_REDO = 0x7fc0beefu;  // last entry of a transform that the warp form leaves to k_ref_distance
constexpr int REF_OCC_DEPTH = 5;  // cube depth the occupancy and field kernels hold in a bitmap
constexpr double REF_FLT_EPS = 1.1920928955078125e-07;  // FLT_EPSILON

// error bits of the status word
constexpr int REF_ERR_WINDOW = 1;  // a rotated occupancy cloud spans more than REF_WIN leaves
constexpr int REF_ERR_DEPTH = 2;   // an occupancy or field cube deeper than REF_OCC_DEPTH
constexpr int REF_ERR_GROW = 4;    // the occupancy cloud left the field's cube (occupancy box wider)

struct RefRot {
  float c1, s1;          // cosf / sinf of theta = (float)(pi / 18)
  float c2[36], s2[36];  // (float)cos((double)(i * theta)), likewise sin
};

struct OctBox {
  double mn[3], mx[3];
  int depth;
};

__device__ __forceinline__ void oct_define(OctBox& b, const float lo[3], const float hi[3], double res) {
  unsigned mv = 2;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double ext = __dsub_rn((double)hi[a], (double)lo[a]);
    const double k = ceil(__ddiv_rn(__dsub_rn(ext, REF_FLT_EPS), res));
    if (k > (double)mv) mv = (unsigned)k;
  }
  int d = 0;
  while (d < 31 && (1u << d) < mv) ++d;
  const double side = __dmul_rn((double)(1u << d), res);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b.mn[a] = (double)lo[a];
    b.mx[a] = (double)hi[a];
    const double over = __ddiv_rn(__dsub_rn(side, __dsub_rn((double)hi[a], (double)lo[a])), 2.0);
    if (over > REF_FLT_EPS) {
      b.mn[a] = __dsub_rn(b.mn[a], over);
      b.mx[a] = __dadd_rn(b.mx[a], over);
    }
  }
  b.depth = d;
}

// Grow until (x, y, z) fits; false past REF_MAX_DEPTH levels.
__device__ bool oct_fit(OctBox& b, float x, float y, float z, double res) {
  const float p[3] = {x, y, z};
  for (int guard = 0; guard <= REF_MAX_DEPTH + 1; ++guard) {
    bool up[3], out = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      up[a] = (double)p[a] >= b.mx[a];
      out = out || up[a] || (double)p[a] < b.mn[a];
    }
    if (!out) return true;
    if (b.depth >= REF_MAX_DEPTH) return false;
    const double side = __dmul_rn((double)(1u << b.depth), res);
#pragma unroll
    for (int a = 0; a < 3; ++a)
      if (!up[a]) b.mn[a] = __dsub_rn(b.mn[a], side);
    b.depth++;
    const double edge = __dsub_rn(__dmul_rn((double)(1u << b.depth), res), REF_FLT_EPS);
#pragma unroll
    for (int a = 0; a < 3; ++a) b.mx[a] = __dadd_rn(b.mn[a], edge);
  }
  return false;
}

__device__ __forceinline__ unsigned oct_key1(const OctBox& b, float p, int a, double res) {
  const unsigned top = (1u << b.depth) - 1u;
  const unsigned v = __double2uint_rz(__ddiv_rn(__dsub_rn((double)p, b.mn[a]), res));
  return v > top ? top : v;
}

// The cube's float view.  For a float p and a double bound c, p < c exactly
// when p < (c rounded up to float), and p >= c exactly when p >= (c rounded
// up): no float lies strictly between c and its upward rounding.  So the
// inside test needs no double arithmetic.
struct OctBoxF {
  float mn_up[3], mx_up[3], mn_f[3];
};

__device__ __forceinline__ void oct_float(const OctBox& b, OctBoxF& f) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    f.mn_up[a] = __double2float_ru(b.mn[a]);
    f.mx_up[a] = __double2float_ru(b.mx[a]);
    f.mn_f[a] = __double2float_rn(b.mn[a]);
  }
}

__device__ __forceinline__ bool oct_outside_f(const OctBoxF& f, float x, float y, float z) {
  return x < f.mn_up[0] || y < f.mn_up[1] || z < f.mn_up[2] || x >= f.mx_up[0] || y >= f.mx_up[1] ||
         z >= f.mx_up[2];
}

// oct_key1 with a float estimate first: y = (p - min) * (1/res) in float is
// within (|min|/res + 3|y|) * 2^-24 of the exact quotient t, so when y is
// farther than four times that from every integer, floor(y) = floor(t) =
// the double-precision key.  Otherwise (a few keys in 10^5) the double path.
__device__ __forceinline__ unsigned oct_key_f(const OctBox& b, const OctBoxF& f, float p, int a, double res,
                                              float inv) {
  const float y = __fmul_rn(__fsub_rn(p, f.mn_f[a]), inv);
  const float fl = floorf(y);
  const float gap = fminf(__fsub_rn(y, fl), __fsub_rn(__fadd_rn(fl, 1.f), y));
  const float margin = __fmul_rn(__fadd_rn(__fadd_rn(__fmul_rn(fabsf(f.mn_f[a]), inv), __fmul_rn(4.f, fabsf(y))), 4.f),
                                 2.4e-7f);
  if (gap > margin && fl >= 0.f && fl < 4194304.f) {
    const unsigned top = (1u << b.depth) - 1u;
    const unsigned v = (unsigned)fl;
    return v > top ? top : v;
  }
  return oct_key1(b, p, a, res);
}

// Morton code of a key (each coordinate < 2^21): the bits of x, y, z
// interleaved with x the high bit of each triple, so ascending codes list the
// leaves depth-first in child order (x << 2 | y << 1 | z) at any depth.
__device__ __forceinline__ unsigned long long spread3(unsigned v) {
  unsigned long long x = v & 0x1fffffu;
  x = (x | x << 32) & 0x1f00000000ffffull;
  x = (x | x << 16) & 0x1f0000ff0000ffull;
  x = (x | x << 8) & 0x100f00f00f00f00full;
  x = (x | x << 4) & 0x10c30c30c30c30c3ull;
  x = (x | x << 2) & 0x1249249249249249ull;
  return x;
}

__device__ __forceinline__ unsigned compact3(unsigned long long x) {
  x &= 0x1249249249249249ull;
  x = (x ^ (x >> 2)) & 0x10c30c30c30c30c3ull;
  x = (x ^ (x >> 4)) & 0x100f00f00f00f00full;
  x = (x ^ (x >> 8)) & 0x1f0000ff0000ffull;
  x = (x ^ (x >> 16)) & 0x1f00000000ffffull;
  x = (x ^ (x >> 32)) & 0x1fffffull;
  return (unsigned)x;
}

__device__ __forceinline__ unsigned long long morton3(unsigned kx, unsigned ky, unsigned kz, int /*depth*/) {
  return (spread3(kx) << 2) | (spread3(ky) << 1) | spread3(kz);
}

__device__ __forceinline__ void demorton3(unsigned long long m, int /*depth*/, unsigned& kx, unsigned& ky,
                                          unsigned& kz) {
  kx = compact3(m >> 2);
  ky = compact3(m >> 1);
  kz = compact3(m);
}

__device__ __forceinline__ float oct_centre(const OctBox& b, unsigned key, int a, double res) {
  return __double2float_rn(__dadd_rn(__dmul_rn(__dadd_rn((double)key, 0.5), res), b.mn[a]));
}

// ((m0*x + m1*y) + m2*z) + m3 per row, each operation rounded.
__device__ __forceinline__ void xf3(const float* M, float& x, float& y, float& z) {
  const float ox = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(M[0], x), __fmul_rn(M[1], y)), __fmul_rn(M[2], z)), M[3]);
  const float oy = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(M[4], x), __fmul_rn(M[5], y)), __fmul_rn(M[6], z)), M[7]);
  const float oz =
      __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(M[8], x), __fmul_rn(M[9], y)), __fmul_rn(M[10], z)), M[11]);
  x = ox, y = oy, z = oz;
}

// C = A B (4x4 row-major float), the four terms summed in index order.
__device__ void mm4(const float* A, const float* B, float* C) {
  float T[16];
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c) {
      float s = __fmul_rn(A[4 * r], B[c]);
      s = __fadd_rn(s, __fmul_rn(A[4 * r + 1], B[4 + c]));
      s = __fadd_rn(s, __fmul_rn(A[4 * r + 2], B[8 + c]));
      s = __fadd_rn(s, __fmul_rn(A[4 * r + 3], B[12 + c]));
      T[4 * r + c] = s;
    }
  for (int i = 0; i < 16; ++i) C[i] = T[i];
}

__device__ __forceinline__ void eye4(float* M) {
  for (int i = 0; i < 16; ++i) M[i] = (i % 5) == 0 ? 1.f : 0.f;
}

// A keypoint's cube for its CTA: worked out by one warp (FP64 is charged per
// warp instruction, a division some 20 of them; with every warp defining the
// cube and dividing for every key the occupancy of 573 keypoints took 86 us a
// pass, 14 us so), keys from floats where they are certain.
struct OctShared {
  OctBox b;
  OctBoxF f;
};
__device__ __forceinline__ void oct_share(OctShared& s, const float lo[3], const float hi[3], float res) {
  if (threadIdx.x < 32) {
    OctBox b;
    oct_define(b, lo, hi, (double)res);
    if (threadIdx.x == 0) {
      s.b = b;
      oct_float(b, s.f);
    }
  }
  __syncthreads();
}

__device__ __forceinline__ bool in_box(float4 p, const float lo[3], const float hi[3]) {
  return p.x >= lo[0] && p.y >= lo[1] && p.z >= lo[2] && p.x <= hi[0] && p.y <= hi[1] && p.z <= hi[2];
}

// ---------------------------------------------------------------------------
// getOccupiedGrid: one CTA per keypoint.  fill == false: count[k] and
// number[k]; fill == true: indices from offsets[k], ascending.
// ---------------------------------------------------------------------------
constexpr int OCC_NT = 256;

__global__ void __launch_bounds__(OCC_NT) k_ref_occ(const float4* __restrict__ cloud, int n,
                                                    const float4* __restrict__ keys, float res, float half,
                                                    bool fill, int* __restrict__ count, int* __restrict__ number,
                                                    const int* __restrict__ offsets, int* __restrict__ indices,
                                                    int* __restrict__ err) {
  __shared__ unsigned s_bm[1024];
  __shared__ int s_wsum[OCC_NT / 32];
  const int k = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const float4 kp = keys[k];
  const float lo[3] = {__fsub_rn(kp.x, half), __fsub_rn(kp.y, half), __fsub_rn(kp.z, half)};
  const float hi[3] = {__fadd_rn(kp.x, half), __fadd_rn(kp.y, half), __fadd_rn(kp.z, half)};
  if (!fill) {
    __shared__ OctShared s_box;
    for (int i = tid; i < 1024; i += OCC_NT) s_bm[i] = 0u;
    oct_share(s_box, lo, hi, res);
    const OctBox& b = s_box.b;
    const OctBoxF bf = s_box.f;
    const float inv = __fdiv_rn(1.f, res);
    const bool deep = b.depth > REF_OCC_DEPTH;
    if (deep && tid == 0) atomicOr(err, REF_ERR_DEPTH);
    int c = 0;
    for (int i = tid; i < n; i += OCC_NT) {
      const float4 p = cloud[i];
      if (!in_box(p, lo, hi)) continue;
      ++c;
      if (deep) continue;
      const unsigned long long m =
          morton3(oct_key_f(b, bf, p.x, 0, (double)res, inv), oct_key_f(b, bf, p.y, 1, (double)res, inv),
                  oct_key_f(b, bf, p.z, 2, (double)res, inv), b.depth);
      atomicOr(&s_bm[(unsigned)(m >> 5)], 1u << (unsigned)(m & 31ull));
    }
    __syncthreads();
    int u = 0;
    for (int i = tid; i < 1024; i += OCC_NT) u += __popc(s_bm[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      c += __shfl_xor_sync(0xffffffffu, c, o);
      u += __shfl_xor_sync(0xffffffffu, u, o);
    }
    __shared__ int s_c[OCC_NT / 32], s_u[OCC_NT / 32];
    if (lane == 0) s_c[w] = c, s_u[w] = u;
    __syncthreads();
    if (tid == 0) {
      int tc = 0, tu = 0;
      for (int i = 0; i < OCC_NT / 32; ++i) tc += s_c[i], tu += s_u[i];
      count[k] = tc;
      number[k] = tu;
    }
    return;
  }
  int base = offsets[k];
  for (int c0 = 0; c0 < n; c0 += OCC_NT) {
    const int i = c0 + tid;
    const bool f = i < n && in_box(cloud[i], lo, hi);
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (lane == 0) s_wsum[w] = __popc(bal);
    __syncthreads();
    int before = 0, tot = 0;
    for (int j = 0; j < OCC_NT / 32; ++j) {
      before += j < w ? s_wsum[j] : 0;
      tot += s_wsum[j];
    }
    if (f) indices[base + before + __popc(bal & lanemask_lt())] = i;
    base += tot;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// get_TSDF's occupied voxels: one CTA per keypoint.  fill == false:
// cnt[k] = leaves - 1 (0 without leaves); fill == true: the integer voxels of
// every leaf but the first, in leaf order, from cell_off[k].
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(OCC_NT) k_ref_tdf_cells(const float4* __restrict__ cloud,
                                                          const float4* __restrict__ keys,
                                                          const int* __restrict__ offsets,
                                                          const int* __restrict__ indices, float res, float half,
                                                          bool fill, int* __restrict__ cnt,
                                                          const int* __restrict__ cell_off, int* __restrict__ occ,
                                                          int* __restrict__ err) {
  __shared__ unsigned s_bm[1024];
  __shared__ int s_ws[OCC_NT / 32];
  const int k = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const float4 kp = keys[k];
  const float lo[3] = {__fsub_rn(kp.x, half), __fsub_rn(kp.y, half), __fsub_rn(kp.z, half)};
  const float hi[3] = {__fadd_rn(kp.x, half), __fadd_rn(kp.y, half), __fadd_rn(kp.z, half)};
  __shared__ OctShared s_box;
  __shared__ int s_ix[3][1 << REF_OCC_DEPTH];  // the field coordinate of a leaf's key
  oct_share(s_box, lo, hi, res);
  const OctBox& b = s_box.b;
  const OctBoxF bf = s_box.f;
  const float inv = __fdiv_rn(1.f, res);
  if (b.depth > REF_OCC_DEPTH) {
    if (tid == 0) {
      atomicOr(err, REF_ERR_DEPTH);
      if (!fill) cnt[k] = 0;
    }
    return;
  }
  if (fill && tid < 3 << REF_OCC_DEPTH) {
    const int a = tid >> REF_OCC_DEPTH;
    const float c = oct_centre(b, (unsigned)(tid & ((1 << REF_OCC_DEPTH) - 1)), a, (double)res);
    s_ix[a][tid & ((1 << REF_OCC_DEPTH) - 1)] = __double2int_rz(__ddiv_rn(__dsub_rn((double)c, (double)lo[a]), (double)res));
  }
  for (int i = tid; i < 1024; i += OCC_NT) s_bm[i] = 0u;
  __syncthreads();
  const int beg = offsets[k], end = offsets[k + 1];
  bool grew = false;
  for (int j = beg + tid; j < end; j += OCC_NT) {
    const float4 p = cloud[indices[j]];
    if (oct_outside_f(bf, p.x, p.y, p.z)) {
      grew = true;
      continue;
    }
    const unsigned long long m =
        morton3(oct_key_f(b, bf, p.x, 0, (double)res, inv), oct_key_f(b, bf, p.y, 1, (double)res, inv),
                oct_key_f(b, bf, p.z, 2, (double)res, inv), b.depth);
    atomicOr(&s_bm[(unsigned)(m >> 5)], 1u << (unsigned)(m & 31ull));
  }
  if (grew) atomicOr(err, REF_ERR_GROW);
  __syncthreads();
  // each thread owns 4 consecutive words (1024 = 4 * OCC_NT)
  unsigned wd[4];
  int mine = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    wd[q] = s_bm[4 * tid + q];
    mine += __popc(wd[q]);
  }
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_ws[w] = incl;
  __syncthreads();
  int before = incl - mine, total = 0;
  for (int j = 0; j < OCC_NT / 32; ++j) {
    before += j < w ? s_ws[j] : 0;
    total += s_ws[j];
  }
  if (!fill) {
    if (tid == 0) cnt[k] = total > 0 ? total - 1 : 0;
    return;
  }
  int rank = before;
  const int out0 = cell_off[k];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    unsigned bits = wd[q];
    while (bits) {
      const int bit = __ffs(bits) - 1;
      bits &= bits - 1u;
      if (rank > 0) {
        const unsigned long long m = (unsigned long long)(4 * tid + q) * 32ull + (unsigned long long)bit;
        unsigned kx, ky, kz;
        demorton3(m, b.depth, kx, ky, kz);
        const unsigned kk[3] = {kx, ky, kz};
        int* o = occ + 3 * (size_t)(out0 + rank - 1);
#pragma unroll
        for (int a = 0; a < 3; ++a) o[a] = s_ix[a][kk[a]];
      }
      ++rank;
    }
  }
}

// ---------------------------------------------------------------------------
// get_Distance: one CTA per pair.
// ---------------------------------------------------------------------------
template <int NT>
struct RefShared {
  unsigned bm[REF_WIN * REF_WIN * REF_WIN / 32];
  int first[NT / 32];
  unsigned long long mmin[NT / 32];
  unsigned kmin[NT / 32][3], kmax[NT / 32][3];
  int u;  // distinct leaves of the current rotation
  float px, py, pz;
};

// get_Distance adds the squared field values of a rotation's leaves (all but
// the first) in float, one by one in the octree's depth-first order, into a
// running score that no rotation resets (matching.h:141,179-189).  Float
// addition does not reassociate, so the leaves are first put in that order:
// a bitonic sort of (Morton code, field value) pairs in shared memory (codes
// are distinct; padding keys are ~0), then one thread adds them in sequence.
// P is a power of two >= 2; `t` / `nt` this thread's index and the number of
// threads sorting; `sync` orders the stages (__syncwarp or __syncthreads).
template <class Sync>
__device__ __forceinline__ void leaf_sort(unsigned long long* key, float* val, int P, int t, int nt, Sync sync) {
  for (int k = 2; k <= P; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int q = t; q < (P >> 1); q += nt) {
        const int i = ((q & ~(j - 1)) << 1) | (q & (j - 1));  // bit j of i clear
        const int l = i | j;
        const unsigned long long a = key[i], b = key[l];
        if ((a > b) == ((i & k) == 0)) {
          key[i] = b;
          key[l] = a;
          const float x = val[i];
          val[i] = val[l];
          val[l] = x;
        }
      }
      sync();
    }
}

// The running score's update for one rotation from its sorted leaves:
// score = (score + v_1^2 + ... + v_{u-1}^2) / (u - 1), each operation a
// float operation rounded to nearest; (size_t)(u - 1) is 2^64 for u = 0.
__device__ __forceinline__ float leaf_running_score(float dtf, const float* val, int u) {
  for (int i = 1; i < u; ++i) dtf = __fadd_rn(dtf, __fmul_rn(val[i], val[i]));
  const float div = u == 0 ? 18446744073709551616.f : (float)(u - 1);
  return __fdiv_rn(dtf, div);
}

struct BlockSync {
  __device__ void operator()() const { __syncthreads(); }
};

__device__ __forceinline__ float field_at(const float* __restrict__ grid, const OctBox& b, unsigned kx, unsigned ky,
                                          unsigned kz, const float lo[3], float res) {
  const unsigned kk[3] = {kx, ky, kz};
  long long ix[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float c = oct_centre(b, kk[a], a, (double)res);
    const float q = __fdiv_rn(__fsub_rn(c, lo[a]), res);
    if (!(q > -2147483648.f && q < 2147483648.f)) return 900.f;
    ix[a] = (long long)__float2int_rz(q);
  }
  const long long idx = ix[1] * REF_DIM + ix[2] * (REF_DIM * REF_DIM) + ix[0];
  return (idx >= 0 && idx < REF_VOL) ? __ldg(grid + idx) : 900.f;
}

template <int NT>
__global__ void __launch_bounds__(NT) k_ref_distance(const float4* __restrict__ mcloud,
                                                     const float4* __restrict__ mkeys,
                                                     const int* __restrict__ moff, const int* __restrict__ midx,
                                                     const float* __restrict__ mtdf,
                                                     const float4* __restrict__ skeys, int ns,
                                                     const int* __restrict__ pair_m,
                                                     const int* __restrict__ pair_s, float res, float half,
                                                     RefRot rot, float* __restrict__ score, float* __restrict__ Tout,
                                                     int* __restrict__ err, int warp_max_points) {
  constexpr int NW = NT / 32;
  constexpr int CAP = NT * REF_PPT;  // distinct leaves <= points
  __shared__ RefShared<NT> sh;
  extern __shared__ unsigned long long s_leaf_key[];  // [CAP] keys, then [CAP] floats
  float* s_leaf_val = reinterpret_cast<float*>(s_leaf_key + CAP);
  const long long p = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int m = pair_m ? pair_m[p] : (int)(p / ns);
  const int s = pair_s ? pair_s[p] : (int)(p % ns);
  const float4 km = mkeys[m], ks = skeys[s];
  float* To = Tout + 16 * p;
  // smaller clouds: only the pairs that the warp form has left
  if (moff[m + 1] - moff[m] <= warp_max_points && __float_as_uint(To[15]) != REFW_REDO) return;
  if (!(isfinite(km.x) && isfinite(km.y) && isfinite(km.z) && isfinite(ks.x) && isfinite(ks.y) &&
        isfinite(ks.z))) {
    if (tid == 0) {
      score[p] = __int_as_float(0x7fc00000);
      eye4(To);
    }
    return;
  }
  const int beg = moff[m], n = moff[m + 1] - beg;
  const float* grid = mtdf + (size_t)m * REF_VOL;
  const double dres = (double)res;
  const float inv = __fdiv_rn(1.f, res);
  const float lo[3] = {__fsub_rn(km.x, half), __fsub_rn(km.y, half), __fsub_rn(km.z, half)};
  const float hi[3] = {__fadd_rn(km.x, half), __fadd_rn(km.y, half), __fadd_rn(km.z, half)};
  float Tm[16], T1[16], T3[16], M[16];
  eye4(Tm);
  Tm[3] = __fsub_rn(km.x, ks.x), Tm[7] = __fsub_rn(km.y, ks.y), Tm[11] = __fsub_rn(km.z, ks.z);
  eye4(T1);
  T1[3] = -km.x, T1[7] = -km.y;
  eye4(T3);
  T3[3] = km.x, T3[7] = km.y;
  {
    float Rs[16];
    eye4(Rs);
    Rs[0] = rot.c1, Rs[4] = rot.s1, Rs[1] = -rot.s1, Rs[5] = rot.c1;
    mm4(T3, Rs, M);
    mm4(M, T1, M);
  }
  float px[REF_PPT], py[REF_PPT], pz[REF_PPT];
#pragma unroll
  for (int q = 0; q < REF_PPT; ++q) {
    const int j = tid + q * NT;
    px[q] = py[q] = pz[q] = 0.f;
    if (j < n) {
      const float4 c = mcloud[midx[beg + j]];
      px[q] = c.x, py[q] = c.y, pz[q] = c.z;
      xf3(Tm, px[q], py[q], pz[q]);
    }
  }
  OctBox b0;
  oct_define(b0, lo, hi, dres);
  float dtf = 0.f, bestf = 100000000.f;
  int best_i = 0;
  bool bad = false;
  for (int it = 0; it < 36 && !bad; ++it) {
    if (it != 0) {
#pragma unroll
      for (int q = 0; q < REF_PPT; ++q)
        if (tid + q * NT < n) xf3(M, px[q], py[q], pz[q]);
    }
    // the tree's growth, point by point in index order: every thread keeps
    // the same cube, grown by the first point outside it until none is
    OctBox b = b0;
    OctBoxF bf;
    oct_float(b, bf);
    for (int round = 0; round < 4 * REF_MAX_DEPTH + 4; ++round) {
      int first = 0x7fffffff;
#pragma unroll
      for (int q = 0; q < REF_PPT; ++q) {
        const int j = tid + q * NT;
        if (j < n && first == 0x7fffffff && oct_outside_f(bf, px[q], py[q], pz[q])) first = j;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
      if (lane == 0) sh.first[w] = first;
      __syncthreads();
      first = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < NW; ++i) first = min(first, sh.first[i]);
      if (first == 0x7fffffff) break;
      if (first % NT == tid) {
        const int q = first / NT;
#pragma unroll
        for (int qq = 0; qq < REF_PPT; ++qq)
          if (qq == q) sh.px = px[qq], sh.py = py[qq], sh.pz = pz[qq];
      }
      __syncthreads();
      if (!oct_fit(b, sh.px, sh.py, sh.pz, dres)) bad = true;
      oct_float(b, bf);
      __syncthreads();
      if (bad) break;
    }
    if (bad) break;
    // leaf keys (as Morton codes), the first leaf, the keys' bounding window
    unsigned long long mc[REF_PPT];
    unsigned long long mmin = ~0ull;
    unsigned kmin[3] = {~0u, ~0u, ~0u}, kmax[3] = {0u, 0u, 0u};
#pragma unroll
    for (int q = 0; q < REF_PPT; ++q) {
      mc[q] = ~0ull;
      if (tid + q * NT < n) {
        const unsigned kx = oct_key_f(b, bf, px[q], 0, dres, inv), ky = oct_key_f(b, bf, py[q], 1, dres, inv),
                       kz = oct_key_f(b, bf, pz[q], 2, dres, inv);
        mc[q] = morton3(kx, ky, kz, b.depth);
        mmin = min(mmin, mc[q]);
        kmin[0] = min(kmin[0], kx), kmin[1] = min(kmin[1], ky), kmin[2] = min(kmin[2], kz);
        kmax[0] = max(kmax[0], kx), kmax[1] = max(kmax[1], ky), kmax[2] = max(kmax[2], kz);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mmin = min(mmin, __shfl_xor_sync(0xffffffffu, mmin, o));
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        kmin[a] = min(kmin[a], __shfl_xor_sync(0xffffffffu, kmin[a], o));
        kmax[a] = max(kmax[a], __shfl_xor_sync(0xffffffffu, kmax[a], o));
      }
    }
    if (lane == 0) {
      sh.mmin[w] = mmin;
#pragma unroll
      for (int a = 0; a < 3; ++a) sh.kmin[w][a] = kmin[a], sh.kmax[w][a] = kmax[a];
    }
    for (int i = tid; i < REF_WIN * REF_WIN * REF_WIN / 32; i += NT) sh.bm[i] = 0u;
    if (tid == 0) sh.u = 0;
    __syncthreads();
    for (int i = 0; i < NW; ++i) {
      mmin = min(mmin, sh.mmin[i]);
#pragma unroll
      for (int a = 0; a < 3; ++a) kmin[a] = min(kmin[a], sh.kmin[i][a]), kmax[a] = max(kmax[a], sh.kmax[i][a]);
    }
    const bool window_ok = n == 0 || (kmax[0] - kmin[0] < (unsigned)REF_WIN && kmax[1] - kmin[1] < (unsigned)REF_WIN &&
                                      kmax[2] - kmin[2] < (unsigned)REF_WIN);
    if (!window_ok && tid == 0) atomicOr(err, REF_ERR_WINDOW);
    // distinct leaves: the thread that sets a leaf's bit reads its field and
    // lists (Morton code, value); the first leaf's value is never added
    if (window_ok) {
#pragma unroll
      for (int q = 0; q < REF_PPT; ++q) {
        if (mc[q] == ~0ull) continue;
        unsigned kx, ky, kz;
        demorton3(mc[q], b.depth, kx, ky, kz);
        const unsigned l = (kx - kmin[0]) + REF_WIN * ((ky - kmin[1]) + REF_WIN * (kz - kmin[2]));
        const unsigned bit = 1u << (l & 31u);
        const unsigned old = atomicOr(&sh.bm[l >> 5], bit);
        if (old & bit) continue;
        const float v = mc[q] == mmin ? 0.f : field_at(grid, b, kx, ky, kz, lo, res);
        const int slot = atomicAdd(&sh.u, 1);
        s_leaf_key[slot] = mc[q];
        s_leaf_val[slot] = v;
      }
    }
    __syncthreads();
    const int u = sh.u;
    int P = 2;
    while (P < u) P <<= 1;
    for (int i = u + tid; i < P; i += NT) s_leaf_key[i] = ~0ull;
    __syncthreads();
    leaf_sort(s_leaf_key, s_leaf_val, P, tid, NT, BlockSync());
    if (tid == 0) {
      dtf = leaf_running_score(dtf, s_leaf_val, u);
      if (dtf < bestf) {
        bestf = dtf;
        best_i = it;
      }
    }
    __syncthreads();
  }
  if (tid != 0) return;
  if (bad) {
    score[p] = __int_as_float(0x7fc00000);
    eye4(To);
    return;
  }
  score[p] = bestf;
  float S[16], R2[16], A[16];
  eye4(S);
  const float cs = __fdiv_rn(km.z, ks.z);
  S[0] = S[5] = S[10] = cs;
  eye4(R2);
  R2[0] = rot.c2[best_i], R2[4] = rot.s2[best_i], R2[1] = -rot.s2[best_i], R2[5] = rot.c2[best_i];
  mm4(S, T3, A);
  mm4(A, R2, A);
  mm4(A, T1, A);
  mm4(A, Tm, A);
  for (int i = 0; i < 16; ++i) To[i] = A[i];
}

// get_Distance, one warp per pair, for occupancy clouds of up to 512 points
// (Q rows of 32; 4 KB of shared memory and less a warp).
//
// What bounds it: issue (and the shuffle / shared-memory pipe next to it):
// about 120 instructions per point and rotation, no FP64 among them.  The
// chip's FP64 rate is low enough that a dozen double operations a rotation
// cost more than everything else, so the cubes are kept in fixed point (a unit
// that follows the leaf, 2^-40 at 0.01; see RefUnit), where the reference's
// double arithmetic is exact:
//  - the bounds of a keypoint's field cube, the leaf edge and FLT_EPSILON are
//    multiples of the unit and below 2^53 of them, so every sum and difference
//    of the growth rule has at most 53 bits and the doubles are never rounded
//    (k_ref_keybox checks it; keypoints that fail, and clouds beyond
//    2^REFW_RANGE_LOG2 leaves of the origin, are left to k_ref_distance);
//  - a float p >= c (c a whole number of units) exactly when floor(p) >= c;
//  - a leaf key is floor((p - min) / res): from a float estimate where that is
//    farther from a whole number than its error, else from whole-number
//    remainders (a quotient that is not whole is more than a double's rounding
//    away from it).
// Per rotation: points turned; the cloud's box (four reductions; z does not
// change) grows the cube (lane a % 3 holds axis a); keys; the leaves' tree
// order as an 18-bit code: 15 Morton bits of the keys' low five bits, and a
// bit per axis for a cloud that crosses a multiple of 32 leaves there, these
// ordered by the highest bit that the crossing changes; codes with the point's
// index sorted in registers (bitonic); equal neighbours dropped; the field
// values, squared, put in that order in shared memory and added one by one.
// Main's clouds (340 x 573 keypoints, clouds of 90 points on average): 62.0 ms
// with double arithmetic per rotation, a bitonic sort of 64-bit Morton codes in
// shared memory and a 32^3 bitmap; 12.0 ms with the growth in whole units and
// a 32-bit sort in registers; 7.0 ms with the growth in leaves, one row of 32
// more per size class instead of powers of two, and no sort where no value is
// read (half the rotations there).
constexpr int REFW_WARPS = 4;
constexpr int REFW_MAX = 512;                 // points of the largest cloud taken
constexpr int REFW_RANGE_LOG2 = 17;           // leaves from the origin

// The unit of the fixed point, 2^-e: a leaf has 2^33 .. 2^34 of them, so all 24
// bits of the resolution are whole units, a coordinate at the end of the
// range has at most 2^51 and a grown cube's bounds stay below 2^53; the
// quotient of a point's offset and the leaf then stays 1 / leaf, more than a
// double's rounding, off the whole numbers it does not meet.  FLT_EPSILON,
// which the growth rule takes off a cube whatever the leaf, is 2^(e - 23) units
// (so e is at least 23, with a shorter range) and has to be a small part of a
// leaf.  A fixed unit of 2^-40 held clouds in metres only: 120 x 400 keypoints,
// 48,000 pairs, took 1.96 ms in metres and 96 in centimetres or millimetres, a
// CTA a pair; 1.9 in all three now (kilometres 3.4).
struct RefUnit {
  float up, down;  // 2^e, 2^-e
  float lim;       // largest coordinate taken (negative: none)
  long long eps;   // FLT_EPSILON in units
};
static RefUnit ref_unit(float res) {
  RefUnit u{1.f, 1.f, -1.f, 0};
  if (!(res >= 1.0e-6f && res <= 0x1p20f)) return u;
  int e = 33 - ilogbf(res);
  if (e < 23) e = 23;
  u.up = ldexpf(1.f, e);
  u.down = ldexpf(1.f, -e);
  u.lim = fminf(ldexpf(res, REFW_RANGE_LOG2), ldexpf(1.f, 51 - e));
  u.eps = 1ll << (e - 23);
  return u;
}

struct RefKeyBox {
  long long mn[3], mx[3];  // the field cube, in units
  float M[6];              // the yaw step about the keypoint: x and y rows, columns 0, 1, 3
  int J[3];                // field coordinate of key k: k + J, truncated toward zero
  int depth, ok, table;    // table: J is not certain, coordinates come from doubles
};

__device__ __forceinline__ long long to_fix(float x, const RefUnit& u) { return __float2ll_rd(x * u.up); }
__device__ __forceinline__ float from_fix_rn(long long v, const RefUnit& u) { return __ll2float_rn(v) * u.down; }
__device__ __forceinline__ float from_fix_ru(long long v, const RefUnit& u) { return __ll2float_ru(v) * u.down; }

__device__ __forceinline__ float warp_min(float x) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float warp_max(float x) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
  return r;
}

// Size classes of the warp form: rows of 32 points.  The last two take the
// clouds whose field coordinates come from a table.
constexpr int REFW_CLASSES = 11;
__host__ __device__ constexpr int refw_rows(int c) {
  constexpr int rows[REFW_CLASSES] = {1, 2, 3, 4, 5, 6, 8, 12, 16, 8, 16};
  return rows[c];
}
__host__ __device__ constexpr int refw_blocks(int c) {  // resident blocks wanted an SM
  return refw_rows(c) <= 2 ? 8 : (refw_rows(c) <= 5 ? 6 : (refw_rows(c) <= 8 ? 5 : 2));
}
__device__ __forceinline__ int refw_class(int n, bool table) {  // n <= REFW_MAX
  int c = table ? 9 : 0;
  while (n > 32 * refw_rows(c)) ++c;
  return c;
}

// Field cube, yaw step and field offsets of every model keypoint; the keys of
// each size class into list[class][n], their number into cls[class].
__global__ void k_ref_keybox(const float4* __restrict__ mkeys, const int* __restrict__ moff, int n, float res,
                             float half, RefUnit un, RefRot rot, RefKeyBox* __restrict__ out,
                             int* __restrict__ list, int* __restrict__ cls) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n) return;
  const int np = moff[m + 1] - moff[m];
  const float4 km = mkeys[m];
  RefKeyBox k;
  const double dres = (double)res;
  const float lim = un.lim;
  const double up = (double)un.up, down = (double)un.down;
  bool ok = half <= lim && fabsf(km.x) <= lim && fabsf(km.y) <= lim && fabsf(km.z) <= lim;  // false for NaN
  const long long r64 = ok ? to_fix(res, un) : 1;
  ok = ok && from_fix_rn(r64, un) == res;
  const float lo[3] = {__fsub_rn(km.x, half), __fsub_rn(km.y, half), __fsub_rn(km.z, half)};
  const float hi[3] = {__fadd_rn(km.x, half), __fadd_rn(km.y, half), __fadd_rn(km.z, half)};
  OctBox b;
  b.depth = 0;
  if (ok) oct_define(b, lo, hi, dres);
  k.table = 0;
  for (int a = 0; a < 3; ++a) {
    k.mn[a] = k.mx[a] = 0;
    k.J[a] = 0;
    if (!ok) continue;
    k.mn[a] = __double2ll_rd(b.mn[a] * up);
    k.mx[a] = __double2ll_rd(b.mx[a] * up);
    ok = ok && (double)k.mn[a] * down == b.mn[a] && (double)k.mx[a] * down == b.mx[a] &&
         from_fix_rn(to_fix(lo[a], un), un) == lo[a] && llabs(k.mx[a] - k.mn[a] - (r64 << b.depth)) <= un.eps;
    // the field coordinate (centre of leaf k - lo) / res = k + num / (2 res):
    // its whole part is certain while the fraction stays clear of 0 and 1
    // (rounding moves it by less than 0.05 in the range)
    const long long num = 2 * (k.mn[a] - to_fix(lo[a], un)) + r64, den = 2 * r64;
    long long q = num / den;
    if (q * den > num) --q;
    const long long fr = num - q * den;
    if (fr * 20 < den * 3 || fr * 20 > den * 17) k.table = 1;
    k.J[a] = (int)q;
  }
  float T1[16], T3[16], M[16], Rs[16];
  eye4(T1);
  T1[3] = -km.x, T1[7] = -km.y;
  eye4(T3);
  T3[3] = km.x, T3[7] = km.y;
  eye4(Rs);
  Rs[0] = rot.c1, Rs[4] = rot.s1, Rs[1] = -rot.s1, Rs[5] = rot.c1;
  mm4(T3, Rs, M);
  mm4(M, T1, M);
  // a turn about a vertical axis: z stays, and x and y take nothing from it
  ok = ok && M[2] == 0.f && M[6] == 0.f && M[8] == 0.f && M[9] == 0.f && M[10] == 1.f && M[11] == 0.f;
  k.M[0] = M[0], k.M[1] = M[1], k.M[2] = M[3], k.M[3] = M[4], k.M[4] = M[5], k.M[5] = M[7];
  k.depth = b.depth;
  k.ok = ok;
  out[m] = k;
  if (np <= REFW_MAX) {
    const int c = refw_class(np, k.table != 0);
    list[(size_t)c * n + atomicAdd(cls + c, 1)] = m;
  }
}

// floor((p - mn) / res) as the reference's doubles give it; est is within a
// few of it.  p lies in the cube.
__device__ __forceinline__ int ref_key_exact(float p, long long mn, long long r64, double dres, int est,
                                             const RefUnit& un) {
  const long long P = to_fix(p, un);
  if (from_fix_rn(P, un) == p) {
    long long r = P - mn - (long long)est * r64;
    while (r < 0) --est, r += r64;
    while (r >= r64) ++est, r -= r64;
    return est;
  }
  return (int)__double2uint_rz(__ddiv_rn(__dsub_rn((double)p, (double)mn * (double)un.down), dres));
}

// Ascending sort of 32 Q words, word i = lane * Q + q: runs of Q sorted in
// each lane, then merged pairwise five times.  A merge compares the runs head
// to tail (lower lanes keep the smaller words), halves the bitonic rest lane
// against lane, and sorts the bitonic Q left in each lane; the halving needs
// only even lengths, so Q need not be a power of two.
__device__ __forceinline__ void cmp_swap(unsigned& a, unsigned& b) {
  const unsigned lo = min(a, b);
  b = max(a, b);
  a = lo;
}
template <int Q, int O, int N>
__device__ __forceinline__ void lane_bitonic(unsigned (&x)[Q]) {  // words O .. O + N - 1, bitonic (any order if N is odd)
  if constexpr (N == 3) {
    cmp_swap(x[O], x[O + 1]);
    cmp_swap(x[O + 1], x[O + 2]);
    cmp_swap(x[O], x[O + 1]);
  } else if constexpr (N == 5) {
    cmp_swap(x[O], x[O + 3]);
    cmp_swap(x[O + 1], x[O + 4]);
    cmp_swap(x[O], x[O + 2]);
    cmp_swap(x[O + 1], x[O + 3]);
    cmp_swap(x[O], x[O + 1]);
    cmp_swap(x[O + 2], x[O + 4]);
    cmp_swap(x[O + 1], x[O + 2]);
    cmp_swap(x[O + 3], x[O + 4]);
    cmp_swap(x[O + 2], x[O + 3]);
  } else if constexpr (N > 1) {
    static_assert(N % 2 == 0, "half-cleaner");
#pragma unroll
    for (int i = 0; i < N / 2; ++i) cmp_swap(x[O + i], x[O + N / 2 + i]);
    lane_bitonic<Q, O, N / 2>(x);
    lane_bitonic<Q, O + N / 2, N / 2>(x);
  }
}
template <int Q, int O, int N>
__device__ __forceinline__ void lane_sort(unsigned (&x)[Q]) {
  if constexpr (N == 3 || N == 5) {
    lane_bitonic<Q, O, N>(x);
  } else if constexpr (N > 1) {
    lane_sort<Q, O, N / 2>(x);
    lane_sort<Q, O + N / 2, N / 2>(x);
#pragma unroll
    for (int i = 0; i < N / 2; ++i) cmp_swap(x[O + i], x[O + N - 1 - i]);
    lane_bitonic<Q, O, N / 2>(x);
    lane_bitonic<Q, O + N / 2, N / 2>(x);
  }
}
template <int Q>
__device__ __forceinline__ void warp_sort(unsigned (&x)[Q], int lane) {
  lane_sort<Q, 0, Q>(x);
#pragma unroll
  for (int m = 1; m <= 5; ++m) {
    {
      const int d = (1 << m) - 1;
      const bool low = (lane & (1 << (m - 1))) == 0;
      unsigned v[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) v[q] = __shfl_xor_sync(0xffffffffu, x[Q - 1 - q], d);
#pragma unroll
      for (int q = 0; q < Q; ++q) x[q] = low ? min(x[q], v[q]) : max(x[q], v[q]);
    }
#pragma unroll
    for (int d = 1 << (m - 1) >> 1; d > 0; d >>= 1) {
      const bool low = (lane & d) == 0;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const unsigned v = __shfl_xor_sync(0xffffffffu, x[q], d);
        x[q] = low ? min(x[q], v) : max(x[q], v);
      }
    }
    lane_bitonic<Q, 0, Q>(x);
  }
}

// One 4x4 product, element lane = 4 r + c in lanes 0..15 (mm4's order).
__device__ __forceinline__ float warp_mm4(float A, float B, int lane) {
  const int r = (lane >> 2) & 3, c = lane & 3;
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float t = __fmul_rn(__shfl_sync(0xffffffffu, A, 4 * r + k), __shfl_sync(0xffffffffu, B, 4 * k + c));
    s = k == 0 ? t : __fadd_rn(s, t);
  }
  return s;
}

// Pairs of size class CLS: all scan keypoints against the n_items / ns model
// keypoints in list, or, with a pair list, its pairs of this class.
template <int CLS>
__global__ void __launch_bounds__(32 * REFW_WARPS, refw_blocks(CLS))
    k_ref_distance_warp(const float4* __restrict__ mcloud, const float4* __restrict__ mkeys,
                        const int* __restrict__ moff, const int* __restrict__ midx, const float* __restrict__ mtdf,
                        const RefKeyBox* __restrict__ boxes, const int* __restrict__ list,
                        const float4* __restrict__ skeys, int ns, const int* __restrict__ pair_m,
                        const int* __restrict__ pair_s, long long n_items, float res, float half, RefUnit un,
                        RefRot rot, float* __restrict__ score, float* __restrict__ Tout, int* __restrict__ err) {
  constexpr int Q = refw_rows(CLS);
  constexpr bool TABLE = CLS >= 9;
  __shared__ unsigned s_bm[REFW_WARPS][REF_WIN * REF_WIN];  // leaves of a cloud that reads no field value
  __shared__ __align__(16) float s_v[REFW_WARPS][32 * Q];
  __shared__ unsigned s_ord[REFW_WARPS][3][64];             // order code of a local key, by axis, above the point index
  __shared__ int s_fld[TABLE ? REFW_WARPS : 1][3][64];      // its share of the field index
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long p = (long long)blockIdx.x * REFW_WARPS + w;
  if (p >= n_items) return;
  int m, sk;
  if (pair_m) {
    m = pair_m[p], sk = pair_s[p];
    const int np = moff[m + 1] - moff[m];
    if (np > REFW_MAX || refw_class(np, boxes[m].table != 0) != CLS) return;
  } else {
    m = list[p / ns], sk = (int)(p % ns);
    p = (long long)m * ns + sk;
  }
  const int beg = moff[m], n = moff[m + 1] - beg;
  const float4 km = mkeys[m], ks = skeys[sk];
  float* To = Tout + 16 * p;
  if (!(isfinite(km.x) && isfinite(km.y) && isfinite(km.z) && isfinite(ks.x) && isfinite(ks.y) && isfinite(ks.z))) {
    if (lane == 0) score[p] = __int_as_float(0x7fc00000);
    if (lane < 16) To[lane] = (lane % 5) == 0 ? 1.f : 0.f;
    return;
  }
  const RefKeyBox* kb = boxes + m;
  const float lim = un.lim;
  const float tx = __fsub_rn(km.x, ks.x), ty = __fsub_rn(km.y, ks.y), tz = __fsub_rn(km.z, ks.z);
  float px[Q], py[Q], pz[Q];
  bool fine = kb->ok != 0;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int j = lane + 32 * q;
    px[q] = py[q] = pz[q] = 0.f;
    if (n > 0) {  // rows past the cloud repeat its first point: the same leaf
      const float4 c = mcloud[midx[beg + (j < n ? j : 0)]];
      px[q] = __fadd_rn(c.x, tx), py[q] = __fadd_rn(c.y, ty), pz[q] = __fadd_rn(c.z, tz);
      fine = fine && fabsf(c.x) <= lim && fabsf(c.y) <= lim && fabsf(c.z) <= lim && fabsf(px[q]) <= lim &&
             fabsf(py[q]) <= lim && fabsf(pz[q]) <= lim;
    }
  }
  if (!__all_sync(0xffffffffu, fine)) {
    if (lane == 0) {
      To[15] = __uint_as_float(REFW_REDO);
      atomicAdd(err + 2, 1);
    }
    return;
  }
  const float* grid = mtdf + (size_t)m * REF_VOL;
  const double dres = (double)res;
  const float inv = __fdiv_rn(1.f, res);
  const long long r64 = to_fix(res, un), eps64 = un.eps;
  const int ax = lane % 3;                               // this lane's axis
  const long long mn0 = kb->mn[ax], mx0 = kb->mx[ax];
  const int J = kb->J[ax], stride = ax == 0 ? 1 : (ax == 1 ? REF_DIM : REF_DIM * REF_DIM);
  const int J0 = kb->J[0], J1 = kb->J[1], J2 = kb->J[2];
  const int depth0 = kb->depth;
  const float m0 = kb->M[0], m1 = kb->M[1], m3 = kb->M[2], m4 = kb->M[3], m5 = kb->M[4], m7 = kb->M[5];
  float zmn = pz[0], zmx = pz[0], far = 0.f;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    zmn = fminf(zmn, pz[q]), zmx = fmaxf(zmx, pz[q]);
    far = fmaxf(far, fabsf(px[q] - km.x) + fabsf(py[q] - km.y));
  }
  zmn = warp_min(zmn), zmx = warp_max(zmx), far = warp_max(far);
  // leaf coordinates: y = (p - mn0) / res - 1/2 by one FMA, off by at most
  // 2^-22 (|c| + |y|); rounding it to a whole number gives the leaf (counted
  // from the field cube's corner) unless y is more than `sure` from it
  const float c_a = -(from_fix_rn(mn0, un) * inv) - 0.5f;
  const float reach = ((ax == 0 ? fabsf(km.x) : (ax == 1 ? fabsf(km.y) : 0.f)) +
                       (ax == 2 ? fmaxf(fabsf(zmn), fabsf(zmx)) : 1.01f * far)) * inv;
  const float sure = 0.5f - warp_max((2.f * fabsf(c_a) + reach + 2.f) * 0x1p-22f + 2.5e-7f * inv);
  const float c0 = __shfl_sync(0xffffffffu, c_a, 0), c1 = __shfl_sync(0xffffffffu, c_a, 1),
              c2 = __shfl_sync(0xffffffffu, c_a, 2);
  constexpr float MAGIC = 12582912.f;  // 1.5 * 2^23: adding it rounds to a whole number, in the low bits
  constexpr int MBITS = 0x4b400000;
  const float zfirst = __shfl_sync(0xffffffffu, pz[0], 0);
  unsigned spread = 0;  // the lane's five bits, every third
#pragma unroll
  for (int i = 0; i < 5; ++i) spread |= ((unsigned)lane >> i & 1u) << (3 * i);
#pragma unroll
  for (int a = 0; a < 3; ++a) s_ord[w][a][lane] = spread << (9 + 2 - a);
  for (int i = lane; i < REF_WIN * REF_WIN; i += 32) s_bm[w][i] = 0u;
  __syncwarp();
  float dtf = 0.f, bestf = 100000000.f;
  int best_i = 0;
  bool bad = false;
  for (int it = 0; it < 36; ++it) {
    if (it != 0) {
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const float x = __fadd_rn(__fadd_rn(__fmul_rn(m0, px[q]), __fmul_rn(m1, py[q])), m3);
        const float y = __fadd_rn(__fadd_rn(__fmul_rn(m4, px[q]), __fmul_rn(m5, py[q])), m7);
        px[q] = x, py[q] = y;
      }
    }
    int u = 0;
    if (n > 0) {
      float xmn = px[0], xmx = px[0], ymn = py[0], ymx = py[0];
#pragma unroll
      for (int q = 1; q < Q; ++q) {
        xmn = fminf(xmn, px[q]), xmx = fmaxf(xmx, px[q]);
        ymn = fminf(ymn, py[q]), ymx = fmaxf(ymx, py[q]);
      }
      xmn = warp_min(xmn), xmx = warp_max(xmx), ymn = warp_min(ymn), ymx = warp_max(ymx);
      const float amn = ax == 0 ? xmn : (ax == 1 ? ymn : zmn), amx = ax == 0 ? xmx : (ax == 1 ? ymx : zmx);
      // this axis: leaves of the cloud's box; K, depth: the grown cube is
      // leaves [-K, -K + 2^depth)
      int kmn, kmx, K = 0, depth = depth0;
      bool near;
      {
        const float y0 = __fmaf_rn(amn, inv, c_a), y1 = __fmaf_rn(amx, inv, c_a);
        const float t0 = __fadd_rn(y0, MAGIC), t1 = __fadd_rn(y1, MAGIC);
        kmn = __float_as_int(t0) - MBITS, kmx = __float_as_int(t1) - MBITS;
        near = fabsf(__fsub_rn(y0, __fsub_rn(t0, MAGIC))) > sure || fabsf(__fsub_rn(y1, __fsub_rn(t1, MAGIC))) > sure;
      }
      near = __any_sync(0xffffffffu, near);
      // growth: the first point outside (in index order) grows the cube until
      // it fits, until no point is outside.  Away from whole numbers the
      // leaves decide (the bounds are whole, up to the FLT_EPSILON that
      // `sure` covers)
      for (int round = 0; !near && round < 2 * REF_MAX_DEPTH; ++round) {
        if (!__any_sync(0xffffffffu, kmn < -K || kmx >= (1 << depth) - K)) break;
        float sx = __shfl_sync(0xffffffffu, px[0], 0), sy = __shfl_sync(0xffffffffu, py[0], 0), sz = zfirst;
        float yp = __fmaf_rn(ax == 0 ? sx : (ax == 1 ? sy : sz), inv, c_a);
        float tp = __fadd_rn(yp, MAGIC);
        int ip = __float_as_int(tp) - MBITS;
        if (!__any_sync(0xffffffffu, ip < -K || ip >= (1 << depth) - K)) {
          // the first point that is outside or too near a bound to tell
          const float flo = (float)-K - sure, fhi = (float)((1 << depth) - K) - 1.f + sure;
          const float lo0 = __shfl_sync(0xffffffffu, flo, 0), lo1 = __shfl_sync(0xffffffffu, flo, 1),
                      lo2 = __shfl_sync(0xffffffffu, flo, 2), hi0 = __shfl_sync(0xffffffffu, fhi, 0),
                      hi1 = __shfl_sync(0xffffffffu, fhi, 1), hi2 = __shfl_sync(0xffffffffu, fhi, 2);
          unsigned first = ~0u;
#pragma unroll
          for (int q = Q - 1; q >= 0; --q) {
            const float y0 = __fmaf_rn(px[q], inv, c0), y1 = __fmaf_rn(py[q], inv, c1), y2 = __fmaf_rn(pz[q], inv, c2);
            if (y0 < lo0 || y0 > hi0 || y1 < lo1 || y1 > hi1 || y2 < lo2 || y2 > hi2) first = (unsigned)(lane + 32 * q);
          }
          first = __reduce_min_sync(0xffffffffu, first);
          const unsigned q0 = first >> 5;
#pragma unroll
          for (int q = 0; q < Q; ++q)
            if ((unsigned)q == q0) sx = px[q], sy = py[q], sz = pz[q];
          const int src = (int)(first & 31u);
          sx = __shfl_sync(0xffffffffu, sx, src);
          sy = __shfl_sync(0xffffffffu, sy, src);
          sz = __shfl_sync(0xffffffffu, sz, src);
          yp = __fmaf_rn(ax == 0 ? sx : (ax == 1 ? sy : sz), inv, c_a);
          tp = __fadd_rn(yp, MAGIC);
          ip = __float_as_int(tp) - MBITS;
        }
        near = __any_sync(0xffffffffu, fabsf(__fsub_rn(yp, __fsub_rn(tp, MAGIC))) > sure);
        while (!near && !bad) {
          const bool up = ip >= (1 << depth) - K;
          if (!__any_sync(0xffffffffu, up || ip < -K)) break;
          if (!up) K += 1 << depth;
          bad = ++depth > REF_MAX_DEPTH;
        }
        if (bad) break;
      }
      if (near && !bad) {
        // some point decides the growth from close to a whole leaf: the same in
        // whole units of 2^-40 m
        long long mn = mn0, mx = mx0;
        const long long bmn = to_fix(amn, un), bmx = to_fix(amx, un);
        K = 0, depth = depth0;
        for (int round = 0; !bad && round < 2 * REF_MAX_DEPTH && __any_sync(0xffffffffu, bmn < mn || bmx >= mx); ++round) {
          const float fmn = from_fix_ru(mn, un), fmx = from_fix_ru(mx, un);
          OctBoxF bf;
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            bf.mn_up[a] = __shfl_sync(0xffffffffu, fmn, a);
            bf.mx_up[a] = __shfl_sync(0xffffffffu, fmx, a);
          }
          unsigned first = ~0u;
#pragma unroll
          for (int q = Q - 1; q >= 0; --q)
            if (oct_outside_f(bf, px[q], py[q], pz[q])) first = (unsigned)(lane + 32 * q);
          first = __reduce_min_sync(0xffffffffu, first);
          const unsigned q0 = first >> 5;
          float sx = 0.f, sy = 0.f, sz = 0.f;
#pragma unroll
          for (int q = 0; q < Q; ++q)
            if ((unsigned)q == q0) sx = px[q], sy = py[q], sz = pz[q];
          const int src = (int)(first & 31u);
          sx = __shfl_sync(0xffffffffu, sx, src);
          sy = __shfl_sync(0xffffffffu, sy, src);
          sz = __shfl_sync(0xffffffffu, sz, src);
          const long long P = to_fix(ax == 0 ? sx : (ax == 1 ? sy : sz), un);
          while (!bad && __any_sync(0xffffffffu, P < mn || P >= mx)) {
            if (P < mx) {
              mn -= r64 << depth;
              K += 1 << depth;
            }
            bad = ++depth > REF_MAX_DEPTH;
            mx = mn + (r64 << depth) - eps64;
          }
        }
        kmn = ref_key_exact(amn, mn, r64, dres, kmn + K, un) - K;
        kmx = ref_key_exact(amx, mn, r64, dres, kmx + K, un) - K;
      }
      if (bad) break;
      if (__any_sync(0xffffffffu, kmx - kmn >= REF_WIN)) {
        if (lane == 0) atomicOr(err, REF_ERR_WINDOW);
      } else {
        // the field index's range over the cloud's box: nothing to read when
        // it lies outside the field, and then the leaves' order does not
        // matter either (every value is 900)
        int flo = kmn + J, fhi = kmx + J;
        flo = (flo + (flo < 0)) * stride, fhi = (fhi + (fhi < 0)) * stride;
        flo = lane < 3 ? flo : 0, fhi = lane < 3 ? fhi : 0;
        const bool inside =
            TABLE || (__reduce_add_sync(0xffffffffu, fhi) >= 0 && __reduce_add_sync(0xffffffffu, flo) < REF_VOL);
        // local keys: from a multiple of 32 of the cube's keys at or below the
        // lowest (0..63), or from the lowest (0..31)
        const int base = inside ? ((kmn + K) & ~31) - K : kmn;
        const int b0 = __shfl_sync(0xffffffffu, base, 0), b1 = __shfl_sync(0xffffffffu, base, 1),
                  b2 = __shfl_sync(0xffffffffu, base, 2);
        if (inside) {
          const unsigned B = (unsigned)((kmn + K) >> 5), chg = B ^ (B + 1u);  // bits that a crossing changes
          const unsigned cx = __shfl_sync(0xffffffffu, chg, 0), cy = __shfl_sync(0xffffffffu, chg, 1),
                         cz = __shfl_sync(0xffffffffu, chg, 2);
          s_ord[w][0][lane + 32] = (spread << 11) | (1u << (24 + (cx >= cy) + (cx >= cz)));
          s_ord[w][1][lane + 32] = (spread << 10) | (1u << (24 + (cy > cx) + (cy >= cz)));
          s_ord[w][2][lane + 32] = (spread << 9) | (1u << (24 + (cz > cx) + (cz > cy)));
          if constexpr (TABLE) {
#pragma unroll 1
            for (int a = 0; a < 3; ++a) {
              const int ba = a == 0 ? b0 : (a == 1 ? b1 : b2);
              const int st = a == 0 ? 1 : (a == 1 ? REF_DIM : REF_DIM * REF_DIM);
              const float lo = __fsub_rn(a == 0 ? km.x : (a == 1 ? km.y : km.z), half);
              const double dmn = (double)__shfl_sync(0xffffffffu, mn0, a) * (double)un.down;
#pragma unroll 1
              for (int l = lane; l < 64; l += 32) {
                const float e = __double2float_rn(__dadd_rn(__dmul_rn(__dadd_rn((double)(ba + l), 0.5), dres), dmn));
                s_fld[TABLE ? w : 0][a][l] = __float2int_rz(__fdiv_rn(__fsub_rn(e, lo), res)) * st;
              }
            }
          }
          __syncwarp();
        }
        // one point: its sort word and squared field value, or its leaf's bit
        const bool neg = __any_sync(0xffffffffu, kmn + J < 0);  // some field coordinate is truncated upward
        auto place = [&](int j, int i0, int i1, int i2, float* sq) -> unsigned {
          const int l0 = (i0 - b0) & 63, l1 = (i1 - b1) & 63, l2 = (i2 - b2) & 63;
          int idx;
          if constexpr (TABLE) {
            idx = s_fld[TABLE ? w : 0][0][l0] + s_fld[TABLE ? w : 0][1][l1] + s_fld[TABLE ? w : 0][2][l2];
          } else {
            int f0 = i0 + J0, f1 = i1 + J1, f2 = i2 + J2;
            if (neg) f0 += f0 < 0, f1 += f1 < 0, f2 += f2 < 0;
            idx = f0 + REF_DIM * f1 + REF_DIM * REF_DIM * f2;
          }
          const float v = (unsigned)idx < (unsigned)REF_VOL ? __ldg(grid + idx) : 900.f;
          *sq = __fmul_rn(v, v);
          return j < n ? s_ord[w][0][l0] + s_ord[w][1][l1] + s_ord[w][2][l2] + (unsigned)j : ~0u;
        };
        auto mark = [&](int i0, int i1, int i2, bool* fresh) -> unsigned {
          const unsigned wd = (unsigned)(((i1 - b1) & 31) + REF_WIN * ((i2 - b2) & 31)), bit = 1u << ((i0 - b0) & 31);
          *fresh = (atomicOr(&s_bm[w][wd], bit) & bit) == 0u;
          return wd;
        };
        unsigned word[Q], close = 0u;  // close: bit q, point too near a whole leaf
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const int j = lane + 32 * q;
          const float y0 = __fmaf_rn(px[q], inv, c0), y1 = __fmaf_rn(py[q], inv, c1), y2 = __fmaf_rn(pz[q], inv, c2);
          const float t0 = __fadd_rn(y0, MAGIC), t1 = __fadd_rn(y1, MAGIC), t2 = __fadd_rn(y2, MAGIC);
          const bool c = fabsf(__fsub_rn(y0, __fsub_rn(t0, MAGIC))) > sure ||
                         fabsf(__fsub_rn(y1, __fsub_rn(t1, MAGIC))) > sure ||
                         fabsf(__fsub_rn(y2, __fsub_rn(t2, MAGIC))) > sure;
          if (c && j < n) close |= 1u << q;
          const int i0 = __float_as_int(t0) - MBITS, i1 = __float_as_int(t1) - MBITS, i2 = __float_as_int(t2) - MBITS;
          if (inside) {
            float sq;
            word[q] = place(j, i0, i1, i2, &sq);
            s_v[w][j] = sq;
          } else {
            bool fresh = false;
            word[q] = 0u;
            if (!c && j < n) word[q] = mark(i0, i1, i2, &fresh);
            u += __popc(__ballot_sync(0xffffffffu, fresh));
          }
        }
        while (__any_sync(0xffffffffu, close != 0u)) {
          const int qq = close ? __ffs(close) - 1 : Q;
          float x = 0.f, y = 0.f, z = 0.f;
#pragma unroll
          for (int q = 0; q < Q; ++q)
            if (q == qq) x = px[q], y = py[q], z = pz[q];
          int i[3];
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const long long mna = __shfl_sync(0xffffffffu, mn0 - (long long)K * r64, a);
            const int ka = __shfl_sync(0xffffffffu, K, a);
            const float pa = a == 0 ? x : (a == 1 ? y : z), ca = a == 0 ? c0 : (a == 1 ? c1 : c2);
            i[a] = 0;
            if (close) i[a] = ref_key_exact(pa, mna, r64, dres, __float2int_rn(__fmaf_rn(pa, inv, ca)) + ka, un) - ka;
          }
          bool fresh = false;
          if (close) {
            unsigned wd;
            if (inside) {
              float sq;
              wd = place(lane + 32 * qq, i[0], i[1], i[2], &sq);
              s_v[w][lane + 32 * qq] = sq;
            } else {
              wd = mark(i[0], i[1], i[2], &fresh);
            }
#pragma unroll
            for (int q = 0; q < Q; ++q) word[q] = q == qq ? wd : word[q];
          }
          u += __popc(__ballot_sync(0xffffffffu, fresh));
          close &= close - 1u;
        }
        if (!inside) {
          __syncwarp();
#pragma unroll
          for (int q = 0; q < Q; ++q) s_bm[w][word[q]] = 0u;
#pragma unroll 8
          for (int i = 1; i < u; ++i) dtf = __fadd_rn(dtf, 810000.f);
        } else {
          warp_sort<Q>(word, lane);
          __syncwarp();
          // distinct leaves after the first keep their value
          const unsigned prev = __shfl_up_sync(0xffffffffu, word[Q - 1], 1);
          float val[Q];
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            const unsigned before = q == 0 ? prev : word[q > 0 ? q - 1 : 0];
            const bool head = (q == 0 && lane == 0) || (word[q] >> 9) != (before >> 9);
            const bool leaf = head && word[q] != ~0u;
            u += __popc(__ballot_sync(0xffffffffu, leaf));
            val[q] = leaf && !(q == 0 && lane == 0) ? s_v[w][word[q] & 511u] : 0.f;
          }
          __syncwarp();
#pragma unroll
          for (int q = 0; q < Q; ++q) s_v[w][lane * Q + q] = val[q];
          __syncwarp();
          const float4* sv = reinterpret_cast<const float4*>(s_v[w]);
          const int n4 = (n + 3) >> 2;
#pragma unroll 4
          for (int i = 0; i < n4; ++i) {
            const float4 v = sv[i];
            dtf = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(dtf, v.x), v.y), v.z), v.w);
          }
        }
        __syncwarp();
      }
    }
    dtf = __fdiv_rn(dtf, u == 0 ? 18446744073709551616.f : (float)(u - 1));
    if (dtf < bestf) {
      bestf = dtf;
      best_i = it;
    }
  }
  if (bad) {  // past REF_MAX_DEPTH levels (the range keeps clouds below it)
    if (lane == 0) {
      To[15] = __uint_as_float(REFW_REDO);
      atomicAdd(err + 2, 1);
    }
    return;
  }
  if (lane == 0) score[p] = bestf;
  // S T3 R2 T1 Tm, one element a lane
  const int r = (lane >> 2) & 3, c = lane & 3;
  const float one = r == c ? 1.f : 0.f;
  const float cs = __fdiv_rn(km.z, ks.z);
  float A = r == c && r < 3 ? cs : one;
  A = warp_mm4(A, lane == 3 ? km.x : (lane == 7 ? km.y : one), lane);
  const float rc = rot.c2[best_i], rs = rot.s2[best_i];
  A = warp_mm4(A, lane == 0 || lane == 5 ? rc : (lane == 4 ? rs : (lane == 1 ? -rs : one)), lane);
  A = warp_mm4(A, lane == 3 ? -km.x : (lane == 7 ? -km.y : one), lane);
  A = warp_mm4(A, lane == 3 ? tx : (lane == 7 ? ty : (lane == 11 ? tz : one)), lane);
  if (lane < 16) To[lane] = A;
}

__global__ void k_ref_sum_counts(const uint32_t* __restrict__ cnt, int n, unsigned long long* __restrict__ out) {
  unsigned long long v = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) v += cnt[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(out, v);
}

__global__ void k_ref_max_count(const int* __restrict__ off, int n, int* __restrict__ out) {
  int v = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    v = max(v, off[i + 1] - off[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) atomicMax(out, v);
}

// ---------------------------------------------------------------------------
// the all-pairs loop's gates (function.h:158-178, as written)
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool ref_gates(float4 km, int mnum, const double* mv3, float4 ks, int snum,
                                          const double* sv3) {
  const float h = __fdiv_rn(km.z, ks.z);
  if (!(h >= 0.f || h <= 1.5f)) return false;
  for (int a = 0; a < 3; ++a) {
    const double r = __ddiv_rn(mv3 ? mv3[a] : 0.16, sv3 ? sv3[a] : 0.16);
    if (r > 3.0 || r < 0.0) return false;
  }
  if (snum == 0) return false;
  const float q = (float)(mnum / snum);
  return !(q > 2.f || q < 0.5f);
}

__global__ void k_ref_gates(const float4* __restrict__ mkeys, const int* __restrict__ mnum,
                            const double* __restrict__ mv3, const float4* __restrict__ skeys,
                            const int* __restrict__ snum, const double* __restrict__ sv3, int ns, long long np,
                            const float* __restrict__ score, float max_score, uint32_t* __restrict__ flags) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < np; p += (long long)gridDim.x * blockDim.x) {
    const int m = (int)(p / ns), s = (int)(p % ns);
    flags[p] = (score[p] < max_score &&
                ref_gates(mkeys[m], mnum[m], mv3 ? mv3 + 3 * (size_t)m : nullptr, skeys[s], snum[s],
                          sv3 ? sv3 + 3 * (size_t)s : nullptr))
                   ? 1u
                   : 0u;
  }
}

__global__ void k_ref_scatter(const uint32_t* __restrict__ flags, const uint32_t* __restrict__ pos, long long np,
                              int cap, int* __restrict__ out) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < np; p += (long long)gridDim.x * blockDim.x)
    if (flags[p] && pos[p] < (uint32_t)cap) out[pos[p]] = (int)p;
}

// ---------------------------------------------------------------------------
// Ransac (function.h:35-109): inliers of every kept pair's transform
// ---------------------------------------------------------------------------
constexpr int RANSAC_NT = 256;

__global__ void __launch_bounds__(RANSAC_NT) k_ref_ransac(const float4* __restrict__ mkeys,
                                                          const float4* __restrict__ skeys, int ns,
                                                          const int* __restrict__ pair_idx, int np,
                                                          const float* __restrict__ score,
                                                          const float* __restrict__ T_all, float inlier,
                                                          float max_des, int* __restrict__ cnt) {
  __shared__ int s_c[RANSAC_NT / 32];
  const int i = blockIdx.x, tid = threadIdx.x;
  float Ti[12];
  const float* src = T_all + 16 * (size_t)pair_idx[i];
#pragma unroll
  for (int e = 0; e < 12; ++e) Ti[e] = src[e];
  int c = 0;
  for (int j = tid; j < np; j += RANSAC_NT) {
    const long long p = pair_idx[j];
    const int m = (int)(p / ns), s = (int)(p % ns);
    const float4 sk = skeys[s], k = mkeys[m];
    float x = sk.x, y = sk.y, z = sk.z;
    xf3(Ti, x, y, z);
    const float dx = __fsub_rn(k.x, x), dy = __fsub_rn(k.y, y), dz = __fsub_rn(k.z, z);
    const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    const float dis = __fsqrt_rn(d2);
    if ((double)dis < (double)inlier && score[p] < max_des) ++c;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((tid & 31) == 0) s_c[tid >> 5] = c;
  __syncthreads();
  if (tid == 0) {
    int t = 0;
    for (int w = 0; w < RANSAC_NT / 32; ++w) t += s_c[w];
    cnt[i] = t;
  }
}

// First position with the most inliers (> 0): out[0] = position or -1, out[1] = inliers.
__global__ void k_ref_argmax(const int* __restrict__ cnt, int np, int* __restrict__ out) {
  __shared__ int s_v[32], s_i[32];
  int bv = 0, bi = -1;
  for (int i = threadIdx.x; i < np; i += blockDim.x)
    if (cnt[i] > bv) bv = cnt[i], bi = i;  // ascending i per thread: first max kept
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int ov = __shfl_xor_sync(0xffffffffu, bv, o), oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > bv || (ov == bv && ov > 0 && oi < bi)) bv = ov, bi = oi;
  }
  if ((threadIdx.x & 31) == 0) s_v[threadIdx.x >> 5] = bv, s_i[threadIdx.x >> 5] = bi;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
      if (s_v[w] > bv || (s_v[w] == bv && bv > 0 && s_i[w] < bi)) bv = s_v[w], bi = s_i[w];
    out[0] = bv > 0 ? bi : -1;
    out[1] = bv;
  }
}

static RefRot ref_rot_tables() {
  RefRot r;
  const float theta = (float)(3.14159265358979323846 / 18);  // M_PI / 18 rounded to float
  r.c1 = cosf(theta);
  r.s1 = sinf(theta);
  for (int i = 0; i < 36; ++i) {
    const float th = (float)i * theta;
    r.c2[i] = (float)cos((double)th);
    r.s2[i] = (float)sin((double)th);
  }
  return r;
}

static rtr_status ref_read_ints(rtr_context* ctx, const int* d, int n, cudaStream_t st, int* h) {
  if (!ctx->h_pin || n > 64) return fail(RTR_ERR_CUDA, "rtr_ref: pinned staging missing");
  RTR_CUDA(cudaMemcpyAsync(ctx->h_pin, d, sizeof(int) * (size_t)n, cudaMemcpyDeviceToHost, st));
  RTR_CUDA(cudaStreamSynchronize(st));
  memcpy(h, ctx->h_pin, sizeof(int) * (size_t)n);
  return RTR_OK;
}

static rtr_status ref_check_err(int e, const char* who) {
  if (e & REF_ERR_DEPTH)
    return fail(RTR_ERR_INVALID_ARG, "%s: the box spans more than %d octree levels (half / res too large)", who,
                REF_OCC_DEPTH);
  if (e & REF_ERR_GROW)
    return fail(RTR_ERR_INVALID_ARG, "%s: occupancy points outside the field's box (occupancy box wider)", who);
  if (e & REF_ERR_WINDOW)
    return fail(RTR_ERR_INVALID_ARG, "%s: a rotated occupancy cloud spans more than %d leaves (occupancy box too "
                "wide for this resolution)", who, REF_WIN);
  return RTR_OK;
}

}  // namespace rtr

using namespace rtr;

extern "C" {

rtr_status rtr_ref_occupancy(rtr_context* ctx, const float* d_cloud, int n, const float* d_keys, int n_keys,
                             float resolution, float half_box, int32_t* d_number, int32_t* d_offsets,
                             int32_t* d_indices, long long cap_indices, long long* h_total, rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && n >= 0 && n_keys >= 0 && h_total, "rtr_ref_occupancy: bad arguments");
  RTR_CHECK_ARG(resolution > 0.f && half_box > 0.f && isfinite(resolution) && isfinite(half_box),
                "rtr_ref_occupancy: resolution and half_box must be positive");
  RTR_CHECK_ARG(2.0 * half_box / resolution <= 30.0, "rtr_ref_occupancy: half_box / resolution above 15");
  *h_total = 0;
  RTR_CHECK_ARG(d_offsets, "rtr_ref_occupancy: NULL offsets");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  if (n_keys == 0) {
    RTR_CUDA(cudaMemsetAsync(d_offsets, 0, sizeof(int32_t), st));
    RTR_CUDA(cudaStreamSynchronize(st));
    return RTR_OK;
  }
  RTR_CHECK_ARG(d_keys && d_number && (n == 0 || d_cloud), "rtr_ref_occupancy: NULL input");
  ScratchPlan plan;
  const size_t o_cnt = plan.add<uint32_t>((size_t)n_keys + 1);
  const size_t o_tiles = plan.add<uint32_t>((size_t)scan_tiles(n_keys + 1));
  const size_t o_err = plan.add<int>(4);
  const size_t o_tot = plan.add<unsigned long long>(1);
  Scratch s;
  RTR_TRY(ensure_scratch(ctx, plan.bytes, st, &s));
  uint32_t* cnt = reinterpret_cast<uint32_t*>(s.base + o_cnt);
  uint32_t* tiles = reinterpret_cast<uint32_t*>(s.base + o_tiles);
  int* err = reinterpret_cast<int*>(s.base + o_err);
  unsigned long long* tot64 = reinterpret_cast<unsigned long long*>(s.base + o_tot);
  ProfScope ps(ctx, st, "ref_occupancy");
  RTR_CUDA(cudaMemsetAsync(err, 0, 4 * sizeof(int), st));
  RTR_CUDA(cudaMemsetAsync(tot64, 0, sizeof(unsigned long long), st));
  RTR_CUDA(cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * ((size_t)n_keys + 1), st));
  const float4* cloud = reinterpret_cast<const float4*>(d_cloud);
  const float4* keys = reinterpret_cast<const float4*>(d_keys);
  k_ref_occ<<<n_keys, OCC_NT, 0, st>>>(cloud, n, keys, resolution, half_box, false, reinterpret_cast<int*>(cnt),
                                       d_number, nullptr, nullptr, err);
  // offsets = exclusive scan over n_keys + 1 counts (the last is 0): offsets[n_keys] = total
  scan_exclusive(cnt, reinterpret_cast<uint32_t*>(d_offsets), tiles, n_keys + 1, n_keys + 1, nullptr, nullptr, st);
  k_ref_sum_counts<<<(n_keys + 255) / 256 < 1024 ? (n_keys + 255) / 256 : 1024, 256, 0, st>>>(cnt, n_keys, tot64);
  RTR_LAUNCHED(3);
  int h[4];
  RTR_TRY(ref_read_ints(ctx, err, 4, st, h));
  RTR_TRY(ref_check_err(h[0], "rtr_ref_occupancy"));
  int h2[2];
  RTR_TRY(ref_read_ints(ctx, reinterpret_cast<const int*>(tot64), 2, st, h2));
  unsigned long long total64 = 0;
  memcpy(&total64, h2, sizeof(total64));
  const long long total = (long long)total64;
  *h_total = total;
  if (total > 0x7fffffffLL)
    return fail(RTR_ERR_CAPACITY, "rtr_ref_occupancy: %lld indices (offsets are 32-bit: at most 2^31 - 1)", total);
  if (total > cap_indices) return fail(RTR_ERR_CAPACITY, "rtr_ref_occupancy: %lld indices, capacity %lld", total,
                                       cap_indices);
  if (total > 0) {
    RTR_CHECK_ARG(d_indices, "rtr_ref_occupancy: NULL indices");
    k_ref_occ<<<n_keys, OCC_NT, 0, st>>>(cloud, n, keys, resolution, half_box, true, nullptr, nullptr, d_offsets,
                                         d_indices, err);
    RTR_LAUNCHED(1);
  }
  RTR_CUDA(cudaGetLastError());
  RTR_CUDA(cudaStreamSynchronize(st));
  return RTR_OK;
}

rtr_status rtr_ref_tdf(rtr_context* ctx, const float* d_cloud, const float* d_keys, int n_keys,
                       const int32_t* d_offsets, const int32_t* d_indices, float resolution, float half_tdf,
                       float* d_tdf, int* h_dim, rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && n_keys >= 0, "rtr_ref_tdf: bad arguments");
  RTR_CHECK_ARG(resolution > 0.f && half_tdf > 0.f && isfinite(resolution) && isfinite(half_tdf),
                "rtr_ref_tdf: resolution and half_tdf must be positive");
  const int dim = (int)(half_tdf / resolution * 2);  // key_point.h:313, in float
  RTR_CHECK_ARG(dim >= 1 && dim <= REF_DIM && 2.0 * half_tdf / resolution <= 31.0,
                "rtr_ref_tdf: dim %d outside [1, 30]", dim);
  if (h_dim) *h_dim = dim;
  if (n_keys == 0) return RTR_OK;
  RTR_CHECK_ARG(d_cloud && d_keys && d_offsets && d_tdf, "rtr_ref_tdf: NULL input or output");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  int h_last = 0;
  RTR_TRY(ref_read_ints(ctx, d_offsets + n_keys, 1, st, &h_last));
  RTR_CHECK_ARG(h_last >= 0, "rtr_ref_tdf: bad offsets");
  RTR_CHECK_ARG(h_last == 0 || d_indices, "rtr_ref_tdf: NULL indices");
  ScratchPlan plan;
  const size_t o_cnt = plan.add<uint32_t>((size_t)n_keys + 1);
  const size_t o_off = plan.add<uint32_t>((size_t)n_keys + 1);
  const size_t o_tiles = plan.add<uint32_t>((size_t)scan_tiles(n_keys + 1));
  const size_t o_err = plan.add<int>(4);
  const size_t o_occ = plan.add<int>(3 * (size_t)(h_last > 0 ? h_last : 1));
  Scratch s;
  RTR_TRY(ensure_scratch(ctx, plan.bytes, st, &s));
  uint32_t* cnt = reinterpret_cast<uint32_t*>(s.base + o_cnt);
  uint32_t* coff = reinterpret_cast<uint32_t*>(s.base + o_off);
  uint32_t* tiles = reinterpret_cast<uint32_t*>(s.base + o_tiles);
  int* err = reinterpret_cast<int*>(s.base + o_err);
  int* occ = reinterpret_cast<int*>(s.base + o_occ);
  ProfScope ps(ctx, st, "ref_tdf");
  RTR_CUDA(cudaMemsetAsync(err, 0, 4 * sizeof(int), st));
  RTR_CUDA(cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * ((size_t)n_keys + 1), st));
  const float4* cloud = reinterpret_cast<const float4*>(d_cloud);
  const float4* keys = reinterpret_cast<const float4*>(d_keys);
  k_ref_tdf_cells<<<n_keys, OCC_NT, 0, st>>>(cloud, keys, d_offsets, d_indices, resolution, half_tdf, false,
                                             reinterpret_cast<int*>(cnt), nullptr, nullptr, err);
  scan_exclusive(cnt, coff, tiles, n_keys + 1, n_keys + 1, nullptr, nullptr, st);
  k_ref_tdf_cells<<<n_keys, OCC_NT, 0, st>>>(cloud, keys, d_offsets, d_indices, resolution, half_tdf, true,
                                             nullptr, reinterpret_cast<const int*>(coff), occ, err);
  RTR_LAUNCHED(3);
  int h[4];
  RTR_TRY(ref_read_ints(ctx, err, 4, st, h));
  RTR_TRY(ref_check_err(h[0], "rtr_ref_tdf"));
  RTR_TRY(rtr_tdf_batch(ctx, occ, reinterpret_cast<const int*>(coff), n_keys, dim, d_tdf, stream));
  RTR_CUDA(cudaStreamSynchronize(st));
  return RTR_OK;
}

}  // extern "C"

// Dynamic shared memory of k_ref_distance<NT>: the sort list of a rotation's
// distinct leaves, 8-byte codes and 4-byte values, one per cloud point.
static size_t ref_leaf_smem(int nt) { return (size_t)nt * REF_PPT * (sizeof(unsigned long long) + sizeof(float)); }

template <int NT>
static rtr_status ref_distance_smem() {
  // the attribute is per function and device; setting it again is harmless
  RTR_CUDA(cudaFuncSetAttribute(k_ref_distance<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)ref_leaf_smem(NT)));
  return RTR_OK;
}

extern "C" {

rtr_status rtr_ref_distance(rtr_context* ctx, const float* d_mcloud, const float* d_mkeys, int n_model,
                            const int32_t* d_moffsets, const int32_t* d_mindices, const float* d_mtdf,
                            const float* d_skeys, int n_scan, const int32_t* d_pair_m, const int32_t* d_pair_s,
                            long long n_pairs, float resolution, float half_tdf, float* d_score, float* d_T,
                            rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && n_model >= 0 && n_scan >= 0, "rtr_ref_distance: bad arguments");
  RTR_CHECK_ARG(resolution > 0.f && half_tdf > 0.f && isfinite(resolution) && isfinite(half_tdf),
                "rtr_ref_distance: resolution and half_tdf must be positive");
  RTR_CHECK_ARG((int)(half_tdf / resolution * 2) == REF_DIM,
                "rtr_ref_distance: the field must be 30^3 voxels (get_Distance reads it as 30^3)");
  const bool all = d_pair_m == nullptr;
  RTR_CHECK_ARG(all == (d_pair_s == nullptr), "rtr_ref_distance: pair_m and pair_s both or neither");
  if (all) n_pairs = (long long)n_model * n_scan;
  RTR_CHECK_ARG(n_pairs >= 0 && n_pairs <= 0x7fffffffLL, "rtr_ref_distance: %lld pairs (at most 2^31 - 1)",
                n_pairs);
  if (n_pairs == 0) return RTR_OK;
  RTR_CHECK_ARG(n_model > 0 && n_scan > 0 && d_mcloud && d_mkeys && d_moffsets && d_mtdf && d_skeys && d_score &&
                    d_T,
                "rtr_ref_distance: NULL input or output");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  ScratchPlan plan;
  // err: [0] error bits, [1] largest cloud, [2] pairs the warp form leaves,
  // [3..] model keypoints per size class
  const size_t o_err = plan.add<int>(3 + REFW_CLASSES);
  const size_t least = plan.bytes;  // without the warp form: every pair a CTA
  const size_t o_box = plan.add<RefKeyBox>((size_t)n_model);
  const size_t o_list = plan.add<int>((size_t)n_model * REFW_CLASSES);
  Scratch s;
  RTR_TRY(ensure_scratch_upto(ctx, plan.bytes, least, st, &s));
  const int warp_max = s.cap >= plan.bytes ? REFW_MAX : -1;
  int* err = reinterpret_cast<int*>(s.base + o_err);
  RefKeyBox* boxes = reinterpret_cast<RefKeyBox*>(s.base + o_box);
  int* list = reinterpret_cast<int*>(s.base + o_list);
  const RefRot rot = ref_rot_tables();
  const RefUnit un = ref_unit(resolution);
  RTR_CUDA(cudaMemsetAsync(err, 0, (3 + REFW_CLASSES) * sizeof(int), st));
  k_ref_max_count<<<(n_model + 255) / 256, 256, 0, st>>>(d_moffsets, n_model, err + 1);
  if (warp_max >= 0)
    k_ref_keybox<<<(n_model + 63) / 64, 64, 0, st>>>(reinterpret_cast<const float4*>(d_mkeys), d_moffsets, n_model,
                                                     resolution, half_tdf, un, rot, boxes, list, err + 3);
  RTR_LAUNCHED(warp_max >= 0 ? 2 : 1);
  int h[3 + REFW_CLASSES];
  RTR_TRY(ref_read_ints(ctx, err, 3 + REFW_CLASSES, st, h));
  const int nmax = h[1];
  if (nmax > 0) RTR_CHECK_ARG(d_mindices, "rtr_ref_distance: NULL indices");
  if (nmax > REF_PPT * 1024)
    return fail(RTR_ERR_CAPACITY, "rtr_ref_distance: an occupancy cloud of %d points (at most %d)", nmax,
                REF_PPT * 1024);
  if (!all) {
    // every pair index inside [0, n_model) x [0, n_scan): checked on the host
    std::vector<int32_t> pm((size_t)n_pairs), ps_((size_t)n_pairs);
    RTR_CUDA(cudaMemcpyAsync(pm.data(), d_pair_m, sizeof(int32_t) * (size_t)n_pairs, cudaMemcpyDeviceToHost, st));
    RTR_CUDA(cudaMemcpyAsync(ps_.data(), d_pair_s, sizeof(int32_t) * (size_t)n_pairs, cudaMemcpyDeviceToHost, st));
    RTR_CUDA(cudaStreamSynchronize(st));
    for (long long i = 0; i < n_pairs; ++i)
      RTR_CHECK_ARG(pm[(size_t)i] >= 0 && pm[(size_t)i] < n_model && ps_[(size_t)i] >= 0 && ps_[(size_t)i] < n_scan,
                    "rtr_ref_distance: pair %lld = (%d, %d) out of range", i, pm[(size_t)i], ps_[(size_t)i]);
  }
  ProfScope ps(ctx, st, "ref_distance");
  const float4* mc = reinterpret_cast<const float4*>(d_mcloud);
  const float4* mk = reinterpret_cast<const float4*>(d_mkeys);
  const float4* sk = reinterpret_cast<const float4*>(d_skeys);
  const unsigned nb = (unsigned)n_pairs;
  // a launch per size class that has clouds, the largest first
#define REF_WARP_CLASS(c)                                                                                            \
  if (h[3 + (c)] > 0) {                                                                                              \
    const long long items = all ? (long long)h[3 + (c)] * n_scan : n_pairs;                                          \
    k_ref_distance_warp<c><<<(unsigned)((items + REFW_WARPS - 1) / REFW_WARPS), 32 * REFW_WARPS, 0, st>>>(           \
        mc, mk, d_moffsets, d_mindices, d_mtdf, boxes, list + (size_t)(c) * n_model, sk, n_scan, d_pair_m, d_pair_s, \
        items, resolution, half_tdf, un, rot, d_score, d_T, err);                                                        \
    RTR_LAUNCHED(1);                                                                                                 \
  }
  REF_WARP_CLASS(10)
  REF_WARP_CLASS(8)
  REF_WARP_CLASS(7)
  REF_WARP_CLASS(9)
  REF_WARP_CLASS(6)
  REF_WARP_CLASS(5)
  REF_WARP_CLASS(4)
  REF_WARP_CLASS(3)
  REF_WARP_CLASS(2)
  REF_WARP_CLASS(1)
  REF_WARP_CLASS(0)
#undef REF_WARP_CLASS
  RTR_CUDA(cudaGetLastError());
  if (nmax <= warp_max) {
    RTR_TRY(ref_read_ints(ctx, err, 4, st, h));
    RTR_TRY(ref_check_err(h[0], "rtr_ref_distance"));
    if (h[2] == 0) return RTR_OK;
  }
  // larger clouds, and the pairs left: a CTA each
  if (nmax <= REF_PPT * 256) {
    RTR_TRY(ref_distance_smem<256>());
    k_ref_distance<256><<<nb, 256, ref_leaf_smem(256), st>>>(mc, mk, d_moffsets, d_mindices, d_mtdf, sk, n_scan,
                                                             d_pair_m, d_pair_s, resolution, half_tdf, rot, d_score,
                                                             d_T, err, warp_max);
  } else if (nmax <= REF_PPT * 512) {
    RTR_TRY(ref_distance_smem<512>());
    k_ref_distance<512><<<nb, 512, ref_leaf_smem(512), st>>>(mc, mk, d_moffsets, d_mindices, d_mtdf, sk, n_scan,
                                                             d_pair_m, d_pair_s, resolution, half_tdf, rot, d_score,
                                                             d_T, err, warp_max);
  } else {
    RTR_TRY(ref_distance_smem<1024>());
    k_ref_distance<1024><<<nb, 1024, ref_leaf_smem(1024), st>>>(mc, mk, d_moffsets, d_mindices, d_mtdf, sk, n_scan,
                                                                d_pair_m, d_pair_s, resolution, half_tdf, rot, d_score,
                                                                d_T, err, warp_max);
  }
  RTR_LAUNCHED(1);
  RTR_CUDA(cudaGetLastError());
  RTR_TRY(ref_read_ints(ctx, err, 4, st, h));
  return ref_check_err(h[0], "rtr_ref_distance");
}

rtr_status rtr_ref_correspond(rtr_context* ctx, const float* d_mkeys, const int32_t* d_mnumber, const double* d_mv3,
                              int n_model, const float* d_skeys, const int32_t* d_snumber, const double* d_sv3,
                              int n_scan, const float* d_score_all, float max_score, int32_t* d_pair_idx, int cap,
                              int* h_n_pairs, rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && n_model >= 0 && n_scan >= 0 && cap >= 0 && h_n_pairs, "rtr_ref_correspond: bad arguments");
  *h_n_pairs = 0;
  const long long np = (long long)n_model * n_scan;
  RTR_CHECK_ARG(np <= (1LL << 30), "rtr_ref_correspond: %lld pairs (at most 2^30)", np);
  if (np == 0) return RTR_OK;
  RTR_CHECK_ARG(d_mkeys && d_mnumber && d_skeys && d_snumber && d_score_all, "rtr_ref_correspond: NULL input");
  RTR_CHECK_ARG(cap == 0 || d_pair_idx, "rtr_ref_correspond: NULL output");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  ScratchPlan plan;
  const size_t o_f = plan.add<uint32_t>((size_t)np + 1);
  const size_t o_p = plan.add<uint32_t>((size_t)np + 1);
  const size_t o_tiles = plan.add<uint32_t>((size_t)scan_tiles((int)np + 1));
  const size_t o_tot = plan.add<uint32_t>(4);
  Scratch s;
  RTR_TRY(ensure_scratch(ctx, plan.bytes, st, &s));
  uint32_t* flags = reinterpret_cast<uint32_t*>(s.base + o_f);
  uint32_t* pos = reinterpret_cast<uint32_t*>(s.base + o_p);
  uint32_t* tiles = reinterpret_cast<uint32_t*>(s.base + o_tiles);
  uint32_t* tot = reinterpret_cast<uint32_t*>(s.base + o_tot);
  ProfScope ps(ctx, st, "ref_correspond");
  RTR_CUDA(cudaMemsetAsync(flags + np, 0, sizeof(uint32_t), st));
  const int nb = (int)((np + 255) / 256 < 65535 ? (np + 255) / 256 : 65535);
  k_ref_gates<<<nb, 256, 0, st>>>(reinterpret_cast<const float4*>(d_mkeys), d_mnumber, d_mv3,
                                  reinterpret_cast<const float4*>(d_skeys), d_snumber, d_sv3, n_scan, np, d_score_all,
                                  max_score, flags);
  scan_exclusive(flags, pos, tiles, (int)np + 1, (int)np + 1, nullptr, tot, st);
  k_ref_scatter<<<nb, 256, 0, st>>>(flags, pos, np, cap, d_pair_idx);
  RTR_LAUNCHED(3);
  RTR_CUDA(cudaGetLastError());
  int h[1];
  RTR_TRY(ref_read_ints(ctx, reinterpret_cast<const int*>(tot), 1, st, h));
  *h_n_pairs = h[0];
  if (h[0] > cap) return fail(RTR_ERR_CAPACITY, "rtr_ref_correspond: %d pairs, capacity %d", h[0], cap);
  return RTR_OK;
}

rtr_status rtr_ref_ransac(rtr_context* ctx, const float* d_mkeys, int n_model, const float* d_skeys, int n_scan,
                          const int32_t* d_pair_idx, int n_pairs, const float* d_score_all, const float* d_T_all,
                          float inlier_dist, float max_des, float* h_T, int* h_inliers, int* h_best,
                          rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && n_model > 0 && n_scan > 0 && n_pairs >= 0 && h_T && h_inliers && h_best,
                "rtr_ref_ransac: bad arguments");
  for (int i = 0; i < 16; ++i) h_T[i] = (i % 5) == 0 ? 1.f : 0.f;
  *h_inliers = 0;
  *h_best = -1;
  if (n_pairs == 0) return RTR_OK;
  RTR_CHECK_ARG(d_mkeys && d_skeys && d_pair_idx && d_score_all && d_T_all, "rtr_ref_ransac: NULL input");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  {
    // every pair index inside the n_model x n_scan table: checked on the host
    std::vector<int32_t> pi((size_t)n_pairs);
    RTR_CUDA(cudaMemcpyAsync(pi.data(), d_pair_idx, sizeof(int32_t) * (size_t)n_pairs, cudaMemcpyDeviceToHost, st));
    RTR_CUDA(cudaStreamSynchronize(st));
    const long long np_all = (long long)n_model * n_scan;
    for (int i = 0; i < n_pairs; ++i)
      RTR_CHECK_ARG(pi[(size_t)i] >= 0 && pi[(size_t)i] < np_all, "rtr_ref_ransac: pair index %d = %d out of range", i,
                    pi[(size_t)i]);
  }
  ScratchPlan plan;
  const size_t o_c = plan.add<int>((size_t)n_pairs);
  const size_t o_o = plan.add<int>(4);
  Scratch s;
  RTR_TRY(ensure_scratch(ctx, plan.bytes, st, &s));
  int* cnt = reinterpret_cast<int*>(s.base + o_c);
  int* out = reinterpret_cast<int*>(s.base + o_o);
  ProfScope ps(ctx, st, "ref_ransac");
  k_ref_ransac<<<n_pairs, RANSAC_NT, 0, st>>>(reinterpret_cast<const float4*>(d_mkeys),
                                              reinterpret_cast<const float4*>(d_skeys), n_scan, d_pair_idx, n_pairs,
                                              d_score_all, d_T_all, inlier_dist, max_des, cnt);
  k_ref_argmax<<<1, 1024, 0, st>>>(cnt, n_pairs, out);
  RTR_LAUNCHED(2);
  RTR_CUDA(cudaGetLastError());
  int h[2];
  RTR_TRY(ref_read_ints(ctx, out, 2, st, h));
  *h_best = h[0];
  *h_inliers = h[1];
  if (h[0] >= 0) {
    int pidx = 0;
    RTR_CUDA(cudaMemcpyAsync(ctx->h_pin, d_pair_idx + h[0], sizeof(int), cudaMemcpyDeviceToHost, st));
    RTR_CUDA(cudaStreamSynchronize(st));
    pidx = ctx->h_pin[0];
    RTR_CUDA(cudaMemcpyAsync(h_T, d_T_all + 16 * (size_t)pidx, 16 * sizeof(float), cudaMemcpyDeviceToHost, st));
    RTR_CUDA(cudaStreamSynchronize(st));
  }
  return RTR_OK;
}

}  // extern "C"
