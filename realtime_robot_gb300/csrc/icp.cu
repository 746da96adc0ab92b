// icp.cu — persistent point-to-point ICP (replaces the PCL
// IterativeClosestPoint used by keyPointICP, function.h:111-148).
//
// One cooperative launch runs every iteration.  Per iteration the source
// points are transformed with the FP32 pose and matched to their exact 1-NN
// in the target grid within max_corr_dist (rejection; most points only show
// that their last neighbour still is the nearest, see k_icp), and each thread
// accumulates the centred sums (dp, dq, dp dq^T, d^2) in FP32 Kahan–Babuška
// accumulators; warps and the block combine them with TwoSum-compensated
// shuffles into one (hi, lo) pair per value per block.  The last block to
// arrive reduces the block pairs (fixed order, FP64 closing), solves the pose
// in FP64 (pose.cuh) and publishes it to the others.  Every wait is bounded by
// a clock64 budget; a block that runs out writes RTR_ERR_TIMEOUT and leaves.
#include <math.h>
#include <algorithm>
#include <atomic>
#include <string.h>

#include "coop_share.h"
#include "grid.cuh"
#include "icp.cuh"
#include "pose.cuh"
#include "search.cuh"

namespace rtr {

constexpr int ICP_THREADS = 256;
constexpr int ICP_WARPS = ICP_THREADS / 32;
constexpr int ICP_NV = 16;  // dp(3) dq(3) dp*dq^T(9) d^2(1)
constexpr size_t ICP_STATE_MAX = size_t(50) << 20;  // points whose matching state a call asks scratch for (1 GB)
constexpr int ICP_CHUNK = 2048;  // points a block matches between two barriers

__device__ __forceinline__ unsigned long long icp_timer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Between iterations nothing may cost the SM its L1: an acquire or a full
// fence invalidates it, and every load of the next iteration (points, table,
// the matching state, all of them hits otherwise) would go to L2.  So a block
// arrives with a release alone, and the new pose is published as twelve
// 64-bit words that carry the iteration beside the value: whoever reads the
// right iteration has the value, in any order.  Only the block that arrives
// last fences, to read the others' sums.  (Two 20k chairs 1583 -> 1387 us,
// the room's recognition 4284 -> 4116 us.)
__device__ __forceinline__ unsigned icp_arrive(unsigned* p) {
  unsigned v;
  asm volatile("atom.add.release.gpu.global.u32 %0, [%1], 1;" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ float centre_of(const GridMeta* m, int a) {
  return 0.5f * (box_lo(m, a) + box_hi(m, a));
}

// One launch serves many problems: block b works on problem blk2prob[b]
// together with that problem's other nblk - 1 blocks; problems never wait on
// one another.
//
// Matching.  The search that found a point's neighbour also found how far away
// every other target point was ("room").  As long as the distance the source
// point has moved since then, subtracted from the room, leaves more than the
// distance to the neighbour as it is now, the neighbour is still the nearest,
// and the point needs no search (for a point without a neighbour: more than
// the bound).  Both sides carry a margin far above their rounding, so the
// correspondences are those of a search from scratch.  Each iteration runs
//   1. a thread per point: is the last answer still certain?  The others
//      queue up in shared memory;
//   2. G lanes per queued point: the search (grid_nn1_from), starting from
//      the last neighbour; a queue keeps every lane busy where single points
//      scattered over the warps would hold up 32 lanes each;
//   3. S lanes per point, 16 / S of the sums each.
// A search per point and iteration, each from the full bound, was over half of
// the kernel.  Per iteration of block 0, matching and sums before and now: two
// 20k chairs 25 and 8 us; 102k points against a 285k-point frame 35 and 10 us;
// 16 refinements of a 9.2k-voxel model in a room 24 and 10 us.
//
// The sums.  Which points a block owns, and the order and the tree in which
// they are added, depend on n, the number of blocks and S alone: point l of a
// pass goes to the same S lanes however the matching is run.  A compensated
// sum in another order differs in its last bits (1e-14), and where a pose's
// small entries are rounded to FP32 for the next iteration that now and then
// becomes an ulp, 1e-8 of the result; so a change of the matching, its lanes
// or its queue leaves every bit of the sums where it was.
// (Runs of eight points, mixed best over the blocks, and a thread per point's
// sums gain nothing: two 20k chairs 1,227 us, 1,197 so; 102k points against a
// 285k-point frame 1,105 and 1,120; 64 pairs 26.3 ms and 25.5.)
// G: lanes cooperating on one source point's 1-NN search; S: lanes sharing a
// point's sums (icp_pick_sum_lanes); OCC: blocks wanted an SM
template <int G, int S, int OCC>
__global__ void __launch_bounds__(ICP_THREADS, OCC) k_icp(const IcpDev* __restrict__ probs,
                                                        const int* __restrict__ blk2prob) {
  const IcpDev& a = probs[blk2prob[blockIdx.x]];
  const int lb = (int)blockIdx.x - a.blk0;
  __shared__ float s_red[ICP_WARPS][ICP_NV][2], s_blk[2 * ICP_WARPS][ICP_NV][2];
  __shared__ int s_cnt[ICP_WARPS];
  __shared__ double s_sum[ICP_NV];
  __shared__ float s_T[12];
  __shared__ int s_pos[ICP_CHUNK];             // matched position of each point of the chunk (-1: none)
  __shared__ unsigned short s_queue[ICP_CHUNK];  // points to search
  __shared__ int s_qn;
  __shared__ int s_last, s_stop;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (a.d_active && a.slot >= *a.d_active) {  // a capacity slot left unused: every block of it leaves
    if (lb == 0 && tid == 0) {
      a.result->iterations = 0;
      a.result->converged = 0;
      a.result->n_corr = 0;
      a.result->fitness = 0.0;
      a.result->status = RTR_OK;
    }
    return;
  }
  const int B = a.nblk;
  BoxView bv = box_view(a.grid);
  if (G <= 4) bv.dense = grid_dense(a.grid, bv.g);
  const GridView& g = bv.g;
  const float r = sqrt_up(a.r2max);
  // Centring: target terms about the target box centre c, source terms about
  // the source box centre moved by the current pose (cp), so the FP32 products
  // stay small even while the clouds are far apart.
  const float c[3] = {centre_of(a.grid.meta, 0), centre_of(a.grid.meta, 1), centre_of(a.grid.meta, 2)};
  const float4 cs = make_float4(centre_of(a.src_meta, 0), centre_of(a.src_meta, 1), centre_of(a.src_meta, 2), 0.f);
  float mag = 0.f;  // the size of the source's coordinates
#pragma unroll
  for (int k = 0; k < 3; ++k) mag += fmaxf(fabsf(box_lo(a.src_meta, k)), fabsf(box_hi(a.src_meta, k)));
  // point l of this block: runs of PPB points dealt out to the blocks in turn
  constexpr int PPB = ICP_THREADS / S;  // points a block sums side by side
  constexpr int NVL = ICP_NV / S;       // sums kept per lane
  static_assert(ICP_CHUNK % PPB == 0, "a chunk is a whole number of passes of the sums");
  const int groups = (a.n_src + PPB - 1) / PPB;
  const int n_loc = lb < groups ? ((groups - lb + B - 1) / B) * PPB : 0;
  auto point_of = [&](int l) { return ((l / PPB) * B + lb) * PPB + (l & (PPB - 1)); };
  const int lg = lane & (G - 1), ls = lane & (S - 1);
  const unsigned gmask = ((1u << G) - 1u) << (lane & ~(G - 1));

  const bool prof0 = a.prof != nullptr && lb == 0 && tid == 0;
  unsigned long long t_it = 0, t_arr = 0;
  for (int it = 0; it < a.max_it; ++it) {
    if (prof0) t_it = icp_timer();
    if (it == 0) {  // later poses arrive in s_T
      if (tid < 12) s_T[tid] = __double2float_rn(a.init[tid]);
      __syncthreads();
    }
    float T[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) T[k] = s_T[k];
    const float4 cp = xform_exact(T, cs);
    // rounding of the search, and of a point's position then and now
    const float margin = bv.margin + 2.0e-6f * (mag + fabsf(T[3]) + fabsf(T[7]) + fabsf(T[11]));
    KSum acc[NVL];  // values ls * NVL ... of the points tid / S, tid / S + PPB, ... in that order
#pragma unroll
    for (int k = 0; k < NVL; ++k) acc[k].init();
    int cnt = 0;
    for (int c0 = 0; c0 < n_loc; c0 += ICP_CHUNK) {
      const int cn = min(ICP_CHUNK, n_loc - c0);
      if (c0 > 0) __syncthreads();  // the last chunk's places are free
      if (tid == 0) s_qn = 0;
      __syncthreads();
      // 1. still certain?  (loop bound rounded up: the ballots need whole warps)
      for (int l = tid; l < ((cn + 31) & ~31); l += ICP_THREADS) {
        const int i = l < cn ? point_of(c0 + l) : a.n_src;
        bool search = false;
        int pos = -1;
        if (i < a.n_src) {
          search = true;
          if (it > 0 && a.anchor) {
            const float4 was = a.anchor[i], p = xform_exact(T, a.src[i]);
            pos = a.last[i];
            float reach = r;
            if (pos >= 0) {
              const float d2 = dist2_exact(p, g.pts[pos]);
              reach = d2 <= a.r2max ? sqrt_up(d2) : __int_as_float(0x7f800000);
            }
            search = !(reach + margin < was.w - sqrt_up(dist2_exact(p, was)));
          }
        }
        if (l < cn) s_pos[l] = pos;
        const unsigned bal = __ballot_sync(0xffffffffu, search);
        int base = 0;
        if (lane == 0 && bal) base = atomicAdd(&s_qn, __popc(bal));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (search) s_queue[base + __popc(bal & lanemask_lt())] = (unsigned short)l;
      }
      __syncthreads();
      // 2. the searches.  A box is widened by what the point moved since its
      // last search, up to half the neighbour's distance (its next nearest
      // is about that much farther) or a fraction of the bound.
      const int qn = s_qn;
      for (int k = tid / G; k < qn; k += ICP_THREADS / G) {
        const int l = s_queue[k], i = point_of(c0 + l), was = s_pos[l];
        const float4 p = xform_exact(T, a.src[i]);
        float extra = 0.f, room;
        if (it > 0 && a.anchor) {
          const float m = 4.f * sqrt_up(dist2_exact(p, a.anchor[i]));
          if (was >= 0)
            extra = fminf(m, fmaxf(0.5f * fminf(sqrt_up(dist2_exact(p, g.pts[was])), r), 0.1f * g.h));
          else
            extra = m < 0.4f * r ? fminf(m, 0.3f * r) : 0.f;
        }
        const int pos = grid_nn1_from<G>(bv, p, a.r2max, r, was, extra, lg, gmask, &room);
        if (lg == 0) {
          s_pos[l] = pos;
          if (a.anchor) {
            a.anchor[i] = make_float4(p.x, p.y, p.z, room);
            a.last[i] = pos;
          }
        }
      }
      __syncthreads();
      // 3. the sums: dp 0-2, dq 3-5, dp dq^T 6-14, d^2 15
      for (int l = tid / S; l < cn; l += PPB) {
        const int i = point_of(c0 + l), pos = s_pos[l];
        if (i >= a.n_src) break;  // and all after it
        if (pos >= 0) {
          const float4 p = xform_exact(T, a.src[i]), q = g.pts[pos];
          const float dp[3] = {__fsub_rn(p.x, cp.x), __fsub_rn(p.y, cp.y), __fsub_rn(p.z, cp.z)};
          const float dq[3] = {__fsub_rn(q.x, c[0]), __fsub_rn(q.y, c[1]), __fsub_rn(q.z, c[2])};
          float val[ICP_NV];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            val[k] = dp[k];
            val[3 + k] = dq[k];
#pragma unroll
            for (int m = 0; m < 3; ++m) val[6 + 3 * k + m] = __fmul_rn(dp[k], dq[m]);
          }
          val[15] = dist2_exact(p, q);
#pragma unroll
          for (int k = 0; k < NVL; ++k) {
            float x = val[k];
#pragma unroll
            for (int o = 1; o < S; ++o)
              if (ls == o) x = val[o * NVL + k];
            acc[k].add(x);
          }
          ++cnt;
        }
        if (a.trace_corr && ls == 0)
          a.trace_corr[(size_t)it * (size_t)a.n_src + (size_t)(a.src_idx ? a.src_idx[i] : i)] =
              pos >= 0 ? pt_index(g.pts[pos]) : -1;
      }
    }
    // compensated sums over the warp's points, halving the values a lane holds
    // with each exchange (lane bit 4 keeps the lower or the upper half, ...):
    // the tree of offsets 16 ... S over all values, at NVL combinations a lane
    {
      float s[NVL], e[NVL];
      int v = ls * NVL;  // the value this lane ends with
#pragma unroll
      for (int k = 0; k < NVL; ++k) {
        s[k] = acc[k].s;
        e[k] = acc[k].c;
      }
#pragma unroll
      for (int off = 16, nv = NVL / 2; nv >= 1; off >>= 1, nv >>= 1) {
        const bool up = (lane & off) != 0;
        if (up) v += nv;
#pragma unroll
        for (int k = 0; k < nv; ++k) {
          const float ks = up ? s[k + nv] : s[k], ke = up ? e[k + nv] : e[k];
          const float os = __shfl_xor_sync(0xffffffffu, up ? s[k] : s[k + nv], off);
          const float oe = __shfl_xor_sync(0xffffffffu, up ? e[k] : e[k + nv], off);
          float t, err;
          two_sum(ks, os, t, err);
          s[k] = t;
          e[k] = __fadd_rn(__fadd_rn(ke, oe), err);
        }
      }
      const float os = __shfl_xor_sync(0xffffffffu, s[0], S), oe = __shfl_xor_sync(0xffffffffu, e[0], S);
      float t, err;
      two_sum(s[0], os, t, err);
      if ((lane & S) == 0) {
        s_red[warp][v][0] = t;
        s_red[warp][v][1] = __fadd_rn(__fadd_rn(e[0], oe), err);
      }
    }
    cnt = ls == 0 ? cnt : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if (lane == 0) s_cnt[warp] = cnt;
    __syncthreads();
    if (tid < ICP_NV) {
      float s = s_red[0][tid][0], cc = s_red[0][tid][1];
      for (int w = 1; w < ICP_WARPS; ++w) {
        float t, e;
        two_sum(s, s_red[w][tid][0], t, e);
        s = t;
        cc = __fadd_rn(__fadd_rn(cc, s_red[w][tid][1]), e);
      }
      a.partial[lb * 32 + tid] = s;
      a.partial[lb * 32 + ICP_NV + tid] = cc;
    }
    if (tid == 0) {
      int tot = 0;
      for (int w = 0; w < ICP_WARPS; ++w) tot += s_cnt[w];
      a.pcount[lb] = tot;
    }
    __syncthreads();
    if (tid == 0) {
      if (prof0) {
        t_arr = icp_timer();
        atomicAdd(a.prof + 0, t_arr - t_it);
      }
      const unsigned t = icp_arrive(a.arrive);
      s_last = (t == (unsigned)(it + 1) * (unsigned)B - 1u) ? 1 : 0;
      if (s_last) __threadfence();
    }
    __syncthreads();
    if (s_last) {
      const unsigned long long t_s0 = a.prof && tid == 0 ? icp_timer() : 0ull;
      // warp 0 lane k: entry k of the current pose (FP64), fetched early
      const double pk = warp != 0 || lane > 15 ? 0.0 : (it == 0 ? a.init[lane] : __ldcg(a.pose64 + lane));
      // Cross-block reduction.  GB300 issues one FP64 warp-instruction per ~16
      // SM cycles, so the tree runs on compensated FP32 pairs (TwoSum, ~48-bit
      // significand) and FP64 closes it: one (double)hi + (double)lo per value.
      // 32 sums of every 32nd block (thread (k, v): value v of those of k and of
      // k + 16, in order; ten blocks' loads in flight, whole lines), then a tree
      // of offsets 16, 8, 4, 2, 1 over them.
      {
        constexpr int KG = ICP_THREADS / ICP_NV;
        const int v = tid & (ICP_NV - 1), kg = tid / ICP_NV;
        float hs[2] = {0.f, 0.f}, lo[2] = {0.f, 0.f};
        int nloc = 0;
        for (int b0 = kg; b0 < B; b0 += 10 * KG) {
          float h[10], l[10];
#pragma unroll
          for (int u = 0; u < 10; ++u) {
            const int b = b0 + KG * u;
            h[u] = b < B ? __ldcg(a.partial + b * 32 + v) : 0.f;
            l[u] = b < B ? __ldcg(a.partial + b * 32 + ICP_NV + v) : 0.f;
            if (v == 0 && b < B) nloc += __ldcg(a.pcount + b);
          }
#pragma unroll
          for (int u = 0; u < 10; ++u) {
            float t, e;
            two_sum(hs[u & 1], h[u], t, e);
            hs[u & 1] = t;
            lo[u & 1] = __fadd_rn(__fadd_rn(lo[u & 1], l[u]), e);
          }
        }
        float t, e;
        two_sum(hs[0], hs[1], t, e);
        s_blk[kg][v][0] = t;
        s_blk[kg][v][1] = __fadd_rn(__fadd_rn(lo[0], lo[1]), e);
        nloc += __shfl_xor_sync(0xffffffffu, nloc, 16);
        if (lane == 0) s_cnt[warp] = nloc;
      }
      __syncthreads();
      if (warp == 0) {
        const int v = lane & (ICP_NV - 1), odd = lane / ICP_NV;
        float h[ICP_WARPS], l[ICP_WARPS];
#pragma unroll
        for (int j = 0; j < ICP_WARPS; ++j) {
          h[j] = s_blk[odd + 2 * j][v][0];
          l[j] = s_blk[odd + 2 * j][v][1];
        }
#pragma unroll
        for (int off = ICP_WARPS / 2; off > 0; off >>= 1)
#pragma unroll
          for (int j = 0; j < off; ++j) {
            float t, e;
            two_sum(h[j], h[j + off], t, e);
            h[j] = t;
            l[j] = __fadd_rn(__fadd_rn(l[j], l[j + off]), e);
          }
        float hs, e;
        two_sum(h[0], __shfl_xor_sync(0xffffffffu, h[0], 16), hs, e);
        const float lo = __fadd_rn(__fadd_rn(l[0], __shfl_xor_sync(0xffffffffu, l[0], 16)), e);
        if (lane < ICP_NV) s_sum[lane] = (double)hs + (double)lo;
        __syncwarp();
      }
      if (a.prof && tid == 0) atomicAdd(a.prof + 4, icp_timer() - t_s0);
      if (warp == 0) {
        // the pose solve and the new pose, on warp 0 without a block barrier:
        // 3-vectors, 3x3 and 4x4 matrices are spread over the lanes (FP64 is
        // charged per warp instruction) and operands come by shuffle
        const unsigned full = 0xffffffffu;
        int n = 0;
#pragma unroll
        for (int w = 0; w < ICP_WARPS; ++w) n += s_cnt[w];
        int stop = it + 1 >= a.max_it ? 1 : 0, converged = 1;
        double fitness = 0.0, np = pk;
        if (it == 0 && a.trace_pose && lane < 16) a.trace_pose[lane] = pk;
        if (n < 3) {
          stop = 1;
          converged = 0;
        } else {
          // 1 / n: the FP32 reciprocal and two Newton steps
          const double dn = (double)n;
          double inv = (double)__frcp_rn((float)n);
          inv = fma(inv, fma(-dn, inv, 1.0), inv);
          inv = fma(inv, fma(-dn, inv, 1.0), inv);
          // centred cross-covariance, entry e in lane e; the rotation likewise
          const int e = lane < 9 ? lane : 8;
          const double r = umeyama_rotation_warp(fma(-(s_sum[e / 3] * inv), s_sum[3 + e % 3], s_sum[6 + e]));
          // lanes 0-2: source mean, 3-5: target mean; then lane i: t_i
          const int v = lane < 6 ? lane : 5;
          const float off = v == 0 ? cp.x : (v == 1 ? cp.y : (v == 2 ? cp.z : (v == 3 ? c[0] : (v == 4 ? c[1] : c[2]))));
          const double mean = fma(s_sum[v], inv, (double)off);
          const int i3 = lane < 3 ? lane : 2;
          double t = __shfl_sync(full, mean, 3 + i3);
#pragma unroll
          for (int k = 0; k < 3; ++k)
            t = fma(-__shfl_sync(full, r, 3 * i3 + k), __shfl_sync(full, mean, k), t);
          // pose <- [r t] pose, entry (lane / 4, lane % 4) in lanes 0-11; its last row stays
          const int ar = lane < 12 ? lane >> 2 : 2, bc = lane & 3;
          double acc = __shfl_sync(full, t, ar) * __shfl_sync(full, pk, 12 + bc);
#pragma unroll
          for (int k = 0; k < 3; ++k)
            acc = fma(__shfl_sync(full, r, 3 * ar + k), __shfl_sync(full, pk, 4 * k + bc), acc);
          if (lane < 12) np = acc;
          fitness = s_sum[15] * inv;
          if (a.eps_t > 0.0) {
            const double t0 = __shfl_sync(full, t, 0), t1 = __shfl_sync(full, t, 1), t2 = __shfl_sync(full, t, 2);
            const double tr = __shfl_sync(full, r, 0) + __shfl_sync(full, r, 4) + __shfl_sync(full, r, 8);
            if (t0 * t0 + t1 * t1 + t2 * t2 < a.eps_t && (a.eps_r <= 0.0 || 0.5 * (tr - 1.0) > a.eps_r)) stop = 1;
          }
        }
        if (lane < 16) {
          a.pose64[lane] = np;
          if (lane < 12) {
            const float f = __double2float_rn(np);
            s_T[lane] = f;
            st_relaxed(a.posew + lane, ((unsigned long long)((unsigned)(it + 1) | (stop ? 0x80000000u : 0u)) << 32) |
                                           __float_as_uint(f));
          }
          if (a.trace_pose) a.trace_pose[(size_t)(it + 1) * 16 + lane] = np;
          a.result->pose[lane] = np;
        }
        if (lane == 0) {
          a.result->fitness = fitness;
          a.result->iterations = it + 1;
          a.result->converged = converged;
          a.result->n_corr = n;
          a.result->status = RTR_OK;
          s_stop = stop;
          if (a.prof) atomicAdd(a.prof + 5, icp_timer() - t_s0);
        }
        if (lane == 0 && a.prof) {
          atomicAdd(a.prof + 1, icp_timer() - t_s0);
          atomicAdd(a.prof + 3, 1ull);
        }
      }
      __syncthreads();
    } else {
      if (tid < 32) {
        const long long t0 = clock64();
        unsigned long long w = 0;
        bool here = lane >= 12, late = false;
        for (;;) {
          if (!here) {
            w = ld_relaxed(a.posew + lane);
            here = (unsigned)((w >> 32) & 0x7fffffffu) >= (unsigned)(it + 1);
          }
          if (__all_sync(0xffffffffu, here)) break;
          late = __any_sync(0xffffffffu, clock64() - t0 > a.budget);
          if (late) break;
          __nanosleep(32);
        }
        if (late) {
          if (lane == 0) {
            atomicExch(a.status, (int)RTR_ERR_TIMEOUT);
            a.result->status = RTR_ERR_TIMEOUT;
            a.result->converged = 0;
            s_stop = 1;
          }
        } else {
          if (lane < 12) s_T[lane] = __uint_as_float((unsigned)w);
          if (lane == 0) s_stop = (int)(w >> 63);
        }
        if (prof0) atomicAdd(a.prof + 2, icp_timer() - t_arr);
      }
      __syncthreads();
    }
    if (s_stop) break;
  }
}

// Sort keys of the source under the initial pose, in the target grid.
__global__ void __launch_bounds__(256) k_src_keys(const float4* __restrict__ src, int n,
                                                  IcpDev a, uint32_t* __restrict__ keys) {
  const GridMeta* m = a.grid.meta;
  float T[12];
#pragma unroll
  for (int k = 0; k < 12; ++k) T[k] = __double2float_rn(a.init[k]);
  const float ox = m->ox, oy = m->oy, oz = m->oz, ih = m->inv_h;
  const int nx = m->nx, ny = m->ny, nz = m->nz;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float4 p = xform_exact(T, src[i]);
    int cx = min(max(q_cell(p.x, ox, ih), 0), nx - 1);
    int cy = min(max(q_cell(p.y, oy, ih), 0), ny - 1);
    int cz = min(max(q_cell(p.z, oz, ih), 0), nz - 1);
    keys[i] = ((uint32_t)cz * (uint32_t)ny + (uint32_t)cy) * (uint32_t)nx + (uint32_t)cx;
  }
}

__global__ void __launch_bounds__(256) k_gather_pts(const float4* __restrict__ pts,
                                                    const uint32_t* __restrict__ order, int n,
                                                    float4* __restrict__ out, int* __restrict__ idx) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t o = order[i];
    out[i] = pts[o];
    idx[i] = (int)o;
  }
}

// Blocks an SM holds of the ICP kernel.  Two with all the registers that the
// pose solve wants, where one call has the GPU: a solve an iteration is on its
// critical path (two 20k chairs 1,295 us; 1,571 with three blocks an SM, 1,816
// with four).  Four, the solve spilling, for workers side by side: other pairs
// fill that wait, and the searches gain from the threads (64 pairs with learned
// pruning 22.8 ms with two and half the SMs' places, 21.1 with four and the
// shares of coop_share.h, which leave every launch its places; six models in
// one room the other way, 28.6 and 30.9 ms).
constexpr int ICP_OCC = 2, ICP_OCC_WORKER = 4;

template <int G, int S, int OCC>
static int icp_per_sm_of() {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_icp<G, S, OCC>, ICP_THREADS, 0);
  return n;
}
template <int OCC>
static int icp_per_sm() {
  return std::min(std::min(icp_per_sm_of<2, 2, OCC>(), icp_per_sm_of<4, 2, OCC>()),
                  std::min(icp_per_sm_of<4, 4, OCC>(), icp_per_sm_of<8, 8, OCC>()));
}

// A worker beside others takes the small form (a worker alone has the GPU).
static bool icp_shared(const rtr_context* ctx) { return ctx->worker && ctx->coop_div > 1; }

// Co-resident blocks of the ICP kernel (the smallest over the group sizes,
// so a plan made for one group size fits every variant).
int icp_max_blocks(rtr_context* ctx) {
  static std::atomic<int> cached[64][2];  // per device; 0 = not yet known
  const int dev = ctx->device, kind = icp_shared(ctx) ? 1 : 0;
  if (dev >= 0 && dev < 64) {
    const int v = cached[dev][kind].load(std::memory_order_relaxed);
    if (v > 0) return v;
  }
  const int per_sm = kind ? icp_per_sm<ICP_OCC_WORKER>() : icp_per_sm<ICP_OCC>();
  const int v = per_sm * ctx->num_sms;
  if (dev >= 0 && dev < 64) cached[dev][kind].store(v, std::memory_order_relaxed);
  return v;
}

// Lanes per searched source point: the tuning override when set, else by the
// points a block has to match.  Few points leave lanes idle and wait on the
// latency of single searches: 8 lanes; many keep the block busy, and what
// counts is instructions: 4, then 2.  Measured (8 / 4 / 2 lanes): two 20k
// chairs, 66 points a block, 1332 / 1352 / 1871 us; 16 refinements of 9.2k
// points, 484 a block, the room's recognition 4196 / 4074 / 4140 us; a batch of
// 64 pairs, thousands a block, 32.8 / 31.2 / 31.2 ms.
int icp_pick_group(const rtr_context* ctx, long long total_pts, int blocks) {
  const int t = ctx->tune_icp_group;
  if (t == 2 || t == 4 || t == 8) return t;
  const long long per_block = total_pts / (blocks > 0 ? blocks : 1);
  return per_block <= 128 ? 8 : (per_block <= 1024 ? 4 : 2);
}

// Lanes that share a point's sums: 8, 4 or 2, the most with which a block takes
// at most four passes over its points (the tuning override sets both).  The
// search's lanes are the same or more, so four pairs are compiled.
static int icp_pick_sum_lanes(const rtr_context* ctx, long long total_pts, int blocks) {
  const int t = ctx->tune_icp_group;
  if (t == 2 || t == 4 || t == 8) return t;
  const long long lanes = (long long)blocks * ICP_THREADS;
  if (total_pts * 8 <= 4 * lanes) return 8;
  return total_pts * 4 <= 4 * lanes ? 4 : 2;
}

template <int OCC>
static rtr_status launch_icp(int G, int S, const IcpDev* d_probs, const int* d_blk2prob, int blocks, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(ICP_THREADS);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (S == 8)  // then G is 8 too
    RTR_CUDA(cudaLaunchKernelEx(&cfg, k_icp<8, 8, OCC>, d_probs, d_blk2prob));
  else if (S == 4)
    RTR_CUDA(cudaLaunchKernelEx(&cfg, k_icp<4, 4, OCC>, d_probs, d_blk2prob));
  else if (G == 4)
    RTR_CUDA(cudaLaunchKernelEx(&cfg, k_icp<4, 2, OCC>, d_probs, d_blk2prob));
  else
    RTR_CUDA(cudaLaunchKernelEx(&cfg, k_icp<2, 2, OCC>, d_probs, d_blk2prob));
  RTR_LAUNCHED(1);
  return RTR_OK;
}

// Problem descriptors reach device memory through kernel parameters (so a
// stream capture records them by value).  init_dev (optional) overrides the
// parameter's initial pose with a pose already on the device.
constexpr int ICP_SETUP_BATCH = 16;
struct IcpSetup {
  IcpDev p[ICP_SETUP_BATCH];
  const double* init_dev[ICP_SETUP_BATCH];
  int n, first;
};

__global__ void k_icp_setup(IcpSetup s, IcpDev* __restrict__ probs, int* __restrict__ blk2prob) {
  const int k = blockIdx.x;
  if (k >= s.n) return;
  const int pid = s.first + k;
  const IcpDev& a = s.p[k];
  for (int b = threadIdx.x; b < a.nblk; b += blockDim.x) blk2prob[a.blk0 + b] = pid;
  if (threadIdx.x == 0) {
    IcpDev d = a;
    if (s.init_dev[k])
      for (int i = 0; i < 16; ++i) d.init[i] = s.init_dev[k][i];
    probs[pid] = d;
    d.arrive[0] = 0u;
    for (int i = 0; i < 12; ++i) d.posew[i] = 0ull;
  }
}

void icp_multi_plan(ScratchPlan& p, int n_probs, int max_blocks, size_t n_state) {
  p.add<IcpDev>(n_probs);
  p.add<int>(max_blocks);
  p.add<double>((size_t)n_probs * 16);
  p.add<unsigned long long>((size_t)n_probs * 16);
  p.add<float>((size_t)max_blocks * 32);
  p.add<int>(max_blocks);
  p.add<unsigned>(n_probs);
  p.add<float4>(n_state);
  p.add<int>(n_state);
}

rtr_status icp_multi(rtr_context* ctx, Scratch& s, std::vector<IcpSpec>& specs, cudaStream_t st) {
  const int M = (int)specs.size();
  if (M == 0) return RTR_OK;
  const int maxb = icp_max_blocks(ctx);
  if (M > maxb) return fail(RTR_ERR_CAPACITY, "icp: %d problems exceed the %d co-resident blocks", M, maxb);
  // a share of the GPU when several contexts run cooperative kernels at once
  int budget = icp_shared(ctx) ? std::min(maxb, coop_share(ctx->num_sms, ctx->coop_div, ctx->coop_gc_per_sm).icp)
                               : maxb;
  if (budget < M) budget = M;
  IcpDev* d_probs = s.take<IcpDev>(M);
  int* d_b2p = s.take<int>(maxb);
  double* pose64 = s.take<double>((size_t)M * 16);
  unsigned long long* posew = s.take<unsigned long long>((size_t)M * 16);
  float* partial = s.take<float>((size_t)maxb * 32);
  int* pcount = s.take<int>(maxb);
  unsigned* sync = s.take<unsigned>(M);
  if (!sync) return fail(RTR_ERR_CAPACITY, "icp: scratch carve");
  // the matching state, of as many problems as the scratch at hand holds it for
  // (the plans of the single-cloud entry points include it up to ICP_STATE_MAX
  // points; a recognition's stages leave far more): without it every point is
  // searched in every iteration
  auto state_fits = [&](size_t n) {
    Scratch t = s;
    return t.take<float4>(n) && t.take<int>(n);
  };
  int with_state = 0;
  size_t n_state = 0;
  while (with_state < M && state_fits(n_state + specs[with_state].dev.n_src))
    n_state += specs[with_state++].dev.n_src;
  float4* anchor = s.take<float4>(n_state);
  int* last = s.take<int>(n_state);
  // apportion blocks: want_i = ceil(n_i * G / threads), scaled to fit
  long long want_total = 0;
  std::vector<long long> want(M);
  for (int i = 0; i < M; ++i) {
    want[i] = ((long long)specs[i].dev.n_src * 8 + ICP_THREADS - 1) / ICP_THREADS;
    if (want[i] < 1) want[i] = 1;
    want_total += want[i];
  }
  std::vector<int> nblk(M);
  int used = 0;
  for (int i = 0; i < M; ++i) {
    long long b = want_total <= budget ? want[i] : (want[i] * (budget - M)) / want_total + 1;
    nblk[i] = (int)(b < 1 ? 1 : b);
    used += nblk[i];
  }
  int blk = 0;
  for (int i = 0; i < M; ++i) {
    IcpDev& d = specs[i].dev;
    d.blk0 = blk;
    d.nblk = nblk[i];
    d.pose64 = pose64 + 16 * i;
    d.posew = posew + 16 * i;
    d.partial = partial + (size_t)blk * 32;
    d.pcount = pcount + blk;
    d.arrive = sync + i;
    d.anchor = i < with_state ? anchor : nullptr;
    d.last = i < with_state ? last : nullptr;
    if (i < with_state) {
      anchor += d.n_src;
      last += d.n_src;
    }
    d.status = ctx->d_status;
    d.budget = ctx->wait_budget_cycles;
    d.prof = i == 0 ? reinterpret_cast<unsigned long long*>(ctx->d_status + 32) : nullptr;
    blk += nblk[i];
  }
  RTR_CUDA(cudaMemsetAsync(ctx->d_status + 32, 0, 6 * sizeof(unsigned long long), st));
  for (int f = 0; f < M; f += ICP_SETUP_BATCH) {
    IcpSetup su;
    memset(&su, 0, sizeof(su));
    su.first = f;
    su.n = M - f < ICP_SETUP_BATCH ? M - f : ICP_SETUP_BATCH;
    for (int k = 0; k < su.n; ++k) {
      su.p[k] = specs[f + k].dev;
      su.init_dev[k] = specs[f + k].init_dev;
    }
    k_icp_setup<<<su.n, 128, 0, st>>>(su, d_probs, d_b2p);
    RTR_LAUNCHED(1);
  }
  RTR_CUDA(cudaGetLastError());
  long long total = 0;
  for (int i = 0; i < M; ++i) total += specs[i].dev.n_src;
  const int G = icp_pick_group(ctx, total, used), S = icp_pick_sum_lanes(ctx, total, used);
  return icp_shared(ctx) ? launch_icp<ICP_OCC_WORKER>(G, S, d_probs, d_b2p, used, st)
                         : launch_icp<ICP_OCC>(G, S, d_probs, d_b2p, used, st);
}

}  // namespace rtr

using namespace rtr;

extern "C" {

void rtr_icp_default_params(rtr_icp_params* p) {
  if (!p) return;
  p->max_iterations = 10;
  p->max_corr_dist = 0.f;
  p->transformation_epsilon = 0.0;
  p->rotation_epsilon = 0.0;
  p->cell_size = 0.f;
  p->record_trace = 0;
}

rtr_status rtr_icp(rtr_context* ctx, const float* d_src, int n_src, const float* d_tgt, int n_tgt,
                   const rtr_icp_params* params, const double* h_init_pose,
                   rtr_icp_result* d_result, double* d_trace_pose, int32_t* d_trace_corr,
                   rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && params && d_result, "rtr_icp: ctx, params and d_result are required");
  RTR_CHECK_ARG(n_src > 0 && n_tgt > 0 && d_src && d_tgt, "rtr_icp: empty source or target");
  RTR_CHECK_ARG(params->max_iterations > 0, "rtr_icp: max_iterations must be > 0");
  RTR_CHECK_ARG(((uintptr_t)d_src & 15) == 0 && ((uintptr_t)d_tgt & 15) == 0,
                "rtr_icp: point arrays must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));

  const unsigned cell_cap = default_cell_cap(n_tgt);
  const int maxb = icp_max_blocks(ctx);
  int blocks = (int)(((long long)n_src * 8 + ICP_THREADS - 1) / ICP_THREADS);
  if (blocks > maxb) blocks = maxb;
  if (blocks < 1) blocks = 1;

  ScratchPlan plan;
  grid_plan(plan, n_tgt, cell_cap);
  plan.add<float4>(n_src);
  plan.add<int>(n_src);
  for (int i = 0; i < 4; ++i) plan.add<uint32_t>(n_src);
  plan.add<uint32_t>(radix_hist_entries(n_src));
  plan.add<GridMeta>(1);
  ScratchPlan least = plan;  // without the matching state
  icp_multi_plan(least, 1, maxb, 0);
  icp_multi_plan(plan, 1, maxb, std::min((size_t)n_src, ICP_STATE_MAX));
  Scratch s;
  RTR_TRY(ensure_scratch_upto(ctx, plan.bytes, least.bytes, st, &s));
  GridBufs gb;
  if (!grid_take(s, n_tgt, cell_cap, &gb)) return fail(RTR_ERR_CAPACITY, "rtr_icp: scratch carve");
  float4* src_sorted = s.take<float4>(n_src);
  int* src_idx = s.take<int>(n_src);
  uint32_t* k0 = s.take<uint32_t>(n_src);
  uint32_t* v0 = s.take<uint32_t>(n_src);
  uint32_t* k1 = s.take<uint32_t>(n_src);
  uint32_t* v1 = s.take<uint32_t>(n_src);
  uint32_t* hist = s.take<uint32_t>(radix_hist_entries(n_src));
  GridMeta* src_meta = s.take<GridMeta>(1);
  if (!src_meta) return fail(RTR_ERR_CAPACITY, "rtr_icp: scratch carve");

  float h = params->cell_size;
  if (!(h > 0.f)) h = params->max_corr_dist > 0.f ? 0.5f * params->max_corr_dist : -1.f;
  {
    ProfScope ps(ctx, st, "grid_build");
    RTR_TRY(grid_build(gb, reinterpret_cast<const float4*>(d_tgt), n_tgt, nullptr, h, st));
  }

  IcpDev a;
  memset(&a, 0, sizeof(a));
  a.grid = grid_dev(gb);
  a.src_meta = src_meta;
  RTR_TRY(bbox_build(src_meta, reinterpret_cast<const float4*>(d_src), n_src, st));
  a.src = src_sorted;
  a.src_idx = src_idx;
  a.n_src = n_src;
  a.max_it = params->max_iterations;
  const float r = params->max_corr_dist;
  a.r2max = (r > 0.f && r < 1e18f) ? r * r : __builtin_inff();
  a.eps_t = params->transformation_epsilon;
  a.eps_r = params->rotation_epsilon;
  for (int k = 0; k < 16; ++k) a.init[k] = h_init_pose ? h_init_pose[k] : ((k % 5) == 0 ? 1.0 : 0.0);
  a.result = d_result;
  a.trace_pose = params->record_trace ? d_trace_pose : nullptr;
  a.trace_corr = params->record_trace ? d_trace_corr : nullptr;

  int nb = (n_src + 255) / 256;
  if (nb > 152 * 8) nb = 152 * 8;
  ProfScope ps_sort(ctx, st, "src_sort");
  k_src_keys<<<nb, 256, 0, st>>>(reinterpret_cast<const float4*>(d_src), n_src, a, k0);
  int bits = 1;
  while (bits < 32 && (1ull << bits) < (unsigned long long)cell_cap) ++bits;
  uint32_t *ks, *vs;
  RTR_TRY(radix_sort_pairs(ctx, k0, v0, k1, v1, hist, n_src, n_src, nullptr, bits, true, st, &ks, &vs));
  k_gather_pts<<<nb, 256, 0, st>>>(reinterpret_cast<const float4*>(d_src), vs, n_src, src_sorted,
                                   src_idx);
  RTR_LAUNCHED(2);
  RTR_CUDA(cudaGetLastError());
  ps_sort.end();
  ProfScope ps(ctx, st, "icp_kernel");
  std::vector<IcpSpec> specs(1);
  specs[0].dev = a;
  specs[0].init_dev = nullptr;
  return icp_multi(ctx, s, specs, st);
}

rtr_status rtr_icp_multi(rtr_context* ctx, const float* d_src, int n_src, const float* d_tgt, int n_tgt,
                         const rtr_icp_params* params, const double* d_init_poses, int n_problems,
                         rtr_icp_result* d_results, rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && params && d_results, "rtr_icp_multi: ctx, params and d_results are required");
  RTR_CHECK_ARG(n_src > 0 && n_tgt > 0 && d_src && d_tgt, "rtr_icp_multi: empty source or target");
  RTR_CHECK_ARG(params->max_iterations > 0, "rtr_icp_multi: max_iterations must be > 0");
  RTR_CHECK_ARG(((uintptr_t)d_src & 15) == 0 && ((uintptr_t)d_tgt & 15) == 0,
                "rtr_icp_multi: point arrays must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  const int maxb = icp_max_blocks(ctx);
  RTR_CHECK_ARG(n_problems >= 1 && n_problems <= maxb, "rtr_icp_multi: n_problems must be in [1, %d]", maxb);
  const unsigned cell_cap = default_cell_cap(n_tgt);
  ScratchPlan plan;
  grid_plan(plan, n_tgt, cell_cap);
  plan.add<GridMeta>(1);
  ScratchPlan least = plan;  // without the matching state
  icp_multi_plan(least, n_problems, maxb, 0);
  icp_multi_plan(plan, n_problems, maxb, std::min((size_t)n_problems * n_src, ICP_STATE_MAX));
  Scratch s;
  RTR_TRY(ensure_scratch_upto(ctx, plan.bytes, least.bytes, st, &s));
  GridBufs gb;
  if (!grid_take(s, n_tgt, cell_cap, &gb)) return fail(RTR_ERR_CAPACITY, "rtr_icp_multi: scratch carve");
  GridMeta* src_meta = s.take<GridMeta>(1);
  if (!src_meta) return fail(RTR_ERR_CAPACITY, "rtr_icp_multi: scratch carve");
  float h = params->cell_size;
  if (!(h > 0.f)) h = params->max_corr_dist > 0.f ? 0.5f * params->max_corr_dist : -1.f;
  ProfScope ps(ctx, st, "icp_multi");
  RTR_TRY(grid_build(gb, reinterpret_cast<const float4*>(d_tgt), n_tgt, nullptr, h, st));
  RTR_TRY(bbox_build(src_meta, reinterpret_cast<const float4*>(d_src), n_src, st));
  std::vector<IcpSpec> specs((size_t)n_problems);
  const float r = params->max_corr_dist;
  for (int k = 0; k < n_problems; ++k) {
    IcpDev& a = specs[(size_t)k].dev;
    memset(&a, 0, sizeof(a));
    a.grid = grid_dev(gb);
    a.src_meta = src_meta;
    a.src = reinterpret_cast<const float4*>(d_src);
    a.src_idx = nullptr;
    a.n_src = n_src;
    a.max_it = params->max_iterations;
    a.r2max = (r > 0.f && r < 1e18f) ? r * r : __builtin_inff();
    a.eps_t = params->transformation_epsilon;
    a.eps_r = params->rotation_epsilon;
    for (int e = 0; e < 16; ++e) a.init[e] = (e % 5) == 0 ? 1.0 : 0.0;
    a.result = d_results + k;
    specs[(size_t)k].init_dev = d_init_poses ? d_init_poses + 16 * (size_t)k : nullptr;
  }
  return icp_multi(ctx, s, specs, st);
}

rtr_status rtr_icp_host(rtr_context* ctx, const float* h_src, int n_src, const float* h_tgt,
                        int n_tgt, const rtr_icp_params* params, const double* h_init_pose,
                        rtr_icp_result* h_result) {
  RTR_CHECK_ARG(ctx && h_src && h_tgt && params && h_result && n_src > 0 && n_tgt > 0,
                "rtr_icp_host: bad arguments");
  RTR_CUDA(cudaSetDevice(ctx->device));
  const size_t bs = (size_t)n_src * 16, bt = (size_t)n_tgt * 16;
  const size_t need = ((bs + 255) & ~size_t(255)) + ((bt + 255) & ~size_t(255)) + 256;
  RTR_TRY(ensure_io(ctx, need));
  char* io = static_cast<char*>(ctx->io);
  float* d_src = reinterpret_cast<float*>(io);
  float* d_tgt = reinterpret_cast<float*>(io + ((bs + 255) & ~size_t(255)));
  rtr_icp_result* d_res =
      reinterpret_cast<rtr_icp_result*>(io + ((bs + 255) & ~size_t(255)) + ((bt + 255) & ~size_t(255)));
  cudaStream_t st = ctx->host_stream;
  RTR_CUDA(cudaMemcpyAsync(d_src, h_src, bs, cudaMemcpyHostToDevice, st));
  RTR_CUDA(cudaMemcpyAsync(d_tgt, h_tgt, bt, cudaMemcpyHostToDevice, st));
  RTR_TRY(rtr_icp(ctx, d_src, n_src, d_tgt, n_tgt, params, h_init_pose, d_res, nullptr, nullptr, st));
  RTR_CUDA(cudaMemcpyAsync(h_result, d_res, sizeof(rtr_icp_result), cudaMemcpyDeviceToHost, st));
  return rtr_context_check(ctx, st);
}

}  // extern "C"

extern "C" rtr_status rtr_icp_stats(rtr_context* ctx, long long* h_stats6) {
  RTR_CHECK_ARG(ctx && h_stats6, "rtr_icp_stats: bad arguments");
  RTR_CUDA(cudaSetDevice(ctx->device));
  RTR_CUDA(cudaDeviceSynchronize());
  RTR_CUDA(cudaMemcpy(h_stats6, ctx->d_status + 32, 6 * sizeof(long long), cudaMemcpyDeviceToHost));
  return RTR_OK;
}
