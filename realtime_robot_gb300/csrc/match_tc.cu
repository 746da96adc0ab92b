// match_tc.cu — descriptor 1-NN on the 5th-generation tensor cores.
//
// d^2(q, b) = |q|^2 + |b|^2 - 2 q.b with the dot product as a BF16 GEMM with
// FP32 accumulation in tensor memory.  Each FP32 descriptor is split into
// hi = bf16(x) and lo = bf16(x - hi); the accumulator sums hi.hi + hi.lo +
// lo.hi (three tcgen05.mma per K step), which leaves |err(q.b)| of order
// 1e-4 |q| |b| (dropped lo.lo, the split's rounding, FP32 accumulation); the
// certification uses TC_ERR * max(|q|, max |b|)^2, which covers that and the
// FP32 norms with margin (unit-norm SHOT vectors: 5e-4).  Inf values, and NaN
// in a query, make a query uncertified; a database row with a NaN never wins
// and is left out.  Per query the epilogue keeps the 8
// smallest approximate distances; an exact FP32 re-rank (sequential sums, as
// the oracle) picks the winner, and a query is certified when its 8th
// approximate distance minus the error bound is still above the exact winner,
// so no unseen descriptor can beat or tie it.  Uncertified queries (near-ties)
// take a band pass: the same GEMM over them lists every row whose d~ is
// within twice the bound of the exact winner (every row that could tie or beat
// it), and exact distances to those rows decide; a band over TC_BAND rows
// falls back to an exact scan of the whole database.  The result is
// bit-identical to the exact matcher.
//
// Kernel layout (one CTA per 128 queries, 6 warps): warp 4 issues TMA loads of
// the K-blocks (32 bf16 = one 64-byte swizzle row) of Q_hi, Q_lo, B_hi, B_lo
// into a 4-stage ring; warp 5 issues tcgen05.mma (M=128, N=256, K=16) into one
// of two TMEM accumulators (2 x 256 columns); warps 0-3 drain the finished
// accumulator with tcgen05.ld (thread = query row) and update the top-8.
// Every mbarrier wait is bounded; on timeout the CTA records RTR_ERR_TIMEOUT,
// stops issuing, waits (bounded) for its in-flight work and frees its TMEM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <string.h>

#include "common.cuh"

namespace rtr {

constexpr int TC_DIM = 352;
constexpr int TC_KPAD = 384;              // 6 K-blocks of 64
// K-blocks of 32 bf16 (one 64-byte swizzle row): 48 KB stages, four of
// them in flight (two 96 KB stages of 64-wide K-blocks ran 3 % slower).
constexpr int TC_KB = 32;
constexpr int TC_NKB = TC_KPAD / TC_KB;
constexpr int TC_SW = TC_KB * 2;          // swizzle row bytes (64)
constexpr int TC_BM = 128;
constexpr int TC_BN = 256;
constexpr int TC_STAGES = 4;
constexpr int TC_TOP = 8;
constexpr int TC_BAND = 256;      // band pass: rows listed per uncertified query
constexpr int TC_BAND_Q = 16384;  // band pass: uncertified queries it takes (the rest: full scan)
constexpr int TC_A_BYTES = TC_BM * TC_KB * 2;   // 8 KB
constexpr int TC_B_BYTES = TC_BN * TC_KB * 2;   // 16 KB
constexpr int TC_STAGE_BYTES = 2 * TC_A_BYTES + 2 * TC_B_BYTES;  // 48 KB
constexpr int TC_KTAIL = TC_DIM / TC_KB;         // the K-block that holds only the norm column (its first)
constexpr int TC_RANGES = 8;                     // most database ranges of the first pass
constexpr int TC_THREADS = 192;
constexpr int TC_ROW = 36;  // floats a row in the epilogue's staging (16-byte stores of 8 rows meet 32 banks)
// Bound on |d~ - d| over max(|q|, max |b|)^2, d the FP32 sequential sum.  BF16
// keeps 8 significant bits: hi is within 2^-8 of x, hi + lo within 2^-16.  The
// dropped lo.lo and the two rests, twice: 2 * 3 * 2^-16 = 9.2e-5; the norm
// column's rest: 1.5e-5; 68 accumulations of 16 products, each term cut at 2^-23
// of the largest: 2.8e-4 (how the tensor cores add is not documented: an
// assumption, ten times what is measured); the sequential sum's own rounding
// (352 terms, d up to 4): 8.4e-5; norms and the last step: 2e-6; 4.7e-4 at
// worst.  Measured at most 2.2e-5 (SHOT rows of the room, Gaussian, sparse,
// offset and badly scaled ones).
constexpr float TC_ERR = 5.0e-4f;
constexpr long long TC_SPIN_LIMIT = 1LL << 26;

// ---------------------------------------------------------------------------
// PTX helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait (`limit` tries, from the context's wait budget); returns false
// (and raises the CTA abort flag) on timeout or when another role aborted
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, volatile int* abort, long long limit) {
  for (long long i = 0; i < limit; ++i) {
    if (mbar_try(b, parity)) return true;
    if (*abort) return false;
  }
  *abort = 1;
  return false;
}
// the drain after an abort: wait for work already issued, up to the fixed
// TC_SPIN_LIMIT tries whatever the budget (a copy or MMA in flight ends by
// itself; this only bounds the wait if the hardware stopped answering)
__device__ __forceinline__ void mbar_drain(uint64_t* b, uint32_t parity) {
  for (long long i = 0; i < TC_SPIN_LIMIT; ++i)
    if (mbar_try(b, parity)) return;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}
// UMMA shared-memory descriptor: K-major, TC_SW-byte swizzle rows, 8-row
// atoms of 8 * TC_SW bytes (SBO), start address in 16-byte units, descriptor
// version 1; layout type 4 = 64-byte swizzle, 2 = 128-byte swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);       // start address
  d |= (uint64_t)1 << 16;                         // LBO (unused for swizzled K-major)
  d |= (uint64_t)((8 * TC_SW) >> 4) << 32;        // SBO
  d |= (uint64_t)1 << 46;                         // version
  d |= (uint64_t)(TC_SW == 128 ? 2 : 4) << 61;    // swizzle mode
  return d;
}
// Instruction descriptor, kind::f16: D = F32, A = B = BF16, K-major, N, M.
__device__ __forceinline__ uint32_t umma_idesc() {
  uint32_t d = 0;
  d |= 1u << 4;                          // D format F32
  d |= 1u << 7;                          // A BF16
  d |= 1u << 10;                         // B BF16
  d |= (uint32_t)(TC_BN >> 3) << 17;     // N
  d |= (uint32_t)(TC_BM >> 4) << 24;     // M
  return d;
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(
          tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accum)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---------------------------------------------------------------------------
// FP32 descriptors -> padded (hi, lo) BF16 rows + FP32 squared norms
// ---------------------------------------------------------------------------
// hi/lo split of each row, padded to TC_KPAD.  Column TC_DIM carries the
// norm term so that the GEMM yields q.b - |b|^2 / 2 directly: 1 in query
// rows, -|b|^2 / 2 (itself split) in database rows.
__global__ void k_split_bf16(const float* __restrict__ x, int n_host, const int* d_n, int n_cap,
                             __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo,
                             float* __restrict__ norm2, unsigned* __restrict__ max_bits, bool is_db,
                             unsigned char* __restrict__ zero_row) {
  static_assert(TC_DIM % 4 == 0 && TC_KPAD == 96 * 4, "a row is 96 groups of four columns");
  const int n = d_n ? min(*d_n, n_cap) : n_host;
  // rows past the last tile that has live ones are never read (the room's
  // scene: 116k rows of 300k; 102 -> 53 us)
  const int end = min(n_cap, (n + TC_BM - 1) / TC_BM * TC_BM);
  const int lane = threadIdx.x & 31;
  const bool v4 = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  for (int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < end; r += gridDim.x * (blockDim.x >> 5)) {
    // lane takes column groups lane, lane + 32, lane + 64: four columns each,
    // one 16-byte load and two 8-byte stores
    float ss = 0.f;
    bool nz = false;
    float4 vv[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int c4 = lane + 32 * k;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < n && c4 < TC_DIM / 4) {
        const float* src = x + (size_t)r * TC_DIM + 4 * c4;
        v = v4 ? __ldg(reinterpret_cast<const float4*>(src)) : make_float4(src[0], src[1], src[2], src[3]);
      }
      vv[k] = v;
      nz |= v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f;
      ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    nz = __any_sync(0xffffffffu, nz);
    // column TC_DIM carries the norm term: 1 in query rows, -|b|^2 / 2 in
    // database rows (zero in padding rows)
    const float tv = r < n ? (is_db ? -0.5f * ss : 1.f) : 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int c4 = lane + 32 * k;
      float4 v = vv[k];
      if (c4 == TC_DIM / 4) v.x = tv;
      const float e[4] = {v.x, v.y, v.z, v.w};
      __nv_bfloat16 h[4], l[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        h[j] = __float2bfloat16_rn(e[j]);
        l[j] = __float2bfloat16_rn(e[j] - __bfloat162float(h[j]));
      }
      uint2 hp, lp;
      hp.x = (unsigned)__bfloat16_as_ushort(h[0]) | ((unsigned)__bfloat16_as_ushort(h[1]) << 16);
      hp.y = (unsigned)__bfloat16_as_ushort(h[2]) | ((unsigned)__bfloat16_as_ushort(h[3]) << 16);
      lp.x = (unsigned)__bfloat16_as_ushort(l[0]) | ((unsigned)__bfloat16_as_ushort(l[1]) << 16);
      lp.y = (unsigned)__bfloat16_as_ushort(l[2]) | ((unsigned)__bfloat16_as_ushort(l[3]) << 16);
      reinterpret_cast<uint2*>(hi + (size_t)r * TC_KPAD)[c4] = hp;
      reinterpret_cast<uint2*>(lo + (size_t)r * TC_KPAD)[c4] = lp;
    }
    if (lane == 0) {
      norm2[r] = ss;
      // the largest norm (ss >= 0), the scale of the error bound.  A row with a
      // NaN never wins and is nowhere in the lists: it sets no scale (a maximum
      // of NaN would leave the bound to the query's norm alone)
      if (max_bits && r < n && ss == ss) atomicMax(max_bits, __float_as_uint(ss));
      if (zero_row) zero_row[r] = (r < n && !nz) ? 1 : 0;
    }
  }
}

// ---------------------------------------------------------------------------
// GEMM + top-8
// ---------------------------------------------------------------------------
struct TcArgs {
  int nq_host;
  const int* d_nq;
  int nq_cap;
  int ndb;
  const float* qn;   // [nq_cap] |q|^2
  int* cand_idx;     // [nq_cap][8]; band pass: [nq_cap][TC_BAND] rows within the threshold
  float* cand_d;     // [nq_cap][8]
  int* more_idx;     // [ranges - 1][nq_cap][8]: the lists of the database ranges after the first
  float* more_d;
  int* status;
  const float* thr;  // band pass: [nq_cap] largest d~ a row may have and still tie the winner
  int* band_n;       // band pass: [nq_cap] rows listed (over TC_BAND: overflowed)
  long long spin_limit;  // tries per mbarrier wait (the context's wait budget)
};

// The band pass over the uncertified queries: per query every row with
// d~ <= thr[q], the first TC_BAND of them listed in band_n[q] (zeroed by the
// caller; a count over TC_BAND means the band overflowed and the row stops
// counting); the grid splits the database into gridDim.y ranges so that a
// few uncertified queries still fill the GPU.
__global__ void __launch_bounds__(TC_THREADS, 1) k_match_band(const __grid_constant__ CUtensorMap mq_hi,
                                                            const __grid_constant__ CUtensorMap mq_lo,
                                                            const __grid_constant__ CUtensorMap mb_hi,
                                                            const __grid_constant__ CUtensorMap mb_lo, TcArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[TC_STAGES], empty_bar[TC_STAGES], acc_full[2], acc_empty[2], drain_bar;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = a.d_nq ? min(*a.d_nq, a.nq_cap) : a.nq_host;
  const int q0 = blockIdx.x * TC_BM;
  if (q0 >= nq) return;  // uniform per CTA, before any barrier or TMEM use
  // database tiles of this CTA: all of them, or (band pass, gridDim.y > 1)
  // one of gridDim.y contiguous ranges
  const int n_all = (a.ndb + TC_BN - 1) / TC_BN;
  const int t_lo = (int)((long long)blockIdx.y * n_all / gridDim.y);
  const int t_hi = (int)((long long)(blockIdx.y + 1) * n_all / gridDim.y);

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < TC_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 128);
    }
    mbar_init(&drain_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 5) {  // allocate 512 TMEM columns (two 128 x 256 FP32 accumulators)
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  volatile int* abort = &abort_flag;
  const long long lim = a.spin_limit;
  int issued = 0;  // producer: stage loads issued

  if (warp == 4) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int it = 0;
      for (int t = t_lo; t < t_hi && !*abort; ++t) {
        for (int kb = 0; kb < TC_NKB && !*abort; ++kb, ++it) {
          const int s = it % TC_STAGES;
          const uint32_t ph = (uint32_t)(it / TC_STAGES) & 1u;
          if (it >= TC_STAGES && !mbar_wait(&empty_bar[s], ph ^ 1u, abort, lim)) break;
          uint8_t* st = smem + s * TC_STAGE_BYTES;
          mbar_expect_tx(&full_bar[s], TC_STAGE_BYTES);
          tma_load_2d(st, &mq_hi, &full_bar[s], kb * TC_KB, q0);
          tma_load_2d(st + TC_A_BYTES, &mq_lo, &full_bar[s], kb * TC_KB, q0);
          tma_load_2d(st + 2 * TC_A_BYTES, &mb_hi, &full_bar[s], kb * TC_KB, t * TC_BN);
          tma_load_2d(st + 2 * TC_A_BYTES + TC_B_BYTES, &mb_lo, &full_bar[s], kb * TC_KB, t * TC_BN);
        }
      }
      issued = it;
    }
  } else if (warp == 5) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      const uint32_t idesc = umma_idesc();
      int it = 0;
      for (int t = t_lo; t < t_hi && !*abort; ++t) {
        const int buf = (t - t_lo) & 1;
        const uint32_t use = (uint32_t)((t - t_lo) >> 1);
        if (t - t_lo >= 2 && !mbar_wait(&acc_empty[buf], (use - 1) & 1u, abort, lim)) break;
        tc_fence_after();
        const uint32_t dcol = tmem + (uint32_t)buf * TC_BN;
        for (int kb = 0; kb < TC_NKB; ++kb, ++it) {
          const int s = it % TC_STAGES;
          const uint32_t ph = (uint32_t)(it / TC_STAGES) & 1u;
          if (!mbar_wait(&full_bar[s], ph, abort, lim)) break;
          tc_fence_after();
          const uint32_t base = smem_u32(smem + s * TC_STAGE_BYTES);
          const uint32_t ah = base, al = base + TC_A_BYTES, bh = base + 2 * TC_A_BYTES,
                         bl = base + 2 * TC_A_BYTES + TC_B_BYTES;
#pragma unroll
          for (int k = 0; k < TC_KB / 16; ++k) {
            const uint32_t off = (uint32_t)k * 32;  // 16 bf16 along K inside the swizzle row
            const uint32_t acc0 = (kb > 0 || k > 0) ? 1u : 0u;
            umma_f16(dcol, umma_desc(ah + off), umma_desc(bh + off), idesc, acc0);
            umma_f16(dcol, umma_desc(ah + off), umma_desc(bl + off), idesc, 1u);
            umma_f16(dcol, umma_desc(al + off), umma_desc(bh + off), idesc, 1u);
          }
          umma_commit(&empty_bar[s]);  // stage free once these MMAs have read it
        }
        umma_commit(&acc_full[buf]);  // accumulator ready
      }
    }
  } else {
    // ---------------- epilogue: warps 0-3, thread = query row ----------------
    // The accumulator holds q.b - |b|^2 / 2.
    const int row = warp * 32 + lane;
    const int q = q0 + row;
    const float qn = q < nq ? a.qn[q] : 0.f;
    {
      // rows past the live queries (stale scratch, any bits) list nothing
      const bool live = q < nq;
      const float thr = live ? a.thr[q] : 0.f;
      int* list = a.cand_idx + (size_t)(live ? q : 0) * TC_BAND;
      bool over = false;  // this row's band already past TC_BAND: count no further
      for (int t = t_lo; t < t_hi; ++t) {
        const int buf = (t - t_lo) & 1;
        const uint32_t use = (uint32_t)((t - t_lo) >> 1);
        if (!mbar_wait(&acc_full[buf], use & 1u, abort, lim)) break;
        tc_fence_after();
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)buf * TC_BN;
        const int valid = min(TC_BN, a.ndb - t * TC_BN);
        for (int c0 = 0; c0 < TC_BN; c0 += 32) {
          float v[32];
          tmem_ld32(taddr + (uint32_t)c0, v);
          const int jb = t * TC_BN + c0;
          const int lim = valid - c0;
          // d~ exactly as the first pass forms it for its candidates
          uint32_t hit = 0;
#pragma unroll
          for (int i = 0; i < 32; ++i) hit |= (i < lim && qn - 2.f * v[i] <= thr) ? (1u << i) : 0u;
          if (live && hit && !over) {
            // one atomic per chunk (CTAs of other database ranges list into the same row)
            int pos = atomicAdd(a.band_n + q, __popc(hit));
            over = pos + __popc(hit) > TC_BAND;
            while (hit && pos < TC_BAND) {
              list[pos++] = jb + __ffs(hit) - 1;
              hit &= hit - 1;
            }
          }
        }
        tc_fence_before();
        mbar_arrive(&acc_empty[buf]);
      }
    }
  }
  // after an abort nothing of this CTA may still be in flight when it frees
  // its TMEM and exits: the MMA issuer waits for every MMA it issued, the
  // producer for the stage loads not yet seen complete (the last ones; each
  // earlier load of a stage completed before the stage was reused)
  __syncthreads();
  if (abort_flag) {
    if (warp == 5 && lane == 0) {
      umma_commit(&drain_bar);
      mbar_drain(&drain_bar, 0u);
    }
    if (warp == 4 && lane == 0)
      for (int i = issued > TC_STAGES ? issued - TC_STAGES : 0; i < issued; ++i)
        mbar_drain(&full_bar[i % TC_STAGES], (uint32_t)(i / TC_STAGES) & 1u);
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) atomicExch(a.status, (int)RTR_ERR_TIMEOUT);
  if (warp == 5) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  }
}

// The first pass: per query the 8 smallest d~ (largest q.b - |b|^2 / 2) of each
// database range (gridDim.y of them, contiguous tiles).
// What bounds it: the tensor cores.  Its 68 MMAs of 128 x 256 x 16 a tile alone
// (nothing loaded, nothing read back) take 401 us for the room's 111k x 3,001,
// the library GEMM's rate; with everything 460 us.  766 us while the epilogue
// inserted under divergence (3,072 columns a row, about 700 insertions a warp
// at 45 instructions in a chain of compares; now about 220 a warp, all lanes at
// once).  Tried and not better: two CTAs a cluster sharing a tile
// (cta_group::2; 483 us against 495 with the same epilogue), eight epilogue
// warps, the next accumulator columns loaded ahead, database boxes of 128 rows
// (+20 us).
__global__ void __launch_bounds__(TC_THREADS, 1) k_match_top(const __grid_constant__ CUtensorMap mq_hi,
                                                            const __grid_constant__ CUtensorMap mq_lo,
                                                            const __grid_constant__ CUtensorMap mb_hi,
                                                            const __grid_constant__ CUtensorMap mb_lo, TcArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[TC_STAGES], empty_bar[TC_STAGES], acc_full[2], acc_empty[2], drain_bar;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nq = a.d_nq ? min(*a.d_nq, a.nq_cap) : a.nq_host;
  const int q0 = blockIdx.x * TC_BM;
  if (q0 >= nq) return;  // uniform per CTA, before any barrier or TMEM use
  // database tiles of this CTA: one of gridDim.y contiguous ranges
  const int n_all = (a.ndb + TC_BN - 1) / TC_BN;
  const int t_lo = (int)((long long)blockIdx.y * n_all / gridDim.y);
  const int t_hi = (int)((long long)(blockIdx.y + 1) * n_all / gridDim.y);
  // every CTA starts at another tile, so that the CTAs, which run in step, do
  // not all read the same rows at the same time (518 -> 495 us)
  const int t_off = (int)(blockIdx.x % (unsigned)max(t_hi - t_lo, 1));
  auto tile = [&](int t) {
    const int r = t + t_off;
    return r < t_hi ? r : r - (t_hi - t_lo);
  };

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < TC_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 128);
    }
    mbar_init(&drain_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 5) {  // allocate 512 TMEM columns (two 128 x 256 FP32 accumulators)
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  volatile int* abort = &abort_flag;
  const long long lim = a.spin_limit;
  int issued = 0;  // producer: stage loads issued

  if (warp == 4) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int it = 0;
      for (int t = t_lo; t < t_hi && !*abort; ++t) {
        for (int kb = 0; kb < TC_NKB && !*abort; ++kb, ++it) {
          const int s = it % TC_STAGES;
          const uint32_t ph = (uint32_t)(it / TC_STAGES) & 1u;
          if (it >= TC_STAGES && !mbar_wait(&empty_bar[s], ph ^ 1u, abort, lim)) break;
          uint8_t* st = smem + s * TC_STAGE_BYTES;
          mbar_expect_tx(&full_bar[s], TC_STAGE_BYTES);
          tma_load_2d(st, &mq_hi, &full_bar[s], kb * TC_KB, q0);
          tma_load_2d(st + TC_A_BYTES, &mq_lo, &full_bar[s], kb * TC_KB, q0);
          tma_load_2d(st + 2 * TC_A_BYTES, &mb_hi, &full_bar[s], kb * TC_KB, tile(t) * TC_BN);
          tma_load_2d(st + 2 * TC_A_BYTES + TC_B_BYTES, &mb_lo, &full_bar[s], kb * TC_KB, tile(t) * TC_BN);
        }
      }
      issued = it;
    }
  } else if (warp == 5) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      const uint32_t idesc = umma_idesc();
      int it = 0;
      for (int t = t_lo; t < t_hi && !*abort; ++t) {
        const int buf = (t - t_lo) & 1;
        const uint32_t use = (uint32_t)((t - t_lo) >> 1);
        if (t - t_lo >= 2 && !mbar_wait(&acc_empty[buf], (use - 1) & 1u, abort, lim)) break;
        tc_fence_after();
        const uint32_t dcol = tmem + (uint32_t)buf * TC_BN;
        for (int kb = 0; kb < TC_NKB; ++kb, ++it) {
          const int s = it % TC_STAGES;
          const uint32_t ph = (uint32_t)(it / TC_STAGES) & 1u;
          if (!mbar_wait(&full_bar[s], ph, abort, lim)) break;
          tc_fence_after();
          const uint32_t base = smem_u32(smem + s * TC_STAGE_BYTES);
          const uint32_t ah = base, al = base + TC_A_BYTES, bh = base + 2 * TC_A_BYTES,
                         bl = base + 2 * TC_A_BYTES + TC_B_BYTES;
          // the tail block: one column that counts, and none in the queries' lo part
          for (int k = 0; k < (kb == TC_KTAIL ? 1 : TC_KB / 16); ++k) {
            const uint32_t off = (uint32_t)k * 32;  // 16 bf16 along K inside the swizzle row
            const uint32_t acc0 = (kb > 0 || k > 0) ? 1u : 0u;
            umma_f16(dcol, umma_desc(ah + off), umma_desc(bh + off), idesc, acc0);
            umma_f16(dcol, umma_desc(ah + off), umma_desc(bl + off), idesc, 1u);
            if (kb != TC_KTAIL) umma_f16(dcol, umma_desc(al + off), umma_desc(bh + off), idesc, 1u);
          }
          umma_commit(&empty_bar[s]);  // stage free once these MMAs have read it
        }
        umma_commit(&acc_full[buf]);  // accumulator ready
      }
    }
  } else {
    // ---------------- epilogue: warps 0-3, thread = query row ----------------
    // The accumulator holds q.b - |b|^2 / 2, so the nearest rows are the
    // largest values: one compare per element, d~ = |q|^2 - 2 acc at the end.
    const int row = warp * 32 + lane;
    const int q = q0 + row;
    const float qn = q < nq ? a.qn[q] : 0.f;
    {
    // The list of 8 is ascending in d~.  A chunk of 32 columns is compared with
    // the list's last value (a subtraction and a funnel shift collect a lane's
    // hits as bits), staged in shared memory, and each lane takes its own hits
    // in column order, all lanes at once: the warp runs as many insertions a
    // chunk as its busiest lane has hits.  An insertion's slots are independent
    // (the middle of the left neighbour, the new value and the slot).
    float ba[TC_TOP];
    int bi[TC_TOP];
#pragma unroll
    for (int s = 0; s < TC_TOP; ++s) {
      ba[s] = -__int_as_float(0x7f800000);
      bi[s] = 0x7fffffff;
    }
    float* stage = reinterpret_cast<float*>(smem + TC_STAGES * TC_STAGE_BYTES) + (size_t)row * TC_ROW;
    for (int t = t_lo; t < t_hi; ++t) {
      const int buf = (t - t_lo) & 1;
      const uint32_t use = (uint32_t)((t - t_lo) >> 1);
      if (!mbar_wait(&acc_full[buf], use & 1u, abort, lim)) break;
      tc_fence_after();
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)buf * TC_BN;
      const int valid = min(TC_BN, a.ndb - tile(t) * TC_BN);
      for (int c0 = 0; c0 < valid; c0 += 32) {
        float v[32];
        tmem_ld32(taddr + (uint32_t)c0, v);
        uint32_t hits = 0;  // bit 31 - i: column i (NaN and ties with the last value: not taken)
#pragma unroll
        for (int i = 0; i < 32; ++i)
          hits = __funnelshift_l(__float_as_uint(__fsub_rn(ba[TC_TOP - 1], v[i])), hits, 1);
        if (valid - c0 < 32) hits &= ~(0xffffffffu >> (valid - c0));
        if (!__any_sync(0xffffffffu, hits)) continue;
#pragma unroll
        for (int i = 0; i < 32; i += 4)
          *reinterpret_cast<float4*>(stage + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        do {
          const int i = hits ? __clz(hits) : 0;
          float x = stage[i];
          x = hits ? x : -__int_as_float(0x7f800000);
          const int xi = tile(t) * TC_BN + c0 + i;
          hits &= 0x7fffffffu >> i;  // (a lane without hits keeps none)
          bool gt[TC_TOP];
#pragma unroll
          for (int s = 0; s < TC_TOP; ++s) gt[s] = x > ba[s];
#pragma unroll
          for (int s = TC_TOP - 1; s > 0; --s) {
            bi[s] = gt[s - 1] ? bi[s - 1] : (gt[s] ? xi : bi[s]);
            ba[s] = gt[s - 1] ? ba[s - 1] : (gt[s] ? x : ba[s]);
          }
          bi[0] = gt[0] ? xi : bi[0];
          ba[0] = gt[0] ? x : ba[0];
        } while (__any_sync(0xffffffffu, hits));
      }
      tc_fence_before();
      mbar_arrive(&acc_empty[buf]);
    }
    if (q < nq) {
      const size_t off = (size_t)a.nq_cap * TC_TOP * (blockIdx.y > 0 ? blockIdx.y - 1 : 0);
      int* ci = blockIdx.y > 0 ? a.more_idx + off : a.cand_idx;
      float* cd = blockIdx.y > 0 ? a.more_d + off : a.cand_d;
#pragma unroll
      for (int s = 0; s < TC_TOP; ++s) {
        ci[(size_t)q * TC_TOP + s] = bi[s] == 0x7fffffff ? -1 : bi[s];
        cd[(size_t)q * TC_TOP + s] = bi[s] == 0x7fffffff ? __int_as_float(0x7f800000) : qn - 2.f * ba[s];
      }
    }
    }
  }
  // after an abort nothing of this CTA may still be in flight when it frees
  // its TMEM and exits: the MMA issuer waits for every MMA it issued, the
  // producer for the stage loads not yet seen complete (the last ones; each
  // earlier load of a stage completed before the stage was reused)
  __syncthreads();
  if (abort_flag) {
    if (warp == 5 && lane == 0) {
      umma_commit(&drain_bar);
      mbar_drain(&drain_bar, 0u);
    }
    if (warp == 4 && lane == 0)
      for (int i = issued > TC_STAGES ? issued - TC_STAGES : 0; i < issued; ++i)
        mbar_drain(&full_bar[i % TC_STAGES], (uint32_t)(i / TC_STAGES) & 1u);
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) atomicExch(a.status, (int)RTR_ERR_TIMEOUT);
  if (warp == 5) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  }
}

// Exact d^2 of one 352-float row pair: sequential sum in k order, each
// operation rounded (the oracle's order).  V4: both rows 16-byte aligned.
template <bool V4>
__device__ __forceinline__ float exact_d2(const float* __restrict__ x, const float* __restrict__ y) {
  float acc = 0.f;
  if (V4) {
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const float4* y4 = reinterpret_cast<const float4*>(y);
#pragma unroll 4
    for (int k = 0; k < TC_DIM / 4; ++k) {
      const float4 a = __ldg(x4 + k), b = __ldg(y4 + k);
      float t = __fsub_rn(a.x, b.x);
      acc = __fadd_rn(acc, __fmul_rn(t, t));
      t = __fsub_rn(a.y, b.y);
      acc = __fadd_rn(acc, __fmul_rn(t, t));
      t = __fsub_rn(a.z, b.z);
      acc = __fadd_rn(acc, __fmul_rn(t, t));
      t = __fsub_rn(a.w, b.w);
      acc = __fadd_rn(acc, __fmul_rn(t, t));
    }
  } else {
    for (int k = 0; k < TC_DIM; ++k) {
      const float t = __fsub_rn(x[k], y[k]);
      acc = __fadd_rn(acc, __fmul_rn(t, t));
    }
  }
  return acc;
}

// Exact FP32 re-rank of the candidates that can still win, and
// certification.  Uncertified queries go to the redo list with their running
// minimum reset.
// A warp takes `per` (4 .. 16) queries, lists the candidates in doubt (one or two a query)
// and handles eight of them at a time: the lanes read each candidate's and its
// query's row together (whole lines, all eight in flight), the squared
// differences go through shared memory, and a lane adds up one candidate's in
// order.  Bound by latency (of the rows, then of the adds): 98 us for the
// room's 111k queries with a lane reading its rows by itself, 67 us now.
constexpr int RR_WARPS = 4;
constexpr int RR_Q = 16;
constexpr int RR_C = 8;
// Queries a warp takes: 16, fewer where a warp would have its chain of
// candidates and others nothing (whole call, us, 4 / 8 / 16 a warp; rows of a
// room: 50 queries 96 / 98 / 104, 6,000 124 / 128 / 134, 111k 668 / 651 / 650;
// every row nine times in the database: 50 118 / 133 / 161, 6,000 135 / 150 /
// 172, 20,000 227 / 235 / 232).
static int rr_queries(int nq) { return nq <= 8000 ? 4 : (nq <= 16000 ? 8 : RR_Q); }
template <bool V4>
__global__ void __launch_bounds__(32 * RR_WARPS)
    k_rerank(const float* __restrict__ q, int nq_host, const int* d_nq, int nq_cap, const float* __restrict__ db, int ndb,
             const int* __restrict__ cand_idx, const float* __restrict__ cand_d, const int* __restrict__ more_idx,
             const float* __restrict__ more_d, int ranges, int per, int* __restrict__ out_idx, float* __restrict__ out_d2,
             int* __restrict__ redo, int* __restrict__ n_redo, unsigned long long* __restrict__ redo_best,
             float* __restrict__ redo_thr, const float* __restrict__ qn, const float* __restrict__ db_max,
             const unsigned long long* __restrict__ zero_best, const unsigned char* __restrict__ qzero) {
  __shared__ __align__(16) float s_term[RR_WARPS][RR_C][TC_DIM + 4];
  __shared__ int s_cand[RR_WARPS][RR_Q * TC_TOP];
  __shared__ unsigned char s_of[RR_WARPS][RR_Q * TC_TOP];
  __shared__ unsigned long long s_best[RR_WARPS][RR_Q];
  __shared__ float s_worst[RR_WARPS][RR_Q], s_bound[RR_WARPS][RR_Q];
  const int nq = d_nq ? min(*d_nq, nq_cap) : nq_host;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, sub = lane >> 3, l8 = lane & 7;
  const int warps = gridDim.x * RR_WARPS;
  const float dbm = *db_max;
  for (int base = (blockIdx.x * RR_WARPS + w) * per; base < nq; base += warps * per) {
    if (lane < per) s_best[w][lane] = ~0ull;
    // |d~ - d| <= err: a candidate whose d~ exceeds the smallest d~ (the
    // first of the ranges' ascending lists) by more than 2 err has an exact
    // distance above that candidate's, so it can neither win nor tie: its
    // exact distance is not computed
    if (lane < per) {
      const int i = base + lane;
      float bound = -__int_as_float(0x7f800000), worst = __int_as_float(0x7f800000);
      if (i < nq && qzero[i] == 0) {
        float first = cand_d[(size_t)i * TC_TOP];
        worst = cand_d[(size_t)i * TC_TOP + TC_TOP - 1];
        for (int r = 0; r + 1 < ranges; ++r) {
          const float* l = more_d + ((size_t)r * nq_cap + i) * TC_TOP;
          first = fminf(first, l[0]);
          worst = fminf(worst, l[TC_TOP - 1]);
        }
        bound = first + 2.f * (TC_ERR * fmaxf(qn[i], dbm));
      }
      s_bound[w][lane] = bound;
      s_worst[w][lane] = worst;
    }
    __syncwarp();
    for (int r = 0; r < ranges; ++r) {
      const int* li = r > 0 ? more_idx + (size_t)(r - 1) * nq_cap * TC_TOP : cand_idx;
      const float* ld = r > 0 ? more_d + (size_t)(r - 1) * nq_cap * TC_TOP : cand_d;
      int cnt = 0;
#pragma unroll
      for (int q0 = 0; q0 < RR_Q; q0 += 4) {
        if (q0 >= per) break;
        const size_t at = (size_t)(base + q0 + sub) * TC_TOP + l8;
        const bool live = base + q0 + sub < nq;
        const int c = live ? li[at] : -1;
        const float d = live ? ld[at] : 0.f;
        // (never read past the database, whatever the first pass left)
        const bool need = c >= 0 && c < ndb && d <= s_bound[w][q0 + sub];
        const unsigned nb = __ballot_sync(0xffffffffu, need);
        if (need) {
          const int e = cnt + __popc(nb & ((1u << lane) - 1u));
          s_cand[w][e] = c;
          s_of[w][e] = (unsigned char)(q0 + sub);
        }
        cnt += __popc(nb);
      }
      __syncwarp();
      for (int b0 = 0; b0 < cnt; b0 += RR_C) {
        const int m = min(RR_C, cnt - b0);
#pragma unroll 4
        for (int j = 0; j < m; ++j) {
          const float* x = q + (size_t)(base + s_of[w][b0 + j]) * TC_DIM;
          const float* y = db + (size_t)s_cand[w][b0 + j] * TC_DIM;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const int v = lane + 32 * k;
            if (v >= TC_DIM / 4) continue;
            float4 a, b;
            if (V4) {
              a = __ldg(reinterpret_cast<const float4*>(x) + v);
              b = __ldg(reinterpret_cast<const float4*>(y) + v);
            } else {
              a = make_float4(x[4 * v], x[4 * v + 1], x[4 * v + 2], x[4 * v + 3]);
              b = make_float4(y[4 * v], y[4 * v + 1], y[4 * v + 2], y[4 * v + 3]);
            }
            a.x = __fsub_rn(a.x, b.x), a.y = __fsub_rn(a.y, b.y), a.z = __fsub_rn(a.z, b.z), a.w = __fsub_rn(a.w, b.w);
            *reinterpret_cast<float4*>(&s_term[w][j][4 * v]) =
                make_float4(__fmul_rn(a.x, a.x), __fmul_rn(a.y, a.y), __fmul_rn(a.z, a.z), __fmul_rn(a.w, a.w));
          }
        }
        __syncwarp();
        if (lane < m) {
          float acc = 0.f;
#pragma unroll 8
          for (int k = 0; k < TC_DIM; k += 4) {
            const float4 t = *reinterpret_cast<const float4*>(&s_term[w][lane][k]);
            acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, t.x), t.y), t.z), t.w);
          }
          // the least (distance, index) of each query; a NaN distance never wins
          if (acc <= __int_as_float(0x7f800000))
            atomicMin(&s_best[w][s_of[w][b0 + lane]],
                      ((unsigned long long)__float_as_uint(acc) << 32) | (unsigned)s_cand[w][b0 + lane]);
        }
        __syncwarp();
      }
    }
    __syncwarp();
    const int i = base + lane;
    if (lane < per && i < nq) {
      const unsigned long long best = s_best[w][lane];
      if (qzero[i] != 0) {
        // an all-zero query ties (up to rounding) with every unit-norm row: its
        // answer is the database's, the row of least exact sequential |b|^2
        // (lowest index on ties), found when the database was split
        const unsigned long long key = *zero_best;
        out_idx[i] = key == ~0ull ? -1 : (int)(unsigned)(key & 0xffffffffull);
        if (out_d2) out_d2[i] = key == ~0ull ? __int_as_float(0x7f800000) : __uint_as_float((unsigned)(key >> 32));
      } else {
        const float bd = best == ~0ull ? __int_as_float(0x7f800000) : __uint_as_float((unsigned)(best >> 32));
        const bool all_seen = ndb < TC_TOP;  // every descriptor was a candidate
        // the bound scales with the norms: |err| <= TC_ERR * max(|q|, |b|max)^2
        const float err = TC_ERR * fmaxf(qn[i], dbm);
        if (all_seen || s_worst[w][lane] - err > bd) {
          out_idx[i] = best == ~0ull ? -1 : (int)(unsigned)(best & 0xffffffffull);
          if (out_d2) out_d2[i] = bd;
        } else {
          const int p = atomicAdd(n_redo, 1);
          redo[p] = i;
          redo_best[p] = ~0ull;
          // a row that ties or beats the exact winner has d~ <= bd + err; the
          // band pass lists rows up to twice that margin
          redo_thr[p] = bd + 2.f * err;
        }
      }
    }
    __syncwarp();  // the lists are reused
  }
}

// The answer for an all-zero query: min over rows of the exact sequential
// sum of (0 - b_k)^2 = b_k^2 (each operation rounded, as exact_d2 with a
// zero row), packed (d^2 bits, index) so that atomicMin keeps the lowest
// index on ties.  Rows with an infinite or NaN sum never win.  It depends on
// the database only: computed when the database is split.
// A block takes 32 rows: all threads bring them to shared memory (coalesced),
// one warp adds them up, a row a lane (rows 353 floats apart: no conflicts).
constexpr int ZB_ROWS = 32;
__global__ void __launch_bounds__(256) k_zero_best(const float* __restrict__ db, int ndb,
                                                   unsigned long long* __restrict__ best) {
  __shared__ float s_row[ZB_ROWS][TC_DIM + 1];
  const int j0 = blockIdx.x * ZB_ROWS, rows = min(ZB_ROWS, ndb - j0);
  for (int i = threadIdx.x; i < rows * TC_DIM; i += blockDim.x) s_row[i / TC_DIM][i % TC_DIM] = db[(size_t)j0 * TC_DIM + i];
  __syncthreads();
  if ((int)threadIdx.x >= rows) return;
  float acc = 0.f;
#pragma unroll 8
  for (int k = 0; k < TC_DIM; ++k) {
    const float t = __fsub_rn(0.f, s_row[threadIdx.x][k]);
    acc = __fadd_rn(acc, __fmul_rn(t, t));
  }
  if (acc < __int_as_float(0x7f800000))
    atomicMin(best, ((unsigned long long)__float_as_uint(acc) << 32) | (unsigned)(j0 + threadIdx.x));
}

__global__ void k_band_gather(const uint4* __restrict__ qhi, const uint4* __restrict__ qlo,
                              const float* __restrict__ qn, const int* __restrict__ redo,
                              const int* __restrict__ n_redo, int cap, uint4* __restrict__ hi2, uint4* __restrict__ lo2,
                              float* __restrict__ qn2) {
  const int n = min(*n_redo, cap);
  constexpr int V = TC_KPAD * 2 / 16;  // uint4 per row
  const int lane = threadIdx.x & 31;
  for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < n; w += gridDim.x * (blockDim.x >> 5)) {
    const int i = redo[w];
    for (int k = lane; k < V; k += 32) {
      hi2[(size_t)w * V + k] = qhi[(size_t)i * V + k];
      lo2[(size_t)w * V + k] = qlo[(size_t)i * V + k];
    }
    if (lane == 0) qn2[w] = qn[i];
  }
}

// Band pass, step 3: exact FP32 distances to the listed rows, a block per
// query and a thread per row (a band holds at most TC_BAND = 256 rows).  The
// band holds every row that can tie or beat the exact winner, so its exact
// minimum (lowest index on ties) is the scan's.  Queries past TC_BAND_Q,
// with a band over TC_BAND rows, or with a non-finite threshold (Inf or NaN
// values) go to the full scan list.
template <bool V4>
__global__ void __launch_bounds__(256) k_band_rerank(const float* __restrict__ q, const float* __restrict__ db,
                                                     const int* __restrict__ redo, const int* __restrict__ n_redo,
                                                     const float* __restrict__ thr, const int* __restrict__ band_idx,
                                                     const int* __restrict__ band_n, int cap, int ndb,
                                                     unsigned long long* __restrict__ redo_best,
                                                     int* __restrict__ full, int* __restrict__ n_full) {
  static_assert(TC_BAND <= 256, "a thread per band row");
  __shared__ unsigned long long s_min[8];
  const int n = *n_redo;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {  // uniform per block
    const int cnt = w < cap ? band_n[w] : TC_BAND + 1;
    if (cnt > TC_BAND || !isfinite(w < cap ? thr[w] : 0.f)) {
      if (threadIdx.x == 0) full[atomicAdd(n_full, 1)] = w;
      continue;
    }
    const int i = redo[w];
    unsigned long long key = ~0ull;
    const int m = threadIdx.x;
    if (m < cnt) {
      const int j = band_idx[(size_t)w * TC_BAND + m];
      if ((unsigned)j < (unsigned)ndb) {  // (out of range only after a timed-out band pass, status set)
        const float d = exact_d2<V4>(q + (size_t)i * TC_DIM, db + (size_t)j * TC_DIM);
        if (d < __int_as_float(0x7f800000)) key = ((unsigned long long)__float_as_uint(d) << 32) | (unsigned)j;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long ok = __shfl_xor_sync(0xffffffffu, key, o);
      key = ok < key ? ok : key;
    }
    if (lane == 0) s_min[warp] = key;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long b = s_min[0];
#pragma unroll
      for (int k = 1; k < 8; ++k) b = s_min[k] < b ? s_min[k] : b;
      redo_best[w] = b;
    }
    __syncthreads();  // s_min is reused by the next query
  }
}

// Exact scan for the queries the band pass could not settle: one CTA per
// (query, 256 database rows), thread per row; the winner is the minimum of
// (d^2 bits, index) packed in 64 bits (d^2 >= 0, so its bits order like the
// value).  A row wins only with d^2 < +inf, as in the sequential scan.
template <bool V4>
__global__ void __launch_bounds__(256) k_match_redo(const float* __restrict__ q, const float* __restrict__ db, int ndb,
                                                    const int* __restrict__ redo, const int* __restrict__ full,
                                                    const int* __restrict__ n_full,
                                                    unsigned long long* __restrict__ redo_best) {
  const int n = *n_full;
  const int rblocks = (ndb + 255) >> 8;
  const int lane = threadIdx.x & 31;
  for (long long item = blockIdx.x; item < (long long)n * rblocks; item += gridDim.x) {
    const int w = full[(int)(item / rblocks)], rb = (int)(item % rblocks);
    const int i = redo[w];
    const int j = rb * 256 + threadIdx.x;
    unsigned long long key = ~0ull;
    if (j < ndb) {
      const float d = exact_d2<V4>(q + (size_t)i * TC_DIM, db + (size_t)j * TC_DIM);
      if (d < __int_as_float(0x7f800000)) key = ((unsigned long long)__float_as_uint(d) << 32) | (unsigned)j;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long ok = __shfl_xor_sync(0xffffffffu, key, o);
      key = ok < key ? ok : key;
    }
    if (lane == 0 && key != ~0ull) atomicMin(redo_best + w, key);
  }
}

__global__ void k_match_redo_out(const int* __restrict__ redo, const int* __restrict__ n_redo,
                                 const unsigned long long* __restrict__ redo_best, int* __restrict__ out_idx,
                                 float* __restrict__ out_d2) {
  const int n = *n_redo;
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < n; w += gridDim.x * blockDim.x) {
    const int i = redo[w];
    const unsigned long long key = redo_best[w];
    out_idx[i] = key == ~0ull ? -1 : (int)(unsigned)(key & 0xffffffffull);
    if (out_d2) out_d2[i] = key == ~0ull ? __int_as_float(0x7f800000) : __uint_as_float((unsigned)(key >> 32));
  }
}

// ---------------------------------------------------------------------------
// host: tensor maps through the driver entry point (no libcuda link)
// ---------------------------------------------------------------------------
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static PFN_encodeTiled get_encode() {
  // resolved once (thread-safe static initialisation)
  static const PFN_encodeTiled fn = []() -> PFN_encodeTiled {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<PFN_encodeTiled>(p);
    return nullptr;
  }();
  return fn;
}

static bool make_map(CUtensorMap* m, const void* base, int rows, int box_rows) {
  PFN_encodeTiled enc = get_encode();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)TC_KPAD, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)TC_KPAD * 2};
  const cuuint32_t box[2] = {(cuuint32_t)TC_KB, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, TC_SW == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

size_t match_tc_bf16_bytes(int rows) { return (size_t)rows * TC_KPAD * 2; }

// rows of the band pass (a multiple of TC_BM)
static int band_rows(int nqp) { return nqp < TC_BAND_Q ? nqp : TC_BAND_Q; }

// mbarrier tries per wait for the context's wait budget (a try is a few
// dozen cycles; the default 2 s budget gives about 2^26 tries)
static long long tc_spin_limit(const rtr_context* ctx) {
  const long long t = ctx->wait_budget_cycles / 64;
  return t < 1 ? 1 : t;
}

// Database ranges of the first pass: the fewest waves of CTAs times tiles of a
// CTA (its start costs about half a tile), where a few queries would leave SMs
// idle.  The lists of the ranges after the first have to fit in the band
// pass's rows.
static int match_ranges(int nqp, int ndb, int bq) {
  const int sms = 152, tiles = (ndb + TC_BN - 1) / TC_BN;
  const long long ctas = nqp / TC_BM;
  int best = 1;
  double cost = 0.0;
  for (int r = 1; r <= TC_RANGES && r <= tiles; ++r) {
    if ((long long)(r - 1) * nqp * TC_TOP * 2 > (long long)bq * TC_BAND) break;
    const double c = (double)((ctas * r + sms - 1) / sms) * ((tiles + r - 1) / r + 0.6);
    if (r == 1 || c < 0.97 * cost) {
      best = r;
      cost = c;
    }
  }
  return best;
}

void match_tc_plan(ScratchPlan& p, int nq_cap, bool with_db, int ndb) {
  const int nqp = ((nq_cap + TC_BM - 1) / TC_BM) * TC_BM;
  p.add<__nv_bfloat16>((size_t)nqp * TC_KPAD);
  p.add<__nv_bfloat16>((size_t)nqp * TC_KPAD);
  p.add<float>(nqp);
  if (with_db) {
    p.add<__nv_bfloat16>((size_t)ndb * TC_KPAD);
    p.add<__nv_bfloat16>((size_t)ndb * TC_KPAD);
    p.add<float>(db_norm_floats(ndb));
  }
  p.add<int>((size_t)nqp * TC_TOP);
  p.add<float>((size_t)nqp * TC_TOP);
  p.add<int>(nqp);
  p.add<unsigned long long>(nqp);
  p.add<int>(4);
  // band pass
  const int bq = band_rows(nqp);
  p.add<float>(nqp);
  p.add<int>(nqp);
  p.add<__nv_bfloat16>((size_t)bq * TC_KPAD);
  p.add<__nv_bfloat16>((size_t)bq * TC_KPAD);
  p.add<float>(bq);
  p.add<int>((size_t)bq * TC_BAND);
  p.add<int>(bq);
  p.add<unsigned char>(nqp);
}

// Splits a descriptor database once (the model side keeps the result).
rtr_status match_tc_prepare_db(const float* db, int ndb, __nv_bfloat16* hi, __nv_bfloat16* lo, float* norm2,
                               cudaStream_t st) {
  int blocks = (ndb + 7) / 8;
  if (blocks > 152 * 16) blocks = 152 * 16;
  if (blocks < 1) blocks = 1;
  // norm2[ndb] receives the largest squared norm (scales the error bound),
  // db_zero_key the answer for an all-zero query
  RTR_CUDA(cudaMemsetAsync(norm2 + ndb, 0, sizeof(float), st));
  RTR_CUDA(cudaMemsetAsync(db_zero_key(norm2, ndb), 0xff, sizeof(unsigned long long), st));
  k_split_bf16<<<blocks, 256, 0, st>>>(db, ndb, nullptr, ndb, hi, lo, norm2, reinterpret_cast<unsigned*>(norm2 + ndb),
                                       true, nullptr);
  k_zero_best<<<ndb > 0 ? (ndb + ZB_ROWS - 1) / ZB_ROWS : 1, 256, 0, st>>>(db, ndb, db_zero_key(norm2, ndb));
  RTR_LAUNCHED(2);
  RTR_CUDA(cudaGetLastError());
  return RTR_OK;
}

rtr_status match_tc_dev(rtr_context* ctx, Scratch& s, const float* q, int nq_cap, const int* d_nq, const float* db,
                        int ndb, const __nv_bfloat16* db_hi, const __nv_bfloat16* db_lo, const float* db_n2,
                        int* out_idx, float* out_d2, cudaStream_t st) {
  const int nqp = ((nq_cap + TC_BM - 1) / TC_BM) * TC_BM;
  __nv_bfloat16* qhi = s.take<__nv_bfloat16>((size_t)nqp * TC_KPAD);
  __nv_bfloat16* qlo = s.take<__nv_bfloat16>((size_t)nqp * TC_KPAD);
  float* qn = s.take<float>(nqp);
  if (!db_hi) {
    __nv_bfloat16* h = s.take<__nv_bfloat16>((size_t)ndb * TC_KPAD);
    __nv_bfloat16* l = s.take<__nv_bfloat16>((size_t)ndb * TC_KPAD);
    float* n2 = s.take<float>(db_norm_floats(ndb));
    if (!n2) return fail(RTR_ERR_CAPACITY, "match_tc: scratch");
    RTR_TRY(match_tc_prepare_db(db, ndb, h, l, n2, st));
    db_hi = h;
    db_lo = l;
    db_n2 = n2;
  }
  int* cidx = s.take<int>((size_t)nqp * TC_TOP);
  float* cd = s.take<float>((size_t)nqp * TC_TOP);
  int* redo = s.take<int>(nqp);
  unsigned long long* redo_best = s.take<unsigned long long>(nqp);
  int* nredo = s.take<int>(4);  // [0] uncertified, [1] left to the full scan
  const int bq = band_rows(nqp);
  float* redo_thr = s.take<float>(nqp);
  int* full = s.take<int>(nqp);
  __nv_bfloat16* hi2 = s.take<__nv_bfloat16>((size_t)bq * TC_KPAD);
  __nv_bfloat16* lo2 = s.take<__nv_bfloat16>((size_t)bq * TC_KPAD);
  float* qn2 = s.take<float>(bq);
  int* band_idx = s.take<int>((size_t)bq * TC_BAND);
  int* band_n = s.take<int>(bq);
  unsigned char* qzero = s.take<unsigned char>(nqp);
  if (!qzero) return fail(RTR_ERR_CAPACITY, "match_tc: scratch");
  int sb = (nqp + 7) / 8;
  if (sb > 152 * 16) sb = 152 * 16;
  {
    ProfScope pp(ctx, st, "match_split");
    k_split_bf16<<<sb, 256, 0, st>>>(q, nq_cap, d_nq, nqp, qhi, qlo, qn, nullptr, false, qzero);
  }
  CUtensorMap m_qh, m_ql, m_bh, m_bl, m_qh2, m_ql2;
  if (!make_map(&m_qh, qhi, nqp, TC_BM) || !make_map(&m_ql, qlo, nqp, TC_BM) || !make_map(&m_bh, db_hi, ndb, TC_BN) ||
      !make_map(&m_bl, db_lo, ndb, TC_BN) || !make_map(&m_qh2, hi2, bq, TC_BM) || !make_map(&m_ql2, lo2, bq, TC_BM))
    return fail(RTR_ERR_CUDA, "match_tc: cuTensorMapEncodeTiled failed");
  const size_t smem = (size_t)TC_STAGES * TC_STAGE_BYTES + 1024;
  const size_t top_smem = smem + TC_BM * TC_ROW * sizeof(float);
  // per call: the attribute is per device, and calls may come from several threads
  RTR_CUDA(cudaFuncSetAttribute(k_match_top, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)top_smem));
  RTR_CUDA(cudaFuncSetAttribute(k_match_band, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // The lists of further ranges lie in the band pass's rows (written after
  // the re-rank has read them).
  const int ranges = match_ranges(nqp, ndb, bq);
  int* more_idx = band_idx;
  float* more_d = reinterpret_cast<float*>(band_idx + (size_t)(ranges - 1) * nq_cap * TC_TOP);
  TcArgs a{nq_cap, d_nq, nq_cap, ndb, qn, cidx, cd, more_idx, more_d, ctx->d_status, nullptr, nullptr,
           tc_spin_limit(ctx)};
  {
    ProfScope pg(ctx, st, "match_gemm");
    k_match_top<<<dim3(nqp / TC_BM, ranges), TC_THREADS, top_smem, st>>>(m_qh, m_ql, m_bh, m_bl, a);
  }
  RTR_CUDA(cudaMemsetAsync(nredo, 0, 2 * sizeof(int), st));
  const int per = rr_queries(nq_cap);
  int rb = (nq_cap + RR_WARPS * per - 1) / (RR_WARPS * per);
  if (rb > 152 * 16) rb = 152 * 16;
  // block per uncertified query (grid-stride over the device-side count)
  const int wb = band_rows(nqp) < 152 * 8 ? band_rows(nqp) : 152 * 8;
  const bool v4 = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(db)) & 15u) == 0;
  // band pass over the uncertified queries: the GEMM again, listing every
  // row within the tie margin, then exact distances to those rows only
  TcArgs ab{bq, nredo, bq, ndb, qn2, band_idx, nullptr, nullptr, nullptr, ctx->d_status, redo_thr, band_n, tc_spin_limit(ctx)};
  ProfScope pr(ctx, st, "match_rerank");
  if (v4)
    k_rerank<true><<<rb, 32 * RR_WARPS, 0, st>>>(q, nq_cap, d_nq, nq_cap, db, ndb, cidx, cd, more_idx, more_d, ranges,
                                                 per, out_idx, out_d2, redo, nredo, redo_best, redo_thr, qn,
                                                 db_n2 + ndb, db_zero_key(db_n2, ndb), qzero);
  else
    k_rerank<false><<<rb, 32 * RR_WARPS, 0, st>>>(q, nq_cap, d_nq, nq_cap, db, ndb, cidx, cd, more_idx, more_d, ranges,
                                                  per, out_idx, out_d2, redo, nredo, redo_best, redo_thr, qn,
                                                  db_n2 + ndb, db_zero_key(db_n2, ndb), qzero);
  pr.end();
  ProfScope pu(ctx, st, "match_uncertified");
  k_band_gather<<<(bq + 7) / 8 < 152 * 2 ? (bq + 7) / 8 : 152 * 2, 256, 0, st>>>(reinterpret_cast<const uint4*>(qhi), reinterpret_cast<const uint4*>(qlo),
                                              qn, redo, nredo, bq, reinterpret_cast<uint4*>(hi2),
                                              reinterpret_cast<uint4*>(lo2), qn2);
  RTR_CUDA(cudaMemsetAsync(band_n, 0, sizeof(int) * bq, st));
  {
    ProfScope pb(ctx, st, "match_band");
    const int n_tiles = (ndb + TC_BN - 1) / TC_BN;
    const dim3 grid(bq / TC_BM, n_tiles < 8 ? n_tiles : 8);
    k_match_band<<<grid, TC_THREADS, smem, st>>>(m_qh2, m_ql2, m_bh, m_bl, ab);
  }
  if (v4) {
    k_band_rerank<true><<<wb, 256, 0, st>>>(q, db, redo, nredo, redo_thr, band_idx, band_n, bq, ndb, redo_best, full,
                                            nredo + 1);
    k_match_redo<true><<<152 * 8, 256, 0, st>>>(q, db, ndb, redo, full, nredo + 1, redo_best);
  } else {
    k_band_rerank<false><<<wb, 256, 0, st>>>(q, db, redo, nredo, redo_thr, band_idx, band_n, bq, ndb, redo_best, full,
                                             nredo + 1);
    k_match_redo<false><<<152 * 8, 256, 0, st>>>(q, db, ndb, redo, full, nredo + 1, redo_best);
  }
  k_match_redo_out<<<4, 256, 0, st>>>(redo, nredo, redo_best, out_idx, out_d2);
  RTR_LAUNCHED(9);
  // keep the number of uncertified queries and of full scans for rtr_match_stats
  RTR_CUDA(cudaMemcpyAsync(ctx->d_status + 8, nredo, 2 * sizeof(int), cudaMemcpyDeviceToDevice, st));
  RTR_CUDA(cudaGetLastError());
  return RTR_OK;
}

// ---------------------------------------------------------------------------
// Keypoint-credibility MLP inference on the tensor cores: 352 -> 128 -> 64
// -> 1 (ReLU, ReLU, sigmoid) with BF16 weights.  Layer 1 is a tcgen05 GEMM:
// each FP32 descriptor is split into three BF16 parts (hi + mid + lo = x up
// to the last part's rounding, 2^-24 of |x|), and the three products with
// the BF16 weights accumulate in FP32 in tensor memory: FP32-level accuracy.
// The epilogue (thread = row) adds the bias, applies the ReLU, runs layer 2
// (64 outputs, FP32 FMAs over the 128 inputs in order), the head and the
// sigmoid, so only the score leaves the CTA.
// ---------------------------------------------------------------------------
constexpr int MLP_TC_IN = 352, MLP_TC_H1 = 128, MLP_TC_H2 = 64;
constexpr int MLP_TC_A_BYTES = TC_BM * TC_KB * 2;     // 8 KB: one part's K-block
constexpr int MLP_TC_B_BYTES = MLP_TC_H1 * TC_KB * 2;  // 8 KB: W1's K-block
constexpr int MLP_TC_STAGE_BYTES = 3 * MLP_TC_A_BYTES + MLP_TC_B_BYTES;  // 32 KB
constexpr int MLP_TC_STAGES = 4;
constexpr int MLP_TC_SMEM = MLP_TC_STAGES * MLP_TC_STAGE_BYTES + 1024;

// hi / mid / lo BF16 parts of each row, padded to TC_KPAD (zero past 352 and
// in padding rows); a warp per row, four columns per lane and 16-byte loads.
__global__ void k_split3_bf16(const float* __restrict__ x, int n_cap_rows, const int* d_n, int n_pad,
                              __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ mid,
                              __nv_bfloat16* __restrict__ lo) {
  const int n = d_n ? min(*d_n, n_cap_rows) : n_cap_rows;
  const int lane = threadIdx.x & 31;
  for (int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < n_pad; r += gridDim.x * (blockDim.x >> 5)) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int c4 = lane + 32 * k;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < n && c4 < MLP_TC_IN / 4) v = __ldg(reinterpret_cast<const float4*>(x + (size_t)r * MLP_TC_IN) + c4);
      const float e[4] = {v.x, v.y, v.z, v.w};
      unsigned short h[4], m[4], l[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat16 bh = __float2bfloat16_rn(e[j]);
        const float r1 = e[j] - __bfloat162float(bh);
        const __nv_bfloat16 bm = __float2bfloat16_rn(r1);
        const __nv_bfloat16 bl = __float2bfloat16_rn(r1 - __bfloat162float(bm));
        h[j] = __bfloat16_as_ushort(bh);
        m[j] = __bfloat16_as_ushort(bm);
        l[j] = __bfloat16_as_ushort(bl);
      }
      const size_t o = (size_t)r * (TC_KPAD / 4) + c4;
      reinterpret_cast<uint2*>(hi)[o] = make_uint2(h[0] | ((unsigned)h[1] << 16), h[2] | ((unsigned)h[3] << 16));
      reinterpret_cast<uint2*>(mid)[o] = make_uint2(m[0] | ((unsigned)m[1] << 16), m[2] | ((unsigned)m[3] << 16));
      reinterpret_cast<uint2*>(lo)[o] = make_uint2(l[0] | ((unsigned)l[1] << 16), l[2] | ((unsigned)l[3] << 16));
    }
  }
}

__device__ __forceinline__ uint32_t umma_idesc_n(int n) {
  uint32_t d = 0;
  d |= 1u << 4;                        // D format F32
  d |= 1u << 7;                        // A BF16
  d |= 1u << 10;                       // B BF16
  d |= (uint32_t)(n >> 3) << 17;       // N
  d |= (uint32_t)(TC_BM >> 4) << 24;   // M
  return d;
}

struct MlpTcArgs {
  int n_cap;
  const int* d_n;
  const float* b1;         // [128]
  const __nv_bfloat16* w2;  // [64][128]
  const float* b2;         // [64]
  const __nv_bfloat16* w3;  // [64]
  const float* b3;         // [1]
  float* score;            // [n]
  int* status;
  long long spin_limit;
};

__global__ void __launch_bounds__(TC_THREADS, 1) k_mlp_tc(const __grid_constant__ CUtensorMap m_hi,
                                                          const __grid_constant__ CUtensorMap m_mid,
                                                          const __grid_constant__ CUtensorMap m_lo,
                                                          const __grid_constant__ CUtensorMap m_w1, MlpTcArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[MLP_TC_STAGES], empty_bar[MLP_TC_STAGES], acc_full, drain_bar;
  __shared__ uint32_t tmem_base;
  __shared__ int abort_flag;
  __shared__ float s_w2[MLP_TC_H1][MLP_TC_H2];  // [input c][output j]
  __shared__ float s_b1[MLP_TC_H1], s_b2[MLP_TC_H2], s_w3[MLP_TC_H2];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = a.d_n ? min(*a.d_n, a.n_cap) : a.n_cap;
  const int q0 = blockIdx.x * TC_BM;
  if (q0 >= n) return;  // uniform per CTA, before any barrier or TMEM use

  for (int i = threadIdx.x; i < MLP_TC_H1 * MLP_TC_H2; i += blockDim.x) {
    const int j = i / MLP_TC_H1, c = i - j * MLP_TC_H1;  // w2 row-major [j][c]
    s_w2[c][j] = __bfloat162float(a.w2[i]);
  }
  for (int i = threadIdx.x; i < MLP_TC_H1; i += blockDim.x) s_b1[i] = a.b1[i];
  for (int i = threadIdx.x; i < MLP_TC_H2; i += blockDim.x) {
    s_b2[i] = a.b2[i];
    s_w3[i] = __bfloat162float(a.w3[i]);
  }
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < MLP_TC_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_full, 1);
    mbar_init(&drain_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 5) {  // 128 TMEM columns: one 128 x 128 FP32 accumulator
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 128;" ::"r"(smem_u32(&tmem_base)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  volatile int* abort = &abort_flag;
  const long long lim = a.spin_limit;
  int issued = 0;

  if (warp == 4) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int kb = 0;
      for (; kb < TC_NKB && !*abort; ++kb) {
        const int s = kb % MLP_TC_STAGES;
        const uint32_t ph = (uint32_t)(kb / MLP_TC_STAGES) & 1u;
        if (kb >= MLP_TC_STAGES && !mbar_wait(&empty_bar[s], ph ^ 1u, abort, lim)) break;
        uint8_t* st = smem + s * MLP_TC_STAGE_BYTES;
        mbar_expect_tx(&full_bar[s], MLP_TC_STAGE_BYTES);
        tma_load_2d(st, &m_hi, &full_bar[s], kb * TC_KB, q0);
        tma_load_2d(st + MLP_TC_A_BYTES, &m_mid, &full_bar[s], kb * TC_KB, q0);
        tma_load_2d(st + 2 * MLP_TC_A_BYTES, &m_lo, &full_bar[s], kb * TC_KB, q0);
        tma_load_2d(st + 3 * MLP_TC_A_BYTES, &m_w1, &full_bar[s], kb * TC_KB, 0);
      }
      issued = kb;
    }
  } else if (warp == 5) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      const uint32_t idesc = umma_idesc_n(MLP_TC_H1);
      bool ok = true;
      for (int kb = 0; kb < TC_NKB; ++kb) {
        const int s = kb % MLP_TC_STAGES;
        const uint32_t ph = (uint32_t)(kb / MLP_TC_STAGES) & 1u;
        if (!mbar_wait(&full_bar[s], ph, abort, lim)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t base = smem_u32(smem + s * MLP_TC_STAGE_BYTES);
        const uint32_t ah = base, am = base + MLP_TC_A_BYTES, al = base + 2 * MLP_TC_A_BYTES,
                       bw = base + 3 * MLP_TC_A_BYTES;
#pragma unroll
        for (int k = 0; k < TC_KB / 16; ++k) {
          const uint32_t off = (uint32_t)k * 32;  // 16 bf16 along K inside the swizzle row
          const uint32_t acc0 = (kb > 0 || k > 0) ? 1u : 0u;
          umma_f16(tmem, umma_desc(ah + off), umma_desc(bw + off), idesc, acc0);
          umma_f16(tmem, umma_desc(am + off), umma_desc(bw + off), idesc, 1u);
          umma_f16(tmem, umma_desc(al + off), umma_desc(bw + off), idesc, 1u);
        }
        umma_commit(&empty_bar[s]);
      }
      if (ok) umma_commit(&acc_full);
    }
  } else {
    // ---------------- epilogue: warps 0-3, thread = row ----------------
    const int row = warp * 32 + lane;
    const int q = q0 + row;
    if (mbar_wait(&acc_full, 0u, abort, lim)) {
      tc_fence_after();
      float h2[MLP_TC_H2];
#pragma unroll
      for (int j = 0; j < MLP_TC_H2; ++j) h2[j] = 0.f;
      const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
      for (int c0 = 0; c0 < MLP_TC_H1; c0 += 32) {
        float v[32];
        tmem_ld32(taddr + (uint32_t)c0, v);
#pragma unroll 4
        for (int i = 0; i < 32; ++i) {
          const float h = fmaxf(v[i] + s_b1[c0 + i], 0.f);
#pragma unroll
          for (int j = 0; j < MLP_TC_H2; ++j) h2[j] = fmaf(h, s_w2[c0 + i][j], h2[j]);
        }
      }
      float z = 0.f;
#pragma unroll
      for (int j = 0; j < MLP_TC_H2; ++j) z = fmaf(fmaxf(h2[j] + s_b2[j], 0.f), s_w3[j], z);
      z += *a.b3;
      if (q < n) a.score[q] = 1.f / (1.f + __expf(-z));
    }
  }
  __syncthreads();
  if (abort_flag) {
    if (warp == 5 && lane == 0) {
      umma_commit(&drain_bar);
      mbar_drain(&drain_bar, 0u);
    }
    if (warp == 4 && lane == 0)
      for (int i = issued > MLP_TC_STAGES ? issued - MLP_TC_STAGES : 0; i < issued; ++i)
        mbar_drain(&full_bar[i % MLP_TC_STAGES], (uint32_t)(i / MLP_TC_STAGES) & 1u);
  }
  tc_fence_before();
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) atomicExch(a.status, (int)RTR_ERR_TIMEOUT);
  if (warp == 5) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 128;" ::"r"(tmem));
  }
}

size_t mlp_tc_bytes(int n_cap) {
  const size_t nqp = (size_t)(((n_cap > 0 ? n_cap : 1) + TC_BM - 1) / TC_BM) * TC_BM;
  ScratchPlan p;
  for (int i = 0; i < 3; ++i) p.add<__nv_bfloat16>(nqp * TC_KPAD);
  return p.bytes;
}

// Scores of rows X[0 .. *d_n) (n_cap rows of capacity).  w1pad: W1 as BF16
// [128][TC_KPAD] with zero columns past 352; theta_b1/b2/b3: the FP32 biases.
rtr_status mlp_tc_score(rtr_context* ctx, Scratch& s, const float* X, int n_cap, const int* d_n,
                        const __nv_bfloat16* w1pad, const float* b1, const __nv_bfloat16* w2, const float* b2,
                        const __nv_bfloat16* w3, const float* b3, float* score, cudaStream_t st) {
  if (n_cap <= 0) return RTR_OK;
  const int nqp = ((n_cap + TC_BM - 1) / TC_BM) * TC_BM;
  __nv_bfloat16* hi = s.take<__nv_bfloat16>((size_t)nqp * TC_KPAD);
  __nv_bfloat16* mid = s.take<__nv_bfloat16>((size_t)nqp * TC_KPAD);
  __nv_bfloat16* lo = s.take<__nv_bfloat16>((size_t)nqp * TC_KPAD);
  if (!lo) return fail(RTR_ERR_CAPACITY, "mlp_tc: scratch");
  int sb = (nqp + 7) / 8;
  if (sb > 152 * 16) sb = 152 * 16;
  k_split3_bf16<<<sb, 256, 0, st>>>(X, n_cap, d_n, nqp, hi, mid, lo);
  CUtensorMap mh, mm, ml, mw;
  if (!make_map(&mh, hi, nqp, TC_BM) || !make_map(&mm, mid, nqp, TC_BM) || !make_map(&ml, lo, nqp, TC_BM) ||
      !make_map(&mw, w1pad, MLP_TC_H1, MLP_TC_H1))
    return fail(RTR_ERR_CUDA, "mlp_tc: cuTensorMapEncodeTiled failed");
  RTR_CUDA(cudaFuncSetAttribute(k_mlp_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, MLP_TC_SMEM));
  MlpTcArgs a{n_cap, d_n, b1, w2, b2, w3, b3, score, ctx->d_status, tc_spin_limit(ctx)};
  k_mlp_tc<<<nqp / TC_BM, TC_THREADS, MLP_TC_SMEM, st>>>(mh, mm, ml, mw, a);
  RTR_LAUNCHED(2);
  RTR_CUDA(cudaGetLastError());
  return RTR_OK;
}

}  // namespace rtr

using namespace rtr;

extern "C" rtr_status rtr_match_stats(rtr_context* ctx, int* h_uncertified) {
  RTR_CHECK_ARG(ctx && h_uncertified, "rtr_match_stats: bad arguments");
  RTR_CUDA(cudaSetDevice(ctx->device));
  RTR_CUDA(cudaDeviceSynchronize());
  RTR_CUDA(cudaMemcpy(h_uncertified, ctx->d_status + 8, sizeof(int), cudaMemcpyDeviceToHost));
  return RTR_OK;
}

extern "C" rtr_status rtr_match_stats_ex(rtr_context* ctx, int* h_uncertified, int* h_full_scans) {
  RTR_CHECK_ARG(ctx && h_uncertified && h_full_scans, "rtr_match_stats_ex: bad arguments");
  RTR_CUDA(cudaSetDevice(ctx->device));
  RTR_CUDA(cudaDeviceSynchronize());
  int h[2];
  RTR_CUDA(cudaMemcpy(h, ctx->d_status + 8, sizeof(h), cudaMemcpyDeviceToHost));
  *h_uncertified = h[0];
  *h_full_scans = h[1];
  return RTR_OK;
}

extern "C" rtr_status rtr_match(rtr_context* ctx, const float* d_query, int n_query, const float* d_db, int n_db,
                                int32_t* d_idx, float* d_d2, rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && n_query >= 0 && n_db >= 0, "rtr_match: bad arguments");
  if (n_query == 0) return RTR_OK;
  RTR_CHECK_ARG(d_query && d_idx, "rtr_match: NULL query or output");
  cudaStream_t st = (cudaStream_t)stream;
  RTR_CUDA(cudaSetDevice(ctx->device));
  if (n_db == 0) {
    RTR_CUDA(cudaMemsetAsync(d_idx, 0xff, (size_t)n_query * 4, st));
    return RTR_OK;
  }
  RTR_CHECK_ARG(d_db != nullptr, "rtr_match: NULL database");
  ScratchPlan p;
  match_tc_plan(p, n_query, true, n_db);
  Scratch s;
  RTR_TRY(ensure_scratch(ctx, p.bytes, st, &s));
  ProfScope ps(ctx, st, "match_tc");
  return match_tc_dev(ctx, s, d_query, n_query, nullptr, d_db, n_db, nullptr, nullptr, nullptr, d_idx, d_d2, st);
}
