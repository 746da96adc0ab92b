// tdf.cu — truncated distance field of occupied voxels.
//
// Replaces ComputeTDF / ComputeTDFWithCuda (kernel.cu:8-106).  For every voxel
// v = (x, y, z) of a dim^3 grid (x fastest), value = min(900, min_i |v - o_i|^2)
// over the integer occupied voxels o_i, stored as float (kernel.cu:20-30).
// All values are integers below 2^24, so the float result is exact and equal to
// the reference's.
//
// Layout here: a thread owns XP voxels of one x-row of one keypoint, so
// dy^2 + dz^2 is computed once per occupied voxel for the XP of them, and the
// occupied list is staged through shared memory in chunks.  The inner step is
// one multiply-add and one minimum per (voxel, occupied voxel):
//   dx^2 + dyz = x^2 + (x * (-2 ox) + (ox^2 + dyz)),
// with x^2 added after the minimum over the list.
//
// What bounds it: with many keypoints the integer pipe; with few, the length
// of one thread's walk over the list on a nearly idle chip.  So a row is cut
// in four (XP = 8) when whole rows (XP = 32) would leave SMs without a block.
// One keypoint, 180 occupied voxels, dim 30 on GB300: a CTA of 1024 threads
// per keypoint with whole rows took 101 us (one SM busy); XP = 8 over 29 CTAs
// takes 5.5 us from device memory and 9.5 us from and to page-locked memory.
#include <string.h>

#include "common.cuh"

namespace rtr {

constexpr int TDF_MAXDIM = 32;
constexpr int TDF_CHUNK = 1024;
constexpr int TDF_THREADS = 128;

// Occupied voxels of keypoint blockIdx.y: occ[3 * offsets[key]) ...
// 3 * offsets[key + 1]), or the n_occ voxels of occ when offsets is NULL.
// extra: one more voxel, (0, 0, dim), after the dim^3 of the grid.
template <int XP>
__global__ void __launch_bounds__(TDF_THREADS) k_tdf(const int* __restrict__ occ, const int* __restrict__ offsets,
                                                     int n_occ, int dim, int extra, float* __restrict__ out) {
  constexpr int PARTS = TDF_MAXDIM / XP;  // threads per row
  __shared__ int4 s_occ[TDF_CHUNK];       // y, z, -2 x, x^2
  const int key = blockIdx.y;
  const int beg = offsets ? offsets[key] : 0, end = offsets ? offsets[key + 1] : n_occ;
  const int rows = dim * dim + extra;
  float* o = out + (size_t)key * ((size_t)dim * dim * dim);
  const int t = (int)(blockIdx.x * TDF_THREADS + threadIdx.x);
  const int row = t / PARTS, x0 = (t % PARTS) * XP;
  const int y = row < dim * dim ? row % dim : 0, z = row < dim * dim ? row / dim : dim;
  const bool live = row < rows && x0 < dim;
  constexpr int FAR = 1 << 28;
  int best[XP];  // min over the list of x (-2 ox) + (ox^2 + dyz)
#pragma unroll
  for (int k = 0; k < XP; ++k) best[k] = FAR;
  for (int c0 = beg; c0 < end; c0 += TDF_CHUNK) {
    const int cn = min(TDF_CHUNK, end - c0);
    __syncthreads();
    for (int i = threadIdx.x; i < cn; i += TDF_THREADS) {
      const int* v = occ + 3 * (size_t)(c0 + i);
      const int ox = v[0], oy = v[1], oz = v[2];
      // a voxel 30 or more cells outside the grid along an axis lowers
      // nothing below 900: it is moved there, which keeps the products small
      const int cx = min(max(ox, -30), dim + 30), cy = min(max(oy, -30), dim + 30), cz = min(max(oz, -30), dim + 30);
      s_occ[i] = make_int4(cy, cz, -2 * cx, cx * cx);
    }
    __syncthreads();
    if (live) {
#pragma unroll 4
      for (int i = 0; i < cn; ++i) {
        const int4 v = s_occ[i];
        const int dy = y - v.x, dz = z - v.y;
        const int dyz = dy * dy + dz * dz;
        const int m = v.z, c = v.w + dyz;
#pragma unroll
        for (int k = 0; k < XP; ++k) best[k] = min(best[k], (x0 + k) * m + c);
      }
    }
  }
  // the CTA's rows are contiguous in the output: written through shared
  // memory, so that every store instruction covers whole lines (the output
  // may be page-locked host memory)
  constexpr int ROWS = TDF_THREADS / PARTS;
  __shared__ float s_out[ROWS * TDF_MAXDIM];
  const int row0 = (int)blockIdx.x * ROWS;
  if (live) {
#pragma unroll
    for (int k = 0; k < XP; ++k) {
      const int x = x0 + k;
      if (x < dim) s_out[(row - row0) * dim + x] = (float)min(900, best[k] + x * x);
    }
  }
  __syncthreads();
  const int nfull = min(ROWS, dim * dim - row0);  // whole rows (below 0: only the extra voxel, or none)
  const int count = max(nfull, 0) * dim + (row0 <= dim * dim && row0 + ROWS > dim * dim ? extra : 0);
  for (int i = threadIdx.x; i < count; i += TDF_THREADS) o[(size_t)row0 * dim + i] = s_out[i];
}

// Whole rows once they alone give three CTAs to every two SMs.  Measured on GB300
// (180 occupied voxels a keypoint, dim 30; whole rows / quarters, us): 1
// keypoint 11.1 / 5.5, 24: 17.7 / 14.5, 32: 17.8 / 19.1, 340: 136 / 158.
static void tdf_launch(const int* occ, const int* offsets, int n_occ, int n_keys, int dim, int extra, float* out,
                       cudaStream_t st) {
  const int rows = dim * dim + extra;
  const int whole = (rows + TDF_THREADS - 1) / TDF_THREADS;
  for (int k0 = 0; k0 < n_keys; k0 += 65535) {  // the grid's y limit
    const int nk = n_keys - k0 < 65535 ? n_keys - k0 : 65535;
    const int* off = offsets ? offsets + k0 : nullptr;
    float* o = out + (size_t)k0 * ((size_t)dim * dim * dim);
    if ((long long)whole * nk >= 3 * 152 / 2)
      k_tdf<32><<<dim3(whole, nk), TDF_THREADS, 0, st>>>(occ, off, n_occ, dim, extra, o);
    else
      k_tdf<8><<<dim3((rows * 4 + TDF_THREADS - 1) / TDF_THREADS, nk), TDF_THREADS, 0, st>>>(occ, off, n_occ, dim,
                                                                                            extra, o);
    RTR_LAUNCHED(1);
  }
}

// Buffers of the host-pointer shim, kept between calls (one host thread at a
// time, as with the reference).  Both directions go through page-locked
// memory that the kernel reads and writes itself: the call is one launch
// between two small host copies, without the four driver copies (and the
// pageable staging behind them) that made up 31 of its 133 us: 25 us now.  A list of
// over TDF_PIN_OCC voxels, which every CTA would read over the host link, is
// copied to the device first.
constexpr int TDF_PIN_OCC = 4096;
struct TdfShim {
  int* pin_occ = nullptr;    // [TDF_PIN_OCC][3], page-locked
  float* pin_tdf = nullptr;  // [27001], page-locked
  int* occ = nullptr;        // device list of a long call
  size_t occ_cap = 0;
};
static TdfShim g_tdf;

}  // namespace rtr

using namespace rtr;

extern "C" {

rtr_status rtr_tdf_batch(rtr_context* ctx, const int* d_occ, const int* d_offsets, int n_keys, int dim,
                         float* d_tdf, rtr_stream_t stream) {
  RTR_CHECK_ARG(ctx && n_keys >= 0, "rtr_tdf_batch: bad arguments");
  RTR_CHECK_ARG(dim >= 1 && dim <= TDF_MAXDIM, "rtr_tdf_batch: dim must be in [1, %d]", TDF_MAXDIM);
  if (n_keys == 0) return RTR_OK;
  RTR_CHECK_ARG(d_offsets && d_tdf, "rtr_tdf_batch: NULL offsets or output");
  RTR_CUDA(cudaSetDevice(ctx->device));
  ProfScope ps(ctx, (cudaStream_t)stream, "tdf");
  tdf_launch(d_occ, d_offsets, 0, n_keys, dim, 0, d_tdf, (cudaStream_t)stream);
  RTR_CUDA(cudaGetLastError());
  return RTR_OK;
}

int ComputeTDFWithCuda(const int* voxel_grid_occ, float* voxel_grid_TDF, int voxel_grid_dim,
                       int num_occ) {
  const int dim = voxel_grid_dim;
  if (dim < 1 || (long long)dim * dim * dim > 27000 || num_occ < 0 || !voxel_grid_TDF ||
      (num_occ > 0 && !voxel_grid_occ)) {
    set_error("ComputeTDFWithCuda: dim^3 must be in [1, 27000] and num_occ >= 0");
    return (int)cudaErrorInvalidValue;
  }
  cudaError_t e = cudaSetDevice(0);
  if (e != cudaSuccess) return (int)e;
  TdfShim& S = g_tdf;
  if (!S.pin_occ && (e = cudaMallocHost(&S.pin_occ, (size_t)TDF_PIN_OCC * 3 * sizeof(int))) != cudaSuccess) {
    S.pin_occ = nullptr;
    return (int)e;
  }
  if (!S.pin_tdf && (e = cudaMallocHost(&S.pin_tdf, 27001 * sizeof(float))) != cudaSuccess) {
    S.pin_tdf = nullptr;
    return (int)e;
  }
  const int* list = S.pin_occ;
  if (num_occ <= TDF_PIN_OCC) {
    if (num_occ > 0) memcpy(S.pin_occ, voxel_grid_occ, (size_t)num_occ * 3 * sizeof(int));
  } else {
    if ((size_t)num_occ > S.occ_cap) {
      if (S.occ) cudaFree(S.occ);
      S.occ = nullptr;
      S.occ_cap = 0;
      if ((e = cudaMalloc(&S.occ, (size_t)num_occ * 3 * sizeof(int))) != cudaSuccess) return (int)e;
      S.occ_cap = (size_t)num_occ;
    }
    if ((e = cudaMemcpy(S.occ, voxel_grid_occ, (size_t)num_occ * 3 * sizeof(int), cudaMemcpyHostToDevice)) !=
        cudaSuccess)
      return (int)e;
    list = S.occ;
  }
  const int vol = dim * dim * dim;
  // the reference kernel's guard lets thread dim^3 write the voxel (0, 0, dim)
  const int extra = vol < 27000 ? 1 : 0;
  tdf_launch(list, nullptr, num_occ, 1, dim, extra, S.pin_tdf, 0);
  if ((e = cudaGetLastError()) != cudaSuccess) return (int)e;
  if ((e = cudaDeviceSynchronize()) != cudaSuccess) return (int)e;
  memcpy(voxel_grid_TDF, S.pin_tdf, (size_t)(vol + extra) * sizeof(float));
  return (int)cudaSuccess;
}

}  // extern "C"
