// grid.cuh — uniform grid (built on device, exact searches) and radix sort.
//
// A grid over n points with cell edge h keeps the points in the order of the
// linear index of their cell (x fastest) and one table of ncells + 1 starts:
// cell c holds points [starts[c], starts[c + 1]), and a run of cells along x
// is one contiguous run of points.  Every size and every bound is computed on
// the device, so a build can sit inside a captured CUDA graph; capacities
// come from the host.
#pragma once
#include <atomic>

#include "common.cuh"

struct GridMeta {
  float ox, oy, oz;      // lower corner of cell (0,0,0)
  float h, inv_h;        // cell edge actually used (>= the requested edge)
  int nx, ny, nz;
  int n;                 // points in the grid
  unsigned ncells;       // nx*ny*nz
  // bounding box as order-preserving unsigned, the lower corner complemented
  // so that both start at zero (cleared by a memset); see box_lo, box_hi
  unsigned nmin[3];
  unsigned bmax[3];
  unsigned ticket;       // blocks of the box reduction that are done
};

struct GridDev {
  const GridMeta* meta;  // device
  const float4* pts;     // points in cell order; w = original index (int bits)
  const uint32_t* starts;  // [ncells + 1]
};

#ifdef __CUDACC__
__device__ __forceinline__ float box_lo(const GridMeta* m, int a) { return ordered_to_float(~m->nmin[a]); }
__device__ __forceinline__ float box_hi(const GridMeta* m, int a) { return ordered_to_float(m->bmax[a]); }
#endif

namespace rtr {

struct GridBufs {
  GridMeta* meta;        // followed by the table in one allocation
  uint32_t* starts;      // [cell_cap + 1]
  uint32_t* tiles;       // tile sums of the table's scan
  float4* pts;
  uint32_t *k0, *v0;     // cell of each point, and its rank there
  uint32_t *k1, *v1, *hist;  // ordered builds only
  int n_cap;
  unsigned cell_cap;
};

// Stable LSD radix sort of (key, value) pairs by the low `bits` bits of key.
// When vals_in is NULL the values are the element indices.  Ping-pongs
// between (k0,v0) and (k1,v1); *k_out/*v_out point at the sorted arrays.
int radix_hist_entries(int n_cap);
// Whether each device schedules a kernel's largest cluster: asked once a kernel
// and device (0: not yet, 1: no, 2: yes).
struct ClusterFit {
  std::atomic<int> known[64] = {};
};
// CTAs of the cluster of `kern` (1,024 threads a CTA) that sorts n_cap items in
// one launch; 0: a grid of tiles (too many items, or ctx asks for it; ctx may be
// NULL).
int cluster_sort_ctas(const rtr_context* ctx, int n_cap, const void* kern, ClusterFit& fit);
// Launches a kernel of clusters of `ctas` CTAs of 1,024 threads (one cluster).
template <class... P, class... A>
inline rtr_status launch_cluster(void (*kern)(P...), int ctas, cudaStream_t st, A... args) {
  if (ctas > 8) RTR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(1024);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  RTR_CUDA(cudaLaunchKernelEx(&cfg, kern, (P)args...));
  return RTR_OK;
}
[[nodiscard]] rtr_status radix_sort_pairs(const rtr_context* ctx, uint32_t* k0, uint32_t* v0, uint32_t* k1,
                                          uint32_t* v1, uint32_t* hist, int n_cap, int n_host, const int* d_n, int bits,
                                          bool vals_iota, cudaStream_t st, uint32_t** k_out, uint32_t** v_out);

// ordered: the points of a cell in ascending original index (a stable sort by
// cell); otherwise in any order (counted into place, a quarter of the time).
void grid_plan(ScratchPlan& plan, int n_cap, unsigned cell_cap, bool ordered = false);
bool grid_take(Scratch& s, int n_cap, unsigned cell_cap, GridBufs* b, bool ordered = false);
// Build the grid over pts[0..n) (n = *d_n when d_n != NULL).  h_req is the
// requested cell edge; if the bounding box needs more than cell_cap cells the
// edge grows until it fits (searches stay exact, only slower).
rtr_status grid_build(const GridBufs& b, const float4* pts, int n_host, const int* d_n, float h_req, cudaStream_t st,
                      bool ordered = false);
// Bounding box only (box_lo, box_hi).
rtr_status bbox_build(GridMeta* m, const float4* pts, int n, cudaStream_t st);
// Same over the first *d_n (<= n_cap) points.
rtr_status bbox_build(GridMeta* m, const float4* pts, int n_cap, const int* d_n, cudaStream_t st);
inline GridDev grid_dev(const GridBufs& b) { return GridDev{b.meta, b.pts, b.starts}; }
inline unsigned default_cell_cap(int n) {
  unsigned c = (unsigned)n * 8u;
  return c < (1u << 18) ? (1u << 18) : c;
}

}  // namespace rtr
