// search.cuh — exact grid searches (device functions).
//
// Ring search: cells are visited in rings of growing Chebyshev radius k around
// the query's cell.  After ring k every unvisited point lies outside the box of
// cells [c-k, c+k], so its distance is at least the distance lb from the query
// to that box's faces (faces on the grid boundary do not count: nothing lies
// beyond them).  The search stops once lb, shrunk by a rounding margin, is
// strictly larger than the current k-th best distance.  Cells whose box is
// farther than the current bound are skipped.  Candidates are compared as
// (d^2, original index), so ties go to the lowest index and the result does not
// depend on the visiting order.
//
// Sorted points carry their original index in the w lane (as int bits), so one
// 16-byte load gives both the coordinates and the tie-break key.
#pragma once
#include <limits.h>

#include "grid.cuh"

struct GridView {
  float ox, oy, oz, h, inv_h;
  int nx, ny, nz;
  const float4* __restrict__ pts;
  const uint32_t* __restrict__ starts;
};

__device__ __forceinline__ GridView load_view(const GridDev& g) {
  GridView v;
  const GridMeta* m = g.meta;
  v.ox = m->ox;
  v.oy = m->oy;
  v.oz = m->oz;
  v.h = m->h;
  v.inv_h = m->inv_h;
  v.nx = m->nx;
  v.ny = m->ny;
  v.nz = m->nz;
  v.pts = g.pts;
  v.starts = g.starts;
  return v;
}

// Points of cell (x, y, z), and of the run of cells x0 .. x1 of row (y, z).
__device__ __forceinline__ uint2 row_span(const GridView& g, int x0, int x1, int y, int z) {
  const unsigned r = ((unsigned)z * (unsigned)g.ny + (unsigned)y) * (unsigned)g.nx;
  return make_uint2(__ldg(g.starts + r + (unsigned)x0), __ldg(g.starts + r + (unsigned)x1 + 1u));
}
__device__ __forceinline__ uint2 cell_span(const GridView& g, int x, int y, int z) { return row_span(g, x, x, y, z); }

__device__ __forceinline__ int pt_index(float4 p) { return __float_as_int(p.w); }

__device__ __forceinline__ int q_cell(float v, float o, float inv_h) {
  float f = __fmul_rn(__fsub_rn(v, o), inv_h);
  f = fminf(fmaxf(f, -1.0e8f), 1.0e8f);
  return (int)floorf(f);
}

// Conservative rounding margin (metres) for bounds near query q.
__device__ __forceinline__ float search_margin(const GridView& g, float4 q, int k) {
  float s = fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fabsf(q.z));
  s = fmaxf(s, fmaxf(fmaxf(fabsf(g.ox), fabsf(g.oy)), fabsf(g.oz)));
  float ext = (float)(max(max(g.nx, g.ny), g.nz) + k + 2) * g.h;
  return 8.0e-6f * (1.0f + s + ext);
}

// True when every point at distance >= (lb - margin) has d^2 > bound.
__device__ __forceinline__ bool beyond(float lb, float margin, float bound) {
  float l = lb - margin;
  return l > 0.f && l * l > bound * 1.000001f + 1e-30f;
}

// Distance from q to the box of cell (x, y, z).
__device__ __forceinline__ float cell_box_dist(const GridView& g, float4 q, int x, int y, int z) {
  float lx = g.ox + (float)x * g.h, ly = g.oy + (float)y * g.h, lz = g.oz + (float)z * g.h;
  float dx = fmaxf(fmaxf(lx - q.x, q.x - (lx + g.h)), 0.f);
  float dy = fmaxf(fmaxf(ly - q.y, q.y - (ly + g.h)), 0.f);
  float dz = fmaxf(fmaxf(lz - q.z, q.z - (lz + g.h)), 0.f);
  return sqrtf(dx * dx + dy * dy + dz * dz);
}

// Lower bound on the distance to any point outside the ring box of radius k;
// +inf when the ring box already covers the whole grid.
__device__ __forceinline__ float ring_bound(const GridView& g, float4 q, int cx, int cy, int cz, int k) {
  float lb = __int_as_float(0x7f800000);
  if (cx - k > 0) lb = fminf(lb, q.x - (g.ox + (float)(cx - k) * g.h));
  if (cx + k < g.nx - 1) lb = fminf(lb, (g.ox + (float)(cx + k + 1) * g.h) - q.x);
  if (cy - k > 0) lb = fminf(lb, q.y - (g.oy + (float)(cy - k) * g.h));
  if (cy + k < g.ny - 1) lb = fminf(lb, (g.oy + (float)(cy + k + 1) * g.h) - q.y);
  if (cz - k > 0) lb = fminf(lb, q.z - (g.oz + (float)(cz - k) * g.h));
  if (cz + k < g.nz - 1) lb = fminf(lb, (g.oz + (float)(cz + k + 1) * g.h) - q.z);
  return lb;
}

// Distance from q to the box spanned by the whole grid.
__device__ __forceinline__ float grid_box_dist(const GridView& g, float4 q) {
  const float hx = g.ox + (float)g.nx * g.h, hy = g.oy + (float)g.ny * g.h, hz = g.oz + (float)g.nz * g.h;
  const float dx = fmaxf(fmaxf(g.ox - q.x, q.x - hx), 0.f);
  const float dy = fmaxf(fmaxf(g.oy - q.y, q.y - hy), 0.f);
  const float dz = fmaxf(fmaxf(g.oz - q.z, q.z - hz), 0.f);
  return sqrtf(dx * dx + dy * dy + dz * dz);
}

__device__ __forceinline__ bool ring_covers(const GridView& g, int cx, int cy, int cz, int k) {
  return cx - k <= 0 && cx + k >= g.nx - 1 && cy - k <= 0 && cy + k >= g.ny - 1 && cz - k <= 0 &&
         cz + k >= g.nz - 1;
}

// Visits every in-grid cell at Chebyshev distance exactly k from (cx, cy, cz):
// rows on a z or y face of the ring are walked in full, the others only at
// x = cx - k and x = cx + k.  The body sees the cell as (x, y, z).
#define RTR_FOR_RING(g, cx, cy, cz, k, ...)                                         \
  {                                                                                 \
    const int z0_ = max((cz) - (k), 0), z1_ = min((cz) + (k), (g).nz - 1);            \
    const int y0_ = max((cy) - (k), 0), y1_ = min((cy) + (k), (g).ny - 1);            \
    for (int z = z0_; z <= z1_; ++z) {                                              \
      const bool zedge_ = (z == (cz) - (k)) || (z == (cz) + (k));                   \
      for (int y = y0_; y <= y1_; ++y) {                                            \
        const bool edge_ = zedge_ || (y == (cy) - (k)) || (y == (cy) + (k));        \
        const int xs_ = edge_ ? max((cx) - (k), 0) : (cx) - (k);                     \
        const int xe_ = edge_ ? min((cx) + (k), (g).nx - 1) : (cx) + (k);            \
        const int st_ = edge_ ? 1 : 2 * (k);                                        \
        for (int x = xs_; x <= xe_; x += st_) {                                     \
          if (x < 0 || x >= (g).nx) continue;                                       \
          __VA_ARGS__                                                               \
        }                                                                           \
      }                                                                             \
    }                                                                               \
  }

__device__ __forceinline__ int first_ring(const GridView& g, int cx, int cy, int cz) {
  int k = 0;
  k = max(k, max(-cx, cx - (g.nx - 1)));
  k = max(k, max(-cy, cy - (g.ny - 1)));
  k = max(k, max(-cz, cz - (g.nz - 1)));
  return k;
}

__device__ __forceinline__ void nn_take(float4 p, unsigned j, float4 q, float& bd, int& bi, int& bpos) {
  const float d2 = dist2_exact(q, p);
  const int id = pt_index(p);
  // a candidate at infinite (or NaN) d^2 is never a neighbour: points with a
  // non-finite coordinate never match
  if (d2 < bd || (d2 == bd && id < bi && d2 < __int_as_float(0x7f800000))) {
    bd = d2;
    bi = id;
    bpos = (int)j;
  }
}

// Group reduction of (bd, bi, bpos) over the G lanes in gmask.
template <int G>
__device__ __forceinline__ void group_best(unsigned gmask, float& bd, int& bi, int& bpos) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const float od = __shfl_xor_sync(gmask, bd, o);
    const int oi = __shfl_xor_sync(gmask, bi, o);
    const int op = __shfl_xor_sync(gmask, bpos, o);
    if (od < bd || (od == bd && oi < bi)) {
      bd = od;
      bi = oi;
      bpos = op;
    }
  }
}

// Same search with G lanes per query (G a power of two <= 32; the lanes of a
// group are contiguous and aligned).  A ring is walked as the (2k+1)^3 cube in
// chunks of 4G entries: each lane fetches four cell entries at once (interior
// and out-of-grid entries are dropped), the group ballots the surviving
// candidate cells and then scans each one's points with all G lanes.  After
// every ring the group agrees on the best (d^2, index), so the ring loop is
// uniform inside the group.  A lane skips a cell only when the cell is beyond
// its own best, which is never better than the group's.
// Exact 1-NN with d^2 <= r2max (r2max = +inf: unbounded); the original index
// (or -1) and the sorted position.
template <int G>
__device__ __forceinline__ void grid_nn1_group(const GridView& g, float4 q, float r2max, int lg,
                                               unsigned gmask, float& bd, int& bi, int& bpos) {
  bd = r2max;
  bi = INT_MAX;
  bpos = -1;
  const int cx = q_cell(q.x, g.ox, g.inv_h), cy = q_cell(q.y, g.oy, g.inv_h),
            cz = q_cell(q.z, g.oz, g.inv_h);
  const int gbase = (threadIdx.x & 31) & ~(G - 1);
  // nothing of the grid within the bound (uniform inside the group)
  if (beyond(grid_box_dist(g, q), search_margin(g, q, 0), r2max)) {
    bi = -1;
    bd = __int_as_float(0x7f800000);
    return;
  }
  for (int k = first_ring(g, cx, cy, cz);; ++k) {
    const float margin = search_margin(g, q, k);
    // the ring's cube clamped to the grid
    const int x0 = max(cx - k, 0), y0 = max(cy - k, 0), z0 = max(cz - k, 0);
    const int ex = min(cx + k, g.nx - 1) - x0 + 1, ey = min(cy + k, g.ny - 1) - y0 + 1,
              ez = min(cz + k, g.nz - 1) - z0 + 1;
    const int vol = (ex > 0 && ey > 0 && ez > 0) ? ex * ey * ez : 0;
    if (vol <= 512) {
      for (int m0 = 0; m0 < vol; m0 += 4 * G) {
        uint2 cc[4];
        bool cand[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int m = m0 + s * G + lg;
          cand[s] = false;
          cc[s] = make_uint2(0u, 0u);
          if (m < vol) {
            const int x = x0 + m % ex, y = y0 + (m / ex) % ey, z = z0 + m / (ex * ey);
            // the cell's box first: a cell beyond the current best is not fetched
            if (max(max(abs(x - cx), abs(y - cy)), abs(z - cz)) == k &&
                !beyond(cell_box_dist(g, q, x, y, z), margin, bd)) {
              cc[s] = cell_span(g, x, y, z);
              cand[s] = cc[s].x < cc[s].y;
            }
          }
        }
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          unsigned bal = __ballot_sync(gmask, cand[s]) >> gbase;
          while (bal) {
            const int src = __ffs(bal) - 1;
            bal &= bal - 1;
            const unsigned b0 = __shfl_sync(gmask, cc[s].x, gbase + src);
            const unsigned b1 = __shfl_sync(gmask, cc[s].y, gbase + src);
            for (unsigned j = b0 + (unsigned)lg; j < b1; j += G) nn_take(g.pts[j], j, q, bd, bi, bpos);
          }
        }
      }
    } else {
      // large rings: walk only the shell, all lanes on the same cell
      RTR_FOR_RING(g, cx, cy, cz, k, {
        const uint2 c = cell_span(g, x, y, z);
        if (c.x < c.y && !beyond(cell_box_dist(g, q, x, y, z), margin, bd))
          for (unsigned j = c.x + (unsigned)lg; j < c.y; j += G) nn_take(g.pts[j], j, q, bd, bi, bpos);
      })
    }
    group_best<G>(gmask, bd, bi, bpos);
    if (ring_covers(g, cx, cy, cz, k)) break;
    if (beyond(ring_bound(g, q, cx, cy, cz, k), margin, bd)) break;
  }
  if (bi == INT_MAX) {
    bi = -1;
    bpos = -1;
    bd = __int_as_float(0x7f800000);
  }
}

// Box searches, for many queries against one grid: what does not depend on
// the query is computed once.  The rounding of a search is covered by the
// margin of the grid plus the query's own part (box_margin).
struct BoxView {
  GridView g;
  float margin;
  float nxm, nym, nzm;  // last cell of each axis
  float hx, hy, hz;     // upper corner
  bool dense;           // many points a cell: large boxes are walked outwards (box_points_ordered)
};
__device__ __forceinline__ BoxView box_view(const GridDev& gd) {
  BoxView b;
  b.g = load_view(gd);
  const GridView& g = b.g;
  b.nxm = (float)(g.nx - 1);
  b.nym = (float)(g.ny - 1);
  b.nzm = (float)(g.nz - 1);
  b.hx = g.ox + (float)g.nx * g.h;
  b.hy = g.oy + (float)g.ny * g.h;
  b.hz = g.oz + (float)g.nz * g.h;
  float s = fmaxf(fmaxf(fabsf(g.ox), fabsf(g.oy)), fabsf(g.oz));
  s = fmaxf(s, fmaxf(fmaxf(fabsf(b.hx), fabsf(b.hy)), fabsf(b.hz)));
  b.dense = false;
  b.margin = 8.0e-6f * (1.0f + s + (float)(max(max(g.nx, g.ny), g.nz) + 3) * g.h);
  return b;
}
__device__ __forceinline__ float box_margin(const BoxView& b, float4 q) {
  return b.margin + 8.0e-6f * fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fabsf(q.z));
}

__device__ __forceinline__ float sqrt_up(float x) {  // >= sqrt(x), by a few parts in 10^6
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r * 1.00001f;
}

// The cells meeting the box q -+ t (t > 0 includes the margin), in cell units.
struct CellBox {
  float ux, uy, uz, tc2;
  int x0, x1, y0, y1, z0, z1;
};
__device__ __forceinline__ CellBox cell_box(const BoxView& v, float4 q, float t) {
  const GridView& g = v.g;
  CellBox c;
  const float ux = c.ux = (q.x - g.ox) * g.inv_h;
  c.uy = (q.y - g.oy) * g.inv_h;
  c.uz = (q.z - g.oz) * g.inv_h;
  const float tc = t * g.inv_h;
  c.tc2 = tc * tc * 1.00001f;
  c.x0 = __float2int_rd(fminf(fmaxf(ux - tc, 0.f), v.nxm));
  c.x1 = __float2int_rd(fminf(fmaxf(ux + tc, 0.f), v.nxm));
  c.y0 = __float2int_rd(fminf(fmaxf(c.uy - tc, 0.f), v.nym));
  c.y1 = __float2int_rd(fminf(fmaxf(c.uy + tc, 0.f), v.nym));
  c.z0 = __float2int_rd(fminf(fmaxf(c.uz - tc, 0.f), v.nzm));
  c.z1 = __float2int_rd(fminf(fmaxf(c.uz + tc, 0.f), v.nzm));
  return c;
}

// Calls body(span) for the rows of the box along x, each one contiguous run of
// points, four rows' spans in flight; a row farther from q than t (by its y
// and z extent) is skipped.  body returns true to stop (after its four rows).
template <typename F>
__device__ __forceinline__ void box_rows(const BoxView& v, const CellBox& c, F body) {
  const int rows = (c.y1 - c.y0 + 1) * (c.z1 - c.z0 + 1);
  int y = c.y0, z = c.z0;
  for (int r0 = 0; r0 < rows; r0 += 4) {
    uint2 s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s[u] = make_uint2(0u, 0u);
      if (r0 + u < rows) {
        const float fy = (float)y, fz = (float)z;
        const float dy = fmaxf(fmaxf(fy - c.uy, c.uy - (fy + 1.f)), 0.f);
        const float dz = fmaxf(fmaxf(fz - c.uz, c.uz - (fz + 1.f)), 0.f);
        if (!(dy * dy + dz * dz > c.tc2)) s[u] = row_span(v.g, c.x0, c.x1, y, z);
        if (++y > c.y1) {
          y = c.y0;
          ++z;
        }
      }
    }
    bool stop = false;
#pragma unroll
    for (int u = 0; u < 4; ++u) stop |= body(s[u]);
    if (stop) return;
  }
}

// The two nearest of the points seen: the best by (d^2, index) and the
// squared distance of the second.
struct Near2 {
  float bd, sd;
  int bi, bpos;
};
__device__ __forceinline__ void near2_take(float4 p, unsigned j, float4 q, Near2& n) {
  const float d2 = dist2_exact(q, p);
  const int id = pt_index(p);
  // a point at infinite (or NaN) d^2 is never a neighbour
  const bool better = d2 < n.bd || (d2 == n.bd && id < n.bi && d2 < __int_as_float(0x7f800000));
  n.sd = fminf(n.sd, better ? n.bd : d2);
  if (better) {
    n.bd = d2;
    n.bi = id;
    n.bpos = (int)j;
  }
}

// Whether a cell with a point in it holds more than DENSE_CELL on average: 32
// points of the grid asked, a lane each.  Where cells hold many, a box scanned
// whole costs far more than its nearest rows: two 400k chairs within 5 cm, cells
// of 1 cm, 20 iterations 20.2 ms, 6.9 walked outwards (13.4 with rings of
// cells); a million points a chair 85 and 26 (36), cells of 2.5 cm 180 and 128
// (120); two 60k desks within 10 cm, 50 iterations, 4.7 and 3.5.  Where they hold
// few, walking outwards is a longer chain: 60k points on 10k 2.9 and 4.0 ms, a
// 640 x 480 frame 1.15 and 1.20 (1.14 with the line at 24 points, 1.21 at 16).
constexpr unsigned DENSE_CELL = 24;
__device__ __forceinline__ bool grid_dense(const GridDev& gd, const GridView& g) {
  const int n = gd.meta->n, lane = threadIdx.x & 31;
  unsigned cnt = 0;
  if (n > 0) {
    const float4 p = g.pts[(int)(((long long)n * lane) >> 5)];
    const int cx = min(max(q_cell(p.x, g.ox, g.inv_h), 0), g.nx - 1), cy = min(max(q_cell(p.y, g.oy, g.inv_h), 0), g.ny - 1),
              cz = min(max(q_cell(p.z, g.oz, g.inv_h), 0), g.nz - 1);
    const uint2 s = cell_span(g, cx, cy, cz);
    cnt = min(s.y - s.x, 8u * DENSE_CELL);
  }
  return __reduce_add_sync(0xffffffffu, cnt) > 32u * DENSE_CELL;
}

// Cell k of lo .. hi in the order centre, centre - 1, centre + 1, ...
__device__ __forceinline__ int cell_outward(int lo, int hi, int centre, int k) {
  const int a = centre - lo, b = hi - centre, m = min(a, b);
  return centre + (k <= 2 * m ? ((k & 1) ? -(k + 1) / 2 : k / 2) : (a > b ? m - k : k - m));
}

// The rows of a larger box from the query outwards, each cut to the cells
// within the second nearest distance that the lane has seen so far: what is
// left out lies beyond it.  Lane lg takes the points j with j mod G = lg,
// whatever its cuts.
template <int G>
__device__ __forceinline__ void box_points_ordered(const BoxView& v, const CellBox& c, float4 q, float margin, int lg,
                                                   Near2& n) {
  const GridView& g = v.g;
  const int yc = min(max(__float2int_rd(c.uy), c.y0), c.y1), zc = min(max(__float2int_rd(c.uz), c.z0), c.z1);
  const int ey = c.y1 - c.y0 + 1, ez = c.z1 - c.z0 + 1;
  float lim2 = c.tc2;
  for (int kz = 0; kz < ez; ++kz) {
    const int z = cell_outward(c.z0, c.z1, zc, kz);
    const float dz = fmaxf(fmaxf((float)z - c.uz, c.uz - ((float)z + 1.f)), 0.f);
    if (dz * dz > lim2) continue;
    for (int k0 = 0; k0 < ey; k0 += 4) {
      uint2 s[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        s[u] = make_uint2(0u, 0u);
        if (k0 + u < ey) {
          const int y = cell_outward(c.y0, c.y1, yc, k0 + u);
          const float dy = fmaxf(fmaxf((float)y - c.uy, c.uy - ((float)y + 1.f)), 0.f);
          const float rest = lim2 - (dy * dy + dz * dz);
          if (rest >= 0.f) {
            const float w = sqrt_up(rest);
            const int x0 = max(c.x0, __float2int_rd(fmaxf(c.ux - w, 0.f)));
            const int x1 = min(c.x1, __float2int_rd(fminf(c.ux + w, v.nxm)));
            if (x0 <= x1) s[u] = row_span(g, x0, x1, y, z);
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        unsigned j = s[u].x + (((unsigned)lg - s[u].x) & (G - 1));
        for (; j + G < s[u].y; j += 2 * G) {
          const float4 p0 = g.pts[j], p1 = g.pts[j + G];
          near2_take(p0, j, q, n);
          near2_take(p1, j + G, q, n);
        }
        if (j < s[u].y) near2_take(g.pts[j], j, q, n);
      }
      const float t = (sqrt_up(n.sd) + margin) * g.inv_h;
      lim2 = fminf(c.tc2, t * t * 1.00001f);
    }
  }
}

// The points of the box's rows into n, spread over the G lanes of the group.
// Up to 4 lanes walk the rows one after another, striding through each row's
// points: fewest instructions, for kernels with enough queries in flight to
// hide that every row is a dependent load (larger boxes over dense cells:
// box_points_ordered).  With 8 lanes and more each lane fetches one row's span,
// a prefix sum over the rows numbers their points, and the lanes stride through
// the numbers, four loads in flight each: a few round trips in all, for kernels
// whose queries are few and wait on one another.  Uniform in the group.
template <int G>
__device__ __forceinline__ void box_points(const BoxView& v, const CellBox& c, float4 q, float margin, int lg,
                                           unsigned gmask, Near2& n) {
  auto take = [&](float4 p, unsigned j) { near2_take(p, j, q, n); };
  if (G <= 4 && v.dense && (c.y1 - c.y0 + 1) * (c.z1 - c.z0 + 1) > 4) {
    box_points_ordered<G>(v, c, q, margin, lg, n);
    return;
  }
  if (G <= 4) {
    box_rows(v, c, [&](uint2 s) {
      unsigned j = s.x + (unsigned)lg;
      for (; j + G < s.y; j += 2 * G) {
        const float4 p0 = v.g.pts[j], p1 = v.g.pts[j + G];
        take(p0, j);
        take(p1, j + G);
      }
      if (j < s.y) take(v.g.pts[j], j);
      return false;
    });
    return;
  }
  const int ey = c.y1 - c.y0 + 1, rows = ey * (c.z1 - c.z0 + 1);
  for (int r0 = 0; r0 < rows; r0 += G) {
    const int r = r0 + lg;
    uint2 s = make_uint2(0u, 0u);
    if (r < rows) {
      const int zi = r / ey, y = c.y0 + r - zi * ey, z = c.z0 + zi;
      const float fy = (float)y, fz = (float)z;
      const float dy = fmaxf(fmaxf(fy - c.uy, c.uy - (fy + 1.f)), 0.f);
      const float dz = fmaxf(fmaxf(fz - c.uz, c.uz - (fz + 1.f)), 0.f);
      if (!(dy * dy + dz * dz > c.tc2)) s = row_span(v.g, c.x0, c.x1, y, z);
    }
    unsigned incl = s.y - s.x;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
      const unsigned t = __shfl_up_sync(gmask, incl, o, G);
      if (lg >= o) incl += t;
    }
    const unsigned total = __shfl_sync(gmask, incl, G - 1, G);
    const unsigned off = s.y - incl;  // point k of the numbering lies at off + k of its row
    for (unsigned k0 = 0; k0 < total; k0 += 4 * G) {
      unsigned j[4];
      float4 p[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const unsigned k = k0 + u * G + (unsigned)lg;
        int row = 0;  // the first row whose points go past k
#pragma unroll
        for (int step = G / 2; step > 0; step >>= 1)
          if (k >= __shfl_sync(gmask, incl, row + step - 1, G)) row += step;
        j[u] = __shfl_sync(gmask, off, row, G) + k;
        if (k < total) p[u] = v.g.pts[j[u]];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k0 + u * G + (unsigned)lg < total) take(p[u], j[u]);
    }
  }
}

// Whether the cells of the box hold no point; the group's lanes share the rows.
template <int G>
__device__ __forceinline__ bool box_empty(const BoxView& v, const CellBox& c, int lg, unsigned gmask) {
  const int ey = c.y1 - c.y0 + 1, rows = ey * (c.z1 - c.z0 + 1);
  bool any = false;
#pragma unroll 4
  for (int r = lg; r < rows; r += G) {
    const int zi = r / ey;
    const uint2 s = row_span(v.g, c.x0, c.x1, c.y0 + r - zi * ey, c.z0 + zi);
    any |= s.x < s.y;
  }
  return !__any_sync(gmask, any);
}

// Exact 1-NN with d^2 <= r2max (r >= its root), G lanes per query (see
// grid_nn1_group; the same neighbour), for queries that come again and move
// little.  cand: the sorted position of any grid point, by choice the last
// answer, or -1.  With a candidate one box of its distance is scanned: where
// it is the answer or close to it, a few rows.  Without one the box grows
// from one cell edge, doubling up to the bound, until something is found, and
// then covers what was found.  *room: every point of the grid but the answer
// (every point, when there is none) is at least that far away.  extra widens
// the last box, so that room comes out useful; and where the bound holds
// nothing, boxes up to eight times it are tried for emptiness (spans only, no
// points), so that a query in the open is told it need not come back soon.  Returns the answer's
// sorted position or -1; uniform in the group.
template <int G>
__device__ __forceinline__ int grid_nn1_from(const BoxView& v, float4 q, float r2max, float r, int cand, float extra,
                                             int lg, unsigned gmask, float* room) {
  const GridView& g = v.g;
  const float inf = __int_as_float(0x7f800000);
  Near2 n;
  const float far = r + extra, margin = box_margin(v, q);
  float tr = 0.f, t;
  if (cand >= 0) {
    t = fminf(sqrt_up(dist2_exact(q, g.pts[cand])), r) + extra + margin;
  } else {
    const float dx = fmaxf(fmaxf(g.ox - q.x, q.x - v.hx), 0.f), dy = fmaxf(fmaxf(g.oy - q.y, q.y - v.hy), 0.f),
                dz = fmaxf(fmaxf(g.oz - q.z, q.z - v.hz), 0.f);
    const float d0 = sqrt_up(dx * dx + dy * dy + dz * dz);  // to the grid's box
    if (d0 * 0.9999f > r + margin) {  // nothing of the grid within the bound
      *room = d0 * 0.9999f - margin;
      return -1;
    }
    tr = fminf(far, d0 + g.h);
    t = tr + margin;
  }
  bool whole;
  for (;;) {
    const CellBox c = cell_box(v, q, t);
    n = Near2{inf, inf, INT_MAX, -1};
    box_points<G>(v, c, q, margin, lg, gmask, n);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      const float od = __shfl_xor_sync(gmask, n.bd, o), os = __shfl_xor_sync(gmask, n.sd, o);
      const int oi = __shfl_xor_sync(gmask, n.bi, o), op = __shfl_xor_sync(gmask, n.bpos, o);
      const bool better = od < n.bd || (od == n.bd && oi < n.bi);
      n.sd = fminf(fminf(n.sd, os), better ? n.bd : od);
      if (better) {
        n.bd = od;
        n.bi = oi;
        n.bpos = op;
      }
    }
    whole = c.x0 == 0 && c.y0 == 0 && c.z0 == 0 && c.x1 == g.nx - 1 && c.y1 == g.ny - 1 && c.z1 == g.nz - 1;
    if (cand >= 0 || whole) break;
    if (n.bpos >= 0) {
      const float need = margin + fminf(sqrt_up(n.bd), far);
      if (need <= t) break;  // all within the answer's distance, or the bound, has been seen
      t = need + extra;
      cand = n.bpos;  // the last box
    } else {
      if (tr >= far) break;
      tr = fminf(far, 2.f * tr);
      t = tr + margin;
    }
  }
  float seen = whole ? inf : t - margin;  // every point closer than this has been seen
  const bool hit = n.bd <= r2max && n.bpos >= 0;
  if (n.bpos < 0 && !whole && seen < 1.0e30f) {
    for (int k = 0; k < 5; ++k) {  // 1.5^5 = 7.6
      const CellBox c = cell_box(v, q, 1.5f * seen + margin);
      if (!box_empty<G>(v, c, lg, gmask)) break;
      seen *= 1.5f;
    }
  }
  *room = fminf(sqrt_up(hit ? n.sd : n.bd) * 0.9999f, seen);
  return hit ? n.bpos : -1;
}

// Whether any point lies within sqrt(r2) of q (d^2 <= r2, finite r2), G lanes
// per query; the same answer as grid_nn1_group finding a neighbour.  The own
// cell first, then rows; every lane stops once the group has found one.  (Rows
// alone begin in a corner of the box, which costs where cells hold many: 20,000
// points of a wall against a million within 10 cm 1,110 us, 230 so, and 128
// instead of 122 where cells hold few.)
template <int G>
__device__ __forceinline__ bool grid_any_within(const BoxView& v, float4 q, float r2, int lg, unsigned gmask) {
  const GridView& g = v.g;
  const float r = sqrt_up(r2) + box_margin(v, q);
  if (g.ox - q.x > r || q.x - v.hx > r || g.oy - q.y > r || q.y - v.hy > r || g.oz - q.z > r || q.z - v.hz > r)
    return false;
  bool found = false;
  const int cx = q_cell(q.x, g.ox, g.inv_h), cy = q_cell(q.y, g.oy, g.inv_h), cz = q_cell(q.z, g.oz, g.inv_h);
  if (cx >= 0 && cy >= 0 && cz >= 0 && cx < g.nx && cy < g.ny && cz < g.nz) {
    const uint2 s = cell_span(g, cx, cy, cz);
    for (unsigned j = s.x + (unsigned)lg; j < s.y && !found; j += G) found = dist2_exact(q, g.pts[j]) <= r2;
    if (G > 1 ? __any_sync(gmask, found) != 0 : found) return true;
  }
  int left = 4;
  box_rows(v, cell_box(v, q, r), [&](uint2 s) {
    for (unsigned j = s.x + (unsigned)lg; j < s.y && !found; j += G) found = dist2_exact(q, g.pts[j]) <= r2;
    if (--left > 0) return false;
    left = 4;
    found = G > 1 ? __any_sync(gmask, found) != 0 : found;
    return found;
  });
  return found;
}

// Exact K-NN (K compile-time), sorted by (d^2, index).  The K nearest by that
// order are unique, so any k <= K of them form the exact k-NN.  The list holds
// (d^2 bits, index) as one word each, ascending; an empty slot is (+inf, 0),
// which no candidate at infinite or NaN d^2 goes below.  The slots of an
// insertion are independent of each other.
constexpr unsigned long long KNN_NONE = 0x7f800000ull << 32;
template <int K>
__device__ __forceinline__ void knn_insert(unsigned long long (&list)[K], float4 q, float4 p) {
  const unsigned long long c =
      ((unsigned long long)__float_as_uint(dist2_exact(q, p)) << 32) | (unsigned)pt_index(p);
  if (!(c < list[K - 1])) return;
  bool lt[K];
#pragma unroll
  for (int s = 0; s < K; ++s) lt[s] = c < list[s];
#pragma unroll
  for (int s = K - 1; s > 0; --s) list[s] = lt[s - 1] ? list[s - 1] : (lt[s] ? c : list[s]);
  list[0] = lt[0] ? c : list[0];
}
template <int K>
__device__ __forceinline__ float knn_worst(const unsigned long long (&list)[K]) {
  return __uint_as_float((unsigned)(list[K - 1] >> 32));
}

// The nearest of the 27 cells around q's (cx, cy, cz) inside the grid: the own
// cell, those beside it, then eight rows, a run of points each, the nearest
// first and cut to the cells that can still hold an entry.  (The own row as one
// run costs where cells hold many: 50,000 queries in a million points of a room,
// k = 16 1,865 us, 1,170 now.)  True when nothing farther can enter the list.
template <int K>
__device__ __forceinline__ bool knn_near(const GridView& g, float4 q, int cx, int cy, int cz,
                                         unsigned long long (&list)[K]) {
  const float margin = search_margin(g, q, 1);
  const float lx = g.ox + (float)cx * g.h, ly = g.oy + (float)cy * g.h, lz = g.oz + (float)cz * g.h;  // the query's cell
  const float xlo = fmaxf(q.x - lx, 0.f), xhi = fmaxf(lx + g.h - q.x, 0.f);
  const float ylo = fmaxf(q.y - ly, 0.f), yhi = fmaxf(ly + g.h - q.y, 0.f);
  const float zlo = fmaxf(q.z - lz, 0.f), zhi = fmaxf(lz + g.h - q.z, 0.f);
#pragma unroll 1
  for (int k = 0; k < 11; ++k) {
    // rows (0, 0) in three parts, (-1, 0), (1, 0), (0, -1), (0, 1) and the corners: two bits each, plus one
    const int r = max(k - 2, 0);
    const int dy = (int)((0x28161u >> (2 * r)) & 3u) - 1, dz = (int)((0x22215u >> (2 * r)) & 3u) - 1;
    const int y = cy + dy, z = cz + dz;
    if (y < 0 || y >= g.ny || z < 0 || z >= g.nz) continue;
    const float ey = dy < 0 ? ylo : (dy > 0 ? yhi : 0.f), ez = dz < 0 ? zlo : (dz > 0 ? zhi : 0.f);
    const float e2 = ey * ey + ez * ez, worst = knn_worst<K>(list);
    if (r > 0 && beyond(sqrtf(e2), margin, worst)) continue;
    const bool left = cx > 0 && k != 0 && k != 2 && !beyond(sqrtf(e2 + xlo * xlo), margin, worst);
    const bool right = cx < g.nx - 1 && k > 1 && !beyond(sqrtf(e2 + xhi * xhi), margin, worst);
    const int xa = k == 2 ? cx + 1 : (left ? cx - 1 : cx), xb = k == 1 ? cx - 1 : (right ? cx + 1 : cx);
    if (xa > xb || (k == 1 && !left)) continue;
    const uint2 span = row_span(g, xa, xb, y, z);
    for (unsigned j = span.x; j < span.y; ++j) knn_insert<K>(list, q, g.pts[j]);
  }
  return ring_covers(g, cx, cy, cz, 1) || beyond(ring_bound(g, q, cx, cy, cz, 1), margin, knn_worst<K>(list));
}

// The K (<= 32) nearest of a finite query by a whole warp, every lane with the
// same q; lane s < K returns entry s (KNN_NONE: none).
// Rows of a box of cells, 32 at a time, a lane a row's ends; their points as
// one sequence, 32 at a time.  The list is held sorted across the lanes: a few
// candidates below its last entry go in one by one, more of them are sorted and
// merged.  The box: the 27 cells around the query's (its own cell where these
// hold many points); once the list is full its last entry bounds the search,
// and one more box, of the cells within that distance, settles it; boxes of 7,
// 15, ... cells a side while it is not full.  So a point far from others costs
// tens of steps, not a chain of single cells, and no lane waits for another
// query's.
__device__ __forceinline__ unsigned long long knn_stage(unsigned long long x, int d, bool low) {
  const unsigned long long o = __shfl_xor_sync(0xffffffffu, x, d);
  return (o < x) == low ? o : x;
}
struct KnnWarp {
  unsigned long long mine, worst, limit;  // entry `lane`; entry K - 1; no entry of the result is above limit
};
// The points of the rows whose ends the lanes hold.
template <int K>
__device__ __forceinline__ void knn_rows(const GridView& g, float4 q, uint2 span, KnnWarp& w) {
  const int lane = threadIdx.x & 31;
  const int len = (int)(span.y - span.x);
  int incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  const int first = (int)span.x - (incl - len);  // point t of the sequence, if in this lane's row: first + t
  for (int t0 = 0; t0 < total; t0 += 32) {
    const int t = t0 + lane;
    int r = 0;  // rows that end at or before t
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      if (__shfl_sync(0xffffffffu, incl, r + o - 1) <= t) r += o;
    const int j = __shfl_sync(0xffffffffu, first, r & 31) + t;
    unsigned long long c = ~0ull;
    if (t < total) {
      const float4 p = g.pts[j];
      c = ((unsigned long long)__float_as_uint(dist2_exact(q, p)) << 32) | (unsigned)pt_index(p);
    }
    // (an entry of the last box's list may be the limit itself)
    const bool in = c < w.worst && c <= w.limit && c < KNN_NONE;
    unsigned m = __ballot_sync(0xffffffffu, in);
    if (__popc(m) <= 6) {
      for (; m; m &= m - 1) {
        const unsigned long long x = __shfl_sync(0xffffffffu, c, __ffs(m) - 1);
        const unsigned long long before = __shfl_up_sync(0xffffffffu, w.mine, 1);
        if (x < w.mine) w.mine = lane > 0 && x < before ? before : x;
      }
    } else {
      c = in ? c : KNN_NONE;
#pragma unroll
      for (int s = 2; s <= 32; s <<= 1)
#pragma unroll
        for (int d = s >> 1; d > 0; d >>= 1) c = knn_stage(c, d, ((lane & d) == 0) == ((lane & s) == 0));
      if (__shfl_sync(0xffffffffu, w.mine, 0) == KNN_NONE) {
        w.mine = c;  // the first candidates
      } else {
        const unsigned long long o = __shfl_sync(0xffffffffu, c, 31 - lane);
        w.mine = o < w.mine ? o : w.mine;  // the 32 least of both, bitonic
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) w.mine = knn_stage(w.mine, d, (lane & d) == 0);
      }
    }
    w.worst = __shfl_sync(0xffffffffu, w.mine, K - 1);
  }
}
constexpr int KNN_DENSE = 128;  // points in 27 cells from which the query's own cell goes first
template <int K>
__device__ __forceinline__ unsigned long long knn_warp(const BoxView& v, float4 q) {
  const GridView& g = v.g;
  const int lane = threadIdx.x & 31;
  const float margin = box_margin(v, q);
  const int cx = min(max(q_cell(q.x, g.ox, g.inv_h), 0), g.nx - 1), cy = min(max(q_cell(q.y, g.oy, g.inv_h), 0), g.ny - 1),
            cz = min(max(q_cell(q.z, g.oz, g.inv_h), 0), g.nz - 1);
  KnnWarp w{KNN_NONE, KNN_NONE, KNN_NONE};
  {
    const int zi = lane / 3, y = cy + lane - 3 * zi - 1, z = cz + zi - 1;
    uint2 span = make_uint2(0u, 0u);
    if (lane < 9 && y >= 0 && y < g.ny && z >= 0 && z < g.nz)
      span = row_span(g, max(cx - 1, 0), min(cx + 1, g.nx - 1), y, z);
    bool own = false;
    if (__reduce_add_sync(0xffffffffu, span.y - span.x) > KNN_DENSE) {
      const uint2 c = cell_span(g, cx, cy, cz);
      own = c.y - c.x >= (unsigned)K;
      if (own) span = lane == 0 ? c : make_uint2(0u, 0u);
    }
    knn_rows<K>(g, q, span, w);
    if (!own && (ring_covers(g, cx, cy, cz, 1) || beyond(ring_bound(g, q, cx, cy, cz, 1), margin,
                                                         __uint_as_float((unsigned)(w.worst >> 32)))))
      return w.mine;
  }
  for (int k = 3;; k = 2 * k + 1) {
    // the cells within the list's last distance, or +-k cells
    const bool full = w.worst < KNN_NONE;
    CellBox c;
    if (full) {
      c = cell_box(v, q, sqrt_up(__uint_as_float((unsigned)(w.worst >> 32))) + margin);
    } else {
      c.x0 = max(cx - k, 0), c.x1 = min(cx + k, g.nx - 1), c.y0 = max(cy - k, 0), c.y1 = min(cy + k, g.ny - 1);
      c.z0 = max(cz - k, 0), c.z1 = min(cz + k, g.nz - 1);
    }
    w.limit = w.worst;
    w.mine = w.worst = KNN_NONE;
    const int ny = c.y1 - c.y0 + 1, rows = ny * (c.z1 - c.z0 + 1);
    for (int r0 = 0; r0 < rows; r0 += 32) {
      uint2 span = make_uint2(0u, 0u);
      if (r0 + lane < rows) {
        const int zi = (r0 + lane) / ny, y = c.y0 + (r0 + lane) - zi * ny, z = c.z0 + zi;
        const float fy = (float)y, fz = (float)z;
        const float dy = fmaxf(fmaxf(fy - c.uy, c.uy - (fy + 1.f)), 0.f), dz = fmaxf(fmaxf(fz - c.uz, c.uz - (fz + 1.f)), 0.f);
        if (!full || !(dy * dy + dz * dz > c.tc2)) span = row_span(g, c.x0, c.x1, y, z);
      }
      knn_rows<K>(g, q, span, w);
    }
    if (full || ring_covers(g, cx, cy, cz, k)) return w.mine;
    if (beyond(ring_bound(g, q, cx, cy, cz, k), margin, __uint_as_float((unsigned)(w.worst >> 32)))) return w.mine;
  }
}

// A query inside the grid takes the 27 cells around it first; further rings,
// and queries outside, go cell by cell.
template <int K>
__device__ __forceinline__ void grid_knn(const GridView& g, float4 q, float (&bd)[K], int (&bi)[K]) {
  unsigned long long list[K];
#pragma unroll
  for (int s = 0; s < K; ++s) list[s] = KNN_NONE;
  const int cx = q_cell(q.x, g.ox, g.inv_h), cy = q_cell(q.y, g.oy, g.inv_h),
            cz = q_cell(q.z, g.oz, g.inv_h);
  int k = first_ring(g, cx, cy, cz);
  bool done = false;
  if (k == 0) {
    done = knn_near<K>(g, q, cx, cy, cz, list);
    k = 2;
  }
  for (; !done; ++k) {
    const float margin = search_margin(g, q, k);
    RTR_FOR_RING(g, cx, cy, cz, k, {
      const uint2 c = cell_span(g, x, y, z);
      if (c.x < c.y && !beyond(cell_box_dist(g, q, x, y, z), margin, knn_worst<K>(list)))
        for (unsigned j = c.x; j < c.y; ++j) knn_insert<K>(list, q, g.pts[j]);
    })
    done = ring_covers(g, cx, cy, cz, k) || beyond(ring_bound(g, q, cx, cy, cz, k), margin, knn_worst<K>(list));
  }
#pragma unroll
  for (int s = 0; s < K; ++s) {
    bd[s] = __uint_as_float((unsigned)(list[s] >> 32));
    bi[s] = list[s] == KNN_NONE ? INT_MAX : (int)(unsigned)list[s];
  }
}
