// rtg_surface.cu -- per-element kernels around the trace:
//   * neighbour lists of overlapping discs (disc_neighborhood.hpp:20-220):
//     uniform grid of cell size 2*r_max, discs counted into its cells and
//     copied in cell order, each disc tests the 27 surrounding cells (nine runs
//     of three) with the reference's predicate distance(c_i, c_j) < r_i + r_j;
//     rows are sorted by id (CSR);
//   * exposed disc area inside the x/y box (disc_bounding_box_intersector.hpp:
//     43-441) and triangle areas (utils.hpp:161-169), one thread per element;
//   * normalised, neighbourhood-smoothed estimates (device.hpp:154-187);
//   * relative error and variance of variance (hit_accumulator.hpp:152-249).
#include <cfloat>
#include <cmath>
#include <cstdint>

#include "rtg_internal.cuh"
#include "rtg_math.cuh"

namespace rtg {

namespace {

inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

struct Grid {
  float org[3];
  float inv_h;
  int dim[3];
};

// Monotone in v, and off by at most 3 * 2^-24 * dim cells (the roundings of the
// difference, of inv_h and of the product).
__device__ __forceinline__ int cell_coord(float v, float org, float inv_h, int dim) {
  const int c = (int)floorf((v - org) * inv_h);
  return c < 0 ? 0 : (c >= dim ? dim - 1 : c);
}

// The cell of every disc and its place among that cell's discs.
__global__ void cell_count_kernel(const float4* __restrict__ dcr, int64_t nd, Grid g, uint32_t* __restrict__ count,
                                  uint2* __restrict__ cell_rank) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nd) return;
  const float4 c = dcr[i];
  const int cx = cell_coord(c.x, g.org[0], g.inv_h, g.dim[0]);
  const int cy = cell_coord(c.y, g.org[1], g.inv_h, g.dim[1]);
  const int cz = cell_coord(c.z, g.org[2], g.inv_h, g.dim[2]);
  const uint32_t cell = (uint32_t)((cz * g.dim[1] + cy) * g.dim[0] + cx);
  cell_rank[i] = make_uint2(cell, atomicAdd(&count[cell], 1u));
}

// The discs in cell order (`start`: the exclusive scan of the counts).
__global__ void cell_place_kernel(const float4* __restrict__ dcr, int64_t nd, const uint32_t* __restrict__ start,
                                  const uint2* __restrict__ cell_rank, float4* __restrict__ cell_disc,
                                  uint32_t* __restrict__ cell_id) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nd) return;
  const uint2 cr = cell_rank[i];
  const uint32_t at = start[cr.x] + cr.y;
  cell_disc[at] = dcr[i];
  cell_id[at] = (uint32_t)i;
}

// check_dist (disc_neighborhood.hpp:190-220): the three axis pre-tests are
// implied by the distance test in IEEE arithmetic and are omitted.
__device__ __forceinline__ bool overlaps(float4 a, float4 b) {
  float d1 = a.x - b.x, d2 = a.y - b.y, d3 = a.z - b.z;
  float dist = sqrtf(d1 * d1 + d2 * d2 + d3 * d3);
  return dist < a.w + b.w;
}

// One thread per disc, in cell order (the lanes of a warp read the same runs).
// FILL = false: the row's length; FILL = true: the row, sorted by id, as ids and
// as disc slots.  Bound by the latency of the nine runs' loads; cells of 2 r_max
// (up to 16 a disc) instead of fewer, wider ones, discs copied in cell order and
// rows sorted in the thread took the pair of launches from 0.15 to 0.06 ms on
// 98 k discs and from 22 to 1.3 ms on 4.19 M.
template <bool FILL>
__global__ void neighbor_kernel(const float4* __restrict__ cell_disc, const uint32_t* __restrict__ cell_id, int64_t nd,
                                Grid g, const uint32_t* __restrict__ start, int64_t* __restrict__ row,
                                const uint32_t* __restrict__ slot_of_id, int32_t* __restrict__ cols,
                                uint32_t* __restrict__ slots) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nd) return;
  const float4 ci = cell_disc[s];
  const uint32_t id = cell_id[s];
  const int cx = cell_coord(ci.x, g.org[0], g.inv_h, g.dim[0]);
  const int cy = cell_coord(ci.y, g.org[1], g.inv_h, g.dim[1]);
  const int cz = cell_coord(ci.z, g.org[2], g.inv_h, g.dim[2]);
  const int x0 = max(cx - 1, 0), x1 = min(cx + 1, g.dim[0] - 1);
  constexpr int kLocal = 32;  // longer rows are sorted where they lie
  int32_t buf[FILL ? kLocal : 1];
  const int64_t out = FILL ? row[id] : 0;
  const int64_t len = FILL ? row[id + 1] - out : 0;
  const bool local = len <= kLocal;
  int64_t cnt = 0;
  for (int z = max(cz - 1, 0); z <= min(cz + 1, g.dim[2] - 1); ++z)
    for (int y = max(cy - 1, 0); y <= min(cy + 1, g.dim[1] - 1); ++y) {
      const int64_t line = ((int64_t)z * g.dim[1] + y) * g.dim[0];
      const uint32_t b = start[line + x0], e = start[line + x1 + 1];
      for (uint32_t q = b; q < e; ++q) {
        if (q == (uint32_t)s || !overlaps(ci, cell_disc[q])) continue;
        if (FILL) {
          if (cnt >= len) continue;  // cannot happen: the same test counted the row
          const int32_t j = (int32_t)cell_id[q];
          if (local) {  // insertion by id
            int k = (int)cnt;
            for (; k > 0 && buf[k - 1] > j; --k) buf[k] = buf[k - 1];
            buf[k] = j;
          } else {
            int64_t k = out + cnt;
            for (; k > out && cols[k - 1] > j; --k) cols[k] = cols[k - 1];
            cols[k] = j;
          }
        }
        ++cnt;
      }
    }
  if (FILL) {
    for (int64_t k = 0; k < len; ++k) {
      const int32_t j = local ? buf[k] : cols[out + k];
      if (local) cols[out + k] = j;
      slots[out + k] = slot_of_id[j];
    }
  } else {
    row[id] = cnt;
  }
}

// ---------------- exposed area (disc_bounding_box_intersector.hpp) ----------
struct BB {
  float lx, ly, hx, hy;
};
struct DBBI {
  BB bb;
  BB t[2][2];
};

__host__ __device__ inline void swapf(float& a, float& b) {
  float t = a;
  a = b;
  b = t;
}

// fill_bboxtransforms / fix_bboxtransforms (lines 265-340)
inline DBBI make_dbbi(float xmin, float ymin, float xmax, float ymax) {
  DBBI g;
  g.bb = BB{xmin, ymin, xmax, ymax};
  g.t[0][0] = g.bb;
  BB c = g.bb;
  swapf(c.lx, c.ly);
  swapf(c.hx, c.hy);
  c.ly *= -1;
  c.hy *= -1;
  g.t[1][0] = c;
  c = g.bb;
  c.lx *= -1;
  c.hx *= -1;
  c.ly *= -1;
  c.hy *= -1;
  g.t[0][1] = c;
  c = g.bb;
  swapf(c.lx, c.ly);
  swapf(c.hx, c.hy);
  c.lx *= -1;
  c.hx *= -1;
  g.t[1][1] = c;
  if (g.bb.lx > g.bb.hx) swapf(g.bb.lx, g.bb.hx);
  if (g.bb.ly > g.bb.hy) swapf(g.bb.ly, g.bb.hy);
  for (int i = 0; i < 2; ++i)
    for (int j = 0; j < 2; ++j) {
      BB& r = g.t[i][j];
      if (r.lx > r.hx) swapf(r.lx, r.hx);
      if (r.ly > r.hy) swapf(r.ly, r.hy);
    }
  return g;
}

struct Approach {
  float approach;
  int swp, refl;
};

// compute_closest_approach(disc, normal, swapXY, reflectX) (lines 372-441)
__device__ float closest_approach1(const DBBI& g, float4 disc, f3 n, int swp, int refl) {
  float xx = swp ? disc.y : disc.x;
  float ny = swp ? n.x : n.y;
  float nz = n.z;
  if (refl) xx = -xx;
  const BB& bb = g.t[swp][refl];
  const float radius = disc.w;
  float xterm = radius * sqrtf(nz * nz + ny * ny);
  if (xx + xterm <= bb.hx) return FLT_MAX;
  if (xx - xterm >= bb.hx) return -FLT_MAX;
  if ((double)xterm <= 1e-9) return FLT_MAX;
  return (bb.hx - xx) * radius / xterm;
}

__device__ f3 neg3(f3 a) { return mk3(-a.x, -a.y, -a.z); }
__device__ f3 scl3(float f, f3 v) { return mk3(v.x * f, v.y * f, v.z * f); }
__device__ f3 add3(f3 a, f3 b) { return mk3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ f3 diff3(f3 a, f3 b) { return mk3(a.x + (-b.x), a.y + (-b.y), a.z + (-b.z)); }
__device__ float dist3(f3 a, f3 b) {
  float d1 = a.x - b.x, d2 = a.y - b.y, d3 = a.z - b.z;
  return sqrtf(d1 * d1 + d2 * d2 + d3 * d3);
}

// compute_area_outside_given_closest_approach (lines 108-263)
__device__ float area_outside(const DBBI& g, float4 disc, f3 dn, const Approach* ao) {
  const float radius = disc.w;
  float area = 0.0f;
  for (int i = 0; i < 4; ++i) {
    const float dd = ao[i].approach;
    if (-radius < dd && dd < radius) {
      double angle = 2 * acos((double)dd / radius);
      double seg = (double)(radius * radius / 2) * (angle - sin(angle));
      area = (float)((double)area + seg);
    }
  }
  for (int i = 0; i < 4; ++i) {
    const Approach& a1 = ao[i];
    const Approach& a2 = ao[(i + 1) % 4];
    const float d1 = a1.approach, d2 = a2.approach;
    const BB& t1 = g.t[a1.swp][a1.refl];
    const BB& t2 = g.t[a2.swp][a2.refl];
    if (!(-radius < d1 && d1 < radius && -radius < d2 && d2 < radius)) continue;
    f3 dp = mk3(disc.x, disc.y, disc.z);
    f3 p1 = mk3(t1.hx, t1.hy, 0), p2 = mk3(t2.hx, t2.hy, 0);
    f3 n1 = normalize3(cross3(sub3(mk3(t1.hx, t1.hy, 0), mk3(t1.hx, t1.hy, 1)),
                              sub3(mk3(t1.hx, t1.ly, 0), mk3(t1.hx, t1.hy, 1))));
    f3 n2 = normalize3(cross3(sub3(mk3(t2.hx, t2.hy, 0), mk3(t2.hx, t2.hy, 1)),
                              sub3(mk3(t2.hx, t2.ly, 0), mk3(t2.hx, t2.hy, 1))));
    if (a1.refl) { p1.y *= -1; n1.y *= -1; p1.x *= -1; n1.x *= -1; }
    if (a2.refl) { p2.y *= -1; n2.y *= -1; p2.x *= -1; n2.x *= -1; }
    if (a1.swp) { p1.y *= -1; n1.y *= -1; swapf(p1.x, p1.y); swapf(n1.x, n1.y); }
    if (a2.swp) { p2.y *= -1; n2.y *= -1; swapf(p2.x, p2.y); swapf(n2.x, n2.y); }
    f3 id1 = normalize3(cross3(dn, n1));
    f3 id2 = normalize3(cross3(dn, n2));
    if (dot3(id1, n2) >= 0) id1 = neg3(id1);
    if (dot3(id2, n1) >= 0) id2 = neg3(id2);
    const float xi = p2.x, yi = p2.y;
    f3 ip = mk3(xi, yi, (dn.x * dp.x + dn.y * dp.y + dn.z * dp.z - dn.x * xi - dn.y * yi) / dn.z);
    if (dist3(dp, ip) >= radius) continue;
    f3 ic1 = diff3(dp, ip);
    float ca1 = dot3(ic1, id1);
    f3 cp1 = add3(ip, scl3(ca1, id1));
    float thc1 = sqrtf(radius * radius - d1 * d1);
    f3 q1 = add3(cp1, scl3(thc1, id1));
    f3 ic2 = diff3(dp, ip);
    float ca2 = dot3(ic2, id2);
    f3 cp2 = add3(ip, scl3(ca2, id2));
    float thc2 = sqrtf(radius * radius - d2 * d2);
    f3 q2 = add3(cp2, scl3(thc2, id2));
    f3 cq1 = diff3(q1, dp), cq2 = diff3(q2, dp);
    float ang = acosf(dot3(cq1, cq2) / len3(cq1) / len3(cq2));
    float oseg = radius * radius / 2 * (ang - sinf(ang));
    f3 k1 = diff3(q1, ip), k2 = diff3(q2, ip);
    float otri = 0.5f * len3(cross3(k1, k2));
    area -= oseg + otri;
  }
  return area;
}

// area_inside (lines 42-76)
__device__ float area_inside(const DBBI& g, float4 disc, float4 nrm) {
  f3 dn = normalize3(mk3(nrm.x, nrm.y, nrm.z));
  const float xx = disc.x, yy = disc.y, r = disc.w;
  if (r <= 0) return 0.0f;
  const float full = r * r * (float)3.14159265358979323846;
  const BB& b = g.bb;
  if ((b.lx <= xx - r && xx + r <= b.hx) && (b.ly <= yy - r && yy + r <= b.hy)) return full;
  if ((xx + r <= b.lx || b.hx <= xx - r) || (yy + r <= b.ly || b.hy <= yy - r)) return 0.0f;
  // order right, bottom, left, top: (swap, reflect) = (0,0) (1,1) (0,1) (1,0)
  Approach ao[4];
  for (int i = 0; i < 4; ++i) ao[i] = Approach{0.0f, 0, 0};
  for (int i = 0; i < 4; ++i) {
    const int swp = (i == 1 || i == 3) ? 1 : 0, refl = (i == 1 || i == 2) ? 1 : 0;
    ao[i].approach = closest_approach1(g, disc, dn, swp, refl);
    ao[i].swp = swp;
    ao[i].refl = refl;
    if (ao[i].approach < -r) break;
  }
  for (int i = 0; i < 4; ++i)
    if (ao[i].approach < -r) return 0.0f;
  return full - area_outside(g, disc, dn, ao);
}

__global__ void area_kernel(const float4* __restrict__ dcr, const float4* __restrict__ dn, int64_t nd,
                            const float4* __restrict__ tv, const uint32_t* __restrict__ tidx, int64_t nt,
                            DBBI g, float* __restrict__ out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nd) {
    out[i] = area_inside(g, dcr[i], dn[i]);
  } else if (i < nd + nt) {
    int64_t t = i - nd;
    float4 a = tv[tidx[3 * t]], b = tv[tidx[3 * t + 1]], c = tv[tidx[3 * t + 2]];
    f3 v0 = mk3(a.x, a.y, a.z);
    f3 e1 = sub3(mk3(b.x, b.y, b.z), v0), e2 = sub3(mk3(c.x, c.y, c.z), v0);
    out[i] = (float)(0.5 * len3(cross3(e1, e2)));
  }
}

// ---------------- normalised smoothed estimates (device.hpp:154-187) --------
// S1 per area of every disc: a disc's value is read once for itself and once
// for every neighbour, and the FP64 division is what these kernels wait for
// (98 k discs: 37 us with a division per neighbour, now 6 + 8).
__global__ void flux_kernel(const double* __restrict__ s1, const float* __restrict__ areas, int64_t nd,
                            double* __restrict__ flux) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nd) flux[i] = s1[i] / areas[i];
}

__global__ void smooth_kernel(const double* __restrict__ s1, const float* __restrict__ areas,
                              const double* __restrict__ flux, int64_t n, int64_t nd, const int64_t* __restrict__ rp,
                              const int32_t* __restrict__ cols, float* __restrict__ est,
                              unsigned long long* __restrict__ maxbits) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double vv = 0.0;
  if (i < n) {
    int64_t deg = 0;
    if (i < nd) {
      vv = flux[i];
      const int64_t q0 = rp[i], q1 = rp[i + 1];
      for (int64_t q = q0; q < q1; ++q) vv += flux[cols[q]];
      deg = q1 - q0;
    } else {
      vv = s1[i] / areas[i];
    }
    vv /= (double)(deg + 1);
    est[i] = (float)vv;
  }
  // maxv tracks only values that compare greater than the running max (0 start)
  double m = (i < n && vv > 0.0) ? vv : 0.0;
  for (int o = 16; o > 0; o >>= 1) {
    double y = __shfl_down_sync(0xFFFFFFFFu, m, o);
    if (y > m) m = y;
  }
  if ((threadIdx.x & 31) == 0 && m > 0.0) atomicMax(maxbits, (unsigned long long)__double_as_longlong(m));
}

__global__ void divide_kernel(float* __restrict__ est, int64_t n, const unsigned long long* __restrict__ maxbits) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double maxv = __longlong_as_double((long long)*maxbits);
  est[i] = (float)((double)est[i] / maxv);
}

__global__ void stats_kernel(const double* __restrict__ s1, const double* __restrict__ s2,
                             const double* __restrict__ s3, const double* __restrict__ s4,
                             const unsigned long long* __restrict__ cnt, int64_t n, unsigned long long total,
                             double* __restrict__ rel, double* __restrict__ vov) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  // get_relative_error (hit_accumulator.hpp:152-186)
  double r = DBL_MAX;
  if (total != 0) {
    double sq = s1[i] * s1[i];
    if (sq != 0) r = sqrt(s2[i] / sq - 1.0 / (double)total);
  }
  rel[i] = r;
  // get_vov (hit_accumulator.hpp:188-249)
  double v = DBL_MAX;
  if (cnt[i] != 0) {
    double a = s1[i], b = s2[i], c = s3[i], d = s4[i];
    double a2 = a * a, a4 = a2 * a2, b2 = b * b;
    unsigned long long nn = total, nn2 = nn * nn, nn3 = nn * nn * nn;
    double num = d - (4 * a * c / nn) + (8 * b * a2 / nn2) - (4 * a4 / nn3) - (b2 / nn);
    double dr2 = nn * b - a2;
    double den2 = dr2 * dr2;
    v = den2 == 0 ? DBL_MAX : num / den2 * nn * nn;
  }
  vov[i] = v;
}

}  // namespace

// Enqueues the discs' cells and the row lengths, scanned into nb_ptr: needs the
// discs by id only, so that it runs before the tree is there.
int count_neighbors(rtg_context* ctx, NeighborWork& w) {
  Geometry& g = ctx->g;
  cudaStream_t st = ctx->stream;
  const int64_t nd = g.nd;
  g.nb_nnz = 0;
  RTG_TRY(dalloc(ctx, g.nb_ptr, (size_t)(nd + 1), "neighbour row pointers"));
  if (nd == 0) return RTG_OK;
  RTG_CUDA(ctx, cudaMemsetAsync(g.nb_ptr.p + nd, 0, sizeof(int64_t), st));
  if (nd == 1) {
    RTG_CUDA(ctx, cudaMemsetAsync(g.nb_ptr.p, 0, sizeof(int64_t), st));
    return RTG_OK;
  }
  // A cell is 1 % wider than the largest distance of an overlap, far more than
  // the rounding of a coordinate (below 2^-8 cells for up to 2^14 a side), so
  // overlapping discs lie at most one cell apart.
  Grid grid;
  double h = 2.02 * (double)g.rmax;
  if (!(h > 0.0)) h = 1.0;
  double ext[3];
  for (int a = 0; a < 3; ++a) ext[a] = (double)g.cmax[a] - (double)g.cmin[a];
  // at most 16 cells a disc; larger cells keep the test exact
  for (;;) {
    double cells = 1.0;
    bool fits = true;
    for (int a = 0; a < 3; ++a) {
      const double n = std::floor(ext[a] / h) + 2.0;
      fits = fits && n <= 16384.0;
      cells *= n;
    }
    if (fits && cells <= 16.0 * (double)nd + 4096.0 && cells < 2.0e9) break;
    h *= 1.25;
  }
  for (int a = 0; a < 3; ++a) {
    grid.org[a] = g.cmin[a];
    grid.dim[a] = (int)std::floor(ext[a] / h) + 2;
  }
  grid.inv_h = (float)(1.0 / h);
  const int64_t ncells = (int64_t)grid.dim[0] * grid.dim[1] * grid.dim[2];
  RTG_TRY(talloc(ctx, w.start, (size_t)(ncells + 1), st, "grid cells"));
  RTG_TRY(talloc(ctx, w.cell_rank, (size_t)nd, st, "grid cells"));
  RTG_TRY(talloc(ctx, w.cell_disc, (size_t)nd, st, "grid discs"));
  RTG_TRY(talloc(ctx, w.cell_id, (size_t)nd, st, "grid ids"));
  cudaMemsetAsync(w.start.p, 0, (size_t)(ncells + 1) * sizeof(uint32_t), st);
  cell_count_kernel<<<blocks_for(nd, 256), 256, 0, st>>>(g.disc_cr_by_id.p, nd, grid, w.start.p, w.cell_rank.p);
  RTG_TRY(exclusive_scan_u32(ctx, w.start.p, ncells + 1, nullptr, st));
  cell_place_kernel<<<blocks_for(nd, 256), 256, 0, st>>>(g.disc_cr_by_id.p, nd, w.start.p, w.cell_rank.p,
                                                         w.cell_disc.p, w.cell_id.p);
  neighbor_kernel<false><<<blocks_for(nd, 128), 128, 0, st>>>(w.cell_disc.p, w.cell_id.p, nd, grid, w.start.p,
                                                              g.nb_ptr.p, nullptr, nullptr, nullptr);
  RTG_CUDA(ctx, cudaGetLastError());
  RTG_TRY(exclusive_scan_i64(ctx, g.nb_ptr.p, nd + 1, nullptr, st));
  for (int a = 0; a < 3; ++a) {
    w.org[a] = grid.org[a];
    w.dim[a] = grid.dim[a];
  }
  w.inv_h = grid.inv_h;
  return RTG_OK;
}

// Enqueues the rows, once the tree's slots are there (waits for the row lengths).
int fill_neighbors(rtg_context* ctx, NeighborWork& w) {
  Geometry& g = ctx->g;
  cudaStream_t st = ctx->stream;
  const int64_t nd = g.nd;
  if (nd == 0) return RTG_OK;
  int64_t nnz = 0;
  RTG_CUDA(ctx, cudaMemcpyAsync(&nnz, g.nb_ptr.p + nd, sizeof nnz, cudaMemcpyDeviceToHost, st));
  RTG_CUDA(ctx, cudaStreamSynchronize(st));
  RTG_TRY(dalloc(ctx, g.nb_idx, (size_t)(nnz > 0 ? nnz : 1), "neighbour columns"));
  RTG_TRY(dalloc(ctx, g.nb_slot, (size_t)(nnz > 0 ? nnz : 1), "neighbour slots"));
  g.nb_nnz = nnz;
  if (nnz == 0) return RTG_OK;
  Grid grid;
  for (int a = 0; a < 3; ++a) {
    grid.org[a] = w.org[a];
    grid.dim[a] = w.dim[a];
  }
  grid.inv_h = w.inv_h;
  neighbor_kernel<true><<<blocks_for(nd, 128), 128, 0, st>>>(w.cell_disc.p, w.cell_id.p, nd, grid, w.start.p,
                                                             g.nb_ptr.p, g.disc_slot.p, g.nb_idx.p, g.nb_slot.p);
  RTG_CUDA(ctx, cudaGetLastError());
  return RTG_OK;
}

void release_neighbors(NeighborWork& w, cudaStream_t st) {
  tfree(w.start, st);
  tfree(w.cell_rank, st);
  tfree(w.cell_disc, st);
  tfree(w.cell_id, st);
}

int compute_areas_into(rtg_context* ctx, cudaStream_t st, const float* box_lo, const float* box_hi, float* out) {
  Geometry& g = ctx->g;
  const int64_t np = g.nd + g.nt;
  DBBI dbbi = make_dbbi(box_lo[0], box_lo[1], box_hi[0], box_hi[1]);
  area_kernel<<<blocks_for(np, 256), 256, 0, st>>>(g.disc_cr_by_id.p, g.disc_n_by_id.p, g.nd, g.tri_v.p,
                                                   g.tri_idx.p, g.nt, dbbi, out);
  RTG_CUDA(ctx, cudaGetLastError());
  return RTG_OK;
}

int compute_areas(rtg_context* ctx, cudaStream_t st, const float* box_lo, const float* box_hi) {
  return compute_areas_into(ctx, st, box_lo, box_hi, ctx->areas.p);
}

int finalize_estimates(rtg_context* ctx, cudaStream_t st) {
  Geometry& g = ctx->g;
  const int64_t np = g.nd + g.nt;
  RTG_TRY(dalloc(ctx, ctx->stat_tmp, (size_t)(2 * np), "estimates"));
  unsigned long long* mx = reinterpret_cast<unsigned long long*>(ctx->stat_tmp.p);
  double* flux = ctx->stat_tmp.p + 1;  // at most 2 np - 1 discs
  RTG_CUDA(ctx, cudaMemsetAsync(mx, 0, sizeof(unsigned long long), st));
  if (g.nd > 0) flux_kernel<<<blocks_for(g.nd, 256), 256, 0, st>>>(ctx->acc.p, ctx->areas.p, g.nd, flux);
  smooth_kernel<<<blocks_for(np, 256), 256, 0, st>>>(ctx->acc.p, ctx->areas.p, flux, np, g.nd, g.nb_ptr.p, g.nb_idx.p,
                                                     ctx->est.p, mx);
  divide_kernel<<<blocks_for(np, 256), 256, 0, st>>>(ctx->est.p, np, mx);
  RTG_CUDA(ctx, cudaGetLastError());
  RTG_CUDA(ctx, cudaStreamSynchronize(st));
  return RTG_OK;
}

int compute_stats(rtg_context* ctx, cudaStream_t st, uint64_t total, double* d_rel, double* d_vov) {
  const int64_t np = ctx->g.nd + ctx->g.nt;
  const double* s = ctx->acc.p;
  stats_kernel<<<blocks_for(np, 256), 256, 0, st>>>(s, s + np, s + 2 * np, s + 3 * np, ctx->cnt.p, np, total,
                                                    d_rel, d_vov);
  RTG_CUDA(ctx, cudaGetLastError());
  return RTG_OK;
}

}  // namespace rtg
