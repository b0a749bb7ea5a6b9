// rtg_lbvh.cu -- GPU LBVH over oriented discs and triangles.
//
// Replaces the Embree scene build of the reference (tracer.hpp:75-100,
// point_cloud_disc_geometry.hpp:178-222, triangle_geometry.hpp:56-99):
//   1. padded primitive boxes and centroid bounds,
//   2. 32-bit Morton codes of the centroids, their bits dealt to the axes by extent,
//   3. stable radix sort (rtg_sort.cu),
//   4. Karras (HPG 2012) binary radix tree over the keys (morton << 32 | rank),
//   5. primitives copied to slot order (LBVH leaf order) for coherent access,
//   6. bottom-up box refit with per-node arrival counters,
//   7. the four-box node of every internal node, and the stack these can need.
// rtg_update_* reruns 1, 5, 6 and 7 only (moved surface, same topology).
// Step 4 can be replaced by PLOC clustering over the same sorted leaves
// (build_ploc), whose trees need fewer node visits per query on irregular
// surfaces and take longer to build.
//
// Leaves hold one primitive; each internal node stores the boxes of both
// children (64 bytes), from which step 7 takes up to four boxes below the node
// in one fetch (QuadNode).
#include <cfloat>
#include <cstdint>
#include <vector>

#include "rtg_internal.cuh"
#include "rtg_math.cuh"

namespace rtg {

namespace {

__device__ __forceinline__ uint32_t fenc(float f) {
  uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float fdec(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Conservative boxes: the extent of the disc or of the triangle, padded so that
// every hit the primitive test accepts lies inside.  A disc reaches r
// sqrt(n_j^2 + n_k^2) / |n| along axis i; its normal may be off unit length by
// 1e-3, and max(1 - n_i^2, n_j^2 + n_k^2) is never below that square (1 - n_i^2
// is where |n| <= 1, the other where |n| >= 1).
constexpr int kBoundsThreads = 256;
__global__ void __launch_bounds__(kBoundsThreads) prim_bounds_kernel(const float4* __restrict__ dcr, const float4* __restrict__ dn, int64_t nd,
                                   const float4* __restrict__ tv, const uint32_t* __restrict__ tidx,
                                   int64_t nt, float* __restrict__ plo, float* __restrict__ phi,
                                   uint32_t* __restrict__ cbounds) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t cmin[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, cmax[3] = {0u, 0u, 0u};
  if (p < nd + nt) {
    float lo[3], hi[3];
    if (p < nd) {
      float4 c = dcr[p], n = dn[p];
      float cc[3] = {c.x, c.y, c.z}, nn[3] = {n.x, n.y, n.z};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float nj = nn[(a + 1) % 3], nk = nn[(a + 2) % 3];
        const float e = fmaxf(1.0f - nn[a] * nn[a], nj * nj + nk * nk);
        float ext = c.w * sqrtf(e);
        float pad = 1e-5f * (fabsf(cc[a]) + c.w) + 1e-4f * c.w;
        lo[a] = cc[a] - ext - pad;
        hi[a] = cc[a] + ext + pad;
      }
    } else {
      int64_t t = p - nd;
      float4 v0 = tv[tidx[3 * t]], v1 = tv[tidx[3 * t + 1]], v2 = tv[tidx[3 * t + 2]];
      float a0[3] = {v0.x, v0.y, v0.z}, a1[3] = {v1.x, v1.y, v1.z}, a2[3] = {v2.x, v2.y, v2.z};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        float l = fminf(a0[a], fminf(a1[a], a2[a])), h = fmaxf(a0[a], fmaxf(a1[a], a2[a]));
        float pad = 1e-5f * (fabsf(l) + fabsf(h)) + 1e-6f * (h - l) + 1e-7f;
        lo[a] = l - pad;
        hi[a] = h + pad;
      }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      plo[3 * p + a] = lo[a];
      phi[3 * p + a] = hi[a];
      cmin[a] = cmax[a] = fenc(0.5f * (lo[a] + hi[a]));
    }
  }
  if (!cbounds) return;
  // one atomic per block and bound (one per primitive kept the L2 atomics busy: 4.2 M discs 0.9 ms)
  __shared__ uint32_t red[kBoundsThreads / 32][6];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const uint32_t l = __reduce_min_sync(0xFFFFFFFFu, cmin[a]), h = __reduce_max_sync(0xFFFFFFFFu, cmax[a]);
    if (lane == 0) {
      red[warp][a] = l;
      red[warp][3 + a] = h;
    }
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    uint32_t v = red[0][threadIdx.x];
    for (int w = 1; w < kBoundsThreads / 32; ++w)
      v = threadIdx.x < 3 ? min(v, red[w][threadIdx.x]) : max(v, red[w][threadIdx.x]);
    if (threadIdx.x < 3) atomicMin(&cbounds[threadIdx.x], v);
    else atomicMax(&cbounds[threadIdx.x], v);
  }
}

// The order of the leaves: 32 bits, each halving the cell along the axis in
// which it is longest by then.  The cells are meant to be as wide as they are
// deep, with two exceptions along z, the axis that sources shine along:
//   - a surface deeper than wide counts as deep as wide.  Paths run down a hole,
//     and flat cells would put more of them in the way: directional source on a
//     disc hole (4 deep, 2 wide) 2.32 ms with this rule, 3.33 without;
//   - in a surface flatter than wide, z counts less by the same ratio again: the
//     height of a sheet follows its place, so a cell of its x and y is flatter
//     still than the whole (4.19 M discs, radix tree: 20.8 ms with this rule, 22.8
//     without).
// Where all centres lie above one another there is no width to go by, and all bits
// go to z.
// Bits that take turns over all three axes, ten each, whatever the extents ->
// this: 2e7 rays onto 4.19 M discs 40.0 -> 20.8 ms (radix tree), 25.1 -> 20.5
// (clustered); 262 k discs with a field 1.03 -> 0.79; 90.6 k discs 0.315 -> 0.271;
// hole, 1e7 rays 43.4 -> 43.0 (radix), 43.0 -> 42.2 (clustered); trenches the same.
__global__ void morton_kernel(const float* __restrict__ plo, const float* __restrict__ phi, int64_t np,
                              const uint32_t* __restrict__ cbounds, uint32_t* __restrict__ keys,
                              uint32_t* __restrict__ vals) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  float u[3], e[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float mn = fdec(cbounds[a]), mx = fdec(cbounds[3 + a]);
    e[a] = mx - mn;
    const float c = 0.5f * (plo[3 * p + a] + phi[3 * p + a]);
    u[a] = e[a] > 0.0f ? fminf(fmaxf((c - mn) / e[a], 0.0f), 0.99999994f) : 0.0f;
  }
  const float wide = fmaxf(e[0], e[1]);
  if (wide > 0.0f) e[2] = e[2] < wide ? e[2] * (e[2] / wide) : wide;
  uint32_t key = 0u;
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    const int a = e[0] >= e[1] ? (e[0] >= e[2] ? 0 : 2) : (e[1] >= e[2] ? 1 : 2);
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (j == a) {
        e[j] *= 0.5f;
        u[j] *= 2.0f;
        const bool upper = u[j] >= 1.0f;
        key = key << 1 | (upper ? 1u : 0u);
        if (upper) u[j] -= 1.0f;
      }
  }
  keys[p] = key;
  vals[p] = (uint32_t)p;
}

// is-disc flag per sorted position (scanned into disc slots)
__global__ void disc_flag_kernel(const uint32_t* __restrict__ sorted_prim, int64_t np, int64_t nd,
                                 uint32_t* __restrict__ flag) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  flag[i] = sorted_prim[i] < (uint32_t)nd ? 1u : 0u;
}

// Leaf references and slot-ordered primitive data.
__global__ void slots_kernel(const uint32_t* __restrict__ sorted_prim, const uint32_t* __restrict__ disc_rank,
                             int64_t np, int64_t nd, const float4* __restrict__ dcr_id,
                             const float4* __restrict__ dn_id, const float4* __restrict__ tv,
                             const uint32_t* __restrict__ tidx, float4* __restrict__ disc,
                             uint32_t* __restrict__ disc_slot, float4* __restrict__ tri,
                             uint32_t* __restrict__ leaf_ref, int32_t* __restrict__ leaf_prim, float4* __restrict__ basis) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const uint32_t p = min(sorted_prim[i], (uint32_t)(np - 1));  // a failed sort (reported) leaves anything here
  // discs before this position: all or none of them where there is one kind only
  const uint32_t ds = disc_rank ? disc_rank[i] : (nd > 0 ? (uint32_t)i : 0u);
  leaf_prim[i] = (int32_t)p;
  if (p < (uint32_t)nd) {
    float4 n = dn_id[p];
    disc[2 * (int64_t)ds] = dcr_id[p];
    disc_slot[p] = ds;
    disc[2 * (int64_t)ds + 1] = make_float4(n.x, n.y, n.z, __int_as_float((int)p));
    leaf_ref[i] = kLeafBit | ds;
    const f3 nv = mk3(n.x, n.y, n.z);
    pack_basis(normal_basis(nv), nv, basis[2 * (int64_t)ds], basis[2 * (int64_t)ds + 1]);
  } else {
    uint32_t ts = (uint32_t)i - ds;
    int64_t t = (int64_t)p - nd;
    float4 a = tv[tidx[3 * t]], b = tv[tidx[3 * t + 1]], c = tv[tidx[3 * t + 2]];
    f3 v0 = mk3(a.x, a.y, a.z);
    f3 e1 = sub3(mk3(b.x, b.y, b.z), v0);
    f3 e2 = sub3(mk3(c.x, c.y, c.z), v0);
    // util::compute_normal + normalize (i_triangle_reader.hpp:22-38)
    f3 n = normalize3(cross3(e1, e2));
    tri[4 * (int64_t)ts] = make_float4(v0.x, v0.y, v0.z, __int_as_float((int)p));
    tri[4 * (int64_t)ts + 1] = make_float4(e1.x, e1.y, e1.z, 0.0f);
    tri[4 * (int64_t)ts + 2] = make_float4(e2.x, e2.y, e2.z, 0.0f);
    tri[4 * (int64_t)ts + 3] = make_float4(n.x, n.y, n.z, 0.0f);
    leaf_ref[i] = kLeafBit | kTriBit | ts;
    pack_basis(normal_basis(n), n, basis[2 * (nd + ts)], basis[2 * (nd + ts) + 1]);
  }
}

__device__ __forceinline__ int kdelta(const uint32_t* __restrict__ m, int64_t n, int64_t i, int64_t j) {
  if (j < 0 || j >= n) return -1;
  uint64_t ki = ((uint64_t)m[i] << 32) | (uint32_t)i;
  uint64_t kj = ((uint64_t)m[j] << 32) | (uint32_t)j;
  return __clzll(ki ^ kj);
}

// Karras 2012, "Maximizing parallelism in the construction of BVHs, octrees,
// and k-d trees": internal node i covers a key range found from the sign of
// the prefix difference and splits at the highest differing bit.
__global__ void karras_kernel(const uint32_t* __restrict__ m, int64_t n, const uint32_t* __restrict__ leaf_ref,
                              Node* __restrict__ nodes, uint32_t* __restrict__ parent) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const int d = (kdelta(m, n, i, i + 1) - kdelta(m, n, i, i - 1)) >= 0 ? 1 : -1;
  const int dmin = kdelta(m, n, i, i - d);
  int64_t lmax = 2;
  while (kdelta(m, n, i, i + lmax * d) > dmin) lmax *= 2;
  int64_t l = 0;
  for (int64_t t = lmax / 2; t >= 1; t /= 2)
    if (kdelta(m, n, i, i + (l + t) * d) > dmin) l += t;
  const int64_t j = i + l * d;
  const int dnode = kdelta(m, n, i, j);
  int64_t s = 0, t = l;
  do {
    t = (t + 1) >> 1;
    if (kdelta(m, n, i, i + (s + t) * d) > dnode) s += t;
  } while (t > 1);
  const int64_t gamma = i + s * d + (d < 0 ? -1 : 0);
  const int64_t first = i < j ? i : j, last = i < j ? j : i;
  uint32_t left, right;
  if (first == gamma) {
    left = leaf_ref[gamma];
    parent[(n - 1) + gamma] = (uint32_t)i;
  } else {
    left = (uint32_t)gamma;
    parent[gamma] = (uint32_t)i;
  }
  if (last == gamma + 1) {
    right = leaf_ref[gamma + 1];
    parent[(n - 1) + gamma + 1] = (uint32_t)i;
  } else {
    right = (uint32_t)(gamma + 1);
    parent[gamma + 1] = (uint32_t)i;
  }
  nodes[i].d = make_uint4(left, right, 0u, 0u);
}


// ---- PLOC: parallel locally-ordered clustering (Meister and Bittner, TVCG
// 2018), an agglomerative build over the Morton-ordered leaves.  Each round,
// every cluster finds the neighbour within kPlocRadius positions whose merged
// box has the smallest surface area (ties: the lower position); mutual pairs
// merge into a new internal node; the survivors are compacted in order.
// Node indices are handed out from the top down, round by round and in
// position order, so the root is node 0 and the layout is deterministic.
constexpr int kPlocRadius = 16;
constexpr int kPlocThreads = 256;
constexpr uint32_t kClusterLeaf = 0x80000000u;  // cluster = sorted leaf index | bit 31, else a node index

__global__ void ploc_init_kernel(const uint32_t* __restrict__ sorted_prim, int64_t n, const float* __restrict__ plo,
                                 const float* __restrict__ phi, uint32_t* __restrict__ cid, float4* __restrict__ blo,
                                 float4* __restrict__ bhi) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t p = min(sorted_prim[i], (uint32_t)(n - 1));
  cid[i] = kClusterLeaf | (uint32_t)i;
  blo[i] = make_float4(plo[3 * p], plo[3 * p + 1], plo[3 * p + 2], 0.0f);
  bhi[i] = make_float4(phi[3 * p], phi[3 * p + 1], phi[3 * p + 2], 0.0f);
}

__device__ __forceinline__ float merged_area(float4 al, float4 ah, float4 bl, float4 bh) {
  const float dx = fmaxf(ah.x, bh.x) - fminf(al.x, bl.x);
  const float dy = fmaxf(ah.y, bh.y) - fminf(al.y, bl.y);
  const float dz = fmaxf(ah.z, bh.z) - fminf(al.z, bl.z);
  return dx * dy + dy * dz + dz * dx;
}

__global__ void __launch_bounds__(kPlocThreads) ploc_nn_kernel(const float4* __restrict__ blo,
                                                               const float4* __restrict__ bhi,
                                                               const uint64_t* __restrict__ state,
                                                               uint32_t* __restrict__ nn) {
  __shared__ float4 slo[kPlocThreads + 2 * kPlocRadius], shi[kPlocThreads + 2 * kPlocRadius];
  const int64_t n = (int64_t)state[0];
  if (n < 2 || (int64_t)blockIdx.x * kPlocThreads >= n) return;
  const int64_t b0 = (int64_t)blockIdx.x * kPlocThreads;
  for (int k = threadIdx.x; k < kPlocThreads + 2 * kPlocRadius; k += kPlocThreads) {
    const int64_t j = b0 - kPlocRadius + k;
    if (j >= 0 && j < n) {
      slo[k] = blo[j];
      shi[k] = bhi[j];
    }
  }
  __syncthreads();
  const int64_t i = b0 + threadIdx.x;
  if (i >= n) return;
  const int li = threadIdx.x + kPlocRadius;
  const float4 al = slo[li], ah = shi[li];
  float best = INFINITY;
  int64_t bj = i > 0 ? i - 1 : i + 1;
  for (int d = -kPlocRadius; d <= kPlocRadius; ++d) {
    const int64_t j = i + d;
    if (d == 0 || j < 0 || j >= n) continue;
    const float a = merged_area(al, ah, slo[li + d], shi[li + d]);
    if (a < best) {
      best = a;
      bj = j;
    }
  }
  nn[i] = (uint32_t)bj;
}

// Per position: (survives << 32) | merges-with-its-higher-mutual-neighbour,
// zero beyond the current cluster count (the scan length is an upper bound).
// The higher member of a mutual pair is absorbed.
__global__ void ploc_flags_kernel(const uint32_t* __restrict__ nn, int64_t bound, const uint64_t* __restrict__ state,
                                  unsigned long long* __restrict__ packed) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= bound) return;
  const int64_t n = (int64_t)state[0];
  if (i >= n) {
    packed[i] = 0ull;
    return;
  }
  if (n < 2) {
    packed[i] = 1ull << 32;
    return;
  }
  const uint32_t j = nn[i];
  const bool mutual = nn[j] == (uint32_t)i;
  const unsigned long long merge = (mutual && (uint32_t)i < j) ? 1ull : 0ull;
  const unsigned long long keep = (mutual && (uint32_t)i > j) ? 0ull : 1ull;
  packed[i] = (keep << 32) | merge;
}

// After the scan: state[0] = surviving clusters, state[1] += merges; a round
// without a merge while clusters remain is recorded in state[2].
__global__ void ploc_update_kernel(const unsigned long long* __restrict__ total, uint64_t* __restrict__ state) {
  const unsigned long long t = *total;
  const uint64_t merges = t & 0xFFFFFFFFull, kept = t >> 32;
  if (merges == 0 && state[0] > 1) state[2] = 1;
  state[0] = kept;
  state[1] += merges;
}

__global__ void ploc_merge_kernel(const uint32_t* __restrict__ nn, int64_t bound,
                                  const uint64_t* __restrict__ state, const uint32_t* __restrict__ cid,
                                  const float4* __restrict__ blo, const float4* __restrict__ bhi,
                                  const unsigned long long* __restrict__ packed, uint32_t n_int,
                                  const uint32_t* __restrict__ leaf_ref, int64_t nleaves, Node* __restrict__ nodes,
                                  uint32_t* __restrict__ parent, uint32_t* __restrict__ cid_out,
                                  float4* __restrict__ blo_out, float4* __restrict__ bhi_out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n = (int64_t)state[0];
  if (i >= bound || i >= n) return;
  if (n < 2) {  // the finished root cluster: carried over unchanged
    cid_out[0] = cid[0];
    blo_out[0] = blo[0];
    bhi_out[0] = bhi[0];
    return;
  }
  const uint32_t j = nn[i];
  const bool mutual = nn[j] == (uint32_t)i;
  if (mutual && (uint32_t)i > j) return;  // absorbed by j
  // positions after compaction (high word) and merge ranks (low word) come
  // from the exclusive scan; nodes are handed out downwards from node_top
  const uint32_t pos = (uint32_t)(packed[i] >> 32);
  const uint32_t rank = (uint32_t)(packed[i] & 0xFFFFFFFFull);
  const uint32_t node_top = n_int - 1u - (uint32_t)state[1];
  if (mutual) {
    const uint32_t idx = node_top - rank;
    const uint32_t a = cid[i], b = cid[j];
    const uint32_t ra = (a & kClusterLeaf) ? leaf_ref[a & ~kClusterLeaf] : a;
    const uint32_t rb = (b & kClusterLeaf) ? leaf_ref[b & ~kClusterLeaf] : b;
    nodes[idx].d = make_uint4(ra, rb, 0u, 0u);
    if (a & kClusterLeaf) parent[(nleaves - 1) + (a & ~kClusterLeaf)] = idx;
    else parent[a] = idx;
    if (b & kClusterLeaf) parent[(nleaves - 1) + (b & ~kClusterLeaf)] = idx;
    else parent[b] = idx;
    const float4 al = blo[i], ah = bhi[i], bl = blo[j], bh = bhi[j];
    cid_out[pos] = idx;
    blo_out[pos] = make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z), 0.0f);
    bhi_out[pos] = make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), 0.0f);
  } else {
    cid_out[pos] = cid[i];
    blo_out[pos] = blo[i];
    bhi_out[pos] = bhi[i];
  }
}

// The last rounds of PLOC in one block: once at most kPlocTailMax clusters
// remain, the rounds are too small to fill the GPU and a launch sequence per
// round (neighbours, flags, scan, merge) costs more than the work.  One block
// of kPlocTailThreads runs every remaining round with the same rules as the
// kernels above -- nearest neighbour within kPlocRadius positions (ties to the
// lower position), mutual pairs merged by the lower member, survivors
// compacted in order, nodes handed out downwards in position order -- so the
// tree is the one the round-by-round launches would build.  Each round merges
// at least the pair of smallest merged area, so the loop ends after at most
// n - 1 rounds (n_int + 1 bounds it); a round without a merge sets state[2]
// and stops.
constexpr uint32_t kPlocTailMax = 8192;  // measured: 2 Ki-8 Ki fastest on the hole (200 k leaves)
constexpr int kPlocTailThreads = 1024;

__global__ void __launch_bounds__(kPlocTailThreads) ploc_tail_kernel(
    uint32_t* __restrict__ cid0, float4* __restrict__ blo0, float4* __restrict__ bhi0, uint32_t* __restrict__ cid1,
    float4* __restrict__ blo1, float4* __restrict__ bhi1, uint32_t* __restrict__ nn, uint64_t* __restrict__ state,
    uint32_t n_int, const uint32_t* __restrict__ leaf_ref, int64_t nleaves, Node* __restrict__ nodes,
    uint32_t* __restrict__ parent) {
  __shared__ uint32_t w_keep[kPlocTailThreads / 32], w_merge[kPlocTailThreads / 32];
  __shared__ uint32_t s_tot[2];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  uint32_t n = (uint32_t)state[0];
  uint32_t allocated = (uint32_t)state[1];
  uint32_t* cid_in = cid0;
  float4* blo_in = blo0;
  float4* bhi_in = bhi0;
  uint32_t* cid_out = cid1;
  float4* blo_out = blo1;
  float4* bhi_out = bhi1;
  bool stalled = false;
  for (uint32_t round = 0; n > 1 && round < n_int + 1u; ++round) {
    for (uint32_t i = tid; i < n; i += kPlocTailThreads) {
      const float4 al = blo_in[i], ah = bhi_in[i];
      float best = INFINITY;
      uint32_t bj = i > 0 ? i - 1 : i + 1;
      for (int d = -kPlocRadius; d <= kPlocRadius; ++d) {
        const int64_t j = (int64_t)i + d;
        if (d == 0 || j < 0 || j >= (int64_t)n) continue;
        const float a = merged_area(al, ah, blo_in[j], bhi_in[j]);
        if (a < best) {
          best = a;
          bj = (uint32_t)j;
        }
      }
      nn[i] = bj;
    }
    __syncthreads();
    // survivors and merges of this thread's run of positions, then their
    // exclusive prefix over the block (positions in order)
    const uint32_t per = (n + kPlocTailThreads - 1) / kPlocTailThreads;
    const uint32_t c0 = min(n, tid * per), c1 = min(n, c0 + per);
    uint32_t keep = 0, merge = 0;
    for (uint32_t i = c0; i < c1; ++i) {
      const uint32_t j = nn[i];
      const bool mutual = nn[j] == i;
      keep += (mutual && i > j) ? 0u : 1u;
      merge += (mutual && i < j) ? 1u : 0u;
    }
    uint32_t ik = keep, im = merge;  // inclusive warp scan
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t k2 = __shfl_up_sync(0xFFFFFFFFu, ik, o), m2 = __shfl_up_sync(0xFFFFFFFFu, im, o);
      if (lane >= (uint32_t)o) {
        ik += k2;
        im += m2;
      }
    }
    if (lane == 31) {
      w_keep[warp] = ik;
      w_merge[warp] = im;
    }
    __syncthreads();
    if (warp == 0) {
      uint32_t tk = lane < kPlocTailThreads / 32 ? w_keep[lane] : 0u, tm = lane < kPlocTailThreads / 32 ? w_merge[lane] : 0u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t k2 = __shfl_up_sync(0xFFFFFFFFu, tk, o), m2 = __shfl_up_sync(0xFFFFFFFFu, tm, o);
        if (lane >= (uint32_t)o) {
          tk += k2;
          tm += m2;
        }
      }
      if (lane < kPlocTailThreads / 32) {  // inclusive prefix over the warps
        w_keep[lane] = tk;
        w_merge[lane] = tm;
      }
      if (lane == kPlocTailThreads / 32 - 1) {
        s_tot[0] = tk;
        s_tot[1] = tm;
      }
    }
    __syncthreads();
    uint32_t pos = (warp > 0 ? w_keep[warp - 1] : 0u) + ik - keep;
    uint32_t rank = (warp > 0 ? w_merge[warp - 1] : 0u) + im - merge;
    const uint32_t kept_total = s_tot[0], merged_total = s_tot[1];
    const uint32_t node_top = n_int - 1u - allocated;
    for (uint32_t i = c0; i < c1; ++i) {
      const uint32_t j = nn[i];
      const bool mutual = nn[j] == i;
      if (mutual && i > j) continue;  // absorbed by j
      if (mutual) {
        const uint32_t idx = node_top - rank++;
        const uint32_t a = cid_in[i], b = cid_in[j];
        const uint32_t ra = (a & kClusterLeaf) ? leaf_ref[a & ~kClusterLeaf] : a;
        const uint32_t rb = (b & kClusterLeaf) ? leaf_ref[b & ~kClusterLeaf] : b;
        nodes[idx].d = make_uint4(ra, rb, 0u, 0u);
        if (a & kClusterLeaf) parent[(nleaves - 1) + (a & ~kClusterLeaf)] = idx;
        else parent[a] = idx;
        if (b & kClusterLeaf) parent[(nleaves - 1) + (b & ~kClusterLeaf)] = idx;
        else parent[b] = idx;
        const float4 al = blo_in[i], ah = bhi_in[i], bl = blo_in[j], bh = bhi_in[j];
        cid_out[pos] = idx;
        blo_out[pos] = make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z), 0.0f);
        bhi_out[pos] = make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), 0.0f);
      } else {
        cid_out[pos] = cid_in[i];
        blo_out[pos] = blo_in[i];
        bhi_out[pos] = bhi_in[i];
      }
      ++pos;
    }
    __syncthreads();  // the outputs are complete before they become the inputs
    if (merged_total == 0) {
      stalled = true;
      break;
    }
    allocated += merged_total;
    n = kept_total;
    uint32_t* tc = cid_in;
    cid_in = cid_out;
    cid_out = tc;
    float4* tl = blo_in;
    blo_in = blo_out;
    blo_out = tl;
    float4* th = bhi_in;
    bhi_in = bhi_out;
    bhi_out = th;
  }
  if (tid == 0) {
    state[0] = n;
    state[1] = allocated;
    if (stalled || n > 1) state[2] = 1;
  }
}

// A box on its way up the tree, with the height (binary levels) of its subtree.
struct __align__(16) NodeBox {
  float lo[3];
  int32_t height;
  float hi[3];
  int32_t unused;
};

__device__ __forceinline__ NodeBox child_box(uint32_t ref, const float4* __restrict__ dn,
                                             const float4* __restrict__ tri, const float* __restrict__ plo,
                                             const float* __restrict__ phi, const NodeBox* node_box) {
  NodeBox b;
  if (ref & kLeafBit) {
    uint32_t slot = ref & kSlotMask;
    int p = (ref & kTriBit) ? __float_as_int(tri[4 * (int64_t)slot].w) : __float_as_int(dn[2 * (int64_t)slot + 1].w);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      b.lo[a] = plo[3 * (int64_t)p + a];
      b.hi[a] = phi[3 * (int64_t)p + a];
    }
    b.height = 0;
  } else {  // written by another block: past L1
    const float4* q = reinterpret_cast<const float4*>(node_box + ref);
    const float4 l = __ldcg(q), h = __ldcg(q + 1);
    b.lo[0] = l.x; b.lo[1] = l.y; b.lo[2] = l.z;
    b.hi[0] = h.x; b.hi[1] = h.y; b.hi[2] = h.z;
    b.height = __float_as_int(l.w);
  }
  b.unused = 0;
  return b;
}

__device__ __forceinline__ void store_boxes(Node& n, const NodeBox& b0, const NodeBox& b1) {
  n.a = make_float4(b0.lo[0], b0.hi[0], b1.lo[0], b1.hi[0]);
  n.b = make_float4(b0.lo[1], b0.hi[1], b1.lo[1], b1.hi[1]);
  n.c = make_float4(b0.lo[2], b0.hi[2], b1.lo[2], b1.hi[2]);
}

// What a build reports: errors of the sort, the structure check and the refit,
// the tree's height, the stack need of its quads.
enum : int { kStSort = 0, kStCheck, kStRefit, kStHeight, kStNeed, kStWords };

// Bottom-up refit: the second thread to reach a node writes both child boxes.
// A serial chain of the tree's height, a node costs one atomic that orders the
// boxes behind it and two dependent loads (a fence on either side of the
// atomic, scalar box loads and the quad nodes on the same chain took 0.16 ms
// for 200 k triangles).
__global__ void refit_kernel(int64_t n, const uint32_t* __restrict__ parent, const float4* __restrict__ dn,
                             const float4* __restrict__ tri, const float* __restrict__ plo,
                             const float* __restrict__ phi, Node* nodes, NodeBox* node_box, unsigned int* flags,
                             unsigned long long* status) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t node = parent[(n - 1) + i];
  for (int iter = 0; iter < 256; ++iter) {
    if ((int64_t)node >= n - 1) break;  // a parent that was never written
    unsigned int old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(flags + node) : "memory");
    if (old == 0) return;
    const uint4 r = __ldcg(&nodes[node].d);
    const NodeBox b0 = child_box(r.x, dn, tri, plo, phi, node_box), b1 = child_box(r.y, dn, tri, plo, phi, node_box);
    store_boxes(nodes[node], b0, b1);
    const int32_t height = max(b0.height, b1.height) + 1;
    if (node == 0) {
      status[kStHeight] = (unsigned long long)height;
      return;
    }
    float4* out = reinterpret_cast<float4*>(node_box + node);
    out[0] = make_float4(fminf(b0.lo[0], b1.lo[0]), fminf(b0.lo[1], b1.lo[1]), fminf(b0.lo[2], b1.lo[2]),
                         __int_as_float(height));
    out[1] = make_float4(fmaxf(b0.hi[0], b1.hi[0]), fmaxf(b0.hi[1], b1.hi[1]), fmaxf(b0.hi[2], b1.hi[2]), 0.0f);
    node = parent[node];
  }
  atomicAdd(&status[kStRefit], 1ull);
}

// Centre and half extent (a bfloat16, rounded up) of [lo, hi] as a QuadNode
// stores them.
__device__ __forceinline__ uint32_t quad_extent(float lo, float hi, float& c) {
  c = 0.5f * lo + 0.5f * hi;
  const float e = fmaxf(__fsub_ru(hi, c), __fsub_ru(c, lo));
  const float h = __fadd_ru(__fmul_ru(e, 1.00000096f), __fmul_ru(fabsf(c), 0x1p-21f));
  return (__float_as_uint(h) + 0xFFFFu) >> 16;
}

// The QuadNode of every binary node: its two children and, as long as there is
// room for `most` boxes, those of the one of largest surface area in its
// place, which saves the query a visit.
__global__ void quad_kernel(const Node* __restrict__ nodes, int64_t n_internal, int most, QuadNode* __restrict__ quads) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_internal) return;
  float lo[4][3], hi[4][3];
  uint32_t ref[4];
  auto open = [&](uint32_t node, int k0, int k1) {
    const Node o = nodes[node];
    const float box0[6] = {o.a.x, o.b.x, o.c.x, o.a.y, o.b.y, o.c.y};
    const float box1[6] = {o.a.z, o.b.z, o.c.z, o.a.w, o.b.w, o.c.w};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[k0][a] = box0[a];
      hi[k0][a] = box0[3 + a];
      lo[k1][a] = box1[a];
      hi[k1][a] = box1[3 + a];
    }
    ref[k0] = o.d.x;
    ref[k1] = o.d.y;
  };
  open((uint32_t)i, 0, 1);
  int n = ref[0] == ref[1] ? 1 : 2;  // a one-primitive tree holds its leaf in both children of the root
  while (n > 1 && n < most) {
    int best = -1;
    float ba = -1.0f;
    for (int k = 0; k < n; ++k) {
      if (ref[k] & kLeafBit) continue;
      const float x = hi[k][0] - lo[k][0], y = hi[k][1] - lo[k][1], z = hi[k][2] - lo[k][2];
      const float area = x * y + y * z + z * x;
      if (area > ba) {
        ba = area;
        best = k;
      }
    }
    if (best < 0 || (int64_t)ref[best] >= n_internal) break;
    open(ref[best], best, n);
    ++n;
  }
  uint32_t h[4][3];
  QuadNode out;
  out.inner = 0u;
  out.unused = 0u;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float c[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      h[k][a] = __float_as_uint(-1e30f) >> 16;
      if (k < n) h[k][a] = quad_extent(lo[k][a], hi[k][a], c[a]);
    }
    out.xy[2 * k] = c[0];
    out.xy[2 * k + 1] = c[1];
    out.z[k] = c[2];
    out.ref[k] = k < n ? ref[k] : kLeafBit;
    if (!(out.ref[k] & kLeafBit)) out.inner += 1u;
  }
  out.half[0] = h[0][0] << 16 | h[1][0];
  out.half[1] = h[0][1] << 16 | h[1][1];
  out.half[2] = h[2][0] << 16 | h[3][0];
  out.half[3] = h[2][1] << 16 | h[3][1];
  out.half[4] = h[0][2] << 16 | h[2][2];
  out.half[5] = h[1][2] << 16 | h[3][2];
  quads[i] = out;
}

// The deepest stack that a traversal of the quads can need: on the way down to
// a leaf, the inner children but one wait at every quad.  One thread per leaf:
// up to the root for the path, then down along the quads on it.
__global__ void quad_need_kernel(int64_t n, const uint32_t* __restrict__ parent, const QuadNode* __restrict__ quads,
                                 unsigned long long* __restrict__ status) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned int need = 0;
  if (i < n) {
    uint32_t path[kMaxDepth];
    int len = 0;
    uint32_t node = parent[(n - 1) + i];
    bool whole = false;
    while (len < kMaxDepth && (int64_t)node < n - 1) {
      path[len++] = node;
      if (node == 0) {
        whole = true;
        break;
      }
      node = parent[node];
    }
    int at = whole ? len - 1 : -1;  // path[at] is the quad to leave; a broken link is the refit's error
    while (at > 0) {
      const uint32_t* r = quads[path[at]].ref;
      const unsigned int inner = quads[path[at]].inner;
      const uint32_t r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3];
      int next = -1;
      for (int k = at - 1; k >= 0 && k >= at - 3; --k)
        if (r0 == path[k] || r1 == path[k] || r2 == path[k] || r3 == path[k]) {
          next = k;
          break;
        }
      if (next < 0) break;  // the leaf itself is a child of this quad
      need += inner - 1;
      at = next;
    }
  }
  need = __reduce_max_sync(0xFFFFFFFFu, need);
  if ((threadIdx.x & 31) == 0 && need) atomicMax(&status[kStNeed], (unsigned long long)need);
}

// Structural check of the tree before any traversal: every child reference is
// in range, and every node except the root has exactly one parent.
// parents: [internal nodes | discs | triangles].
__global__ void validate_kernel(const Node* __restrict__ nodes, int64_t n_internal, int64_t nd, int64_t nt,
                                unsigned int* __restrict__ parents, unsigned long long* __restrict__ errors) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_internal) return;
  const uint4 d = nodes[i].d;
  const uint32_t ch[2] = {d.x, d.y};
  for (int k = 0; k < 2; ++k) {
    const uint32_t r = ch[k];
    const int64_t slot = r & kSlotMask;
    int64_t at = -1;
    if (r & kLeafBit) {
      if (r & kTriBit) at = slot < nt ? n_internal + nd + slot : -1;
      else at = slot < nd ? n_internal + slot : -1;
    } else if (!(r & kTriBit) && slot != 0 && slot < n_internal) {
      at = slot;
    }
    if (at >= 0) atomicAdd(&parents[at], 1u);
    else atomicAdd(errors, 1ull);
  }
}

// Every entry has one parent but the root (entry 0), which has none.
__global__ void count_check_kernel(const unsigned int* __restrict__ c, int64_t n,
                                   unsigned long long* __restrict__ errors) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (c[i] != (i == 0 ? 0u : 1u)) atomicAdd(errors, 1ull);
}

__global__ void single_leaf_kernel(const uint32_t* __restrict__ leaf_ref, const float4* __restrict__ dn,
                                   const float4* __restrict__ tri, const float* __restrict__ plo,
                                   const float* __restrict__ phi, Node* nodes) {
  uint32_t r = leaf_ref[0];
  const NodeBox b = child_box(r, dn, tri, plo, phi, nullptr);
  store_boxes(nodes[0], b, b);
  nodes[0].d = make_uint4(r, r, 0u, 0u);
}

inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

// Enqueues the structure check of the links.
int check_tree(rtg_context* ctx, unsigned long long* status, cudaStream_t st) {
  Geometry& g = ctx->g;
  const int64_t np = g.nd + g.nt, ni = np - 1;
  if (np < 2) return RTG_OK;
  DBuf<unsigned int> parents;
  RTG_TRY(talloc(ctx, parents, (size_t)(ni + np), st, "tree check"));
  cudaMemsetAsync(parents.p, 0, (size_t)(ni + np) * sizeof(unsigned int), st);
  validate_kernel<<<blocks_for(ni, 256), 256, 0, st>>>(g.nodes.p, ni, g.nd, g.nt, parents.p, status + kStCheck);
  count_check_kernel<<<blocks_for(ni + np, 256), 256, 0, st>>>(parents.p, ni + np, status + kStCheck);
  tfree(parents, st);
  RTG_CUDA(ctx, cudaGetLastError());
  return RTG_OK;
}

// Binary tree over the np sorted leaves by PLOC (see ploc_* kernels): writes
// the child references of nodes [0, np-1) and the parent array; boxes come
// from the refit that follows.
int build_ploc(rtg_context* ctx, const uint32_t* d_sorted_prim, cudaStream_t st) {
  Geometry& g = ctx->g;
  const int64_t n = g.nd + g.nt;
  DBuf<uint32_t> cid[2], nn;
  DBuf<float4> blo[2], bhi[2];
  DBuf<int64_t> packed, total;
  DBuf<uint64_t> state;  // [0] clusters, [1] nodes allocated, [2] stall flag
  auto cleanup = [&]() {
    for (int q = 0; q < 2; ++q) {
      tfree(cid[q], st);
      tfree(blo[q], st);
      tfree(bhi[q], st);
    }
    tfree(nn, st);
    tfree(packed, st);
    tfree(total, st);
    tfree(state, st);
  };
  int rc = RTG_OK;
  for (int q = 0; q < 2 && rc == RTG_OK; ++q) {
    rc = talloc(ctx, cid[q], (size_t)n, st, "PLOC clusters");
    if (rc == RTG_OK) rc = talloc(ctx, blo[q], (size_t)n, st, "PLOC boxes");
    if (rc == RTG_OK) rc = talloc(ctx, bhi[q], (size_t)n, st, "PLOC boxes");
  }
  if (rc == RTG_OK) rc = talloc(ctx, nn, (size_t)n, st, "PLOC neighbours");
  if (rc == RTG_OK) rc = talloc(ctx, packed, (size_t)n, st, "PLOC scan");
  if (rc == RTG_OK) rc = talloc(ctx, total, 1, st, "PLOC totals");
  if (rc == RTG_OK) rc = talloc(ctx, state, 3, st, "PLOC state");
  if (rc != RTG_OK) {
    cleanup();
    return rc;
  }
  const uint64_t init[3] = {(uint64_t)n, 0, 0};
  cudaMemcpyAsync(state.p, init, sizeof init, cudaMemcpyHostToDevice, st);
  ploc_init_kernel<<<blocks_for(n, 256), 256, 0, st>>>(d_sorted_prim, n, g.prim_lo.p, g.prim_hi.p, cid[0].p,
                                                        blo[0].p, bhi[0].p);
  const uint32_t n_int = (uint32_t)(n - 1);
  int64_t bound = n;  // the cluster count is only read back between chunks of rounds
  int q = 0;
  uint64_t h[3] = {(uint64_t)n, 0, 0};
  for (int chunk = 0; h[0] > 1; ++chunk) {
    if (chunk > 10000) {
      rc = set_error(ctx, RTG_ERR_INTERNAL, "PLOC did not converge");
      break;
    }
    if (h[0] <= kPlocTailMax) {  // the remaining rounds in one block
      ploc_tail_kernel<<<1, kPlocTailThreads, 0, st>>>(cid[q].p, blo[q].p, bhi[q].p, cid[q ^ 1].p, blo[q ^ 1].p,
                                                        bhi[q ^ 1].p, nn.p, state.p, n_int, g.leaf_ref.p, n,
                                                        g.nodes.p, g.parent.p);
    }
    for (int r = 0; r < 4 && rc == RTG_OK && h[0] > kPlocTailMax; ++r) {
      const unsigned nb = (unsigned)((bound + kPlocThreads - 1) / kPlocThreads);
      ploc_nn_kernel<<<nb, kPlocThreads, 0, st>>>(blo[q].p, bhi[q].p, state.p, nn.p);
      ploc_flags_kernel<<<blocks_for(bound, 256), 256, 0, st>>>(nn.p, bound, state.p,
                                                                (unsigned long long*)packed.p);
      rc = exclusive_scan_i64(ctx, packed.p, bound, total.p, st);
      if (rc != RTG_OK) break;
      ploc_merge_kernel<<<blocks_for(bound, 256), 256, 0, st>>>(
          nn.p, bound, state.p, cid[q].p, blo[q].p, bhi[q].p, (const unsigned long long*)packed.p, n_int,
          g.leaf_ref.p, n, g.nodes.p, g.parent.p, cid[q ^ 1].p, blo[q ^ 1].p, bhi[q ^ 1].p);
      ploc_update_kernel<<<1, 1, 0, st>>>((const unsigned long long*)total.p, state.p);
      q ^= 1;
    }
    if (rc != RTG_OK) break;
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, state.p, sizeof h, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
      rc = check_cuda(ctx, e, "PLOC round");
      break;
    }
    if (h[2] != 0 || h[1] > n_int) {
      rc = set_error(ctx, RTG_ERR_INTERNAL, "PLOC round without progress");
      break;
    }
    bound = (int64_t)h[0];
  }
  if (rc == RTG_OK && h[1] != n_int) rc = set_error(ctx, RTG_ERR_INTERNAL, "PLOC node count mismatch");
  cudaStreamSynchronize(st);
  cleanup();
  return rc;
}

int run_bounds(rtg_context* ctx, uint32_t* d_cbounds, cudaStream_t st) {
  Geometry& g = ctx->g;
  const int64_t np = g.nd + g.nt;
  RTG_TRY(dalloc(ctx, g.prim_lo, (size_t)(3 * np), "primitive boxes"));
  RTG_TRY(dalloc(ctx, g.prim_hi, (size_t)(3 * np), "primitive boxes"));
  prim_bounds_kernel<<<blocks_for(np, kBoundsThreads), kBoundsThreads, 0, st>>>(
      g.disc_cr_by_id.p, g.disc_n_by_id.p, g.nd, g.tri_v.p, g.tri_idx.p, g.nt, g.prim_lo.p, g.prim_hi.p, d_cbounds);
  RTG_CUDA(ctx, cudaGetLastError());
  return RTG_OK;
}

// Slot-ordered primitive data from the sorted primitive order.
int run_slots(rtg_context* ctx, const uint32_t* d_sorted_prim, cudaStream_t st) {
  Geometry& g = ctx->g;
  const int64_t np = g.nd + g.nt;
  DBuf<uint32_t> rank;  // discs before each sorted position, where discs and triangles mix
  if (g.nd > 0 && g.nt > 0) {
    RTG_TRY(talloc(ctx, rank, (size_t)np, st, "disc ranks"));
    disc_flag_kernel<<<blocks_for(np, 256), 256, 0, st>>>(d_sorted_prim, np, g.nd, rank.p);
    const int rc = exclusive_scan_u32(ctx, rank.p, np, nullptr, st);
    if (rc != RTG_OK) {
      tfree(rank, st);
      return rc;
    }
  }
  slots_kernel<<<blocks_for(np, 256), 256, 0, st>>>(d_sorted_prim, rank.p, np, g.nd, g.disc_cr_by_id.p,
                                                    g.disc_n_by_id.p, g.tri_v.p, g.tri_idx.p, g.disc.p, g.disc_slot.p,
                                                    g.tri.p, g.leaf_ref.p, g.leaf_prim.p, g.basis.p);
  tfree(rank, st);
  RTG_CUDA(ctx, cudaGetLastError());
  return RTG_OK;
}

// Enqueues the boxes, the quads and their stack need over the current links.
int run_refit(rtg_context* ctx, unsigned long long* status, cudaStream_t st) {
  Geometry& g = ctx->g;
  const int64_t np = g.nd + g.nt, ni = np > 1 ? np - 1 : 1;
  g.wide_current = false;  // the wide tree's boxes follow the binary ones: now, or before a trace that wants it
  RTG_TRY(dalloc(ctx, g.quads, (size_t)ni, "quad nodes"));
  if (np == 1) {
    single_leaf_kernel<<<1, 1, 0, st>>>(g.leaf_ref.p, g.disc.p, g.tri.p, g.prim_lo.p, g.prim_hi.p, g.nodes.p);
    quad_kernel<<<1, 1, 0, st>>>(g.nodes.p, 1, 4, g.quads.p);
    RTG_CUDA(ctx, cudaGetLastError());
    return RTG_OK;
  }
  DBuf<NodeBox> node_box;
  RTG_TRY(dalloc(ctx, g.refit_flags, (size_t)ni, "refit flags"));
  RTG_TRY(talloc(ctx, node_box, (size_t)ni, st, "node boxes"));
  cudaMemsetAsync(g.refit_flags.p, 0, sizeof(unsigned int) * ni, st);
  refit_kernel<<<blocks_for(np, 256), 256, 0, st>>>(np, g.parent.p, g.disc.p, g.tri.p, g.prim_lo.p, g.prim_hi.p,
                                                    g.nodes.p, node_box.p, g.refit_flags.p, status);
  tfree(node_box, st);
  quad_kernel<<<blocks_for(ni, 128), 128, 0, st>>>(g.nodes.p, ni, 4, g.quads.p);
  quad_need_kernel<<<blocks_for(np, 256), 256, 0, st>>>(np, g.parent.p, g.quads.p, status);
  RTG_CUDA(ctx, cudaGetLastError());
  return RTG_OK;
}

// Waits for the build and reads its report.
int read_status(rtg_context* ctx, const unsigned long long* status, unsigned long long* h, cudaStream_t st) {
  RTG_CUDA(ctx, cudaMemcpyAsync(h, status, kStWords * sizeof *h, cudaMemcpyDeviceToHost, st));
  RTG_CUDA(ctx, cudaStreamSynchronize(st));
  return RTG_OK;
}

// Takes over the height and the stack need of a good build.  Quads that could
// outgrow the largest stack (a clustering with many inner siblings down a deep
// path) are made again of two boxes each, which need no more than the height.
int take_shape(rtg_context* ctx, const unsigned long long* h, cudaStream_t st) {
  Geometry& g = ctx->g;
  const int64_t np = g.nd + g.nt;
  if (np == 1) {
    g.depth = 1;
    g.quad_stack = 0;
    return RTG_OK;
  }
  g.depth = (int32_t)h[kStHeight];
  g.quad_stack = (int32_t)h[kStNeed];
  if (g.quad_stack > kMaxStack) {
    quad_kernel<<<blocks_for(np - 1, 128), 128, 0, st>>>(g.nodes.p, np - 1, 2, g.quads.p);
    RTG_CUDA(ctx, cudaGetLastError());
    g.quad_stack = g.depth;
  }
  return RTG_OK;
}

int build_status(rtg_context* ctx, const unsigned long long* h) {
  if (h[kStSort]) return set_error(ctx, RTG_ERR_INTERNAL, "radix sort did not finish");
  if (h[kStCheck])
    return set_error(ctx, RTG_ERR_INTERNAL, "LBVH check failed: " + std::to_string(h[kStCheck]) + " bad links");
  if (h[kStRefit]) return set_error(ctx, RTG_ERR_INTERNAL, "LBVH refit exceeded its depth limit");
  if (h[kStHeight] > (unsigned long long)kMaxDepth)
    return set_error(ctx, RTG_ERR_INTERNAL, "LBVH deeper than 256 levels");
  return RTG_OK;
}

}  // namespace

int build_lbvh(rtg_context* ctx) {
  Geometry& g = ctx->g;
  cudaStream_t st = ctx->stream;
  const int64_t np = g.nd + g.nt;
  if (np <= 0) return set_error(ctx, RTG_ERR_NO_GEOMETRY, "no primitives");
  if (np > (int64_t)kSlotMask) return set_error(ctx, RTG_ERR_INVALID_ARGUMENT, "too many primitives");
  DBuf<uint32_t> cb, pairs;  // centroid bounds; keys | values | scratch for both
  DBuf<unsigned long long> status;
  auto cleanup = [&]() { tfree(cb, st); tfree(pairs, st); tfree(status, st); };
  int rc = RTG_OK;
  do {
    if ((rc = talloc(ctx, cb, 6, st, "centroid bounds")) != RTG_OK) break;
    if ((rc = talloc(ctx, status, kStWords, st, "build status")) != RTG_OK) break;
    if ((rc = talloc(ctx, pairs, (size_t)(4 * np), st, "morton pairs")) != RTG_OK) break;
    uint32_t *keys = pairs.p, *vals = pairs.p + np, *tk = pairs.p + 2 * np, *tv = pairs.p + 3 * np;
    cudaMemsetAsync(cb.p, 0xFF, 3 * sizeof(uint32_t), st);
    cudaMemsetAsync(cb.p + 3, 0, 3 * sizeof(uint32_t), st);
    cudaMemsetAsync(status.p, 0, kStWords * sizeof(unsigned long long), st);
    if ((rc = run_bounds(ctx, cb.p, st)) != RTG_OK) break;
    morton_kernel<<<blocks_for(np, 256), 256, 0, st>>>(g.prim_lo.p, g.prim_hi.p, np, cb.p, keys, vals);
    if ((rc = radix_sort_pairs(ctx, keys, vals, tk, tv, np, 32, status.p + kStSort, st)) != RTG_OK) break;
    if ((rc = dalloc(ctx, g.disc, (size_t)(2 * (g.nd ? g.nd : 1)), "disc slots")) != RTG_OK) break;
    if ((rc = dalloc(ctx, g.disc_slot, (size_t)(g.nd ? g.nd : 1), "disc slot map")) != RTG_OK) break;
    if ((rc = dalloc(ctx, g.tri, (size_t)(4 * (g.nt ? g.nt : 1)), "triangle slots")) != RTG_OK) break;
    if ((rc = dalloc(ctx, g.basis, (size_t)(2 * np), "normal bases")) != RTG_OK) break;
    if ((rc = dalloc(ctx, g.leaf_ref, (size_t)np, "leaf references")) != RTG_OK) break;
    if ((rc = dalloc(ctx, g.leaf_prim, (size_t)np, "leaf primitives")) != RTG_OK) break;
    const int64_t nn = np > 1 ? np - 1 : 1;
    if ((rc = dalloc(ctx, g.nodes, (size_t)nn, "LBVH nodes")) != RTG_OK) break;
    if ((rc = dalloc(ctx, g.parent, (size_t)(2 * np), "LBVH parents")) != RTG_OK) break;
    // slots first: the builders read the leaf references
    if ((rc = run_slots(ctx, vals, st)) != RTG_OK) break;
    unsigned long long h[kStWords] = {};
    // PLOC first; a clustering deeper than the traversal stacks allow (possible
    // for degenerate inputs) falls back to the Karras tree, whose depth is
    // bounded by the key length
    for (bool karras = g.builder != kBuilderPloc || np == 1;; karras = true) {
      if (np > 1) {
        cudaMemsetAsync(g.parent.p, 0xFF, 2 * np * sizeof(uint32_t), st);
        if (karras) {
          karras_kernel<<<blocks_for(np - 1, 256), 256, 0, st>>>(keys, np, g.leaf_ref.p, g.nodes.p, g.parent.p);
        } else if ((rc = build_ploc(ctx, vals, st)) != RTG_OK) {
          break;
        }
        if ((rc = check_tree(ctx, status.p, st)) != RTG_OK) break;
      }
      if ((rc = run_refit(ctx, status.p, st)) != RTG_OK) break;
      if ((rc = read_status(ctx, status.p, h, st)) != RTG_OK) break;
      const bool deep = h[kStRefit] != 0 || h[kStHeight] > (unsigned long long)kMaxDepth;
      if (karras || h[kStSort] || h[kStCheck] || !deep) break;
      cudaMemsetAsync(status.p, 0, kStWords * sizeof(unsigned long long), st);
    }
    if (rc == RTG_OK) rc = build_status(ctx, h);
    if (rc == RTG_OK) rc = take_shape(ctx, h, st);
    if (rc == RTG_OK && wants_wide(ctx)) rc = build_wide(ctx, st);
  } while (0);
  if (rc != RTG_OK) cudaStreamSynchronize(st);
  cleanup();
  g.root = 0;
  return rc;
}

int refit_lbvh(rtg_context* ctx) {
  Geometry& g = ctx->g;
  cudaStream_t st = ctx->stream;
  RTG_TRY(run_bounds(ctx, nullptr, st));
  // keep the leaf order: recompute slot data from the sorted primitive order
  const int64_t np = g.nd + g.nt;
  DBuf<uint32_t> order;
  DBuf<unsigned long long> status;
  int rc = talloc(ctx, order, (size_t)np, st, "leaf order");
  if (rc == RTG_OK) rc = talloc(ctx, status, kStWords, st, "build status");
  unsigned long long h[kStWords] = {};
  if (rc == RTG_OK) {
    cudaMemcpyAsync(order.p, g.leaf_prim.p, np * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st);
    cudaMemsetAsync(status.p, 0, kStWords * sizeof(unsigned long long), st);
    rc = run_slots(ctx, order.p, st);
  }
  if (rc == RTG_OK) rc = run_refit(ctx, status.p, st);
  if (rc == RTG_OK) rc = read_status(ctx, status.p, h, st);
  if (rc == RTG_OK) rc = build_status(ctx, h);
  if (rc == RTG_OK) rc = take_shape(ctx, h, st);
  if (rc == RTG_OK && wants_wide(ctx)) rc = build_wide(ctx, st);
  if (rc != RTG_OK) cudaStreamSynchronize(st);
  tfree(order, st);
  tfree(status, st);
  return rc;
}

}  // namespace rtg
