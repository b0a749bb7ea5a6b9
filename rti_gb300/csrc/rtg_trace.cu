// rtg_trace.cu -- launches of the path kernel for one context (forward trace
// and adjoint replays), and the explicit-ray closest-hit kernel.
#include <algorithm>

#include "rtg_path.cuh"

namespace rtg {

namespace {

constexpr int kQueryThreads = 128;

// Closest hits of explicit rays, `share` of them a warp, bound as a trace's
// queries are.  The stack follows the tree's need, and the wide traversal is
// compiled in only where it runs.  Whole calls of 262 144 rays, before -> now: hole of 31 k triangles 479 -> 219 us,
// trench of 98 k discs 488 -> 198, 4.19 M discs 707 -> 379; 1000 rays 106 -> 81.
// 768, 1280 and 1536 threads an SM: 230, 224, 245 us for the hole.
template <int STACK, bool WIDE>
__global__ void __launch_bounds__(kQueryThreads, 1024 / kQueryThreads)
    closest_hit_kernel(const SceneView s, const float* __restrict__ rays, int64_t n, int share, float tnear,
                       int32_t* __restrict__ prim, float* __restrict__ tout, unsigned long long* errors) {
  const int lane = threadIdx.x & 31;
  const int64_t i = ((int64_t)blockIdx.x * (kQueryThreads / 32) + threadIdx.x / 32) * share + lane;
  if (lane >= share || i >= n) return;
  const float* r = rays + 6 * i;
  float t;
  int id;
  uint32_t ref;
  uint32_t e = 0;
  if (closest_hit<STACK, 0, WIDE>(s, mk3(r[0], r[1], r[2]), mk3(r[3], r[4], r[5]), tnear, fmaxf(tnear, 0.0f), t, id,
                                  ref, e)) {
    prim[i] = id;
    tout[i] = t;
  } else {
    prim[i] = -1;
    tout[i] = 0.0f;
  }
  if (e) atomicAdd(errors, (unsigned long long)e);
}

// Ordered launches: a counting sort of the rays by the cell that they start in,
// so that a warp's paths, and those in flight around them, visit the same
// nodes.  A cell is one of 64 x 64 parts of the source rectangle (in Morton order)
// and a quarter turn of the direction, all of them high bits of the source draw.
// The rays are sorted in pieces, one after the other in the order that the launch
// takes them: of more rays a cell holds so many that all paths in flight deposit on
// the same few primitives.  4e8 rays, sorted as one piece -> in pieces of 2^25, one
// launch -> a launch for each piece, which lets the GPU run empty after each:
// directional source on a disc hole 295 -> 221 -> 219 ms, hole of 200 k triangles
// 1256 -> 1280 -> 1362, trench 437 -> 439 -> 442, 4.19 M discs 313 -> 317 -> 317 (in
// ascending order 279, 1295, 444, 413).
constexpr int kCellBits = 6, kTurnBits = 2, kCells = 1 << (2 * kCellBits + kTurnBits);
constexpr uint64_t kOrderPiece = 1u << 25;   // rays sorted at once
constexpr uint64_t kOrderMax = 1u << 29;     // rays of one launch (2 GB of ids)
constexpr uint64_t kOrderKept = 128u << 20;  // bytes that a context keeps for its next ordered launch

__device__ __forceinline__ uint32_t spread_bits(uint32_t v) {  // 6 bits to every second place
  v = (v | v << 4) & 0x0F0Fu;
  v = (v | v << 2) & 0x3333u;
  return (v | v << 1) & 0x5555u;
}
__device__ __forceinline__ uint32_t source_cell(const TraceParams& p, uint32_t j) {
  const uint4 u = draw4(p.seed, p.ray_begin + j, 0xFFFFFFFFu, p.job);
  const uint32_t place = spread_bits(u.x >> (32 - kCellBits)) << 1 | spread_bits(u.y >> (32 - kCellBits));
  return place << kTurnBits | u.z >> (32 - kTurnBits);
}
// One thread per ray of the piece that begins with the launch's ray `first`, bound
// by the atomics on the cells (2e7 rays: 0.12 ms to count, 0.23 ms to place; the
// trace of these takes 13 to 16 ms).
__global__ void order_count_kernel(const __grid_constant__ TraceParams p, uint32_t first, uint32_t n,
                                   uint32_t* __restrict__ cells) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) atomicAdd(&cells[source_cell(p, first + j)], 1u);
}
__global__ void order_place_kernel(const __grid_constant__ TraceParams p, uint32_t first, uint32_t n,
                                   uint32_t* __restrict__ cells, uint32_t* __restrict__ order) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) order[first + atomicAdd(&cells[source_cell(p, first + j)], 1u)] = first + j;
}

template <int TPB>
PathKernel forward_kernel(int stack, bool shared, bool wide) {
  if (stack <= 32) return kernel_for<kModeForward, false, TPB, 32>(shared, wide);
  if (stack <= 64) return kernel_for<kModeForward, false, TPB, 64>(shared, wide);
  return kernel_for<kModeForward, false, TPB, 256>(shared, wide);
}

// The adjoint replays run with 128 threads and a 64- or 256-entry stack.
PathKernel pick_kernel(int mode, int tpb, int stack, bool shared, bool wide, int& tpb_out) {
  if (mode == kModeAdjGlobal) {
    tpb_out = 128;
    if (stack <= 64) return kernel_for<kModeAdjGlobal, false, 128, 64>(shared, wide);
    return wide ? trace_paths_kernel<kModeAdjGlobal, false, 128, 256, false, true>
                : trace_paths_kernel<kModeAdjGlobal, false, 128, 256>;
  }
  if (mode == kModeAdjField) {
    tpb_out = 128;
    if (stack <= 64) return kernel_for<kModeAdjField, false, 128, 64>(shared, wide);
    return wide ? trace_paths_kernel<kModeAdjField, false, 128, 256, false, true>
                : trace_paths_kernel<kModeAdjField, false, 128, 256>;
  }
  if (mode == kModeLogged) {  // a debugging trace: one configuration, both trees
    tpb_out = 128;
    return trace_paths_kernel<kModeLogged, false, 128, 256, false, true>;
  }
  if (mode == kModeWindow) {
    tpb_out = 128;
    if (stack <= 64)
      return wide ? trace_paths_kernel<kModeWindow, false, 128, 64, false, true>
                  : trace_paths_kernel<kModeWindow, false, 128, 64>;
    return wide ? trace_paths_kernel<kModeWindow, false, 128, 256, false, true>
                : trace_paths_kernel<kModeWindow, false, 128, 256>;
  }
  tpb_out = tpb;
  if (tpb == 64) return forward_kernel<64>(stack, shared, wide);
  if (tpb == 256) return forward_kernel<256>(stack, shared, wide);
  tpb_out = 128;
  return forward_kernel<128>(stack, shared, wide);
}

}  // namespace

namespace {

__global__ void s1_fixed_kernel(double* s1, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) reinterpret_cast<long long*>(s1)[i] = __double2ll_rn(s1[i] * 4294967296.0);
}

__global__ void s1_double_kernel(double* s1, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) s1[i] = (double)reinterpret_cast<const long long*>(s1)[i] * (1.0 / 4294967296.0);
}

}  // namespace

int s1_to_fixed(rtg_context* ctx, double* s1, int64_t n, cudaStream_t st) {
  if (n <= 0) return RTG_OK;
  s1_fixed_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(s1, n);
  RTG_CUDA(ctx, cudaGetLastError());
  return RTG_OK;
}

int s1_to_double(rtg_context* ctx, double* s1, int64_t n, cudaStream_t st) {
  if (n <= 0) return RTG_OK;
  s1_double_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(s1, n);
  RTG_CUDA(ctx, cudaGetLastError());
  return RTG_OK;
}

// Whether what the queries of ctx read outgrows the L2 cache: about 96 bytes a disc (a
// third of the four-box nodes can be met, 32 of them; the record; the normal's basis)
// and 128 a triangle, which is what the binary nodes and the records take.
bool outgrows_l2(const rtg_context* ctx) {
  int l2 = 0;
  if (cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, ctx->device) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  const Geometry& g = ctx->g;
  const size_t bytes = g.nodes.n * sizeof(Node) + (g.disc.n + g.tri.n) * sizeof(float4);
  return l2 > 0 && bytes > (size_t)l2;
}

bool shared_stack(rtg_context* ctx, const rtg_launch_config& lc) {
  if (lc.stack_memory == RTG_STACK_SHARED) return true;
  if (lc.stack_memory == RTG_STACK_LOCAL) return false;
  return outgrows_l2(ctx);
}

int stack_for(int requested, int tree_depth) {
  const int need = requested > tree_depth ? requested : tree_depth;
  if (need <= 32) return 32;
  if (need <= 64) return 64;
  return 256;
}

// The paths that each warp holds in a launch of nrays.  A warp's time per
// segment grows with the paths in it, since they part ways: alone a path takes
// a third of what 32 take together.  So a launch that the GPU could hold at
// once is spread over 16 warps an SM before any warp gets more.  Packed warps
// -> 8, 16, 24, 32 warps an SM: 1024 rays into a trench of 1500 discs 266 -> 174,
// 176, 177, 176 us; 16 384 into one of 98 k discs 698 -> 606, 546, 657, 557; 50 000
// onto 4.19 M discs 323 -> 321, 311, 315, 335; from 78 000 rays on (32 paths a
// warp) nothing changes.
int warp_share(uint64_t nrays, int sms) {
  const uint64_t warps = 16 * (uint64_t)sms;
  return (int)std::min<uint64_t>(32, std::max<uint64_t>(1, nrays / warps + (nrays % warps != 0)));
}

uint64_t spread_rays(TraceParams& p, uint64_t nrays, int tpb, int sms) {
  p.lanes = p.plain ? 32 : warp_share(nrays, sms);
  p.packet = std::min(p.packet, p.lanes);
  const uint64_t held = (uint64_t)(tpb / 32) * p.lanes;
  return std::max<uint64_t>(1, nrays / held + (nrays % held != 0));
}

int check_launch_config(rtg_context* ctx, const rtg_launch_config& lc) {
  auto bad = [&](const char* m) { return set_error(ctx, RTG_ERR_INVALID_ARGUMENT, m); };
  if (lc.threads_per_block != 64 && lc.threads_per_block != 128 && lc.threads_per_block != 256)
    return bad("threads_per_block must be 64, 128 or 256");
  if (lc.packet < 1 || lc.packet > 32) return bad("packet must be in 1..32");
  if (lc.stack_depth != 0 && lc.stack_depth != 32 && lc.stack_depth != 64 && lc.stack_depth != 256)
    return bad("stack_depth must be 0, 32, 64 or 256");
  if (lc.scheduling != RTG_SCHED_MEGAKERNEL && lc.scheduling != RTG_SCHED_WAVEFRONT &&
      lc.scheduling != RTG_SCHED_PLAIN)
    return bad("scheduling must be RTG_SCHED_MEGAKERNEL, RTG_SCHED_WAVEFRONT or RTG_SCHED_PLAIN");
  if (lc.leaf_tests != RTG_LEAF_IMMEDIATE && lc.leaf_tests != RTG_LEAF_POSTPONED)
    return bad("leaf_tests must be RTG_LEAF_IMMEDIATE or RTG_LEAF_POSTPONED");
  if (lc.stack_memory != RTG_STACK_AUTO && lc.stack_memory != RTG_STACK_LOCAL && lc.stack_memory != RTG_STACK_SHARED)
    return bad("stack_memory must be RTG_STACK_AUTO, RTG_STACK_LOCAL or RTG_STACK_SHARED");
  return RTG_OK;
}

bool use_wide(const rtg_context* ctx) {
  const Geometry& g = ctx->g;
  return g.wide_current && g.n_wnodes > 0 && g.wide_stack <= 256 && wants_wide(ctx);
}

int traversal_depth(const rtg_context* ctx) {
  return use_wide(ctx) ? ctx->g.wide_stack : ctx->g.quad_stack;
}

SceneView scene_view(rtg_context* ctx) {
  const Geometry& g = ctx->g;
  SceneView s{};
  const bool wide = use_wide(ctx);
  s.wnodes = wide ? g.wnodes.p : nullptr;
  s.n_wnodes = wide ? g.n_wnodes : 0u;
  s.disc = g.disc.p;
  s.nd = (int32_t)g.nd;
  s.tri = g.tri.p;
  s.nt = (int32_t)g.nt;
  s.quads = g.quads.p;
  s.basis = g.basis.p;
  s.root = g.root;
  s.nb_ptr = g.nd > 0 ? g.nb_ptr.p : nullptr;
  s.nb_slot = g.nb_slot.p;
  s.sticking_field = ctx->sticking_field.p;
  // a valid query visits each node at most once (< 2 x primitives)
  const uint64_t automatic = std::min<uint64_t>(4 * (uint64_t)(g.nd + g.nt) + 64, 0xFFFFFFFFull);
  s.max_visits = (uint32_t)(ctx->visit_limit ? std::min<uint64_t>(ctx->visit_limit, automatic) : automatic);
  return s;
}

namespace {

// Whether a launch takes its rays by the cells they start in.  It does where
// paths that start together share memory that others would evict, on a surface
// that outgrows the L2 cache, and where they stay together for long, in a surface
// as deep as it is wide; on a flat surface that the cache holds they only meet in
// their deposits.  Ascending ids -> ordered, launch and sort, in us:
//   4.19 M discs                1e6 rays 1226 -> 1123, 4e6 4279 -> 3515, 1.6e7 16540 -> 12998
//   their field adjoint         5e6 rays 5940 -> 4840
//   directional, disc hole      1e6 rays 995 -> 907, 2e6 1624 -> 1412, 4e6 3031 -> 2405, 1.6e7 11329 -> 8668
//   trench                      1e6 rays 2048 -> 2070, 2e6 3215 -> 3239, 4e6 5600 -> 5415, 1.6e7 19640 -> 19140
//   hole, 200 k triangles       1e6 rays the same, 4e6 23200 -> 22830, 1.6e7 63170 -> 61080
//   flat, 262 k discs           1e6 rays 790 -> 818, 4e6 2708 -> 2789, 1.6e7 10979 -> 11284: not ordered
// (up to 4e8 rays: at kOrderPiece)
bool wants_order(const rtg_context* ctx, const TraceParams& p, uint64_t nrays) {
  if (nrays < 1u << 20) return false;
  if (outgrows_l2(ctx)) return true;
  const float wide = std::max(p.box_hi[0] - p.box_lo[0], p.box_hi[1] - p.box_lo[1]);
  return nrays >= 1u << 21 && p.box_hi[2] - p.box_lo[2] >= wide;
}

// The size of equal parts of n, as few as keep each within most.
uint64_t equal_parts(uint64_t n, uint64_t most) {
  const uint64_t parts = n / most + (n % most != 0);
  return n / parts + (n % parts != 0);
}

// A capture of another stream has no part in the pool, so it may go on meanwhile:
// the calls are made with this thread's capture mode relaxed.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  RelaxedCapture(const RelaxedCapture&) = delete;
  RelaxedCapture& operator=(const RelaxedCapture&) = delete;
};

// The cells and the ids of an ordered launch, taken from the context's pool and
// given back to it in the order of the stream, so that the call only enqueues: a
// buffer of cudaMalloc made a larger launch than before wait for the one before it,
// and broke a capture that another stream had open in the global mode.  The pool
// keeps kOrderKept bytes between launches (mapping 80 MB anew takes 0.3 ms of the
// 16 ms of 2e7 rays onto 4.19 M discs, 12 MB 0.18 ms of the 2 of 3e6) and gives
// them up in release_kept.
struct OrderRoom {
  uint32_t* p = nullptr;
  cudaStream_t st;
  explicit OrderRoom(cudaStream_t s) : st(s) {}
  ~OrderRoom() {
    if (!p) return;
    const RelaxedCapture relaxed;
    cudaFreeAsync(p, st);
  }
  OrderRoom(const OrderRoom&) = delete;
  OrderRoom& operator=(const OrderRoom&) = delete;

  // Whether there is room.  Without it, or while the stream is being captured (a
  // graph would hold the room for as long as it lives), the launch takes its rays in
  // ascending order.
  bool take(rtg_context* ctx, uint64_t rays) {
    const RelaxedCapture relaxed;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone &&
        !injected_alloc_failure(ctx) && make_pool(ctx) &&
        cudaMallocFromPoolAsync((void**)&p, (kCells + (size_t)rays) * sizeof(uint32_t), ctx->order_pool, st) == cudaSuccess)
      return true;
    cudaGetLastError();
    p = nullptr;
    return false;
  }

 private:
  static bool make_pool(rtg_context* ctx) {
    if (ctx->order_pool) return true;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = ctx->device;
    if (cudaMemPoolCreate(&ctx->order_pool, &props) != cudaSuccess) {
      ctx->order_pool = nullptr;
      return false;
    }
    uint64_t keep = kOrderKept;
    int off = 0;  // a trace and a replay on two streams do not wait for each other's room
    cudaMemPoolSetAttribute(ctx->order_pool, cudaMemPoolAttrReleaseThreshold, &keep);
    cudaMemPoolSetAttribute(ctx->order_pool, cudaMemPoolReuseAllowInternalDependencies, &off);
    return true;
  }
};

}  // namespace

int launch_trace(rtg_context* ctx, const TraceParams& p_in, cudaStream_t st, int mode) {
  const rtg_launch_config& lc = ctx->lc;
  TraceParams p = p_in;
  p.packet = lc.packet;
  const uint64_t nrays = p.ray_end - p.ray_begin;
  // the window deposit has a kernel of its own (megakernel or plain schedule),
  // so has a trace that fills the segment log
  if (mode == kModeForward && p.window) mode = kModeWindow;
  if (mode == kModeForward && p.log.rec) mode = kModeLogged;
  // the window's interval queries visit the quads, whichever tree the closest hits use
  const int need = mode == kModeWindow ? std::max(ctx->g.quad_stack, traversal_depth(ctx)) : traversal_depth(ctx);
  const int stack = stack_for(lc.stack_depth, need);
  if (mode == kModeForward && lc.scheduling == RTG_SCHED_WAVEFRONT) {
    // a job table of one entry
    Wavefront& wf = ctx->wf;
    RTG_TRY(dalloc(ctx, wf.one_job, 1, "wavefront job"));
    RTG_TRY(dalloc(ctx, wf.one_prefix, 2, "wavefront prefix"));
    const uint64_t pre[2] = {0, nrays};
    RTG_CUDA(ctx, cudaMemcpyAsync(wf.one_job.p, &p, sizeof p, cudaMemcpyHostToDevice, st));
    RTG_CUDA(ctx, cudaMemcpyAsync(wf.one_prefix.p, pre, sizeof pre, cudaMemcpyHostToDevice, st));
    RTG_CUDA(ctx, cudaStreamSynchronize(st));  // the host copies above are locals
    return launch_wavefront(ctx, p, wf.one_job.p, wf.one_prefix.p, 1, nrays, st, lc, traversal_depth(ctx));
  }
  int tpb = 128, sms = 0, per_sm = 0;
  PathKernel kern = pick_kernel(mode, lc.threads_per_block, stack, shared_stack(ctx, lc), p.s.wnodes != nullptr, tpb);
  p.plain = (mode == kModeForward || mode == kModeWindow) && lc.scheduling == RTG_SCHED_PLAIN ? 1 : 0;
  RTG_CUDA(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
  RTG_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, tpb, 0));
  if (per_sm < 1) per_sm = 1;
  // one launch, or several of more ordered rays than a launch may have
  uint64_t chunk = nrays;
  OrderRoom room(st);
  // the context's own traces and replays only: two batches that share a scene's context may launch from two threads,
  // and must not both make its pool
  const bool own = p.tally == ctx->d_tally || p.tally == ctx->d_tally_adj;
  bool ordered = own && mode != kModeLogged && wants_order(ctx, p, nrays);
  if (ordered) {
    chunk = equal_parts(nrays, kOrderMax);
    ordered = room.take(ctx, chunk);
    if (!ordered) chunk = nrays;
  }
  const uint64_t end = p.ray_end;
  for (uint64_t begin = p.ray_begin; begin < end;) {
    const uint64_t n = std::min(chunk, end - begin);  // begin + chunk may pass 2^64
    p.ray_begin = begin;
    p.ray_end = begin + n;
    if (ordered) {
      uint32_t *cells = room.p, *order = room.p + kCells;
      p.order = order;
      const uint64_t piece = equal_parts(n, kOrderPiece);
      for (uint64_t first = 0; first < n; first += piece) {
        const uint32_t m = (uint32_t)std::min(piece, n - first);
        const unsigned grid = (m + 255) / 256;
        RTG_CUDA(ctx, cudaMemsetAsync(cells, 0, kCells * sizeof(uint32_t), st));
        order_count_kernel<<<grid, 256, 0, st>>>(p, (uint32_t)first, m, cells);
        RTG_TRY(exclusive_scan_u32(ctx, cells, kCells, nullptr, st));
        order_place_kernel<<<grid, 256, 0, st>>>(p, (uint32_t)first, m, cells, order);
      }
    }
    if (begin != p_in.ray_begin)
      RTG_CUDA(ctx, cudaMemsetAsync(&p.tally->next_ray, 0, sizeof(unsigned long long), st));
    uint64_t blocks = (uint64_t)sms * per_sm;
    const uint64_t full = spread_rays(p, n, tpb, sms);
    if (full < blocks || p.plain) blocks = full;
    if (blocks > 0x7FFFFFFFull) return set_error(ctx, RTG_ERR_INVALID_ARGUMENT, "too many rays for a plain launch");
    kern<<<(unsigned)blocks, tpb, 0, st>>>(p, nullptr, nullptr, 0);
    RTG_CUDA(ctx, cudaGetLastError());
    begin += n;
  }
  return RTG_OK;
}

int launch_closest_hit(rtg_context* ctx, const float* d_rays, int64_t n, float tnear, int32_t* d_prim, float* d_t,
                       unsigned long long* d_errors, cudaStream_t st) {
  if (n <= 0) return RTG_OK;
  const SceneView s = scene_view(ctx);
  const int stack = stack_for(0, traversal_depth(ctx));
  int sms = 0;
  RTG_CUDA(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
  const int share = warp_share((uint64_t)n, sms);
  const int64_t held = (int64_t)(kQueryThreads / 32) * share, blocks = (n + held - 1) / held;
  if (blocks > 0x7FFFFFFFll) return set_error(ctx, RTG_ERR_INVALID_ARGUMENT, "too many rays for one launch");
  auto kern = s.wnodes ? closest_hit_kernel<256, true>
              : stack <= 32 ? closest_hit_kernel<32, false>
              : stack <= 64 ? closest_hit_kernel<64, false>
                            : closest_hit_kernel<256, false>;
  kern<<<(unsigned)blocks, kQueryThreads, 0, st>>>(s, d_rays, n, share, tnear, d_prim, d_t, d_errors);
  RTG_CUDA(ctx, cudaGetLastError());
  return RTG_OK;
}

}  // namespace rtg
