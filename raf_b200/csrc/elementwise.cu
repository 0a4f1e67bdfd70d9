// SGD-momentum and Adam update kernels (single pass, HBM-bound: every byte is
// touched once), raf.op.cast / group_cast and fuse_tensor / defuse_tensor.
#include <cmath>
#include <type_traits>

#include "common.h"
#include "symm_dev.cuh"
#include "update_core.cuh"

namespace rafb200 {

// ---- update kernels -----------------------------------------------------------
// Bound: HBM.  One block per kSpanElems elements and no loop: the block scheduler replaces a
// finished block at once, so the SMs stay level, and a block's loads overlap its neighbours'
// stores.  Against 8 resident blocks an SM that stride over the items (the last of 5.3 rounds was
// 27 % full): ResNet-50 SGD, 25,557,032 elements, 87.9 -> 80.8 us, and 77.2 us (6.6 TB/s) with the
// next step's blocks placed and their table rows read while this step's last blocks finish.
// Adam, one tensor of 44,353,792 elements with bf16 gradients: 215 -> 186 us (6.7 TB/s) with AdamOp::vec's
// straight-line arithmetic, 204 us without it (any operand outside its ranges); 194 us as the 292 tensors
// of a shard of GPT-2-medium.
// The minimum of resident blocks is the largest without a spill: six blocks are 40 registers, with
// which Adam spills (16-bit gradients 194 against 186 us; fp32, 16 Mi elements, 81 against 74 us).
constexpr int kSpanUnroll = 2;
constexpr int kSpanElems = kPassElems * kSpanUnroll;           // 2048
constexpr int kSpansPerChunk = kChunkElems / kSpanElems;       // list items cover two spans
template <int NSTATE>
constexpr int kMinBlocks = NSTATE == 1 ? 6 : 5;

template <int NSTATE, typename GT, typename OT, typename Op>
__global__ void __launch_bounds__(kBlockThreads, kMinBlocks<NSTATE>)
    update_list_kernel(const TensorDesc* __restrict__ descs, const Item* __restrict__ items, Op op) {
  Policies pol;
  pol.init();
  grid_dependency_trigger();
  // The tables are written by copies, never by a kernel: they are in place before the kernel in
  // front of this one has started, and may be read while it still runs.
  const Item item = items[blockIdx.x / kSpansPerChunk];
  const TensorDesc d = descs[item.tensor_phase & kTensorMask];
  grid_dependency_wait();
  const int64_t start = (int64_t)item.chunk * kChunkElems + (blockIdx.x % kSpansPerChunk) * kSpanElems;
  const int64_t left = d.numel - start;
  if (left <= 0) return;
  update_span<NSTATE, GT, OT, kSpanUnroll>(d, start, left < kSpanElems ? (int)left : kSpanElems, op, pol);
}

// The same update with the collectives inside (n > 1, symmetric memory; no counterpart in the
// reference): the gradient is the sum over ranks of the chunk, read through the multicast
// address or peer by peer at TensorDesc's symmetric offset (kept in first_chunk / nchunks) and
// also written to the rank's local gradient block; the model-dtype copy goes into every rank's
// parameter buffer.  The symmetric layout is 16-byte aligned and zero-padded per row block.
// Bound: the latency of the loads over the links, so resident blocks count: 80 registers for Adam, three
// blocks an SM (AdamOp::vec left alone takes 96 and two blocks); SGD has 48 without a bound.  Buffers of
// two / three "ranks" on one GPU, 44,353,792 elements, bf16: 312 / 369 us, with two blocks 354 / 431 us.
// Passes in flight per thread: four were measured slower (128 registers, half the resident blocks).
constexpr int kFusedUnroll = 2;
template <int NSTATE, typename GT, typename OT, typename Op>
__global__ void __launch_bounds__(kBlockThreads, NSTATE == 2 ? 3 : 0)
    update_list_fused_kernel(const TensorDesc* __restrict__ descs, const Item* __restrict__ items,
                             uint32_t nitems, Op op, LansFuse fu) {
  constexpr int kDT = sizeof(GT) == 4 ? RAFB200_F32 : (std::is_same<GT, __half>::value ? RAFB200_F16 : RAFB200_BF16);
  Policies pol;
  pol.init();
  const int tid = threadIdx.x;
  for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x) {
    const Item item = items[it];
    const TensorDesc d = descs[item.tensor_phase & kTensorMask];
    const ChunkView c = chunk_view(d, item.chunk, sizeof(GT), sizeof(OT));
    const size_t sym = ((((size_t)d.nchunks) << 32) | d.first_chunk) + (size_t)item.chunk * kChunkElems * sizeof(GT);
    GT* gred = const_cast<GT*>(static_cast<const GT*>(c.g));
    OT* out = static_cast<OT*>(c.out);
    const int len4 = c.len & ~(kVec - 1);
    for (int base = 0; base < len4; base += kFusedUnroll * kPassElems) {
      F4 rg[kFusedUnroll], rp[kFusedUnroll], rm[kFusedUnroll], rv[kFusedUnroll];
      uint32_t bits[kFusedUnroll][4];
#pragma unroll
      for (int u = 0; u < kFusedUnroll; ++u) {
        const int e = base + u * kPassElems + tid * kVec;
        if (sizeof(GT) == 2) {
          // 16-bit gradients: a pair of lanes shares one 16-byte access (eight elements); the even
          // lane makes it - the row block's zero padding covers a missing partner - and hands the
          // upper half over.  Every lane of the warp takes part in the exchange.
          uint4 raw = make_uint4(0, 0, 0, 0);
          if ((tid & 1) == 0 && e < len4) {
            const size_t off = sym + (size_t)e * sizeof(GT);
            if (fu.g_mc) {
              raw = mc_ld_reduce<kDT>(fu.g_mc + off);
            } else {
              float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
              for (int q = 0; q < fu.world; ++q) accumulate<kDT>(acc, peer_ld(fu.g_peer[q] + off));
              raw = round_once<kDT>(acc);
            }
          }
          const uint32_t hi0 = __shfl_sync(0xffffffffu, raw.z, (tid & 31) & ~1);
          const uint32_t hi1 = __shfl_sync(0xffffffffu, raw.w, (tid & 31) & ~1);
          bits[u][0] = (tid & 1) ? hi0 : raw.x;
          bits[u][1] = (tid & 1) ? hi1 : raw.y;
          bits[u][2] = bits[u][3] = 0;
          float f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
          accumulate<kDT>(f, make_uint4(bits[u][0], bits[u][1], 0u, 0u));
#pragma unroll
          for (int j = 0; j < 4; ++j) rg[u].x[j] = f[j];
        }
        if (e < len4) {
          if (sizeof(GT) == 4)
            reduced4<kDT>(fu.g_mc, fu.g_peer, fu.world, sym + (size_t)e * sizeof(GT), rg[u].x, bits[u]);
          rp[u] = Elem<float>::template load4<kStream>(c.p + e, pol);
          rm[u] = Elem<float>::template load4<kStream>(c.m + e, pol);
          if (NSTATE == 2) rv[u] = Elem<float>::template load4<kStream>(c.v + e, pol);
          else rv[u] = f4_zero();
        }
      }
#pragma unroll
      for (int u = 0; u < kFusedUnroll; ++u) {
        const int e = base + u * kPassElems + tid * kVec;
        if (e < len4) {
          if (sizeof(GT) == 4) *reinterpret_cast<uint4*>(gred + e) = make_uint4(bits[u][0], bits[u][1], bits[u][2], bits[u][3]);
          else *reinterpret_cast<uint2*>(gred + e) = make_uint2(bits[u][0], bits[u][1]);
          op.vec(rg[u], rp[u], rm[u], rv[u]);
          Elem<float>::template store4<kDefault>(c.p + e, rp[u], pol);
          Elem<float>::template store4<kDefault>(c.m + e, rm[u], pol);
          if (NSTATE == 2) Elem<float>::template store4<kDefault>(c.v + e, rv[u], pol);
          if (out) {
            if (fu.fuse_ag) store4_everywhere<OT>(fu.p_mc, fu.p_peer, fu.world, fu.rank, out + e, rp[u]);
            else Elem<OT>::template store4<kDefault>(out + e, rp[u], pol);
          }
        }
      }
    }
    // the last one to three elements of a tensor: element by element, peer by peer
    for (int e = len4 + tid; e < c.len; e += kBlockThreads) {
      float acc = 0.f;
      for (int q = 0; q < fu.world; ++q)
        acc += Elem<GT>::to_f32(*reinterpret_cast<const volatile GT*>(fu.g_peer[q] + sym + (size_t)e * sizeof(GT)));
      const GT rounded = Elem<GT>::from_f32(acc);
      gred[e] = rounded;
      float gg = Elem<GT>::to_f32(rounded);
      float pp = c.p[e], mm = c.m[e], vv = NSTATE == 2 ? c.v[e] : 0.f;
      op(gg, pp, mm, vv);
      c.p[e] = pp;
      c.m[e] = mm;
      if (NSTATE == 2) c.v[e] = vv;
      if (out) {
        if (fu.fuse_ag) store1_everywhere<OT>(fu.p_peer, fu.world, fu.rank, out + e, pp);
        else out[e] = Elem<OT>::from_f32(pp);
      }
    }
  }
}

// One tensor described by value.
template <int NSTATE, typename GT, typename OT, typename Op>
__global__ void __launch_bounds__(kBlockThreads, kMinBlocks<NSTATE>)
    update_flat_kernel(TensorDesc d, Op op) {
  Policies pol;
  pol.init();
  grid_dependency_trigger();
  grid_dependency_wait();
  const int64_t start = (int64_t)blockIdx.x * kSpanElems;
  const int64_t left = d.numel - start;
  update_span<NSTATE, GT, OT, kSpanUnroll>(d, start, left < kSpanElems ? (int)left : kSpanElems, op, pol);
}

// SGD from (x, dx, v) to (x1, v1): the operator's own form, which leaves its inputs alone.
// One pass over 20 bytes an element instead of two clones and an in-place update (36 bytes,
// three launches); in place when x1 == x and v1 == v.
template <typename GT>
__global__ void __launch_bounds__(kBlockThreads)
    sgd_to_kernel(const GT* g, const float* x, const float* v, float* x1, float* v1, int64_t n, bool aligned,
                  SgdOp op) {
  Policies pol;
  pol.init();
  grid_dependency_trigger();
  grid_dependency_wait();
  const int64_t start = (int64_t)blockIdx.x * kPassElems + threadIdx.x * kVec;
  if (aligned && start + kVec <= n) {
    const F4 gg = Elem<GT>::template load4<kStream>(g + start, pol);
    F4 pp = Elem<float>::template load4<kStream>(x + start, pol);
    F4 mm = Elem<float>::template load4<kStream>(v + start, pol), unused = f4_zero();
    op.vec(gg, pp, mm, unused);
    Elem<float>::template store4<kDefault>(x1 + start, pp, pol);
    Elem<float>::template store4<kDefault>(v1 + start, mm, pol);
    return;
  }
#pragma unroll
  for (int j = 0; j < kVec; ++j) {
    const int64_t e = start + j;
    if (e >= n) return;
    float pp = x[e], mm = v[e], unused = 0.f;
    op(Elem<GT>::to_f32(g[e]), pp, mm, unused);
    x1[e] = pp;
    v1[e] = mm;
  }
}

// Tensors described by value, for callers without a tensor list: what an eager loop updates in
// one launch.  `end` counts spans: block b works on the tensor with end[i - 1] <= b < end[i].
template <int CAP>
struct Rows {
  const void* g[CAP];
  float* p[CAP];
  float* m[CAP];
  uint32_t end[CAP];
  uint32_t numel[CAP];  // below 2^31; the top bit set = vector accesses allowed
};
constexpr int kMaxRows = 512;  // 16 KB of the 32 KB a launch's parameters may take

template <typename GT, int CAP>
__global__ void __launch_bounds__(kBlockThreads, kMinBlocks<1>)
    sgd_rows_kernel(const __grid_constant__ Rows<CAP> rows, int k, SgdOp op) {
  Policies pol;
  pol.init();
  grid_dependency_trigger();
  int lo = 0, hi = k - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (blockIdx.x < rows.end[mid]) hi = mid;
    else lo = mid + 1;
  }
  TensorDesc d{};
  d.g = rows.g[lo];
  d.p = rows.p[lo];
  d.m = rows.m[lo];
  d.flags = (rows.numel[lo] >> 31) ? kFlagAligned : 0u;
  const int64_t n = rows.numel[lo] & 0x7fffffffu;
  const int64_t start = (int64_t)(blockIdx.x - (lo ? rows.end[lo - 1] : 0u)) * kSpanElems;
  grid_dependency_wait();
  update_span<1, GT, float, kSpanUnroll>(d, start, n - start < kSpanElems ? (int)(n - start) : kSpanElems, op, pol);
}

static int grid_for(uint32_t nitems, int device) {
  static int sm_count[64] = {0};
  if (device < 0 || device >= 64) device = 0;
  if (sm_count[device] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0)
      n = 148;
    sm_count[device] = n;
  }
  // 8 resident blocks of 256 threads per SM; a multiple of the SM count.
  uint32_t cap = (uint32_t)sm_count[device] * 8u;
  return (int)(nitems < cap ? (nitems ? nitems : 1) : cap);
}

// Items [first, first + n) of the list, all of them unless the caller cuts the list into groups.
template <int NSTATE, typename Op, typename GT>
static int launch_list_out(const rafb200_tensor_list_s* l, const Op& op, uint32_t first, uint32_t n, cudaStream_t s) {
  if (l->fuse.fuse_rs) {
    const int grid = grid_for(l->n_items, l->device);
    switch (l->out_dtype) {
      case RAFB200_F32:
        update_list_fused_kernel<NSTATE, GT, float><<<grid, kBlockThreads, 0, s>>>(l->dev_desc, l->dev_items, l->n_items, op, l->fuse);
        break;
      case RAFB200_F16:
        update_list_fused_kernel<NSTATE, GT, __half><<<grid, kBlockThreads, 0, s>>>(l->dev_desc, l->dev_items, l->n_items, op, l->fuse);
        break;
      default:
        update_list_fused_kernel<NSTATE, GT, __nv_bfloat16><<<grid, kBlockThreads, 0, s>>>(l->dev_desc, l->dev_items, l->n_items, op, l->fuse);
        break;
    }
    RAFB200_CUDA(cudaGetLastError());
    return RAFB200_OK;
  }
  const unsigned blocks = n * kSpansPerChunk;
  const Item* items = l->dev_items + first;
  switch (l->out_dtype) {
    case RAFB200_F32:
      RAFB200_CUDA(launch_dependent(update_list_kernel<NSTATE, GT, float, Op>, blocks, kBlockThreads, 0, s, l->dev_desc, items, op));
      break;
    case RAFB200_F16:
      RAFB200_CUDA(launch_dependent(update_list_kernel<NSTATE, GT, __half, Op>, blocks, kBlockThreads, 0, s, l->dev_desc, items, op));
      break;
    default:
      RAFB200_CUDA(launch_dependent(update_list_kernel<NSTATE, GT, __nv_bfloat16, Op>, blocks, kBlockThreads, 0, s, l->dev_desc, items, op));
      break;
  }
  return RAFB200_OK;
}

template <int NSTATE, typename Op>
static int launch_list(const rafb200_tensor_list_s* l, const Op& op, uint32_t first, uint32_t n, cudaStream_t s) {
  if (n == 0) return RAFB200_OK;
  switch (l->g_dtype) {
    case RAFB200_F32: return launch_list_out<NSTATE, Op, float>(l, op, first, n, s);
    case RAFB200_F16: return launch_list_out<NSTATE, Op, __half>(l, op, first, n, s);
    default: return launch_list_out<NSTATE, Op, __nv_bfloat16>(l, op, first, n, s);
  }
}

template <typename GT>
static int launch_flat_sgd_out(const TensorDesc& d, int out_dtype, const SgdOp& op, cudaStream_t s) {
  const unsigned grid = (unsigned)((d.numel + kSpanElems - 1) / kSpanElems);
  switch (out_dtype) {
    case RAFB200_F32:
      RAFB200_CUDA(launch_dependent(update_flat_kernel<1, GT, float, SgdOp>, grid, kBlockThreads, 0, s, d, op));
      break;
    case RAFB200_F16:
      RAFB200_CUDA(launch_dependent(update_flat_kernel<1, GT, __half, SgdOp>, grid, kBlockThreads, 0, s, d, op));
      break;
    default:
      RAFB200_CUDA(launch_dependent(update_flat_kernel<1, GT, __nv_bfloat16, SgdOp>, grid, kBlockThreads, 0, s, d, op));
      break;
  }
  return RAFB200_OK;
}

bool pointers_aligned(const void* g, int g_dtype, const void* p, const void* m, const void* v,
                      const void* out, int out_dtype) {
  auto ok = [](const void* ptr, int bytes) { return (reinterpret_cast<uintptr_t>(ptr) % bytes) == 0; };
  bool a = ok(g, g_dtype == RAFB200_F32 ? 16 : 8) && ok(p, 16) && ok(m, 16);
  if (v) a = a && ok(v, 16);
  if (out) a = a && ok(out, out_dtype == RAFB200_F32 ? 16 : 8);
  return a;
}

template <typename GT>
static int launch_sgd_to(const float* x, const void* dx, const float* v, float* x1, float* v1, int64_t n, bool aligned,
                         const SgdOp& op, cudaStream_t s) {
  const unsigned grid = (unsigned)((n + kPassElems - 1) / kPassElems);
  RAFB200_CUDA(launch_dependent(sgd_to_kernel<GT>, grid, kBlockThreads, 0, s, static_cast<const GT*>(dx), x, v, x1, v1, n,
                                aligned, op));
  return RAFB200_OK;
}

// One launch over k >= 1 tensors, none empty, at most CAP of them.
template <typename GT, int CAP>
static int launch_sgd_rows(int k, float* const* x, const void* const* dx, int dx_dtype, float* const* v,
                           const int64_t* numel, const SgdOp& op, cudaStream_t s) {
  Rows<CAP> rows;
  uint64_t end = 0;
  for (int i = 0; i < k; ++i) {
    rows.g[i] = dx[i];
    rows.p[i] = x[i];
    rows.m[i] = v[i];
    end += (uint64_t)((numel[i] + kSpanElems - 1) / kSpanElems);
    rows.end[i] = (uint32_t)end;
    rows.numel[i] = (uint32_t)numel[i] |
                    (pointers_aligned(dx[i], dx_dtype, x[i], v[i], nullptr, nullptr, RAFB200_F32) ? 0x80000000u : 0u);
  }
  RAFB200_CUDA(launch_dependent(sgd_rows_kernel<GT, CAP>, (unsigned)end, kBlockThreads, 0, s, rows, k, op));
  return RAFB200_OK;
}

// The parameter block of a launch is copied whole: the smaller table where it is enough.
template <typename GT>
static int launch_sgd_many(int k, float* const* x, const void* const* dx, int dx_dtype, float* const* v,
                           const int64_t* numel, const SgdOp& op, cudaStream_t s) {
  if (k <= 64) return launch_sgd_rows<GT, 64>(k, x, dx, dx_dtype, v, numel, op, s);
  return launch_sgd_rows<GT, kMaxRows>(k, x, dx, dx_dtype, v, numel, op, s);
}

// Bias corrections exactly as the reference's host code computes them
// (src/op/dialect/cuda/lans.cc:100-105: float base, int exponent -> double pow).
void bias_corrections(float beta1, float beta2, int step, int bias_correction, float* bc1,
                      float* bc2) {
  *bc1 = 1.0f;
  *bc2 = 1.0f;
  if (bias_correction == 1) {
    *bc1 = static_cast<float>(1 - std::pow(static_cast<double>(beta1), static_cast<double>(step)));
    *bc2 = static_cast<float>(1 - std::pow(static_cast<double>(beta2), static_cast<double>(step)));
  }
}

// ---- cast ----------------------------------------------------------------------
template <typename ST, typename DT>
__global__ void __launch_bounds__(kBlockThreads)
    cast_kernel(const ST* __restrict__ src, DT* __restrict__ dst, int64_t n, bool aligned) {
  Policies pol;
  pol.init();
  const int64_t n4 = aligned ? (n & ~(int64_t)3) : 0;
  for (int64_t e = ((int64_t)blockIdx.x * kBlockThreads + threadIdx.x) * 4; e < n4;
       e += (int64_t)gridDim.x * kBlockThreads * 4) {
    F4 v = Elem<ST>::template load4<kStream>(src + e, pol);
    Elem<DT>::template store4<kDefault>(dst + e, v, pol);
  }
  for (int64_t e = n4 + (int64_t)blockIdx.x * kBlockThreads + threadIdx.x; e < n;
       e += (int64_t)gridDim.x * kBlockThreads)
    dst[e] = Elem<DT>::from_f32(Elem<ST>::to_f32(src[e]));
}

template <typename ST>
static int launch_cast_dst(const void* src, void* dst, int dst_dtype, int64_t n, bool aligned,
                           int grid, cudaStream_t s) {
  switch (dst_dtype) {
    case RAFB200_F32:
      cast_kernel<ST, float><<<grid, kBlockThreads, 0, s>>>((const ST*)src, (float*)dst, n, aligned);
      break;
    case RAFB200_F16:
      cast_kernel<ST, __half><<<grid, kBlockThreads, 0, s>>>((const ST*)src, (__half*)dst, n, aligned);
      break;
    default:
      cast_kernel<ST, __nv_bfloat16><<<grid, kBlockThreads, 0, s>>>((const ST*)src, (__nv_bfloat16*)dst, n, aligned);
      break;
  }
  RAFB200_CUDA(cudaGetLastError());
  return RAFB200_OK;
}

static int cast_impl(const void* src, int src_dtype, void* dst, int dst_dtype, int64_t n,
                     cudaStream_t s) {
  if (n == 0) return RAFB200_OK;
  int device = 0;
  cudaGetDevice(&device);
  auto ok = [](const void* ptr, int dt) {
    return (reinterpret_cast<uintptr_t>(ptr) % (dt == RAFB200_F32 ? 16 : 8)) == 0;
  };
  const bool aligned = ok(src, src_dtype) && ok(dst, dst_dtype);
  const int64_t per_block = (int64_t)kBlockThreads * 4;
  const int64_t blocks = (n + per_block - 1) / per_block;
  const int grid = grid_for((uint32_t)(blocks > (1 << 30) ? (1 << 30) : blocks), device);
  switch (src_dtype) {
    case RAFB200_F32: return launch_cast_dst<float>(src, dst, dst_dtype, n, aligned, grid, s);
    case RAFB200_F16: return launch_cast_dst<__half>(src, dst, dst_dtype, n, aligned, grid, s);
    default: return launch_cast_dst<__nv_bfloat16>(src, dst, dst_dtype, n, aligned, grid, s);
  }
}

// ---- batched movers (group_cast, fuse_tensor, defuse_tensor) ------------------------
// Bound: HBM, and for a bucket of small tensors the launch.  The tensors travel in the launch
// parameters; one block per span of one tensor, found by bisection over the running span counts
// (a grid as wide as the largest tensor for every tensor left most blocks of a ragged list empty).
template <int CAP>
struct CopyRows {
  const void* src[CAP];
  void* dst[CAP];
  int64_t count[CAP];  // elements of a cast, bytes of a copy
  uint32_t end[CAP];   // spans of tensors 0 .. i
};
constexpr int kFewRows = 64;  // launches with no more tensors pass the smaller table

template <int CAP>
__device__ __forceinline__ int row_of(const CopyRows<CAP>& r, int k) {
  int lo = 0, hi = k - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (blockIdx.x < r.end[mid]) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

constexpr int kCastUnroll = 4;
constexpr int kCastSpan = kPassElems * kCastUnroll;  // elements per block
template <typename ST, typename DT, int CAP>
__global__ void __launch_bounds__(kBlockThreads) group_cast_kernel(const __grid_constant__ CopyRows<CAP> rows, int k) {
  Policies pol;
  pol.init();
  grid_dependency_trigger();
  const int t = row_of(rows, k);
  const int64_t start = (int64_t)(blockIdx.x - (t ? rows.end[t - 1] : 0u)) * kCastSpan;
  const ST* src = static_cast<const ST*>(rows.src[t]) + start;
  DT* dst = static_cast<DT*>(rows.dst[t]) + start;
  const int64_t left = rows.count[t] - start;
  const int len = left < kCastSpan ? (int)left : kCastSpan;
  const bool aligned = (reinterpret_cast<uintptr_t>(src) % (sizeof(ST) * 4) == 0) &&
                       (reinterpret_cast<uintptr_t>(dst) % (sizeof(DT) * 4) == 0);
  const int len4 = aligned ? (len & ~3) : 0;
  grid_dependency_wait();
  F4 v[kCastUnroll];
#pragma unroll
  for (int u = 0; u < kCastUnroll; ++u) {
    const int e = u * kPassElems + threadIdx.x * kVec;
    if (e < len4) v[u] = Elem<ST>::template load4<kStream>(src + e, pol);
  }
#pragma unroll
  for (int u = 0; u < kCastUnroll; ++u) {
    const int e = u * kPassElems + threadIdx.x * kVec;
    if (e < len4) Elem<DT>::template store4<kDefault>(dst + e, v[u], pol);
  }
  for (int e = len4 + threadIdx.x; e < len; e += kBlockThreads) dst[e] = Elem<DT>::from_f32(Elem<ST>::to_f32(src[e]));
}

// 16 bytes that start `sh` bytes (1 .. 15) into the two aligned words a, b.
__device__ __forceinline__ uint4 shifted(uint4 a, uint4 b, int sh) {
  const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  const int r = (sh & 3) * 8;
  uint4 o;
#define RAFB200_SHIFTED(Q)                       \
  case Q:                                        \
    o.x = __funnelshift_r(w[Q], w[Q + 1], r);     \
    o.y = __funnelshift_r(w[Q + 1], w[Q + 2], r); \
    o.z = __funnelshift_r(w[Q + 2], w[Q + 3], r); \
    o.w = __funnelshift_r(w[Q + 3], w[Q < 3 ? Q + 4 : 7], r); \
    break;
  switch (sh >> 2) {
    RAFB200_SHIFTED(0)
    RAFB200_SHIFTED(1)
    RAFB200_SHIFTED(2)
    default:
      RAFB200_SHIFTED(3)
  }
#undef RAFB200_SHIFTED
  return o;
}

// Byte copies.  Where source and destination lie differently to 16 bytes (a tensor of odd size
// in front of this one in the flat buffer), the destination is still written in aligned 16-byte
// words: each is cut out of the two aligned source words it spans.  Words of which a source half
// would lie outside the tensor, and the bytes before the first and after the last word, go
// byte by byte.  48 ragged fp32 tensors, 13.5 MB, packed and unpacked through the operators: 222.5 -> 46.8 us.
constexpr int kCopyUnroll = 2;
constexpr int kCopySpan = kBlockThreads * 16 * kCopyUnroll;  // bytes per block
template <int CAP>
__global__ void __launch_bounds__(kBlockThreads) group_copy_kernel(const __grid_constant__ CopyRows<CAP> rows, int k) {
  Policies pol;
  pol.init();
  grid_dependency_trigger();
  const int t = row_of(rows, k);
  const int64_t start = (int64_t)(blockIdx.x - (t ? rows.end[t - 1] : 0u)) * kCopySpan;
  const char* const row = static_cast<const char*>(rows.src[t]);
  const char* const row_end = row + rows.count[t];
  const int64_t left = rows.count[t] - start;
  const int len = left < kCopySpan ? (int)left : kCopySpan;
  const char* src = row + start;
  char* dst = static_cast<char*>(rows.dst[t]) + start;
  int head = (int)(-reinterpret_cast<intptr_t>(dst) & 15);
  if (head > len) head = len;
  const int nv = (len - head) >> 4;
  const int sh = (int)(reinterpret_cast<uintptr_t>(src + head) & 15);
  grid_dependency_wait();
  uint4 v[kCopyUnroll];
  bool whole[kCopyUnroll];
#pragma unroll
  for (int u = 0; u < kCopyUnroll; ++u) {
    const int i = threadIdx.x + u * kBlockThreads;
    const char* s = src + head + (size_t)i * 16 - sh;
    whole[u] = i < nv && (sh == 0 || (s >= row && s + 32 <= row_end));
    if (whole[u]) v[u] = sh == 0 ? ld16<kStream>(s, pol) : shifted(ld16<kDefault>(s, pol), ld16<kDefault>(s + 16, pol), sh);
  }
#pragma unroll
  for (int u = 0; u < kCopyUnroll; ++u) {
    const int i = threadIdx.x + u * kBlockThreads;
    if (whole[u]) {
      st16<kDefault>(dst + head + (size_t)i * 16, v[u], pol);
    } else if (i < nv) {
      for (int j = 0; j < 16; ++j) dst[head + i * 16 + j] = src[head + i * 16 + j];
    }
  }
  if ((int)threadIdx.x < head) dst[threadIdx.x] = src[threadIdx.x];
  const int tail = head + nv * 16 + threadIdx.x;
  if (tail < len) dst[tail] = src[tail];
}

// Calls `launch(rows, k, spans)` for the tensors in groups that fit a table; empty ones are left out.
template <int CAP, typename Launch>
static int for_each_group(int k, const void* const* src, void* const* dst, const int64_t* numel, int64_t scale, int span,
                          Launch launch) {
  CopyRows<CAP> rows;
  for (int i = 0; i < k; ++i)  // before the first launch: a refused call has done nothing
    RAFB200_REQUIRE(numel[i] >= 0 && (numel[i] == 0 || (src[i] && dst[i])), "tensor %d of %d: NULL or of negative size", i, k);
  int n = 0;
  uint64_t spans = 0;
  for (int i = 0; i < k; ++i) {
    const int64_t count = numel[i] * scale;
    const uint64_t mine = (uint64_t)((count + span - 1) / span);
    if (n == CAP || (n > 0 && spans + mine >= (1ull << 31))) {
      if (int rc = launch(rows, n, (unsigned)spans)) return rc;
      n = 0;
      spans = 0;
    }
    if (count == 0) continue;
    spans += mine;
    rows.src[n] = src[i];
    rows.dst[n] = dst[i];
    rows.count[n] = count;
    rows.end[n++] = (uint32_t)spans;
  }
  return n ? launch(rows, n, (unsigned)spans) : (int)RAFB200_OK;
}

template <typename ST, typename DT, int CAP>
static int group_cast_rows(int k, const void* const* src, void* const* dst, const int64_t* numel, cudaStream_t s) {
  return for_each_group<CAP>(k, src, dst, numel, 1, kCastSpan, [&](const CopyRows<CAP>& r, int n, unsigned spans) {
    RAFB200_CUDA(launch_dependent(group_cast_kernel<ST, DT, CAP>, spans, kBlockThreads, 0, s, r, n));
    return (int)RAFB200_OK;
  });
}

template <typename ST, typename DT>
static int group_cast_any(int k, const void* const* src, void* const* dst, const int64_t* numel, cudaStream_t s) {
  return k <= kFewRows ? group_cast_rows<ST, DT, kFewRows>(k, src, dst, numel, s)
                       : group_cast_rows<ST, DT, kMaxRows>(k, src, dst, numel, s);
}

template <typename ST>
static int group_cast_dst(int k, const void* const* src, void* const* dst, int dst_dtype, const int64_t* numel,
                          cudaStream_t s) {
  switch (dst_dtype) {
    case RAFB200_F32: return group_cast_any<ST, float>(k, src, dst, numel, s);
    case RAFB200_F16: return group_cast_any<ST, __half>(k, src, dst, numel, s);
    default: return group_cast_any<ST, __nv_bfloat16>(k, src, dst, numel, s);
  }
}

template <int CAP>
static int group_copy_rows(int k, const void* const* src, void* const* dst, const int64_t* numel, int elem_size,
                           cudaStream_t s) {
  return for_each_group<CAP>(k, src, dst, numel, elem_size, kCopySpan, [&](const CopyRows<CAP>& r, int n, unsigned spans) {
    RAFB200_CUDA(launch_dependent(group_copy_kernel<CAP>, spans, kBlockThreads, 0, s, r, n));
    return (int)RAFB200_OK;
  });
}

static int group_copy(int k, const void* const* src, void* const* dst, const int64_t* numel, int elem_size,
                      cudaStream_t s) {
  return k <= kFewRows ? group_copy_rows<kFewRows>(k, src, dst, numel, elem_size, s)
                       : group_copy_rows<kMaxRows>(k, src, dst, numel, elem_size, s);
}

int copy_many(int k, const void* const* src, void* const* dst, const int64_t* bytes, cudaStream_t s) {
  return group_copy(k, src, dst, bytes, 1, s);
}

// The list's update on part of its work items (item i = 4096 elements, tensor by tensor).
int sgd_list_items(rafb200_tensor_list_s* list, uint32_t first, uint32_t n, float learning_rate, float mu,
                   float weight_decay, float grad_scale, cudaStream_t s) {
  RAFB200_REQUIRE(list->bound, "rafb200_sgd_list: bind the tensor list first");
  SgdOp op{learning_rate, mu, weight_decay, grad_scale};
  return launch_list<1>(list, op, first, n, s);
}

int adam_list_items(rafb200_tensor_list_s* list, uint32_t first, uint32_t n, int step, float learning_rate,
                    float beta1, float beta2, float eps, int bias_correction, float weight_decay, int mode,
                    float grad_scale, cudaStream_t s) {
  RAFB200_REQUIRE(list->bound && list->has_v, "rafb200_adam: bind g, p, m and v first");
  RAFB200_REQUIRE(step >= 1, "rafb200_adam: step counts from 1");
  AdamOp op;
  op.lr = learning_rate;
  op.beta1 = beta1;
  op.beta2 = beta2;
  op.beta3 = 1 - beta1;
  op.one_minus_beta2 = 1 - beta2;
  op.eps = eps;
  bias_corrections(beta1, beta2, step, bias_correction, &op.bc1, &op.bc2);
  op.wd = weight_decay;
  op.gscale = grad_scale;
  op.mode = mode;
  // the branch-free form of AdamOp::vec: see the ranges there
  op.y1 = 1.0f / op.bc1;
  op.y2 = 1.0f / op.bc2;
  auto within = [](float x, float lo, float hi) { return x >= lo && x <= hi; };
  op.fast = within(op.bc1, 0x1p-20f, 1.0f) && within(op.bc2, 0x1p-20f, 1.0f) && within(eps, 0x1p-40f, 1.0f);
  return launch_list<2>(list, op, first, n, s);
}

}  // namespace rafb200

using namespace rafb200;

extern "C" {

int rafb200_sgd(float* x, const void* dx, int dx_dtype, float* v, int64_t numel,
                float learning_rate, float mu, float weight_decay, float grad_scale, void* out,
                int out_dtype, void* stream) {
  RAFB200_REQUIRE(numel >= 0, "rafb200_sgd: negative numel");
  RAFB200_REQUIRE(dtype_valid(dx_dtype) && dtype_valid(out_dtype), "rafb200_sgd: bad dtype");
  if (numel == 0) return RAFB200_OK;
  RAFB200_REQUIRE(x && dx && v, "rafb200_sgd: x, dx and v must not be NULL");
  RAFB200_REQUIRE((numel + kSpanElems - 1) / kSpanElems < (int64_t)1 << 31,
                  "rafb200_sgd: tensor too large");
  TensorDesc d{};
  d.g = dx;
  d.p = x;
  d.m = v;
  d.v = nullptr;
  d.out = out;
  d.numel = numel;
  d.flags = pointers_aligned(dx, dx_dtype, x, v, nullptr, out, out_dtype) ? kFlagAligned : 0;
  SgdOp op{learning_rate, mu, weight_decay, grad_scale};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dx_dtype) {
    case RAFB200_F32: return launch_flat_sgd_out<float>(d, out_dtype, op, s);
    case RAFB200_F16: return launch_flat_sgd_out<__half>(d, out_dtype, op, s);
    default: return launch_flat_sgd_out<__nv_bfloat16>(d, out_dtype, op, s);
  }
}

int rafb200_sgd_to(const float* x, const void* dx, int dx_dtype, const float* v, float* x1, float* v1, int64_t numel,
                   float learning_rate, float mu, void* stream) {
  RAFB200_REQUIRE(numel >= 0, "rafb200_sgd_to: negative numel");
  RAFB200_REQUIRE(dtype_valid(dx_dtype), "rafb200_sgd_to: bad dtype");
  if (numel == 0) return RAFB200_OK;
  RAFB200_REQUIRE(x && dx && v && x1 && v1, "rafb200_sgd_to: NULL argument");
  RAFB200_REQUIRE((numel + kPassElems - 1) / kPassElems < (int64_t)1 << 31, "rafb200_sgd_to: tensor too large");
  const bool aligned = pointers_aligned(dx, dx_dtype, x, v, x1, v1, RAFB200_F32);
  const SgdOp op{learning_rate, mu, 0.0f, 1.0f};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dx_dtype) {
    case RAFB200_F32: return launch_sgd_to<float>(x, dx, v, x1, v1, numel, aligned, op, s);
    case RAFB200_F16: return launch_sgd_to<__half>(x, dx, v, x1, v1, numel, aligned, op, s);
    default: return launch_sgd_to<__nv_bfloat16>(x, dx, v, x1, v1, numel, aligned, op, s);
  }
}

int rafb200_sgd_many(int k, float* const* x, const void* const* dx, int dx_dtype, float* const* v,
                     const int64_t* numel, float learning_rate, float mu, void* stream) {
  RAFB200_REQUIRE(k >= 0 && (k == 0 || (x && dx && v && numel)), "rafb200_sgd_many: bad arguments");
  RAFB200_REQUIRE(dtype_valid(dx_dtype), "rafb200_sgd_many: bad dtype");
  for (int i = 0; i < k; ++i) {
    RAFB200_REQUIRE(numel[i] >= 0 && numel[i] < (1ll << 31), "rafb200_sgd_many: numel[%d] must be in [0, 2^31)", i);
    RAFB200_REQUIRE(numel[i] == 0 || (x[i] && dx[i] && v[i]), "rafb200_sgd_many: NULL pointer for tensor %d", i);
  }
  const SgdOp op{learning_rate, mu, 0.0f, 1.0f};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  for (int i = 0; i < k;) {
    if (numel[i] == 0) {
      ++i;
      continue;
    }
    int n = 1;  // a run of tensors with elements
    while (i + n < k && n < kMaxRows && numel[i + n] > 0) ++n;
    int rc;
    switch (dx_dtype) {
      case RAFB200_F32: rc = launch_sgd_many<float>(n, x + i, dx + i, dx_dtype, v + i, numel + i, op, s); break;
      case RAFB200_F16: rc = launch_sgd_many<__half>(n, x + i, dx + i, dx_dtype, v + i, numel + i, op, s); break;
      default: rc = launch_sgd_many<__nv_bfloat16>(n, x + i, dx + i, dx_dtype, v + i, numel + i, op, s); break;
    }
    if (rc != RAFB200_OK) return rc;
    i += n;
  }
  return RAFB200_OK;
}

int rafb200_sgd_list(rafb200_tensor_list_t list, float learning_rate, float mu,
                     float weight_decay, float grad_scale, void* stream) {
  RAFB200_REQUIRE(list, "rafb200_sgd_list: NULL list");
  return sgd_list_items(list, 0, list->n_items, learning_rate, mu, weight_decay, grad_scale,
                        static_cast<cudaStream_t>(stream));
}

int rafb200_adam(rafb200_tensor_list_t list, int step, const float* step_dev,
                 float learning_rate, float beta1, float beta2, float eps, int bias_correction,
                 float weight_decay, int mode, float grad_scale, void* stream) {
  RAFB200_REQUIRE(list, "rafb200_adam: NULL list");
  RAFB200_REQUIRE(step_dev == nullptr,
                  "rafb200_adam: a device-resident step is only supported by rafb200_lans");
  return adam_list_items(list, 0, list->n_items, step, learning_rate, beta1, beta2, eps, bias_correction, weight_decay,
                         mode, grad_scale, static_cast<cudaStream_t>(stream));
}

int rafb200_cast(const void* src, int src_dtype, void* dst, int dst_dtype, int64_t numel,
                 void* stream) {
  RAFB200_REQUIRE(dtype_valid(src_dtype) && dtype_valid(dst_dtype), "rafb200_cast: bad dtype");
  RAFB200_REQUIRE(numel >= 0 && (numel == 0 || (src && dst)), "rafb200_cast: bad arguments");
  return cast_impl(src, src_dtype, dst, dst_dtype, numel, static_cast<cudaStream_t>(stream));
}

int rafb200_group_cast(int k, const void* const* src, int src_dtype, void* const* dst,
                       int dst_dtype, const int64_t* numel, void* stream) {
  RAFB200_REQUIRE(k >= 0 && (k == 0 || (src && dst && numel)), "rafb200_group_cast: bad arguments");
  RAFB200_REQUIRE(dtype_valid(src_dtype) && dtype_valid(dst_dtype), "rafb200_group_cast: bad dtype");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (src_dtype) {
    case RAFB200_F32: return group_cast_dst<float>(k, src, dst, dst_dtype, numel, s);
    case RAFB200_F16: return group_cast_dst<__half>(k, src, dst, dst_dtype, numel, s);
    default: return group_cast_dst<__nv_bfloat16>(k, src, dst, dst_dtype, numel, s);
  }
}

int rafb200_fuse_tensor(int k, const void* const* src, const int64_t* numel, const int64_t* offsets,
                        int elem_size, void* flat, void* stream) {
  RAFB200_REQUIRE(k >= 0 && elem_size > 0 && (k == 0 || (src && numel && offsets && flat)),
                  "rafb200_fuse_tensor: bad arguments");
  std::vector<void*> dst(k);
  for (int i = 0; i < k; ++i) dst[i] = static_cast<char*>(flat) + offsets[i] * elem_size;
  return group_copy(k, src, dst.data(), numel, elem_size, static_cast<cudaStream_t>(stream));
}

int rafb200_defuse_tensor(int k, void* const* dst, const int64_t* numel, const int64_t* offsets,
                          int elem_size, const void* flat, void* stream) {
  RAFB200_REQUIRE(k >= 0 && elem_size > 0 && (k == 0 || (dst && numel && offsets && flat)),
                  "rafb200_defuse_tensor: bad arguments");
  std::vector<const void*> src(k);
  for (int i = 0; i < k; ++i) src[i] = static_cast<const char*>(flat) + offsets[i] * elem_size;
  return group_copy(k, src.data(), dst, numel, elem_size, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
