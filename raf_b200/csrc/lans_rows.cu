// raf.op.lans for callers that come without a tensor list: the eager operator, which is given its
// tensors anew on every call (src/op/dialect/cuda/lans.cc:25-165, python/raf/optim/lans.py:87-99).
//
// The persistent kernel of lans.cu wants a schedule in device memory: four allocations, three blocking
// copies and a synchronisation to read its error word made a call on a network of 2,477 elements
// cost 1.0 ms (8.5 us now).  Here the addresses travel in the launch parameters and no block waits for
// another one, so there is nothing to allocate but the sums, nothing to upload and nothing to check:
//   - tensors of at most kBlockElems elements each: one launch, one block per tensor; it sums, waits at
//     its own barrier and goes on;
//   - otherwise three launches over the whole list, one span of 2048 elements per block: ||g||; stage 1
//     with m, v and the three sums; stage 2, which computes the directions again from the stored m
//     and v (the same bits).  The order of the stream is the only barrier.
// Bound: host work of the launches for small lists; HBM for large ones, at 48 bytes an element (g three times,
// p twice read, m and v read, written and read again, p written) against the 28 of the persistent kernel, part of it
// from L2 (126 MB).  One tensor of 1 Mi elements 14.6 us (the bound list kernel 28.4), twelve of them 97 (91), 31 of
// 4 Mi 915 us (1065), one of 64 Mi 477 us (549).
#include <cmath>

#include "common.h"
#include "update_core.cuh"

namespace rafb200 {

void bias_corrections(float beta1, float beta2, int step, int bias_correction, float* bc1, float* bc2);
bool pointers_aligned(const void* g, int g_dtype, const void* p, const void* m, const void* v, const void* out,
                      int out_dtype);

constexpr int kRowUnroll = 2;
constexpr int kRowSpan = kPassElems * kRowUnroll;  // 2048 elements per block of the three-launch form
// Device time of a call, one launch against a memset and three.  One to eight tensors: 7.5 us at 1000 elements, 10 at
// 8192, 13.1 to 14 at 16384 against 10.4 from 16385 on, so up to 3.6 us are lost above 8192.  31 tensors: 13.8
// against 12.3.  148: 14.4 against 19.0, and 12.4 us of host time less a call.  400: 52 against 51 (21 at 1000).  The
// line lies where the many tensors of a network still gain; one by the number of tensors would be better for few.
constexpr int kBlockElems = 16384;
constexpr int kOneBlockThreads = 1024;
constexpr int kLansMaxRows = 512;  // 20 KB of the 32 KB a launch's parameters may take
constexpr int kLansFewRows = 64;

struct LansRowsParams {
  LansStage1 s1;
  float lr;
};

template <int CAP>
struct LansRows {
  const float* g[CAP];
  float* p[CAP];
  float* m[CAP];
  float* v[CAP];
  uint32_t end[CAP];    // spans of tensors 0 .. i
  uint32_t numel[CAP];  // below 2^31; the top bit set = vector accesses allowed
};

struct LansRow {
  const float* g;
  float *p, *m, *v;
  int n;  // elements from the pointers on
  bool vec;
};

// Four values from element e, zeros past the end.
__device__ __forceinline__ F4 row_load(const float* a, int e, const LansRow& r, const Policies& pol) {
  if (r.vec && e + kVec <= r.n) return Elem<float>::load4<kDefault>(a + e, pol);
  F4 x;
#pragma unroll
  for (int j = 0; j < kVec; ++j) x.x[j] = e + j < r.n ? a[e + j] : 0.f;
  return x;
}
__device__ __forceinline__ void row_store(float* a, int e, const F4& x, const LansRow& r, const Policies& pol) {
  if (r.vec && e + kVec <= r.n) {
    Elem<float>::store4<kDefault>(a + e, x, pol);
    return;
  }
#pragma unroll
  for (int j = 0; j < kVec; ++j)
    if (e + j < r.n) a[e + j] = x.x[j];
}

// N sums over the block: fp32 inside a warp, double across the warps; in every thread.
template <int N, int THREADS>
__device__ __forceinline__ void row_sums(const float (&x)[N], double (&total)[N]) {
  __shared__ float part[N][THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float s = warp_sum(x[i]);
    if (lane == 0) part[i][warp] = s;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    total[i] = 0.0;
    for (int w = 0; w < THREADS / 32; ++w) total[i] += (double)part[i][w];
  }
}

__device__ __forceinline__ float row_norm_sum(const LansRow& r, int e, float gscale, const Policies& pol) {
  const F4 g = row_load(r.g, e, r, pol);
  float acc = 0.f;
#pragma unroll
  for (int j = 0; j < kVec; ++j) {
    const float x = g.x[j] * gscale;
    acc = fmaf(x, x, acc);
  }
  return acc;
}

// Stage 1 of four elements: m and v stored, the three sums of squares advanced.
template <int MODE>
__device__ __forceinline__ void row_stage1(const LansRow& r, int e, const LansStage1& s1, float cs, float (&acc)[3],
                                           const Policies& pol) {
  const F4 g = row_load(r.g, e, r, pol), p = row_load(r.p, e, r, pol);
  F4 m = row_load(r.m, e, r, pol), v = row_load(r.v, e, r, pol);
#pragma unroll
  for (int j = 0; j < kVec; ++j) {
    float um, ug;
    s1.template apply<MODE>(g.x[j], p.x[j], m.x[j], v.x[j], cs, um, ug);
    if (e + j >= r.n) um = ug = 0.f;  // zeros past the end: 0 / (0 + eps) is no number without an eps
    acc[0] = fmaf(p.x[j], p.x[j], acc[0]);
    acc[1] = fmaf(um, um, acc[1]);
    acc[2] = fmaf(ug, ug, acc[2]);
  }
  row_store(r.m, e, m, r, pol);
  row_store(r.v, e, v, r, pol);
}

// Stage 2 of four elements, the directions computed again from the m and v of stage 1.
template <int MODE>
__device__ __forceinline__ void row_stage2(const LansRow& r, int e, const LansStage1& s1, float cs, float ratio_m,
                                           float ratio_g, const Policies& pol) {
  const F4 g = row_load(r.g, e, r, pol), m = row_load(r.m, e, r, pol), v = row_load(r.v, e, r, pol);
  F4 p = row_load(r.p, e, r, pol);
#pragma unroll
  for (int j = 0; j < kVec; ++j) {
    float um, ug;
    s1.template directions<MODE>(s1.template scaled<MODE>(g.x[j], p.x[j], cs), p.x[j], m.x[j], v.x[j], um, ug);
    p.x[j] = fmaf(ratio_g, ug, fmaf(ratio_m, um, p.x[j]));
  }
  row_store(r.p, e, p, r, pol);
}

// -beta1 * lr * ||p|| / ||update_m|| and -beta3 * lr * ||p|| / ||update_g|| (multi_tensor_lans.cu:347-353)
__device__ __forceinline__ void row_ratios(const LansRowsParams& P, float pn, float umn, float ugn, float* rm, float* rg) {
  const float a = (umn != 0.0f && pn != 0.0f) ? mul(P.lr, fdiv(pn, umn)) : P.lr;
  const float b = (ugn != 0.0f && pn != 0.0f) ? mul(P.lr, fdiv(pn, ugn)) : P.lr;
  *rm = -mul(a, P.s1.beta1);
  *rg = -mul(b, P.s1.beta3);
}

template <int CAP>
__device__ __forceinline__ LansRow row_at(const LansRows<CAP>& rows, int i, int64_t start, int most) {
  const int64_t n = rows.numel[i] & 0x7fffffffu;
  return LansRow{rows.g[i] + start, rows.p[i] + start, rows.m[i] + start, rows.v[i] + start,
                 n - start < most ? (int)(n - start) : most, (rows.numel[i] >> 31) != 0};
}

// ---- one block per tensor ---------------------------------------------------------------
template <int MODE, int CAP>
__global__ void __launch_bounds__(kOneBlockThreads)
    lans_block_kernel(const __grid_constant__ LansRows<CAP> rows, const LansRowsParams P) {
  Policies pol;
  pol.init();
  grid_dependency_trigger();
  const LansRow r = row_at(rows, (int)blockIdx.x, 0, kBlockElems);
  grid_dependency_wait();
  float cs = P.s1.gscale;
  if (P.s1.normalize) {
    float acc[1] = {0.f};
    for (int e = threadIdx.x * kVec; e < r.n; e += kOneBlockThreads * kVec) acc[0] += row_norm_sum(r, e, P.s1.gscale, pol);
    double total[1];
    row_sums<1, kOneBlockThreads>(acc, total);
    cs = P.s1.grad_multiplier(sqrtf((float)total[0]));
  }
  float acc[3] = {0.f, 0.f, 0.f};
  for (int e = threadIdx.x * kVec; e < r.n; e += kOneBlockThreads * kVec) row_stage1<MODE>(r, e, P.s1, cs, acc, pol);
  double total[3];
  row_sums<3, kOneBlockThreads>(acc, total);
  float rm, rg;
  row_ratios(P, sqrtf((float)total[0]), sqrtf((float)total[1]), sqrtf((float)total[2]), &rm, &rg);
  // a thread reads the m and v that it has stored itself
  for (int e = threadIdx.x * kVec; e < r.n; e += kOneBlockThreads * kVec) row_stage2<MODE>(r, e, P.s1, cs, rm, rg, pol);
}

// ---- three launches -----------------------------------------------------------------------
// PHASE 0: ||g||^2 of every tensor into sums[4 t]; 1: stage 1, the other three sums; 2: stage 2.
template <int PHASE, int MODE, int CAP>
__global__ void __launch_bounds__(kBlockThreads)
    lans_phase_kernel(const __grid_constant__ LansRows<CAP> rows, int k, const LansRowsParams P, double* sums) {
  Policies pol;
  pol.init();
  grid_dependency_trigger();
  int lo = 0, hi = k - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (blockIdx.x < rows.end[mid]) hi = mid;
    else lo = mid + 1;
  }
  const LansRow r = row_at(rows, lo, (int64_t)(blockIdx.x - (lo ? rows.end[lo - 1] : 0u)) * kRowSpan, kRowSpan);
  double* mine = sums + 4 * lo;
  grid_dependency_wait();
  if (PHASE == 0) {
    float acc[1] = {0.f};
#pragma unroll
    for (int u = 0; u < kRowUnroll; ++u) acc[0] += row_norm_sum(r, u * kPassElems + threadIdx.x * kVec, P.s1.gscale, pol);
    double total[1];
    row_sums<1, kBlockThreads>(acc, total);
    if (threadIdx.x == 0) atomicAdd(&mine[0], total[0]);
    return;
  }
  const float cs = P.s1.normalize ? P.s1.grad_multiplier(sqrtf((float)mine[0])) : P.s1.gscale;
  if (PHASE == 1) {
    float acc[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int u = 0; u < kRowUnroll; ++u)
      row_stage1<MODE>(r, u * kPassElems + threadIdx.x * kVec, P.s1, cs, acc, pol);
    double total[3];
    row_sums<3, kBlockThreads>(acc, total);
    if (threadIdx.x < 3) atomicAdd(&mine[1 + threadIdx.x], threadIdx.x == 0 ? total[0] : threadIdx.x == 1 ? total[1] : total[2]);
    return;
  }
  float rm, rg;
  row_ratios(P, sqrtf((float)mine[1]), sqrtf((float)mine[2]), sqrtf((float)mine[3]), &rm, &rg);
#pragma unroll
  for (int u = 0; u < kRowUnroll; ++u)
    row_stage2<MODE>(r, u * kPassElems + threadIdx.x * kVec, P.s1, cs, rm, rg, pol);
}

// k >= 1 tensors, none empty, at most CAP of them and fewer than 2^31 spans.
template <int MODE, int CAP>
static int launch_lans_rows(int k, const float* const* g, float* const* p, float* const* m, float* const* v,
                            const int64_t* numel, const LansRowsParams& P, double* sums, cudaStream_t s) {
  LansRows<CAP> rows;
  uint64_t end = 0;
  int64_t largest = 0;
  for (int i = 0; i < k; ++i) {
    rows.g[i] = g[i];
    rows.p[i] = p[i];
    rows.m[i] = m[i];
    rows.v[i] = v[i];
    end += (uint64_t)((numel[i] + kRowSpan - 1) / kRowSpan);
    rows.end[i] = (uint32_t)end;
    rows.numel[i] = (uint32_t)numel[i] |
                    (pointers_aligned(g[i], RAFB200_F32, p[i], m[i], v[i], nullptr, RAFB200_F32) ? 0x80000000u : 0u);
    if (numel[i] > largest) largest = numel[i];
  }
  if (largest <= kBlockElems) {
    RAFB200_CUDA(launch_dependent(lans_block_kernel<MODE, CAP>, (unsigned)k, kOneBlockThreads, 0, s, rows, P));
    return RAFB200_OK;
  }
  const unsigned grid = (unsigned)end;
  RAFB200_CUDA(cudaMemsetAsync(sums, 0, (size_t)k * 4 * sizeof(double), s));
  if (P.s1.normalize)
    RAFB200_CUDA(launch_dependent(lans_phase_kernel<0, MODE, CAP>, grid, kBlockThreads, 0, s, rows, k, P, sums));
  RAFB200_CUDA(launch_dependent(lans_phase_kernel<1, MODE, CAP>, grid, kBlockThreads, 0, s, rows, k, P, sums));
  RAFB200_CUDA(launch_dependent(lans_phase_kernel<2, MODE, CAP>, grid, kBlockThreads, 0, s, rows, k, P, sums));
  return RAFB200_OK;
}

}  // namespace rafb200

using namespace rafb200;

extern "C" {

int rafb200_lans_many(int k, const float* const* g, float* const* p, float* const* m, float* const* v,
                      const int64_t* numel, int step, float learning_rate, float beta1, float beta2, float eps,
                      int bias_correction, float weight_decay, int grad_averaging, int mode, int normalize_grad,
                      float grad_scale, void* workspace, size_t workspace_bytes, void* stream) {
  RAFB200_REQUIRE(k >= 0 && (k == 0 || (g && p && m && v && numel)), "rafb200_lans_many: bad arguments");
  RAFB200_REQUIRE(step >= 1, "rafb200_lans_many: step counts from 1");
  RAFB200_REQUIRE(mode == 0 || mode == 1, "rafb200_lans_many: mode must be 0 (L2) or 1 (decoupled)");
  for (int i = 0; i < k; ++i) {
    RAFB200_REQUIRE(numel[i] >= 0 && numel[i] < (1ll << 31), "rafb200_lans_many: numel[%d] must be in [0, 2^31)", i);
    RAFB200_REQUIRE(numel[i] == 0 || (g[i] && p[i] && m[i] && v[i]), "rafb200_lans_many: NULL pointer for tensor %d", i);
  }
  RAFB200_REQUIRE(workspace && workspace_bytes >= 32 * (size_t)kLansMaxRows && reinterpret_cast<uintptr_t>(workspace) % 16 == 0,
                  "rafb200_lans_many: a workspace of %d bytes, 16-byte aligned, is required", 32 * kLansMaxRows);
  LansRowsParams P{};
  float bc1, bc2;
  bias_corrections(beta1, beta2, step, bias_correction, &bc1, &bc2);
  P.s1.beta1 = beta1;
  P.s1.beta2 = beta2;
  P.s1.beta3 = (grad_averaging == 1) ? 1 - beta1 : 1.0f;  // lans.cc:106-109
  P.s1.one_minus_beta2 = 1 - beta2;
  P.s1.eps = eps;
  P.s1.inv_bc1 = 1.0f / bc1;
  P.s1.inv_bc2 = 1.0f / bc2;
  P.s1.wd = weight_decay;
  P.s1.gscale = grad_scale;
  P.s1.mode = mode;
  P.s1.normalize = normalize_grad ? 1 : 0;
  P.lr = learning_rate;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  double* sums = static_cast<double*>(workspace);
  for (int i = 0; i < k;) {
    if (numel[i] == 0) {
      ++i;
      continue;
    }
    int n = 0;  // a run of tensors with elements; 512 of them have fewer than 2^30 spans
    while (i + n < k && n < kLansMaxRows && numel[i + n] > 0) ++n;
    int rc;
    if (n <= kLansFewRows)
      rc = mode ? launch_lans_rows<1, kLansFewRows>(n, g + i, p + i, m + i, v + i, numel + i, P, sums, s)
                : launch_lans_rows<0, kLansFewRows>(n, g + i, p + i, m + i, v + i, numel + i, P, sums, s);
    else
      rc = mode ? launch_lans_rows<1, kLansMaxRows>(n, g + i, p + i, m + i, v + i, numel + i, P, sums, s)
                : launch_lans_rows<0, kLansMaxRows>(n, g + i, p + i, m + i, v + i, numel + i, P, sums, s);
    if (rc != RAFB200_OK) return rc;
    i += n;
  }
  return RAFB200_OK;
}

}  // extern "C"
