// Building blocks of the update kernels: the per-element arithmetic of SGD, Adam and LANS,
// and the walk of a block over one span of a tensor with 16-byte accesses (scalar ones for
// unaligned tensors and ragged tails).
#pragma once
#include "common.h"
#include "vec_io.cuh"

namespace rafb200 {

constexpr int kVec = 4;                              // elements per thread per pass
constexpr int kPassElems = kBlockThreads * kVec;     // 1024
constexpr uint32_t kFlagAligned = 1u;  // vector accesses allowed (16 B fp32, 8 B 16-bit arrays)
constexpr uint32_t kFlagBulk = 2u;     // every array is 16-byte aligned: TMA bulk copies allowed

// ---- per-element arithmetic -------------------------------------------------
// All three follow the reference expression by expression; see the C ABI
// header for the citations.  Every operation is a separately rounded fp32 op.

struct SgdOp {
  float lr, mu, wd, gscale;
  // v1 = mu*v0 + dx ; x1 = x0 - lr*v1      (python/raf/_tvm_op/sgd.py:21-29)
  __device__ __forceinline__ void operator()(float g, float& p, float& m, float& /*v*/) const {
    if (gscale != 1.0f) g = mul(g, gscale);
    if (wd != 0.0f) g = add(g, mul(wd, p));
    float v1 = add(mul(mu, m), g);
    p = sub(p, mul(lr, v1));
    m = v1;
  }
  __device__ __forceinline__ void vec(const F4& g, F4& p, F4& m, F4& v) const {
#pragma unroll
    for (int j = 0; j < 4; ++j) (*this)(g.x[j], p.x[j], m.x[j], v.x[j]);
  }
};

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Correctly rounded a/b and sqrt(x) without a branch, for operands far from overflow and
// underflow (AdamOp::vec checks).  The library forms test every operand and branch, which keeps
// the elements a thread holds from being interleaved.
// a/b: P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor"
// (1990): with y = RN(1/b) and q within one unit of a/b, RN(q + RN(a - b*q) * y) is RN(a/b).  The
// first step brings a*y (up to 1.5 units off) within one unit, the second one rounds.
__device__ __forceinline__ float div_by(float a, float b, float y) {
  float q = mul(a, y);
  q = fmaf(fmaf(-b, q, a), y, q);
  return fmaf(fmaf(-b, q, a), y, q);
}
// RN(1/b): one step of Newton's method for 1/y - b, y + y * (1 - b * y) with the bracket in one rounding, on
// the hardware's approximation.  That it rounds correctly is a property of that approximation:
// tests/test_adam_arithmetic_gpu.py compares every one of the 2^23 significands, at exponents
// -60 .. 60, with __frcp_rn.
__device__ __forceinline__ float rcp_rn(float b) {
  const float y = rcp_approx(b);
  return fmaf(fmaf(-b, y, 1.0f), y, y);
}
// RN(sqrt(x)): one step of Newton's method for g^2 - x, g + (x - g * g) / (2 g) with the bracket in one rounding, from
// g = x * y and 1 / (2 g) = y / 2, y the hardware's approximation of 1 / sqrt(x).  Compared with
// __fsqrt_rn for every float from 2^-100 to 2^100 by the same test.  x must not be zero.
__device__ __forceinline__ float sqrt_rn(float x) {
  const float y = rsqrt_approx(x);
  const float g = mul(x, y), h = mul(0.5f, y);
  return fmaf(fmaf(-g, g, x), h, g);
}

// (m / bc1) / (sqrt(v / bc2) + eps) for any operands; a call, so that it costs the kernels no registers
static __device__ __noinline__ float adam_ratio(float m, float v, float bc1, float bc2, float eps) {
  return fdiv(fdiv(m, bc1), add(fsqrt(fdiv(v, bc2)), eps));
}

struct AdamOp {
  float lr, beta1, beta2, beta3, one_minus_beta2, eps, bc1, bc2, wd, gscale;
  int mode;
  float y1, y2;  // RN(1/bc1), RN(1/bc2)
  int fast;      // bc1, bc2 and eps allow vec() its branch-free form
  __device__ __forceinline__ void moments(float& g, float p, float& m, float& v) const {
    if (gscale != 1.0f) g = mul(g, gscale);
    if (mode == 0) g = add(g, mul(wd, p));
    m = add(mul(m, beta1), mul(beta3, g));
    v = add(mul(v, beta2), mul(mul(one_minus_beta2, g), g));
  }
  __device__ __forceinline__ void finish(float update, float& p) const {
    if (mode != 0) update = add(update, mul(wd, p));
    p = sub(p, mul(lr, update));
  }
  __device__ __forceinline__ void operator()(float g, float& p, float& m, float& v) const {
    moments(g, p, m, v);
    finish(adam_ratio(m, v, bc1, bc2, eps), p);
  }
  // Four elements at once.  Two exact divisions by per-call constants, one by the denominator and
  // one square root per element: with the library forms the Adam kernel issues more than HBM
  // can feed (44,353,792 elements bf16: 204 us against 186).  Here the operands of all four are
  // tested once and the arithmetic is straight-line code with the same bits.  The test:
  // m is +0 or 2^-80 .. 2^60 in size, v is +0 or 2^-100 .. 2^40, and the host has seen bc1, bc2 in
  // 2^-20 .. 1 and eps in 2^-40 .. 1: every quotient is then a normal number or zero, every
  // remainder exact, and the denominator lies within 2^-40 .. 2^31.
  __device__ __forceinline__ void vec(const F4& gi, F4& p, F4& m, F4& v) const {
    bool ok = fast != 0;
    F4 g = gi;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      moments(g.x[j], p.x[j], m.x[j], v.x[j]);
      const unsigned mb = __float_as_uint(m.x[j]), vb = __float_as_uint(v.x[j]);
      ok &= (mb == 0u) | ((mb & 0x7fffffffu) - 0x17800000u < 0x46000000u);  // 2^-80 <= |m| < 2^60
      ok &= (vb == 0u) | (vb - 0x0d800000u < 0x46000000u);                  // 2^-100 <= v < 2^40
    }
    if (__builtin_expect(ok, 1)) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float vh = div_by(v.x[j], bc2, y2);
        const float denom = add(vh == 0.0f ? 0.0f : sqrt_rn(vh), eps);
        finish(div_by(div_by(m.x[j], bc1, y1), denom, rcp_rn(denom)), p.x[j]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) finish(adam_ratio(m.x[j], v.x[j], bc1, bc2, eps), p.x[j]);
    }
  }
};

// LANS stage 1 (src/op/dialect/cuda/kernels/multi_tensor_lans.cu:281-306).
// The reference divides five times and takes one square root per element; at
// 28 bytes per element that is more arithmetic than a B200 SM can issue in the
// time HBM delivers the data (two passes need it).  The divisions by values
// that are constant per call or per tensor (bias corrections, ||g||+eps) become
// multiplications by reciprocals computed once, the two divisions by the
// denominator share one reciprocal, and sqrt / reciprocal use the 1-ulp hardware
// approximations (flush-to-zero forms: the square root's argument only matters
// when it is far above the denormal range, and the reciprocal's is >= eps).
// Each substitution moves a result by at most about one unit
// in the last place (1.2e-7 relative); the tests bound the total against the
// exact restatement at 2e-6 for m and v and far less for p.
struct LansStage1 {
  float beta1, beta2, beta3, one_minus_beta2, eps, inv_bc1, inv_bc2, wd, gscale;
  int mode, normalize;
  // Multiplier that turns a raw gradient element into the scaled gradient:
  // grad_scale / (||g|| + eps) when gradients are normalised and ||g|| != 0.
  __device__ __forceinline__ float grad_multiplier(float gnorm) const {
    if (normalize && gnorm != 0.0f) return gscale * fdiv(1.0f, add(gnorm, eps));
    return gscale;
  }
  // in: g (raw), p, m, v, cs = grad_multiplier   out: m, v updated; um, ug.
  // MODE is the `mode` argument (0 = L2, 1 = decoupled weight decay) as a compile-time
  // constant: with the choice made once per chunk, the arithmetic of the elements a thread
  // holds is one straight line of code that the compiler can interleave.
  template <int MODE>
  __device__ __forceinline__ float scaled(float g, float p, float cs) const {
    const float sg = g * cs;
    return MODE == 0 ? fmaf(wd, p, sg) : sg;
  }
  // update_m and update_g from the new m and v
  template <int MODE>
  __device__ __forceinline__ void directions(float sg, float p, float m, float v, float& um, float& ug) const {
    const float r = rcp_approx(sqrt_approx(v * inv_bc2) + eps);
    if (MODE == 0) {
      um = (m * inv_bc1) * r;
      ug = sg * r;
    } else {
      const float sp = wd * p;
      um = fmaf(m * inv_bc1, r, sp);
      ug = fmaf(sg, r, sp);
    }
  }
  template <int MODE>
  __device__ __forceinline__ void apply(float g, float p, float& m, float& v, float cs, float& um,
                                        float& ug) const {
    const float sg = scaled<MODE>(g, p, cs);
    m = fmaf(beta3, sg, m * beta1);
    v = fmaf(one_minus_beta2 * sg, sg, v * beta2);
    directions<MODE>(sg, p, m, v, um, ug);
  }
};

// ---- the element-wise update of a span --------------------------------------------
// One block's share: `len` elements (<= kBlockThreads * 4 * UNROLL) of one tensor from element
// `start`.  Every load of the span is issued before the first use: 256 threads with UNROLL = 2
// keep 24 to 32 KB in flight per block, and six to eight blocks of them an SM.
template <int NSTATE, typename GT, typename OT, int UNROLL, typename Op>
__device__ __forceinline__ void update_span(const TensorDesc& d, int64_t start, int len, const Op& op,
                                            const Policies& pol) {
  const GT* g = static_cast<const GT*>(d.g) + start;
  float* p = d.p + start;
  float* m = d.m + start;
  float* v = NSTATE == 2 ? d.v + start : nullptr;
  OT* out = d.out ? static_cast<OT*>(d.out) + start : nullptr;
  const int tid = threadIdx.x;
  int done = 0;
  if (d.flags & kFlagAligned) {
    const int len4 = len & ~(kVec - 1);
    F4 rg[UNROLL], rp[UNROLL], rm[UNROLL], rv[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int e = u * kPassElems + tid * kVec;
      if (e < len4) {
        rg[u] = Elem<GT>::template load4<kStream>(g + e, pol);
        rp[u] = Elem<float>::template load4<kStream>(p + e, pol);
        rm[u] = Elem<float>::template load4<kStream>(m + e, pol);
        if (NSTATE == 2) rv[u] = Elem<float>::template load4<kStream>(v + e, pol);
        else rv[u] = f4_zero();
      }
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int e = u * kPassElems + tid * kVec;
      if (e < len4) {
        op.vec(rg[u], rp[u], rm[u], rv[u]);
        Elem<float>::template store4<kDefault>(p + e, rp[u], pol);
        Elem<float>::template store4<kDefault>(m + e, rm[u], pol);
        if (NSTATE == 2) Elem<float>::template store4<kDefault>(v + e, rv[u], pol);
        if (out) Elem<OT>::template store4<kDefault>(out + e, rp[u], pol);
      }
    }
    done = len4;
  }
  for (int e = done + tid; e < len; e += kBlockThreads) {
    float gg = Elem<GT>::to_f32(g[e]);
    float pp = p[e], mm = m[e], vv = NSTATE == 2 ? v[e] : 0.f;
    op(gg, pp, mm, vv);
    p[e] = pp;
    m[e] = mm;
    if (NSTATE == 2) v[e] = vv;
    if (out) out[e] = Elem<OT>::from_f32(pp);
  }
}

// What a chunk of the list (fused kernel) covers.
struct ChunkView {
  const void* g;
  float* p;
  float* m;
  float* v;
  void* out;
  int len;       // elements in this chunk
};

__device__ __forceinline__ ChunkView chunk_view(const TensorDesc& d, uint32_t chunk, int g_size,
                                                int out_size) {
  ChunkView c;
  const int64_t start = (int64_t)chunk * kChunkElems;
  const int64_t left = d.numel - start;
  c.len = left < kChunkElems ? (int)left : kChunkElems;
  c.g = static_cast<const char*>(d.g) + start * g_size;
  c.p = d.p + start;
  c.m = d.m + start;
  c.v = d.v ? d.v + start : nullptr;
  c.out = d.out ? static_cast<char*>(d.out) + start * out_size : nullptr;
  return c;
}

}  // namespace rafb200
