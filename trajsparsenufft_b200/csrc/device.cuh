// Device helpers shared by the sm_100a kernels: complex arithmetic, asynchronous copies,
// ldmatrix / warp sparse MMA wrappers, FP16 hi+residual split.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tsn {
namespace dev {

// Complex add / subtract as one paired FP32 instruction (sm_100 FADD2; each lane rounds
// exactly like the scalar add).
__host__ __device__ __forceinline__ float2 cadd(float2 a, float2 b) {
#ifdef __CUDA_ARCH__
  return __fadd2_rn(a, b);
#else
  return make_float2(a.x + b.x, a.y + b.y);
#endif
}
__host__ __device__ __forceinline__ float2 csub(float2 a, float2 b) {
#ifdef __CUDA_ARCH__
  return __fadd2_rn(a, make_float2(-b.x, -b.y));
#else
  return make_float2(a.x - b.x, a.y - b.y);
#endif
}
__host__ __device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a * conj(b)
__host__ __device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
// y + a x with a in FP64 and one rounding per component. The CG step lengths are applied so: a
// step length rounded to FP32 leaves 6e-8 of the dominant direction in the residual, which
// ten iterations turn into 5e-5 of the image (FP64 restatement of the solve, 128^2, 4 coils;
// 1.5e-6 with every vector in FP32 and the step lengths in FP64).
__device__ __forceinline__ float2 axpy64(double a, float2 x, float2 y) {
  return make_float2(static_cast<float>(fma(a, static_cast<double>(x.x), static_cast<double>(y.x))),
                     static_cast<float>(fma(a, static_cast<double>(x.y), static_cast<double>(y.y))));
}
__host__ __device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__host__ __device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Programmatic dependent launch. pdl_wait blocks until the kernel this one was launched
// behind (with cudaLaunchAttributeProgrammaticStreamSerialization) has completed and its
// writes are visible; pdl_trigger lets the next such kernel of the stream start its prologue.
// Both return at once in a kernel launched without the attribute.  A kernel reads nothing
// that an earlier kernel may write, and writes nothing, before pdl_wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(smem_dst)), "l"(gmem_src));
}
// The same to a shared address.
__device__ __forceinline__ void cp_async16_u32(uint32_t smem_dst, const void* gmem_src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_dst), "l"(gmem_src) : "memory");
}
// 16-byte copy to a shared address, or (skip != 0) a 16-byte zero fill without a global read.
__device__ __forceinline__ void cp_async16_or_zero(uint32_t smem_dst, const void* gmem_src, uint32_t skip) {
  asm volatile("{ .reg .pred p; setp.ne.u32 p, %2, 0; cp.async.cg.shared.global [%0], [%1], 16, p; }\n" ::"r"(smem_dst),
               "l"(gmem_src), "r"(skip)
               : "memory");
}
// base + 16 units, in one instruction
__device__ __forceinline__ const uint8_t* offset16(const uint8_t* base, uint32_t units) {
  uint64_t a;
  asm("mad.wide.u32 %0, %1, 16, %2;" : "=l"(a) : "r"(units), "l"(base));
  return reinterpret_cast<const uint8_t*>(a);
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Four transposed 8x8 b16 matrices (rows addressed by lanes 0-7, 8-15, 16-23, 24-31).
__device__ __forceinline__ void ldmatrix_x4_trans_u32(uint32_t (&r)[4], uint32_t smem_row) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(smem_row)
               : "memory");
}

// Warp-level 2:4 sparse MMA m16n8k32, FP16 inputs, FP32 accumulate, metadata selector 0.
__device__ __forceinline__ void mma_sp_16832(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[4],
                                             uint32_t meta) {
  asm volatile(
      "mma.sp::ordered_metadata.sync.aligned.m16n8k32.row.col.f32.f16.f16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9,%10,%11}, {%0,%1,%2,%3}, %12, 0x0;\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(meta));
}

// The same product from a zero accumulator.
__device__ __forceinline__ void mma_sp_16832_zero(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[4],
                                                  uint32_t meta) {
  asm volatile(
      "mma.sp::ordered_metadata.sync.aligned.m16n8k32.row.col.f32.f16.f16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9,%10,%11}, {%13,%13,%13,%13}, %12, 0x0;\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(meta), "f"(0.f));
}

// FP32 value -> FP16 high part + FP16 residual (value - float(high)), the reference's
// split2 panel (reference_sparse_solver.py:66-76, integrated_complex_to_split2_half_rows).
__device__ __forceinline__ void split_hi_res(float v, __half& hi, __half& res) {
  hi = __float2half_rn(v);
  res = __float2half_rn(v - __half2float(hi));
}

__device__ __forceinline__ uint32_t pack_half2(__half lo, __half hi) {
  return static_cast<uint32_t>(__half_as_ushort(lo)) | (static_cast<uint32_t>(__half_as_ushort(hi)) << 16);
}

// Complex (re, im) -> packed FP16 high parts (re low, im high) and packed FP16 residuals:
// split_hi_res on each component, with the paired conversions (same rounding, same bits).
__device__ __forceinline__ void split_hi_res2(float re, float im, uint32_t& hi, uint32_t& res) {
  const __half2 h = __floats2half2_rn(re, im);
  const float2 back = __half22float2(h);
  const __half2 r = __floats2half2_rn(re - back.x, im - back.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  res = *reinterpret_cast<const uint32_t*>(&r);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  return v;
}

// Deterministic block sum of one double per thread (fixed order), returned to every thread.
// `scratch` holds 32 doubles; it may be reused at once.
__device__ __forceinline__ double block_sum(double v, double* scratch) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  double t = 0.0;
  for (int w = 0; w < nw; ++w) t += scratch[w];
  __syncthreads();
  return t;
}

// Warp sums of four doubles per lane in six exchanges instead of twenty: each halving of the
// lanes also halves the values a lane keeps. Lanes 0, 8, 16, 24 (and the seven after each)
// return the sums of a, b, c, d.
__device__ __forceinline__ double warp_sum4(double a, double b, double c, double d) {
  const int lane = threadIdx.x & 31;
  const bool upper = lane & 16, odd = lane & 8;
  double k0 = upper ? c : a, k1 = upper ? d : b;
  k0 += __shfl_xor_sync(0xFFFFFFFFu, upper ? a : c, 16);
  k1 += __shfl_xor_sync(0xFFFFFFFFu, upper ? b : d, 16);
  double k = odd ? k1 : k0;
  k += __shfl_xor_sync(0xFFFFFFFFu, odd ? k0 : k1, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) k += __shfl_xor_sync(0xFFFFFFFFu, k, o);
  return k;
}

// Power-of-two scale bringing rms to ~target (FP16 rounding commutes with it): the nearest
// power (on the logarithm) of target / rms, from the exponent of 2 (target / rms)^2. Every CTA
// of a row stage waits for it, so no square root, logarithm or power is taken.
__device__ __forceinline__ float pow2_scale(double sum_sq, double count, float target) {
  if (!(sum_sq > 0.0) || !isfinite(sum_sq)) return 1.0f;
  const double q = 2.0 * static_cast<double>(target) * target * count / sum_sq;
  const int e = (((__double2hiint(q) >> 20) & 0x7FF) - 1023) >> 1;  // floor(log2(q) / 2)
  return __int_as_float((min(max(e, -100), 100) + 127) << 23);
}

}  // namespace dev
}  // namespace tsn
