// f32x4.h -- four FP32 values of a lane: 16-byte loads and stores, and arithmetic with
// the packed two-value instructions (add, mul, fma .rn.f32x2: each half rounded as the
// scalar instruction rounds it, two values an issue slot).
#pragma once
#ifdef __CUDACC__
namespace ads {

struct alignas(16) F4 {
  float2 a, b;
};
__device__ __forceinline__ float2 add2(float2 x, float2 y) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, r;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "add.rn.f32x2 r, x, y;\n\tmov.b64 {%0, %1}, r;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 x, float2 y) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, r;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "mul.rn.f32x2 r, x, y;\n\tmov.b64 {%0, %1}, r;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y));
  return r;
}
__device__ __forceinline__ float2 fma2(float2 x, float2 y, float2 z) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z, r;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
      "mov.b64 z, {%6, %7};\n\tfma.rn.f32x2 r, x, y, z;\n\tmov.b64 {%0, %1}, r;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y), "f"(z.x), "f"(z.y));
  return r;
}
__device__ __forceinline__ float2 sub2(float2 x, float2 y) {  // x - y
  return fma2(y, make_float2(-1.f, -1.f), x);
}

// A 16-byte load / store at a 32-bit element offset of a field, predicated.
__device__ __forceinline__ F4 ld4(const float* p, int o, bool on) {
  F4 x;
  x.a.x = x.a.y = x.b.x = x.b.y = 0.f;
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t"
      "@q ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "+f"(x.a.x), "+f"(x.a.y), "+f"(x.b.x), "+f"(x.b.y)
      : "l"(p + o), "r"((unsigned)on));
  return x;
}
__device__ __forceinline__ void st4(float* p, int o, const F4& x) {
  *reinterpret_cast<float4*>(p + o) = make_float4(x.a.x, x.a.y, x.b.x, x.b.y);
}
__device__ __forceinline__ float ld1v(const float* p, int o, bool on) {
  float a = 0.f;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.global.f32 %0, [%1];\n\t}"
               : "+f"(a)
               : "l"(p + o), "r"((unsigned)on));
  return a;
}

__device__ __forceinline__ F4 add4(const F4& x, const F4& y) { return {add2(x.a, y.a), add2(x.b, y.b)}; }
__device__ __forceinline__ F4 sub4(const F4& x, const F4& y) { return {sub2(x.a, y.a), sub2(x.b, y.b)}; }
__device__ __forceinline__ F4 mul4(const F4& x, const F4& y) { return {mul2(x.a, y.a), mul2(x.b, y.b)}; }
__device__ __forceinline__ F4 fma4(const F4& x, const F4& y, const F4& z) {
  return {fma2(x.a, y.a, z.a), fma2(x.b, y.b, z.b)};
}

}  // namespace ads
#endif
