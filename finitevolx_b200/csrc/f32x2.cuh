// Packed FP32 pairs (Blackwell f32x2 arithmetic): two independent values per
// instruction, each lane an IEEE round-to-nearest FP32 operation, the same as
// its scalar form.
#pragma once
#include "fvx_common.cuh"

namespace fvx {

typedef unsigned long long f32x2;
DEV f32x2 f2_pack(float x, float y) {
  f32x2 r;
  asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
DEV float2 f2_unpack(f32x2 a) {
  float2 r;
  asm("mov.b64 {%0,%1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
DEV f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// The same on float2 values.
DEV float2 f2fma(float2 a, float2 b, float2 c) {
  return f2_unpack(f2_fma(f2_pack(a.x, a.y), f2_pack(b.x, b.y), f2_pack(c.x, c.y)));
}
DEV float2 f2add(float2 a, float2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(f2_pack(a.x, a.y)), "l"(f2_pack(b.x, b.y)));
  return f2_unpack(d);
}
DEV float2 f2sub(float2 a, float2 b) {
  f32x2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(f2_pack(a.x, a.y)), "l"(f2_pack(b.x, b.y)));
  return f2_unpack(d);
}
DEV float2 f2mul(float2 a, float2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(f2_pack(a.x, a.y)), "l"(f2_pack(b.x, b.y)));
  return f2_unpack(d);
}
DEV float2 f2s(float c) { return make_float2(c, c); }

}  // namespace fvx
