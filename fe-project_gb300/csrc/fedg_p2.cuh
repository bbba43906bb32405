// fedg_p2.cuh -- two float pairs side by side: the pair arithmetic of fedg_f2.cuh on the packed FP32
// instructions (add/sub/mul/fma.rn.f32x2), one instruction for the same operation on two nodes.
//
// The packed instructions retire the same number of FP32 results per cycle as the scalar ones (63
// packed against 120-125 scalar instructions per cycle and SM, measured with register-only loops), but
// take half the issue slots, and one thread's two independent chains overlap their latencies.  Kernels
// bound by issue or by the latency of the compensated sums gain from both; the arithmetic of each node
// is the same sequence of roundings as the scalar pair operation's.
#pragma once
#include "fedg_f2.cuh"

namespace fedg {

typedef unsigned long long u64x;  // two floats: .lo (node A), .hi (node B)

__device__ __forceinline__ u64x pk(float a, float b) {
  u64x r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpk(u64x v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ u64x pk1(float a) { return pk(a, a); }
__device__ __forceinline__ u64x xadd(u64x a, u64x b) {
  u64x d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64x xsub(u64x a, u64x b) {
  u64x d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64x xmul(u64x a, u64x b) {
  u64x d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64x xfma(u64x a, u64x b, u64x c) {
  u64x d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// the pairs of two nodes: h = (hA, hB), l = (lA, lB); 16 bytes in memory
struct p2 {
  u64x h, l;
};
struct __align__(16) p2m {  // p2 in memory: one 16-byte access
  u64x h, l;
};
__device__ __forceinline__ p2 ld(const p2m& m) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&m);
  return {v.x, v.y};
}
__device__ __forceinline__ void st(p2m& m, p2 v) { *reinterpret_cast<ulonglong2*>(&m) = make_ulonglong2(v.h, v.l); }

__device__ __forceinline__ p2 p2_of(f2 a, f2 b) { return {pk(a.h, b.h), pk(a.l, b.l)}; }
__device__ __forceinline__ p2 p2_dup(f2 a) { return {pk1(a.h), pk1(a.l)}; }
__device__ __forceinline__ p2 p2_dup(float2 a) { return {pk1(a.x), pk1(a.y)}; }
__device__ __forceinline__ p2 p2_of(float2 a, float2 b) { return {pk(a.x, b.x), pk(a.y, b.y)}; }
__device__ __forceinline__ f2 p2_a(p2 v) { return {unpk(v.h).x, unpk(v.l).x}; }
__device__ __forceinline__ f2 p2_b(p2 v) { return {unpk(v.h).y, unpk(v.l).y}; }
__device__ __forceinline__ p2 p2_zero() { return {0ull, 0ull}; }

__device__ __forceinline__ p2 p2_two_sum(u64x a, u64x b) {
  const u64x s = xadd(a, b);
  const u64x bb = xsub(s, a);
  return {s, xadd(xsub(a, xsub(s, bb)), xsub(b, bb))};
}
__device__ __forceinline__ p2 p2_fast_two_sum(u64x a, u64x b) {
  const u64x s = xadd(a, b);
  return {s, xsub(b, xsub(s, a))};
}
__device__ __forceinline__ p2 operator+(p2 a, p2 b) {
  const p2 s = p2_two_sum(a.h, b.h);
  return p2_fast_two_sum(s.h, xadd(s.l, xadd(a.l, b.l)));
}
__device__ __forceinline__ p2 operator-(p2 a, p2 b) {
  // two-sum of a.h and -b.h
  const u64x s = xsub(a.h, b.h);
  const u64x bb = xsub(s, a.h);
  const u64x e = xsub(xsub(a.h, xsub(s, bb)), xadd(b.h, bb));
  return p2_fast_two_sum(s, xadd(e, xsub(a.l, b.l)));
}
__device__ __forceinline__ p2 p2_add_x(p2 a, u64x b) {
  const p2 s = p2_two_sum(a.h, b);
  return p2_fast_two_sum(s.h, xadd(s.l, a.l));
}
__device__ __forceinline__ p2 operator*(p2 a, p2 b) {
  const u64x p = xmul(a.h, b.h);
  // the product's error: a.h b.h - p = -(p - a.h b.h), and p - x y needs a negated factor, so the
  // sign is taken on p (exact)
  u64x e = xfma(a.h, b.h, p ^ 0x8000000080000000ull);
  e = xfma(a.h, b.l, e);
  e = xfma(a.l, b.h, e);
  return p2_fast_two_sum(p, e);
}
__device__ __forceinline__ p2 p2_mul_x(p2 a, u64x b) {
  const u64x p = xmul(a.h, b);
  u64x e = xfma(a.h, b, p ^ 0x8000000080000000ull);
  e = xfma(a.l, b, e);
  return p2_fast_two_sum(p, e);
}
// exact scaling by a power of two or a sign
__device__ __forceinline__ p2 p2_scale(p2 a, u64x s) { return {xmul(a.h, s), xmul(a.l, s)}; }
__device__ __forceinline__ p2 p2_neg(p2 a) { return {a.h ^ 0x8000000080000000ull, a.l ^ 0x8000000080000000ull}; }
__device__ __forceinline__ p2 p2_recip(p2 d) {
  const float2 dh = unpk(d.h);
  const u64x y = pk(__fdividef(1.f, dh.x), __fdividef(1.f, dh.y));
  const p2 t = p2_mul_x(d, y);
  const u64x e = xsub(xsub(pk1(1.f), t.h), t.l);
  return p2_fast_two_sum(y, xmul(y, e));
}
__device__ __forceinline__ p2 p2_split(double a, double b) { return p2_of(f2_split(a), f2_split(b)); }
// the same normalised (h the nearest float; f2_split truncates), for values that enter reciprocals and products
// whose l l term is dropped
__device__ __forceinline__ p2 p2_split_n(double a, double b) {
  const p2 v = p2_split(a, b);
  return p2_fast_two_sum(v.h, v.l);
}

// compensated dot-product accumulator (f2acc)
struct p2acc {
  u64x s = 0ull, c = 0ull;
  __device__ __forceinline__ void add(p2 d, p2 x) {
    const u64x p = xmul(d.h, x.h);
    u64x e = xfma(d.h, x.h, p ^ 0x8000000080000000ull);
    e = xfma(d.h, x.l, e);
    e = xfma(d.l, x.h, e);
    const p2 t = p2_two_sum(s, p);
    s = t.h;
    c = xadd(c, xadd(t.l, e));
  }
  __device__ __forceinline__ p2 get() const { return p2_fast_two_sum(s, c); }
};

}  // namespace fedg
