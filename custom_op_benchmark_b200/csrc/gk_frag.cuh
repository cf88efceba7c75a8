// Register fragments: the elements of one slot (4, 8 or 16 bytes of a feature row) held by a lane in the accumulation
// type, and the few operations the kernels do on them.  float accumulators are kept as pairs in 64-bit registers so
// that products and sums go through the packed fma.rn.f32x2 of sm_100 (two IEEE fused multiply-adds per instruction,
// the same rounding as two scalar ones): a 16-byte slot of four floats is two instructions instead of four, one of
// eight bfloat16 four instead of eight.
#pragma once
#include "gk_common.cuh"

namespace gk {

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(float& a, float& b, f32x2 v) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// two bfloat16 of a 32-bit word (element 0 in the low half) as two floats
__device__ __forceinline__ f32x2 widen2(uint32_t w) { return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }

// 2^x.  float: the hardware approximation (relative error about 2^-22); double: exp2().
__device__ __forceinline__ float gk_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ double gk_exp2(double x) { return exp2(x); }
__device__ __forceinline__ float gk_log2(float x) { return log2f(x); }
__device__ __forceinline__ double gk_log2(double x) { return log2(x); }
constexpr double kLog2e = 1.4426950408889634074;
constexpr double kLn2 = 0.69314718055994530942;

// ---------------------------------------------------------------------------------------
// Fragment of V accumulators (A = float or double)
// ---------------------------------------------------------------------------------------
template <typename A, int V> struct Frag;

template <int V> struct Frag<float, V> {
  static_assert(V == 1 || V % 2 == 0, "one float or pairs");
  static constexpr int P = V == 1 ? 1 : V / 2;
  f32x2 p[P];   // V == 1: the float sits in the low half, the high half is zero
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < P; ++i) p[i] = 0ull;
  }
  __device__ __forceinline__ void get(float (&x)[V]) const {
    if constexpr (V == 1) {
      float hi;
      unpack2(x[0], hi, p[0]);
    } else {
#pragma unroll
      for (int i = 0; i < P; ++i) unpack2(x[2 * i], x[2 * i + 1], p[i]);
    }
  }
  __device__ __forceinline__ void set(const float (&x)[V]) {
    if constexpr (V == 1) {
      p[0] = pack2(x[0], 0.f);
    } else {
#pragma unroll
      for (int i = 0; i < P; ++i) p[i] = pack2(x[2 * i], x[2 * i + 1]);
    }
  }
  __device__ __forceinline__ void scale(float s) {
    const f32x2 ss = pack2(s, s);
#pragma unroll
    for (int i = 0; i < P; ++i) p[i] = mul2(p[i], ss);
  }
  __device__ __forceinline__ void axpy(float s, const Frag& x) {
    const f32x2 ss = pack2(s, s);
#pragma unroll
    for (int i = 0; i < P; ++i) p[i] = fma2(ss, x.p[i], p[i]);
  }
  __device__ __forceinline__ void add(const Frag& x) {
#pragma unroll
    for (int i = 0; i < P; ++i) p[i] = add2(p[i], x.p[i]);
  }
  // this * wa + x * wb
  __device__ __forceinline__ void blend(float wa, const Frag& x, float wb) {
    const f32x2 aa = pack2(wa, wa), bb = pack2(wb, wb);
#pragma unroll
    for (int i = 0; i < P; ++i) p[i] = fma2(x.p[i], bb, mul2(p[i], aa));
  }
};

template <int V> struct Frag<double, V> {
  double p[V];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < V; ++i) p[i] = 0.0;
  }
  __device__ __forceinline__ void get(double (&x)[V]) const {
#pragma unroll
    for (int i = 0; i < V; ++i) x[i] = p[i];
  }
  __device__ __forceinline__ void set(const double (&x)[V]) {
#pragma unroll
    for (int i = 0; i < V; ++i) p[i] = x[i];
  }
  __device__ __forceinline__ void scale(double s) {
#pragma unroll
    for (int i = 0; i < V; ++i) p[i] *= s;
  }
  __device__ __forceinline__ void axpy(double s, const Frag& x) {
#pragma unroll
    for (int i = 0; i < V; ++i) p[i] = fma(s, x.p[i], p[i]);
  }
  __device__ __forceinline__ void add(const Frag& x) {
#pragma unroll
    for (int i = 0; i < V; ++i) p[i] += x.p[i];
  }
  __device__ __forceinline__ void blend(double wa, const Frag& x, double wb) {
#pragma unroll
    for (int i = 0; i < V; ++i) p[i] = p[i] * wa + x.p[i] * wb;
  }
};

// sum of the products of W fragments; every kernel forms its dot products here, so that two kernels that multiply
// the same rows get the same bits
template <int V, int W>
__device__ __forceinline__ float frag_dot(const Frag<float, V> (&a)[W], const Frag<float, V> (&b)[W]) {
  f32x2 s = mul2(a[0].p[0], b[0].p[0]);
#pragma unroll
  for (int i = 0; i < W; ++i)
#pragma unroll
    for (int j = (i == 0 ? 1 : 0); j < Frag<float, V>::P; ++j) s = fma2(a[i].p[j], b[i].p[j], s);
  float lo, hi;
  unpack2(lo, hi, s);
  return lo + hi;
}
template <int V, int W>
__device__ __forceinline__ double frag_dot(const Frag<double, V> (&a)[W], const Frag<double, V> (&b)[W]) {
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < W; ++i)
#pragma unroll
    for (int j = 0; j < V; ++j) s = fma(a[i].p[j], b[i].p[j], s);
  return s;
}

// raw slot bytes -> fragment
template <int SB> struct SlotWord;
template <> struct SlotWord<16> { using type = uint4; };
template <> struct SlotWord<8> { using type = uint2; };
template <> struct SlotWord<4> { using type = uint32_t; };

template <typename T, int SB>
__device__ __forceinline__ void frag_unpack(Frag<typename AccOf<T>::type, SB / (int)sizeof(T)>& f,
                                            const typename SlotWord<SB>::type& word) {
  constexpr int V = SB / (int)sizeof(T);
  union { typename SlotWord<SB>::type m; T t[V]; uint32_t w[SB / 4]; f32x2 d[SB >= 8 ? SB / 8 : 1]; } u;
  u.m = word;
  if constexpr (sizeof(T) == 2) {
#pragma unroll
    for (int i = 0; i < V / 2; ++i) f.p[i] = widen2(u.w[i]);
  } else if constexpr (sizeof(T) == 4 && V == 1) {
    f.p[0] = pack2(__uint_as_float(u.w[0]), 0.f);
  } else if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int i = 0; i < V / 2; ++i) f.p[i] = u.d[i];
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) f.p[i] = to_acc<T>(u.t[i]);
  }
}
// Loads of gathered rows.  volatile: a slot is refilled where it was last read, not before.
__device__ __forceinline__ void ldg_word(uint4& v, const void* p) {
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
}
__device__ __forceinline__ void ldg_word(uint2& v, const void* p) {
  asm volatile("ld.global.nc.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
}
__device__ __forceinline__ void ldg_word(uint32_t& v, const void* p) { asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p)); }

// Shared memory by its 32-bit address.  volatile: these loads stay behind the waits for the asynchronous copies.
__device__ __forceinline__ void lds(uint4& v, unsigned at) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at));
}
__device__ __forceinline__ void lds(uint2& v, unsigned at) {
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(at));
}
__device__ __forceinline__ void lds(uint32_t& v, unsigned at) { asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at)); }
__device__ __forceinline__ void lds(float& v, unsigned at) { asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at)); }
__device__ __forceinline__ void lds(double& v, unsigned at) { asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at)); }
__device__ __forceinline__ void lds(__nv_bfloat16& v, unsigned at) {
  uint16_t t;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(t) : "r"(at));
  v = __ushort_as_bfloat16(t);
}
__device__ __forceinline__ void lds2(float& a, float& b, unsigned at) {
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(b) : "r"(at));
}
__device__ __forceinline__ void lds2(double& a, double& b, unsigned at) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(a), "=d"(b) : "r"(at));
}
// raw slot bytes -> fragment, from shared memory
template <typename T, int SB>
__device__ __forceinline__ void frag_lds(Frag<typename AccOf<T>::type, SB / (int)sizeof(T)>& f, unsigned at) {
  if constexpr (sizeof(T) == 4 && SB == 16) {
    float a, b, c, d;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(a), "=f"(b), "=f"(c), "=f"(d) : "r"(at));
    f.p[0] = pack2(a, b);
    f.p[1] = pack2(c, d);
  } else if constexpr (sizeof(T) == 4 && SB == 8) {
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(f.p[0]) : "r"(at));
  } else {
    typename SlotWord<SB>::type w;
    lds(w, at);
    frag_unpack<T, SB>(f, w);
  }
}
// fragment -> V elements of T, one store of SB bytes
template <typename T, int SB>
__device__ __forceinline__ void frag_stg(void* p, const Frag<typename AccOf<T>::type, SB / (int)sizeof(T)>& f) {
  constexpr int V = SB / (int)sizeof(T);
  typename AccOf<T>::type x[V];
  f.get(x);
  union { typename SlotWord<SB>::type m; T t[V]; } u;
#pragma unroll
  for (int i = 0; i < V; ++i) u.t[i] = from_acc<T>(x[i]);
  *reinterpret_cast<typename SlotWord<SB>::type*>(p) = u.m;
}
// partial records: accumulators as they are
template <typename A, int V>
__device__ __forceinline__ void frag_save(A* p, const Frag<A, V>& f) {
  A x[V];
  f.get(x);
  if constexpr (V * sizeof(A) % 16 == 0) {
    union { uint4 m[V * sizeof(A) / 16]; A t[V]; } u;
#pragma unroll
    for (int i = 0; i < V; ++i) u.t[i] = x[i];
#pragma unroll
    for (int i = 0; i < (int)(V * sizeof(A) / 16); ++i) reinterpret_cast<uint4*>(p)[i] = u.m[i];
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) p[i] = x[i];
  }
}
template <typename A, int V>
__device__ __forceinline__ void frag_load_raw(Frag<A, V>& f, const A* p) {
  A x[V];
  if constexpr (V * sizeof(A) % 16 == 0) {
    union { uint4 m[V * sizeof(A) / 16]; A t[V]; } u;
#pragma unroll
    for (int i = 0; i < (int)(V * sizeof(A) / 16); ++i) u.m[i] = reinterpret_cast<const uint4*>(p)[i];
#pragma unroll
    for (int i = 0; i < V; ++i) x[i] = u.t[i];
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) x[i] = p[i];
  }
  f.set(x);
}

}  // namespace gk
