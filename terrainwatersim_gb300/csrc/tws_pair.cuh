// tws_pair.cuh -- two cells at a time: packed f32x2 arithmetic shared by the
// kernels that keep a lane's adjacent cells together (row sweep, mesh).
#pragma once
#include "tws_device.cuh"

namespace tws {

// A lane's two cells as one packed f32x2 operand, kept in a 64-bit register (its
// low half is the lane's first column): values that stay packed from one row to
// the next then cost no moves to line their halves up.
typedef unsigned long long pair_t;
__device__ __forceinline__ pair_t pk(float x, float y) {
  pair_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 un(pair_t p) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p));
  return r;
}
__device__ __forceinline__ pair_t add2(pair_t a, pair_t b) {
  pair_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ pair_t sub2(pair_t a, pair_t b) {
  pair_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// a * b rounded, with -0 added: the product's own bits (x + -0 = x for every x,
// -0 included), as a fused multiply-add that no later sum can be contracted
// with.  `nz` must reach the kernel as data (StepArgs::neg_zero).
__device__ __forceinline__ pair_t prod2(pair_t a, pair_t b, pair_t nz) {
  pair_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(nz));
  return r;
}
__device__ __forceinline__ pair_t max0p(pair_t v) {
  const float2 f = un(v);
  return pk(max0_fast(f.x), max0_fast(f.y));
}

// d / t per half, rounded to nearest, for t up to kDivMaxT and d in
// [kDivMinD, t): nothing on the way then overflows or leaves the normal range.
// Markstein's division (IBM J. Res. Dev. 34, 1990): a reciprocal refined to
// its correct rounding with one Newton step in fused arithmetic, a quotient
// within an ulp, and the exact remainder's correction.  The tests compare it with
// the correctly rounded quotient over that range, at its limits and for the
// quotients closest to a rounding boundary (tests/test_division_gpu.py).
// `nt` is -t.
constexpr float kDivMinD = 0x1p-100f, kDivMaxT = 0x1p20f;
__device__ __forceinline__ pair_t fma2(pair_t a, pair_t b, pair_t c) {
  pair_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ pair_t div2(pair_t d, pair_t t, pair_t nt) {
  const float2 tv = un(t);
  float y0, y1;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(tv.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y1) : "f"(tv.y));
  pair_t y = pk(y0, y1);
  y = fma2(fma2(nt, y, pk(1.0f, 1.0f)), y, y);
  pair_t q;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(q) : "l"(d), "l"(y));
  return fma2(fma2(nt, q, d), y, q);
}

// A lane's four cells: columns 0, 1 and 2, 3.
struct Quad {
  pair_t p[2];
};
#define TWS_QUAD_OP(name, op)                                     \
  __device__ __forceinline__ Quad name(const Quad& a, const Quad& b) { \
    return Quad{{op(a.p[0], b.p[0]), op(a.p[1], b.p[1])}};          \
  }
TWS_QUAD_OP(add4, add2)
TWS_QUAD_OP(sub4, sub2)
#undef TWS_QUAD_OP
__device__ __forceinline__ Quad prod4(const Quad& a, pair_t b, pair_t nz) {
  return Quad{{prod2(a.p[0], b, nz), prod2(a.p[1], b, nz)}};
}
__device__ __forceinline__ Quad prod4(const Quad& a, const Quad& b, pair_t nz) {
  return Quad{{prod2(a.p[0], b.p[0], nz), prod2(a.p[1], b.p[1], nz)}};
}
__device__ __forceinline__ Quad max0q(const Quad& v) {
  return Quad{{max0p(v.p[0]), max0p(v.p[1])}};
}
__device__ __forceinline__ float4 un4(const Quad& v) {
  const float2 l = un(v.p[0]), h = un(v.p[1]);
  return make_float4(l.x, l.y, h.x, h.y);
}
__device__ __forceinline__ Quad pk4(float x, float y, float z, float w) {
  return Quad{{pk(x, y), pk(z, w)}};
}
__device__ __forceinline__ Quad load_quad(const unsigned char* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return Quad{{v.x, v.y}};
}
__device__ __forceinline__ void store_quad(unsigned char* p, const Quad& v) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.p[0], v.p[1]);
}
// One 32-byte store (whole sectors; the address is a multiple of 32).
__device__ __forceinline__ void store32(void* p, float a, float b, float c, float d, float e,
                                        float f, float g, float h) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a), "f"(b),
               "f"(c), "f"(d), "f"(e), "f"(f), "f"(g), "f"(h)
               : "memory");
}

// The four outflow channels (+x, -x, +y, -y) of a lane's four cells.
struct Flux4 {
  Quad x, y, z, w;
};

// The factors that keep the outflows `out` (their sum) of four cells within
// their depths d (flowUpdate.comp:55-62): d / total where total = out * c > d,
// else 1, which leaves a cell's bits.  d / total of a dry cell (d = +-0) is d
// itself, so most of a shore needs no division.  cc2 = (c, c), ncc2 = (-c, -c).
__device__ __forceinline__ Quad outflow_factors(const Quad& out, const Quad& dq, pair_t cc2,
                                                pair_t ncc2, pair_t nz) {
  const Quad tq = prod4(out, cc2, nz);
  const float4 t4 = un4(tq), d4 = un4(dq);
  const float t[4] = {t4.x, t4.y, t4.z, t4.w}, d[4] = {d4.x, d4.y, d4.z, d4.w};
  float f[4];
  bool div[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const bool over = t[c] > d[c];
    f[c] = over ? d[c] : 1.0f;
    div[c] = over & (d[c] != 0.0f);
  }
  if (div[0] | div[1] | div[2] | div[3]) {
    bool far = fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3])) > kDivMaxT;
#pragma unroll
    for (int c = 0; c < 4; ++c) far |= div[c] & (d[c] < kDivMinD);
    if (!far) {
      const Quad nt = prod4(out, ncc2, nz);
      const float2 lo = un(div2(dq.p[0], tq.p[0], nt.p[0]));
      const float2 hi = un(div2(dq.p[1], tq.p[1], nt.p[1]));
      f[0] = div[0] ? lo.x : f[0];
      f[1] = div[1] ? lo.y : f[1];
      f[2] = div[2] ? hi.x : f[2];
      f[3] = div[3] ? hi.y : f[3];
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (div[c]) f[c] = fdiv(d[c], t[c]);
    }
  }
  return pk4(f[0], f[1], f[2], f[3]);
}

// The same for two cells.
__device__ __forceinline__ pair_t outflow_factors2(pair_t out, pair_t d2, pair_t cc2, pair_t ncc2,
                                                   pair_t nz) {
  const pair_t t2 = prod2(out, cc2, nz);
  const float2 t = un(t2), d = un(d2);
  const bool over0 = t.x > d.x, over1 = t.y > d.y;
  float f0 = over0 ? d.x : 1.0f, f1 = over1 ? d.y : 1.0f;
  const bool div0 = over0 & (d.x != 0.0f), div1 = over1 & (d.y != 0.0f);
  if (div0 | div1) {
    const bool far = (fmaxf(t.x, t.y) > kDivMaxT) | (div0 & (d.x < kDivMinD)) |
                     (div1 & (d.y < kDivMinD));
    if (!far) {
      const float2 q = un(div2(d2, t2, prod2(out, ncc2, nz)));
      f0 = div0 ? q.x : f0;
      f1 = div1 ? q.y : f1;
    } else {
      if (div0) f0 = fdiv(d.x, t.x);
      if (div1) f1 = fdiv(d.y, t.y);
    }
  }
  return pk(f0, f1);
}

// add_rain on two cells side by side, without a branch: TwoSum's sum and error,
// then one ulp toward d + rate with the probability that makes it exact.  h0 and
// h1 are the cells' rain_hash32(x ^ rain_hash32(y)); a cell that is not in the
// disk keeps its depth.
__device__ __forceinline__ pair_t rain2(pair_t d2, float rate, uint32_t h0, uint32_t h1, bool in0,
                                        bool in1) {
  const pair_t rate2 = pk(rate, rate);
  const pair_t s2 = add2(d2, rate2), bp = sub2(s2, d2);
  const float2 e = un(add2(sub2(d2, sub2(s2, bp)), sub2(rate2, bp)));
  const float2 d = un(d2), s = un(s2);
  auto pick = [&](uint32_t hc, float dc, float sc, float ec, bool in) {
    const uint32_t sb = __float_as_uint(sc);
    const float next = __uint_as_float(((sc > 0.0f) == (ec > 0.0f)) ? sb + 1u : sb - 1u);
    const uint32_t h = rain_hash32(__float_as_uint(dc) ^ hc);
    const float u = fmul(__uint2float_rn(h >> 8), 0x1p-24f);
    const float o = fmul(u, fabsf(fsub(next, sc))) < fabsf(ec) ? next : sc;
    return in ? o : dc;
  };
  return pk(pick(h0, d.x, s.x, e.x, in0), pick(h1, d.y, s.y, e.y, in1));
}

}  // namespace tws
