// alpha m in f64, rounded to nearest even, on the integer pipes: the normalised min-sum's
// scaling of a row's two magnitudes.
//
// GB300 has two FP64 lanes per SM and clock: a warp's FP64 instruction holds its quarter of the
// pipe for 64 cycles, in which the integer pipes issue 64 instructions.  A min-sum row of D edges
// takes 2 D additions and two of these products on the FP64 pipe; formed from four 32 x 32
// bit products (about 28 instructions), the products leave it to the additions.
//
// The 53-bit significands' product P lies in [2^104, 2^106); its upper 53 bits Q and the
// remainder below them decide the rounding, and Q added to the exponent field carries into
// it when rounding overflows.  Factors that are not positive and normal, or products near the
// ends of the exponent range, take the multiplication instruction.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SC_HD __host__ __device__ __forceinline__
#else
#define SC_HD inline
#endif

namespace cbk {

struct ScaleF64 {
  double alpha;
  uint32_t a0, a1;  // the low word and the high bits (with the leading one) of alpha's significand
  int32_t ea;       // alpha's exponent; 1 << 20 when the products take the instruction
};

SC_HD uint64_t sc_bits(double x) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
SC_HD double sc_from_bits(uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}

SC_HD ScaleF64 make_scale(double alpha) {
  const uint64_t b = sc_bits(alpha);
  const uint32_t hi = (uint32_t)(b >> 32), e = hi >> 20;  // the sign counts as a large exponent
  ScaleF64 s;
  s.alpha = alpha;
  s.a0 = (uint32_t)b;
  s.a1 = (hi & 0xfffffu) | 0x100000u;
  s.ea = e >= 1 && e <= 2046 ? (int32_t)e - 1023 : 1 << 20;
  return s;
}

// RN(alpha m) for m >= 0 (zero, subnormal and infinite included)
SC_HD double scaled(const ScaleF64& s, double m) {
  const uint64_t mb = sc_bits(m);
  const uint32_t lo = (uint32_t)mb, hi = (uint32_t)(mb >> 32), em = hi >> 20;
  // m normal and the product's exponent, less one and one more, normal too
  if (em - 1u >= 2046u || em + (uint32_t)s.ea - 2u >= 2043u) {
    if (mb == 0 && s.ea != 1 << 20) return m;
#if defined(__CUDA_ARCH__)
    return __dmul_rn(s.alpha, m);
#else
    return s.alpha * m;
#endif
  }
  const uint32_t mh = (hi & 0xfffffu) | 0x100000u;
  const uint64_t t0 = (uint64_t)lo * s.a0;
  const uint64_t t1 = (uint64_t)lo * s.a1 + (t0 >> 32);
  const uint64_t t2 = (uint64_t)mh * s.a0 + (uint32_t)t1;
  const uint64_t t3 = (uint64_t)mh * s.a1 + (t1 >> 32) + (t2 >> 32);  // P >> 64
  const uint32_t p1 = (uint32_t)t2, p0 = (uint32_t)t0;                // its lower words
  const uint32_t c = (uint32_t)(t3 >> 41), sh = 12 - c;               // P >= 2^105
  // Q = P >> (52 + c); the remainder's upper word, its last bit set for what lies below
  const uint64_t q = (t3 << sh) | (p1 >> (32 - sh));
  const uint32_t rem = (p1 << sh) | (p0 != 0);
  const uint64_t up = rem > 0x80000000u - ((uint32_t)q & 1u);
  const uint32_t er = em + (uint32_t)s.ea + c - 1u;  // Q's leading one adds the last 1
  return sc_from_bits(((uint64_t)er << 52) + q + up);
}

}  // namespace cbk
