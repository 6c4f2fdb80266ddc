// Host GF(2^128) loops of the transcript side (host_bulk.h). They are in a unit
// of the host compiler's own so that an Arm host's PMULL is inlined into them:
// a product through host_field.h's call costs 4.1 ns on a Grace core, one in
// these loops 3.2 ns, one of a dot product (reduced once) 1.9 ns; the 128 x 128
// bit transpose 1.1 us against about 45 us bit by bit.
#include "host_bulk.h"

#if FLOCK_HOST_PMULL
#include <arm_neon.h>
#endif

namespace hf {

namespace {

#if FLOCK_HOST_PMULL
inline void clmul_in(uint64_t a, uint64_t b, uint64_t& lo, uint64_t& hi) {
  const uint64x2_t v = vreinterpretq_u64_p128(vmull_p64((poly64_t)a, (poly64_t)b));
  lo = vgetq_lane_u64(v, 0);
  hi = vgetq_lane_u64(v, 1);
}
#else
inline void clmul_in(uint64_t a, uint64_t b, uint64_t& lo, uint64_t& hi) { clmul(a, b, lo, hi); }
#endif

// Unreduced sum of products: lo * lo at bit 0, hi * hi at bit 128, and the sum
// of all three Karatsuba products at bit 64.
struct Wide {
  uint64_t l0 = 0, l1 = 0, h0 = 0, h1 = 0, m0 = 0, m1 = 0;
  void add(F a, F b) {
    uint64_t x, y;
    clmul_in(a.lo, b.lo, x, y);
    l0 ^= x; l1 ^= y;
    clmul_in(a.hi, b.hi, x, y);
    h0 ^= x; h1 ^= y;
    clmul_in(a.lo ^ a.hi, b.lo ^ b.hi, x, y);
    m0 ^= x; m1 ^= y;
  }
  F value() const { return reduce(l0, l1 ^ m0 ^ l0 ^ h0, h0 ^ m1 ^ l1 ^ h1, h1); }
};

inline F mul(F a, F b) {
  Wide w;
  w.add(a, b);
  return w.value();
}

}  // namespace

F dot(const F* a, const F* b, size_t n) {
  Wide w;
  for (size_t i = 0; i < n; i++) w.add(a[i], b[i]);
  return w.value();
}

void scale(const F* a, F c, size_t n, F* out) {
  for (size_t i = 0; i < n; i++) out[i] = mul(a[i], c);
}

void bind_pairs(F* v, size_t half, F r) {
  for (size_t j = 0; j < half; j++) v[j] = v[2 * j] + mul(r, v[2 * j] + v[2 * j + 1]);
}

void bind_halves(F* v, size_t half, F r) {
  for (size_t j = 0; j < half; j++) v[j] = v[j] + mul(r, v[j + half] + v[j]);
}

void weighted_round(const F* a, const F* b, const F* eq, size_t pairs, F* g1, F* gi) {
  Wide s1, si;
  for (size_t j = 0; j < pairs; j++) {
    const F a0 = a[2 * j], a1 = a[2 * j + 1], b0 = b[2 * j], b1 = b[2 * j + 1];
    s1.add(eq[j], mul(a1, b1));
    si.add(eq[j], mul(a0 + a1, b0 + b1));
  }
  *g1 = s1.value();
  *gi = si.value();
}

void halves_round(const F* w, const F* g, size_t half, F* e1, F* ei) {
  Wide s1, si;
  for (size_t j = 0; j < half; j++) {
    s1.add(w[j + half], g[j + half]);
    si.add(w[j] + w[j + half], g[j] + g[j + half]);
  }
  *e1 = s1.value();
  *ei = si.value();
}

std::vector<F> eq_table(const std::vector<F>& r) {
  std::vector<F> t((size_t)1 << r.size());
  t[0] = F::one();
  for (size_t i = 0; i < r.size(); i++) {
    const size_t h = (size_t)1 << i;
    for (size_t j = 0; j < h; j++) {
      const F vr = mul(t[j], r[i]);
      t[j + h] = vr;
      t[j] += vr;
    }
  }
  return t;
}

std::vector<F> transpose128(const std::vector<F>& v) {
  // four 64x64 blocks, each by six rounds of masked swaps
  std::vector<F> u(128);
  for (int rb = 0; rb < 2; rb++)
    for (int cb = 0; cb < 2; cb++) {
      uint64_t x[64];
      for (int i = 0; i < 64; i++) x[i] = cb ? v[64 * rb + i].hi : v[64 * rb + i].lo;
      uint64_t mask = 0x00000000FFFFFFFFull;
      for (int s = 32; s; s >>= 1, mask ^= mask << s)
        for (int i = 0; i < 64; i = ((i | s) + 1) & ~s) {
          const uint64_t t = ((x[i] >> s) ^ x[i | s]) & mask;
          x[i] ^= t << s;
          x[i | s] ^= t;
        }
      for (int i = 0; i < 64; i++) (rb ? u[64 * cb + i].hi : u[64 * cb + i].lo) = x[i];
    }
  return u;
}

}  // namespace hf
