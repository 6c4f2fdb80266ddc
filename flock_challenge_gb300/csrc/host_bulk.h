// Loops over GF(2^128) values on the host: the small sumcheck tails, openings
// and claim checks of the prover and the verifier.
#pragma once
#include <cstddef>
#include <vector>

#include "host_field.h"

namespace hf {

// sum_i a[i] b[i]
F dot(const F* a, const F* b, size_t n);
// out[i] = c a[i]
void scale(const F* a, F c, size_t n, F* out);
// v[j] = v[2j] + r (v[2j] + v[2j + 1]) for j < half
void bind_pairs(F* v, size_t half, F r);
// v[j] = v[j] + r (v[j] + v[j + half]) for j < half
void bind_halves(F* v, size_t half, F r);
// g1 = sum_j eq[j] a[2j+1] b[2j+1], gi = sum_j eq[j] (a[2j] + a[2j+1]) (b[2j] + b[2j+1])
void weighted_round(const F* a, const F* b, const F* eq, size_t pairs, F* g1, F* gi);
// e1 = sum_j w[j+half] g[j+half], ei = sum_j (w[j] + w[j+half]) (g[j] + g[j+half])
void halves_round(const F* w, const F* g, size_t half, F* e1, F* ei);
// t[i] = prod_k (bit k of i ? r[k] : 1 + r[k])
std::vector<F> eq_table(const std::vector<F>& r);
// Bit i of out[b] = bit b of v[i] (128 x 128).
std::vector<F> transpose128(const std::vector<F>& v);

}  // namespace hf
