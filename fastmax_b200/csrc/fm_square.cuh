// The polynomial of the scores as a square and a rest, for kernels that need both f and f'.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#include "fm_common.cuh"

namespace fm {

// f(s) = a0 + a1 c s + a2 (c s)^2 = t^2 + rest with t = root c s + shift, and f'(s) = 2 root c t, where c is the heads' scale.  A
// pair of scores costs t = fma(s, root c, shift), P = fma(t, t, rest), E' = t (w - dvec): four packed operations where the
// polynomial and its derivative cost five.  P is what is multiplied, so it is rounded to bf16 where f lies; 2 root c multiplies
// grad_k's accumulator in the end.  (With a2 c^2 left out of P as well, it was rounded where f / (a2 c^2) lies: the error of
// grad_v was 2.75e-3 to 3.07e-3, by the mantissa of a2 c^2, instead of 2.75e-3, and
// inputs 1e10 apart overflowed.  Then t is an addition: the wide kernel took 60.0 us instead of 62.3 for 168 row tiles of 3500
// unmasked columns, 154 / 154 for 1176 causal ones, 252.7 / 249.7 for 1176 unmasked ones.)
// shift and rest stand twice in 64 bits, as packed operations take them from a kernel's parameters, without a register.
struct Square {
  uint64_t shift, rest;
  float root;
};

// Whether t^2 and the rest cancel by less than a factor of 16 (four of float32's 24 bits), which does not depend on the scale: a2 has
// to be positive and a1^2 / (4 a2) at most 16 |a0|.  Else the polynomial is evaluated as it stands.  Error of grad_v, square /
// polynomial, at a0 = a1 = 1 (the line lies at a2 = 1/64): 1e-5 3.3e-3 / 2.8e-3, 1e-6 1.2e-2, 1e-7 9e-2.
inline bool square_form(float a0, float a1, float a2, Square* sq) {
  *sq = Square{};
  const double b = a1, a = a2, lift = b * b / (4.0 * a);
  if (!(a > 0.0) || !(lift <= 16.0 * std::fabs((double)a0)) || !std::isfinite(a) || !std::isfinite(a0)) return false;
  const double root = std::sqrt(a);
  const auto twice = [](double x) {
    const float f = (float)x;
    uint32_t bits;
    std::memcpy(&bits, &f, sizeof bits);
    return (uint64_t)bits << 32 | bits;
  };
  *sq = {twice(b / (2.0 * root)), twice(a0 - lift), (float)root};
  return true;
}

}  // namespace fm
