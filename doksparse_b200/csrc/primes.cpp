// Next prime above a 64-bit number, on the host: every new table draws one prime near its size and one near 2^60 per
// key element, and finding them in Python (16 us and 218 us each) took longer than building a small table.
#include <stdint.h>
#include <initializer_list>
#include "../../include/doksparse.h"

typedef unsigned __int128 u128;

namespace {

// Montgomery arithmetic modulo an odd n (P. L. Montgomery, "Modular multiplication without trial division", 1985).
struct Mont {
  uint64_t n, neg_inv, one, r2;
  explicit Mont(uint64_t m) : n(m) {
    uint64_t inv = m;                                   // Newton: each step doubles the correct low bits (3 to start with)
    for (int i = 0; i < 5; i++) inv *= 2 - m * inv;
    neg_inv = 0 - inv;
    one = (uint64_t)(((u128)1 << 64) % m);
    r2 = (uint64_t)((u128)one * one % m);
  }
  uint64_t reduce(u128 t) const {
    const uint64_t q = (uint64_t)t * neg_inv;
    const u128 qn = (u128)q * n;
    const bool carry_low = (uint64_t)t != 0;            // the low halves cancel to 0 with a carry unless both are 0
    const u128 hi = (u128)(uint64_t)(t >> 64) + (uint64_t)(qn >> 64) + carry_low;
    return (uint64_t)(hi >= n ? hi - n : hi);
  }
  uint64_t mul(uint64_t a, uint64_t b) const { return reduce((u128)a * b); }
};

const uint16_t SMALL[] = {3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67, 71, 73, 79, 83, 89, 97,
                          101, 103, 107, 109, 113, 127, 131, 137, 139, 149, 151, 157, 163, 167, 173, 179, 181, 191, 193};

// Miller-Rabin; the first twelve primes as bases decide every n below 3.3e24 (J. Sorenson and J. Webster, "Strong
// pseudoprimes to twelve prime bases", 2015), so this is exact for 64-bit numbers.
bool is_prime(uint64_t n) {
  if (n < 2) return false;
  if (n % 2 == 0) return n == 2;
  for (uint16_t p : SMALL) if (n % p == 0) return n == p;
  if (n < 193ull * 193ull) return true;
  const Mont m(n);
  const uint64_t minus_one = n - m.one;
  const int s = __builtin_ctzll(n - 1);
  const uint64_t d = (n - 1) >> s;
  for (uint64_t base : {2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37}) {
    const uint64_t b = m.mul(base, m.r2);
    uint64_t x = m.one;
    for (int i = 63 - __builtin_clzll(d); i >= 0; i--) {
      x = m.mul(x, x);
      if ((d >> i) & 1) x = m.mul(x, b);
    }
    if (x == m.one || x == minus_one) continue;
    bool composite = true;
    for (int r = 1; r < s && composite; r++) {
      x = m.mul(x, x);
      if (x == minus_one) composite = false;
    }
    if (composite) return false;
  }
  return true;
}

}  // namespace

extern "C" uint64_t dok_next_prime(uint64_t n) {
  if (n < 2) return 2;
  for (uint64_t c = (n + 1) | 1; c > n; c += 2) if (is_prime(c)) return c;
  return 0;                                             // above the largest 64-bit prime
}
