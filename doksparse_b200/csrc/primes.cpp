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

// Miller-Rabin with the seven bases that J. Sinclair found to decide every 64-bit number (2011, verified against the list of
// strong pseudoprimes to base 2 by J. Feitsma); n is odd and has no factor below 197.
bool is_prime(uint64_t n) {
  const Mont m(n);
  const uint64_t minus_one = n - m.one;
  const int s = __builtin_ctzll(n - 1);
  const uint64_t d = (n - 1) >> s;
  for (uint64_t base : {2ull, 325ull, 9375ull, 28178ull, 450775ull, 9780504ull, 1795265022ull}) {
    base %= n;
    if (base == 0) continue;
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
  if (n < 193 * 193) {                                  // the small primes decide
    for (uint64_t c = (n + 1) | 1;; c += 2) {
      bool prime = true;
      for (uint16_t p : SMALL) {
        if ((uint32_t)p * p > c) break;
        if (c % p == 0) { prime = false; break; }
      }
      if (prime) return c;
    }
  }
  for (uint64_t first = (n + 1) | 1; first > n; first += 2 * 256) {       // 256 odd candidates, those with a small factor struck out
    bool struck[256] = {};
    for (uint16_t p : SMALL) {
      // first + 2 i = 0 (mod p): i = -first / 2 = (p - first % p) * (p + 1) / 2
      for (uint32_t i = (uint32_t)((p - first % p) % p * ((p + 1u) / 2) % p); i < 256; i += p) struck[i] = true;
    }
    for (uint32_t i = 0; i < 256; i++) {
      const uint64_t c = first + 2 * i;
      if (c < first) return 0;                          // above the largest 64-bit prime
      if (!struck[i] && is_prime(c)) return c;
    }
  }
  return 0;
}
