// Host-side helpers of the library: the random generator the reference
// draws from, its Gaussian transform, and the per-particle constants the
// reference computes on the host.
#pragma once
#include <cmath>
#include <cstdint>
#include <random>
#include <vector>

namespace mdsc {

// The reference's generator is GSL's MT19937 (v25/classes.hpp:150-181,
// v25/main.cpp:209-211): init_genrand seeding with seed 0 mapped to 4357,
// uniform = 32-bit output / 2^32.  std::mt19937 implements the same
// generator and seeding.
class Mt19937 {
 public:
  // MT19937 (Matsumoto & Nishimura, ACM TOMACS 8(1), 1998) with GSL's state
  // layout and seeding, so that a state read from the reference's generator
  // files continues the same sequence: 624 words and the position of the
  // next word; a seed of 0 means 4357 (gsl_rng_set).
  static constexpr int kN = 624;
  explicit Mt19937(unsigned long seed = 1) { seed_with(seed); }
  void seed_with(unsigned long seed) {
    uint32_t s = (uint32_t)(seed & 0xffffffffUL);
    if (s == 0) s = 4357u;
    mt_[0] = s;
    for (int i = 1; i < kN; ++i) mt_[i] = 1812433253u * (mt_[i - 1] ^ (mt_[i - 1] >> 30)) + (uint32_t)i;
    mti_ = kN;
  }
  uint32_t next() {
    if (mti_ >= kN) refill();
    uint32_t y = mt_[mti_++];
    y ^= y >> 11;
    y ^= (y << 7) & 0x9d2c5680u;
    y ^= (y << 15) & 0xefc60000u;
    y ^= y >> 18;
    return y;
  }
  double uniform() { return (double)next() / 4294967296.0; }
  void discard(unsigned long long n) {
    for (unsigned long long k = 0; k < n; ++k) next();
  }
  void get_state(uint32_t* mt, int* mti) const {
    for (int i = 0; i < kN; ++i) mt[i] = mt_[i];
    *mti = mti_;
  }
  bool set_state(const uint32_t* mt, int mti) {
    if (mti < 0 || mti > kN) return false;
    for (int i = 0; i < kN; ++i) mt_[i] = mt[i];
    mti_ = mti;
    return true;
  }

 private:
  void refill() {
    constexpr uint32_t kUpper = 0x80000000u, kLower = 0x7fffffffu, kMatrix = 0x9908b0dfu;
    constexpr int kM = 397;
    auto turn = [&](int k, int next, int from) {
      const uint32_t y = (mt_[k] & kUpper) | (mt_[next] & kLower);
      mt_[k] = mt_[from] ^ (y >> 1) ^ ((0u - (y & 1)) & kMatrix);
    };
    for (int k = 0; k < kN - kM; ++k) turn(k, k + 1, k + kM);
    for (int k = kN - kM; k < kN - 1; ++k) turn(k, k + 1, k + kM - kN);
    turn(kN - 1, 0, kM - 1);
    mti_ = 0;
  }
  uint32_t mt_[kN];
  int mti_ = kN;
};

// gauss(1, rnd1, rnd2): Box-Muller as v25/functions.cpp:1149-1156 does it
inline void box_muller(double& rnd1, double& rnd2) {
  const double a = std::sqrt(-2 * std::log(rnd1)) * std::cos(2 * M_PI * rnd2);
  const double b = std::sqrt(-2 * std::log(rnd1)) * std::sin(2 * M_PI * rnd2);
  rnd1 = a;
  rnd2 = b;
}

// Spherocyl::set_inertia, v25/classes.cpp:175-185
inline void spherocyl_inertia(double L, double D, double mass, double I[3]) {
  const double R = D / 2, Rsq = R * R, Rft = Rsq * Rsq, Lsq = L * L;
  const double vol = M_PI * Rsq * (L + 3. * R / 4);
  const double mdens = mass / vol;
  I[0] = mdens * M_PI * (Lsq * L * Rsq / 12 + Lsq * Rsq * R / 3 + L * Rft / 4 + 8. * Rft * R / 15);
  I[1] = I[0];
  I[2] = mdens * M_PI * (L * Rft / 2 + 8. * Rft * R / 15);
}

// A set of the integers 0..n-1 that shrinks: the k-th smallest that remains,
// and removal.  Bits in words of 64; per 16 words the running counts of the
// bits left, 16-bit numbers four to a word, and per 16 of those groups the
// same again, so a lookup is three steps without branches (each counts the
// fields not above k, by the parallel comparison of broadword selection,
// S. Vigna, "Broadword implementation of rank/select queries", 2008) after a
// pass over n / 16384 totals, and a removal takes one from the running counts
// behind it.  32,768 integers drawn and removed one by one, on the host of a
// GB300: a binary indexed tree 90 ns apiece, this 50.
class RankSet {
 public:
  explicit RankSet(int n)
      : bits_((size_t)((n >> 14) + 1) * 256, 0), in16_(bits_.size() / 16), in256_(bits_.size() / 256), total_(in256_.size(), 0) {
    for (int w = 0; w < (n + 63) / 64; ++w) bits_[w] = n - 64 * w >= 64 ? ~0ull : (1ull << (n - 64 * w)) - 1;
    for (size_t b = 0; b < total_.size(); ++b) {
      int outer = 0;
      for (int g = 0; g < 16; ++g) {
        int inner = 0;
        for (int w = 0; w < 16; ++w) {
          inner += __builtin_popcountll(bits_[256 * b + 16 * g + w]);
          in16_[16 * b + g].f[w >> 2] |= (uint64_t)inner << (16 * (w & 3));
        }
        outer += inner;
        in256_[b].f[g >> 2] |= (uint64_t)outer << (16 * (g & 3));
      }
      total_[b] = outer + (b ? total_[b - 1] : 0);
    }
  }
  void remove(int i) {
    bits_[i >> 6] &= ~(1ull << (i & 63));
    in16_[i >> 10].take(i >> 6 & 15);
    in256_[i >> 14].take(i >> 10 & 15);
    const int b = i >> 14, m = (int)total_.size();
    for (int q = 0; q < m; ++q) total_[q] -= q >= b;
  }
  // the k-th (0-based) remaining integer; there are more than k
  int kth(int k) const {
    int b = 0;
    const int m = (int)total_.size();
    for (int q = 0; q < m; ++q) b += total_[q] <= k;
    k -= b ? total_[b - 1] : 0;
    const int g = 16 * b + in256_[b].find(k);
    const int w = 16 * g + in16_[g].find(k);
    return 64 * w + select(bits_[w], k);
  }

 private:
  static constexpr uint64_t kOnes = 0x0001000100010001ull, kHigh = kOnes << 15;
  // running counts of 16 parts (each below 2^15)
  struct Counts {
    uint64_t f[4] = {0, 0, 0, 0};
    // the part that holds the k-th element, k reduced to its place there
    int find(int& k) const {
      const uint64_t kk = (uint64_t)k * kOnes | kHigh;
      uint64_t le = 0;  // per field: how many of the four counts there are not above k
      for (int q = 0; q < 4; ++q) le += ((kk - f[q]) & kHigh) >> 15;
      const int part = (int)(le * kOnes >> 48);
      const int q = part - 1;
      k -= part ? (int)(f[q >> 2] >> (16 * (q & 3)) & 0xffff) : 0;
      return part;
    }
    void take(int part) {
      for (int q = 0; q < 4; ++q) {
        const int from = part - 4 * q;  // fields from here on lose one
        f[q] -= from <= 0 ? kOnes : (from > 3 ? 0 : kOnes << (16 * from));
      }
    }
  };
  // position of the k-th set bit of x
  static int select(uint64_t x, int k) {
    constexpr uint64_t L = 0x0101010101010101ull, H = L << 7;
    uint64_t s = x - (x >> 1 & 0x5555555555555555ull);
    s = (s & 0x3333333333333333ull) + (s >> 2 & 0x3333333333333333ull);
    s = ((s + (s >> 4)) & 0x0f0f0f0f0f0f0f0full) * L;  // running counts of the bytes
    const int b = 8 * (int)((((((uint64_t)k * L | H) - s) & H) >> 7) * L >> 56);  // the byte that holds it, in bits
    k -= b ? (int)(s >> (b - 8) & 0xff) : 0;
    unsigned y = (unsigned)(x >> b & 0xff);
    int pos = b, c = (int)(0x4332322132212110ull >> (4 * (y & 15)) & 7), up = -(k >= c);  // bits of the low nibble
    pos += up & 4, k -= up & c, y >>= up & 4;
    c = (int)((y & 1) + (y >> 1 & 1)), up = -(k >= c);
    pos += up & 2, k -= up & c, y >>= up & 2;
    return pos + (k >= (int)(y & 1));
  }
  std::vector<uint64_t> bits_;
  std::vector<Counts> in16_, in256_;
  std::vector<int> total_;
};

}  // namespace mdsc
