// Host check of the tensor-core Poseidon2 (whirlaway_b200/csrc/poseidon2_tc.cuh compiles for the
// host too, with the matrix products restated over the same byte tables): every word of the
// permutation against p2_permute_fd, and the ranges that the fp64 and 64-bit steps rely on, for
// random, zero and largest round constants and states. Built and run by tests/test_poseidon2_tc.py.
#include <algorithm>
#include <cstdio>
#include <random>

#include "poseidon2_tc.cuh"
using namespace kb;

static long bad = 0, range = 0;

template <int W>
const P2TcTab<W>& tab() {
  static const P2TcTab<W> t = p2lin::make_tab<W>();
  return t;
}
// Accumulators of A (one row of words) times the B operand of n rows at table word `base`.
template <int W>
void product(int base, int ks, int n_rows, const uint32_t* words, uint32_t* acc) {
  for (int n = 0; n < n_rows; n++)
    for (int j = 0; j < 8 * ks; j++) {
      const uint32_t b = tab<W>().w[base + ((j >> 2) * n_rows + n) * 4 + (j & 3)];
      for (int a = 0; a < 4; a++) acc[n] += ((words[j] >> (8 * a)) & 255) * ((b >> (8 * a)) & 255);
    }
}
template <int W>
uint32_t sbox(double zb, uint32_t k) {
  if (zb < 4503599627370496.0 || zb >= 9007199254740992.0 || std::fabs(zb - fb_magic<W>()) >= 137438953472.0) range++;
  const uint32_t r0 = fb_sbox<W>(zb, 0), r = fb_sbox<W>(zb, k);
  const int64_t t = int64_t(r0) + int32_t(k);  // a word, before and after the share is added
  if (r0 < P / 2 - P / 64 || r0 > P + P / 2 + P / 64 || t < 0 || t >= 2 * int64_t(P) || uint32_t(t) != r) range++;
  return r;
}
template <int W>
void permute(const uint32_t* s, const P2ConstsTc<W>& c, uint32_t* out) {
  using T = P2TcTab<W>;
  double z[W];
  uint32_t w[W], words[8 * (T::KS + T::KX)] = {};
  for (int i = 0; i < W; i++) w[i] = s[i] + c.in[i];
  for (int r = 0; r < 4; r++) {
    fb_mds<W>(w, z);
    for (int i = 0; i < W; i++) w[i] = sbox<W>(z[i], c.init[r][i]);
  }
  fb_mds<W>(w, z);
  for (int i = 0; i < W; i++) {
    words[i] = fb_word<W>(z[i]);
    if (words[i] >= 2 * uint64_t(P)) range++;
  }
  uint32_t y[T::N1] = {};
  product<W>(0, T::KS, T::N1, words, y);
  int32_t x[T::RP];
  x[0] = part_cube(kb::umin(words[0], words[0] - P) + c.rc0);
  auto group = [&](int g) {  // the group's x words, and their products into the later outputs
    for (int j = 0; j < 8; j++) words[W + 8 * g + j] = 8 * g + j < T::RP ? uint32_t(x[8 * g + j]) + P : 0;
    uint32_t a[T::N3] = {};
    product<W>(4 * (T::E1 + T::E2), 1, T::N3, words + W + 8 * g, a);
    for (int n = 32 * (g + 1); n < T::N1; n++) y[n] += a[n - 32 * (g + 1)];
  };
  part_chain<W, 0, 0, 8>(y, c, x);
  group(0);
  part_chain<W, 8, 0, 8>(y + 32, c, x + 8);
  group(1);
  part_chain<W, 16, 0, T::O1 - 16>(y + 64, c, x + 16);
  group(2);
  for (int j = 0; j < T::RP; j++)
    if (std::fabs(double(x[j])) > 0.51 * P) range++;
  uint32_t acc[T::N2] = {};
  product<W>(4 * T::E1, T::KS + T::KX, T::N2, words, acc);
  for (uint32_t a : acc) range += a >= (1u << 24);
  for (uint32_t a : y) range += a >= (1u << 24);
  for (int i = 0; i < W; i++)
    w[i] = fb_sbox_word(limb_word(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3], c.mid[i]), c.term[0][i]);
  for (int r = 1; r < 4; r++) {
    fb_mds<W>(w, z);
    for (int i = 0; i < W; i++) w[i] = sbox<W>(z[i], c.term[r][i]);
  }
  fb_mds<W>(w, z);
  for (int i = 0; i < W; i++) {
    const uint32_t q = fb_word<W>(z[i]);
    out[i] = kb::umin(q, q - P);
  }
}
template <int W>
void check(std::mt19937_64& g) {
  for (int t = 0; t < 12; t++) {
    P2Consts<W> m;
    auto pick = [&] { return t == 0 ? 0u : t == 1 ? P - 1 : uint32_t(g() % P); };
    for (int i = 0; i < 4 * W; i++) m.ext_init[i] = pick(), m.ext_term[i] = pick();
    for (uint32_t& v : m.internal) v = pick();
    const P2ConstsTc<W> c = p2_consts_tc(m);
    const P2ConstsFd<W> ref = p2_consts_fd(m);
    for (int it = 0; it < 1500; it++) {
      uint32_t s[W], r[W], o[W];
      for (int i = 0; i < W; i++)
        s[i] = it == 0 ? 0 : it == 1 ? P - 1 : it == 2 ? (i & 1 ? P - 1 : 0) : it < 10 ? (g() & 1 ? 0 : P - 1) : g() % P;
      std::copy(s, s + W, r);
      p2_permute_fd<W>(r, ref);
      if (it % 7 == 0)
        for (uint32_t& v : s) v = v ? v : P;  // p stands for zero
      permute<W>(s, c, o);
      for (int i = 0; i < W; i++) bad += o[i] != r[i];
    }
  }
}
int main() {
  std::mt19937_64 g(5);
  check<16>(g);
  check<24>(g);
  std::printf("wrong words %ld, out of range %ld\n", bad, range);
  return bad || range;
}
