// Host check of the extension-field vectors (host_vec.cpp) against the scalar operations of
// kb.cuh, for random and largest coordinates and every length from 0. Built by tests/test_host_vec.py.
#include <cstdio>
#include <random>
#include <vector>

#include "host_vec.h"
using namespace wl;
using kb::ef;

int main() {
  std::mt19937_64 g(3);
  long bad = 0;
  auto pick = [&](int mode) {
    ef e;
    for (uint32_t& c : e.c) c = mode == 0 ? kb::P - 1 : mode == 1 ? (g() & 1 ? kb::P - 1 : 0) : uint32_t(g() % kb::P);
    return e;
  };
  auto eq = [&](const ef& a, const ef& b) { bad += !kb::ef_eq(a, b); };
  for (int mode = 0; mode < 6; mode++)
    for (size_t n : {size_t(0), size_t(1), size_t(2), size_t(3), size_t(4), size_t(5), size_t(7), size_t(46), size_t(64)}) {
      std::vector<ef> a(2 * n + 1), b(2 * n + 1);
      std::vector<uint32_t> f(3 * n + 1);
      for (auto& x : a) x = pick(mode);
      for (auto& x : b) x = pick(mode);
      for (auto& x : f) x = mode == 0 ? kb::P - 1 : uint32_t(g() % kb::P);
      const ef s = pick(mode);
      std::vector<ef> o(n + 1);
      hv_scale(a.data(), n, s, o.data());
      for (size_t i = 0; i < n; i++) eq(o[i], kb::ef_mul(a[i], s));
      std::vector<ef> m(b.begin(), b.begin() + n);
      hv_mac(a.data(), n, s, m.data());
      for (size_t i = 0; i < n; i++) eq(m[i], kb::ef_add(b[i], kb::ef_mul(a[i], s)));
      std::vector<ef> mb(b.begin(), b.begin() + n);
      hv_mac_base(s, f.data(), n, mb.data());
      for (size_t i = 0; i < n; i++) eq(mb[i], kb::ef_add(b[i], kb::ef_mul_f(s, f[i])));
      ef d = kb::ef_zero(), db = d, t[3] = {d, d, d}, u[3], v = kb::ef_one();
      for (size_t i = 0; i < n; i++) d = kb::ef_add(d, kb::ef_mul(a[i], b[i])), db = kb::ef_add(db, kb::ef_mul_f(a[i], f[3 * i]));
      eq(hv_dot(a.data(), b.data(), n), d);
      eq(hv_dot_base(a.data(), f.data(), 3, n), db);
      for (size_t i = 0; i < n; i++) {
        const ef ah = kb::ef_sub(kb::ef_add(a[i + n], a[i + n]), a[i]), bh = kb::ef_sub(kb::ef_add(b[i + n], b[i + n]), b[i]);
        t[0] = kb::ef_add(t[0], kb::ef_mul(a[i], b[i]));
        t[1] = kb::ef_add(t[1], kb::ef_mul(a[i + n], b[i + n]));
        t[2] = kb::ef_add(t[2], kb::ef_mul(ah, bh));
      }
      hv_pair_sums(a.data(), b.data(), n, u);
      for (int z = 0; z < 3; z++) eq(u[z], t[z]);
      std::vector<ef> c = a;
      hv_fold(c.data(), n, s);
      for (size_t i = 0; i < n; i++) eq(c[i], kb::ef_lerp(a[i], a[i + n], s));
      hv_powers(s, n, o.data());
      for (size_t i = 0; i < n; i++, v = kb::ef_mul(v, s)) eq(o[i], v);
    }
  std::printf("wrong values: %ld\n", bad);
  return bad != 0;
}
