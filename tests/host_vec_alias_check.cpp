// Host check of the extension-field vectors (host_vec.cpp) where arguments overlap as they do in the
// prover: a scaled copy in place or behind its source, a factor that is an entry of the vector, a
// fold in place. argv[1]: 1 when the vector forms are to run, 0 for the scalar ones. Built by
// tests/test_host_vec_forms.py.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "host_vec.h"
using namespace wl;
using kb::ef;

int main(int argc, char** argv) {
  if (argc < 2 || hv_vectorised() != (std::atoi(argv[1]) != 0)) {
    std::printf("the other form runs\n");
    return 2;
  }
  std::mt19937_64 g(5);
  long bad = 0;
  for (size_t n : {size_t(1), size_t(2), size_t(5), size_t(8), size_t(31)})
    for (int mode = 0; mode < 4; mode++) {
      std::vector<ef> a(2 * n);
      for (ef& e : a)
        for (uint32_t& c : e.c) c = mode == 0 ? kb::P - 1 : mode == 1 ? (g() & 1 ? kb::P - 1 : 0) : uint32_t(g() % kb::P);
      const ef s = a[n / 2];
      std::vector<ef> want(n);
      for (size_t i = 0; i < n; i++) want[i] = kb::ef_mul(a[i], s);
      std::vector<ef> v = a;
      hv_scale(v.data(), n, v[n / 2], v.data());  // in place, the factor among the entries
      for (size_t i = 0; i < n; i++) bad += !kb::ef_eq(v[i], want[i]);
      v = a;
      hv_scale(v.data(), n, s, v.data() + n);  // behind its source
      for (size_t i = 0; i < n; i++) bad += !kb::ef_eq(v[n + i], want[i]) || !kb::ef_eq(v[i], a[i]);
      v = a;
      hv_mac(v.data(), n, v[n], v.data() + n);  // the factor among the sums
      for (size_t i = 0; i < n; i++) bad += !kb::ef_eq(v[n + i], kb::ef_add(a[n + i], kb::ef_mul(a[i], a[n])));
      v = a;
      hv_fold(v.data(), n, v[0]);
      for (size_t i = 0; i < n; i++) bad += !kb::ef_eq(v[i], kb::ef_lerp(a[i], a[n + i], a[0]));
    }
  std::printf("wrong values: %ld\n", bad);
  return bad != 0;
}
