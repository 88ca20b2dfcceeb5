// Extension-field vectors on the host (host_vec.cpp): AVX-512 when the CPU has it, else scalar.
#pragma once
#include <cstddef>
#include <cstdint>

#include "kb.cuh"

namespace wl {
bool hv_vectorised();  // which of the two runs
void hv_scale(const kb::ef* a, size_t n, const kb::ef& s, kb::ef* out);  // out[i] = a[i] s (out may be a)
void hv_mac(const kb::ef* a, size_t n, const kb::ef& s, kb::ef* out);    // out[i] += a[i] s
void hv_mac_base(const kb::ef& a, const uint32_t* f, size_t n, kb::ef* out);  // out[i] += a f[i]
kb::ef hv_dot(const kb::ef* a, const kb::ef* b, size_t n);               // sum a[i] b[i]
void hv_fold(kb::ef* t, size_t half, const kb::ef& r);                   // t[i] += r (t[i + half] - t[i])
// Round sums of the product of two tables: at 0, 1 and 2 of the leading variable.
void hv_pair_sums(const kb::ef* g, const kb::ef* e, size_t half, kb::ef* s);
void hv_powers(const kb::ef& x, size_t n, kb::ef* out);                  // out[i] = x^i
kb::ef hv_dot_base(const kb::ef* a, const uint32_t* f, size_t stride, size_t n);  // sum a[i] f[i stride]
}  // namespace wl
