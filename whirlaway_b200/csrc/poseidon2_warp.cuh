// One Poseidon2-16 permutation in one warp, for the places where a single permutation's latency
// is the cost: the device transcript (finish.cuh) and the narrow top of a Merkle tree. Word
// (lane & 15) of the state is in lanes i and i + 16; words are canonical (not Montgomery).
//
// Full rounds: the S-box and the biased fp64 words of poseidon2_tc.cuh (50 clocks from word to
// word, against 72 for two Montgomery products), the external layer by two rounds of shuffles.
//
// Partial rounds: the S-boxes of word 0 are the serial chain. With T_r the sum of words 1..15
// before round r, x_r the S-box output and S_r = T_r + x_r,
//   word 0:  y_(r+1) = T_r - x_r  (V_0 = -2),    word i:  v_i <- V_i v_i + S_r,
//   T_(r+1) = sum_i V_i v_i + 15 S_r,
// so the sum over the words needs only products V_i v_i that do not wait for round r's S-box: it
// is two warp reductions of 16-bit halves (each total below 2^20) beside the chain, which is one
// cube and one subtraction a round. Word 0 is carried in every lane.
//
// Measured in one warp: 3.6 K clocks a permutation; 5.1 K with Montgomery products and the sum on
// the chain, 23 K with the whole state in every lane. The partial rounds unrolled, as a warp's
// instructions issue in order and the reductions of one round fill the gaps of the next one's
// S-box (4.5 K rolled, 4.0 K in fours). Collecting each round's linear part in a lane of its own
// instead (coefficients from a table) took 2.0 K for the partial rounds against 2.0 K, and 1.3 K
// more to set up.
#pragma once
#include "poseidon2_tc.cuh"

namespace kb {

// x is within p/2 + 2^9 of zero, so WARP_HALF + T - x is a word for T in [0, p).
constexpr uint32_t WARP_HALF = P / 2 + (1u << 22);

// Shares of the full rounds' constants (see P2ConstsTc), the partial rounds' constants less
// WARP_HALF (the first one as it is) and the internal diagonal (Montgomery form).
struct alignas(16) P2WarpConsts {
  uint32_t in[16], init[4][16], mid[16], term[4][16];
  uint32_t diag[16], rc[P2Consts<16>::RP];
};
inline P2WarpConsts p2_warp_consts(const P2Consts<16>& m) {
  const P2ConstsTc<16> t = p2_consts_tc(m);
  P2WarpConsts c{};
  std::memcpy(c.in, t.in, sizeof c.in);
  std::memcpy(c.init, t.init, sizeof c.init);
  std::memcpy(c.term, t.term, sizeof c.term);
  for (int i = 0; i < 16; i++) c.mid[i] = t.mid[i] - P, c.diag[i] = p2_diag<16>(i);
  for (int r = 0; r < P2Consts<16>::RP; r++)
    c.rc[r] = sub(from_mont(m.internal[r]), r ? WARP_HALF : 0u);
  return c;
}

#ifdef __CUDACC__
// Copies the constants into shared memory (all threads of the block; a barrier must follow).
__device__ __forceinline__ void p2_warp_load(P2WarpConsts& sh, const P2WarpConsts* __restrict__ c) {
  static_assert(sizeof(P2WarpConsts) % 16 == 0, "16-byte pieces");
  for (int t = threadIdx.x; t < int(sizeof(P2WarpConsts) / 16); t += blockDim.x)
    reinterpret_cast<uint4*>(&sh)[t] = __ldg(reinterpret_cast<const uint4*>(c) + t);
}

// The external layer on words in (0, 2p), as a biased word. Lane i's M4 row is 2 x_i +
// 3 x_(i+1) + x_(i+2) + x_(i+3) within its chunk of four; then the sum over the four chunks.
__device__ __forceinline__ double warp_mds(uint32_t w, int i) {
  constexpr unsigned ALL = 0xffffffffu;
  const int base = i & ~3;
  const uint32_t b = __shfl_sync(ALL, w, base | ((i + 1) & 3), 16);
  const uint32_t c = __shfl_sync(ALL, w, base | ((i + 2) & 3), 16);
  const uint32_t d = __shfl_sync(ALL, w, base | ((i + 3) & 3), 16);
  const double y = (fb_fma(fb_pair(w), 2.0, -2.0 * FB_2_52) + fb_fma(fb_pair(b), 3.0, -3.0 * FB_2_52)) +
                   ((fb_pair(c) - FB_2_52) + (fb_pair(d) - FB_2_52));
  const double y4 = __shfl_xor_sync(ALL, y, 4, 16), y8 = __shfl_xor_sync(ALL, y, 8, 16);
  const double y12 = __shfl_xor_sync(ALL, y, 12, 16);
  return (y4 + y8) + (y12 + fb_fma(y, 2.0, fb_magic<16>() - 35.0 * double(P)));
}
// The canonical residue of a biased z.
__device__ __forceinline__ uint32_t warp_word(double z) {
  const uint32_t w = fb_word<16>(z);
  return umin(w, w - P);
}

static __device__ __noinline__ uint32_t p2_warp_permute(uint32_t v, const P2WarpConsts& c) {
  constexpr unsigned ALL = 0xffffffffu;
  constexpr int RP = P2Consts<16>::RP;
  const int lane = threadIdx.x & 31, i = lane & 15;
  uint32_t w = v + c.in[i];
#pragma unroll 1
  for (int r = 0; r < 4; r++) w = fb_sbox<16>(warp_mds(w, i), c.init[r][i]);
  v = warp_word(warp_mds(w, i));
  const uint32_t d = c.diag[i];
  const bool contrib = lane >= 1 && lane < 16;
  // the words' sum from its 16-bit halves, plus 15 s, reduced with 2^31 = 2^24 - 1 (mod p): the
  // total is below 2^36, so the folded value is below 2p
  auto total = [](uint32_t lo, uint32_t hi, uint32_t s) {
    const uint64_t t = uint64_t(hi) * 65536u + (uint64_t(s) * 15u + lo);
    const uint32_t f = (uint32_t(t) & 0x7fffffffu) + uint32_t(t >> 31) * 0xffffffu;
    return umin(f, f - P);
  };
  uint32_t y = __shfl_sync(ALL, v, 0) + c.rc[0];  // the S-box input, a word
  w = contrib ? v : 0u;
  uint32_t T = total(__reduce_add_sync(ALL, w & 0xffffu), __reduce_add_sync(ALL, w >> 16), 0u);
#pragma unroll 20
  for (int r = 0; r < RP; r++) {
    const uint32_t m = mul(v, d);
    w = contrib ? m : 0u;
    const uint32_t lo = __reduce_add_sync(ALL, w & 0xffffu), hi = __reduce_add_sync(ALL, w >> 16);
    // T_r + the next round's constant (none after the last round)
    const uint32_t tc = (r + 1 < RP ? add(T, c.rc[r + 1]) : sub(T, WARP_HALF)) + WARP_HALF;
    const uint32_t x = uint32_t(part_cube(y));  // signed, within p/2 + 2^9
    y = tc - x;
    const uint32_t S = add(T, umin(x, x + P));
    v = m + S;  // below 2p
    T = total(lo, hi, S);
  }
  if (i == 0) v = y;
  v = umin(v, v - P);
  w = fb_sbox_word(v + c.mid[i], c.term[0][i]);
#pragma unroll 1
  for (int r = 1; r < 4; r++) w = fb_sbox<16>(warp_mds(w, i), c.term[r][i]);
  return warp_word(warp_mds(w, i));
}
#endif

}  // namespace kb
