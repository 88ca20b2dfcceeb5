// Poseidon2 (widths 16 and 24) with the partial rounds' linear algebra on the fifth-generation
// tensor cores, for hashing many rows at once: a block of 128 threads runs 128 permutations.
//
// Partial rounds. Between the full rounds only word 0 passes an S-box: with x_r its output in
// round r, word 0 at the next round and the state after all RP rounds are linear in the entry
// words s_1.. and in x_0 .. x_r. So the RP internal layers (W words each) become
//   y_(r+1) = [sum_i A(r, i) s_i] + sum_(j <= r) tau_(r-j) x_j,   x_r = (y_r + rc_r)^3,
//   s_out   = G s_in + H x,
// where the bracket for every r at once, and the last line, are products of a constant matrix
// with the words of 128 permutations: u8 x u8 -> s32 tcgen05.mma over byte limbs, exact. The
// sum over the x_j is triangular: within groups of 8 rounds it runs on the integer pipe (wide
// multiply-adds), and a finished group's x_j are multiplied into the accumulators of all later
// outputs, where they cost no further reduction.
//
// Byte limbs: the words as they lie in shared memory are the A operand (byte a of word j is
// reduction index 4j + a); B holds byte b of coef(o, j) 2^(8a) 2^32 mod p for output o, so an
// accumulator is below 192 * 255^2 < 2^24, v = sum_b acc_b 2^(8b) < 2^49, and one Montgomery
// reduction of v gives the output word. A thread's accumulators are its own lane of tensor
// memory, so a permutation's words never leave its thread but for the A operand.
//
// Full rounds. Words enter the external layer as 32-bit integers; its sums run on fp64 values
// that are exact integers, biased so that no conversion is spent on them: every output carries
// MAGIC = (row sum of the external matrix) 2^47, which lies in [2^52, 2^53), so the low 32 bits
// of its mantissa are the word mod 2^32.
//  * The S-box of z takes both quotients by p from the fp64 pipe: with C = 1/sqrt(p),
//    u = (z - MAGIC) C is one fused multiply-add (MAGIC C and 2^52 C are exact: C has 47
//    bits), and round(u u) = round(z^2 / p), round((w C) u) = round(w z / p) one more each.
//    The rounding constant is lowered by one, so both residues come out positive and enter
//    fp64 by pairing them with the exponent word of 2^52.
//  * The round constants cost nothing: the second residue's multiply-add also adds the word's
//    share of M^-1 rc, the vector that the following external layer M maps to the next round's
//    constants.
// That is 4 fp64 instructions and 4 integer multiplies per S-box.
//
// Measured (33.5M width-24 permutations, the leaves of 2^22 rows): 6.8 ms against 10.3 ms for
// one thread per permutation with the internal layers word by word (p2_permute_fd): 4,870 instead
// of 8,960 instructions a permutation, the leaf's own work included. What bounds it is register bandwidth: an S-box
// reads 22 32-bit operands, the fp64 pipe's pairs among them, and takes 14-15 clocks a warp and
// scheduler where its pipes (fp64 and integer multiply, 8 clocks each) would allow 9 to 10.
// Without the groups of 8 rounds: 7.3 ms; with mma.sync in place of tcgen05.mma: 9.5 ms, since
// m16n8k32 takes 8 clocks of the pipe that fp64 shares; blocks that stay resident and loop over
// tiles: 5% slower, as the blocks of an SM then run in step and want the same pipe at a time.
#pragma once
#include "poseidon2.cuh"

namespace kb {

// ---------------------------------------------------------------- linear form of the partial rounds
namespace p2lin {
constexpr uint64_t mulm(uint64_t a, uint64_t b) { return a * b % P; }
// Canonical internal diagonal.
template <int W>
constexpr uint32_t diag(int i) {
  return uint32_t(mulm(p2_diag<W>(i), detail::cpow(uint64_t(R_MOD_P), P - 2)));
}
template <int W>
struct Lin {
  static constexpr int RP = P2Consts<W>::RP;
  uint32_t a[RP][W] = {};    // y_(r+1) from s_i (column 0 zero)
  uint32_t g[W][W] = {};     // state after RP rounds from s_i (column 0 zero)
  uint32_t tau[RP] = {};     // y_(r+1) from x_(r - m) at m
  uint32_t h[W][RP] = {};    // state after RP rounds from x_j
};
template <int W>
constexpr Lin<W> make_lin() {
  constexpr int RP = Lin<W>::RP;
  Lin<W> l;
  uint64_t d[W] = {};
  for (int i = 0; i < W; i++) d[i] = diag<W>(i);
  for (int e = 0; e < W; e++) {  // e = 0: the impulse x_0 = 1 from the zero state; else s_e = 1
    uint64_t s[W] = {};
    if (e) s[e] = 1;
    for (int r = 0; r < RP; r++) {
      const uint64_t x0 = e == 0 && r == 0 ? 1 : 0;
      uint64_t sum = x0;
      for (int i = 1; i < W; i++) sum += s[i];
      sum %= P;
      s[0] = (d[0] * x0 + sum) % P;
      for (int i = 1; i < W; i++) s[i] = (d[i] * s[i] + sum) % P;
      if (e) {
        l.a[r][e] = uint32_t(s[0]);
      } else {
        l.tau[r] = uint32_t(s[0]);
        for (int k = 0; k < W; k++) l.h[k][RP - 1 - r] = uint32_t(s[k]);  // r + 1 rounds after x_(RP-1-r)
      }
    }
    if (e)
      for (int k = 0; k < W; k++) l.g[k][e] = uint32_t(s[k]);
  }
  return l;
}
template <int W>
inline constexpr Lin<W> LIN = make_lin<W>();

// tau_m 2^32 mod p in [-p/2, p/2].
template <int W, int M>
struct Tau {
  static constexpr uint32_t u = uint32_t((uint64_t(LIN<W>.tau[M]) << 32) % P);
  static constexpr int32_t v = u > P / 2 ? int32_t(int64_t(u) - int64_t(P)) : int32_t(u);
};
}  // namespace p2lin

// The B operands as tcgen05.mma reads them from shared memory: K-major, no swizzle, in core
// matrices of 8 rows (columns n of B) x 16 bytes. 16-byte piece c of row n, the words j = 4c ..
// 4c + 3, lies at entry c N + n, so core matrices are 128 bytes apart along n and 16 N bytes
// apart along k. Row n = 4 o + b holds byte b of the coefficients of output o.
template <int W>
struct P2TcTab {
  static constexpr int RP = P2Consts<W>::RP;
  static constexpr int KS = W / 8;                       // k-steps of 32 bytes over the state words
  static constexpr int KX = (RP + 7) / 8;                // and over the x words
  static constexpr int O1 = RP - 1;                      // outputs of stage 1: y_1 .. y_(RP-1)
  static constexpr int N1 = (4 * O1 + 15) / 16 * 16;     // rows of the B operands
  static constexpr int N2 = 4 * W;
  static constexpr int N3 = N1 - 32;                     // x of 8 rounds into the outputs after them
  static constexpr int E1 = 2 * KS * N1, E2 = 2 * (KS + KX) * N2, E3 = 2 * N3;  // 16-byte entries
  alignas(16) uint32_t w[(E1 + E2 + E3) * 4] = {};  // read 16 bytes at a time
};
namespace p2lin {
// Coefficient of word j in output o of stage 1 (y_1 .. y_(RP-1) from the state), stage 2 (the
// state after the partial rounds) or stage 3 (output 8 + o of stage 1 from x_0 .. x_7; the same
// for any 8 consecutive rounds).
template <int W>
constexpr uint32_t coef(int stage, int o, int j) {
  constexpr int RP = Lin<W>::RP;
  if (stage == 3) return 8 + o - j < RP ? LIN<W>.tau[8 + o - j] : 0;
  if (stage == 1) return o < RP - 1 && j < W ? LIN<W>.a[o][j] : 0;
  if (j < W) return LIN<W>.g[o][j];
  return j - W < RP ? LIN<W>.h[o][j - W] : 0;
}
template <int W>
constexpr P2TcTab<W> make_tab() {
  using T = P2TcTab<W>;
  P2TcTab<W> t;
  for (int stage = 1; stage <= 3; stage++) {
    const int words = 8 * (stage == 1 ? T::KS : stage == 2 ? T::KS + T::KX : 1);
    const int n_rows = stage == 1 ? T::N1 : stage == 2 ? T::N2 : T::N3;
    uint32_t* base = t.w + 4 * (stage == 1 ? 0 : stage == 2 ? T::E1 : T::E1 + T::E2);
    for (int j = 0; j < words; j++)
      for (int o = 0; o < n_rows / 4; o++) {
        uint64_t v = mulm(coef<W>(stage, o, j), R_MOD_P);  // 2^32 coef: a Montgomery reduction follows
        uint32_t by[4] = {};  // by[b]: byte b of v 2^(8a), a = 0..3
        for (int a = 0; a < 4; a++) {
          for (int b = 0; b < 4; b++) by[b] |= uint32_t((v >> (8 * b)) & 0xff) << (8 * a);
          v = (v << 8) % P;
        }
        for (int b = 0; b < 4; b++) base[((j >> 2) * n_rows + 4 * o + b) * 4 + (j & 3)] = by[b];
      }
  }
  return t;
}
}  // namespace p2lin

// ---------------------------------------------------------------- fp64 pieces
constexpr double FB_C = 0x1.6b7612eb1adc0p-16;  // 1 / sqrt(p) in 47 bits: C^2 p = 1 - 2^-48.06
constexpr double FB_2_52 = 4503599627370496.0, FB_2_47 = 140737488355328.0;
constexpr double FB_RND = FQ_ROUND, FB_RND1 = FQ_ROUND - 1.0;
// The external matrix (J + I) (x) M4 has row sum 7 fb_rows(): M4's is 7, J + I's is W/4 + 1.
template <int W>
constexpr double fb_rows() { return W / 4 + 1; }
template <int W>
constexpr double fb_magic() { return 7.0 * fb_rows<W>() * FB_2_47; }  // in [2^52, 2^53)

KB_HD double fb_fma(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}
KB_HD uint32_t fb_lo(double x) {
#ifdef __CUDA_ARCH__
  return uint32_t(__double2loint(x));
#else
  uint64_t bits;
  std::memcpy(&bits, &x, sizeof bits);
  return uint32_t(bits);
#endif
}
KB_HD double fb_pair(uint32_t u) {  // 2^52 + u
#ifdef __CUDA_ARCH__
  return __hiloint2double(0x43300000, int(u));
#else
  return FB_2_52 + double(u);
#endif
}
// z^3 + k from the low word zi of z and u = z / sqrt(p), |z| < 2^37: the residue of z^3 in
// (p/3, 5p/3), so for k in [-p/3, p/3] a word.
KB_HD uint32_t fb_cube(uint32_t zi, double u, uint32_t k) {
  const uint32_t w = zi * zi - fb_lo(fb_fma(u, u, FB_RND1)) * P;
  const double wc = fb_fma(fb_pair(w), FB_C, -FB_2_52 * FB_C);
  return (w * zi + k) - fb_lo(fb_fma(wc, u, FB_RND1)) * P;
}
// The S-box of a biased word, and of a plain word below 2^32.
template <int W>
KB_HD uint32_t fb_sbox(double zb, uint32_t k) {
  return fb_cube(fb_lo(zb), fb_fma(zb, FB_C, -fb_magic<W>() * FB_C), k);
}
KB_HD uint32_t fb_sbox_word(uint32_t z, uint32_t k) {
  return fb_cube(z, fb_fma(fb_pair(z), FB_C, -FB_2_52 * FB_C), k);
}
// The residue of a biased word in (0, 2p): round(z / p) is off by less than one half more
// (the constant's own rounding), and the quotient is lowered by one.
template <int W>
KB_HD uint32_t fb_word(double zb) {
  return fb_lo(zb) - fb_lo(fb_fma(zb, FQ_INV_P, FB_RND1 - fb_magic<W>() * FQ_INV_P)) * P;
}

// Addends of the full rounds (see the top of the file) and of the partial rounds. Words enter
// an external layer in (0, 2p): an input word in [0, p] takes a share in [0, p), an S-box output
// in (p/2, 3p/2) (its second product is small enough for that) one in [-p/2, p/2).
template <int W>
struct P2ConstsTc {
  static constexpr int RP = P2Consts<W>::RP;
  uint32_t in[W];       // added to the input words
  uint32_t init[4][W];  // added to the S-box outputs of initial full round r
  uint32_t mid[W];      // p + the first terminal round's constants, added as the partial rounds end
  uint32_t term[4][W];  // added to the S-box outputs of terminal full round r
  uint32_t rc0;         // the first partial round's constant
  uint64_t radd[RP - 1];  // (rc_(o+1) - PART_K) 2^32 mod p, added to stage-1 output o
};
// Offset that keeps y + rc, as the triangular sum leaves it, a 32-bit unsigned value: with at
// most four products after the last fold the sum's high word is within PART_H of zero.
constexpr uint32_t PART_H = 1080000000u, PART_K = P + PART_H;

// a with M a = v, M = (J + I) (x) M4 the external matrix: M^-1 = (I - J / (W/4 + 1)) (x) M4^-1.
template <int W>
inline void external_inverse(const uint32_t* v, uint32_t* a) {
  // M4^-1 by Gauss-Jordan elimination mod p
  struct Inv {
    uint64_t m[4][4];
    uint64_t q;
    Inv() {
      const int64_t M[4][4] = {{2, 3, 1, 1}, {1, 2, 3, 1}, {1, 1, 2, 3}, {3, 1, 1, 2}};
      uint64_t w[4][8];
      for (int i = 0; i < 4; i++)
        for (int j = 0; j < 8; j++) w[i][j] = j < 4 ? uint64_t(M[i][j]) : uint64_t(j - 4 == i);
      for (int c = 0; c < 4; c++) {
        int p = c;
        while (w[p][c] == 0) p++;
        for (int j = 0; j < 8; j++) std::swap(w[p][j], w[c][j]);
        const uint64_t iv = detail::cpow(w[c][c], P - 2);
        for (int j = 0; j < 8; j++) w[c][j] = w[c][j] * iv % P;
        for (int i = 0; i < 4; i++) {
          const uint64_t f = w[i][c];
          if (i == c || !f) continue;
          for (int j = 0; j < 8; j++) w[i][j] = (w[i][j] + (P - f) * w[c][j]) % P;
        }
      }
      for (int i = 0; i < 4; i++)
        for (int j = 0; j < 4; j++) m[i][j] = w[i][4 + j];
      q = detail::cpow(W / 4 + 1, P - 2);
    }
  };
  static const Inv inv;
  uint64_t t[W], sum[4] = {};
  for (int c = 0; c < W; c += 4)
    for (int i = 0; i < 4; i++) {
      uint64_t s = 0;
      for (int j = 0; j < 4; j++) s += inv.m[i][j] * v[c + j] % P;
      t[c + i] = s % P;
      sum[i] += t[c + i];
    }
  for (int i = 0; i < 4; i++) sum[i] = sum[i] % P * inv.q % P;
  for (int i = 0; i < W; i++) a[i] = uint32_t((t[i] + P - sum[i & 3]) % P);
}

template <int W>
inline P2ConstsTc<W> p2_consts_tc(const P2Consts<W>& m) {
  P2ConstsTc<W> c{};
  uint32_t rc[W], a[W];
  auto shares = [&](const uint32_t* k) {  // of every word in M^-1 rc
    for (int i = 0; i < W; i++) rc[i] = from_mont(k[i]);
    external_inverse<W>(rc, a);
  };
  shares(m.ext_init);
  for (int i = 0; i < W; i++) c.in[i] = a[i];
  for (int r = 0; r < 3; r++) {
    shares(m.ext_init + (r + 1) * W);
    for (int i = 0; i < W; i++) c.init[r][i] = a[i] < P / 2 ? a[i] : a[i] - P;
    shares(m.ext_term + (r + 1) * W);
    for (int i = 0; i < W; i++) c.term[r][i] = a[i] < P / 2 ? a[i] : a[i] - P;
  }
  for (int i = 0; i < W; i++) c.mid[i] = P + from_mont(m.ext_term[i]);
  c.rc0 = from_mont(m.internal[0]);
  for (int o = 0; o < P2Consts<W>::RP - 1; o++) {
    const uint64_t rcv = from_mont(m.internal[o + 1]);
    c.radd[o] = uint32_t(((rcv + 2 * uint64_t(P) - PART_K) % P << 32) % P);
  }
  return c;
}

// M4 on four values.
KB_HD void fb_m4(const double* x, double* y) {
  const double t01 = x[0] + x[1], t23 = x[2] + x[3], t = t01 + t23;
  const double tx1 = t + x[1], tx3 = t + x[3];
  y[0] = tx1 + t01;
  y[1] = fb_fma(2.0, x[2], tx1);
  y[2] = tx3 + t23;
  y[3] = fb_fma(2.0, x[0], tx3);
}
// External layer: M4 applied to every chunk plus the column sums. The sums are formed in 64-bit
// integers; as fp64 they take the offset that turns a word's exponent pairing (2^52) into the
// bias rows 2^47 and the words' own centring by p, so that the outputs are biased words.
template <int W>
KB_HD void fb_column_sums(const uint32_t* w, double* sum) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    uint64_t t = uint64_t(w[k]) + w[4 + k];
#pragma unroll
    for (int j = 2; j < W / 4; j++) t += w[4 * j + k];
#ifdef __CUDA_ARCH__
    const double td = __hiloint2double(0x43300000 | int(t >> 32), int(uint32_t(t)));
#else
    const double td = FB_2_52 + double(t);
#endif
    sum[k] = td + (fb_rows<W>() * (FB_2_47 - double(P)) - 2.0 * FB_2_52);
  }
}
template <int W>
KB_HD void fb_mds(const uint32_t* w, double* z) {
  double sum[4];
  fb_column_sums<W>(w, sum);
#pragma unroll
  for (int c = 0; c < W; c += 4) {
    double x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) x[k] = fb_pair(w[c + k]) + sum[k];
    fb_m4(x, z + c);
  }
}

// add + sum_b a_b 2^(8b) of an output's four byte accumulators (below 2^24).
KB_HD uint64_t limb_sum(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint64_t add) {
  const uint32_t lo = a0 + (a1 << 8), hi = a2 + (a3 << 8);
  return uint64_t(hi) * 65536u + add + lo;
}
// The triangular sum of one partial round: 2^32 (y + rc) from its stage-1 sum and the x of the
// N rounds since the last group of 8 (signed, |x| <= 0.51 p), reduced to an unsigned word
// congruent to y + rc. With more than four products the 64-bit sum is folded with
// 2^32 = 2^25 - 2 (mod p) so that four follow the fold: it then stays below 2^62 (1 + 2^-10),
// within PART_H 2^32.
template <int W, int N, int J>
KB_HD void part_mac(int64_t& acc, const int32_t* x) {
  if constexpr (J < N) {
    acc += int64_t(x[J]) * p2lin::Tau<W, N - 1 - J>::v;
    if constexpr (J + 1 == N - 4) acc = int64_t(int32_t(acc >> 32)) * ((1 << 25) - 2) + int64_t(uint32_t(acc));
    part_mac<W, N, J + 1>(acc, x);
  }
}
template <int W, int N>
KB_HD uint32_t part_sum(uint64_t init, const int32_t* x) {
  static_assert(N <= 8, "one fold");
  int64_t acc = int64_t(init);
  part_mac<W, N, 0>(acc, x);
  return uint32_t(uint64_t(acc) >> 32) - umulhi(uint32_t(acc) * PINV, P) + PART_K;
}
// x = v^3 as a signed residue within 0.51 p, for the unsigned word v.
KB_HD int32_t part_cube(uint32_t v) {
  const double u = fb_fma(fb_pair(v), FB_C, -FB_2_52 * FB_C);
  const uint32_t w = v * v - fb_lo(fb_fma(u, u, FB_RND1)) * P;
  const double wc = fb_fma(fb_pair(w), FB_C, -FB_2_52 * FB_C);
  return int32_t(w * v - fb_lo(fb_fma(wc, u, FB_RND)) * P);
}
// x[I + 1] .. x[M] from the accumulators of the group's outputs I .. M - 1 and x[0] .. x[I]
// (indices within the group of 8 rounds that starts at round R0).
template <int W, int R0, int I, int M>
KB_HD void part_chain(const uint32_t* acc, const P2ConstsTc<W>& c, int32_t* x) {
  if constexpr (I < M) {
    const uint32_t* a = acc + 4 * I;
    x[I + 1] = part_cube(part_sum<W, I + 1>(limb_sum(a[0], a[1], a[2], a[3], c.radd[R0 + I]), x));
    part_chain<W, R0, I + 1, M>(acc, c, x);
  }
}
// One output word of stage 2 plus add - p, for add in [p, 2p): a word in (0, 2p + 2^17).
KB_HD uint32_t limb_word(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t add) {
  const uint64_t v = limb_sum(a0, a1, a2, a3, 0);
  return uint32_t(v >> 32) - umulhi(uint32_t(v) * PINV, P) + add;
}

// ---------------------------------------------------------------- waits that run out
// A thread's account of its block's matrix products, each of which completes one phase of the
// mbarrier: the parity of the phase to wait for, and whether a wait of this thread ran out. From
// then on the parity stays at that phase, and as the block starts no product once a thread's wait
// has run out (tc_product), that one is the last and the only one that may still be running.
struct TcPhase {
  uint32_t parity = 0;
  bool expired = false;
  KB_HD void waited(bool done) {
    if (done) parity ^= 1;
    else expired = true;
  }
};

#ifdef __CUDACC__
// ---------------------------------------------------------------- one tile of 128 permutations
// A block is one tile: 128 threads, one permutation each, thread t on row t of the A operand and
// lane t of the accumulators in tensor memory. Shared memory holds the B operands (copied once
// per block), the A operand (words of the rows: 16-byte piece c of row t at entry 128 c + t, so
// a warp's stores are contiguous) and the mbarrier that the matrix products arrive on.
constexpr int TC_ROWS = 128;
constexpr int TC_COLS = 128;  // tensor memory columns of a tile (a power of two >= N1, N2)
template <int W>
struct P2TcShared {
  using T = P2TcTab<W>;
  static constexpr int EA = 2 * (T::KS + T::KX) * TC_ROWS;  // 16-byte entries of A
  uint64_t bar;
  uint32_t tmem;
  uint4 b[T::E1 + T::E2 + T::E3];
  uint4 a[EA];
};
template <int W>
__device__ const P2TcTab<W> g_p2_tc_tab = p2lin::make_tab<W>();

// A wait on the mbarrier gives up after this many clocks (about two seconds).
constexpr long long TC_WAIT_CLOCKS = 4000000000ll;

__device__ __forceinline__ uint32_t tc_smem(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

// Loads the B operands. All threads; ends with a barrier. A block that has begun with one width
// may go on with the other on the same bytes (the mbarrier and the accumulators stay).
template <int W>
__device__ __forceinline__ void p2_tc_load(P2TcShared<W>& sh) {
  using T = P2TcTab<W>;
  const uint4* src = reinterpret_cast<const uint4*>(g_p2_tc_tab<W>.w);
  for (int i = threadIdx.x; i < T::E1 + T::E2 + T::E3; i += TC_ROWS) sh.b[i] = src[i];
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Sets the mbarrier up, allocates the tile's accumulators and loads the B operands.
template <int W>
__device__ __forceinline__ void p2_tc_begin(P2TcShared<W>& sh) {
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&sh.tmem)),
                 "r"(TC_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&sh.bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  p2_tc_load(sh);
}
// Waits for the phase of the given parity; false when TC_WAIT_CLOCKS have passed without it.
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity) {
  uint32_t done = 0;
  const long long t0 = clock64();
  do {
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
  } while (!done && clock64() - t0 < TC_WAIT_CLOCKS);
  return done;
}
// Frees the accumulators. A product whose wait ran out may still read shared memory and write the
// accumulators, so it is waited for once more (with the same limit) before they and the block go;
// the block then counts as one that ran out.
template <int W>
__device__ __forceinline__ void p2_tc_end(P2TcShared<W>& sh, const TcPhase& ph, unsigned* timeouts) {
  if (ph.expired) tc_wait(tc_smem(&sh.bar), ph.parity);
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  const bool expired = __syncthreads_or(ph.expired);
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem), "r"(TC_COLS));
  }
  if (threadIdx.x == 0 && expired) atomicAdd(timeouts, 1u);
}
// Shared-memory matrix descriptor: K-major, no swizzle; lbo / sbo are the byte distances of core
// matrices along k and along the rows.
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return uint64_t((addr & 0x3ffff) >> 4) | uint64_t(lbo >> 4) << 16 | uint64_t(sbo >> 4) << 32 | uint64_t(1) << 46;
}
// D = A B (ADD: D += A B) over KT k-steps: u8 x u8 -> s32, M = 128 rows, N columns from column
// `col` of the accumulators; a and b are the operands' first entries (b has NB rows). The block
// has written A; one thread issues the products, and every thread waits for them. Once a wait of any
// thread has run out the block issues none: the results are void (p2_tc_end counts them).
template <int W, int KT, int N, int NB, bool ADD>
__device__ __forceinline__ void tc_product(P2TcShared<W>& sh, const uint4* a, const uint4* b, int col, TcPhase& ph) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  const bool stop = __syncthreads_or(ph.expired);
  if (threadIdx.x == 0 && !stop) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // instruction descriptor: D s32 (2 at bit 4), A and B unsigned 8 bit, both K-major
    constexpr uint32_t idesc = 2u << 4 | uint32_t(N / 8) << 17 | uint32_t(TC_ROWS / 16) << 24;
    const uint32_t sa = tc_smem(a), sb = tc_smem(b), d = sh.tmem + col;
#pragma unroll
    for (int ks = 0; ks < KT; ks++) {
      const uint64_t da = tc_desc(sa + ks * 2 * TC_ROWS * 16, TC_ROWS * 16, 128);
      const uint64_t db = tc_desc(sb + ks * 2 * NB * 16, NB * 16, 128);
      asm volatile(
          "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
          "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
          "l"(da), "l"(db), "r"(idesc), "r"(ADD ? 1 : ks)
          : "memory");
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(&sh.bar))
                 : "memory");
  }
  __syncwarp();
  if (!stop) ph.waited(tc_wait(tc_smem(&sh.bar), ph.parity));
  __syncwarp();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// 32 accumulator columns of this thread's row, from column `col`.
__device__ __forceinline__ void tc_load32(uint32_t tmem, int col, uint32_t* r) {
  const uint32_t addr = tmem + ((threadIdx.x & ~31u) << 16) + col;
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr));
}
__device__ __forceinline__ void tc_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
template <int NW>
__device__ __forceinline__ void tc_store_words(uint4* a, const uint32_t* w) {
#pragma unroll
  for (int q = 0; q < NW / 4; q++) a[q * TC_ROWS + threadIdx.x] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
}
// The partial rounds' S-boxes in groups of 8: within a group the triangular sum runs on the
// integer pipe, and when a group is done its x words are multiplied into the accumulators of
// all later outputs, so that no sum has more than 8 terms.
template <int W, int G>
__device__ __forceinline__ void tc_chain(P2TcShared<W>& sh, const P2ConstsTc<W>& c, TcPhase& ph, int32_t* x) {
  using T = P2TcTab<W>;
  constexpr int R0 = 8 * G, M = T::O1 - R0 < 8 ? T::O1 - R0 : 8;
  uint32_t r[32];
  tc_load32(sh.tmem, 4 * R0, r);
  tc_load_wait();
  part_chain<W, R0, 0, M>(r, c, x + R0);
  uint32_t xs[8];
#pragma unroll
  for (int j = 0; j < 8; j++) xs[j] = R0 + j < T::RP ? uint32_t(x[R0 + j]) + P : 0u;
  uint4* xa = sh.a + 2 * (T::KS + G) * TC_ROWS;
  tc_store_words<8>(xa, xs);
  if constexpr (R0 + 8 < T::O1) {
    tc_product<W, 1, T::N1 - 4 * (R0 + 8), T::N3, true>(sh, xa, sh.b + T::E1 + T::E2, 4 * (R0 + 8), ph);
    tc_chain<W, G + 1>(sh, c, ph, x);
  }
}

// The permutation on words in [0, p] (canonical, or p for zero). Every thread of the block calls
// it. On return `out` holds the first 8 words of the state (first8 false: the last 8), in
// (0, 2p); the other words are not formed.
template <int W>
__device__ __forceinline__ void p2_permute_tc(const uint32_t* s, const P2ConstsTc<W>& c, P2TcShared<W>& sh,
                                              TcPhase& ph, bool first8, uint32_t* out) {
  using T = P2TcTab<W>;
  uint32_t w[W];
  double z[W];
#pragma unroll
  for (int i = 0; i < W; i++) w[i] = s[i] + c.in[i];
#pragma unroll 1
  for (int r = 0; r < 4; r++) {
    fb_mds<W>(w, z);
#pragma unroll
    for (int i = 0; i < W; i++) w[i] = fb_sbox<W>(z[i], c.init[r][i]);
  }
  fb_mds<W>(w, z);
  int32_t x[T::RP];
#pragma unroll
  for (int i = 0; i < W; i++) w[i] = fb_word<W>(z[i]);
  tc_store_words<W>(sh.a, w);
  x[0] = part_cube(umin(w[0], w[0] - P) + c.rc0);
  tc_product<W, T::KS, T::N1, T::N1, false>(sh, sh.a, sh.b, 0, ph);
  tc_chain<W, 0>(sh, c, ph, x);
  static_assert((T::O1 - 1) / 8 + 1 == T::KX, "the last group stores the last x words");
  tc_product<W, T::KS + T::KX, T::N2, T::N2, false>(sh, sh.a, sh.b + T::E1, 0, ph);
#pragma unroll
  for (int g = 0; g < W / 8; g++) {
    uint32_t r[32];
    tc_load32(sh.tmem, 32 * g, r);
    tc_load_wait();
#pragma unroll
    for (int i = 0; i < 8; i++)
      w[8 * g + i] = fb_sbox_word(limb_word(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3], c.mid[8 * g + i]),
                                  c.term[0][8 * g + i]);
  }
#pragma unroll 1
  for (int r = 1; r < 4; r++) {
    fb_mds<W>(w, z);
#pragma unroll
    for (int i = 0; i < W; i++) w[i] = fb_sbox<W>(z[i], c.term[r][i]);
  }
  // the last external layer, for the two chunks asked for
  double sum[4];
  fb_column_sums<W>(w, sum);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    double xh[4], y[4];
#pragma unroll
    for (int k = 0; k < 4; k++) xh[k] = fb_pair(first8 ? w[4 * h + k] : w[W - 8 + 4 * h + k]) + sum[k];
    fb_m4(xh, y);
#pragma unroll
    for (int k = 0; k < 4; k++) out[4 * h + k] = fb_word<W>(y[k]);
  }
}
#endif

}  // namespace kb
