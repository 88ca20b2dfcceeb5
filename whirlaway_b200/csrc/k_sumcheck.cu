// Sumcheck kernels: the AIR zerocheck (univariate-skip first round over the base field,
// later rounds over the extension field), the folds between rounds, the inner-phase
// helpers and the standalone a*b - c zerocheck. They compute the sums of
// crates/sumcheck/src/prove.rs:97-335 (sc_round / compute_over_hypercube) and the folds of
// crates/utils/src/multilinear.rs; the transcript work between rounds stays on the host.
//
// Column conventions: the witness is column-major (column c at wit + c * 2^n, Montgomery).
// "up" columns replace the last row by the one before it and "down" columns shift by one
// row and repeat the last (crates/air/src/utils.rs:140-160); neither is materialised.
// Folded columns are extension-field arrays, column c at cols + c * len.
#include <algorithm>
#include <map>
#include <mutex>
#include "finish.cuh"
#include "kernels.h"
#include "limb_mma.cuh"

namespace wl {

namespace {
using namespace kb;

__device__ __forceinline__ size_t up_row(size_t i, size_t N) { return i == N - 1 ? N - 2 : i; }
__device__ __forceinline__ size_t down_row(size_t i, size_t N) { return i == N - 1 ? N - 1 : i + 1; }

// ------------------------------------------------------------------ eq tables
// out[x] = prod_i (x_i ? r_i : 1 - r_i), x_1 = most significant bit of x.
// eq(pt, x) for x < 2^nvars, x's leading bit pairing with pt[0]. A block writes 2^EQ_BLK_BITS
// consecutive entries: x = (block << nbits) + (a << nb) + b, eq = H * A[a] * B[b], where A and
// B are tables over the block's two groups of low variables (<= 16 entries each, built in
// shared memory) and H is the product over the block's high variables (a product tree).
// The tree and the tables are a chain of a dozen products before the block's one product per
// entry, so a large table's block writes 2^EQ_BIG_BITS entries: H joins a third table C of 16
// entries, C x A is formed once (one product a thread), and each thread writes 16 entries. From
// EQ_BIG_VARS variables on that leaves 128 blocks or more. 2^20 entries: 52 us with blocks of
// 2^8, 31 here; the a*b - c sumcheck of 2^24 1324 to 1277 us.
constexpr int EQ_MAX_VARS = 32;
constexpr int EQ_BLK_BITS = 8;
constexpr int EQ_BIG_BITS = 12, EQ_BIG_VARS = 19;
constexpr int EQ_THREADS = 1 << EQ_BLK_BITS;
__host__ __device__ inline int eq_block_bits(int nvars) {
  return nvars >= EQ_BIG_VARS ? EQ_BIG_BITS : nvars < EQ_BLK_BITS ? nvars : EQ_BLK_BITS;
}
__device__ __forceinline__ void eq_table_block(const ef* __restrict__ pt, int nvars, size_t xhi, ef* __restrict__ out) {
  __shared__ ef r1[EQ_MAX_VARS], r0[EQ_MAX_VARS], fac[EQ_MAX_VARS], A[16], B[16], C[16], CA[256];
  const int nbits = eq_block_bits(nvars), low = nbits < EQ_BLK_BITS ? nbits : EQ_BLK_BITS, nc = nbits - low;
  const int nhi = nvars - nbits, ia = nhi + nc, na = low / 2, nb = low - na;
  const int tid = threadIdx.x;
  for (int i = tid; i < nvars; i += blockDim.x) {
    const ef r = pt[i];
    r1[i] = r;
    r0[i] = ef_sub(ef_one(), r);
  }
  __syncthreads();
  if (tid < nhi) fac[tid] = ((xhi >> (nhi - 1 - tid)) & 1) ? r1[tid] : r0[tid];
  if (tid >= 64 && tid - 64 < (1 << na)) {
    const int a = tid - 64;
    ef v = ef_one();
    for (int i = 0; i < na; i++) v = ef_mul(v, ((a >> (na - 1 - i)) & 1) ? r1[ia + i] : r0[ia + i]);
    A[a] = v;
  }
  if (tid >= 96 && tid - 96 < (1 << nb)) {
    const int b = tid - 96;
    ef v = ef_one();
    for (int i = 0; i < nb; i++) v = ef_mul(v, ((b >> (nb - 1 - i)) & 1) ? r1[ia + na + i] : r0[ia + na + i]);
    B[b] = v;
  }
  if (nc && tid >= 128 && tid - 128 < (1 << nc)) {
    const int c = tid - 128;
    ef v = ef_one();
    for (int i = 0; i < nc; i++) v = ef_mul(v, ((c >> (nc - 1 - i)) & 1) ? r1[nhi + i] : r0[nhi + i]);
    C[c] = v;
  }
  __syncthreads();
  for (int len = nhi; len > 1;) {
    const int m = (len + 1) >> 1;
    if (tid < len - m) fac[tid] = ef_mul(fac[tid], fac[tid + m]);
    __syncthreads();
    len = m;
  }
  if (nc) {  // 12 bits: four each in C, A and B
    if (tid < 16) C[tid] = ef_mul(fac[0], C[tid]);
    __syncthreads();
    CA[tid] = ef_mul(C[tid >> 4], A[tid & 15]);
    __syncthreads();
    const ef b = B[tid & 15];
#pragma unroll 1
    for (int q = 0; q < 16; q++) out[(xhi << nbits) + q * 256 + tid] = ef_mul(CA[q * 16 + (tid >> 4)], b);
    return;
  }
  // the block's factor joins A first: one product per entry
  if (nhi) {
    if (tid < (1 << na)) A[tid] = ef_mul(fac[0], A[tid]);
    __syncthreads();
  }
  if (tid < (1 << nbits)) out[(xhi << nbits) + tid] = ef_mul(A[tid >> nb], B[tid & ((1 << nb) - 1)]);
}

__global__ void __launch_bounds__(EQ_THREADS) k_eq_table(const ef* __restrict__ pt, int nvars, ef* __restrict__ out) {
  eq_table_block(pt, nvars, blockIdx.x, out);
}
// Several tables in one launch, their points in the kernel's arguments: a proof makes two dozen
// small tables, and each used to take a copy of its point, a launch, and where it belonged into a
// larger array a copy of the table. A proof of 2^12 rows: 22 launches, 22 uploads and 8 copies
// become 11 launches (3.14 to 3.08 ms; 2^16 rows 5.17 to 5.06 ms).
__global__ void __launch_bounds__(EQ_THREADS) k_eq_tables(const __grid_constant__ EqTables e) {
  int t = 0;
  while (t + 1 < e.n && int(blockIdx.x) >= e.first[t + 1]) t++;
  eq_table_block(e.pt + e.off[t], e.nvars[t], size_t(int(blockIdx.x) - e.first[t]), e.out[t]);
}

__global__ void k_eq_table_f(const uint32_t* __restrict__ pts, int npts, int nvars, uint32_t* __restrict__ out) {
  size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  size_t n = size_t(npts) << nvars;
  if (i >= n) return;
  size_t p = i >> nvars;
  uint32_t x = uint32_t(i & ((size_t(1) << nvars) - 1));
  uint32_t v = R_MOD_P;
  for (int k = 0; k < nvars; k++) {
    uint32_t r = pts[p * nvars + k];
    bool bit = (x >> (nvars - 1 - k)) & 1;
    v = mul(v, bit ? r : sub(R_MOD_P, r));
  }
  out[i] = v;
}

__global__ void k_reduce_partials(const ef* __restrict__ partial, int nblk, int k, ef* __restrict__ out) {
  __shared__ ef scratch[32];
  const int j = blockIdx.x;
  ef acc = ef_zero();
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) acc = ef_add(acc, partial[size_t(b) * k + j]);
  acc = block_reduce_ef(acc, scratch);
  if (threadIdx.x == 0) out[j] = acc;
}

// ------------------------------------------------------------------ AIR zerocheck
constexpr int ZC0_X = 32;
constexpr int ZC0_STAGES = 2;   // input groups in flight
constexpr int ZC0_GROUP = 8;    // inputs per staged group (one block barrier per group)
constexpr int ZC0_PAD = 20;     // words per x in a staged column tile (16 values + padding)

__device__ __forceinline__ void cp_async4(uint32_t* smem, const uint32_t* gmem) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem));
}
__device__ __forceinline__ void cp_async16(uint32_t* smem, const uint32_t* gmem) {  // 16-byte aligned
  unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// The batched constraint sum_i alpha_i C_i is rewritten as
//   sum_i gamma_i cube(u_i) - sum_i alpha_i col_(17+i),
// since constraint i is (a linear map of an S-box layer) minus its committed column 17 + i:
// the full rounds' linear map moves onto the weights (gamma = MDS^T alpha, the host's betas)
// and the partial rounds' weight is alpha itself. Each cube input u_i is an affine function
// of the row: a committed column plus a round constant (the inputs of beginning and ending
// rounds 1..3), or, for the 52 others, MDS of the inputs (beginning round 0), the partial
// chain's state word 0 (the 20 partial rounds) and the state after the chain (ending round
// 0). The extension to a point z is linear and keeps constants (the Lagrange weights sum to
// one), so k_zc0_rows computes those 52 inputs once per row, and the committed-column term,
// which is linear, once per row as well (weighted by L_j(z) after its sum over x); per
// point z only the 148 cube inputs are extended, cubed and weighted.

// Source of cube input i: computed input q[qcol] (round constant included), or committed
// column 1 + i (qcol < 0) plus the round constant zc0_rc.
__device__ __forceinline__ int zc0_qcol(int i) {
  if (i < 16) return i;             // beginning round 0
  if (i < 64) return -1;            // beginning rounds 1..3: columns 17..64
  if (i < 100) return i - 48;       // partial rounds (q 16..35), ending round 0 (q 36..51)
  return -1;                        // ending rounds 1..3: columns 101..148
}
__device__ __forceinline__ uint32_t zc0_rc(const AirConsts& K, int i) {
  if (i >= 16 && i < 64) return K.begin[(i - 16) / 16 + 1][i & 15];
  if (i >= 100) return K.end[(i - 100) / 16 + 1][(i - 100) & 15];
  return 0u;
}

// The constant operands of k_zc0_eval_mma as its lanes hold them: the Lagrange weights,
// frags[((mt * 32 + lane) * 4 + b) * 8 + 4 kk + o] = byte b of L_j(z) 2^(8a + 16) in byte a, z = 16 mt + g + 8 (o & 1), j = 8 kk + t + 4 (o >> 1); and the
// weights gamma, frags[ZC0_FRAG_G + (grp * 32 + lane) * 8 + 2 b + h] = the same of the Montgomery
// form of 2^(8a) times coefficient g of gamma_i, i = 8 grp + 2t + h (zero past the last input).
constexpr int ZC0_GRPS = (AIR_NC + 7) / 8;
constexpr int ZC0_FRAG_G = 2 * 32 * 32;
static_assert(ZC0_FRAG_G + ZC0_GRPS * 32 * 8 == ZC0_FRAG_WORDS, "operand table");
template <int E>  // w[b] = byte b of v 2^(8a + E - 32), a = 0..3 (v in Montgomery form)
__device__ __forceinline__ void limb_columns(uint32_t v, uint32_t (&w)[4]) {
  uint32_t m[4];
#pragma unroll
  for (int a = 0; a < 4; a++) m[a] = kb::mul(v, uint32_t(kb::detail::cpow(2, 8 * a + E)));
#pragma unroll
  for (int b = 0; b < 4; b++)
    w[b] = ((m[0] >> (8 * b)) & 0xffu) | (((m[1] >> (8 * b)) & 0xffu) << 8) | (((m[2] >> (8 * b)) & 0xffu) << 16) |
           (((m[3] >> (8 * b)) & 0xffu) << 24);
}
__device__ void zc0_fragments(int nz, int nsk, const uint32_t* __restrict__ lw, const ef* __restrict__ alphas,
                              const ef* __restrict__ betas, uint32_t* __restrict__ frags) {
  for (int e = threadIdx.x; e < 2 * 32 * 8; e += blockDim.x) {
    const int lane = (e >> 3) & 31, kk = (e >> 2) & 1, o = e & 3;
    const int z = 16 * (e >> 8) + (lane >> 2) + 8 * (o & 1), j = 8 * kk + (lane & 3) + 4 * (o >> 1);
    uint32_t w[4];
    limb_columns<16>(z < nz && j < nsk ? lw[z * nsk + j] : 0u, w);
#pragma unroll
    for (int b = 0; b < 4; b++) frags[(e >> 3) * 32 + b * 8 + 4 * kk + o] = w[b];
  }
  for (int e = threadIdx.x; e < ZC0_GRPS * 32 * 2; e += blockDim.x) {
    const int lane = (e >> 1) & 31, i = 8 * (e >> 6) + 2 * (lane & 3) + (e & 1);
    const ef* gm = i < 64 ? betas + i : i < 84 ? alphas + i : betas + i - 20;
    uint32_t w[4];
    limb_columns<32>(i < AIR_NC ? gm->c[lane >> 2] : 0u, w);
#pragma unroll
    for (int b = 0; b < 4; b++) frags[ZC0_FRAG_G + (e >> 1) * 8 + 2 * b + (e & 1)] = w[b];
  }
}

// One thread per row r = j S + x, reading the row's up row. Writes q[c * N + r]:
//   c < 16       MDS(inputs)_c + rc_begin[0][c]
//   16 <= c < 36 state word 0 before partial round c - 16, plus its round constant
//   36 <= c < 52 state after the 20 partial rounds, plus rc_end[0]
// and the committed-column term -L_j(z) sum_r eq[x] sum_i alpha_i col_(17+i) of the block's
// rows as partial[blockIdx.x * nz + z]; arow[r] = sum_i alpha_i col_(17+i) (the later rounds
// carry its fold as one more column).
// A thread's row is one chain: 37 steps of four column products, then 20 partial rounds, each
// waiting for its loads. The loads run ZC0R_AHEAD words (4 in the rounds) ahead of their use:
// 2^12 rows 38 us before, 25 after; 2^20 rows 424 us both ways (other warps hid the waits).
// A table whose rows in blocks of 256 leave SMs idle runs in blocks of 64.
constexpr int ZC0R_THREADS = 256;
constexpr int ZC0R_SMALL = 64;
constexpr int ZC0R_AHEAD = 12;  // a multiple of 4
__global__ void __launch_bounds__(ZC0R_THREADS) k_zc0_rows(const uint32_t* __restrict__ wit, int log_n, int k,
                                                           int nz, const uint32_t* __restrict__ lw,
                                                           const ef* __restrict__ eq,
                                                           const ef* __restrict__ alphas_g,
                                                           const ef* __restrict__ betas_g,
                                                           const __grid_constant__ AirConsts K,
                                                           uint32_t* __restrict__ q, ef* __restrict__ partial,
                                                           ef* __restrict__ arow, uint32_t* __restrict__ frags) {
  if (blockIdx.x == gridDim.x - 1) {
    zc0_fragments(nz, 1 << k, lw, alphas_g, betas_g, frags);
    return;
  }
  __shared__ ef alphas[AIR_NC];
  __shared__ ef scratch[32];
  __shared__ ef total;
  __shared__ ef rows[ZC0R_THREADS], sums[16];
  for (int i = threadIdx.x; i < AIR_NC; i += blockDim.x) alphas[i] = alphas_g[i];
  __syncthreads();
  const int lS = log_n - k;
  const size_t N = size_t(1) << log_n;
  const size_t rb = size_t(blockIdx.x) * blockDim.x;
  const size_t r = rb + threadIdx.x;
  ef c = ef_zero();
  if (r < N) {
    const uint32_t* row = wit + up_row(r, N);
    EfMacF m;
    m.init();
    // ZC0R_AHEAD column loads in flight ahead of the products that use them
    uint32_t v[ZC0R_AHEAD];
#pragma unroll
    for (int e = 0; e < ZC0R_AHEAD; e++) v[e] = __ldg(row + size_t(17 + e) * N);
#pragma unroll 1
    for (int i = 0; i < AIR_NC; i += 4) {
      uint32_t u[4];
#pragma unroll
      for (int e = 0; e < 4; e++) u[e] = v[e];
#pragma unroll
      for (int e = 0; e + 4 < ZC0R_AHEAD; e++) v[e] = v[e + 4];
      if (i + ZC0R_AHEAD < AIR_NC) {
#pragma unroll
        for (int e = 0; e < 4; e++) v[ZC0R_AHEAD - 4 + e] = __ldg(row + size_t(17 + i + ZC0R_AHEAD + e) * N);
      }
#pragma unroll
      for (int e = 0; e < 4; e++) m.mac(alphas[i + e], u[e]);
      m.flush();
    }
    uint32_t s[16];
#pragma unroll
    for (int t = 0; t < 16; t++) s[t] = __ldg(row + size_t(1 + t) * N);
    mds_light<16>(s);
    uint32_t* qr = q + r;
#pragma unroll
    for (int t = 0; t < 16; t++) qr[size_t(t) * N] = add(s[t], K.begin[0][t]);
#pragma unroll
    for (int t = 0; t < 16; t++) s[t] = __ldg(row + size_t(65 + t) * N);
    uint32_t post[4];
#pragma unroll
    for (int e = 0; e < 4; e++) post[e] = __ldg(row + size_t(81 + e) * N);
#pragma unroll 1
    for (int pr = 0; pr < 20; pr++) {
      const uint32_t p0 = post[0];
#pragma unroll
      for (int e = 0; e < 3; e++) post[e] = post[e + 1];
      if (pr + 4 < 20) post[3] = __ldg(row + size_t(81 + pr + 4) * N);
      qr[size_t(16 + pr) * N] = add(s[0], K.partial[pr]);
      internal_layer_with0<16>(s, p0);
    }
#pragma unroll
    for (int t = 0; t < 16; t++) qr[size_t(36 + t) * N] = add(s[t], K.end[0][t]);
    const ef a = m.value();
    arow[r] = a;
    c = ef_mul(a, eq[r & ((size_t(1) << lS) - 1)]);
  }
  const int nsk = 1 << k;
  const int S = lS < 16 ? 1 << lS : 1 << 16;  // only compared with the block
  if (S >= int(blockDim.x)) {  // one skip index j in the block: reduce, then weight
    const ef tot = block_reduce_ef(c, scratch);
    if (threadIdx.x == 0) total = tot;
    __syncthreads();
    const int j = int(rb >> lS);
    for (int z = threadIdx.x; z < nz; z += blockDim.x)
      partial[size_t(blockIdx.x) * nz + z] = ef_sub(ef_zero(), ef_mul_f(total, lw[size_t(z) * nsk + j]));
  } else {  // S divides the block: sum the rows of each j, then weight the sums per point
    rows[threadIdx.x] = c;
    __syncthreads();
    const int j0 = int(rb >> lS), nj = min(int(blockDim.x), int(N - rb)) >> lS;
    for (int e = threadIdx.x; e < nj * 8; e += blockDim.x) {
      uint32_t v = 0;
      for (int i = 0; i < S; i++) v = add(v, rows[((e >> 3) << lS) + i].c[e & 7]);
      sums[e >> 3].c[e & 7] = v;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nz * 8; e += blockDim.x) {
      uint32_t v = 0;
      for (int j = 0; j < nj; j++) v = add(v, kb::mul(sums[j].c[e & 7], lw[size_t(e >> 3) * nsk + j0 + j]));
      partial[size_t(blockIdx.x) * nz + (e >> 3)].c[e & 7] = kb::neg(v);
    }
  }
}

// The 148 cube inputs of every row x are extended from their values at rows j S + x, j < 2^k,
// to the points z by the Lagrange weights L_j(z), cubed, weighted by gamma and summed, weighted
// by eq[x]. Both contractions run on the tensor cores as byte-limb integer products.
// Extension: u(z) = sum_j L_j(z) v_j(x) with rows z, reduction index (j, a) over the 16 points j
// and the 4 bytes a of v_j(x), columns the 8 inputs of a group, one product per byte b of
// M(j, z, a) = L_j(z) 2^(8a + 16). The staged words [input][j][x] are the B operand as they lie
// (byte a of word j is k = 4j + a). The accumulators start from the two halves of the round
// constant times 2^16 (bytes 0 and 2). With acc_b <= 64 255^2 + 2^16, the sum sum_b acc_b 2^(8b) =
// lo + 2^16 hi, lo and hi below 1.07 10^9, is congruent to 2^16 times the cube input; since
// p = 1 mod 2^16, dividing by 2^16 takes hi + (lo >> 16) - (lo mod 2^16) (p - 1) / 2^16, which
// lies in (-p, 1.08 10^9): one small multiply where a Montgomery reduction takes two wide ones.
// Weights: sum_i gamma_i cube_i with rows z, reduction index (i, a) over the inputs and the bytes
// of the cube, columns (coefficient n of gamma, byte b). The lane that ends the extension with
// inputs 2t, 2t + 1 of rows g, g + 8 needs exactly these words as its A operand when k-slot t
// stands for input 2t and slot t + 4 for 2t + 1, so the cubes never leave their lane; they need
// not be reduced either (any word congruent to the cube serves, here below 2p).
// A block holds 8 x and the 32 point slots; warp (z-tile mt, xg) takes x = 2 xg, 2 xg + 1: per
// group of 8 inputs and x, 8 products for the extension and 4 for the weights. The values are
// staged by a cp.async pipeline, 8 inputs per stage, a warp per input and 16 bytes per lane;
// weights of j >= 2^k are zero, so unstaged entries contribute nothing.
// 2^20 rows: 1.23 ms with the weights as 8 multiply-adds per cube on the multiply pipe, 0.94 with
// both contractions here, 0.88 with the division by 2^16, 0.78 with 16-byte staging (4-byte pieces
// took a quarter of the instructions); 2^16 rows 0.101 -> 0.064. Bound by latency at 16 warps an SM
// (the operands held in registers allow no more): 45% of issue slots, multiply pipe 55%.
// A block walks 19 groups of inputs one after the other; with too few x blocks to fill the chip
// (2 an SM) the groups are split over blockIdx.y, each block with its own partial sums: 2^12 rows
// on the multiply pipe 110 us without the split, 17 with it.
constexpr int ZC0_FILL = 2 * 148;
constexpr int ZC0M_WARPS = 8;
constexpr int ZE_X = 8;
constexpr int ZE_IN = 16 * ZE_X + 12;  // words per staged input (8-byte reads of lanes (g, t): every bank twice)
__global__ void __launch_bounds__(ZC0M_WARPS * 32, 2) k_zc0_eval_mma(const uint32_t* __restrict__ wit,
                                                                    const uint32_t* __restrict__ q, int log_n,
                                                                    int k, int nz, const ef* __restrict__ eq,
                                                                    const uint32_t* __restrict__ frags,
                                                                    const __grid_constant__ AirConsts K,
                                                                    ef* __restrict__ partial) {
  __shared__ __align__(16) uint32_t tile[ZC0_STAGES][8 * ZE_IN];
  __shared__ ef sums[ZE_X][32];
  __shared__ int rcs[ZC0_GRPS * 8];  // the round constants times 2^16
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3, mt = warp & 1, xg = warp >> 1;
  for (int i = tid; i < ZC0_GRPS * 8; i += ZC0M_WARPS * 32) rcs[i] = i < AIR_NC ? int(kb::mul(zc0_rc(K, i), uint32_t(kb::detail::cpow(2, 48)))) : 0;
  const size_t N = size_t(1) << log_n, S = N >> k;
  const size_t x0 = size_t(blockIdx.x) * ZE_X;
  uint32_t af[4][2][4];
#pragma unroll
  for (int b = 0; b < 4; b++)
#pragma unroll
    for (int kk = 0; kk < 2; kk++) {
      const uint4 v = reinterpret_cast<const uint4*>(frags)[(mt * 32 + lane) * 8 + b * 2 + kk];
      af[b][kk][0] = v.x;
      af[b][kk][1] = v.y;
      af[b][kk][2] = v.z;
      af[b][kk][3] = v.w;
    }
  // staged piece of this thread: x0 + 4 h .. + 3 of row block j of its warp's input of each group;
  // one by one where the block is cut short or holds row N - 1, whose up row is N - 2 (committed
  // columns only)
  const int j = lane >> 1, h = lane & 1;
  const bool stage = j < (1 << k), whole = x0 + ZE_X <= S && S % 4 == 0;
  const size_t row = size_t(j) * S + x0 + 4 * h;
  const int per = (ZC0_GRPS + gridDim.y - 1) / gridDim.y, g0 = blockIdx.y * per, g1 = min(g0 + per, ZC0_GRPS);
  auto issue = [&](int grp) {
    const int i = 8 * grp + warp;
    if (stage && i < AIR_NC && grp < g1) {
      const int qc = zc0_qcol(i);
      const uint32_t* col = qc >= 0 ? q + size_t(qc) * N : wit + size_t(1 + i) * N;
      uint32_t* dst = tile[grp % ZC0_STAGES] + warp * ZE_IN + j * ZE_X + 4 * h;
      if (whole && (qc >= 0 || row + 4 != N)) {
        cp_async16(dst, col + row);
      } else {
        for (int e = 0; e < 4; e++) {
          const size_t r = row + e;
          if (x0 + 4 * h + e < S) cp_async4(dst + e, col + (r == N - 1 && qc < 0 ? N - 2 : r));
        }
      }
    }
    cp_async_commit();
  };
  for (int grp = g0; grp < g0 + ZC0_STAGES - 1; grp++) issue(grp);
  int acc2[2][4][4];
#pragma unroll
  for (int xq = 0; xq < 2; xq++)
#pragma unroll
    for (int b = 0; b < 4; b++)
#pragma unroll
      for (int o = 0; o < 4; o++) acc2[xq][b][o] = 0;
#pragma unroll 1
  for (int grp = g0; grp < g1; grp++) {
    const uint4* gf = reinterpret_cast<const uint4*>(frags + ZC0_FRAG_G) + (grp * 32 + lane) * 2;
    const uint4 gl = __ldg(gf), gh = __ldg(gf + 1);
    const uint32_t gb[4][2] = {{gl.x, gl.y}, {gl.z, gl.w}, {gh.x, gh.y}, {gh.z, gh.w}};
    cp_async_wait<ZC0_STAGES - 2>();
    __syncthreads();  // group grp landed for every thread; the slot of group grp - 1 is free
    issue(grp + ZC0_STAGES - 1);
    const int rc[2] = {rcs[8 * grp + 2 * t], rcs[8 * grp + 2 * t + 1]};
    uint2 vw[4];  // words j = t, t + 4, t + 8, t + 12 of input g at the warp's two x
#pragma unroll
    for (int e = 0; e < 4; e++)
      vw[e] = *reinterpret_cast<const uint2*>(tile[grp % ZC0_STAGES] + g * ZE_IN + (t + 4 * e) * ZE_X + 2 * xg);
#pragma unroll
    for (int xq = 0; xq < 2; xq++) {
      const uint32_t v0 = xq ? vw[0].y : vw[0].x, v1 = xq ? vw[1].y : vw[1].x;
      const uint32_t v2 = xq ? vw[2].y : vw[2].x, v3 = xq ? vw[3].y : vw[3].x;
      int acc[4][4];
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const int r0 = b == 0 ? rc[0] & 0xffff : b == 2 ? rc[0] >> 16 : 0;
        const int r1 = b == 0 ? rc[1] & 0xffff : b == 2 ? rc[1] >> 16 : 0;
        mma_u8_16832_from(acc[b], af[b][0], v0, v1, r0, r1, r0, r1);
        mma_u8_16832_from(acc[b], af[b][1], v2, v3, acc[b][0], acc[b][1], acc[b][2], acc[b][3]);
      }
      uint32_t w[4];  // (z, input) = (g, 2t), (g, 2t + 1), (g + 8, 2t), (g + 8, 2t + 1)
#pragma unroll
      for (int o = 0; o < 4; o++) {
        const uint32_t lo = uint32_t(acc[0][o]) + (uint32_t(acc[1][o]) << 8);
        const uint32_t hi = uint32_t(acc[2][o]) + (uint32_t(acc[3][o]) << 8);
        const uint32_t r = hi + (lo >> 16) + kb::P - (lo & 0xffffu) * ((kb::P - 1) >> 16);
        const uint32_t u = kb::umin(r, r - kb::P);
        w[o] = kb::mul_lazy(kb::mul_lazy(u, u), u);
      }
      const uint32_t ca[4] = {w[0], w[2], w[1], w[3]};
#pragma unroll
      for (int b = 0; b < 4; b++)
        mma_u8_16832_from(acc2[xq][b], ca, gb[b][0], gb[b][1], acc2[xq][b][0], acc2[xq][b][1], acc2[xq][b][2],
                          acc2[xq][b][3]);
    }
  }
  cp_async_wait<0>();
  // lane (g, t) holds coefficients 2t, 2t + 1 of rows z = 16 mt + g and + 8 (acc2 < 2^26 each)
#pragma unroll
  for (int xq = 0; xq < 2; xq++)
#pragma unroll
    for (int o = 0; o < 4; o++)
      sums[2 * xg + xq][16 * mt + g + 8 * (o >> 1)].c[2 * t + (o & 1)] =
          kb::redc(uint64_t(uint32_t(acc2[xq][0][o])) + (uint64_t(uint32_t(acc2[xq][1][o])) << 8) +
                   (uint64_t(uint32_t(acc2[xq][2][o])) << 16) + (uint64_t(uint32_t(acc2[xq][3][o])) << 24));
  __syncthreads();
  if (x0 + warp < S) sums[warp][lane] = ef_mul(sums[warp][lane], eq[x0 + warp]);
  else sums[warp][lane] = ef_zero();
  __syncthreads();
  const int z = tid >> 3, n = tid & 7;
  if (z >= nz) return;
  uint32_t s = 0;
#pragma unroll
  for (int x = 0; x < ZE_X; x++) s = add(s, sums[x][z].c[n]);
  partial[(size_t(blockIdx.y) * gridDim.x + blockIdx.x) * nz + z].c[n] = s;
}

// out[x] = sum_j sel[j] * a[j S + x] for the block's 32 x of an extension-field table a that is
// already read at up rows (the committed-column combination of k_zc0_rows). Warp w takes j = w,
// w + 8 of all 32 x; the eight sums of an x are added through shared memory, one coefficient of
// one x per thread.
__device__ void zc0_fold_arow(const ef* __restrict__ a, int log_n, int k, const ef* __restrict__ sel,
                              ef* __restrict__ out, ef* sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t S = size_t(1) << (log_n - k), x0 = size_t(blockIdx.x) * ZC0_X, x = x0 + lane;
  EfMacE m;
  m.init();
  if (x < S)
    for (int j = warp; j < (1 << k); j += ZC0M_WARPS) m.mac(sel[j], a[size_t(j) * S + x]);
  sums[warp * ZC0_X + lane] = m.value();
  __syncthreads();
  const int xl = threadIdx.x >> 3, c = threadIdx.x & 7;
  uint32_t v = 0;
#pragma unroll
  for (int w = 0; w < ZC0M_WARPS; w++) v = add(v, sums[w * ZC0_X + xl].c[c]);
  if (x0 + xl < S) out[x0 + xl].c[c] = v;
}

// The columns the rounds >= 1 carry: the 148 cube inputs, first the ZC0_NQ computed ones in
// q's order, then the committed ones in constraint order (zc_wit_col), and last the
// committed-column combination.
__device__ __forceinline__ int zc_wit_col(int c) { return c < 100 ? c - 35 : c + 1; }

// out[(c - cb) * S + x] = sum_j sel[j] * v_c[j * S + x] for the cube inputs cb <= c < ce (either
// all computed, src = q, or all committed, src = the witness at up rows), on the tensor cores as
// in k_zc0_eval_mma: rows x, reduction index (j, a) over the 16 points and the 4 bytes of
// v_c[j S + x] (the staged [x][j] words as they lie), columns (n, b) for the 8 coefficients n
// of sel[j] and the 4 bytes b of the Montgomery form of sel[j]_n 2^(8a). Each lane ends with
// all limbs of coefficients 2t, 2t + 1 of rows g, g + 8; one Montgomery reduction each. A
// block holds 32 x and walks the columns in staged groups of ZC0_GROUP; warp (tile, slot)
// takes columns slot and slot + 4 of each group. The up row of row N - 1 is N - 2. The groups are
// split over blockIdx.y as in k_zc0_eval_mma (no sum to join here); with arow, the last
// blockIdx.y folds it as column ce: 2^12 rows 24 + 17 us as two launches of 8 and 1 blocks over
// all 166 columns, 5 us in one.
__global__ void __launch_bounds__(ZC0M_WARPS * 32) k_zc0_fold_mma(const uint32_t* __restrict__ src, int log_n,
                                                                 int k, int cb, int ce,
                                                                 const ef* __restrict__ sel,
                                                                 const ef* __restrict__ arow,
                                                                 ef* __restrict__ out) {
  __shared__ __align__(16) uint32_t tile[ZC0_STAGES][ZC0_GROUP][ZC0_X * ZC0_PAD];
  constexpr int NT = ZC0M_WARPS * 32;
  if (arow && blockIdx.y == gridDim.y - 1) {
    zc0_fold_arow(arow, log_n, k, sel, out + (size_t(ce - cb) << (log_n - k)), reinterpret_cast<ef*>(tile));
    return;
  }
  const bool comp = ce <= ZC0_NQ;  // computed inputs: the columns of src, already read at up rows
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3, mt = warp & 1, slot = warp >> 1;
  const int nsk = 1 << k;
  const size_t N = size_t(1) << log_n;
  const size_t S = N >> k;
  const size_t x0 = size_t(blockIdx.x) * ZC0_X;
  // B fragments: bf[b][kk][h] packs, in byte a, byte b of the Montgomery form of
  // sel[j]_n 2^(8a) for j = 8 kk + 4 h + t and coefficient n = g (the lane's B column)
  uint32_t bf[4][2][2];
#pragma unroll
  for (int kk = 0; kk < 2; kk++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int j = 8 * kk + 4 * h + t;
      const uint32_t v = j < nsk ? sel[j].c[g] : 0u;
      uint32_t m[4];
#pragma unroll
      for (int a = 0; a < 4; a++) m[a] = kb::mul(v, uint32_t(kb::detail::cpow(2, 8 * a + 32)));
#pragma unroll
      for (int b = 0; b < 4; b++)
        bf[b][kk][h] = ((m[0] >> (8 * b)) & 0xffu) | (((m[1] >> (8 * b)) & 0xffu) << 8) |
                       (((m[2] >> (8 * b)) & 0xffu) << 16) | (((m[3] >> (8 * b)) & 0xffu) << 24);
    }
  constexpr int NE = (16 * ZC0_X + NT - 1) / NT;
  uint32_t srow[NE], sdst[NE];
  bool sval[NE];
#pragma unroll
  for (int e = 0; e < NE; e++) {
    const int idx = tid + e * NT;
    const int j = idx / ZC0_X, xl = idx % ZC0_X;
    size_t xx = x0 + xl;
    if (xx >= S) xx = 0;
    sval[e] = idx < 16 * ZC0_X && j < nsk;
    const size_t row = size_t(j) * S + xx;
    srow[e] = uint32_t(row == N - 1 && !comp ? N - 2 : row);
    sdst[e] = uint32_t(xl * ZC0_PAD + j);
  }
  const int ng = (ce - cb + ZC0_GROUP - 1) / ZC0_GROUP;
  const int splits = gridDim.y - (arow ? 1 : 0), per = (ng + splits - 1) / splits;
  const int g0 = blockIdx.y * per, g1 = min(g0 + per, ng);
  auto issue = [&](int grp) {
#pragma unroll
    for (int cc = 0; cc < ZC0_GROUP; cc++) {
      const int c = cb + ZC0_GROUP * grp + cc;
      if (c < ce && grp < g1) {
        const uint32_t* col = src + size_t(comp ? c : zc_wit_col(c)) * N;
        uint32_t* dst = tile[grp % ZC0_STAGES][cc];
#pragma unroll
        for (int e = 0; e < NE; e++)
          if (sval[e]) cp_async4(dst + sdst[e], col + srow[e]);
      }
    }
    cp_async_commit();
  };
  for (int grp = g0; grp < g0 + ZC0_STAGES - 1; grp++) issue(grp);
  const size_t xa = x0 + 16 * mt + g, xb = xa + 8;
#pragma unroll 1
  for (int grp = g0; grp < g1; grp++) {
    cp_async_wait<ZC0_STAGES - 2>();
    __syncthreads();  // group grp landed for every thread; the slot of group grp - 1 is free
    issue(grp + ZC0_STAGES - 1);
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const int cc = slot + 4 * r;
      const int c = cb + ZC0_GROUP * grp + cc;
      if (c >= ce) break;
      const uint32_t* r0 = tile[grp % ZC0_STAGES][cc] + (16 * mt + g) * ZC0_PAD;
      const uint32_t* r1 = r0 + 8 * ZC0_PAD;
      int acc[4][4];
#pragma unroll
      for (int b = 0; b < 4; b++)
#pragma unroll
        for (int o = 0; o < 4; o++) acc[b][o] = 0;
#pragma unroll
      for (int kk = 0; kk < 2; kk++) {
        const uint32_t af[4] = {r0[8 * kk + t], r1[8 * kk + t], r0[8 * kk + t + 4], r1[8 * kk + t + 4]};
#pragma unroll
        for (int b = 0; b < 4; b++) mma_u8_16832(acc[b], af, bf[b][kk][0], bf[b][kk][1]);
      }
      uint32_t res[4];
#pragma unroll
      for (int o = 0; o < 4; o++) {
        const uint32_t lo = uint32_t(acc[0][o]) + (uint32_t(acc[1][o]) << 8);  // < 2^31
        const uint32_t hi = uint32_t(acc[2][o]) + (uint32_t(acc[3][o]) << 8);  // < 2^31
        res[o] = kb::redc(uint64_t(lo) + (uint64_t(hi) << 16));
      }
      if (xa < S) reinterpret_cast<uint2*>(out + size_t(c - cb) * S + xa)[t] = make_uint2(res[0], res[1]);
      if (xb < S) reinterpret_cast<uint2*>(out + size_t(c - cb) * S + xb)[t] = make_uint2(res[2], res[3]);
    }
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------------------ zerocheck rounds >= 1
// The batched constraint at the points z = 0, 2, 3 of every x < 2^(m-1), weighted by eq[x]: the
// 148 cube inputs and the committed-column combination are the carried columns (each an affine
// function of the row, so their values at z are lo + z (hi - lo) of the folded columns, lo, hi
// at x and 2^(m-1) + x), and the constraint is sum_c gamma_c cube(u_c + rc_c) minus the
// combination: no linear layer is left in these rounds, and 149 columns are folded, not 166.
// (Carrying the 165 witness columns instead needs the MDS of the inputs and the chain of the 20
// partial rounds at every point: for 2^20 rows the six rounds of 2^10 points and more took 1.73 ms
// and the ten smaller ones 0.21 ms; here 1.09 and 0.11 ms. 2^12 rows: 8 rounds 135, here 74 us.)
// A warp holds 32 x, one z and every fourth column of its block's share; the three z of a block
// read the same lines (L1 hit rate 95%). Bound by the wide multiplies: about 240 per column and
// point (square, product, weight, reductions) keep the multiply pipe 85% busy. Columns are split
// over blockIdx.y until the grid is two waves of 2 blocks an SM (six waves measured 1.16 ms: more
// epilogues, and their partial sums need a second reduction), so a round of few x has one column
// per warp and takes the latency of one term.
constexpr int ZCS_COLS = 4;                          // columns at a time in a block
constexpr int ZCS_THREADS = 3 * ZCS_COLS * 32;
struct ZcCols {  // columns [0, split) at a, the rest at b
  const ef *a, *b;
  int split;
  __device__ __forceinline__ const ef* col(int c, size_t len) const {
    return c < split ? a + size_t(c) * len : b + size_t(c - split) * len;
  }
};
__device__ __forceinline__ uint32_t zc_const(int c, const AirConsts& K) {
  if (c < 52) return 0u;  // the computed inputs include theirs
  return c < 100 ? K.begin[(c - 52) / 16 + 1][(c - 52) & 15] : K.end[(c - 100) / 16 + 1][(c - 100) & 15];
}
__global__ void __launch_bounds__(ZCS_THREADS, 2) k_zc_sbox(ZcCols cols, int m, const ef* __restrict__ eq,
                                                            const ef* __restrict__ gam,
                                                            const __grid_constant__ AirConsts K,
                                                            ef* __restrict__ partial) {
  __shared__ ef red[3][ZCS_COLS];
  const size_t len = size_t(1) << m, half = len >> 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, zi = warp % 3, cg = warp / 3;
  const size_t x = size_t(blockIdx.x) * 32 + lane;
  const bool valid = x < half;
  const size_t xs = valid ? x : 0;
  auto at = [&](const ef* col) {  // the column's value at the warp's z
    ef lo = col[xs];
    if (zi) {
      const ef d = ef_sub(col[xs + half], lo);
      const ef d2 = ef_add(d, d);
      lo = ef_add(lo, zi == 1 ? d2 : ef_add(d2, d));
    }
    return lo;
  };
  EfMacE acc;
  acc.init();
#pragma unroll 1
  for (int c = blockIdx.y * ZCS_COLS + cg; c < AIR_NC; c += gridDim.y * ZCS_COLS) {
    const ef u = ef_add_f(at(cols.col(c, len)), zc_const(c, K));
    acc.mac3(ef_cube(u), gam[2 * c], gam[2 * c + 1]);
  }
  ef v = acc.value();
  if (blockIdx.y == 0 && cg == 0) v = ef_sub(v, at(cols.col(AIR_NC, len)));
  v = warp_reduce_ef(valid ? ef_mul(v, eq[xs]) : ef_zero());
  if (lane == 0) red[zi][cg] = v;
  __syncthreads();
  if (threadIdx.x < 24) {
    const int z = threadIdx.x >> 3, n = threadIdx.x & 7;
    uint32_t s = red[z][0].c[n];
#pragma unroll
    for (int g = 1; g < ZCS_COLS; g++) s = add(s, red[z][g].c[n]);
    partial[(size_t(blockIdx.y) * gridDim.x + blockIdx.x) * 3 + z].c[n] = s;
  }
}

// Folds every column at the challenge (*r, or rv when r is null) and, in the extra column
// slot, sums the next round's eq table out of the current one.
__global__ void k_fold_cols(const ef* __restrict__ in, ef* __restrict__ out, size_t half, int ncols,
                            const ef* __restrict__ r, ef rv, const ef* __restrict__ eq_in, ef* __restrict__ eq_out,
                            size_t eq_half) {
  const size_t x = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int c = blockIdx.y;
  if (c == ncols) {
    if (x < eq_half) eq_out[x] = ef_add(eq_in[x], eq_in[x + eq_half]);
    return;
  }
  if (x >= half) return;
  const ef* src = in + size_t(c) * 2 * half;
  out[size_t(c) * half + x] = ef_lerp(src[x], src[half + x], r ? *r : rv);
}

// lo + r (hi - lo) for the 16 values of a warp's tile on the tensor cores (byte-limb value
// form): r d = sum_e d_e (X^e r), so the product is a matrix product with rows = values,
// reduction index = (coefficient e of d, byte a), columns = (n, b) for the 8 coefficients n and
// 4 bytes b of the Montgomery form of (X^e r)_n 2^(8a) (the lane's B fragments, fold_frag).
// One k32 step: four mma per 16 values; acc_b < 32 255^2, one reduction per coefficient.
__device__ __forceinline__ void fold_frag(const ef& r, int g, int t, uint32_t (&bf)[4][2]) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int e = t + 4 * h;
    // (X^e r)_g = r_(g - e), times 3 where X^8 = 3 wraps it
    const uint32_t w = g >= e ? r.c[g - e] : kb::add(kb::dbl(r.c[g - e + 8]), r.c[g - e + 8]);
    uint32_t m[4];
#pragma unroll
    for (int a = 0; a < 4; a++) m[a] = kb::mul(w, uint32_t(kb::detail::cpow(2, 8 * a + 32)));
#pragma unroll
    for (int b = 0; b < 4; b++)
      bf[b][h] = ((m[0] >> (8 * b)) & 0xffu) | (((m[1] >> (8 * b)) & 0xffu) << 8) |
                 (((m[2] >> (8 * b)) & 0xffu) << 16) | (((m[3] >> (8 * b)) & 0xffu) << 24);
  }
}
__device__ __forceinline__ void lerp16_mma(const ef* __restrict__ lo, const ef* __restrict__ hi, ef* __restrict__ out,
                                           uint32_t nv, const uint32_t (&bf)[4][2], int g, int t) {
  const uint32_t* l32 = reinterpret_cast<const uint32_t*>(lo);
  const uint32_t* h32 = reinterpret_cast<const uint32_t*>(hi);
  const bool va = uint32_t(g) < nv, vb = uint32_t(g + 8) < nv;
  auto dw = [&](int row, int e, bool v) -> uint32_t { return v ? kb::sub(h32[row * 8 + e], l32[row * 8 + e]) : 0u; };
  const uint32_t af[4] = {dw(g, t, va), dw(g + 8, t, vb), dw(g, t + 4, va), dw(g + 8, t + 4, vb)};
  int acc[4][4];
#pragma unroll
  for (int b = 0; b < 4; b++) {
#pragma unroll
    for (int o = 0; o < 4; o++) acc[b][o] = 0;
    mma_u8_16832(acc[b], af, bf[b][0], bf[b][1]);
  }
  auto prod = [&](int o) {
    return kb::redc(uint64_t(uint32_t(acc[0][o])) + (uint64_t(uint32_t(acc[1][o])) << 8) +
                    (uint64_t(uint32_t(acc[2][o])) << 16) + (uint64_t(uint32_t(acc[3][o])) << 24));
  };
  // lane (g, t) holds coefficients 2t, 2t + 1 of rows g and g + 8
  if (va) {
    const uint2 l = reinterpret_cast<const uint2*>(lo + g)[t];
    reinterpret_cast<uint2*>(out + g)[t] = make_uint2(kb::add(l.x, prod(0)), kb::add(l.y, prod(1)));
  }
  if (vb) {
    const uint2 l = reinterpret_cast<const uint2*>(lo + g + 8)[t];
    reinterpret_cast<uint2*>(out + g + 8)[t] = make_uint2(kb::add(l.x, prod(2)), kb::add(l.y, prod(3)));
  }
}
// k_fold_cols with the challenge by value, 16 values per warp on the tensor cores; the extra
// column slot (blockIdx.y == ncols) sums the next eq table as k_fold_cols does.
// The challenge comes by value (rv) or, when rptr is set, from device memory (a challenge
// sampled on the device by the round-finishing kernel).
__global__ void __launch_bounds__(256) k_fold_cols_mma(ZcCols in, ef* __restrict__ out, size_t half,
                                                      int ncols, ef rv, const ef* __restrict__ rptr,
                                                      const ef* __restrict__ eq_in, ef* __restrict__ eq_out,
                                                      size_t eq_half) {
  const int c = blockIdx.y;
  if (c == ncols) {
    for (size_t x = size_t(blockIdx.x) * blockDim.x + threadIdx.x; x < eq_half; x += size_t(gridDim.x) * blockDim.x)
      eq_out[x] = ef_add(eq_in[x], eq_in[x + eq_half]);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  size_t x0 = (size_t(blockIdx.x) * 8 + warp) * 16;
  if (x0 >= half) return;  // whole warp
  uint32_t bf[4][2];
  fold_frag(rptr ? *rptr : rv, g, t, bf);
  const ef* src = in.col(c, 2 * half);
  for (; x0 < half; x0 += size_t(gridDim.x) * 128) {
    const uint32_t nv = half - x0 < 16 ? uint32_t(half - x0) : 16u;
    lerp16_mma(src + x0, src + half + x0, out + size_t(c) * half + x0, nv, bf, g, t);
  }
}
// lo + r (hi - lo) for two tables with the challenge by value: blockIdx.y selects (a, oa) or (b, ob).
__global__ void __launch_bounds__(256) k_fold2_mma(const ef* __restrict__ a, const ef* __restrict__ b,
                                                  ef* __restrict__ oa, ef* __restrict__ ob, size_t half, ef rv,
                                                  const ef* __restrict__ rptr) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const size_t x0 = (size_t(blockIdx.x) * 8 + warp) * 16;
  if (x0 >= half) return;  // whole warp
  uint32_t bf[4][2];
  fold_frag(rptr ? *rptr : rv, g, t, bf);
  const ef* src = blockIdx.y ? b : a;
  ef* dst = blockIdx.y ? ob : oa;
  const uint32_t nv = half - x0 < 16 ? uint32_t(half - x0) : 16u;
  lerp16_mma(src + x0, src + half + x0, dst + x0, nv, bf, g, t);
}

// Per (column c, j < 2^k, x_hi): eq_hi[x_hi] * sum_{x_lo} eq_lo[x_lo] * up_c[j S + x] (and the
// same for down), x = x_hi 2^ll + x_lo, with eq(tail, x) = eq_hi(x_hi) eq_lo(x_lo) factored so
// every warp reads the same small eq_lo table. One warp per x_hi; 2^ll is a multiple of 32
// or smaller than 32. Outputs pu/pd[(c * 2^k + j) * nhi + x_hi].
constexpr int IS_WARPS = 8;
__global__ void __launch_bounds__(IS_WARPS * 32) k_inner_sums(const uint32_t* __restrict__ wit, int log_n, int k,
                                                              int ll, const ef* __restrict__ eq_hi,
                                                              const ef* __restrict__ eq_lo, ef* __restrict__ pu,
                                                              ef* __restrict__ pd) {
  // columns c0 and c0 + 1 (when it exists) share each eq_lo load
  const size_t N = size_t(1) << log_n, S = N >> k;
  const int c0 = 2 * blockIdx.x, j = blockIdx.y;
  const bool two = c0 + 1 < AIR_W;
  const uint32_t nhi = 1u << (log_n - k - ll);
  const uint32_t xh = blockIdx.z * IS_WARPS + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (xh >= nhi) return;
  const uint32_t nlo = 1u << ll;
  const uint32_t* col0 = wit + size_t(c0) * N + size_t(j) * S + (size_t(xh) << ll);
  const uint32_t* col1 = two ? col0 + N : col0;
  const bool last = j == gridDim.y - 1 && xh == nhi - 1;  // holds the wrapped row N - 1
  EfMacF u0, d0, u1, d1;
  u0.init();
  d0.init();
  u1.init();
  d1.init();
  uint32_t xl = lane;
  for (; xl + 96 < nlo; xl += 128) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint32_t x = xl + 32 * q;
      const ef e = eq_lo[x];
      const bool wrap = last && x == nlo - 1;
      const uint32_t xu = wrap ? x - 1 : x, xd = wrap ? x : x + 1;
      u0.mac(e, col0[xu]);
      d0.mac(e, col0[xd]);
      u1.mac(e, col1[xu]);
      d1.mac(e, col1[xd]);
    }
    u0.flush();
    d0.flush();
    u1.flush();
    d1.flush();
  }
  for (; xl < nlo; xl += 32) {
    const ef e = eq_lo[xl];
    const bool wrap = last && xl == nlo - 1;
    const uint32_t xu = wrap ? xl - 1 : xl, xd = wrap ? xl : xl + 1;
    u0.mac(e, col0[xu]);
    d0.mac(e, col0[xd]);
    u1.mac(e, col1[xu]);
    d1.mac(e, col1[xd]);
    u0.flush();
    d0.flush();
    u1.flush();
    d1.flush();
  }
  const ef su0 = warp_reduce_ef(u0.value()), sd0 = warp_reduce_ef(d0.value());
  const ef su1 = warp_reduce_ef(u1.value()), sd1 = warp_reduce_ef(d1.value());
  if (lane == 0) {
    const ef h = eq_hi[xh];
    size_t o = (size_t(c0) * gridDim.y + j) * nhi + xh;
    pu[o] = ef_mul(su0, h);
    pd[o] = ef_mul(sd0, h);
    if (two) {
      o = (size_t(c0 + 1) * gridDim.y + j) * nhi + xh;
      pu[o] = ef_mul(su1, h);
      pd[o] = ef_mul(sd1, h);
    }
  }
}

// ---- inner sums on the tensor cores
// A sum of products of 31-bit values is exact in integer matrix products over byte limbs:
// with x = sum_a 2^(8a) x_a and e = sum_b 2^(8b) e_b (bytes), sum_k x e = sum_(a,b) 2^(8(a+b))
// sum_k x_a e_b, and each inner sum of 4096 byte products stays below 2^28. The witness
// segments of 2^ll rows are the rows of A (u32 values, split into 4 byte matrices in
// registers), the eq_lo weights the columns of B: 16 columns, the 8 coefficients of eq_lo[x]
// (up sums) and of eq_lo[x - 1] (down sums, shifted by one row), as 4 byte matrices
// prepared once (k_eq_limbs). Each m16n8k32 u8 product adds 16 x 8 x 32 byte products into
// s32 accumulators; warp b of a block holds the 4 x 2 tiles of B limb b for a 16-row tile.
// The limb products are recombined by diagonal (a + b = d, below 2^30), weighted by
// 2^(8d) mod p (7 wide products, below 4 p^2) and reduced once: the Montgomery values give
// the Montgomery product. The row boundary terms (the down sum's element past the segment,
// the wrapped last row) are added on the CUDA cores.
// limbs[(b * 16 + n) * nlo + x] = byte b of column n of B at row x: n < 8 coefficient n of
// eq_lo[x], n >= 8 coefficient n - 8 of eq_lo[x - 1] (zero at x = 0).
__global__ void k_eq_limbs(const ef* __restrict__ eq_lo, int nlo, uint8_t* __restrict__ limbs) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= 16 * nlo) return;
  const int n = idx / nlo, x = idx - n * nlo;
  uint32_t v = 0;
  if (n < 8) v = eq_lo[x].c[n];
  else if (x > 0) v = eq_lo[x - 1].c[n - 8];
#pragma unroll
  for (int b = 0; b < 4; b++) limbs[(size_t(b) * 16 + n) * nlo + x] = uint8_t(v >> (8 * b));
}
constexpr int ISM_WARPS = 4;  // one per B limb
constexpr int ISM_STAGES = 4;  // chunks of 32 values in flight per tile
constexpr int ISM_ROW = 48;    // words per staged row (32 + 16: conflict-free 16-byte fragment reads)
constexpr int CS_WARPS = 4;   // warps of the kernels whose warps own whole tiles

// Sum over the limb pairs of column value (row, col), from the per-pair accumulators
// cs[a][b][row][col]: diagonals a + b = d (below 4 * 2^12 * 255^2 < 2^31) weighted by
// 2^(8d) mod p, then one Montgomery reduction (the sum stays below 4 p^2).
template <int C>
__device__ __forceinline__ uint32_t limb_recombine(const int (&cs)[4][4][16][C], int row, int col) {
  constexpr uint32_t W8[7] = {uint32_t(kb::detail::cpow(2, 0)),  uint32_t(kb::detail::cpow(2, 8)),
                              uint32_t(kb::detail::cpow(2, 16)), uint32_t(kb::detail::cpow(2, 24)),
                              uint32_t(kb::detail::cpow(2, 32)), uint32_t(kb::detail::cpow(2, 40)),
                              uint32_t(kb::detail::cpow(2, 48))};  // 2^(8d) mod p
  uint64_t v = 0;
#pragma unroll
  for (int d = 0; d < 7; d++) {
    uint32_t dd = 0;
#pragma unroll
    for (int a = 0; a < 4; a++)
      if (d - a >= 0 && d - a < 4) dd += uint32_t(cs[a][d - a][row][col]);
    v += kb::wmul(dd, W8[d]);
  }
  return kb::redc(v);
}
template <int NT, int C>
__device__ __forceinline__ void limb_store(int (&cs)[4][4][16][C], const int (&acc)[4][NT][4], int b, int g, int t) {
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int nt = 0; nt < NT; nt++) {
      cs[a][b][g][nt * 8 + 2 * t] = acc[a][nt][0];
      cs[a][b][g][nt * 8 + 2 * t + 1] = acc[a][nt][1];
      cs[a][b][g + 8][nt * 8 + 2 * t] = acc[a][nt][2];
      cs[a][b][g + 8][nt * 8 + 2 * t + 1] = acc[a][nt][3];
    }
}

__global__ void __launch_bounds__(ISM_WARPS * 32) k_inner_sums_mma(const uint32_t* __restrict__ wit, int log_n, int k,
                                                                  int ll, const ef* __restrict__ eq_hi,
                                                                  const ef* __restrict__ eq_lo,
                                                                  const uint8_t* __restrict__ limbs,
                                                                  ef* __restrict__ pu, ef* __restrict__ pd) {
  __shared__ int cs[4][4][16][17];  // [a][b][row][col], padded
  __shared__ ef up_s[16], dn_s[16];
  __shared__ __align__(16) uint32_t ism_a[ISM_STAGES][16][ISM_ROW];
  const size_t N = size_t(1) << log_n, S = N >> k;
  const uint32_t nsk = 1u << k, nhi = 1u << (log_n - k - ll), nlo = 1u << ll;
  const uint32_t M = uint32_t(AIR_W) * nsk * nhi;
  const uint32_t m0 = blockIdx.x * 16;
  const int lane = threadIdx.x & 31, b = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  auto row_base = [&](uint32_t m) -> size_t {
    const uint32_t xh = m % nhi, cj = m / nhi, j = cj % nsk, c = cj / nsk;
    return size_t(c) * N + size_t(j) * S + (size_t(xh) << ll);
  };
  // The tile's 16 segments stream through shared memory in chunks of 32 values (one 16-byte
  // cp.async per thread and chunk, ISM_STAGES chunks in flight), so the four warps (one per
  // limb of B) read each value from HBM once; rows past M are zero-filled.
  {
    const int crow = threadIdx.x >> 3, cpiece = threadIdx.x & 7;  // 16 rows x 8 pieces
    const uint32_t mr = m0 + crow;
    const bool cval = mr < M;
    const uint32_t* csrc = wit + (cval ? row_base(mr) : 0) + 4 * cpiece;
    const unsigned cdst0 = (unsigned)__cvta_generic_to_shared(&ism_a[0][crow][4 * cpiece]);
    const unsigned cstage = sizeof(ism_a[0]);
    const uint32_t nch = nlo >> 5;
    auto issue = [&](uint32_t c) {
      if (c < nch) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(cdst0 + (c % ISM_STAGES) * cstage),
                     "l"(csrc + 32 * c), "r"(cval ? 16 : 0));
      }
      asm volatile("cp.async.commit_group;\n" ::);
    };
    for (int c = 0; c < ISM_STAGES - 1; c++) issue(c);
    int acc[4][2][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[a][nt][q] = 0;
    const uint32_t* lb = reinterpret_cast<const uint32_t*>(limbs + size_t(b) * 16 * nlo);
    const uint32_t lstride = nlo >> 2;
#pragma unroll 1
    for (uint32_t c = 0; c < nch; c++) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(ISM_STAGES - 2));
      __syncthreads();  // chunk c landed for every thread; the slot of chunk c - 1 is free
      issue(c + ISM_STAGES - 1);
      const uint32_t(&X)[16][ISM_ROW] = ism_a[c % ISM_STAGES];
      const uint4 q0 = *reinterpret_cast<const uint4*>(&X[g][4 * t]);
      const uint4 q1 = *reinterpret_cast<const uint4*>(&X[g + 8][4 * t]);
      const uint4 q2 = *reinterpret_cast<const uint4*>(&X[g][16 + 4 * t]);
      const uint4 q3 = *reinterpret_cast<const uint4*>(&X[g + 8][16 + 4 * t]);
      uint32_t l0[4], l1[4], l2[4], l3[4];
      byte_transpose4(q0, l0);
      byte_transpose4(q1, l1);
      byte_transpose4(q2, l2);
      byte_transpose4(q3, l3);
      uint32_t bf[2][2];
#pragma unroll
      for (int nt = 0; nt < 2; nt++) {
        const uint32_t* col = lb + size_t(nt * 8 + g) * lstride + (c << 3) + t;
        bf[nt][0] = __ldg(col);
        bf[nt][1] = __ldg(col + 4);
      }
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const uint32_t af[4] = {l0[a], l1[a], l2[a], l3[a]};
#pragma unroll
        for (int nt = 0; nt < 2; nt++) mma_u8_16832(acc[a][nt], af, bf[nt][0], bf[nt][1]);
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    limb_store<2>(cs, acc, b, g, t);
  }
  __syncthreads();
  // recombination: 256 (row, column) values, two per thread
  for (int e = threadIdx.x; e < 256; e += ISM_WARPS * 32) {
    const int row = e >> 4, col = e & 15;
    const uint32_t r = limb_recombine(cs, row, col);
    if (col < 8) up_s[row].c[col] = r;
    else dn_s[row].c[col - 8] = r;
  }
  __syncthreads();
  if (threadIdx.x < 16) {
    const uint32_t m = m0 + threadIdx.x;
    if (m < M) {
      const uint32_t xh = m % nhi, cj = m / nhi, j = cj % nsk, c = cj / nsk;
      const size_t base = size_t(c) * N + size_t(j) * S + (size_t(xh) << ll);
      const uint32_t* col = wit + size_t(c) * N;
      const bool last = j == nsk - 1 && xh == nhi - 1;  // the segment holding row N - 1
      const ef el = eq_lo[nlo - 1];
      ef up = up_s[threadIdx.x], dn = dn_s[threadIdx.x];
      if (last) {
        // up row of N - 1 is N - 2; down row of N - 1 is N - 1
        up = ef_add(up, ef_mul_f(el, kb::sub(col[N - 2], col[N - 1])));
        dn = ef_add(dn, ef_mul_f(el, col[N - 1]));
      } else {
        dn = ef_add(dn, ef_mul_f(el, wit[base + nlo]));
      }
      const ef h = eq_hi[xh];
      pu[m] = ef_mul(up, h);
      pd[m] = ef_mul(dn, h);
    }
  }
}

// The same inner sums with the tile staged by the bulk-copy (TMA) engine: one thread issues,
// per chunk, one cp.async.bulk of 128 bytes for each of the 16 segments, completing on the
// chunk's mbarrier (expected bytes set by the same thread); all threads wait on the mbarrier's
// phase before reading the chunk. ISB_STAGES chunks are in flight. Every wait is bounded: a
// wait that runs out counts a pipeline timeout (the host checks the counter after the inner
// sums and fails the proof) and the kernel stops consuming. Rows past M copy segment m0's data
// (their results are never stored). The B fragments of the next chunk are loaded from L2
// while the current chunk is multiplied.
constexpr int ISB_STAGES = 6;
constexpr uint32_t PIPE_WAIT_LIMIT = 1u << 20;  // try_wait rounds (each a bounded hardware wait)

__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity) {
  for (uint32_t i = 0; i < PIPE_WAIT_LIMIT; i++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__global__ void __launch_bounds__(ISM_WARPS * 32) k_inner_sums_bulk(const uint32_t* __restrict__ wit, int log_n, int k,
                                                                   int ll, const ef* __restrict__ eq_hi,
                                                                   const ef* __restrict__ eq_lo,
                                                                   const uint8_t* __restrict__ limbs,
                                                                   ef* __restrict__ pu, ef* __restrict__ pd,
                                                                   unsigned* __restrict__ timeouts) {
  __shared__ int cs[4][4][16][17];  // [a][b][row][col], padded
  __shared__ ef up_s[16], dn_s[16];
  __shared__ __align__(128) uint32_t isb_a[ISB_STAGES][16][ISM_ROW];
  __shared__ __align__(8) uint64_t bars[ISB_STAGES];
  __shared__ int stop;
  const size_t N = size_t(1) << log_n, S = N >> k;
  const uint32_t nsk = 1u << k, nhi = 1u << (log_n - k - ll), nlo = 1u << ll;
  const uint32_t M = uint32_t(AIR_W) * nsk * nhi;
  const uint32_t m0 = blockIdx.x * 16;
  const int lane = threadIdx.x & 31, b = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  auto row_base = [&](uint32_t m) -> size_t {
    const uint32_t xh = m % nhi, cj = m / nhi, j = cj % nsk, c = cj / nsk;
    return size_t(c) * N + size_t(j) * S + (size_t(xh) << ll);
  };
  const uint32_t nch = nlo >> 5;
  const unsigned bar0 = (unsigned)__cvta_generic_to_shared(&bars[0]);
  const unsigned dst0 = (unsigned)__cvta_generic_to_shared(&isb_a[0][0][0]);
  if (threadIdx.x == 0) {
    stop = 0;
    for (int st = 0; st < ISB_STAGES; st++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar0 + 8 * st));
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  // issued by thread 0 only: chunk c into slot c % ISB_STAGES
  auto issue = [&](uint32_t c) {
    if (c >= nch) return;
    const uint32_t slot = c % ISB_STAGES;
    const unsigned bar = bar0 + 8 * slot;
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // earlier reads of the slot come first
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(16u * 128u) : "memory");
    for (int row = 0; row < 16; row++) {
      const uint32_t m = m0 + row < M ? m0 + row : m0;
      const uint32_t* src = wit + row_base(m) + 32 * size_t(c);
      const unsigned dst = dst0 + ((slot * 16 + row) * ISM_ROW) * 4;
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 128, [%2];\n" ::"r"(dst),
          "l"(src), "r"(bar)
          : "memory");
    }
  };
  if (threadIdx.x == 0)
    for (int c = 0; c < ISB_STAGES - 1; c++) issue(c);
  int acc[4][2][4];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[a][nt][q] = 0;
  const uint32_t* lb = reinterpret_cast<const uint32_t*>(limbs + size_t(b) * 16 * nlo);
  const uint32_t lstride = nlo >> 2;
  uint32_t bf[2][2], bfn[2][2];
  auto load_b = [&](uint32_t c, uint32_t (&f)[2][2]) {
#pragma unroll
    for (int nt = 0; nt < 2; nt++) {
      const uint32_t* col = lb + size_t(nt * 8 + g) * lstride + (c << 3) + t;
      f[nt][0] = __ldg(col);
      f[nt][1] = __ldg(col + 4);
    }
  };
  load_b(0, bf);
  uint32_t consumed = 0;
#pragma unroll 1
  for (uint32_t c = 0; c < nch; c++) {
    if (!mbar_wait_bounded(bar0 + 8 * (c % ISB_STAGES), (c / ISB_STAGES) & 1)) {
      atomicAdd(timeouts, 1u);
      stop = 1;
    }
    __syncthreads();  // chunk c landed; every thread is done with the slot of chunk c - 1
    if (stop) break;
    if (threadIdx.x == 0) issue(c + ISB_STAGES - 1);
    if (c + 1 < nch) load_b(c + 1, bfn);
    const uint32_t(&X)[16][ISM_ROW] = isb_a[c % ISB_STAGES];
    const uint4 q0 = *reinterpret_cast<const uint4*>(&X[g][4 * t]);
    const uint4 q1 = *reinterpret_cast<const uint4*>(&X[g + 8][4 * t]);
    const uint4 q2 = *reinterpret_cast<const uint4*>(&X[g][16 + 4 * t]);
    const uint4 q3 = *reinterpret_cast<const uint4*>(&X[g + 8][16 + 4 * t]);
    uint32_t l0[4], l1[4], l2[4], l3[4];
    byte_transpose4(q0, l0);
    byte_transpose4(q1, l1);
    byte_transpose4(q2, l2);
    byte_transpose4(q3, l3);
#pragma unroll
    for (int a = 0; a < 4; a++) {
      const uint32_t af[4] = {l0[a], l1[a], l2[a], l3[a]};
#pragma unroll
      for (int nt = 0; nt < 2; nt++) mma_u8_16832(acc[a][nt], af, bf[nt][0], bf[nt][1]);
    }
#pragma unroll
    for (int nt = 0; nt < 2; nt++) bf[nt][0] = bfn[nt][0], bf[nt][1] = bfn[nt][1];
    consumed = c + 1;
  }
  if (consumed < nch) {
    // a wait ran out: let the copies already issued land (bounded) before the block exits
    const uint32_t issued = min(nch, consumed + ISB_STAGES - 1);
    for (uint32_t c = consumed; c < issued; c++) mbar_wait_bounded(bar0 + 8 * (c % ISB_STAGES), (c / ISB_STAGES) & 1);
    return;
  }
  limb_store<2>(cs, acc, b, g, t);
  __syncthreads();
  for (int e = threadIdx.x; e < 256; e += ISM_WARPS * 32) {
    const int row = e >> 4, col = e & 15;
    const uint32_t r = limb_recombine(cs, row, col);
    if (col < 8) up_s[row].c[col] = r;
    else dn_s[row].c[col - 8] = r;
  }
  __syncthreads();
  if (threadIdx.x < 16) {
    const uint32_t m = m0 + threadIdx.x;
    if (m < M) {
      const uint32_t xh = m % nhi, cj = m / nhi, j = cj % nsk, c = cj / nsk;
      const size_t base = size_t(c) * N + size_t(j) * S + (size_t(xh) << ll);
      const uint32_t* col = wit + size_t(c) * N;
      const bool last = j == nsk - 1 && xh == nhi - 1;  // the segment holding row N - 1
      const ef el = eq_lo[nlo - 1];
      ef up = up_s[threadIdx.x], dn = dn_s[threadIdx.x];
      if (last) {
        up = ef_add(up, ef_mul_f(el, kb::sub(col[N - 2], col[N - 1])));
        dn = ef_add(dn, ef_mul_f(el, col[N - 1]));
      } else {
        dn = ef_add(dn, ef_mul_f(el, wit[base + nlo]));
      }
      const ef h = eq_hi[xh];
      pu[m] = ef_mul(up, h);
      pd[m] = ef_mul(dn, h);
    }
  }
}

// WHIR partial evaluation on the tensor cores: rows m = (u, v_hi) are the segments
// T[m 2^ll .. m 2^ll + 2^ll) of the packed table (zero past t_len), B the 8 coefficients of
// lo (limbs[(b * 8 + n) * nlo + x]). Each warp owns a 16-row tile (16 consecutive v_hi of one
// u) and all 4 x 4 limb pairs, so every segment value is loaded and split into limbs once;
// its rows' dot products times hi[v_hi], summed, are partial[(v_hi / 16) * 2^lu + u].
// Short tables give v_hi 6 variables so that this form runs: 2^12 rows 41 + 12 us on
// k_mle_partial_base and its sum (fewer than 16 v_hi), 7 + 4 + 3 us here.
__global__ void __launch_bounds__(CS_WARPS * 32) k_mle_partial_mma(const uint32_t* __restrict__ T, size_t t_len,
                                                                  int lu, int lh, int ll,
                                                                  const ef* __restrict__ hi,
                                                                  const uint8_t* __restrict__ limbs,
                                                                  ef* __restrict__ partial) {
  __shared__ int cs_all[CS_WARPS][4][4][16][9];
  __shared__ ef rows_all[CS_WARPS][16];
  const uint32_t nhi = 1u << lh, nlo = 1u << ll;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  int(&cs)[4][4][16][9] = cs_all[warp];
  const uint32_t m0 = (blockIdx.x * CS_WARPS + warp) * 16;  // 16 rows of one u (16 divides nhi)
  if (m0 >= (1u << (lu + lh))) return;  // whole warp (no block barrier below)
  const size_t ba = size_t(m0 + g) << ll, bb = size_t(m0 + g + 8) << ll;
  const bool va = ba < t_len, vb = bb < t_len;  // t_len is a multiple of 2^ll
  const uint32_t* pa = T + (va ? ba : 0) + 4 * t;
  const uint32_t* pb = T + (vb ? bb : 0) + 4 * t;
  const uint32_t* lw = reinterpret_cast<const uint32_t*>(limbs);
  const uint32_t lstride = nlo >> 2;
  int acc[4][4][4];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[a][b][q] = 0;
  const uint4 zero4 = make_uint4(0, 0, 0, 0);
  // the next step's values are requested before this step's products (two steps in flight)
  uint4 n0 = va ? __ldg(reinterpret_cast<const uint4*>(pa)) : zero4;
  uint4 n1 = vb ? __ldg(reinterpret_cast<const uint4*>(pb)) : zero4;
  uint4 n2 = va ? __ldg(reinterpret_cast<const uint4*>(pa + 16)) : zero4;
  uint4 n3 = vb ? __ldg(reinterpret_cast<const uint4*>(pb + 16)) : zero4;
#pragma unroll 1
  for (uint32_t k0 = 0; k0 < nlo; k0 += 32) {
    const uint4 q0 = n0, q1 = n1, q2 = n2, q3 = n3;
    if (k0 + 32 < nlo) {
      n0 = va ? __ldg(reinterpret_cast<const uint4*>(pa + k0 + 32)) : zero4;
      n1 = vb ? __ldg(reinterpret_cast<const uint4*>(pb + k0 + 32)) : zero4;
      n2 = va ? __ldg(reinterpret_cast<const uint4*>(pa + k0 + 48)) : zero4;
      n3 = vb ? __ldg(reinterpret_cast<const uint4*>(pb + k0 + 48)) : zero4;
    }
    uint32_t l0[4], l1[4], l2[4], l3[4];
    byte_transpose4(q0, l0);
    byte_transpose4(q1, l1);
    byte_transpose4(q2, l2);
    byte_transpose4(q3, l3);
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const uint32_t* col = lw + size_t(b * 8 + g) * lstride + (k0 >> 2) + t;
      const uint32_t b0 = __ldg(col), b1 = __ldg(col + 4);
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const uint32_t af[4] = {l0[a], l1[a], l2[a], l3[a]};
        mma_u8_16832(acc[a][b], af, b0, b1);
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) {
      cs[a][b][g][2 * t] = acc[a][b][0];
      cs[a][b][g][2 * t + 1] = acc[a][b][1];
      cs[a][b][g + 8][2 * t] = acc[a][b][2];
      cs[a][b][g + 8][2 * t + 1] = acc[a][b][3];
    }
  __syncwarp();
#pragma unroll
  for (int e = lane; e < 128; e += 32) rows_all[warp][e >> 3].c[e & 7] = limb_recombine(cs, e >> 3, e & 7);
  __syncwarp();
  const uint32_t u = m0 >> lh, vh0 = m0 & (nhi - 1);
  ef v = lane < 16 ? ef_mul(rows_all[warp][lane], hi[vh0 + lane]) : ef_zero();
  v = warp_reduce_ef(v);
  if (lane == 0) partial[size_t(vh0 >> 4) * (size_t(1) << lu) + u] = v;
}
// limbs[(b * 8 + n) * nlo + x] = byte b of coefficient n of lo[x].
__global__ void k_lo_limbs(const ef* __restrict__ lo, int nlo, uint8_t* __restrict__ limbs) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= 8 * nlo) return;
  const int n = idx / nlo, x = idx - n * nlo;
  const uint32_t v = lo[x].c[n];
#pragma unroll
  for (int b = 0; b < 4; b++) limbs[(size_t(b) * 8 + n) * nlo + x] = uint8_t(v >> (8 * b));
}

// Weighted column sums on the tensor cores: out[m] = sum_(k < K) w[k] A[m][k] for extension
// weights w and base-field A, by byte-limb matrix products (as the inner sums) with the rows
// m on the M side and the short K (<= 192) in chunks of 32. A[m][k] sits at
// src[k * kstride + m] (consecutive rows are consecutive words, so every load of a warp reads
// whole sectors). Used for the batched column (the witness columns, kstride N). The same form
// was measured slower than the CUDA-core kernels for the WHIR table g (K = 128) and for the
// round-0 fold (K = 2^k <= 16, padded to 32): their loads dominate, and the CUDA-core
// kernels read two rows per load.
// Each warp owns a 16-row tile and all 4 x 4 limb pairs; limbs[(b * 8 + n) * Kp + k] holds
// byte b of coefficient n of w[k] (zero for k >= K).
__global__ void __launch_bounds__(CS_WARPS * 32) k_colsum_mma(const uint32_t* __restrict__ src, size_t M, int K,
                                                             int Kp, size_t kstride,
                                                             const uint8_t* __restrict__ limbs, ef* __restrict__ out) {
  __shared__ int cs_all[CS_WARPS][4][4][16][9];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  int(&cs)[4][4][16][9] = cs_all[warp];
  const size_t m0 = (size_t(blockIdx.x) * CS_WARPS + warp) * 16;
  if (m0 >= M) return;  // whole warp (no block barrier below)
  const size_t ra = m0 + g, rb = m0 + g + 8;
  const bool va = ra < M, vb = rb < M;
  auto load = [&](size_t m, bool vm, int kk) -> uint32_t {
    return (vm && kk < K) ? __ldg(src + size_t(kk) * kstride + m) : 0u;
  };
  int acc[4][4][4];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[a][b][q] = 0;
  const uint32_t* lw = reinterpret_cast<const uint32_t*>(limbs);
  const int lstride = Kp >> 2;
  // the next step's values are requested before this step's products (two steps in flight)
  auto load_step = [&](int k0, uint4 (&q)[4]) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int kb0 = k0 + 16 * h + 4 * t;
      q[2 * h] = make_uint4(load(ra, va, kb0), load(ra, va, kb0 + 1), load(ra, va, kb0 + 2), load(ra, va, kb0 + 3));
      q[2 * h + 1] =
          make_uint4(load(rb, vb, kb0), load(rb, vb, kb0 + 1), load(rb, vb, kb0 + 2), load(rb, vb, kb0 + 3));
    }
  };
  uint4 nq[4];
  load_step(0, nq);
#pragma unroll 1
  for (int k0 = 0; k0 < Kp; k0 += 32) {
    uint4 q[4];
#pragma unroll
    for (int i = 0; i < 4; i++) q[i] = nq[i];
    if (k0 + 32 < Kp) load_step(k0 + 32, nq);
    uint32_t l[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++) byte_transpose4(q[i], l[i]);
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const uint32_t* col = lw + size_t(b * 8 + g) * lstride + (k0 >> 2) + t;
      const uint32_t b0 = __ldg(col), b1 = __ldg(col + 4);
#pragma unroll
      for (int a = 0; a < 4; a++) {
        const uint32_t af[4] = {l[0][a], l[1][a], l[2][a], l[3][a]};
        mma_u8_16832(acc[a][b], af, b0, b1);
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) {
      cs[a][b][g][2 * t] = acc[a][b][0];
      cs[a][b][g][2 * t + 1] = acc[a][b][1];
      cs[a][b][g + 8][2 * t] = acc[a][b][2];
      cs[a][b][g + 8][2 * t + 1] = acc[a][b][3];
    }
  __syncwarp();
  uint32_t* o = reinterpret_cast<uint32_t*>(out);
#pragma unroll
  for (int e = lane; e < 128; e += 32) {
    const int row = e >> 3, col = e & 7;
    if (m0 + row < M) o[(m0 + row) * 8 + col] = limb_recombine(cs, row, col);
  }
}
// limbs[(b * 8 + n) * Kp + k] = byte b of coefficient n of w[k] (zero for k >= K).
__global__ void k_w_limbs(const ef* __restrict__ w, int K, int Kp, uint8_t* __restrict__ limbs) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= 8 * Kp) return;
  const int n = idx / Kp, x = idx - n * Kp;
  const uint32_t v = x < K ? w[x].c[n] : 0u;
#pragma unroll
  for (int b = 0; b < 4; b++) limbs[(size_t(b) * 8 + n) * Kp + x] = uint8_t(v >> (8 * b));
}

// out[c] = sum_j sel[j] * sum_h partial[(c * nsk + j) * nh + h]; one warp per column.
__global__ void k_combine_sel(const ef* __restrict__ partial, const ef* __restrict__ sel, int nsk, int nh, int ncols,
                              ef* __restrict__ out) {
  const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (c >= ncols) return;
  ef acc = ef_zero();
  for (int idx = lane; idx < nsk * nh; idx += 32)
    acc = ef_add(acc, ef_mul(sel[idx / nh], partial[size_t(c) * nsk * nh + idx]));
  acc = warp_reduce_ef(acc);
  if (lane == 0) out[c] = acc;
}

// ------------------------------------------------------------------ inner phase
// out[row] = sum_c eqc[c] * wit[c][row]; two adjacent rows per thread (8-byte loads).
__global__ void k_batch_cols(const uint32_t* __restrict__ wit, int log_n, const ef* __restrict__ eqc_g,
                             ef* __restrict__ out) {
  __shared__ ef eqc[AIR_W + 3];
  for (int i = threadIdx.x; i < AIR_W + 3; i += blockDim.x) eqc[i] = i < AIR_W ? eqc_g[i] : ef_zero();
  __syncthreads();
  const size_t N = size_t(1) << log_n;
  const size_t row = (size_t(blockIdx.x) * blockDim.x + threadIdx.x) * 2;
  if (row >= N) return;
  EfMacF m0, m1;
  m0.init();
  m1.init();
#pragma unroll 2
  for (int c = 0; c < AIR_W; c += 4) {
    uint2 v[4];
#pragma unroll
    for (int q = 0; q < 4; q++)
      v[q] = c + q < AIR_W ? __ldg(reinterpret_cast<const uint2*>(wit + size_t(c + q) * N + row)) : make_uint2(0, 0);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      m0.mac(eqc[c + q], v[q].x);
      m1.mac(eqc[c + q], v[q].y);
    }
    m0.flush();
    m1.flush();
  }
  out[row] = m0.value();
  out[row + 1] = m1.value();
}

constexpr int SUB_THREADS = 256, SUB_PER_THREAD = 16;

// partial[(chunk * 2^k + j) * 2 + {0,1}] = sum_x eqt[x] * B[up/down(j S + x)] over the chunk's x
__global__ void k_sub_evals(const ef* __restrict__ B, int log_n, int k, const ef* __restrict__ eqt,
                            ef* __restrict__ partial) {
  __shared__ ef scratch[32];
  const size_t N = size_t(1) << log_n, S = N >> k;
  const int j = blockIdx.y;
  const size_t chunk = blockIdx.x;
  ef u = ef_zero(), d = ef_zero();
  for (int q = 0; q < SUB_PER_THREAD; q++) {
    size_t x = (chunk * SUB_PER_THREAD + q) * SUB_THREADS + threadIdx.x;
    if (x < S) {
      size_t i = size_t(j) * S + x;
      const ef e = eqt[x];
      u = ef_add(u, ef_mul(e, B[up_row(i, N)]));
      d = ef_add(d, ef_mul(e, B[down_row(i, N)]));
    }
  }
  u = block_reduce_ef(u, scratch);
  d = block_reduce_ef(d, scratch);
  if (threadIdx.x == 0) {
    size_t o = (chunk * gridDim.y + j) * 2;
    partial[o] = u;
    partial[o + 1] = d;
  }
}

// A[y] = up-shift matrix row + alpha2 * down-shift matrix row, folded at the point whose
// eq table is e (crates/air/src/uni_skip_utils.rs:5-34).
__global__ void k_inner_mle(const ef* __restrict__ e, int log_n, const ef* __restrict__ alpha2, ef* __restrict__ out) {
  const size_t N = size_t(1) << log_n;
  const size_t y = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (y >= N) return;
  const ef last = e[N - 1];
  ef mu = e[y];
  if (y == N - 2) mu = ef_add(mu, last);
  if (y == N - 1) mu = ef_zero();
  ef md = y >= 1 ? e[y - 1] : ef_zero();
  if (y == N - 1) md = ef_add(md, last);
  out[y] = ef_add(mu, ef_mul(*alpha2, md));
}

constexpr int PROD_THREADS = 256;
// points per thread: 8 for large tables, fewer for small ones so that latency, not a
// serial loop, bounds the small rounds
int prod_per_thread(size_t half) { return half >= (size_t(1) << 19) ? 8 : half >= (size_t(1) << 16) ? 2 : 1; }

__global__ void k_prod_eval(const ef* __restrict__ a, const ef* __restrict__ b, size_t half, int per,
                            ef* __restrict__ partial) {
  __shared__ ef scratch[32];
  ef s0 = ef_zero(), s2 = ef_zero();
  for (int q = 0; q < per; q++) {
    size_t x = (size_t(blockIdx.x) * per + q) * PROD_THREADS + threadIdx.x;
    if (x < half) {
      ef al = a[x], ah = a[x + half], bl = b[x], bh = b[x + half];
      s0 = ef_add(s0, ef_mul(al, bl));
      ef a2 = ef_sub(ef_add(ah, ah), al), b2 = ef_sub(ef_add(bh, bh), bl);
      s2 = ef_add(s2, ef_mul(a2, b2));
    }
  }
  s0 = block_reduce_ef(s0, scratch);
  s2 = block_reduce_ef(s2, scratch);
  if (threadIdx.x == 0) {
    partial[size_t(blockIdx.x) * 2] = s0;
    partial[size_t(blockIdx.x) * 2 + 1] = s2;
  }
}


// ------------------------------------------------------------------ fold fused with the next round
// The fold of the previous round at its challenge (lo + r (hi - lo), the challenge read from
// device memory where the round-finishing kernel left it) fused with this round's sums, so
// every table is read once per round: thread x of this round (x < h, the tables' new length
// being 2h) reads old entries x, x + h, x + 2h, x + 3h, writes the two folded entries x and
// x + h, and accumulates the round polynomial's values. Grid-stride; one partial per block.
constexpr int FE_THREADS = FIN_MAX_THREADS;
__device__ __forceinline__ ef fe_lerp(const ef* t, size_t i, size_t L, const ef& r) {
  const ef lo = t[i];
  return ef_add(lo, ef_mul(r, ef_sub(t[i + L], lo)));
}
// Product sumcheck (NS = 2: values at 0 and 2; the inner sumcheck) and WHIR folding sumcheck
// (NS = 3: values at 0, 1, 2) on the pair of tables (a, b).
template <int NS>
__global__ void __launch_bounds__(FE_THREADS) k_pair_fold_eval(const ef* __restrict__ a, const ef* __restrict__ b,
                                                               const ef* __restrict__ rptr, ef* __restrict__ na,
                                                               ef* __restrict__ nb, size_t h,
                                                               ef* __restrict__ partial, const FinArgs fin) {
  __shared__ ef scratch[32];
  const ef r = *rptr;
  const size_t L = 2 * h;
  ef s0 = ef_zero(), s1 = ef_zero(), s2 = ef_zero();
  for (size_t x = size_t(blockIdx.x) * blockDim.x + threadIdx.x; x < h; x += size_t(gridDim.x) * blockDim.x) {
    const ef al = fe_lerp(a, x, L, r), ah = fe_lerp(a, x + h, L, r);
    const ef bl = fe_lerp(b, x, L, r), bh = fe_lerp(b, x + h, L, r);
    na[x] = al;
    na[x + h] = ah;
    nb[x] = bl;
    nb[x + h] = bh;
    s0 = ef_add(s0, ef_mul(al, bl));
    if (NS == 3) s1 = ef_add(s1, ef_mul(ah, bh));
    s2 = ef_add(s2, ef_mul(ef_sub(ef_add(ah, ah), al), ef_sub(ef_add(bh, bh), bl)));
  }
  s0 = block_reduce_ef(s0, scratch);
  if (threadIdx.x == 0) partial[size_t(blockIdx.x) * NS] = s0;
  __syncthreads();
  if (NS == 3) {
    s1 = block_reduce_ef(s1, scratch);
    if (threadIdx.x == 0) partial[size_t(blockIdx.x) * NS + 1] = s1;
    __syncthreads();
  }
  s2 = block_reduce_ef(s2, scratch);
  if (threadIdx.x == 0) partial[size_t(blockIdx.x) * NS + NS - 1] = s2;
  if (fin.st) fin_last_block(NS == 2 ? FIN_PROD : FIN_WHIR, fin, partial, NS);
}
// The a*b - c zerocheck's rounds >= 2: three columns (column q of old length 4h at q 4h, of new
// length 2h at q 2h) and the eq table (old length 2h, the leading variable summed out into the
// new table of length h); values at z = 0 and 2 of (A B - C) eq.
__global__ void __launch_bounds__(FE_THREADS) k_abc_fold_eval(const ef* __restrict__ cols, const ef* __restrict__ rptr,
                                                              const ef* __restrict__ eq_prev, ef* __restrict__ nc,
                                                              ef* __restrict__ eq_new, size_t h,
                                                              ef* __restrict__ partial, const FinArgs fin) {
  __shared__ ef scratch[32];
  const ef r = *rptr;
  const size_t L = 2 * h;
  ef s0 = ef_zero(), s2 = ef_zero();
  for (size_t x = size_t(blockIdx.x) * blockDim.x + threadIdx.x; x < h; x += size_t(gridDim.x) * blockDim.x) {
    ef lo[3], t[3];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const ef* col = cols + size_t(q) * 2 * L;
      lo[q] = fe_lerp(col, x, L, r);
      const ef hi = fe_lerp(col, x + h, L, r);
      nc[size_t(q) * L + x] = lo[q];
      nc[size_t(q) * L + x + h] = hi;
      t[q] = ef_sub(ef_add(hi, hi), lo[q]);
    }
    const ef e = ef_add(eq_prev[x], eq_prev[x + h]);
    eq_new[x] = e;
    s0 = ef_add(s0, ef_mul(ef_sub(ef_mul(lo[0], lo[1]), lo[2]), e));
    s2 = ef_add(s2, ef_mul(ef_sub(ef_mul(t[0], t[1]), t[2]), e));
  }
  s0 = block_reduce_ef(s0, scratch);
  if (threadIdx.x == 0) partial[size_t(blockIdx.x) * 2] = s0;
  __syncthreads();
  s2 = block_reduce_ef(s2, scratch);
  if (threadIdx.x == 0) partial[size_t(blockIdx.x) * 2 + 1] = s2;
  if (fin.st) fin_last_block(FIN_EQSC3, fin, partial, 2);
}

// ------------------------------------------------------------------ the last rounds of a phase
// Once a phase's tables fit the shared memory of one block or cluster, all rounds that remain run
// in one launch: fold at the last challenge, the round's sums, the finish, and again, with the tables
// folded in place and the phase state kept in shared memory between the rounds. As a launch of
// its own such a round also cost a kernel boundary, a count of blocks through device memory and
// the reload of all it needs: 26.6 us a round of the a*b - c sumcheck, 16.4 us here on average
// over its last nine (9.3 us of each the finish, which is one warp's serial work).
//
// Eight lanes form one extension product (fin_mul), here as in the finish. With one thread per
// product the last rounds have one warp walk through a dozen products in turn, and their code, a
// few hundred instructions each, does not stay in the instruction cache from round to round:
// 20.3 us a round. For many points the other form needs half the instructions, so the tail
// holds at most 256 points in a block: from 512 on its first round would take longer (23 us a round
// on average with 256 threads) than the several blocks of a separate launch.
//
// h is the number of points of the first round. With fold_in the tables come in at length 4h
// (the eq table at 2h), to be folded at challenge *ch0; else at length 2h (h), to be evaluated as
// they are.
//
// From more than TAIL_BLOCK_H = 256 up to TAIL_MAX_H points the launch is a cluster of
// TAIL_CLUSTER blocks (CL): block c holds the entries x = c (mod TAIL_CLUSTER), so every fold stays
// in its block; a round's partial sums go to block 0's shared memory, which finishes the round and
// writes the challenge into the others'. The fold that leaves 2 TAIL_BLOCK_H entries writes them
// to block 0, which goes on alone. Such a round as a launch of its own, on 2 to 8 blocks: 27 us
// (product), 31 (WHIR), 28 (a*b - c); here 14 to 18. The line: with 4096 points (512 a block) the
// round took 32 and 44 us, as eight lanes per product issue more than twice the instructions of one
// thread per product. Loading the first fold's entries eight at a time changed nothing.
constexpr int TAIL_THREADS = 512;
constexpr int TAIL_GROUPS = TAIL_THREADS / 8;
constexpr uint32_t TAIL_BLOCK_H = 256;
constexpr uint32_t TAIL_CLUSTER = uint32_t(TAIL_MAX_H) / TAIL_BLOCK_H;
static_assert(TAIL_CLUSTER <= 8, "portable cluster size");
__shared__ ef tail_red[TAIL_CLUSTER][3];  // block 0: every block's sums of the round

__device__ __forceinline__ uint32_t cl_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// The address of block `rank`'s copy of a shared-memory object.
template <class T>
__device__ __forceinline__ T* cl_map(T* p, uint32_t rank) {
  uint64_t r;
  asm("mapa.u64 %0, %1, %2;" : "=l"(r) : "l"(p), "r"(rank));
  return reinterpret_cast<T*>(r);
}

// Adds the groups' sums acc[z] (coordinate lane & 7) over the block into fin_sm.red and finishes
// the round on warp 0 (with cl, over the cluster's blocks and on block 0's). fin_sm.chal is valid
// for every thread on return.
template <int NS>
__device__ __forceinline__ void tail_finish(int kind, const FinArgs& fin, const uint32_t* acc, bool cl, uint32_t rank) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int z = 0; z < NS; z++) {
    uint32_t v = kb::add(acc[z], __shfl_xor_sync(FIN_FULL, acc[z], 8));
    v = kb::add(v, __shfl_xor_sync(FIN_FULL, v, 16));
    if (lane < 8) fin_sm.tmp[z * (TAIL_THREADS / 32) + w].c[lane] = v;
  }
  __syncthreads();
  if (w == 0) {
    const int z = lane >> 3, k = lane & 7;
    if (z < NS) {
      uint32_t v = 0;
#pragma unroll
      for (int u = 0; u < TAIL_THREADS / 32; u++) v = kb::add(v, fin_sm.tmp[z * (TAIL_THREADS / 32) + u].c[k]);
      (cl ? cl_map(&tail_red[rank][z], 0) : &fin_sm.red[z])->c[k] = v;
    }
    __syncwarp();
  }
  if (cl) cl_sync();
  if (w == 0 && rank == 0) {
    const int z = lane >> 3, k = lane & 7;
    if (cl && z < NS) {
      uint32_t v = 0;
#pragma unroll
      for (uint32_t c = 0; c < TAIL_CLUSTER; c++) v = kb::add(v, tail_red[c][z].c[k]);
      fin_sm.red[z].c[k] = v;
    }
    __syncwarp();
    fin_round(kind, fin);
    __syncwarp();
    if (cl)
      for (uint32_t c = 1 + (lane >> 3); c < TAIL_CLUSTER; c += 4) cl_map(&fin_sm.chal, c)->c[k] = fin_sm.chal.c[k];
  }
  if (cl) cl_sync();
  else __syncthreads();
}
// The entries of a table that a block holds: x_0, x_0 + m, ... of the whole table.
struct TailMap {
  uint32_t m = 1, x0 = 0;
};
// Entries [0, n) of each of NT tables (length 2n at src + q sstride, in the places of sm) folded at r
// (coordinate lane & 7) into dst + q dstride (places of dm); dst may be src, as an entry that is
// written is read only by the group that writes it.
template <int NT>
__device__ __forceinline__ void tail_fold(const ef* src, size_t sstride, ef* dst, size_t dstride, uint32_t n, uint32_t r,
                                          TailMap sm = {}, TailMap dm = {}) {
  const uint32_t g = threadIdx.x >> 3, k = threadIdx.x & 7;
#pragma unroll 1
  for (uint32_t t0 = 0; t0 < NT * n; t0 += TAIL_GROUPS) {
    const uint32_t t = t0 + g;
    const bool on = t < NT * n;
    const uint32_t q = on ? t / n : 0, x = on ? t - q * n : 0;
    const ef* s = src + q * sstride + x * sm.m + sm.x0;
    const uint32_t lo = s[0].c[k], hi = s[n * sm.m].c[k];
    const uint32_t v = kb::add(lo, fin_mul(r, kb::sub(hi, lo)));
    if (on) dst[q * dstride + x * dm.m + dm.x0].c[k] = v;
  }
}
// The same entries copied.
template <int NT>
__device__ __forceinline__ void tail_copy(const ef* src, size_t sstride, ef* dst, size_t dstride, uint32_t n,
                                          TailMap sm = {}) {
  for (uint32_t t = threadIdx.x; t < NT * n * 8; t += TAIL_THREADS) {
    const uint32_t e = t >> 3, q = e / n, x = e - q * n;
    dst[q * dstride + x].c[t & 7] = src[q * sstride + x * sm.m + sm.x0].c[t & 7];
  }
}

// Product (NS = 2) and WHIR (NS = 3) rounds; the tables folded at the last challenge go to oa, ob.
template <int NS, bool CL>
__global__ void __launch_bounds__(TAIL_THREADS, 1)
    k_pair_tail(const ef* __restrict__ a, const ef* __restrict__ b, uint32_t h, bool fold_in,
                const ef* __restrict__ ch0, int rounds, ef* __restrict__ oa, ef* __restrict__ ob, const FinArgs fin) {
  extern __shared__ __align__(16) char tail_smem[];
  const uint32_t rank = CL ? cl_rank() : 0, g = threadIdx.x >> 3, k = threadIdx.x & 7;
  bool cl = CL;
  TailMap mp{CL ? TAIL_CLUSTER : 1u, rank};
  if (CL) h /= TAIL_CLUSTER;  // this block's points
  uint32_t stride = 2 * h;
  ef *sa = reinterpret_cast<ef*>(tail_smem), *sb = sa + stride;
  ef* const joined = sb + stride;  // CL, block 0: the joined tables, 2 TAIL_BLOCK_H entries each
  constexpr int kind = NS == 2 ? FIN_PROD : FIN_WHIR;
  if (rank == 0) fin_load(kind, fin);
  if (fold_in) {
    const uint32_t r = ch0->c[k];
    tail_fold<1>(a, 0, sa, 0, 2 * h, r, mp);
    tail_fold<1>(b, 0, sb, 0, 2 * h, r, mp);
  } else {
    tail_copy<1>(a, 0, sa, 0, 2 * h, mp);
    tail_copy<1>(b, 0, sb, 0, 2 * h, mp);
  }
  if (CL) cl_sync();  // every block runs: from here its shared memory may be written
  else __syncthreads();
#pragma unroll 1
  for (int t = 0;; t++, h >>= 1) {
    uint32_t acc[NS];
#pragma unroll
    for (int z = 0; z < NS; z++) acc[z] = 0;
#pragma unroll 1
    for (uint32_t x0 = 0; x0 < h; x0 += TAIL_GROUPS) {
      const uint32_t x = x0 + g;
      const bool on = x < h;
      const uint32_t al = on ? sa[x].c[k] : 0u, ah = on ? sa[x + h].c[k] : 0u;
      const uint32_t bl = on ? sb[x].c[k] : 0u, bh = on ? sb[x + h].c[k] : 0u;
      acc[0] = kb::add(acc[0], fin_mul(al, bl));
      if (NS == 3) acc[1] = kb::add(acc[1], fin_mul(ah, bh));
      acc[NS - 1] = kb::add(acc[NS - 1], fin_mul(kb::sub(kb::dbl(ah), al), kb::sub(kb::dbl(bh), bl)));
    }
    tail_finish<NS>(kind, fin, acc, cl, rank);
    if (t == rounds - 1) break;
    if (CL && cl && h * TAIL_CLUSTER == 2 * TAIL_BLOCK_H) {
      tail_fold<2>(sa, stride, cl_map(joined, 0), 2 * TAIL_BLOCK_H, h, fin_sm.chal.c[k], {}, mp);
      cl_sync();
      if (rank) return;
      cl = false;
      mp = {};
      h *= TAIL_CLUSTER;
      stride = 2 * TAIL_BLOCK_H;
      sa = joined;
      sb = joined + stride;
    } else {
      tail_fold<2>(sa, stride, sa, stride, h, fin_sm.chal.c[k]);
      __syncthreads();
    }
  }
  tail_fold<1>(sa, 0, oa, 0, h, fin_sm.chal.c[k], {}, mp);
  tail_fold<1>(sb, 0, ob, 0, h, fin_sm.chal.c[k], {}, mp);
  if (rank == 0 && threadIdx.x < 32) fin_commit(fin);
}

// The a*b - c zerocheck's rounds, to the end; the three columns folded at the last challenge go
// to oc (column q at q times the last round's points).
template <bool CL>
__global__ void __launch_bounds__(TAIL_THREADS, 1)
    k_abc_tail(const ef* __restrict__ cols, const ef* __restrict__ eq_in, uint32_t h, bool fold_in,
               const ef* __restrict__ ch0, int rounds, ef* __restrict__ oc, const FinArgs fin) {
  extern __shared__ __align__(16) char tail_smem[];
  const uint32_t rank = CL ? cl_rank() : 0, g = threadIdx.x >> 3, k = threadIdx.x & 7;
  bool cl = CL;
  TailMap mp{CL ? TAIL_CLUSTER : 1u, rank};
  const uint32_t whole = h;
  if (CL) h /= TAIL_CLUSTER;  // this block's points
  uint32_t stride = 2 * h;
  ef *sc = reinterpret_cast<ef*>(tail_smem), *se = sc + 3 * stride;
  ef* const joined = se + h;  // CL, block 0: the joined columns (2 TAIL_BLOCK_H entries each) and eq table
  if (rank == 0) fin_load(FIN_EQSC3, fin);
  if (fold_in) {
    tail_fold<3>(cols, size_t(4) * whole, sc, stride, stride, ch0->c[k], mp);
    for (uint32_t i = threadIdx.x; i < 8 * h; i += TAIL_THREADS) {
      const uint32_t x = (i >> 3) * mp.m + mp.x0;
      se[i >> 3].c[k] = kb::add(eq_in[x].c[k], eq_in[x + whole].c[k]);
    }
  } else {
    tail_copy<3>(cols, size_t(2) * whole, sc, stride, stride, mp);
    tail_copy<1>(eq_in, 0, se, 0, h, mp);
  }
  if (CL) cl_sync();  // every block runs: from here its shared memory may be written
  else __syncthreads();
  const int round0 = fin_sm.st.round;
#pragma unroll 1
  for (int t = 0;; t++, h >>= 1) {
    // the eq challenge of a round after the first of the launch
    if (t && rank == 0 && threadIdx.x >= TAIL_THREADS - 16)
      (threadIdx.x < TAIL_THREADS - 8 ? fin_sm.r : fin_sm.rinv).c[k] =
          (threadIdx.x < TAIL_THREADS - 8 ? fin.req : fin.rinv)[round0 + t].c[k];
    uint32_t acc[2] = {0, 0};
#pragma unroll 1
    for (uint32_t x0 = 0; x0 < h; x0 += TAIL_GROUPS) {
      const uint32_t x = x0 + g;
      const bool on = x < h;
      uint32_t lo[3], d[3];
#pragma unroll
      for (int q = 0; q < 3; q++) {
        lo[q] = on ? sc[q * stride + x].c[k] : 0u;
        const uint32_t hi = on ? sc[q * stride + x + h].c[k] : 0u;
        d[q] = kb::sub(kb::dbl(hi), lo[q]);
      }
      const uint32_t e = on ? se[x].c[k] : 0u;
      acc[0] = kb::add(acc[0], fin_mul(kb::sub(fin_mul(lo[0], lo[1]), lo[2]), e));
      acc[1] = kb::add(acc[1], fin_mul(kb::sub(fin_mul(d[0], d[1]), d[2]), e));
    }
    tail_finish<2>(FIN_EQSC3, fin, acc, cl, rank);
    if (t == rounds - 1) break;
    const bool join = CL && cl && h * TAIL_CLUSTER == 2 * TAIL_BLOCK_H;
    ef* dst = join ? cl_map(joined, 0) : sc;
    ef* edst = join ? dst + 6 * TAIL_BLOCK_H : se;
    const TailMap dm = join ? mp : TailMap{};
    tail_fold<3>(sc, stride, dst, join ? 2 * TAIL_BLOCK_H : stride, h, fin_sm.chal.c[k], {}, dm);
    // the eq table without its leading variable (in place: an entry written is read by the same
    // thread only)
    for (uint32_t i = threadIdx.x; i < 4 * h; i += TAIL_THREADS)
      edst[(i >> 3) * dm.m + dm.x0].c[k] = kb::add(se[i >> 3].c[k], se[(i >> 3) + h / 2].c[k]);
    if (join) {
      cl_sync();
      if (rank) return;
      cl = false;
      mp = {};
      h *= TAIL_CLUSTER;
      stride = 2 * TAIL_BLOCK_H;
      sc = joined;
      se = joined + 6 * TAIL_BLOCK_H;
    } else {
      __syncthreads();
    }
  }
  tail_fold<3>(sc, stride, oc, size_t(h) * mp.m, h, fin_sm.chal.c[k], {}, mp);
  if (rank == 0 && threadIdx.x < 32) fin_commit(fin);
}

// ------------------------------------------------------------------ a*b - c

// Round 0 of the a*b - c zerocheck: for every point z of the skipped variables' extension and
// every x, v_z(x) = A_z(x) B_z(x) - C_z(x) with A_z(x) = sum_j L_j(z) a[j S + x] (and B, C the
// same), weighted by eq(x). Grid-stride over x, one thread per x at a time, all nz points per
// thread: each value is read once (a, b, c and eq(x) coalesced), the points' products stay in
// registers, and each thread keeps nz extension accumulators that one block reduction sums at
// the end (one partial per block and point).
// The inputs are the caller's canonical words, read as they are: lw and sel come multiplied by
// 2^32 once more than Montgomery form, which makes the weighted sums Montgomery values (a pass
// that copied and converted the three columns took 0.13 ms of a 2^24 proof). Any 32-bit word is
// taken for its residue.
__device__ __forceinline__ uint32_t abc_in(uint32_t x) {
  x = kb::umin(x, x - P);
  return kb::umin(x, x - P);  // 2^32 < 3 p
}
constexpr int ABC_X = 32;
constexpr int ABC0_THREADS = 256;
template <int K>
__global__ void __launch_bounds__(ABC0_THREADS, 2) k_abc0_eval(const uint32_t* __restrict__ a,
                                                           const uint32_t* __restrict__ b,
                                                           const uint32_t* __restrict__ c, size_t S,
                                                           const uint32_t* __restrict__ lw,
                                                           const ef* __restrict__ eq, ef* __restrict__ partial) {
  constexpr int NSK = 1 << K, NZ = NSK - 1;
  __shared__ uint32_t w_s[NZ * NSK];
  __shared__ ef scratch[32];
  for (int i = threadIdx.x; i < NZ * NSK; i += blockDim.x) w_s[i] = lw[i];
  __syncthreads();
  ef acc[NZ];
#pragma unroll
  for (int z = 0; z < NZ; z++) acc[z] = ef_zero();
  for (size_t x = size_t(blockIdx.x) * blockDim.x + threadIdx.x; x < S; x += size_t(gridDim.x) * blockDim.x) {
    uint32_t va[NSK], vb[NSK], vc[NSK];
#pragma unroll
    for (int j = 0; j < NSK; j++) {
      va[j] = abc_in(a[size_t(j) * S + x]);
      vb[j] = abc_in(b[size_t(j) * S + x]);
      vc[j] = abc_in(c[size_t(j) * S + x]);
    }
    const ef e = eq[x];
#pragma unroll
    for (int z = 0; z < NZ; z++) {
      const uint32_t* wz = w_s + z * NSK;
      uint64_t sa[2] = {0, 0}, sb[2] = {0, 0}, sc[2] = {0, 0};
#pragma unroll
      for (int j = 0; j < NSK; j++)
        sa[j >> 2] += wmul(wz[j], va[j]), sb[j >> 2] += wmul(wz[j], vb[j]), sc[j >> 2] += wmul(wz[j], vc[j]);
      auto fin = [](const uint64_t* s) { return NSK > 4 ? add(redc(s[0]), redc(s[1])) : redc(s[0]); };
      acc[z] = ef_add(acc[z], ef_mul_f(e, sub(mul(fin(sa), fin(sb)), fin(sc))));
    }
  }
#pragma unroll
  for (int z = 0; z < NZ; z++) {
    const ef t = block_reduce_ef(acc[z], scratch);
    if (threadIdx.x == 0) partial[size_t(blockIdx.x) * NZ + z] = t;
    __syncthreads();  // scratch is reused by the next point
  }
}

// One thread per (x, point) with the block spanning the points: the form for 4 skipped
// variables (15 points, too many to keep per thread).
__global__ void k_abc0_eval_points(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b,
                            const uint32_t* __restrict__ c, size_t S, int nsk, int nz, const uint32_t* __restrict__ lw,
                            const ef* __restrict__ eq, ef* __restrict__ partial) {
  __shared__ uint32_t w_s[32 * 16];
  const int tid = threadIdx.y * ABC_X + threadIdx.x;
  for (int i = tid; i < nz * nsk; i += ABC_X * blockDim.y) w_s[i] = lw[i];
  __syncthreads();
  const size_t x = size_t(blockIdx.x) * ABC_X + threadIdx.x;
  const int zi = threadIdx.y;
  ef res = ef_zero();
  if (x < S && zi < nz) {
    const uint32_t* wz = w_s + zi * nsk;
    uint64_t sa[4] = {0, 0, 0, 0}, sb[4] = {0, 0, 0, 0}, sc[4] = {0, 0, 0, 0};
    for (int j = 0; j < nsk; j++) {
      size_t i = size_t(j) * S + x;
      sa[j & 3] += wmul(wz[j], abc_in(a[i]));
      sb[j & 3] += wmul(wz[j], abc_in(b[i]));
      sc[j & 3] += wmul(wz[j], abc_in(c[i]));
    }
    auto fin = [](uint64_t* s) { return add(add(redc(s[0]), redc(s[1])), add(redc(s[2]), redc(s[3]))); };
    uint32_t v = sub(mul(fin(sa), fin(sb)), fin(sc));
    res = ef_mul_f(eq[x], v);
  }
  res = warp_reduce_ef(res);
  if (threadIdx.x == 0 && zi < nz) partial[size_t(blockIdx.x) * nz + zi] = res;
}

// sum_j sel[j] src[j S + x], the loads first.
template <int NSK>
__device__ __forceinline__ ef abc_fold0(const uint32_t* __restrict__ src, size_t S, size_t x, const ef* sel) {
  uint32_t v[NSK];
#pragma unroll
  for (int j = 0; j < NSK; j++) v[j] = src[size_t(j) * S + x];
  EfMacF m;
  m.init();
#pragma unroll
  for (int j = 0; j < NSK; j++) {
    m.mac(sel[j], abc_in(v[j]));
    if ((j & 3) == 3 && j + 1 < NSK) m.flush();
  }
  return m.value();
}
template <int NSK>
__global__ void k_abc0_fold(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b,
                            const uint32_t* __restrict__ c, size_t S, const ef* __restrict__ sel_g,
                            ef* __restrict__ out) {
  __shared__ ef sel[NSK];
  if (threadIdx.x < NSK) sel[threadIdx.x] = sel_g[threadIdx.x];
  __syncthreads();
  const size_t x = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (x >= S) return;
  const uint32_t* src = blockIdx.y == 0 ? a : blockIdx.y == 1 ? b : c;
  out[size_t(blockIdx.y) * S + x] = abc_fold0<NSK>(src, S, x, sel);
}
// The same with round 1 in one pass: thread x folds entries x and x + h of every column (h = S/2),
// sums the eq table's leading variable out and adds round 1's values at 0 and 2; the last block
// finishes the round. The folded columns are then written once and not read again before round
// 2's fold. For 2^24 values and three skips: 0.24 ms, against 0.33 ms in four launches (fold, eq
// table, sums, finish).
template <int NSK>
__global__ void __launch_bounds__(FE_THREADS, 2)
    k_abc0_fold_eval(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, const uint32_t* __restrict__ c,
                     size_t S, const ef* __restrict__ sel_g, const ef* __restrict__ eq, ef* __restrict__ out,
                     ef* __restrict__ eq_new, ef* __restrict__ partial, const FinArgs fin) {
  __shared__ ef scratch[32];
  __shared__ ef sel[NSK];
  if (threadIdx.x < NSK) sel[threadIdx.x] = sel_g[threadIdx.x];
  __syncthreads();
  const size_t h = S / 2;
  ef s0 = ef_zero(), s2 = ef_zero();
  for (size_t x = size_t(blockIdx.x) * blockDim.x + threadIdx.x; x < h; x += size_t(gridDim.x) * blockDim.x) {
    // column q's entry x, and its value at 2 of the leading variable
    auto column = [&](const uint32_t* src, int q, ef& lo, ef& at2) {
      lo = abc_fold0<NSK>(src, S, x, sel);
      out[size_t(q) * S + x] = lo;
      const ef hi = abc_fold0<NSK>(src, S, x + h, sel);
      out[size_t(q) * S + x + h] = hi;
      at2 = ef_sub(ef_add(hi, hi), lo);
    };
    ef p0, p2, lo, at2;
    column(a, 0, p0, p2);
    column(b, 1, lo, at2);
    p0 = ef_mul(p0, lo);
    p2 = ef_mul(p2, at2);
    column(c, 2, lo, at2);
    const ef e = ef_add(eq[x], eq[x + h]);
    eq_new[x] = e;
    s0 = ef_add(s0, ef_mul(ef_sub(p0, lo), e));
    s2 = ef_add(s2, ef_mul(ef_sub(p2, at2), e));
  }
  s0 = block_reduce_ef(s0, scratch);
  if (threadIdx.x == 0) partial[size_t(blockIdx.x) * 2] = s0;
  __syncthreads();
  s2 = block_reduce_ef(s2, scratch);
  if (threadIdx.x == 0) partial[size_t(blockIdx.x) * 2 + 1] = s2;
  fin_last_block(FIN_EQSC3, fin, partial, 2);
}

__global__ void k_abc_eval_ef(const ef* __restrict__ cols, int m, const ef* __restrict__ eq, ef* __restrict__ partial) {
  const size_t len = size_t(1) << m, half = len >> 1;
  const size_t x = size_t(blockIdx.x) * 32 + threadIdx.x;
  const int zi = threadIdx.y;  // z = 0 or 2
  ef res = ef_zero();
  if (x < half) {
    ef v[3];
    for (int q = 0; q < 3; q++) {
      ef lo = cols[q * len + x], hi = cols[q * len + half + x];
      v[q] = zi == 0 ? lo : ef_sub(ef_add(hi, hi), lo);
    }
    res = ef_mul(ef_sub(ef_mul(v[0], v[1]), v[2]), eq[x]);
  }
  res = warp_reduce_ef(res);
  if (threadIdx.x == 0) partial[size_t(blockIdx.x) * 2 + zi] = res;
}
}  // namespace

// ------------------------------------------------------------------ launchers
void launch_eq_table(const ef* point, int nvars, ef* out, cudaStream_t s) {
  if (nvars > EQ_MAX_VARS) throw std::invalid_argument("eq table: too many variables");
  k_eq_table<<<(unsigned)(size_t(1) << (nvars - eq_block_bits(nvars))), EQ_THREADS, 0, s>>>(point, nvars, out);
  WL_LAUNCH_CHECK();
}
bool EqTables::add(const ef* point, int nv, ef* table) {
  if (nv > EQ_MAX_VARS) throw std::invalid_argument("eq table: too many variables");
  const int used = n ? off[n - 1] + nvars[n - 1] : 0;
  if (n == MAX_TABLES || used + nv > MAX_VARS) return false;
  off[n] = used;
  nvars[n] = nv;
  out[n] = table;
  for (int i = 0; i < nv; i++) pt[used + i] = point[i];
  if (!n) first[0] = 0;
  first[n + 1] = first[n] + (1 << (nv - eq_block_bits(nv)));
  n++;
  return true;
}
void launch_eq_tables(const EqTables& e, cudaStream_t s) {
  if (!e.n) return;
  k_eq_tables<<<(unsigned)e.first[e.n], EQ_THREADS, 0, s>>>(e);
  WL_LAUNCH_CHECK();
}
void launch_eq_table_f(const uint32_t* pts, int npts, int nvars, uint32_t* out, cudaStream_t s) {
  size_t n = size_t(npts) << nvars;
  if (!n) return;
  k_eq_table_f<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(pts, npts, nvars, out);
  WL_LAUNCH_CHECK();
}
void launch_reduce_partials(const ef* partial, int nblk, int k, ef* out, cudaStream_t s) {
  k_reduce_partials<<<k, 256, 0, s>>>(partial, nblk, k, out);
  WL_LAUNCH_CHECK();
}

static int zc0_tiles(int log_n, int k, int xs) {  // blocks of xs x
  size_t S = size_t(1) << (log_n - k);
  return (int)((S + xs - 1) / xs);
}
static int zc0_splits(int tiles, int groups) {
  const int want = std::min(std::max(ZC0_FILL / tiles, 1), groups);
  const int per = (groups + want - 1) / want;
  return (groups + per - 1) / per;  // no empty range
}
int zc0_blocks(int log_n, int k) {
  const int tiles = zc0_tiles(log_n, k, ZE_X);
  return tiles * zc0_splits(tiles, ZC0_GRPS);
}
static int zc0_row_threads(int log_n) { return (size_t(1) << log_n) < size_t(148) * ZC0R_THREADS ? ZC0R_SMALL : ZC0R_THREADS; }
int zc0_row_blocks(int log_n) {
  const int t = zc0_row_threads(log_n);
  return (int)(((size_t(1) << log_n) + t - 1) / t);
}
void launch_zc0_rows(const uint32_t* wit, int log_n, int k, int nz, const uint32_t* lw, const ef* eq,
                     const ef* alphas, const ef* betas, const AirConsts& K, uint32_t* q, ef* partial, ef* arow,
                     cudaStream_t s) {
  if (nz > 32) throw std::invalid_argument("zc0_rows: at most 32 points");
  k_zc0_rows<<<zc0_row_blocks(log_n) + 1, zc0_row_threads(log_n), 0, s>>>(
      wit, log_n, k, nz, lw, eq, alphas, betas, K, q, partial, arow, q + (size_t(ZC0_NQ) << log_n));
  WL_LAUNCH_CHECK();
}
void launch_zc0_eval(const uint32_t* wit, const uint32_t* q, int log_n, int k, int nz, const ef* eq,
                     const AirConsts& K, ef* partial, cudaStream_t s) {
  if (nz > 32) throw std::invalid_argument("zc0_eval: at most 32 points");
  const int tiles = zc0_tiles(log_n, k, ZE_X);
  k_zc0_eval_mma<<<dim3(tiles, zc0_splits(tiles, ZC0_GRPS)), ZC0M_WARPS * 32, 0, s>>>(
      wit, q, log_n, k, nz, eq, q + (size_t(ZC0_NQ) << log_n), K, partial);
  WL_LAUNCH_CHECK();
}
void launch_zc0_fold(const uint32_t* src, int log_n, int k, int cb, int ce, const ef* sel, const ef* arow, ef* out,
                     cudaStream_t s) {
  size_t S = size_t(1) << (log_n - k);
  if (S < 2) throw std::invalid_argument("zc0_fold: at least 2 points per skip block");
  const int tiles = zc0_tiles(log_n, k, ZC0_X), splits = zc0_splits(tiles, (ce - cb + ZC0_GROUP - 1) / ZC0_GROUP);
  k_zc0_fold_mma<<<dim3(tiles, splits + (arow ? 1 : 0)), ZC0M_WARPS * 32, 0, s>>>(src, log_n, k, cb, ce, sel, arow,
                                                                                 out);
  WL_LAUNCH_CHECK();
}
// x blocks of 32, and the split of the columns that gives at least ZCS_FILL blocks.
constexpr int ZCS_FILL = 2 * 2 * 148;
static dim3 zcs_grid(int m) {
  const size_t bx = ((size_t(1) << (m - 1)) + 31) / 32;
  constexpr int most = AIR_NC / ZCS_COLS;  // one column per warp
  const int want = (int)std::min<size_t>((ZCS_FILL + bx - 1) / bx, most);
  const int per = (most + want - 1) / want;
  return dim3((unsigned)bx, (unsigned)((most + per - 1) / per));
}
bool zc_eval_is_dense(int m) { return zcs_grid(m).y < unsigned(AIR_NC / ZCS_COLS); }
int zc_ef_blocks(int m) {
  const dim3 g = zcs_grid(m);
  return (int)(g.x * g.y);
}
std::vector<ef> zc_gammas(const std::vector<ef>& alphas, const std::vector<ef>& betas) {
  std::vector<ef> g(2 * AIR_NC);
  for (int c = 0; c < AIR_NC; c++) {
    const ef v = c < 16   ? betas[c]
                 : c < 36 ? alphas[c + 48]   // partial round c - 16: constraint 64 + (c - 16)
                 : c < 52 ? betas[c + 28]    // ending round 0
                 : c < 100 ? betas[c - 36]   // beginning rounds 1..3
                           : betas[c - 20];  // ending rounds 1..3
    g[2 * c] = v;
    g[2 * c + 1] = kb::ef_add(kb::ef_add(v, v), v);
  }
  return g;
}
void launch_zc_eval_ef(const ef* cols, const ef* cols2, int m, const ef* eq, const ef* gammas, const AirConsts& K,
                       ef* partial, cudaStream_t s) {
  k_zc_sbox<<<zcs_grid(m), ZCS_THREADS, 0, s>>>(ZcCols{cols, cols2, cols2 ? ZC0_NQ : ZC_COLS}, m, eq, gammas, K,
                                                partial);
  WL_LAUNCH_CHECK();
}
void launch_fold_cols(const ef* in, ef* out, int ncols, size_t half, const ef* r, cudaStream_t s, const ef* eq_in,
                      ef* eq_out, size_t eq_half) {
  const size_t width = eq_in && eq_half > half ? eq_half : half;
  dim3 grid((unsigned)((width + 255) / 256), ncols + (eq_in ? 1 : 0));
  k_fold_cols<<<grid, 256, 0, s>>>(in, out, half, ncols, r, ef_zero(), eq_in, eq_out, eq_half);
  WL_LAUNCH_CHECK();
}
// 128 values of a column at a time per block; a block of a large table goes on to further ones (up
// to FOLD_TILES) while at least FOLD_FILL blocks are left, as forming the challenge's operand costs
// a warp about as much as a tile: the folds of 2^20 rows 0.40 ms with one tile a block, 0.32 so.
constexpr size_t FOLD_TILES = 8, FOLD_FILL = 8 * 148;
static dim3 fold_cols_grid(int ncols, size_t half, bool eq) {
  const size_t tiles = std::max<size_t>((half + 127) / 128, 1);
  const size_t per = std::min(std::max<size_t>(tiles * size_t(ncols) / FOLD_FILL, 1), FOLD_TILES);
  return dim3((unsigned)((tiles + per - 1) / per), ncols + (eq ? 1 : 0));
}
void launch_fold_cols_at(const ef* in, ef* out, int ncols, size_t half, const ef& r, cudaStream_t s, const ef* eq_in,
                         ef* eq_out, size_t eq_half, const ef* in2, int split) {
  const dim3 grid = fold_cols_grid(ncols, half, eq_in != nullptr);
  k_fold_cols_mma<<<grid, 256, 0, s>>>(ZcCols{in, in2, in2 ? split : ncols}, out, half, ncols, r, nullptr, eq_in, eq_out, eq_half);
  WL_LAUNCH_CHECK();
}
void launch_fold_cols_dev(const ef* in, ef* out, int ncols, size_t half, const ef* r_dev, cudaStream_t s,
                          const ef* eq_in, ef* eq_out, size_t eq_half, const ef* in2, int split) {
  const dim3 grid = fold_cols_grid(ncols, half, eq_in != nullptr);
  k_fold_cols_mma<<<grid, 256, 0, s>>>(ZcCols{in, in2, in2 ? split : ncols}, out, half, ncols, ef_zero(), r_dev, eq_in, eq_out, eq_half);
  WL_LAUNCH_CHECK();
}
void launch_inner_sums(const uint32_t* wit, int log_n, int k, int ll, const ef* eq_hi, const ef* eq_lo,
                       const ef* sel, ef* out_up, ef* out_down, uint8_t* limbs, cudaStream_t s, int plan,
                       unsigned* timeouts) {
  // out_up / out_down hold AIR_W results followed by AIR_W * 2^k * 2^(log_n - k - ll) partials.
  const int nsk = 1 << k;
  const int nh = 1 << (log_n - k - ll);
  ef* pu = out_up + AIR_W;
  ef* pd = out_down + AIR_W;
  if (limbs && ll >= INNER_MMA_MIN_LL && ll <= 12) {  // 2^12 byte products per s32 sum
    const int nlo = 1 << ll;
    k_eq_limbs<<<(16 * nlo + 255) / 256, 256, 0, s>>>(eq_lo, nlo, limbs);
    WL_LAUNCH_CHECK();
    const uint32_t M = uint32_t(AIR_W) * nsk * nh;
    if (plan == 1 && timeouts)
      k_inner_sums_bulk<<<(M + 15) / 16, ISM_WARPS * 32, 0, s>>>(wit, log_n, k, ll, eq_hi, eq_lo, limbs, pu, pd,
                                                                 timeouts);
    else
      k_inner_sums_mma<<<(M + 15) / 16, ISM_WARPS * 32, 0, s>>>(wit, log_n, k, ll, eq_hi, eq_lo, limbs, pu, pd);
  } else {
    k_inner_sums<<<dim3((AIR_W + 1) / 2, nsk, (nh + IS_WARPS - 1) / IS_WARPS), IS_WARPS * 32, 0, s>>>(
        wit, log_n, k, ll, eq_hi, eq_lo, pu, pd);
  }
  WL_LAUNCH_CHECK();
  k_combine_sel<<<(AIR_W + 7) / 8, 256, 0, s>>>(pu, sel, nsk, nh, AIR_W, out_up);
  WL_LAUNCH_CHECK();
  k_combine_sel<<<(AIR_W + 7) / 8, 256, 0, s>>>(pd, sel, nsk, nh, AIR_W, out_down);
  WL_LAUNCH_CHECK();
}
size_t colsum_limb_bytes(int K) { return K > 192 ? 0 : size_t(32) * ((K + 31) / 32 * 32); }
void launch_batch_cols_mma(const uint32_t* wit, int log_n, const ef* eqc, ef* out, uint8_t* limbs, cudaStream_t s) {
  const size_t N = size_t(1) << log_n;
  const int K = AIR_W, Kp = (K + 31) / 32 * 32;
  k_w_limbs<<<(8 * Kp + 255) / 256, 256, 0, s>>>(eqc, K, Kp, limbs);
  WL_LAUNCH_CHECK();
  const size_t tiles = (N + 15) / 16;
  k_colsum_mma<<<(unsigned)((tiles + CS_WARPS - 1) / CS_WARPS), CS_WARPS * 32, 0, s>>>(wit, N, K, Kp, N, limbs, out);
  WL_LAUNCH_CHECK();
}
size_t mle_partial_scratch_bytes(int lu, int lh, int ll) {
  if (ll < INNER_MMA_MIN_LL || ll > 12 || lh < 4) return 0;
  return (sizeof(ef) << (lu + lh - 4)) + (size_t(32) << ll);
}
bool launch_mle_partial_mma(const uint32_t* T, size_t t_len, int lu, int lh, int ll, const ef* hi, const ef* lo,
                            ef* out, void* scratch, cudaStream_t s) {
  if (!scratch || !mle_partial_scratch_bytes(lu, lh, ll) || t_len % (size_t(1) << ll)) return false;
  ef* partial = static_cast<ef*>(scratch);
  uint8_t* limbs = reinterpret_cast<uint8_t*>(partial + (size_t(1) << (lu + lh - 4)));
  const int nlo = 1 << ll;
  k_lo_limbs<<<(8 * nlo + 255) / 256, 256, 0, s>>>(lo, nlo, limbs);
  WL_LAUNCH_CHECK();
  const uint32_t tiles = 1u << (lu + lh - 4);
  k_mle_partial_mma<<<(tiles + CS_WARPS - 1) / CS_WARPS, CS_WARPS * 32, 0, s>>>(T, t_len, lu, lh, ll, hi, limbs,
                                                                               partial);
  WL_LAUNCH_CHECK();
  launch_reduce_partials(partial, 1 << (lh - 4), 1 << lu, out, s);
  return true;
}
void launch_batch_cols(const uint32_t* wit, int log_n, const ef* eqc, ef* out, cudaStream_t s) {
  if (log_n < 1) throw std::invalid_argument("batch_cols: at least 2 rows");
  size_t N = size_t(1) << log_n;
  k_batch_cols<<<(unsigned)((N / 2 + 255) / 256), 256, 0, s>>>(wit, log_n, eqc, out);
  WL_LAUNCH_CHECK();
}
int sub_eval_blocks(int log_n, int k) {
  size_t S = size_t(1) << (log_n - k);
  size_t per = size_t(SUB_THREADS) * SUB_PER_THREAD;
  return (int)((S + per - 1) / per);
}
void launch_sub_evals(const ef* B, int log_n, int k, const ef* alpha2, const ef* eqt, ef* partial, cudaStream_t s) {
  (void)alpha2;
  dim3 grid(sub_eval_blocks(log_n, k), 1u << k);
  k_sub_evals<<<grid, SUB_THREADS, 0, s>>>(B, log_n, k, eqt, partial);
  WL_LAUNCH_CHECK();
}
void launch_inner_mle(const ef* e, int log_n, const ef* alpha2, ef* out, cudaStream_t s) {
  size_t N = size_t(1) << log_n;
  k_inner_mle<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(e, log_n, alpha2, out);
  WL_LAUNCH_CHECK();
}
int prod_blocks(size_t half) {
  size_t per = size_t(PROD_THREADS) * prod_per_thread(half);
  return (int)((half + per - 1) / per);
}
void launch_prod_eval(const ef* a, const ef* b, size_t half, ef* partial, cudaStream_t s) {
  k_prod_eval<<<prod_blocks(half), PROD_THREADS, 0, s>>>(a, b, half, prod_per_thread(half), partial);
  WL_LAUNCH_CHECK();
}
void launch_fold2_at(const ef* a, const ef* b, ef* oa, ef* ob, size_t half, const ef& r, cudaStream_t s) {
  k_fold2_mma<<<dim3((unsigned)((half + 127) / 128), 2), 256, 0, s>>>(a, b, oa, ob, half, r, nullptr);
  WL_LAUNCH_CHECK();
}
void launch_fold2_dev(const ef* a, const ef* b, ef* oa, ef* ob, size_t half, const ef* r_dev, cudaStream_t s) {
  k_fold2_mma<<<dim3((unsigned)((half + 127) / 128), 2), 256, 0, s>>>(a, b, oa, ob, half, ef_zero(), r_dev);
  WL_LAUNCH_CHECK();
}

int fold_eval_blocks(size_t h) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return (int)std::max<size_t>(1, std::min<size_t>((h + FE_THREADS - 1) / FE_THREADS, size_t(sms) * 4));
}
void launch_pair_fold_eval(int nsums, const ef* a, const ef* b, const ef* r_dev, ef* na, ef* nb, size_t h,
                           ef* partial, const FinArgs* fin, cudaStream_t s) {
  const int g = fold_eval_blocks(h);
  const FinArgs f = fin ? *fin : FinArgs{};
  if (nsums == 2)
    k_pair_fold_eval<2><<<g, FE_THREADS, 0, s>>>(a, b, r_dev, na, nb, h, partial, f);
  else if (nsums == 3)
    k_pair_fold_eval<3><<<g, FE_THREADS, 0, s>>>(a, b, r_dev, na, nb, h, partial, f);
  else
    throw std::invalid_argument("fold-evaluate: 2 or 3 sums");
  WL_LAUNCH_CHECK();
}
namespace {
// Opts a kernel into `bytes` of dynamic shared memory, once per device.
template <class K>
void tail_smem_limit(K kernel, size_t bytes) {
  if (bytes <= 32 * 1024) return;  // beside the static part, within the default 48 KB
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> done;
  int dev = 0;
  WL_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  size_t& d = done[{dev, reinterpret_cast<const void*>(kernel)}];
  if (d >= bytes) return;
  WL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)));
  d = bytes;
}
}  // namespace

// One block up to TAIL_BLOCK_H points, else a cluster (local tables and the joined ones); entries per
// point: `per` in the round's tables.
template <class K, class... A>
static void launch_tail(K one, K cluster, size_t h, size_t per, cudaStream_t s, A... args) {
  const bool cl = h > TAIL_BLOCK_H;
  const size_t smem = sizeof(ef) * per * (cl ? h / TAIL_CLUSTER + TAIL_BLOCK_H : h);
  tail_smem_limit(cl ? cluster : one, smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cl ? TAIL_CLUSTER : 1);
  cfg.blockDim = dim3(TAIL_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = TAIL_CLUSTER;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cl ? 1 : 0;
  WL_CUDA(cudaLaunchKernelEx(&cfg, cl ? cluster : one, args...));
}
static void tail_check(size_t h, int rounds) {
  if (h < 1 || h > TAIL_MAX_H || (h & (h - 1)) || rounds < 1 || (h >> (rounds - 1)) < 1)
    throw std::invalid_argument("sumcheck tail: size");
}
void launch_pair_tail(int nsums, const ef* a, const ef* b, size_t h, const ef* fold_ch, int rounds, ef* oa, ef* ob,
                      const FinArgs& fin, cudaStream_t s) {
  tail_check(h, rounds);
  if (nsums == 2)
    launch_tail(k_pair_tail<2, false>, k_pair_tail<2, true>, h, 4, s, a, b, uint32_t(h), fold_ch != nullptr, fold_ch,
                rounds, oa, ob, fin);
  else
    launch_tail(k_pair_tail<3, false>, k_pair_tail<3, true>, h, 4, s, a, b, uint32_t(h), fold_ch != nullptr, fold_ch,
                rounds, oa, ob, fin);
}
void launch_abc_tail(const ef* cols, const ef* eq_in, size_t h, const ef* fold_ch, int rounds, ef* oc,
                     const FinArgs& fin, cudaStream_t s) {
  tail_check(h, rounds);
  launch_tail(k_abc_tail<false>, k_abc_tail<true>, h, 7, s, cols, eq_in, uint32_t(h), fold_ch != nullptr, fold_ch, rounds,
              oc, fin);
}

void launch_abc_fold_eval(const ef* cols, const ef* r_dev, const ef* eq_prev, ef* nc, ef* eq_new, size_t h, ef* partial,
                          const FinArgs* fin, cudaStream_t s) {
  const FinArgs f = fin ? *fin : FinArgs{};
  if (fin && (!f.req || !f.rinv)) throw std::invalid_argument("fold-evaluate: eq-factor rounds need their eq challenges");
  k_abc_fold_eval<<<fold_eval_blocks(h), FE_THREADS, 0, s>>>(cols, r_dev, eq_prev, nc, eq_new, h, partial, f);
  WL_LAUNCH_CHECK();
}

int abc0_blocks(int log_n, int k) {
  const size_t S = size_t(1) << (log_n - k);
  if (k > 3) return (int)((S + ABC_X - 1) / ABC_X);
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return (int)std::max<size_t>(1, std::min<size_t>((S + ABC0_THREADS - 1) / ABC0_THREADS, size_t(sms) * 2));
}
void launch_abc0_eval(const uint32_t* a, const uint32_t* b, const uint32_t* c, int log_n, int k, int nz,
                      const uint32_t* lw, const ef* eq, ef* partial, cudaStream_t s) {
  const size_t S = size_t(1) << (log_n - k);
  const int nb = abc0_blocks(log_n, k);
  if (k < 1 || k > 4 || nz != (1 << k) - 1) throw std::invalid_argument("abc round 0: skips 1..4");
  if (k == 1) k_abc0_eval<1><<<nb, ABC0_THREADS, 0, s>>>(a, b, c, S, lw, eq, partial);
  if (k == 2) k_abc0_eval<2><<<nb, ABC0_THREADS, 0, s>>>(a, b, c, S, lw, eq, partial);
  if (k == 3) k_abc0_eval<3><<<nb, ABC0_THREADS, 0, s>>>(a, b, c, S, lw, eq, partial);
  if (k == 4) k_abc0_eval_points<<<nb, dim3(ABC_X, nz), 0, s>>>(a, b, c, S, 1 << k, nz, lw, eq, partial);
  WL_LAUNCH_CHECK();
}
void launch_abc0_fold(const uint32_t* a, const uint32_t* b, const uint32_t* c, int log_n, int k, const ef* sel,
                      ef* out, cudaStream_t s) {
  const size_t S = size_t(1) << (log_n - k);
  const dim3 grid((unsigned)((S + 255) / 256), 3);
  if (k < 1 || k > 4) throw std::invalid_argument("abc round 0: skips 1..4");
  if (k == 1) k_abc0_fold<2><<<grid, 256, 0, s>>>(a, b, c, S, sel, out);
  if (k == 2) k_abc0_fold<4><<<grid, 256, 0, s>>>(a, b, c, S, sel, out);
  if (k == 3) k_abc0_fold<8><<<grid, 256, 0, s>>>(a, b, c, S, sel, out);
  if (k == 4) k_abc0_fold<16><<<grid, 256, 0, s>>>(a, b, c, S, sel, out);
  WL_LAUNCH_CHECK();
}
int abc0_fold_eval_blocks(int log_n, int k) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t h = size_t(1) << (log_n - k - 1);
  return (int)std::max<size_t>(1, std::min<size_t>((h + FE_THREADS - 1) / FE_THREADS, size_t(sms) * 2));
}
void launch_abc0_fold_eval(const uint32_t* a, const uint32_t* b, const uint32_t* c, int log_n, int k, const ef* sel,
                           const ef* eq, ef* out, ef* eq_new, ef* partial, const FinArgs& fin, cudaStream_t s) {
  const size_t S = size_t(1) << (log_n - k);
  const int nb = abc0_fold_eval_blocks(log_n, k);
  if (k < 1 || k > 4 || S < 2) throw std::invalid_argument("abc round 0: skips 1..4");
  if (k == 1) k_abc0_fold_eval<2><<<nb, FE_THREADS, 0, s>>>(a, b, c, S, sel, eq, out, eq_new, partial, fin);
  if (k == 2) k_abc0_fold_eval<4><<<nb, FE_THREADS, 0, s>>>(a, b, c, S, sel, eq, out, eq_new, partial, fin);
  if (k == 3) k_abc0_fold_eval<8><<<nb, FE_THREADS, 0, s>>>(a, b, c, S, sel, eq, out, eq_new, partial, fin);
  if (k == 4) k_abc0_fold_eval<16><<<nb, FE_THREADS, 0, s>>>(a, b, c, S, sel, eq, out, eq_new, partial, fin);
  WL_LAUNCH_CHECK();
}
void launch_abc_eval_ef(const ef* cols, int m, const ef* eq, ef* partial, cudaStream_t s) {
  size_t half = size_t(1) << (m - 1);
  k_abc_eval_ef<<<(unsigned)((half + 31) / 32), dim3(32, 2), 0, s>>>(cols, m, eq, partial);
  WL_LAUNCH_CHECK();
}

}  // namespace wl
