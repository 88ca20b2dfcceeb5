// Batched Merkle-path checks for the verifier (the GPU part of wl_verify_batch_device). The
// host replays each proof's transcript with its Merkle openings deferred (verify_air_proof
// with a deferral list); the openings of all proofs are then checked here, one thread per
// opening: the leaf sponge over the opened row (PaddingFreeSponge over Poseidon2-24, rate 16,
// 8 absorptions), then one 2-to-1 compression (Poseidon2-16) per level of its path, and the
// comparison with the root. The words are the proofs' canonical proof_data, so the
// permutations run in the canonical domain, as the prover's trees are built.
#include "kernels.h"

namespace wl {

namespace {

// 128 openings a block, one per thread, on the tensor-core permutations: the sponges with the
// width-24 one, then the paths with the width-16 one on the same shared memory. The matrix products need the whole block, so threads past the last
// opening repeat it, and every thread runs as many levels as the block's longest path; `cur`
// keeps its value past the end of a path.
union VerifyShared {
  kb::P2TcShared<24> p24;
  kb::P2TcShared<16> p16;
};
__global__ void __launch_bounds__(kb::TC_ROWS, 4)
    k_check_openings(const uint32_t* __restrict__ words, const OpeningCheck* __restrict__ ops, int n,
                     const __grid_constant__ kb::P2ConstsTc<24> c24, const __grid_constant__ kb::P2ConstsTc<16> c16,
                     uint8_t* __restrict__ ok, unsigned* __restrict__ timeouts) {
  extern __shared__ __align__(16) char verify_smem[];
  VerifyShared& sh = *reinterpret_cast<VerifyShared*>(verify_smem);
  __shared__ int levels;
  const int i = blockIdx.x * kb::TC_ROWS + threadIdx.x;
  const OpeningCheck op = ops[i < n ? i : n - 1];
  if (threadIdx.x == 0) levels = 0;
  kb::p2_tc_begin<24>(sh.p24);
  atomicMax(&levels, op.ll);
  kb::TcPhase ph;
  uint32_t s[24], cur[8];
#pragma unroll
  for (int j = 0; j < 8; j++) cur[j] = 0;
#pragma unroll 1
  for (int ch = 0; ch < 8; ch++) {
#pragma unroll
    for (int j = 0; j < 16; j++) s[j] = words[op.row + 16 * ch + j];
#pragma unroll
    for (int j = 0; j < 8; j++) s[16 + j] = cur[j];
    kb::p2_permute_tc<24>(s, c24, sh.p24, ph, ch == 7, cur);
#pragma unroll
    for (int j = 0; j < 8; j++) cur[j] = kb::umin(cur[j], cur[j] - kb::P);
  }
  __syncthreads();  // every thread is done with the width-24 operands
  kb::p2_tc_load<16>(sh.p16);
#pragma unroll 1
  for (int l = 0; l < levels; l++) {
    const bool on = l < op.ll;
    const uint32_t* sib = words + op.path + size_t(on ? l : 0) * 8;
    uint32_t t[16], o[8];
    const bool right = (op.q >> l) & 1;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const uint32_t b = op.ll ? sib[j] : 0u;
      t[j] = right ? b : cur[j];
      t[8 + j] = right ? cur[j] : b;
    }
    kb::p2_permute_tc<16>(t, c16, sh.p16, ph, true, o);
#pragma unroll
    for (int j = 0; j < 8; j++) cur[j] = on ? kb::umin(o[j], o[j] - kb::P) : cur[j];
  }
  kb::p2_tc_end<16>(sh.p16, ph, timeouts);
  bool same = true;
#pragma unroll
  for (int j = 0; j < 8; j++) same = same && cur[j] == words[op.root + j];
  if (i < n) ok[i] = same ? 1 : 0;
}

}  // namespace

void launch_check_openings(const uint32_t* words, const OpeningCheck* ops, int n, const kb::P24Consts& p24,
                           const kb::P16Consts& p16, uint8_t* ok, unsigned* timeouts, cudaStream_t s) {
  if (n <= 0) return;
  WL_CUDA(cudaFuncSetAttribute(k_check_openings, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(VerifyShared))));
  k_check_openings<<<(n + kb::TC_ROWS - 1) / kb::TC_ROWS, kb::TC_ROWS, sizeof(VerifyShared), s>>>(
      words, ops, n, kb::p2_consts_tc(p24), kb::p2_consts_tc(p16), ok, timeouts);
  WL_LAUNCH_CHECK();
}

}  // namespace wl
