// tcgen05 / tensor-memory / tiled-TMA wrappers and the arguments shared by the two fused decode + GEMM kernels: gemm_kernel
// (st_gemm.cu: one CTA per tile, and the grouped form) and pair_kernel (st_gemm_pair.cu: CTA pairs, for more tokens).
#pragma once
#include <cuda.h>

#include "st_common.cuh"
#include "st_host.h"

namespace st {

constexpr int NDEC = 8;                      // decode warps of a group = records per k-tile
constexpr int A_COLS = 32;                   // tensor-memory columns of a decoded weight tile: 128 rows x 64 BF16
constexpr int PAIR = 2;                      // k-tiles per decode step
constexpr int RAW_SLOT = NDEC * PAIR * REC;  // 24832 B: the sixteen records of a pair of k-tiles
constexpr int MAXL_GEMM = 4;                 // matrices in one list launch

struct GemmArgs {
  const int* eo; const uint32_t* el;
  uint16_t* Y; float* Yf; int* status;
  // grouped (mixture of experts): per-expert weight tensor maps and escape tables, pairs in moe_align layout
  const CUtensorMap* maps; const long long* eop; const long long* elp;
  const int* sorted; const int* bexp; const int* npost; int E;
  long long M;
  int B, NG, NT, KS, RB, TT, astages, xstages, rstages, bar_off, tmem_cols, rb0;                    // (rb0: first row block of the launch)
  // CTA pairs: first (row pair, token tile) unit of the launch and the one after its last, clusters that share them, tokens of
  // the first MMA of a k-step (all of NT up to 256), rows of an activation box
  int tile0, tile1, nclusters, n1, box;
  // list of matrices that share the activations (q / k / v, gate / up as separate trees): member of each row block
  int nlist; int rbend[MAXL_GEMM];            // first row block after each member in the concatenation
  const int* leo[MAXL_GEMM]; const uint32_t* lel[MAXL_GEMM]; uint16_t* lY[MAXL_GEMM]; float* lYf[MAXL_GEMM];
  long long lM[MAXL_GEMM];
};
struct WMaps { CUtensorMap m[MAXL_GEMM]; };   // weight tensor maps: one, or one per member of a list

// st_gemm_pair.cu: Y = X W^T for more than 128 tokens; a holds the matrix (or list), M, B, NG and the status word.  -1 and nothing
// launched when its estimated time is not less than us
int pair_gemm(GemmArgs& a, const WMaps& wmaps, const void* X, const char* who, double us, cudaStream_t stream);
// st_gemm.cu: activations [rows, N] BF16 as boxes of 64 columns x box_rows rows with the 128-byte swizzle
int make_xmap(CUtensorMap* map, const void* X, long long rows, long long N, int box_rows, const char* who);

#ifdef __CUDACC__
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               :: "r"(smem_addr(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               :: "r"(smem_addr(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar)) : "memory");
}
// CG: CTAs that work on one accumulator tile (every tcgen05 instruction of a kernel names the same number)
template <int CG>
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  if (CG == 1) asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_addr(slot)), "r"(cols) : "memory");
  else asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_addr(slot)), "r"(cols) : "memory");
}
template <int CG>
__device__ __forceinline__ void tmem_relinquish() {
  if (CG == 1) asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  else asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
template <int CG>
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
  if (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(addr), "r"(cols) : "memory");
  else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_addr(bar)) : "memory");
}
// the same for a CTA pair: arrives at the barrier of this offset in every CTA of the cluster named by `ctas` (a bit per rank)
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar, uint16_t ctas) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               :: "r"(smem_addr(bar)), "h"(ctas) : "memory");
}
// D[128 CG x n] (+)= A B^T with A (128 rows of each CTA x 16 BF16: eight 32-bit columns) in tensor memory, B in shared memory
// (CG = 2: n / 2 rows of it in each CTA, at the same offset)
template <int CG>
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint32_t a_tmem, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  if (CG == 1)
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 :: "r"(d_tmem), "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}"
                 :: "r"(d_tmem), "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
// a tiled load into this CTA's shared memory whose bytes are counted on a barrier of either CTA of the pair (`bar`: an address
// in the cluster's shared window)
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               :: "r"(smem_addr(dst)), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// One arrival at a barrier of any CTA of the cluster, behind tcgen05.fence::before_thread_sync.  What it announces lives in tensor
// memory and is ordered by that fence and the waiter's fence::after_thread_sync, so it need not release generic memory: with
// .release.cluster the warp waits for all its memory traffic first (1000 to 1400 cycles per arrival in pair_kernel, as long as
// decoding two records)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" :: "r"(bar) : "memory");
}
// a decoded record (16 rows x 64 BF16 as four mma A fragments) -> 16 lanes x 32 columns of tensor memory.  16x128b: lane
// (g, t) holds column t of rows g (even registers) and g + 8 (odd), each register pair four columns further: exactly
// (A[s][0], A[s][1]) = k 16 s + 2t, (A[s][2], A[s][3]) = k 16 s + 8 + 2t
__device__ __forceinline__ void tmem_st_frag(uint32_t taddr, const uint32_t (&A)[4][4]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               :: "r"(taddr), "r"(A[0][0]), "r"(A[0][1]), "r"(A[0][2]), "r"(A[0][3]), "r"(A[1][0]), "r"(A[1][1]),
                  "r"(A[1][2]), "r"(A[1][3]), "r"(A[2][0]), "r"(A[2][1]), "r"(A[2][2]), "r"(A[2][3]), "r"(A[3][0]),
                  "r"(A[3][1]), "r"(A[3][2]), "r"(A[3][3]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// shared-memory matrix descriptor: K-major operand, 128-byte swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}


// instruction descriptor: D fp32, A and B bf16, both K-major, N = n, M = m rows (128, of a CTA pair 256)
__host__ __device__ constexpr uint32_t mma_idesc(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
#endif

}  // namespace st
