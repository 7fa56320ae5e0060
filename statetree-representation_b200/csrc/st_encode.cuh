// One warp turns a 16 x 64 BF16 block into a state-tree record: shared by the weight encoder and the KV append of whole
// pages.  The inverse of decode_frag: lane (g, t) holds the block as mma.m16n8k16 A fragments, which is exactly the part of
// the record it writes (16 + 16 leaf bytes, 16 state bytes), so nothing is exchanged but the row maxima, and the record
// leaves as three 16-byte stores per lane.  (Rows of eight values per lane, bytes placed through
// shared memory: 57 us for 4096 x 12288, most of it two-byte stores with four-way bank conflicts; this: 31 us.)
#pragma once
#include "st_common.cuh"

namespace st {

struct EncFrag {
  uint32_t A[4][4];      // [s][q]: q = 0: row g, columns 16 s + 2t, + 1; 1: row g + 8; 2, 3: the same rows, columns + 8
  uint32_t node[2];      // largest exponent of row g, of row g + 8
  uint32_t leaf[4][2], state[4][2];   // [s][row half]: bytes = columns 16 s + 2t, + 1, + 8, + 9
  uint32_t esc;          // bit 8 s + 4 r + j: value j (byte order above) of k-step s, row half r, escapes
};

constexpr int ENC_ROW = 144;                   // staged row: 128 bytes and a pad that keeps ldmatrix free of bank conflicts
constexpr int ENC_STAGE = 16 * ENC_ROW;        // bytes of shared memory a warp stages a block in

// A 16 x 64 block as mma A fragments.  src = first value of its first row, rows `stride` values apart; 4-byte aligned.
// Rows that are 16-byte aligned (ALIGNED, or found out here) come as four 16-byte loads per lane and go through `stage`
// (ENC_STAGE bytes, 16-byte aligned, the warp's own), where ldmatrix picks up the fragments; others as sixteen 4-byte loads of
// half a sector each.
__device__ __forceinline__ bool block_aligned(const uint16_t* src, long long stride) {
  return ((reinterpret_cast<uintptr_t>(src) | (uintptr_t)(stride * 2)) & 15u) == 0u;
}
// the two halves of the aligned form: the loads (a caller may have other look-ups in flight with them), then the fragments
__device__ __forceinline__ void request_block(uint4 (&v)[4], const uint16_t* src, long long stride, int lane) {
  const uint16_t* const p = src + (lane >> 3) * stride + (lane & 7) * 8;
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const uint4*>(p + 4 * i * stride);
}
__device__ __forceinline__ void place_block(uint32_t (&A)[4][4], const uint4 (&v)[4], uint8_t* stage, int lane) {
  uint8_t* const to = stage + (lane >> 3) * ENC_ROW + (lane & 7) * 16;
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(to + 4 * i * ENC_ROW) = v[i];
  __syncwarp();
  // lane l names row l % 16 of the two 8-column halves l / 16: matrices in the order of the fragment registers
  const uint32_t from = smem_addr(stage) + (uint32_t)((lane & 15) * ENC_ROW + (lane >> 4) * 16);
#pragma unroll
  for (int s = 0; s < 4; ++s) ldmatrix_x4_stored(from + 32 * s, A[s][0], A[s][1], A[s][2], A[s][3]);
  __syncwarp();                                                  // (the stage is reused)
}

template <bool ALIGNED>
__device__ __forceinline__ void load_block(uint32_t (&A)[4][4], const uint16_t* src, long long stride, uint8_t* stage, int lane) {
  if (ALIGNED || block_aligned(src, stride)) {
    uint4 v[4];
    request_block(v, src, stride, lane);
    place_block(A, v, stage, lane);
    return;
  }
  const uint16_t* const p0 = src + (lane >> 2) * stride + 2 * (lane & 3);
  const uint16_t* const p1 = p0 + 8 * stride;
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      A[s][q] = *reinterpret_cast<const uint32_t*>(((q & 1) ? p1 : p0) + 16 * s + 8 * (q >> 1));
}

// e.A -> the rest of the fragment
__device__ __forceinline__ void enc_finish(EncFrag& e) {
  e.esc = 0u;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    // the exponents of a pair stay in place (bits 7..14 of each half) for the maximum of two 16-bit lanes
    uint32_t m = 0u;
#pragma unroll
    for (int s = 0; s < 4; ++s) m = __vmaxu2(__vmaxu2(m, e.A[s][r] & 0x7F807F80u), e.A[s][2 + r] & 0x7F807F80u);
    m = __vmaxu2(m, __shfl_xor_sync(FULL, m, 1));
    m = __vmaxu2(m, __shfl_xor_sync(FULL, m, 2));
    const uint32_t node = max(m & 0xFFFFu, m >> 16) >> 7, node4 = node * 0x01010101u;
    e.node[r] = node;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      // rotating a pair left by one turns it into [leaf, exponent] bytes: leaf = mantissa << 1 | sign of the pair partner
      const uint32_t a = __funnelshift_l(e.A[s][r], e.A[s][r], 1), b = __funnelshift_l(e.A[s][2 + r], e.A[s][2 + r], 1);
      uint32_t leaf = __byte_perm(a, b, 0x6420), st = node4 - __byte_perm(a, b, 0x7531);
      if (((st & 0xF0F0F0F0u) | (((st & 0x0F0F0F0Fu) + 0x01010101u) & 0x10101010u)) != 0u) {
        // escapes (distance over 14): mantissa and sign are stored as zero, the state as 15
        const uint32_t out = __vcmpgtu4(st, 0x0E0E0E0Eu);
        leaf &= ~(out & 0xFEFEFEFEu) & ~(__byte_perm(out, 0u, 0x2301) & 0x01010101u);
        st = (st & ~out) | (out & 0x0F0F0F0Fu);
        e.esc |= ((out & 1u) | (out >> 7 & 2u) | (out >> 14 & 4u) | (out >> 21 & 8u)) << (8 * s + 4 * r);
      }
      e.leaf[s][r] = leaf;
      e.state[s][r] = st;
    }
  }
}

template <bool ALIGNED>
__device__ __forceinline__ EncFrag enc_block(const uint16_t* src, long long stride, uint8_t* stage, int lane) {
  EncFrag e;
  load_block<ALIGNED>(e.A, src, stride, stage, lane);
  enc_finish(e);
  return e;
}

// the record's 1552 bytes; rec 16-byte aligned (global memory)
__device__ __forceinline__ void enc_write(uint8_t* const rec, const EncFrag& e, int lane) {
  uint4* const out = reinterpret_cast<uint4*>(rec) + lane;
  out[0] = make_uint4(e.leaf[0][0], e.leaf[0][1], e.leaf[1][0], e.leaf[1][1]);
  out[32] = make_uint4(e.leaf[2][0], e.leaf[2][1], e.leaf[3][0], e.leaf[3][1]);
  out[64] = make_uint4(e.state[0][0] | e.state[0][1] << 4, e.state[1][0] | e.state[1][1] << 4,
                       e.state[2][0] | e.state[2][1] << 4, e.state[3][0] | e.state[3][1] << 4);
  if ((lane & 3) == 0) *reinterpret_cast<uint16_t*>(rec + 1536 + 2 * (lane >> 2)) = (uint16_t)(e.node[0] | e.node[1] << 8);
}

// escapes of rows g and g + 8 (the same in the four lanes of a row)
__device__ __forceinline__ int2 enc_row_counts(const EncFrag& e) {
  uint32_t n = (uint32_t)__popc(e.esc & 0x0F0F0F0Fu) | (uint32_t)__popc(e.esc & 0xF0F0F0F0u) << 16;
  n += __shfl_xor_sync(FULL, n, 1);
  n += __shfl_xor_sync(FULL, n, 2);
  return make_int2((int)(n & 0xFFFFu), (int)(n >> 16));
}

// Visits the record's escapes: f(escapes in the rows before, position inside the row, row, column, bits), called by the
// lane that holds the value; positions follow (row, column) order.  Returns their number.  For records that have some.
template <typename F>
__device__ __forceinline__ int enc_escapes(const EncFrag& e, int lane, F f) {
  const int g = lane >> 2, t = lane & 3;
  const int2 cnt = enc_row_counts(e);
  int before0 = cnt.x, before1 = cnt.y;                          // inclusive over the rows (lanes 4 apart), then exclusive
#pragma unroll
  for (int d = 4; d < 32; d <<= 1) {
    const int a = __shfl_up_sync(FULL, before0, d), b = __shfl_up_sync(FULL, before1, d);
    if (lane >= d) { before0 += a; before1 += b; }
  }
  const int total0 = __shfl_sync(FULL, before0, 31), total = total0 + __shfl_sync(FULL, before1, 31);
  before0 -= cnt.x;
  before1 += total0 - cnt.y;
#pragma unroll 1
  for (int r = 0; r < 2; ++r) {
    // the row's escapes as one bit per column, lo = columns 0..31, hi = 32..63
    uint32_t lo = 0u, hi = 0u;
    const uint32_t mine = e.esc >> (4 * r);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const uint32_t b = mine >> (8 * s) & 0xFu;
      const uint32_t m = ((b & 3u) | (b >> 2) << 8) << (2 * t);
      if (s < 2) lo |= m << (16 * s);
      else hi |= m << (16 * (s - 2));
    }
    lo |= __shfl_xor_sync(FULL, lo, 1); hi |= __shfl_xor_sync(FULL, hi, 1);
    lo |= __shfl_xor_sync(FULL, lo, 2); hi |= __shfl_xor_sync(FULL, hi, 2);
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (mine >> (8 * s + j) & 1u) {
          const int col = 16 * s + 8 * (j >> 1) + 2 * t + (j & 1);
          const uint32_t below = (1u << (col & 31)) - 1u;
          const int in_row = col < 32 ? __popc(lo & below) : __popc(lo) + __popc(hi & below);
          const uint32_t pair = r ? e.A[s][2 * (j >> 1) + 1] : e.A[s][2 * (j >> 1)];
          f(r ? before1 : before0, in_row, g + 8 * r, col, (j & 1) ? pair >> 16 : pair & 0xFFFFu);
        }
  }
  return total;
}

}  // namespace st
