// BF16 matrix -> state tree: records, escape lists and the kernels' side tables, and the check of a tree against the
// matrix it was built from.
//
// Bound: HBM.  st_encode reads the matrix once (2 B per weight) and writes the records once (1.52 B); the escape passes
// touch only the records that have escapes.  4096 x 12288 on a B200: st_encode 57 us (177 MB, 3.1 TB/s), the two prefix
// sums 15 us, st_encode_lists 16 us, st_dec_check 36 us (nothing dense is written back).  TreeLinear.from_weight of that
// matrix with its check takes 0.25 ms; with the torch formulation (format._encode_chunk, still the CPU path: ~60 passes over
// 32- and 64-bit copies, then a sort of the escapes and a dense decode to compare) it took 3.7 ms.
#include "../../include/statetree_b200.h"
#include "st_common.cuh"
#include "st_host.h"

namespace {
using namespace st;

constexpr int ENC_WARPS = 8;

// Lane (q, seg) = (lane / 8, lane % 8) of a warp holds columns 8 seg .. 8 seg + 7 of the rows q, q + 4, q + 8, q + 12 of
// the record: rows r and r + 8, which share state bytes, meet in one lane.
struct EncLane {
  uint32_t v[4][4];      // [i] row q + 4 i as four BF16 pairs
  uint32_t top[4];       // the row's node: largest exponent of its 64 values
  uint32_t out[4];       // bit c: value 8 seg + c of row q + 4 i escapes (exponent more than 14 below the node)
};
__device__ __forceinline__ EncLane enc_load(const uint16_t* W, long long N, long long tile, int G, int lane) {
  EncLane e;
  const int q = lane >> 3, seg = lane & 7;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint4 x = *reinterpret_cast<const uint4*>(W + (tile * 16 + q + 4 * i) * N + (long long)G * 64 + seg * 8);
    e.v[i][0] = x.x; e.v[i][1] = x.y; e.v[i][2] = x.z; e.v[i][3] = x.w;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t top = 0;
#pragma unroll
    for (int p = 0; p < 4; ++p) top = max(top, max((e.v[i][p] >> 7) & 0xFFu, (e.v[i][p] >> 23) & 0xFFu));
#pragma unroll
    for (int o = 4; o; o >>= 1) top = max(top, __shfl_xor_sync(FULL, top, o));
    e.top[i] = top;
    uint32_t out = 0;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      if (top - ((e.v[i][p] >> 7) & 0xFFu) > 14u) out |= 1u << (2 * p);
      if (top - ((e.v[i][p] >> 23) & 0xFFu) > 14u) out |= 2u << (2 * p);
    }
    e.out[i] = out;
  }
  return e;
}

// One warp per record.  rowcnt uint8 [M, N/64]: escapes of each row's 64 values; reccnt int32 [records + 1]: escapes of
// each record behind a leading zero (its inclusive prefix sum is the offset table eo).
__global__ void __launch_bounds__(ENC_WARPS * 32) encode_kernel(const uint16_t* __restrict__ W, long long N, int NG,
                                                                long long nrec, uint8_t* __restrict__ tree,
                                                                uint8_t* __restrict__ rowcnt, int* __restrict__ reccnt) {
  __shared__ __align__(16) uint8_t s_rec[ENC_WARPS][REC];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = lane >> 3, seg = lane & 7;
  const long long r = (long long)blockIdx.x * ENC_WARPS + warp;
  if (r == 0 && lane == 0) reccnt[0] = 0;
  if (r >= nrec) return;
  const long long tile = r / NG;
  const int G = (int)(r % NG);
  const EncLane e = enc_load(W, N, tile, G, lane);
  uint8_t* const rec = s_rec[warp];
  const int s = seg >> 1, hi = seg & 1;                          // k-step of the columns, their half of it
  uint32_t cnt = 0;                                              // escapes of the lane's four rows, one byte each
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    cnt |= (uint32_t)__popc(e.out[i]) << (8 * i);
    const int row = q + 4 * i;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      // leaf = mantissa << 1 | sign of the pair partner; an escaped value's mantissa and sign are stored as zero
      const uint32_t v0 = (e.out[i] >> (2 * t)) & 1u ? 0u : e.v[i][t] & 0xFFFFu;
      const uint32_t v1 = (e.out[i] >> (2 * t + 1)) & 1u ? 0u : e.v[i][t] >> 16;
      const uint32_t l0 = (v0 & 0x7Fu) << 1 | v1 >> 15, l1 = (v1 & 0x7Fu) << 1 | v0 >> 15;
      *reinterpret_cast<uint16_t*>(rec + (s >> 1) * 512 + ((row & 7) * 4 + t) * 16 + ((s & 1) * 2 + (row >> 3)) * 4 + 2 * hi) =
          (uint16_t)(l0 | l1 << 8);
    }
    if (seg == 0) rec[1536 + 2 * (row & 7) + (row >> 3)] = (uint8_t)e.top[i];
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {                                  // rows q + 4 i (low nibbles) and q + 4 i + 8 (high)
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      uint32_t b = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = i + 2 * h;
        const uint32_t d0 = (e.out[k] >> (2 * t)) & 1u ? 15u : e.top[k] - ((e.v[k][t] >> 7) & 0xFFu);
        const uint32_t d1 = (e.out[k] >> (2 * t + 1)) & 1u ? 15u : e.top[k] - ((e.v[k][t] >> 23) & 0xFFu);
        b |= (d0 | d1 << 8) << (4 * h);
      }
      *reinterpret_cast<uint16_t*>(rec + 1024 + ((q + 4 * i) * 4 + t) * 16 + s * 4 + 2 * hi) = (uint16_t)b;
    }
  }
#pragma unroll
  for (int o = 4; o; o >>= 1) cnt += __shfl_xor_sync(FULL, cnt, o);          // per row (at most 64 each: no carry)
  if (seg == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) rowcnt[(tile * 16 + q + 4 * i) * NG + G] = (uint8_t)(cnt >> (8 * i));
  }
  int total = (int)((cnt & 0xFFu) + (cnt >> 8 & 0xFFu) + (cnt >> 16 & 0xFFu) + (cnt >> 24));
  total += __shfl_xor_sync(FULL, total, 8);
  total += __shfl_xor_sync(FULL, total, 16);
  if (lane == 0) reccnt[r + 1] = total;
  __syncwarp();
  uint4* const out = reinterpret_cast<uint4*>(tree + r * REC);
  for (int i = lane; i < REC / 16; i += 32) out[i] = reinterpret_cast<const uint4*>(rec)[i];
}

// One warp per GEMV unit (up to eight consecutive records of a tile): the unit's escape block and, for the records that
// have escapes, the list entries in record order (el) and the row-major lists of the format (rows, cols, bits).
// roff int32 [M, N/64] = inclusive prefix sum of rowcnt in row-major order.
__global__ void __launch_bounds__(ENC_WARPS * 32) encode_lists_kernel(
    const uint16_t* __restrict__ W, long long N, int NG, int CPT, long long units, const uint8_t* __restrict__ rowcnt,
    const int* __restrict__ roff, const int* __restrict__ eo, uint32_t* __restrict__ el, uint32_t* __restrict__ eb,
    int* __restrict__ rows, int* __restrict__ cols, uint16_t* __restrict__ bits) {
  __shared__ uint32_t s_eb[ENC_WARPS][16];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = lane >> 3, seg = lane & 7;
  const long long u = (long long)blockIdx.x * ENC_WARPS + warp;
  if (u >= units) return;
  const long long tile = u / CPT;
  const int c = (int)(u % CPT), G0 = c * 8, nrec = min(8, NG - G0);
  const int* const off = eo + tile * NG + G0;
  const int mine = off[min(lane, nrec)];
  const int first = __shfl_sync(FULL, mine, 0), end = __shfl_sync(FULL, mine, nrec);
  const int next = __shfl_down_sync(FULL, mine, 1);
  const unsigned mask = __ballot_sync(FULL, lane < nrec && next > mine);
  uint32_t* const blk = s_eb[warp];
  if (lane < 16) blk[lane] = lane == 0 ? (uint32_t)(end - first) | mask << 16 : (lane == 1 ? (uint32_t)first : 0u);
  __syncwarp();
  for (unsigned m = mask; m; m &= m - 1) {
    const int k = __ffs(m) - 1, G = G0 + k;
    const EncLane e = enc_load(W, N, tile, G, lane);
    int at = __shfl_sync(FULL, mine, k);                         // entries of this record so far
#pragma unroll
    for (int row = 0; row < 16; ++row) {                         // rows in order; lanes 8 (row % 4) .. + 7 hold row `row`
      const int i = row >> 2;
      const uint32_t o = q == (row & 3) ? e.out[i] : 0u;
      uint32_t n = (uint32_t)__popc(o);
      if (!__any_sync(FULL, n != 0u)) continue;
      uint32_t incl = n;                                         // prefix over the lanes = over the columns
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t p = __shfl_up_sync(FULL, incl, d);
        if (lane >= d) incl += p;
      }
      const long long rg = (tile * 16 + row) * NG + G;
      const int rbase = roff[rg] - (int)rowcnt[rg];
      uint32_t pos = incl - n;
      for (uint32_t b = o; b; b &= b - 1, ++pos) {
        const int cc = __ffs(b) - 1, col = seg * 8 + cc;
        uint32_t pair = 0;
#pragma unroll
        for (int p = 0; p < 4; ++p) pair = (cc >> 1) == p ? e.v[i][p] : pair;
        const uint32_t val = (cc & 1) ? pair >> 16 : pair & 0xFFFFu;
        const uint32_t entry = val << 16 | (uint32_t)(G & 7) << 10 | (uint32_t)row << 6 | (uint32_t)col;
        el[at + pos] = entry;
        const int in_unit = at + (int)pos - first;
        if (in_unit < 14) blk[2 + in_unit] = entry;
        rows[rbase + pos] = (int)(tile * 16 + row);
        cols[rbase + pos] = G * 64 + col;
        bits[rbase + pos] = (uint16_t)val;
      }
      at += (int)__shfl_sync(FULL, incl, 31);
    }
  }
  __syncwarp();
  if (lane < 16) eb[u * 16 + lane] = blk[lane];
}

// decodes every record and compares it with the matrix; *bad counts the warps that found a difference
__global__ void __launch_bounds__(256) dec_check_kernel(const uint8_t* __restrict__ tree, const int* __restrict__ eo,
                                                        const uint32_t* __restrict__ el, long long nrec, int NG, long long N,
                                                        const uint16_t* __restrict__ W, int* __restrict__ bad) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= nrec) return;
  uint32_t A[4][4];
  decode_frag(load_rec_global(tree + r * REC, lane), A);
  const uint16_t* const src = W + (r / NG) * 16 * N + (r % NG) * 64;
  uint32_t diff = 0;
  const int lo = __ldg(eo + r), hi = __ldg(eo + r + 1);
  for (int base = lo; base < hi; base += 32) {
    const int n = min(32, hi - base);
    const uint32_t ent = (lane < n) ? __ldg(el + base + lane) : 0u;
    for (int i = 0; i < n; ++i) patch_entry(A, __shfl_sync(FULL, ent, i), lane);
  }
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      diff |= A[s][q] ^ __ldg(reinterpret_cast<const uint32_t*>(src + (g + 8 * (q & 1)) * N + 16 * s + 8 * (q >> 1) + 2 * t));
  if (__any_sync(FULL, diff != 0u) && lane == 0) atomicAdd(bad, 1);
}

int shape_ok(const char* who, int64_t M, int64_t N) {
  ST_REQUIRE(M > 0 && N > 0 && M % 16 == 0 && N % 64 == 0, "%s: M %% 16 and N %% 64 must be 0 (got %lld x %lld)", who,
             (long long)M, (long long)N);
  ST_REQUIRE((M / 16) * (N / 64) < (1ll << 31), "%s: too many records", who);
  return 0;
}
}  // namespace

extern "C" int st_encode(const void* W, int64_t M, int64_t N, void* tree, uint8_t* rowcnt, int32_t* reccnt, void* stream) {
  if (int e = shape_ok("st_encode", M, N)) return e;
  ST_REQUIRE(W && tree && rowcnt && reccnt, "st_encode: null pointer");
  ST_REQUIRE(st::aligned16(W) && st::aligned16(tree), "st_encode: W and tree must be 16-byte aligned");
  const long long nrec = (M / 16) * (N / 64);
  encode_kernel<<<(unsigned)((nrec + ENC_WARPS - 1) / ENC_WARPS), ENC_WARPS * 32, 0, (cudaStream_t)stream>>>(
      (const uint16_t*)W, N, (int)(N / 64), nrec, (uint8_t*)tree, rowcnt, reccnt);
  ST_LAUNCH_CHECK("st_encode launch");
  return 0;
}

extern "C" int st_encode_lists(const void* W, int64_t M, int64_t N, const uint8_t* rowcnt, const int32_t* roff,
                               const int32_t* eo, uint32_t* el, uint32_t* eb, int32_t* rows, int32_t* cols, int16_t* bits,
                               void* stream) {
  if (int e = shape_ok("st_encode_lists", M, N)) return e;
  ST_REQUIRE(W && rowcnt && roff && eo && el && eb && rows && cols && bits, "st_encode_lists: null pointer");
  ST_REQUIRE(st::aligned16(W), "st_encode_lists: W must be 16-byte aligned");
  const int NG = (int)(N / 64), CPT = (NG + 7) / 8;
  const long long units = (M / 16) * CPT;
  encode_lists_kernel<<<(unsigned)((units + ENC_WARPS - 1) / ENC_WARPS), ENC_WARPS * 32, 0, (cudaStream_t)stream>>>(
      (const uint16_t*)W, N, NG, CPT, units, rowcnt, roff, eo, el, eb, rows, cols, (uint16_t*)bits);
  ST_LAUNCH_CHECK("st_encode_lists launch");
  return 0;
}

extern "C" int st_dec_check(const void* tree, const int32_t* eo, const uint32_t* el, int64_t M, int64_t N, const void* W,
                            int32_t* bad, void* stream) {
  if (int e = shape_ok("st_dec_check", M, N)) return e;
  ST_REQUIRE(tree && eo && el && W && bad, "st_dec_check: null pointer");
  ST_REQUIRE(st::aligned16(tree) && st::aligned16(W), "st_dec_check: tree and W must be 16-byte aligned");
  const long long nrec = (M / 16) * (N / 64);
  dec_check_kernel<<<(unsigned)((nrec + 7) / 8), 256, 0, (cudaStream_t)stream>>>(
      (const uint8_t*)tree, eo, el, nrec, (int)(N / 64), N, (const uint16_t*)W, bad);
  ST_LAUNCH_CHECK("st_dec_check launch");
  return 0;
}
