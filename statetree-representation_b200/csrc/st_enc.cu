// BF16 matrix -> state tree: records, escape lists and the kernels' side tables, and the check of a tree against the
// matrix it was built from.
//
// Bound: HBM.  st_encode reads the matrix once (2 B per weight) and writes the records once (1.52 B); the escape passes
// touch only the records that have escapes.  4096 x 12288 on a B200, each launch by itself: st_encode 31 us (177 MB, 5.7 TB/s; 37
// with 4-byte loads), st_encode_offsets 8.5 us (two torch.cumsum with their type conversion 25), st_encode_lists 28 us,
// st_dec_check 28 us (33 with 4-byte loads; nothing dense is written back), st_lists_check 6 us (the stored lists and the escape
// blocks).  TreeLinear.from_weight with its checks and one decode of that matrix take 0.18 ms; with the torch formulation
// (format._encode_chunk, still the CPU path: ~60 passes over 32- and 64-bit copies, then a sort of the escapes
// and a dense decode to compare) 3.7 ms.
#include "../../include/statetree_b200.h"
#include "st_encode.cuh"
#include "st_host.h"

namespace {
using namespace st;

constexpr int ENC_WARPS = 8;

// One warp per record.  rowcnt uint8 [M, N/64]: escapes of each row's 64 values; reccnt int32 [records + 1]: escapes of
// each record behind a leading zero (its inclusive prefix sum is the offset table eo).
__global__ void __launch_bounds__(ENC_WARPS * 32) encode_kernel(const uint16_t* __restrict__ W, long long N, int NG,
                                                                long long nrec, uint8_t* __restrict__ tree,
                                                                uint8_t* __restrict__ rowcnt, int* __restrict__ reccnt) {
  __shared__ __align__(16) uint8_t s_stage[ENC_WARPS][ENC_STAGE];
  const int lane = threadIdx.x & 31;
  const long long r = (long long)blockIdx.x * ENC_WARPS + (threadIdx.x >> 5);
  if (r == 0 && lane == 0) reccnt[0] = 0;
  if (r >= nrec) return;
  const long long tile = r / NG;
  const int G = (int)(r % NG);
  const EncFrag e = enc_block<true>(W + tile * 16 * N + (long long)G * 64, N, s_stage[threadIdx.x >> 5], lane);
  enc_write(tree + r * REC, e, lane);
  int2 cnt = make_int2(0, 0);
  int total = 0;
  if (__any_sync(FULL, e.esc != 0u)) {
    cnt = enc_row_counts(e);
    total = cnt.x + cnt.y;                                       // per row pair; over the eight of them (lanes 4 apart)
    total += __shfl_xor_sync(FULL, total, 4);
    total += __shfl_xor_sync(FULL, total, 8);
    total += __shfl_xor_sync(FULL, total, 16);
  }
  if ((lane & 3) == 0) {
    rowcnt[(tile * 16 + (lane >> 2)) * NG + G] = (uint8_t)cnt.x;
    rowcnt[(tile * 16 + 8 + (lane >> 2)) * NG + G] = (uint8_t)cnt.y;
  }
  if (lane == 0) reccnt[r + 1] = total;
}

// One warp per GEMV unit (up to eight consecutive records of a tile): the unit's escape block and, for the records that
// have escapes, the list entries in record order (el) and the row-major lists of the format (rows, cols, bits).
// roff int32 [M, N/64] = inclusive prefix sum of rowcnt in row-major order.
__global__ void __launch_bounds__(ENC_WARPS * 32, 4) encode_lists_kernel(
    const uint16_t* __restrict__ W, long long N, int NG, int CPT, long long units, const uint8_t* __restrict__ rowcnt,
    const int* __restrict__ roff, const int* __restrict__ eo, uint32_t* __restrict__ el, uint32_t* __restrict__ eb,
    int* __restrict__ rows, int* __restrict__ cols, uint16_t* __restrict__ bits) {
  __shared__ uint32_t s_eb[ENC_WARPS][16];
  __shared__ __align__(16) uint8_t s_stage[ENC_WARPS][ENC_STAGE];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
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
    const EncFrag e = enc_block<true>(W + tile * 16 * N + (long long)G * 64, N, s_stage[warp], lane);
    const int at = __shfl_sync(FULL, mine, k);                   // first entry of this record
    enc_escapes(e, lane, [&](int before, int in_row, int row, int col, uint32_t val) {
      const uint32_t entry = val << 16 | (uint32_t)(G & 7) << 10 | (uint32_t)row << 6 | (uint32_t)col;
      const int pos = at + before + in_row, in_unit = pos - first;
      el[pos] = entry;
      if (in_unit < 14) blk[2 + in_unit] = entry;
      const long long rg = (tile * 16 + row) * NG + G;
      const int rpos = roff[rg] - (int)rowcnt[rg] + in_row;
      rows[rpos] = (int)(tile * 16 + row);
      cols[rpos] = G * 64 + col;
      bits[rpos] = (uint16_t)val;
    });
  }
  __syncwarp();
  if (lane < 16) eb[u * 16 + lane] = blk[lane];
}

// Inclusive prefix sums of the two count arrays (rowcnt: n8 bytes -> roff; reccnt: n32 ints -> eo), in two launches without a CTA
// that waits for another: the sums of chunks of SCAN_CHUNK values, then every CTA adds up the sums before its chunk and scans it.
// The chunks of rowcnt come first, those of reccnt after them.
constexpr int SCAN_CHUNK = 4096;                 // 16 values a thread
struct ScanArgs {
  const uint8_t* c8; const int* c32; long long n8, n32; int chunks8;
  int* sums; int* out8; int* out32;
};
// this thread's sixteen values of the CTA's chunk (zeros behind the array's end; n8 is a multiple of 16, as M is)
__device__ __forceinline__ void scan_values(const ScanArgs& a, int (&v)[16], long long& at, bool& bytes) {
  bytes = (int)blockIdx.x < a.chunks8;
  at = (long long)(bytes ? blockIdx.x : blockIdx.x - a.chunks8) * SCAN_CHUNK + threadIdx.x * 16;
  if (bytes) {                                   // (rowcnt is 16-byte aligned, chunks are multiples of 16)
    const uint4 w = at < a.n8 ? *reinterpret_cast<const uint4*>(a.c8 + at) : make_uint4(0u, 0u, 0u, 0u);
    const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = (int)(ws[i >> 2] >> (8 * (i & 3)) & 0xFFu);
    return;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = at + i < a.n32 ? a.c32[at + i] : 0;
}
__global__ void __launch_bounds__(256) scan_sums_kernel(const ScanArgs a) {
  __shared__ int s_sum[8];
  int v[16], sum = 0;
  long long at;
  bool bytes;
  scan_values(a, v, at, bytes);
#pragma unroll
  for (int i = 0; i < 16; ++i) sum += v[i];
  sum = __reduce_add_sync(FULL, sum);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) sum += s_sum[w];
    a.sums[blockIdx.x] = sum;
  }
}
__global__ void __launch_bounds__(256) scan_kernel(const ScanArgs a) {
  __shared__ int s_before[8], s_warp[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int v[16];
  long long at;
  bool bytes;
  scan_values(a, v, at, bytes);
  int before = 0;                                // the chunks of the same array before this one
  for (int b = (bytes ? 0 : a.chunks8) + threadIdx.x; b < (int)blockIdx.x; b += 256) before += a.sums[b];
  before = __reduce_add_sync(FULL, before);
#pragma unroll
  for (int i = 1; i < 16; ++i) v[i] += v[i - 1];
  int upto = v[15];                              // inclusive over the warp's threads
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(FULL, upto, o);
    if (lane >= o) upto += n;
  }
  if (lane == 31) s_warp[warp] = upto;
  if (lane == 0) s_before[warp] = before;
  __syncthreads();
  int add = upto - v[15];
#pragma unroll
  for (int w = 0; w < 8; ++w) add += s_before[w] + (w < warp ? s_warp[w] : 0);
  int* const out = (bytes ? a.out8 : a.out32) + at;
  const long long left = (bytes ? a.n8 : a.n32) - at;
#pragma unroll
  for (int i = 0; i < 16; i += 4) {
    if (i + 4 <= left) {
      *reinterpret_cast<int4*>(out + i) = make_int4(v[i] + add, v[i + 1] + add, v[i + 2] + add, v[i + 3] + add);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i + k < left) out[i + k] = v[i + k] + add;
    }
  }
}

// decodes every record and compares it with the matrix; *bad counts the warps that found a difference
__global__ void __launch_bounds__(256) dec_check_kernel(const uint8_t* __restrict__ tree, const int* __restrict__ eo,
                                                        const uint32_t* __restrict__ el, long long nrec, int NG, long long N,
                                                        const uint16_t* __restrict__ W, int* __restrict__ bad) {
  __shared__ __align__(16) uint8_t s_stage[8][ENC_STAGE];
  const int lane = threadIdx.x & 31;
  const long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= nrec) return;
  uint32_t A[4][4], want[4][4];
  const RecRegs rec = load_rec_global(tree + r * REC, lane);
  load_block<true>(want, W + (r / NG) * 16 * N + (r % NG) * 64, N, s_stage[threadIdx.x >> 5], lane);
  decode_frag(rec, A);
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
    for (int q = 0; q < 4; ++q) diff |= A[s][q] ^ want[s][q];
  if (__any_sync(FULL, diff != 0u) && lane == 0) atomicAdd(bad, 1);
}

// Are the lists a checkpoint stores (rows, cols, bits: n entries) the matrix's escapes, and are eo / el / eb the tables those
// lists give?  dec_check_kernel has shown that the records and the entries that eo and el name decode to W; here every stored
// entry must lie inside the matrix, follow its predecessor in (row, col) order, hold the matrix's bits and be found in its own
// record's part of el.  eo partitions n entries, so stored and listed entries are then the same set, and a tree read back
// from the stored lists decodes to W too.  eb: every word as the unit's part of eo and el gives it.
// A thread takes one stored entry (a binary search over its record's few entries) and one word of eb.  Nothing is trusted:
// offsets and positions are checked before they are followed.  4096 x 12288 with 8000 escapes: from_weight 236 -> 244 us.
__global__ void __launch_bounds__(256) lists_check_kernel(const int* __restrict__ rows, const int* __restrict__ cols,
                                                          const uint16_t* __restrict__ bits, int n, const int* __restrict__ eo,
                                                          const uint32_t* __restrict__ el, const uint32_t* __restrict__ eb,
                                                          long long M, long long N, int NG, int CPT, long long units,
                                                          const uint16_t* __restrict__ W, int* __restrict__ bad) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  bool ok = true;
  if (i < n) {
    const int r = rows[i], c = cols[i];
    ok = r >= 0 && r < M && c >= 0 && c < N;
    if (ok && i > 0) ok = rows[i - 1] < r || (rows[i - 1] == r && cols[i - 1] < c);
    if (ok) {
      const long long rec = (long long)(r >> 4) * NG + (c >> 6);
      const uint32_t want = (uint32_t)bits[i] << 16 | (uint32_t)((c >> 6) & 7) << 10 | (uint32_t)(r & 15) << 6 | (uint32_t)(c & 63);
      int lo = eo[rec], hi = eo[rec + 1];
      ok = bits[i] == W[(long long)r * N + c] && lo >= 0 && lo < hi && hi <= n;
      if (ok) {
        while (hi - lo > 1) {                                    // entries of a record are in (row, col) order: bits 0..9
          const int mid = (lo + hi) >> 1;
          if ((el[mid] & 0x3FFu) <= (want & 0x3FFu)) lo = mid;
          else hi = mid;
        }
        ok = el[lo] == want;
      }
    }
  }
  if (i < units * 16) {
    const long long u = i >> 4, tile = u / CPT;
    const int word = (int)(i & 15), G0 = (int)(u % CPT) * 8, nrec = min(8, NG - G0);
    const int* const off = eo + tile * NG + G0;
    const int first = off[0], end = off[nrec];
    bool sound = first >= 0 && first <= end && end <= n && (u > 0 || first == 0) && (u + 1 < units || end == n);
    uint32_t want = 0u;
    if (word == 0) {
      want = (uint32_t)(end - first);
      for (int k = 0; k < nrec; ++k) {
        sound = sound && off[k] <= off[k + 1];
        if (off[k] < off[k + 1]) want |= 1u << (16 + k);
      }
    } else if (word == 1) {
      want = (uint32_t)first;
    } else if (sound && word - 2 < end - first) {
      want = el[first + word - 2];
    }
    ok = ok && sound && eb[i] == want;
  }
  if (__any_sync(FULL, !ok) && (threadIdx.x & 31) == 0) atomicAdd(bad, 1);
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

extern "C" int st_lists_check(const int32_t* rows, const int32_t* cols, const int16_t* bits, int64_t n, const int32_t* eo,
                              const uint32_t* el, const uint32_t* eb, int64_t M, int64_t N, const void* W, int32_t* bad,
                              void* stream) {
  if (int e = shape_ok("st_lists_check", M, N)) return e;
  ST_REQUIRE(n >= 0 && n < (1ll << 31), "st_lists_check: number of entries");
  ST_REQUIRE(eo && el && eb && W && bad && (n == 0 || (rows && cols && bits)), "st_lists_check: null pointer");
  const int NG = (int)(N / 64), CPT = (NG + 7) / 8;
  const long long units = (M / 16) * CPT, threads = units * 16 > n ? units * 16 : n;
  lists_check_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      rows, cols, (const uint16_t*)bits, (int)n, eo, el, eb, M, N, NG, CPT, units, (const uint16_t*)W, bad);
  ST_LAUNCH_CHECK("st_lists_check launch");
  return 0;
}

extern "C" int64_t st_encode_offsets_workspace_bytes(int64_t M, int64_t N) {
  if (M <= 0 || N <= 0 || M % 16 || N % 64) return -1;
  const long long n8 = M * (N / 64), n32 = (M / 16) * (N / 64) + 1;
  return ((n8 + SCAN_CHUNK - 1) / SCAN_CHUNK + (n32 + SCAN_CHUNK - 1) / SCAN_CHUNK) * 4;
}

extern "C" int st_encode_offsets(const uint8_t* rowcnt, const int32_t* reccnt, int64_t M, int64_t N, int32_t* roff, int32_t* eo,
                                 void* ws, int64_t ws_bytes, void* stream) {
  if (int e = shape_ok("st_encode_offsets", M, N)) return e;
  ST_REQUIRE(rowcnt && reccnt && roff && eo && ws, "st_encode_offsets: null pointer");
  ST_REQUIRE(st::aligned16(rowcnt) && st::aligned16(roff) && st::aligned16(eo), "st_encode_offsets: 16-byte alignment");
  const int64_t need = st_encode_offsets_workspace_bytes(M, N);
  ST_REQUIRE(ws_bytes >= need, "st_encode_offsets: workspace of %lld bytes needed", (long long)need);
  ScanArgs a;
  a.c8 = rowcnt; a.c32 = reccnt; a.n8 = M * (N / 64); a.n32 = (M / 16) * (N / 64) + 1;
  a.chunks8 = (int)((a.n8 + SCAN_CHUNK - 1) / SCAN_CHUNK);
  a.sums = (int*)ws; a.out8 = roff; a.out32 = eo;
  const unsigned grid = (unsigned)(need / 4);
  scan_sums_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(a);
  ST_LAUNCH_CHECK("st_encode_offsets launch");
  scan_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(a);
  ST_LAUNCH_CHECK("st_encode_offsets launch");
  return 0;
}
