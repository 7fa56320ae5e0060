// Fused tree-decode + GEMM for more than 128 tokens on CTA pairs (tcgen05 cta_group::2) of sm_100a.
//   Y[B, M] = X[B, N] W[M, N]^T,  W as state-tree records, fp32 accumulation in tensor memory, BF16 output.
//
// Two CTAs (two SMs) multiply 256 rows of W by one tile of NT <= 384 tokens: each decodes the records of its own 128 rows into
// its own tensor memory, each loads HALF of the activation rows into its shared memory, and one tcgen05.mma (256 x NT x 16)
// reads both halves.  Warp roles of a CTA:
//   16 decode warps, in two groups of eight (group g takes every second pair of k-tiles): records -> mma fragment registers ->
//              escapes patched -> one tcgen05.st.16x128b.x8 per record, as in st_gemm.cu; they also run the epilogue
//   record producer: one 3-D tiled TMA load per pair of k-tiles (sixteen 1552-byte records) into a ring
//   activation producer: tiled TMA loads of this CTA's half of the tile's rows, 128-byte swizzle; the bytes of both CTAs are
//              counted on the barrier of the pair's first CTA
//   MMA issuer (first CTA only): one elected lane issues the MMAs; tcgen05.commit frees a slot in both CTAs
//
// The clusters are persistent: cluster c takes the (row pair, token tile) units c, c + C, ... and its rings run on across them.
// The decode warps fill the first weight tiles of the next unit BEFORE they empty the accumulator of the last one, so between two
// units the tensor cores wait for the accumulator to be read, not for a pipeline to start: a unit costs 0.9 us beyond its pairs of
// k-tiles (1.3 and 1.37 us each at 352 and 384 tokens; one to three units of 8 to 32 pairs on every cluster).
// A k range may be split over 2 to 4 pairs of one cluster (KS): they park their fp32 tiles in shared memory and add them in rank
// order through distributed shared memory; such a cluster has one unit.
//
// Why pairs: with one CTA per tile (what this kernel replaced) the shared-memory port was the limit beyond ~200 tokens: records
// in and out and the whole activation tile in and out, 3.1 KB + 32 B x tokens per record at 128 B per cycle: 800 cycles per
// k-tile at 304 tokens against 608 of MMAs.  A pair halves the activation part.
// Measured, us per launch in a graph, one CTA per tile / pairs (weights from HBM): 24576 x 4096 at 384, 512, 1024, 1536 rows 91 / 68,
// 104 / 82, 191 / 143, 259 / 211; 6144 x 4096 at 1024 52 / 38; 4096 x 12288 at 700, 1024, 1536 87 / 56, 92 / 79, 126 / 107; 2048 x
// 2048 at 300 13.5 / 10.1.  What bounds it now: from some 250 tokens per tile the MMAs (1.41 PFLOP/s at 1024 rows; under a power
// cap that holds for long the clock, as for any GEMM), below the decode, ~900 cycles per pair of k-tiles of integer work.
#include <stdlib.h>
#include <string.h>

#include "st_tc.cuh"

namespace {
using namespace st;

constexpr int DG = 2;                                            // decode groups
constexpr int NDW = DG * NDEC;                                   // decode warps
constexpr int THREADS = (NDW + 3) * 32;
constexpr int W_RAW = NDW, W_X = NDW + 1, W_MMA = NDW + 2;       // role warps
constexpr int TMEM_COLS = 512;
constexpr int NT_MAX = 384;                                      // 384 accumulator columns + 4 weight tiles of 32 fill TMEM
constexpr int SMEM_BYTES = 216 * 1024;

constexpr int BATCH = 2;                                         // chunks a warp holds at once (three spill)
constexpr int CSTEP = (NDW / 4) * 16;                            // columns between two chunks of 16 of a decode warp's share

// One warp's share of a unit whose whole k range this CTA has: chunks c0, c0 + CSTEP, ... of 16 columns.  Two chunks at a time
// are read and rounded (two tokens of a row per register) before any is stored, the last of them after the accumulator has been
// handed back.  out: this warp's 32 rows of the unit's first token; rows are M values apart.  Lanes pair up (even: column c, odd:
// column c + 1, two rows each) so that a store instruction writes 4 bytes per lane, 64 bytes per column.
__device__ __forceinline__ void store_unit(uint32_t acc, int c0, int NT, int ncol, uint16_t* out, float* outf, long long M,
                                        uint32_t accfree) {
  const int lane = threadIdx.x & 31;
  if (outf) {
#pragma unroll 1
    for (int c = c0; c < NT; c += CSTEP) {
      uint32_t v[16];
      tmem_ld16(acc + (uint32_t)c, v);
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (c + j < ncol) outf[(size_t)(c + j) * M + lane] = __uint_as_float(v[j]);
    }
  }
#pragma unroll 1
  for (; c0 < NT; c0 += BATCH * CSTEP) {
    uint32_t packed[BATCH][8];
#pragma unroll
    for (int h = 0; h < BATCH; ++h) {
      const int c = c0 + h * CSTEP;
      if (c < NT) {
        uint32_t v[16];
        tmem_ld16(acc + (uint32_t)c, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) packed[h][j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
      }
    }
    if (c0 + BATCH * CSTEP >= NT) {                                  // this warp has read its share: the next unit may accumulate
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(accfree);
    }
    uint16_t* p = out + (size_t)(c0 + (lane & 1)) * M + (lane & ~1);
#pragma unroll
    for (int h = 0; h < BATCH; ++h) {
      const int left = ncol - (c0 + h * CSTEP) - (lane & 1);     // this lane's columns 0, 2, .. of the chunk that exist
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t got = __shfl_xor_sync(FULL, packed[h][j], 1);
        const uint32_t two = (lane & 1) ? __byte_perm(got, packed[h][j], 0x7632) : __byte_perm(packed[h][j], got, 0x5410);
        if (2 * j < left) *reinterpret_cast<uint32_t*>(p + (size_t)(2 * j) * M) = two;
      }
      p += (size_t)CSTEP * M;
    }
  }
}

// *Slot parity.*  An mbarrier tells only its current phase from the previous one, so a waiter must never be two phases away.
// The two decode groups alternate pairs of k-tiles, counted over all units of the cluster, so every A slot and record slot
// belongs to one group (whose own program order guarantees that): both counts are even.
__global__ void __launch_bounds__(THREADS, 1)
pair_kernel(const GemmArgs a, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ WMaps wmaps) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);   // (stays a shared-memory pointer to the compiler)
  const int NT = a.NT, SA = a.astages, SX = a.xstages, R = a.rstages;
  const int nbox = a.n1 < NT ? 2 : 1;            // MMAs per k-step = activation boxes per k-tile
  const int XT = nbox * a.box * 128;             // bytes of this CTA's share of an activation tile
  uint8_t* rawring = smem + (size_t)SX * XT;                         // [R] record slots
  uint64_t* aready = reinterpret_cast<uint64_t*>(smem + a.bar_off);  // [SA] both CTAs' weight tiles are in tensor memory (first CTA)
  uint64_t* aempty = aready + SA;                                    // [SA] the MMAs that read the slot have completed
  uint64_t* xfull = aempty + SA;                                     // [SX] both halves of the activation tile landed (first CTA)
  uint64_t* xempty = xfull + SX;                                     // [SX] the MMAs that read it have completed
  uint64_t* rfull = xempty + SX;                                     // [R] records landed
  uint64_t* rempty = rfull + R;                                      // [R] records copied to registers
  uint64_t* accfull = rempty + R;                                    // the unit's MMAs have completed
  uint64_t* accfree = accfull + 1;                                   // both CTAs have read the accumulator (first CTA)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accfree + 1);

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(FULL, tid >> 5, 0);   // (a warp-uniform value to the compiler)
  const int CS = 2 * a.KS, rank = blockIdx.x % CS, cluster = blockIdx.x / CS;
  const int ks = rank >> 1, half = rank & 1;
  const uint32_t first_rank = (uint32_t)(rank & ~1);             // the pair's first CTA: its barriers serve both
  // units of this cluster; the token tiles of a row pair run next to each other (its records come from HBM once)
  const int unit0 = a.tile0 + cluster, nunits = unit0 < a.tile1 ? (a.tile1 - unit0 + a.nclusters - 1) / a.nclusters : 0;
  // whole pairs of k-tiles; an odd last tile is paired with one beyond the matrix, which both tensor maps fill with zeros
  const int pairs = (a.NG + PAIR - 1) / PAIR;
  const int p0 = (int)((long long)pairs * ks / a.KS), np = (int)((long long)pairs * (ks + 1) / a.KS) - p0;
  const int k0 = p0 * PAIR;
  const int total = nunits * np;                                 // pairs of k-tiles over all units

  // row block of this CTA in unit u, the list member it belongs to and its row block inside that member
  struct Rows { int rb, m, lrb; };
  auto rows_of = [&](int unit) {
    Rows r;
    r.rb = unit / a.TT * 2 + half;
    r.m = 0;
    r.lrb = r.rb;
    if (a.nlist > 0) {
      while (r.m + 1 < a.nlist && r.rb >= a.rbend[r.m]) ++r.m;
      r.lrb = r.rb - (r.m ? a.rbend[r.m - 1] : 0);
    }
    return r;
  };
  // records of pair i (of the unit's np) through a 3-D view of the tree [row tile][column group][194 x u64]; a row block beyond
  // an odd count is beyond the map and reads zeros
  int r_unit = -1, r_lrb = 0;
  const CUtensorMap* r_map = nullptr;
  auto load_records = [&](int unit, int i, int r) {
    if (unit != r_unit) {
      const Rows rw = rows_of(unit);
      r_unit = unit; r_lrb = rw.lrb; r_map = &wmaps.m[rw.m];
    }
    if (elect_one()) {
      mbar_expect_tx(rfull + r, (uint32_t)RAW_SLOT);
      tma_load_3d(rawring + (size_t)r * RAW_SLOT, r_map, 0, k0 + PAIR * i, r_lrb * 8, rfull + r);
    }
    __syncwarp();
  };

  // Set-up, spread over the role warps.  The record producer prepares the barriers (a lane each) and sends the first ring
  // fill off before the cluster synchronises: weights depend on no earlier kernel.
  int r_tile = unit0, r_i = 0;                                   // the record producer's next pair
  auto r_next = [&] { if (++r_i == np) { r_i = 0; r_tile += a.nclusters; } };
  if (warp == W_RAW) {
    for (int b = lane; b < 2 * (SA + SX + R) + 2; b += 32) {
      int count = 1;                                             // aempty, xfull, xempty, rfull, accfull
      if (b < SA) count = 2 * NDEC;                              // aready: the group's warps of both CTAs
      else if (b >= 2 * (SA + SX) + R && b < 2 * (SA + SX + R)) count = NDEC;     // rempty: the group's warps
      else if (b == 2 * (SA + SX + R) + 1) count = 2 * NDW;      // accfree: every decode warp of both CTAs
      mbar_init(aready + b, count);
    }
    fence_barrier_init();
    __syncwarp();
    for (int j = 0; j < min(total, R); ++j) { load_records(r_tile, r_i, j); r_next(); }
  } else if (warp == W_X) {
    if (elect_one()) asm volatile("prefetch.tensormap [%0];" :: "l"(&xmap) : "memory");
  } else if (warp == W_MMA) {
    tmem_alloc<2>(tmem_slot, (uint32_t)TMEM_COLS);
    tmem_relinquish<2>();
  }
  tc_fence_before();
  cluster_sync_all();                                            // barriers of both CTAs exist
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tmem_a = tmem + (uint32_t)NT;                   // the weight tiles' columns follow the accumulator (NT % 32 == 0)
  pdl_launch_dependents();

  if (warp == W_RAW) {
    // ---------------------------------------------------------------- record producer, behind the first ring fill
    for (int j = R, r = 0, k = 1; j < total; ++j, r = (r + 1 == R ? 0 : r + 1), k += (r == 0)) {
      if (!mbar_wait_look(rempty + r, (uint32_t)(k - 1) & 1u)) { if (lane == 0) atomicExch(a.status, ERR_WAIT_EMPTY); break; }
      load_records(r_tile, r_i, r);
      r_next();
    }
  } else if (warp == W_X) {
    // ---------------------------------------------------------------- activation producer.  The activations are the only
    // input an earlier kernel of the stream may still be writing: this thread is the one that waits for it, and everything
    // that touches the output is downstream of the first activation tile.
    pdl_wait();
    int s = 0, k = 0;
    bool ok = true;
    for (int n = 0; ok && n < nunits; ++n) {
      const int tok = (unit0 + n * a.nclusters) % a.TT * NT;
      const int y0 = tok + half * (a.n1 >> 1), y1 = tok + a.n1 + half * ((NT - a.n1) >> 1);
      for (int i = 0; i < np * PAIR; ++i) {
        if (k > 0 && !mbar_wait_look(xempty + s, (uint32_t)(k - 1) & 1u)) {
          if (lane == 0) atomicExch(a.status, ERR_WAIT_EMPTY);
          ok = false;
          break;
        }
        if (elect_one()) {
          const uint32_t bar = map_to_cta(smem_addr(xfull + s), first_rank);
          if (half == 0) mbar_expect_tx(xfull + s, (uint32_t)(2 * XT));
          uint8_t* dst = smem + (size_t)s * XT;
          tma_load_2d_pair(dst, &xmap, (k0 + i) * 64, y0, bar);
          if (nbox == 2) tma_load_2d_pair(dst + a.box * 128, &xmap, (k0 + i) * 64, y1, bar);
        }
        __syncwarp();
        if (++s == SX) { s = 0; ++k; }
      }
    }
  } else if (warp == W_MMA) {
    if (half == 0) {
      // -------------------------------------------------------------- MMA issuer.  The whole warp waits; one elected lane issues
      const int n2 = NT - a.n1;
      const uint32_t idesc = mma_idesc(256, a.n1), idesc2 = mma_idesc(256, n2 ? n2 : 32);
      const uint16_t both = (uint16_t)(3u << first_rank);
      int xs = 0, s = 0;
      uint32_t xph = 0u, sph = 0u;
      bool ok = true;
      for (int n = 0; ok && n < nunits; ++n) {
        if (n > 0) ok = mbar_wait_look(accfree, (uint32_t)(n - 1) & 1u);
        for (int i = 0; ok && i < np; ++i) {
          ok = mbar_wait_look(aready + s, sph);
          tc_fence_after();
#pragma unroll
          for (int h = 0; h < PAIR; ++h) {
            ok = ok && mbar_wait_look(xfull + xs, xph);
            if (!ok) break;
            tc_fence_after();
            const uint64_t db = smem_desc_sw128(smem_addr(smem + (size_t)xs * XT));
            const uint32_t ta = tmem_a + (uint32_t)((s * PAIR + h) * A_COLS);
            if (elect_one()) {
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                tc_mma<2>(tmem, ta + 8 * j, db + 2 * j, idesc, (i || h || j) ? 1u : 0u);
                if (n2)
                  tc_mma<2>(tmem + (uint32_t)a.n1, ta + 8 * j, db + 2 * j + (uint64_t)(a.box * 8), idesc2, (i || h || j) ? 1u : 0u);
              }
              tc_commit_pair(xempty + xs, both);
              if (h == PAIR - 1) tc_commit_pair(aempty + s, both);
            }
            __syncwarp();
            if (++xs == SX) { xs = 0; xph ^= 1u; }
          }
          if (++s == SA) { s = 0; sph ^= 1u; }
        }
        if (!ok && lane == 0) atomicExch(a.status, ERR_WAIT_MMA);
        if (elect_one()) tc_commit_pair(accfull, both);           // arrives when every MMA of the unit has completed
        __syncwarp();
      }
    }
  } else {
    // ---------------------------------------------------------------- decode warps: group g = warp / 8 takes the pairs
    // g, g + 2, ... of the cluster's units in order.  A warp reaches only the 32 tensor-memory lanes of its quadrant
    // (warp % 4), i.e. the two 16-row tiles 2 (warp % 4) and 2 (warp % 4) + 1: warps w and w + 4 of a group take one each.
    const int grp = warp / NDEC, w8 = warp % NDEC, rec = 2 * (w8 & 3) + (w8 >> 2);
    const uint32_t my_a = tmem_a + ((uint32_t)(rec * 16) << 16);
    const uint8_t* const my_raw = rawring + rec * (PAIR * REC);
    const int q4 = warp & 3, cg = warp >> 2;                     // epilogue: TMEM lane quadrant, column share of the warp
    // The two records of a pair are neighbours in memory order, so their escapes are one run of the list.  It is fetched
    // one step ahead: the list offsets come 32 pairs at a time (lane l holds those of pair eo_base + l) and the first 32
    // entries of the next pair are requested before this pair is decoded, so no global-load latency sits between the
    // records landing and the tiles being handed to the tensor core
    const int last = a.NG - k0;                                  // records of a row tile from k0 on
    const int* my_eo = nullptr;
    const uint32_t* el = nullptr;
    int e_unit = -1, e_live = 0, eo_base = 0, eo_lo = 0, eo_hi = 0;
    unsigned emask = 0u;                                         // bit l: pair eo_base + l of this warp has escapes
    auto load_offsets = [&](int first) {
      eo_base = first;
      const int j = (first + lane) * PAIR;
      const bool in = e_live && j < last;
      eo_lo = in ? __ldg(my_eo + j) : 0;
      eo_hi = in ? __ldg(my_eo + min(j + PAIR, last)) : 0;
      emask = __ballot_sync(FULL, eo_hi > eo_lo);
    };
    int lo = 0, hi = 0;
    uint32_t ent = 0u;
    auto fetch_escapes = [&](int unit, int i) {                  // (el, lo, hi, ent) of pair i of a unit
      lo = hi = 0;
      if (unit != e_unit) {
        const Rows rw = rows_of(unit);
        e_unit = unit;
        e_live = rw.rb < a.RB;                                   // (beyond an odd number of row blocks: zero records)
        el = a.nlist > 0 ? a.lel[rw.m] : a.el;
        my_eo = (a.nlist > 0 ? a.leo[rw.m] : a.eo) + (size_t)(rw.lrb * 8 + rec) * a.NG + k0;
        load_offsets(i);
      } else if (i - eo_base >= 32) {
        load_offsets(i);
      }
      const int off = i - eo_base;
      if ((emask >> off) & 1u) {                                 // most pairs have none: one bit test
        lo = __shfl_sync(FULL, eo_lo, off);
        hi = __shfl_sync(FULL, eo_hi, off);
        if (lane < hi - lo) ent = __ldg(el + lo + lane);
      }
    };
    // reads unit n's accumulator and stores it (KS == 1) or parks it over the idle rings
    auto finish = [&](int n) {
      if (!mbar_wait_look(accfull, (uint32_t)n & 1u)) {
        if (lane == 0) atomicExch(a.status, ERR_WAIT_ACC);
        return false;
      }
      __syncwarp();
      tc_fence_after();
      const int unit = unit0 + n * a.nclusters, tok0 = unit % a.TT * NT;
      const Rows rw = rows_of(unit);
      uint16_t* const Yp = a.nlist > 0 ? a.lY[rw.m] : a.Y;
      float* const Yfp = a.nlist > 0 ? a.lYf[rw.m] : a.Yf;
      const long long Mp = a.nlist > 0 ? a.lM[rw.m] : a.M;
      const int ncol = rw.rb < a.RB ? min(NT, a.B - tok0) : 0;    // token columns that exist
      const uint32_t my_acc = tmem + ((uint32_t)(q4 * 32) << 16);   // this lane's row is q4 * 32 + lane
      if (a.KS > 1) {
        float* const stg = reinterpret_cast<float*>(smem);       // [NT][128] fp32
        for (int c0 = cg * 16; c0 < NT; c0 += CSTEP) {
          uint32_t v[16];
          tmem_ld16(my_acc + (uint32_t)c0, v);
#pragma unroll
          for (int j = 0; j < 16; ++j) stg[(size_t)(c0 + j) * 128 + q4 * 32 + lane] = __uint_as_float(v[j]);
        }
        return true;
      }
      const size_t at = (size_t)tok0 * Mp + (size_t)rw.lrb * 128 + q4 * 32;
      store_unit(my_acc, cg * 16, NT, ncol, Yp + at, Yfp ? Yfp + at : nullptr, Mp, map_to_cta(smem_addr(accfree), first_rank));
      return true;
    };
    int unit = unit0, n = 0, i = grp, done = 0;                  // unit n of the cluster, pair i of it
    bool ok = true;
    auto step = [&](int& un, int& nn, int& ii) { while (ii >= np) { ii -= np; un += a.nclusters; ++nn; } };
    step(unit, n, i);
    if (grp < total) fetch_escapes(unit, i);
    int s = grp, r = grp;                                        // A slot, record slot (both counts are even and at least 2)
    uint32_t sph = 0u, rph = 0u;
    bool first = true;                                           // the A slot has not been used yet: nothing to wait for
    for (int j = grp; j < total; j += DG) {
      if (!mbar_wait(rfull + r, rph)) {
        if (lane == 0) atomicExch(a.status, ERR_WAIT_FULL);
        ok = false;
        break;
      }
      RecRegs rr[PAIR];
#pragma unroll
      for (int h = 0; h < PAIR; ++h) rr[h] = load_rec_shared(my_raw + r * RAW_SLOT + h * REC, lane);
      const int clo = lo, chi = hi, cn = n, ci = i;
      const uint32_t cent = ent;
      const uint32_t* const cel = el;
      i += DG;
      step(unit, n, i);
      lo = hi = 0;
      if (j + DG < total) fetch_escapes(unit, i);
      __syncwarp();
      if (lane == 0) mbar_arrive(rempty + r);                     // the slot can be refilled while we decode
      r += DG; if (r >= R) { r -= R; rph ^= 1u; }
#pragma unroll
      for (int h = 0; h < PAIR; ++h) {
        uint32_t A[4][4];
        decode_frag(rr[h], A);
        if (clo < chi) {                                          // entries of record h: bits 10..12 = column group % 8
          const uint32_t want = (uint32_t)(k0 + ci * PAIR + h) & 7u;
          for (int base = clo; base < chi; base += 32) {
            const uint32_t mine = base == clo ? cent : (lane < chi - base ? __ldg(cel + base + lane) : 0u);
            unsigned m = __ballot_sync(FULL, lane < chi - base && ((mine >> 10) & 7u) == want);
            while (m) {
              const int src = __ffs(m) - 1;
              m &= m - 1;
              patch_entry(A, __shfl_sync(FULL, mine, src), lane);
            }
          }
        }
        if (h == 0) {
          if (!first) ok = mbar_wait(aempty + s, sph ^ 1u);        // the MMAs of the slot's last use are done
          __syncwarp();
          if (!ok) break;
          tc_fence_after();
        }
        tmem_st_frag(my_a + (uint32_t)((s * PAIR + h) * A_COLS), A);
      }
      if (!ok) {
        if (lane == 0) atomicExch(a.status, ERR_WAIT_EMPTY);
        break;
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_addr(aready + s), first_rank));
      s += DG; if (s >= SA) { s -= SA; sph ^= 1u; first = false; }
      for (; ok && done < cn; ++done) ok = finish(done);          // the units before this pair's
      if (!ok) break;
    }
    for (; ok && done < nunits; ++done) ok = finish(done);
  }
  tc_fence_before();
  __syncwarp();
  cluster_sync_all();                                            // parked tiles are visible; nobody's shared memory is read any more
  if (a.KS > 1) {
    if (warp < NDW && nunits > 0) {
      // -------------------------------------------------------------- add the KS tiles of this half, rank order
      const int unit = unit0, tok0 = unit % a.TT * NT;
      const Rows rw = rows_of(unit);
      uint16_t* const Yp = a.nlist > 0 ? a.lY[rw.m] : a.Y;
      float* const Yfp = a.nlist > 0 ? a.lYf[rw.m] : a.Yf;
      const long long Mp = a.nlist > 0 ? a.lM[rw.m] : a.M;
      const int ncol = rw.rb < a.RB ? min(NT, a.B - tok0) : 0;
      const int c_lo = (int)((long long)ncol * ks / a.KS), c_end = (int)((long long)ncol * (ks + 1) / a.KS);
      const uint32_t mine = smem_addr(smem);
      // CPP columns per pass, every partial tile's float4 requested before the first add: distributed-shared-memory reads
      // have a long latency, so the loads of a pass must all be in flight together
      constexpr int CPP = 4;
      for (int c = c_lo + warp; c < c_end; c += CPP * NDW) {
        float4 v[CPP][4];
#pragma unroll
        for (int h = 0; h < CPP; ++h)
#pragma unroll
          for (int p = 0; p < 4; ++p)
            if (p < a.KS && c + h * NDW < c_end) {
              const uint32_t at = (uint32_t)(((c + h * NDW) * 128 + 4 * lane) * 4);
              v[h][p] = p == ks ? *reinterpret_cast<const float4*>(smem + at)
                                : ld_cluster_f4(map_to_cta(mine + at, (uint32_t)(2 * p + half)));
            }
#pragma unroll
        for (int h = 0; h < CPP; ++h) {
          const int cc = c + h * NDW;
          if (cc >= c_end) break;
          float4 sum = v[h][0];
#pragma unroll
          for (int p = 1; p < 4; ++p)
            if (p < a.KS) { sum.x += v[h][p].x; sum.y += v[h][p].y; sum.z += v[h][p].z; sum.w += v[h][p].w; }
          const size_t o = (size_t)(tok0 + cc) * Mp + (size_t)rw.lrb * 128 + 4 * lane;
          uint2 packed;
          packed.x = pack_bf16(sum.x, sum.y);
          packed.y = pack_bf16(sum.z, sum.w);
          *reinterpret_cast<uint2*>(Yp + o) = packed;
          if (Yfp) *reinterpret_cast<float4*>(Yfp + o) = sum;
        }
      }
    }
    __syncwarp();
    cluster_sync_all();                                          // nobody leaves while a peer still reads its tile
  }
  if (warp == W_MMA) {
    __syncwarp();
    tmem_dealloc<2>(tmem, (uint32_t)TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------------ host side
int set_attr() {                                                 // once per device: opt in to the large dynamic shared memory
  static bool set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !set[dev]) {
    if (int e = st::cuda_fail(cudaFuncSetAttribute(pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES),
                              "st_gemm: shared memory attribute"))
      return e;
    set[dev] = true;
  }
  return 0;
}

// clusters of 2 ks CTAs that are resident at once (a cluster lives inside one GPC: sizes that do not divide a GPC's SM count
// strand SMs); asked from the driver once per device and size
int resident_clusters(int ks, int sms) {
  static int cache[64][5] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return sms / (2 * ks);
  if (cache[dev][ks] == 0) {
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * ks * sms));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)(2 * ks);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (set_attr() != 0 || cudaOccupancyMaxActiveClusters(&n, pair_kernel, &cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = sms / (2 * ks);                                        // no answer (no device): assume perfect packing
    }
    cache[dev][ks] = n;
  }
  return cache[dev][ks];
}

struct PairPlan {
  int NT, TT, n1, box, astages, xstages, rstages, bar_off;
  int tile1, KS;                                                 // units [0, tile1) unsplit, the rest in a launch split KS ways
  size_t smem;
};

void rings(PairPlan& p) {
  p.n1 = p.NT <= 256 ? p.NT : (p.NT / 2 + 31) & ~31;             // MMA widths: multiples of 32
  p.box = p.n1 / 2;
  const size_t xt = (size_t)(p.n1 < p.NT ? 2 : 1) * p.box * 128;
  const size_t stg = (size_t)p.NT * 128 * 4;                      // the parked accumulator tile reuses the rings
  const size_t slack = 1024 /* alignment */ + 512 /* barriers */;
  const size_t budget = SMEM_BYTES - slack;
  p.astages = (TMEM_COLS - p.NT) / (PAIR * A_COLS);
  if (p.astages > 4) p.astages = 4;
  p.astages &= ~1;                                                // slot parity: see the kernel
  // activation tiles: enough to cover the L2 latency (four if they fit beside four record slots); the rest of the shared
  // memory goes to the record ring, which covers the HBM latency
  p.xstages = 4;
  p.rstages = (int)((budget - p.xstages * xt) / RAW_SLOT);
  if (p.rstages > 6) p.rstages = 6;
  p.rstages &= ~1;
  p.xstages = (int)((budget - (size_t)p.rstages * RAW_SLOT) / xt);
  if (p.xstages > 8) p.xstages = 8;
  size_t ring = p.xstages * xt + (size_t)p.rstages * RAW_SLOT;
  if (ring < stg) ring = stg;
  ring = (ring + 15) & ~(size_t)15;
  p.bar_off = (int)ring;
  p.smem = ring + slack;
}

// Token tiles and split of the k range: the least estimated time in us (`time`), fitted to launches of 6144, 4096, 24576 and 12288 x
// 4096 / 12288 / 2048 matrices in a graph at 129 to 2000 tokens: start-up and drain (which the next launch hides where SMs are free),
// per pair of k-tiles the larger of the decode and a time that grows with the token tile, more when every SM streams, and the epilogue
// of a split (adding KS tiles through distributed shared memory).  Units beyond the resident clusters run in waves, in one launch or,
// when it is the faster, the full waves unsplit and the rest in a second launch with a split.
// What the plan is expected to take, which decides between this kernel and the one-CTA one: `expected`, the same terms fitted with
// the one-CTA kernel's so that the ratio of the two is met (st_gemm.cu).  Up to half of the SMs, the next launch's clusters start
// beside this one's; further waves of a split start anew.  (Choosing the plan by it was no better: 34 of 520 sizes slower by more
// than 3 %, 40 faster.)
// One token tile and between one and two waves: all of it in one launch, or the full wave and a split rest, by `expected` too.  us in
// two launches / in one: 24576 x 1024 at 200 tokens 25.4 / 18.6, 24576 x 2048 at 330 42.5 / 36.9, 28672 x 2048 at 300 42.8 / 37.0,
// 28672 x 4096 73.8 / 67.1, 24576 x 4096 at 330 65.5 / 65.5, 20480 x 2048 at 384 41.9 / 41.9 (one launch was never the slower one at the
// 81 sizes where it is estimated to be the faster).
PairPlan make_plan(long long M, int NG, long long B, double& us) {
  const int sms = st::sm_count(), RP = (int)((M / 128 + 1) / 2), pairs = (NG + PAIR - 1) / PAIR;
  const int C = resident_clusters(1, sms);
  const int ksmax = pairs / 4 < 1 ? 1 : (pairs / 4 > 4 ? 4 : pairs / 4);
  PairPlan best = {};
  us = 1e30;
  auto expected = [&](long long u, int ks, int nt) {
    const int slots = resident_clusters(ks, sms), per = (pairs + ks - 1) / ks;
    const double waves = (double)((u + slots - 1) / slots), load = (double)(u < slots ? u : slots) * ks / C;
    const double pair = 0.214 + 0.0019 * nt > 0.576 ? 0.214 + 0.0019 * nt : 0.576;
    const double end = ks > 1 ? 1.44 + ks * (0.0065 * nt - 0.3) + 7.1 * (waves - 1.0) / waves : 0.0063 * nt - 0.66;
    return 1.66 + 2.77 * load + (load > 0.5 ? 1.5 : 0.0) + waves * (per * (pair + 0.17 * load) + end);
  };
  int tt_lo = (int)((B + NT_MAX - 1) / NT_MAX), tt_hi = (int)((B + 127) / 128), ks_lo = 1, ks_hi = ksmax;
#ifdef ST_TUNE                                                   // development builds may force both
  if (const char* f = getenv("STATETREE_PAIR_TT")) if (atoi(f) >= tt_lo && atoi(f) > 0) tt_lo = tt_hi = atoi(f);
  if (const char* f = getenv("STATETREE_PAIR_KS")) if (atoi(f) > 0) ks_lo = ks_hi = atoi(f) < ksmax ? atoi(f) : ksmax;
#endif
  for (int tt = tt_lo; tt <= tt_hi; ++tt) {
    const int per = (int)((B + tt - 1) / tt), nt = (per + 31) & ~31;   // MMA widths: multiples of 32
    if (nt > NT_MAX) continue;
    const long long units = (long long)RP * tt, full = units / C * C, rest = units - full;
    const double pair = 0.25 + 0.00175 * nt > 0.52 ? 0.25 + 0.00175 * nt : 0.52;
    auto time = [&](long long u, int ks) {
      const int slots = resident_clusters(ks, sms);
      const double waves = (double)((u + slots - 1) / slots), load = (double)(u < slots ? u : slots) * ks / C;
      return 2.0 + 4.5 * load + waves * (((pairs + ks - 1) / ks) * (pair + 0.13 * load) + (ks > 1 ? ks * (1.0 + 0.0045 * nt) : 0.3));
    };
    for (int ks = ks_lo; ks <= ks_hi; ++ks) {
      double t;
      long long tile1 = 0;                                       // units of the unsplit launch
      if (full == 0) {
        t = time(units, ks);
      } else if (ks == 1 && (tt > 1 || full > C || rest == 0)) {
        t = time(units, 1);
        tile1 = units;
      } else if (rest > 0) {
        t = time(full, 1) + time(rest, ks);
        tile1 = full;
      } else {
        continue;
      }
      if (t < us - 1e-9) { us = t; best.NT = nt; best.TT = tt; best.tile1 = (int)tile1; best.KS = ks; }
    }
  }
  if (best.TT == 0) return best;
  const long long units = (long long)RP * best.TT;
  us = (best.tile1 > 0 ? expected(best.tile1, 1, best.NT) : 0.0) +
       (units > best.tile1 ? expected(units - best.tile1, best.KS, best.NT) + (best.tile1 > 0 ? 5.0 : 0.0) : 0.0);
  if (tt_lo == 1 && ks_lo == 1 && RP > C && RP < 2 * C) {
    const int nt = (int)((B + 31) & ~31ll);
    const double one = expected(RP, 1, nt);
    if (one < 0.97 * us) { us = one; best.NT = nt; best.TT = 1; best.tile1 = RP; best.KS = 1; }
  }
  rings(best);
  return best;
}

int launch(const PairPlan& p, GemmArgs& a, int tile0, int tile1, int KS, const CUtensorMap& xmap, const WMaps& wmaps,
           cudaStream_t stream) {
  const int C = resident_clusters(1, st::sm_count()), units = tile1 - tile0;
  a.tile0 = tile0; a.tile1 = tile1; a.KS = KS;
  a.nclusters = KS > 1 || units < C ? units : C;                  // (a split cluster parks its tile over the rings: one unit)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(a.nclusters * 2 * KS));
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)(2 * KS);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = st::pdl_enabled() ? 2 : 1;
  return st::cuda_fail(cudaLaunchKernelEx(&cfg, pair_kernel, a, xmap, wmaps), "st_gemm launch");
}
}  // namespace

int st::pair_gemm(GemmArgs& a, const WMaps& wmaps, const void* X, const char* who, double us, cudaStream_t stream) {
  double mine;
  const PairPlan p = make_plan(a.M, a.NG, a.B, mine);
  if (mine >= us) return -1;
  ST_REQUIRE((a.M / 256 + 1) * (long long)p.TT * 8 < (1ll << 31), "%s: grid too large", who);
  if (int e = set_attr()) return e;
  CUtensorMap xmap;
  if (int e = make_xmap(&xmap, X, a.B, (long long)a.NG * 64, p.box, who)) return e;
  a.NT = p.NT; a.TT = p.TT; a.n1 = p.n1; a.box = p.box; a.RB = (int)(a.M / 128);
  a.astages = p.astages; a.xstages = p.xstages; a.rstages = p.rstages; a.bar_off = p.bar_off; a.tmem_cols = TMEM_COLS;
  const int units = (a.RB + 1) / 2 * p.TT;
  if (p.tile1 > 0)
    if (int e = launch(p, a, 0, p.tile1, 1, xmap, wmaps, stream)) return e;
  return p.tile1 < units ? launch(p, a, p.tile1, units, p.KS, xmap, wmaps, stream) : 0;
}
