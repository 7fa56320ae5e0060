// Fused tree-decode + GEMM on the 5th-generation tensor cores (tcgen05 / TMEM) of sm_100a, one CTA per tile of at most 320 tokens,
// and its grouped (mixture-of-experts) form.  More than 128 tokens go to CTA pairs (st_gemm_pair.cu) where those are the faster ones.
//   Y[B, M] = X[B, N] W[M, N]^T,  W as state-tree records, fp32 accumulation in tensor memory, BF16 output.
//
// One CTA computes a 128-row block of W against one tile of NT tokens over a contiguous range of 64-column k-tiles.
// Warp roles:
//   8 DG decode warps, in DG groups of eight (group g takes the k-tile pairs g, g + DG, ...): each warp turns the two
//              records of its 16 rows into mma-fragment registers (five integer ops per four weights), patches escapes,
//              and writes each 16 x 64 BF16 sub-tile into TENSOR MEMORY with one tcgen05.st.16x128b.x8: a record is stored in mma.m16n8k16
//              A-fragment order, which is that instruction's register layout, so the A operand never touches shared
//              memory (no stmatrix, no proxy fence, no operand read by the tensor core)
//   record producer: one 3-D tiled TMA load per pair of k-tiles brings the sixteen 1552-byte records of the block's eight
//              16-row tiles into a ring
//   activation producer: tiled TMA loads of X[tok0 .. tok0 + NT, 64 cols] with the 128-byte swizzle
//   MMA issuer: one elected thread issues four tcgen05.mma (128 x NT x 16, kind::f16; two halves beyond 256 tokens) per
//              k-tile, A from tensor memory, B from shared memory, D in tensor memory; tcgen05.commit frees the stage
// Epilogue: a CTA that owns its whole k range stores BF16 straight from tcgen05.ld registers; the CTAs that split a k
// range form a thread-block cluster, park their fp32 tiles in shared memory and add them through distributed shared
// memory in rank order (deterministic), then store BF16.
// The grouped (mixture-of-experts) variant runs the same pipeline per (block of NT routed pairs, 128-row block): the
// block's expert selects the weight tensor map and escape tables, the activation tile comes from rows gathered in
// block order, the MMA width and the activation loads cover only the pairs the block really holds, and the result rows
// are scattered back to their pair indices.
// Every mbarrier wait is bounded; a wait that runs out sets the device status word and the CTA leaves after
// releasing its tensor memory.
#include <stdlib.h>
#include <string.h>

#include <mutex>

#include "../../include/statetree_b200.h"
#include "st_tc.cuh"

namespace {
using namespace st;

constexpr int MAXL = MAXL_GEMM;              // matrices in one list launch
#define GW mbar_wait_look
constexpr int XBOX_GROUPED = 32;             // rows per activation load of the grouped variant
template <int DG> constexpr int gemm_threads() { return (DG * NDEC + 3) * 32; }

// Three rings.  The RAW ring (R slots of sixteen records) faces HBM: its depth sets the bytes in flight.  The A ring (SA
// slots of two decoded weight tiles in tensor memory) covers the decode -> MMA hand-over, the X ring (SX activation tiles
// of one k-tile in shared memory) the L2 latency of the activation loads.
//
// Why pairs: a decode warp's time per step is ~250 cycles of decoding per record and ~700 cycles of barrier looks, slot
// hand-overs and escape bookkeeping per step, whatever the step holds (cycle counters around each part, 6144 x 4096): one
// record per step cost 1000 cycles, i.e. 63 per record and SM with sixteen warps.
//
// DG = 1 (token tiles up to 128): eight decode warps, at most half of an SM's shared memory, registers and tensor memory,
// so two CTAs share an SM: one CTA's start-up, drain and epilogue run under the other's main loop, and the next launch's
// CTAs become resident (and start streaming weights) as soon as any CTA of this launch leaves.
// DG = 2 (tiles of up to 320 tokens): one CTA per SM, sixteen decode warps.
//
// Measured, the four projections of a layer (6144, 4096, 24576 x 4096 and 4096 x 12288) in a graph, us per layer: 64 rows
// 108 -> 85, 300 rows 251 -> 153 (was: A through shared memory by stmatrix, one record per step, 64 / 128 / 256-token
// tiles, an issuer under a lane test).  What bounds it now: up to ~128 tokens HBM plus ~5 us per launch of start-up, drain
// and the split's epilogue; beyond, the shared-memory port (records in and out, activation tile in and out:
// 3.1 KB + 32 B x tokens per record at 128 B per cycle; 800 cycles per k-tile at 304 tokens against 608 of MMAs).
//
// *Slot parity.*  An mbarrier tells only its current phase from the previous one, so a waiter must never be two phases
// away.  With two decode groups that alternate pairs every A slot and record slot has to belong to one group (whose own
// program order guarantees that): both counts are even when DG = 2.
//
// The KS CTAs that split the k range of one (row block, token tile) form a thread-block cluster (blockIdx.x % KS is
// the rank).  After its main loop every CTA parks its fp32 accumulator tile in its own shared memory; after a cluster
// barrier CTA j adds the KS tiles for its share of the token columns through distributed shared memory, in rank
// order (bit-identical from run to run), and stores BF16.  No partial sums travel through global memory.
template <int DG, bool GROUPED>
__global__ void __launch_bounds__(gemm_threads<DG>(), DG == 1 ? 2 : 1)
gemm_kernel(const GemmArgs a, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ WMaps wmaps) {
  constexpr int NDW = DG * NDEC;                                              // decode warps
  constexpr int W_RAW = NDW, W_X = NDW + 1, W_MMA = NDW + 2;                  // role warps
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_used[4], s_row[128];          // grouped: pairs per 32 entries of the block, result row of each entry
  uint8_t* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);   // (stays a shared-memory pointer to the compiler)
  const int NT = a.NT, SA = a.astages, SX = a.xstages, R = a.rstages;
  const int XT = NT * 128;                       // bytes of an activation tile
  uint8_t* rawring = smem + (size_t)SX * XT;                         // [R] record slots
  uint64_t* aready = reinterpret_cast<uint64_t*>(smem + a.bar_off);  // [SA] the slot's weight tiles are in tensor memory
  uint64_t* aempty = aready + SA;                                    // [SA] the MMAs that read the slot have completed
  uint64_t* xfull = aempty + SA;                                     // [SX] activation tile landed
  uint64_t* xempty = xfull + SX;                                     // [SX] the MMAs that read it have completed
  uint64_t* rfull = xempty + SX;                                     // [R] records landed
  uint64_t* rempty = rfull + R;                                      // [R] records copied to registers
  uint64_t* accbar = rempty + R;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accbar + 1);

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(FULL, tid >> 5, 0);   // (a warp-uniform value to the compiler)
  // unit of this CTA.  Dense: the token tiles of a row block run next to each other (its records then come from HBM once
  // and from L2 for the other tiles); grouped: the row blocks of a pair block do (they share the gathered activations)
  const int ks = blockIdx.x % a.KS, rt = blockIdx.x / a.KS;
  const bool tiles = DG == 2 && !GROUPED && a.TT > 1;            // (up to 128 tokens are one tile)
  const int rb = GROUPED ? rt % a.RB : a.rb0 + (tiles ? rt / a.TT : rt), tt = GROUPED ? rt / a.RB : (tiles ? rt % a.TT : 0);
  // whole pairs of k-tiles; an odd last tile is paired with one beyond the matrix, which both tensor maps fill with zeros
  const int pairs = (a.NG + PAIR - 1) / PAIR;
  const int p0 = (int)((long long)pairs * ks / a.KS), np = (int)((long long)pairs * (ks + 1) / a.KS) - p0;
  const int k0 = p0 * PAIR;
  const int tok0 = tt * NT;
  // the matrix this CTA multiplies by: the one of the call, or (grouped) the expert of pair block tt
  const int* eo = a.eo;
  const uint32_t* el = a.el;
  const CUtensorMap* wm = &wmaps.m[0];
  int lrb = rb;                                                  // row block inside its matrix
  uint16_t* Yp = a.Y;
  float* Yfp = a.Yf;
  long long Mp = a.M;
  int ncol = GROUPED ? NT : min(NT, a.B - tok0);                 // token columns that exist
  if (!GROUPED && a.nlist > 0) {                                 // a list: the member this row block belongs to
    int m = 0;
    while (m + 1 < a.nlist && rb >= a.rbend[m]) ++m;
    lrb = rb - (m ? a.rbend[m - 1] : 0);
    eo = a.leo[m]; el = a.lel[m]; wm = &wmaps.m[m];
    Yp = a.lY[m]; Yfp = a.lYf[m]; Mp = a.lM[m];
  }
  if (GROUPED) {
    pdl_wait();                                                  // the block table comes from an earlier kernel
    // (the three lookups are requested together: a chain of them would be most of a short CTA's start-up)
    const int npost = a.npost[0], expert = a.bexp[tt];
    int p = -1;
    if (tid < NT) p = a.sorted[tok0 + tid];
    if (tok0 >= npost) return;                                   // beyond the blocks the routing filled
    if (expert < 0 || expert >= a.E) return;                     // another rank's expert
    eo = reinterpret_cast<const int*>(a.eop[expert]);
    el = reinterpret_cast<const uint32_t*>(a.elp[expert]);
    wm = a.maps + expert;
    if (tid == 0) asm volatile("prefetch.tensormap [%0];" :: "l"(wm) : "memory");
    if (tid < NT) {
      const bool pair = p >= 0 && p < a.B;
      s_row[tid] = pair ? p : -1;
      const int used = __reduce_max_sync(FULL, pair ? tid + 1 : 0);
      if (lane == 0) s_used[warp] = used;
    }
  }

  // Set-up, spread over the role warps.  The record producer prepares the barriers (a lane each) and sends the first ring
  // fill off before the block synchronises: weights depend on no earlier kernel.
  auto load_records = [&](int i, int r) {
    // one tiled TMA load per pair of k-tiles fetches sixteen records (row tiles rb * 8 .. + 7, column groups k0 + 2 i and
    // + 1) through a 3-D view of the tree [row tile][column group][194 x u64]; separate bulk copies would cost far more
    if (elect_one()) {
      mbar_expect_tx(rfull + r, (uint32_t)RAW_SLOT);
      tma_load_3d(rawring + (size_t)r * RAW_SLOT, wm, 0, k0 + PAIR * i, lrb * 8, rfull + r);
    }
    __syncwarp();
  };
  if (warp == W_RAW) {
    if (!GROUPED && elect_one()) asm volatile("prefetch.tensormap [%0];" :: "l"(wm) : "memory");
    for (int b = lane; b < 2 * (SA + SX + R) + 1; b += 32) {
      int count = 1;                                             // aempty, xfull, xempty, rfull, accbar
      if (b < SA || (b >= 2 * (SA + SX) + R && b < 2 * (SA + SX + R))) count = NDEC;   // aready, rempty: one arrival per decode warp
      mbar_init(aready + b, count);
    }
    fence_barrier_init();
    __syncwarp();
    for (int i = 0; i < min(np, R); ++i) load_records(i, i);
  } else if (warp == W_X) {
    if (elect_one()) asm volatile("prefetch.tensormap [%0];" :: "l"(&xmap) : "memory");
  } else if (warp == W_MMA) {
    tmem_alloc<1>(tmem_slot, (uint32_t)a.tmem_cols);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (GROUPED) {                                                 // pairs in the block: one past the last that is not padding
    ncol = 0;
    for (int w = 0; w * 32 < NT; ++w) ncol = max(ncol, s_used[w]);
  }
  const int nmma = GROUPED ? (max(ncol, 1) + 15) & ~15 : NT;     // token columns the MMAs cover
  const uint32_t tmem = *tmem_slot;
  const uint32_t tmem_a = tmem + (uint32_t)((NT + 31) & ~31);    // the weight tiles' columns follow the accumulator
  pdl_launch_dependents();

  if (warp == W_RAW) {
    // ---------------------------------------------------------------- record producer, behind the first ring fill
    for (int i = R, r = 0, k = 1; i < np; ++i, r = (r + 1 == R ? 0 : r + 1), k += (r == 0)) {
      if (!GW(rempty + r, (uint32_t)(k - 1) & 1u)) { if (lane == 0) atomicExch(a.status, ERR_WAIT_EMPTY); break; }
      load_records(i, r);
    }
  } else if (warp == W_X) {
    // ---------------------------------------------------------------- activation producer.  The activations are the
    // only input an earlier kernel of the stream may still be writing: with programmatic dependent launch the CTA
    // starts (and its record producer streams weights) under the tail of that kernel, and this thread is the one that
    // waits for it.  Everything that touches the output is downstream of the first activation tile.
    pdl_wait();
    const int box = GROUPED ? XBOX_GROUPED : (NT > 256 ? NT / 2 : NT);       // rows per load
    const int nbox = GROUPED ? (nmma + XBOX_GROUPED - 1) / XBOX_GROUPED : (NT > 256 ? 2 : 1);
    for (int i = 0, s = 0, k = 0; i < np * PAIR; ++i, s = (s + 1 == SX ? 0 : s + 1), k += (s == 0)) {
      if (k > 0 && !GW(xempty + s, (uint32_t)(k - 1) & 1u)) { if (lane == 0) atomicExch(a.status, ERR_WAIT_EMPTY); break; }
      if (elect_one()) {
        mbar_expect_tx(xfull + s, (uint32_t)(nbox * box * 128));
        for (int b = 0; b < nbox; ++b)
          tma_load_2d(smem + (size_t)s * XT + (size_t)b * box * 128, &xmap, (k0 + i) * 64, tok0 + b * box, xfull + s);
      }
      __syncwarp();
    }
  } else if (warp == W_MMA) {
    // ---------------------------------------------------------------- MMA issuer.  The whole warp waits; one elected
    // lane issues.  The loop must stay warp-uniform: tensor-core and TMA instructions take their operands from uniform
    // registers, and under a lane test (`if (lane == 0)`) the compiler has to serialise over the lanes around each one
    // (measured: ~1000 cycles for the four MMAs and the commit of a k-tile instead of < 200).
    // beyond 256 tokens one MMA cannot cover the tile: two, of (up to 16 tokens) different width
    const int half = NT > 256 ? ((NT / 2 + 15) & ~15) : 0;
    const uint32_t idesc = mma_idesc(128, half ? half : nmma), idesc2 = mma_idesc(128, half ? NT - half : 16);
    int xs = 0, xk = 0;
    bool ok = true;
    for (int i = 0, s = 0, k = 0; ok && i < np; ++i, s = (s + 1 == SA ? 0 : s + 1), k += (s == 0)) {
      ok = GW(aready + s, (uint32_t)k & 1u);
      tc_fence_after();
#pragma unroll
      for (int h = 0; h < PAIR; ++h) {
        ok = ok && GW(xfull + xs, (uint32_t)xk & 1u);
        if (!ok) break;
        const uint64_t db = smem_desc_sw128(smem_addr(smem + (size_t)xs * XT));
        const uint32_t ta = tmem_a + (uint32_t)((s * PAIR + h) * A_COLS);
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            tc_mma<1>(tmem, ta + 8 * j, db + 2 * j, idesc, (i || h || j) ? 1u : 0u);
            if (half)
              tc_mma<1>(tmem + (uint32_t)half, ta + 8 * j, db + 2 * j + (uint64_t)(half * 8), idesc2, (i || h || j) ? 1u : 0u);
          }
          tc_commit(xempty + xs);
          if (h == PAIR - 1) tc_commit(aempty + s);
        }
        __syncwarp();
        if (++xs == SX) { xs = 0; ++xk; }
      }
    }
    if (!ok && lane == 0) atomicExch(a.status, ERR_WAIT_MMA);
    if (elect_one()) tc_commit(accbar);                           // arrives when every MMA has completed
    __syncwarp();
  } else {
    // ---------------------------------------------------------------- decode warps: group g = warp / 8 takes the
    // pairs i = g, g + DG, ...  A warp reaches only the 32 tensor-memory lanes of its quadrant (warp % 4), i.e. the two
    // 16-row tiles 2 (warp % 4) and 2 (warp % 4) + 1: warps w and w + 4 of a group take one each.
    const int grp = warp / NDEC, w8 = warp % NDEC, rec = 2 * (w8 & 3) + (w8 >> 2);
    const uint32_t my_a = tmem_a + ((uint32_t)(rec * 16) << 16);
    const uint8_t* const my_raw = rawring + rec * (PAIR * REC);
    const int* const my_eo = eo + (size_t)(lrb * 8 + rec) * a.NG + k0;
    const int last = a.NG - k0;                                    // records of this row tile from k0 on
    // The two records of a pair are neighbours in memory order, so their escapes are one run of the list.  It is fetched
    // one pair ahead: the list offsets come 32 pairs at a time (lane l holds those of pair eo_base + l) and the first 32
    // entries of the next pair are requested before this pair is decoded, so no global-load latency sits between the
    // records landing and the tiles being handed to the tensor core
    int eo_base = 0, eo_lo = 0, eo_hi = 0;
    unsigned emask = 0u;                                           // bit l: pair eo_base + l of this warp has escapes
    auto load_offsets = [&](int first) {
      eo_base = first;
      const int j = (first + lane) * PAIR;
      eo_lo = j < last ? __ldg(my_eo + j) : 0;
      eo_hi = j < last ? __ldg(my_eo + min(j + PAIR, last)) : 0;
      emask = __ballot_sync(FULL, eo_hi > eo_lo);
    };
    int lo = 0, hi = 0;
    uint32_t ent = 0u;
    auto fetch_escapes = [&](int i) {                              // (lo, hi, ent) of pair i
      lo = hi = 0;
      if (i >= np) return;
      if (i - eo_base >= 32) load_offsets(i);
      const int off = i - eo_base;
      if ((emask >> off) & 1u) {                                  // most pairs have none: one bit test
        lo = __shfl_sync(FULL, eo_lo, off);
        hi = __shfl_sync(FULL, eo_hi, off);
        if (lane < hi - lo) ent = __ldg(el + lo + lane);
      }
    };
    load_offsets(grp);
    fetch_escapes(grp);
    int s = grp % SA, r = grp % R;                                 // A slot, record slot
    uint32_t sph = (uint32_t)(grp / SA) & 1u, rph = (uint32_t)(grp / R) & 1u;
    bool first = grp < SA;                                         // the slot has not been used yet: nothing to wait for
    for (int i = grp; i < np; i += DG) {
      if (!mbar_wait(rfull + r, rph)) {
        if (lane == 0) atomicExch(a.status, ERR_WAIT_FULL);
        break;
      }
      RecRegs rr[PAIR];
#pragma unroll
      for (int h = 0; h < PAIR; ++h) rr[h] = load_rec_shared(my_raw + r * RAW_SLOT + h * REC, lane);
      const int clo = lo, chi = hi;
      const uint32_t cent = ent;
      fetch_escapes(i + DG);
      __syncwarp();
      if (lane == 0) mbar_arrive(rempty + r);                     // the slot can be refilled while we decode
      r += DG; if (r >= R) { r -= R; rph ^= 1u; }
      bool ok = true;
#pragma unroll
      for (int h = 0; h < PAIR; ++h) {
        uint32_t A[4][4];
        decode_frag(rr[h], A);
        if (clo < chi) {                                          // entries of record h: bits 10..12 = column group % 8
          const uint32_t want = (uint32_t)(k0 + i * PAIR + h) & 7u;
          for (int base = clo; base < chi; base += 32) {
            const uint32_t mine = base == clo ? cent : (lane < chi - base ? __ldg(el + base + lane) : 0u);
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
      if (lane == 0) mbar_arrive(aready + s);
      s += DG; if (s >= SA) { s -= SA; sph ^= 1u; first = false; }
    }
    // ---------------------------------------------------------------- epilogue 1: accumulator -> registers
    __syncwarp();
    const bool acc_ok = GW(accbar, 0u);
    if (!acc_ok && lane == 0) atomicExch(a.status, ERR_WAIT_ACC);
    __syncwarp();
    tc_fence_after();
    const int q4 = warp & 3, cg = warp >> 2;                     // TMEM lane quadrant, column share of the warp
    float* stg = reinterpret_cast<float*>(smem);                 // [NT][128] fp32, over the (now idle) rings
    for (int c0 = cg * 16; c0 < nmma; c0 += (NDW / 4) * 16) {
      uint32_t v[16];
      tmem_ld16(tmem + ((uint32_t)(q4 * 32) << 16) + (uint32_t)c0, v);
      if (!GROUPED && a.KS > 1) {
#pragma unroll
        for (int j = 0; j < 16; ++j) stg[(size_t)(c0 + j) * 128 + q4 * 32 + lane] = __uint_as_float(v[j]);
      } else {
        // whole k range: this lane holds row q4 * 32 + lane of 16 token columns.  Lanes pair up (even: column j, odd:
        // column j + 1, two rows each) so that a store instruction writes 4 bytes per lane, 64 bytes per column
        const long long m0 = (long long)lrb * 128 + q4 * 32 + (lane & ~1);
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          const uint32_t give = (lane & 1) ? v[j] : v[j + 1], keep = (lane & 1) ? v[j + 1] : v[j];
          const uint32_t got = __shfl_xor_sync(FULL, give, 1);
          const float x0 = __uint_as_float((lane & 1) ? got : keep), x1 = __uint_as_float((lane & 1) ? keep : got);
          const int c = c0 + j + (lane & 1);
          if (c < ncol && acc_ok) {
            long long row = tok0 + c;
            if (GROUPED) row = s_row[c];                           // result rows go back to their pair index
            if (!GROUPED || row >= 0) {
              *reinterpret_cast<uint32_t*>(Yp + (size_t)row * Mp + m0) = pack_bf16(x0, x1);
              if (Yfp) *reinterpret_cast<float2*>(Yfp + (size_t)row * Mp + m0) = make_float2(x0, x1);
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncwarp();
  if (GROUPED || a.KS == 1) {
    __syncthreads();
  } else {
    cluster_sync_all();                                          // every CTA of the cluster has parked its tile
    if (warp < NDW) {
      // -------------------------------------------------------------- epilogue 2: add the KS tiles, rank order
      const int c_lo = (int)((long long)ncol * ks / a.KS), c_end = (int)((long long)ncol * (ks + 1) / a.KS);
      const uint32_t mine = smem_addr(smem);
      // CPP columns per pass, every partial tile's float4 requested before the first add: distributed-shared-memory
      // reads have a long latency, so the loads of a pass must all be in flight together
      constexpr int CPP = DG;                                    // (DG = 2 has up to twice the columns; DG = 1 takes 63 registers of the 88 it may)
      for (int c = c_lo + warp; c < c_end; c += CPP * NDW) {
        float4 v[CPP][8];
#pragma unroll
        for (int h = 0; h < CPP; ++h)
#pragma unroll
          for (int p = 0; p < 8; ++p)
            if (p < a.KS && c + h * NDW < c_end)
              v[h][p] = ld_cluster_f4(map_to_cta(mine + (uint32_t)(((c + h * NDW) * 128 + 4 * lane) * 4), (uint32_t)p));
#pragma unroll
        for (int h = 0; h < CPP; ++h) {
          const int cc = c + h * NDW;
          if (cc >= c_end) break;
          float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int p = 0; p < 8; ++p)
            if (p < a.KS) { sum.x += v[h][p].x; sum.y += v[h][p].y; sum.z += v[h][p].z; sum.w += v[h][p].w; }
          const size_t o = (size_t)(tok0 + cc) * Mp + lrb * 128 + 4 * lane;
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
    tmem_dealloc<1>(tmem, (uint32_t)a.tmem_cols);
  }
}

// ------------------------------------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

struct GemmPlan {
  int RB1, KS1;                                                  // the first RB1 row blocks go out in a launch of their own, split KS1 ways
  int NT, TT, RB, KS, DG, astages, xstages, rstages, bar_off, tmem_cols;
  size_t smem;
};

template <int DG, bool GROUPED>
int gemm_attr() {                                                // once per device: opt in to the large dynamic shared memory
  static bool set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !set[dev]) {
    if (int e = st::cuda_fail(cudaFuncSetAttribute(gemm_kernel<DG, GROUPED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   DG == 1 ? 113 * 1024 : 220 * 1024), "st_gemm: shared memory attribute"))
      return e;
    set[dev] = true;
  }
  return 0;
}

// CTAs that can be resident at once when launched as clusters of ks: a cluster lives inside one GPC, so sizes that do not
// divide a GPC's SM count strand SMs (one CTA per SM: clusters of 3 fit 45 times, not 49).  Asked from the driver once per
// (device, cluster size, kernel).  The driver's answer assumes one CTA per SM for every kernel that allocates tensor
// memory; the DG = 1 kernel takes half of an SM's, and two do share an SM (start times of 296 such CTAs: all at once).
template <int DG>
long long resident_ctas(int ks, size_t smem, int sms) {
  static int cache[64][9] = {};
  const int per_sm = DG == 1 ? 2 : 1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (ks == 1 || dev < 0 || dev >= 64) return (long long)sms * per_sm;
  if (cache[dev][ks] == 0) {
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ks * sms));
    cfg.blockDim = dim3(gemm_threads<DG>());
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (gemm_attr<DG, false>() != 0 || cudaOccupancyMaxActiveClusters(&n, gemm_kernel<DG, false>, &cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = sms / ks;                                              // no answer (no device): assume perfect packing
    }
    cache[dev][ks] = n;
  }
  return (long long)cache[dev][ks] * ks * per_sm;
}

// rings for a token tile of NT
void gemm_rings(GemmPlan& p) {
  const size_t xt = (size_t)p.NT * 128;
  const size_t stg = (size_t)p.NT * 128 * 4;                      // the parked accumulator tile reuses the rings
  const size_t slack = 1024 /* alignment */ + 512 /* barriers */;
  const int acc = (p.NT + 31) & ~31;
  p.DG = p.NT <= 128 ? 1 : 2;
  p.tmem_cols = p.DG == 1 ? 256 : 512;
  const size_t budget = (p.DG == 1 ? 112 : 216) * 1024 - slack;
  p.astages = (p.tmem_cols - acc) / (PAIR * A_COLS);
  if (p.astages > 4) p.astages = 4;
  if (p.DG == 2) p.astages &= ~1;                                 // slot parity: see the kernel
  // activation tiles: enough to cover the L2 latency (four if they fit beside two record slots); the rest of the shared
  // memory goes to the record ring, which covers the HBM latency
  p.xstages = 4;
  while (p.xstages > 2 && p.xstages * xt + 2 * RAW_SLOT > budget) --p.xstages;
  p.rstages = (int)((budget - p.xstages * xt) / RAW_SLOT);
  if (p.rstages > 6) p.rstages = 6;
  if (p.DG == 2) p.rstages &= ~1;
  p.xstages = (int)((budget - (size_t)p.rstages * RAW_SLOT) / xt);
  if (p.xstages > 6) p.xstages = 6;
  size_t ring = p.xstages * xt + (size_t)p.rstages * RAW_SLOT;
  if (ring < stg) ring = stg;
  ring = (ring + 15) & ~(size_t)15;
  p.bar_off = (int)ring;
  p.smem = ring + slack;
}

constexpr int NT_MAX = 320;                                      // 320 accumulator columns + 4 weight tiles of 32 fill TMEM

GemmPlan gemm_plan(long long M, int NG, long long B, double& us) {
  GemmPlan p;
  // the fewest token tiles (every tile decodes the records again), of equal width
  p.TT = (int)((B + NT_MAX - 1) / NT_MAX);
  p.NT = (int)(((B + p.TT - 1) / p.TT + 15) & ~15);               // MMA widths: multiples of 16
  p.RB = (int)(M / 128);
  const int sms = st::sm_count();
  gemm_rings(p);
  // Split of the k range = cluster size (<= 8): the least estimated time in us, fitted to launches of the four projection
  // shapes of a 4096 / 12288 model (and 12288, 3072, 2048 x 2048) in a graph (16 to 192 row blocks, 16 to 304 tokens, splits 1 to
  // 8; within 15 %):
  //   start-up + drain, the epilogue (grows with the tiles to add through distributed shared memory), and per pair of
  //   k-tiles a time that grows with the CTAs that stream at once (two per SM) or with the token tile (one per SM).
  // A grid larger than the CTAs that are resident at once runs in waves.
  const int pairs = (NG + PAIR - 1) / PAIR, ksmax = pairs / 4 < 1 ? 1 : (pairs / 4 > 8 ? 8 : pairs / 4);
  auto estimate = [&](int rows, int ks) {
    const double ctas = (double)rows * p.TT * ks;
    const double slots = (double)(p.DG == 1 ? resident_ctas<1>(ks, p.smem, sms) : resident_ctas<2>(ks, p.smem, sms));
    if (slots <= 0) return 1e30;
    const double waves = ctas <= slots ? 1.0 : (double)(long long)((ctas + slots - 1) / slots);
    const double per_cta = (double)((pairs + ks - 1) / ks), load = ctas < slots ? ctas : slots;
    if (p.DG == 1) return waves * (per_cta * (0.45 + 0.0024 * load) * (1.0 + 0.0015 * (p.NT - 16)) + 3.0 + 0.3 * ks * p.NT / 64.0);
    const double pair = 0.785 * p.NT / 304.0 > 0.5 ? 0.785 * p.NT / 304.0 : 0.5;
    return waves * (per_cta * (pair + 0.1 * load / sms) + 6.0 + 0.3 * ks * p.NT / 64.0);
  };
  auto best_split = [&](int rows, double& t) {
    int best = 1;
    t = 1e30;
    for (int ks = 1; ks <= ksmax; ++ks) {
#ifdef ST_TUNE                                                   // development builds may force a split
      if (const char* f = getenv("STATETREE_GEMM_KS")) if (atoi(f) > 0 && atoi(f) != ks) continue;
#endif
      const double e = estimate(rows, ks);
      if (e < t - 1e-9) { t = e; best = ks; }
    }
    return best;
  };
  p.KS = best_split(p.RB, us);
  p.RB1 = 0;
  p.KS1 = 1;
  // One CTA per SM: a last wave that is nearly empty costs as much as a full one (192 row blocks at 300 tokens: 148 + 44).
  // Then the full waves go out unsplit and the rest of the row blocks in a second launch with a split of its own.  (One token tile:
  // with several of them CTA pairs were ahead of such a form at 780 of 790 sizes.)
  if (p.DG == 2 && p.TT == 1 && p.RB > sms) {
    const int rows1 = p.RB / sms * sms;
    double rest;
    if (rows1 < p.RB) {
      const int ks2 = best_split(p.RB - rows1, rest);
      const double both = estimate(rows1, 1) + rest + 1.0;
      if (both < us) { p.RB1 = rows1; p.KS1 = 1; p.KS = ks2; us = both; }
    }
  }
  // One CTA per SM: what the plan is expected to take next to CTA pairs.  The same terms, fitted so that the ratio of the two kernels'
  // times is met at 3900 sizes (8 to 296 row blocks, 1024 to 12288 columns, 129 to 2000 tokens): within 4 %, standard deviation.
  // Up to half of the SMs, the next launch's CTAs start beside this one's.
  if (p.DG == 2) {
    auto expected = [&](int rows, int ks) {
      const double ctas = (double)rows * p.TT * ks, slots = (double)resident_ctas<2>(ks, p.smem, sms);
      const double waves = (double)(long long)((ctas + slots - 1) / slots), part = (ctas < slots ? ctas : slots) / sms;
      const double per_cta = (double)((pairs + ks - 1) / ks), split = ks > 1 ? 0.91 + 0.159 * ks * p.NT / 64.0 : 0.0;
      return -3.25 + 2.2 * part + (part > 0.5 ? 0.77 : 0.0) + waves * (per_cta * (0.332 + 0.0019 * p.NT + 0.156 * part) + 5.97 + split);
    };
    us = expected(p.RB - p.RB1, p.KS) + (p.RB1 > 0 ? expected(p.RB1, p.KS1) + 4.4 : 0.0);
  }
  return p;
}

template <int DG, bool GROUPED>
int gemm_launch(const GemmPlan& p, const GemmArgs& a, const CUtensorMap& xmap, const WMaps& wmaps, cudaStream_t stream) {
  if (int e = gemm_attr<DG, GROUPED>()) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.RB * p.TT * p.KS));
  cfg.blockDim = dim3(gemm_threads<DG>());
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)p.KS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = st::pdl_enabled() ? 2 : 1;
  return st::cuda_fail(cudaLaunchKernelEx(&cfg, gemm_kernel<DG, GROUPED>, a, xmap, wmaps),
                       GROUPED ? "st_moe_group_gemm launch" : "st_gemm launch");
}
void plan_args(GemmArgs& a, const GemmPlan& p) {
  a.NT = p.NT; a.KS = p.KS; a.RB = p.RB; a.TT = p.TT;
  a.astages = p.astages; a.xstages = p.xstages; a.rstages = p.rstages; a.bar_off = p.bar_off; a.tmem_cols = p.tmem_cols;
}

// one matrix or a list (a names them, B, the rows of all members as M, NG and the status word)
int dense_gemm(GemmArgs& a, const WMaps& wmaps, const void* X, const char* who, cudaStream_t stream) {
  ST_REQUIRE(a.M / 128 * 8 * ((a.B + NT_MAX - 1) / NT_MAX) < (1ll << 31), "%s: grid too large", who);
  double us;
  const GemmPlan plan = gemm_plan(a.M, a.NG, a.B, us);
  // More than 128 tokens: CTA pairs where they are expected to be the faster ones.  Measured, us, this kernel / CTA pairs:
  //   2048 x 2048   at 300 tokens 11.2 / 10.1, 321 11.1 / 12.7        4096 x 4096   at 300 17.5 / 20.2, 321 19.0 / 20.4
  //   4608 x 3584   at 321 18.2 / 22.3, 900 32.4 / 29.7               4096 x 12288  at 300 32.3 / 42.1
  //   6144 x 4096   at 321 28.2 / 24.8                                4608 x 12288  at 512 56.9 / 77.0
  // Few row blocks split over up to eight CTAs here and over up to four pairs there, of which fifteen find room at once; with many
  // tiles a pair halves the activations' part of the shared-memory traffic.  Two launches here (between full waves of one token tile)
  // stay unless pairs are an eighth faster: tests/test_gpu_weights.py expects them of 192 row blocks of 2048 columns, where pairs in
  // one launch take 27.1 us against 30.5 at 136 tokens.
  if (plan.DG == 2) {
    const int done = pair_gemm(a, wmaps, X, who, (plan.RB1 > 0 ? 0.88 : 0.98) * us, stream);
    if (done >= 0) return done;
  }
  CUtensorMap xmap;
  if (int e = make_xmap(&xmap, X, a.B, (long long)a.NG * 64, plan.NT > 256 ? plan.NT / 2 : plan.NT, who)) return e;
  GemmPlan p = plan;
  auto go = [&] {
    plan_args(a, p);
    return p.DG == 1 ? gemm_launch<1, false>(p, a, xmap, wmaps, stream) : gemm_launch<2, false>(p, a, xmap, wmaps, stream);
  };
  a.rb0 = 0;
  if (plan.RB1 > 0) {
    p.RB = plan.RB1;
    p.KS = plan.KS1;
    if (int e = go()) return e;
    p.RB = plan.RB - plan.RB1;
    p.KS = plan.KS;
    a.rb0 = plan.RB1;
  }
  return go();
}

// a tree [M/16][N/64][1552 B] as 194 x u64 rows, boxes of eight row tiles of two column groups
int make_wmap(CUtensorMap* map, const void* tree, long long M, long long N, const char* who) {
  EncodeTiledFn enc = encode_fn();
  ST_REQUIRE(enc != nullptr, "%s: cuTensorMapEncodeTiled is not available from the driver", who);
  const cuuint64_t wd[3] = {194u, (cuuint64_t)(N / 64), (cuuint64_t)(M / 16)};
  const cuuint64_t wst[2] = {(cuuint64_t)REC, (cuuint64_t)(N / 64) * REC};
  const cuuint32_t wbox[3] = {194u, (cuuint32_t)PAIR, 8u};
  const cuuint32_t we[3] = {1u, 1u, 1u};
  const CUresult wr = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, const_cast<void*>(tree), wd, wst, wbox, we,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  ST_REQUIRE(wr == CUDA_SUCCESS, "%s: cuTensorMapEncodeTiled (tree) failed (%d)", who, (int)wr);
  return 0;
}

}  // namespace

// activations [rows, N] BF16 as boxes of 64 columns x `box_rows` rows with the 128-byte swizzle
int st::make_xmap(CUtensorMap* map, const void* X, long long rows, long long N, int box_rows, const char* who) {
  EncodeTiledFn enc = encode_fn();
  ST_REQUIRE(enc != nullptr, "%s: cuTensorMapEncodeTiled is not available from the driver", who);
  const cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)N * 2};
  const cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1u, 1u};
  const CUresult cr = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(X), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  ST_REQUIRE(cr == CUDA_SUCCESS, "%s: cuTensorMapEncodeTiled failed (%d)", who, (int)cr);
  return 0;
}

extern "C" int64_t st_gemm_workspace_bytes(int64_t M, int64_t N, int64_t B) {
  if (M <= 0 || N <= 0 || M % 128 || N % 64 || B < 1) return -1;
  return 0;                                                      // split partial sums stay in shared memory
}

extern "C" int st_gemm(const void* tree, const int32_t* eo, const uint32_t* el, const void* X, void* Y, float* Yf32,
                       int64_t B, int64_t M, int64_t N, void* ws, int64_t ws_bytes, int32_t* cnt, void* stream) {
  ST_REQUIRE(M > 0 && N > 0 && M % 128 == 0 && N % 64 == 0,
             "st_gemm: M %% 128 and N %% 64 must be 0 (got %lld x %lld)", (long long)M, (long long)N);
  ST_REQUIRE(B >= 1 && B < (1ll << 24), "st_gemm: batch out of range");
  ST_REQUIRE(tree && eo && el && X && Y && cnt, "st_gemm: null pointer");
  ST_REQUIRE(st::aligned16(tree) && st::aligned16(X), "st_gemm: tree and X must be 16-byte aligned");
  (void)ws; (void)ws_bytes;
  WMaps wmaps;
  memset(&wmaps, 0, sizeof(wmaps));
  if (int e = make_wmap(&wmaps.m[0], tree, M, N, "st_gemm")) return e;
  GemmArgs a = {};
  a.eo = eo; a.el = el; a.Y = (uint16_t*)Y; a.Yf = Yf32;
  a.status = st::status_ptr();
  ST_REQUIRE(a.status != nullptr, "st_gemm: no device status word");
  a.M = M; a.B = (int)B; a.NG = (int)(N / 64);
  return dense_gemm(a, wmaps, X, "st_gemm", (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------------------- list of matrices
extern "C" int st_gemm_list(int64_t n, const void* const* trees, const int32_t* const* eo, const uint32_t* const* el,
                            const void* X, void* const* Y, float* const* Yf32, int64_t B, const int64_t* M, int64_t N,
                            int32_t* cnt, void* stream) {
  const char* who = "st_gemm_list";
  ST_REQUIRE(n >= 1 && n <= MAXL, "%s: 1 to %d matrices per call (got %lld)", who, MAXL, (long long)n);
  ST_REQUIRE(trees && eo && el && X && Y && M && cnt, "%s: null pointer", who);
  ST_REQUIRE(N > 0 && N % 64 == 0, "%s: N %% 64 must be 0", who);
  ST_REQUIRE(B >= 1 && B < (1ll << 24), "%s: batch out of range", who);
  ST_REQUIRE(st::aligned16(X), "%s: X must be 16-byte aligned", who);
  GemmArgs a = {};
  WMaps wmaps;
  memset(&wmaps, 0, sizeof(wmaps));
  long long total = 0;
  for (int i = 0; i < (int)n; ++i) {
    ST_REQUIRE(trees[i] && eo[i] && el[i] && Y[i], "%s: null pointer in member %d", who, i);
    ST_REQUIRE(st::aligned16(trees[i]), "%s: tree of member %d must be 16-byte aligned", who, i);
    ST_REQUIRE(M[i] > 0 && M[i] % 128 == 0, "%s: rows of member %d must be a positive multiple of 128", who, i);
    if (int e = make_wmap(&wmaps.m[i], trees[i], M[i], N, who)) return e;
    a.leo[i] = eo[i]; a.lel[i] = el[i]; a.lY[i] = (uint16_t*)Y[i]; a.lYf[i] = Yf32 ? Yf32[i] : nullptr; a.lM[i] = M[i];
    total += M[i];
    a.rbend[i] = (int)(total / 128);
  }
  a.nlist = (int)n;
  a.eo = eo[0]; a.el = el[0]; a.Y = (uint16_t*)Y[0];
  a.status = st::status_ptr();
  ST_REQUIRE(a.status != nullptr, "%s: no device status word", who);
  a.M = total; a.B = (int)B; a.NG = (int)(N / 64);
  return dense_gemm(a, wmaps, X, who, (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------------------------- grouped (MoE)
extern "C" int64_t st_moe_tensor_map_bytes(void) { return (int64_t)sizeof(CUtensorMap); }

extern "C" int st_moe_tensor_maps(const int64_t* trees_host, int64_t E, int64_t M, int64_t N, void* maps_dev,
                                  void* stream) {
  ST_REQUIRE(E >= 1 && E <= 4096 && M > 0 && N > 0 && M % 128 == 0 && N % 64 == 0,
             "st_moe_tensor_maps: 1..4096 experts of M %% 128 == 0 rows and N %% 64 == 0 columns");
  ST_REQUIRE(trees_host && maps_dev && ((uintptr_t)maps_dev & 63u) == 0, "st_moe_tensor_maps: null or unaligned pointer");
  static thread_local CUtensorMap staging[4096];
  for (int64_t e = 0; e < E; ++e) {
    const void* tree = reinterpret_cast<const void*>(trees_host[e]);
    ST_REQUIRE(tree != nullptr && st::aligned16(tree), "st_moe_tensor_maps: tree %lld is null or unaligned", (long long)e);
    if (int r = make_wmap(&staging[e], tree, M, N, "st_moe_tensor_maps")) return r;
  }
  // pageable source: the copy is staged by the driver before the call returns, so `staging` may be reused at once
  return st::cuda_fail(cudaMemcpyAsync(maps_dev, staging, (size_t)E * sizeof(CUtensorMap), cudaMemcpyHostToDevice,
                                       (cudaStream_t)stream), "st_moe_tensor_maps: copy");
}

extern "C" int st_moe_group_gemm(const void* maps, const int64_t* eop, const int64_t* elp, int64_t E, const void* Xg,
                                 const int32_t* sorted, const int32_t* bexp, const int32_t* npost, int64_t nblk,
                                 int64_t bs, void* Y, float* Yf32, int64_t S, int64_t M, int64_t N, void* stream) {
  ST_REQUIRE(M > 0 && N > 0 && M % 128 == 0 && N % 64 == 0, "st_moe_group_gemm: M %% 128 and N %% 64 must be 0");
  ST_REQUIRE(bs == 64 || bs == 128, "st_moe_group_gemm: block size must be 64 or 128 (got %lld)", (long long)bs);
  ST_REQUIRE(E >= 1 && S >= 0 && nblk >= 0, "st_moe_group_gemm: sizes");
  if (S == 0 || nblk == 0) return 0;
  ST_REQUIRE(maps && eop && elp && Xg && sorted && bexp && npost && Y, "st_moe_group_gemm: null pointer");
  ST_REQUIRE(((uintptr_t)maps & 63u) == 0 && st::aligned16(Xg), "st_moe_group_gemm: maps 64-byte, Xg 16-byte aligned");
  GemmPlan p;
  p.NT = (int)bs;
  p.TT = (int)nblk;
  p.RB = (int)(M / 128);
  p.KS = 1;
  gemm_rings(p);
  ST_REQUIRE((long long)p.RB * p.TT < (1ll << 31), "st_moe_group_gemm: grid too large");
  CUtensorMap xmap;
  WMaps unused;
  if (int e = make_xmap(&xmap, Xg, nblk * bs, N, XBOX_GROUPED, "st_moe_group_gemm")) return e;
  memset(&unused, 0, sizeof(unused));
  GemmArgs a = {};
  a.Y = (uint16_t*)Y; a.Yf = Yf32;
  a.maps = reinterpret_cast<const CUtensorMap*>(maps); a.eop = (const long long*)eop; a.elp = (const long long*)elp;
  a.sorted = sorted; a.bexp = bexp; a.npost = npost; a.E = (int)E;
  a.status = st::status_ptr();
  ST_REQUIRE(a.status != nullptr, "st_moe_group_gemm: no device status word");
  a.M = M; a.B = (int)S; a.NG = (int)(N / 64);
  plan_args(a, p);
  return gemm_launch<1, true>(p, a, xmap, unused, (cudaStream_t)stream);
}
