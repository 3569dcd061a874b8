// Streaming trellis GEMM for decode widths (1..64 activation rows) on sm_100a.
//
//   raw[rows][cols] = A[rows][k] (fp16, prepared beforehand in global memory)  x  W'[k][cols] (EXL3 tiles, decoded in
//   registers)
//
// One CTA = 8 consumer warps + 1 producer warp and is persistent over a list of work units. A unit is a block of
// <= 8 output tiles (128 columns) x a run of k-tiles of one matrix. The producer moves the compressed tiles with ONE tiled
// TMA copy per ring stage (a 3-D tensor map over the trellis: x = bytes along the tile row, y = k-tile, z = expert; box =
// 8 tiles x SG_KS k-tiles) and the unit's A rows with 1-D bulk copies into one of a few A slots, always one unit ahead
// of the tiles; completion is signalled on mbarriers by transaction count. It runs ahead across unit boundaries, so HBM
// stays busy and the consumers never wait for an operand that could have been fetched earlier. The producer warp shares
// its scheduler with consumer warps that are always ready to issue, so every instruction it needs per stage delays the
// stream: one copy instruction per stage (instead of one per k-tile) is what keeps the ring full. Each consumer warp owns one output tile:
// per k-tile it reads its lane window (3 words) from the ring, decodes 8 weights per lane, rounds them with two
// constant-matrix MMAs and issues one mma.m16n8k16 per 8 activation rows; accumulators are fp32 registers. Only compressed bytes cross HBM.
//
// The "problem" type P supplies the unit list and the operand / result addresses:
//   bool P::units_final() const                        // the unit list does not depend on the preceding kernel's output
//   int  P::num_units() const
//   Unit P::unit(int u) const                         // where the tiles are, how many k-steps, K, rows, ...
//   const CUtensorMap *P::tmap(int i) const            // tensor map i over a trellis (see make_trellis_map)
//   int  P::row_index(const Unit&, int i) const       // which operand / result row the unit's i-th row is
//   const __half *P::a_row(const Unit&, int idx) const  // global address of that row's first element of the unit's k range
//   float *P::out_base(const Unit&) const               // raw output of the unit: element (row idx, unit column c) is
//   int P::out_row_off(const Unit&, int idx) const      //   out_base(un)[out_row_off(un, idx) + c]
#pragma once
#include <cuda.h>

#include "exl3_decode.cuh"
#include "pipeline.cuh"

namespace ijah {

#ifndef SG_KS_STEPS
#define SG_KS_STEPS 16
#endif
#ifndef SG_CTAS_PER_SM
#define SG_CTAS_PER_SM 2
#endif
constexpr int SG_WARPS = 8;               // consumer warps = output tiles per unit
constexpr int SG_THREADS = 32 * (SG_WARPS + 1);
constexpr int SG_KS = SG_KS_STEPS;        // k-steps per ring stage
constexpr int SG_CTAS = SG_CTAS_PER_SM;   // persistent CTAs per SM
constexpr int SG_MAX_STAGES = 16;
constexpr int SG_MAX_ASLOTS = 4;
constexpr int SG_DESC_UNIT_BYTES = 128;   // shared-memory room for one unit descriptor
constexpr int SG_DESC_BYTES = SG_DESC_UNIT_BYTES + 64 * 4;  // + the row indices of up to 64 rows

struct UnitBase {
  int map;             // which of the problem's tensor maps (P::tmap) holds the unit's tiles
  int x, y, z;         // box coordinates of the unit's first stage: x in 8-byte elements (= n0 * 4K), y = first k-tile, z = expert
  int kc;              // k-tiles in this unit
  int ntiles;          // output tiles (1..8)
  int K;               // bits per weight
  int nrows;           // live activation rows (<= 8 * MT)
};

// What the consumer warps need of a unit; the producer writes it into the unit's A slot together with one output row
// offset per activation row, so the consumers never touch the unit list nor do any address arithmetic beyond one add.
struct UnitDesc {
  float *out;
  int kc, ntiles, K, nrows;
};

struct StreamLayout {  // dynamic shared memory carve-up (host computes, kernel mirrors)
  int stages;          // ring stages
  int stage_bytes;     // SG_KS * 8 * 32 * Kmax
  int lda;             // A row stride in halfs (16 per k-tile + 8 pad: keeps ldmatrix rows on distinct banks)
  int arows;           // rows per A slot
  int aslots;          // A slots (units the producer may run ahead)
  __host__ __device__ size_t ring_off() const { return 512 + SG_MAX_ASLOTS * SG_DESC_BYTES; }
  __host__ __device__ size_t slot_bytes() const { return (size_t)arows * lda * 2; }
  __host__ __device__ size_t a_off() const { return ring_off() + (size_t)stages * stage_bytes; }
  __host__ __device__ size_t total() const { return a_off() + (size_t)aslots * slot_bytes() + 64; }  // (the last row's fragment load may cover one k-tile more)
};

// shared-memory loads with the constant part of the address as an immediate (no address arithmetic per tile)
template <int OFF>
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(addr), "n"(OFF));
  return v;
}
template <int OFF>
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4+%5];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr), "n"(OFF));
}

// Two k-tiles (I and I + 1 of a stage) for one output tile. The tensor core computes D^T = W'^T * X^T: the decoded tile is the
// A operand (16 output columns x 16 k), the activations are the B operand (16 k x 8 rows), one ldmatrix.x4 for both k-tiles.
// The codebook function yields every weight as a pair of fp16 summands (lo, hi) in one register (dec8_raw).
//   EX (default): two constant-matrix MMAs per tile (round_pairs) round and pack the lane's 8 pairs into the tile's A fragment of
//                 fp16(lo + hi), the weights as the format defines them; one MMA per 8 rows multiplies them.
//   !EX (opt-in): the pairs are multiplied as they are: a pair takes the place of two k elements, against (v, v) made from
//                 the activation fragment, so a tile takes two MMAs (even inputs: slots 0, 4, 2, 6; odd: 1, 5, 3, 7) and the
//                 accumulator receives lo * v + hi * v, the sum of the summands unrounded.
// MT = number of 8-row groups (1, 2, 4, 8); a_row[g] is the ldmatrix address of row group g for k-tile 0 of the stage,
// tile I sits I * 32 bytes further in the A rows. acc[g] = D^T fragment of group g: (column gq, rows 2q, 2q+1), (column gq + 8, ..).
// The loop is bound by instruction issue and the half-rate integer pipe, the tensor pipe has room (35 % busy): K5, block of 64
// rows, gate / up launch: one half add per weight and (w, w) against (v, 0) pairs in doubled activation rows took 54.8
// instructions per tile and 340 us, rounding on the tensor core takes 44.7 and 301 us (both under ncu).
constexpr uint32_t SG_A_TILE_BYTES = 16 * 2;  // one k-tile of one prepared activation row

// (v, v) of both halves of an activation fragment register
__device__ __forceinline__ uint32_t dup_lo(uint32_t v) { return __byte_perm(v, 0u, 0x1010); }
__device__ __forceinline__ uint32_t dup_hi(uint32_t v) { return __byte_perm(v, 0u, 0x3232); }

template <bool EX>
__device__ __forceinline__ void tile_frag(const uint32_t (&r)[8], const PairSum &ps, uint32_t (&f)[EX ? 4 : 8]) {
  if constexpr (EX) {
    uint32_t lo[2], hi[2];  // k 0-7 and k 8-15 of the fragment
    round_pairs(lo, r[0], r[4], r[1], r[5], ps);
    round_pairs(hi, r[2], r[6], r[3], r[7], ps);
    f[0] = lo[0]; f[1] = lo[1]; f[2] = hi[0]; f[3] = hi[1];
  } else {
    f[0] = r[0]; f[1] = r[4]; f[2] = r[2]; f[3] = r[6];
    f[4] = r[1]; f[5] = r[5]; f[6] = r[3]; f[7] = r[7];
  }
}
template <bool EX>
__device__ __forceinline__ void tile_mma(float (&acc)[4], const uint32_t (&f)[EX ? 4 : 8], uint32_t x0, uint32_t x1) {
  if constexpr (EX) {
    mma_16816(acc, f, x0, x1);
  } else {
    const uint32_t even[4] = {f[0], f[1], f[2], f[3]}, odd[4] = {f[4], f[5], f[6], f[7]};
    mma_16816(acc, even, dup_lo(x0), dup_lo(x1));
    mma_16816(acc, odd, dup_hi(x0), dup_hi(x1));
  }
}

template <int K, bool EX, int MT, int I>
__device__ __forceinline__ void pair_mma(const uint32_t (&wa)[3], const uint32_t (&wb)[3], uint32_t la, const McgConst &mc, const PairSum &ps,
                                         const uint32_t (&a_row)[MT], float (&acc)[MT][4]) {
  uint32_t r[8], fa[EX ? 4 : 8], fb[EX ? 4 : 8];
  dec8_raw<K>(wa[0], wa[1], wa[2], la, mc, r);
  tile_frag<EX>(r, ps, fa);
  dec8_raw<K>(wb[0], wb[1], wb[2], la, mc, r);
  tile_frag<EX>(r, ps, fb);
#pragma unroll
  for (int g = 0; g < MT; g++) {
    uint32_t x[4];
    ldsm4<I * (int)SG_A_TILE_BYTES>(x, a_row[g]);
    tile_mma<EX>(acc[g], fa, x[0], x[1]);
    tile_mma<EX>(acc[g], fb, x[2], x[3]);
  }
}
// Groups of SG_HALF k-tiles starting at tile B: all window words are loaded first (3 * SG_HALF independent shared loads in
// flight), then decoded and multiplied in pairs of tiles. Groups keep the window words at 12 registers; the other warps of
// the SM cover the shared-memory latency at the start of each group.
constexpr int SG_HALF = 4;
constexpr int SG_GROUPS = SG_KS / SG_HALF;

// the groups G .. of a full stage, one after the other
template <int K, bool EX, int MT, int G>
__device__ __forceinline__ void stage_groups(uint32_t p0, uint32_t p1, uint32_t p2, uint32_t la, const McgConst &mc, const PairSum &ps,
                                             const uint32_t (&a_row)[MT], float (&acc)[MT][4]) {
  if constexpr (G < SG_GROUPS) {
    constexpr int B = G * SG_HALF, KSTEP = SG_WARPS * Codec<K>::TILE_BYTES;
    static_assert(SG_HALF == 4, "two pairs of tiles per group");
    uint32_t w[SG_HALF][3];
    w[0][0] = lds32<(B + 0) * KSTEP>(p0); w[0][1] = lds32<(B + 0) * KSTEP>(p1); w[0][2] = lds32<(B + 0) * KSTEP>(p2);
    w[1][0] = lds32<(B + 1) * KSTEP>(p0); w[1][1] = lds32<(B + 1) * KSTEP>(p1); w[1][2] = lds32<(B + 1) * KSTEP>(p2);
    w[2][0] = lds32<(B + 2) * KSTEP>(p0); w[2][1] = lds32<(B + 2) * KSTEP>(p1); w[2][2] = lds32<(B + 2) * KSTEP>(p2);
    w[3][0] = lds32<(B + 3) * KSTEP>(p0); w[3][1] = lds32<(B + 3) * KSTEP>(p1); w[3][2] = lds32<(B + 3) * KSTEP>(p2);
    pair_mma<K, EX, MT, B>(w[0], w[1], la, mc, ps, a_row, acc);
    pair_mma<K, EX, MT, B + 2>(w[2], w[3], la, mc, ps, a_row, acc);
    stage_groups<K, EX, MT, G + 1>(p0, p1, p2, la, mc, ps, a_row, acc);
  }
}
// the n < SG_KS tiles of a short last stage, one at a time
template <int K, bool EX, int MT>
__device__ __forceinline__ void stage_tail(uint32_t p0, uint32_t p1, uint32_t p2, uint32_t la, const McgConst &mc, const PairSum &ps,
                                           const uint32_t (&a_row)[MT], float (&acc)[MT][4], int n) {
  constexpr uint32_t KSTEP = SG_WARPS * Codec<K>::TILE_BYTES;
#pragma unroll 1
  for (int i = 0; i < n; i++) {
    uint32_t r[8], f[EX ? 4 : 8];
    dec8_raw<K>(lds32<0>(p0 + i * KSTEP), lds32<0>(p1 + i * KSTEP), lds32<0>(p2 + i * KSTEP), la, mc, r);
    tile_frag<EX>(r, ps, f);
#pragma unroll
    for (int g = 0; g < MT; g++) {
      uint32_t x[4];
      ldsm4<0>(x, a_row[g] + i * SG_A_TILE_BYTES);
      tile_mma<EX>(acc[g], f, x[0], x[1]);
    }
  }
}

// The consumer side of the ring, all in registers: stage index and parity, the shared-memory addresses of the barriers
// (empty[s] sits SG_MAX_STAGES * 8 bytes after full[s]) and of the warp's tile inside stage 0.
struct RingCursor {
  uint32_t full;          // address of full[0]
  uint32_t tile0;         // address of this warp's tile of k-step 0 in stage 0
  uint32_t stage_bytes;
  uint32_t nstages, stage, phase;
  __device__ __forceinline__ void advance() {
    const uint32_t nx = stage + 1u, wrap = nx == nstages ? 1u : 0u;
    stage = wrap ? 0u : nx;
    phase ^= wrap;
  }
};
constexpr uint32_t SG_EMPTY_OFF = SG_MAX_STAGES * 8;

// All k-steps of one unit for one warp: 8 * MT activation rows, accumulators zeroed here, results stored to
// out[rowoff[row] + col]. Returns false if a bounded wait gave up. The steady-state loop (full stages of a live warp) is
// straight-line code between one wait and one arrive; a short last stage and the warps without a tile (units narrower
// than 8 tiles) take their own loops.
template <int K, bool EX, int MT>
__device__ __forceinline__ bool consume_unit(const UnitDesc &d, RingCursor &rc, bool live, int lane, const McgConst &mc, const PairSum &ps, uint32_t a_addr,
                                             uint32_t lda_bytes, const int *rowoff, int col, int *status) {
  const uint32_t lane0 = lane == 0 ? 1u : 0u;
  const int nfull = d.kc / SG_KS, rem = d.kc - nfull * SG_KS;
  if (!live) {
    for (int s = 0; s < nfull + (rem ? 1 : 0); s++) {
      const uint32_t bar = rc.full + rc.stage * 8u;
      if (!mbar_wait_poll(bar, rc.phase)) { atomicExch(status, 2); return false; }
      mbar_arrive_if(bar + SG_EMPTY_OFF, lane0);
      rc.advance();
    }
    return true;
  }
  float acc[MT][4];
#pragma unroll
  for (int m = 0; m < MT; m++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[m][j] = 0.0f;
  // ldmatrix.x4 row addresses of an 8-row group: lanes 8j .. 8j+7 give rows 0-7 at byte 16 j of a pair of k-tiles. A dead row (its results are never stored) reads the
  // unit's row 0 again: the same address as a live lane, i.e. a broadcast. (A separate zero row sat at the same offset
  // modulo 128 bytes as row 0 and cost every ldmatrix a two-way bank conflict: 4 of 14 load wavefronts per tile.)
  uint32_t a_row[MT];
  {
    const uint32_t lkof = (uint32_t)(lane >> 3) * 16u;
#pragma unroll
    for (int m = 0; m < MT; m++) {
      const int r = m * 8 + (lane & 7);
      a_row[m] = a_addr + (uint32_t)(r < d.nrows ? r : 0) * lda_bytes + lkof;
    }
  }
  const typename Codec<K>::Lane L = Codec<K>::lane(lane);
  const uint32_t d1 = L.o1 - L.o0, d2 = L.o2 - L.o0, t0 = rc.tile0 + L.o0;
  for (int s = 0; s < nfull; s++) {
    const uint32_t bar = rc.full + rc.stage * 8u;
    if (!mbar_wait_poll(bar, rc.phase)) { atomicExch(status, 2); return false; }
    const uint32_t p0 = t0 + rc.stage * rc.stage_bytes, p1 = p0 + d1, p2 = p0 + d2;
    stage_groups<K, EX, MT, 0>(p0, p1, p2, L.a, mc, ps, a_row, acc);
#pragma unroll
    for (int m = 0; m < MT; m++) a_row[m] += SG_KS * SG_A_TILE_BYTES;
    __syncwarp();
    mbar_arrive_if(bar + SG_EMPTY_OFF, lane0);
    rc.advance();
  }
  if (rem) {  // a short last stage
    const uint32_t bar = rc.full + rc.stage * 8u;
    if (!mbar_wait_poll(bar, rc.phase)) { atomicExch(status, 2); return false; }
    const uint32_t p0 = t0 + rc.stage * rc.stage_bytes, p1 = p0 + d1, p2 = p0 + d2;
    stage_tail<K, EX, MT>(p0, p1, p2, L.a, mc, ps, a_row, acc, rem);
    __syncwarp();
    mbar_arrive_if(bar + SG_EMPTY_OFF, lane0);
    rc.advance();
  }
  const int q = lane & 3;
#pragma unroll
  for (int m = 0; m < MT; m++) {
    const int r0 = m * 8 + 2 * q;
    if (r0 < d.nrows) {
      float *o = d.out + rowoff[r0] + col;
      o[0] = acc[m][0];
      o[8] = acc[m][2];
    }
    if (r0 + 1 < d.nrows) {
      float *o = d.out + rowoff[r0 + 1] + col;
      o[0] = acc[m][1];
      o[8] = acc[m][3];
    }
  }
  return true;
}

template <bool EX, int MT>
__device__ __forceinline__ bool consume_any(const UnitDesc &d, RingCursor &rc, bool live, int warp, int lane, const McgConst &mc, const PairSum &ps, uint32_t a_addr,
                                            uint32_t lda_bytes, const int *rowoff, int col, int *status) {
  const uint32_t ring0 = rc.tile0;  // address of stage 0; the warp's tile offset depends on the unit's K
#define SG_CASE(KK)                                                                                              \
  case KK: {                                                                                                     \
    rc.tile0 = ring0 + (uint32_t)warp * Codec<KK>::TILE_BYTES;                                                   \
    const bool ok = consume_unit<KK, EX, MT>(d, rc, live, lane, mc, ps, a_addr, lda_bytes, rowoff, col, status); \
    rc.tile0 = ring0;                                                                                            \
    return ok;                                                                                                   \
  }
  switch (d.K) {
    SG_CASE(4)
    SG_CASE(5)
    SG_CASE(6)
    SG_CASE(7)
    default:
      SG_CASE(8)
  }
#undef SG_CASE
}

template <class P, int MT, bool EX>
__global__ void __launch_bounds__(SG_THREADS, SG_CTAS) stream_gemm_kernel(const __grid_constant__ P prob, const StreamLayout lay, int *status) {
  static_assert(sizeof(UnitDesc) <= SG_DESC_UNIT_BYTES, "unit descriptor too large for its shared-memory slot");
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t *full = reinterpret_cast<uint64_t *>(smem);
  uint64_t *empty = full + SG_MAX_STAGES;
  uint64_t *a_full = empty + SG_MAX_STAGES;
  uint64_t *a_empty = a_full + SG_MAX_ASLOTS;
  unsigned char *desc = smem + 512;  // per A slot: the unit descriptor, then the output row offsets of its rows
  unsigned char *ring = smem + lay.ring_off();
  unsigned char *aslot = smem + lay.a_off();

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < lay.stages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], SG_WARPS);
    }
    for (int s = 0; s < lay.aslots; s++) {
      mbar_init(&a_full[s], 1);
      mbar_init(&a_empty[s], SG_WARPS);
    }
    mbar_fence_init();
  }
  __syncthreads();

  if (warp == SG_WARPS) {
    // ---------------------------------------------------------------- producer (one warp)
    // Only this warp reads the unit list from global memory; the consumers get each unit's descriptor and output row
    // offsets through shared memory together with the A rows, so no consumer ever waits on a global load. Per ring stage
    // the producer executes one wait, one expect_tx and ONE tensor copy (lane 0); per unit, one unit AHEAD of the tiles it
    // is streaming, the descriptor and one bulk copy per activation row (lane i copies row i).
    //
    // Start-up under programmatic dependent launch: the A rows (and for some problems the unit list itself) are written
    // by the preceding kernel, the compressed weights are not. A problem whose unit list is final when the kernel is
    // launched (P::units_final()) streams the first unit's weight stages into the fresh ring before it waits for
    // the predecessor, so the ring is full when the A rows arrive.
    pdl_launch();  // the successor's CTAs only take resources this grid has released; they wait for its completion themselves
    uint32_t stage = 0, phase = 0;
    int slot = 0;
    uint32_t aphase = 0;
    int u = blockIdx.x;
    typename P::Unit un;
    int nunits = 0, k_pre = 0;
    const uint64_t wpol = l2_evict_first_policy();
    const uint32_t full_a = smem_u32(full), ring_a = smem_u32(ring), nstages = (uint32_t)lay.stages;
    // one stage of unit `t`, k-tiles [k, k + SG_KS): the box is always full size (what lies beyond the unit, the matrix or
    // its last column tile is zero-filled or simply not used), so the byte count depends on K only
    auto issue_stage = [&](const typename P::Unit &t, int k) {
      if (lane == 0) {
        const uint32_t bar = full_a + stage * 8u;
        mbar_arrive_expect_tx_a(bar, (uint32_t)(SG_KS * SG_WARPS * 32) * (uint32_t)t.K);
        tma_load_3d(ring_a + stage * (uint32_t)lay.stage_bytes, prob.tmap(t.map), t.x, t.y + k, t.z, bar, wpol);
      }
      if (++stage == nstages) { stage = 0; phase ^= 1u; }
    };
    // descriptor, output row offsets and A rows of unit `t` into the next A slot
    auto issue_rows = [&](const typename P::Unit &t) -> bool {
      const int i0 = lane < t.nrows ? prob.row_index(t, lane) : 0;
      const int i1 = lane + 32 < t.nrows ? prob.row_index(t, lane + 32) : 0;
      if (!mbar_wait(&a_empty[slot], aphase ^ 1u, status, 3)) return false;
      UnitDesc *du = reinterpret_cast<UnitDesc *>(desc + (size_t)slot * SG_DESC_BYTES);
      int *doff = reinterpret_cast<int *>(desc + (size_t)slot * SG_DESC_BYTES + SG_DESC_UNIT_BYTES);
      doff[lane] = lane < t.nrows ? prob.out_row_off(t, i0) : 0;
      doff[lane + 32] = lane + 32 < t.nrows ? prob.out_row_off(t, i1) : 0;
      const uint32_t rowb = (uint32_t)t.kc * SG_A_TILE_BYTES;
      __syncwarp();
      if (lane == 0) {
        *du = UnitDesc{prob.out_base(t), t.kc, t.ntiles, t.K, t.nrows};
        mbar_arrive_expect_tx(&a_full[slot], (uint32_t)t.nrows * rowb);  // release: descriptor and offsets are visible
      }
      __syncwarp();
      unsigned char *adst = aslot + (size_t)slot * lay.slot_bytes();
      if (lane < t.nrows) bulk_g2s(adst + (size_t)lane * lay.lda * 2, prob.a_row(t, i0), rowb, &a_full[slot]);
      if (lane + 32 < t.nrows) bulk_g2s(adst + (size_t)(lane + 32) * lay.lda * 2, prob.a_row(t, i1), rowb, &a_full[slot]);
      if (++slot == lay.aslots) { slot = 0; aphase ^= 1u; }
      return true;
    };
    if (prob.units_final()) {
      nunits = prob.num_units();
      if (u < nunits) {
        un = prob.unit(u);
        for (; k_pre < un.kc && k_pre < SG_KS * lay.stages; k_pre += SG_KS) issue_stage(un, k_pre);  // fresh ring: no empty-wait needed
      }
      pdl_wait();
    } else {
      pdl_wait();
      nunits = prob.num_units();
      if (u < nunits) un = prob.unit(u);
    }
    if (u < nunits && !issue_rows(un)) return;
    while (u < nunits) {
      const int u_next = u + gridDim.x;
      typename P::Unit nx;
      if (u_next < nunits) {  // the next unit's rows go out before this unit's remaining tiles: they arrive stages early
        nx = prob.unit(u_next);
        if (!issue_rows(nx)) return;
      }
      for (int k = k_pre; k < un.kc; k += SG_KS) {
#ifdef SG_PRODUCER_SLEEP_NS
        if (!mbar_wait_sleep(&empty[stage], phase ^ 1u, status, 1, SG_PRODUCER_SLEEP_NS)) return;
#else
        if (!mbar_wait(&empty[stage], phase ^ 1u, status, 1)) return;
#endif
        issue_stage(un, k);
      }
      k_pre = 0;
      un = nx;
      u = u_next;
    }
    return;
  }

  // ------------------------------------------------------------------ consumers (8 warps)
  RingCursor rc;
  rc.full = smem_u32(full); rc.tile0 = smem_u32(ring);
  rc.stage_bytes = (uint32_t)lay.stage_bytes; rc.nstages = (uint32_t)lay.stages; rc.stage = 0u; rc.phase = 0u;
  int slot = 0;
  uint32_t aphase = 0;
  const uint32_t a0_addr = smem_u32(aslot), slot_bytes = (uint32_t)lay.slot_bytes(), lda_bytes = (uint32_t)lay.lda * 2u;
  const uint32_t afull_a = smem_u32(a_full), aempty_a = smem_u32(a_empty);
  const McgConst mc = McgConst::load();
  const PairSum ps = PairSum::make(lane);
  const int col = warp * 16 + (lane >> 2);

  if (!prob.units_final()) pdl_wait();  // the unit count is the predecessor's output
  const int nunits = prob.num_units();
  for (int u = blockIdx.x; u < nunits; u += gridDim.x) {
    if (!mbar_wait_a(afull_a + (uint32_t)slot * 8u, aphase, status, 4)) return;
    const UnitDesc d = *reinterpret_cast<const UnitDesc *>(desc + (size_t)slot * SG_DESC_BYTES);
    const int *rowoff = reinterpret_cast<const int *>(desc + (size_t)slot * SG_DESC_BYTES + SG_DESC_UNIT_BYTES);
    if (!consume_any<EX, MT>(d, rc, warp < d.ntiles, warp, lane, mc, ps, a0_addr + (uint32_t)slot * slot_bytes, lda_bytes, rowoff, col, status))
      return;
    // the stores above read the slot's row offsets: only now may it be refilled
    __syncwarp();
    if (lane == 0) mbar_arrive_a(aempty_a + (uint32_t)slot * 8u);
    if (++slot == lay.aslots) { slot = 0; aphase ^= 1u; }
  }
}

}  // namespace ijah
