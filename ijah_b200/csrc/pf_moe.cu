// Prefill MoE kernels. See pf_moe.cuh.
#include <algorithm>

#include "common.hpp"
#include "exl3_decode.cuh"
#include "pf_moe.cuh"
#include "stream_gemm.cuh"
#include "umma.cuh"

namespace ijah {

// =============================================================================================== grouped trellis GEMM
// out[pos][col] = sum_k act[pos][k] * W'_e[k][col] for one work item = (expert, <= 256 sorted rows, 256 output columns).
//
// The contraction runs on the 5th-generation tensor core with the rows as M = 128 and all 256 columns as N, K = 16 per
// instruction; the accumulator of 128 rows is one half of TMEM. An item of at most 128 rows takes one half, so the epilogue of
// one item overlaps the MMAs of the next; an item of more rows takes both and multiplies every decoded weight with both groups
// of rows. One CTA per SM, warp-specialised:
//   warp 0        weights: two tiled TMA copies per stage (4 k-tiles x 2 x 8 column tiles) into the ring
//   warp 1        issues tcgen05.mma (one thread) when a stage's decoded weights and activations are present
//   warps 2-5     epilogue: tcgen05.ld the accumulators, store the live rows
//   warps 6-29    decoders, three groups of eight: a group takes every third stage; each of its warps decodes two column tiles
//                 of the stage's k-tiles with the same register decode as the decode-width kernels and writes fp16 into the
//                 MMA's shared-memory layout
//   warp 30       activations: one bulk copy per stage and group of 128 rows (the operands are stored stage by stage)
// so every expert tile is decoded once per 256 rows instead of once per 16/32-row window. The two kinds of copies have warps of
// their own because each must run as far ahead as its own buffers allow.
// What bounds it is the latency of one decoder's way through a stage, not a pipe: with sixteen decoders of four tiles per stage
// (cycle counters, 8 rows) a stage took 2016 cycles, 1154 of them decoding, the rest waits, fence and arrivals, at 36 % of the
// issue slots. Twenty-four decoders that pass the barriers once per eight tiles keep more work in flight (prefill block of
// 333 tokens 1211 -> 1154 us); with the decode taken out of a copy the block took 874 us, with the MMAs 975: both sides are close. Warp 1 shares its
// scheduler with them, so each of its instructions costs several times its issue slot (634 cycles for eight MMAs with M = 128
// columns): hence N = 256, descriptors that are one addition away from the last and all barriers of a stage polled at once by
// different lanes. The warps that mostly wait sleep between polls.
constexpr int PG_KS = 4;                      // k-tiles per stage
constexpr int PG_RING_MAX = 8;                // compressed-tile stages (as many as fit)
constexpr int PG_A = 3;                       // decoded-weight stages = decoder groups
constexpr int PG_B = 4;                       // activation slots (128 rows of one stage)
constexpr int PG_DW = 8;                      // decoder warps per group; PG_A groups: group g fills decoded stage g
constexpr int PG_THREADS = 32 * (7 + PG_A * PG_DW);
constexpr int PG_A_STAGE = PG_KS * 2 * 4096;  // [ks][khalf][32 groups of 8 columns][128 B]
constexpr int PG_B_SLOT = 16 * 1024;          // [row group][8 k-chunks][128 B]

struct PgGemm {
  alignas(64) CUtensorMap w_routed[2], w_shared[2];  // trellises per projection: boxes of 8 column tiles x PG_KS k-tiles
  const PfItem *items;
  const int *nitems;
  const __half *act[2];                   // blocked activations per projection
  float *out[2];                          // output base per projection; element (pos, col) at out + pos * ldo + col
  int ldo, in, IT, OT, Kx, Ks;
  int groups;                             // 8-row groups of the blocked operands
  int ring;                               // ring stages
};

struct PgSmem {
  uint64_t ring_full[PG_RING_MAX], ring_empty[PG_RING_MAX];
  uint64_t a_full[PG_A], a_empty[PG_A];
  uint64_t b_full[PG_B], b_empty[PG_B];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
};

// A decoder warp's view of the two rings: its group's next ring stage, the parities of that and of the group's decoded stage
struct PgCursor {
  uint32_t rs, rph, aph;
};

// The stages first, first + PG_A, .. of one item for one decoder warp (column tiles dw and dw + 8): straight-line code for one
// K, so that the lane's constants of the other four do not compete for registers (with the choice of K inside the stage loop
// they spilled).
template <int K>
__device__ __forceinline__ bool pg_decode_item(const PgSmem *sm, uint32_t ring, uint32_t ring_stage_bytes, uint32_t nring, uint32_t abuf, int group,
                                               PgCursor &cu, int first, int nst, int dw, int lane, int *status) {
  const typename Codec<K>::Lane L = Codec<K>::lane(lane);
  const McgConst mc = McgConst::load();
  const PairSum ps = PairSum::make(lane);
  constexpr int KSTEP = 8 * Codec<K>::TILE_BYTES;  // a ring stage is two boxes [k-tile][8 column tiles]
  const uint32_t tile0 = ring + (uint32_t)(dw * Codec<K>::TILE_BYTES) + L.o0, d1 = L.o1 - L.o0, d2 = L.o2 - L.o0;
  // lane (q, c) = (lane & 3, lane >> 2) writes k (2q, 2q + 1) and (2q + 8, 2q + 9) of columns c and c + 8
  const uint32_t dst = abuf + (uint32_t)(group * PG_A_STAGE + dw * 256 + lane * 4);
  const uint32_t bars = smem_u32(sm);
  const uint32_t rfull = bars + (uint32_t)offsetof(PgSmem, ring_full), rempty = bars + (uint32_t)offsetof(PgSmem, ring_empty);
  const uint32_t afull = bars + (uint32_t)offsetof(PgSmem, a_full) + group * 8u, aempty = bars + (uint32_t)offsetof(PgSmem, a_empty) + group * 8u;
  const uint32_t lane0 = lane == 0 ? 1u : 0u;
  const bool odd = lane & 1;
#pragma unroll 1
  for (int st = first; st < nst; st += PG_A) {
    // even lanes wait for the tiles, odd ones for the place to write to: one latency for both
    if (!__all_sync(0xFFFFFFFFu, mbar_wait_a(odd ? aempty : rfull + cu.rs * 8u, odd ? cu.aph ^ 1u : cu.rph, status, 17))) return false;
    __syncwarp();
    static_assert(PG_KS == 4, "four k-tiles per stage");
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t p0 = tile0 + cu.rs * ring_stage_bytes + h * PG_KS * KSTEP, p1 = p0 + d1, p2 = p0 + d2;
      uint32_t w[4][3];
      w[0][0] = lds32<0 * KSTEP>(p0); w[0][1] = lds32<0 * KSTEP>(p1); w[0][2] = lds32<0 * KSTEP>(p2);
      w[1][0] = lds32<1 * KSTEP>(p0); w[1][1] = lds32<1 * KSTEP>(p1); w[1][2] = lds32<1 * KSTEP>(p2);
      w[2][0] = lds32<2 * KSTEP>(p0); w[2][1] = lds32<2 * KSTEP>(p1); w[2][2] = lds32<2 * KSTEP>(p2);
      w[3][0] = lds32<3 * KSTEP>(p0); w[3][1] = lds32<3 * KSTEP>(p1); w[3][2] = lds32<3 * KSTEP>(p2);
#pragma unroll
      for (int ks = 0; ks < PG_KS; ks++) {
        uint32_t r[8], lo[2], hi[2];
        dec8_raw<K>(w[ks][0], w[ks][1], w[ks][2], L.a, mc, r);
        round_pairs(lo, r[0], r[4], r[1], r[5], ps);
        round_pairs(hi, r[2], r[6], r[3], r[7], ps);
        const uint32_t d = dst + ks * 8192 + h * 2048;  // (the offsets below are immediates)
        asm volatile(
            "st.shared.u32 [%0], %1;\n\tst.shared.u32 [%0+4096], %2;\n\tst.shared.u32 [%0+128], %3;\n\tst.shared.u32 [%0+4224], %4;"
            ::"r"(d), "r"(lo[0]), "r"(hi[0]), "r"(lo[1]), "r"(hi[1])
            : "memory");
      }
    }
    fence_proxy_async_smem();  // the tensor core reads what these ordinary stores wrote
    __syncwarp();
    mbar_arrive_if(afull, lane0);
    mbar_arrive_if(rempty + cu.rs * 8u, lane0);
    cu.rs += PG_A;
    if (cu.rs >= nring) { cu.rs -= nring; cu.rph ^= 1u; }
    cu.aph ^= 1u;
  }
  return true;
}

__global__ void __launch_bounds__(PG_THREADS, 1) pf_gemm_kernel(const __grid_constant__ PgGemm g, int *status) {
  extern __shared__ __align__(1024) unsigned char pf_smem[];
  unsigned char *smem = pf_smem;
  PgSmem *sm = reinterpret_cast<PgSmem *>(smem);
  const int ring_stage_bytes = PG_KS * 16 * 32 * max(g.Kx, g.Ks);
  unsigned char *abuf = smem + 1024;
  unsigned char *bbuf = abuf + (size_t)PG_A * PG_A_STAGE;
  unsigned char *ring = bbuf + (size_t)PG_B * PG_B_SLOT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < g.ring; s++) { mbar_init(&sm->ring_full[s], 1); mbar_init(&sm->ring_empty[s], PG_DW); }
    for (int s = 0; s < PG_A; s++) { mbar_init(&sm->a_full[s], PG_DW); mbar_init(&sm->a_empty[s], 1); }
    for (int s = 0; s < PG_B; s++) { mbar_init(&sm->b_full[s], 1); mbar_init(&sm->b_empty[s], 1); }
    for (int b = 0; b < 2; b++) { mbar_init(&sm->acc_full[b], 1); mbar_init(&sm->acc_empty[b], 4); }
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(&sm->tmem_base, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sm->tmem_base;
  const int nitems = *g.nitems;
  const int nst = g.IT / PG_KS;

  if (warp == 0) {
    // ------------------------------------------------------------------------------------------ weights
    int rs = 0;
    uint32_t rph = 0;
    const uint64_t pol = l2_evict_first_policy();
    const uint32_t ring_a = smem_u32(ring);
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
      const int expert = g.items[it].expert, proj = g.items[it].proj, ngpair = g.items[it].ngpair;
      const int K = expert < 0 ? g.Ks : g.Kx, x0 = ngpair * 16 * 4 * K;
      const CUtensorMap *map = expert < 0 ? &g.w_shared[proj] : &g.w_routed[proj];
      const uint32_t box = (uint32_t)(PG_KS * 8 * 32) * (uint32_t)K;
      for (int st = 0; st < nst; st++) {
        if (!mbar_wait_sleep(&sm->ring_empty[rs], rph ^ 1u, status, 11, 40)) goto out;
        if (lane == 0) {
          const uint32_t bar = smem_u32(&sm->ring_full[rs]), dst = ring_a + (uint32_t)(rs * ring_stage_bytes);
          mbar_arrive_expect_tx_a(bar, 2u * box);
          tma_load_3d(dst, map, x0, st * PG_KS, max(expert, 0), bar, pol);
          tma_load_3d(dst + box, map, x0 + 8 * 4 * K, st * PG_KS, max(expert, 0), bar, pol);
        }
        __syncwarp();
        if (++rs == g.ring) { rs = 0; rph ^= 1u; }
      }
    }
  } else if (warp == 6 + PG_A * PG_DW) {
    // ------------------------------------------------------------------------------------------ activations
    int bs = 0;
    uint32_t bph = 0;
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
      const int row0 = g.items[it].row0, nrows = g.items[it].nrows;
      const __half *act = g.act[g.items[it].proj] + (size_t)(row0 >> 3) * 512;
      for (int st = 0; st < nst; st++)
        for (int r0 = 0; r0 < nrows; r0 += PF_NTOK) {
          if (!mbar_wait_sleep(&sm->b_empty[bs], bph ^ 1u, status, 12, 40)) goto out;
          if (lane == 0) {
            const uint32_t bytes = (uint32_t)((min(PF_NTOK, nrows - r0) + 7) >> 3) * 1024u;
            mbar_arrive_expect_tx(&sm->b_full[bs], bytes);
            bulk_g2s(bbuf + (size_t)bs * PG_B_SLOT, act + ((size_t)st * g.groups + (r0 >> 3)) * 512, bytes, &sm->b_full[bs]);
          }
          __syncwarp();
          if (++bs == PG_B) { bs = 0; bph ^= 1u; }
        }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------------------------------ MMA issuer
    int as = 0, bs = 0, half = 0;
    uint32_t aph = 0, bph = 0, cph[2] = {0, 0};
    const uint64_t w0 = umma_smem_desc(smem_u32(abuf), 4096, 128), x0 = umma_smem_desc(smem_u32(bbuf), 128, 1024);
    const uint32_t afull = smem_u32(&sm->a_full[0]), bfull = smem_u32(&sm->b_full[0]);
    constexpr uint32_t idesc = umma_idesc_f16(128, PF_NCOL);
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
      const int nsub = g.items[it].nrows > PF_NTOK ? 2 : 1;
      for (int s = 0; s < nsub; s++) {
        const int h = half ^ s;
        if (!mbar_wait(&sm->acc_empty[h], (h ? cph[1] : cph[0]) ^ 1u, status, 13)) goto out;
        if (h) cph[1] ^= 1u; else cph[0] ^= 1u;
      }
      for (int st = 0; st < nst; st++) {
        // lanes 0, 1, 2 (mod 4) poll the decoded weights and the activations of one or two groups of rows
        const int bs1 = bs + 1 == PG_B ? 0 : bs + 1;
        const uint32_t bph1 = bs + 1 == PG_B ? bph ^ 1u : bph;
        const int which = lane & 3;
        const uint32_t bar = which == 1 ? bfull + bs * 8u : which == 2 && nsub == 2 ? bfull + bs1 * 8u : afull + as * 8u;
        const uint32_t par = which == 1 ? bph : which == 2 && nsub == 2 ? bph1 : aph;
        if (!__all_sync(0xFFFFFFFFu, mbar_wait_a(bar, par, status, 14))) goto out;
        __syncwarp();
        tc_fence_after_sync();
        if (elect_one()) {
          const uint64_t wd = w0 + (uint32_t)as * (uint32_t)(PG_A_STAGE >> 4);
          uint64_t xd = x0 + (uint32_t)bs * (uint32_t)(PG_B_SLOT >> 4);
          uint32_t d = tmem + (uint32_t)half * 256u;
          umma_f16_ss(d, xd, wd, idesc, st > 0 ? 1u : 0u);
#pragma unroll
          for (int ks = 1; ks < PG_KS; ks++) umma_f16_ss(d, xd + ks * 16, wd + ks * 512, idesc, 1u);
          umma_commit(&sm->b_empty[bs]);  // a slot may be overwritten once these MMAs have read it
          if (nsub == 2) {
            if (st == nst - 1) umma_commit(&sm->acc_full[half]);
            xd = x0 + (uint32_t)bs1 * (uint32_t)(PG_B_SLOT >> 4);
            d = tmem + (uint32_t)(half ^ 1) * 256u;
            umma_f16_ss(d, xd, wd, idesc, st > 0 ? 1u : 0u);
#pragma unroll
            for (int ks = 1; ks < PG_KS; ks++) umma_f16_ss(d, xd + ks * 16, wd + ks * 512, idesc, 1u);
            umma_commit(&sm->b_empty[bs1]);
          }
          umma_commit(&sm->a_empty[as]);
          if (st == nst - 1) umma_commit(&sm->acc_full[half ^ (nsub - 1)]);
        }
        __syncwarp();
        for (int s = 0; s < nsub; s++)
          if (++bs == PG_B) { bs = 0; bph ^= 1u; }
        if (++as == PG_A) { as = 0; aph ^= 1u; }
      }
      half ^= nsub & 1;
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------------------------------------ epilogue
    const int qd = warp & 3;  // TMEM lanes 32 qd .. 32 qd + 31 are this warp's
    int half = 0;
    uint32_t cph[2] = {0, 0};
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
      const int proj = g.items[it].proj, ngpair = g.items[it].ngpair, row0 = g.items[it].row0, nall = g.items[it].nrows;
      for (int r0 = 0; r0 < nall; r0 += PF_NTOK) {
        if (!mbar_wait_sleep(&sm->acc_full[half], half ? cph[1] : cph[0], status, 16, 200)) goto out;
        if (half) cph[1] ^= 1u; else cph[0] ^= 1u;
        tc_fence_after_sync();
        const int row = r0 + qd * 32 + lane;  // TMEM lane = row, column = column
        if (r0 + qd * 32 < nall) {
          float *o = g.out[proj] + (size_t)(row0 + row) * g.ldo + ngpair * PF_NCOL;
#pragma unroll 1
          for (int c0 = 0; c0 < PF_NCOL; c0 += 32) {
            uint32_t r[32];
            tmem_ld_32x32(tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)half * 256u + (uint32_t)c0, r);
            if (row < nall) {
#pragma unroll
              for (int j = 0; j < 8; j++)
                reinterpret_cast<uint4 *>(o + c0)[j] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
            }
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm->acc_empty[half]);
        half ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------------------------------------ decoders
    const int group = (warp - 6) / PG_DW, dw = (warp - 6) % PG_DW;
    PgCursor cu{(uint32_t)group, 0u, 0u};
    int first = group;  // the group's first stage of the item: the stages of all items are dealt to the groups in turn
    const uint32_t ring_a = smem_u32(ring), abuf_a = smem_u32(abuf), rsb = (uint32_t)ring_stage_bytes, nr = (uint32_t)g.ring;
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
      const int K = g.items[it].expert < 0 ? g.Ks : g.Kx;
      bool ok;
      switch (K) {
        case 4: ok = pg_decode_item<4>(sm, ring_a, rsb, nr, abuf_a, group, cu, first, nst, dw, lane, status); break;
        case 5: ok = pg_decode_item<5>(sm, ring_a, rsb, nr, abuf_a, group, cu, first, nst, dw, lane, status); break;
        case 6: ok = pg_decode_item<6>(sm, ring_a, rsb, nr, abuf_a, group, cu, first, nst, dw, lane, status); break;
        case 7: ok = pg_decode_item<7>(sm, ring_a, rsb, nr, abuf_a, group, cu, first, nst, dw, lane, status); break;
        default: ok = pg_decode_item<8>(sm, ring_a, rsb, nr, abuf_a, group, cu, first, nst, dw, lane, status); break;
      }
      if (!ok) break;
      first -= nst % PG_A;  // (stage nst + x of this item is stage x of the next)
      if (first < 0) first += PG_A;
    }
  }
out:
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

static void launch_pf_gemm(PgGemm &g, int *status, cudaStream_t st) {
  IJ_CHECK(g.IT % PG_KS == 0 && g.OT % 16 == 0 && g.in % 64 == 0, "prefill GEMM needs in %% 64 == 0 and out %% 256 == 0 (in %d, out %d)", g.in, g.OT * 16);
  const size_t fixed = 1024 + (size_t)PG_A * PG_A_STAGE + (size_t)PG_B * PG_B_SLOT, stage = (size_t)PG_KS * 16 * 32 * std::max(g.Kx, g.Ks);
  g.ring = (int)std::min<size_t>(PG_RING_MAX, (226 * 1024 - fixed) / stage);  // 6 at K5, 4 at K8 (at least PG_A: a group's stages are PG_A apart)
  IJ_CUDA(cudaFuncSetAttribute(pf_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));  // per device: every launch
  pf_gemm_kernel<<<sm_count(), PG_THREADS, fixed + g.ring * stage, st>>>(g, status);
  IJ_CUDA(cudaGetLastError());
}

// (the routing, sorting, operand and finishing kernels follow)

// =============================================================================================== router
// logits[n][0 .. E) = x . W^T (bf16 W, f32 x) on tensor cores without giving up f32 accuracy: x is split into three bf16
// terms (x = hi + mid + lo to 2^-24), each multiplied with the bf16 weights by mma.sync.m16n8k16 (products exact, f32
// accumulate). 128 tokens x 128 experts per CTA, 8 warps of 32 x 64, k in steps of 32 through double-buffered shared
// memory (rows padded to 80 bytes: conflict-free ldmatrix). Reference: the router GEMM of the chunked prefill
// (kernels/prefill/pf_gemm.metal:159-186). The shared expert's gate logit (column E) is a plain dot product in
// pf_route_kernel.
constexpr int LG_T = 128, LG_K = 32, LG_LD = LG_K + 8;              // halfs per staged row
constexpr int LG_PLANE = LG_T * LG_LD, LG_BUF = 4 * LG_PLANE;       // x hi, mid, lo, W
constexpr int LG_SMEM = 2 * LG_BUF * 2;                             // bytes
constexpr int LG_SPLITS = 8;                                        // most k-splits

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t bf16_rn_bits(float v) {
  const uint32_t u = __float_as_uint(v);
  return (u + 0x7FFFu + ((u >> 16) & 1u)) >> 16;
}
// (a, b) -> packed bf16 pairs of the three terms
__device__ __forceinline__ void split3(float a, float b, uint32_t &hi, uint32_t &mid, uint32_t &lo) {
  const uint32_t ah = bf16_rn_bits(a), bh = bf16_rn_bits(b);
  const float a1 = a - __uint_as_float(ah << 16), b1 = b - __uint_as_float(bh << 16);
  const uint32_t am = bf16_rn_bits(a1), bm = bf16_rn_bits(b1);
  const float a2 = a1 - __uint_as_float(am << 16), b2 = b1 - __uint_as_float(bm << 16);
  hi = ah | (bh << 16);
  mid = am | (bm << 16);
  lo = bf16_rn_bits(a2) | (bf16_rn_bits(b2) << 16);
}

__global__ void __launch_bounds__(256) pf_logits_kernel(const PfParams p, float *part, int nk) {
  extern __shared__ __align__(16) unsigned char lg_smem[];
  uint16_t *sm = reinterpret_cast<uint16_t *>(lg_smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t0 = blockIdx.x * LG_T, c0 = blockIdx.y * LG_T, H = p.H;
  const int k_first = blockIdx.z * nk * LG_K;  // this split's first input
  const int wm = warp >> 1, wn = warp & 1;  // warp tile: tokens 32 wm .. +31, experts 64 wn .. +63
  // loads. x: thread -> rows (tid >> 3) + 32 j, floats 4 (tid & 7) .. +3; W: rows (tid >> 2) + 64 j, 16-byte chunk tid & 3
  const int xr = tid >> 3, xc = (tid & 7) * 4, wr = tid >> 2, wc = (tid & 3) * 8;
  const float *xsrc[4];
  const uint16_t *wsrc[2];
#pragma unroll
  for (int j = 0; j < 4; j++) xsrc[j] = p.x + (size_t)min(t0 + xr + 32 * j, p.n - 1) * H + k_first + xc;
#pragma unroll
  for (int j = 0; j < 2; j++) wsrc[j] = p.router + (size_t)min(c0 + wr + 64 * j, p.E - 1) * H + k_first + wc;
  float4 xv[4];
  auto load_x = [&](int ks) {
#pragma unroll
    for (int j = 0; j < 4; j++) xv[j] = *reinterpret_cast<const float4 *>(xsrc[j] + ks * LG_K);
  };
  auto load_w = [&](int ks, int buf) {
    const uint32_t dst = smem_u32(sm + buf * LG_BUF + 3 * LG_PLANE);
#pragma unroll
    for (int j = 0; j < 2; j++)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (uint32_t)(((wr + 64 * j) * LG_LD + wc) * 2)), "l"(wsrc[j] + ks * LG_K) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto stash_x = [&](int buf) {
    uint16_t *b = sm + buf * LG_BUF;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      uint32_t h0, m0, l0, h1, m1, l1;
      split3(xv[j].x, xv[j].y, h0, m0, l0);
      split3(xv[j].z, xv[j].w, h1, m1, l1);
      const int o = (xr + 32 * j) * LG_LD + xc;
      *reinterpret_cast<uint2 *>(b + o) = make_uint2(h0, h1);
      *reinterpret_cast<uint2 *>(b + LG_PLANE + o) = make_uint2(m0, m1);
      *reinterpret_cast<uint2 *>(b + 2 * LG_PLANE + o) = make_uint2(l0, l1);
    }
  };
  float acc[2][8][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[i][j][q] = 0.0f;
  load_x(0);
  load_w(0, 0);
  stash_x(0);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // ldmatrix lane offsets (in halfs): A rows (lane & 15), k half (lane >> 4); B rows (lane & 7) + 8 ((lane >> 4) & 1), k half (lane >> 3) & 1
  const int a_off = (32 * wm + (lane & 15)) * LG_LD + (lane >> 4) * 8;
  const int b_off = (64 * wn + (lane & 7) + ((lane >> 4) & 1) * 8) * LG_LD + ((lane >> 3) & 1) * 8;
  nk = min(nk, (H - k_first) / LG_K);
  for (int ks = 0; ks < nk; ks++) {
    const int buf = ks & 1;
    if (ks + 1 < nk) {
      load_x(ks + 1);
      load_w(ks + 1, buf ^ 1);  // that buffer was last read one step ago, before the barrier below
    }
    const uint32_t base = smem_u32(sm + buf * LG_BUF);
#pragma unroll
    for (int kk = 0; kk < LG_K; kk += 16) {
      uint32_t bfr[4][4];  // per pair of expert tiles: b0, b1 of tile 2 j, b0, b1 of tile 2 j + 1
#pragma unroll
      for (int j = 0; j < 4; j++) ldmatrix_x4(bfr[j], base + (uint32_t)((3 * LG_PLANE + b_off + j * 16 * LG_LD + kk) * 2));
#pragma unroll
      for (int t = 0; t < 3; t++) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
          uint32_t afr[4];
          ldmatrix_x4(afr, base + (uint32_t)((t * LG_PLANE + a_off + i * 16 * LG_LD + kk) * 2));
#pragma unroll
          for (int j = 0; j < 4; j++) {
            mma_bf16_16816(acc[i][2 * j], afr, bfr[j][0], bfr[j][1]);
            mma_bf16_16816(acc[i][2 * j + 1], afr, bfr[j][2], bfr[j][3]);
          }
        }
      }
    }
    if (ks + 1 < nk) {
      stash_x(buf ^ 1);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
  }
  const int g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int hh = 0; hh < 2; hh++) {
      const int t = t0 + 32 * wm + 16 * i + g + 8 * hh;
      if (t >= p.n) continue;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int c = c0 + 64 * wn + 8 * j + 2 * q;
        float *dst = part + ((size_t)blockIdx.z * p.n + t) * (p.E + 1) + c;
        if (c < p.E) dst[0] = acc[i][j][2 * hh];
        if (c + 1 < p.E) dst[1] = acc[i][j][2 * hh + 1];
      }
    }
}

// top-k on the logits (ties -> lowest index), weights = softmax over the k selected; one warp per token
__global__ void __launch_bounds__(256) pf_route_kernel(const PfParams p, const float *part, int nsplit) {
  __shared__ float sl[8][1024];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = blockIdx.x * 8 + warp;
  if (t >= p.n) return;
  float *s = sl[warp];
  const int E = p.E, k = p.topk;
  if (nsplit == 1) {
    for (int i = lane; i < E; i += 32) s[i] = p.logits[(size_t)t * (E + 1) + i];
  } else {  // the router GEMM's k-splits, added in their order
    for (int i = lane; i < E; i += 32) {
      float v[LG_SPLITS];
#pragma unroll
      for (int j = 0; j < LG_SPLITS; j++) v[j] = j < nsplit ? part[((size_t)j * p.n + t) * (E + 1) + i] : 0.0f;
#pragma unroll
      for (int j = 1; j < LG_SPLITS; j++) v[0] += v[j];
      s[i] = v[0];
      p.logits[(size_t)t * (E + 1) + i] = v[0];
    }
  }
  if (p.has_shared) {  // the shared expert's gate logit: x[t] . w_sg
    float g = 0.0f;
    for (int i = lane * 8; i < p.H; i += 256) {
      const float4 a = *reinterpret_cast<const float4 *>(p.x + (size_t)t * p.H + i), b = *reinterpret_cast<const float4 *>(p.x + (size_t)t * p.H + i + 4);
      const uint4 u = *reinterpret_cast<const uint4 *>(p.sgate + i);
      g += a.x * __uint_as_float(u.x << 16) + a.y * __uint_as_float(u.x & 0xFFFF0000u) + a.z * __uint_as_float(u.y << 16) +
           a.w * __uint_as_float(u.y & 0xFFFF0000u) + b.x * __uint_as_float(u.z << 16) + b.y * __uint_as_float(u.z & 0xFFFF0000u) +
           b.z * __uint_as_float(u.w << 16) + b.w * __uint_as_float(u.w & 0xFFFF0000u);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xFFFFFFFFu, g, o);
    if (lane == 0) p.logits[(size_t)t * (E + 1) + E] = g;
  }
  __syncwarp();
  float myv = 0.0f, top = 0.0f;
  int myi = 0;
  for (int r = 0; r < k; r++) {
    float best = -INFINITY;
    int bi = 0x7FFFFFFF;
    for (int i = lane; i < E; i += 32) {
      const float v = s[i];
      if (v > best || bi == 0x7FFFFFFF) { best = v; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xFFFFFFFFu, best, o);
      const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, o);
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (r == 0) top = best;
    if (lane == r) { myv = best; myi = bi; }
    if ((bi & 31) == lane) s[bi] = -INFINITY;
    __syncwarp();
  }
  float pr = lane < k ? expf(myv - top) : 0.0f, sum = pr;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
  if (lane < k) {
    p.route[(size_t)t * 2 * k + lane] = (uint32_t)myi;
    p.route[(size_t)t * 2 * k + k + lane] = __float_as_uint(pr / sum);
  }
}

// =============================================================================================== sort by expert
// Deterministic counting sort of the n * topk slots by expert (reference kernels/prefill/pf_moe.metal:29-83), three passes:
//   pf_hist_kernel   one warp per block of PS_BLOCK consecutive slots: per-expert counts of the block
//   pf_scan_kernel   per expert, exclusive scan of the counts over the blocks (a warp per expert); then one CTA lays out
//                    the experts' position ranges (padded to 8 rows, the granule of the blocked operand layout) and
//                    writes the work items
//   pf_place_kernel  the same warps walk their block in slot order: rank of a slot among its expert's slots = the block's
//                    base + earlier equals in the block (warp match), position = expert offset + rank
constexpr int PS_BLOCK = 256;
__global__ void __launch_bounds__(32) pf_hist_kernel(const PfParams p, int *hist) {
  __shared__ int cnt[1024];
  const int b = blockIdx.x, lane = threadIdx.x, k = p.topk;
  for (int e = lane; e < p.E; e += 32) cnt[e] = 0;
  __syncwarp();
  for (int i = lane; i < PS_BLOCK; i += 32) {
    const int s = b * PS_BLOCK + i;
    if (s < p.S) {
      const int e = (int)p.route[(size_t)(s / k) * 2 * k + s % k];
      if (e >= p.e0 && e < p.e0 + p.ecount) atomicAdd(&cnt[e], 1);  // slots of experts held elsewhere are not placed
    }
  }
  __syncwarp();
  for (int e = lane; e < p.E; e += 32) hist[(size_t)b * p.E + e] = cnt[e];
}

// hist[b][e] -> exclusive scan over b (in place), cnt[e] = total; one warp per expert
__global__ void __launch_bounds__(256) pf_blockscan_kernel(const PfParams p, int *hist, int nb) {
  const int e = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (e >= p.E) return;
  int run = 0;
  for (int b0 = 0; b0 < nb; b0 += 32) {
    const int b = b0 + lane, v = b < nb ? hist[(size_t)b * p.E + e] : 0;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xFFFFFFFFu, inc, o);
      if (lane >= o) inc += a;
    }
    if (b < nb) hist[(size_t)b * p.E + e] = run + inc - v;
    run += __shfl_sync(0xFFFFFFFFu, inc, 31);
  }
  if (lane == 0) p.cnt[e] = run;
}

__device__ __forceinline__ int block_excl_scan(int v, int *warp_tot, int *total) {  // blockDim = 1024, all threads call
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int s = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xFFFFFFFFu, s, o);
    if (lane >= o) s += a;
  }
  __syncthreads();
  if (lane == 31) warp_tot[warp] = s;
  __syncthreads();
  if (warp == 0) {
    int t = warp_tot[lane], ts = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xFFFFFFFFu, ts, o);
      if (lane >= o) ts += a;
    }
    warp_tot[lane] = ts - t;
    if (lane == 31) *total = ts;
  }
  __syncthreads();
  return warp_tot[warp] + s - v;
}

__global__ void __launch_bounds__(1024) pf_scan_kernel(const PfParams p) {
  __shared__ int wt[32], tot8, totp;
  __shared__ int s_pb[1024], s_off[1024], s_cnt[1024];
  const int e = threadIdx.x, E = p.E;
  const int c = e < E ? p.cnt[e] : 0, c8 = (c + 7) & ~7, np = (c + PF_PASS - 1) / PF_PASS;
  const int o = block_excl_scan(c8, wt, &tot8);
  const int pb = block_excl_scan(np, wt, &totp);
  if (e < E) p.off[e] = o;
  s_pb[e] = e < E ? pb : 0x7FFFFFFF;
  s_off[e] = o;
  s_cnt[e] = c;
  const int nsh = p.has_shared ? p.sh_rows : 0, shp = (nsh + PF_PASS - 1) / PF_PASS;
  if (e == 0) {
    p.off[E] = tot8;
    p.off[E + 1] = tot8 + ((nsh + 7) & ~7);
    p.nitems[0] = (totp + shp) * 2 * (p.I / PF_NCOL);
    p.nitems[1] = (totp + shp) * (p.H / PF_NCOL);
  }
  __syncthreads();
  // one thread per item (a thread that writes all items of a pass one after the other made this kernel 35 to 53 us long).
  // The expert of pass q is the last one whose first pass is <= q (experts without rows share the first-pass index of the
  // next expert that has some); passes beyond the routed ones are the shared expert's.
  auto pass_item = [&](int q, int proj, int ngpair) {
    if (q >= totp) {
      const int j = q - totp;
      return PfItem{-1, proj, ngpair, tot8 + j * PF_PASS, min(PF_PASS, nsh - j * PF_PASS), {0, 0, 0}};
    }
    int lo = 0, hi = 1024;  // first index with s_pb > q
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (s_pb[mid] <= q) lo = mid + 1; else hi = mid;
    }
    const int ex = lo - 1, j = q - s_pb[ex];
    return PfItem{ex - p.e0, proj, ngpair, s_off[ex] + j * PF_PASS, min(PF_PASS, s_cnt[ex] - j * PF_PASS), {0, 0, 0}};  // expert index into the local stacks
  };
  const int GU = p.I / PF_NCOL, DN = p.H / PF_NCOL;
  for (int i = threadIdx.x; i < (totp + shp) * 2 * GU; i += blockDim.x) {
    const int q = i / (2 * GU), j = i - q * 2 * GU;
    p.items_gu[i] = pass_item(q, j / GU, j % GU);
  }
  for (int i = threadIdx.x; i < (totp + shp) * DN; i += blockDim.x) p.items_d[i] = pass_item(i / DN, 0, i % DN);
}

// order[pos] = slot (S + t for the shared expert's row of token t, -1 = padding), inv[slot] = pos, seid[pos] = expert
// (E = shared). order / seid are pre-set to -1 by the launcher. Blocks 0 .. nb-1 place the routed slots, the rest the shared rows.
__global__ void __launch_bounds__(32) pf_place_kernel(const PfParams p, int *order, const int *hist, int nb) {
  __shared__ int base[1024];
  const int b = blockIdx.x, lane = threadIdx.x, k = p.topk;
  if (b >= nb) {
    if (!p.has_shared) return;
    for (int j = (b - nb) * PS_BLOCK + lane; j < min(p.sh_rows, (b - nb + 1) * PS_BLOCK); j += 32) {
      const int pos = p.off[p.E] + j;
      order[pos] = p.S + p.sh_row0 + j;
      p.seid[pos] = p.E;
    }
    return;
  }
  for (int e = lane; e < p.E; e += 32) base[e] = hist[(size_t)b * p.E + e] + p.off[e];
  __syncwarp();
  const uint32_t lt = (1u << lane) - 1u;
  for (int i = lane; i < PS_BLOCK; i += 32) {  // 32 consecutive slots per round, rounds in slot order
    const int s = b * PS_BLOCK + i;
    const int er = s < p.S ? (int)p.route[(size_t)(s / k) * 2 * k + s % k] : -1;
    const bool on = er >= p.e0 && er < p.e0 + p.ecount;
    if (s < p.S && !on) p.inv[s] = -1;
    const int e = on ? er : -1 - lane;
    const uint32_t same = __match_any_sync(0xFFFFFFFFu, e);
    if (on) {
      const int pos = base[e] + __popc(same & lt);
      order[pos] = s;
      p.inv[s] = pos;
      p.seid[pos] = e;
    }
    __syncwarp();
    if (on && (same & lt) == 0) base[e] += __popc(same);  // the first lane of each expert advances its base
    __syncwarp();
  }
}

// The elementwise kernels below give four lanes one 128-element chunk of a row (fwht128_quad) and a warp the same chunk of the
// eight rows of one row group of the blocked layout, whose rows all belong to one expert: what the warp writes of a core matrix
// is then 128 contiguous bytes without a detour through shared memory, and the scale vectors are one broadcast per warp.
// Prefill of 4096 tokens, Zipf routing: with one warp per row and 20 shuffles per chunk the three were bound by the shuffle pipe
// and took 199 + 115 + 137 us; now 153 + 111 + 120, about twice what their f32 partial results and operands take at the DRAM rate.
constexpr float PF_HS = 0.08838834764831845f;  // 1 / sqrt(128)

// v[4 i + j] = element 16 i + 4 l + j of the lane's chunk of an f32 row
__device__ __forceinline__ void quad_load(float (&v)[32], const float *chunk, int lane) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const float4 a = *reinterpret_cast<const float4 *>(chunk + 16 * i + 4 * (lane & 3));
    v[4 * i] = a.x; v[4 * i + 1] = a.y; v[4 * i + 2] = a.z; v[4 * i + 3] = a.w;
  }
}
// v *= the halfs of a scale vector's chunk, elements in the order of quad_load
__device__ __forceinline__ void quad_scale_in(float (&v)[32], const __half *chunk, int lane) {
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const uint2 h = *reinterpret_cast<const uint2 *>(chunk + 16 * i + 4 * (lane & 3));
    const float2 f0 = __half22float2(*reinterpret_cast<const __half2 *>(&h.x)), f1 = __half22float2(*reinterpret_cast<const __half2 *>(&h.y));
    v[4 * i] *= f0.x; v[4 * i + 1] *= f0.y; v[4 * i + 2] *= f1.x; v[4 * i + 3] *= f1.y;
  }
}
// v *= the halfs of a scale vector's chunk, 32 elements from quad_first(lane) on (the order after the transform)
__device__ __forceinline__ void quad_scale_out(float (&v)[32], const __half *chunk, int lane) {
  const uint4 *src = reinterpret_cast<const uint4 *>(chunk + quad_first(lane));
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const uint4 u = src[c];
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[j]));
      v[8 * c + 2 * j] *= f.x; v[8 * c + 2 * j + 1] *= f.y;
    }
  }
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}
// fp16(v) into a blocked operand of `groups` row groups: chunk `chunk` of position pos (a lane's run lies within one stage)
__device__ __forceinline__ void quad_store_blocked(const float (&v)[32], __half *base, int pos, int chunk, int lane, int groups) {
  __half *dst = base + blocked_index(pos, chunk * 128 + quad_first(lane), groups);
#pragma unroll
  for (int c = 0; c < 4; c++)
    *reinterpret_cast<uint4 *>(dst + 64 * c) = make_uint4(pack2(v[8 * c], v[8 * c + 1]), pack2(v[8 * c + 2], v[8 * c + 3]),
                                                         pack2(v[8 * c + 4], v[8 * c + 5]), pack2(v[8 * c + 6], v[8 * c + 7]));
}
__device__ __forceinline__ void quad_zero(float (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 32; j++) v[j] = 0.0f;
}

// gate / up operands: xh[pos] = fp16(H128(x[token(pos)] * suh[expert(pos)])) (reference kernels/prefill/pf_moe.metal:88-104);
// padding positions are written as zeros. One warp per (row group, PF_PREP_CHUNKS chunks): the rows' metadata is fetched once
// and a chunk's activations are on their way while the chunk before is transformed.
constexpr int PF_PREP_CHUNKS = 4;
__global__ void __launch_bounds__(256, 2) pf_prep_kernel(const PfParams p, const int *order) {
  const int lane = threadIdx.x & 31, H = p.H, nc = H / 128, runs = (nc + PF_PREP_CHUNKS - 1) / PF_PREP_CHUNKS;
  const int job = blockIdx.x * 8 + (threadIdx.x >> 5), group = job / runs, c0 = (job - group * runs) * PF_PREP_CHUNKS;
  if (group * 8 >= p.pos_cap) return;
  const int pos = group * 8 + (lane >> 2);  // pos_cap is a multiple of 8
  const int slot = pos < p.off[p.E + 1] ? order[pos] : -1;
  const bool shared = slot >= p.S;
  const int t = slot < 0 ? 0 : shared ? slot - p.S : slot / p.topk;
  const int e = (slot < 0 || shared) ? 0 : p.seid[pos] - p.e0;
  const __half *const sg = shared ? p.sgt.suh : p.gate.suh + (size_t)e * H, *const su = shared ? p.sup.suh : p.up.suh + (size_t)e * H;
  const float *const xr = p.x + (size_t)t * H;
  const int c1 = min(nc, c0 + PF_PREP_CHUNKS);
  float nx[32];
  quad_zero(nx);
  if (slot >= 0) quad_load(nx, xr + c0 * 128, lane);
#pragma unroll 1
  for (int c = c0; c < c1; c++) {
    float x[32], v[32];
#pragma unroll
    for (int j = 0; j < 32; j++) x[j] = nx[j];
    if (slot >= 0 && c + 1 < c1) quad_load(nx, xr + (c + 1) * 128, lane);
#pragma unroll
    for (int j = 0; j < 32; j++) v[j] = x[j];
    if (slot >= 0) quad_scale_in(v, sg + c * 128, lane);  // (a padding row stays zero whatever the scales are)
    fwht128_quad(v, lane, PF_HS);
    quad_store_blocked(v, p.xh_g, pos, c, lane, p.pos_cap / 8);
#pragma unroll
    for (int j = 0; j < 32; j++) v[j] = x[j];
    if (slot >= 0) quad_scale_in(v, su + c * 128, lane);
    fwht128_quad(v, lane, PF_HS);
    quad_store_blocked(v, p.xh_u, pos, c, lane, p.pos_cap / 8);
  }
}

// down operand: SwiGLU of the finished gate / up, times suh_down, H128, fp16 (reference pf_moe.metal:107-125). One warp per
// (row group, chunk).
__global__ void __launch_bounds__(256, 3) pf_mid_kernel(const PfParams p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, I = p.I, nc = I / 128;
  const int job = blockIdx.x * 8 + warp, group = job / nc, chunk = job - group * nc;
  if (group * 8 >= p.pos_cap) return;
  const int pos = group * 8 + (lane >> 2);
  const int e = pos < p.off[p.E + 1] ? p.seid[pos] : -1;
  const bool live = e >= 0, shared = e == p.E;
  const int el = shared || !live ? 0 : e - p.e0;
  const int o = chunk * 128;
  float g[32], u[32];
  quad_zero(g);
  quad_zero(u);
  if (live) {
    const float *raw = p.raw_gu + (size_t)pos * 2 * I + o;
    quad_load(g, raw, lane);
    quad_load(u, raw + I, lane);
  }
  fwht128_quad(g, lane, PF_HS);
  fwht128_quad(u, lane, PF_HS);
  if (live) {
    quad_scale_out(g, (shared ? p.sgt.svh : p.gate.svh + (size_t)el * I) + o, lane);
    quad_scale_out(u, (shared ? p.sup.svh : p.up.svh + (size_t)el * I) + o, lane);
#pragma unroll
    for (int j = 0; j < 32; j++) g[j] = g[j] / (1.0f + expf(-g[j])) * u[j];
    quad_scale_out(g, (shared ? p.sdn.suh : p.down.suh + (size_t)el * I) + o, lane);
  }
  fwht128_quad_runs(g, lane, PF_HS);
#pragma unroll
  for (int r = 0; r < 4; r++)
    *reinterpret_cast<uint4 *>(p.xh_d + blocked_index(pos, o + quad_run(lane, r), p.pos_cap / 8)) =
        make_uint4(pack2(g[8 * r], g[8 * r + 1]), pack2(g[8 * r + 2], g[8 * r + 3]), pack2(g[8 * r + 4], g[8 * r + 5]), pack2(g[8 * r + 6], g[8 * r + 7]));
}

// finish: one CTA per (token, 1024 columns), one warp per slot + one for the shared expert: every warp finishes its slot's
// eight chunks (H128, svh, routing weight) into shared memory, then the CTA sums the slots in slot order
// (reference pf_moe.metal:129-161). A lane's 32 contiguous values go to shared memory in 16-byte pieces XORed with the number
// of their 128-byte line, so neither the writes nor the reads of the sum meet in a bank.
constexpr int PF_FQ = 1024;
__global__ void __launch_bounds__(32 * 17, 2) pf_finish_kernel(const PfParams p) {
  extern __shared__ __align__(16) float vals_dyn[];  // [slots][PF_FQ]; the block has one warp per slot, at least 4 warps
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q0 = blockIdx.x * PF_FQ, t = blockIdx.y, H = p.H, k = p.topk;
  const int nslots = k + (p.has_shared ? 1 : 0);
  const int ncol = min(PF_FQ, H - q0);
  if (warp < nslots) {
    const bool shared = warp == k;
    const int pos = shared ? (t >= p.sh_row0 && t < p.sh_row0 + p.sh_rows ? p.off[p.E] + t - p.sh_row0 : -1) : p.inv[t * k + warp];
    const int o = (lane >> 2) * 128;  // this quad's chunk
    const bool on = pos >= 0 && o < ncol;
    float v[32];
    quad_zero(v);
    if (on) quad_load(v, p.raw_d + (size_t)pos * H + q0 + o, lane);
    fwht128_quad(v, lane, PF_HS);
    const int first = o + quad_first(lane);
    if (on) {
      const int e = shared ? 0 : (int)p.route[(size_t)t * 2 * k + warp] - p.e0;
      const float w = shared ? 1.0f / (1.0f + expf(-p.logits[(size_t)t * (p.E + 1) + p.E])) : __uint_as_float(p.route[(size_t)t * 2 * k + k + warp]);
      quad_scale_out(v, (shared ? p.sdn.svh : p.down.svh + (size_t)e * H) + q0 + o, lane);
      if (shared) {
        float4 *dst = reinterpret_cast<float4 *>(p.sho + (size_t)t * H + q0 + first);
#pragma unroll
        for (int c = 0; c < 8; c++) dst[c] = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
      }
#pragma unroll
      for (int j = 0; j < 32; j++) v[j] *= w;
    }  // else: a slot computed on another rank, or a row whose shared expert runs elsewhere: zeros
    float *line = vals_dyn + warp * PF_FQ + first;
#pragma unroll
    for (int c = 0; c < 8; c++)
      *reinterpret_cast<float4 *>(line + 4 * (c ^ ((first >> 5) & 7))) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
  }
  __syncthreads();
  for (int c = threadIdx.x * 4; c < ncol; c += blockDim.x * 4) {
    const int at = (c & ~31) + 4 * (((c >> 2) & 7) ^ ((c >> 5) & 7));
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int s = 0; s < nslots; s++) {
      const float4 v = *reinterpret_cast<const float4 *>(vals_dyn + s * PF_FQ + at);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    *reinterpret_cast<float4 *>(p.y + (size_t)t * H + q0 + c) = acc;
  }
}

// =============================================================================================== one Linear, many rows
// y[n][out] = x[n][in] @ W for n > 64 rows (reference: t6::record_prefill, kernels/trunk6/trunk6.mm:385-492, which
// decodes W' densely once per chunk and runs an fp16 GEMM): the same grouped GEMM with a single group that holds all
// rows, i.e. every tile is decoded once per 128 rows straight into the tensor core's operand layout.
__global__ void __launch_bounds__(256) pfl_prep_kernel(const float *__restrict__ x, const __half *__restrict__ suh, __half *xh, int n, int n8, int in) {
  const int lane = threadIdx.x & 31, nc = in / 128, job = blockIdx.x * 8 + (threadIdx.x >> 5), group = job / nc, chunk = job - group * nc;
  if (group * 8 >= n8) return;
  const int r = group * 8 + (lane >> 2);
  float v[32];
  quad_zero(v);
  if (r < n) {
    quad_load(v, x + (size_t)r * in + chunk * 128, lane);
    quad_scale_in(v, suh + chunk * 128, lane);
  }
  fwht128_quad(v, lane, PF_HS);
  quad_store_blocked(v, xh, r, chunk, lane, n8 / 8);
}

__global__ void pfl_items_kernel(PfItem *items, int *nitems, int n, int ncb, int rows) {
  const int passes = (n + rows - 1) / rows, total = passes * ncb;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int pass = i / ncb, cb = i - pass * ncb;
    items[i] = PfItem{-1, 0, cb, pass * rows, min(rows, n - pass * rows), {0, 0, 0}};
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *nitems = total;
}

// one warp per (row, eight chunks)
__global__ void __launch_bounds__(256) pfl_finish_kernel(const float *__restrict__ raw, const __half *__restrict__ svh, float *y, int n, int out) {
  const int lane = threadIdx.x & 31, nc = out / 128;
  const long job = ((long)blockIdx.x * 8 + (threadIdx.x >> 5)) * 8 + (lane >> 2);
  const int r = (int)(job / nc), o = (int)(job - (long)r * nc) * 128;
  const bool on = r < n;
  float v[32];
  quad_zero(v);
  if (on) quad_load(v, raw + (size_t)r * out + o, lane);
  fwht128_quad(v, lane, PF_HS);
  if (!on) return;
  quad_scale_out(v, svh + o, lane);
  float4 *dst = reinterpret_cast<float4 *>(y + (size_t)r * out + o + quad_first(lane));
#pragma unroll
  for (int c = 0; c < 8; c++) dst[c] = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
}

size_t pf_linear_scratch_bytes(int in, int out, int n) {
  const size_t n8 = ((size_t)n + 7) & ~(size_t)7, passes = ((size_t)n + PF_NTOK - 1) / PF_NTOK;
  return n8 * in * 2 + n8 * out * 4 + passes * (out / PF_NCOL) * sizeof(PfItem) + 1024;
}

void launch_pf_linear(const void *trellis, const void *suh, const void *svh, int in, int out, int K, const float *x, int n, float *y,
                      void *scratch, int *status, cudaStream_t st) {
  IJ_CHECK(in % 128 == 0 && out % 256 == 0, "prefill Linear needs in %% 128 == 0 and out %% 256 == 0 (%d -> %d)", in, out);
  IJ_CHECK(K >= 4 && K <= 8, "EXL3 bits per weight %d outside 4..8", K);
  IJ_CHECK(n >= 1 && n <= 65535 * 8, "prefill Linear: %d rows", n);
  const size_t n8 = ((size_t)n + 7) & ~(size_t)7, passes = ((size_t)n + PF_NTOK - 1) / PF_NTOK;
  char *base = (char *)scratch;
  __half *xh = (__half *)base;
  float *raw = (float *)(base + n8 * in * 2);
  PfItem *items = (PfItem *)(base + n8 * in * 2 + n8 * out * 4);
  int *nitems = (int *)((char *)items + passes * (out / PF_NCOL) * sizeof(PfItem));
  nitems = (int *)(((uintptr_t)nitems + 15) & ~(uintptr_t)15);
  pfl_prep_kernel<<<(int)((n8 / 8 * (in / 128) + 7) / 8), 256, 0, st>>>(x, (const __half *)suh, xh, n, (int)n8, in);
  // rows per item: 256 halve the decode, 128 make twice as many items; the fewer rounds of the persistent grid decide (an item of
  // 256 rows is weighed as 1.25 of 128: the decode is the same, the MMAs and the results double)
  const int ncb = out / PF_NCOL, sms = sm_count();
  auto rounds = [&](int rows) { return ((n + rows - 1) / rows * ncb + sms - 1) / sms; };
  const int rows = rounds(PF_PASS) * 1.25 <= rounds(PF_NTOK) ? PF_PASS : PF_NTOK;
  pfl_items_kernel<<<8, 256, 0, st>>>(items, nitems, n, ncb, rows);
  IJ_CUDA(cudaGetLastError());
  PgGemm g{};
  g.items = items; g.nitems = nitems;
  make_trellis_map(&g.w_shared[0], trellis, 1, in / 16, out / 16, K, PG_KS);
  g.act[0] = xh;
  g.out[0] = raw;
  g.groups = (int)(n8 / 8); g.ldo = out; g.in = in; g.IT = in / 16; g.OT = out / 16; g.Kx = K; g.Ks = K;
  launch_pf_gemm(g, status, st);
  pfl_finish_kernel<<<(int)(((size_t)n * (out / 128) + 63) / 64), 256, 0, st>>>(raw, (const __half *)svh, y, n, out);
  IJ_CUDA(cudaGetLastError());
}

// =============================================================================================== host side
size_t pf_pos_cap(int n, int topk, int E, bool has_shared) {
  return (((size_t)n * topk + 8 * (size_t)E + (has_shared ? n : 0) + 15) / 8) * 8;
}

void launch_pf_moe(const PfParams &p, int *status, cudaStream_t st) {
  IJ_CHECK(p.E <= 1024 && p.topk <= 16 && p.H % 256 == 0 && p.I % 256 == 0, "prefill: unsupported dims E %d top_k %d H %d I %d", p.E, p.topk, p.H, p.I);
  IJ_CHECK(p.n >= 1 && p.n <= 65535, "prefill: %d tokens outside 1..65535", p.n);
  const int groups = p.pos_cap / 8;
  IJ_CUDA(cudaMemsetAsync(p.order, 0xFF, (size_t)p.pos_cap * 4, st));
  IJ_CUDA(cudaMemsetAsync(p.seid, 0xFF, (size_t)p.pos_cap * 4, st));
  IJ_CHECK(p.H % LG_K == 0, "prefill: hidden %d must be a multiple of %d", p.H, LG_K);
  if (!p.external_route) {
    IJ_CUDA(cudaFuncSetAttribute(pf_logits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LG_SMEM));
    // k-splits until every SM has two CTAs: a step of the k loop is a memory round trip, 64 of them in a row took 110 us for 333
    // tokens (12 CTAs) and 117 for 4096 (128). The partial sums lie where the down products come later.
    const int tiles = ((p.n + LG_T - 1) / LG_T) * ((p.E + LG_T - 1) / LG_T), steps = p.H / LG_K;
    int nsplit = std::max(1, std::min(std::min(LG_SPLITS, 2 * sm_count() / tiles), steps));
    while (nsplit > 1 && (size_t)nsplit * p.n * (p.E + 1) > (size_t)p.pos_cap * p.H) nsplit--;
    const int nk = (steps + nsplit - 1) / nsplit;
    nsplit = (steps + nk - 1) / nk;
    float *part = nsplit > 1 ? p.raw_d : p.logits;
    pf_logits_kernel<<<dim3((p.n + LG_T - 1) / LG_T, (p.E + LG_T - 1) / LG_T, nsplit), 256, LG_SMEM, st>>>(p, part, nk);
    pf_route_kernel<<<(p.n + 7) / 8, 256, 0, st>>>(p, part, nsplit);
  } else {
    IJ_CHECK(!p.has_shared, "prefill: caller-routed pairs carry no shared expert");
  }
  IJ_CHECK(p.e0 >= 0 && p.ecount >= 0 && p.e0 + p.ecount <= p.E, "prefill: bad expert slice");
  IJ_CHECK(p.sh_row0 >= 0 && p.sh_rows >= 0 && p.sh_row0 + p.sh_rows <= p.n, "prefill: shared rows [%d, %d) outside [0, %d)", p.sh_row0, p.sh_row0 + p.sh_rows, p.n);
  const int nb = (p.S + PS_BLOCK - 1) / PS_BLOCK, nbs = p.has_shared ? (p.sh_rows + PS_BLOCK - 1) / PS_BLOCK : 0;
  pf_hist_kernel<<<nb, 32, 0, st>>>(p, p.hist);
  pf_blockscan_kernel<<<(p.E + 7) / 8, 256, 0, st>>>(p, p.hist, nb);
  pf_scan_kernel<<<1, 1024, 0, st>>>(p);
  pf_place_kernel<<<nb + nbs, 32, 0, st>>>(p, p.order, p.hist, nb);
  pf_prep_kernel<<<(groups * ((p.H / 128 + PF_PREP_CHUNKS - 1) / PF_PREP_CHUNKS) + 7) / 8, 256, 0, st>>>(p, p.order);
  IJ_CUDA(cudaGetLastError());
  PgGemm g{};
  g.items = p.items_gu; g.nitems = p.nitems;
  const bool routed = p.ecount > 0;  // (no items name a stack that is not there)
  const int HT = p.H / 16, IT = p.I / 16;
  if (routed) {
    make_trellis_map(&g.w_routed[0], p.gate.trellis, p.ecount, HT, IT, p.Kx, PG_KS);
    make_trellis_map(&g.w_routed[1], p.up.trellis, p.ecount, HT, IT, p.Kx, PG_KS);
  }
  if (p.has_shared) {
    make_trellis_map(&g.w_shared[0], p.sgt.trellis, 1, HT, IT, p.Ks, PG_KS);
    make_trellis_map(&g.w_shared[1], p.sup.trellis, 1, HT, IT, p.Ks, PG_KS);
  }
  g.act[0] = p.xh_g; g.act[1] = p.xh_u;
  g.out[0] = p.raw_gu; g.out[1] = p.raw_gu + p.I;
  g.groups = groups; g.ldo = 2 * p.I; g.in = p.H; g.IT = p.H / 16; g.OT = p.I / 16; g.Kx = p.Kx; g.Ks = p.has_shared ? p.Ks : p.Kx;
  launch_pf_gemm(g, status, st);
  pf_mid_kernel<<<(groups * (p.I / 128) + 7) / 8, 256, 0, st>>>(p);
  IJ_CUDA(cudaGetLastError());
  PgGemm d{};
  d.items = p.items_d; d.nitems = p.nitems + 1;
  if (routed) make_trellis_map(&d.w_routed[0], p.down.trellis, p.ecount, IT, HT, p.Kx, PG_KS);
  if (p.has_shared) make_trellis_map(&d.w_shared[0], p.sdn.trellis, 1, IT, HT, p.Ks, PG_KS);
  d.act[0] = p.xh_d;
  d.out[0] = p.raw_d;
  d.groups = groups; d.ldo = p.H; d.in = p.I; d.IT = p.I / 16; d.OT = p.H / 16; d.Kx = p.Kx; d.Ks = g.Ks;
  launch_pf_gemm(d, status, st);
  const int fslots = p.topk + (p.has_shared ? 1 : 0);  // one warp per slot; caller-routed pairs bring a single slot per row
  // up to 17 slots of 4 KB (per device: every launch)
  IJ_CUDA(cudaFuncSetAttribute(pf_finish_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 17 * PF_FQ * 4));
  pf_finish_kernel<<<dim3((p.H + PF_FQ - 1) / PF_FQ, p.n), 32 * std::max(fslots, 4), (size_t)fslots * PF_FQ * 4, st>>>(p);
  IJ_CUDA(cudaGetLastError());
}

// =============================================================================================== all-to-all helpers
// Stable counting sort of the n * k (token, slot) pairs of a route array by owner rank (= expert id / per): packed row `at`
// of the dispatch buffer takes pair p, send_token[at] = its token, send_route[at] = (id, weight bits), pos[p] = at,
// counts[d] = pairs going to rank d. One CTA; every thread owns a contiguous run of pairs, the ranks are placed one
// after the other with a block-wide exclusive scan each (at most 16 ranks).
__global__ void __launch_bounds__(1024) pairs_by_owner_kernel(const uint32_t *__restrict__ route, int n, int k, int per, int world,
                                                              int *__restrict__ send_token, uint32_t *__restrict__ send_route,
                                                              int *__restrict__ pos, long long *__restrict__ counts) {
  __shared__ int wsum[32];
  const int P = n * k, tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int chunk = (P + T - 1) / T, lo = min(P, tid * chunk), hi = min(P, lo + chunk);
  int start = 0;
  for (int d = 0; d < world; d++) {
    int mine = 0;
    for (int pr = lo; pr < hi; pr++) mine += (int)(route[(size_t)(pr / k) * 2 * k + pr % k] / (uint32_t)per) == d ? 1 : 0;
    int inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xFFFFFFFFu, inc, o);
      if (lane >= o) inc += a;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < T / 32; w++) {
      before += w < warp ? wsum[w] : 0;
      total += wsum[w];
    }
    int at = start + before + inc - mine;
    for (int pr = lo; pr < hi; pr++) {
      const size_t r = (size_t)(pr / k) * 2 * k + pr % k;
      const uint32_t id = route[r];
      if ((int)(id / (uint32_t)per) == d) {
        send_token[at] = pr / k;
        send_route[2 * at] = id;
        send_route[2 * at + 1] = route[r + k];
        pos[pr] = at;
        at++;
      }
    }
    if (tid == 0) counts[d] = total;
    start += total;
    __syncthreads();
  }
}
void launch_pairs_by_owner(const uint32_t *route, int n, int k, int per, int world, int *send_token, uint32_t *send_route, int *pos,
                           long long *counts, cudaStream_t st) {
  IJ_CHECK(n >= 1 && k >= 1 && per >= 1 && world >= 1 && world <= 16, "pairs_by_owner: n %d k %d experts per rank %d ranks %d", n, k, per, world);
  pairs_by_owner_kernel<<<1, 1024, 0, st>>>(route, n, k, per, world, send_token, send_route, pos, counts);
  IJ_CUDA(cudaGetLastError());
}

// dst[i] = src[idx[i]] (rows of H floats, H a multiple of 4): packs the (token, slot) pairs of one destination rank after
// the other for the dispatch all-to-all. One CTA per output row.
__global__ void __launch_bounds__(256) rows_gather_kernel(const float4 *__restrict__ src, const int *__restrict__ idx, float4 *__restrict__ dst, int q) {
  const size_t i = blockIdx.x, r = (size_t)idx[i];
  for (int c = threadIdx.x; c < q; c += blockDim.x) dst[i * q + c] = __ldg(src + r * q + c);
}
void launch_rows_gather(const float *src, const int *idx, int n_out, int H, float *dst, cudaStream_t st) {
  IJ_CHECK(H % 4 == 0 && (((uintptr_t)src | (uintptr_t)dst) & 15) == 0, "rows_gather: rows of a multiple of 4 floats, 16-byte aligned");
  if (n_out <= 0) return;
  rows_gather_kernel<<<n_out, 256, 0, st>>>(reinterpret_cast<const float4 *>(src), idx, reinterpret_cast<float4 *>(dst), H / 4);
  IJ_CUDA(cudaGetLastError());
}

// y[t] = ((slot[pos[t][0]] + slot[pos[t][1]]) + .. + slot[pos[t][k-1]]) + base[t]: the combine of the all-to-all prefill on a
// token's home rank. The slots are added in slot order and the shared expert's term last, as pf_finish_kernel does on one
// GPU, so the result is bit-identical to it. pos < 0 skips a slot.
__global__ void __launch_bounds__(256) slots_combine_kernel(const float4 *__restrict__ slot, const int *__restrict__ pos, const float4 *__restrict__ base,
                                                            float4 *__restrict__ y, int k, int q) {
  const size_t t = blockIdx.x;
  for (int c = threadIdx.x; c < q; c += blockDim.x) {
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int s = 0; s < k; s++) {
      const int ps = pos[t * k + s];
      if (ps >= 0) {
        const float4 v = __ldg(slot + (size_t)ps * q + c);
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
    }
    if (base != nullptr) {
      const float4 b = base[t * q + c];
      acc.x += b.x; acc.y += b.y; acc.z += b.z; acc.w += b.w;
    }
    y[t * q + c] = acc;
  }
}
void launch_slots_combine(const float *slot, const int *pos, const float *base, float *y, int n, int k, int H, cudaStream_t st) {
  IJ_CHECK(H % 4 == 0 && (((uintptr_t)slot | (uintptr_t)base | (uintptr_t)y) & 15) == 0, "slots_combine: rows of a multiple of 4 floats, 16-byte aligned");
  IJ_CHECK(n >= 1 && k >= 1, "slots_combine: %d tokens, %d slots", n, k);
  slots_combine_kernel<<<n, 256, 0, st>>>(reinterpret_cast<const float4 *>(slot), pos, reinterpret_cast<const float4 *>(base),
                                          reinterpret_cast<float4 *>(y), k, H / 4);
  IJ_CUDA(cudaGetLastError());
}

}  // namespace ijah
