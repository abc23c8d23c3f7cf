// Backward gated scan with 17 to 64 states, chunked form on tcgen05 tensor cores: the walk in reverse time of bwd_tc.cu
// (whose notation is used here; the adjoint of naju/scan.py:79-93 as written out in naju/cuda/naju_cuda.cu:85-144, dB and dC
// in the Gram form of naju/chunk_bwd_triton.py:20-99) on chunks of Q = 32 steps:
//
//   Yt[d,t] = sum_{s<=t} G[t,s] wt[d,s] + <C_t, h[d]>            gt[d,s] = sum_{t>=s} G[t,s] al[d,t] + <B_s, lt[d]>
//   dL[d,n] = sum_t al[d,t] C[t,n]                               M2[t,s] = sum_d al[d,t] wt[d,s]
//   dC[t,n] = sum_d al[d,t] h[d,n] + sum_{s<=t} M2[t,s] B[s,n]   dB[s,n] = sum_d wt[d,s] lt[d,n] + sum_{t>=s} M2[t,s] C[t,n]
//   r_t = r_{t+1} + al_t Yt_t - wt_t gt_t,   d f_logit = (1-f_t) r_t,   du = i_t R_t gt_t + D_skip dy_t,   d i_logit = wt_t (1-i_t) gt_t
//
// What bounds it: the recurrent kernel does 14 N operations per channel and step on the CUDA cores (64 states: 13.9 ms for
// 8 x 8192 x 4096, 32 states 11.6 ms; 4.75 and 3.36 ms here).  Here they are MMAs, and a tile is a chain of phases: gates, MMAs, sweep.
// Every operand is in three bf16 terms, all 24 bits of an fp32 significand, as the recurrent kernel computes in fp32 throughout; of
// the nine products of two such operands the six that reach 24 bits are taken, the smallest first (an accumulating MMA truncates).
// A channel's row is [al 32 | wt 32 | h NS | lt NS] three times: with 64 states 147 KB for 128 channels, so a chunk is 32 steps and
// there is one set of rows.
//   warps 0-15   main warps, four threads per channel: group g owns steps [8g, 8g+8) of every chunk, gates and sweep;
//                everything per step stays in registers in between.
//   warps 16-23  carry warps, two threads per channel with half of the states each: adjoint carry, h and lt rows from the
//                checkpoints, the seed of the r recurrence; the dC / dB partial rows.
//   warp 24      operand builder: C and B rows, G = C B^T, then the masked M2 operand of the second MMA round.
//   warp 25      TMA producer.     warp 26  MMA issuer.
// The second round adds tril(M2) B and tril(M2)^T C onto the cross-channel sums where they lie in TMEM.
// Stands down unless the forward ran chunked and met no deep-gate tile (nor a value that is not finite).  Where a gradient that comes in
// is not finite, a product with one of the masks' zeros would reach steps that it must not: the kernel says so in the header
// (`redo`), and the recurrent kernel launched behind it does the work over.  Every wait is bounded.
#include "common.cuh"
#include "params.h"
#include "tc_common.cuh"
#include "tma_host.h"

namespace naju {
namespace wideb {

using namespace tcx;

constexpr int Q = 32, NGRP = 4, SLAB = Q / NGRP, RING = 4, NCARRY = 256;
constexpr int W_CARRY = 16, W_BUILD = 24, W_PROD = 25, W_MMA = 26, NTHREADS = 27 * 32;
static_assert(W_BUILD % 4 == 0, "the builder warp reads accumulator rows 0-31");

struct Maps {
  CUtensorMap u, fl, il, dy, bm, cm;
};

template <int NS>
struct Smem {
  static constexpr int NC = NS / 8;
  // channel row (bf16, chunks of 8): term k from chunk k * R_TERM on
  static constexpr int R_A = 0, R_W = 4, R_H = 8, R_L = 8 + NC, R_TERM = 8 + 2 * NC;
  static constexpr uint32_t SBO_R = 3 * R_TERM * 128, ROWS_BYTES = 16 * SBO_R;
  static constexpr int BG_C = 0, BG_G = NC;                           // rows t: [C NS | g1 32 | g2 32 | g3 32]
  static constexpr uint32_t SBO_BG = (NC + 12) * 128, BG_BYTES = 4 * SBO_BG;
  static constexpr uint32_t SBO_BB = NC * 128, BB_BYTES = 4 * SBO_BB;
  static constexpr uint32_t SBO_M = 12 * 128, M_BYTES = 4 * SBO_M;    // M2 operand rows t: [m1 32 | m2 32 | m3 32]
  static constexpr uint32_t BC_BYTES = Q * NS * 2;
  static constexpr uint32_t one = SLAB * kDT * 2, slab_bytes = 4 * one;  // u | f_logit | i_logit | dy
  static constexpr uint32_t off_ring = 0;
  // The 32 rows of the C and M2 operands are addressed as 128, and M2's MN-major view starts four chunks early: all of
  // it lies inside shared memory.
  static constexpr uint32_t off_BG = off_ring + RING * slab_bytes;   // [2]
  static constexpr uint32_t off_BB = off_BG + 2 * BG_BYTES;          // [2]
  static constexpr uint32_t off_bc = off_BB + 2 * BB_BYTES;          // [B raw | C raw]
  static constexpr uint32_t off_M = off_bc + 2 * BC_BYTES;
  static constexpr uint32_t off_rows = off_M + M_BYTES;
  static constexpr uint32_t total = off_rows + ROWS_BYTES;
  static_assert(total + 8192 <= 232448, "with the static arrays, within an SM's 227 KB");
  static_assert(RING >= NGRP, "a group waits for its slab by parity: the slot's previous use was filled before the group's own previous slab");
  static_assert(off_M >= 4 * 128 && off_M + 16 * SBO_M <= total && off_BG + BG_BYTES + 16 * SBO_BG <= total, "");
  // (dL sits directly before gt: one MMA with the B operand [C | g1] feeds both)
  static constexpr uint32_t TM_Y = 0, TM_DL = 32, TM_G = 32 + NS, TM_GB = 64 + NS, TM_X = 96 + NS, TM_U = TM_X + 32, TM_V = TM_U + NS,
                            TMEM_COLS = 512;
  static_assert(TM_V + NS <= TMEM_COLS, "");
};

struct Bars {
  unsigned long long full[RING], empty[RING];
  unsigned long long bc_full, bc_empty;
  unsigned long long lprod[NGRP];      // a group's retention product is published          (counts are in warps)
  unsigned long long ssum[NGRP];       // a group's sum of r-increments is published
  unsigned long long part[NGRP];       // a group's operand-row chunks written
  unsigned long long rq_ready;         // the chunk's retention product is published
  unsigned long long h_full, lt_full;  // h rows / lt rows written
  unsigned long long seed_ready[2];    // seed of the r recurrence published
  unsigned long long ops_full[2];      // C | g1 | g2 and B rows of a tile built
  unsigned long long g_full[2];        // the builder's own MMA is complete
  unsigned long long d1_full, d4_full; // MMA rounds complete: first (Yt, gt, dL), cross-channel
  unsigned long long d5_full[2];       // second round (and with it every read of the tile's BG / BB)
  unsigned long long m2_full;          // M2 operand written
  unsigned long long x_free;           // second-round results read
  unsigned long long acc_free;         // Yt, gt, dL read
};

template <bool UTM, int NS>
__global__ void __launch_bounds__(NTHREADS, 1)
bwd_wide_kernel(const BwdParams p, const __grid_constant__ Maps maps) {
  using SM = Smem<NS>;
  using T16 = __nv_bfloat16;
  constexpr int NSH = NS / 2;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ Bars bars;
  __shared__ unsigned int s_tmem;
  __shared__ float s_L[NGRP][kDT];       // retention product of a group's steps (as 1 / prod f)
  __shared__ float s_S[NGRP][kDT];       // sum of the r-increments of a group's steps
  __shared__ float s_Rend[kDT];          // 1 / (retention product of the whole chunk)
  __shared__ float s_seed[2][2][kDT];    // r at the chunk end, <lam, x_end>: each half of the states' share

  pdl_wait();
  // stand down unless the forward ran in the chunked form and met no deep-gate tile
  if ((*p.fwd_form & 3) != 1) return;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t sbase = smem_u32(smem);
  const int ctiles = p.B * p.ndt, nchunks = p.nchunks;
  const int x_first = static_cast<int>(blockIdx.x), x_step = static_cast<int>(gridDim.x);
  const int ntotal = (x_first < ctiles ? (ctiles - x_first + x_step - 1) / x_step : 0) * nchunks;

  if (tid == 0) {
    if (blockIdx.x == 0) p.hdr->form = NAJU_FORM_TC_WALK;
    for (int i = 0; i < RING; ++i) {
      mbar_init(smem_u32(&bars.full[i]), 1);
      mbar_init(smem_u32(&bars.empty[i]), 4);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&bars.seed_ready[i]), NCARRY / 32);
      mbar_init(smem_u32(&bars.ops_full[i]), 1);
      mbar_init(smem_u32(&bars.g_full[i]), 1);
      mbar_init(smem_u32(&bars.d5_full[i]), 1);
    }
    for (int i = 0; i < NGRP; ++i) {
      mbar_init(smem_u32(&bars.lprod[i]), 4);
      mbar_init(smem_u32(&bars.ssum[i]), 4);
      mbar_init(smem_u32(&bars.part[i]), 4);
    }
    mbar_init(smem_u32(&bars.bc_full), 1);
    mbar_init(smem_u32(&bars.bc_empty), 1);
    mbar_init(smem_u32(&bars.rq_ready), 4);
    mbar_init(smem_u32(&bars.h_full), NCARRY / 32);
    mbar_init(smem_u32(&bars.lt_full), NCARRY / 32);
    mbar_init(smem_u32(&bars.d1_full), 1);
    mbar_init(smem_u32(&bars.d4_full), 1);
    mbar_init(smem_u32(&bars.m2_full), 1);
    mbar_init(smem_u32(&bars.x_free), 4);
    mbar_init(smem_u32(&bars.acc_free), 16 + NCARRY / 32);
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(smem_u32(&s_tmem), SM::TMEM_COLS);
  // the upper triangles of g1 / g2 and of M2 are never written: clear the shared operands once
  for (uint32_t i = tid * 16; i < 2 * (SM::BG_BYTES + SM::BB_BYTES); i += NTHREADS * 16)
    *reinterpret_cast<uint4*>(smem + SM::off_BG + i) = make_uint4(0, 0, 0, 0);
  for (uint32_t i = tid * 16; i < SM::M_BYTES; i += NTHREADS * 16)
    *reinterpret_cast<uint4*>(smem + SM::off_M + i) = make_uint4(0, 0, 0, 0);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  auto timeout = [&]() { atomicOr(&p.hdr->status, NAJU_ST_MMA_TIMEOUT); };

  if (warp == W_PROD) {
    // ===================================================================== TMA producer
    if (lane == 0) {
      uint32_t slab = 0;
      int it = 0;
      for (int x = x_first; x < ctiles; x += x_step) {
        const int b = x / p.ndt, d0 = (x - b * p.ndt) * kDT;
        for (int ci = 0; ci < nchunks; ++ci, ++it) {
          const int t0 = (nchunks - 1 - ci) * Q;
          if (it >= 1 && !mbar_wait(smem_u32(&bars.bc_empty), (it & 1) ^ 1)) timeout();
          {
            const uint32_t bar = smem_u32(&bars.bc_full), dst = sbase + SM::off_bc;
            mbar_arrive_expect_tx(bar, 2 * SM::BC_BYTES);
            tma_load_3d(dst, &maps.bm, 0, t0, b, bar);
            tma_load_3d(dst + SM::BC_BYTES, &maps.cm, 0, t0, b, bar);
          }
          for (int k = 0; k < NGRP; ++k, ++slab) {
            const uint32_t slot = slab % RING, ph = (slab / RING) & 1;
            if (slab >= RING && !mbar_wait(smem_u32(&bars.empty[slot]), ph ^ 1)) timeout();
            const uint32_t bar = smem_u32(&bars.full[slot]), dst = sbase + SM::off_ring + slot * SM::slab_bytes;
            mbar_arrive_expect_tx(bar, SM::slab_bytes);
            if (UTM) tma_load_3d(dst, &maps.u, t0 + k * SLAB, d0, b, bar);   // lands as [channel][step]
            else tma_load_3d(dst, &maps.u, d0, t0 + k * SLAB, b, bar);
            tma_load_3d(dst + SM::one, &maps.fl, d0, t0 + k * SLAB, b, bar);
            tma_load_3d(dst + 2 * SM::one, &maps.il, d0, t0 + k * SLAB, b, bar);
            tma_load_3d(dst + 3 * SM::one, &maps.dy, d0, t0 + k * SLAB, b, bar);
          }
        }
      }
    }
  } else if (warp == W_BUILD) {
    // ===================================================================== operand builder (lane = step)
    // Trip k builds the shared operands of tile k (one tile ahead of the MMAs), then the M2 operand of tile k-1.
    const int t = lane;
    const uint32_t idG = umma_idesc(128, Q, 1);
    // row t of a 32 x 32 accumulator block, masked to s <= t, in three bf16 terms of four chunks each
    auto tril_rows = [&](uint32_t tcol, unsigned char* row) {
#pragma unroll
      for (int c16 = 0; c16 < 2; ++c16) {
        uint32_t x[16];
        tmem_ld16_async(tcol + 16 * c16, x);
        tmem_ld_wait16(x);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c8 = 2 * c16 + h;
          if (c8 <= (t >> 3)) {
            uint32_t v[3][4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int s = 8 * c8 + 2 * k;
              split3(make_float2(s <= t ? __uint_as_float(x[8 * h + 2 * k]) : 0.f,
                                 s + 1 <= t ? __uint_as_float(x[8 * h + 2 * k + 1]) : 0.f), v[0][k], v[1][k], v[2][k]);
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) *reinterpret_cast<uint4*>(row + (4 * k + c8) * 128) = make_uint4(v[k][0], v[k][1], v[k][2], v[k][3]);
          }
        }
        __syncwarp();
      }
    };
    for (int it = 0; it <= ntotal; ++it) {
      if (it < ntotal) {
        const int st = it & 1;
        const uint32_t par = (it >> 1) & 1;
        if (!mbar_wait(smem_u32(&bars.bc_full), it & 1)) timeout();
        // every MMA of the tile two back that reads BG / BB (or the M2 operand) is complete
        if (it >= 2 && !mbar_wait(smem_u32(&bars.d5_full[st]), par ^ 1)) timeout();
        unsigned char* s_BG = smem + SM::off_BG + st * SM::BG_BYTES;
        unsigned char* s_BB = smem + SM::off_BB + st * SM::BB_BYTES;
        const unsigned char* raw = smem + SM::off_bc;
#pragma unroll 4
        for (int i = lane; i < Q * SM::NC; i += 32) {
          const int r = i / SM::NC, k = i % SM::NC;
          *reinterpret_cast<uint4*>(s_BB + op_off16(r, k * 8, SM::SBO_BB)) = *reinterpret_cast<const uint4*>(raw + i * 16);
          *reinterpret_cast<uint4*>(s_BG + op_off16(r, (SM::BG_C + k) * 8, SM::SBO_BG)) =
              *reinterpret_cast<const uint4*>(raw + SM::BC_BYTES + i * 16);
        }
        fence_async_smem();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          tc_fence_after();
          mbar_arrive(smem_u32(&bars.bc_empty));  // the raw rows have been read
          const uint64_t dC = umma_desc(sbase + SM::off_BG + st * SM::BG_BYTES, 128, SM::SBO_BG),
                         dB = umma_desc(sbase + SM::off_BB + st * SM::BB_BYTES, 128, SM::SBO_BB);
#pragma unroll
          for (int k = 0; k < NS / 16; ++k) umma_bf16(tmem + SM::TM_GB, dC + k * 16, dB + k * 16, idG, k > 0);
          umma_commit(smem_u32(&bars.g_full[st]));
        }
        __syncwarp();
        if (!mbar_wait(smem_u32(&bars.g_full[st]), par)) timeout();
        __syncwarp();
        tc_fence_after();
        tril_rows(tmem + SM::TM_GB, s_BG + static_cast<uint32_t>(t >> 3) * SM::SBO_BG + static_cast<uint32_t>(t & 7) * 16 + SM::BG_G * 128);
        fence_async_smem();
        tc_fence_before();
        mbar_arrive_warp(smem_u32(&bars.ops_full[st]));
      }
      if (it >= 1) {
        // (and with it the second round of tile it-2, the M2 operand's last reader: it was issued before)
        if (!mbar_wait(smem_u32(&bars.d4_full), (it - 1) & 1)) timeout();
        __syncwarp();
        tc_fence_after();
        tril_rows(tmem + SM::TM_X, smem + SM::off_M + static_cast<uint32_t>(t >> 3) * SM::SBO_M + static_cast<uint32_t>(t & 7) * 16);
        fence_async_smem();
        tc_fence_before();
        mbar_arrive_warp(smem_u32(&bars.m2_full));
      }
    }
  } else if (warp == W_MMA) {
    // ===================================================================== MMA issuer
    if (lane == 0) {
      const uint32_t aR = sbase + SM::off_rows, aM = sbase + SM::off_M;
      auto idesc = [](int N, uint32_t a_mn, uint32_t b_mn) { return umma_idesc(128, N, 1) | (a_mn << 15) | (b_mn << 16); };
      const uint32_t iKK = idesc(Q, 0, 0), iKM = idesc(Q, 0, 1), iKMc = idesc(NS + Q, 0, 1), iKMn = idesc(NS, 0, 1),
                     iMMx = idesc(Q + 2 * NS, 1, 1), iMMn = idesc(NS, 1, 1);
      // K-major: LBO = bytes between 16-byte K chunks, SBO = bytes between 8-row groups.  MN-major: LBO = bytes between
      // groups of 8 along K, SBO = bytes between 8-element chunks along M / N.
      const uint64_t dRk = umma_desc(aR, 128, SM::SBO_R), dRm = umma_desc(aR, SM::SBO_R, 128);
      // M2: K-major as is; MN-major starting four chunks early, so that column s lands in accumulator row 32+s (V's)
      const uint64_t dMk = umma_desc(aM, 128, SM::SBO_M), dMm = umma_desc(aM - 4 * 128, SM::SBO_M, 128);
      auto off = [](uint32_t bytes) { return static_cast<uint64_t>(bytes >> 4); };
      for (int it = 0; it < ntotal; ++it) {
        const int st = it & 1;
        const uint32_t par = it & 1, par2 = (it >> 1) & 1;
        const uint32_t aBG = sbase + SM::off_BG + st * SM::BG_BYTES, aBB = sbase + SM::off_BB + st * SM::BB_BYTES;
        const uint64_t dGk = umma_desc(aBG, 128, SM::SBO_BG), dGm = umma_desc(aBG, SM::SBO_BG, 128);   // C | g1 | g2 | g3
        const uint64_t dBk = umma_desc(aBB, 128, SM::SBO_BB), dBm = umma_desc(aBB, SM::SBO_BB, 128);   // B rows
        if (!mbar_wait(smem_u32(&bars.ops_full[st]), par2)) timeout();
        if (it >= 1 && !mbar_wait(smem_u32(&bars.acc_free), par ^ 1)) timeout();
        if (!mbar_wait(smem_u32(&bars.h_full), par)) timeout();
        tc_fence_after();
        // chunk `c` of term `k` of the channel rows / of g
        auto row = [](int k, int c) { return static_cast<uint32_t>(k * SM::R_TERM + c) * 128; };
        auto gch = [](int k, int c) { return static_cast<uint32_t>(SM::BG_G + 4 * k + c) * 128; };
        // Yt = (h1 + h2 + h3).C   (K = n)
#pragma unroll
        for (int k = 2; k >= 0; --k)
#pragma unroll
          for (int ks = 0; ks < NS / 16; ++ks)
            umma_bf16(tmem + SM::TM_Y, dRk + off(row(k, SM::R_H + 2 * ks)), dGk + off((SM::BG_C + 2 * ks) * 128), iKK, k < 2 || ks > 0);
        for (int g = 0; g < NGRP; ++g)
          if (!mbar_wait(smem_u32(&bars.part[g]), par)) timeout();
        tc_fence_after();
        // dL += (al1 + al2 + al3).C and gt += the products of al and g^T, those with g1 in one instruction with dL's: [dL | gt] += al.[C | g1]
        auto al_cg = [&](int k) {
#pragma unroll
          for (int ks = 0; ks < Q / 16; ++ks)
            umma_bf16(tmem + SM::TM_DL, dRk + off(row(k, SM::R_A + 2 * ks)), dGm + off(2 * ks * SM::SBO_BG), iKMc, k < 2 || ks > 0);
        };
        auto al_g = [&](int k, int j) {
#pragma unroll
          for (int ks = 0; ks < Q / 16; ++ks)
            umma_bf16(tmem + SM::TM_G, dRk + off(row(k, SM::R_A + 2 * ks)), dGm + off(2 * ks * SM::SBO_BG + gch(j, 0)), iKM, 1u);
        };
        // Yt += the products of wt and g   (K = s)
        auto w_g = [&](int k, int j) {
#pragma unroll
          for (int ks = 0; ks < Q / 16; ++ks)
            umma_bf16(tmem + SM::TM_Y, dRk + off(row(k, SM::R_W + 2 * ks)), dGk + off(gch(j, 2 * ks)), iKK, 1u);
        };
        al_cg(2);
        al_g(0, 2);
        al_g(1, 1);
        w_g(2, 0);
        w_g(0, 2);
        w_g(1, 1);
        al_cg(1);
        al_g(0, 1);
        w_g(1, 0);
        w_g(0, 1);
        al_cg(0);
        w_g(0, 0);
        // gt += (l1 + l2 + l3).B   (K = n)
        if (!mbar_wait(smem_u32(&bars.lt_full), par)) timeout();
        tc_fence_after();
#pragma unroll
        for (int k = 2; k >= 0; --k)
#pragma unroll
          for (int ks = 0; ks < NS / 16; ++ks)
            umma_bf16(tmem + SM::TM_G, dRk + off(row(k, SM::R_L + 2 * ks)), dBk + off(2 * ks * 128), iKK, 1u);
        umma_commit(smem_u32(&bars.d1_full));  // the reverse sweep can start
        // cross-channel: X += [al | wt]^T . [wt | h | lt]   (K = 16 channels per step), once the previous tile's second-round
        // results, which lie in the same columns, have been read
        if (it >= 1 && !mbar_wait(smem_u32(&bars.x_free), par ^ 1)) timeout();
        tc_fence_after();
        auto cross = [&](int k, int j, bool first) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_bf16(tmem + SM::TM_X, dRm + off(2 * ks * SM::SBO_R + row(k, SM::R_A)), dRm + off(2 * ks * SM::SBO_R + row(j, SM::R_W)), iMMx,
                      !first || ks > 0);
        };
        cross(2, 0, true);
        cross(0, 2, false);
        cross(1, 1, false);
        cross(1, 0, false);
        cross(0, 1, false);
        cross(0, 0, false);
        umma_commit(smem_u32(&bars.d4_full));
        // second round, onto U (accumulator rows 0-31: steps) and V (rows 32-63)
        if (!mbar_wait(smem_u32(&bars.m2_full), par)) timeout();
        tc_fence_after();
#pragma unroll
        for (int k = 2; k >= 0; --k)
#pragma unroll
          for (int ks = 0; ks < Q / 16; ++ks) {
            // dC[t,n] += sum_s M2[t,s] B[s,n]
            umma_bf16(tmem + SM::TM_U, dMk + off((4 * k + 2 * ks) * 128), dBm + off(2 * ks * SM::SBO_BB), iKMn, 1u);
            // dB[32+s,n] += sum_t M2[t,s] C[t,n]
            umma_bf16(tmem + SM::TM_V, dMm + off(2 * ks * SM::SBO_M + 4 * k * 128), dGm + off(2 * ks * SM::SBO_BG), iMMn, 1u);
          }
        umma_commit(smem_u32(&bars.d5_full[st]));
      }
    }
  } else if (warp >= W_CARRY && warp < W_BUILD) {
    // ===================================================================== carry warps
    const int half = (warp - W_CARRY) >> 2, cid = (warp & 3) * 32 + lane, n0 = half * NSH;
    const uint32_t trow = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    unsigned char* my_row = smem + SM::off_rows + static_cast<uint32_t>(cid >> 3) * SM::SBO_R + static_cast<uint32_t>(cid & 7) * 16 +
                            half * (NSH / 8) * 128;
    float lam[NSH];   // adjoint entering the current chunk from the future
    auto split_chunk = [&](const float (&v)[8], int c) {
      uint32_t o[3][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) split3(make_float2(v[2 * j], v[2 * j + 1]), o[0][j], o[1][j], o[2][j]);
#pragma unroll
      for (int k = 0; k < 3; ++k) *reinterpret_cast<uint4*>(my_row + (k * SM::R_TERM + c) * 128) = make_uint4(o[k][0], o[k][1], o[k][2], o[k][3]);
    };
    auto state_row = [&](int xx, int c) { return p.ckS + ((static_cast<int64_t>(c) * ctiles + xx) * kDT + cid) * NS + n0; };
    // this thread's share of <lam, state at the end of chunk c of channel tile xx>
    auto seed_of = [&](int xx, int c) {
      const float4* src = reinterpret_cast<const float4*>(state_row(xx, c));
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < NSH / 4; ++k) {
        const float4 v = __ldg(src + k);
        s = fmaf(lam[4 * k], v.x, fmaf(lam[4 * k + 1], v.y, fmaf(lam[4 * k + 2], v.z, fmaf(lam[4 * k + 3], v.w, s))));
      }
      return s;
    };
    // h rows of the tile whose chunk is entered with the state at the end of chunk c (h0 below chunk 0)
    auto post_h = [&](int xx, int c) {
      const int bb = xx / p.ndt, dd = (xx - bb * p.ndt) * kDT + cid;
      const float* src = c >= 0 ? state_row(xx, c) : nullptr;
      // (64 states: sixteen in flight at a time, 2343 -> 2237 us at B=8, T=4096, D=4096, with the prefetch below and two-term operands; 32 states:
      // eight, 1477 us against 1514)
      constexpr int PER = NS == 64 ? 2 : 1;
#pragma unroll
      for (int k = 0; k < NSH / 8; k += PER) {
        float v[PER][8];
        if (c >= 0) {
          float4 a[2 * PER];
#pragma unroll
          for (int j = 0; j < 2 * PER; ++j) a[j] = __ldg(reinterpret_cast<const float4*>(src) + 2 * k + j);
#pragma unroll
          for (int j = 0; j < 2 * PER; ++j) {
            float* o = &v[j >> 1][4 * (j & 1)];
            o[0] = a[j].x; o[1] = a[j].y; o[2] = a[j].z; o[3] = a[j].w;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8 * PER; ++j) {
            const int n = n0 + 8 * k + j;
            v[j >> 3][j & 7] = (p.h0 != nullptr && dd < p.D && n < p.N) ? p.h0[(static_cast<int64_t>(bb) * p.D + dd) * p.N + n] : 0.f;
          }
        }
#pragma unroll
        for (int j = 0; j < PER; ++j) split_chunk(v[j], SM::R_H + k + j);
      }
      fence_async_smem();
      mbar_arrive_warp(smem_u32(&bars.h_full));
    };
    auto post_seed = [&](int jt, float s) {
      s_seed[jt & 1][half][cid] = s;
      mbar_arrive_warp(smem_u32(&bars.seed_ready[jt & 1]));
    };
    // adjoint entering the last chunk of channel tile xx
    auto load_lam = [&](int xx) {
      const int bb = xx / p.ndt, dd = (xx - bb * p.ndt) * kDT + cid;
#pragma unroll
      for (int n = 0; n < NSH; ++n)
        lam[n] = (p.dhT != nullptr && dd < p.D && n0 + n < p.N) ? p.dhT[(static_cast<int64_t>(bb) * p.D + dd) * p.N + n0 + n] : 0.f;
    };
    int x = x_first, ci = 0;
    if (ntotal > 0) {
      load_lam(x);
      post_h(x, nchunks - 2);
      post_seed(0, seed_of(x, nchunks - 1));
    }
#pragma unroll 1
    for (int it = 0; it < ntotal; ++it) {
      const int b = x / p.ndt, dt = x - b * p.ndt, d = dt * kDT + cid;
      const int c = nchunks - 1 - ci, t0 = c * Q;
      const uint32_t par = it & 1, st = it & 1, par2 = (it >> 1) & 1;
      const bool more = it + 1 < ntotal;
      // the states the next tile's h rows come from, towards L2 while there is time
      if (NS == 64 && c > 1) asm volatile("prefetch.global.L2 [%0];" ::"l"(state_row(x, c - 2)));
      // ---- the chunk's retention product is known: lt rows
      if (!mbar_wait(smem_u32(&bars.rq_ready), par)) timeout();
      const float Rend = s_Rend[cid];
      const float PQ = __frcp_rn(Rend);
#pragma unroll
      for (int k = 0; k < NSH / 8; ++k) {
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          lam[8 * k + j] *= PQ;
          v[j] = lam[8 * k + j];
        }
        split_chunk(v, SM::R_L + k);
      }
      fence_async_smem();
      mbar_arrive_warp(smem_u32(&bars.lt_full));
      {   // (behind the arrival: the tile's chain does not wait for it, 0.23 ms of 4.9)
        float2 z = make_float2(0.f, 0.f);
#pragma unroll
        for (int n = 0; n < NSH; n += 2) z = watch(z, make_float2(lam[n], lam[n + 1]), kOverState);
        // (the forward's product of the same gates was below kRMax; its order of multiplication is another)
        if (!(Rend < kRMax) || !(z.x + z.y == 0.f)) atomicOr(&p.hdr->redo, 1);
      }
      // ---- first round complete: adjoint leaving the chunk
      if (!mbar_wait(smem_u32(&bars.d1_full), par)) timeout();
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int k = 0; k < NSH / 16; ++k) {
        uint32_t dl[16];
        tmem_ld16_async(trow + SM::TM_DL + n0 + 16 * k, dl);
        tmem_ld_wait16(dl);
#pragma unroll
        for (int n = 0; n < 16; ++n) lam[16 * k + n] += __uint_as_float(dl[n]);
      }
      tc_fence_before();
      mbar_arrive_warp(smem_u32(&bars.acc_free));
      // next tile: the chunk before this one (its r recurrence ends at <lam, state entering this chunk>), or the last
      // chunk of the next channel tile
      const int xn = c > 0 ? x : x + x_step, cn = c > 0 ? c - 1 : nchunks - 1;
      if (c == 0) {
        if (p.dh0 != nullptr && d < p.D) {
          float* o = p.dh0 + (static_cast<int64_t>(b) * p.D + d) * p.N;
#pragma unroll
          for (int n = 0; n < NSH; ++n)
            if (n0 + n < p.N) o[n0 + n] = lam[n];
        }
        if (more) load_lam(xn);
      }
      float seed = 0.f;
      if (more) seed = seed_of(xn, cn);
      // ---- cross-channel block complete, and with it every MMA that reads the channel rows
      if (!mbar_wait(smem_u32(&bars.d4_full), par)) timeout();
      if (more) {
        post_h(xn, cn - 1);
        post_seed(it + 1, seed);
      }
      // ---- second round complete: dC (accumulator rows 0-31) and dB (rows 32-63), one row per step of the chunk
      if ((warp & 3) < 2) {
        if (!mbar_wait(smem_u32(&bars.d5_full[st]), par2)) timeout();
        __syncwarp();
        tc_fence_after();
        const bool isC = (warp & 3) == 0;
        float* dst = (isC ? p.dCpart : p.dBpart) + ((static_cast<int64_t>(b) * p.T + t0 + lane) * p.ndt + dt) * NS + n0;
#pragma unroll
        for (int k = 0; k < NSH / 16; ++k) {
          uint32_t v[16];
          tmem_ld16_async(trow + (isC ? SM::TM_U : SM::TM_V) + n0 + 16 * k, v);
          tmem_ld_wait16(v);
          if (t0 + lane < p.T)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              reinterpret_cast<float4*>(dst + 16 * k)[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                                                       __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
          __syncwarp();
        }
        tc_fence_before();
        mbar_arrive_warp(smem_u32(&bars.x_free));
      }
      if (++ci == nchunks) {
        ci = 0;
        x += x_step;
      }
    }
  } else if (warp < W_CARRY) {
    // ===================================================================== main warps
    const int grp = warp >> 2;                     // owns steps [8 grp, 8 grp + 8) of every chunk
    const int cid = (warp & 3) * 32 + lane;        // channel within the tile
    const uint32_t trow = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + SLAB * grp;
    unsigned char* my_row = smem + SM::off_rows + static_cast<uint32_t>(cid >> 3) * SM::SBO_R + static_cast<uint32_t>(cid & 7) * 16;
    const float2 kk = make_float2(kNegLog2e, kNegLog2e), one2 = make_float2(1.f, 1.f);
    constexpr int H = SLAB / 2;
    int it = 0;
    for (int x = x_first; x < ctiles; x += x_step) {
      const int b = x / p.ndt, dt = x - b * p.ndt, d0 = dt * kDT, d = d0 + cid;
      const bool d_ok = d < p.D;
      const float Dv = d_ok ? __ldg(p.Dskip + d) : 0.f;
      float dDsum = 0.f, dDlow = 0.f;   // (the sum over the chunks and what its additions dropped)
#pragma unroll 1
      for (int ci = 0; ci < nchunks; ++ci, ++it) {
        const int t0 = (nchunks - 1 - ci) * Q, nvalid = p.T - t0 - SLAB * grp;   // real steps among this thread's
        const uint32_t par = it & 1;
        const uint32_t sidx = static_cast<uint32_t>(it) * NGRP + grp, slot = sidx % RING, ph = (sidx / RING) & 1;
        if (!mbar_wait(smem_u32(&bars.full[slot]), ph)) timeout();
        const unsigned char* sl = smem + SM::off_ring + slot * SM::slab_bytes;
        const T16* s_u = reinterpret_cast<const T16*>(sl) + cid;             // [step][channel]
        const T16* s_ut = reinterpret_cast<const T16*>(sl) + cid * SLAB;      // [channel][step] (time-contiguous u)
        const T16* s_fl = reinterpret_cast<const T16*>(sl + SM::one) + cid;
        const T16* s_il = reinterpret_cast<const T16*>(sl + 2 * SM::one) + cid;
        const T16* s_dy = reinterpret_cast<const T16*>(sl + 3 * SM::one) + cid;
        // ---------------- gates (1): retention of the own steps, a_j = e^{-f_logit_j}, L_j = prod_{i<=j} (1 + a_i).  Steps past
        // the end of the sequence (they arrive as zeros) are made neutral: f = 1.
        float2 av[H], L[H];
#pragma unroll
        for (int j2 = 0; j2 < H; ++j2) {
          const float2 fl2 = mul2(make_float2(ld_as_f32(s_fl, (2 * j2) * kDT), ld_as_f32(s_fl, (2 * j2 + 1) * kDT)), kk);
          av[j2] = make_float2(fast_ex2(fl2.x), fast_ex2(fl2.y));
        }
        if (nvalid < SLAB) {
#pragma unroll
          for (int j2 = 0; j2 < H; ++j2) {
            if (2 * j2 >= nvalid) av[j2].x = 0.f;
            if (2 * j2 + 1 >= nvalid) av[j2].y = 0.f;
          }
        }
        {
          float run = 1.f;
#pragma unroll
          for (int j2 = 0; j2 < H; ++j2) {
            const float2 qv = add2(av[j2], one2);
            L[j2] = mul2(make_float2(run, run), make_float2(qv.x, qv.x * qv.y));
            run = L[j2].y;
          }
        }
        // (the readers of the previous tile's products arrived on `part` before the d1_full waited for below)
        s_L[grp][cid] = L[H - 1].y;
        mbar_arrive_warp(smem_u32(&bars.lprod[grp]));
        // ---------------- gates (2): R_t = (products of the groups before) x L_j
        float Rstart = 1.f;
        for (int g2 = 0; g2 < grp; ++g2) {
          if (!mbar_wait(smem_u32(&bars.lprod[g2]), par)) timeout();
          Rstart *= s_L[g2][cid];
        }
        if (grp == NGRP - 1) {
          s_Rend[cid] = Rstart * L[H - 1].y;      // the whole chunk's product, for the carry warps
          mbar_arrive_warp(smem_u32(&bars.rq_ready));
        }
        const float2 Rs2 = make_float2(Rstart, Rstart);
        float2 alr[H], wtr[H], cf[H], cm[H], cu[H];
        uint32_t dyp[H];
        float dDc = 0.f;
#pragma unroll
        for (int j2 = 0; j2 < H; ++j2) {
          const float2 il2 = mul2(make_float2(fmaxf(ld_as_f32(s_il, (2 * j2) * kDT), -80.f), fmaxf(ld_as_f32(s_il, (2 * j2 + 1) * kDT), -80.f)), kk);
          const float2 bq = make_float2(fast_ex2(il2.x), fast_ex2(il2.y));
          const float2 opb = add2(bq, one2);                      // 1 / i_t
          const float2 u2 = UTM ? ld_pair_as_f32(s_ut + 2 * j2) : make_float2(ld_as_f32(s_u, (2 * j2) * kDT), ld_as_f32(s_u, (2 * j2 + 1) * kDT));
          const float2 dy2 = make_float2(ld_as_f32(s_dy, (2 * j2) * kDT), ld_as_f32(s_dy, (2 * j2 + 1) * kDT));
          const float2 R = mul2(Rs2, L[j2]);
          const float2 Rprev = make_float2(j2 == 0 ? Rstart : Rstart * L[j2 == 0 ? 0 : j2 - 1].y, R.x);
          const float2 P = make_float2(fast_rcp(R.x), fast_rcp(R.y));          // 1 / R_t
          const float2 ig = make_float2(fast_rcp(opb.x), fast_rcp(opb.y));     // i_t
          cu[j2] = mul2(ig, R);                                   // i_t R_t
          wtr[j2] = mul2(u2, cu[j2]);
          alr[j2] = mul2(dy2, P);
          cf[j2] = mul2(mul2(av[j2], Rprev), P);                  // 1 - f_t
          cm[j2] = mul2(bq, ig);                                  // 1 - i_t
          dDc = fmaf(dy2.x, u2.x, fmaf(dy2.y, u2.y, dDc));
          dyp[j2] = __byte_perm(__float_as_uint(dy2.x), __float_as_uint(dy2.y), 0x7632);
        }
        mbar_arrive_warp(smem_u32(&bars.empty[slot]));   // the slab has been read
        {
          const float s = dDsum + dDc, v = s - dDsum;
          dDlow += (dDsum - (s - v)) + (dDc - v);
          dDsum = s;
        }
        // the channel rows are free once every MMA of the previous tile that reads them is complete
        if (it >= 1 && !mbar_wait(smem_u32(&bars.d4_full), par ^ 1)) timeout();
        {
          auto put = [&](const float2 (&v)[H], int c) {
            uint32_t o[3][H];
#pragma unroll
            for (int j2 = 0; j2 < H; ++j2) split3(v[j2], o[0][j2], o[1][j2], o[2][j2]);
#pragma unroll
            for (int k = 0; k < 3; ++k) *reinterpret_cast<uint4*>(my_row + (k * SM::R_TERM + c + grp) * 128) = make_uint4(o[k][0], o[k][1], o[k][2], o[k][3]);
          };
          put(alr, SM::R_A);
          put(wtr, SM::R_W);
        }
        fence_async_smem();
        tc_fence_before();
        mbar_arrive_warp(smem_u32(&bars.part[grp]));
        {
          float2 za = make_float2(0.f, 0.f), zw = za;
#pragma unroll
          for (int j2 = 0; j2 < H; ++j2) {
            za = watch(za, alr[j2], kOverGrad);
            zw = watch(zw, wtr[j2], kOverW);
          }
          if (!(za.x + za.y + zw.x + zw.y == 0.f)) atomicOr(&p.hdr->redo, 1);
        }

        const int64_t row0 = (static_cast<int64_t>(b) * p.T + t0 + SLAB * grp) * p.D + d;
        const int nout = d_ok ? nvalid : 0;
        // ---------------- sweep (1), once the first MMA round is complete: z_t = al_t Yt_t - wt_t gt_t and its suffix sums
        // over the own steps; du and d i_logit need gt only
        if (!mbar_wait(smem_u32(&bars.d1_full), par)) timeout();
        __syncwarp();
        tc_fence_after();
        float2 S[H];
        {
          uint32_t y8[8], g8[8];
          tmem_ld8_async(trow + SM::TM_Y, y8);
          tmem_ld8_async(trow + SM::TM_G, g8);
          tmem_ld_wait8(y8, g8);
          tc_fence_before();
          mbar_arrive_warp(smem_u32(&bars.acc_free));      // Yt and gt have been read
          float run = 0.f;
          float2 wg[H];
#pragma unroll
          for (int j2 = H - 1; j2 >= 0; --j2) {
            wg[j2] = mul2(wtr[j2], f2(g8[2 * j2], g8[2 * j2 + 1]));
            const float2 z = fma2(alr[j2], f2(y8[2 * j2], y8[2 * j2 + 1]), make_float2(-wg[j2].x, -wg[j2].y));
            const float s1 = run + z.y;
            run = s1 + z.x;
            S[j2] = make_float2(run, s1);
          }
          s_S[grp][cid] = run;
          mbar_arrive_warp(smem_u32(&bars.ssum[grp]));
          T16* gdu = UTM ? reinterpret_cast<T16*>(p.du) + static_cast<int64_t>(b) * p.u_sb + static_cast<int64_t>(d) * p.u_sd + t0 + SLAB * grp
                         : reinterpret_cast<T16*>(p.du) + row0;
          T16* gdil = reinterpret_cast<T16*>(p.dil) + row0;
          const float2 Dv2 = make_float2(Dv, Dv);
          uint32_t pk[H];
#pragma unroll
          for (int j2 = 0; j2 < H; ++j2) {
            float2 du = mul2(cu[j2], f2(g8[2 * j2], g8[2 * j2 + 1]));
            if (Dv != 0.f) du = fma2(Dv2, make_float2(bf16lo_f32(dyp[j2]), bf16hi_f32(dyp[j2])), du);
            const float2 dil = mul2(cm[j2], wg[j2]);
            pk[j2] = pack_bf16x2(du.x, du.y);
            const uint32_t pi = pack_bf16x2(dil.x, dil.y);
            if (2 * j2 < nout) {
              if (!UTM) reinterpret_cast<unsigned short*>(gdu)[static_cast<int64_t>(2 * j2) * p.D] = static_cast<unsigned short>(pk[j2]);
              reinterpret_cast<unsigned short*>(gdil)[static_cast<int64_t>(2 * j2) * p.D] = static_cast<unsigned short>(pi);
            }
            if (2 * j2 + 1 < nout) {
              if (!UTM) reinterpret_cast<unsigned short*>(gdu)[static_cast<int64_t>(2 * j2 + 1) * p.D] = static_cast<unsigned short>(pk[j2] >> 16);
              reinterpret_cast<unsigned short*>(gdil)[static_cast<int64_t>(2 * j2 + 1) * p.D] = static_cast<unsigned short>(pi >> 16);
            }
          }
          if constexpr (UTM) {   // this thread's steps of du are 16 adjacent bytes of its channel's row
            if (nout >= SLAB) *reinterpret_cast<uint4*>(gdu) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            else
#pragma unroll
              for (int e = 0; e < SLAB; ++e)
                if (e < nout) reinterpret_cast<unsigned short*>(gdu)[e] = static_cast<unsigned short>(e & 1 ? pk[e >> 1] >> 16 : pk[e >> 1] & 0xFFFFu);
          }
        }
        // ---------------- sweep (2): r_t = seed + (sums of the groups after) + S_t
        if (!mbar_wait(smem_u32(&bars.seed_ready[it & 1]), (it >> 1) & 1)) timeout();
        float rstart = s_seed[it & 1][0][cid] + s_seed[it & 1][1][cid];
        for (int g2 = NGRP - 1; g2 > grp; --g2) {
          if (!mbar_wait(smem_u32(&bars.ssum[g2]), par)) timeout();
          rstart += s_S[g2][cid];
        }
        T16* gdfl = reinterpret_cast<T16*>(p.dfl) + row0;
        const float2 rs2 = make_float2(rstart, rstart);
#pragma unroll
        for (int j2 = 0; j2 < H; ++j2) {
          const float2 dfl = mul2(cf[j2], add2(S[j2], rs2));
          if (2 * j2 < nout) gdfl[static_cast<int64_t>(2 * j2) * p.D] = from_f32<T16>(dfl.x);
          if (2 * j2 + 1 < nout) gdfl[static_cast<int64_t>(2 * j2 + 1) * p.D] = from_f32<T16>(dfl.y);
        }
      }
      // channel tile done: D_skip partials (one row per group and batch row)
      p.dDpart[static_cast<int64_t>(grp * p.B + b) * (p.ndt * kDT) + d] = dDsum + dDlow;
    }
  }
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, SM::TMEM_COLS);
}

}  // namespace wideb

namespace {
template <bool UTM, int NS>
int launch_bwd_wide_t(const BwdParams& p, const Geometry& g, const wideb::Maps& maps, cudaStream_t st) {
  auto kern = wideb::bwd_wide_kernel<UTM, NS>;
  constexpr size_t smem = wideb::Smem<NS>::total;
  static std::atomic<unsigned long long> ok{0};
  const int rc = allow_smem(kern, smem, ok);
  if (rc != 0) return rc;
  const int64_t ctiles = static_cast<int64_t>(g.B) * g.ndt, sms = tmah::sm_count();
  return launch_pdl(kern, dim3(static_cast<unsigned>(ctiles < sms ? ctiles : sms)), dim3(wideb::NTHREADS), smem, st, p, maps);
}
}  // namespace

// Tensor-core backward of 17 to 64 states; returns -1000 if this problem cannot take it or has too few channel tiles to
// fill the GPU.  fp32 logits stay with the recurrent kernel: their gradients are fp32, and two-term operands are not.
int launch_bwd_wide(const BwdParams& p, const Geometry& g, int act, int gate, int bc, void* stream) {
  if (!(g.N > 16 && g.NS <= 64 && g.TC == wideb::Q && act == NAJU_BF16 && gate == NAJU_BF16 && bc == NAJU_BF16)) return -1000;
  if (!wide_walk_pays(g, tmah::sm_count())) return -1000;
  wideb::Maps maps;
  // (du, in u's layout, leaves in 16-byte pieces where that is time-contiguous)
  const bool ok = (p.u_sd == 1 || (reinterpret_cast<uintptr_t>(p.du) & 15) == 0) &&
      (p.u_sd > 1 ? tmah::make_map_tmajor(&maps.u, p.u, act, g.B, g.T, g.D, p.u_sb, p.u_sd, wideb::SLAB, kDT)
                  : tmah::make_map(&maps.u, p.u, act, g.B, g.T, g.D, p.u_sb, p.u_st, kDT, wideb::SLAB)) &&
      tmah::make_map(&maps.fl, p.fl, gate, g.B, g.T, g.D, p.fl_sb, p.fl_st, kDT, wideb::SLAB) &&
      tmah::make_map(&maps.il, p.il, gate, g.B, g.T, g.D, p.il_sb, p.il_st, kDT, wideb::SLAB) &&
      tmah::make_map(&maps.dy, p.dy, act, g.B, g.T, g.D, static_cast<int64_t>(g.T) * g.D, g.D, kDT, wideb::SLAB) &&
      tmah::make_map(&maps.bm, p.Bm, bc, g.B, g.T, g.N, p.bm_sb, p.bm_st, g.NS, wideb::Q) &&
      tmah::make_map(&maps.cm, p.Cm, bc, g.B, g.T, g.N, p.cm_sb, p.cm_st, g.NS, wideb::Q);
  if (!ok) return -1000;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (g.NS == 64) return p.u_sd > 1 ? launch_bwd_wide_t<true, 64>(p, g, maps, st) : launch_bwd_wide_t<false, 64>(p, g, maps, st);
  return p.u_sd > 1 ? launch_bwd_wide_t<true, 32>(p, g, maps, st) : launch_bwd_wide_t<false, 32>(p, g, maps, st);
}

}  // namespace naju
