// Forward gated scan with 17 to 64 states, chunked form on tcgen05 tensor cores: persistent, TMA-fed, warp-specialised.
//
// The mathematics is the 16-state walk's (fwd_tc3.cu; recurrence of naju/scan.py:79-93) on chunks of Q = 32 steps:
//     y_t   = P_t [ <C_t, h> + sum_{s<=t} (C_t . B_s) wt_s ] + D_skip u_t,   wt_s = sigmoid(i_s) u_s / P_s
//     x_end = P_Q [ h + sum_s wt_s B_s ]
// as GEMMs with M = 128 channels (bf16 operands, fp32 accumulators in TMEM):
//     D2[128 x NS] = (w1 + w2 + w3) . B^T                                                   chunk-local state increment
//     D1[128 x 32] = sum of w_i . g_j, i + j <= 4, + (h1 + h2 + h3) . C                     pre-scaled outputs
// with wt, tril(C B^T) = g and h in three bf16 terms each, all 24 bits of an fp32 significand: these problems are the recurrent
// kernels' otherwise, whose arithmetic is fp32 throughout.  (Two-term operands, 16 bits, showed through y's rounding to 16 bits.)
//
// What bounds it: the recurrent kernel does N multiply-adds and N loads' worth of B and C per channel and step on the
// CUDA cores (64 states: 6.7 ms for 8 x 8192 x 4096, 32 states 3.9 ms); here that work is MMAs, and what is left per
// step is the gates and a tile's hand-offs: 2.25 and 1.52 ms, 4.4 and 3.0 us a tile (with two-term
// operands and nothing watched for 1.93 and 1.35 ms).
// Chunks are 32 steps, half the 16-state kernel's, because the carried rows are four times as wide; two sets of
// main warps take the even and the odd tiles, so that one set's gates run while the other waits for its MMAs.
//   warps 0-15   main warps: set s = warp / 8 takes the tiles of its parity, its half g steps [16g, 16g+16), a thread one
//                channel.  Gates -> operand rows; then, when the tile's MMAs are complete, its outputs (P_t and u_t are
//                still in registers).
//   warps 16-23  carry warps: two threads per channel, half of the states each: D2 -> carry (registers), checkpoint,
//                carry-in row of the next tile; deep-gate tiles.
//   warp 24      operand builder: C and B rows into operand layout, G = C B^T by an MMA of its own, masked and split.
//   warp 25      TMA producer: u / f_logit / i_logit in 16-step slabs, the chunk's raw B and C rows.
//   warp 26      MMA issuer.
// A tile whose retention product falls below 2^-80 in any channel runs as the exact recurrence in the carry warps.
// Every wait is bounded.
#include "fwd_common.cuh"
#include "tc_common.cuh"
#include "tma_host.h"

namespace naju {
namespace wide {

using namespace tcx;

constexpr int Q = 32, SLAB = 16, NSLAB = 2;
constexpr int W_CARRY = 16, W_BUILD = 24, W_PROD = 25, W_MMA = 26, NTHREADS = 27 * 32, NCARRY = 256;
static_assert(W_BUILD % 4 == 0, "the builder warp reads accumulator rows 0-31");
constexpr int AW_W1 = 0, AW_W2 = 4, AW_W3 = 8;                  // operand rows [w1 32 | w2 32 | w3 32], per stage
constexpr uint32_t SBO_AW = 12 * 128, AW_BYTES = 16 * SBO_AW;

struct Maps {
  CUtensorMap u, fl, il, bm, cm;
};

template <typename TG, int NS>
struct Smem {
  static constexpr int NC = NS / 8;                                  // 16-byte chunks of a state row
  static constexpr int AH_H1 = 0, AH_H2 = NC, AH_H3 = 2 * NC;        // carry-in rows [h1 NS | h2 NS | h3 NS]
  static constexpr uint32_t SBO_AH = 3 * NC * 128, AH_BYTES = 16 * SBO_AH;
  static constexpr int B1_C = 0, B1_G1 = NC, B1_G2 = NC + 4, B1_G3 = NC + 8;   // rows t: [C NS | g1 32 | g2 32 | g3 32]
  static constexpr uint32_t SBO_B1 = (NC + 12) * 128, B1_BYTES = 4 * SBO_B1;
  static constexpr uint32_t SBO_BB = NC * 128, BB_BYTES = 4 * SBO_BB;  // rows s: [B NS]
  static constexpr uint32_t BC_BYTES = Q * NS * 2;
  static constexpr uint32_t slab_bytes = SLAB * kDT * (2 + 2 * sizeof(TG));
  static constexpr int RING = sizeof(TG) == 2 ? 6 : 4;
  static constexpr uint32_t off_ring = 0;
  // The builder's MMA addresses the 32 C rows of a stage as a 128-row operand: what follows must be readable.
  static constexpr uint32_t off_B1 = off_ring + RING * slab_bytes;     // [2]
  static constexpr uint32_t off_BB = off_B1 + 2 * B1_BYTES;            // [2]
  static constexpr uint32_t off_bc = off_BB + 2 * BB_BYTES;            // [2 tiles][B raw | C raw]
  static constexpr uint32_t off_AH = off_bc + 4 * BC_BYTES;
  static constexpr uint32_t off_AW = off_AH + AH_BYTES;                // [2]
  static constexpr uint32_t total = off_AW + 2 * AW_BYTES;
  static_assert(Q * kDT * 4 <= AW_BYTES, "a tile taken by the exact path uses its own operand rows as scratch");
  static_assert(RING >= 4, "a half waits for its slab by parity: the slot's previous use was filled before the half's own previous slab");
  static_assert(total + 4096 <= 232448, "with the static arrays, within an SM's 227 KB");
  static_assert(off_B1 + B1_BYTES + 16 * SBO_B1 <= total, "the 128-row view of a stage's C rows stays inside shared memory");
  // (D2's largest term has an accumulator of its own, see the MMA issuer)
  static constexpr uint32_t TM_D1 = 0, TM_D2 = 32, TM_D2S = 32 + NS, TM_G = 32 + 2 * NS, TM_STAGE = 64 + 2 * NS,
                            TMEM_COLS = NS == 64 ? 512 : 256;
  static_assert(2 * TM_STAGE <= TMEM_COLS, "");
};

struct Bars {
  unsigned long long full[6], empty[6];
  unsigned long long bc_full[2], bc_empty[2];
  unsigned long long lprod[2];         // the first half's retention products are published
  unsigned long long part[2][NSLAB];   // operand-row chunks of one slab written
  unsigned long long g_full[2];        // the builder's own MMA is complete
  unsigned long long ops_full[2];      // builder -> MMA issuer
  unsigned long long d2_full[2];       // D2 complete
  unsigned long long h_ready;          // carry-in row written
  unsigned long long d1_full[2];       // D1 complete, every operand of the tile read
  unsigned long long y_read[2];        // main warps have read D1
  unsigned long long acc_free[2];      // carry warps have read D2 and s_Rend and written the deep flag
};

// Exact recurrence of one tile straight from global memory (deep gates, or something that is not finite), by the carry
// threads, each with its NSH states from n0 on; the second half's share of y goes through shared memory.
template <typename TA, typename TG, int NSH>
__device__ __noinline__ void exact_tile(const FwdParams& p, const TileCoord& tc, int q, int half, float* s_deep, float (&hw)[NSH], float& Pw) {
  const TA* gu = reinterpret_cast<const TA*>(p.u) + tc.b * p.u_sb + static_cast<int64_t>(tc.t0) * p.u_st + tc.d * p.u_sd;
  const TG* gf = reinterpret_cast<const TG*>(p.fl) + tc.b * p.fl_sb + static_cast<int64_t>(tc.t0) * p.fl_st + tc.d;
  const TG* gi = reinterpret_cast<const TG*>(p.il) + tc.b * p.il_sb + static_cast<int64_t>(tc.t0) * p.il_st + tc.d;
  const int n0 = half * NSH;
  const int64_t bbase = tc.b * p.bm_sb + static_cast<int64_t>(tc.t0) * p.bm_st + n0;
  const int64_t cbase = tc.b * p.cm_sb + static_cast<int64_t>(tc.t0) * p.cm_st + n0;
  const float Dv = tc.d_ok ? p.Dskip[tc.d] : 0.f;
  TA* gy = reinterpret_cast<TA*>(p.y) + (static_cast<int64_t>(tc.b) * p.T + tc.t0) * p.D + tc.d;
  if (half == 0) bar_sync<4, NCARRY>();   // the other half's share is there
  for (int t = 0; t < tc.len; ++t) {
    float f = 1.f, w = 0.f, ut = 0.f;
    if (tc.d_ok) {
      ut = to_f32(gu[t * p.u_st]);
      f = sigmoid_f(to_f32(gf[t * p.fl_st]));
      w = sigmoid_f(to_f32(gi[t * p.il_st])) * ut;
    }
    Pw *= f;
    float acc = 0.f;
#pragma unroll
    for (int n = 0; n < NSH; ++n) {
      const float bv = n0 + n < p.N ? load_dyn(p.Bm, p.bc_dtype, bbase + t * p.bm_st + n) : 0.f;
      const float cv = n0 + n < p.N ? load_dyn(p.Cm, p.bc_dtype, cbase + t * p.cm_st + n) : 0.f;
      hw[n] = fmaf(f, hw[n], w * bv);
      acc = fmaf(cv, hw[n], acc);
    }
    if (half == 1) s_deep[t * kDT + q] = acc;
    else if (tc.d_ok) gy[static_cast<int64_t>(t) * p.D] = from_f32<TA>(fmaf(Dv, ut, acc + s_deep[t * kDT + q]));
  }
  if (half == 1) bar_sync<4, NCARRY>();
  bar_sync<4, NCARRY>();                  // s_deep may be written again
}

template <typename TA, typename TG, bool UTM, int NS>
__global__ void __launch_bounds__(NTHREADS, 1)
fwd_wide_kernel(const FwdParams p, const __grid_constant__ Maps maps) {
  using SM = Smem<TG, NS>;
  constexpr int NSH = NS / 2;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ Bars bars;
  __shared__ int s_stage_deep[2];
  __shared__ int s_bad[2];           // some w of the stage's tile is too large for the factorised form, or not finite
  __shared__ int s_bad_bc[4];        // some B or C of tile `it & 3` is
  __shared__ unsigned int s_tmem;
  __shared__ float s_L[2][kDT];      // retention product of a tile's first 16 steps (as 1 / prod f)
  __shared__ float s_Rend[2][kDT];   // 1 / (retention product of the whole chunk)

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t sbase = smem_u32(smem);
  const int nchunks = p.nchunks, ctiles = p.B * p.ndt;
  const int x_first = static_cast<int>(blockIdx.x), x_step = static_cast<int>(gridDim.x);
  const int ntotal = (x_first < ctiles ? (ctiles - x_first + x_step - 1) / x_step : 0) * nchunks;

  if (tid < 2) s_bad[tid] = 0;
  if (tid == 0) {
    for (int i = 0; i < SM::RING; ++i) {
      mbar_init(smem_u32(&bars.full[i]), 1);
      mbar_init(smem_u32(&bars.empty[i]), 4);      // (arrival counts are in warps)
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&bars.bc_full[i]), 1);
      mbar_init(smem_u32(&bars.bc_empty[i]), 1);
      mbar_init(smem_u32(&bars.lprod[i]), 4);
      for (int k = 0; k < NSLAB; ++k) mbar_init(smem_u32(&bars.part[i][k]), 4);
      mbar_init(smem_u32(&bars.g_full[i]), 1);
      mbar_init(smem_u32(&bars.ops_full[i]), 1);
      mbar_init(smem_u32(&bars.d2_full[i]), 1);
      mbar_init(smem_u32(&bars.d1_full[i]), 1);
      mbar_init(smem_u32(&bars.y_read[i]), 8);
      mbar_init(smem_u32(&bars.acc_free[i]), NCARRY / 32);
    }
    mbar_init(smem_u32(&bars.h_ready), NCARRY / 32);
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(smem_u32(&s_tmem), SM::TMEM_COLS);
  // the upper triangle of g1 / g2 is never written again: clear the shared operands once
  for (uint32_t i = tid * 16; i < 2 * (SM::B1_BYTES + SM::BB_BYTES); i += NTHREADS * 16)
    *reinterpret_cast<uint4*>(smem + SM::off_B1 + i) = make_uint4(0, 0, 0, 0);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  pdl_wait();   // nothing above touches global memory
  if (blockIdx.x == 0 && tid == 0) {
    atomicOr(p.fwd_form, 1);  // tell the backward how the forward ran
    p.hdr->form = NAJU_FORM_TC_WALK;
  }
  auto timeout = [&]() { atomicOr(&p.hdr->status, NAJU_ST_MMA_TIMEOUT); };

  if (warp == W_PROD) {
    // ===================================================================== TMA producer
    if (lane == 0) {
      uint32_t slab = 0;
      int it = 0;
      for (int x = x_first; x < ctiles; x += x_step) {
        const int b = x / p.ndt, d0 = (x - b * p.ndt) * kDT;
        for (int c = 0; c < nchunks; ++c, ++it) {
          const int t0 = c * Q, rb = it & 1;
          if (it >= 2 && !mbar_wait(smem_u32(&bars.bc_empty[rb]), ((it >> 1) & 1) ^ 1)) timeout();
          {
            const uint32_t bar = smem_u32(&bars.bc_full[rb]), dst = sbase + SM::off_bc + rb * 2 * SM::BC_BYTES;
            mbar_arrive_expect_tx(bar, 2 * SM::BC_BYTES);
            tma_load_3d(dst, &maps.bm, 0, t0, b, bar);
            tma_load_3d(dst + SM::BC_BYTES, &maps.cm, 0, t0, b, bar);
          }
          for (int k = 0; k < NSLAB; ++k, ++slab) {
            const uint32_t slot = slab % SM::RING, ph = (slab / SM::RING) & 1;
            if (slab >= SM::RING && !mbar_wait(smem_u32(&bars.empty[slot]), ph ^ 1)) timeout();
            const uint32_t bar = smem_u32(&bars.full[slot]), dst = sbase + SM::off_ring + slot * SM::slab_bytes;
            mbar_arrive_expect_tx(bar, SM::slab_bytes);
            // (a time-contiguous u is mapped (T, D, B): its slab lands as [channel][step])
            if (UTM) tma_load_3d(dst, &maps.u, t0 + k * SLAB, d0, b, bar);
            else tma_load_3d(dst, &maps.u, d0, t0 + k * SLAB, b, bar);
            tma_load_3d(dst + SLAB * kDT * 2, &maps.fl, d0, t0 + k * SLAB, b, bar);
            tma_load_3d(dst + SLAB * kDT * (2 + sizeof(TG)), &maps.il, d0, t0 + k * SLAB, b, bar);
          }
        }
      }
    }
  } else if (warp == W_BUILD) {
    // ===================================================================== operand builder (lane = step)
    const int t = lane;
    const uint32_t idG = umma_idesc(128, Q, 1);
    for (int it = 0; it < ntotal; ++it) {
      const int st = it & 1;
      const uint32_t par = (it >> 1) & 1;
      if (!mbar_wait(smem_u32(&bars.bc_full[st]), par)) timeout();
      // stage st: the MMAs of the tile two back have read B1 / BB
      if (it >= 2 && !mbar_wait(smem_u32(&bars.d1_full[st]), par ^ 1)) timeout();
      unsigned char* s_B1 = smem + SM::off_B1 + st * SM::B1_BYTES;
      unsigned char* s_BB = smem + SM::off_BB + st * SM::BB_BYTES;
      const unsigned char* raw = smem + SM::off_bc + st * 2 * SM::BC_BYTES;
      // 16-byte pieces: eight lanes take a row's neighbours in turn (the raw rows are read without bank conflicts)
      uint32_t bad = 0;
#pragma unroll 4
      for (int i = lane; i < Q * SM::NC; i += 32) {
        const int r = i / SM::NC, k = i % SM::NC;
        const uint4 bv = *reinterpret_cast<const uint4*>(raw + i * 16), cv = *reinterpret_cast<const uint4*>(raw + SM::BC_BYTES + i * 16);
        *reinterpret_cast<uint4*>(s_BB + op_off16(r, k * 8, SM::SBO_BB)) = bv;
        *reinterpret_cast<uint4*>(s_B1 + op_off16(r, (SM::B1_C + k) * 8, SM::SBO_B1)) = cv;
        bad |= too_large_bf16x8(bv) | too_large_bf16x8(cv);
      }
      // (four slots: the carry warps are at most two tiles behind)
      const bool bad_bc = __any_sync(0xffffffffu, bad != 0);
      if (lane == 0) s_bad_bc[it & 3] = bad_bc ? 1 : 0;
      fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        tc_fence_after();
        mbar_arrive(smem_u32(&bars.bc_empty[st]));  // the raw rows have been read
        // G[t, s] = <C_t, B_s> (of the 128 rows 32 are real; the others are never read)
        const uint64_t dC = umma_desc(sbase + SM::off_B1 + st * SM::B1_BYTES, 128, SM::SBO_B1),
                       dB = umma_desc(sbase + SM::off_BB + st * SM::BB_BYTES, 128, SM::SBO_BB);
#pragma unroll
        for (int k = 0; k < NS / 16; ++k) umma_bf16(tmem + st * SM::TM_STAGE + SM::TM_G, dC + k * 16, dB + k * 16, idG, k > 0);
        umma_commit(smem_u32(&bars.g_full[st]));
      }
      __syncwarp();
      if (!mbar_wait(smem_u32(&bars.g_full[st]), par)) timeout();
      __syncwarp();
      tc_fence_after();
      unsigned char* row = s_B1 + static_cast<uint32_t>(t >> 3) * SM::SBO_B1 + static_cast<uint32_t>(t & 7) * 16;
#pragma unroll
      for (int c16 = 0; c16 < 2; ++c16) {
        uint32_t x[16];
        tmem_ld16_async(tmem + st * SM::TM_STAGE + SM::TM_G + 16 * c16, x);
        tmem_ld_wait16(x);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c8 = 2 * c16 + h;
          if (c8 <= (t >> 3)) {
            uint32_t g1[4], g2[4], g3[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int s = 8 * c8 + 2 * k;
              split3(make_float2(s <= t ? __uint_as_float(x[8 * h + 2 * k]) : 0.f,
                                 s + 1 <= t ? __uint_as_float(x[8 * h + 2 * k + 1]) : 0.f), g1[k], g2[k], g3[k]);
            }
            *reinterpret_cast<uint4*>(row + (SM::B1_G1 + c8) * 128) = make_uint4(g1[0], g1[1], g1[2], g1[3]);
            *reinterpret_cast<uint4*>(row + (SM::B1_G2 + c8) * 128) = make_uint4(g2[0], g2[1], g2[2], g2[3]);
            *reinterpret_cast<uint4*>(row + (SM::B1_G3 + c8) * 128) = make_uint4(g3[0], g3[1], g3[2], g3[3]);
          }
        }
      }
      fence_async_smem();
      tc_fence_before();
      mbar_arrive_warp(smem_u32(&bars.ops_full[st]));
    }
  } else if (warp == W_MMA) {
    // ===================================================================== MMA issuer
    if (lane == 0) {
      const uint32_t idN = umma_idesc(128, NS, 1) | (1u << 16), id32 = umma_idesc(128, Q, 1);
      auto off = [](uint32_t bytes) { return static_cast<uint64_t>(bytes >> 4); };
      const uint64_t dAH = umma_desc(sbase + SM::off_AH, 128, SM::SBO_AH);
      for (int it = 0; it < ntotal; ++it) {
        const int st = it & 1;
        const uint32_t par = (it >> 1) & 1;
        const uint64_t dAW = umma_desc(sbase + SM::off_AW + st * AW_BYTES, 128, SBO_AW);
        const uint64_t dB1 = umma_desc(sbase + SM::off_B1 + st * SM::B1_BYTES, 128, SM::SBO_B1);
        // the B rows read MN-major (N = state contiguous, K = step)
        const uint64_t dBB = umma_desc(sbase + SM::off_BB + st * SM::BB_BYTES, SM::SBO_BB, 128);
        const uint32_t tst = tmem + st * SM::TM_STAGE;
        if (!mbar_wait(smem_u32(&bars.ops_full[st]), par)) timeout();
        // every reader of the stage's accumulators of two tiles back is done
        if (it >= 2 && !mbar_wait(smem_u32(&bars.y_read[st]), par ^ 1)) timeout();
        if (it >= 2 && !mbar_wait(smem_u32(&bars.acc_free[st]), par ^ 1)) timeout();
        if (!mbar_wait(smem_u32(&bars.part[st][0]), par)) timeout();
        if (!mbar_wait(smem_u32(&bars.part[st][1]), par)) timeout();
        tc_fence_after();
        // D2: the small terms in an accumulator of their own, added up by the carry warps.  (An accumulating MMA truncates;
        // w1 . B alone hardly has bits to lose.)
#pragma unroll
        for (int ks = 0; ks < NSLAB; ++ks) {
          const uint64_t bb = dBB + off(2 * ks * SM::SBO_BB);
          umma_bf16(tst + SM::TM_D2S, dAW + off((AW_W3 + 2 * ks) * 128), bb, idN, ks > 0);
          umma_bf16(tst + SM::TM_D2, dAW + off((AW_W1 + 2 * ks) * 128), bb, idN, ks > 0);
        }
#pragma unroll
        for (int ks = 0; ks < NSLAB; ++ks) umma_bf16(tst + SM::TM_D2S, dAW + off((AW_W2 + 2 * ks) * 128), dBB + off(2 * ks * SM::SBO_BB), idN, 1u);
        umma_commit(smem_u32(&bars.d2_full[st]));
        // D1: the products of terms that reach 24 bits, the smallest first
        auto wg = [&](int w, int g, bool first) {
#pragma unroll
          for (int ks = 0; ks < NSLAB; ++ks)
            umma_bf16(tst + SM::TM_D1, dAW + off((w + 2 * ks) * 128), dB1 + off((g + 2 * ks) * 128), id32, !first || ks > 0);
        };
        wg(AW_W3, SM::B1_G1, true);
        wg(AW_W1, SM::B1_G3, false);
        wg(AW_W2, SM::B1_G2, false);
        wg(AW_W2, SM::B1_G1, false);
        wg(AW_W1, SM::B1_G2, false);
        wg(AW_W1, SM::B1_G1, false);
        // (the accumulators of a tile that the exact path takes are junk and are never read)
        if (!mbar_wait(smem_u32(&bars.h_ready), it & 1)) timeout();
        tc_fence_after();
#pragma unroll
        for (int term = 2; term >= 0; --term)
#pragma unroll
          for (int k = 0; k < NS / 16; ++k)
            umma_bf16(tst + SM::TM_D1, dAH + off((term * SM::NC + 2 * k) * 128), dB1 + off((SM::B1_C + 2 * k) * 128), id32, 1u);
        umma_commit(smem_u32(&bars.d1_full[st]));
      }
    }
  } else if (warp >= W_CARRY && warp < W_BUILD) {
    // ===================================================================== carry warps
    const int half = (warp - W_CARRY) >> 2, q = (warp & 3) * 32 + lane, n0 = half * NSH;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    unsigned char* h_row = smem + SM::off_AH + static_cast<uint32_t>(q >> 3) * SM::SBO_AH + static_cast<uint32_t>(q & 7) * 16;
    float hc[NSH];    // states entering the current chunk
    float Pc = 1.f;   // cumulative decay
    auto write_h_row = [&]() {
#pragma unroll
      for (int k = 0; k < NSH / 8; ++k) {
        uint32_t h1[4], h2[4], h3[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split3(make_float2(hc[8 * k + 2 * j], hc[8 * k + 2 * j + 1]), h1[j], h2[j], h3[j]);
        const int ch = half * (NSH / 8) + k;
        *reinterpret_cast<uint4*>(h_row + (SM::AH_H1 + ch) * 128) = make_uint4(h1[0], h1[1], h1[2], h1[3]);
        *reinterpret_cast<uint4*>(h_row + (SM::AH_H2 + ch) * 128) = make_uint4(h2[0], h2[1], h2[2], h2[3]);
        *reinterpret_cast<uint4*>(h_row + (SM::AH_H3 + ch) * 128) = make_uint4(h3[0], h3[1], h3[2], h3[3]);
      }
      fence_async_smem();
      tc_fence_before();
      mbar_arrive_warp(smem_u32(&bars.h_ready));
    };
    auto load_h0 = [&](int x) {
      const int b = x / p.ndt, d = (x - b * p.ndt) * kDT + q;
#pragma unroll
      for (int n = 0; n < NSH; ++n)
        hc[n] = (p.h0 != nullptr && d < p.D && n0 + n < p.N) ? p.h0[(static_cast<int64_t>(b) * p.D + d) * p.N + n0 + n] : 0.f;
      Pc = 1.f;
    };
    // Not 0 if a state entering the current chunk is too large or not finite.  Looked at where states come in and behind the exact
    // path only: what the factorised path takes leaves them finite, and here they are on the chain from tile to tile (0.15 ms of
    // 2.4 at B=8, T=8192, D=4096, N=64).
    float hz = 0.f;
    auto check_states = [&]() {
      float2 z = make_float2(0.f, 0.f);
#pragma unroll
      for (int n = 0; n < NSH; n += 2) z = watch(z, make_float2(hc[n], hc[n + 1]), kOverState);
      hz = z.x + z.y;
    };
    if (x_first < ctiles) {
      load_h0(x_first);
      write_h_row();
      check_states();
    }
    int it = 0;
    for (int x = x_first; x < ctiles; x += x_step) {
      TileCoord tcd;
      tcd.per_chunk = ctiles;
      tcd.rem = x;
      tcd.b = x / p.ndt;
      tcd.dt = x - tcd.b * p.ndt;
      tcd.d0 = tcd.dt * kDT;
      tcd.cols = min(kDT, p.D - tcd.d0);
      tcd.d = tcd.d0 + q;
      tcd.d_ok = tcd.d < p.D;
      for (int c = 0; c < nchunks; ++c, ++it) {
        const int st = it & 1;
        const uint32_t par = (it >> 1) & 1;
        if (!mbar_wait(smem_u32(&bars.d2_full[st]), par)) timeout();
        // (the writers of s_Rend and s_bad arrived on `part`, the writer of s_bad_bc on `ops_full`)
        if (!mbar_wait(smem_u32(&bars.part[st][0]), par)) timeout();
        if (!mbar_wait(smem_u32(&bars.part[st][1]), par)) timeout();
        if (!mbar_wait(smem_u32(&bars.ops_full[st]), par)) timeout();
        const float Rend = s_Rend[st][q];
        // The exact path takes a tile with deep gates, and one with a value that is not finite: every step of a channel meets
        // the others' in an MMA, masked by zeros.
        const bool deep = bar_or<2, NCARRY>(!(Rend < kRMax) || !(hz == 0.f) || (s_bad[st] | s_bad_bc[it & 3]) != 0);
        if (tid == W_CARRY * 32) {
          s_stage_deep[st] = deep ? 1 : 0;
          s_bad[st] = 0;
        }
        tc_fence_after();
        if (deep) {
          if (tid == W_CARRY * 32) atomicOr(p.fwd_form, 2);
          tcd.c = c;
          tcd.tile = static_cast<int64_t>(c) * ctiles + x;
          tcd.t0 = c * Q;
          tcd.len = min(Q, p.T - tcd.t0);
          // (copies: what a call takes by reference lives in local memory everywhere)
          const TileCoord at = tcd;
          float hw[NSH], Pw = Pc;
#pragma unroll
          for (int n = 0; n < NSH; ++n) hw[n] = hc[n];
          if (!mbar_wait(smem_u32(&bars.d1_full[st]), par)) timeout();   // the operand rows are scratch now
          exact_tile<TA, TG, NSH>(p, at, q, half, reinterpret_cast<float*>(smem + SM::off_AW + st * AW_BYTES), hw, Pw);
#pragma unroll
          for (int n = 0; n < NSH; ++n) hc[n] = hw[n];
          Pc = Pw;
          check_states();
        } else {
          const float P = __frcp_rn(Rend), Pl = P * fmaf(-P, Rend, 1.f);   // (P + Pl = 1 / Rend)
#pragma unroll
          for (int k = 0; k < NSH / 8; ++k) {
            uint32_t sr[8], ss[8];
            tmem_ld8_async(tmem + st * SM::TM_STAGE + lane_off + SM::TM_D2 + n0 + 8 * k, sr);
            tmem_ld8_async(tmem + st * SM::TM_STAGE + lane_off + SM::TM_D2S + n0 + 8 * k, ss);
            tmem_ld_wait8(sr, ss);
#pragma unroll
            for (int n = 0; n < 8; ++n)
              hc[8 * k + n] = fmaf(P, __uint_as_float(sr[n]), fmaf(P, __uint_as_float(ss[n]), fmaf(Pl, __uint_as_float(sr[n]), P * hc[8 * k + n])));
          }
          Pc *= P;
        }
        tc_fence_before();
        mbar_arrive_warp(smem_u32(&bars.acc_free[st]));
        // this tile's MMAs have read the carry-in row: the next tile's, which they wait for, before anything else
        if (!mbar_wait(smem_u32(&bars.d1_full[st]), par)) timeout();
        if (c + 1 < nchunks) write_h_row();
        // the chunk-end state: checkpoint, the last chunk's also the final state
        const int64_t slot = (static_cast<int64_t>(c) * ctiles + x) * kDT + q;
        float4* dstS = reinterpret_cast<float4*>(p.ckS + slot * NS + n0);
#pragma unroll
        for (int k = 0; k < NSH / 4; ++k) dstS[k] = make_float4(hc[4 * k], hc[4 * k + 1], hc[4 * k + 2], hc[4 * k + 3]);
        if (half == 0) p.ckP[slot] = Pc;
        if (c + 1 == nchunks) {
          if (tcd.d_ok) {
            const int64_t ch = static_cast<int64_t>(tcd.b) * p.D + tcd.d;
            if (p.hT != nullptr)
#pragma unroll
              for (int n = 0; n < NSH; ++n)
                if (n0 + n < p.N) p.hT[ch * p.N + n0 + n] = hc[n];
            if (p.pT != nullptr && half == 0) p.pT[ch] = Pc;
          }
          if (x + x_step >= ctiles) continue;
          load_h0(x + x_step);
          write_h_row();
          check_states();
        }
      }
    }
  } else if (warp < W_CARRY) {
    // ===================================================================== main warps
    const int set = warp >> 3, g = (warp >> 2) & 1;   // tiles of this parity, steps [16 g, 16 g + 16)
    const int q = (warp & 3) * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const float2 kk = make_float2(kNegLog2e, kNegLog2e), one2 = make_float2(1.f, 1.f);
    const int st = set;
    unsigned char* a_row = smem + SM::off_AW + st * AW_BYTES + static_cast<uint32_t>(q >> 3) * SBO_AW + static_cast<uint32_t>(q & 7) * 16;
    int x = x_first, c = set;
#pragma unroll 1
    for (int it = set; it < ntotal; it += 2, c += 2) {
      while (c >= nchunks) {
        c -= nchunks;
        x += x_step;
      }
      const uint32_t par = (it >> 1) & 1;
      const int b = x / p.ndt, d = (x - b * p.ndt) * kDT + q, t0 = c * Q, nvalid = p.T - t0 - SLAB * g;
      const uint32_t sidx = static_cast<uint32_t>(it) * NSLAB + g, slot = sidx % SM::RING, ph = (sidx / SM::RING) & 1;
      if (!mbar_wait(smem_u32(&bars.full[slot]), ph)) timeout();
      const unsigned char* sl = smem + SM::off_ring + slot * SM::slab_bytes;
      const TA* s_u = reinterpret_cast<const TA*>(sl) + q;           // [step][channel]
      const TA* s_ut = reinterpret_cast<const TA*>(sl) + q * SLAB;    // [channel][step] (time-contiguous u)
      const TG* s_fl = reinterpret_cast<const TG*>(sl + SLAB * kDT * 2) + q;
      const TG* s_il = s_fl + SLAB * kDT;
      // ---- retention of the own 16 steps: L_j = prod_{i<=j} (1 + e^{-f_logit_i})
      float2 L[SLAB / 2];
      {
        float2 qv[SLAB / 2];
#pragma unroll
        for (int j2 = 0; j2 < SLAB / 2; ++j2) {
          const float2 fl2 = mul2(make_float2(ld_as_f32(s_fl, (2 * j2) * kDT), ld_as_f32(s_fl, (2 * j2 + 1) * kDT)), kk);
          qv[j2] = add2(make_float2(fast_ex2(fl2.x), fast_ex2(fl2.y)), one2);
        }
        // steps past the end of the sequence arrive as zeros: neutral (f = 1, u = 0)
        if (nvalid < SLAB) {
#pragma unroll
          for (int j2 = 0; j2 < SLAB / 2; ++j2) {
            if (2 * j2 >= nvalid) qv[j2].x = 1.f;
            if (2 * j2 + 1 >= nvalid) qv[j2].y = 1.f;
          }
        }
        float run = 1.f;
#pragma unroll
        for (int j2 = 0; j2 < SLAB / 2; ++j2) {
          L[j2] = mul2(make_float2(run, run), make_float2(qv[j2].x, qv[j2].x * qv[j2].y));
          run = L[j2].y;
        }
      }
      float Rstart = 1.f;
      if (g == 0) {
        s_L[st][q] = L[SLAB / 2 - 1].y;
        mbar_arrive_warp(smem_u32(&bars.lprod[st]));
      } else {
        if (!mbar_wait(smem_u32(&bars.lprod[st]), par)) timeout();
        Rstart = s_L[st][q];
        s_Rend[st][q] = Rstart * L[SLAB / 2 - 1].y;
      }
      const float2 Rs2 = make_float2(Rstart, Rstart);
      float2 Pv[SLAB / 2];
      float2 uv[SLAB / 2];
      float2 wz = make_float2(0.f, 0.f);
#pragma unroll
      for (int j8 = 0; j8 < SLAB / 8; ++j8) {
        uint32_t w1[4], w2[4], w3[4];
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const int j2 = 4 * j8 + jj;
          // (the floor of the exact kernels' gate: e^80 is finite, and so is its reciprocal's product with R)
          const float2 il2 = mul2(make_float2(fmaxf(ld_as_f32(s_il, (2 * j2) * kDT), -80.f), fmaxf(ld_as_f32(s_il, (2 * j2 + 1) * kDT), -80.f)), kk);
          const float2 opb = add2(make_float2(fast_ex2(il2.x), fast_ex2(il2.y)), one2);   // 1 / i_t
          uv[j2] = UTM ? ld_pair_as_f32(s_ut + 2 * j2) : make_float2(ld_as_f32(s_u, (2 * j2) * kDT), ld_as_f32(s_u, (2 * j2 + 1) * kDT));
          const float2 R = mul2(Rs2, L[j2]);
          Pv[j2] = make_float2(fast_rcp(R.x), fast_rcp(R.y));           // P_t = 1 / R_t
          // (u_t i_t R_t; the reciprocal's last bit goes into the product: the final state's error against 64 bits stays the recurrent
          // kernel's with it)
          const float2 ig = make_float2(fast_rcp(opb.x), fast_rcp(opb.y)), iR = mul2(ig, R);
          const float2 w = mul2(uv[j2], fma2(iR, fma2(make_float2(-opb.x, -opb.y), ig, one2), iR));
          wz = watch(wz, w, kOverW);
          split3(w, w1[jj], w2[jj], w3[jj]);
        }
        const int ch = 2 * g + j8;
        *reinterpret_cast<uint4*>(a_row + (AW_W1 + ch) * 128) = make_uint4(w1[0], w1[1], w1[2], w1[3]);
        *reinterpret_cast<uint4*>(a_row + (AW_W2 + ch) * 128) = make_uint4(w2[0], w2[1], w2[2], w2[3]);
        *reinterpret_cast<uint4*>(a_row + (AW_W3 + ch) * 128) = make_uint4(w3[0], w3[1], w3[2], w3[3]);
      }
      if (!(wz.x + wz.y == 0.f)) s_bad[st] = 1;
      mbar_arrive_warp(smem_u32(&bars.empty[slot]));   // the slab has been read
      fence_async_smem();
      tc_fence_before();
      mbar_arrive_warp(smem_u32(&bars.part[st][g]));
      const float Dv = d < p.D ? __ldg(p.Dskip + d) : 0.f;
      const int nout = d < p.D ? nvalid : 0;
      TA* gy = reinterpret_cast<TA*>(p.y) + (static_cast<int64_t>(b) * p.T + t0 + SLAB * g) * p.D + d;
      // ---- the tile's outputs
      if (!mbar_wait(smem_u32(&bars.acc_free[st]), par)) timeout();   // (the deep flag's writer arrived here)
      if (!mbar_wait(smem_u32(&bars.d1_full[st]), par)) timeout();
      tc_fence_after();
      if (s_stage_deep[st] == 0) {
        uint32_t v[16];
        __syncwarp();
        tmem_ld16_async(tmem + st * SM::TM_STAGE + lane_off + SM::TM_D1 + SLAB * g, v);
        tmem_ld_wait16(v);
        const float2 Dv2 = make_float2(Dv, Dv);
#pragma unroll
        for (int j2 = 0; j2 < SLAB / 2; ++j2) {
          float2 y = mul2(Pv[j2], make_float2(__uint_as_float(v[2 * j2]), __uint_as_float(v[2 * j2 + 1])));
          if (Dv != 0.f) y = fma2(Dv2, uv[j2], y);
          if (2 * j2 < nout) gy[static_cast<int64_t>(2 * j2) * p.D] = from_f32<TA>(y.x);
          if (2 * j2 + 1 < nout) gy[static_cast<int64_t>(2 * j2 + 1) * p.D] = from_f32<TA>(y.y);
        }
      }
      tc_fence_before();
      mbar_arrive_warp(smem_u32(&bars.y_read[st]));
    }
  }
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, SM::TMEM_COLS);
  finish_forward<TA>(p);
}

}  // namespace wide

namespace {
template <typename TG, bool UTM, int NS>
int launch_wide_t(const FwdParams& p, const Geometry& g, const wide::Maps& maps, cudaStream_t st) {
  auto kern = wide::fwd_wide_kernel<__nv_bfloat16, TG, UTM, NS>;
  constexpr size_t smem = wide::Smem<TG, NS>::total;
  static std::atomic<unsigned long long> ok{0};
  int rc = allow_smem(kern, smem, ok);
  if (rc == 0) rc = launch_init(p.hdr, 256, p.fwd_form, st);
  if (rc != 0) return rc;
  const int64_t ctiles = static_cast<int64_t>(g.B) * g.ndt, sms = tmah::sm_count();
  return launch_pdl(kern, dim3(static_cast<unsigned>(ctiles < sms ? ctiles : sms)), dim3(wide::NTHREADS), smem, st, p, maps);
}
}  // namespace

// Tensor-core forward of 17 to 64 states; returns -1000 if this problem cannot take it, or if it has too few channel
// tiles to fill the GPU by walking them (the recurrent kernel spreads over time as well).
int launch_fwd_wide(const FwdParams& p, const Geometry& g, int act, int gate, int bc, void* stream) {
  if (!(g.N > 16 && g.NS <= 64 && g.TC == wide::Q && act == NAJU_BF16 && bc == NAJU_BF16 && (gate == NAJU_BF16 || gate == NAJU_F32))) return -1000;
  if (g.ntiles >= (1LL << 31)) return -1000;
  if (!wide_walk_pays(g, tmah::sm_count())) return -1000;
  wide::Maps maps;
  const bool ok =
      (p.u_sd > 1 ? tmah::make_map_tmajor(&maps.u, p.u, act, g.B, g.T, g.D, p.u_sb, p.u_sd, wide::SLAB, kDT)
                  : tmah::make_map(&maps.u, p.u, act, g.B, g.T, g.D, p.u_sb, p.u_st, kDT, wide::SLAB)) &&
      tmah::make_map(&maps.fl, p.fl, gate, g.B, g.T, g.D, p.fl_sb, p.fl_st, kDT, wide::SLAB) &&
      tmah::make_map(&maps.il, p.il, gate, g.B, g.T, g.D, p.il_sb, p.il_st, kDT, wide::SLAB) &&
      tmah::make_map(&maps.bm, p.Bm, bc, g.B, g.T, g.N, p.bm_sb, p.bm_st, g.NS, wide::Q) &&
      tmah::make_map(&maps.cm, p.Cm, bc, g.B, g.T, g.N, p.cm_sb, p.cm_st, g.NS, wide::Q);
  if (!ok) return -1000;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool utm = p.u_sd > 1;
  if (g.NS == 64) {
    if (gate == NAJU_F32) return utm ? launch_wide_t<float, true, 64>(p, g, maps, st) : launch_wide_t<float, false, 64>(p, g, maps, st);
    return utm ? launch_wide_t<__nv_bfloat16, true, 64>(p, g, maps, st) : launch_wide_t<__nv_bfloat16, false, 64>(p, g, maps, st);
  }
  if (gate == NAJU_F32) return utm ? launch_wide_t<float, true, 32>(p, g, maps, st) : launch_wide_t<float, false, 32>(p, g, maps, st);
  return utm ? launch_wide_t<__nv_bfloat16, true, 32>(p, g, maps, st) : launch_wide_t<__nv_bfloat16, false, 32>(p, g, maps, st);
}

}  // namespace naju
