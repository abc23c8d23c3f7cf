// Backward gated scan, exact recurrent form: every gradient in one reverse-time pass,
// without materialising the state history.
//
// Adjoint of naju/scan.py:79-93 as written out in naju/cuda/naju_cuda.cu:85-144:
//   xbar_t = dy_t C_t + f_{t+1} xbar_{t+1}
//   dC_t[n] = sum_d dy_t x_t[n]          dB_t[n] = sum_d xbar_t[n] w_t      (w = i u)
//   g_t = <xbar_t, B_t>   du_t = i_t g_t + D_skip dy_t   d i_logit_t = g_t w_t (1 - i_t)
//   d f_logit_t = (1 - f_t) r_t,  r_t = <xbar_t, x_t> - w_t g_t
// (the last line is the division-free form naju/chunk_bwd_triton.py:90-91 uses).
//
// r_t obeys a scalar recurrence, r_t = r_{t+1} + dy_t <C_t, x_t> - w_t g_t, seeded at the
// chunk end by r = <carry_in, x_end>.  That removes the need to hold x_t and xbar_t at the
// same time: a tile (TC steps x 128 channels; a thread owns four channels x K states, simt_common.cuh) is
// walked once forward from the chunk-start state the forward saved (states, dC, dy*cx, the adjoint
// aggregate) and once in reverse (adjoint, dB, g, r); the elementwise gradients follow from g and r in a
// pass over the tile that reads the logits again (they are still in L2).  The adjoint carry crosses chunks
// by the same bounded decoupled look-back as the forward, run towards later chunks.
// Shared memory holds the gates of kSB = 32 steps; the 64-step chunks of the tensor-core kernels, whose
// checkpoints this kernel takes over when their backward stands down, go through it in two pieces.
// dB/dC are reduced over the tile's channels in registers, by a fixed-order warp reduce-scatter and across
// the warps, and written as per-channel-tile partials; a finalize kernel adds those (deterministic).
#include <algorithm>

#include "simt_common.cuh"
#include "tma_host.h"

namespace naju {

using namespace simt;

template <int NS>
struct BwdShape : Shape<NS> {
  // steps between two cross-warp flushes of the dB / dC partial sums
  static constexpr int G = NS == 16 ? 16 : NS == 32 ? 8 : 8;
  static constexpr int part_floats = Shape<NS>::W * G * NS;
};

template <typename TA, typename TG, int NS, int NH>
__global__ void __launch_bounds__(Shape<NS>::NT, NS == 128 ? 1 : NS == 64 ? 2 : NH == 2 ? 2 : 3)
bwd_simt_kernel(const BwdParams p) {
  using S = BwdShape<NS>;
  constexpr int K = S::K, L = S::L, GW = S::GW, W = S::W, NT = S::NT, G = S::G, TC = NH * kSB;
  using RG = ReduceGroups<K, L, GW>;
  extern __shared__ __align__(16) float sm[];
  float* s_f = sm;                       // [kSB][128] retention; du on its way out of a time-contiguous layout
  float* s_w = s_f + kSB * kDT;          // [kSB][128] i u
  float* s_dy = s_w + kSB * kDT;         // [kSB][128] dy; g replaces it in the reverse walk
  float* s_a = s_dy + kSB * kDT;         // [TC][128] dy_t <C_t, x_t>; r replaces it in the reverse walk
  float* s_B = s_a + TC * kDT;           // [TC][NS]
  float* s_C = s_B + TC * NS;            // [TC][NS]
  float* s_part = s_C + TC * NS;         // [W][G][NS]; also the dD partials [W][128]
  __shared__ unsigned int s_ticket;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  // the tensor-core backward was launched for this call and has done the work
  if (tc_did_it(p)) return;
  if (blockIdx.x == 0 && tid == 0) p.hdr->form = NAJU_FORM_RECURRENT;

  const int q = lane % L, g = lane / L, chan0 = (warp * GW + g) * kC, my_ch = chan0 + chan_of<L>(q);
  const bool ch_writer = L == 4 || (q % (L / 4)) == 0;
  const int part_n = q * K + RG::base(g);
  const bool part_writer = !RG::dup || (g & 1) == 0;
  const int per_chunk = p.B * p.ndt;

  // Persistent CTAs: each takes tile tickets (reverse-time-major, so the chunk a tile waits on is
  // always held by a running CTA or done) until they run out.  The grid is a few CTAs per SM, which
  // also makes the stand-down above cost a few microseconds instead of one CTA launch per tile.
  for (;;) {
    __syncthreads();  // the previous tile is done with shared memory (and with s_ticket)
    if (tid == 0) s_ticket = atomicAdd(&p.hdr->ticket, 1u);
    __syncthreads();
    const int order = static_cast<int>(s_ticket / per_chunk);  // 0 = last chunk in time
    const int rem = static_cast<int>(s_ticket % per_chunk);
    if (order >= p.nchunks) return;
    const int c = p.nchunks - 1 - order;
    const int b = rem / p.ndt, dt = rem % p.ndt;
    const int64_t tile = static_cast<int64_t>(c) * per_chunk + rem;
    const int t0 = c * TC, len = min(TC, p.T - t0), d0 = dt * kDT, cols = min(kDT, p.D - d0), d = d0 + chan0;
    const int64_t slot0 = tile * kDT + chan0, bd0 = static_cast<int64_t>(b) * p.D + d;
    const int64_t part_row0 = (static_cast<int64_t>(b) * p.T + t0) * p.ndt + dt;  // + t*ndt
    float4 dd = make_float4(0.f, 0.f, 0.f, 0.f);

    auto stage = [&](int h, float4& dd) {
      if (p.u_sd > 1) {
        load_tmajor<TA, NT>(s_w, reinterpret_cast<const TA*>(p.u) + b * p.u_sb + t0 + h * kSB + static_cast<int64_t>(d0) * p.u_sd,
                            p.u_sd, len - h * kSB, cols, tid);
        __syncthreads();
      }
      stage_gates<TA, TG, NT, true>(p, s_f, s_w, s_dy, b, t0 + h * kSB, len - h * kSB, d0, tid, dd);
    };
    // the partial sums of steps [h kSB + tg, + G) over the tile's channels, summed over the warps
    auto flush = [&](float* part, int t_first) {
      __syncthreads();
      for (int e = tid; e < G * NS; e += NT) {
        const int gg = e / NS, n = e % NS;
        if (t_first + gg < len) {
          float s = 0.f;
#pragma unroll
          for (int wq = 0; wq < W; ++wq) s += s_part[(wq * G + gg) * NS + n];
          part[(part_row0 + static_cast<int64_t>(t_first + gg) * p.ndt) * NS + n] = s;
        }
      }
      __syncthreads();
    };
    auto chunk_start_state = [&](float (&v)[kC][K]) {   // the forward's inclusive state of the previous chunk, or h0
      if (c == 0) get_user_state<K>(p.h0, bd0, d, p.D, p.N, q, v);
      else get_state<NS, K>(p.ckS, slot0 - static_cast<int64_t>(per_chunk) * kDT, q, v);
    };

    float x[kC][K];
    {
      StageBC<NS, NT, TC> bc;
      bc.load(p, b, t0, len, tid);
      chunk_start_state(x);
      stage(0, dd);
      bc.store(p, s_B, s_C, b, t0, len, tid);
    }
    __syncthreads();

    // ---------------- forward walk: states, dC partials, a_t, adjoint aggregate
    float lam[kC][K], P[kC];
    [[maybe_unused]] float xh[NH == 2 ? kC : 1][NH == 2 ? K : 1];   // state between the two pieces
#pragma unroll
    for (int k = 0; k < kC; ++k) {
      P[k] = 1.f;
#pragma unroll
      for (int n = 0; n < K; ++n) lam[k][n] = 0.f;
    }
#pragma unroll 1
    for (int h = 0; h < NH; ++h) {
      if (h > 0) {
        if constexpr (NH == 2)
#pragma unroll
          for (int k = 0; k < kC; ++k)
#pragma unroll
            for (int n = 0; n < K; ++n) xh[k][n] = x[k][n];
        stage(h, dd);
        __syncthreads();
      }
#pragma unroll 1
      for (int tg = 0; tg < kSB; tg += G) {
#pragma unroll 2
        for (int gg = 0; gg < G; ++gg) {
          const int tl = tg + gg, t = h * kSB + tl;
          float f[kC], w[kC], y[kC], Bv[K], Cv[K], cx[kC], dc[K];
          lds_row<kC>(s_f + tl * kDT + chan0, f);
          lds_row<kC>(s_w + tl * kDT + chan0, w);
          lds_row<kC>(s_dy + tl * kDT + chan0, y);
          lds_row<K>(s_B + t * NS + q * K, Bv);
          lds_row<K>(s_C + t * NS + q * K, Cv);
#pragma unroll
          for (int k = 0; k < kC; ++k) {
            P[k] *= f[k];
            const float pdy = P[k] * y[k];
            cx[k] = 0.f;
#pragma unroll
            for (int n = 0; n < K; ++n) {
              x[k][n] = fmaf(f[k], x[k][n], w[k] * Bv[n]);
              cx[k] = fmaf(Cv[n], x[k][n], cx[k]);
              lam[k][n] = fmaf(pdy, Cv[n], lam[k][n]);
              dc[n] = k == 0 ? y[0] * x[0][n] : fmaf(y[k], x[k][n], dc[n]);
            }
            cx[k] *= y[k];
          }
          const float a = reduce_states<L>(cx, q);
          if (ch_writer) s_a[t * kDT + my_ch] = a;
          RG::run(dc, g);
          if (part_writer)
#pragma unroll
            for (int j = 0; j < RG::count; ++j) s_part[(warp * G + gg) * NS + part_n + j] = dc[j];
        }
        flush(p.dCpart, h * kSB + tg);
      }
    }
    {
      // dD partials: a thread holds the sums of four channels over its rows
      *reinterpret_cast<float4*>(s_part + warp * kDT + 4 * lane) = dd;
      __syncthreads();
      for (int e = tid; e < kDT; e += NT) {
        float s = 0.f;
#pragma unroll
        for (int wq = 0; wq < W; ++wq) s += s_part[wq * kDT + e];
        p.dDpart[(static_cast<int64_t>(c) * p.B + b) * (p.ndt * kDT) + d0 + e] = s;
      }
    }

    // ---------------- adjoint carry-in by decoupled look-back towards later chunks
    float carry[kC][K];
    if (c == p.nchunks - 1) {
      get_user_state<K>(p.dhT, bd0, d, p.D, p.N, q, carry);
    } else {
      if (c > 0) {   // (nobody looks back to chunk 0)
        put_state<NS, K>(p.aggL, slot0, q, lam);
        if (q == 0) *reinterpret_cast<float4*>(p.aggP + slot0) = make_float4(P[0], P[1], P[2], P[3]);
        __syncthreads();
        if (tid == 0) {
          __threadfence();
          st_release(p.flags + tile, 1);
        }
      }
      float accP[kC];
      const int64_t src = look_back<NS, K, NH == 2 ? 4 : 1>(p.flags, p.aggP, p.aggL, p.inclL, tile + per_chunk, per_chunk, p.nchunks - 1 - c, chan0,
                                           q, lane, carry, accP);
      if (src < 0) atomicOr(&p.hdr->status, NAJU_ST_LOOKBACK_TIMEOUT);
    }
    // inclusive adjoint leaving this chunk towards earlier time: lam + P * carry_in
    {
#pragma unroll
      for (int k = 0; k < kC; ++k)
#pragma unroll
        for (int n = 0; n < K; ++n) lam[k][n] = fmaf(P[k], carry[k][n], lam[k][n]);
      if (c > 0) {
        put_state<NS, K>(p.inclL, slot0, q, lam);
        __syncthreads();
        if (tid == 0) {
          __threadfence();
          st_release(p.flags + tile, 2);
        }
      } else {
        __syncthreads();
        if (p.dh0 != nullptr) put_user_state<K>(p.dh0, bd0, d, p.D, p.N, q, lam);
      }
    }

    // ---------------- reverse walk
    float r;   // of channel my_ch
    {
      float v[kC];
#pragma unroll
      for (int k = 0; k < kC; ++k) {
        v[k] = 0.f;
#pragma unroll
        for (int n = 0; n < K; ++n) v[k] = fmaf(carry[k][n], x[k][n], v[k]);
      }
      r = reduce_states<L>(v, q);
    }
#pragma unroll 1
    for (int h = NH - 1; h >= 0; --h) {
      if (h < NH - 1) {
        float4 again = make_float4(0.f, 0.f, 0.f, 0.f);
        stage(h, again);
        __syncthreads();
      }
#pragma unroll 1
      for (int tg = kSB - G; tg >= 0; tg -= G) {
#pragma unroll 2
        for (int gg = G - 1; gg >= 0; --gg) {
          const int tl = tg + gg, t = h * kSB + tl;
          float f[kC], w[kC], y[kC], Bv[K], Cv[K], gs[kC], db[K];
          lds_row<kC>(s_f + tl * kDT + chan0, f);
          lds_row<kC>(s_w + tl * kDT + chan0, w);
          lds_row<kC>(s_dy + tl * kDT + chan0, y);
          lds_row<K>(s_B + t * NS + q * K, Bv);
          lds_row<K>(s_C + t * NS + q * K, Cv);
          const float a = s_a[t * kDT + my_ch], wm = s_w[tl * kDT + my_ch];
          // Deep retention gate: r_t = f_t <xbar_t, x_{t-1}> is then far smaller than the two
          // terms whose difference the recurrence forms, so it is computed directly instead,
          // from x_{t-1} re-walked from the start of the piece (rare; cost O(t) for this warp).
          float r_exact = 0.f;
          bool deep_m = false;
          if (__any_sync(0xffffffffu, fminf(fminf(f[0], f[1]), fminf(f[2], f[3])) < kDeepGate)) {
            float xp[kC][K], v[kC];
            if (h == 0) chunk_start_state(xp);
            else if constexpr (NH == 2)
#pragma unroll
              for (int k = 0; k < kC; ++k)
#pragma unroll
                for (int n = 0; n < K; ++n) xp[k][n] = xh[k][n];
#pragma unroll 1
            for (int tt = 0; tt < tl; ++tt) {
              float f2[kC], w2[kC], B2[K];
              lds_row<kC>(s_f + tt * kDT + chan0, f2);
              lds_row<kC>(s_w + tt * kDT + chan0, w2);
              lds_row<K>(s_B + (h * kSB + tt) * NS + q * K, B2);
#pragma unroll
              for (int k = 0; k < kC; ++k)
#pragma unroll
                for (int n = 0; n < K; ++n) xp[k][n] = fmaf(f2[k], xp[k][n], w2[k] * B2[n]);
            }
#pragma unroll
            for (int k = 0; k < kC; ++k) {
              v[k] = 0.f;
#pragma unroll
              for (int n = 0; n < K; ++n) v[k] = fmaf(fmaf(Cv[n], y[k], carry[k][n]), xp[k][n], v[k]);
            }
            const float dot = reduce_states<L>(v, q);
            const float fm = s_f[tl * kDT + my_ch];
            r_exact = fm * dot;
            deep_m = fm < kDeepGate;
          }
#pragma unroll
          for (int k = 0; k < kC; ++k) {
            gs[k] = 0.f;
#pragma unroll
            for (int n = 0; n < K; ++n) {
              const float dx = fmaf(Cv[n], y[k], carry[k][n]);
              gs[k] = fmaf(dx, Bv[n], gs[k]);
              db[n] = k == 0 ? dx * w[0] : fmaf(dx, w[k], db[n]);
              carry[k][n] = f[k] * dx;
            }
          }
          const float gm = reduce_states<L>(gs, q);
          r += a - wm * gm;
          if (deep_m) r = r_exact;
          __syncwarp();   // the group's lanes have read dy and a of this step
          if (ch_writer) {
            s_dy[tl * kDT + my_ch] = gm;
            s_a[t * kDT + my_ch] = r;
          }
          RG::run(db, g);
          if (part_writer)
#pragma unroll
            for (int j = 0; j < RG::count; ++j) s_part[(warp * G + gg) * NS + part_n + j] = db[j];
        }
        flush(p.dBpart, h * kSB + tg);
      }
      // ---------------- the elementwise gradients of this piece, four channels of one step per thread
      const int v = 4 * lane, n = p.D - d0 - v, th = t0 + h * kSB, lenh = len - h * kSB;
      const int64_t row0 = (static_cast<int64_t>(b) * p.T + th) * p.D + d0 + v;
      const TG* fl = reinterpret_cast<const TG*>(p.fl) + b * p.fl_sb + static_cast<int64_t>(th) * p.fl_st + d0 + v;
      const TG* il = reinterpret_cast<const TG*>(p.il) + b * p.il_sb + static_cast<int64_t>(th) * p.il_st + d0 + v;
      const TA* dy = reinterpret_cast<const TA*>(p.dy) + row0;
      TG* dfl = reinterpret_cast<TG*>(p.dfl) + row0;
      TG* dil = reinterpret_cast<TG*>(p.dil) + row0;
      TA* du = reinterpret_cast<TA*>(p.du) + row0;
      const bool vf = vec4_ok(fl, p.fl_st), vi = vec4_ok(il, p.il_st), vy = vec4_ok(dy, p.D), vof = vec4_ok(dfl, p.D),
                 voi = vec4_ok(dil, p.D), vou = vec4_ok(du, p.D);
      const float4 Dv = load4(p.Dskip + d0 + v, n, vec4_ok(p.Dskip + d0 + v, 4));
      const bool skip = Dv.x != 0.f || Dv.y != 0.f || Dv.z != 0.f || Dv.w != 0.f;
#pragma unroll 2
      for (int tl = warp; tl < min(kSB, lenh); tl += W) {
        const float4 fv = load4(fl + static_cast<int64_t>(tl) * p.fl_st, n, vf);
        const float4 iv = load4(il + static_cast<int64_t>(tl) * p.il_st, n, vi);
        const float4 gg = *reinterpret_cast<const float4*>(s_dy + tl * kDT + v);
        const float4 rr = *reinterpret_cast<const float4*>(s_a + (h * kSB + tl) * kDT + v);
        const float4 ww = *reinterpret_cast<const float4*>(s_w + tl * kDT + v);
        const Gate i0 = gate(iv.x), i1 = gate(iv.y), i2 = gate(iv.z), i3 = gate(iv.w);
        float4 o = make_float4(i0.s * gg.x, i1.s * gg.y, i2.s * gg.z, i3.s * gg.w);
        if (skip) {
          const float4 y = load4(dy + static_cast<int64_t>(tl) * p.D, n, vy);
          o = make_float4(fmaf(Dv.x, y.x, o.x), fmaf(Dv.y, y.y, o.y), fmaf(Dv.z, y.z, o.z), fmaf(Dv.w, y.w, o.w));
        }
        if (p.u_sd > 1) *reinterpret_cast<float4*>(s_f + tl * kDT + v) = o;
        else store4(du + static_cast<int64_t>(tl) * p.D, o, n, vou);
        store4(dfl + static_cast<int64_t>(tl) * p.D,
               make_float4(gate(fv.x).one_minus * rr.x, gate(fv.y).one_minus * rr.y, gate(fv.z).one_minus * rr.z,
                           gate(fv.w).one_minus * rr.w), n, vof);
        store4(dil + static_cast<int64_t>(tl) * p.D,
               make_float4(gg.x * ww.x * i0.one_minus, gg.y * ww.y * i1.one_minus, gg.z * ww.z * i2.one_minus,
                           gg.w * ww.w * i3.one_minus), n, voi);
      }
      if (p.u_sd > 1) {   // du in the layout of a time-contiguous u
        __syncthreads();
        store_tmajor<TA, NT>(reinterpret_cast<TA*>(p.du) + b * p.u_sb + th + static_cast<int64_t>(d0) * p.u_sd, s_f, p.u_sd,
                             min(kSB, lenh), cols, tid);
      }
      if (h > 0) __syncthreads();   // the next piece is staged over this one
    }
  }
}

// ------------------------------------------------------------------------------ finalize
// dB[row][n] = sum_k part[row][k][n] for n < N (and dC), written in the caller's dtype; dD[d] = the sum over its
// partial rows.  One launch: blocks [0, ndd) take 32 channels of dD each (the longest chains first), then nbc take dB and nbc dC, in a
// fixed order throughout.  If a bounded wait of this call or of its forward ran out (or `inject` asks for it),
// every output is overwritten with all-ones bytes (NaN) instead.
struct PoisonList {
  void* ptr[4];
  unsigned long long bytes[4];
};

__global__ void __launch_bounds__(256) finalize_kernel(const BwdParams p, void* __restrict__ dB, void* __restrict__ dC,
                                                       float* __restrict__ dD, int NS, int nbc, int ndd, int dd_rows, int dd_rows_tc,
                                                       int inject, const PoisonList list) {
  __shared__ float red[8][33];
  pdl_wait();
  const int blk = static_cast<int>(blockIdx.x) - ndd;
  float sum = 0.f;
  const int64_t i = static_cast<int64_t>(blk < nbc ? blk : blk - nbc) * 256 + threadIdx.x;
  const bool mine = blk >= 0 && i < static_cast<int64_t>(p.B) * p.T * p.N;
  if (mine) {   // (before the status is looked at: the loads need not wait for it)
    const int64_t row = i < (1ll << 32) ? static_cast<uint32_t>(i) / static_cast<uint32_t>(p.N) : i / p.N;
    const float* src = (blk < nbc ? p.dBpart : p.dCpart) + row * p.ndt * NS + (i - row * p.N);
#pragma unroll 8
    for (int k = 0; k < p.ndt; ++k) sum += __ldcg(src + static_cast<int64_t>(k) * NS);   // (not the read-only path: the writer may overlap this kernel's start)
  }
  if (inject && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&p.hdr->status, NAJU_ST_LOOKBACK_TIMEOUT);
  const bool bad = inject || *reinterpret_cast<volatile int*>(&p.hdr->status) != 0 || (*p.fwd_form & 4) != 0;
  const float nan = __int_as_float(-1);
  if (bad) {
    for (int k = 0; k < 4; ++k)
      for (unsigned long long e = static_cast<unsigned long long>(blockIdx.x) * 256 + threadIdx.x; e < list.bytes[k];
           e += static_cast<unsigned long long>(gridDim.x) * 256)
        static_cast<unsigned char*>(list.ptr[k])[e] = 0xFF;
  }
  if (blk >= 0) {
    if (mine) store_dyn(blk < nbc ? dB : dC, p.bc_dtype, i, bad ? nan : sum);
    return;
  }
  // the tensor-core backward writes four partial rows per rank and batch row, the recurrent one per chunk
  const int rows = tc_did_it(p) ? dd_rows_tc : dd_rows;
  const int dl = threadIdx.x & 31, rl = threadIdx.x >> 5, d = static_cast<int>(blockIdx.x) * 32 + dl, ld = p.ndt * kDT;
  float s = 0.f;
  if (d < p.D)
#pragma unroll 4
    for (int r = rl; r < rows; r += 8) s += p.dDpart[static_cast<int64_t>(r) * ld + d];
  red[rl][dl] = s;
  __syncthreads();
  if (rl == 0 && d < p.D) {
    float tot = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) tot += red[k][dl];
    dD[d] = bad ? nan : tot;
  }
}

int launch_bwd_finalize(const BwdParams& p, const Geometry& g, int act, int gate, void* dB, void* dC, float* dD, bool inject,
                        void* stream) {
  const int64_t ntd = static_cast<int64_t>(g.B) * g.T * g.D, nbc = (static_cast<int64_t>(g.B) * g.T * g.N + 255) / 256;
  const int ndd = (g.D + 31) / 32;
  const int64_t blocks = 2 * nbc + ndd;
  if (blocks > 0x7fffffff) return NAJU_E_SHAPE;
  PoisonList list = {{p.du, p.dfl, p.dil, p.dh0},
                     {static_cast<unsigned long long>(ntd) * dtype_size(act), static_cast<unsigned long long>(ntd) * dtype_size(gate),
                      static_cast<unsigned long long>(ntd) * dtype_size(gate),
                      p.dh0 ? static_cast<unsigned long long>(g.B) * g.D * g.N * 4 : 0ull}};
  return launch_pdl(finalize_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, static_cast<cudaStream_t>(stream), p, dB,
                    dC, dD, g.NS, static_cast<int>(nbc), ndd, g.nchunks * g.B, 4 * p.tc_launched * g.B, inject ? 1 : 0, list);
}

template <typename TA, typename TG, int NS, int NH>
static int launch_nh(const BwdParams& p, const Geometry& g, cudaStream_t st) {
  using S = BwdShape<NS>;
  constexpr size_t smem = 4 * (static_cast<size_t>(kSB) * kDT * (3 + NH) + 2 * static_cast<size_t>(NH) * kSB * NS +
                               std::max(S::part_floats, S::W * kDT));
  auto kern = bwd_simt_kernel<TA, TG, NS, NH>;
  static std::atomic<unsigned long long> allowed{0};
  const int rc = allow_smem(kern, smem, allowed);
  if (rc != 0) return rc;
  // persistent grid: what fits on the GPU at once (the look-back needs every waiting CTA's
  // predecessors to be resident or done, which ticket order guarantees for any grid size)
  static std::atomic<int> per_sm_cache{0};
  int per_sm = per_sm_cache.load(std::memory_order_relaxed);
  if (per_sm == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, S::NT, smem) != cudaSuccess || per_sm < 1) per_sm = 1;
    per_sm_cache.store(per_sm, std::memory_order_relaxed);
  }
  const int64_t grid = std::min<int64_t>(g.ntiles, static_cast<int64_t>(tmah::sm_count()) * per_sm);
  return launch_pdl(kern, dim3(static_cast<unsigned>(grid)), dim3(S::NT), smem, st, p);
}

template <typename TA, typename TG>
static int launch_types(const BwdParams& p, const Geometry& g, cudaStream_t st) {
  if (g.NS == 16) {
    if constexpr (sizeof(TA) == 2)
      if (g.TC == 64) return launch_nh<TA, TG, 16, 2>(p, g, st);
    return launch_nh<TA, TG, 16, 1>(p, g, st);
  }
  if (g.NS == 32) return launch_nh<TA, TG, 32, 1>(p, g, st);
  if (g.NS == 64) return launch_nh<TA, TG, 64, 1>(p, g, st);
  return launch_nh<TA, TG, 128, 1>(p, g, st);
}

int launch_bwd_simt(const BwdParams& p, const Geometry& g, int act, int gate, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (act == NAJU_F32 && gate == NAJU_F32) return launch_types<float, float>(p, g, st);
  if (act == NAJU_BF16 && gate == NAJU_BF16) return launch_types<__nv_bfloat16, __nv_bfloat16>(p, g, st);
  if (act == NAJU_BF16 && gate == NAJU_F32) return launch_types<__nv_bfloat16, float>(p, g, st);
  if (act == NAJU_F16 && gate == NAJU_F16) return launch_types<__half, __half>(p, g, st);
  if (act == NAJU_F16 && gate == NAJU_F32) return launch_types<__half, float>(p, g, st);
  return NAJU_E_DTYPE;
}

}  // namespace naju
