// Forward gated scan, exact recurrent form (any gate logit).
//
//   x_t[n] = f_t x_{t-1}[n] + (i_t u_t) B_t[n],   y_t = sum_n C_t[n] x_t[n] + D_skip u_t
//   (naju/scan.py:79-93 of the reference project)
//
// One CTA owns a tile of TC time steps x 128 channels of one batch row; a thread owns four channels x K
// states (simt_common.cuh).  The gates of the tile are staged in shared memory and walked twice:
//   pass 1  local scan from a zero state -> (P, S) = (product of f, chunk-end state)
//   carry   decoupled look-back over the preceding chunks of the same channel tile:
//           each chunk publishes its aggregate (P, S) and, once its own carry-in is known,
//           its inclusive state; a chunk folds aggregates backwards until it meets an
//           inclusive state.  Tiles are handed out by an atomic ticket in time-major order,
//           so every predecessor is already running; every wait is bounded.
//   pass 2  scan again from the true carry-in, emitting y.
// The first chunk knows its carry-in and skips pass 1.  The inclusive chunk-end states double as the
// checkpoints the backward restarts from.
#include "fwd_common.cuh"
#include "simt_common.cuh"

namespace naju {

using namespace simt;

template <typename TA, typename TG, int NS, int TC>
__global__ void __launch_bounds__(Shape<NS>::NT, NS == 128 ? 1 : NS == 64 ? 2 : 4) fwd_simt_kernel(const FwdParams p) {
  using S = Shape<NS>;
  constexpr int K = S::K, L = S::L, NT = S::NT;
  extern __shared__ __align__(16) float sm[];
  float* s_f = sm;                    // [TC][128]
  float* s_w = s_f + TC * kDT;        // [TC][128]; y replaces w behind pass 2
  float* s_B = s_w + TC * kDT;        // [TC][NS]
  float* s_C = s_B + TC * NS;         // [TC][NS]
  __shared__ unsigned int s_ticket;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  if (tid == 0) {
    s_ticket = atomicAdd(&p.hdr->ticket, 1u);
    if (blockIdx.x == 0) p.hdr->form = NAJU_FORM_RECURRENT;
  }
  __syncthreads();
  const int per_chunk = p.B * p.ndt;
  const int64_t tile = s_ticket;
  const int c = static_cast<int>(tile / per_chunk), rem = static_cast<int>(tile - static_cast<int64_t>(c) * per_chunk);
  const int b = rem / p.ndt, d0 = (rem - b * p.ndt) * kDT, t0 = c * TC, len = min(TC, p.T - t0), cols = min(kDT, p.D - d0);

  // ---- stage the tile
  StageBC<NS, NT, TC> bc;
  bc.load(p, b, t0, len, tid);
  if (p.u_sd > 1) {
#pragma unroll
    for (int h = 0; h < TC / kSB; ++h)
      load_tmajor<TA, NT>(s_w + h * kSB * kDT,
                          reinterpret_cast<const TA*>(p.u) + b * p.u_sb + t0 + h * kSB + static_cast<int64_t>(d0) * p.u_sd,
                          p.u_sd, len - h * kSB, cols, tid);
    __syncthreads();
  }
  float4 dd = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int h = 0; h < TC / kSB; ++h)
    stage_gates<TA, TG, NT, false>(p, s_f + h * kSB * kDT, s_w + h * kSB * kDT, nullptr, b, t0 + h * kSB, len - h * kSB, d0, tid, dd);
  bc.store(p, s_B, s_C, b, t0, len, tid);
  __syncthreads();

  const int q = lane % L, g = lane / L, chan0 = (warp * S::GW + g) * kC, d = d0 + chan0;
  const int64_t slot0 = tile * kDT + chan0, bd0 = static_cast<int64_t>(b) * p.D + d;
  const float* my_f = s_f + chan0;
  const float* my_w = s_w + chan0;
  const float* my_B = s_B + q * K;
  const float* my_C = s_C + q * K;

  float x[kC][K], P[kC], Pin[kC];
#pragma unroll
  for (int k = 0; k < kC; ++k) Pin[k] = P[k] = 1.f;
  if (c == 0) {
    get_user_state<K>(p.h0, bd0, d, p.D, p.N, q, x);
  } else {
    // ---- pass 1
#pragma unroll
    for (int k = 0; k < kC; ++k)
#pragma unroll
      for (int n = 0; n < K; ++n) x[k][n] = 0.f;
#pragma unroll 4
    for (int t = 0; t < TC; ++t) {
      float f[kC], w[kC], Bv[K];
      lds_row<kC>(my_f + t * kDT, f);
      lds_row<kC>(my_w + t * kDT, w);
      lds_row<K>(my_B + t * NS, Bv);
#pragma unroll
      for (int k = 0; k < kC; ++k) {
        P[k] *= f[k];
#pragma unroll
        for (int n = 0; n < K; ++n) x[k][n] = fmaf(f[k], x[k][n], w[k] * Bv[n]);
      }
    }
    // ---- carry: publish the aggregate, fold the predecessors', publish the inclusive state
    put_state<NS, K>(p.aggS, slot0, q, x);
    if (q == 0) *reinterpret_cast<float4*>(p.aggP + slot0) = make_float4(P[0], P[1], P[2], P[3]);
    __syncthreads();
    if (tid == 0) {
      __threadfence();  // cumulative: orders every thread's stores above (seen through the barrier)
      st_release(p.flags + tile, 1);
    }
    float h[kC][K];
    const int64_t src = look_back<NS, K, 1>(p.flags, p.aggP, p.aggS, p.ckS, tile - per_chunk, -per_chunk, c, chan0, q, lane, h, Pin);
    if (src < 0) {
      atomicOr(&p.hdr->status, NAJU_ST_LOOKBACK_TIMEOUT);
    } else {
      const float4 pi = __ldcg(reinterpret_cast<const float4*>(p.ckP + src * kDT + chan0));
      Pin[0] *= pi.x; Pin[1] *= pi.y; Pin[2] *= pi.z; Pin[3] *= pi.w;
    }
    float e[kC][K];
#pragma unroll
    for (int k = 0; k < kC; ++k)
#pragma unroll
      for (int n = 0; n < K; ++n) {
        e[k][n] = fmaf(P[k], h[k][n], x[k][n]);
        x[k][n] = h[k][n];
      }
    put_state<NS, K>(p.ckS, slot0, q, e);
    if (q == 0)
      *reinterpret_cast<float4*>(p.ckP + slot0) = make_float4(P[0] * Pin[0], P[1] * Pin[1], P[2] * Pin[2], P[3] * Pin[3]);
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      st_release(p.flags + tile, 2);
    }
  }
  // ---- pass 2 (a y replaces the w of its step and channel: the group's lanes have read it by then)
  const int ych = chan0 + chan_of<L>(q);
  const bool ywriter = L == 4 || (q % (L / 4)) == 0;
#pragma unroll 4
  for (int t = 0; t < TC; ++t) {
    float f[kC], w[kC], Bv[K], Cv[K], acc[kC];
    lds_row<kC>(my_f + t * kDT, f);
    lds_row<kC>(my_w + t * kDT, w);
    lds_row<K>(my_B + t * NS, Bv);
    lds_row<K>(my_C + t * NS, Cv);
#pragma unroll
    for (int k = 0; k < kC; ++k) {
      if (c == 0) P[k] *= f[k];
      acc[k] = 0.f;
#pragma unroll
      for (int n = 0; n < K; ++n) {
        x[k][n] = fmaf(f[k], x[k][n], w[k] * Bv[n]);
        acc[k] = fmaf(Cv[n], x[k][n], acc[k]);
      }
    }
    const float y = reduce_states<L>(acc, q);
    if (ywriter) s_w[t * kDT + ych] = y;
  }
  if (c == 0) {
    put_state<NS, K>(p.ckS, slot0, q, x);
    if (q == 0) *reinterpret_cast<float4*>(p.ckP + slot0) = make_float4(P[0], P[1], P[2], P[3]);
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      st_release(p.flags + tile, 2);
    }
  } else {
    __syncthreads();
  }
  if (c == p.nchunks - 1) {
    if (p.hT != nullptr) put_user_state<K>(p.hT, bd0, d, p.D, p.N, q, x);
    if (p.pT != nullptr && q == 0)
#pragma unroll
      for (int k = 0; k < kC; ++k)
        if (d + k < p.D) p.pT[bd0 + k] = P[k] * Pin[k];
  }
  // ---- y out
  {
    const int v = 4 * lane, n = p.D - d0 - v;
    TA* y = reinterpret_cast<TA*>(p.y) + (static_cast<int64_t>(b) * p.T + t0) * p.D + d0 + v;
    const TA* u = reinterpret_cast<const TA*>(p.u) + b * p.u_sb + static_cast<int64_t>(t0) * p.u_st + (d0 + v) * p.u_sd;
    const bool vy = vec4_ok(y, p.D), vu = p.u_sd == 1 && vec4_ok(u, p.u_st);
    const float4 Dv = load4(p.Dskip + d0 + v, n, vec4_ok(p.Dskip + d0 + v, 4));
    const bool skip = Dv.x != 0.f || Dv.y != 0.f || Dv.z != 0.f || Dv.w != 0.f;
#pragma unroll 4
    for (int t = warp; t < len; t += S::W) {
      float4 o = *reinterpret_cast<const float4*>(s_w + t * kDT + v);
      if (skip) {
        const TA* ut = u + static_cast<int64_t>(t) * p.u_st;
        float4 uu;
        if (p.u_sd == 1) uu = load4(ut, n, vu);
        else uu = make_float4(n > 0 ? to_f32(ut[0]) : 0.f, n > 1 ? to_f32(ut[p.u_sd]) : 0.f,
                              n > 2 ? to_f32(ut[2 * p.u_sd]) : 0.f, n > 3 ? to_f32(ut[3 * p.u_sd]) : 0.f);
        o = make_float4(fmaf(Dv.x, uu.x, o.x), fmaf(Dv.y, uu.y, o.y), fmaf(Dv.z, uu.z, o.z), fmaf(Dv.w, uu.w, o.w));
      }
      store4(y + static_cast<int64_t>(t) * p.D, o, n, vy);
    }
  }
  finish_forward<TA>(p);
}

template <typename TA, typename TG, int NS, int TC>
static int launch_tc(const FwdParams& p, const Geometry& g, cudaStream_t st) {
  constexpr size_t smem = static_cast<size_t>(TC) * kDT * 8 + 2 * static_cast<size_t>(TC) * NS * 4;
  auto kern = fwd_simt_kernel<TA, TG, NS, TC>;
  static std::atomic<unsigned long long> allowed{0};
  int rc = allow_smem(kern, smem, allowed);
  if (rc == 0) rc = launch_init(p.hdr, static_cast<size_t>(256 + g.ntiles * 4), p.fwd_form, st);
  if (rc != 0) return rc;
  return launch_pdl(kern, dim3(static_cast<unsigned>(g.ntiles)), dim3(Shape<NS>::NT), smem, st, p);
}

template <typename TA, typename TG>
static int launch_types(const FwdParams& p, const Geometry& g, cudaStream_t st) {
  if (g.NS == 16) {
    // (64-step chunks belong to the types that the tensor-core kernels take, see params.h, and to problems too large for
    // naju_b200_fwd_noalloc()'s workspace with 32)
    return g.TC == 64 ? launch_tc<TA, TG, 16, 64>(p, g, st) : launch_tc<TA, TG, 16, 32>(p, g, st);
  }
  if (g.NS == 32) return g.TC == 64 ? launch_tc<TA, TG, 32, 64>(p, g, st) : launch_tc<TA, TG, 32, 32>(p, g, st);
  if (g.NS == 64) return launch_tc<TA, TG, 64, 32>(p, g, st);
  return launch_tc<TA, TG, 128, 32>(p, g, st);
}

int launch_fwd_simt(const FwdParams& p, const Geometry& g, int act, int gate, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (act == NAJU_F32 && gate == NAJU_F32) return launch_types<float, float>(p, g, st);
  if (act == NAJU_BF16 && gate == NAJU_BF16) return launch_types<__nv_bfloat16, __nv_bfloat16>(p, g, st);
  if (act == NAJU_BF16 && gate == NAJU_F32) return launch_types<__nv_bfloat16, float>(p, g, st);
  if (act == NAJU_F16 && gate == NAJU_F16) return launch_types<__half, __half>(p, g, st);
  if (act == NAJU_F16 && gate == NAJU_F32) return launch_types<__half, float>(p, g, st);
  return NAJU_E_DTYPE;
}

}  // namespace naju
