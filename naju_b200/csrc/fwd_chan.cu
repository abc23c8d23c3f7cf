// Forward gated scan, exact recurrent form, for 16 states and 16-bit inputs: the kernel of fwd_simt.cu (which see for the
// recurrence, naju/scan.py:79-93, and for how the carry crosses tiles) with one channel and all of its states per thread
// and the tile staged as it is, in 16 bits.
//
// A tile then takes 6 bytes of shared memory per step and channel, or 10 with fp32 logits, instead of fwd_simt.cu's 8 fp32
// bytes plus its fp32 rows, enough CTAs fit to hide the walk's latency, and with 16 states the broadcasts of B and C do not
// yet bound it: B=8, T=16384, D=2048, bf16 2.2 ms against 3.5 ms there.  With fp32 tiles, or more states, it is the other
// way round (B=2, T=4096, D=1001, fp32: 252 against 159 us), so those stay there.
#include "lookback_common.cuh"

namespace naju {

template <typename TA, typename TG, int NS, int TC>
__global__ void __launch_bounds__(kThreads) fwd_chan_kernel(const FwdParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TA* s_u = reinterpret_cast<TA*>(smem_raw);            // [TC][128]; reused for y
  TG* s_fl = reinterpret_cast<TG*>(s_u + TC * kDT);     // [TC][128]
  TG* s_il = s_fl + TC * kDT;                           // [TC][128]
  float* s_B = reinterpret_cast<float*>(s_il + TC * kDT);  // [TC][NS]
  float* s_C = s_B + TC * NS;                              // [TC][NS]
  __shared__ unsigned int s_ticket;

  const int tid = threadIdx.x;
  pdl_wait();
  if (tid == 0) {
    s_ticket = atomicAdd(&p.hdr->ticket, 1u);
    if (blockIdx.x == 0) p.hdr->form = NAJU_FORM_RECURRENT;
  }
  __syncthreads();
  TileCoord tc;
  decode_tile<TC>(s_ticket, p.B, p.T, p.D, p.nchunks, p.ndt, tid, tc);
  const int b = tc.b, t0 = tc.t0, len = tc.len, d0 = tc.d0, cols = tc.cols;

  // ---- stage the tile
  load_tile_async(s_u, reinterpret_cast<const TA*>(p.u) + b * p.u_sb + t0 * p.u_st + d0, p.u_st,
                  len, cols, tid);
  load_tile_async(s_fl, reinterpret_cast<const TG*>(p.fl) + b * p.fl_sb + t0 * p.fl_st + d0,
                  p.fl_st, len, cols, tid);
  load_tile_async(s_il, reinterpret_cast<const TG*>(p.il) + b * p.il_sb + t0 * p.il_st + d0,
                  p.il_st, len, cols, tid);
  cp_async_commit();
  load_bc_tile<NS>(s_B, p.Bm, p.bc_dtype, b * p.bm_sb + t0 * p.bm_st, p.bm_st, len, p.N, tid);
  load_bc_tile<NS>(s_C, p.Cm, p.bc_dtype, b * p.cm_sb + t0 * p.cm_st, p.cm_st, len, p.N, tid);
  cp_async_wait_all();
  __syncthreads();

  float x[NS], h[NS];
  float P, Pin;
  tile_pass1<TA, TG, NS>(s_u, s_fl, s_il, s_B, len, tid, x, P);
  carry_lookback<NS>(p, tc, tid, x, P, h, Pin);
  const float Dv = tc.d_ok ? p.Dskip[tc.d] : 0.f;
  tile_pass2<TA, TG, NS>(s_u, s_fl, s_il, s_B, s_C, len, tid, Dv, h);
  write_final<NS>(p, tc, h, P * Pin);
  __syncthreads();
  store_tile(reinterpret_cast<TA*>(p.y) + (static_cast<int64_t>(b) * p.T + t0) * p.D + d0, s_u,
             static_cast<int64_t>(p.D), len, cols, tid);
  finish_forward<TA>(p);
}

template <typename TA, typename TG, int TC>
static int launch_chan_tc(const FwdParams& p, const Geometry& g, cudaStream_t st) {
  constexpr int NS = 16;
  constexpr size_t smem = static_cast<size_t>(TC) * kDT * (sizeof(TA) + 2 * sizeof(TG)) + 2 * static_cast<size_t>(TC) * NS * 4;
  auto kern = fwd_chan_kernel<TA, TG, NS, TC>;
  static std::atomic<unsigned long long> allowed{0};
  int rc = allow_smem(kern, smem, allowed);
  if (rc == 0) rc = launch_init(p.hdr, static_cast<size_t>(256 + g.ntiles * 4), p.fwd_form, st);
  if (rc != 0) return rc;
  return launch_pdl(kern, dim3(static_cast<unsigned>(g.ntiles)), dim3(kThreads), smem, st, p);
}

template <typename TA, typename TG>
static int launch_chan_t(const FwdParams& p, const Geometry& g, cudaStream_t st) {
  return g.TC == 64 ? launch_chan_tc<TA, TG, 64>(p, g, st) : launch_chan_tc<TA, TG, 32>(p, g, st);
}

// -1000: not its problem (state width, 32-bit u, time-contiguous u).
int launch_fwd_chan(const FwdParams& p, const Geometry& g, int act, int gate, void* stream) {
  if (g.NS != 16 || p.u_sd > 1) return -1000;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (act == NAJU_BF16) return gate == NAJU_F32 ? launch_chan_t<__nv_bfloat16, float>(p, g, st) : launch_chan_t<__nv_bfloat16, __nv_bfloat16>(p, g, st);
  if (act == NAJU_F16) return gate == NAJU_F32 ? launch_chan_t<__half, float>(p, g, st) : launch_chan_t<__half, __half>(p, g, st);
  return -1000;
}

}  // namespace naju
