// Single-token recurrent state update for decode: one iteration of the scan recurrence
// (naju/scan.py:87-91 of the reference project, which has no decode entry point).
//
//   state[b,d,n] <- f state[b,d,n] + (i u) B[b,n];   y[b,d] = sum_n C[b,n] state[b,d,n] + D_skip u
//
// HBM streaming of the fp32 state (read once, written once): 8 N bytes per channel against 8 to 16 of
// everything else.  A thread owns four consecutive states of kIter channels, so all of its state loads
// (16 bytes each) are in flight at once and the row's B and C are read once for all of them, as one
// vector each; the N/4 lanes that share a channel are adjacent, so a warp touches contiguous
// 512-byte spans and the readout is a short shuffle reduction.  Decode calls follow one another layer by
// layer, each too short to hide a launch: the kernel lets its successor's blocks launch early and waits
// for its predecessor itself (programmatic dependent launch).
#include "common.cuh"
#include "params.h"

namespace naju {

constexpr int kStepBlock = 128;

// four consecutive elements of a row of B or C as floats (`vec`: one 8- or 16-byte load)
template <typename TB>
__device__ __forceinline__ void load_row4(const TB* __restrict__ p, int n0, int N, bool vec, float (&v)[4]) {
  if (vec) {
    if constexpr (sizeof(TB) == 4) {
      const float4 t = __ldg(reinterpret_cast<const float4*>(p + n0));
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
      const uint2 t = __ldg(reinterpret_cast<const uint2*>(p + n0));
      TB e[4];
      *reinterpret_cast<uint2*>(e) = t;
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = to_f32(e[k]);
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = n0 + k < N ? to_f32(p[n0 + k]) : 0.f;
  }
}

// Block = kStepBlock threads of one batch row (blockIdx.y); lpc lanes per channel (a power of two, at
// least N/4); kIter channels per thread, kStepBlock / lpc apart.  kWhole: a channel's states come in
// 16-byte pieces (N % 4 == 0).  kN: N at compile time, or 0.  Lanes beyond the last channel or state read in-bounds duplicates and
// write nothing, so that no load of the batch sits behind a branch (with branches around them the
// loads were issued one iteration at a time: 18.9 us against 13 us at 256 sequences x 2048 channels).
template <typename TA, typename TG, typename TB, int kIter, bool kWhole, int kN>
__global__ void __launch_bounds__(kStepBlock) step_kernel(float* __restrict__ state, const TA* __restrict__ u,
                                                   const TG* __restrict__ fl, const TG* __restrict__ il,
                                                   const TB* __restrict__ Bm, const TB* __restrict__ Cm,
                                                   const float* __restrict__ Dskip, TA* __restrict__ y, int D, int N_,
                                                   int lpc_log2_, bool vec, int64_t u_sb, int64_t fl_sb, int64_t il_sb,
                                                   int64_t bm_sb, int64_t cm_sb) {
  pdl_launch_dependents();
  const int N = kN > 0 ? kN : N_;
  const int lpc_log2 = kN == 0 ? lpc_log2_ : kN <= 4 ? 0 : kN <= 8 ? 1 : kN <= 16 ? 2 : kN <= 32 ? 3 : kN <= 64 ? 4 : 5;
  const int b = blockIdx.y, q = threadIdx.x & ((1 << lpc_log2) - 1);
  const int per_pass = kStepBlock >> lpc_log2;
  const int d0 = blockIdx.x * per_pass * kIter + (static_cast<int>(threadIdx.x) >> lpc_log2);
  const bool mine = 4 * q < N;
  const int n0 = mine ? 4 * q : 0;
  float* srow = state + static_cast<int64_t>(b) * D * N + n0;
  u += b * u_sb;
  fl += b * fl_sb;
  il += b * il_sb;
  pdl_wait();
  float4 s[kIter];
  float ut[kIter], xf[kIter], xi[kIter], bv[4], cv[4];
#pragma unroll
  for (int k = 0; k < kIter; ++k) {
    const int d = min(d0 + k * per_pass, D - 1);
    const float* sp = srow + static_cast<int64_t>(d) * N;
    if constexpr (kWhole) {
      s[k] = *reinterpret_cast<const float4*>(sp);
    } else {
      s[k].x = sp[0];
      s[k].y = sp[min(1, N - 1 - n0)];
      s[k].z = sp[min(2, N - 1 - n0)];
      s[k].w = sp[min(3, N - 1 - n0)];
    }
    ut[k] = to_f32(u[d]);
    xf[k] = to_f32(fl[d]);
    xi[k] = to_f32(il[d]);
  }
  load_row4(Bm + b * bm_sb, n0, N, vec, bv);
  load_row4(Cm + b * cm_sb, n0, N, vec, cv);
#pragma unroll
  for (int k = 0; k < kIter; ++k) {
    const int d = d0 + k * per_pass;
    const float f = sigmoid_f(xf[k]);
    const float w = sigmoid_f(xi[k]) * ut[k];
    s[k].x = fmaf(f, s[k].x, w * bv[0]);
    s[k].y = fmaf(f, s[k].y, w * bv[1]);
    s[k].z = fmaf(f, s[k].z, w * bv[2]);
    s[k].w = fmaf(f, s[k].w, w * bv[3]);
    float part = s[k].x * cv[0];
    part = fmaf(s[k].y, cv[1], part);
    part = fmaf(s[k].z, cv[2], part);
    part = fmaf(s[k].w, cv[3], part);
    if (!mine) part = 0.f;
    if (d < D && mine) {
      float* sp = srow + static_cast<int64_t>(d) * N;
      if constexpr (kWhole) {
        *reinterpret_cast<float4*>(sp) = s[k];
      } else {
        sp[0] = s[k].x;
        if (n0 + 1 < N) sp[1] = s[k].y;
        if (n0 + 2 < N) sp[2] = s[k].z;
        if (n0 + 3 < N) sp[3] = s[k].w;
      }
    }
    // lanes sharing a channel are adjacent and their number divides 32
#pragma unroll
    for (int m = (1 << lpc_log2) >> 1; m >= 1; m >>= 1) part += __shfl_xor_sync(0xffffffffu, part, m);
    if (d < D && q == 0) y[static_cast<int64_t>(b) * D + d] = from_f32<TA>(fmaf(Dskip[d], ut[k], part));
  }
}

template <typename TA, typename TG, typename TB, int kIter, bool kWhole, int kN>
static int launch_iter(const naju_scan_desc& d, float* state, const void* u, const void* fl, const void* il, const void* Bm,
                       const void* Cm, const float* Dskip, void* y, int lpc_log2, cudaStream_t st) {
  const int span = (kStepBlock >> lpc_log2) * kIter;
  auto aligned4 = [](const void* p, int64_t sb) {
    return reinterpret_cast<uintptr_t>(p) % (4 * sizeof(TB)) == 0 && sb % 4 == 0;
  };
  const bool vec = d.N % 4 == 0 && aligned4(Bm, d.bm_sb) && aligned4(Cm, d.cm_sb);
  for (int b0 = 0; b0 < d.B; b0 += 65535) {   // (grid.y limit)
    const int nb = d.B - b0 < 65535 ? d.B - b0 : 65535;
    const dim3 grid(static_cast<unsigned>((d.D + span - 1) / span), static_cast<unsigned>(nb));
    const int rc = launch_pdl(step_kernel<TA, TG, TB, kIter, kWhole, kN>, grid, dim3(kStepBlock), 0, st,
                              state + static_cast<int64_t>(b0) * d.D * d.N, static_cast<const TA*>(u) + b0 * d.u_sb,
                              static_cast<const TG*>(fl) + b0 * d.fl_sb, static_cast<const TG*>(il) + b0 * d.il_sb,
                              static_cast<const TB*>(Bm) + b0 * d.bm_sb, static_cast<const TB*>(Cm) + b0 * d.cm_sb, Dskip,
                              static_cast<TA*>(y) + static_cast<int64_t>(b0) * d.D, d.D, d.N, lpc_log2, vec, d.u_sb, d.fl_sb,
                              d.il_sb, d.bm_sb, d.cm_sb);
    if (rc != 0) return rc;
  }
  return 0;
}

template <typename TA, typename TG, typename TB>
static int launch_t(const naju_scan_desc& d, float* state, const void* u, const void* fl, const void* il, const void* Bm,
                    const void* Cm, const float* Dskip, void* y, cudaStream_t st) {
  int lpc_log2 = 0;
  while ((4 << lpc_log2) < d.N) ++lpc_log2;  // 1..32 lanes
  // Two channels per thread once the grid stays at several blocks per SM with them: below that the call is
  // bound by latency and more blocks are all there is.  (256 sequences x 2048 channels x 16 states: one
  // channel per thread 14.9 us, two 13.2, four 13.7, eight 14.7; reading and writing the state in place
  // and nothing else takes 14.4.)
  const int64_t blocks1 = static_cast<int64_t>(d.B) * ((static_cast<int64_t>(d.D) << lpc_log2) / kStepBlock);
  // The usual widths have N, and with it every address and the readout's shuffles, at compile time
  // (16.7 us with run-time ones at that size).
  if (d.N % 4 != 0) return launch_iter<TA, TG, TB, 1, false, 0>(d, state, u, fl, il, Bm, Cm, Dskip, y, lpc_log2, st);
  if (blocks1 <= 148 * 16) return launch_iter<TA, TG, TB, 1, true, 0>(d, state, u, fl, il, Bm, Cm, Dskip, y, lpc_log2, st);
  switch (d.N) {
    case 8: return launch_iter<TA, TG, TB, 2, true, 8>(d, state, u, fl, il, Bm, Cm, Dskip, y, lpc_log2, st);
    case 16: return launch_iter<TA, TG, TB, 2, true, 16>(d, state, u, fl, il, Bm, Cm, Dskip, y, lpc_log2, st);
    case 32: return launch_iter<TA, TG, TB, 2, true, 32>(d, state, u, fl, il, Bm, Cm, Dskip, y, lpc_log2, st);
    case 64: return launch_iter<TA, TG, TB, 2, true, 64>(d, state, u, fl, il, Bm, Cm, Dskip, y, lpc_log2, st);
    case 128: return launch_iter<TA, TG, TB, 2, true, 128>(d, state, u, fl, il, Bm, Cm, Dskip, y, lpc_log2, st);
    default: return launch_iter<TA, TG, TB, 2, true, 0>(d, state, u, fl, il, Bm, Cm, Dskip, y, lpc_log2, st);
  }
}

template <typename TA, typename TG>
static int launch_bc(const naju_scan_desc& d, float* state, const void* u, const void* fl, const void* il, const void* Bm,
                     const void* Cm, const float* Dskip, void* y, cudaStream_t st) {
  if (d.bc_dtype == NAJU_F32) return launch_t<TA, TG, float>(d, state, u, fl, il, Bm, Cm, Dskip, y, st);
  if (d.bc_dtype == NAJU_BF16) return launch_t<TA, TG, __nv_bfloat16>(d, state, u, fl, il, Bm, Cm, Dskip, y, st);
  return launch_t<TA, TG, __half>(d, state, u, fl, il, Bm, Cm, Dskip, y, st);
}

int launch_step(const naju_scan_desc& d, float* state, const void* u, const void* fl, const void* il,
                const void* Bm, const void* Cm, const float* Dskip, void* y, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int a = d.act_dtype, g = d.gate_dtype;
  if (a == NAJU_F32 && g == NAJU_F32) return launch_bc<float, float>(d, state, u, fl, il, Bm, Cm, Dskip, y, st);
  if (a == NAJU_BF16 && g == NAJU_BF16) return launch_bc<__nv_bfloat16, __nv_bfloat16>(d, state, u, fl, il, Bm, Cm, Dskip, y, st);
  if (a == NAJU_BF16 && g == NAJU_F32) return launch_bc<__nv_bfloat16, float>(d, state, u, fl, il, Bm, Cm, Dskip, y, st);
  if (a == NAJU_F16 && g == NAJU_F16) return launch_bc<__half, __half>(d, state, u, fl, il, Bm, Cm, Dskip, y, st);
  if (a == NAJU_F16 && g == NAJU_F32) return launch_bc<__half, float>(d, state, u, fl, il, Bm, Cm, Dskip, y, st);
  return NAJU_E_DTYPE;
}

}  // namespace naju
