// Building blocks shared by the forward kernels.
#pragma once

#include "common.cuh"
#include "params.h"

namespace naju {

// Tile coordinates handed out by the time-major ticket.
struct TileCoord {
  int64_t tile;
  int c, rem, b, dt, per_chunk, t0, len, d0, cols, d;
  bool d_ok;
};

template <int TC>
__device__ __forceinline__ bool decode_tile(unsigned ticket, int B, int T, int D, int nchunks,
                                            int ndt, int tid, TileCoord& tc) {
  tc.tile = ticket;
  tc.per_chunk = B * ndt;
  tc.c = static_cast<int>(ticket / tc.per_chunk);
  tc.rem = static_cast<int>(ticket % tc.per_chunk);
  tc.b = tc.rem / ndt;
  tc.dt = tc.rem % ndt;
  tc.t0 = tc.c * TC;
  tc.len = min(TC, T - tc.t0);
  tc.d0 = tc.dt * kDT;
  tc.cols = min(kDT, D - tc.d0);
  tc.d = tc.d0 + tid;
  tc.d_ok = tc.d < D;
  return tc.c < nchunks;
}

// Carry across chunks.  In: (P, S) the tile's local aggregate.  Out: h = state entering the
// chunk, Pin = product of f from t=0 to the chunk start.  Publishes the aggregate, resolves
// the carry-in by bounded decoupled look-back and publishes the inclusive chunk-end state
// (the backward's checkpoint).  Must be called by all threads of the CTA.
// NAMED = false: all threads of the CTA take part (__syncthreads).  NAMED = true: only the first
// 128 threads do (named barrier 1), for kernels whose other warps have other roles.
template <bool NAMED>
__device__ __forceinline__ void carry_sync() {
  if constexpr (NAMED) asm volatile("bar.sync 1, 128;" ::: "memory");
  else __syncthreads();
}

template <int NS, bool NAMED = false>
__device__ __forceinline__ void carry_lookback(const FwdParams& p, const TileCoord& tc, int tid,
                                               const float (&S)[NS], float P, float (&h)[NS],
                                               float& Pin) {
  const int64_t slot = tc.tile * kDT + tid;
  Pin = 1.f;
  if (tc.c == 0) {
#pragma unroll
    for (int n = 0; n < NS; ++n)
      h[n] = (p.h0 != nullptr && tc.d_ok && n < p.N)
                 ? p.h0[(static_cast<int64_t>(tc.b) * p.D + tc.d) * p.N + n] : 0.f;
  } else {
    p.aggP[slot] = P;
    float4* dstS = reinterpret_cast<float4*>(p.aggS + slot * NS);
#pragma unroll
    for (int q = 0; q < NS / 4; ++q)
      dstS[q] = make_float4(S[4 * q], S[4 * q + 1], S[4 * q + 2], S[4 * q + 3]);
    carry_sync<NAMED>();
    if (tid == 0) {
      __threadfence();  // cumulative: orders every thread's stores above (seen through the barrier)
      st_release(p.flags + tc.tile, 1);
    }

    float accP = 1.f;
#pragma unroll
    for (int n = 0; n < NS; ++n) h[n] = 0.f;
    for (int j = tc.c - 1; j >= 0; --j) {
      const int64_t jt = static_cast<int64_t>(j) * tc.per_chunk + tc.rem;
      const int64_t js = jt * kDT + tid;
      const int st = wait_flag(p.flags + jt);
      if (st == 0) {
        atomicOr(&p.hdr->status, NAJU_ST_LOOKBACK_TIMEOUT);
        break;
      }
      const float4* src = reinterpret_cast<const float4*>((st == 2 ? p.ckS : p.aggS) + js * NS);
#pragma unroll
      for (int q = 0; q < NS / 4; ++q) {
        const float4 v = __ldcg(src + q);
        h[4 * q + 0] = fmaf(accP, v.x, h[4 * q + 0]);
        h[4 * q + 1] = fmaf(accP, v.y, h[4 * q + 1]);
        h[4 * q + 2] = fmaf(accP, v.z, h[4 * q + 2]);
        h[4 * q + 3] = fmaf(accP, v.w, h[4 * q + 3]);
      }
      if (st == 2) {
        Pin = accP * __ldcg(p.ckP + js);
        break;
      }
      accP *= __ldcg(p.aggP + js);
    }
  }
  float4* dstS = reinterpret_cast<float4*>(p.ckS + slot * NS);
#pragma unroll
  for (int q = 0; q < NS / 4; ++q)
    dstS[q] = make_float4(fmaf(P, h[4 * q + 0], S[4 * q + 0]), fmaf(P, h[4 * q + 1], S[4 * q + 1]),
                          fmaf(P, h[4 * q + 2], S[4 * q + 2]), fmaf(P, h[4 * q + 3], S[4 * q + 3]));
  p.ckP[slot] = P * Pin;
  carry_sync<NAMED>();
  if (tid == 0) {
    __threadfence();
    st_release(p.flags + tc.tile, 2);
  }
}

// final state / total decay outputs of the last chunk
template <int NS>
__device__ __forceinline__ void write_final(const FwdParams& p, const TileCoord& tc,
                                            const float (&xend)[NS], float Ptot) {
  if (tc.c == p.nchunks - 1 && tc.d_ok) {
    if (p.hT != nullptr) {
      float* o = p.hT + (static_cast<int64_t>(tc.b) * p.D + tc.d) * p.N;
#pragma unroll
      for (int n = 0; n < NS; ++n)
        if (n < p.N) o[n] = xend[n];
    }
    if (p.pT != nullptr) p.pT[static_cast<int64_t>(tc.b) * p.D + tc.d] = Ptot;
  }
}

// End of a forward kernel, called by every thread of every CTA after its last write.  The last CTA to
// get here looks at the status word: if a bounded wait ran out anywhere (or `inject` asks for it), it
// overwrites every output with all-ones bytes (NaN in fp32, bf16 and fp16 alike) and marks the checkpoints, so
// that a timeout can never pass for a result; no host round trip and no extra launch is needed for that.
template <typename TA>
__device__ __forceinline__ void finish_forward(const FwdParams& p) {
  __shared__ int s_bad;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_bad = 0;
    if (atomicAdd(&p.hdr->done, 1u) == gridDim.x - 1) {
      __threadfence();
      if (p.inject) atomicOr(&p.hdr->status, NAJU_ST_LOOKBACK_TIMEOUT);
      if (*reinterpret_cast<volatile int*>(&p.hdr->status) != 0) {
        s_bad = 1;
        atomicOr(p.fwd_form, 4);
      }
    }
  }
  __syncthreads();
  if (!s_bad) return;
  auto fill = [&](void* ptr, int64_t bytes) {
    if (ptr != nullptr)
      for (int64_t i = threadIdx.x; i < bytes; i += blockDim.x) static_cast<unsigned char*>(ptr)[i] = 0xFF;
  };
  fill(p.y, static_cast<int64_t>(p.B) * p.T * p.D * static_cast<int64_t>(sizeof(TA)));
  fill(p.hT, static_cast<int64_t>(p.B) * p.D * p.N * 4);
  fill(p.pT, static_cast<int64_t>(p.B) * p.D * 4);
}

}  // namespace naju
