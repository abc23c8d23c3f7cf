// Building blocks shared by the forward kernels.
#pragma once

#include "common.cuh"
#include "params.h"

namespace naju {

// Coordinates of a tile: chunk c of channel tile (batch row b, 128 channels from d0).  tile = c * per_chunk + rem.
struct TileCoord {
  int64_t tile;
  int c, rem, b, dt, per_chunk, t0, len, d0, cols, d;
  bool d_ok;
};

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
