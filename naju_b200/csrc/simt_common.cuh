// Building blocks of the exact recurrent kernels (fwd_simt.cu, bwd_simt.cu).
//
// A thread owns kC = 4 adjacent channels x K states.  The B_t / C_t values it reads from shared memory
// then serve four channels and the gates of a step serve K states: with one channel and all states per
// thread the shared-memory broadcasts alone cost more cycles than the arithmetic (a 128-bit shared load
// takes an SM 2.5 to 4 cycles, four FMA instructions take one).  Sums over the channels are formed in
// registers over the thread's four first, sums over the states over its K first; what is left goes
// through short shuffle reduce-scatters.  The L = NS / K lanes that share four channels are adjacent;
// a CTA of L warps covers the 128 channels of a tile.
//
// The gates are evaluated elementwise when a piece of the tile is staged (all threads, no serial chain)
// and the walks along time read them as fp32 from shared memory.
#pragma once

#include "common.cuh"
#include "params.h"

namespace naju {

// Below this retention the difference form of d f_logit loses more than ~3e-5 relative
// accuracy (it matches the f_logit >= -5 envelope of naju/chunk_triton.py:200).
constexpr float kDeepGate = 0.0078125f;

// Whether the backward's work is done: asked behind pdl_wait(), when the tensor-core backward, if there was one, has completed.
__device__ __forceinline__ bool tc_did_it(const BwdParams& p) {
  return p.tc_launched && (*p.fwd_form & 3) == 1 && *reinterpret_cast<volatile int*>(&p.hdr->redo) == 0;
}

namespace simt {

constexpr int kC = 4;    // channels per thread
constexpr int kSB = 32;  // steps staged at a time

template <int NS>
struct Shape {
  static constexpr int K = NS == 16 ? 4 : 8;            // states per thread
  static constexpr int L = NS / K;                      // lanes per group of four channels
  static constexpr int GW = 32 / L;                     // groups per warp
  static constexpr int W = kDT / (kC * GW);             // warps
  static constexpr int NT = 32 * W;
};

// ---------------------------------------------------------------- four adjacent channels of one step
template <typename T>
__device__ __forceinline__ float4 load4(const T* __restrict__ p, int n, bool vec) {
  if (vec && n >= 4) {
    if constexpr (sizeof(T) == 4) {
      return __ldg(reinterpret_cast<const float4*>(p));
    } else {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
      T e[4];
      *reinterpret_cast<uint2*>(e) = v;
      return make_float4(to_f32(e[0]), to_f32(e[1]), to_f32(e[2]), to_f32(e[3]));
    }
  }
  return make_float4(n > 0 ? to_f32(p[0]) : 0.f, n > 1 ? to_f32(p[1]) : 0.f, n > 2 ? to_f32(p[2]) : 0.f,
                     n > 3 ? to_f32(p[3]) : 0.f);
}

template <typename T>
__device__ __forceinline__ void store4(T* __restrict__ p, float4 v, int n, bool vec) {
  if (vec && n >= 4) {
    if constexpr (sizeof(T) == 4) {
      *reinterpret_cast<float4*>(p) = v;
    } else {
      T e[4] = {from_f32<T>(v.x), from_f32<T>(v.y), from_f32<T>(v.z), from_f32<T>(v.w)};
      *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(e);
    }
    return;
  }
  if (n > 0) p[0] = from_f32<T>(v.x);
  if (n > 1) p[1] = from_f32<T>(v.y);
  if (n > 2) p[2] = from_f32<T>(v.z);
  if (n > 3) p[3] = from_f32<T>(v.w);
}

template <typename T>
__device__ __forceinline__ bool vec4_ok(const T* base, int64_t row_stride) {
  return (reinterpret_cast<uintptr_t>(base) % (4 * sizeof(T))) == 0 && row_stride % 4 == 0;
}

// Whether 16 bytes of consecutive steps can be moved at once in a time-contiguous tensor.
template <typename T>
__device__ __forceinline__ bool vec_steps_ok(const T* base, int64_t sd) {
  return (reinterpret_cast<uintptr_t>(base) & 15) == 0 && sd * static_cast<int64_t>(sizeof(T)) % 16 == 0;
}

// A time-contiguous source (element (step r, channel c) at src[c * sd + r]) into a [kSB][128] fp32 tile:
// thread = channel, 16 bytes of its steps at a time (element by element where the layout does not allow that).  `len` steps are
// real; the rest become zero.
template <typename T, int NT>
__device__ __forceinline__ void load_tmajor(float* __restrict__ dst, const T* __restrict__ src, int64_t sd, int len,
                                            int cols, int tid) {
  constexpr int E = 16 / sizeof(T);
  const bool vec = vec_steps_ok(src, sd);
  for (int i = tid; i < kDT * (kSB / E); i += NT) {
    const int c = i % kDT, r0 = (i / kDT) * E;
    T e[E];
    if (vec && c < cols && r0 + E <= len) {
      *reinterpret_cast<uint4*>(e) = __ldg(reinterpret_cast<const uint4*>(src + c * sd + r0));
    } else {
#pragma unroll
      for (int k = 0; k < E; ++k) e[k] = (c < cols && r0 + k < len) ? src[c * sd + r0 + k] : from_f32<T>(0.f);
    }
#pragma unroll
    for (int k = 0; k < E; ++k) dst[(r0 + k) * kDT + c] = to_f32(e[k]);
  }
}
template <typename T, int NT>
__device__ __forceinline__ void store_tmajor(T* __restrict__ dst, const float* __restrict__ src, int64_t sd, int len,
                                             int cols, int tid) {
  constexpr int E = 16 / sizeof(T);
  const bool vec = vec_steps_ok(dst, sd);
  for (int i = tid; i < kDT * (kSB / E); i += NT) {
    const int c = i % kDT, r0 = (i / kDT) * E;
    if (c >= cols || r0 >= len) continue;
    T e[E];
#pragma unroll
    for (int k = 0; k < E; ++k) e[k] = from_f32<T>(src[(r0 + k) * kDT + c]);
    if (vec && r0 + E <= len) {
      *reinterpret_cast<uint4*>(dst + c * sd + r0) = *reinterpret_cast<const uint4*>(e);
    } else {
      for (int k = 0; k < E; ++k)
        if (r0 + k < len) dst[c * sd + r0 + k] = e[k];
    }
  }
}

// B and C rows of a tile as fp32 [STEPS][NS], zero padded in both directions.  load() only issues the global
// loads (16 bytes each; all of a thread's are in flight together and with whatever is loaded next), store()
// converts them into shared memory.  Rows that are not whole 16-byte pieces (N < NS, odd strides) are read
// element by element in store().
template <int NS, int NT, int STEPS>
struct StageBC {
  static constexpr int MAXV = (STEPS * NS / 4 + NT - 1) / NT;   // 16-byte pieces per thread and tensor, fp32
  uint4 vb[MAXV], vc[MAXV];
  bool vec;

  template <typename P>
  __device__ __forceinline__ void load(const P& p, int b, int t0, int len, int tid) {
    const int es = p.bc_dtype == NAJU_F32 ? 4 : 2, e = 16 / es, ppr = NS / e;   // elements per piece, pieces per row
    const char* Bp = static_cast<const char*>(p.Bm) + (b * p.bm_sb + static_cast<int64_t>(t0) * p.bm_st) * es;
    const char* Cp = static_cast<const char*>(p.Cm) + (b * p.cm_sb + static_cast<int64_t>(t0) * p.cm_st) * es;
    vec = p.N == NS && (reinterpret_cast<uintptr_t>(Bp) & 15) == 0 && (reinterpret_cast<uintptr_t>(Cp) & 15) == 0 &&
          ((p.bm_st | p.cm_st) * es & 15) == 0;
    if (!vec) return;
#pragma unroll
    for (int k = 0; k < MAXV; ++k) {
      const int i = tid + k * NT, r = i / ppr, o = (i - r * ppr) * 16;
      vb[k] = vc[k] = make_uint4(0, 0, 0, 0);
      if (r < min(len, STEPS)) {
        vb[k] = __ldg(reinterpret_cast<const uint4*>(Bp + r * p.bm_st * es + o));
        vc[k] = __ldg(reinterpret_cast<const uint4*>(Cp + r * p.cm_st * es + o));
      }
    }
  }

  template <typename T>
  __device__ __forceinline__ static void put(float* dst, const uint4& v) {
    constexpr int E = 16 / sizeof(T);
    T e[E];
    *reinterpret_cast<uint4*>(e) = v;
#pragma unroll
    for (int k = 0; k < E; k += 4)
      *reinterpret_cast<float4*>(dst + k) = make_float4(to_f32(e[k]), to_f32(e[k + 1]), to_f32(e[k + 2]), to_f32(e[k + 3]));
  }

  template <typename P>
  __device__ __forceinline__ void store(const P& p, float* s_B, float* s_C, int b, int t0, int len, int tid) {
    if (vec) {
      const int e = p.bc_dtype == NAJU_F32 ? 4 : 8;
#pragma unroll
      for (int k = 0; k < MAXV; ++k) {
        const int i = tid + k * NT;
        if (i * e >= STEPS * NS) break;
        if (p.bc_dtype == NAJU_F32) { put<float>(s_B + i * 4, vb[k]); put<float>(s_C + i * 4, vc[k]); }
        else if (p.bc_dtype == NAJU_BF16) { put<__nv_bfloat16>(s_B + i * 8, vb[k]); put<__nv_bfloat16>(s_C + i * 8, vc[k]); }
        else { put<__half>(s_B + i * 8, vb[k]); put<__half>(s_C + i * 8, vc[k]); }
      }
      return;
    }
    for (int e = tid; e < STEPS * NS; e += NT) {
      const int r = e / NS, n = e % NS;
      const bool ok = n < p.N && r < len;
      s_B[e] = ok ? load_dyn(p.Bm, p.bc_dtype, b * p.bm_sb + static_cast<int64_t>(t0 + r) * p.bm_st + n) : 0.f;
      s_C[e] = ok ? load_dyn(p.Cm, p.bc_dtype, b * p.cm_sb + static_cast<int64_t>(t0 + r) * p.cm_st + n) : 0.f;
    }
  }
};

// Stages kSB steps: f = sigmoid(f_logit) and w = sigmoid(i_logit) u into s_f / s_w ([step][128] fp32) and, with
// BWD, dy into s_dy; accumulates sum_t dy_t u_t of the thread's four channels into dd.  Steps past `len`
// become neutral (f = 1, w = dy = 0).  With a time-contiguous u, s_w must already hold u.
template <typename TA, typename TG, int NT, bool BWD, typename P>
__device__ __forceinline__ void stage_gates(const P& p, float* __restrict__ s_f, float* __restrict__ s_w,
                                            float* __restrict__ s_dy, int b, int t0, int len, int d0, int tid, float4& dd) {
  constexpr int RP = NT / 32, BATCH = kSB / RP < 4 ? kSB / RP : 4;
  const int v = tid & 31, c = 4 * v, n = p.D - d0 - c;
  const bool utm = p.u_sd > 1;
  const TA* u = reinterpret_cast<const TA*>(p.u) + b * p.u_sb + static_cast<int64_t>(t0) * p.u_st + d0 + c;
  const TG* fl = reinterpret_cast<const TG*>(p.fl) + b * p.fl_sb + static_cast<int64_t>(t0) * p.fl_st + d0 + c;
  const TG* il = reinterpret_cast<const TG*>(p.il) + b * p.il_sb + static_cast<int64_t>(t0) * p.il_st + d0 + c;
  const TA* dy = nullptr;
  if constexpr (BWD) dy = reinterpret_cast<const TA*>(p.dy) + (static_cast<int64_t>(b) * p.T + t0) * p.D + d0 + c;
  const bool vu = vec4_ok(u, p.u_st), vf = vec4_ok(fl, p.fl_st), vi = vec4_ok(il, p.il_st), vy = BWD && vec4_ok(dy, p.D);
#pragma unroll 1
  for (int r0 = tid >> 5; r0 < kSB; r0 += RP * BATCH) {
    float4 uu[BATCH], ff[BATCH], ii[BATCH], yy[BATCH];
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      const int r = r0 + k * RP, nn = r < len ? n : 0;
      uu[k] = utm ? *reinterpret_cast<const float4*>(s_w + r * kDT + c)
                  : load4(u + static_cast<int64_t>(r) * p.u_st, nn, vu);
      ff[k] = load4(fl + static_cast<int64_t>(r) * p.fl_st, nn, vf);
      ii[k] = load4(il + static_cast<int64_t>(r) * p.il_st, nn, vi);
      if constexpr (BWD) yy[k] = load4(dy + static_cast<int64_t>(r) * p.D, nn, vy);
    }
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      const int r = r0 + k * RP;
      float4 f = make_float4(1.f, 1.f, 1.f, 1.f);
      if (r < len) f = make_float4(sigmoid_f(ff[k].x), sigmoid_f(ff[k].y), sigmoid_f(ff[k].z), sigmoid_f(ff[k].w));
      const float4 w = make_float4(sigmoid_f(ii[k].x) * uu[k].x, sigmoid_f(ii[k].y) * uu[k].y,
                                   sigmoid_f(ii[k].z) * uu[k].z, sigmoid_f(ii[k].w) * uu[k].w);
      *reinterpret_cast<float4*>(s_f + r * kDT + c) = f;
      *reinterpret_cast<float4*>(s_w + r * kDT + c) = w;
      if constexpr (BWD) {
        *reinterpret_cast<float4*>(s_dy + r * kDT + c) = yy[k];
        dd.x = fmaf(yy[k].x, uu[k].x, dd.x);
        dd.y = fmaf(yy[k].y, uu[k].y, dd.y);
        dd.z = fmaf(yy[k].z, uu[k].z, dd.z);
        dd.w = fmaf(yy[k].w, uu[k].w, dd.w);
      }
    }
  }
}

// ---------------------------------------------------------------- shuffle reductions
// Sum of v[0..3] over the L adjacent lanes of a group; lane q of the group ends up with the total of entry
// chan_of(q) (with L > 4 several lanes hold the same one).
template <int L>
__device__ __forceinline__ int chan_of(int q) {
  return L == 4 ? q : (q / (L / 4)) & 3;
}
template <int L>
__device__ __forceinline__ float reduce_states(float (&v)[kC], int q) {
  const bool up = (q & (L / 2)) != 0;
  const float a = (up ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], L / 2);
  const float b = (up ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], L / 2);
  const bool up2 = (q & (L / 4)) != 0;
  float s = (up2 ? b : a) + __shfl_xor_sync(0xffffffffu, up2 ? a : b, L / 4);
#pragma unroll
  for (int m = L / 8; m >= 1; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
  return s;
}

// Sum of v[0..K) over the GW groups of a warp (lanes L apart): on return the lane holds, in v[0..count), the
// totals of entries base + j.
template <int K, int L, int GW>
struct ReduceGroups {
  static constexpr int count = K / GW > 0 ? K / GW : 1;
  static constexpr bool dup = GW > K;   // pairs of lanes end up with the same totals
  __device__ static __forceinline__ int base(int g) {
    int b = 0, cnt = K;
#pragma unroll
    for (int m = GW / 2; m >= 1; m >>= 1)
      if (cnt > 1) {
        cnt >>= 1;
        if (g & m) b += cnt;
      }
    return b;
  }
  __device__ static __forceinline__ void run(float (&v)[K], int g) {
    int cnt = K;
#pragma unroll
    for (int m = GW / 2; m >= 1; m >>= 1) {
      if (cnt > 1) {
        const int half = cnt >> 1;
        const bool up = (g & m) != 0;
#pragma unroll
        for (int j = 0; j < K / 2; ++j)
          if (j < half) v[j] = (up ? v[j + half] : v[j]) + __shfl_xor_sync(0xffffffffu, up ? v[j] : v[j + half], m * L);
        cnt = half;
      } else {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], m * L);
      }
    }
  }
};

template <int K>
__device__ __forceinline__ void lds_row(const float* __restrict__ s, float (&v)[K]) {
#pragma unroll
  for (int q = 0; q < K / 4; ++q) {
    const float4 t = reinterpret_cast<const float4*>(s)[q];
    v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
  }
}

// ---------------------------------------------------------------- carry between tiles
// K states of four channels to / from a [slot][NS] array (slot = tile * 128 + channel).
template <int NS, int K>
__device__ __forceinline__ void put_state(float* __restrict__ a, int64_t slot0, int q, const float (&x)[kC][K]) {
#pragma unroll
  for (int c = 0; c < kC; ++c)
#pragma unroll
    for (int k = 0; k < K / 4; ++k)
      *reinterpret_cast<float4*>(a + (slot0 + c) * NS + q * K + 4 * k) =
          make_float4(x[c][4 * k], x[c][4 * k + 1], x[c][4 * k + 2], x[c][4 * k + 3]);
}
template <int NS, int K>
__device__ __forceinline__ void get_state(const float* __restrict__ a, int64_t slot0, int q, float (&x)[kC][K]) {
#pragma unroll
  for (int c = 0; c < kC; ++c)
#pragma unroll
    for (int k = 0; k < K / 4; ++k) {
      const float4 v = __ldcg(reinterpret_cast<const float4*>(a + (slot0 + c) * NS + q * K + 4 * k));
      x[c][4 * k] = v.x; x[c][4 * k + 1] = v.y; x[c][4 * k + 2] = v.z; x[c][4 * k + 3] = v.w;
    }
}
// ... of the caller's [B][D][N] state tensors (NULL = zeros)
template <int K>
__device__ __forceinline__ void get_user_state(const float* __restrict__ h, int64_t bd0, int d, int D, int N, int q,
                                               float (&x)[kC][K]) {
#pragma unroll
  for (int c = 0; c < kC; ++c)
#pragma unroll
    for (int k = 0; k < K; ++k)
      x[c][k] = (h != nullptr && d + c < D && q * K + k < N) ? h[(bd0 + c) * N + q * K + k] : 0.f;
}
template <int K>
__device__ __forceinline__ void put_user_state(float* __restrict__ h, int64_t bd0, int d, int D, int N, int q,
                                               const float (&x)[kC][K]) {
#pragma unroll
  for (int c = 0; c < kC; ++c)
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (d + c < D && q * K + k < N) h[(bd0 + c) * N + q * K + k] = x[c][k];
}

// Bounded decoupled look-back of one warp.  Predecessor i (0 = nearest) is tile tile0 + i * step, i < count; the
// farthest one always publishes an inclusive state.  Flags: 0 not yet, 1 aggregate (P, S) published, 2 inclusive
// state published.  On return acc = fold of the aggregates onto the first inclusive state met and accP the product
// of the P's folded (without that tile's own); *incl_tile = that tile, or -1 when the wait ran out.
// A window of 32 flags is looked at together, one per lane, so a long run of published aggregates costs one
// round trip of flag reads, not one per tile; DEPTH aggregates are fetched together.  (More than one where registers
// are left only: B=4, T=2048, D=1024, N=16, fp32 backward 208 us with one, 264 with two.)
template <int NS, int K, int DEPTH>
__device__ __forceinline__ int64_t look_back(const int* __restrict__ flags, const float* __restrict__ aggP,
                                             const float* __restrict__ agg, const float* __restrict__ incl, int64_t tile0,
                                             int64_t step, int count, int chan0, int q, int lane, float (&acc)[kC][K],
                                             float (&accP)[kC]) {
#pragma unroll
  for (int c = 0; c < kC; ++c) {
    accP[c] = 1.f;
#pragma unroll
    for (int k = 0; k < K; ++k) acc[c][k] = 0.f;
  }
  int done = 0, spins = 0;
  for (;;) {
    const int i = done + lane;
    const int st = i < count ? ld_acquire(flags + tile0 + i * step) : 0;
    const unsigned ready = __ballot_sync(0xffffffffu, st != 0), inc = __ballot_sync(0xffffffffu, st == 2);
    __syncwarp();
    const int nready = ready == 0xffffffffu ? 32 : __ffs(~ready) - 1;
    const int first_inc = inc ? __ffs(inc) - 1 : 32;
    const int n = min(nready, first_inc + 1);
    for (int k = 0; k < n; k += DEPTH) {
      float v[DEPTH][kC][K];
      float4 pv[DEPTH];
#pragma unroll
      for (int m = 0; m < DEPTH; ++m) {
        if (k + m >= n) break;
        const int64_t t = tile0 + (done + k + m) * step;
        const bool last = k + m == first_inc;
        get_state<NS, K>(last ? incl : agg, t * kDT + chan0, q, v[m]);
        pv[m] = last ? make_float4(1.f, 1.f, 1.f, 1.f) : __ldcg(reinterpret_cast<const float4*>(aggP + t * kDT + chan0));
      }
#pragma unroll
      for (int m = 0; m < DEPTH; ++m) {
        if (k + m >= n) break;
        const float pc[kC] = {pv[m].x, pv[m].y, pv[m].z, pv[m].w};
#pragma unroll
        for (int c = 0; c < kC; ++c) {
#pragma unroll
          for (int j = 0; j < K; ++j) acc[c][j] = fmaf(accP[c], v[m][c][j], acc[c][j]);
          accP[c] *= pc[c];
        }
        if (k + m == first_inc) return tile0 + (done + k + m) * step;
      }
    }
    done += n;
    if (n == 0) {
      if (++spins > kSpinLimit) return -1;
      __nanosleep(64);
    }
  }
}

}  // namespace simt
}  // namespace naju
