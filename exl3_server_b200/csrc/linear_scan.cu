// Linear recurrences with a matrix state per head, and what stands around them.
//
// State S [dk, dv] per (sequence, head), float32, kept in the cache's per-sequence state between steps.
//
//   mode 0, a decay per token and key channel and a bonus for the current token:
//       o_t = S^T r_t + (sum_i r_ti u_i k_ti) v_t
//       S  <- diag(w_t) S + k_t v_t^T,        w_t = exp(-exp(wraw_t + w0))
//   mode 1, one decay per head (retention):
//       S  <- decay_h S + k_t v_t^T
//       o_t = S^T r_t
//
// A block owns one (row of the batch, head): thread j keeps column j of S in shared memory and walks the row's tokens
// in order; r, k and the decays of eight tokens at a time are staged in shared memory.  The state is read from and
// written back to the row's slot, so a sequence cut into steps in any way walks the same chain of sums.
//
// Rows that bring many tokens are cut into chunks of LS_CHUNK tokens that run side by side, as the element-wise
// recurrence of recurrent.cu does: over a chunk S_out = diag(A) S_in + B with A the product of the chunk's decays
// and B the chunk's own scan from zero.  A first launch leaves (A, B) per chunk, a second folds the (A, B) of the
// chunks before its own, in order, into its start and walks its chunk.  That changes roundings only.  The row's last
// chunk leaves the new state in the slot while the others may still be starting, so the first launch also copies the
// state of every row that has more than one chunk into the scratch, and the second launch starts from that copy.
//
// Everything but the element types of r, k, v (a projection's output) is float32.
#include "api.h"
#include "common.cuh"

namespace exl3 {

__device__ inline float ls_load(const void* p, int dtype, int64_t i) {
  return dtype == DT_F32 ? static_cast<const float*>(p)[i]
                         : __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}
__device__ inline float ls_load_act(const void* p, int dtype, int64_t i) {
  return dtype == DT_F32 ? __ldcg(static_cast<const float*>(p) + i)
                         : __bfloat162float(__ldcg(static_cast<const __nv_bfloat16*>(p) + i));
}
// what the projections' outputs go through before they enter the recurrence: 0 nothing, 1 silu
__device__ inline float ls_in(float x, int act) { return act == 1 ? x / (1.0f + expf(-x)) : x; }
__device__ inline void ls_store(void* p, int dtype, int64_t i, float v) {
  if (dtype == DT_F32) static_cast<float*>(p)[i] = v;
  else static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
}

// ---- token shift ---------------------------------------------------------------------------------------------------

__global__ void __launch_bounds__(256)
token_shift_kernel(const void* h, int h_dtype, const void* __restrict__ mu, int mu_dtype, int n_mix, float* prev,
                   const int* __restrict__ tok_seq, const int* __restrict__ row_start,
                   const int* __restrict__ slot_ids, void* out, int out_dtype, int T, int H) {
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x;
  const int b = __ldcg(tok_seq + t);
  const int first = __ldcg(row_start + b), end = __ldcg(row_start + b + 1);
  float* st = prev + (int64_t)__ldcg(slot_ids + b) * H;
  for (int c = threadIdx.x; c < H; c += blockDim.x) {
    const float x = ls_load_act(h, h_dtype, (int64_t)t * H + c);
    float before;
    if (t == first) {
      // the same thread reads the entry and then leaves the row's last h of this step in it
      before = __ldcg(st + c);
      st[c] = ls_load_act(h, h_dtype, (int64_t)(end - 1) * H + c);
    } else {
      before = ls_load_act(h, h_dtype, (int64_t)(t - 1) * H + c);
    }
    const float d = before - x;
    for (int s = 0; s < n_mix; ++s)
      ls_store(out, out_dtype, ((int64_t)s * T + t) * H + c, fmaf(d, ls_load(mu, mu_dtype, (int64_t)s * H + c), x));
  }
}

// Eight consecutive values as floats from float32 or bfloat16 storage, through L2; and back.
__device__ inline void ls_load8(const float* p, float (&v)[8]) {
  float a[4], b[4];
  load_vec_cg(p, a);
  load_vec_cg(p + 4, b);
#pragma unroll
  for (int e = 0; e < 4; ++e) { v[e] = a[e]; v[4 + e] = b[e]; }
}
__device__ inline void ls_load8(const __nv_bfloat16* p, float (&v)[8]) { load_vec_cg(p, v); }
__device__ inline void ls_store8(float* p, const float (&v)[8]) {
  const float a[4] = {v[0], v[1], v[2], v[3]}, b[4] = {v[4], v[5], v[6], v[7]};
  store_vec(p, a);
  store_vec(p + 4, b);
}
__device__ inline void ls_store8(__nv_bfloat16* p, const float (&v)[8]) { store_vec(p, v); }

// Token shift with eight features a thread (H a multiple of 8, float32 mu).
template <typename TH, typename TO>
__global__ void __launch_bounds__(256)
token_shift_vec_kernel(const TH* h, const float* __restrict__ mu, int n_mix, float* prev, const int* __restrict__ tok_seq,
                       const int* __restrict__ row_start, const int* __restrict__ slot_ids, TO* out, int T, int H) {
  pdl_wait();
  pdl_trigger();
  const int t = blockIdx.x;
  const int b = __ldcg(tok_seq + t);
  const int first = __ldcg(row_start + b), end = __ldcg(row_start + b + 1);
  float* st = prev + (int64_t)__ldcg(slot_ids + b) * H;
  for (int c = threadIdx.x * 8; c < H; c += blockDim.x * 8) {
    float x[8], before[8];
    ls_load8(h + (int64_t)t * H + c, x);
    if (t == first) {
      float last[8];
      ls_load8(st + c, before);
      ls_load8(h + (int64_t)(end - 1) * H + c, last);
      ls_store8(st + c, last);
    } else {
      ls_load8(h + (int64_t)(t - 1) * H + c, before);
    }
    for (int s = 0; s < n_mix; ++s) {
      float m[8], o[8];
      load_vec(mu + (int64_t)s * H + c, reinterpret_cast<float(&)[4]>(m[0]));
      load_vec(mu + (int64_t)s * H + c + 4, reinterpret_cast<float(&)[4]>(m[4]));
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = fmaf(before[e] - x[e], m[e], x[e]);
      ls_store8(out + ((int64_t)s * T + t) * H + c, o);
    }
  }
}

// ---- the scan ------------------------------------------------------------------------------------------------------

constexpr int LS_STAGE = 8;                      // tokens staged in shared memory at a time
constexpr int LS_CHUNK = 64;                     // tokens of a chunk when a row's tokens run side by side

struct ScanArgs {
  const void* r; int64_t r_ld; const void* k; int64_t k_ld; int rk_dtype;
  const void* v; int64_t v_ld; int v_dtype;
  const void* wraw; int64_t w_ld; int w_dtype;
  const void* w0; const void* u; int wu_dtype;
  const float* decay;
  float* state; const int* slot_ids; const int* row_start;
  float* out; float* ab; float* snap;
  int heads, dk, dv, places, chunk;              // chunk: tokens of a chunk, LS_CHUNK or (the wide kernel) as lw_chunk says
  int act;                                       // see ls_in
};

// Chunk j of batch row b has a place of its own among floor(T / chunk) + B + 1 places.
__device__ inline int ls_place(int chunk, int t0, int b, int j) { return t0 / chunk + b + j; }

// phase 0: a row's tokens of the step, from its state, state written back.
// phase 1: a chunk from zero, (A, B) to scratch (no output; the row's last chunk does nothing).
// phase 2: the chunks before folded into the state, then the chunk; the row's last chunk writes the state.
template <int MODE>
__global__ void linear_scan_kernel(ScanArgs a, int phase) {
  extern __shared__ float ls_sm[];
  const int dk = a.dk, dv = a.dv;
  float* S = ls_sm;                              // [dk][dv]
  float* sr = S + dk * dv;                       // [LS_STAGE][dk]
  float* sk = sr + LS_STAGE * dk;                // [LS_STAGE][dk]
  float* sw = sk + LS_STAGE * dk;                // [LS_STAGE][dk] decays (mode 0)
  float* sb = sw + LS_STAGE * dk;                // [LS_STAGE] bonus factors (mode 0)
  float* sA = sb + LS_STAGE;                     // [dk] product of decays (phase 1)
  pdl_wait();
  pdl_trigger();
  const int hd = blockIdx.x, c = blockIdx.y, b = blockIdx.z;
  const int t0 = __ldcg(a.row_start + b), t1 = __ldcg(a.row_start + b + 1);
  int lo = t0, hi = t1;
  if (phase == 1) {
    lo = t0 + c * LS_CHUNK;
    hi = lo + LS_CHUNK;
    if (hi >= t1) return;                        // the row's last chunk has nobody after it
  } else if (phase == 2) {
    lo = t0 + c * LS_CHUNK;
    hi = min(lo + LS_CHUNK, t1);
    if (lo >= t1) return;
  }
  const int j = threadIdx.x;
  const bool col = j < dv;
  float* st = a.state + ((int64_t)__ldcg(a.slot_ids + b) * a.heads + hd) * dk * dv;
  const int64_t rec = (int64_t)dk + (int64_t)dk * dv;      // floats of one (place, head): A then B
  float* snap = a.snap + ((int64_t)b * a.heads + hd) * dk * dv;
  if (phase == 1) {
    if (col) for (int i = 0; i < dk; ++i) S[i * dv + j] = 0.0f;
    for (int i = j; i < dk; i += blockDim.x) sA[i] = 1.0f;
    if (c == 0 && col) for (int i = 0; i < dk; ++i) snap[i * dv + j] = __ldcg(st + i * dv + j);
  } else {
    // a row of several chunks starts from the copy that the first launch took
    const float* from = (phase == 2 && t1 - t0 > LS_CHUNK) ? snap : st;
    if (col) for (int i = 0; i < dk; ++i) S[i * dv + j] = __ldcg(from + i * dv + j);
    if (phase == 2 && col) {
      for (int p = 0; p < c; ++p) {              // the chunks before this one, in order
        const float* ab = a.ab + ((int64_t)ls_place(LS_CHUNK, t0, b, p) * a.heads + hd) * rec;
        for (int i = 0; i < dk; ++i) S[i * dv + j] = fmaf(__ldcg(ab + i), S[i * dv + j], __ldcg(ab + dk + i * dv + j));
      }
    }
  }
  const float gamma = MODE == 1 ? a.decay[hd] : 0.0f;
  for (int s0 = lo; s0 < hi; s0 += LS_STAGE) {
    const int n = min(LS_STAGE, hi - s0);
    __syncthreads();                             // the stage before has been used
    for (int idx = threadIdx.x; idx < n * dk; idx += blockDim.x) {
      const int tt = idx / dk, i = idx - tt * dk;
      const int64_t t = s0 + tt;
      sr[idx] = ls_in(ls_load_act(a.r, a.rk_dtype, t * a.r_ld + (int64_t)hd * dk + i), a.act);
      sk[idx] = ls_in(ls_load_act(a.k, a.rk_dtype, t * a.k_ld + (int64_t)hd * dk + i), a.act);
      if (MODE == 0) {
        const float z = ls_load_act(a.wraw, a.w_dtype, t * a.w_ld + (int64_t)hd * dk + i) +
                        ls_load(a.w0, a.wu_dtype, (int64_t)hd * dk + i);
        sw[idx] = expf(-expf(z));
      }
    }
    __syncthreads();
    if (MODE == 0) {
      // the bonus factor sum_i r_i u_i k_i of each staged token, a warp a token
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
      for (int tt = warp; tt < n; tt += nw) {
        float acc = 0.0f;
        for (int i = lane; i < dk; i += 32)
          acc = fmaf(sr[tt * dk + i] * ls_load(a.u, a.wu_dtype, (int64_t)hd * dk + i), sk[tt * dk + i], acc);
        acc = warp_sum(acc);
        if (lane == 0) sb[tt] = acc;
      }
      if (phase == 1)
        for (int i = threadIdx.x; i < dk; i += blockDim.x) {
          float p = sA[i];
          for (int tt = 0; tt < n; ++tt) p *= sw[tt * dk + i];
          sA[i] = p;
        }
      __syncthreads();
    } else if (phase == 1) {
      for (int i = threadIdx.x; i < dk; i += blockDim.x) {
        float p = sA[i];
        for (int tt = 0; tt < n; ++tt) p *= gamma;
        sA[i] = p;
      }
    }
    if (col) {
      for (int tt = 0; tt < n; ++tt) {
        const int64_t t = s0 + tt;
        const float vj = ls_in(ls_load_act(a.v, a.v_dtype, t * a.v_ld + (int64_t)hd * dv + j), a.act);
        const float* rr = sr + tt * dk;
        const float* kk = sk + tt * dk;
        float acc = 0.0f;
        if (MODE == 0) {
          const float* ww = sw + tt * dk;
#pragma unroll 4
          for (int i = 0; i < dk; ++i) {
            const float s = S[i * dv + j];
            acc = fmaf(rr[i], s, acc);
            S[i * dv + j] = fmaf(ww[i], s, kk[i] * vj);
          }
          acc = fmaf(sb[tt], vj, acc);
        } else {
#pragma unroll 4
          for (int i = 0; i < dk; ++i) {
            const float s = fmaf(gamma, S[i * dv + j], kk[i] * vj);
            S[i * dv + j] = s;
            acc = fmaf(rr[i], s, acc);
          }
        }
        if (phase != 1) a.out[t * ((int64_t)a.heads * dv) + (int64_t)hd * dv + j] = acc;
      }
    }
  }
  if (phase == 1) {
    __syncthreads();
    float* ab = a.ab + ((int64_t)ls_place(LS_CHUNK, t0, b, c) * a.heads + hd) * rec;
    for (int i = threadIdx.x; i < dk; i += blockDim.x) ab[i] = sA[i];
    if (col) for (int i = 0; i < dk; ++i) ab[dk + i * dv + j] = S[i * dv + j];
  } else if (hi == t1 && col) {
    for (int i = 0; i < dk; ++i) st[i * dv + j] = S[i * dv + j];
  }
}

// The same with the state in registers, for key sizes of 16, 32, 64 and 128 and up to 128 values a head.  A column of
// S is cut over LS_Q threads (a quarter of the key channels each), so a token costs a thread DK / 4 steps of its chain
// instead of DK and a block has four times the warps to hide its loads behind; the four partial sums of an output
// meet in shared memory once per stage of eight tokens.  r, k and the decays are read four at a time.  (With the whole
// state in shared memory a token cost a warp five shared-memory instructions per key channel, which bounded the
// kernel: 8,192 tokens of 32 heads of 64 x 64 took 0.94 ms a launch.)
constexpr int LS_Q = 4;
constexpr int LS_MAX_DV = 128;

template <int MODE, int DK, int PHASE>
__global__ void __launch_bounds__(LS_Q * LS_MAX_DV, DK <= 64 ? 2 : 1) linear_scan_reg_kernel(ScanArgs a, int) {
  constexpr int phase = PHASE;                       // 1 (a chunk's summary) needs neither r nor the outputs
  constexpr int DKQ = DK / LS_Q;
  __shared__ __align__(16) float sr[LS_STAGE * DK];
  __shared__ __align__(16) float sk[LS_STAGE * DK];
  __shared__ __align__(16) float sw[MODE == 0 ? LS_STAGE * DK : 4];
  __shared__ float sb[LS_STAGE];
  __shared__ float sA[DK];
  extern __shared__ float ls_acc[];                  // [LS_STAGE][LS_Q][dvr] partial outputs
  const int dv = a.dv;
  const int dvr = blockDim.x / LS_Q;                 // dv rounded up to whole warps
  pdl_wait();
  pdl_trigger();
  const int hd = blockIdx.x, c = blockIdx.y, b = blockIdx.z;
  const int t0 = __ldcg(a.row_start + b), t1 = __ldcg(a.row_start + b + 1);
  int lo = t0, hi = t1;
  if (phase == 1) {
    lo = t0 + c * LS_CHUNK;
    hi = lo + LS_CHUNK;
    if (hi >= t1) return;
  } else if (phase == 2) {
    lo = t0 + c * LS_CHUNK;
    hi = min(lo + LS_CHUNK, t1);
    if (lo >= t1) return;
  }
  const int q = threadIdx.x / dvr, j = threadIdx.x - q * dvr;
  const bool col = j < dv;
  const int i0 = q * DKQ;                            // this thread's key channels: i0 .. i0 + DKQ - 1
  float* st = a.state + ((int64_t)__ldcg(a.slot_ids + b) * a.heads + hd) * DK * dv;
  const int64_t rec = (int64_t)DK + (int64_t)DK * dv;
  float* snap = a.snap + ((int64_t)b * a.heads + hd) * DK * dv;
  float S[DKQ];
  if (phase == 1) {
#pragma unroll
    for (int i = 0; i < DKQ; ++i) S[i] = 0.0f;
    for (int i = threadIdx.x; i < DK; i += blockDim.x) sA[i] = 1.0f;
    if (c == 0 && col) {
#pragma unroll
      for (int i = 0; i < DKQ; ++i) snap[(i0 + i) * dv + j] = __ldcg(st + (i0 + i) * dv + j);
    }
  } else {
    const float* from = (phase == 2 && t1 - t0 > LS_CHUNK) ? snap : st;
#pragma unroll
    for (int i = 0; i < DKQ; ++i) S[i] = col ? __ldcg(from + (i0 + i) * dv + j) : 0.0f;
    if (phase == 2 && col) {
#pragma unroll 2
      for (int p = 0; p < c; ++p) {                  // the chunks before this one, in order
        const float* ab = a.ab + ((int64_t)ls_place(LS_CHUNK, t0, b, p) * a.heads + hd) * rec;
#pragma unroll
        for (int i = 0; i < DKQ; ++i) S[i] = fmaf(__ldcg(ab + i0 + i), S[i], __ldcg(ab + DK + (i0 + i) * dv + j));
      }
    }
  }
  const float gamma = MODE == 1 ? a.decay[hd] : 0.0f;
  // A stage's r, k and decay inputs come into registers a stage ahead, so that their way from memory passes under the
  // stage before's arithmetic instead of standing in front of the barrier (a block has at least 128 threads, so
  // PER values a thread cover a stage).
  constexpr int PER = LS_STAGE * DK / 128;
  float pr[PER], pk[PER], pw[MODE == 0 ? PER : 1];
  auto fetch = [&](int s0) {
    const int n = min(LS_STAGE, hi - s0);
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      const int idx = threadIdx.x + e * blockDim.x;
      if (idx < n * DK) {
        const int tt = idx / DK, i = idx - tt * DK;
        const int64_t t = s0 + tt;
        if (phase != 1) pr[e] = ls_load_act(a.r, a.rk_dtype, t * a.r_ld + (int64_t)hd * DK + i);
        pk[e] = ls_load_act(a.k, a.rk_dtype, t * a.k_ld + (int64_t)hd * DK + i);
        if (MODE == 0) pw[e] = ls_load_act(a.wraw, a.w_dtype, t * a.w_ld + (int64_t)hd * DK + i);
      }
    }
  };
  fetch(lo);
  for (int s0 = lo; s0 < hi; s0 += LS_STAGE) {
    const int n = min(LS_STAGE, hi - s0);
    __syncthreads();                                 // the stage before has been used, its outputs written
#pragma unroll
    for (int e = 0; e < PER; ++e) {
      const int idx = threadIdx.x + e * blockDim.x;
      if (idx < n * DK) {
        if (phase != 1) sr[idx] = ls_in(pr[e], a.act);
        sk[idx] = ls_in(pk[e], a.act);
        if (MODE == 0) sw[idx] = expf(-expf(pw[e] + ls_load(a.w0, a.wu_dtype, (int64_t)hd * DK + idx % DK)));
      }
    }
    // the values of the stage's tokens, asked for before the barrier
    float vj[LS_STAGE];
#pragma unroll
    for (int tt = 0; tt < LS_STAGE; ++tt)
      vj[tt] = (col && tt < n) ? ls_in(ls_load_act(a.v, a.v_dtype, (int64_t)(s0 + tt) * a.v_ld + (int64_t)hd * dv + j), a.act) : 0.0f;
    __syncthreads();
    if (s0 + LS_STAGE < hi) fetch(s0 + LS_STAGE);
    if (MODE == 0) {
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
      for (int tt = warp; phase != 1 && tt < n; tt += nw) {
        float acc = 0.0f;
        for (int i = lane; i < DK; i += 32)
          acc = fmaf(sr[tt * DK + i] * ls_load(a.u, a.wu_dtype, (int64_t)hd * DK + i), sk[tt * DK + i], acc);
        acc = warp_sum(acc);
        if (lane == 0) sb[tt] = acc;
      }
      if (phase == 1)
        for (int i = threadIdx.x; i < DK; i += blockDim.x) {
          float p = sA[i];
          for (int tt = 0; tt < n; ++tt) p *= sw[tt * DK + i];
          sA[i] = p;
        }
      __syncthreads();
    } else if (phase == 1) {
      for (int i = threadIdx.x; i < DK; i += blockDim.x) {
        float p = sA[i];
        for (int tt = 0; tt < n; ++tt) p *= gamma;
        sA[i] = p;
      }
    }
#pragma unroll
    for (int tt = 0; tt < LS_STAGE; ++tt) {
      if (tt < n) {
        const float4* rr = reinterpret_cast<const float4*>(sr + tt * DK + i0);
        const float4* kk = reinterpret_cast<const float4*>(sk + tt * DK + i0);
        float acc0 = 0.0f, acc1 = 0.0f;
        if (MODE == 0) {
          const float4* ww = reinterpret_cast<const float4*>(sw + tt * DK + i0);
#pragma unroll
          for (int i4 = 0; i4 < DKQ / 4; ++i4) {
            const float4 r4 = rr[i4], k4 = kk[i4], w4 = ww[i4];
            if (phase != 1) {
              acc0 = fmaf(r4.x, S[4 * i4 + 0], acc0); acc1 = fmaf(r4.y, S[4 * i4 + 1], acc1);
              acc0 = fmaf(r4.z, S[4 * i4 + 2], acc0); acc1 = fmaf(r4.w, S[4 * i4 + 3], acc1);
            }
            S[4 * i4 + 0] = fmaf(w4.x, S[4 * i4 + 0], k4.x * vj[tt]);
            S[4 * i4 + 1] = fmaf(w4.y, S[4 * i4 + 1], k4.y * vj[tt]);
            S[4 * i4 + 2] = fmaf(w4.z, S[4 * i4 + 2], k4.z * vj[tt]);
            S[4 * i4 + 3] = fmaf(w4.w, S[4 * i4 + 3], k4.w * vj[tt]);
          }
          if (q == 0) acc0 = fmaf(sb[tt], vj[tt], acc0);          // the bonus, once
        } else {
#pragma unroll
          for (int i4 = 0; i4 < DKQ / 4; ++i4) {
            const float4 r4 = rr[i4], k4 = kk[i4];
            S[4 * i4 + 0] = fmaf(gamma, S[4 * i4 + 0], k4.x * vj[tt]);
            S[4 * i4 + 1] = fmaf(gamma, S[4 * i4 + 1], k4.y * vj[tt]);
            S[4 * i4 + 2] = fmaf(gamma, S[4 * i4 + 2], k4.z * vj[tt]);
            S[4 * i4 + 3] = fmaf(gamma, S[4 * i4 + 3], k4.w * vj[tt]);
            if (phase != 1) {
              acc0 = fmaf(r4.x, S[4 * i4 + 0], acc0); acc1 = fmaf(r4.y, S[4 * i4 + 1], acc1);
              acc0 = fmaf(r4.z, S[4 * i4 + 2], acc0); acc1 = fmaf(r4.w, S[4 * i4 + 3], acc1);
            }
          }
        }
        if (phase != 1) ls_acc[(tt * LS_Q + q) * dvr + j] = acc0 + acc1;
      }
    }
    if (phase != 1) {
      __syncthreads();
      // the four parts of every output of the stage, summed in the order of the key channels
      for (int idx = threadIdx.x; idx < n * dv; idx += blockDim.x) {
        const int tt = idx / dv, jj = idx - tt * dv;
        const float* pa = ls_acc + tt * LS_Q * dvr + jj;
        a.out[(int64_t)(s0 + tt) * ((int64_t)a.heads * dv) + (int64_t)hd * dv + jj] =
            ((pa[0] + pa[dvr]) + pa[2 * dvr]) + pa[3 * dvr];
      }
    }
  }
  if (phase == 1) {
    __syncthreads();
    float* ab = a.ab + ((int64_t)ls_place(LS_CHUNK, t0, b, c) * a.heads + hd) * rec;
    for (int i = threadIdx.x; i < DK; i += blockDim.x) ab[i] = sA[i];
    if (col) {
#pragma unroll
      for (int i = 0; i < DKQ; ++i) ab[DK + (i0 + i) * dv + j] = S[i];
    }
  } else if (hi == t1 && col) {
#pragma unroll
    for (int i = 0; i < DKQ; ++i) st[(i0 + i) * dv + j] = S[i];
  }
}

// The same for key sizes of 64 and up to 128 values a head in sixteens, with 16-byte rows.  A thread has two columns of S
// and a quarter of their key channels, as eight pairs of channels: a token costs it 48 paired fma (one and a product for the
// update, one for the output) and 13 reads of shared memory for r, k, the decays and v.  The quarters of a column are lanes
// of one warp (a quarter's eight lanes side by side: with the quarters side by side the same loop took 157 us instead of
// 115), so an output's four parts meet in two shuffles and no barrier; sixteen tokens are staged at a time,
// read 16 bytes a thread a stage ahead and widened (the decays' exponentials taken) on their way into shared memory.
// Bound by what a warp does for one token after the other (some 270 cycles alone on its SM): rows of 520, 120, 300,
// 400, 200, 350, 450 and 320 tokens with 32 heads of 64 x 64 and decays 114 us (the kernel above, in chunks: 368), with 16
// heads of 64 x 128 127 us (280); one row of 8,192 tokens 474 (1,546) and 349 us (1,284).  Sixteen columns of eight channels,
// or eight of four, a thread's work cut differently at the same sum: 119 and 150 us for the first of these.
constexpr int LW_DK = 64, LW_STAGE = 16, LW_Q = 4, LW_COLS = 2, LW_PAIRS = LW_DK / LW_Q / 2;
// A staged row: the quarters 20 floats apart, so that the four addresses of a warp's read do not collide.
constexpr int LW_QP = LW_DK / LW_Q + 4, LW_ROW = LW_Q * LW_QP;
__device__ inline int lw_at(int i) { return i / (LW_DK / LW_Q) * LW_QP + i % (LW_DK / LW_Q); }

__device__ inline unsigned long long lw_dup(float v) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ inline unsigned long long lw_mul(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ inline unsigned long long lw_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ inline float2 lw_split(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ inline unsigned long long lw_pair(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}

// The tokens of a chunk of a row of n: a step's, a multiple of LS_CHUNK, or (LW_BY_ROW) what the row's own length gives:
// up to LW_CUTS chunks of some sixty-fours, rows of up to 128 tokens whole.  Places are counted in the shortest chunks.
constexpr int LW_BY_ROW = -1, LW_CUTS = 16;
__device__ inline int lw_chunk(int chunk, int n) {
  if (chunk != LW_BY_ROW) return chunk;
  return n <= 2 * LS_CHUNK ? max(n, 1) : (n + LS_CHUNK * LW_CUTS - 1) / (LS_CHUNK * LW_CUTS) * LS_CHUNK;
}
__host__ __device__ inline int lw_place_len(int chunk) { return chunk == LW_BY_ROW ? LS_CHUNK : chunk; }

// TK: element type of r, k; TV: of v and the raw decays.  PHASE as above.
template <int MODE, int PHASE, typename TK, typename TV>
__global__ void __launch_bounds__(LW_Q * LS_MAX_DV / LW_COLS, MODE == 0 ? 1 : 2) linear_scan_wide_kernel(ScanArgs a) {
  constexpr int VK = Elem<TK>::vec, VV = Elem<TV>::vec;
  __shared__ __align__(16) float sr[LW_STAGE * LW_ROW];
  __shared__ __align__(16) float sk[LW_STAGE * LW_ROW];
  __shared__ __align__(16) float sw[MODE == 0 ? LW_STAGE * LW_ROW : 4];
  __shared__ __align__(16) float sv[LW_STAGE * LS_MAX_DV];
  __shared__ float sb[LW_STAGE];
  __shared__ float su[MODE == 0 ? LW_DK : 1], sw0[MODE == 0 ? LW_DK : 1];
  const int tid = threadIdx.x, lane = tid & 31, dv = a.dv, threads = blockDim.x;
  const int hd = blockIdx.x, c = blockIdx.y, b = blockIdx.z;
  if (MODE == 0 && tid < LW_DK) {
    su[tid] = ls_load(a.u, a.wu_dtype, (int64_t)hd * LW_DK + tid);
    sw0[tid] = ls_load(a.w0, a.wu_dtype, (int64_t)hd * LW_DK + tid);
  }
  pdl_wait();
  pdl_trigger();
  const int t0 = __ldcg(a.row_start + b), t1 = __ldcg(a.row_start + b + 1);
  int lo = t0, hi = t1;
  const int chunk = PHASE == 0 ? 0 : lw_chunk(a.chunk, t1 - t0);
  if (PHASE == 1) {
    lo = t0 + c * chunk;
    hi = lo + chunk;
    if (hi >= t1) return;
  } else if (PHASE == 2) {
    lo = t0 + c * chunk;
    hi = min(lo + chunk, t1);
    if (lo >= t1) return;
  }
  const int q = lane >> 3, j = ((tid >> 5) * 8 + (lane & 7)) * LW_COLS;    // columns j, j + 1; channels 16 q .. 16 q + 15
  float* st = a.state + ((int64_t)__ldcg(a.slot_ids + b) * a.heads + hd) * LW_DK * dv;
  const int64_t rec = (int64_t)LW_DK + (int64_t)LW_DK * dv;
  float* snap = a.snap + ((int64_t)b * a.heads + hd) * LW_DK * dv;
  unsigned long long S[LW_COLS][LW_PAIRS];
  float decays = 1.0f;                                                      // phase 1: channel tid's product
  // a matrix's part of this thread: pairs of channels of both columns
  auto pairs_of = [&](const float* from, auto&& f) {
#pragma unroll
    for (int p = 0; p < LW_PAIRS; ++p) {
      const int i = q * (LW_DK / LW_Q) + 2 * p;
      const float2 x = __ldcg(reinterpret_cast<const float2*>(from + (int64_t)i * dv + j));
      const float2 y = __ldcg(reinterpret_cast<const float2*>(from + (int64_t)(i + 1) * dv + j));
      const unsigned long long v[LW_COLS] = {lw_pair(x.x, y.x), lw_pair(x.y, y.y)};
      f(p, i, v);
    }
  };
  auto take = [&](int p, int, const unsigned long long (&v)[LW_COLS]) {
#pragma unroll
    for (int m = 0; m < LW_COLS; ++m) S[m][p] = v[m];
  };
  auto put_pairs = [&](float* to) {
#pragma unroll
    for (int p = 0; p < LW_PAIRS; ++p) {
      const int i = q * (LW_DK / LW_Q) + 2 * p;
      const float2 c0 = lw_split(S[0][p]), c1 = lw_split(S[1][p]);
      *reinterpret_cast<float2*>(to + (int64_t)i * dv + j) = make_float2(c0.x, c1.x);
      *reinterpret_cast<float2*>(to + (int64_t)(i + 1) * dv + j) = make_float2(c0.y, c1.y);
    }
  };
  if (PHASE == 1) {
    if (c == 0) {
      pairs_of(st, take);
      put_pairs(snap);
    }
#pragma unroll
    for (int p = 0; p < LW_PAIRS; ++p)
#pragma unroll
      for (int m = 0; m < LW_COLS; ++m) S[m][p] = 0;
  } else {
    pairs_of((PHASE == 2 && t1 - t0 > chunk) ? snap : st, take);
    if (PHASE == 2) {
#pragma unroll 1
      for (int e = 0; e < c; ++e) {                                         // the chunks before this one, in order
        const float* ab = a.ab + ((int64_t)ls_place(lw_place_len(a.chunk), t0, b, e) * a.heads + hd) * rec;
        pairs_of(ab + LW_DK, [&](int p, int i, const unsigned long long (&v)[LW_COLS]) {
          const float2 w = __ldcg(reinterpret_cast<const float2*>(ab + i));
          const unsigned long long ww = lw_pair(w.x, w.y);
#pragma unroll
          for (int m = 0; m < LW_COLS; ++m) S[m][p] = lw_fma(ww, S[m][p], v[m]);
        });
      }
    }
  }
  const float gamma = MODE == 1 ? a.decay[hd] : 0.0f;
  const unsigned long long gamma2 = lw_dup(gamma);

  // a stage's inputs a stage ahead in registers, 16 bytes a thread
  constexpr int NK = LW_STAGE * LW_DK / VK, NW = LW_STAGE * LW_DK / VV;     // pieces of r or k, of the raw decays
  constexpr int HK = NK / 128, HW = NW / 128, HV = LW_STAGE / (2 * VV);     // a block has 2 dv >= 128 threads
  uint4 pr[HK], pk[HK], pw[MODE == 0 ? HW : 1], pv[HV];
  const int vpieces = dv / VV;                                              // of a token's values
  auto fetch = [&](int s0) {
    const int n = min(LW_STAGE, hi - s0);
#pragma unroll
    for (int e = 0; e < HK; ++e) {
      const int idx = tid + e * threads, tt = idx / (LW_DK / VK), i = idx % (LW_DK / VK) * VK;
      if (idx < NK && tt < n) {
        if (PHASE != 1) pr[e] = load_raw_cg(static_cast<const TK*>(a.r) + (int64_t)(s0 + tt) * a.r_ld + hd * LW_DK + i);
        pk[e] = load_raw_cg(static_cast<const TK*>(a.k) + (int64_t)(s0 + tt) * a.k_ld + hd * LW_DK + i);
      }
    }
    if (MODE == 0) {
#pragma unroll
      for (int e = 0; e < HW; ++e) {
        const int idx = tid + e * threads, tt = idx / (LW_DK / VV), i = idx % (LW_DK / VV) * VV;
        if (idx < NW && tt < n) pw[e] = load_raw_cg(static_cast<const TV*>(a.wraw) + (int64_t)(s0 + tt) * a.w_ld + hd * LW_DK + i);
      }
    }
#pragma unroll
    for (int e = 0; e < HV; ++e) {
      const int idx = tid + e * threads, tt = idx / vpieces;
      if (tt < n) pv[e] = load_raw_cg(static_cast<const TV*>(a.v) + (int64_t)(s0 + tt) * a.v_ld + (int64_t)hd * dv + (idx - tt * vpieces) * VV);
    }
  };
  fetch(lo);
#pragma unroll 1
  for (int s0 = lo; s0 < hi; s0 += LW_STAGE) {
    const int n = min(LW_STAGE, hi - s0);
    __syncthreads();                                                        // the stage before has been used
#pragma unroll
    for (int e = 0; e < HK; ++e) {
      const int idx = tid + e * threads, tt = idx / (LW_DK / VK), i = idx % (LW_DK / VK) * VK;
      float bonus = 0.0f;
      if (idx < NK && tt < n) {
        float x[VK], y[VK];
        unpack_raw(pk[e], y, (const TK*)nullptr);
#pragma unroll
        for (int z = 0; z < VK; ++z) y[z] = ls_in(y[z], a.act);
#pragma unroll
        for (int z = 0; z < VK; z += 4)
          *reinterpret_cast<float4*>(sk + tt * LW_ROW + lw_at(i + z)) = make_float4(y[z], y[z + 1], y[z + 2], y[z + 3]);
        if (PHASE != 1) {
          unpack_raw(pr[e], x, (const TK*)nullptr);
#pragma unroll
          for (int z = 0; z < VK; ++z) {
            x[z] = ls_in(x[z], a.act);
            if (MODE == 0) bonus = fmaf(x[z] * su[i + z], y[z], bonus);
          }
#pragma unroll
          for (int z = 0; z < VK; z += 4)
            *reinterpret_cast<float4*>(sr + tt * LW_ROW + lw_at(i + z)) = make_float4(x[z], x[z + 1], x[z + 2], x[z + 3]);
        }
      }
      if (MODE == 0 && PHASE != 1) {                                        // a token's pieces are neighbours in a warp
#pragma unroll
        for (int o = LW_DK / VK / 2; o > 0; o >>= 1) bonus += __shfl_xor_sync(0xffffffffu, bonus, o);
        if (idx < NK && tt < n && i == 0) sb[tt] = bonus;
      }
    }
    if (MODE == 0) {
#pragma unroll
      for (int e = 0; e < HW; ++e) {
        const int idx = tid + e * threads, tt = idx / (LW_DK / VV), i = idx % (LW_DK / VV) * VV;
        if (idx < NW && tt < n) {
          float x[VV];
          unpack_raw(pw[e], x, (const TV*)nullptr);
#pragma unroll
          for (int z = 0; z < VV; ++z) x[z] = expf(-expf(x[z] + sw0[i + z]));
#pragma unroll
          for (int z = 0; z < VV; z += 4)
            *reinterpret_cast<float4*>(sw + tt * LW_ROW + lw_at(i + z)) = make_float4(x[z], x[z + 1], x[z + 2], x[z + 3]);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < HV; ++e) {
      const int idx = tid + e * threads, tt = idx / vpieces;
      if (tt < n) {
        float x[VV];
        unpack_raw(pv[e], x, (const TV*)nullptr);
#pragma unroll
        for (int z = 0; z < VV; ++z) x[z] = ls_in(x[z], a.act);
#pragma unroll
        for (int z = 0; z < VV; z += 4)
          *reinterpret_cast<float4*>(sv + tt * LS_MAX_DV + (idx - tt * vpieces) * VV + z) =
              make_float4(x[z], x[z + 1], x[z + 2], x[z + 3]);
      }
    }
    __syncthreads();
    if (s0 + LW_STAGE < hi) fetch(s0 + LW_STAGE);
    if (PHASE == 1 && tid < LW_DK) {
      for (int tt = 0; tt < n; ++tt)
        decays *= MODE == 0 ? sw[tt * LW_ROW + lw_at(tid)] : gamma;
    }
    const bool odd = q & 1;                                                 // the column whose output ends up in this lane
    float* to = a.out + (int64_t)s0 * a.heads * dv + (int64_t)hd * dv + j + (odd ? 1 : 0);
#pragma unroll 2
    for (int tt = 0; tt < n; ++tt) {
      const float* rt = sr + tt * LW_ROW + q * LW_QP;
      const float* kt = sk + tt * LW_ROW + q * LW_QP;
      const float* wt = MODE == 0 ? sw + tt * LW_ROW + q * LW_QP : nullptr;
      const float2 v = *reinterpret_cast<const float2*>(sv + tt * LS_MAX_DV + j);
      const unsigned long long vv[LW_COLS] = {lw_dup(v.x), lw_dup(v.y)};
      unsigned long long o[LW_COLS] = {0, 0};
#pragma unroll
      for (int h = 0; h < LW_PAIRS / 2; ++h) {
        const ulonglong2 k2 = *reinterpret_cast<const ulonglong2*>(kt + h * 4);
        const ulonglong2 w2 = MODE == 0 ? *reinterpret_cast<const ulonglong2*>(wt + h * 4) : make_ulonglong2(gamma2, gamma2);
        const ulonglong2 r2 = PHASE != 1 ? *reinterpret_cast<const ulonglong2*>(rt + h * 4) : make_ulonglong2(0, 0);
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          const unsigned long long kp = z ? k2.y : k2.x, wp = z ? w2.y : w2.x, rp = z ? r2.y : r2.x;
          const int p = 2 * h + z;
#pragma unroll
          for (int m = 0; m < LW_COLS; ++m) {
            if (MODE == 0 && PHASE != 1) o[m] = lw_fma(rp, S[m][p], o[m]);  // the output sees the state before the token
            S[m][p] = lw_fma(wp, S[m][p], lw_mul(kp, vv[m]));
            if (MODE == 1 && PHASE != 1) o[m] = lw_fma(rp, S[m][p], o[m]);
          }
        }
      }
      if (PHASE != 1) {
        // lanes of odd quarters go on with the second column, of even ones with the first; then both halves
        const float2 e0 = lw_split(o[0]), e1 = lw_split(o[1]);
        const float y0 = e0.x + e0.y, y1 = e1.x + e1.y;
        float out = (odd ? y1 : y0) + __shfl_xor_sync(0xffffffffu, odd ? y0 : y1, 8);
        out += __shfl_xor_sync(0xffffffffu, out, 16);
        if (MODE == 0) out = fmaf(sb[tt], odd ? v.y : v.x, out);            // the bonus
        if (q < 2) to[(int64_t)tt * a.heads * dv] = out;
      }
    }
  }
  if (PHASE == 1) {
    float* ab = a.ab + ((int64_t)ls_place(lw_place_len(a.chunk), t0, b, c) * a.heads + hd) * rec;
    if (tid < LW_DK) ab[tid] = decays;
    put_pairs(ab + LW_DK);
  } else if (hi == t1) {
    put_pairs(st);
  }
}

// ---- per-head norm and gate ------------------------------------------------------------------------------------------

__global__ void __launch_bounds__(128)
head_norm_gate_kernel(const float* o, const void* __restrict__ w, int w_dtype, const void* gate, int gate_dtype,
                      int64_t gate_ld, int gate_kind, float eps, void* out, int out_dtype, int n_items, int heads, int dv) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);       // (token, head)
  if (item >= n_items) return;
  const int t = item / heads, hd = item - t * heads;
  const float* src = o + (int64_t)item * dv;
  float ss = 0.0f;
  for (int e = lane; e < dv; e += 32) {
    const float x = __ldcg(src + e);
    ss += x * x;
  }
  ss = warp_sum(ss);
  const float inv = 1.0f / sqrtf(ss / (float)dv + eps);
  for (int e = lane; e < dv; e += 32) {
    float x = __ldcg(src + e) * inv;
    if (w) x *= ls_load(w, w_dtype, (int64_t)hd * dv + e);
    if (gate) {
      const float g = ls_load_act(gate, gate_dtype, (int64_t)t * gate_ld + (int64_t)hd * dv + e);
      x *= (gate_kind == 1 ? 1.0f : g) / (1.0f + expf(-g));
    }
    ls_store(out, out_dtype, (int64_t)item * dv + e, x);
  }
}

// The same for wide heads (all heads normed together make one of heads * dv values): a block per (token, head), the
// head's values kept in registers between the sum of squares and the output (up to HN_WIDE_PER values a thread; what is
// beyond is read again).
constexpr int HN_WIDE_THREADS = 512, HN_WIDE_PER = 8;

__global__ void __launch_bounds__(HN_WIDE_THREADS)
head_norm_gate_wide_kernel(const float* o, const void* __restrict__ w, int w_dtype, const void* gate, int gate_dtype,
                           int64_t gate_ld, int gate_kind, float eps, void* out, int out_dtype, int heads, int dv) {
  __shared__ float red[32];
  pdl_wait();
  pdl_trigger();
  const int item = blockIdx.x;
  const int t = item / heads, hd = item - t * heads;
  const float* src = o + (int64_t)item * dv;
  float x[HN_WIDE_PER];
  float ss = 0.0f;
#pragma unroll
  for (int i = 0; i < HN_WIDE_PER; ++i) {
    const int e = threadIdx.x + i * HN_WIDE_THREADS;
    x[i] = e < dv ? __ldcg(src + e) : 0.0f;
    ss = fmaf(x[i], x[i], ss);
  }
  for (int e = threadIdx.x + HN_WIDE_PER * HN_WIDE_THREADS; e < dv; e += HN_WIDE_THREADS) {
    const float v = __ldcg(src + e);
    ss = fmaf(v, v, ss);
  }
  ss = block_sum(ss, red);
  const float inv = 1.0f / sqrtf(ss / (float)dv + eps);
  auto emit = [&](int e, float v) {
    v *= inv;
    if (w) v *= ls_load(w, w_dtype, (int64_t)hd * dv + e);
    if (gate) {
      const float g = ls_load_act(gate, gate_dtype, (int64_t)t * gate_ld + (int64_t)hd * dv + e);
      v *= (gate_kind == 1 ? 1.0f : g) / (1.0f + expf(-g));
    }
    ls_store(out, out_dtype, (int64_t)item * dv + e, v);
  };
#pragma unroll
  for (int i = 0; i < HN_WIDE_PER; ++i) {
    const int e = threadIdx.x + i * HN_WIDE_THREADS;
    if (e < dv) emit(e, x[i]);
  }
  for (int e = threadIdx.x + HN_WIDE_PER * HN_WIDE_THREADS; e < dv; e += HN_WIDE_THREADS) emit(e, __ldcg(src + e));
}

// The same with four values a lane (dv a multiple of 4, at most 128 a head: one piece a lane), float32 weight.  LANES: of a
// head, 16 where they are enough (a warp then has two heads).  Bound by its bytes and the chain of a load, a sum and a store:
// 101,216 heads of 64 with gates in bfloat16, 52 MB, 16.9 us = 0.47 of the copy rate (32 lanes a head and a gate a load: 30),
// 50,608 heads of 128 16.5 us (17.2).  Gates or outputs that do not lie on four of their size go one by one (gate_vec, out_vec):
// 14.8 us for the heads of 64 with float32 gates off 16 bytes, 14.3 on them (back to back; the general kernel 37.8).
template <typename TG, typename TO, int LANES>
__global__ void __launch_bounds__(128)
head_norm_gate_vec_kernel(const float* o, const float* __restrict__ w, const TG* gate, int64_t gate_ld, int gate_kind,
                          float eps, TO* out, int n_items, int heads, int dv, bool gate_vec, bool out_vec) {
  pdl_wait();
  pdl_trigger();
  const int item = blockIdx.x * (blockDim.x / LANES) + threadIdx.x / LANES;    // the threads may be more than 2^32
  const int t = item / heads, hd = item - t * heads;
  const int e = threadIdx.x % LANES * 4;
  const bool mine = item < n_items && e < dv;
  float x[4] = {0.0f, 0.0f, 0.0f, 0.0f}, g[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (mine) {
    load_vec_cg(o + (int64_t)item * dv + e, x);
    if (gate) {                                                          // through L2: a kernel of this step wrote it
      const TG* from = gate + (int64_t)t * gate_ld + (int64_t)hd * dv + e;
      if (!gate_vec) {
#pragma unroll
        for (int i = 0; i < 4; ++i) g[i] = ls_load_act(from, Elem<TG>::code, i);
      } else if constexpr (sizeof(TG) == 4) {
        load_vec_cg(from, g);
      } else {
        const uint2 raw = __ldcg(reinterpret_cast<const uint2*>(from));
        g[0] = __uint_as_float(raw.x << 16); g[1] = __uint_as_float(raw.x & 0xffff0000u);
        g[2] = __uint_as_float(raw.y << 16); g[3] = __uint_as_float(raw.y & 0xffff0000u);
      }
    }
  }
  float ss = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3];
#pragma unroll
  for (int s = LANES / 2; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
  const float inv = 1.0f / sqrtf(ss / (float)dv + eps);
  if (mine) {
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[i] = x[i] * inv;
      if (w) v[i] *= w[(int64_t)hd * dv + e + i];
      if (gate) v[i] *= (gate_kind == 1 ? 1.0f : g[i]) / (1.0f + (sizeof(TO) == 4 ? expf(-g[i]) : __expf(-g[i])));
    }
    TO* to = out + (int64_t)item * dv + e;
    if (!out_vec) {
#pragma unroll
      for (int i = 0; i < 4; ++i) Elem<TO>::store(to + i, v[i]);
    } else if constexpr (sizeof(TO) == 4) {
      *reinterpret_cast<float4*>(to) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
      __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
      *reinterpret_cast<uint2*>(to) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
    }
  }
}

}  // namespace exl3

using namespace exl3;

// Sizes that the wide kernel takes (with 16-byte rows: else the kernels above run).
static bool ls_wide(int dk, int dv) { return dk == LW_DK && dv % 16 == 0 && dv >= 64 && dv <= LS_MAX_DV; }

static int ls_sm_count() {
  static thread_local int dev_of = -1, count = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev != dev_of) {
    if (cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) count = 148;
    dev_of = dev;
  }
  return count;
}

// Tokens of a chunk, 0 for rows that are walked whole.  The kernels above take chunks of 64 of every row beyond 128 tokens: their
// blocks are too few to fill the GPU with whole rows (four rows of 2,048 tokens off 16 bytes, 32 heads of 64 x 64: whole 2,001
// us, in chunks 1,113).  The wide kernel walks rows whole while they keep half the SMs busy
// for as long as the longest one takes (the eight rows above: whole 114 us, in chunks of 64 / 128
// / 256 132 / 126 / 171; four rows of 2,048 287 against 448 / 366 / 356); else chunks leave two blocks an SM, since every chunk
// pays for folding the ones before it (one row of 8,192: chunks of 64 747 us, of 256 378, of 896 470, whole 1,137).  With
// float32 values each row is cut by its own length alone, so that its bits do not depend on the rows beside it: the eight rows
// in float32 135 us (whole 119), four rows of 2,048 364 (327), one of 8,192 401.
static int ls_chunk_len(bool wide, int v_dtype, int T, int heads, int max_new) {
  if (max_new <= 2 * LS_CHUNK) return 0;
  if (!wide) return LS_CHUNK;
  if (v_dtype == DT_F32) return LW_BY_ROW;
  const int64_t work = (int64_t)T * heads, sms = ls_sm_count();
  if (2 * work >= sms * max_new) return 0;
  const int64_t len = (work / (2 * sms) + LS_CHUNK - 1) / LS_CHUNK * LS_CHUNK;
  return len < LS_CHUNK ? LS_CHUNK : (len >= max_new ? 0 : (int)len);
}

static size_t ls_scratch_bytes(int chunk, int B, int T, int heads, int dk, int dv) {
  if (chunk == 0) return 0;
  return ((size_t)(T / lw_place_len(chunk) + B + 1) * heads * ((size_t)dk + (size_t)dk * dv) + (size_t)B * heads * dk * dv) *
         sizeof(float);
}

// Enough for either kernel: the shortest chunks take the most.
extern "C" size_t exl3_linear_scan_scratch_bytes(int B, int T, int heads, int dk, int dv, int max_new) {
  return ls_scratch_bytes(ls_chunk_len(false, DT_F32, T, heads, max_new), B, T, heads, dk, dv);
}

extern "C" int exl3_token_shift(const void* h, int h_dtype, const void* mu, int mu_dtype, int n_mix, float* prev,
                                const int* tok_seq, const int* row_start, const int* slot_ids, void* out,
                                int out_dtype, int T, int H, cudaStream_t stream) {
  if (T == 0) return 0;
  if (T < 0 || H < 1 || n_mix < 1 || prev == nullptr) {
    set_error("token_shift: bad sizes T=%d H=%d mixes=%d", T, H, n_mix);
    return ERR_BAD_ARGUMENT;
  }
  const bool vec = H % 8 == 0 && mu_dtype == DT_F32 && h_dtype == out_dtype && aligned16(h) && aligned16(mu) &&
                   aligned16(prev) && aligned16(out);
  const dim3 threads(H >= 2048 ? 256 : 128);
  if (vec && h_dtype == DT_BF16)
    launch_pdl(token_shift_vec_kernel<__nv_bfloat16, __nv_bfloat16>, dim3(T), threads, 0, stream,
               static_cast<const __nv_bfloat16*>(h), static_cast<const float*>(mu), n_mix, prev, tok_seq, row_start,
               slot_ids, static_cast<__nv_bfloat16*>(out), T, H);
  else if (vec && h_dtype == DT_F32)
    launch_pdl(token_shift_vec_kernel<float, float>, dim3(T), threads, 0, stream, static_cast<const float*>(h),
               static_cast<const float*>(mu), n_mix, prev, tok_seq, row_start, slot_ids, static_cast<float*>(out), T, H);
  else
    launch_pdl(token_shift_kernel, dim3(T), dim3(H >= 1024 ? 256 : 128), 0, stream, h, h_dtype, mu, mu_dtype, n_mix,
               prev, tok_seq, row_start, slot_ids, out, out_dtype, T, H);
  return launch_status("token_shift");
}

extern "C" int exl3_linear_scan(int mode, const void* r, int64_t r_ld, const void* k, int64_t k_ld, int rk_dtype,
                                const void* v, int64_t v_ld, int v_dtype, const void* wraw, int64_t w_ld, int w_dtype,
                                const void* w0, const void* u, int wu_dtype, const float* decay, float* state,
                                const int* slot_ids, const int* row_start, float* out, int B, int T, int heads, int dk,
                                int dv, int max_new, int in_act, float* scratch, size_t scratch_bytes, cudaStream_t stream) {
  if (B == 0 || T == 0) return 0;
  if (B < 0 || T < 0 || heads < 1 || dk < 1 || dv < 1 || dv > 1024 || B > 65535 || mode < 0 || mode > 1 ||
      (mode == 0 && (wraw == nullptr || w0 == nullptr || u == nullptr)) || (mode == 1 && decay == nullptr) || in_act < 0 || in_act > 1) {
    set_error("linear_scan: bad arguments mode=%d rows=%d tokens=%d heads=%d dk=%d dv=%d", mode, B, T, heads, dk, dv);
    return ERR_BAD_ARGUMENT;
  }
  size_t smem = ((size_t)dk * dv + 3 * (size_t)LS_STAGE * dk + LS_STAGE + dk) * sizeof(float);
  if (smem > 200 * 1024) {
    set_error("linear_scan: a state of %d x %d per head does not fit shared memory", dk, dv);
    return ERR_UNSUPPORTED;
  }
  void (*kernel)(ScanArgs, int) = mode == 0 ? linear_scan_kernel<0> : linear_scan_kernel<1>;
  // key sizes of 16, 32, 64 and 128 with up to 128 values a head: the state in registers
  bool regs = dv <= LS_MAX_DV;
  void (*by_phase[3])(ScanArgs, int) = {kernel, kernel, kernel};
#define EXL3_SCAN(DKV)                                                                                            \
  case DKV:                                                                                                       \
    for (int ph = 0; ph < 3; ++ph)                                                                                \
      by_phase[ph] = mode == 0 ? (ph == 0 ? linear_scan_reg_kernel<0, DKV, 0> : ph == 1 ? linear_scan_reg_kernel<0, DKV, 1> \
                                                                                         : linear_scan_reg_kernel<0, DKV, 2>) \
                               : (ph == 0 ? linear_scan_reg_kernel<1, DKV, 0> : ph == 1 ? linear_scan_reg_kernel<1, DKV, 1> \
                                                                                         : linear_scan_reg_kernel<1, DKV, 2>); \
    break;
  if (regs) {
    switch (dk) {
      EXL3_SCAN(16) EXL3_SCAN(32) EXL3_SCAN(64) EXL3_SCAN(128)
      default: regs = false;
    }
  }
#undef EXL3_SCAN
  const int dvr = (dv + 31) / 32 * 32;
  if (regs) smem = (size_t)LS_STAGE * LS_Q * dvr * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) {
      set_error("linear_scan: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(e));
      return (int)e;
    }
  }
  ScanArgs a;
  a.r = r; a.r_ld = r_ld; a.k = k; a.k_ld = k_ld; a.rk_dtype = rk_dtype; a.v = v; a.v_ld = v_ld; a.v_dtype = v_dtype;
  a.wraw = wraw; a.w_ld = w_ld; a.w_dtype = w_dtype; a.w0 = w0; a.u = u; a.wu_dtype = wu_dtype; a.decay = decay;
  a.state = state; a.slot_ids = slot_ids; a.row_start = row_start; a.out = out; a.ab = scratch;
  a.act = in_act;
  a.heads = heads; a.dk = dk; a.dv = dv;
  const int vk = rk_dtype == DT_F32 ? 4 : 8, vv = v_dtype == DT_F32 ? 4 : 8;
  const bool wide = ls_wide(dk, dv) && r_ld % vk == 0 && k_ld % vk == 0 && v_ld % vv == 0 && aligned16(r) && aligned16(k) &&
                    aligned16(v) && aligned16(state) && aligned16(out) && aligned16(scratch) &&
                    (mode == 1 || (w_dtype == v_dtype && w_ld % vv == 0 && aligned16(wraw)));
  a.chunk = ls_chunk_len(wide, v_dtype, T, heads, max_new);
  a.places = a.chunk != 0 ? T / lw_place_len(a.chunk) + B + 1 : 0;
  a.snap = scratch ? scratch + (size_t)a.places * heads * ((size_t)dk + (size_t)dk * dv) : nullptr;
  const int threads = regs ? LS_Q * dvr : dvr;
  auto go = [&](int phase, int chunks) {
    const dim3 grid(heads, chunks, B);
    if (!wide) {
      launch_pdl(by_phase[phase], grid, dim3(threads), smem, stream, a, phase);
      return;
    }
#define EXL3_WIDE(M, TK, TV)                                                                                          \
  launch_pdl(phase == 0 ? linear_scan_wide_kernel<M, 0, TK, TV> : phase == 1 ? linear_scan_wide_kernel<M, 1, TK, TV>  \
                                                                              : linear_scan_wide_kernel<M, 2, TK, TV>, \
             grid, dim3(LW_Q * dv / LW_COLS), 0, stream, a)
#define EXL3_WIDE_TYPES(M)                                                                    \
  if (rk_dtype == DT_F32 && v_dtype == DT_F32) EXL3_WIDE(M, float, float);                    \
  else if (rk_dtype == DT_F32) EXL3_WIDE(M, float, __nv_bfloat16);                            \
  else if (v_dtype == DT_F32) EXL3_WIDE(M, __nv_bfloat16, float);                             \
  else EXL3_WIDE(M, __nv_bfloat16, __nv_bfloat16);
    if (mode == 0) { EXL3_WIDE_TYPES(0) } else { EXL3_WIDE_TYPES(1) }
#undef EXL3_WIDE_TYPES
#undef EXL3_WIDE
  };
  if (a.chunk != 0) {
    int chunks = ceil_div(max_new, lw_place_len(a.chunk));
    if (a.chunk == LW_BY_ROW && chunks > LW_CUTS) chunks = LW_CUTS;
    if (scratch == nullptr || ls_scratch_bytes(a.chunk, B, T, heads, dk, dv) > scratch_bytes || chunks > 65535) {
      set_error("linear_scan: scratch of %zu bytes is too small for %d tokens", scratch_bytes, T);
      return ERR_SCRATCH;
    }
    go(1, chunks);
    int rc = launch_status("linear_scan (chunks)");
    if (rc) return rc;
    go(2, chunks);
    return launch_status("linear_scan (fold)");
  }
  go(0, 1);
  return launch_status("linear_scan");
}

extern "C" int exl3_head_norm_gate(const float* o, const void* w, int w_dtype, const void* gate, int gate_dtype,
                                   int64_t gate_ld, int gate_kind, float eps, void* out, int out_dtype, int T, int heads,
                                   int dv, cudaStream_t stream) {
  if (T == 0) return 0;
  if (T < 0 || heads < 1 || dv < 1 || gate_kind < 0 || gate_kind > 1) { set_error("head_norm_gate: bad sizes"); return ERR_BAD_ARGUMENT; }
  const int items = T * heads;
  const bool vec = dv % 4 == 0 && dv <= 128 && (w == nullptr || w_dtype == DT_F32) && aligned16(o) &&
                   (gate == nullptr || gate_ld % 4 == 0);
  // four gates, four outputs at once where they lie on their own size
  auto on_four = [](const void* p, int dtype) { return (reinterpret_cast<uintptr_t>(p) & (dtype == DT_F32 ? 15u : 7u)) == 0; };
  const bool gate_vec = on_four(gate, gate_dtype), out_vec = on_four(out, out_dtype);
  const float* wf = static_cast<const float*>(w);
  const dim3 grid(ceil_div(items, 4)), threads(128);
  if (dv > 256)
    launch_pdl(head_norm_gate_wide_kernel, dim3(items), dim3(HN_WIDE_THREADS), 0, stream, o, w, w_dtype, gate, gate_dtype,
               gate_ld, gate_kind, eps, out, out_dtype, heads, dv);
  else if (vec && ((gate_dtype == DT_BF16 && out_dtype == DT_BF16) || (gate_dtype == DT_F32 && (out_dtype == DT_BF16 || out_dtype == DT_F32)))) {
    const dim3 g16(ceil_div(items, 8));
#define EXL3_HNG(TG, TO)                                                                                                \
  if (dv <= 64)                                                                                                         \
    launch_pdl(head_norm_gate_vec_kernel<TG, TO, 16>, g16, threads, 0, stream, o, wf, static_cast<const TG*>(gate), gate_ld, \
               gate_kind, eps, static_cast<TO*>(out), items, heads, dv, gate_vec, out_vec);                                        \
  else                                                                                                                  \
    launch_pdl(head_norm_gate_vec_kernel<TG, TO, 32>, grid, threads, 0, stream, o, wf, static_cast<const TG*>(gate), gate_ld, \
               gate_kind, eps, static_cast<TO*>(out), items, heads, dv, gate_vec, out_vec);
    if (gate_dtype == DT_BF16) { EXL3_HNG(__nv_bfloat16, __nv_bfloat16) }
    else if (out_dtype == DT_BF16) { EXL3_HNG(float, __nv_bfloat16) }
    else { EXL3_HNG(float, float) }
#undef EXL3_HNG
  }
  else
    launch_pdl(head_norm_gate_kernel, grid, threads, 0, stream, o, w, w_dtype, gate, gate_dtype, gate_ld, gate_kind, eps,
               out, out_dtype, items, heads, dv);
  return launch_status("head_norm_gate");
}
