// Plain matrix product on the CUDA cores: y[M,N] = x[M,K] . w[N,K]^T (+ bias).
//
// This is the true 32-bit path of every projection (no tensor cores, no
// reduced-precision mode) and the fallback for sizes the fast kernels refuse.
// The reference keeps weights as (in, out) and calls a library matmul
// (src/model.cpp:549-552); the checkpoint's (out, in) order is kept here.
//
// One order of summation for every output, whatever M, N, the kernel or what else is in the batch.  K is cut into
// pieces of 8; piece q belongs to lane q mod 16.  A lane walks its pieces from K = 0 upward, one fma a product, the even
// and the odd features on an accumulator each (neighbours in memory, so a pair of them is one fma.rn.f32x2 without any
// packing), and adds the two at its end; lanes 4g .. 4g + 3 are added in order to group g's sum, and the four groups'
// sums in order.  So half a warp that streams a row of w has a lane of the sum in every thread (32 bytes each), four
// groups of threads that share a tile of outputs have a group of lanes each, and both give the same bits.  (Against one
// accumulator over all of K the chains are also shorter: at K = 4,096 the
// error against 64 bits is 2.1e-7, not 1.1e-6.)
#include "api.h"
#include "common.cuh"
#include <algorithm>

namespace exl3 {

constexpr int GS_PIECE = 8;                          // features of a piece
constexpr int GS_LANES = 16;                         // lanes of an output's sum
constexpr int GS_GROUPS = 4, GS_GROUP_LANES = 4;     // and how they are added up

__device__ inline void gs_cp16(void* smem, const void* gmem, bool ok) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  const int bytes = ok ? 16 : 0;                     // nothing read, zeros written
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}
__device__ inline void gs_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ inline void gs_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// an element as it lies in memory, and its value
__device__ inline uint32_t gs_raw(const float* p) { return __ldcg(reinterpret_cast<const uint32_t*>(p)); }
__device__ inline uint32_t gs_raw(const __nv_bfloat16* p) { return __ldcg(reinterpret_cast<const unsigned short*>(p)); }
template <typename T> __device__ inline float gs_value(uint32_t raw) { return __uint_as_float(sizeof(T) == 4 ? raw : raw << 16); }

// two products on two accumulators: lo += a.lo * b.lo, hi += a.hi * b.hi
__device__ inline void gs_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ inline float gs_both(unsigned long long acc) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(acc));
  return lo + hi;
}

// Many rows: a block has a tile of 64 x 64 outputs, and (SPLIT 4) each of its four groups of 128 threads (8 x 4 outputs a
// thread) a quarter of the lanes: the groups walk different pieces of K with rings and barriers of their own, and meet once at the
// end.  So a narrow output (1,024 columns at some hundred rows: fewer tiles than SMs) still has sixteen warps an SM.  The
// sums of finished lanes wait in shared memory, which leaves the registers to the pairs of accumulators.  With many tiles, or
// with K too short for all lanes, a block has one group that walks all of them (SPLIT 1), four blocks an SM, whose starts and ends
// run beside one another: 2,000 x 8,192 (rows, columns) x 64 88 us (four groups 142; one accumulator over K 103), x 1,024 928 (976).
// Bound by the fma pipe and by what shared memory returns (12 reads of 8 bytes a lane, 128 bytes a cycle, for 32 paired fma)
// about equally: 525 x 8,192 x 1,024 (rows, columns, K) 278 us, 32 TFLOP/s; 525 x 1,024 x 4,096 130 us (one accumulator and 4 x 4
// outputs a thread, an element a load: 442 and 390 us; this kernel with scalar fma and the lanes' sums in registers 302 and 140).
constexpr int GT_TILE = 64, GT_GROUP = 128;
constexpr int GT_PITCH = GS_PIECE + 4;               // floats; rows 48 bytes apart: the reads of 8 rows do not collide
constexpr int GT_STAGE_FLOATS = 2 * GT_TILE * GT_PITCH;
constexpr int GT_OUT_PITCH = GT_TILE + 8;
// SPLIT: groups of threads in a block, GS_GROUPS or 1.
template <int SPLIT> constexpr int gt_stages() { return SPLIT == 1 ? 3 : 4; }
template <int SPLIT> constexpr int gt_ring_floats() { return SPLIT * gt_stages<SPLIT>() * GT_STAGE_FLOATS; }
template <int SPLIT> constexpr int gt_smem() {                // the ring, sums of lanes, with one group also sums of groups
  return (gt_ring_floats<SPLIT>() + (SPLIT == 1 ? 2 : SPLIT) * GT_GROUP * 32) * 4;
}
static_assert(GS_GROUPS * GT_TILE * GT_OUT_PITCH <= gt_ring_floats<GS_GROUPS>(), "the groups' sums go where the rings were");

// VEC: float32, K % 4 == 0 and 16-byte aligned operands (16-byte asynchronous copies); else element by element, the loads of a
// stage in registers while the stage before is worked on: 1,000 x 8,192 x 1,020 in bfloat16 616 us, x 1,023 in float32 616
// (one accumulator in blocks of 64 x 64 765 and 762; every load waited for before the stage, two threads a row, 968 and 922).
template <typename TI, typename TO, bool VEC, int SPLIT>
__global__ void __launch_bounds__(SPLIT * GT_GROUP, SPLIT == 1 ? 4 : 1)
gemm_simt_kernel(const TI* __restrict__ x, const TI* __restrict__ w, const TI* __restrict__ bias,
                 TO* __restrict__ y, int M, int N, int K) {
  constexpr int THREADS = SPLIT * GT_GROUP, STAGES = gt_stages<SPLIT>(), GROUP_LANES = GS_LANES / SPLIT;
  extern __shared__ __align__(16) float gt_smem[];
  pdl_wait();
  pdl_trigger();
  const int g = threadIdx.x / GT_GROUP, t = threadIdx.x % GT_GROUP;
  // a warp has 4 x 8 threads: its reads of x are four rows, of w eight, a wavefront each
  const int tx = (t & 7) + (t >> 6) * 8, ty = ((t >> 3) & 3) + ((t >> 5) & 1) * 4;
  const int m0 = blockIdx.y * GT_TILE, n0 = blockIdx.x * GT_TILE;
  float* ring = gt_smem + g * STAGES * GT_STAGE_FLOATS;
  float4* sums = reinterpret_cast<float4*>(gt_smem + gt_ring_floats<SPLIT>()) + threadIdx.x;   // [8][threads], this thread's own
  float4* totals = sums + 8 * THREADS;                        // the same of finished groups of lanes (SPLIT 1)
  const int pieces = (K + GS_PIECE - 1) / GS_PIECE;
  const int first_lane = g * GROUP_LANES, last_lane = first_lane + GROUP_LANES;

  // One stage: one piece of the 64 rows of x and of w.  16 bytes a thread and operand, half a row, asynchronously; or, element by
  // element, a feature of every sixteenth row (a warp's loads then share their sectors), asked for before the stage in hand is
  // worked on and stored behind it.
  const int fr = VEC ? t >> 1 : t >> 3, fk = VEC ? (t & 1) * 4 : t & 7;
  const bool in_m = m0 + fr < M, in_n = n0 + fr < N;
  const TI* xr = x + (int64_t)(in_m ? m0 + fr : 0) * K + (VEC ? 0 : fk);
  const TI* wr = w + (int64_t)(in_n ? n0 + fr : 0) * K + (VEC ? 0 : fk);
  struct Ahead { uint32_t x[4], w[4]; };
  auto ask = [&](Ahead& v, int q) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const bool in_k = q * GS_PIECE + fk < K;
      const int64_t at = (int64_t)e * 16 * K + q * GS_PIECE;
      v.x[e] = in_k && m0 + fr + 16 * e < M ? gs_raw(xr + at) : 0u;
      v.w[e] = in_k && n0 + fr + 16 * e < N ? gs_raw(wr + at) : 0u;
    }
  };
  auto put = [&](const Ahead& v, int slot) {
    float* a = ring + slot * GT_STAGE_FLOATS + fr * GT_PITCH + fk;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      a[e * 16 * GT_PITCH] = gs_value<TI>(v.x[e]);
      a[(GT_TILE + e * 16) * GT_PITCH] = gs_value<TI>(v.w[e]);
    }
  };
  auto copy = [&](int slot, int q) {
    float* a = ring + slot * GT_STAGE_FLOATS + fr * GT_PITCH + fk;
    const int k = q * GS_PIECE + fk;
    const bool in_k = k < K;
    gs_cp16(a, xr + (in_k ? k : 0), in_k && in_m);
    gs_cp16(a + GT_TILE * GT_PITCH, wr + (in_k ? k : 0), in_k && in_n);
  };
  // the group's stages in order: lane by lane, each from its first piece on
  int fl = first_lane, fq = fl;                               // the next stage to fill
  auto fill_next = [&](int slot, Ahead& v) {
    const bool more = fl < last_lane && fq < pieces;
    if (more) {
      if constexpr (VEC) copy(slot, fq);
      else ask(v, fq);
      fq += GS_LANES;
      if (fq >= pieces) { ++fl; fq = fl; }
    }
    if (VEC) gs_commit();
    return more;
  };
  {
    Ahead v[STAGES - 1];
    bool some[STAGES - 1];
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) some[s] = fill_next(s, v[s]);
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s)
      if (!VEC && some[s]) put(v[s], s);
  }

  unsigned long long acc[8][4];
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (SPLIT > 1) sums[i * THREADS] = zero;
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
  }
  int slot = 0;
  for (int lane = first_lane; lane < last_lane && lane < pieces; ++lane) {
    for (int q = lane; q < pieces; q += GS_LANES) {
      if (VEC) gs_wait<STAGES - 2>();
      asm volatile("bar.sync %0, 128;" ::"r"(1 + g) : "memory");
      const int last = slot == 0 ? STAGES - 1 : slot - 1;  // the slot that was read last
      Ahead v;
      const bool some = fill_next(last, v);
      const float* a = ring + slot * GT_STAGE_FLOATS + ty * GT_PITCH;
      const float* b = ring + slot * GT_STAGE_FLOATS + (GT_TILE + tx) * GT_PITCH;
      slot = slot + 1 == STAGES ? 0 : slot + 1;
#pragma unroll
      for (int h = 0; h < GS_PIECE / 2; ++h) {
        unsigned long long av[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) av[i] = *reinterpret_cast<const unsigned long long*>(a + i * 8 * GT_PITCH + h * 2);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const unsigned long long bv = *reinterpret_cast<const unsigned long long*>(b + j * 16 * GT_PITCH + h * 2);
#pragma unroll
          for (int i = 0; i < 8; ++i) gs_fma2(acc[i][j], av[i], bv);
        }
      }
      if (!VEC && some) put(v, last);
    }
    // a lane is finished: to its group's sum, and with one group of threads a finished group's to the total
    const bool first = SPLIT == 1 && lane % GS_GROUP_LANES == 0;
    const bool ends = SPLIT == 1 && (lane % GS_GROUP_LANES == GS_GROUP_LANES - 1 || lane + 1 >= pieces);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float4 v = first ? zero : sums[i * THREADS];
      v.x += gs_both(acc[i][0]); v.y += gs_both(acc[i][1]); v.z += gs_both(acc[i][2]); v.w += gs_both(acc[i][3]);
      if (ends && lane >= GS_GROUP_LANES) {
        const float4 u = totals[i * THREADS];
        v.x = u.x + v.x; v.y = u.y + v.y; v.z = u.z + v.z; v.w = u.w + v.w;
      }
      (ends ? totals : sums)[i * THREADS] = v;
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    }
  }
  if (VEC) gs_wait<0>();
  if constexpr (SPLIT == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = m0 + ty + 8 * i;
      const float4 v4 = totals[i * THREADS];
      const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + tx + 16 * j;
        if (m < M && n < N) Elem<TO>::store(y + (int64_t)m * N + n, bias ? v[j] + Elem<TI>::load(bias + n) : v[j]);
      }
    }
    return;
  }
  __syncthreads();                                            // every ring has been read
  float* mine = gt_smem + g * GT_TILE * GT_OUT_PITCH + ty * GT_OUT_PITCH + tx;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float4 v = sums[i * THREADS];
    float* o = mine + 8 * i * GT_OUT_PITCH;
    o[0] = v.x; o[16] = v.y; o[32] = v.z; o[48] = v.w;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < GT_TILE * GT_TILE; idx += THREADS) {
    const int r = idx >> 6, c = idx & 63;
    if (m0 + r >= M || n0 + c >= N) continue;
    const float* p = gt_smem + r * GT_OUT_PITCH + c;
    constexpr int G = GT_TILE * GT_OUT_PITCH;
    float v = ((p[0] + p[G]) + p[2 * G]) + p[3 * G];
    if (bias) v += Elem<TI>::load(bias + n0 + c);
    Elem<TO>::store(y + (int64_t)(m0 + r) * N + n0 + c, v);
  }
}

// Few rows in float32: half a warp streams R rows of w against MR rows of x, a thread a lane of every sum.  The block's
// segment of x (1,024 features) is in shared memory, the two 16-byte halves of the pieces in planes of their own so that
// the threads' reads do not collide; a row's next U pieces of 512 bytes are in flight in registers, the first of them before
// the wait for the kernel before.  Bound by reading w, with eight rows by the chain of a block's segments: 8,192 x 1,024 (columns, K) takes 5.6 / 8.3 / 11.4 us
// for 1 / 3 / 8 rows (5.2 of bytes; the tiles alone: 98 us for any), 1,024 x 4,096 4.8 / 8.7 / 16.2 us (382).
constexpr int GF_WARPS = 8, GF_SEG = 1024;

// a lane's piece of a row of w (zeros beyond K)
template <bool V8>
__device__ inline void gf_load_w(const float* p, int k, int K, unsigned long long (&v)[4]) {
  if constexpr (V8) {
    if (k < K) {
      asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3]) : "l"(p + k));
    } else {
      v[0] = v[1] = v[2] = v[3] = 0;
    }
  } else {
    const ulonglong2 z = make_ulonglong2(0, 0);
    const ulonglong2 a = k < K ? *reinterpret_cast<const ulonglong2*>(p + k) : z;
    const ulonglong2 b = k + 4 < K ? *reinterpret_cast<const ulonglong2*>(p + k + 4) : z;
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
}

template <int MR, int R, int U, bool V8>
__global__ void __launch_bounds__(GF_WARPS * 32)
gemm_simt_few_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                     float* __restrict__ y, int M, int N, int K) {
  constexpr int STEP = GS_LANES * GS_PIECE;                   // features of a warp's step
  constexpr int STEPS = GF_SEG / STEP;                        // of a segment of x
  static_assert(STEPS % U == 0, "the register ring starts a segment at its start");
  extern __shared__ __align__(16) float gf_smem[];            // [2][MR][STEPS][2 planes][16 lanes][4]; later the lanes' sums
  const int tid32 = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lane = tid32 & (GS_LANES - 1), half = tid32 / GS_LANES;
  const int m0 = blockIdx.y * MR;
  const int w0 = (blockIdx.x * GF_WARPS + warp) * 2 * R, n0 = w0 + half * R;   // the warp's first row of w, and this half's
  const float* wr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) wr[r] = w + (int64_t)min(n0 + r, N - 1) * K;    // rows beyond N repeat the last one

  unsigned long long wv[U][R][4];
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int r = 0; r < R; ++r) gf_load_w<V8>(wr[r], u * STEP + lane * GS_PIECE, K, wv[u][r]);
  pdl_wait();
  pdl_trigger();

  const int segs = (K + GF_SEG - 1) / GF_SEG;
  auto fetch = [&](int seg) {
    if (seg < segs) {
      float* to = gf_smem + (seg & 1) * MR * GF_SEG;
      for (int i = threadIdx.x; i < MR * (GF_SEG / 4); i += GF_WARPS * 32) {
        const int m = i / (GF_SEG / 4), f = i % (GF_SEG / 4);          // f: 16 bytes of the segment
        const int k = seg * GF_SEG + f * 4;
        const bool ok = m0 + m < M && k < K;
        gs_cp16(to + m * GF_SEG + (f / (2 * GS_LANES)) * STEP + (f & 1) * (STEP / 2) + ((f / 2) % GS_LANES) * 4,
                x + (ok ? (int64_t)(m0 + m) * K + k : 0), ok);
      }
    }
    gs_commit();
  };
  unsigned long long acc[R][MR];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m < MR; ++m) acc[r][m] = 0;
  fetch(0);
  for (int seg = 0; seg < segs; ++seg) {
    fetch(seg + 1);
    gs_wait<1>();
    __syncthreads();
    const float* xs = gf_smem + (seg & 1) * MR * GF_SEG + lane * 4;
#pragma unroll
    for (int s = 0; s < STEPS; ++s) {
      unsigned long long cur[R][4];
      const int k = seg * GF_SEG + s * STEP + lane * GS_PIECE;
#pragma unroll
      for (int r = 0; r < R; ++r) {
#pragma unroll
        for (int e = 0; e < 4; ++e) cur[r][e] = wv[s % U][r][e];
        gf_load_w<V8>(wr[r], k + U * STEP, K, wv[s % U][r]);
      }
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(xs + m * GF_SEG + s * STEP);
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(xs + m * GF_SEG + s * STEP + STEP / 2);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          gs_fma2(acc[r][m], a.x, cur[r][0]);
          gs_fma2(acc[r][m], a.y, cur[r][1]);
          gs_fma2(acc[r][m], b.x, cur[r][2]);
          gs_fma2(acc[r][m], b.y, cur[r][3]);
        }
      }
    }
    __syncthreads();                                          // the segment has been read
  }
  gs_wait<0>();
  // a thread per output adds its lanes in the order above
  constexpr int OUTS = 2 * R * MR, PITCH = GS_LANES + 1;
  float* part = gf_smem + warp * OUTS * PITCH;
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m < MR; ++m) part[((half * R + r) * MR + m) * PITCH + lane] = gs_both(acc[r][m]);
  __syncwarp();
  for (int o = tid32; o < OUTS; o += 32) {
    const int n = w0 + o / MR, m = m0 + o % MR;
    if (n >= N || m >= M) continue;
    const float* p = part + o * PITCH;
    float v = 0.0f;
#pragma unroll
    for (int g = 0; g < GS_GROUPS; ++g) {
      float s = 0.0f;
#pragma unroll
      for (int l = 0; l < GS_GROUP_LANES; ++l) s += p[g * GS_GROUP_LANES + l];
      v = g == 0 ? s : v + s;
    }
    if (bias) v += bias[n];
    y[(int64_t)m * N + n] = v;
  }
}

static int gs_sm_count() {
  static thread_local int dev_of = -1, count = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev != dev_of) {
    cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
    dev_of = dev;
  }
  return count;
}

template <typename Kern>
static int gs_allow_smem(Kern kernel, size_t smem) {
  if (smem <= 48 * 1024) return 0;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) {
    set_error("gemm_simt: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(e));
    return (int)e;
  }
  return 0;
}

// The three kernels give the same bits, so a call takes the one that models of their times, fitted to 1,304 sizes (K of 4 to 4,096, 8
// to 32,000 columns, 1 to 2,000 rows), call the fastest.  In us, streamed / tiles of four groups / of one: 300 rows x 1,024 columns,
// K 4,096: 110 / 131 / 200; 300 x 8,192, K 64: 160 / 27 / 20; 8 x 8,192, K 64: 10 / 6.5 / 6.9; 2,000 x 8,192, K 64: - / 142 / 88,
// K 1,024: - / 976 / 928.

// Tiles: with four groups of lanes a wave is one tile an SM; with one group up to four tiles an SM share what one of them would
// have alone (whole waves after one another, or the last one by how many an SM gets).
static double gs_tiles_us(int M, int N, int K, bool vec, int split) {
  const double tiles = (double)ceil_div(M, GT_TILE) * ceil_div(N, GT_TILE), sms = gs_sm_count();
  if (split > 1)
    return 1.0 + ceil(tiles / sms) * (vec ? std::min(2.0 + 0.047 * K, 3.5 + 0.0305 * K) : std::min(2.6 + 0.085 * K, 4.6 + 0.039 * K));
  const double full = vec ? 2.6 + 0.127 * K : std::min(2.5 + 0.19 * K, 8.9 + 0.1465 * K);
  const double alone = vec ? std::min(1.9 + 0.075 * K, 5.4 + 0.048 * K) : std::min(2.4 + 0.0945 * K, 6.0 + 0.067 * K);
  const double start = vec ? std::min(4.4, 0.6 + 0.06 * K) : 2.5, waves = floor(tiles / (4 * sms));
  const int an_sm = (int)ceil((tiles - waves * 4 * sms) / sms);
  return waves * full + (an_sm == 0 ? 0.0 : std::max(alone, an_sm == 1 ? 0.0 : (0.1 + 0.25 * an_sm) * full + start));
}

template <typename TI, typename TO, bool VEC, int SPLIT>
static int launch_tiles(const void* x, const void* w, const void* bias, void* y, int M, int N, int K, cudaStream_t stream) {
  const dim3 grid(ceil_div(N, GT_TILE), ceil_div(M, GT_TILE));
  if (grid.y > 65535) { set_error("gemm_simt: M=%d is too large", M); return ERR_UNSUPPORTED; }
  auto kernel = gemm_simt_kernel<TI, TO, VEC, SPLIT>;
  int rc = gs_allow_smem(kernel, gt_smem<SPLIT>());
  if (rc) return rc;
  launch_pdl(kernel, grid, dim3(SPLIT * GT_GROUP), gt_smem<SPLIT>(), stream, static_cast<const TI*>(x),
             static_cast<const TI*>(w), static_cast<const TI*>(bias), static_cast<TO*>(y), M, N, K);
  return launch_status("gemm_simt");
}

template <typename TI, typename TO, bool VEC>
static int launch(const void* x, const void* w, const void* bias, void* y, int M, int N, int K, cudaStream_t stream) {
  return gs_tiles_us(M, N, K, VEC, 1) < gs_tiles_us(M, N, K, VEC, GS_GROUPS)
             ? launch_tiles<TI, TO, VEC, 1>(x, w, bias, y, M, N, K, stream)
             : launch_tiles<TI, TO, VEC, GS_GROUPS>(x, w, bias, y, M, N, K, stream);
}

template <int MR, int R, int U, bool V8>
static int launch_few(const float* x, const float* w, const float* bias, float* y, int M, int N, int K,
                      cudaStream_t stream) {
  const size_t ring = (size_t)2 * MR * GF_SEG * 4, parts = (size_t)GF_WARPS * 2 * R * MR * (GS_LANES + 1) * 4;
  const size_t smem = ring > parts ? ring : parts;
  int rc = gs_allow_smem(gemm_simt_few_kernel<MR, R, U, V8>, smem);
  if (rc) return rc;
  const dim3 grid(ceil_div(N, GF_WARPS * 2 * R), ceil_div(M, MR));
  launch_pdl(gemm_simt_few_kernel<MR, R, U, V8>, grid, dim3(GF_WARPS * 32), smem, stream, x, w, bias, y, M, N, K);
  return launch_status("gemm_simt_few");
}

// Rows of w a half warp: as many as leave every SM eight warps, so that the reads of x are shared.
static int gs_few_w_rows(int M, int N, int MR) {
  const int rows_an_sm = N / gs_sm_count() * ceil_div(M, MR);
  return rows_an_sm >= 64 ? 4 : rows_an_sm >= 32 ? 2 : 1;
}
static int gs_few_x_rows(int M) { return M <= 2 ? M : M <= 4 ? 4 : 8; }

template <int MR, bool V8>
static int launch_few_rows(const float* x, const float* w, const float* bias, float* y, int M, int N, int K,
                           cudaStream_t stream) {
  switch (gs_few_w_rows(M, N, MR)) {
    case 4: return launch_few<MR, 4, 2, V8>(x, w, bias, y, M, N, K, stream);
    case 2: return launch_few<MR, 2, 4, V8>(x, w, bias, y, M, N, K, stream);
    default: return launch_few<MR, 1, 8, V8>(x, w, bias, y, M, N, K, stream);
  }
}

// The streaming kernel: a lane's chain over K, or by pairs of a row of w and up to eight of x.
static double gs_few_us(int M, int N, int K) {
  const int MR = gs_few_x_rows(M);
  if (MR < 8) return std::max(1.7 + 0.0007 * sqrt((double)MR) * K, 2.0 + (0.1 * MR + 0.0006 * K) * 1e-3 * N);
  const double pairs = (double)ceil_div(M, 8) * N, rows_an_sm = pairs / gs_sm_count();
  const double spread = rows_an_sm >= 128 ? 1.0 : rows_an_sm >= 64 ? 1.6 : rows_an_sm >= 32 || pairs > 8000 ? 1.8 : 2.8;
  // a pair: whole segments of K, and every eight rows read w again, from L2 while it fits there
  const double pair = K < GF_SEG ? 0.5 + 0.00012 * K : 0.1 + ((double)N * K > 2.5e7 ? 0.00073 : 0.00053) * GF_SEG * ceil_div(K, GF_SEG);
  return std::max(std::max(4.6, 1.6 + 0.0035 * K), 2.0 + pair * 1e-3 * spread * pairs);
}

}  // namespace exl3

using namespace exl3;

extern "C" int exl3_gemm_simt(const void* x, const void* w, const void* bias, void* y, int in_dtype,
                              int out_dtype, int M, int N, int K, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  if (M < 0 || N < 0 || K < 1) { set_error("gemm_simt: bad sizes M=%d N=%d K=%d", M, N, K); return ERR_BAD_ARGUMENT; }
  if (in_dtype == DT_F32 && out_dtype == DT_F32) {
    if (K % 4 != 0 || !aligned16(x) || !aligned16(w)) return launch<float, float, false>(x, w, bias, y, M, N, K, stream);
    if (M > 65535 || gs_few_us(M, N, K) > std::min(gs_tiles_us(M, N, K, true, 1), gs_tiles_us(M, N, K, true, GS_GROUPS)))
      return launch<float, float, true>(x, w, bias, y, M, N, K, stream);
    const float *xf = static_cast<const float*>(x), *wf = static_cast<const float*>(w), *bf = static_cast<const float*>(bias);
    float* yf = static_cast<float*>(y);
    const bool v8 = K % 8 == 0 && (reinterpret_cast<uintptr_t>(w) & 31u) == 0;
    if (M == 1)
      return v8 ? launch_few_rows<1, true>(xf, wf, bf, yf, M, N, K, stream) : launch_few_rows<1, false>(xf, wf, bf, yf, M, N, K, stream);
    if (M == 2)
      return v8 ? launch_few_rows<2, true>(xf, wf, bf, yf, M, N, K, stream) : launch_few_rows<2, false>(xf, wf, bf, yf, M, N, K, stream);
    if (M <= 4)
      return v8 ? launch_few_rows<4, true>(xf, wf, bf, yf, M, N, K, stream) : launch_few_rows<4, false>(xf, wf, bf, yf, M, N, K, stream);
    return v8 ? launch_few_rows<8, true>(xf, wf, bf, yf, M, N, K, stream) : launch_few_rows<8, false>(xf, wf, bf, yf, M, N, K, stream);
  }
  if (in_dtype == DT_BF16 && out_dtype == DT_BF16)
    return launch<__nv_bfloat16, __nv_bfloat16, false>(x, w, bias, y, M, N, K, stream);
  if (in_dtype == DT_BF16 && out_dtype == DT_F32)
    return launch<__nv_bfloat16, float, false>(x, w, bias, y, M, N, K, stream);
  set_error("gemm_simt: unsupported element types in=%d out=%d", in_dtype, out_dtype);
  return ERR_UNSUPPORTED;
}

// y[M, N] = x[M, K] . w[N, K]^T (+ bias) in float32 for a handful of output features and many rows (a few gates or
// scores per token): a warp a row of x, the lanes striding K in 16-byte pieces, four output features at a time over
// the same pieces of x; the row of x and the few rows of w stay in L1 and L2.  One order of summation per (row,
// feature), whatever M.
namespace exl3 {

constexpr int FEW_WARPS = 8;

template <typename T>
__global__ void __launch_bounds__(FEW_WARPS * 32)
gemm_few_out_kernel(const T* __restrict__ x, int64_t ldx, const T* __restrict__ w, const T* __restrict__ bias,
                    float* __restrict__ y, int M, int N, int K) {
  constexpr int VEC = Elem<T>::vec;
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int m = blockIdx.x * FEW_WARPS + (threadIdx.x >> 5);
  if (m >= M) return;
  const T* xr = x + (int64_t)m * ldx;
  const int pieces = K / VEC;
  for (int n0 = 0; n0 < N; n0 += 4) {
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int p = lane; p < pieces; p += 32) {
      float xv[VEC];
      load_vec_cg(xr + (int64_t)p * VEC, xv);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (n0 + u < N) {
          float wv[VEC];
          load_vec(w + (int64_t)(n0 + u) * K + (int64_t)p * VEC, wv);
#pragma unroll
          for (int e = 0; e < VEC; ++e) acc[u] = fmaf(xv[e], wv[e], acc[u]);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float v = warp_sum(acc[u]);
      if (lane == 0 && n0 + u < N) y[(int64_t)m * N + n0 + u] = v + (bias ? Elem<T>::load(bias + n0 + u) : 0.0f);
    }
  }
}

}  // namespace exl3

extern "C" int exl3_gemm_few_out(const void* x, int64_t ldx, const void* w, const void* bias, float* y, int in_dtype,
                                 int M, int N, int K, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  const int vec = in_dtype == DT_F32 ? 4 : 8;
  if (M < 0 || N < 0 || K < 1 || (in_dtype != DT_F32 && in_dtype != DT_BF16) || K % vec != 0 || ldx % vec != 0 ||
      !aligned16(x) || !aligned16(w)) {
    set_error("gemm_few_out: needs float32 or bfloat16 inputs, K and the pitch of x in 16-byte pieces, got M=%d N=%d K=%d", M,
              N, K);
    return ERR_BAD_ARGUMENT;
  }
  const dim3 grid(ceil_div(M, FEW_WARPS));
  if (in_dtype == DT_F32)
    launch_pdl(gemm_few_out_kernel<float>, grid, dim3(FEW_WARPS * 32), 0, stream, static_cast<const float*>(x), ldx,
               static_cast<const float*>(w), static_cast<const float*>(bias), y, M, N, K);
  else
    launch_pdl(gemm_few_out_kernel<__nv_bfloat16>, grid, dim3(FEW_WARPS * 32), 0, stream,
               static_cast<const __nv_bfloat16*>(x), ldx, static_cast<const __nv_bfloat16*>(w),
               static_cast<const __nv_bfloat16*>(bias), y, M, N, K);
  return launch_status("gemm_few_out");
}
