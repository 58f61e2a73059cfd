// Sampling with filters on the device: the reference's sampler (sample_token,
// src/model.cpp:667-757) step for step.
//
//   penalties over the context, then
//   the 2048 largest logits in descending order (ties: the smaller index first),
//   p[i] = exp(logit[i] / T - max) as float32, sums in float64,
//   min-p: cut before the first candidate whose share is below min_p * the largest share,
//   top-k: at most k candidates,
//   top-p: cut after the first candidate at which the running share reaches top_p,
//   and the token at which the running sum of what is kept reaches u * its total.
//
// Only the chosen ids cross to the host; with the sampler on the host a step
// carries the whole rows there (vocabulary x 4 bytes each) and sorts them.
//
// The candidates are found without sorting the vocabulary: a radix select over
// the float bits (digits of 11, 11 and 10 bits) gives the 2048th largest value;
// when several tokens share that value the select goes on over their indices, so
// exactly 2048 tokens pass.  They are sorted (bitonic, 64-bit keys: value bits
// above, inverted index below, all different).
//
// A row is the work of a cluster of up to eight blocks.  Each reads its part of
// the row once, with the penalties applied on the way, and keeps the keys in
// shared memory, where the passes of the select find them (the first pass's
// histogram is taken while the row is read); a pass's histograms
// meet through distributed shared memory (every block adds all of them up and
// finds the same digit), and the passing keys are dealt out to the blocks in equal
// shares.  Each sorts its share, every block reads all the shares, and a key's place
// among all of them goes with it into the first block, which draws.  Bound by the chain of
// passes and barriers (of 42 us with one block sorting: the row 4.4, three passes 5 to 6 each,
// the collection 4.4, the sort of 2,048 13.6, the draw 4): 32 rows of 122,753 take 34 us, one row 31.
// (One block a row that reads it five times: 105 us, and the penalties were a copy of the logits and a kernel of 16 us.)
#include "api.h"
#include "common.cuh"

#include <math.h>
#include <string.h>

#include <algorithm>

namespace exl3 {

constexpr int SF_THREADS = 1024;
constexpr int SF_CAP = 2048;                     // candidates: max(top_k, 2048) in the reference; top_k above it is refused here

// float bits -> unsigned keys in the floats' order
__device__ inline uint32_t sf_key(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ inline float sf_value(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct SfRow {            // one row's options, as the host gives them (float64 [R, 5])
  double temperature, top_k, top_p, min_p, u;
};

// The options of a call's rows.  Up to so many rows come as a parameter of the kernel: no buffer to make and to copy (some
// 25 us of the host's time a call).
constexpr int SF_DIRECT_ROWS = 64;
struct SfBatch {
  SfRow rows[SF_DIRECT_ROWS];
  int* counts_of[SF_DIRECT_ROWS];
  float params_of[SF_DIRECT_ROWS][3];
  __device__ SfRow row(int r) const { return rows[r]; }
  __device__ const int* counts(int r) const { return counts_of[r]; }
  __device__ const float* params(int r) const { return params_of[r]; }
};
// Or they lie in buffers on the device.  (A type of its own: 4 KB of parameters that nobody reads cost a launch 1 us.)
struct SfTables {
  const SfRow* rows;
  int* const* counts_of;                         // null: no row has penalties
  const float* params_of;
  __device__ SfRow row(int r) const { return rows[r]; }
  __device__ const int* counts(int r) const { return counts_of ? counts_of[r] : nullptr; }
  __device__ const float* params(int r) const { return params_of + 3 * r; }
};

// the model of a launch's time (sf_launch): a wave of rows with 8 / 4 / 2 / 1 blocks a row, and a token of a block's part
constexpr double SF_FIXED_US[4] = {26.5, 23.0, 24.5, 28.0}, SF_AGAIN_FIXED_US = 6.0;
constexpr double SF_STAGED_US = 0.00032, SF_AGAIN_US = 0.00033, SF_AGAIN_PENALTIES_US = 0.00066, SF_AGAIN_FAR_US = 0.00075, SF_PENALTIES_US = 2.1;
constexpr double SF_NEAR_BYTES = 100e6;          // logits and counts of the rows under way that L2 holds
constexpr int SF_BINS = 2048;
constexpr int SF_BLOCKS = 8;                     // of a row, at most
constexpr int SF_HEAD_BYTES = (2 * SF_BINS * 4) + 2 * (SF_CAP * 8);     // histograms, candidates, this block's own
constexpr int SF_SMEM_MOST = 200 * 1024;                                // with the staged part of a row

__device__ inline uint32_t sf_remote(const void* mine, uint32_t rank) {
  uint32_t addr;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(rank));
  return addr;
}
__device__ inline void sf_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ inline unsigned long long sf_max(unsigned long long a, unsigned long long b) { return a > b ? a : b; }
__device__ inline unsigned long long sf_min(unsigned long long a, unsigned long long b) { return a < b ? a : b; }

// A logit with its token's penalties (src/model.cpp:672-686).
__device__ inline float sf_penalised(float x, int count, float rep, float presence, float frequency) {
  if (count <= 0) return x;
  if (rep != 1.0f) x = x > 0.0f ? __fdiv_rn(x, rep) : __fmul_rn(x, rep);
  if (presence != 0.0f) x = __fsub_rn(x, presence);
  if (frequency != 0.0f) x = __fsub_rn(x, __fmul_rn(frequency, (float)count));
  return x;
}

// of_rows: the rows' options, per row a pointer to its token counts [V] (null: the row has no penalties) and three numbers:
// repetition, presence, frequency.  host_out: null, or a page-locked copy of out.  count_now: no two rows share their counts,
// so a row's token joins them at once; else they are only read, and the chosen tokens join them in a kernel of their own, after
// every row has been drawn (2 us for 32 rows).  STAGED: the block's part of the row is kept in shared memory;
// else (parts too long for that) every pass reads it again, 16 bytes a load: one block a row takes 76 us for 122,753
// tokens (4 bytes a load, and 64-bit keys compared in every pass: 107), 142 for 320,001.  PENALTIES: there may be counts.
template <bool STAGED, bool PENALTIES, typename ROWS>
__global__ void __launch_bounds__(SF_THREADS)
sample_filtered_kernel(const float* __restrict__ logits, const __grid_constant__ ROWS of_rows, int* __restrict__ out, int V,
                       int blocks, int* host_out, bool count_now) {
  extern __shared__ __align__(16) unsigned char sf_smem[];
  unsigned* hists = reinterpret_cast<unsigned*>(sf_smem);                                      // [2][SF_BINS]
  unsigned long long* cand = reinterpret_cast<unsigned long long*>(sf_smem + 2 * SF_BINS * 4);  // this block's share of them
  unsigned long long* found = cand + SF_CAP;                                                   // those of this block's tokens
  uint32_t* keys = reinterpret_cast<uint32_t*>(sf_smem + SF_HEAD_BYTES);                       // this block's part of the row
  float* probs = reinterpret_cast<float*>(found);            // and once the block's own candidates are
  __shared__ double warp_tot[SF_THREADS / 32];
  __shared__ unsigned warp_cnt[SF_THREADS / 32];
  __shared__ unsigned sel_digit, sel_remaining, sel_same, n_cand, n_found, at_cand;
  __shared__ int first_below, first_hit, first_draw;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row_id = blockIdx.x / blocks, rank = blockIdx.x % blocks;
  const float* row = logits + (int64_t)row_id * V;
  const SfRow o = of_rows.row(row_id);
  const int M = V < SF_CAP ? V : SF_CAP;
  const int* count = PENALTIES ? of_rows.counts(row_id) : nullptr;
  float rep = 1.0f, presence = 0.0f, frequency = 0.0f;
  if (count) {
    const float* params = of_rows.params(row_id);
    rep = params[0];
    presence = params[1];
    frequency = params[2];
  }
  // the row's token, from the thread that knows it; all of the row's blocks have read its counts by then
  auto chosen = [&](int t) {
    out[row_id] = t;
    if (host_out) host_out[row_id] = t;
    if (count && count_now && t >= 0 && t < V) atomicAdd(const_cast<int*>(count) + t, 1);
  };
  const int slots = SF_CAP / blocks;             // a block's share of the candidates (blocks is a power of two)
  const int per = (V + blocks - 1) / blocks;
  const int first = min(V, rank * per), n = min(V, first + per) - first;
  // f(value's key, place in the row) for every token of this block's part
  auto for_each = [&](auto&& f) {
    if constexpr (STAGED) {
      const uint4* keys4 = reinterpret_cast<const uint4*>(keys);
#pragma unroll 2
      for (int j = tid; j < n / 4; j += SF_THREADS) {
        const uint4 k = keys4[j];
        const int i = first + 4 * j;
        f(k.x, i);
        f(k.y, i + 1);
        f(k.z, i + 2);
        f(k.w, i + 3);
      }
      for (int i = n / 4 * 4 + tid; i < n; i += SF_THREADS) f(keys[i], first + i);
    } else {
      // 16-byte loads, four of a thread on their way, with penalties two and as many of the counts (parts start at any
      // multiple of 4 bytes: the pieces before and after the aligned part go one by one)
      constexpr int AHEAD = PENALTIES ? 2 : 4;
      const float* part = row + first;
      auto key_of = [&](float x, int c) {
        if constexpr (PENALTIES) return sf_key(sf_penalised(x, c, rep, presence, frequency));
        else return sf_key(x);
      };
      auto counted = [&](int i) { return PENALTIES && count ? count[first + i] : 0; };
      const int head = min(n, (int)((4 - ((reinterpret_cast<uintptr_t>(part) >> 2) & 3)) & 3)), n_vec = (n - head) / 4;
      const float4* part4 = reinterpret_cast<const float4*>(part + head);
      auto one = [&](int i) { f(key_of(part[i], counted(i)), first + i); };
      if (tid < head) one(tid);
#pragma unroll 1
      for (int j0 = tid; j0 < n_vec; j0 += SF_THREADS * AHEAD) {
        float4 x[AHEAD];
        int c[AHEAD][4];
#pragma unroll
        for (int a = 0; a < AHEAD; ++a) {
          const int j = j0 + a * SF_THREADS;
          if (j < n_vec) {
            x[a] = part4[j];
#pragma unroll
            for (int e = 0; e < 4; ++e) c[a][e] = counted(head + 4 * j + e);
          }
        }
#pragma unroll
        for (int a = 0; a < AHEAD; ++a) {
          const int j = j0 + a * SF_THREADS, i = first + head + 4 * j;
          if (j < n_vec) {
            f(key_of(x[a].x, c[a][0]), i);
            f(key_of(x[a].y, c[a][1]), i + 1);
            f(key_of(x[a].z, c[a][2]), i + 2);
            f(key_of(x[a].w, c[a][3]), i + 3);
          }
        }
      }
      for (int i = head + 4 * n_vec + tid; i < n; i += SF_THREADS) one(i);
    }
  };
  for (int b = tid; b < SF_BINS; b += SF_THREADS) hists[b] = 0;
  for (int i = tid; i < slots; i += SF_THREADS) cand[i] = 0ull;         // padding sorts last
  if (tid == 0) n_cand = n_found = 0;
  __syncthreads();
  if constexpr (STAGED) {
    // the select's first histogram on the way, where there is a select
    constexpr int AHEAD = 8;
    for (int i0 = tid; i0 < n; i0 += SF_THREADS * AHEAD) {
      float x[AHEAD];
      int c[AHEAD];
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) {
        const int i = i0 + a * SF_THREADS;
        x[a] = i < n ? row[first + i] : 0.0f;
        c[a] = i < n && count ? count[first + i] : 0;
      }
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) {
        const int i = i0 + a * SF_THREADS;
        if (i < n) {
          const uint32_t key = sf_key(sf_penalised(x[a], c[a], rep, presence, frequency));
          keys[i] = key;
          if (V > SF_CAP) atomicAdd(hists + (key >> 21), 1u);
        }
      }
    }
    __syncthreads();
  }

  // ---- the M largest (value, then smaller index): radix select on the composite key -------------
  unsigned long long thresh = 0;                 // everything passes when the row is no longer than the cap
  if (V > SF_CAP) {
    unsigned remaining = (unsigned)M;
    // the value's three digits; the index's three only when tokens with the threshold's value are too many
    for (int pass = 0; pass < 6; ++pass) {
      const int at[6] = {53, 42, 32, 21, 10, 0}, wide[6] = {11, 11, 10, 11, 11, 10};
      const int shift = at[pass], bits = wide[pass];
      unsigned* hist = hists + (pass & 1) * SF_BINS;
      if (pass > 0) {
        // nobody reads this one any more: the blocks have met since
        for (int b = tid; b < SF_BINS; b += SF_THREADS) hist[b] = 0;
        __syncthreads();
      }
      const unsigned digit_mask = (1u << bits) - 1u;
      const uint32_t want = (uint32_t)(thresh >> 32);
      if (STAGED && pass == 0) {
        // taken above
      } else if (pass < 3) {
        const uint32_t mask = pass == 0 ? 0u : ~0u << (shift - 32 + bits);
        for_each([&](uint32_t key, int) {
          if (((key ^ want) & mask) == 0) atomicAdd(hist + ((key >> (shift - 32)) & digit_mask), 1u);
        });
      } else {
        const uint32_t mask = pass == 3 ? 0u : ~0u << (shift + bits), low = (uint32_t)thresh;
        for_each([&](uint32_t key, int i) {
          if (key == want && ((~(uint32_t)i ^ low) & mask) == 0) atomicAdd(hist + ((~(uint32_t)i >> shift) & digit_mask), 1u);
        });
      }
      sf_cluster_sync();
      // all blocks' histograms, from the largest digit down, two bins a thread
      const int hi = SF_BINS - 1 - 2 * tid;
      unsigned n1 = 0, n0 = 0;                    // bins hi and hi - 1
      {
        unsigned lo_bin[SF_BLOCKS], hi_bin[SF_BLOCKS];      // all asked for before the first is added
#pragma unroll
        for (int b = 0; b < SF_BLOCKS; ++b) {
          lo_bin[b] = hi_bin[b] = 0;
          if (b < blocks)
            asm volatile("ld.shared::cluster.v2.u32 {%0, %1}, [%2];" : "=r"(lo_bin[b]), "=r"(hi_bin[b]) : "r"(sf_remote(hist + hi - 1, b)));
        }
#pragma unroll
        for (int b = 0; b < SF_BLOCKS; ++b) { n1 += hi_bin[b]; n0 += lo_bin[b]; }
      }
      unsigned run = n1 + n0;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, run, s);
        if (lane >= s) run += v;
      }
      if (lane == 31) warp_cnt[warp] = run;
      __syncthreads();
      const unsigned before = run - (n1 + n0) + __reduce_add_sync(0xffffffffu, lane < warp ? warp_cnt[lane] : 0u);
      if (before < remaining && before + n1 >= remaining) {
        sel_digit = hi;
        sel_remaining = remaining - before;      // how many of this digit's tokens still pass
        sel_same = n1;
      } else if (before + n1 < remaining && before + n1 + n0 >= remaining) {
        sel_digit = hi - 1;
        sel_remaining = remaining - before - n1;
        sel_same = n0;
      }
      __syncthreads();
      remaining = sel_remaining;
      thresh |= (unsigned long long)sel_digit << shift;
      // if all tokens with this value pass, their indices need no select: the threshold is (value, any index)
      if (shift == 32 && sel_same == remaining) break;
      __syncthreads();                            // before the next pass's sums
    }
  }
  const uint32_t least = (uint32_t)(thresh >> 32);
  for_each([&](uint32_t key, int i) {
    if (key >= least) {
      const unsigned long long c = ((unsigned long long)key << 32) | ~(uint32_t)i;
      if (c >= thresh) {
        const unsigned k = atomicAdd(&n_found, 1u);
        if (k < (unsigned)SF_CAP) found[k] = c;
      }
    }
  });
  if (V <= SF_CAP) sf_cluster_sync();             // the first block's candidates are cleared (else the select has met)
  __syncthreads();
  if (tid == 0)
    asm volatile("atom.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(at_cand) : "r"(sf_remote(&n_cand, 0)), "r"(n_found) : "memory");
  __syncthreads();
  for (unsigned i = tid; i < n_found; i += SF_THREADS) {
    const unsigned at = at_cand + i;               // equal shares for the blocks
    if (at < (unsigned)SF_CAP)
      asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(sf_remote(cand + (at & (slots - 1)), at / slots)), "l"(found[i]) : "memory");
  }
  sf_cluster_sync();                              // all candidates are there

  // ---- sorted descending: each block its share, bitonic, two neighbours a thread: partners up to 32 places away are in
  // the same warp, only the farther ones go through shared memory.  Then a candidate's place among all of them is the
  // sum of its places in the blocks' shares: with four blocks 7 us, one block sorting all of them 13.6 --------------
  {
    const bool mine = 2 * tid < slots;            // whole warps: a share is 256 slots or more
    unsigned long long a = mine ? cand[2 * tid] : 0ull, b = mine ? cand[2 * tid + 1] : 0ull;
    for (int k = 2; k <= slots; k <<= 1) {
      const bool desc = ((2 * tid) & k) == 0;     // the same for both places: k >= 2
      for (int j = k >> 1; j >= 64; j >>= 1) {
        __syncthreads();
        if (mine) {
          cand[2 * tid] = a;
          cand[2 * tid + 1] = b;
        }
        __syncthreads();
        if (mine) {
          const unsigned long long pa = cand[(2 * tid) ^ j], pb = cand[(2 * tid + 1) ^ j];
          const bool larger = desc == (((2 * tid) & j) == 0);
          a = larger ? sf_max(a, pa) : sf_min(a, pa);
          b = larger ? sf_max(b, pb) : sf_min(b, pb);
        }
      }
      if (mine) {
        for (int j = min(k >> 1, 32); j >= 2; j >>= 1) {
          const unsigned long long pa = __shfl_xor_sync(0xffffffffu, a, j >> 1), pb = __shfl_xor_sync(0xffffffffu, b, j >> 1);
          const bool larger = desc == (((2 * tid) & j) == 0);
          a = larger ? sf_max(a, pa) : sf_min(a, pa);
          b = larger ? sf_max(b, pb) : sf_min(b, pb);
        }
        const unsigned long long top = sf_max(a, b), low = sf_min(a, b);
        a = desc ? top : low;
        b = desc ? low : top;
      }
    }
    __syncthreads();
    if (mine) {
      cand[2 * tid] = a;
      cand[2 * tid + 1] = b;
    }
    __syncthreads();
  }
  unsigned long long* sorted = cand;
  double* acc = reinterpret_cast<double*>(sf_smem);            // running sums of probs: the histograms' place
  if (blocks > 1) {
    sf_cluster_sync();                            // every share is sorted
    // all shares side by side in `found`
    for (int i = tid; i < SF_CAP; i += SF_THREADS) {
      unsigned long long c;
      asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(c) : "r"(sf_remote(cand + (i & (slots - 1)), i / slots)));
      found[i] = c;
    }
    unsigned* places = reinterpret_cast<unsigned*>(cand + slots);      // (a share is half of cand at most)
    if (tid < slots) places[tid] = 0;
    __syncthreads();
    // SF_THREADS / slots = blocks / 2 groups of threads, a group two of the shares
    const int e = tid & (slots - 1), group = tid / slots, groups = blocks >> 1;
    const unsigned long long c = cand[e];
    const unsigned long long *s0 = found + group * slots, *s1 = found + (group + groups) * slots;
    int p0 = 0, p1 = 0;                           // how many of a share are larger
    for (int step = slots >> 1; step > 0; step >>= 1) {
      if (s0[p0 + step - 1] > c) p0 += step;
      if (s1[p1 + step - 1] > c) p1 += step;
    }
    if (s0[p0] > c) ++p0;
    if (s1[p1] > c) ++p1;
    atomicAdd(places + e, (unsigned)(p0 + p1));
    __syncthreads();
    sorted = reinterpret_cast<unsigned long long*>(sf_smem);   // the first block's histograms' place: nobody reads those any more
    acc = reinterpret_cast<double*>(cand);
    if (tid < slots && c != 0ull)                 // (padding has no place: nobody looks at it)
      asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(sf_remote(sorted + places[e], 0)), "l"(c) : "memory");
    sf_cluster_sync();                            // and nobody reads another block any more
    if (rank != 0) return;
  }
  auto token_of = [&](int i) { return (int)(~(unsigned)(sorted[i] & 0xffffffffull)); };
  if (!(o.temperature > 0.0)) {                  // greedy: the first maximum
    if (tid == 0) chosen(token_of(0));
    return;
  }

  // ---- probabilities as the reference rounds them, their running sums in float64 ------------------
  const float inv_t = __fdiv_rn(1.0f, (float)o.temperature);
  const float maxl = __fmul_rn(sf_value((uint32_t)(sorted[0] >> 32)), inv_t);
  for (int i = tid; i < SF_CAP; i += SF_THREADS)
    probs[i] = i < M ? expf(__fsub_rn(__fmul_rn(sf_value((uint32_t)(sorted[i] >> 32)), inv_t), maxl)) : 0.0f;
  __syncthreads();
  {
    // inclusive scan: two neighbours per thread, then warps, then the warps' totals
    const int i0 = 2 * tid;
    const double a0 = (double)probs[i0], a1 = a0 + (double)probs[i0 + 1];
    double run = a1;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, run, s);
      if ((tid & 31) >= s) run += v;
    }
    if ((tid & 31) == 31) warp_tot[tid >> 5] = run;
    __syncthreads();
    if (tid < 32) {
      double t = warp_tot[tid];
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, t, s);
        if (tid >= s) t += v;
      }
      warp_tot[tid] = t;
    }
    __syncthreads();
    const double before = (tid >> 5) > 0 ? warp_tot[(tid >> 5) - 1] : 0.0;
    acc[i0] = before + (run - a1) + a0;
    acc[i0 + 1] = before + run;
  }
  if (tid == 0) { first_below = M; first_hit = M; first_draw = M; }
  __syncthreads();
  const double total = acc[M - 1];
  if (!(total > 0.0)) {
    if (tid == 0) chosen(token_of(0));
    return;
  }
  int keep = M;
  if (o.min_p > 0.0) {
    const double th = o.min_p * ((double)probs[0] / total);
    for (int i = tid; i < M; i += SF_THREADS)
      if ((double)probs[i] / total < th) atomicMin(&first_below, i);
    __syncthreads();
    keep = first_below < 1 ? 1 : first_below;
  }
  const int top_k = (int)o.top_k;
  if (top_k > 0 && top_k < keep) keep = top_k;
  if (o.top_p < 1.0) {
    for (int i = tid; i < keep; i += SF_THREADS)
      if (acc[i] / total >= o.top_p) atomicMin(&first_hit, i);
    __syncthreads();
    if (first_hit < keep) keep = first_hit + 1;
  }
  const double r = o.u * acc[keep - 1];
  for (int i = tid; i < keep; i += SF_THREADS)
    if (acc[i] >= r) atomicMin(&first_draw, i);
  __syncthreads();
  if (tid == 0) chosen(token_of(first_draw < keep ? first_draw : keep - 1));
}

// Penalties over a row's context (src/model.cpp:672-686).  counts[r] points to the row's token counts [V]
// (how often each token occurs in its context so far), or is null for a row without penalties.
__global__ void sample_penalties_kernel(float* __restrict__ logits, int V, const int* const* __restrict__ counts,
                                        const float* __restrict__ params /* [R, 3]: repetition, presence, frequency */) {
  const int row = blockIdx.y;
  const int* c = counts[row];
  if (c == nullptr) return;
  const int tok = blockIdx.x * blockDim.x + threadIdx.x;
  if (tok >= V) return;
  const int count = c[tok];
  if (count <= 0) return;
  float* x = logits + (int64_t)row * V + tok;
  *x = sf_penalised(*x, count, params[3 * row], params[3 * row + 1], params[3 * row + 2]);
}

// The chosen tokens join their rows' contexts (rows that share their counts may have chosen the same token).
__global__ void sample_count_kernel(int* const* __restrict__ counts, const int* __restrict__ ids, int R, int V) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= R || counts[row] == nullptr) return;
  const int t = ids[row];
  if (t >= 0 && t < V) atomicAdd(counts[row] + t, 1);
}

struct SfCounts { int* at[SF_DIRECT_ROWS]; };
__global__ void sample_count_batch_kernel(const __grid_constant__ SfCounts counts, const int* __restrict__ ids, int R, int V) {
  const int row = threadIdx.x;
  if (row >= R || counts.at[row] == nullptr) return;
  const int t = ids[row];
  if (t >= 0 && t < V) atomicAdd(counts.at[row] + t, 1);
}

}  // namespace exl3

using namespace exl3;

// Clusters of b blocks (2, 4 or 8), a block an SM, that run at once; the GPU's, so asked for once.
static int sf_clusters_at_once(int b, int sms) {
  struct Table { int n[SF_BLOCKS + 1]; };
  static const Table table = [sms] {
    Table t = {};
    auto kernel = sample_filtered_kernel<true, true, SfTables>;
    const bool fine = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SF_SMEM_MOST) == cudaSuccess;
    for (int c = 2; c <= SF_BLOCKS; c *= 2) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(c * sms);
      cfg.blockDim = dim3(SF_THREADS);
      cfg.dynamicSmemBytes = SF_SMEM_MOST;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = c;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      if (!fine || cudaOccupancyMaxActiveClusters(&t.n[c], kernel, &cfg) != cudaSuccess || t.n[c] < 1) t.n[c] = std::max(1, sms / c);
    }
    cudaGetLastError();
    return t;
  }();
  return table.n[b];
}

// rows: float64 [R, 5] on the device: temperature (<= 0: greedy), top_k (0: off, at most 2048), top_p, min_p and
// the row's uniform number in [0, 1).  out: int32 [R].  counts (may be null): as in exl3_sample_penalties, with params;
// the penalties are applied as the logits are read, and the chosen tokens are counted when all rows have been drawn.
template <typename ROWS>
static int sf_launch(const float* logits, const ROWS& of_rows, int* out, int R, int V, bool penalties, int* host_out, bool count_now,
                     cudaStream_t stream) {
  // Blocks a row.  An SM holds one block, and a cluster must fit into a group of SMs, so the driver says how many clusters run
  // at once; a wave of rows takes 23 to 28 us (2 more with penalties) and, for a token of a block's part, 0.32 ns, or where the part is
  // too long for shared memory and read in every pass 6 us and 0.33 ns (with penalties 0.66 where L2 holds the rows under way, else 0.75:
  // 256 rows of 50,257 take one block a row, 133 us, and not two, 144; 75 of 320,001 two, 237, and not one, 266).  With 8 / 4 / 2 / 1 blocks: one row of 32,000
  // 27.8 / 25.7 / 29.6 / 38 us, 64 rows 131 / 52 / 30 / 38; 8 rows of 122,753 31.8 / 33.1 / 49 / 76, 16 rows 60 / 33 / 49 / 76,
  // 148 rows 299 / 157 / 98 / 77; 100 rows of 320,001 289 / 200 / 168 / 163.
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  constexpr size_t MOST = SF_SMEM_MOST - SF_HEAD_BYTES;
  int blocks = 8;
  double best = 0.0;
  for (int b = 8, i = 0; b >= 1; b /= 2, ++i) {
    const int each = ceil_div(V, b);
    const int at_once = b == 1 ? sms : sf_clusters_at_once(b, sms);
    const double waves = (double)((R + at_once - 1) / at_once);
    const bool kept = (size_t)each * 4 <= MOST;
    const bool near = 8.0 * V * std::min(R, at_once) < SF_NEAR_BYTES;
    const double a_token = kept ? SF_STAGED_US : !penalties ? SF_AGAIN_US : near ? SF_AGAIN_PENALTIES_US : SF_AGAIN_FAR_US;
    const double cost = waves * (SF_FIXED_US[i] + (kept ? penalties ? SF_PENALTIES_US : 0.0 : SF_AGAIN_FIXED_US) + a_token * each);
    if (b == 8 || cost < best) {
      best = cost;
      blocks = b;
    }
  }
  const size_t part = (size_t)ceil_div(V, blocks) * 4;
  const bool staged = part <= MOST;
  auto kernel = staged ? sample_filtered_kernel<true, true, ROWS>
                       : penalties ? sample_filtered_kernel<false, true, ROWS> : sample_filtered_kernel<false, false, ROWS>;
  const size_t smem = SF_HEAD_BYTES + (staged ? part : 0);
  // The limit belongs to the function and not to this call: the same number from every thread, whatever its rows take, or a
  // thread with shorter rows would lower it between another one's setting it and its launch.
  const int limit = staged ? SF_SMEM_MOST : SF_HEAD_BYTES;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
  if (e != cudaSuccess) {
    set_error("sample_filtered: %d bytes of shared memory refused: %s", limit, cudaGetErrorString(e));
    return (int)e;
  }
  if ((long long)R * blocks > 0x7fffffffll) { set_error("sample_filtered: %d rows are too many", R); return ERR_UNSUPPORTED; }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(R * blocks);
  cfg.blockDim = dim3(SF_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = blocks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = blocks > 1 ? 1 : 0;               // without a cluster blocks are spread over the SMs first
  cudaLaunchKernelEx(&cfg, kernel, logits, of_rows, out, V, blocks, host_out, count_now);
  return launch_status("sample_filtered");
}

extern "C" int exl3_sample_rows(const float* logits, const double* rows, int* const* counts, const float* params, int* out,
                                int R, int V, cudaStream_t stream) {
  if (R == 0) return 0;
  if (R < 0 || V < 1 || rows == nullptr || (counts != nullptr && params == nullptr)) {
    set_error("sample_filtered: bad sizes rows=%d vocab=%d, or penalties without their constants", R, V);
    return ERR_BAD_ARGUMENT;
  }
  const SfTables tables = {reinterpret_cast<const SfRow*>(rows), counts, params};
  int rc = sf_launch(logits, tables, out, R, V, counts != nullptr, nullptr, false, stream);
  if (rc || counts == nullptr) return rc;
  return exl3_sample_count(counts, out, R, V, stream);
}

extern "C" int exl3_sample_direct_rows() { return SF_DIRECT_ROWS; }

// The reference's generator (src/model.cpp:656-665) behind its step: a state's number in [0, 1).
static double sf_uniform(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

// The same for up to exl3_sample_direct_rows() rows whose options are on the host.  packed: float64 [R, 7] = temperature,
// top_k, top_p, min_p, repetition, presence and frequency penalty; uint64 [R], the generators' states after their step (not
// looked at for greedy rows); uint64 [R], the addresses of the rows' token counts (0: no penalties).  shared_counts: rows may
// have the same counts.  host_out: null, or page-locked int32 [R] that gets the ids as well.
extern "C" int exl3_sample_batch(const float* logits, const void* packed, int R, int V, int shared_counts, int* out,
                                 int* host_out, cudaStream_t stream) {
  if (R == 0) return 0;
  if (R < 0 || R > SF_DIRECT_ROWS || V < 1 || packed == nullptr) {
    set_error("sample_batch: rows=%d (at most %d) vocab=%d", R, SF_DIRECT_ROWS, V);
    return ERR_BAD_ARGUMENT;
  }
  const unsigned char* at = static_cast<const unsigned char*>(packed);
  SfBatch batch = {};
  bool penalties = false;
  for (int r = 0; r < R; ++r) {
    double o[7];
    unsigned long long state, counts;
    memcpy(o, at + (size_t)r * 56, 56);
    memcpy(&state, at + (size_t)R * 56 + (size_t)r * 8, 8);
    memcpy(&counts, at + (size_t)R * 64 + (size_t)r * 8, 8);
    batch.rows[r] = {o[0], o[1], o[2], o[3], o[0] <= 0.0 ? 0.0 : sf_uniform(state)};
    batch.counts_of[r] = reinterpret_cast<int*>(counts);
    for (int i = 0; i < 3; ++i) batch.params_of[r][i] = (float)o[4 + i];
    penalties |= counts != 0;
  }
  int rc = sf_launch(logits, batch, out, R, V, penalties, host_out, !shared_counts, stream);
  if (rc || !penalties || !shared_counts) return rc;
  SfCounts c = {};
  memcpy(c.at, batch.counts_of, sizeof(c.at));
  sample_count_batch_kernel<<<1, SF_DIRECT_ROWS, 0, stream>>>(c, out, R, V);
  return launch_status("sample_count");
}

extern "C" int exl3_sample_filtered(const float* logits, const double* rows, int* out, int R, int V,
                                    cudaStream_t stream) {
  return exl3_sample_rows(logits, rows, nullptr, nullptr, out, R, V, stream);
}

extern "C" int exl3_sample_filtered_cap() { return SF_CAP; }

// counts: R device pointers (null: the row has no penalties) to int32 [V] token counts of the rows' contexts;
// params: float32 [R, 3] (repetition, presence, frequency penalty).  Changes logits in place.
extern "C" int exl3_sample_penalties(float* logits, int R, int V, const int* const* counts, const float* params,
                                     cudaStream_t stream) {
  if (R == 0) return 0;
  if (R < 0 || R > 65535 || V < 1) { set_error("sample_penalties: bad sizes rows=%d vocab=%d", R, V); return ERR_BAD_ARGUMENT; }
  sample_penalties_kernel<<<dim3(ceil_div(V, 256), R), 256, 0, stream>>>(logits, V, counts, params);
  return launch_status("sample_penalties");
}

// counts[r][ids[r]] += 1 for the rows that keep counts.
extern "C" int exl3_sample_count(int* const* counts, const int* ids, int R, int V, cudaStream_t stream) {
  if (R == 0) return 0;
  if (R < 0 || V < 1) { set_error("sample_count: bad sizes rows=%d vocab=%d", R, V); return ERR_BAD_ARGUMENT; }
  sample_count_kernel<<<ceil_div(R, 128), 128, 0, stream>>>(counts, ids, R, V);
  return launch_status("sample_count");
}
