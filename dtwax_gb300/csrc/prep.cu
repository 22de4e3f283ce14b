// Kernels around the sDTW sweep: the reference-squiggle builder, the per-read
// window + z-score normaliser, the reset of the result keys and the finalize
// step that turns per-strand (score, end column) keys into read results.
#include <algorithm>

#include "dtwx_internal.h"

namespace dtwx {

// Layout of the public dtwx_result (include/dtwx.h); the host checks sizeof.
struct ResultRec {
  float score;
  float score_fwd;
  float score_rev;
  int32_t strand;
  int64_t end_pos;
  int32_t call;
  int32_t n_samples;
};
static_assert(sizeof(ResultRec) == 32, "dtwx_result layout");

constexpr int kBlock = 256;

__device__ __forceinline__ int base2(unsigned char c) {
  switch (c) {
    case 'A': case 'a': return 0;
    case 'C': case 'c': return 1;
    case 'G': case 'g': return 2;
    case 'T': case 't': return 3;
    default: return -1;
  }
}

// Block-wide sum of doubles (deterministic order for a fixed block size).
__device__ double block_sum(double v, double *sh) {
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r += sh[i];
    sh[32] = r;
  }
  __syncthreads();
  r = sh[32];
  __syncthreads();
  return r;
}

// ---------------------------------------------------------------- reference builder
// Follows src/include/load_reference.hpp:33-128 (6-mer levels of the forward
// strand and of the reverse complement, z-scored per strand) and
// scripts/sdtw.py:101-116.  Statistics are FP64 over the valid k-mers; k-mers
// with a non-ACGT base become 0 and are left out.
//
// A strand has at most 4,096 different levels, so the statistics come from a
// histogram of its k-mer codes and the z-scores from a table of 4,096: the
// FP64 work (a division per level and strand) no longer grows with the genome.
// What remains is bound by the 24 bytes that a column writes in five layouts:
// 5 Mb, FP64 sums and divisions per position 427 us of kernels, now 120 us (histogram 42,
// statistics 24, z-scores 52; 18 us for the bytes).
//
// work layout: counts (uint32 [2][4096]), stats (double [2][2]: mean, sd),
// z-scored levels (float [2][4096]).

constexpr int kCodesPerThread = 16;
constexpr int kCodeSpan = kBlock * kCodesPerThread;  // columns of a CTA's turn
constexpr uint32_t kNoCode = 0xffffffffu;

// Columns [j0, j0 + kCodeSpan) of both strands: calls f(column, forward code,
// reverse code) with column j0 + t + 256 * i for thread t, kNoCode where a base
// is not ACGT.  seq_f and seq_r stage the bases as 0..3, or 4.
template <typename F>
__device__ __forceinline__ void for_codes(const unsigned char *seq, int64_t L, int64_t m, int64_t j0,
                                          unsigned char *seq_f, unsigned char *seq_r, F f) {
  __syncthreads();
  for (int i = threadIdx.x; i < kCodeSpan + kKmer - 1; i += kBlock) {
    // reverse complement: rc[t] = comp(seq[L-1-t]); comp of code c is 3-c
    const int64_t jf = j0 + i, jr = L - 1 - (j0 + i);
    const int bf = jf < L ? base2(seq[jf]) : -1, br = jr >= 0 ? base2(seq[jr]) : -1;
    seq_f[i] = (unsigned char)(bf < 0 ? 4 : bf);
    seq_r[i] = (unsigned char)(br < 0 ? 4 : 3 - br);
  }
  __syncthreads();
#pragma unroll 4
  for (int i = 0; i < kCodesPerThread; ++i) {
    const int t = threadIdx.x + kBlock * i;
    if (j0 + t >= m) break;
    uint32_t cf = 0, cr = 0, bad_f = 0, bad_r = 0;
#pragma unroll
    for (int k = 0; k < kKmer; ++k) {
      const uint32_t bf = seq_f[t + k], br = seq_r[t + k];
      bad_f |= bf, bad_r |= br;
      cf = (cf << 2) | (bf & 3u);
      cr = (cr << 2) | (br & 3u);
    }
    f(j0 + t, (bad_f & 4u) ? kNoCode : cf, (bad_r & 4u) ? kNoCode : cr);
  }
}

// Occurrences of every k-mer code on both strands.
__global__ void __launch_bounds__(kBlock) kmer_histogram_kernel(const unsigned char *seq, int64_t L, int64_t m,
                                                                uint32_t *counts) {
  __shared__ uint32_t hist[2 * kTableSize];
  __shared__ unsigned char seq_f[kCodeSpan + kKmer], seq_r[kCodeSpan + kKmer];
  for (int i = threadIdx.x; i < 2 * kTableSize; i += kBlock) hist[i] = 0;
  for (int64_t j0 = (int64_t)blockIdx.x * kCodeSpan; j0 < m; j0 += (int64_t)gridDim.x * kCodeSpan)
    for_codes(seq, L, m, j0, seq_f, seq_r, [&](int64_t, uint32_t cf, uint32_t cr) {
      if (cf != kNoCode) atomicAdd(&hist[cf], 1u);
      if (cr != kNoCode) atomicAdd(&hist[kTableSize + cr], 1u);
    });
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * kTableSize; i += kBlock)
    if (hist[i]) atomicAdd(&counts[i], hist[i]);
}

// Mean and standard deviation of a strand's levels (one CTA per strand), two passes.
__global__ void __launch_bounds__(kBlock) level_stats_kernel(const uint32_t *counts, const double *table,
                                                             double *stats) {
  __shared__ double sh[33];
  const uint32_t *n = counts + blockIdx.x * kTableSize;
  double s = 0, c = 0;
  for (int i = threadIdx.x; i < kTableSize; i += kBlock) {
    if (!n[i]) continue;
    s += (double)n[i] * table[i];
    c += (double)n[i];
  }
  s = block_sum(s, sh);
  c = block_sum(c, sh);
  const double mean = c > 0 ? s / c : 0.0;
  double q = 0;
  for (int i = threadIdx.x; i < kTableSize; i += kBlock) {
    const double d = table[i] - mean;
    if (n[i]) q += (double)n[i] * (d * d);
  }
  q = block_sum(q, sh);
  if (threadIdx.x == 0) {
    const double sd = c > 0 ? sqrt(q / c) : 1.0;
    stats[2 * blockIdx.x] = mean;
    stats[2 * blockIdx.x + 1] = sd > 0 ? sd : 1.0;
  }
}

// The z-scored level of every code, FP32 (blockIdx.y: strand).
__global__ void level_table_kernel(const double *table, const double *stats, float *z) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const double mean = stats[2 * blockIdx.y], sd = stats[2 * blockIdx.y + 1];
  z[blockIdx.y * kTableSize + i] = (float)((table[i] - mean) / sd);
}

// Writes the z-scored levels: FP16 pairs (fwd[j], rev[j]) and FP32 planes.
// PAIRED: column j < m holds k-mer j of each strand.  CONCAT: one sequence
// fwd||rev of 2m columns, stored in both strand slots (the FP32 sweep then
// aligns only plane 0).  Columns past the last (up to m_pad) are zero.
__global__ void __launch_bounds__(kBlock) zscore_pairs_kernel(const unsigned char *seq, int64_t L, int64_t m,
                                                              int64_t m_pad, int concat, const float *z,
                                                              __half2 *ref16, float *ref32, __half *ref16p,
                                                              float *fwd32, float *rev32) {
  __shared__ float lev[2 * kTableSize];
  __shared__ unsigned char seq_f[kCodeSpan + kKmer], seq_r[kCodeSpan + kKmer];
  for (int i = threadIdx.x; i < 2 * kTableSize; i += kBlock) lev[i] = z[i];
  const auto column = [&](int64_t j, float a, float b) {
    ref32[j] = a;          // fwd plane
    ref32[m_pad + j] = b;  // rev plane
    ref16[j] = __floats2half2_rn(a, b);
    ref16p[j] = __float2half_rn(a);  // FP16 planes (MIXED precision)
    ref16p[m_pad + j] = __float2half_rn(b);
  };
  for (int64_t j0 = (int64_t)blockIdx.x * kCodeSpan; j0 < m; j0 += (int64_t)gridDim.x * kCodeSpan)
    for_codes(seq, L, m, j0, seq_f, seq_r, [&](int64_t j, uint32_t cf, uint32_t cr) {
      const float a = cf == kNoCode ? 0.f : lev[cf], b = cr == kNoCode ? 0.f : lev[kTableSize + cr];
      fwd32[j] = a;
      rev32[j] = b;
      if (!concat) {
        column(j, a, b);
      } else {
        column(j, a, a);
        column(m + j, b, b);
      }
    });
  for (int64_t j = (concat ? 2 * m : m) + (int64_t)blockIdx.x * kBlock + threadIdx.x; j < m_pad;
       j += (int64_t)gridDim.x * kBlock)
    column(j, 0.f, 0.f);
}

size_t build_reference_work_bytes() {
  return sizeof(uint32_t) * 2 * kTableSize + sizeof(double) * 4 + sizeof(float) * 2 * kTableSize;
}

cudaError_t launch_build_reference(const char *d_seq, int64_t L, const double *d_table, int64_t m,
                                   int64_t m_pad, int concat, void *d_work, __half2 *d_ref16,
                                   float *d_ref32, __half *d_ref16p, float *d_fwd32, float *d_rev32,
                                   cudaStream_t s) {
  uint32_t *counts = static_cast<uint32_t *>(d_work);
  double *stats = reinterpret_cast<double *>(counts + 2 * kTableSize);
  float *z = reinterpret_cast<float *>(stats + 4);
  const unsigned char *seq = reinterpret_cast<const unsigned char *>(d_seq);
  const int grid = (int)std::min<int64_t>((m + kCodeSpan - 1) / kCodeSpan, 152 * 5);
  const cudaError_t e = cudaMemsetAsync(counts, 0, sizeof(uint32_t) * 2 * kTableSize, s);
  if (e != cudaSuccess) return e;
  kmer_histogram_kernel<<<grid, kBlock, 0, s>>>(seq, L, m, counts);
  level_stats_kernel<<<2, kBlock, 0, s>>>(counts, d_table, stats);
  level_table_kernel<<<dim3(kTableSize / 64, 2), 64, 0, s>>>(d_table, stats, z);
  zscore_pairs_kernel<<<grid, kBlock, 0, s>>>(seq, L, m, m_pad, concat, z, d_ref16, d_ref32, d_ref16p, d_fwd32,
                                              d_rev32);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- normaliser
// Per read: y = (x - mean) / sqrt(var + eps) over the window, population
// variance, two passes (src/include/normalizer.cu:370-413 uses cuDNN batch norm
// in SPATIAL mode with eps 1e-4 for the same formula).  int16 input is first
// scaled to pA: (raw + add) * mul.
//
// 64-bit accuracy without the FP64 pipe, which has 1/64 of the FP32 rate here
// (2,048 reads of 1,000 to 8,000 samples, one dtwx_normalize call after the
// other: 244 us with FP64 passes, now 49 on reads that come from HBM and 42 on
// the same 37 MB again and again, which L2 holds; 11 us for the bytes): sums,
// deviations and products are unevaluated pairs of floats
// (error-free sums and FMA products, Knuth and Dekker), about 48 bits, and
// the mean, variance and reciprocal root of a read are FP64 in one warp, with as
// few instructions as they take: a warp's total converted by each warp, added by
// one thread and divided twice cost 6 us more, and a third of the time of
// short reads (4,096 of 200 to 400 samples: 47 us, 32 now; 120 with FP64 passes).
// Accuracy: the mean is good to about 2^-47 of its own size, which is an absolute
// error of every result, so a value whose deviation is as small as 2^-22 of the
// mean may miss the FP32 nearest to the 64-bit value; the largest error of a read
// does not change.  (11 kinds of input, 200 to 40,000 samples, against 80 bits:
// the same errors as with FP64 passes in 42 of 44; 592 of 2,000 values spread
// 1e-5 about 90 rounded better, 986 of 40,000 spread 1 about 1e6 worse, by at most
// 0.16 units.)  Reads with samples of 2^40 or more, none above 2^-40,
// NaN or infinity, or a deviation whose squares leave the FP32 range take the
// FP64 passes.  The samples of a read are read once and kept in shared memory
// (up to kNormStaged of them).

constexpr int kNormStaged = 11776;  // 46 KB: with the reductions within the 48 KB that need no opt-in

// s + e == a + b exactly, s the rounded sum.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// x - (m0 + m1 + m2) as a pair, |e| about half a unit of d.  (The mean in three
// parts: two lose bits where the samples lie far from zero for their spread.)
__device__ __forceinline__ void deviation(float x, float m0, float m1, float m2, float &d, float &e) {
  float a, b;
  two_sum(x, -m0, a, b);
  two_sum(a, -m1, d, e);
  e += b - m2;
}

// A sum as an unevaluated pair.
struct PairSum {
  float h = 0.f, l = 0.f;
  __device__ __forceinline__ void add(float x) {
    float e;
    two_sum(h, x, h, e);
    l += e;
  }
  __device__ __forceinline__ void warp_reduce() {
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
      const float oh = __shfl_xor_sync(0xffffffffu, h, m), ol = __shfl_xor_sync(0xffffffffu, l, m);
      add(oh);
      l += ol;
    }
  }
};

// Total of the warps' sums, in FP64: `part` holds a pair per warp; every lane of
// the calling warp gets it.  (Eight lanes convert and add at once: an FP64
// instruction holds its pipe 16 cycles for one lane as for 32.)
__device__ __forceinline__ double warps_total(const float2 *part, int lane) {
  double v = 0.0;
  if (lane < kBlock / 32) v = (double)part[lane].x + (double)part[lane].y;
#pragma unroll
  for (int m = kBlock / 64; m >= 1; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}

template <typename T>
__global__ void __launch_bounds__(kBlock) normalize_kernel(const T *src, const int64_t *src_off,
                                                           const int64_t *dst_off, const int32_t *dst_len,
                                                           const float *scale_mul,
                                                           const float *scale_add, float eps,
                                                           float *dst, int staged) {
  extern __shared__ float stage[];
  __shared__ double sh[33];
  __shared__ uint32_t sh_max[kBlock / 32];
  __shared__ float sh_part[4];
  __shared__ float2 sh_pair[kBlock / 32];
  const int r = blockIdx.x;
  const int n = dst_len[r];
  if (n <= 0) return;
  const T *x = src + src_off[r];
  float *y = dst + dst_off[r];
  const float mul = scale_mul ? scale_mul[r] : 1.f;
  const float add = scale_add ? scale_add[r] : 0.f;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const auto sample = [&](int i) { return ((float)x[i] + add) * mul; };
  const bool keep = n <= staged;
  const auto get = [&](int i) { return keep ? stage[i] : sample(i); };

  double rn = 0.0;  // of warp 0, whose division overlaps the loads of the others
  if (warp == 0) rn = 1.0 / (double)n;

  // pass 1: sum, and the largest magnitude (NaN and infinity above all others)
  PairSum s;
  uint32_t top = 0;
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += kBlock) {
    const float v = sample(i);
    if (keep) stage[i] = v;
    top = max(top, __float_as_uint(v) & 0x7fffffffu);
    s.add(v);
  }
  s.warp_reduce();
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) {
    sh_pair[warp] = make_float2(s.h, s.l);
    sh_max[warp] = top;
  }
  __syncthreads();
  top = 0;
  for (int i = 0; i < kBlock / 32; ++i) top = max(top, sh_max[i]);
  constexpr uint32_t kBig = (127u + 40u) << 23, kSmall = (127u - 40u) << 23;
  bool wild = top >= kBig || top < kSmall;
  if (!wild) {
    if (warp == 0) {
      double mean = warps_total(sh_pair, lane) * rn;
      if (lane == 0) {
        sh_part[0] = (float)mean;
        mean -= (double)sh_part[0];
        sh_part[1] = (float)mean;
        sh_part[2] = (float)(mean - (double)sh_part[1]);
      }
    }
    __syncthreads();
    const float m0 = sh_part[0], m1 = sh_part[1], m2 = sh_part[2];

    // pass 2: squared deviations
    PairSum q;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += kBlock) {
      float d, e;
      deviation(get(i), m0, m1, m2, d, e);
      const float p = __fmul_rn(d, d);
      q.add(p);
      q.l += fmaf(2.f * d, e, fmaf(d, d, -p));
    }
    q.warp_reduce();
    if (lane == 0) sh_pair[warp] = make_float2(q.h, q.l);
    __syncthreads();
    if (warp == 0) {
      const double var = warps_total(sh_pair, lane) * rn;
      const double inv = rsqrt(var + (double)eps);
      if (lane == 0) {
        sh_part[0] = (float)inv;
        sh_part[1] = (float)(inv - (double)(float)inv);
        sh_part[3] = (float)var;
      }
    }
    __syncthreads();
    const float ih = sh_part[0], il = sh_part[1];
    // squares below the FP32 range (a deviation of 2^-60 and less next to no eps)
    wild = sh_part[3] < 0x1p-80f && eps < 0x1p-60f;
    if (!wild) {
#pragma unroll 4
      for (int i = threadIdx.x; i < n; i += kBlock) {
        float d, e;
        deviation(get(i), m0, m1, m2, d, e);
        const float p = __fmul_rn(d, ih);
        y[i] = p + fmaf(e, ih, fmaf(d, il, fmaf(d, ih, -p)));
      }
      return;
    }
  }
  __syncthreads();
  double sd = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) sd += (double)get(i);
  const double mean = block_sum(sd, sh) / (double)n;
  double q = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double d = (double)get(i) - mean;
    q += d * d;
  }
  const double var = block_sum(q, sh) / (double)n;
  const double inv = 1.0 / sqrt(var + (double)eps);
  for (int i = threadIdx.x; i < n; i += blockDim.x) y[i] = (float)(((double)get(i) - mean) * inv);
}

cudaError_t launch_normalize(const void *src, int is_i16, const int64_t *src_off,
                             const int64_t *dst_off, const int32_t *dst_len, const float *scale_mul,
                             const float *scale_add, int n_reads, int max_len, float eps, float *dst,
                             cudaStream_t s) {
  if (n_reads <= 0) return cudaSuccess;
  const int staged = max_len <= kNormStaged ? max_len : kNormStaged;
  const size_t smem = sizeof(float) * (size_t)(staged > 0 ? staged : 1);
  if (is_i16)
    normalize_kernel<int16_t><<<n_reads, kBlock, smem, s>>>(static_cast<const int16_t *>(src), src_off, dst_off,
                                                            dst_len, scale_mul, scale_add, eps, dst, staged);
  else
    normalize_kernel<float><<<n_reads, kBlock, smem, s>>>(static_cast<const float *>(src), src_off, dst_off, dst_len,
                                                          scale_mul, scale_add, eps, dst, staged);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- reset / finalize

__global__ void reset_kernel(unsigned long long *keys, int n_keys, int32_t *counter, int32_t *err,
                             int32_t *halo_read, int n_halo) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_keys) keys[i] = ~0ull;
  if (i < n_halo) halo_read[i] = 0;
  if (i == 0 && counter) *counter = 0;
  if (i == 0 && err) *err = 0;
}

cudaError_t launch_reset(unsigned long long *keys, int n_keys, int32_t *counter, int32_t *err, int32_t *halo_read,
                         int n_halo, cudaStream_t s) {
  const int most = n_keys > n_halo ? n_keys : n_halo, n = most > 1 ? most : 1;
  reset_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, s>>>(keys, n_keys, counter, err, halo_read, n_halo);
  return cudaGetLastError();
}

// The min/argmin of the last DP row was reduced inside the sweep into one key
// per read and strand: (orderable score << 32) | end column, combined with
// atomicMin, so the smallest score wins and ties go to the smallest column.
// Here the two strands are combined (ties: forward strand) and the call is
// made: target when score < threshold (calc_classification_threshold.py:52).
__global__ void finalize_kernel(const unsigned long long *keys, const int32_t *n_samples,
                                int n_reads, int concat, int64_t m_fwd, float threshold,
                                const int32_t *err, ResultRec *out) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n_reads) return;
  ResultRec o;
  const int32_t ns = n_samples ? n_samples[r] : 1;
  o.n_samples = ns;
  const unsigned long long kf = keys[2 * r], kr = keys[2 * r + 1];
  const float inf = __int_as_float(0x7f800000);
  float sf = kf == ~0ull ? inf : ordered_to_float((uint32_t)(kf >> 32));
  float sr = kr == ~0ull ? inf : ordered_to_float((uint32_t)(kr >> 32));
  const int64_t ef = kf == ~0ull ? -1 : (int64_t)(uint32_t)(kf & 0xffffffffu);
  const int64_t er = kr == ~0ull ? -1 : (int64_t)(uint32_t)(kr & 0xffffffffu);
  if (!concat) {
    const bool rev = sr < sf || (sr == sf && er < ef);
    o.score_fwd = sf;
    o.score_rev = sr;
    o.score = rev ? sr : sf;
    o.strand = rev ? 1 : 0;
    o.end_pos = rev ? er : ef;
  } else {
    // one sequence fwd||rev: the column tells the strand
    o.score = sf;
    o.score_fwd = sf;
    o.score_rev = sf;
    o.strand = ef >= m_fwd ? 1 : 0;
    o.end_pos = ef >= m_fwd ? ef - m_fwd : ef;
  }
  o.call = ns <= 0 ? -1 : (o.score < threshold ? 1 : 0);
  if (ns <= 0) {
    o.score = o.score_fwd = o.score_rev = inf;
    o.end_pos = -1;
    o.strand = 0;
  }
  const int32_t e = err ? *err : 0;
  if (e != 0) {
    // a bounded wait gave up or a task was refused: the keys are incomplete
    o.score = o.score_fwd = o.score_rev = __int_as_float(0x7fc00000);
    o.end_pos = -1;
    o.strand = e;
    o.call = kCallDeviceError;
  }
  out[r] = o;
}

cudaError_t launch_finalize(const unsigned long long *keys, const int32_t *n_samples, int n_reads,
                            int concat, int64_t m_fwd, float threshold, const int32_t *err,
                            void *d_results, cudaStream_t s) {
  if (n_reads <= 0) return cudaSuccess;
  finalize_kernel<<<(n_reads + kBlock - 1) / kBlock, kBlock, 0, s>>>(
      keys, n_samples, n_reads, concat, m_fwd, threshold, err, static_cast<ResultRec *>(d_results));
  return cudaGetLastError();
}

}  // namespace dtwx
