// sDTW kernels for sm_103a: the persistent batched kernel (FP16 half2 with a
// running-minimum offset, or FP32) and the issue-rate probe used as roofline.
//
// Recurrence (src/include/DTW.cu:37-39 with -DNO_REF_DEL; scripts/sdtw.py:205-225):
//   D[i][j] = (r_j - q_i)^2 + min(D[i-1][j], D[i-1][j-1]),   free start (row -1 = 0),
//   D[i][0] = D[i-1][0] + (r_0 - q_i)^2,   result = min_j D[n-1][j] and its column.
//
// Layout of the work.  A row depends only on the previous row (there is no
// horizontal term), so the 32 lanes of a warp sweep the SAME row together; lane
// l owns the S consecutive columns x + l*S .. x + l*S + S-1 of a 32*S-column
// "strip", keeps them in registers, and receives the diagonal predecessor of
// its first column from lane l-1 by one __shfl_up_sync per row.  Lane 0 takes
// it from the seam column written by the strip to the left.
//
// A work item is (task, chunk): the task's rows against output columns
// [a, b) of the reference.  The warps of a CTA form a team (team.cuh): the
// strips of [x0, b) are handed out left to right, and the warp of strip s + 1
// runs a window of 32 rows behind the warp of strip s, whose last column
// reaches it through a seam buffer in global scratch.  An item therefore lasts
// about as long as its strips divided by the team's warps, not as long as one
// warp takes for all of them.  Each warp stages its strip's slice of the
// reference into shared memory by a TMA tensor copy and reads it into
// registers once per strip.  Chunks are independent: a chunk starting at a > 0
// recomputes a halo of >= n columns to its left, with +inf entering at the
// halo's left edge; that error moves right one column per row, so it never
// reaches column a.  Halo strips stop at the last row that can still influence
// column a.  In the NH instances they are narrower than the chunk's own
// strips, so the swept halo follows that shrinking triangle more closely.
//
// FP16: cells are __half2 (fwd strand in .x, rev in .y).  Every kRescaleRows
// rows each strip subtracts its own row minimum from its cells and adds it to
// an FP32 offset, so the cells near the minimum stay small and precise.  The
// seam value crossing into the next strip is re-based by the difference of the
// two strips' offsets (one per epoch of kRescaleRows rows).
//
// MIXED: the differences r - q run in FP16 half2 (two adjacent columns of one
// strand per instruction) and the path cost is FP32: each cell is one
// mixed-precision FMA d*d + min(...) with f16 d and an f32 addend and result.
#include "dtwx_internal.h"

#include <algorithm>
#include <atomic>
#include <cuda/std/cstdint>

#include "team.cuh"

namespace dtwx {

// ---------------------------------------------------------------- precision policies
// Every policy keeps one 32-bit register per cell so that selects, shuffles
// and seam stores are single instructions.  FP16 packs the two strands of a
// column into one __half2 (fwd in .x, rev in .y) and a work item covers both;
// FP32 and MIXED keep one strand per cell and a work item covers one strand.
// RV is the register type of the reference (RB bytes per column).

template <int PREC> struct Pol;

template <> struct Pol<0> {  // FP16 pairs
  using V = __half2;
  using RV = __half2;
  static constexpr int RB = 4;       // reference bytes per column
  static constexpr int STRANDS = 1;  // work items per (task, chunk)
  __device__ __forceinline__ static V inf() { return __half2half2(__ushort_as_half((unsigned short)0x7c00u)); }
  __device__ __forceinline__ static V zero() { return __half2half2(__ushort_as_half((unsigned short)0)); }
  __device__ __forceinline__ static V cell(V r, V q, V a, V b) {
    const V d = __hsub2(r, q);
    return __hfma2(d, d, __hmin2(a, b));
  }
  __device__ __forceinline__ static V vmin(V a, V b) { return __hmin2(a, b); }
  __device__ __forceinline__ static V shfl(V v, int src) { return __shfl_sync(FULL_MASK, v, src); }
  __device__ __forceinline__ static V shfl_up(V v) { return __shfl_up_sync(FULL_MASK, v, 1); }
  __device__ __forceinline__ static V shfl_xor(V v, int m) { return __shfl_xor_sync(FULL_MASK, v, m); }
  __device__ __forceinline__ static V sel(bool p, V a, V b) { return p ? a : b; }
  __device__ __forceinline__ static V from_bits(uint32_t u) {
    V v;
    memcpy(&v, &u, 4);
    return v;
  }
  // a query sample as the cells take it: (q, q)
  using QW = __half2;
  __device__ __forceinline__ static QW qw(float q) { return __float2half2_rn(q); }
};

template <> struct Pol<1> {  // FP32, one strand
  using V = float;
  using RV = float;
  static constexpr int RB = 4;
  static constexpr int STRANDS = 2;
  __device__ __forceinline__ static V inf() { return __int_as_float(0x7f800000); }
  __device__ __forceinline__ static V zero() { return 0.f; }
  __device__ __forceinline__ static V cell(V r, V q, V a, V b) {
    const float d = r - q;
    return fmaf(d, d, fminf(a, b));
  }
  __device__ __forceinline__ static V vmin(V a, V b) { return fminf(a, b); }
  __device__ __forceinline__ static V shfl(V v, int src) { return __shfl_sync(FULL_MASK, v, src); }
  __device__ __forceinline__ static V shfl_up(V v) { return __shfl_up_sync(FULL_MASK, v, 1); }
  __device__ __forceinline__ static V shfl_xor(V v, int m) { return __shfl_xor_sync(FULL_MASK, v, m); }
  __device__ __forceinline__ static V sel(bool p, V a, V b) { return p ? a : b; }
  __device__ __forceinline__ static V from_bits(uint32_t u) { return __uint_as_float(u); }
  using QW = float;
  __device__ __forceinline__ static QW qw(float q) { return q; }
};

template <> struct Pol<2> {  // MIXED: FP16 differences, FP32 path cost, one strand
  using V = float;
  using RV = __half2;                // two adjacent columns of one strand
  static constexpr int RB = 2;
  static constexpr int STRANDS = 2;
  __device__ __forceinline__ static V inf() { return __int_as_float(0x7f800000); }
  __device__ __forceinline__ static V zero() { return 0.f; }
  __device__ __forceinline__ static V vmin(V a, V b) { return fminf(a, b); }
  __device__ __forceinline__ static V shfl(V v, int src) { return __shfl_sync(FULL_MASK, v, src); }
  __device__ __forceinline__ static V shfl_up(V v) { return __shfl_up_sync(FULL_MASK, v, 1); }
  __device__ __forceinline__ static V shfl_xor(V v, int m) { return __shfl_xor_sync(FULL_MASK, v, m); }
  __device__ __forceinline__ static V sel(bool p, V a, V b) { return p ? a : b; }
  __device__ __forceinline__ static V from_bits(uint32_t u) { return __uint_as_float(u); }
  using QW = __half2;
  __device__ __forceinline__ static QW qw(float q) { return __float2half2_rn(q); }
};

// d*d + c with d in FP16 and c, the result in FP32, one rounding (PTX
// fma.rn.f32.f16, sm_100 and later).
__device__ __forceinline__ float fma_sq_f16(__half d, float c) {
  float r;
  asm("fma.rn.f32.f16 %0, %1, %1, %2;" : "=f"(r) : "h"(__half_as_ushort(d)), "f"(c));
  return r;
}

template <typename T>
__device__ __forceinline__ T bits_as(uint32_t u) {
  T v;
  memcpy(&v, &u, 4);
  return v;
}

// ---------------------------------------------------------------- TMA / mbarrier helpers

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Bounded wait on an mbarrier phase: at most `limit` polls; false when the
// wait gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, uint32_t limit) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Lane-0 actions as predicated PTX: every lane executes the same instruction
// stream (the action is masked by a predicate), so the compiler never sees a
// lane-dependent branch it could use to duplicate the whole strip loop into a
// lane-0 copy and a lanes-1..31 copy.
__device__ __forceinline__ void mbar_init_if(uint64_t *bar, uint32_t count, uint32_t pred) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p mbarrier.init.shared::cta.b64 [%0], %1;\n\t}" ::"r"(
          smem_u32(bar)),
      "r"(count), "r"(pred)
      : "memory");
}

__device__ __forceinline__ void tma_issue_if(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1,
                                             uint32_t bytes, uint32_t pred) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t"
      "@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%4], %6;\n\t"
      "@p cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];\n\t}" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_u32(bar)), "r"(pred), "r"(bytes)
      : "memory");
}

// 32-bit shared-memory store by the lanes whose pred is set, as predicated PTX.
__device__ __forceinline__ void st_shared_if(uint32_t addr, uint32_t v, uint32_t pred) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.shared.b32 [%0], %1;\n\t}" ::"r"(addr), "r"(v),
               "r"(pred)
               : "memory");
}

__device__ __forceinline__ uint32_t ld_shared_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

// N = 2 or 4 consecutive 32-bit words from shared memory.
template <int N>
__device__ __forceinline__ void ld_shared_words(uint32_t addr, uint32_t (&v)[N]) {
  static_assert(N == 2 || N == 4, "one vector load");
  if constexpr (N == 2)
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(addr) : "memory");
  else
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(addr)
                 : "memory");
}

__device__ __forceinline__ void st_shared_u32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

__device__ __forceinline__ void st_shared_v4_if(uint32_t addr, uint4 v, uint32_t pred) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t@p st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n\t}" ::"r"(addr),
      "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(pred)
      : "memory");
}

// Byte offset of logical byte b of a tile written by TMA with 128-byte
// swizzling: the 16-byte chunk index inside each 128-byte row is XOR-ed with
// the row index modulo 8.
__device__ __forceinline__ uint32_t swz128(uint32_t b) {
  const uint32_t row = b >> 7;
  const uint32_t chunk = (b >> 4) & 7u;
  return (row << 7) | ((chunk ^ (row & 7u)) << 4) | (b & 15u);
}

// ---------------------------------------------------------------- ref strip -> registers
// Lane l's slice of a strip: NW consecutive 32-bit words at byte (l*NW)*4
// (S columns: NW = S for 4-byte columns, S/2 for FP16 columns of one strand).

template <int NW, typename RV>
__device__ __forceinline__ void regs_from_smem(const unsigned char *tile, int lane, RV (&R)[NW]) {
  static_assert((NW * 4) % 16 == 0, "lane slice must be 16-byte aligned");
#pragma unroll
  for (int k = 0; k < NW; k += 4) {
    const uint32_t b = (uint32_t)((lane * NW + k) * 4);
    const uint4 v = *reinterpret_cast<const uint4 *>(tile + swz128(b));
    R[k] = bits_as<RV>(v.x);
    R[k + 1] = bits_as<RV>(v.y);
    R[k + 2] = bits_as<RV>(v.z);
    R[k + 3] = bits_as<RV>(v.w);
  }
}

// Contiguous words from global memory (FP16 pairs, one FP32 strand plane, or
// one FP16 strand plane).
template <int NW, typename RV>
__device__ __forceinline__ void regs_from_global(const void *base, int lane, RV (&R)[NW]) {
  const uint4 *g = reinterpret_cast<const uint4 *>(reinterpret_cast<const uint32_t *>(base) + lane * NW);
#pragma unroll
  for (int k = 0; k < NW; k += 4) {
    const uint4 v = __ldg(g + k / 4);
    R[k] = bits_as<RV>(v.x);
    R[k + 1] = bits_as<RV>(v.y);
    R[k + 2] = bits_as<RV>(v.z);
    R[k + 3] = bits_as<RV>(v.w);
  }
}

// FP32 strand `strand` out of interleaved (fwd, rev) float pairs, of which
// `cols` (even) may be read; columns past them are past the reference too.
template <int S>
__device__ __forceinline__ void regs_from_pairs(const float2 *pairs, int64_t x, int64_t cols, int lane, int strand,
                                                float (&R)[S]) {
  const int64_t c0 = x + (int64_t)lane * S;
  const float4 *g = reinterpret_cast<const float4 *>(pairs + c0);
#pragma unroll
  for (int k = 0; k < S; k += 2) {
    const float4 v = c0 + k < cols ? __ldg(g + k / 2) : make_float4(0.f, 0.f, 0.f, 0.f);
    R[k] = strand ? v.y : v.x;
    R[k + 1] = strand ? v.w : v.z;
  }
}

// Bit image of a cell and back (both policies use 32-bit cells).
template <int PREC>
__device__ __forceinline__ uint32_t cell_bits(typename Pol<PREC>::V v) {
  uint32_t u;
  memcpy(&u, &v, 4);
  return u;
}

// Bit image of a query sample as the policy's cells take it, and back.
template <int PREC>
__device__ __forceinline__ uint32_t qw_bits(float q) {
  const typename Pol<PREC>::QW w = Pol<PREC>::qw(q);
  uint32_t u;
  memcpy(&u, &w, 4);
  return u;
}
template <int PREC>
__device__ __forceinline__ typename Pol<PREC>::QW qw_from(uint32_t u) {
  return bits_as<typename Pol<PREC>::QW>(u);
}

// All-ones on lane 0, zero elsewhere, from an opaque move: the optimiser cannot
// see which lanes hold which value, so it cannot split the row loop into a
// lane-0 copy and a lanes-1..31 copy (which halves the active lanes of every
// cell instruction).
__device__ __forceinline__ uint32_t lane0_mask(int lane) {
  uint32_t m = lane == 0 ? 0xffffffffu : 0u;
  asm volatile("mov.b32 %0, %0;" : "+r"(m));
  return m;
}

// One DP row of this lane's S columns.  The previous row is in D; columns are
// updated from right to left so D[k-1] still holds the previous row when
// column k reads it.  The diagonal predecessor of column 0 comes from lane-1
// (shuffle) or, on lane 0, from the seam column of the strip to the left,
// merged in with the lane-0 bit mask.
template <int S, int PREC>
__device__ __forceinline__ void sweep_row(typename Pol<PREC>::V (&D)[S], const typename Pol<PREC>::V (&R)[S],
                                          typename Pol<PREC>::V qq, typename Pol<PREC>::V seam, uint32_t m0) {
  using P = Pol<PREC>;
  const typename P::V up = P::shfl_up(D[S - 1]);
  const typename P::V left = P::from_bits((cell_bits<PREC>(up) & ~m0) | (cell_bits<PREC>(seam) & m0));
  if constexpr (PREC == 1) {
    // two columns per packed FP32 operation: the cell's three issue slots become
    // two, with the bits of the scalar operations
    const float2 nq = make_float2(-qq, -qq);
#pragma unroll
    for (int k = S - 2; k >= 0; k -= 2) {
      const float2 m = make_float2(fminf(D[k], k > 0 ? D[k - 1] : left), fminf(D[k + 1], D[k]));
      const float2 d = __fadd2_rn(make_float2(R[k], R[k + 1]), nq);
      const float2 c = __ffma2_rn(d, d, m);
      D[k] = c.x;
      D[k + 1] = c.y;
    }
  } else {
#pragma unroll
    for (int k = S - 1; k >= 1; --k) D[k] = P::cell(R[k], qq, D[k], D[k - 1]);
    D[0] = P::cell(R[0], qq, D[0], left);
  }
}

// The MIXED row: reference columns 2k and 2k+1 of the lane share one half2,
// so one HSUB2 gives both differences; each cell is one FP32-result FMA.
template <int S>
__device__ __forceinline__ void sweep_row_mixed(float (&D)[S], const __half2 (&R)[S / 2], __half2 qq, float seam,
                                                uint32_t m0) {
  const float up = __shfl_up_sync(FULL_MASK, D[S - 1], 1);
  const float left = __uint_as_float((__float_as_uint(up) & ~m0) | (__float_as_uint(seam) & m0));
#pragma unroll
  for (int k = S / 2 - 1; k >= 0; --k) {
    const __half2 d = __hsub2(R[k], qq);
    D[2 * k + 1] = fma_sq_f16(__high2half(d), fminf(D[2 * k + 1], D[2 * k]));
    D[2 * k] = fma_sq_f16(__low2half(d), fminf(D[2 * k], k > 0 ? D[2 * k - 1] : left));
  }
}

// ---------------------------------------------------------------- the persistent kernel

// One DP row for the policy: FP16 pairs and FP32 share sweep_row, MIXED has its own.
template <int S, int PREC>
__device__ __forceinline__ void row(typename Pol<PREC>::V (&D)[S],
                                    const typename Pol<PREC>::RV (&R)[S * Pol<PREC>::RB / 4],
                                    typename Pol<PREC>::QW qq, typename Pol<PREC>::V seam, uint32_t m0) {
  if constexpr (PREC == 2)
    sweep_row_mixed<S>(D, R, qq, seam, m0);
  else
    sweep_row<S, PREC>(D, R, qq, seam, m0);
}

// Register cap per instance: the S cells and S reference elements of a lane
// plus about 40 registers of bookkeeping, rounded to 128 or 168 (16 or 12
// warps/SM).
template <int S, int PREC>
constexpr int sdtw_reg_cap() { return S + S * Pol<PREC>::RB / 4 + 40 <= 128 ? 128 : 168; }

// ---------------------------------------------------------------- work items

// The item's geometry: its columns [a, b), where its halo starts and its strips.
struct Item {
  int64_t a, b, x0;
  int nh, nstrips;
};
template <int W, int WH>
__device__ __forceinline__ Item item_geometry(const SdtwParams &p, int chunk, int n) {
  Item g;
  const int64_t C = (int64_t)p.chunk_strips * W;
  g.a = (int64_t)chunk * C;
  g.b = min(g.a + C, p.m);
  g.x0 = g.a;
  if (chunk > 0) {
    const int64_t halo = ((int64_t)n + WH - 1) / WH * WH;
    g.x0 = g.a - halo > 0 ? g.a - halo : 0;
  }
  g.nh = (int)((g.a - g.x0) / WH);
  g.nstrips = g.nh + (int)((g.b - g.a + W - 1) / W);
  return g;
}

// ---------------------------------------------------------------- row state

// Row "-1" of a resumed strip's columns [c0, c0 + SC) of this lane, and the
// frame offset (FP16 cells: the strip's minimum).
template <int SC, int PREC, bool ST16>
__device__ __forceinline__ void load_row_state(typename Pol<PREC>::V (&D)[SC], float2 &O, const float *plane0,
                                               int64_t m_pad, int strand, int64_t c0) {
  if constexpr (PREC == 0) {
    float mx = __int_as_float(0x7f800000), my = mx;
    if constexpr (ST16) {
      // FP16 row state: half2 cells relative to the offset of their 512-column
      // group (the saving strip's frame); re-based onto this strip's minimum
      const uint4 *hc = reinterpret_cast<const uint4 *>(reinterpret_cast<const __half2 *>(plane0) + c0);
      const float2 *og = reinterpret_cast<const float2 *>(plane0 + m_pad);
#pragma unroll
      for (int k = 0; k < SC / 4; ++k) {
        const uint4 u = hc[k];
        D[4 * k] = bits_as<__half2>(u.x);
        D[4 * k + 1] = bits_as<__half2>(u.y);
        D[4 * k + 2] = bits_as<__half2>(u.z);
        D[4 * k + 3] = bits_as<__half2>(u.w);
      }
#pragma unroll
      for (int k = 0; k < SC; ++k) {
        const float2 o = og[(c0 + k) >> 9];
        const float2 v = __half22float2(D[k]);
        mx = fminf(mx, v.x + o.x);
        my = fminf(my, v.y + o.y);
      }
    } else {
      // two passes over the saved planes: strip minimum first, then the cells
      const float4 *f0 = reinterpret_cast<const float4 *>(plane0 + c0);
      const float4 *f1 = reinterpret_cast<const float4 *>(plane0 + m_pad + c0);
#pragma unroll
      for (int k = 0; k < SC / 4; ++k) {
        const float4 u = f0[k], v = f1[k];
        mx = fminf(mx, fminf(fminf(u.x, u.y), fminf(u.z, u.w)));
        my = fminf(my, fminf(fminf(v.x, v.y), fminf(v.z, v.w)));
      }
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
      mx = fminf(mx, __shfl_xor_sync(FULL_MASK, mx, m));
      my = fminf(my, __shfl_xor_sync(FULL_MASK, my, m));
    }
    O = make_float2(mx, my);
    if constexpr (ST16) {
      const float2 *og = reinterpret_cast<const float2 *>(plane0 + m_pad);
#pragma unroll
      for (int k = 0; k < SC; ++k) {
        const float2 o = og[(c0 + k) >> 9];
        const float2 v = __half22float2(D[k]);
        D[k] = __floats2half2_rn(v.x + o.x - mx, v.y + o.y - my);
      }
    } else {
      const float4 *f0 = reinterpret_cast<const float4 *>(plane0 + c0);
      const float4 *f1 = reinterpret_cast<const float4 *>(plane0 + m_pad + c0);
#pragma unroll
      for (int k = 0; k < SC / 4; ++k) {
        const float4 u = f0[k], v = f1[k];
        D[4 * k] = __floats2half2_rn(u.x - mx, v.x - my);
        D[4 * k + 1] = __floats2half2_rn(u.y - mx, v.y - my);
        D[4 * k + 2] = __floats2half2_rn(u.z - mx, v.z - my);
        D[4 * k + 3] = __floats2half2_rn(u.w - mx, v.w - my);
      }
    }
  } else {
    const float4 *f = reinterpret_cast<const float4 *>(plane0 + (int64_t)strand * m_pad + c0);
#pragma unroll
    for (int k = 0; k < SC / 4; ++k) {
      const float4 u = f[k];
      D[4 * k] = u.x;
      D[4 * k + 1] = u.y;
      D[4 * k + 2] = u.z;
      D[4 * k + 3] = u.w;
    }
  }
}

// The last row of this lane's columns, back to the read's row state.
template <int S, int PREC, bool ST16>
__device__ __forceinline__ void save_row_state(const typename Pol<PREC>::V (&D)[S], float2 O, float *plane0,
                                               int64_t m_pad, int strand, int64_t c0) {
  if constexpr (PREC == 0 && ST16) {
    // half2 cells in this strip's frame, the frame offset once per 512-column group
    uint4 *hc = reinterpret_cast<uint4 *>(reinterpret_cast<__half2 *>(plane0) + c0);
#pragma unroll
    for (int k = 0; k < S / 4; ++k)
      hc[k] = make_uint4(cell_bits<0>(D[4 * k]), cell_bits<0>(D[4 * k + 1]), cell_bits<0>(D[4 * k + 2]),
                         cell_bits<0>(D[4 * k + 3]));
    float2 *og = reinterpret_cast<float2 *>(plane0 + m_pad);
    og[c0 >> 9] = O;  // every lane of the strip stores the same value
    og[(c0 + S - 1) >> 9] = O;
  } else if constexpr (PREC == 0) {
    float4 *f0 = reinterpret_cast<float4 *>(plane0 + c0);
    float4 *f1 = reinterpret_cast<float4 *>(plane0 + m_pad + c0);
#pragma unroll
    for (int k = 0; k < S / 4; ++k) {
      const float2 v0 = __half22float2(D[4 * k]), v1 = __half22float2(D[4 * k + 1]);
      const float2 v2 = __half22float2(D[4 * k + 2]), v3 = __half22float2(D[4 * k + 3]);
      f0[k] = make_float4(v0.x + O.x, v1.x + O.x, v2.x + O.x, v3.x + O.x);
      f1[k] = make_float4(v0.y + O.y, v1.y + O.y, v2.y + O.y, v3.y + O.y);
    }
  } else {
    float4 *f = reinterpret_cast<float4 *>(plane0 + (int64_t)strand * m_pad + c0);
#pragma unroll
    for (int k = 0; k < S / 4; ++k) f[k] = make_float4(D[4 * k], D[4 * k + 1], D[4 * k + 2], D[4 * k + 3]);
  }
}

// Wait until the resumed halos that start from the saved row of columns
// [x, x + W) have read it: the halos of the chunks to the right of this one
// that reach column x.  Those chunks have lower item numbers: they were handed
// out before this one (tickets), or belong to a CTA that started before this one
// (ORDERED below), and their halo strips depend on nothing of it.  Bounded; it
// gives up before the waits of team_wait that can be behind it (at a third of a
// microsecond a poll or more: a tenth of a second and 5 us a row).
template <int W, int WH>
__device__ __forceinline__ bool wait_halo_readers(const SdtwParams &p, const Item &g, int64_t x, int item, int chunk,
                                                  int n, uint32_t abort_addr) {
  for (int c = chunk + 1; c < p.n_chunks; ++c) {
    const Item h = item_geometry<W, WH>(p, c, n);
    if (h.x0 >= x + W) break;
    const uint32_t limit = (1u << 18) + 16u * (uint32_t)min(n, 1 << 23);
    bool done = false;
    for (uint32_t it = 0; it < limit && !done; ++it) {
      int32_t v;
      asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(&p.halo_read[item - (c - chunk)]) : "memory");
      done = __all_sync(FULL_MASK, v >= h.nh);
      if (!done) {
        if (__any_sync(FULL_MASK, ld_shared_volatile(abort_addr) != 0)) return false;
        __nanosleep(100);
      }
    }
    if (!done) return false;
  }
  return true;
}

__device__ __forceinline__ uint64_t ld_shared_u64(uint32_t addr) {
  uint64_t v;
  asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared_u64(uint32_t addr, uint64_t v) {
  asm volatile("st.volatile.shared.u64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}

// ---------------------------------------------------------------- one strip

// What a strip's sweep is given besides its columns (all warp-uniform).
struct Strip {
  int64_t x;         // first column
  int rows;          // rows to sweep: n, or fewer in a halo strip
  int n;             // rows of the read
  int strand;
  bool first;        // leftmost strip of its item
  bool resume;
  const float *q;
  const float *st_plane0;
  uint32_t seq;      // its place in the CTA's sequence
  char *in_b, *out_b;          // seam columns of the left neighbour and of this strip
  uint32_t prog_in, prog_out;  // their progress words
};

// Sweeps SC cells per lane through the strip's rows; the last row is left in
// D, its frame in O.  False when a wait gave up.
template <int SC, int PREC, bool ST16, typename OnLoaded>
__device__ __forceinline__ bool sweep_strip(const SdtwParams &p, const Strip &st, typename Pol<PREC>::V (&D)[SC],
                                            float2 &O, int lane, uint32_t m0, uint32_t is31, uint32_t wb,
                                            const unsigned char *slot, uint64_t *bar, uint32_t &phase,
                                            uint32_t spin_limit, uint32_t abort_addr, OnLoaded on_loaded) {
  using P = Pol<PREC>;
  using V = typename P::V;
  using RV = typename P::RV;
  constexpr int RB = P::RB;           // reference bytes per column
  constexpr int NW = SC * RB / 4;     // reference words per lane
  constexpr int K = kRescaleRows;
  // rows per group of the window loop, and how their seam cells leave it, by
  // what the instruction schedule measured (64 strips of one read per item,
  // Tcell/s): FP16 pairs, 4 rows and one 16-byte store 18.1, a store per row
  // 15.2, 2 rows 15.8; FP32, 4 rows and a store per row 12.9, one 16-byte
  // store 12.6, 2 rows 12.6; MIXED, 2 rows and a store per row 13.4, 4 rows 12.9
  constexpr int kRows = PREC == 2 ? 2 : 4;
  const int n = st.n, rows = st.rows;
  const bool first = st.first;
  const float *q = st.q;
  const int64_t off_pos = seam_offsets_pos(4, p.max_rows);
  const V *seam_in = reinterpret_cast<const V *>(st.in_b);
  const float2 *off_in = reinterpret_cast<const float2 *>(st.in_b + off_pos);
  V *seam_out = reinterpret_cast<V *>(st.out_b);
  float2 *off_out = reinterpret_cast<float2 *>(st.out_b + off_pos);

  // -- initial row ("row -1"): zeros (free start) or the saved row state
  O = make_float2(0.f, 0.f);  // FP16 frame offsets (fwd, rev)
  if (st.resume) {
    load_row_state<SC, PREC, ST16>(D, O, st.st_plane0, p.m_pad, st.strand, st.x + (int64_t)lane * SC);
    on_loaded();
  } else {
#pragma unroll
    for (int k = 0; k < SC; ++k) D[k] = P::zero();
  }

  // -- reference strip into registers (after the row state: fewer live registers)
  RV R[NW];
  // column offset of this item's strand in a planar reference (FP32 planes, or MIXED FP16 planes)
  const int64_t ref_plane = (PREC == 2 || (PREC == 1 && p.ref_layout == 1)) ? (int64_t)st.strand * p.m_pad : 0;
  if (p.use_tma) {
    // every lane waits (acquire of the TMA bytes); the give-up decision is warp-uniform
    if (!__all_sync(FULL_MASK, mbar_wait(bar, phase, spin_limit))) return false;
    phase ^= 1u;
    regs_from_smem<NW, RV>(slot, lane, R);
    __syncwarp();
  } else if constexpr (PREC == 1) {
    if (p.ref_layout == 0)
      regs_from_pairs<SC>(reinterpret_cast<const float2 *>(p.ref_plain), st.x, p.m_pad, lane, st.strand, R);
    else
      regs_from_global<NW, RV>(reinterpret_cast<const float *>(p.ref_plain) + ref_plane + st.x, lane, R);
  } else if constexpr (PREC == 2) {
    regs_from_global<NW, RV>(reinterpret_cast<const __half *>(p.ref_plain) + ref_plane + st.x, lane, R);
  } else {
    regs_from_global<NW, RV>(reinterpret_cast<const __half2 *>(p.ref_plain) + st.x, lane, R);
  }

  // uniform stores (every lane writes the same value): no lane-dependent branch
  seam_out[0] = P::shfl(D[SC - 1], 31);
  if constexpr (PREC == 0) off_out[0] = O;

  // the left neighbour's first window: seam rows -1 .. 31, offsets 0 and 1
  const uint64_t tag_in = (uint64_t)st.seq << 32;
  if (!first && !team_wait(st.prog_in, tag_in | 1u, abort_addr, n)) return false;

  // -- row sweep, 32 rows per window.  The window's query samples, its incoming
  // seam values (already re-based into this strip's frame; delta changes only
  // at a rescale, which ends a window) and its outgoing ones pass through three
  // 128-byte shared buffers: four rows take one 16-byte broadcast load of each
  // and one 16-byte store by lane 31, where a shuffle per row and value cost
  // four times as many issue slots.
  const V vinf = P::inf();
  uint32_t qb = qw_bits<PREC>(lane < n ? q[lane] : 0.f);
  V swin = (!first && lane < rows) ? seam_in[lane] : vinf;
  if constexpr (PREC == 0) {
    // re-base by the offset of the left strip's frame relative to this strip's
    const float2 oi = first ? O : off_in[0];
    swin = __hadd2(swin, __float22half2_rn(make_float2(oi.x - O.x, oi.y - O.y)));
  }
  V *so = seam_out + 1;  // seam value of row i goes to seam_out[i + 1]
  uint32_t win = 0;      // windows complete
  for (int i0 = 0; i0 < rows; i0 += kWarp) {
    st_shared_u32(wb + 4u * (uint32_t)lane, qb);
    st_shared_u32(wb + 128u + 4u * (uint32_t)lane, cell_bits<PREC>(swin));
    __syncwarp();
    // the next window's seam values come from the left neighbour's next window.
    // FP32 cells fetch them ahead of this window's rows if it is complete by now;
    // FP16 and MIXED fetch them after the rows (the registers that would hold them
    // cost the rows more: 16.8 against 18.1 and 12.6 against 13.4 Tcell/s)
    const int r = i0 + kWarp + lane;
    const bool more = !first && i0 + kWarp < rows;
    const bool ahead = PREC == 1 && more && team_ready(st.prog_in, tag_in | (win + 2));
    V sn = vinf;
    float2 off_next = O;
    if (ahead && r < rows) sn = seam_in[r];
    V sout;
    if (rows - i0 >= kWarp) {
      if constexpr (PREC == 0) {
#pragma unroll 1
        for (int g = 0; g < kWarp / 4; ++g) {
          const uint4 qv = ld_shared_v4(wb + 16u * (uint32_t)g), sv = ld_shared_v4(wb + 128u + 16u * (uint32_t)g);
          uint4 ov;
          row<SC, PREC>(D, R, qw_from<PREC>(qv.x), P::from_bits(sv.x), m0);
          ov.x = cell_bits<PREC>(D[SC - 1]);
          row<SC, PREC>(D, R, qw_from<PREC>(qv.y), P::from_bits(sv.y), m0);
          ov.y = cell_bits<PREC>(D[SC - 1]);
          row<SC, PREC>(D, R, qw_from<PREC>(qv.z), P::from_bits(sv.z), m0);
          ov.z = cell_bits<PREC>(D[SC - 1]);
          row<SC, PREC>(D, R, qw_from<PREC>(qv.w), P::from_bits(sv.w), m0);
          ov.w = cell_bits<PREC>(D[SC - 1]);
          st_shared_v4_if(wb + 256u + 16u * (uint32_t)g, ov, is31);
        }
      } else {
#pragma unroll 1
        for (int g = 0; g < kWarp; g += kRows) {
          uint32_t qv[kRows], sv[kRows];
          ld_shared_words(wb + 4u * (uint32_t)g, qv);
          ld_shared_words(wb + 128u + 4u * (uint32_t)g, sv);
#pragma unroll
          for (int j = 0; j < kRows; ++j) {
            row<SC, PREC>(D, R, qw_from<PREC>(qv[j]), P::from_bits(sv[j]), m0);
            st_shared_if(wb + 256u + 4u * (uint32_t)(g + j), cell_bits<PREC>(D[SC - 1]), is31);
          }
        }
      }
      __syncwarp();
      sout = P::from_bits(ld_shared_u32(wb + 256u + 4u * (uint32_t)lane));
      if constexpr (PREC == 0) {
        // rescale: subtract this strip's row minimum (one epoch = 32 rows)
        // (four partial minima: a single chain of SC dependent minima would
        // stall the warp once per window)
        V mq[4] = {D[0], D[1], D[2], D[3]};
#pragma unroll
        for (int k = 4; k < SC; ++k) mq[k & 3] = __hmin2(mq[k & 3], D[k]);
        V mn = __hmin2(__hmin2(mq[0], mq[1]), __hmin2(mq[2], mq[3]));
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) mn = __hmin2(mn, P::shfl_xor(mn, m));
#pragma unroll
        for (int k = 0; k < SC; ++k) D[k] = __hsub2(D[k], mn);
        const float2 mf = __half22float2(mn);
        O.x += mf.x;
        O.y += mf.y;
        const int e = (i0 + kWarp) / K;
        off_out[e] = O;  // warp-uniform value, stored by every lane
        sout = P::sel(lane == kWarp - 1, D[SC - 1], sout);  // the seam leaves in the new frame
      }
      so[lane] = sout;
    } else {
      const int cnt = rows - i0;
      for (int il = 0; il < cnt; ++il) {
        row<SC, PREC>(D, R, qw_from<PREC>(ld_shared_u32(wb + 4u * (uint32_t)il)),
                      P::from_bits(ld_shared_u32(wb + 128u + 4u * (uint32_t)il)), m0);
        st_shared_if(wb + 256u + 4u * (uint32_t)il, cell_bits<PREC>(D[SC - 1]), is31);
      }
      __syncwarp();
      // lanes >= cnt write +inf into the buffer's 32-entry slack past the rows
      so[lane] = lane < cnt ? P::from_bits(ld_shared_u32(wb + 256u + 4u * (uint32_t)lane)) : vinf;
    }
    so += kWarp;
    // (the samples' load goes out before the publish for FP16 pairs, 3 % on narrow
    // chunks, and after it for the others, 4 % on FP32)
    float qn = 0.f;
    if constexpr (PREC == 0) qn = r < n ? q[r] : 0.f;
    ++win;
    team_publish(st.prog_out, st.seq, win);
    if (more && !ahead) {
      if (!team_wait(st.prog_in, tag_in | (win + 1), abort_addr, n)) return false;
      if (r < rows) sn = seam_in[r];
      if constexpr (PREC == 0) off_next = off_in[win];
    }
    if constexpr (PREC != 0) qn = r < n ? q[r] : 0.f;
    qb = qw_bits<PREC>(qn);
    swin = sn;
    if constexpr (PREC == 0) {
      if (!first) swin = __hadd2(swin, __float22half2_rn(make_float2(off_next.x - O.x, off_next.y - O.y)));
    }
  }
  if (rows < n) {
    // rows this halo strip skipped can no longer reach column a: keep them
    // inert (whole 32-entry groups; the buffers have 32 entries of slack)
    for (int rr = rows + 1; rr <= n; rr += kWarp) seam_out[rr + lane] = vinf;
    if constexpr (PREC == 0) {
      for (int e = rows / K + 1; e <= n / K; e += kWarp) off_out[e + lane] = O;
    }
  }
  return true;
}

// The NO_REF_DEL sweep.  (The REF_DEL recurrence runs the anti-diagonal
// kernels of refdel.cu.)
// ST16: FP16 cells whose serving row state is FP16 (p.state_fp16); a separate
// instance, so the other instances carry none of its registers.
// NH: halo strips kNarrowHaloCells wide (FP16 pairs, p.narrow_halo).
// ORDERED: dealt batches that resume and save rows.  Their items wait for items
// of lower number (wait_halo_readers), so a CTA's number is a ticket, taken when
// it starts, and its items are consecutive: whatever it waits for is its own or
// belongs to a CTA that started before it, and the wait ends even while another
// kernel keeps the remaining CTAs off the GPU.  An instance of its own: its few
// registers cost the others' rows 2 % (192 FP32 reads of 2,000 samples against
// 1 Mb: 61.0 ms, 62.1 with it).
template <int S, int PREC, bool ST16, bool NH, bool ORDERED>
__global__ void __maxnreg__((sdtw_reg_cap<S, PREC>())) sdtw_kernel(
    const __grid_constant__ CUtensorMap tmap, const SdtwParams p) {
  using P = Pol<PREC>;
  using V = typename P::V;
  constexpr bool PAIRS = PREC == 0;           // both strands in one cell (FP16)
  constexpr int W = kWarp * S;                // columns per strip
  constexpr int RB = P::RB;                   // reference bytes per column
  constexpr int STRIP_BYTES = W * RB;
  constexpr int SH = NH ? kNarrowHaloCells : S;  // cells per lane in halo strips
  constexpr int WH = kWarp * SH;
  // dealt batches (p.deal): not in the FP16 instance of wide chunks, which has
  // many items and whose rows lose 6 % to the registers of the first round
  constexpr bool DEAL = PREC != 0 || NH;
  static_assert(S % SH == 0 && SH % 8 == 0, "halo strips must tile the chunk start");
  static_assert(!ORDERED || DEAL, "only a dealt batch has an order of CTAs");
  static_assert(!NH || PREC == 0, "narrow halo strips are built for FP16 pairs");
  static_assert(STRIP_BYTES % 1024 == 0, "strip tile must keep 1024-byte alignment");
  static_assert(S % 8 == 0, "row state and reference move in 16-byte groups");
  static_assert(!ST16 || PREC == 0, "the FP16 row state is built for FP16 cells");

  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  const uint32_t m0 = lane0_mask(lane);
  // per warp: a reference strip tile, its mbarrier and three 128-byte windows
  // (query samples, seam in, seam out); per CTA: the team's state and
  // two progress words a warp
  unsigned char *const slot = smem + warp * STRIP_BYTES;
  uint64_t *const bar = reinterpret_cast<uint64_t *>(smem + nwarps * STRIP_BYTES) + 2 * warp;
  const uint32_t wb = smem_u32(smem + nwarps * (STRIP_BYTES + 16)) + 384u * (uint32_t)warp;
  unsigned char *const team_p = smem + nwarps * (STRIP_BYTES + 16 + 384);
  const uint32_t team = smem_u32(team_p);
  const uint32_t prog = team + kTeamStateBytes;
  const int nbuf = p.seam_buffers ? p.seam_buffers : 2 * nwarps;
  uint32_t is31 = lane == kWarp - 1 ? 1u : 0u;
  asm volatile("mov.b32 %0, %0;" : "+r"(is31));  // opaque to the optimiser, like lane0_mask

  const uint32_t is0 = m0 & 1u;  // 1 on lane 0 (opaque to the optimiser)
  if (p.use_tma) {
    mbar_init_if(bar, 1, is0);
    fence_mbar_init();
  }
  for (int i = threadIdx.x; i < (int)kTeamStateBytes / 4 + 4 * nwarps; i += blockDim.x)
    reinterpret_cast<uint32_t *>(team_p)[i] = 0;
  __syncthreads();
  uint32_t phase = 0;  // parity of the tile's next completion

  const uint32_t lock_a = team, abort_a = team + 4, item_a = team + 8, next_a = team + 12, total_a = team + 16,
                 seq_a = team + 20, dealt_a = team + 24, end_a = team + 28;
  const int64_t seam_half = p.seam_stride / 2;
  char *const seam_base = p.seam + (int64_t)blockIdx.x * nbuf * seam_half;
  // FP32 and MIXED split each (task, chunk) into one work item per strand
  const int nstr = !PAIRS ? (p.strands > 0 ? p.strands : 2) : 1;
  const int per_task = p.n_chunks * nstr;
  const int64_t n_items = (int64_t)p.n_tasks * per_task;
  const uint32_t spin_limit = p.spin_limit ? p.spin_limit : kSpinLimit;

  // Strips of an item (none of one with nothing to do or that is refused).
  const auto item_strips = [&](int item) -> int {
    const int tr = item / per_task;
    const int n = p.tasks[p.order ? p.order[tr] : tr].n;
    if (n <= 0 || n > p.max_rows) {
      if (n > p.max_rows) atomicOr(p.err, kErrBadTask);  // every lane: same bit
      return 0;
    }
    const int rem = item - tr * per_task;
    return item_geometry<W, WH>(p, p.n_chunks - 1 - (!PAIRS ? rem % p.n_chunks : rem), n).nstrips;
  };

  // A dealt batch's first round: warp w takes the strip that p.deal_warps
  // gives it, walking the CTA's items to find it; the warp with the last one
  // leaves the cursor behind it.
  // FP16 pairs keep it in the word beside the warp's mbarrier: in registers it
  // lived through every row (4 reads of 1,600 samples against 5 Mb: 4.26 to
  // 4.22 ms).  FP32 and MIXED keep it in registers, which their schedule
  // takes better (192 reads of 2,000 samples against 1 Mb: 60.8 and 58.4 ms,
  // 61.4 and 59.2 through shared memory); an ordered deal of MIXED cells takes
  // the word better (three steps of a read of 1,600 samples a step against
  // 120 kb: 577 us, 633 in registers).
  constexpr bool FIRST_SHARED = PREC == 0 || (ORDERED && PREC == 2);
  const uint32_t first_a = smem_u32(bar + 1);
  if constexpr (DEAL && FIRST_SHARED) st_shared_u64(first_a, 0);
  int first_item = -1, first_s = 0;
  uint32_t first_seq = 0;
  if constexpr (ORDERED) {
    if (warp == 0) {
      const int64_t cta = __shfl_sync(FULL_MASK, ticket_if(p.counter, is0), 0);
      st_shared_volatile(dealt_a, (uint32_t)(cta * n_items / gridDim.x));
      st_shared_volatile(end_a, (uint32_t)((cta + 1) * n_items / gridDim.x));
    }
    __syncthreads();
  }
  if (DEAL && (ORDERED || p.deal)) {
    int pos = 0;
    while (pos < 15 && (int)((p.deal_warps >> (4 * pos)) & 15u) != warp) ++pos;
    int at = 0, total = 0, dealt = 0;
    int64_t item = blockIdx.x, end = n_items;
    int step = gridDim.x;
    if constexpr (ORDERED) {
      item = ld_shared_volatile(dealt_a);
      end = ld_shared_volatile(end_a);
      step = 1;
      __syncthreads();  // (every warp has read the first item)
    }
    for (; item < end; item += step) {
      ++dealt;
      total = item_strips((int)item);
      if (pos < at + total) break;
      at += total;
    }
    if (item < end) {
      first_item = (int)item;
      first_s = pos - at;
      first_seq = (uint32_t)pos;
    } else {
      first_item = (int)n_items;  // fewer strips than warps
    }
    if (pos == nwarps - 1) {
      st_shared_volatile(item_a, (uint32_t)first_item);
      st_shared_volatile(next_a, (uint32_t)(first_s + 1));
      st_shared_volatile(total_a, (uint32_t)total);
      st_shared_volatile(seq_a, (uint32_t)nwarps);
      st_shared_volatile(dealt_a, (uint32_t)(ORDERED ? item + 1 : dealt));
    }
    if constexpr (FIRST_SHARED)  // (strips of a first round: at most 16)
      st_shared_u64(first_a, (uint64_t)(0x80000000u | first_seq << 8 | (uint32_t)first_s) << 32 | (uint32_t)first_item);
    __syncthreads();
  }

  for (;;) {
    // -- the next strip of the CTA's sequence, under the team's lock.  Every
    // lane runs the same instructions (only the atomics are lane 0's).
    int item = -1, s = 0;
    uint32_t seq = 0;
    if constexpr (DEAL && !FIRST_SHARED) {
      item = first_item, s = first_s, seq = first_seq;
      first_item = -1;
    } else if constexpr (DEAL) {
      const uint64_t f = ld_shared_u64(first_a);
      if (f) {
        item = (int)(uint32_t)f;
        s = (int)(f >> 32 & 0xff);
        seq = (uint32_t)(f >> 40 & 0xff);
        __syncwarp();
        st_shared_u64(first_a, 0);
      }
    }
    if (item < 0) {
      if (!team_lock(lock_a, abort_a, is0)) {
        atomicOr(p.err, kErrWaitTimeout);  // every lane: same bit
        st_shared_volatile(abort_a, 1);
        return;
      }
      item = (int)ld_shared_volatile(item_a);
      s = (int)ld_shared_volatile(next_a);
      int total = (int)ld_shared_volatile(total_a);
      seq = ld_shared_volatile(seq_a);
      while (s >= total && item < n_items) {
        if constexpr (ORDERED) {
          item = (int)ld_shared_volatile(dealt_a);
          if (item >= (int)ld_shared_volatile(end_a)) item = (int)n_items;
          __syncwarp();
          st_shared_volatile(dealt_a, (uint32_t)(item + 1));
          __syncwarp();
        } else if (DEAL && p.deal) {
          const uint32_t dealt = ld_shared_volatile(dealt_a);
          item = (int)(blockIdx.x + dealt * gridDim.x);
          __syncwarp();
          st_shared_volatile(dealt_a, dealt + 1);
          __syncwarp();
        } else {
          item = __shfl_sync(FULL_MASK, ticket_if(p.counter, is0), 0);
        }
        if (item >= n_items) break;
        s = 0;
        total = item_strips(item);
      }
      __syncwarp();
      st_shared_volatile(item_a, (uint32_t)(item < n_items ? item : (int)n_items));
      st_shared_volatile(next_a, (uint32_t)(s + 1));
      st_shared_volatile(total_a, (uint32_t)total);
      st_shared_volatile(seq_a, seq + 1);
      team_unlock(lock_a);
    }
    if (item >= n_items) break;

    const int tr = item / per_task;
    const int rem = item - tr * per_task;
    // Chunks go from right to left: a resumed chunk's halo reads the saved row
    // of the columns to its left before their own chunks overwrite it.
    const int strand = !PAIRS ? rem / p.n_chunks : 0;
    const int chunk = p.n_chunks - 1 - (rem - strand * p.n_chunks);
    const Task t = p.tasks[p.order ? p.order[tr] : tr];
    const int n = t.n;
    const Item g = item_geometry<W, WH>(p, chunk, n);
    const bool save = (t.flags & kTaskSaveState) != 0 && p.state != nullptr;
    const bool halo = s < g.nh;  // left of column a: no result

    Strip st;
    st.x = halo ? g.x0 + (int64_t)s * WH : g.a + (int64_t)(s - g.nh) * W;
    st.n = n;
    st.rows = n;
    if (halo) {
      // rows that can still reach column a
      const int64_t lim = (int64_t)n - 1 - (g.a - st.x - WH);
      st.rows = (int)(lim < 0 ? 0 : (lim > n ? n : lim));
    }
    st.strand = strand;
    st.first = s == 0;
    st.resume = (t.flags & kTaskResume) != 0;
    st.q = p.query + t.q_off;
    // planar row state: strand s of this read at state + state_off + s*m_pad
    st.st_plane0 = p.state ? p.state + t.state_off : nullptr;
    st.seq = seq;
    const uint32_t buf = seq % (uint32_t)nbuf;
    const uint32_t buf_in = buf ? buf - 1 : (uint32_t)nbuf - 1;
    st.out_b = seam_base + buf * seam_half;
    st.in_b = seam_base + buf_in * seam_half;
    st.prog_out = prog + 8 * buf;
    st.prog_in = prog + 8 * buf_in;

    // the buffer's last writer and its reader (the strip after it) must be
    // done; the reader may end first, where it begins another item
    bool ok = true;
    if (seq >= (uint32_t)nbuf) {
      const uint32_t last = seq - (uint32_t)nbuf;
      ok = team_wait(st.prog_out, ((uint64_t)(last + 1) << 32) | kStripDone, abort_a, p.max_rows) &&
           team_wait(prog + 8 * ((buf + 1) % (uint32_t)nbuf), ((uint64_t)(last + 2) << 32) | kStripDone, abort_a,
                     p.max_rows);
    }
    if (ok && p.use_tma) {
      // the test hook p.stall_item withholds this copy (and its arrival) for
      // one item's first strip: the wait for it then runs out with no copy in flight
      const int64_t ref_plane = (PREC == 2 || (PREC == 1 && p.ref_layout == 1)) ? (int64_t)strand * p.m_pad : 0;
      fence_proxy_async_smem();
      tma_issue_if(slot, &tmap, bar, 0, (int)((ref_plane + st.x) * RB / 128), STRIP_BYTES,
                   is0 & (s > 0 || item + 1 != p.stall_item ? 1u : 0u));
    }
    // a resumed halo strip counts itself in once it has read its row state
    const auto on_loaded = [&]() {
      if (halo && p.halo_read) {
        __threadfence();
        __syncwarp();
        red_add_if(&p.halo_read[item], 1, is0);
      }
    };

    bool swept = false;
    if constexpr (SH != S) {
      if (halo) {
        V D[SH];
        float2 O;
        if (ok)
          ok = sweep_strip<SH, PREC, ST16>(p, st, D, O, lane, m0, is31, wb, slot, bar, phase, spin_limit,
                                                  abort_a, on_loaded);
        swept = true;
      }
    }
    if (!swept) {
      V D[S];
      float2 O;
      if (ok)
        ok = sweep_strip<S, PREC, ST16>(p, st, D, O, lane, m0, is31, wb, slot, bar,
                                                                    phase, spin_limit, abort_a, on_loaded);
      if (ok && !halo) {
        const int64_t c0 = st.x + (int64_t)lane * S;
        float bestx = __int_as_float(0x7f800000), besty = bestx;
        int64_t colx = -1, coly = -1;
#pragma unroll
        for (int k = 0; k < S; ++k) {
          const int64_t col = c0 + k;
          if constexpr (PREC == 0) {
            const float2 v = __half22float2(D[k]);
            const float vx = v.x + O.x, vy = v.y + O.y;
            if (col < g.b) {
              if (vx < bestx) { bestx = vx; colx = col; }
              if (vy < besty) { besty = vy; coly = col; }
            }
          } else {
            if (col < g.b && D[k] < bestx) { bestx = D[k]; colx = col; }
          }
        }
        if (save) {
          // wait for the halo strips of the chunks to the right that start from
          // this strip's saved row (handed out before this chunk)
          if (p.halo_read && st.resume) ok = wait_halo_readers<W, WH>(p, g, st.x, item, chunk, n, abort_a);
          if (ok)
            save_row_state<S, PREC, ST16>(D, O, p.state + t.state_off, p.m_pad, strand, c0);
        }
        warp_argmin(bestx, colx);
        const int64_t base = 2 * (int64_t)t.out_slot;
        if constexpr (PREC == 0) {
          warp_argmin(besty, coly);
          red_min_if(&p.keys[base + 0], make_key(bestx, colx), is0 & (colx >= 0 ? 1u : 0u));
          red_min_if(&p.keys[base + 1], make_key(besty, coly), is0 & (coly >= 0 ? 1u : 0u));
        } else {
          red_min_if(&p.keys[base + strand], make_key(bestx, colx), is0 & (colx >= 0 ? 1u : 0u));
        }
      }
    }
    if (!ok) {
      atomicOr(p.err, kErrWaitTimeout);  // every lane: same bit
      st_shared_volatile(abort_a, 1);
      return;
    }
    team_publish(st.prog_out, seq, kStripDone);
  }
}

// ---------------------------------------------------------------- instances / launch

// Lets an instance take the shared memory of its largest CTA.  The limit belongs
// to the function on the device, not to a launch: every caller sets the same
// value, so that threads with CTAs of different sizes do not take it from each
// other between their call here and their launch.
constexpr int kMostWarps = 16;
template <int S, int PREC, typename F>
static cudaError_t allow_smem(F fn) {
  static_assert(kMostWarps * (kWarp * S * Pol<PREC>::RB + 512) + 2048 <= 227 * 1024, "shared memory of an SM");
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)sdtw_smem_bytes(PREC, S, kMostWarps));
}

template <int S, int PREC, bool ST16 = false, bool NH = false, bool ORDERED = false>
static cudaError_t launch_inst(int warps, int grid, const SdtwParams &p, const CUtensorMap *tmap,
                               cudaStream_t s) {
  constexpr bool kDeals = PREC != 0 || NH;
  if constexpr (kDeals && !ORDERED) {
    if (p.deal && p.halo_read) return launch_inst<S, PREC, ST16, NH, true>(warps, grid, p, tmap, s);
  }
  const size_t smem = sdtw_smem_bytes(PREC, S, warps);
  auto fn = sdtw_kernel<S, PREC, ST16, NH, ORDERED>;
  const cudaError_t e = allow_smem<S, PREC>(fn);
  if (e != cudaSuccess) return e;
  CUtensorMap dummy;
  if (!tmap) {
    memset(&dummy, 0, sizeof(dummy));
    tmap = &dummy;
  }
  fn<<<grid, warps * kWarp, smem, s>>>(*tmap, p);
  return cudaGetLastError();
}

template <int S, int PREC, bool ST16 = false, bool NH = false>
static int occ_inst(int warps) {
  int n = 0;
  const size_t smem = sdtw_smem_bytes(PREC, S, warps);
  auto fn = sdtw_kernel<S, PREC, ST16, NH, false>;
  if (allow_smem<S, PREC>(fn) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, warps * kWarp, smem) != cudaSuccess) return 0;
  return n;
}

int sdtw_pair_bytes(int precision, bool ref_del) {
  // the FP16-pair REF_DEL kernel passes its seam column as absolute FP32 pairs
  return precision == 0 && ref_del ? 8 : 4;
}

int sdtw_ref_bytes(int precision) { return precision == 2 ? 2 : 4; }

size_t sdtw_smem_bytes(int precision, int cells_per_thread, int warps_per_cta) {
  const size_t strip = (size_t)kWarp * cells_per_thread * sdtw_ref_bytes(precision);
  // per warp: a strip tile, its mbarrier (16 bytes), three windows, two progress words; per CTA: the team's state
  return 1024 /* alignment slack */ + warps_per_cta * (strip + 16 + 384 + 16) + kTeamStateBytes;
}

bool sdtw_instance_exists(int precision, int S, bool ref_del) {
  if (ref_del) return (precision == 1 && (S == 16 || S == 32)) || (precision == 0 && S == 32);
  if (precision == 0) return S == 32 || S == 48;
  if (precision == 2) return S == 32 || S == 48 || S == 64;
  return S == 16 || S == 32 || S == 48;
}

#define DTWX_DISPATCH(PREC, S, CALL) \
  if (precision == PREC && cells_per_thread == S) return CALL<S, PREC>
#define DTWX_DISPATCH_ST16(S, CALL) \
  if (precision == 0 && cells_per_thread == S) return CALL<S, 0, true>
#define DTWX_DISPATCH_NH(S, ST16, CALL) \
  if (precision == 0 && cells_per_thread == S) return CALL<S, 0, ST16, true>

cudaError_t launch_sdtw(int precision, int cells_per_thread, int warps_per_cta, int grid,
                        const SdtwParams &p, const CUtensorMap *tmap, cudaStream_t s) {
  if (p.ref_del) {
    // the anti-diagonal kernels of refdel.cu
    return launch_refdel(precision, cells_per_thread, warps_per_cta, grid, p, s);
  }
  if (p.narrow_halo) {
    if (p.state_fp16) {
      DTWX_DISPATCH_NH(32, true, launch_inst)(warps_per_cta, grid, p, tmap, s);
      DTWX_DISPATCH_NH(48, true, launch_inst)(warps_per_cta, grid, p, tmap, s);
    } else {
      DTWX_DISPATCH_NH(32, false, launch_inst)(warps_per_cta, grid, p, tmap, s);
      DTWX_DISPATCH_NH(48, false, launch_inst)(warps_per_cta, grid, p, tmap, s);
    }
    return cudaErrorInvalidValue;
  }
  if (p.state_fp16) {
    DTWX_DISPATCH_ST16(32, launch_inst)(warps_per_cta, grid, p, tmap, s);
    DTWX_DISPATCH_ST16(48, launch_inst)(warps_per_cta, grid, p, tmap, s);
    return cudaErrorInvalidValue;
  }
  DTWX_DISPATCH(0, 32, launch_inst)(warps_per_cta, grid, p, tmap, s);
  DTWX_DISPATCH(0, 48, launch_inst)(warps_per_cta, grid, p, tmap, s);
  DTWX_DISPATCH(1, 16, launch_inst)(warps_per_cta, grid, p, tmap, s);
  DTWX_DISPATCH(1, 32, launch_inst)(warps_per_cta, grid, p, tmap, s);
  DTWX_DISPATCH(1, 48, launch_inst)(warps_per_cta, grid, p, tmap, s);
  DTWX_DISPATCH(2, 32, launch_inst)(warps_per_cta, grid, p, tmap, s);
  DTWX_DISPATCH(2, 48, launch_inst)(warps_per_cta, grid, p, tmap, s);
  DTWX_DISPATCH(2, 64, launch_inst)(warps_per_cta, grid, p, tmap, s);
  return cudaErrorInvalidValue;
}

static int query_ctas_per_sm(int precision, int cells_per_thread, int warps_per_cta, bool ref_del) {
  if (ref_del) {
    return refdel_ctas_per_sm(precision, cells_per_thread, warps_per_cta);
  }
  DTWX_DISPATCH(0, 32, occ_inst)(warps_per_cta);
  DTWX_DISPATCH(0, 48, occ_inst)(warps_per_cta);
  DTWX_DISPATCH(1, 16, occ_inst)(warps_per_cta);
  DTWX_DISPATCH(1, 32, occ_inst)(warps_per_cta);
  DTWX_DISPATCH(1, 48, occ_inst)(warps_per_cta);
  DTWX_DISPATCH(2, 32, occ_inst)(warps_per_cta);
  DTWX_DISPATCH(2, 48, occ_inst)(warps_per_cta);
  DTWX_DISPATCH(2, 64, occ_inst)(warps_per_cta);
  return 0;
}

// A property of the compiled instance on this GPU model, asked several times
// per call while a shape is picked: the occupancy API is asked once.
int sdtw_ctas_per_sm(int precision, int cells_per_thread, int warps_per_cta, bool ref_del) {
  static std::atomic<int8_t> known[2][3][5][kMostWarps + 1];  // 0: not asked yet, else 1 + CTAs
  const int c = cells_per_thread / 16;
  if (precision < 0 || precision > 2 || c < 1 || c > 4 || cells_per_thread != 16 * c || warps_per_cta < 1 ||
      warps_per_cta > kMostWarps)
    return 0;
  std::atomic<int8_t> &k = known[ref_del ? 1 : 0][precision][c][warps_per_cta];
  int8_t v = k.load(std::memory_order_relaxed);
  if (v == 0) {
    v = (int8_t)(1 + std::min(query_ctas_per_sm(precision, cells_per_thread, warps_per_cta, ref_del), 100));
    if (v > 1) k.store(v, std::memory_order_relaxed);  // (an error is asked again)
  }
  return v - 1;
}

// ---------------------------------------------------------------- issue-rate probe
// Runs only the cell update of the sweep (sub, min, fma over a register row of
// 32 pairs, next row from the previous one) with no shuffles, seams or memory:
// the instruction-issue ceiling of the recurrence on this device.

template <int PREC>
__device__ __forceinline__ typename Pol<PREC>::V probe_value(float a, float b) {
  if constexpr (PREC == 0)
    return __floats2half2_rn(a, b);
  else
    return a;
}

// MIXED: the same row with half2 reference pairs and FP32 cells.
__global__ void __launch_bounds__(256) peak_probe_mixed_kernel(int iters, float *sink) {
  constexpr int S = 32;
  __half2 R[S / 2];
  float D[S];
  const float t = (float)(threadIdx.x & 7) * 0.01f;
#pragma unroll
  for (int k = 0; k < S / 2; ++k) R[k] = __floats2half2_rn(t + 0.06f * k, t - 0.042f * k);
#pragma unroll
  for (int k = 0; k < S; ++k) D[k] = 0.f;
  float qf = 0.25f + t;
  for (int it = 0; it < iters; ++it) {
    const __half2 qq = __float2half2_rn(qf);
#pragma unroll
    for (int k = S / 2 - 1; k >= 0; --k) {
      const __half2 d = __hsub2(R[k], qq);
      D[2 * k + 1] = fma_sq_f16(__high2half(d), fminf(D[2 * k + 1], D[2 * k]));
      D[2 * k] = fma_sq_f16(__low2half(d), fminf(D[2 * k], k > 0 ? D[2 * k - 1] : D[S - 1]));
    }
    qf = fmaf(qf, 0.999f, 0.0137f);
  }
  float acc = D[0];
#pragma unroll
  for (int k = 1; k < S; ++k) acc = fminf(acc, D[k]);
  if (acc == 12345.678f) sink[threadIdx.x] = acc;
}

template <int PREC>
__global__ void __launch_bounds__(256) peak_probe_kernel(int iters, float *sink) {
  using P = Pol<PREC>;
  using V = typename P::V;
  constexpr int S = 32;
  V R[S], D[S];
  const float t = (float)(threadIdx.x & 7) * 0.01f;
#pragma unroll
  for (int k = 0; k < S; ++k) {
    R[k] = probe_value<PREC>(t + 0.03f * k, t - 0.021f * k);  // distinct strands and columns
    D[k] = P::zero();
  }
  float qf = 0.25f + t;
  for (int it = 0; it < iters; ++it) {
    const V qq = probe_value<PREC>(qf, qf);
#pragma unroll
    for (int k = S - 1; k >= 1; --k) D[k] = P::cell(R[k], qq, D[k], D[k - 1]);
    D[0] = P::cell(R[0], qq, D[0], D[S - 1]);
    // a new query sample every row, as in the sweep: (r - q)^2 cannot be hoisted
    qf = fmaf(qf, 0.999f, 0.0137f);
  }
  V acc = D[0];
#pragma unroll
  for (int k = 1; k < S; ++k) acc = P::vmin(acc, D[k]);
  float f;
  if constexpr (PREC == 0)
    f = __low2float(acc) + __high2float(acc);
  else
    f = acc;
  if (f == 12345.678f) sink[threadIdx.x] = f;  // keeps the loop alive
}

cudaError_t launch_peak_probe(int precision, int grid, int block, int iters, float *sink,
                              cudaStream_t s) {
  if (precision == 0)
    peak_probe_kernel<0><<<grid, block, 0, s>>>(iters, sink);
  else if (precision == 2)
    peak_probe_mixed_kernel<<<grid, block, 0, s>>>(iters, sink);
  else
    peak_probe_kernel<1><<<grid, block, 0, s>>>(iters, sink);
  return cudaGetLastError();
}

}  // namespace dtwx
