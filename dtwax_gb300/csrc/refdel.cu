// The REF_DEL recurrence on FP32 cells and on FP16 pairs (src/include/DTW.cu:
// 23-29, the build without -DNO_REF_DEL; scripts/sdtw.py keeps no such
// variant):
//
//   D[i][j] = (r_j - q_i)^2 + min(D[i-1][j], D[i-1][j-1], D[i][j-1])
//
// with the free start of sDTW (row -1 is zero, or the saved row of a resumed
// read) and +inf left of column 0.
//
// The left predecessor chains the cells of one row, so a warp sweeps a strip
// of 32*S columns along anti-diagonals instead of row by row:
// * lane l owns S consecutive columns and, at step t, computes rows
//   2(t - l) and 2(t - l) + 1 of them from left to right, so the horizontal
//   chain stays inside the lane;
// * the left predecessors of its first column are lane l-1's last cells of
//   the same rows, which lane l-1 computed at step t-1 (two shuffles per
//   step), and the diagonal one of the first row is the value received one
//   step earlier;
// * lane 0 takes both from the seam column of the strip to the left, and lane
//   31 writes the seam column for the strip to its right.
// Each step a lane computes two consecutive rows, interleaved (two dependency
// chains).  A cell costs one subtraction, one three-input minimum (FP16 pairs: two
// minima) and one FMA.  A strip
// takes ceil(n / 2) + 31 steps; in the first and last 31 some lanes have no
// rows and keep their cells, so after the last step every lane holds row
// n - 1.
//
// A horizontal run can cross any column, so a task is one work item (per
// strand for FP32 cells) of all its strips (the host launches it with one
// chunk).  The p.team_warps warps of a team sweep an item's strips as a
// pipeline: the strip to the right runs about 64 rows behind, fed by the seam
// column through global scratch.
//
// Query samples, incoming and outgoing seam values pass through shared memory,
// 32 rows (a window of 16 steps) at a time.
//
// FP16 pairs: one item covers both strands (fwd in .x, rev in .y).  FP16 keeps
// the path cost in range with running-minimum frames, one per lane: lane l
// holds its cells relative to a float2 offset O_l, its own minimum at the last
// rescale (the end of a window, all lanes at the same step).  A value crossing
// from lane l-1 is re-based by O_{l-1} - O_l in FP32 and rounded to FP16 at the
// magnitude of the result.  With horizontal moves allowed, neighbouring frames
// differ by at most the cost of a horizontal run, so the re-based values stay
// in range.  Lane 0 re-bases the left strip's seam column, which travels as
// absolute FP32 pairs.
#include "team.cuh"

namespace dtwx {

namespace {

constexpr int kWindowSteps = 16;             // steps (2 rows each) of a window
constexpr int kWindowRows = 2 * kWindowSteps;
constexpr int kQueryRing = 128;              // samples a warp keeps: its lanes span 64 rows, a window adds 32
constexpr int kMaxWarps = 16;                // warps of the largest CTA

// Three-input minimum of the ALU (PTX min with three operands, sm_100 and
// later): the two minima of a cell in one issue slot.  The ALU takes 2 cycles
// for either, so with two of them the cell was bound there.
__device__ __forceinline__ float min3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <int PREC> struct Cells;
template <> struct Cells<1> {  // FP32, one strand
  using V = float;
  using Seam = float;   // a seam value
  using Q = float;      // a query sample
  __device__ __forceinline__ static Q q(float x) { return x; }
  // (a packed add of two columns' differences takes one issue slot less and is
  // 3 % slower here)
  __device__ __forceinline__ static V cell(V r, Q q, V up, V diag, V left) {
    const float d = r - q;
    return fmaf(d, d, min3(up, diag, left));
  }
};
template <> struct Cells<0> {  // FP16 pairs
  using V = __half2;
  using Seam = float2;
  using Q = __half;
  __device__ __forceinline__ static Q q(float x) { return __float2half_rn(x); }
  __device__ __forceinline__ static V cell(V r, Q q, V up, V diag, V left) {
    const __half2 d = __hsub2(r, __half2half2(q));
    return __hfma2(d, d, __hmin2(__hmin2(up, diag), left));
  }
};

// One step of one lane: its S cells of two consecutive rows r and r + 1,
// left to right, interleaved.  Row r + 1's cell k needs row r's cells k and
// k - 1 and its own cell k - 1, so the two rows are two dependency chains one
// cell apart, which doubles the instruction-level parallelism of the lane.
// D holds row r - 1 on entry and the last valid row on exit.  diag0 is the
// left neighbour's cell on row r - 1, left0 / left1 on rows r / r + 1;
// left0 returns this lane's last cell of row r.  ONE: row r + 1 does not exist,
// so the cells stay on row r.
template <int PREC, int S, bool ONE>
__device__ __forceinline__ void refdel_step2(typename Cells<PREC>::V (&D)[S], const typename Cells<PREC>::V (&R)[S],
                                             typename Cells<PREC>::Q q0, typename Cells<PREC>::Q q1,
                                             typename Cells<PREC>::V diag0, typename Cells<PREC>::V &left0,
                                             typename Cells<PREC>::V left1) {
  using C = Cells<PREC>;
  using V = typename C::V;
  V diag1 = left0;
#pragma unroll
  for (int k = 0; k < S; ++k) {
    const V up = D[k];
    const V a = C::cell(R[k], q0, up, diag0, left0);
    const V b = C::cell(R[k], q1, a, diag1, left1);
    D[k] = ONE ? a : b;
    diag0 = up;
    left0 = a;
    diag1 = a;
    left1 = b;
  }
}

__device__ __forceinline__ __half2 rebase(float2 v, float2 dl) {
  return __floats2half2_rn(v.x + dl.x, v.y + dl.y);
}

template <typename T> __device__ __forceinline__ T inf_value();
template <> __device__ __forceinline__ float inf_value<float>() { return __int_as_float(0x7f800000); }
template <> __device__ __forceinline__ float2 inf_value<float2>() {
  return make_float2(inf_value<float>(), inf_value<float>());
}

// A lane's state of one strip.
template <int PREC, int S> struct Lane {
  typename Cells<PREC>::V D[S], R[S];
  typename Cells<PREC>::V last_a;     // its last cell of the pair's first row (after each step)
  typename Cells<PREC>::V diag_next;  // the left neighbour's last cell, received one step earlier
  float2 O, dl;                       // FP16: this lane's frame; what re-bases a value arriving on its left
};

// Step `st`: lane l computes row pair st - l.  q2: its two samples; s2: lane 0's
// two seam values; o2: lane 31's place for its own two.
template <int PREC, int S, bool RAMP>
__device__ __forceinline__ void refdel_step(Lane<PREC, S> &L, int st, int n, int lane,
                                            const typename Cells<PREC>::Q *q2, const typename Cells<PREC>::Seam *s2,
                                            typename Cells<PREC>::Seam *o2) {
  using V = typename Cells<PREC>::V;
  const int r = 2 * (st - lane);  // this lane's rows r, r + 1
  const auto q0 = q2[0], q1 = q2[1];
  const auto s0 = s2[0], s1 = s2[1];
  const V ua = __shfl_up_sync(FULL_MASK, L.last_a, 1);
  const V ub = __shfl_up_sync(FULL_MASK, L.D[S - 1], 1);
  V left0, left1;
  if constexpr (PREC == 0) {
    left0 = rebase(lane == 0 ? s0 : __half22float2(ua), L.dl);
    left1 = rebase(lane == 0 ? s1 : __half22float2(ub), L.dl);
  } else {
    left0 = lane == 0 ? s0 : ua;
    left1 = lane == 0 ? s1 : ub;
  }
  const V diag0 = L.diag_next;
  L.diag_next = left1;
  if constexpr (RAMP) {
    // first and last 31 steps: a lane whose rows do not exist (yet) keeps its
    // cells.  (No shuffle in here: the lanes part.)
    if ((unsigned)(r + 1) < (unsigned)n)
      refdel_step2<PREC, S, false>(L.D, L.R, q0, q1, diag0, left0, left1);
    else if ((unsigned)r < (unsigned)n)
      refdel_step2<PREC, S, true>(L.D, L.R, q0, q1, diag0, left0, left1);
    __syncwarp();
  } else {
    refdel_step2<PREC, S, false>(L.D, L.R, q0, q1, diag0, left0, left1);
  }
  L.last_a = left0;
  if (lane == kWarp - 1) {
    if constexpr (PREC == 0) {
      const float2 va = __half22float2(left0), vb = __half22float2(L.D[S - 1]);
      o2[0] = make_float2(va.x + L.O.x, va.y + L.O.y);
      o2[1] = make_float2(vb.x + L.O.x, vb.y + L.O.y);
    } else {
      o2[0] = left0;
      o2[1] = L.D[S - 1];
    }
  }
}

// 128 registers: 16 warps per SM, at the price of 40 to 60 bytes a thread spilled
// outside the steps at 32 cells per lane.  (512 reads of 2,000 samples against
// 48 kb, FP32 at 32 cells: 12.0 ms; 12.95 with 168 registers and 12 warps.)
constexpr int kRefDelRegs = 128;

template <int PREC, int S>
__global__ void __maxnreg__(kRefDelRegs) sdtw_refdel_kernel(const SdtwParams p) {
  static_assert(S % 4 == 0, "row state moves in 16-byte groups");
  using C = Cells<PREC>;
  using V = typename C::V;
  using Seam = typename C::Seam;
  using Q = typename C::Q;
  constexpr bool PAIRS = PREC == 0;
  constexpr int W = kWarp * S;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  const uint32_t is0 = lane == 0 ? 1u : 0u;
  const float inf = inf_value<float>();

  __shared__ TeamState team_state[kMaxWarps];
  __shared__ uint64_t team_prog[2 * kMaxWarps];
  __shared__ __align__(16) Q q_ring[kMaxWarps][kQueryRing];
  __shared__ __align__(16) Seam seam_win[kMaxWarps][2][kWindowRows];  // in, out
  for (int i = threadIdx.x; i < (int)(sizeof(team_state) / 4); i += blockDim.x)
    reinterpret_cast<uint32_t *>(team_state)[i] = 0;
  for (int i = threadIdx.x; i < 2 * kMaxWarps; i += blockDim.x) team_prog[i] = 0;
  __syncthreads();

  // this warp's team: its state, its 2 * k seam buffers and their progress words
  const int k = p.team_warps;
  const int my_team = warp / k;
  const uint32_t team = static_cast<uint32_t>(__cvta_generic_to_shared(&team_state[my_team]));
  const uint32_t prog = static_cast<uint32_t>(__cvta_generic_to_shared(&team_prog[2 * k * my_team]));
  const uint32_t lock_a = team, abort_a = team + 4, item_a = team + 8, next_a = team + 12, seq_a = team + 20;
  const uint32_t nbuf = 2u * (uint32_t)k;
  char *const seam_base = p.seam + ((int64_t)blockIdx.x * nwarps + my_team * k) * p.seam_stride;
  const int64_t seam_half = p.seam_stride / 2;
  Q *const qr = q_ring[warp];
  Seam *const sin_w = seam_win[warp][0];
  Seam *const out_w = seam_win[warp][1];

  const int nstr = PAIRS ? 1 : (p.strands > 0 ? p.strands : 2);
  const int64_t n_items = (int64_t)p.n_tasks * nstr;
  const int strips = (int)((p.m + W - 1) / W);
  if (warp % k == 0) st_shared_volatile(next_a, (uint32_t)strips);  // the first strip handed out begins an item
  __syncthreads();

  for (;;) {
    // -- the next strip of the team's sequence (its items one after the other)
    bool ok = team_lock(lock_a, abort_a, is0);
    if (!ok) {
      atomicOr(p.err, kErrWaitTimeout);  // every lane: same bit
      st_shared_volatile(abort_a, 1);
      return;
    }
    int item = (int)ld_shared_volatile(item_a);
    int s = (int)ld_shared_volatile(next_a);
    const uint32_t seq = ld_shared_volatile(seq_a);
    while (s >= strips && item < n_items) {
      item = __shfl_sync(FULL_MASK, ticket_if(p.counter, is0), 0);
      if (item >= n_items) break;
      const int n = p.tasks[p.order ? p.order[item / nstr] : item / nstr].n;
      if (n > p.max_rows) atomicOr(p.err, kErrBadTask);  // every lane: same bit
      if (n > 0 && n <= p.max_rows) s = 0;
    }
    __syncwarp();
    st_shared_volatile(item_a, (uint32_t)(item < n_items ? item : (int)n_items));
    st_shared_volatile(next_a, (uint32_t)(s + 1));
    st_shared_volatile(seq_a, seq + 1);
    team_unlock(lock_a);
    if (item >= n_items) break;

    const int strand = PAIRS ? 0 : item % nstr;
    const int tr = item / nstr;
    const Task t = p.tasks[p.order ? p.order[tr] : tr];
    const int n = t.n;
    const float *q = p.query + t.q_off;
    const bool resume = (t.flags & kTaskResume) != 0 && p.state != nullptr;
    const bool save = (t.flags & kTaskSaveState) != 0 && p.state != nullptr;
    // planar FP32 reference and row state: strand s at s * m_pad
    const int64_t plane = (int64_t)strand * p.m_pad;
    const int64_t c0 = (int64_t)s * W + (int64_t)lane * S;
    const bool first = s == 0;
    const uint32_t buf = seq % nbuf, buf_in = buf ? buf - 1 : nbuf - 1;
    const uint32_t prog_out = prog + 8 * buf, prog_in = prog + 8 * buf_in;
    // seam column of the left strip: row -1 at [0], row i at [i + 1]
    const Seam *seam_in = reinterpret_cast<const Seam *>(seam_base + buf_in * seam_half);
    Seam *seam_out = reinterpret_cast<Seam *>(seam_base + buf * seam_half);

    // the buffer's last writer and its reader (the strip after it) must be
    // done; the reader may end first, where it begins another item
    if (seq >= nbuf) {
      const uint32_t last = seq - nbuf;
      ok = team_wait(prog_out, ((uint64_t)(last + 1) << 32) | kStripDone, abort_a, p.max_rows) &&
           team_wait(prog + 8 * ((buf + 1) % nbuf), ((uint64_t)(last + 2) << 32) | kStripDone, abort_a, p.max_rows);
    }

    Lane<PREC, S> L;
    L.O = make_float2(0.f, 0.f);
    if (resume) {
      // FP32 row state (fwd plane, rev plane at m_pad); FP16: the frame is the lane's minimum
      if constexpr (PAIRS) {
        const float4 *f0 = reinterpret_cast<const float4 *>(p.state + t.state_off + c0);
        const float4 *f1 = reinterpret_cast<const float4 *>(p.state + t.state_off + p.m_pad + c0);
        float mx = inf, my = inf;
#pragma unroll
        for (int j = 0; j < S / 4; ++j) {
          const float4 u = f0[j], v = f1[j];
          mx = fminf(mx, fminf(fminf(u.x, u.y), fminf(u.z, u.w)));
          my = fminf(my, fminf(fminf(v.x, v.y), fminf(v.z, v.w)));
        }
        L.O = make_float2(isinf(mx) ? 0.f : mx, isinf(my) ? 0.f : my);
#pragma unroll
        for (int j = 0; j < S / 4; ++j) {
          const float4 u = f0[j], v = f1[j];
          L.D[4 * j] = __floats2half2_rn(u.x - L.O.x, v.x - L.O.y);
          L.D[4 * j + 1] = __floats2half2_rn(u.y - L.O.x, v.y - L.O.y);
          L.D[4 * j + 2] = __floats2half2_rn(u.z - L.O.x, v.z - L.O.y);
          L.D[4 * j + 3] = __floats2half2_rn(u.w - L.O.x, v.w - L.O.y);
        }
      } else {
        const float4 *f = reinterpret_cast<const float4 *>(p.state + t.state_off + plane + c0);
#pragma unroll
        for (int j = 0; j < S / 4; ++j) {
          const float4 u = f[j];
          L.D[4 * j] = u.x, L.D[4 * j + 1] = u.y, L.D[4 * j + 2] = u.z, L.D[4 * j + 3] = u.w;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < S; ++j) memset(&L.D[j], 0, sizeof(V));
    }
    {
      // one word per column: an FP16 pair, or one strand's FP32 level
      const uint4 *g = reinterpret_cast<const uint4 *>(static_cast<const uint32_t *>(p.ref_plain) + plane + c0);
#pragma unroll
      for (int j = 0; j < S / 4; ++j) {
        const uint4 u = __ldg(g + j);
        memcpy(&L.R[4 * j], &u.x, 4);
        memcpy(&L.R[4 * j + 1], &u.y, 4);
        memcpy(&L.R[4 * j + 2], &u.z, 4);
        memcpy(&L.R[4 * j + 3], &u.w, 4);
      }
    }
    if (lane == kWarp - 1) {
      if constexpr (PAIRS) {
        const float2 v = __half22float2(L.D[S - 1]);
        seam_out[0] = make_float2(v.x + L.O.x, v.y + L.O.y);
      } else {
        seam_out[0] = L.D[S - 1];
      }
    }
    const auto set_dl = [&]() {
      // from lane l-1: that lane's frame minus this one; on lane 0, from the
      // absolute seam column: minus this frame
      const float ox = __shfl_up_sync(FULL_MASK, L.O.x, 1), oy = __shfl_up_sync(FULL_MASK, L.O.y, 1);
      L.dl = lane == 0 ? make_float2(-L.O.x, -L.O.y) : make_float2(ox - L.O.x, oy - L.O.y);
    };

    const uint64_t tag_in = (uint64_t)seq << 32;
    if (ok && !first) ok = team_wait(prog_in, tag_in | (uint32_t)min(n, kWindowRows), abort_a, n);
    const V up0 = __shfl_up_sync(FULL_MASK, L.D[S - 1], 1);  // every lane takes part in the shuffle
    const Seam in0 = ok && !first ? seam_in[0] : inf_value<Seam>();
    if constexpr (PAIRS) {
      set_dl();
      L.diag_next = rebase(lane == 0 ? in0 : __half22float2(up0), L.dl);
    } else {
      L.diag_next = lane == 0 ? in0 : up0;
    }
    L.last_a = L.D[S - 1];

    // a strip takes ceil(n / 2) + 31 steps, 16 to a window: before its steps a
    // window brings in the query samples and seam values of the 32 rows that
    // lane 0 begins in it, after them it takes out the 32 that lane 31 ended
    const int steps = ((n + 1) >> 1) + kWarp - 1;
    for (int st0 = 0; ok && st0 < steps; st0 += kWindowSteps) {
      const int r = 2 * st0 + lane;
      if (!first && st0 > 0) ok = team_wait(prog_in, tag_in | (uint32_t)min(n, 2 * st0 + kWindowRows), abort_a, n);
      if (!ok) break;
      qr[r & (kQueryRing - 1)] = C::q(r < n ? q[r] : 0.f);
      sin_w[lane] = !first && r < n ? seam_in[r + 1] : inf_value<Seam>();
      __syncwarp();
      if (st0 >= kWarp - 1 && 2 * (st0 + kWindowSteps) <= n) {
#pragma unroll 4
        for (int i = 0; i < kWindowSteps; ++i)
          refdel_step<PREC, S, false>(L, st0 + i, n, lane, qr + ((2 * (st0 + i - lane)) & (kQueryRing - 1)),
                                      sin_w + 2 * i, out_w + 2 * i);
      } else {
        const int cnt = min(kWindowSteps, steps - st0);
#pragma unroll 1
        for (int i = 0; i < cnt; ++i)
          refdel_step<PREC, S, true>(L, st0 + i, n, lane, qr + ((2 * (st0 + i - lane)) & (kQueryRing - 1)),
                                     sin_w + 2 * i, out_w + 2 * i);
      }
      __syncwarp();
      const int ro = r - 2 * (kWarp - 1);  // lane 31's rows of this window
      if ((unsigned)ro < (unsigned)n) seam_out[ro + 1] = out_w[lane];
      if constexpr (PAIRS) {
        if (st0 + kWindowSteps <= steps) {
          // rescale (every lane at the same step): subtract this lane's minimum
          __half2 mq[4] = {L.D[0], L.D[1], L.D[2], L.D[3]};
#pragma unroll
          for (int j = 4; j < S; ++j) mq[j & 3] = __hmin2(mq[j & 3], L.D[j]);
          const __half2 mn = __hmin2(__hmin2(mq[0], mq[1]), __hmin2(mq[2], mq[3]));
          float2 mf = __half22float2(mn);
          mf.x = isinf(mf.x) ? 0.f : mf.x;  // all-infinite cells stay as they are
          mf.y = isinf(mf.y) ? 0.f : mf.y;
          const __half2 ms = __floats2half2_rn(mf.x, mf.y);  // exact: the components are FP16 values
#pragma unroll
          for (int j = 0; j < S; ++j) L.D[j] = __hsub2(L.D[j], ms);
          L.last_a = __hsub2(L.last_a, ms);
          L.diag_next = __hsub2(L.diag_next, ms);
          L.O.x += mf.x;
          L.O.y += mf.y;
          set_dl();
        }
      }
      const int done = 2 * (st0 + kWindowSteps) - 2 * (kWarp - 1);  // rows lane 31 has ended
      if (done > 0) team_publish(prog_out, seq, (uint32_t)min(done, n));
    }
    if (!ok) {
      atomicOr(p.err, kErrWaitTimeout);  // every lane: same bit
      st_shared_volatile(abort_a, 1);
      return;
    }
    team_publish(prog_out, seq, kStripDone);

    // every lane now holds row n - 1 of its columns
    float bestx = inf, besty = inf;
    int64_t colx = -1, coly = -1;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const int64_t col = c0 + j;
      if (col < p.m) {
        if constexpr (PAIRS) {
          const float2 v = __half22float2(L.D[j]);
          const float vx = v.x + L.O.x, vy = v.y + L.O.y;
          if (vx < bestx) bestx = vx, colx = col;
          if (vy < besty) besty = vy, coly = col;
        } else if (L.D[j] < bestx) {
          bestx = L.D[j], colx = col;
        }
      }
    }
    if (save) {
      if constexpr (PAIRS) {
        float4 *f0 = reinterpret_cast<float4 *>(p.state + t.state_off + c0);
        float4 *f1 = reinterpret_cast<float4 *>(p.state + t.state_off + p.m_pad + c0);
#pragma unroll
        for (int j = 0; j < S / 4; ++j) {
          const float2 v0 = __half22float2(L.D[4 * j]), v1 = __half22float2(L.D[4 * j + 1]);
          const float2 v2 = __half22float2(L.D[4 * j + 2]), v3 = __half22float2(L.D[4 * j + 3]);
          f0[j] = make_float4(v0.x + L.O.x, v1.x + L.O.x, v2.x + L.O.x, v3.x + L.O.x);
          f1[j] = make_float4(v0.y + L.O.y, v1.y + L.O.y, v2.y + L.O.y, v3.y + L.O.y);
        }
      } else {
        float4 *f = reinterpret_cast<float4 *>(p.state + t.state_off + plane + c0);
#pragma unroll
        for (int j = 0; j < S / 4; ++j)
          f[j] = make_float4(L.D[4 * j], L.D[4 * j + 1], L.D[4 * j + 2], L.D[4 * j + 3]);
      }
    }
    warp_argmin(bestx, colx);
    const int64_t base = 2 * (int64_t)t.out_slot;
    red_min_if(&p.keys[base + strand], make_key(bestx, colx), is0 & (colx >= 0 ? 1u : 0u));
    if constexpr (PAIRS) {
      warp_argmin(besty, coly);
      red_min_if(&p.keys[base + 1], make_key(besty, coly), is0 & (coly >= 0 ? 1u : 0u));
    }
  }
}

template <int PREC, int S>
cudaError_t launch_refdel_inst(int warps, int grid, const SdtwParams &p, cudaStream_t s) {
  sdtw_refdel_kernel<PREC, S><<<grid, warps * kWarp, 0, s>>>(p);
  return cudaGetLastError();
}

template <int PREC, int S>
int occ_refdel_inst(int warps) {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, sdtw_refdel_kernel<PREC, S>, warps * kWarp, 0) != cudaSuccess)
    return 0;
  return n;
}

}  // namespace

cudaError_t launch_refdel(int precision, int cells_per_thread, int warps_per_cta, int grid, const SdtwParams &p,
                          cudaStream_t s) {
  if (warps_per_cta > kMaxWarps || p.team_warps < 1 || warps_per_cta % p.team_warps) return cudaErrorInvalidValue;
  if (precision == 1 && cells_per_thread == 16) return launch_refdel_inst<1, 16>(warps_per_cta, grid, p, s);
  if (precision == 1 && cells_per_thread == 32) return launch_refdel_inst<1, 32>(warps_per_cta, grid, p, s);
  if (precision == 0 && cells_per_thread == 32) return launch_refdel_inst<0, 32>(warps_per_cta, grid, p, s);
  return cudaErrorInvalidValue;
}

int refdel_ctas_per_sm(int precision, int cells_per_thread, int warps_per_cta) {
  if (precision == 1 && cells_per_thread == 16) return occ_refdel_inst<1, 16>(warps_per_cta);
  if (precision == 1 && cells_per_thread == 32) return occ_refdel_inst<1, 32>(warps_per_cta);
  if (precision == 0 && cells_per_thread == 32) return occ_refdel_inst<0, 32>(warps_per_cta);
  return 0;
}

}  // namespace dtwx
