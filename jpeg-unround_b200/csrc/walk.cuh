// The whole iteration as one walk down the picture (sm_100a): the dual step D_n with the
// relaxation, from x~_n and s_{n-1} to s_n, and the primal step P_{n+1} on s_n, x~_{n+1}, in one
// pass over HBM (TGV: 9 planes read and 9 written a sample, against 9 + 8 and then 3 + 1 in two
// launches). Of an iteration with a record, the tilde duals of D_n (KEEP 2) or zeta, v and G's terms of
// P_{n+1} (KEEP 1) are written beside; one with both takes sweep.cu and kernels.cu.
//
// A CTA owns a strip of 32 canvas columns (64 with one channel) and walks down strip_rows rows
// of it in chunks of 8 rows, its warps specialised:
//
//   warps 0-3  the dual step: a warp two rows of the chunk, a half-warp a row, a lane two
//              neighbouring columns, whose arithmetic goes by the packed binary32 operations
//              (fma.rn.f32x2 and the like: each half rounded as the operation of one sample), so
//              that a sample takes half the instructions. First x_n, w~, w_n and p_n; w- and p_n
//              go to shared memory; after a barrier of these warps the r step and
//              v = x_n + tau gamma div p_n take the left and upper neighbours' from there
//   warp 4     the bulk-tensor copies; and w- and p1_n of the column left of the strip, a lane per
//              row and channel, a chunk ahead
//   warps 5-   the proximal map, a warp a channel (with one channel, a half of the strip)
//
// Two rows at a time come into shared memory, one box (every plane of the state, and of x~ behind
// it; the strip and 4 columns either side), into a ring of 9: a chunk's rows and the row below, and
// the whole next chunk, so that its copies have a chunk's time; a chunk's rows are given back once
// its w- and p_n are made. v goes to the proximal maps' warps through tiles in two turns, and they
// write x~_{n+1}; a warp never waits for the whole CTA.
//
// Each value is made from the same operands by the same operations as in the two launches
// (dual_strip of sweep.cu, primal_block_row of kernels.cu; which product of a sum is fused is
// written out), so the iterates are theirs bit for bit. Every wait is bounded: one that runs out
// sets the error word, the other warps see it and leave, and the copies in flight are waited for.
// On every path a slot that a copy went to is waited for before its barrier is armed again and before
// the CTA leaves: a chunk's slots by the warps that read them, before they arrive at `drained`, which
// the copying warp waits for before it fills one again or leaves; slot 0, of which strips at the top
// read nothing, by warp 0; after a wait that ran out, all that are on their way by the copying warp. (No
// warp waited for slot 0 at first: its barrier could be armed in an unfinished phase, or a copy land in
// the shared memory of a CTA that had left. Four solves on four streams reported a failed launch.)
//
// What bounds it: instructions, not memory. A chunk of three channels takes 3,900
// warp-instructions (5.4 a sample with a strip's start; the two launches take 10.5) over 8 warps, two CTAs an SM by
// shared memory; they issue at 1.7 an SM and cycle, held by the latency of dependent operations and
// by instruction fetch, so that code size counts (the edges' tests are folded into addresses, and
// what is rarely run is not inlined: 4032x3024 TV 331 -> 261 us). Its rows are there when a chunk
// begins: of 56 looks at the ring, 55 need no wait. A launch's CTAs start on the places that the one
// before leaves (programmatic dependent launch) and wait for its end with their barriers and
// factors ready: 1-5 us of an iteration (160x120 5.2 -> 3.7, 2048^2 of three channels 174 -> 168).
// They let the next launch's in only after their own wait, so that one launch waits at a time: let in at
// once, launches wait in chains, as deep as small grids leave places, and hold those of other solves.
// Measured, an iteration before (two or three launches, in graphs of eight) and after: TV grey
// 160x120 12.6 -> 3.7 us, 512^2 13.3 -> 4.5; TGV grey 512^2 18.4 -> 8.4, 2048^2 74 -> 64; TGV 4:2:0
// 768x512 36.7 -> 18.2, 2048^2 200 -> 167; TV 4:2:0 1919x1083 63.2 -> 43.9, 2048^2 101 (two CTAs an
// SM, a barrier for each tile) -> 84.
#pragma once

#include <algorithm>
#include <atomic>
#include <type_traits>

#include <cuda.h>

#include "dct.cuh"
#include "kernels.hpp"
#include "prox.cuh"
#include "tma.cuh"

namespace urb {

namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kHalo = 4;  // columns loaded either side of the strip (16-byte aligned start)
constexpr int kChunk = 8;     // rows of a chunk
constexpr int kDual = 4;      // the dual step's warps, two rows of a chunk each
// Warps 0-3 the dual step's, 4 the copies' and the left column's, then a warp for the proximal map
// of each channel (with one channel, of each half of the strip).
template <int C>
constexpr int walk_threads() {
  return 32 * (kDual + 1 + (C == 1 ? 2 : C));
}
constexpr int kSlots = 9;     // of the ring, two rows each: a chunk's and the row below, and the next chunk's

constexpr int round32(int n) { return (n + 31) / 32 * 32; }

// CTAs an SM holds: by shared memory (TGV: 112 KB of three channels, 62 KB of one), else by
// registers; TV of three channels with two: 8% slower at 2048x2048, 14% at 1919x1083.
template <bool TGV, int C>
constexpr int walk_ctas() {
  return C == 1 ? (TGV ? 3 : 4) : (TGV ? 2 : 3);
}

// Two neighbouring samples of a row, as the packed binary32 operations take them: each lane of
// a pair rounded as the operation of single samples.
using Pair = unsigned long long;
__device__ __forceinline__ Pair pair(float x, float y) {
  Pair p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(x), "f"(y));
  return p;
}
__device__ __forceinline__ Pair pair(float x) { return pair(x, x); }
__device__ __forceinline__ float first(Pair p) {
  float x;
  asm("{\n .reg .f32 y;\n mov.b64 {%0, y}, %1;\n}\n" : "=f"(x) : "l"(p));
  return x;
}
__device__ __forceinline__ float second(Pair p) {
  float y;
  asm("{\n .reg .f32 x;\n mov.b64 {x, %0}, %1;\n}\n" : "=f"(y) : "l"(p));
  return y;
}
__device__ __forceinline__ Pair add2(Pair a, Pair b) {
  Pair p;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(a), "l"(b));
  return p;
}
__device__ __forceinline__ Pair sub2(Pair a, Pair b) {
  Pair p;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(a), "l"(b));
  return p;
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
  Pair p;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(a), "l"(b));
  return p;
}
__device__ __forceinline__ Pair fma2(Pair a, Pair b, Pair c) {
  Pair p;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p) : "l"(a), "l"(b), "l"(c));
  return p;
}
// A ball's scale: radius / |p| beyond it, 1 within. `inside` is just below the radius's square, so
// that a square at most that is within without the root and the quotient. The pair's root and
// quotient, each correctly rounded, go by Markstein's sequences of fused multiply-adds (P. W.
// Markstein, IBM J. Res. Dev. 34, 1990) from the approximate 1 / sqrt, both halves at once: 14
// packed operations against two square roots and two divisions. Their one exception, a divisor
// whose significand is all ones, and squares and radii far from 1 (`usual` false), where an
// intermediate could leave the range, take sqrtf and the division. Equal to those on every float
// of six octaves above the radius, for each of 600 radii (tests/ball_check.cu).
// A solve's radii are usual (walk_takes). The unrolled solve takes any(): of a tiny one, whose square
// rounds coarsely or to 0, `inside` is negative and the norm decides; a negative one projects beyond its
// square and leaves what lies within, as the adjoint has it.
struct Ball {
  float radius, inside;
  bool usual;
  __device__ explicit Ball(float r) : radius(r), inside(r * r * 0.999999f), usual(r > 1e-12f && r < 1e12f) {}
  static __device__ __forceinline__ Ball any(float r) {
    Ball ball(r);
    ball.inside = r * r * 0.999999f - 1e-25f;
    return ball;
  }
};

__device__ __forceinline__ float ball(float square, const Ball& B) {
  if (square <= B.inside) return 1.0f;
  const float norm = sqrtf(square);
  return norm > B.radius ? B.radius / norm : 1.0f;
}

__device__ __forceinline__ Pair ball2(Pair square, const Ball& B) {
  const float x = first(square), y = second(square);
  if (x <= B.inside && y <= B.inside) return pair(1.0f);
  const float ax = fmaxf(x, B.inside), ay = fmaxf(y, B.inside);
  const Pair a = pair(ax, ay), minus_one = pair(-1.0f), radius = pair(B.radius);
  float sx, sy;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(sx) : "f"(ax));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(sy) : "f"(ay));
  const Pair s = pair(sx, sy);
  Pair g = mul2(a, s), h = mul2(s, pair(-0.5f));  // sqrt(a), -1 / (2 sqrt(a)), approximately
  const Pair r = fma2(h, g, pair(0.5f));
  g = fma2(g, r, g);
  h = fma2(h, r, h);
  const Pair norm = fma2(fma2(g, g, mul2(a, minus_one)), h, g), minus_norm = mul2(norm, minus_one);
  Pair inverse = mul2(h, pair(-2.0f));
  inverse = fma2(inverse, fma2(inverse, minus_norm, pair(1.0f)), inverse);
  const Pair q = mul2(radius, inverse), scale = fma2(fma2(q, minus_norm, radius), inverse, q);
  const float nx = first(norm), ny = second(norm);
  const bool exception = (__float_as_uint(nx) | 0xff800000u) == 0xffffffffu || (__float_as_uint(ny) | 0xff800000u) == 0xffffffffu;
  if (!B.usual || exception || !(fmaxf(ax, ay) < 1e24f)) return pair(ball(x, B), ball(y, B));
  return pair(nx > B.radius ? first(scale) : 1.0f, ny > B.radius ? second(scale) : 1.0f);
}

// The CTA's shared memory, in floats, every part 128-byte aligned.
template <bool TGV, int C, int CR>
struct WalkLayout {
  static constexpr int F = TGV ? 8 : 3;  // state planes a channel: x, p1, p2 (+ w1, w2, r11, r22, r12)
  static constexpr int L = lane_columns(C);
  static constexpr int WIDTH = 32 * L;
  static constexpr int SPAN = WIDTH + 2 * kHalo;
  static constexpr int PLANE = 2 * SPAN;  // a plane's rows in a slot
  static constexpr int SLOT = round32((F + 1) * C * PLANE);
  // The exchange: -w-1, -w-2, p1_n and p2_n (TV: p1_n, p2_n) of each row of a chunk and of the
  // row above it: rows 0-6, and row 7 in two turns. Column 4 + j of the strip; columns 2 and 3 the
  // left neighbour's, in turns.
  static constexpr int Q = TGV ? 4 : 2;
  static constexpr int ROW = Q * C * (WIDTH + 4);
  static constexpr int EXCHANGE = kSlots * SLOT;
  static constexpr int LUMA = EXCHANGE + round32((kChunk + 1) * ROW);  // v of channel 0, two chunks
  static constexpr int CHROMA = LUMA + 2 * kChunk * WIDTH;             // v of channels 1 and 2, two bands
  static constexpr int FLOATS = CHROMA + 2 * (C - 1) * 8 * CR * WIDTH;
};

// A component's factors in shared memory; those of MMSE centres and of a slack's cost, where it
// has them (`general`), are read from `all`.
struct WalkFactors {
  float4 plain[64];
  float4 flat[64];
  const ProxFactors* all;
  int general;
};

// A block row's levels and flat flag at a lane (row m of its block), read ahead of their use.
struct Ahead {
  int4 levels;
  std::int16_t dc;
  std::uint8_t flat;
  bool in;
};

template <int PR, int PC>
__device__ __forceinline__ Ahead look_ahead(const IterationParams& P, int c, int j, int i, int lane) {
  const ComponentDevice& D = P.component[c];
  const int vbx = j / (8 * PC), vby = i / (8 * PR), m = lane % (8 * PC) / PC;
  Ahead a;
  a.in = j < P.dual.g.columns && vby < D.block_rows && vbx < D.block_columns;
  a.levels = make_int4(0, 0, 0, 0);
  a.dc = 0;
  a.flat = 0;
  if (a.in) {
    const std::size_t block = static_cast<std::size_t>(vby) * D.block_columns + vbx;
    a.levels = __ldg(reinterpret_cast<const int4*>(D.levels + block * 64 + m * 8));
    a.dc = __ldg(D.levels + block * 64);
    a.flat = __ldg(D.flat + block);
  }
  return a;
}

__device__ __noinline__ void general_row(float (&coef)[8], int4 levels, int m, bool flat, const ProxFactors& F);

// The proximal map of a block row of a component at the lane's column: v down the column from
// `tile` (32 columns, rows WIDTH apart), x~ of the next iteration out. As primal_block_row
// (kernels.cu). The transposes go through the tile, whose v is in registers by then: entry (k, m)
// of a block at row k, column m ^ k of the block's eight, so that a warp's accesses along either
// fall into different banks.
// With KEEP, zeta and v are written and G's terms added to `sum` (of the component `D`, v of the
// tile's first row at `v_out`).
template <int PR, int PC, int WIDTH, bool KEEP>
__device__ __forceinline__ void prox_rows(float* tile, const Ahead& a, const WalkFactors& F, float* next, int pitch, int lane, bool column_in, const ComponentDevice& D, std::size_t block,
                                          float* v_out, bool counted, double& sum) {
  constexpr int BH = 8 * PR, LANES = 8 * PC;
  const int in_block = lane % LANES, m = in_block / PC, cell = in_block % PC, leader = lane - cell;
  float* const t = tile + lane / LANES * 8;
  auto entry = [&](int k, int n) -> float& { return t[k * WIDTH + (n ^ k)]; };
  float v[BH];
#pragma unroll
  for (int r = 0; r < BH; ++r) v[r] = tile[r * WIDTH + lane];
  const float middle = (static_cast<float>(a.dc) * F.plain[0].x + 1024.0f) * 0.125f;
  float mean[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    if constexpr (PR == 1 && PC == 1) {
      mean[r] = v[r] - middle;
    } else {
      float column = v[PR * r];
#pragma unroll
      for (int k = 1; k < PR; ++k) column += v[PR * r + k];
      float total = 0.0f;
#pragma unroll
      for (int k = 0; k < PC; ++k) {
        const float part = __shfl_sync(kAll, column, leader + k);
        total = k == 0 ? part : total + part;
      }
      mean[r] = total / static_cast<float>(PR * PC) - middle;
    }
  }
  float col[8], row[8], coef[8], zeta[8];
  forward8(mean, col);
  __syncwarp();
  if (cell == 0) {
#pragma unroll
    for (int k = 0; k < 8; ++k) entry(k, m) = col[k];
  }
  __syncwarp();
#pragma unroll
  for (int u = 0; u < 8; ++u) row[u] = entry(m, u);
  forward8(row, coef);
  const int words[4] = {a.levels.x, a.levels.y, a.levels.z, a.levels.w};
  auto level_at = [&](int u) -> int { return static_cast<std::int16_t>(words[u >> 1] >> (16 * (u & 1))); };
  if (F.general == 0) {
    // prox_at of midpoint centres without a slack's cost.
    const float4* table = (a.flat != 0 ? F.flat : F.plain) + m * 8;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float4 f = table[u ^ m];  // prox_slot: Q, r, t r, (1/2 + s) Q
      const float level = u == 0 && m == 0 ? 0.0f : static_cast<float>(level_at(u));
      const float centre = level * f.x;
      const float z = fmaf(f.z, centre, coef[u] * f.y);
      zeta[u] = clamp_to(z, centre - f.w, centre + f.w);
    }
  } else {
#pragma unroll
    for (int u = 0; u < 8; ++u) zeta[u] = coef[u];
    general_row(zeta, a.levels, m, a.flat != 0, *F.all);
  }
  if constexpr (KEEP) {
    if (a.in && cell == 0) {
      float4* to = reinterpret_cast<float4*>(D.zeta + block * 64 + m * 8);
      to[0] = make_float4(zeta[0], zeta[1], zeta[2], zeta[3]);
      to[1] = make_float4(zeta[4], zeta[5], zeta[6], zeta[7]);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int k = m * 8 + u;
        double absolute = zeta[u];  // DC is kept centred (less q Q + 1024)
        if (k == 0) absolute += static_cast<double>(level_at(0)) * D.constants->step[0] + 1024.0;
        if (counted) sum += value_term(absolute, level_at(u), k, a.flat != 0, *D.constants);
      }
    }
    if (column_in) {
#pragma unroll
      for (int r = 0; r < BH; ++r) v_out[static_cast<std::size_t>(r) * pitch] = v[r];
    }
  }
  inverse8(zeta, row);
  __syncwarp();
  if (cell == 0) {
#pragma unroll
    for (int k = 0; k < 8; ++k) entry(m, k) = row[k];
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; ++k) col[k] = entry(k, m);
  float back[8];
  inverse8(col, back);
  if (column_in) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
#pragma unroll
      for (int k = 0; k < PR; ++k) {
        const int rr = PR * r + k;
        float out;
        if constexpr (PR == 1 && PC == 1) {
          out = a.in ? back[r] + middle : v[rr];
        } else {
          out = a.in ? v[rr] + (back[r] - mean[r]) : v[rr];
        }
        next[static_cast<std::size_t>(rr) * pitch] = out;
      }
    }
  }
}

// The CTA's barriers. full: a slot's bytes are in; drained: a chunk's rows are read (by the dual
// step's warps and the left column's), in turns; go: the second part of a chunk may run, in turns
// (its left column is made, and the proximal maps' warps are done with the tiles it writes);
// luma, chroma: a tile of v is whole.
struct WalkBarriers {
  std::uint64_t full[kSlots];
  std::uint64_t drained[2];
  std::uint64_t go[2];
  std::uint64_t luma[2];
  std::uint64_t chroma[2];
};

// A barrier of the dual step's warps; whether any of their threads says so.
__device__ __forceinline__ bool any_of_dual(bool said) {
  int any;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.or.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(any)
      : "r"(static_cast<int>(said)), "n"(32 * kDual)
      : "memory");
  return any != 0;
}

__device__ __forceinline__ void dual_barrier() {
  asm volatile("barrier.cta.sync 1, %0;" ::"n"(32 * kDual) : "memory");
}

// Waits for a phase of a barrier that has not come at once, until another warp of the CTA has given
// up or the tries run out.
__device__ __noinline__ bool wait_longer(std::uint64_t* bar, unsigned parity, const volatile int* failed, int tries) {
  for (int k = 0; k < tries; ++k) {
    if (barrier_try(bar, parity)) return true;
    if ((k & 15) == 15 && *failed != 0) return false;
  }
  return false;
}

__device__ __forceinline__ bool wait_unless(std::uint64_t* bar, unsigned parity, const volatile int* failed,
                                            int tries = static_cast<int>(kWaitLimit)) {
  return (tries > 0 && barrier_try(bar, parity)) || wait_longer(bar, parity, failed, tries);
}

// prox_at of a row of a block with MMSE centres or a slack's cost.
__device__ __noinline__ void general_row(float (&coef)[8], int4 levels, int m, bool flat, const ProxFactors& F) {
  const int words[4] = {levels.x, levels.y, levels.z, levels.w};
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    coef[u] = prox_at(coef[u], static_cast<std::int16_t>(words[u >> 1] >> (16 * (u & 1))), m * 8 + u, flat, F);
  }
}

// RAGGED: a canvas that is not whole blocks (pictures of samples): a strip's last chunk may reach past
// the last row, and the last pair of an odd number of columns past the last column.
template <bool TGV, int C, bool COUPLED, int CR, int CC, int KEEP, bool UNROLLED = false, bool RAGGED = false>
struct Walk {
  using W = WalkLayout<TGV, C, CR>;
  static constexpr int L = W::L, SPAN = W::SPAN, WIDTH = W::WIDTH, XS = WIDTH + 4;
  // One channel's kernels of sweep.cu relax p and r, and take the square of p, with the other
  // product fused.
  static constexpr bool REST_FIRST = C == 1;
  static constexpr bool SQUARE_2 = TGV && C == 1 && !UNROLLED;
  // The unrolled solve's kernels relax w with the first product fused.
  static constexpr bool REST_FIRST_W = !UNROLLED;

  const IterationParams& Q;
  float* const shared;
  const int x0, i0, i1;
  // Of the unrolled solve: the picture, and its parameters (UnrolledWalk).
  const int image = 0;
  const float image_tau = 0.0f, image_sigma = 0.0f, image_alpha1 = 0.0f, image_alpha0 = 0.0f;

  __device__ __forceinline__ float tau(int c) const { return UNROLLED ? image_tau : Q.dual.tau[c]; }
  __device__ __forceinline__ float sigma(int c) const { return UNROLLED ? image_sigma : Q.dual.sigma[c]; }
  __device__ __forceinline__ float radius() const { return UNROLLED ? image_alpha1 : Q.dual.radius; }
  __device__ __forceinline__ float radius0() const { return UNROLLED ? image_alpha0 : Q.dual.radius0; }
  static __device__ __forceinline__ Ball ball_of(float r) {
    if constexpr (UNROLLED) {
      return Ball::any(r);
    } else {
      return Ball(r);
    }
  }
  // Row i of the picture among the rows of a plane; an offset within a plane in bytes.
  using Offset = std::conditional_t<UNROLLED, std::size_t, unsigned>;
  __device__ __forceinline__ Offset plane_row(int i) const {
    return UNROLLED ? static_cast<Offset>(image) * Q.dual.g.rows + i : static_cast<Offset>(i);
  }

  // A plane of a slot: a field's, or x~'s.
  static __device__ __forceinline__ int at(int field, int c) { return (field * C + c) * W::PLANE; }
  static __device__ __forceinline__ int tilde(int c) { return at(W::F, c); }
  static __device__ __forceinline__ int exchange(int q, int c) { return (q * C + c) * XS + 4; }

  // ---- The dual step's first part at the lane's row i: x_n, w_n, p_n written, -w- and p_n kept
  // for the second part and left in the exchange row `to`. `own` the row in
  // its slot, `down` the row below in its.
  struct Kept {
    Pair xn[C], pn1[C], pn2[C], nb1[C], nb2[C], r11[C], r22[C], r12[C];
  };

  // Past the last column or row a forward difference is 0: the neighbour's place is the own one
  // there (`next` the offset of the column right of the pair, `down` the row itself).
  template <bool FIRST>
  __device__ __forceinline__ void first_part(Kept& k, const float* own, const float* down, int part, int across, int i,
                                             float* to) const {
    const DualParams& P = Q.dual;
    const int o = kHalo + 32 * part + across, j = x0 + 32 * part + across;
    const bool valid = j < P.g.columns && (!RAGGED || i < P.g.rows);  // the pair, or its first sample
    const bool alone = RAGGED && j + 1 >= P.g.columns;               // the second past the last column
    const int next = j + 2 < P.g.columns ? o + 2 : o + 1;
    const Offset here = (plane_row(FIRST ? 0 : i) * P.g.pitch + j) * 4u;
    const Pair rho = pair(P.rho), rest = pair(P.rest), minus_two = pair(-2.0f);
    auto own_at = [&](int offset) -> Pair { return *reinterpret_cast<const Pair*>(own + offset + o); };
    auto right_of = [&](int offset, Pair p) -> Pair {
      return pair(alone ? first(p) : second(p), own[offset + next]);
    };
    auto down_at = [&](int offset) -> Pair { return *reinterpret_cast<const Pair*>(down + offset + o); };
    auto put = [&](float* base, int c, Pair p) {
      if (!FIRST && valid) *reinterpret_cast<Pair*>(reinterpret_cast<char*>(base + c * P.g.plane) + here) = p;
    };
    Pair step_p1[C], step_p2[C], old_p1[C], old_p2[C];
    Pair square_p = 0;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      // -x-, of the pair, of its right and of its lower neighbours.
      const Pair xt = own_at(tilde(c)), x = own_at(at(0, c));
      const Pair bar = fma2(xt, minus_two, x);
      const float right = fmaf(own[tilde(c) + next], -2.0f, own[at(0, c) + next]);
      const Pair below = fma2(down_at(tilde(c)), minus_two, down_at(at(0, c)));
      const Pair gx = sub2(bar, pair(alone ? first(bar) : second(bar), right));
      const Pair gy = sub2(bar, below);
      k.xn[c] = fma2(rho, xt, mul2(rest, x));
      put(P.out.x, c, k.xn[c]);
      old_p1[c] = own_at(at(1, c));
      old_p2[c] = own_at(at(2, c));
      const Pair sigma_c = pair(sigma(c));
      if constexpr (!TGV) {
        step_p1[c] = fma2(sigma_c, gx, old_p1[c]);
        step_p2[c] = fma2(sigma_c, gy, old_p2[c]);
      } else {
        // w~ = w + tau (p + div2 r), -w-.
        const Pair tau_c = pair(tau(c));
        const Pair r11 = own_at(at(5, c)), r22 = own_at(at(6, c)), r12 = own_at(at(7, c));
        k.r11[c] = r11;
        k.r22[c] = r22;
        k.r12[c] = r12;
        const Pair d1 = add2(sub2(right_of(at(5, c), r11), r11), sub2(down_at(at(7, c)), r12));
        const Pair d2 = add2(sub2(right_of(at(7, c), r12), r12), sub2(down_at(at(6, c)), r22));
        const Pair w1 = own_at(at(3, c)), w2 = own_at(at(4, c));
        const Pair t1 = fma2(tau_c, add2(old_p1[c], d1), w1), t2 = fma2(tau_c, add2(old_p2[c], d2), w2);
        put(P.out.w1, c, REST_FIRST_W ? fma2(rest, w1, mul2(rho, t1)) : fma2(rho, t1, mul2(rest, w1)));
        put(P.out.w2, c, REST_FIRST_W ? fma2(rest, w2, mul2(rho, t2)) : fma2(rho, t2, mul2(rest, w2)));
        if constexpr (KEEP == 2) {
          put(P.tilde.w1, c, t1);
          put(P.tilde.w2, c, t2);
        }
        k.nb1[c] = fma2(t1, minus_two, w1);
        k.nb2[c] = fma2(t2, minus_two, w2);
        step_p1[c] = fma2(sigma_c, add2(gx, k.nb1[c]), old_p1[c]);
        step_p2[c] = fma2(sigma_c, add2(gy, k.nb2[c]), old_p2[c]);
      }
      if constexpr (COUPLED) {
        const Pair square = fma2(step_p1[c], step_p1[c], mul2(step_p2[c], step_p2[c]));
        square_p = c == 0 ? square : add2(square_p, square);
      }
    }
    const Ball unit = ball_of(radius());
    Pair scale = 0;
    if constexpr (COUPLED) scale = ball2(square_p, unit);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      if constexpr (!COUPLED) {
        const Pair a = SQUARE_2 ? step_p2[c] : step_p1[c], b = SQUARE_2 ? step_p1[c] : step_p2[c];
        scale = ball2(fma2(a, a, mul2(b, b)), unit);
      }
      const Pair q1 = mul2(step_p1[c], scale), q2 = mul2(step_p2[c], scale);
      k.pn1[c] = REST_FIRST ? fma2(rest, old_p1[c], mul2(rho, q1)) : fma2(rho, q1, mul2(rest, old_p1[c]));
      k.pn2[c] = REST_FIRST ? fma2(rest, old_p2[c], mul2(rho, q2)) : fma2(rho, q2, mul2(rest, old_p2[c]));
      put(P.out.p1, c, k.pn1[c]);
      put(P.out.p2, c, k.pn2[c]);
      if (KEEP == 2 && P.tilde.p1 != nullptr) {  // p~: TV's records and the partial gap's
        put(P.tilde.p1, c, q1);
        put(P.tilde.p2, c, q2);
      }
      auto leave = [&](int q, Pair p) {
        *reinterpret_cast<Pair*>(to + exchange(q, c) + 32 * part + across) = p;
      };
      leave(0, k.pn1[c]);
      leave(1, k.pn2[c]);
      if constexpr (TGV) {
        leave(2, k.nb1[c]);
        leave(3, k.nb2[c]);
      }
    }
  }

  // ---- The second part: r_n from w- of the pixel and of its left and upper neighbours, and v of
  // the next primal step. `here` and `above` the exchange rows of the pixel's row and of the row
  // above, `before` the exchange column of the left neighbour of the pair.
  __device__ __forceinline__ void second_part(const Kept& k, const float* own_row, const float* above_row, int before,
                                              int part, int across, int i, float* luma, float* chroma) const {
    const DualParams& P = Q.dual;
    const int j = x0 + 32 * part + across;
    const bool has_down = i + 1 < P.g.rows;
    const bool valid = j < P.g.columns && (!RAGGED || i < P.g.rows);
    const bool has_right = j + 2 < P.g.columns;  // of the pair's second sample
    const bool alone = RAGGED && j + 1 >= P.g.columns;
    const Offset here = (plane_row(i) * P.g.pitch + j) * 4u;
    const Pair rho = pair(P.rho), rest = pair(P.rest), two = pair(2.0f);
    auto across_or_0 = [&](Pair p) -> Pair {
      return pair(alone ? 0.0f : first(p), has_right ? second(p) : 0.0f);
    };
    auto down_or_0 = [&](Pair p) -> Pair { return has_down ? p : pair(0.0f); };
    auto put = [&](float* base, int c, Pair p) {
      if (valid) *reinterpret_cast<Pair*>(reinterpret_cast<char*>(base + c * P.g.plane) + here) = p;
    };
    auto above_at = [&](int q, int c) -> Pair {
      return *reinterpret_cast<const Pair*>(above_row + exchange(q, c) + 32 * part + across);
    };
    auto left_of = [&](int q, int c, Pair p) -> Pair { return pair(own_row[exchange(q, c) + before], first(p)); };
    if constexpr (TGV) {
      const Ball unit = ball_of(radius0());
      Pair r11[C], r22[C], r12[C];
      Pair square = 0;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const Pair l1 = left_of(2, c, k.nb1[c]), l2 = left_of(3, c, k.nb2[c]);
        const Pair u1 = above_at(2, c), u2 = above_at(3, c);
        const Pair exx = sub2(l1, across_or_0(k.nb1[c])), eyy = sub2(u2, down_or_0(k.nb2[c]));
        const Pair exy = mul2(pair(0.5f), add2(sub2(u1, down_or_0(k.nb1[c])), sub2(l2, across_or_0(k.nb2[c]))));
        const Pair sigma_c = pair(sigma(c));
        r11[c] = fma2(sigma_c, exx, k.r11[c]);
        r22[c] = fma2(sigma_c, eyy, k.r22[c]);
        r12[c] = fma2(sigma_c, exy, k.r12[c]);
        const Pair own = fma2(two, mul2(r12[c], r12[c]), fma2(r11[c], r11[c], mul2(r22[c], r22[c])));
        square = !COUPLED || c == 0 ? own : add2(square, own);
        if constexpr (!COUPLED) {
          const Pair scale = ball2(square, unit);
          r11[c] = mul2(r11[c], scale);
          r22[c] = mul2(r22[c], scale);
          r12[c] = mul2(r12[c], scale);
        }
      }
      Pair scale = 0;
      if constexpr (COUPLED) scale = ball2(square, unit);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        if constexpr (COUPLED) {
          r11[c] = mul2(r11[c], scale);
          r22[c] = mul2(r22[c], scale);
          r12[c] = mul2(r12[c], scale);
        }
        auto relaxed = [&](Pair t, Pair old) -> Pair {
          return REST_FIRST ? fma2(rest, old, mul2(rho, t)) : fma2(rho, t, mul2(rest, old));
        };
        put(P.out.r11, c, relaxed(r11[c], k.r11[c]));
        put(P.out.r22, c, relaxed(r22[c], k.r22[c]));
        put(P.out.r12, c, relaxed(r12[c], k.r12[c]));
        if constexpr (KEEP == 2) {
          put(P.tilde.r11, c, r11[c]);
          put(P.tilde.r22, c, r22[c]);
          put(P.tilde.r12, c, r12[c]);
        }
      }
    }
    // v = x_n + tau gamma div p_n, backward differences.
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const Pair dy = sub2(down_or_0(k.pn2[c]), above_at(1, c));
      const Pair dx = sub2(across_or_0(k.pn1[c]), left_of(0, c, k.pn1[c]));
      float* to = c == 0 ? luma : chroma + (c - 1) * 8 * CR * WIDTH;
      *reinterpret_cast<Pair*>(to + 32 * part + across) = fma2(pair(tau(c)), add2(dy, dx), k.xn[c]);
    }
  }

  // ---- Warps 0-3. False where a wait ran out.
  __device__ __forceinline__ bool dual_warp(WalkBarriers& bars, const volatile int* failed, int warp, int lane) const {
    const DualParams& P = Q.dual;
    const int half = lane >> 4, across = 2 * (lane & 15);
    float* const rows = shared + W::EXCHANGE;          // of the chunk
    auto row_of = [&](int r, int k) -> float* { return rows + (r < kChunk - 1 ? r : r + (k & 1)) * W::ROW; };
    const int chunks = (i1 - i0) / kChunk;
    // Slot n holds rows i0 - 2 + 2 n and the next.
    auto slot = [&](int n) -> const float* { return shared + n % kSlots * W::SLOT; };
    const int tries = static_cast<int>(min(P.ring_wait_limit, kWaitLimit));
    auto ready = [&](int n) { return wait_unless(&bars.full[n % kSlots], (n / kSlots) & 1, failed, tries); };
    // The row above the strip: its -w- and p2_n, as a chunk's row 7 before the first (0 above the
    // canvas). Slot 0 is waited for there too: no slot is filled again, and no CTA leaves, before what
    // was on its way to it has landed.
    bool good = true;
    if (warp == 0) {
      float* const to = row_of(kChunk - 1, 1);
      good = __all_sync(kAll, ready(0) && ready(1));
      if (i0 > 0) {
        if (good) {
          Kept kept[L];
#pragma unroll
          for (int h = 0; h < L; ++h) {
            first_part<true>(kept[h], slot(0) + SPAN, slot(1), h, across, i0 - 1, to);
          }
        }
      } else {
        for (int k = lane; k < W::ROW; k += 32) to[k] = 0.0f;
      }
    }
    for (int k = 0; k < chunks; ++k) {
      const int n = 1 + kDual * k + warp;
      const int i = i0 + kChunk * k + 2 * warp + half;
      good = good && ready(n) && ready(n + 1);
      good = __all_sync(kAll, good);
      Kept kept[L];
      if (good) {
        const float* own = slot(n) + half * SPAN;
        const float* down = i + 1 >= P.g.rows ? own : half == 0 ? own + SPAN : slot(n + 1);
        float* const to = row_of(2 * warp + half, k);
#pragma unroll
        for (int h = 0; h < L; ++h) {
          first_part<false>(kept[h], own, down, h, across, i, to);
        }
        __syncwarp();
        if (lane == 0) barrier_arrive(&bars.drained[k & 1]);
        good = wait_unless(&bars.go[k & 1], (k >> 1) & 1, failed);
      }
      if (any_of_dual(!good)) return false;
      {
        const int row = 2 * warp + half;
        const float* own_row = row_of(row, k);
        const float* above_row = row == 0 ? row_of(kChunk - 1, k + 1) : rows + (row - 1) * W::ROW;
        float* const luma = shared + W::LUMA + ((k & 1) * kChunk + row) * WIDTH;
        float* const chroma =
            shared + W::CHROMA + ((k / CR & 1) * (C - 1) * 8 * CR + k % CR * kChunk + row) * WIDTH;
#pragma unroll
        for (int h = 0; h < L; ++h) {
          const int before = h == 0 && across == 0 ? -1 - (k & 1) : 32 * h + across - 1;
          second_part(kept[h], own_row, above_row, before, h, across, i, luma, chroma);
        }
      }
      __syncwarp();
      if (lane == 0) {
        barrier_arrive(&bars.luma[k & 1]);
        if constexpr (C > 1) barrier_arrive(&bars.chroma[k / CR & 1]);
      }
      dual_barrier();  // the exchange is read before the next chunk's is written
    }
    return true;
  }

  // ---- The side warp's look at the left column: -w- and p1_n at column x0 - 1 of chunk k's rows (0
  // left of the canvas), a lane per row and channel.
  __device__ __forceinline__ bool left_column(WalkBarriers& bars, const volatile int* failed, int k, int lane) const {
    const DualParams& P = Q.dual;
    bool good = true;
#pragma unroll
    for (int s = 0; s <= kDual; ++s) {
      const int n = 1 + kDual * k + s;
      good = good && wait_unless(&bars.full[n % kSlots], (n / kSlots) & 1, failed);
    }
    if (!__all_sync(kAll, good)) return false;
    const int row = lane / C, c = lane % C, ii = i0 + kChunk * k + row, o = kHalo - 1;
    const bool mine = lane < kChunk * C;
    float nb1 = 0.0f, nb2 = 0.0f, step1 = 0.0f, step2 = 0.0f, old1 = 0.0f, square = 0.0f;
    if (mine && x0 > 0) {
      const int n = 1 + kDual * k + row / 2;
      const float* a = shared + n % kSlots * W::SLOT + row % 2 * SPAN + o;
      const float* d = row % 2 == 0 ? a + SPAN : shared + (n + 1) % kSlots * W::SLOT + o;
      const bool lower = ii + 1 < P.g.rows;  // the column to the right is the strip's first
      auto S = [&](const float* from, int field) -> float { return from[at(field, c)]; };
      auto X = [&](const float* from) -> float { return from[tilde(c)]; };
      if constexpr (TGV) {
        const float r11 = S(a, 5), r22 = S(a, 6), r12 = S(a, 7), w1 = S(a, 3), w2 = S(a, 4);
        const float d1 = __fadd_rn(__fsub_rn(S(a + 1, 5), r11), lower ? __fsub_rn(S(d, 7), r12) : 0.0f);
        const float d2 = __fadd_rn(__fsub_rn(S(a + 1, 7), r12), lower ? __fsub_rn(S(d, 6), r22) : 0.0f);
        nb1 = fmaf(fmaf(tau(c), __fadd_rn(S(a, 1), d1), w1), -2.0f, w1);
        nb2 = fmaf(fmaf(tau(c), __fadd_rn(S(a, 2), d2), w2), -2.0f, w2);
      }
      const float bar = fmaf(X(a), -2.0f, S(a, 0));
      const float gx = __fsub_rn(bar, fmaf(X(a + 1), -2.0f, S(a + 1, 0)));
      const float gy = lower ? __fsub_rn(bar, fmaf(X(d), -2.0f, S(d, 0))) : 0.0f;
      old1 = S(a, 1);
      step1 = fmaf(sigma(c), TGV ? __fadd_rn(gx, nb1) : gx, old1);
      step2 = fmaf(sigma(c), TGV ? __fadd_rn(gy, nb2) : gy, S(a, 2));
      const float s = SQUARE_2 ? step2 : step1, t = SQUARE_2 ? step1 : step2;
      square = fmaf(s, s, __fmul_rn(t, t));
    }
    if constexpr (COUPLED) {
      float total = 0.0f;
#pragma unroll
      for (int m = 0; m < C; ++m) {
        const float one = __shfl_sync(kAll, square, (lane - c + m) & 31);
        total = m == 0 ? one : __fadd_rn(total, one);
      }
      square = total;
    }
    if (mine) {
      const float q1 = __fmul_rn(step1, ball(square, ball_of(radius())));
      float* to = shared + W::EXCHANGE + (row < kChunk - 1 ? row : row + (k & 1)) * W::ROW - 1 - (k & 1);
      to[exchange(0, c)] =
          REST_FIRST ? fmaf(P.rest, old1, __fmul_rn(P.rho, q1)) : fmaf(P.rho, q1, __fmul_rn(P.rest, old1));
      if constexpr (TGV) {
        to[exchange(2, c)] = nb1;
        to[exchange(3, c)] = nb2;
      }
    }
    __syncwarp();
    if (lane == 0) {
      barrier_arrive(&bars.go[k & 1]);
      barrier_arrive(&bars.drained[k & 1]);
    }
    return true;
  }

  // ---- Warp 4: the copies, slots n = 0 .. (i1 - i0) / 2 + 1, each once the rows it held are drained; and the left column of each chunk, a chunk ahead.
  __device__ __forceinline__ bool copy_warp(const CUtensorMap* map, WalkBarriers& bars, const volatile int* failed, int lane,
                                            int& issued) const {
    const int chunks = (i1 - i0) / kChunk, slots = (i1 - i0) / 2 + 2;
    auto issue_to = [&](int end) {
      for (; issued < min(end, slots); ++issued) {
        if (lane == 0) {
          const int s = issued % kSlots;
          barrier_expect(&bars.full[s], (W::F + 1) * C * W::PLANE * 4);
          if constexpr (UNROLLED) {
            load_fields(shared + s * W::SLOT, map, &bars.full[s], x0 - kHalo, i0 - 2 + 2 * issued, image);
          } else {
            load_box(shared + s * W::SLOT, map, &bars.full[s], x0 - kHalo, i0 - 2 + 2 * issued, 0);
          }
        }
      }
    };
    // Nothing of the state is read or written before the launch before this one is done: every other
    // warp waits for rows that are copied from here on. Only then may the next launch's CTAs take the
    // places that this one's leave (to wait here, with what does not depend on it done): one launch
    // waits at a time, never a chain of them.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    issue_to(kSlots);
    if (!left_column(bars, failed, 0, lane)) return false;
    for (int k = 0; k < chunks; ++k) {
      if (!__all_sync(kAll, wait_unless(&bars.drained[k & 1], (k >> 1) & 1, failed))) return false;
      issue_to(kSlots + 1 + kDual * (k + 1));
      // The left column of chunk k is read once v of the chunk is made; the next goes beside it.
      if (k > 0 && !__all_sync(kAll, wait_unless(&bars.luma[(k - 1) & 1], ((k - 1) >> 1) & 1, failed))) return false;
      if (k + 1 < chunks && !left_column(bars, failed, k + 1, lane)) return false;
    }
    return true;
  }

  // ---- The other warps: the proximal map of channel c (its part of the strip), block row by block
  // row of it, the levels looked up one ahead. When one of its two tiles is full, the other is free:
  // the chunks that fill it may go.
  template <int PR, int PC>
  __device__ __forceinline__ bool prox_warp(WalkBarriers& bars, const volatile int* failed, const WalkFactors& F, int c,
                                            int part, int lane, double& sum) const {
    constexpr int BH = 8 * PR;
    const int j = x0 + 32 * part + lane, pitch = Q.dual.g.pitch;
    std::uint64_t* const full = c == 0 ? bars.luma : bars.chroma;
    float* const tile = shared + (c == 0 ? W::LUMA : W::CHROMA + (c - 1) * BH * WIDTH) + 32 * part;
    const int stride = c == 0 ? BH * WIDTH : (C - 1) * BH * WIDTH;
    float* next = Q.next + c * Q.dual.g.plane + static_cast<std::size_t>(i0) * pitch + j;
    auto let_go = [&](int band) {
#pragma unroll
      for (int k = 0; k < PR; ++k) {
        if (lane == 0) barrier_arrive(&bars.go[(band * PR + k) & 1]);
      }
    };
    let_go(0);
    Ahead ahead = look_ahead<PR, PC>(Q, c, j, i0, lane);
    for (int i = i0, b = 0; i < i1; i += BH, ++b) {
      const Ahead now = ahead;
      if (i + BH < i1) ahead = look_ahead<PR, PC>(Q, c, j, i + BH, lane);
      if (!__all_sync(kAll, wait_unless(&full[b & 1], (b >> 1) & 1, failed))) return false;
      let_go(b + 1);
      const ComponentDevice& D = Q.component[c];
      const std::size_t block = static_cast<std::size_t>(i / BH) * D.block_columns + j / (8 * PC);
      prox_rows<PR, PC, WIDTH, KEEP == 1>(tile + (b & 1) * stride, now, F, next, pitch, lane, j < Q.dual.g.columns, D,
                                          block, Q.v + (next - Q.next), Q.dual.g.recorded_row(i), sum);
      __syncwarp();
      next += static_cast<std::size_t>(BH) * pitch;
    }
    return true;
  }
};

template <bool TGV, int C, bool COUPLED, int CR, int CC, int KEEP>
__global__ void __launch_bounds__(walk_threads<C>(), walk_ctas<TGV, C>())
    walk_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ IterationParams Q) {
  using W = WalkLayout<TGV, C, CR>;
  extern __shared__ __align__(128) float shared[];
  __shared__ __align__(8) WalkBarriers bars;
  __shared__ WalkFactors factors[C];
  __shared__ int failed;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const ProxFactors* all = Q.component[c].factors;
    const float4* from = all->plain;  // and `flat` behind it
    float4* to = factors[c].plain;
    for (int k = tid; k < 128; k += walk_threads<C>()) to[k] = __ldg(from + k);
    if (tid == 0) {
      factors[c].all = all;
      factors[c].general = all->mmse != 0 || all->costed != 0;
    }
  }
  if (tid == 0) {
    for (int s = 0; s < kSlots; ++s) barrier_init(&bars.full[s], 1);
    for (int s = 0; s < 2; ++s) {
      barrier_init(&bars.drained[s], kDual + 1);
      barrier_init(&bars.go[s], 1 + (C == 1 ? 2 : C));
      barrier_init(&bars.luma[s], kDual);
      barrier_init(&bars.chroma[s], kDual * CR);
    }
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int i0 = blockIdx.y * Q.strip_rows;
  const Walk<TGV, C, COUPLED, CR, CC, KEEP> walk{Q, shared, static_cast<int>(blockIdx.x) * W::WIDTH, i0,
                                           min(i0 + Q.strip_rows, Q.dual.g.rows)};
  bool good = true;
  int issued = 0;
  if (warp < kDual) {
    good = walk.dual_warp(bars, &failed, warp, lane);
  } else if (warp == kDual) {
    good = walk.copy_warp(&map, bars, &failed, lane, issued);
  } else {
    const int z = warp - kDual - 1;
    double sum = 0.0;  // G's terms
    if constexpr (C == 1) {
      good = walk.template prox_warp<1, 1>(bars, &failed, factors[0], 0, z, lane, sum);
    } else if (CR * CC == 1 || z == 0) {
      good = walk.template prox_warp<1, 1>(bars, &failed, factors[z], z, 0, lane, sum);
    } else {
      good = walk.template prox_warp<CR, CC>(bars, &failed, factors[z], z, 0, lane, sum);
    }
    if constexpr (KEEP == 1) {
#pragma unroll
      for (int offset = 16; offset > 0; offset >>= 1) sum += __shfl_down_sync(kAll, sum, offset);
      const int cta = blockIdx.x + gridDim.x * blockIdx.y;
      if (lane == 0) Q.partials[C == 1 ? 0 : z][C == 1 ? 2 * cta + z : cta] = sum;
    }
  }
  if (!good) {
    *static_cast<volatile int*>(&failed) = 1;
    if (lane == 0 && Q.dual.error != nullptr) atomicExch(Q.dual.error, 1);
    // No copy may still write into shared memory when the CTA leaves.
    for (int n = max(issued - kSlots, 0); n < issued; ++n) barrier_wait(&bars.full[n % kSlots], (n / kSlots) & 1);
  }
}

// The strip height that finishes the walk soonest: its CTAs in waves of the CTAs the device
// holds, each as long as its rows and its start and end (about two chunks).
int walk_rows(const Geometry& g, int ctas, int width, int band) {
  const long long strips = (g.columns + width - 1) / width;
  int best = band;
  long long best_cost = -1;
  for (int height = band; height <= 512; height += band) {
    const long long items = strips * ((g.rows + height - 1) / height);
    const long long cost = (items + ctas - 1) / ctas * (height + 2 * kChunk);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = height;
    }
  }
  return best;
}

// A walk of a picture by `kernel` (`bytes` of shared memory, strips of `width` columns, heights of whole
// bands) with the arguments `map` and `args`, whose strip height, in `step`, is set here. *grid: its CTAs.
template <typename Args>
cudaError_t launch_strips(void (*kernel)(CUtensorMap, Args), int threads, std::size_t bytes, int width, int band,
                          const CUtensorMap& map, Args& args, IterationParams& step, std::atomic<int> (&resident)[64],
                          cudaStream_t s, int* ctas_of_grid = nullptr) {
  // Once per device: the shared-memory size above 48 KB, and how many CTAs the device holds.
  int device = 0;
  cudaGetDevice(&device);
  int ctas = resident[device & 63].load();
  if (ctas == 0) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    int per_sm = 0, sms = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, bytes);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) return e;
    ctas = std::max(1, per_sm * sms);
    resident[device & 63].store(ctas);
  }
  const Geometry& g = step.dual.g;
  // The last picture's strip height: the same for all of a solve's launches.
  thread_local struct {
    int rows = 0, columns = 0, ctas = 0, width = 0, band = 0, height = 0;
  } last;
  if (last.rows != g.rows || last.columns != g.columns || last.ctas != ctas || last.width != width || last.band != band) {
    last = {g.rows, g.columns, ctas, width, band, walk_rows(g, ctas, width, band)};
  }
  step.strip_rows = last.height;
  const dim3 grid((g.columns + width - 1) / width, (g.rows + step.strip_rows - 1) / step.strip_rows);
  if (ctas_of_grid != nullptr) *ctas_of_grid = static_cast<int>(grid.x * grid.y);
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = bytes;
  config.stream = s;
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &early;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, map, args);
}

template <bool TGV, int C, bool COUPLED, int CR, int CC, int KEEP>
cudaError_t launch_one(const CUtensorMap& map, const IterationParams& p, cudaStream_t s, int* partials) {
  using W = WalkLayout<TGV, C, CR>;
  static std::atomic<int> resident[64] = {};
  IterationParams q = p;
  const cudaError_t e = launch_strips(walk_kernel<TGV, C, COUPLED, CR, CC, KEEP>, walk_threads<C>(),
                                      W::FLOATS * sizeof(float), W::WIDTH, 8 * CR, map, q, q, resident, s, partials);
  if (partials != nullptr && C == 1) *partials *= 2;
  return e;
}

template <bool TGV, bool COUPLED, int KEEP>
cudaError_t launch_cells(const CUtensorMap& map, const IterationParams& p, int cr, int cc, cudaStream_t s, int* partials) {
  if (cr == 1 && cc == 1) return launch_one<TGV, 3, COUPLED, 1, 1, KEEP>(map, p, s, partials);
  if (cr == 1 && cc == 2) return launch_one<TGV, 3, COUPLED, 1, 2, KEEP>(map, p, s, partials);
  if (cr == 2 && cc == 1) return launch_one<TGV, 3, COUPLED, 2, 1, KEEP>(map, p, s, partials);
  if (cr == 2 && cc == 2) return launch_one<TGV, 3, COUPLED, 2, 2, KEEP>(map, p, s, partials);
  return cudaErrorInvalidValue;
}

template <int KEEP>
cudaError_t launch_keep(const CUtensorMap& map, const IterationParams& p, bool tgv, bool coupled, int cr, int cc,
                        cudaStream_t s, int* partials) {
  if (p.dual.g.channels == 1) {
    return tgv ? launch_one<true, 1, false, 1, 1, KEEP>(map, p, s, partials)
               : launch_one<false, 1, false, 1, 1, KEEP>(map, p, s, partials);
  }
  if (p.dual.g.channels != 3) return cudaErrorInvalidValue;
  if (tgv) {
    return coupled ? launch_cells<true, true, KEEP>(map, p, cr, cc, s, partials)
                   : launch_cells<true, false, KEEP>(map, p, cr, cc, s, partials);
  }
  return coupled ? launch_cells<false, true, KEEP>(map, p, cr, cc, s, partials)
                 : launch_cells<false, false, KEEP>(map, p, cr, cc, s, partials);
}

}  // namespace

}  // namespace urb
