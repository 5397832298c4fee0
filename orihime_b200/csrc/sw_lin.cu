// Soft Smith-Waterman forward / adjoint in the scaled linear domain (sm_100a),
// local alignment with linear or affine gaps.  Compiled as part of sw_capi.cu
// after sw_kernels.cu, whose band decomposition, task queue, cross-band
// buffers, polling and pair finish this file reuses.
//
// What bounds it.  4096 ragged pairs fill every warp slot: the forward moves
// about 7 GB (scores and checkpoints) in 1.68 ms, two thirds of the measured
// copy rate, and the adjoint is bound by instruction issue and dependent
// results (3.12 ms).  A small batch is bound by the latency of one step of one
// warp: about 120 ns at 4 columns per lane and 160 at 8 (180 and 390 before
// the steps were packed and their bounds, address and frame arithmetic cut),
// times the steps of the longest chain of bands.
//
// Why a linear domain
// -------------------
// Every term of the reference recurrence is positive, so instead of
// log-sum-exp over scaled log values (one ex2 per term, one lg2 per state:
// 14 MUFU ops per affine cell forward, 15 more in the adjoint) the DP can run
// on the exponentials themselves.  With E = 2^(s k) (k = log2(e) / T),
// G_o = 2^(go k), G_e = 2^(ge k) the local affine recurrence of
// src/sw_affine/kernels_cpu.cpp:94-196 becomes
//     M[i,j] = E[i,j] * (M + I + D)[i-1,j-1] + E[i,j]      (the "+ E": a fresh start)
//     I[i,j] = G_o * M[i-1,j] + G_e * I[i-1,j]
//     D[i,j] = G_o * M[i,j-1] + G_e * D[i,j-1]
//     Z      = 1 + sum over all cells and states,  S = T ln Z,
// and the linear one (src/sw/kernels_cpu.cpp:70-160)
//     A[i,j] = E[i,j] * (A[i-1,j-1] + 1) + G (A[i-1,j] + A[i,j-1]).
// The adjoint is the outside recursion beta = dZ/d(cell) over the successors,
//     beta_M = 1 + t(i+1,j+1) + G_o (beta_I(i+1,j) + beta_D(i,j+1)),  t = E * beta_M,
//     beta_I = 1 + t(i+1,j+1) + G_e beta_I(i+1,j),   beta_D = 1 + t + G_e beta_D(i,j+1),
// with the map P = M beta_M / Z (linear: E (A_diag + 1) beta / Z) and the
// parameter gradients as expected transition counts.  One ex2 per cell
// (the emission E), the rest multiply-adds.
//
// Range
// -----
// Values span far more than fp32's exponent range, so each lane keeps its R
// columns of a row as float mantissas under one power-of-two frame:
// value = m * 2^e.  A step computes its row in the frame et = max of its
// inputs' normalised frames (the lane's previous row, the left lane's row and
// the left lane's previous row), which makes every converted input <= 1;
// then the row's sum gives the normalised frame n = et + exponent(sum) in
// which the row is <= 1.  Within a lane rows are never rescaled: the raw
// values keep the compute frame et and every use scales them by
// 2^(frame - target) (a power-of-two factor built from the exponent bits,
// folded into the gap factors).  What a lane passes on is normalised.  Frames
// are floored at 0: the empty alignment's weight 1 is always representable
// and Z >= 1.  Scores are within |s|/T <= 80 (the host's domain check), so
// E <= 2^115.4 and a step's raw values stay below 2^122.
//
// What is lost.  A lane's columns share one frame, so a column more than 126
// bits below the lane's row is dropped (fewer by what a row of the lane gained
// in one step: its own values are converted in one factor).  It matters where
// the dropped column's path would later have caught up, which takes matches
// worth those bits inside the lane.  Scores with a standard deviation of 1 to
// 6 T never came near it at 4 columns, 6 T to 9 T did without a wrong result.
// Pairs of 512 with a wrong map (more than 1e-3 off the log domain), scores
// 3 N(0, 1), gap -1 (linear, the worse model), 600 x 172 / 500 x 384, at 2, 4
// and 8 columns per lane:
//   T = 0.5    0 / 0     0 / 0      1 / 0
//   T = 0.35   0 / 0     0 / 0    335 / 45
//   T = 0.25   0 / 0    75 / 6    511 / 460
// 172 x 600, wide instead of tall: none.  At a deviation of 25 T (the domain
// check lets scores up to 80 T pass) most pairs are wrong at 4 columns and many
// at 2.  Splitting the lane's own conversions into two factors saves none of
// them (the same counts in a restatement of the step): what is lost there is
// the frame's range itself.  Nothing detects it; the padded entry points and
// ragged.cols_limit choose the columns by the temperature, and a call beyond
// that needs the log domain (swb_options).
//
// The kernels run when every transition factor is at most 1 (gaps <= 0);
// otherwise the host uses the log-domain kernels of sw_kernels.cu.
#include "sw_kernels.cuh"

namespace swb {

// 2^d for an integer d <= 127 (0 for d < -126): frame conversion factors.
// Conversions go to a frame at least as large as the source's normalised
// frame, so d <= 126 always (a raw value's frame exceeds its normalised frame
// by at most 126, when the values are below 1).
__device__ __forceinline__ float p2i(int d) {
  d = max(d, -127);
  return __int_as_float((d + 127) << 23);
}
// 2^d for any integer d, saturated to [0, 2^127].
__device__ __forceinline__ float p2any(int d) {
  d = min(max(d, -127), 127);
  return __int_as_float((d + 127) << 23);
}
// Upper bound k of log2 of a non-negative float: m <= 2^k, tight within a
// factor 2 for normal m (0 and subnormals give -126).
__device__ __forceinline__ int fexp(float m) {
  return (int)((__float_as_uint(m) >> 23) & 0xffu) - 126;
}

constexpr float XMAX = 118.f;   // scaled scores above this are clamped (|s|/T <= 80 gives 115.4)

// Quiet chunks of the adjoint: every posterior in the chunk and every flow
// out of it below 2^-SWB_LQUIET (relative to Z).  At 45 the posterior mass a
// pair can lose over all its chunks stays below ~1e-9.
#ifndef SWB_LQUIET
#define SWB_LQUIET 45
#endif

// Asynchronous global -> shared copy (cp.async): the adjoint stages the next
// chunk's checkpoint while it runs the current chunk, so it occupies no
// registers in between.
__device__ __forceinline__ void lcp16(float* dst, const float* src, int src_size) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(src_size)
               : "memory");
}
__device__ __forceinline__ void lcp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void lcp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---------------------------------------------------------------------------
// whole-chunk row pieces
// ---------------------------------------------------------------------------
// In the skewed wavefront lane l works on row t - l + 1 at step t, so one
// store of every lane touches 32 rows: 32 cache lines per warp instruction.
// Over a checkpoint chunk (C steps), though, row i is worked on by C
// adjacent lanes, whose columns are one contiguous piece of 4 C R bytes.  The
// adjoint writes the map rows of a quiet chunk (zeros) in whole row pieces:
// round `it`, item k = 32 it + lane is float4 h of lane l at step cu with
// q = k % NI, rho = k / NI, cu = q / HR, h = q % HR, l = rho - (C - 1) + cu;
// its row is kc C + cu - l + 1.  Every (cu, l, h) is one item; NI
// consecutive items are one row piece.
template <int R> struct Pieces {
  static constexpr int HR = R / 4;                    // float4 per lane and row
  static constexpr int NI = C_STEPS * HR;             // items per row piece
  static constexpr int ROWS = 32 + C_STEPS - 1;       // rows a chunk touches
  static constexpr int ROUNDS = (ROWS * NI + 31) / 32;
};

// Zero chunk kc's map rows of a band (a quiet chunk) in whole row pieces.
// Rows outside [1, L1] are not written; every column up to the row pitch is.
// The rounds run as a loop: unrolled, their per-lane item indices would stay
// live in registers across the adjoint.
template <int R>
__device__ __forceinline__ void zero_chunk_rows(const Pair& pr, int kc, int col0, int lane) {
  using P = Pieces<R>;
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
  for (int it = 0; it < P::ROUNDS; ++it) {
    const int k = it * 32 + lane;
    const int rho = k / P::NI, q = k - rho * P::NI;
    const int cu = q / P::HR, h = q - cu * P::HR;
    const int l = rho - (C_STEPS - 1) + cu;
    if (rho < P::ROWS && l >= 0 && l < 32) {
      const int i = kc * C_STEPS + cu - l + 1;
      const int col = col0 + R * l + 4 * h;
      if (i >= 1 && i <= pr.L1 && col < pr.ld) {
        float* dst = pr.m + (size_t)(i - 1) * pr.ld + col;
        if (pr.vec) {
          *reinterpret_cast<float4*>(dst) = z;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (col + e < pr.ld) dst[e] = 0.f;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// packed columns
// ---------------------------------------------------------------------------
// A lane's R columns are kept as R / 2 float2 pairs (k, k + R/2), so that one
// packed fp32 instruction (fma.rn.f32x2 and its kin, the same rounding per
// component) works on two columns, and the diagonal inputs of pair k are
// simply pair k - 1 of the row above: only pair 0 has to be put together.
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
// column c of a row of pairs
template <int H> __device__ __forceinline__ float& col(float2 (&p)[H], int c) {
  return c < H ? p[c < H ? c : 0].x : p[c >= H ? c - H : 0].y;
}
// Sum over the columns, a short tree.
template <int H> __device__ __forceinline__ float sum2(const float2 (&p)[H]) {
  float2 s[H];
#pragma unroll
  for (int k = 0; k < H; ++k) s[k] = p[k];
#pragma unroll
  for (int h = 1; h < H; h *= 2)
#pragma unroll
    for (int k = 0; k + h < H; k += 2 * h) s[k] = add2(s[k], s[k + h]);
  return s[0].x + s[0].y;
}
// 2^d as bits for d + 127 given: 0 below the exponent range.
__device__ __forceinline__ float p2b(int d127) { return __int_as_float(max(d127, 0) << 23); }

// Checkpoint floats per lane (CKF, padded to float4), one checkpoint record
// (LREC: CK4 groups of [lane][4]) and adjoint shared-memory floats per lane
// per step (FW).  A band's checkpoint region holds ceil(nchunks / ck_every)
// records, then one float per chunk: the chunk's largest normalised alpha
// frame (the adjoint's quiet-chunk test).  A record keeps M and I of the
// lane's row (linear: A), D of its first column, the left lane's diagonal sum
// and two frames; the rest of D, the column sums and the normalised frame are
// rebuilt with the forward's own operations, bit for bit: 20 floats per lane
// at 8 columns per lane (12 for the linear gap).
template <int NS, int R> struct LDims {
  static constexpr int H = R / 2;
  static constexpr int CKV = NS == 3 ? 2 * R + 4 : R + 3;
  static constexpr int CKF = (CKV + 3) / 4 * 4;
  static constexpr int CK4 = CKF / 4;
  static constexpr int LREC = CKF * 32;
  // affine: M, I, D (raw) and the scaled score per column; linear: A, the
  // emission part E (A_diag + 1), and the scaled score; then the frame e
  static constexpr int NF = NS == 3 ? 4 : 3;
  static constexpr int FW = NF * R + 1;
};

// Lane state of the forward wavefront.
template <int NS, int R> struct LState {
  static constexpr int H = R / 2;
  float2 v[NS == 3 ? 2 : 1][H];    // raw M and I (linear: A) of the lane's latest row (frame e)
  float2 c[NS == 3 ? H : 1];       // affine: the row's column sums (M + I) + D (frame e)
  float ds;                        // the left lane's column sum (linear: A) of that row, last column (frame nd)
  float od, oc;                    // out to the right lane, in the normalised frame n: D of the column after
                                   // the last, the last column's sum
  int e, n, nd;                    // raw frame, normalised frame, the left lane's normalised frame of that row
};

// Exponent bound of a non-negative sum: x <= 2^(sexp(x) - 126).
__device__ __forceinline__ int sexp(float x) { return (int)(__float_as_uint(x) >> 23); }

template <int NS, int R>
__device__ __forceinline__ void lstate_zero(LState<NS, R>& s) {
  constexpr int H = R / 2;
#pragma unroll
  for (int k = 0; k < H; ++k) {
    s.v[0][k] = dup2(0.f);
    if constexpr (NS == 3) { s.v[1][k] = dup2(0.f); s.c[k] = dup2(0.f); }
  }
  s.ds = 0.f; s.od = 0.f; s.oc = 0.f;
  s.e = 0; s.n = 0; s.nd = 0;
}

// Columns past the pair (DM): 0 the band has none, 1 it may have some and they
// are masked without a branch, 2 a warp-uniform branch on whether it has any.
// The kernels at 8 columns per lane, which run with every scheduler full,
// keep one copy of their steps (2, and no copy for chunks inside the pair):
// with several the instruction cache misses cost more than the branches
// (4096 ragged pairs, forward + adjoint: 7.0 ms against 5.0).  The narrower
// ones run few warps, and there a branch costs its latency.
template <int R> __host__ __device__ constexpr bool split_code() { return R < 8; }
template <int DM> __device__ __forceinline__ bool masks(bool has_dead) {
  return DM == 1 || (DM == 2 && has_dead);
}

// D of a row from its first column's D and the row's M: D runs along the
// lane's columns, one fma per column on that chain; `od` is the next lane's
// first D.  Columns past the pair get 0.
template <int NS, int R, int DM>
__device__ __forceinline__ void ldchain(const float2 (&m)[R / 2], float d0, float gO, float gE, int nlive, bool hd,
                                        float2 (&d)[R / 2], float& od) {
  constexpr int H = R / 2;
  float2 t[H];
#pragma unroll
  for (int k = 0; k < H; ++k) t[k] = mul2(dup2(gO), m[k]);
  col(d, 0) = d0;
#pragma unroll
  for (int c = 1; c < R; ++c) col(d, c) = fmaf(gE, col(d, c - 1), col(t, c - 1));
  od = fmaf(gE, col(d, R - 1), col(t, R - 1));
  if (masks<DM>(hd)) {
#pragma unroll
    for (int c = 0; c < R; ++c)
      if (c >= nlive) col(d, c) = 0.f;
  }
}

// The normalised frame of a row from its raw frame e and sum rs (which bounds
// every value of the row: all are >= 0), and the outputs in it.  The outputs
// are normalised here, not by the receiver: its factor reaches down to 2^-126
// only, and a raw value can stand up to 2^115 above its frame, so a value
// 2^-12 below the receiver's row could become 0 there (affine pairs of 32 to
// 1000 at T = 0.25, 4 columns per lane: 4 of 400 lost paths that way, 1 this
// way; 600 x 172, linear: 39 and 23 of 512).  The two products,
// with the split scale of the adjoint's posteriors, cost up to 3 % of a call
// (64 x 1024^2 883 -> 909 us, 1 x 1023 x 2047 752 -> 754); by the receiver,
// which then needs e as well, they cost as much or more.
template <int NS, typename S>
__device__ __forceinline__ void lnormal(S& s, int e, float rs) {
  s.n = max(e - 126 + sexp(rs), 0);
  const float f = p2b(e - s.n + 127);
  if constexpr (NS == 3) s.od *= f;
  s.oc *= f;
}

template <int NS, int R>
__device__ __forceinline__ void lck_store(float* rec, int lane, const LState<NS, R>& s, float d0) {
  using L = LDims<NS, R>;
  constexpr int H = R / 2;
  float x[L::CKF];
#pragma unroll
  for (int q = 0; q < (NS == 3 ? 2 : 1); ++q)
#pragma unroll
    for (int k = 0; k < H; ++k) { x[q * R + 2 * k] = s.v[q][k].x; x[q * R + 2 * k + 1] = s.v[q][k].y; }
  constexpr int V = NS == 3 ? 2 * R : R;
  x[V] = s.ds;
  x[V + 1] = __int_as_float(s.e);
  x[V + 2] = __int_as_float(s.nd);
  if constexpr (NS == 3) x[V + 3] = d0;
#pragma unroll
  for (int f = L::CKV; f < L::CKF; ++f) x[f] = 0.f;
#pragma unroll
  for (int g = 0; g < L::CK4; ++g)
    reinterpret_cast<float4*>(rec + g * 128)[lane] = make_float4(x[4 * g], x[4 * g + 1], x[4 * g + 2], x[4 * g + 3]);
}

// Restores the lane state of a record (`rec` + lane: global or staged in
// shared memory), rebuilding D, the sums and the normalised frame with the
// operations lcells used for that row; `d` is the row's D.
template <int NS, int R, int DM>
__device__ __forceinline__ void lck_restore(const float* rec, int lane, LState<NS, R>& s, float gO, float gE,
                                            int nlive, bool hd, float2 (&d)[R / 2]) {
  using L = LDims<NS, R>;
  constexpr int H = R / 2;
  float x[L::CKF];
#pragma unroll
  for (int g = 0; g < L::CK4; ++g) {
    const float4 y = reinterpret_cast<const float4*>(rec + g * 128)[lane];
    x[4 * g] = y.x; x[4 * g + 1] = y.y; x[4 * g + 2] = y.z; x[4 * g + 3] = y.w;
  }
#pragma unroll
  for (int q = 0; q < (NS == 3 ? 2 : 1); ++q)
#pragma unroll
    for (int k = 0; k < H; ++k) s.v[q][k] = make_float2(x[q * R + 2 * k], x[q * R + 2 * k + 1]);
  constexpr int V = NS == 3 ? 2 * R : R;
  s.ds = x[V];
  s.e = __float_as_int(x[V + 1]);
  s.nd = __float_as_int(x[V + 2]);
  float rs;
  if constexpr (NS == 3) {
    ldchain<NS, R, DM>(s.v[0], x[V + 3], gO, gE, nlive, hd, d, s.od);
#pragma unroll
    for (int k = 0; k < H; ++k) s.c[k] = add2(add2(s.v[0][k], s.v[1][k]), d[k]);
    s.oc = s.c[H - 1].y;
    rs = sum2(s.c);
  } else {
    s.od = 0.f;
    s.oc = s.v[0][H - 1].y;
    rs = sum2(s.v[0]);
  }
  lnormal<NS>(s, s.e, rs);
}

// One step of the forward wavefront for one lane: (xd, xc) are the left
// lane's outputs of this row in its normalised frame xn, E the emissions
// 2^(s k) (0 past the pair).  Updates the state to this row in the
// frame et (its raw frame from then on) and returns the row's sum over its
// columns and states in `rs`.
// Affine: M, I and `d` = D; linear: A and `d` = the emission part.
template <int NS, int R, int DM>
__device__ __forceinline__ void lcells(LState<NS, R>& s, float xd, float xc, int xn,
                                       const float2 (&E)[R / 2], float gO, float gE, int nlive, bool hd,
                                       float2 (&d)[R / 2], float& rs) {
  constexpr int H = R / 2;
  // the row's frame is at least every input's normalised frame, so that every
  // converted input is <= 1 (a raw value's frame exceeds its normalised frame
  // by at most 126)
  const int et = max(max(s.n, xn), s.nd);
  const int q = 127 - et;
  const float fU = p2b(s.e + q), fL = p2b(xn + q), fD = p2b(s.nd + q);
  s.nd = xn;
  const float2 fU2 = dup2(fU), st2 = dup2(p2b(q));   // st: the fresh-start term 1 in frame et
  if constexpr (NS == 3) {
    float2 m[H];
#pragma unroll
    for (int k = 0; k < H; ++k) {
      const float2 p = k == 0 ? make_float2(s.ds, s.c[H - 1].x) : s.c[k > 0 ? k - 1 : 0];
      m[k] = mul2(E[k], fma2(k == 0 ? make_float2(fD, fU) : fU2, p, st2));
    }
    const float2 gOu = dup2(gO * fU), gEu = dup2(gE * fU);
#pragma unroll
    for (int k = 0; k < H; ++k) s.v[1][k] = fma2(gOu, s.v[0][k], mul2(gEu, s.v[1][k]));
    ldchain<NS, R, DM>(m, xd * fL, gO, gE, nlive, hd, d, s.od);
#pragma unroll
    for (int k = 0; k < H; ++k) {
      s.v[0][k] = m[k];
      s.c[k] = add2(add2(m[k], s.v[1][k]), d[k]);
    }
    s.ds = xc;
    s.oc = s.c[H - 1].y;
    rs = sum2(s.c);
  } else {
    const float2 gU = dup2(gO * fU);
    float2 x[H];
#pragma unroll
    for (int k = 0; k < H; ++k) {
      const float2 p = k == 0 ? make_float2(s.ds, s.v[0][H - 1].x) : s.v[0][k > 0 ? k - 1 : 0];
      d[k] = mul2(E[k], fma2(k == 0 ? make_float2(fD, fU) : fU2, p, st2));
    }
#pragma unroll
    for (int k = 0; k < H; ++k) x[k] = fma2(gU, s.v[0][k], d[k]);
    s.ds = xc;
    col(s.v[0], 0) = fmaf(gO, xc * fL, col(x, 0));
#pragma unroll
    for (int c = 1; c < R; ++c) col(s.v[0], c) = fmaf(gO, col(s.v[0], c - 1), col(x, c));
    if (masks<DM>(hd)) {
#pragma unroll
      for (int c = 0; c < R; ++c)
        if (c >= nlive) { col(s.v[0], c) = 0.f; col(d, c) = 0.f; }
    }
    s.oc = s.v[0][H - 1].y;
    rs = sum2(s.v[0]);
  }
  // the row sum over columns and states is the row's partition term
  s.e = et;
  lnormal<NS>(s, et, rs);
}

// Scaled scores and emissions of one step as pairs: clamped at XMAX, NEG
// (E = 0) in columns past the pair.
template <int R, int DM>
__device__ __forceinline__ void lemit(const float (&sb)[R], float k, int nlive, bool hd, float2 (&xs)[R / 2],
                                      float2 (&E)[R / 2]) {
  constexpr int H = R / 2;
  float x[R];
#pragma unroll
  for (int c = 0; c < R; c += 2) {
    const float2 t = mul2(make_float2(sb[c], sb[c + 1]), dup2(k));
    x[c] = fminf(t.x, XMAX);
    x[c + 1] = fminf(t.y, XMAX);
  }
  if (masks<DM>(hd)) {
#pragma unroll
    for (int c = 0; c < R; ++c)
      if (c >= nlive) x[c] = NEG;
  }
#pragma unroll
  for (int j = 0; j < H; ++j) {
    xs[j] = make_float2(x[j], x[j + H]);
    E[j] = make_float2(ex2(x[j]), ex2(x[j + H]));
  }
}

// A lane's walk down (or up) the rows of its columns: whole float4 (float2 at
// 2 columns) pieces when rows are 16-byte aligned (vec; a piece may reach past
// the pair but not past the row pitch), else one load per column.  A row
// outside the pair leaves `o` as it was: those values are finite and unused.
// `fetch` loads without any test, for chunks whose rows are inside for every
// lane (`inside`): a lane past the pair then reads on into the next rows,
// which must still belong to the pair, and its columns are not used.
template <int R> struct Rows {
  static constexpr int Q = R >= 4 ? 4 : 2;   // columns per piece
  const float* base;   // row 1, the lane's first column
  long long ld;
  int L1, l1a, l1b;    // rows; rows of the first and second piece (0: past the pitch)
  int nlive;
  int last;            // the last row whose band width can be read whole
  bool vec;
  __device__ __forceinline__ void init(const Pair& pr, int jl, int col0) {
    base = pr.s + jl;
    ld = pr.ld;
    L1 = pr.L1;
    vec = pr.vec;
    nlive = min(max(pr.L2 - jl, 0), R);
    l1a = jl + Q <= pr.ld ? L1 : 0;
    l1b = jl + 2 * Q <= pr.ld ? L1 : 0;
    const int over = col0 + 32 * R - pr.ld;   // floats past the row's end
    last = over > 0 ? L1 - (over + pr.ld - 1) / pr.ld : L1;
  }
  // chunk kc's rows are inside the pair for every lane, and reading the whole
  // band's width of each stays within it
  __device__ __forceinline__ bool inside(int kc) const { return kc >= 32 / C_STEPS && (kc + 1) * C_STEPS <= last; }
  template <bool VEC> __device__ __forceinline__ void fetch(const float* p, float (&o)[R]) const {
    if constexpr (VEC && R == 2) {
      const float2 v = __ldg(reinterpret_cast<const float2*>(p));
      o[0] = v.x; o[1] = v.y;
    } else if constexpr (VEC) {
#pragma unroll
      for (int h = 0; h < R / 4; ++h) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(p) + h);
        o[4 * h] = v.x; o[4 * h + 1] = v.y; o[4 * h + 2] = v.z; o[4 * h + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int c = 0; c < R; ++c) o[c] = __ldg(p + c);
    }
  }
  __device__ __forceinline__ const float* at(int i) const { return base + (long long)(i - 1) * ld; }
  __device__ __forceinline__ void load(const float* p, int i, float (&o)[R]) const {
    if (vec) {
      if ((unsigned)(i - 1) < (unsigned)l1a) {
        if constexpr (R == 2) {
          const float2 v = __ldg(reinterpret_cast<const float2*>(p));
          o[0] = v.x; o[1] = v.y;
        } else {
          const float4 v = __ldg(reinterpret_cast<const float4*>(p));
          o[0] = v.x; o[1] = v.y; o[R > 2 ? 2 : 0] = v.z; o[R > 3 ? 3 : 0] = v.w;
        }
      }
      if constexpr (R == 8) {
        if ((unsigned)(i - 1) < (unsigned)l1b) {
          const float4 v = __ldg(reinterpret_cast<const float4*>(p) + 1);
          o[4] = v.x; o[5] = v.y; o[6] = v.z; o[7] = v.w;
        }
      }
    } else if ((unsigned)(i - 1) < (unsigned)L1) {
#pragma unroll
      for (int c = 0; c < R; ++c)
        if (c < nlive) o[c] = __ldg(p + c);
    }
  }
};

// Writes a row of the map for the lane's columns (a row inside the pair):
// columns past the pair hold 0, and those inside the row pitch are written.
template <int R>
__device__ __forceinline__ void store_pairs(float* dst, int jl, const Pair& pr, float2 (&v)[R / 2]) {
  constexpr int H = R / 2;
  if (pr.vec) {
    if constexpr (R == 2) {
      if (jl + 2 <= pr.ld) *reinterpret_cast<float2*>(dst) = v[0];
    } else if constexpr (R == 4) {
      if (jl + 4 <= pr.ld) *reinterpret_cast<float4*>(dst) = make_float4(v[0].x, v[H > 1 ? 1 : 0].x, v[0].y, v[H > 1 ? 1 : 0].y);
    } else {
      if (jl + 4 <= pr.ld) reinterpret_cast<float4*>(dst)[0] = make_float4(v[0].x, v[H > 1 ? 1 : 0].x, v[H > 2 ? 2 : 0].x, v[H > 3 ? 3 : 0].x);
      if (jl + 8 <= pr.ld) reinterpret_cast<float4*>(dst)[1] = make_float4(v[0].y, v[H > 1 ? 1 : 0].y, v[H > 2 ? 2 : 0].y, v[H > 3 ? 3 : 0].y);
    }
  } else {
    if (jl + R <= pr.ld) {
#pragma unroll
      for (int c = 0; c < R; ++c) dst[c] = col(v, c);
    } else {
#pragma unroll
      for (int c = 0; c < R; ++c)
        if (jl + c < pr.ld) dst[c] = col(v, c);
    }
  }
}

// *p (0 where !ok), a strong load; no branch.
__device__ __forceinline__ float ld_poll_if(const float* p, bool ok) {
  float v;
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %2, 0;\n mov.b32 %0, 0;\n @p ld.relaxed.gpu.global.f32 %0, [%1];\n}"
               : "=&f"(v) : "l"(p), "r"((int)ok));
  return v;
}

// Edge records, one per row of a band: the last lane's outputs of the row.
// Affine: one float4 (od, oc, normalised frame, 0); linear: one float2 (oc,
// normalised frame).  A band's records start at the next
// 16-byte boundary of its edge slice (2 NS floats per row hold them with the
// padding; slices start at even offsets).
template <int NS> struct LEdge {
  __device__ static __forceinline__ float* base(float* edge, size_t off) {
    return edge + (NS == 3 ? (off + 3) / 4 * 4 : off);
  }
  __device__ static __forceinline__ void put(float* b, int i, float od, float oc, int n) {
    if constexpr (NS == 3) reinterpret_cast<float4*>(b)[i - 1] = make_float4(od, oc, __int_as_float(n), 0.f);
    else reinterpret_cast<float2*>(b)[i - 1] = make_float2(oc, __int_as_float(n));
  }
  // record i (0 where !ok), a strong load; no branch
  __device__ static __forceinline__ float4 get(const float* b, int i, bool ok) {
    float4 v;
    if constexpr (NS == 3) {
      asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %5, 0;\n mov.b32 %0, 0;\n mov.b32 %1, 0;\n mov.b32 %2, 0;\n"
                   " mov.b32 %3, 0;\n @p ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];\n}"
                   : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w) : "l"(b + 4 * (size_t)(i - 1)), "r"((int)ok));
    } else {
      v.z = 0.f; v.w = 0.f;
      asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %3, 0;\n mov.b32 %0, 0;\n mov.b32 %1, 0;\n"
                   " @p ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];\n}"
                   : "=&f"(v.x), "=&f"(v.y) : "l"(b + 2 * (size_t)(i - 1)), "r"((int)ok));
    }
    return v;
  }
  __device__ static __forceinline__ bool missing(const float4& v) {
    if constexpr (NS == 3)
      return is_sentinel(v.x) || is_sentinel(v.y) || is_sentinel(v.z);
    else
      return is_sentinel(v.x) || is_sentinel(v.y);
  }
  // (od, oc, n) of a resolved record
  __device__ static __forceinline__ float4 open(const float4& v) {
    if constexpr (NS == 3) return v;
    return make_float4(0.f, v.x, v.y, 0.f);
  }
  // Bounded wait for record i; on expiry the status word and the pair's flag
  // are set and the record reads as 0.
  __device__ static __noinline__ float4 wait(const float* b, int i, uint64_t deadline, unsigned* status,
                                             unsigned* flag) {
    for (int tries = 0;; ++tries) {
      const float4 v = get(b, i, true);
      if (!missing(v)) return v;
      if (gtimer() > deadline) {
        mark_timeout(status, flag);
        return make_float4(0.f, 0.f, 0.f, 0.f);
      }
      if (tries > 16) __nanosleep(SWB_POLL_SLEEP);
    }
  }
};

// Scaled scores of one step, clamped at XMAX; NEG in columns past the pair
// (E = 0 there).  Rows outside the pair hold scores 0 (load_row).
template <int R>
__device__ __forceinline__ void lscores(const float (&sb)[R], float k, int nlive, bool has_dead,
                                        float (&xs)[R]) {
#pragma unroll
  for (int c = 0; c < R; ++c) xs[c] = fminf(__fmul_rn(sb[c], k), XMAX);
  if (has_dead) {
#pragma unroll
    for (int c = 0; c < R; ++c)
      if (c >= nlive) xs[c] = NEG;
  }
}

// Parameters of a linear-domain launch: the launch's floats, or read from the
// device parameter array when there is one (a stream capture with tensor
// parameters: each replay reads their current values).  k and the transition
// factors are formed exactly as the host forms them.  ok is false for a
// temperature that is not finite and positive or a positive gap: the linear
// domain needs every transition factor <= 1.
struct LParams {
  float go, ge, T, k, xgo, xge;
  bool ok;
};
template <int NS>
__device__ __forceinline__ LParams lparams(const Args& a) {
  LParams p{a.go, a.ge, a.T, a.k, a.xgo, a.xge, true};
  if (a.dparams) {
    p.go = a.dparams[0];
    p.ge = NS == 3 ? a.dparams[1] : 0.f;
    p.T = a.dparams[NS == 3 ? 2 : 1];
    p.k = 1.4426950408889634f / p.T;
    p.xgo = (float)exp2((double)p.go * (double)p.k);
    p.xge = (float)exp2((double)p.ge * (double)p.k);
    p.ok = p.T > 0.f && p.T < INFINITY && p.go * p.k <= 0.f && p.ge * p.k <= 0.f;
  }
  return p;
}

// ---------------------------------------------------------------------------
// forward band task
// ---------------------------------------------------------------------------

// Score prefetch distance of the tangent kernels' forward (steps).
constexpr int FPF = C_STEPS;
// Score prefetch distance of the sweeps (steps): each row is requested this
// many steps ahead; the narrow kernels, whose steps are shorter, look further.
template <int R> __host__ __device__ constexpr int fwd_ahead() { return R == 8 ? 4 : 8; }
// Steps per block of the forward: the left band's records are passed a block
// at a time (about 220 cycles a time in a lone warp).
template <int R> __host__ __device__ constexpr int fwd_block() { return split_code<R>() ? 2 * C_STEPS : C_STEPS; }

// Forward wavefront of one band: per-lane partition sums (Kahan over the rows,
// in the lane's largest normalised frame), the left-to-right edge records and,
// every C steps, a checkpoint of the lane state plus the chunk's largest
// normalised frame.  The band's partition partial is (frame, mantissa sum):
// Z_band = sum * 2^frame.
//
// The left band's records of a block (WB steps) pass through shared memory,
// where lane 0 reads the one of each step.  They are requested two blocks
// ahead and put there one block ahead, two buffers in turn, so a block whose
// records had been written by then starts without waiting for anything.
//
// DM (see above): 1 also where rows are not 16-byte aligned.
template <int NS, int R, int DM>
__device__ void lfwd_band(const Args& a, const LParams& lp, const Place& w, int lane,
                          uint64_t deadline, float4* sedge) {
  using LD = LDims<NS, R>;
  using LE = LEdge<NS>;
  constexpr int H = R / 2, AH = fwd_ahead<R>(), WB = fwd_block<R>();
  check_lengths(a, w, lane);
  if (!lp.ok && w.band == 0 && lane == 0) {
    atomicOr(a.status, ERR_BAD_PARAMS);
    atomicOr(a.pair_done + w.p, PAIR_TIMEOUT);
  }
  const Pair& pr = w.pr;
  const int L1 = pr.L1, L2 = pr.L2;
  const int band = w.band;
  const size_t slot = w.slot0 + band;
  const int col0 = band * 32 * R;
  float* part = a.part + 2 * (size_t)slot;
  if (!(L1 > 0 && col0 < L2)) {
    if (lane == 0) { part[0] = 0.f; part[1] = (band == 0) ? 1.f : 0.f; }
    return;
  }
  const int jl = col0 + lane * R;
  const int nlive = min(max(L2 - jl, 0), R);
  const bool hd = col0 + 32 * R > L2;
  const float k = lp.k, gO = lp.xgo, gE = lp.xge;
  float* eout = LE::base(a.edge, w.ed0 + (size_t)band * w.edb);
  const bool fault = a.fault_inject && band > 0;
  const float* ein = (band > 0 && !fault) ? LE::base(a.edge, w.ed0 + (size_t)(band - 1) * w.edb) : nullptr;
  const bool keep_ck = a.ckpt != nullptr;
  float* ck = keep_ck ? a.ckpt + w.ck0 + (size_t)band * w.ckb : nullptr;
  const int nch = band_chunks(L1);
  const int KC = a.ck_every;
  float* ckmax = keep_ck ? ck + (size_t)((nch + KC - 1) / KC) * LD::LREC : nullptr;
  int next_ck = 0;   // the next chunk whose record is kept

  LState<NS, R> s;
  lstate_zero(s);
  float2 d[H];
#pragma unroll
  for (int j = 0; j < H; ++j) d[j] = dup2(0.f);
  // partition: the row sums in the frame ze (the largest normalised frame so
  // far), Kahan-compensated
  float zm = (band == 0 && lane == 0) ? 1.f : 0.f, zc = 0.f;   // M[0,0]: the empty alignment
  int ze = 0;
  auto zadd = [&](float v) {
    const float y = v - zc, t = zm + y;
    zc = (t - zm) - y;
    zm = t;
  };

  // lane u < WB holds the left band's edge record lane 0 needs at step u of a
  // block: `ea` of the next block, `eb` of the one after
  auto get_edge = [&](int bl) {
    const int ie = bl * WB + lane + 1;
    return LE::get(ein, ie, ein && lane < WB && ie <= L1);
  };
  float4 ea = get_edge(0), eb = get_edge(1);
  bool ready = false;   // this block's records are in shared memory
  Rows<R> rows;
  rows.init(pr, jl, col0);
  const float* src = rows.at(1 - lane);
  float sb[AH][R];   // per-lane score ring, AH steps ahead
#pragma unroll
  for (int u = 0; u < AH; ++u) {
#pragma unroll
    for (int c = 0; c < R; ++c) sb[u][c] = 0.f;
    rows.load(src, u - lane + 1, sb[u]);
    src += rows.ld;
  }

  int i = 1 - lane;   // the lane's row at the next step
#pragma unroll 1
  for (int bl = 0; bl * WB < nch * C_STEPS; ++bl) {
    float4* se = sedge + (bl & 1) * WB;
    __syncwarp();   // the buffers: the last block's reads are done, its writes are seen
    if (!ready) {
      // wait for the block's records: lane u < WB polls its own until the left
      // band has written it (one bounded wait per block, not per row); fault
      // injection waits on a word nobody writes and substitutes zeros
      const int ie = bl * WB + lane + 1;
      const bool mine = lane < WB && ie <= L1;
      if (fault) {
        if (mine)
          poll_value(a.never_written, ld_poll(a.never_written), deadline, a.status, a.pair_done + w.p, 0.f);
      } else if (ein && mine && LE::missing(ea)) {
        ea = LE::wait(ein, ie, deadline, a.status, a.pair_done + w.p);
      }
      __syncwarp();
      if (lane < WB) se[lane] = LE::open(ea);
      __syncwarp();
    }
    // the next block's records, if they are there (fault injection: never)
    ready = __all_sync(FULL, !LE::missing(eb)) && !fault;
    if (ready && lane < WB) sedge[((bl + 1) & 1) * WB + lane] = LE::open(eb);
    ea = eb;
    eb = get_edge(bl + 2);
    const bool in_block = rows.inside(bl * (WB / C_STEPS)) && rows.inside((bl + 1) * (WB / C_STEPS) - 1 + AH / C_STEPS);
#pragma unroll
    for (int h = 0; h < WB / C_STEPS; ++h) {
    const int kc = bl * (WB / C_STEPS) + h;
    if (keep_ck && kc == next_ck && kc < nch) {
      lck_store<NS, R>(ck, lane, s, col(d, 0));
      ck += LD::LREC;
      next_ck += KC;
    }
    int cmx = -(1 << 30);   // largest normalised frame of the lane's live rows in this chunk
    float rsv[C_STEPS];
    int ev[C_STEPS];
    // the chunk's steps.  Inside chunks (every lane on a row of the pair, now
    // and for the rows requested) run without a branch, so that the steps'
    // loads, emissions and chains overlap
    auto steps = [&](auto inside_c, auto vec_c) {
      constexpr bool IN = decltype(inside_c)::value, VEC = decltype(vec_c)::value;
      constexpr int DD = IN || DM == 2 ? DM : 1;
#pragma unroll
      for (int cu = 0; cu < C_STEPS; ++cu) {
        const bool act = IN || (unsigned)(i + cu - 1) < (unsigned)L1;
        const float4 e4 = se[h * C_STEPS + cu];   // 0 where there is no left band
        float xd = 0.f;
        if constexpr (NS == 3) {
          xd = __shfl_up_sync(FULL, s.od, 1);
          xd = lane == 0 ? e4.x : xd;
        }
        float xc = __shfl_up_sync(FULL, s.oc, 1);
        int xn = __shfl_up_sync(FULL, s.n, 1);
        xc = lane == 0 ? e4.y : xc;
        xn = lane == 0 ? __float_as_int(e4.z) : xn;
        float2 xs[H], E[H];
        lemit<R, DD>(sb[(h * C_STEPS + cu) % AH], k, nlive, hd, xs, E);
        if constexpr (IN) rows.template fetch<VEC>(src, sb[(h * C_STEPS + cu) % AH]);
        else rows.load(src, i + cu + AH, sb[(h * C_STEPS + cu) % AH]);
        src += rows.ld;
        rsv[cu] = 0.f;
        ev[cu] = 0;
        if (act) {
          lcells<NS, R, DD>(s, xd, xc, xn, E, gO, gE, nlive, hd, d, rsv[cu]);
          ev[cu] = s.e;
          cmx = max(cmx, s.n);
          if (lane == 31) LE::put(eout, i + cu, s.od, s.oc, s.n);
        }
      }
    };
    bool done = false;
    if constexpr (split_code<R>()) {
      if (in_block) {
        done = true;
        if (DM != 1 || rows.vec) steps(std::true_type{}, std::true_type{});
        else if constexpr (DM == 1) steps(std::true_type{}, std::false_type{});
      }
    }
    if (!done) steps(std::false_type{}, std::false_type{});
    i += C_STEPS;
    {
      const int zn = max(ze, cmx);
      const float f = p2b(ze - zn + 127);
      zm *= f;
      zc *= f;
#pragma unroll
      for (int cu = 0; cu < C_STEPS; ++cu) zadd(rsv[cu] * p2b(ev[cu] - zn + 127));
      ze = zn;
    }
    if (keep_ck) {
      cmx = __reduce_max_sync(FULL, cmx);
      if (lane == 0 && kc < nch) ckmax[kc] = __int_as_float(cmx);
    }
    }
  }
  // warp-combine (frame, sum) pairs, fixed shuffle tree
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int z2 = __shfl_xor_sync(FULL, ze, o);
    const float m2 = __shfl_xor_sync(FULL, zm, o);
    const int m = max(ze, z2);
    zm = zm * p2i(ze - m) + m2 * p2i(z2 - m);
    ze = m;
  }
  if (lane == 0) { part[0] = (float)ze; part[1] = zm; }
}

#ifndef SWB_LFWD_MINB
#define SWB_LFWD_MINB 4
#endif
template <int NS, int R>
__global__ void __launch_bounds__(128, (R >= 8 ? 4 : SWB_LFWD_MINB)) lfwd_kernel(Args a) {
  __shared__ float4 s_edge[4][2 * fwd_block<R>()];   // per warp: the left band's records of two blocks
  const int lane = threadIdx.x & 31;
  const LParams lp = lparams<NS>(a);
  const uint64_t deadline = gtimer() + a.spin_limit_ns;
  const int ntasks = (a.layout == 0) ? a.B * a.nb : a.ntasks;
  while (true) {
    int task = 0;
    if (lane == 0) task = (int)atomicAdd(a.counters + 0, 1u);
    task = __shfl_sync(FULL, task, 0);
    if (task >= ntasks) break;
    const Place w = place_of<NS, R>(a, task, false);
    // a band whose last columns lie past the pair takes the variant that masks them
    float4* se = s_edge[threadIdx.x >> 5];
    if constexpr (!split_code<R>()) lfwd_band<NS, R, 2>(a, lp, w, lane, deadline, se);
    else if ((w.band + 1) * 32 * R > w.pr.L2 || !w.pr.vec) lfwd_band<NS, R, 1>(a, lp, w, lane, deadline, se);
    else lfwd_band<NS, R, 0>(a, lp, w, lane, deadline, se);
  }
}

// ---------------------------------------------------------------------------
// partition of a pair
// ---------------------------------------------------------------------------

// Z of pair w as (integer frame ze, mantissa zm): Z = zm * 2^ze, combined
// from the band partials in a fixed order (deterministic).
__device__ __forceinline__ void lpair_z(const Args& a, const Place& w, int lane, int& ze, float& zm) {
  int ref = 0;
  float s = 0.f;
  for (int b = lane; b < w.nb; b += 32) {
    const float* q = a.part + 2 * (w.slot0 + b);
    const int r2 = (int)q[0];
    const float s2 = q[1];
    if (s2 > 0.f) {
      const int m = max(ref, r2);
      s = s * p2i(ref - m) + s2 * p2i(r2 - m);
      ref = m;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const int r2 = __shfl_xor_sync(FULL, ref, o);
    const float s2 = __shfl_xor_sync(FULL, s, o);
    const int m = max(ref, r2);
    s = s * p2i(ref - m) + s2 * p2i(r2 - m);
    ref = m;
  }
  ze = ref;
  zm = s;
}

// S' = log2 Z as a double-float (Sh, Sl): the integer part joins the frame
// exactly and lg2 sees only the mantissa.
__device__ __forceinline__ void lz_log2(int ze, float zm, float& Sh, float& Sl) {
  const unsigned bits = __float_as_uint(zm);
  const int e = (int)((bits >> 23) & 0xffu) - 127;
  if (zm > 0.f && e > -127 && e < 128) {
    float h, l;
    two_sum((float)ze, (float)e, h, l);
    Sh = h;
    Sl = l + lg2(__uint_as_float((bits & 0x7fffffu) | 0x3f800000u));
  } else {
    Sh = (float)ze;
    Sl = lg2(zm);
  }
}

// Value-only calls: one warp per pair folds the band partials into S.
template <int NS, int R>
__global__ void __launch_bounds__(128) lvalue_kernel(Args a) {
  const int lane = threadIdx.x & 31;
  const int q = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (q >= a.B) return;
  Place w;
  if (a.layout == 0) {
    w = place_of<NS, R>(a, q * a.nb, false);
  } else {
    const long long* pw = a.plan_pairs + (size_t)q * PLAN_PAIR_WORDS;
    w.p = q;
    w.nb = (int)pw[PW_NB];
    w.slot0 = (size_t)pw[PW_SLOT0];
  }
  if (a.pair_done[w.p] & PAIR_TIMEOUT) {   // a bounded wait of this pair expired
    if (lane == 0) a.value[w.p] = __int_as_float(0x7fc00000);
    return;
  }
  int ze;
  float zm, Sh, Sl;
  lpair_z(a, w, lane, ze, zm);
  lz_log2(ze, zm, Sh, Sl);
  if (lane == 0) a.value[w.p] = (Sh + Sl) * (1.f / lparams<NS>(a).k);
}

// ---------------------------------------------------------------------------
// adjoint band task
// ---------------------------------------------------------------------------

// Shared memory per adjoint warp (floats): one chunk of recomputed fields,
// the staged checkpoint of the next chunk, then the chunk's cross-band
// records as float4 per step: the left band's edge records (lane 0,
// recompute) and the right band's push records (lane 31, outside recursion).
// The next chunk's score rows wait in registers.
template <int NS, int R>
__host__ __device__ constexpr int lbwd_smem_floats() {
  return (C_STEPS * LDims<NS, R>::FW + LDims<NS, R>::CKF) * 32 + 2 * C_STEPS * 4;
}

// Lane state of the outside recursion: the row below and the right
// neighbour's held value.
template <int R> struct BState {
  static constexpr int H = R / 2;
  float2 b[H];      // beta_I (linear: beta) of the lane's latest row, raw (frame fb)
  float2 t[H];      // t = E beta_M of that row (normalised frame nb)
  float ht, ob;     // the right neighbour's held t (frame hn); beta_D (beta) of column 0 (frame nb)
  int fb, nb, hn;
};
template <int R> __device__ __forceinline__ void bstate_zero(BState<R>& s) {
#pragma unroll
  for (int k = 0; k < R / 2; ++k) { s.b[k] = dup2(0.f); s.t[k] = dup2(0.f); }
  s.ht = 0.f; s.ob = 0.f;
  s.fb = 0; s.nb = 0; s.hn = 0;
}

// The state as a record ([group][lane][4] floats).
template <int R> struct BDims {
  static constexpr int BKF = (2 * R + 5 + 3) / 4 * 4;
  static constexpr int BREC = BKF * 32;
};
template <int R>
__device__ __forceinline__ void bstate_store(float* rec, int lane, const BState<R>& s) {
  constexpr int H = R / 2, K = BDims<R>::BKF;
  float x[K];
#pragma unroll
  for (int k = 0; k < H; ++k) {
    x[2 * k] = s.b[k].x; x[2 * k + 1] = s.b[k].y;
    x[R + 2 * k] = s.t[k].x; x[R + 2 * k + 1] = s.t[k].y;
  }
  x[2 * R] = s.ht;
  x[2 * R + 1] = s.ob;
  x[2 * R + 2] = __int_as_float(s.fb);
  x[2 * R + 3] = __int_as_float(s.nb);
  x[2 * R + 4] = __int_as_float(s.hn);
#pragma unroll
  for (int f = 2 * R + 5; f < K; ++f) x[f] = 0.f;
#pragma unroll
  for (int g = 0; g < K / 4; ++g)
    reinterpret_cast<float4*>(rec + g * 128)[lane] = make_float4(x[4 * g], x[4 * g + 1], x[4 * g + 2], x[4 * g + 3]);
}
template <int R>
__device__ __forceinline__ void bstate_load(const float* rec, int lane, BState<R>& s) {
  constexpr int H = R / 2, K = BDims<R>::BKF;
  float x[K];
#pragma unroll
  for (int g = 0; g < K / 4; ++g) {
    const float4 y = reinterpret_cast<const float4*>(rec + g * 128)[lane];
    x[4 * g] = y.x; x[4 * g + 1] = y.y; x[4 * g + 2] = y.z; x[4 * g + 3] = y.w;
  }
#pragma unroll
  for (int k = 0; k < H; ++k) {
    s.b[k] = make_float2(x[2 * k], x[2 * k + 1]);
    s.t[k] = make_float2(x[R + 2 * k], x[R + 2 * k + 1]);
  }
  s.ht = x[2 * R];
  s.ob = x[2 * R + 1];
  s.fb = __float_as_int(x[2 * R + 2]);
  s.nb = __float_as_int(x[2 * R + 3]);
  s.hn = __float_as_int(x[2 * R + 4]);
}

// The gradient sums of a band are formed per segment of kSeg chunks (per lane
// plain within a chunk and compensated over the chunks, then a shuffle tree)
// and folded over the segments, last one first, with compensation: the adjoint
// of a whole band and the segment kernel give the same bits.
constexpr int kSeg = 4;
struct BandSum {
  KSum a, b, m;
  __device__ __forceinline__ void add(float x, float y, float z) {
    if (x != 0.f || y != 0.f || z != 0.f) { a.add(x); b.add(y); m.add(z); }
  }
};

// End of a segment: its gradient partials; the pair's last segment folds them
// (lane l the bands l, l + 32, ...; then the bands in order).
template <int NS>
__device__ __forceinline__ void lfinish_seg(const Args& a, const Place& w, int lane, int seg, float Sh, float Sl,
                                            float g0, float g1, float ps, PParams pp) {
  const int p = w.p;
  unsigned done = 0;
  if (lane == 0) {
    reinterpret_cast<float4*>(a.spart)[(w.slot0 + w.band) * a.nseg + seg] = make_float4(g0, g1, ps, 0.f);
    __threadfence();
    done = atomicAdd(a.pair_done + p, 1u);
  }
  done = __shfl_sync(FULL, done, 0);
  if ((done & ~PAIR_TIMEOUT) != (unsigned)(w.nb * a.nseg) - 1) return;
  __threadfence();
  double o = 0., e = 0., m = 0.;
  for (int b0 = 0; b0 < w.nb; b0 += 32) {
    BandSum s;
    if (b0 + lane < w.nb) {
      const float* x = a.spart + 4 * (w.slot0 + b0 + lane) * a.nseg;
      for (int q = a.nseg - 1; q >= 0; --q) s.add(ld_poll(x + 4 * q), ld_poll(x + 4 * q + 1), ld_poll(x + 4 * q + 2));
    }
    for (int b = 0; b < min(32, w.nb - b0); ++b) {
      o += __shfl_sync(FULL, s.a.s, b);
      e += __shfl_sync(FULL, s.b.s, b);
      m += __shfl_sync(FULL, s.m.s, b);
    }
  }
  if (lane != 0) return;
  if (done & PAIR_TIMEOUT) {   // a bounded wait of this pair expired
    const float nan = __int_as_float(0x7fc00000);
    a.value[p] = nan; a.g_open[p] = nan; a.g_T[p] = nan;
    if (a.g_ext) a.g_ext[p] = nan;
    return;
  }
  a.value[p] = (Sh + Sl) * (1.f / pp.k);   // 1 / k = T ln 2
  a.g_open[p] = (float)o;
  if (a.g_ext) a.g_ext[p] = NS == 3 ? (float)e : 0.f;
  a.g_T[p] = dS_dT(Sh, Sl, m, o, scaled<true>(pp.go, pp.k), NS == 3 ? e : 0., scaled<true>(pp.ge, pp.k));
}

// One row of the outside recursion for one lane: (rb, rt, rn) are the right
// lane's beta_D (linear: beta) of its column 0, its t and its normalised
// frame; live: the row is inside the pair.  Returns, in the frame `ft`: vm =
// beta_M (beta), sr = beta_I below + beta_D right and br = beta_D right per
// column.  The state moves on with bfinish.
template <int NS, int R, int DM>
__device__ __forceinline__ void bcells(const BState<R>& s, float rb, int rn, bool live, float gO, float gE,
                                       float gX, int nlive, bool hd, int& ft, float& fB,
                                       float2 (&vm)[R / 2], float2 (&vi)[R / 2], float2 (&sr)[R / 2],
                                       float2 (&br)[R / 2], float& vd0, float& mx) {
  constexpr int H = R / 2;
  // frames: the row is computed in ft >= every input's normalised frame
  ft = max(max(s.nb, rn), s.hn);
  const int q = 127 - ft;
  fB = p2b(s.fb + q);
  const float fT = p2b(s.nb + q), fR = p2b(rn + q), fH = p2b(s.hn + q);
  const float one = live ? p2b(q) : 0.f;
  float2 base[H];
#pragma unroll
  for (int k = 0; k < H; ++k) {   // 1 plus the diagonal successor's t
    float2 oc = dup2(one);
    if (masks<DM>(hd)) oc = make_float2(k < nlive ? one : 0.f, k + H < nlive ? one : 0.f);
    base[k] = k == H - 1 ? fma2(make_float2(fT, fH), make_float2(s.t[0].y, s.ht), oc)
                         : fma2(dup2(fT), s.t[k < H - 1 ? k + 1 : 0], oc);
  }
  const float b0 = fR * rb;   // right successor's beta_D (beta) of the last column
  float2 v[H];                // beta_D (beta) per column
  if constexpr (NS == 3) {
    col(v, R - 1) = fmaf(gE, b0, col(base, R - 1));
#pragma unroll
    for (int c = R - 2; c >= 0; --c) col(v, c) = fmaf(gE, col(v, c + 1), col(base, c));
  } else {
    float2 x[H];
    const float2 gOb = dup2(gO * fB);
#pragma unroll
    for (int k = 0; k < H; ++k) x[k] = fma2(gOb, s.b[k], base[k]);
    col(v, R - 1) = fmaf(gO, b0, col(x, R - 1));
#pragma unroll
    for (int c = R - 2; c >= 0; --c) col(v, c) = fmaf(gO, col(v, c + 1), col(x, c));
  }
  vd0 = v[0].x;
#pragma unroll
  for (int k = 0; k < H; ++k) {
    br[k] = k == H - 1 ? make_float2(v[0].y, b0) : v[k < H - 1 ? k + 1 : 0];
    sr[k] = fma2(dup2(fB), s.b[k], br[k]);
  }
  float2 m[H];
  if constexpr (NS == 3) {
    const float2 gEb = dup2(gE * fB);
#pragma unroll
    for (int k = 0; k < H; ++k) {
      vm[k] = fma2(dup2(gO), sr[k], base[k]);
      vi[k] = fma2(gEb, s.b[k], base[k]);
      m[k] = fma2(dup2(gX), sr[k], base[k]);   // >= beta_M, beta_I, beta_D
    }
  } else {
#pragma unroll
    for (int k = 0; k < H; ++k) { vm[k] = v[k]; vi[k] = v[k]; m[k] = v[k]; }
  }
  float x[R];
#pragma unroll
  for (int c = 0; c < R; ++c) x[c] = col(m, c);
#pragma unroll
  for (int h = 1; h < R; h *= 2)
#pragma unroll
    for (int c = 0; c + h < R; c += 2 * h) x[c] = fmaxf(x[c], x[c + h]);
  mx = x[0];
}

// The state after the row: t = E beta_M in the row's normalised frame, 0 in a
// row outside the pair (!live), whose E is of whatever score a load left there:
// t takes part in the quiet-chunk test of its warp, and the kernels' leftovers
// differ (and, after a quiet run that a record not written yet ended, depend on
// timing).
template <int R>
__device__ __forceinline__ void bfinish(BState<R>& s, int ft, float mx, bool live, const float2 (&vm)[R / 2],
                                        const float2 (&vi)[R / 2], float vd0, const float2 (&E)[R / 2],
                                        float rt, int rn) {
  constexpr int H = R / 2;
  const int nn = max(ft - 126 + sexp(mx), 0);
  const float bs = p2b(ft - nn + 127), ts = live ? bs : 0.f;
#pragma unroll
  for (int k = 0; k < H; ++k) {
    s.t[k] = mul2(mul2(vm[k], dup2(ts)), E[k]);
    s.b[k] = vi[k];
  }
  s.fb = ft;
  s.nb = nn;
  s.ob = vd0 * bs;
  s.ht = rt;
  s.hn = rn;
}

// ---- quiet chunks.  For a cell u of a chunk, alpha_u beta_u / Z sums, over
// the chunk cells x where u's continuations stay inside, terms
// alpha_x (1 + w beta_out) / Z (alpha_u W(u -> x) <= alpha_x: all weights are
// positive), where beta_out are the successors outside the chunk: the row
// below, the right neighbour's held t and, for lane 31, the right band's
// records.  With at most 2^9 cells, alpha_x <= 2^ckm and
// 1 + w beta_out <= 4 max(1, inflow), every posterior in the chunk and every
// flow across its top and left edges is below 2^-SWB_LQUIET when
// ckm + 11 + max(log2 inflow, 0) < log2 Z - SWB_LQUIET.  Such a chunk has zero
// map rows and zero records to the left band, and passes zero beta up: the
// flows it drops are among those bounded.  The right band's records are
// resolved first, so the decision does not depend on timing.  zlog: log2 of Z
// less SWB_LQUIET; pb: lane u < C the record of backward step u. ----
template <int R>
__device__ __forceinline__ bool lquiet(const BState<R>& s, int ckm, const float (&pb)[3], int lane, int zlog) {
  int inl = s.hn + fexp(s.ht);
  float mb = 0.f, mt = 0.f;   // largest beta and t of the row below
#pragma unroll
  for (int j = 0; j < R / 2; ++j) {
    mb = fmaxf(mb, fmaxf(s.b[j].x, s.b[j].y));
    mt = fmaxf(mt, fmaxf(s.t[j].x, s.t[j].y));
  }
  inl = max(inl, max(s.fb + fexp(mb), s.nb + fexp(mt)));
  if (lane < C_STEPS) inl = max(inl, __float_as_int(pb[2]) + fexp(fmaxf(pb[0], pb[1])));
  return __all_sync(FULL, ckm + 11 + max(inl, 0) < zlog);
}
// ---- quiet run.  After a quiet chunk only lane 31's held t (pt, pn) and the
// right band's records enter the chunks above, so one round of loads decides
// the next 32 / C chunks: lane l takes chunk kn - l / C at backward step
// l % C (lane 31's row there), checking that record and the one of the row
// below (lane l - 1's; lane 0: the held t).  A record not written yet ends
// the run; that chunk is then decided by lquiet from the same values, so
// results do not depend on timing.  Returns how many chunks from kn down (not
// below k_lo) are quiet; r1, rn: the lane's record's t and frame. ----
__device__ __forceinline__ int lquiet_run(const float* pin, size_t Lm, int L1, const float* ckmax, int kn, int k_lo,
                                          int lane, float pt, int pn, int zlog, float& r1, int& rn) {
  constexpr int RUN = 32 / C_STEPS;
  const int j = lane / C_STEPS, u = lane - j * C_STEPS;
  const int kq = kn - j;
  float r0 = 0.f;
  int cm = -(1 << 30);
  bool written = true;
  r1 = 0.f;
  rn = 0;
  if (kq >= k_lo) {
    const int ir = kq * C_STEPS + C_STEPS - 1 - u - 30;
    if (pin && ir >= 1 && ir <= L1) {
      r0 = ld_poll(pin + 0 * (Lm + 1) + ir);
      r1 = ld_poll(pin + 1 * (Lm + 1) + ir);
      const float r2 = ld_poll(pin + 2 * (Lm + 1) + ir);
      written = !is_sentinel(r0) && !is_sentinel(r1) && !is_sentinel(r2);
      rn = __float_as_int(r2);
    }
    cm = __float_as_int(ckmax[kq]);
  }
  const int lg = written ? rn + fexp(fmaxf(r0, r1)) : 0;
  const int lgu = __shfl_up_sync(FULL, lg, 1);
  const bool wu = __shfl_up_sync(FULL, (int)written, 1) != 0;
  const int lgb = lane == 0 ? pn + fexp(pt) : lgu;
  const bool wb = lane == 0 || wu;
  const bool q = kq >= k_lo && written && wb && cm + 11 + max(max(lg, lgb), 0) < zlog;
  const unsigned ball = __ballot_sync(FULL, q);
  constexpr unsigned grp = (1u << C_STEPS) - 1u;
  int n = 0;
  while (n < RUN && kn - n >= k_lo && ((ball >> (n * C_STEPS)) & grp) == grp) ++n;
  return n;
}
// Zero records to the left band for the rows of chunk kq (lane 0's).
__device__ __forceinline__ void zero_push(float* pout, size_t Lm, int L1, int kq, int lane) {
  const int i = kq * C_STEPS + lane + 1;
  if (pout && lane < C_STEPS && i <= L1) {
    pout[0 * (Lm + 1) + i] = 0.f;
    pout[1 * (Lm + 1) + i] = 0.f;
    pout[2 * (Lm + 1) + i] = 0.f;
  }
}

// Per band, checkpoint chunks in reverse.  Each chunk restores its checkpoint
// and recomputes C steps of the forward, keeping every cell's raw values and
// scaled score (and each step's frame) in shared memory; then the outside
// recursion runs the same C steps backwards.  Lane l + 1 is one step ahead of
// lane l (it processes row i one step earlier); a lane receives from its right
// neighbour that row's beta_D (beta, linear) of column 0 in the neighbour's
// normalised frame, its t = E beta_M of column 0 and the frame, and holds
// the t for one more step (it is the diagonal successor of the next row).
// Lane 0 passes the same three values to the left band through the push
// buffer; lane 31 reads the right band's.  No atomics; the map is written row
// by row (a quiet chunk writes its zero rows in whole row pieces); the
// gradient sums are folded per pair in band order.
//
// SEG: one segment of the band, chunks [k_lo, k_hi), starting from the state
// the outside sweep (lbeta_band) kept for it; every record it reads has been
// written by then, and it passes none on.
template <int NS, int R, bool SPARSE, int DM, bool SEG = false>
__device__ void lbwd_band(const Args& a, const LParams& lp, const Place& w, int lane, float* sm,
                          uint64_t deadline, int seg = 0) {
  using LD = LDims<NS, R>;
  using LE = LEdge<NS>;
  constexpr int H = R / 2;
  constexpr int CKF = LD::CKF, LREC = LD::LREC, FW = LD::FW, NPF = 3;
  const Pair& pr = w.pr;
  const int L1 = pr.L1, L2 = pr.L2;
  const int band = w.band;
  const int col0 = band * 32 * R;
  int ze;
  float zm, Sh, Sl;
  lpair_z(a, w, lane, ze, zm);
  lz_log2(ze, zm, Sh, Sl);
  const PParams pp{lp.go, lp.ge, lp.T, lp.k};
  const int nch = band_chunks(L1);
  const int k_lo = SEG ? seg * kSeg : 0, k_hi = SEG ? min(k_lo + kSeg, nch) : nch;
  if (!(L1 > 0 && col0 < L2) || k_lo >= k_hi) {
    if constexpr (SEG) lfinish_seg<NS>(a, w, lane, seg, Sh, Sl, 0.f, 0.f, 0.f, pp);
    else finish_pair_p<NS, 0, true>(a, w, lane, Sh, Sl, 0.f, 0.f, 0.f, pp);
    return;
  }
  const float invZ = 1.f / zm;
  const int jl = col0 + lane * R;
  const int nlive = min(max(L2 - jl, 0), R);
  const bool hd = col0 + 32 * R > L2;
  const float k = lp.k, gO = lp.xgo, gE = lp.xge, gX = fmaxf(gO, gE);
  const size_t Lm = (size_t)w.Lm;
  const float* ein = (band > 0) ? LE::base(a.edge, w.ed0 + (size_t)(band - 1) * w.edb) : nullptr;
  float* pout = (!SEG && band > 0) ? a.bpush + w.bp0 + (size_t)band * w.bpb : nullptr;
  const bool right_live = (col0 + 32 * R) < L2 && (band + 1) < w.nb;
  const float* pin = right_live ? a.bpush + w.bp0 + (size_t)(band + 1) * w.bpb : nullptr;
  const float* ck = a.ckpt + w.ck0 + (size_t)band * w.ckb;
  const int KC = SPARSE ? a.ck_every : 1;   // checkpoint records every KC chunks
  const float* ckmax = ck + (size_t)((nch + KC - 1) / KC) * LREC;

  // ---- chunk-ahead prefetch state: the next chunk's checkpoint is staged in
  // shared memory (cp.async), its score rows and records wait in registers ----
  float* stg_ck = sm + C_STEPS * FW * 32;   // [CK4][lane][4]
  float4* s_eb = reinterpret_cast<float4*>(stg_ck + CKF * 32);   // [C] edge records
  float4* s_pb = s_eb + C_STEPS;                                 // [C] push records
  Rows<R> rows;
  rows.init(pr, jl, col0);
  float nsb[C_STEPS][R];   // the next chunk's score rows, requested a chunk ahead
#pragma unroll
  for (int u = 0; u < C_STEPS; ++u)
#pragma unroll
    for (int c = 0; c < R; ++c) nsb[u][c] = 0.f;
  int ckm;                 // the next chunk's largest normalised alpha frame
  float4 ebr;              // lane u < C: left-band edge record of lane 0's row at recompute step u
  float pbc[NPF], pbn[NPF];// lane u < C: right-band record lane 31 needs at backward step u
  auto load_ck = [&](int kc) {   // the record at or before chunk kc, and kc's alpha frame
    const float* rec = ck + (size_t)(SPARSE ? kc / KC : kc) * LREC;
#pragma unroll
    for (int g = 0; g < LD::CK4; ++g) lcp16(stg_ck + g * 128 + lane * 4, rec + g * 128 + lane * 4, 16);
    lcp_commit();
    ckm = __float_as_int(ckmax[kc]);
  };
  auto get_edge = [&](int kc) {
    const int i = kc * C_STEPS + lane + 1;
    return LE::get(ein, i, ein && lane < C_STEPS && i <= L1);
  };
  auto load_pb = [&](int kc, float (&dst)[NPF]) {
    const int i = kc * C_STEPS + C_STEPS - 1 - lane - 30;   // lane 31's row at backward step lane
    const bool ok = pin && lane < C_STEPS && i >= 1 && i <= L1;
#pragma unroll
    for (int f = 0; f < NPF; ++f) dst[f] = ok ? ld_poll(pin + f * (Lm + 1) + i) : 0.f;
  };
  auto load_sb = [&](int kc) {
    const int i0 = kc * C_STEPS - lane + 1;
    const float* src = rows.at(i0);
    if (rows.vec && rows.inside(kc)) {
#pragma unroll
      for (int u = 0; u < C_STEPS; ++u) {
        rows.template fetch<true>(src, nsb[u]);
        src += rows.ld;
      }
    } else if (split_code<R>() && rows.inside(kc)) {
#pragma unroll
      for (int u = 0; u < C_STEPS; ++u) {
        rows.template fetch<false>(src, nsb[u]);
        src += rows.ld;
      }
    } else {
#pragma unroll
      for (int u = 0; u < C_STEPS; ++u) {
        rows.load(src, i0 + u, nsb[u]);
        src += rows.ld;
      }
    }
  };
  load_ck(k_hi - 1);
  ebr = get_edge(k_hi - 1);
  load_sb(k_hi - 1);
  load_pb(k_hi - 1, pbc);
#pragma unroll
  for (int f = 0; f < NPF; ++f) pbn[f] = 0.f;

  BState<R> bs;
  if constexpr (SEG) bstate_load<R>(a.bck + ((w.slot0 + band) * a.nseg + seg) * BDims<R>::BREC, lane, bs);
  else bstate_zero(bs);
  BandSum gsum;
  KSum gA, gB, gS;            // the lane's sums over the segment's chunks
  auto flush = [&]() {        // at the end of a segment
    float v0 = gA.s, v1 = gB.s, v2 = gS.s;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v0 += __shfl_xor_sync(FULL, v0, o);
      v1 += __shfl_xor_sync(FULL, v1, o);
      v2 += __shfl_xor_sync(FULL, v2, o);
    }
    gsum.add(v0, v1, v2);
    gA = KSum(); gB = KSum(); gS = KSum();
  };

  // log2 of Z is at least zlog; a chunk is quiet (below) when every cell's
  // posterior and every flow out of it is below 2^-SWB_LQUIET
  const int zlog = ze + fexp(zm) - 1 - SWB_LQUIET;
#pragma unroll 1
  for (int kc = k_hi - 1; kc >= k_lo; --kc) {
    const int t0 = kc * C_STEPS;
    lcp_wait_all();   // this chunk's staged checkpoint
    __syncwarp();
    if constexpr (!SEG) {   // the right band's records of this chunk
      const bool miss = is_sentinel(pbc[0]) || is_sentinel(pbc[1]) || is_sentinel(pbc[2]);
      if (__any_sync(FULL, miss) && miss) {
        const int ir = kc * C_STEPS + C_STEPS - 1 - lane - 30;   // as in load_pb
        FieldVec<NPF> x;
#pragma unroll
        for (int f = 0; f < NPF; ++f) x.v[f] = pbc[f];
        x = poll_fields_v<NPF, 0>(x, pin + ir, Lm + 1, deadline, a.status, a.pair_done + w.p);
#pragma unroll
        for (int f = 0; f < NPF; ++f) pbc[f] = x.v[f];
      }
      __syncwarp();
    }
    const bool quiet = lquiet<R>(bs, ckm, pbc, lane, zlog);
#ifdef SWB_COUNT_QUIET   // measurement builds: quiet and computed chunks in header words 8, 9
    if (lane == 0) atomicAdd(a.counters + (quiet ? 8 : 9), 1u);
#endif
    if (quiet) {
      auto zero_chunk = [&](int kq) {   // zero map rows and records
        if constexpr (R % 4 == 0) zero_chunk_rows<R>(pr, kq, col0, lane);
        else {
          for (int cu = 0; cu < C_STEPS; ++cu) {
            const int i = kq * C_STEPS + cu - lane + 1;
            float z[R];
#pragma unroll
            for (int c = 0; c < R; ++c) z[c] = 0.f;
            if (i >= 1 && i <= L1) store_row<R>(pr, i, jl, z);
          }
        }
        zero_push(pout, Lm, L1, kq, lane);
      };
      zero_chunk(kc);
      // the row above the chunk sees zero beta; lane 31 keeps the right
      // band's t of its top chunk row as the held diagonal successor
      float pt = __shfl_sync(FULL, pbc[1], C_STEPS - 1);
      int pn = __shfl_sync(FULL, __float_as_int(pbc[2]), C_STEPS - 1);
      int kn = kc - 1;
      while (kn >= k_lo) {
        float r1;
        int rn;
        const int n = lquiet_run(pin, Lm, L1, ckmax, kn, k_lo, lane, pt, pn, zlog, r1, rn);
        for (int m = 0; m < n; ++m) zero_chunk(kn - m);
        if (n > 0) {   // lane 31's held t: the record of its top row of the last zeroed chunk
          pt = __shfl_sync(FULL, r1, n * C_STEPS - 1);
          pn = __shfl_sync(FULL, rn, n * C_STEPS - 1);
        }
        kn -= n;
        if (n < 32 / C_STEPS) break;
      }
      if (!SEG && kc / kSeg != (kn + (kn < 0 ? -kSeg + 1 : 0)) / kSeg) flush();   // the run left the segment
      bstate_zero(bs);
      bs.ht = lane == 31 ? pt : 0.f;
      bs.hn = lane == 31 ? pn : 0;
      if (kn >= k_lo) {   // inputs of the next chunk to run
        load_ck(kn);
        ebr = get_edge(kn);
        load_sb(kn);
        load_pb(kn, pbc);
      }
      kc = kn + 1;   // the loop continues with chunk kn
      continue;
    }
    // ---- restore the checkpoint and recompute the chunk ----
    LState<NS, R> st;
    float2 d[H];
#pragma unroll
    for (int j = 0; j < H; ++j) d[j] = dup2(0.f);
    lck_restore<NS, R, DM>(stg_ck, lane, st, gO, gE, nlive, hd, d);
    if (lane < C_STEPS) s_eb[lane] = LE::open(ebr);
    __syncwarp();   // the staged checkpoint is read before the next chunk's copy is issued
    if constexpr (SPARSE) {
      if (kc % KC != 0) {
        // sparse checkpoints: the restored state is that of chunk kc - kc % KC;
        // run the forward over the chunks in between (the same steps as the
        // forward kernel, so the state reached is bit for bit the same)
        const int k0 = kc - kc % KC;
        float ab[PF][R];
        int i = k0 * C_STEPS - lane + 1;
        const float* src = rows.at(i);
#pragma unroll
        for (int u = 0; u < PF; ++u) {
#pragma unroll
          for (int c = 0; c < R; ++c) ab[u][c] = 0.f;
          rows.load(src, i + u, ab[u]);
          src += rows.ld;
        }
#pragma unroll 1
        for (int ka = k0; ka < kc; ++ka) {
          float4 er = LE::open(get_edge(ka));
#pragma unroll 1
          for (int u0 = 0; u0 < C_STEPS; u0 += PF)
#pragma unroll
          for (int u = 0; u < PF; ++u) {
            const int cu = u0 + u;
            const bool act = (unsigned)(i - 1) < (unsigned)L1;
            float xd = 0.f;
            if constexpr (NS == 3) xd = __shfl_up_sync(FULL, st.od, 1);
            float xc = __shfl_up_sync(FULL, st.oc, 1);
            int xn = __shfl_up_sync(FULL, st.n, 1);
            const float e0 = __shfl_sync(FULL, er.x, cu), e1 = __shfl_sync(FULL, er.y, cu);
            const float e2 = __shfl_sync(FULL, er.z, cu);
            if (lane == 0) { xd = e0; xc = e1; xn = __float_as_int(e2); }
            float2 xs[H], E[H];
            lemit<R, DM>(ab[u], k, nlive, hd, xs, E);
            rows.load(src, i + PF, ab[u]);
            src += rows.ld;
            float rs;
            if (act) lcells<NS, R, DM>(st, xd, xc, xn, E, gO, gE, nlive, hd, d, rs);
            ++i;
          }
        }
      }
    }
    auto recompute = [&](auto inside_c) {
      constexpr bool IN = decltype(inside_c)::value;
#pragma unroll
    for (int cu = 0; cu < C_STEPS; ++cu) {
      const int i = t0 + cu - lane + 1;
      const bool act = IN || (unsigned)(i - 1) < (unsigned)L1;
      float xd = 0.f;
      if constexpr (NS == 3) xd = __shfl_up_sync(FULL, st.od, 1);
      float xc = __shfl_up_sync(FULL, st.oc, 1);
      int xn = __shfl_up_sync(FULL, st.n, 1);
      if (lane == 0) {
        const float4 e4 = s_eb[cu];
        xd = e4.x; xc = e4.y; xn = __float_as_int(e4.z);
      }
      float2 xs[H], E[H];
      lemit<R, DM>(nsb[cu], k, nlive, hd, xs, E);
      float rs;
      if (act) lcells<NS, R, DM>(st, xd, xc, xn, E, gO, gE, nlive, hd, d, rs);
      float* ent = sm + (size_t)cu * FW * 32;
      // field g's R columns as pairs: [g][quad][lane][4] (2 columns: [g][lane][2])
      auto put = [&](int g, const float2 (&x)[H]) {
        if constexpr (R == 2) {
          reinterpret_cast<float2*>(ent + g * 64)[lane] = x[0];
        } else {
#pragma unroll
          for (int h = 0; h < H / 2; ++h)
            reinterpret_cast<float4*>(ent + g * R * 32 + h * 128)[lane] =
                make_float4(x[2 * h].x, x[2 * h].y, x[2 * h + 1].x, x[2 * h + 1].y);
        }
      };
      put(0, st.v[0]);
      if constexpr (NS == 3) put(1, st.v[1]);
      put(LD::NF - 2, d);
      put(LD::NF - 1, xs);
      ent[LD::NF * R * 32 + lane] = __int_as_float(st.e);
    }
    };
    const bool in = kc >= 32 / C_STEPS && (kc + 1) * C_STEPS <= L1;   // every lane on a row of the pair
    if (split_code<R>() && in) recompute(std::true_type{});
    else recompute(std::false_type{});
    if (kc > k_lo) {   // prefetch the next chunk's inputs while the outside recursion runs
      load_ck(kc - 1);
      ebr = get_edge(kc - 1);
      load_sb(kc - 1);
      load_pb(kc - 1, pbn);
    }
    if (lane < C_STEPS) s_pb[lane] = make_float4(pbc[0], pbc[1], pbc[2], 0.f);
    __syncwarp();
    float cA = 0.f, cB = 0.f;   // this chunk's plain sums
    float2 cS = dup2(0.f);
    int i = t0 + C_STEPS - lane;
    float* mrow = pr.m + (long long)(i - 1) * pr.ld + jl;
    // ---- outside recursion over the chunk, last step first ----
#pragma unroll 1
    for (int cu = 0; cu < C_STEPS; ++cu) {
      const bool act = (unsigned)(i - 1) < (unsigned)L1;
      const float* ent = sm + (size_t)(C_STEPS - 1 - cu) * FW * 32;
      // the right neighbour's latest row (row i): beta_D / beta of its column
      // 0, its t and frame; lane 31 takes the right band's record of row i
      float rb = __shfl_down_sync(FULL, bs.ob, 1);
      float rt = __shfl_down_sync(FULL, bs.t[0].x, 1);
      int rn = __shfl_down_sync(FULL, bs.nb, 1);
      if (lane == 31) {   // resolved at the chunk's start (the quiet-chunk test polls them)
        const float4 p4 = s_pb[cu];
        rb = p4.x; rt = p4.y; rn = __float_as_int(p4.z);
      }
      auto get = [&](int g, float2 (&x)[H]) {
        if constexpr (R == 2) {
          x[0] = reinterpret_cast<const float2*>(ent + g * 64)[lane];
        } else {
#pragma unroll
          for (int h = 0; h < H / 2; ++h) {
            const float4 y = reinterpret_cast<const float4*>(ent + g * R * 32 + h * 128)[lane];
            x[2 * h] = make_float2(y.x, y.y);
            x[2 * h + 1] = make_float2(y.z, y.w);
          }
        }
      };
      const int ea = __float_as_int(ent[LD::NF * R * 32 + lane]);
      float2 fm[H], fd[H], xs[H], E[H];
      get(0, fm);
      get(LD::NF - 2, fd);
      get(LD::NF - 1, xs);
#pragma unroll
      for (int j = 0; j < H; ++j) E[j] = make_float2(ex2(xs[j].x), ex2(xs[j].y));
      int ft;
      float fB, vd0, mx;
      float2 vm[H], vi[H], sr[H], br[H], P[H];
      bcells<NS, R, DM>(bs, rb, rn, act, gO, gE, gX, nlive, hd, ft, fB, vm, vi, sr, br, vd0, mx);
      // raw alpha (frame ea) times raw beta (frame ft), over Z: half of the
      // scale on each.  Both may stand up to 2^115 above their frames, where
      // the whole scale would be 0 and their product infinite.
      const int sh = ea + ft - ze, sha = sh >> 1;
      const float fA = p2any(sha), fZ = p2any(sh - sha) * invZ;
      float2 so = dup2(0.f);
#pragma unroll
      for (int j = 0; j < H; ++j) {
        fm[j] = mul2(fm[j], dup2(fA));
        fd[j] = mul2(fd[j], dup2(fA));
        const float2 p = mul2(NS == 3 ? fm[j] : fd[j], mul2(vm[j], dup2(fZ)));
        P[j] = make_float2(fminf(p.x, 1.f), fminf(p.y, 1.f));   // a posterior: rounding may pass 1
        so = fma2(fm[j], sr[j], so);
        cS = fma2(P[j], xs[j], cS);
      }
      cA = fmaf((so.x + so.y) * fZ, gO, cA);
      if constexpr (NS == 3) {
        float2 fi[H];
        get(1, fi);
        float2 sxi = dup2(0.f), sxd = dup2(0.f);
#pragma unroll
        for (int j = 0; j < H; ++j) {
          sxi = fma2(fi[j], bs.b[j], sxi);
          sxd = fma2(fd[j], br[j], sxd);
        }
        cB = fmaf(fmaf((sxi.x + sxi.y) * fA, fB, sxd.x + sxd.y) * fZ, gE, cB);
      }
      bfinish<R>(bs, ft, mx, act, vm, vi, vd0, E, rt, rn);
      if (act) {
        store_pairs<R>(mrow, jl, pr, P);
        if (lane == 0 && pout) {
          pout[0 * (Lm + 1) + i] = bs.ob;
          pout[1 * (Lm + 1) + i] = bs.t[0].x;
          pout[2 * (Lm + 1) + i] = __int_as_float(bs.nb);
        }
      }
      --i;
      mrow -= pr.ld;
    }
#pragma unroll
    for (int f = 0; f < NPF; ++f) pbc[f] = pbn[f];
    gA.add(cA);
    if constexpr (NS == 3) gB.add(cB);
    gS.add(cS.x + cS.y);
    if (!SEG && kc % kSeg == 0) flush();
    __syncwarp();
  }
  if constexpr (SEG) {
    flush();
    lfinish_seg<NS>(a, w, lane, seg, Sh, Sl, gsum.a.s, gsum.b.s, gsum.m.s, pp);
  } else {
    finish_pair_p<NS, 0, true>(a, w, lane, Sh, Sl, gsum.a.s, gsum.b.s, gsum.m.s, pp);
  }
}

// ---------------------------------------------------------------------------
// the outside sweep and the segments
// ---------------------------------------------------------------------------
// In a batch too small to fill the GPU the adjoint's time is its longest
// chain: per band, chunk after chunk, a restore, a recompute and an outside
// pass.  There the outside recursion, which needs nothing of alpha but the
// quiet-chunk test, runs as a sweep of its own (lbeta_kernel) that skips the
// quiet chunks and keeps its state at the top of every kSeg-th chunk; then
// every (band, segment) recomputes its chunks and writes its map rows
// independently of the others (lseg_kernel).  The decisions, the states and
// the sums are the adjoint's, so the results are its results bit for bit.

template <int NS, int R, int DM>
__device__ void lbeta_band(const Args& a, const LParams& lp, const Place& w, int lane, uint64_t deadline,
                           float4* spush) {
  using LD = LDims<NS, R>;
  constexpr int H = R / 2, AH = fwd_ahead<R>(), SUB = AH / C_STEPS, NPF = 3;
  const Pair& pr = w.pr;
  const int L1 = pr.L1, L2 = pr.L2;
  const int band = w.band;
  const int col0 = band * 32 * R;
  if (!(L1 > 0 && col0 < L2)) return;
  int ze;
  float zm;
  lpair_z(a, w, lane, ze, zm);
  const int zlog = ze + fexp(zm) - 1 - SWB_LQUIET;
  const int jl = col0 + lane * R;
  const int nlive = min(max(L2 - jl, 0), R);
  const bool hd = col0 + 32 * R > L2;
  const float k = lp.k, gO = lp.xgo, gE = lp.xge, gX = fmaxf(gO, gE);
  const size_t Lm = (size_t)w.Lm;
  float* pout = (band > 0) ? a.bpush + w.bp0 + (size_t)band * w.bpb : nullptr;
  const bool right_live = (col0 + 32 * R) < L2 && (band + 1) < w.nb;
  const float* pin = right_live ? a.bpush + w.bp0 + (size_t)(band + 1) * w.bpb : nullptr;
  const int nch = band_chunks(L1), KC = a.ck_every;
  const float* ckmax = a.ckpt + w.ck0 + (size_t)band * w.ckb + (size_t)((nch + KC - 1) / KC) * LD::LREC;
  float* rec = a.bck + (w.slot0 + band) * (size_t)a.nseg * BDims<R>::BREC;

  BState<R> bs;
  bstate_zero(bs);
  auto get_push = [&](int kc) {   // lane u < C: the right band's record lane 31 needs at backward step u
    const int i = kc * C_STEPS + C_STEPS - 1 - lane - 30;
    FieldVec<NPF> x;
    const bool ok = pin && lane < C_STEPS && i >= 1 && i <= L1;
#pragma unroll
    for (int f = 0; f < NPF; ++f) x.v[f] = ld_poll_if(pin + f * (Lm + 1) + i, ok);
    return x;
  };
  // the state at the top of a segment whose chunks above were quiet
  auto store_zero = [&](int kq, float pt, int pn) {
    BState<R> z;
    bstate_zero(z);
    z.ht = lane == 31 ? pt : 0.f;
    z.hn = lane == 31 ? pn : 0;
    bstate_store<R>(rec + (size_t)(kq / kSeg) * BDims<R>::BREC, lane, z);
  };
  Rows<R> rows;
  rows.init(pr, jl, col0);
  float sb[AH][R];
#pragma unroll
  for (int u = 0; u < AH; ++u)
#pragma unroll
    for (int c = 0; c < R; ++c) sb[u][c] = 0.f;
  int kc = nch - 1;
  FieldVec<NPF> ea, eb;
  int ckm = 0, i = 0;
  const float* src = rows.base;
  // chunk kc's inputs, at the start and after a quiet run
  auto prime = [&]() {
    i = (kc + 1) * C_STEPS - lane;   // the lane's row at the next step
    src = rows.at(i);
    ea = get_push(kc);
    eb = get_push(kc - 1);
    ckm = __float_as_int(ckmax[kc]);
#pragma unroll
    for (int u = 0; u < AH; ++u) {
      rows.load(src, i - u, sb[u]);
      src -= rows.ld;
    }
  };
  // one chunk; true after a quiet one (kc moved past the quiet run)
  auto chunk = [&](auto sub_c) -> bool {
    constexpr int S0 = decltype(sub_c)::value * C_STEPS;
    const bool miss = is_sentinel(ea.v[0]) || is_sentinel(ea.v[1]) || is_sentinel(ea.v[2]);
    if (__any_sync(FULL, miss)) {
      if (miss)
        ea = poll_fields_v<NPF, 0>(ea, pin + (kc * C_STEPS + C_STEPS - 1 - lane - 30), Lm + 1, deadline, a.status,
                                   a.pair_done + w.p);
      __syncwarp();
    }
    if (kc == nch - 1 || (kc + 1) % kSeg == 0) bstate_store<R>(rec + (size_t)(kc / kSeg) * BDims<R>::BREC, lane, bs);
    if (lquiet<R>(bs, ckm, ea.v, lane, zlog)) {
      zero_push(pout, Lm, L1, kc, lane);
      float pt = __shfl_sync(FULL, ea.v[1], C_STEPS - 1);
      int pn = __shfl_sync(FULL, __float_as_int(ea.v[2]), C_STEPS - 1);
      int kn = kc - 1;
      while (kn >= 0) {
        float r1;
        int rn;
        const int n = lquiet_run(pin, Lm, L1, ckmax, kn, 0, lane, pt, pn, zlog, r1, rn);
        for (int m = 0; m < n; ++m) {
          if ((kn - m + 1) % kSeg == 0) store_zero(kn - m, pt, pn);
          zero_push(pout, Lm, L1, kn - m, lane);
          pt = __shfl_sync(FULL, r1, m * C_STEPS + C_STEPS - 1);
          pn = __shfl_sync(FULL, rn, m * C_STEPS + C_STEPS - 1);
        }
        kn -= n;
        if (n < 32 / C_STEPS) break;
      }
      bstate_zero(bs);
      bs.ht = lane == 31 ? pt : 0.f;
      bs.hn = lane == 31 ? pn : 0;
      kc = kn;
      return true;
    }
    if (lane < C_STEPS) spush[lane] = make_float4(ea.v[0], ea.v[1], ea.v[2], 0.f);
    __syncwarp();
    ea = eb;
    eb = get_push(kc - 2);
    if (kc > 0) ckm = __float_as_int(ckmax[kc - 1]);
    auto steps = [&](auto inside_c, auto vec_c) {
      constexpr bool IN = decltype(inside_c)::value, VEC = decltype(vec_c)::value;
      constexpr int DD = IN ? DM : 1;
#pragma unroll
      for (int cu = 0; cu < C_STEPS; ++cu) {
        const bool act = IN || (unsigned)(i - cu - 1) < (unsigned)L1;
        const float4 p4 = spush[cu];
        float rb = __shfl_down_sync(FULL, bs.ob, 1);
        float rt = __shfl_down_sync(FULL, bs.t[0].x, 1);
        int rn = __shfl_down_sync(FULL, bs.nb, 1);
        rb = lane == 31 ? p4.x : rb;
        rt = lane == 31 ? p4.y : rt;
        rn = lane == 31 ? __float_as_int(p4.z) : rn;
        float2 xs[H], E[H];
        lemit<R, DD>(sb[S0 + cu], k, nlive, hd, xs, E);
        if constexpr (IN) rows.template fetch<VEC>(src, sb[S0 + cu]);
        else rows.load(src, i - cu - AH, sb[S0 + cu]);
        src -= rows.ld;
        int ft;
        float fB, vd0, mx;
        float2 vm[H], vi[H], sr[H], br[H];
        bcells<NS, R, DD>(bs, rb, rn, act, gO, gE, gX, nlive, hd, ft, fB, vm, vi, sr, br, vd0, mx);
        bfinish<R>(bs, ft, mx, act, vm, vi, vd0, E, rt, rn);
        if (act && lane == 0 && pout) {
          pout[0 * (Lm + 1) + i - cu] = bs.ob;
          pout[1 * (Lm + 1) + i - cu] = bs.t[0].x;
          pout[2 * (Lm + 1) + i - cu] = __int_as_float(bs.nb);
        }
      }
    };
    if (rows.inside(kc) && rows.inside(kc - SUB)) {
      if (DM != 1 || rows.vec) steps(std::true_type{}, std::true_type{});
      else if constexpr (DM == 1) steps(std::true_type{}, std::false_type{});
    } else {
      steps(std::false_type{}, std::false_type{});
    }
    i -= C_STEPS;
    --kc;
    __syncwarp();   // spush is free for the next chunk
    return false;
  };
  bool jumped = true;
#pragma unroll 1
  while (kc >= 0) {
    if (jumped) prime();
    jumped = chunk(std::integral_constant<int, 0>{});
    if constexpr (SUB > 1) {
      if (!jumped && kc >= 0) jumped = chunk(std::integral_constant<int, 1 % SUB>{});
    }
  }
}

template <int NS, int R>
__global__ void __launch_bounds__(128) lbeta_kernel(Args a) {
  __shared__ float4 s_push[4][C_STEPS];
  const int lane = threadIdx.x & 31;
  const LParams lp = lparams<NS>(a);
  const uint64_t deadline = gtimer() + a.spin_limit_ns;
  const int ntasks = a.B * a.nb;
  while (true) {
    int task = 0;
    if (lane == 0) task = (int)atomicAdd(a.counters + 1, 1u);
    task = __shfl_sync(FULL, task, 0);
    if (task >= ntasks) break;
    const Place w = place_of<NS, R>(a, task, true);
    if ((w.band + 1) * 32 * R > w.pr.L2 || !w.pr.vec)
      lbeta_band<NS, R, 1>(a, lp, w, lane, deadline, s_push[threadIdx.x >> 5]);
    else
      lbeta_band<NS, R, 0>(a, lp, w, lane, deadline, s_push[threadIdx.x >> 5]);
    __syncwarp();
  }
}

// The segments of every band (a.nseg per band): one warp each.
template <int NS, int R, bool SPARSE>
__global__ void __launch_bounds__(32) lseg_kernel(Args a) {
  extern __shared__ float smem[];
  const int lane = threadIdx.x;
  const LParams lp = lparams<NS>(a);
  const int ntasks = a.B * a.nb * a.nseg;
  for (int task = blockIdx.x; task < ntasks; task += gridDim.x) {
    const int slot = task / a.nseg, seg = task - slot * a.nseg;
    const Place w = place_of<NS, R>(a, slot, false);
    if constexpr (!split_code<R>()) lbwd_band<NS, R, SPARSE, 2, true>(a, lp, w, lane, smem, 0, seg);
    else if ((w.band + 1) * 32 * R > w.pr.L2) lbwd_band<NS, R, SPARSE, 1, true>(a, lp, w, lane, smem, 0, seg);
    else lbwd_band<NS, R, SPARSE, 0, true>(a, lp, w, lane, smem, 0, seg);
    lcp_wait_all();
    __syncwarp();
  }
}

// Before a separate adjoint launch on a workspace the forward filled: the
// adjoint task counter to 0 and the pairs' completion counts to 0, keeping
// the failure flags the forward set.
__global__ void adjoint_reset_kernel(unsigned* counters, unsigned* pair_done, int B) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) counters[1] = 0u;
  if (i < B) pair_done[i] &= PAIR_TIMEOUT;
}

// SPARSE: checkpoints every a.ck_every chunks (the chunks between are
// recomputed); otherwise every chunk (a.ck_every must be 1).
template <int NS, int R, int WARPS, bool SPARSE = false>
__global__ void __launch_bounds__(32 * WARPS) lbwd_kernel(Args a) {
  extern __shared__ float smem[];
  const int lane = threadIdx.x & 31;
  const int wi = threadIdx.x >> 5;
  float* sm = smem + (size_t)wi * lbwd_smem_floats<NS, R>();
  const LParams lp = lparams<NS>(a);
  const uint64_t deadline = gtimer() + a.spin_limit_ns;
  const int ntasks = (a.layout == 0) ? a.B * a.nb : a.ntasks;
  while (true) {
    int task = 0;
    if (lane == 0) task = (int)atomicAdd(a.counters + 1, 1u);
    task = __shfl_sync(FULL, task, 0);
    if (task >= ntasks) break;
    const Place w = place_of<NS, R>(a, task, true);
    if constexpr (!split_code<R>()) lbwd_band<NS, R, SPARSE, 2>(a, lp, w, lane, sm, deadline);
    else if ((w.band + 1) * 32 * R > w.pr.L2) lbwd_band<NS, R, SPARSE, 1>(a, lp, w, lane, sm, deadline);
    else lbwd_band<NS, R, SPARSE, 0>(a, lp, w, lane, sm, deadline);
  }
}

}  // namespace swb
