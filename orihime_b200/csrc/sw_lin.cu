// Soft Smith-Waterman forward / adjoint in the scaled linear domain (sm_100a),
// local alignment with linear or affine gaps.  Compiled as part of sw_capi.cu
// after sw_kernels.cu, whose band decomposition, task queue, cross-band
// buffers, polling and pair finish this file reuses.
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
// which the row is <= 1.  Rows are never rescaled: the raw values keep the
// compute frame et and every use scales them by 2^(frame - target) (a
// power-of-two factor built from the exponent bits, folded into the gap
// factors).  Frames are floored at 0: the empty alignment's weight 1 is
// always representable and Z >= 1, so values below 2^-149 of it are dropped,
// as the reference drops exponentials below e^-88 of their LSE's maximum.
// Scores are within |s|/T <= 80 (the host's domain check), so E <= 2^115.4
// and a step's raw values stay below 2^122.
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

// Columns past the pair (DM): 0 the band has none, 1 it may have some and they
// are masked without a branch, 2 a warp-uniform branch on whether it has any.
// Kernels that run with every scheduler full keep one copy of their steps (2,
// and no copy for chunks inside the pair): with several the instruction cache
// misses cost more than the branches (4096 ragged pairs at 8 columns per lane,
// forward + adjoint: 7.0 ms against 5.0).  The sweeps of small batches (SPLIT)
// run a warp or two per scheduler, and there a branch costs its latency.
template <int DM> __device__ __forceinline__ bool masks(bool has_dead) {
  return DM == 1 || (DM == 2 && has_dead);
}

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

// Model variants (template argument GM, as in sw_kernels.cu): 0 the local
// models, 1 the global ones, 2 Saigo-Vert.  Against the recurrences above:
// * global (soft Needleman-Wunsch): no fresh start and one end, the cell
//   (L1, L2); A[i,j] = E A_diag + G (A_up + A_left), and with affine gaps also
//   I from D above and D from I on the left, at the open factor.  Row 0 and
//   column 0 hold the boundary gaps.  Frames are not floored at 0 (there is no
//   weight 1 to keep), ZF stands for "no value yet".
// * Saigo-Vert: D also from I on the left (open factor), and only M ends.
constexpr int ZF_NONE = -(1 << 28);
template <int GM> __host__ __device__ constexpr int zero_frame() { return GM == 1 ? ZF_NONE : 0; }
template <int GM> __device__ __forceinline__ int floor_frame(int n) { return GM == 1 ? n : max(n, 0); }
// Frames in cross-band records are biased so that no word is the sentinel.
template <int GM> __host__ __device__ constexpr int frame_bias() { return GM ? (1 << 29) : 0; }

// ---- spread.  A lane keeps its columns of a row under one frame, so a value
// far enough below the row's largest loses bits or all of it.  The
// double-float log-domain kernels do not, so the models that they otherwise
// serve (GM 1 and 2) place their rows HEADROOM bits higher in fp32's range
// (scores up to XHEAD fit on top of it), which leaves 2^-174 below a row's
// inputs, and watch what is left; a pair in which it may have mattered is run
// again in the log domain:
// * the forward flags a pair when a raw value of some lane's row is below
//   2^-SPREAD (Saigo-Vert: values below 2^-45 of the empty alignment do not
//   count, as any continuation of theirs weighs less than a fresh start), or
//   when a score passes XHEAD;
// * the adjoint flags a pair when a raw value of beta is below 2^-SPREAD where
//   it may count: where 2^-126 of the row's frame times the row's alpha is
//   over 2^-45 of Z (with a bit of its own: bands of the pair that have not
//   started must not stop, their neighbours wait for them).
// Of 1024 pairs of 32 to 1024 rows and columns at T = 0.5, one or two come
// within 2^-110 of a row's largest value, and each such pair run again costs a
// whole chain of log-domain steps; hence the headroom.
template <int GM> __host__ __device__ constexpr int headroom() { return GM ? 48 : 0; }
template <int GM> __host__ __device__ constexpr float score_max() { return GM ? 70.f : XMAX; }
constexpr int SPREAD = 124;
__device__ __forceinline__ void flag_redo(const Args& a, int p, int lane, unsigned flag) {
  if (lane == 0) {
    atomicOr(a.pair_done + p, flag);
    atomicOr(a.status + 1, 1u);
  }
}
__device__ __forceinline__ unsigned ld_flag(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ bool redo_set(const Args& a, int p) { return (ld_flag(a.pair_done + p) & PAIR_REDO) != 0; }
// Smallest live column of a row of sums.
template <int DM, int H> __device__ __forceinline__ float min2(const float2 (&p)[H], int nlive, bool hd) {
  float m = INFINITY;
#pragma unroll
  for (int k = 0; k < H; ++k) {
    const bool x = !masks<DM>(hd) || k < nlive, y = !masks<DM>(hd) || k + H < nlive;
    m = fminf(m, fminf(x ? p[k].x : INFINITY, y ? p[k].y : INFINITY));
  }
  return m;
}

// Lane state of the forward wavefront.
template <int NS, int R> struct LState {
  static constexpr int H = R / 2;
  float2 v[NS == 3 ? 2 : 1][H];    // raw M and I (linear: A) of the lane's latest row (frame e)
  float2 c[NS == 3 ? H : 1];       // affine: the row's column sums (M + I) + D (frame e)
  float ds;                        // the left lane's column sum (linear: A) of that row, last column (frame e)
  float od, oc;                    // out to the right lane: D of the column after the last, the last column's sum
  int e, n, nd;                    // raw frame, normalised frame, the left lane's normalised frame of that row
};

// Exponent bound of a non-negative sum: x <= 2^(sexp(x) - 126).
__device__ __forceinline__ int sexp(float x) { return (int)(__float_as_uint(x) >> 23); }

template <int NS, int R, int GM>
__device__ __forceinline__ void lstate_zero(LState<NS, R>& s) {
  constexpr int H = R / 2;
#pragma unroll
  for (int k = 0; k < H; ++k) {
    s.v[0][k] = dup2(0.f);
    if constexpr (NS == 3) { s.v[1][k] = dup2(0.f); s.c[k] = dup2(0.f); }
  }
  s.ds = 0.f; s.od = 0.f; s.oc = 0.f;
  s.e = zero_frame<GM>(); s.n = s.e; s.nd = s.e;
}

// 2^x as a mantissa in (0.5, 1] under the frame e (x may be far out of range).
__device__ __forceinline__ float split2(double x, int& e) {
  const double f = ceil(x);
  e = (int)f;
  return exp2f((float)(x - f));
}
// log2 of the boundary gap of length n >= 1 (affine: open, then extensions).
template <int NS> __device__ __forceinline__ double gap_log2(const LParams& lp, int n) {
  const double o = (double)lp.go * (double)lp.k;
  return NS == 3 ? o + (double)(n - 1) * ((double)lp.ge * (double)lp.k) : (double)n * o;
}

// Global alignment: the lane's columns of row 0 (jl columns lie to the left).
template <int NS, int R, int DM>
__device__ __forceinline__ void lstate_row0(LState<NS, R>& s, float2 (&d)[R / 2], const LParams& lp, int jl,
                                            int nlive, bool hd) {
  constexpr int H = R / 2;
  lstate_zero<NS, R, 1>(s);
  if (nlive > 0) {
    split2(gap_log2<NS>(lp, jl + 1), s.e);
    float2 x[H];
#pragma unroll
    for (int c = 0; c < R; ++c) {   // D as ldchain rebuilds it from its first column
      if (NS == 3 && c > 0) col(x, c) = lp.xge * col(x, c - 1);
      else col(x, c) = exp2f((float)(gap_log2<NS>(lp, jl + 1 + c) - (double)s.e));
    }
    if (masks<DM>(hd)) {
#pragma unroll
      for (int c = 0; c < R; ++c)
        if (c >= nlive) col(x, c) = 0.f;
    }
#pragma unroll
    for (int k = 0; k < H; ++k) {
      if constexpr (NS == 3) { d[k] = x[k]; s.c[k] = x[k]; }
      else s.v[0][k] = x[k];
    }
    const double left = jl > 0 ? gap_log2<NS>(lp, jl) : 0.0;   // the cell (0, jl)
    s.ds = exp2f((float)(left - (double)s.e));
    s.nd = (int)ceil(left);
    s.n = s.e - 126 + sexp(sum2(x));
    s.oc = x[H - 1].y;
  }
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

// What D opens from: M, and I where the model lets D follow I.
template <int R, int GM>
__device__ __forceinline__ void dsource(const float2 (&m)[R / 2], const float2 (&iv)[R / 2], float2 (&o)[R / 2]) {
#pragma unroll
  for (int k = 0; k < R / 2; ++k) o[k] = GM ? add2(m[k], iv[k]) : m[k];
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
template <int NS, int R, int DM, int GM>
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
    float2 ds[H];
    dsource<R, GM>(s.v[0], s.v[1], ds);
    ldchain<NS, R, DM>(ds, x[V + 3], gO, gE, nlive, hd, d, s.od);
#pragma unroll
    for (int k = 0; k < H; ++k) s.c[k] = add2(add2(s.v[0][k], s.v[1][k]), d[k]);
    s.oc = s.c[H - 1].y;
    rs = sum2(s.c);
  } else {
    s.od = 0.f;
    s.oc = s.v[0][H - 1].y;
    rs = sum2(s.v[0]);
  }
  s.n = floor_frame<GM>(s.e - 126 + sexp(rs));
}

// One step of the forward wavefront for one lane: (xd, xc) are the left
// lane's outputs of this row in its raw frame xe (normalised frame xn), E the
// emissions 2^(s k) (0 past the pair).  Updates the state to this row in the
// frame et (its raw frame from then on) and returns the row's sum over its
// columns and states in `rs`.
// Affine: M, I and `d` = D; linear: A and `d` = the emission part.
template <int NS, int R, int DM, int GM>
__device__ __forceinline__ void lcells(LState<NS, R>& s, float xd, float xc, int xe, int xn,
                                       const float2 (&E)[R / 2], float gO, float gE, int nlive, bool hd,
                                       float2 (&d)[R / 2], float& rs) {
  constexpr int H = R / 2;
  // the row's frame is at least every input's normalised frame, so that every
  // converted input is <= 1 (a raw value's frame exceeds its normalised frame
  // by at most 126)
  int et = max(max(s.n, xn), s.nd);
  if constexpr (GM != 0) et = max(max(et - headroom<GM>(), s.e - 127), xe - 127);   // (conversions stay below 2^128)
  s.nd = xn;
  const int q = 127 - et;
  const float fU = p2b(s.e + q), fL = p2b(xe + q);
  const float2 fU2 = dup2(fU), st2 = dup2(GM == 1 ? 0.f : p2b(q));   // st: the fresh-start term 1 in frame et
  if constexpr (NS == 3) {
    float2 m[H];
#pragma unroll
    for (int k = 0; k < H; ++k) {
      const float2 p = k == 0 ? make_float2(s.ds, s.c[H - 1].x) : s.c[k > 0 ? k - 1 : 0];
      m[k] = GM == 1 ? mul2(E[k], mul2(fU2, p)) : mul2(E[k], fma2(fU2, p, st2));
    }
    const float2 gOu = dup2(gO * fU), gEu = dup2(gE * fU);
#pragma unroll
    for (int k = 0; k < H; ++k)   // I opens from M above (global: and from D above)
      s.v[1][k] = fma2(gOu, GM == 1 ? add2(s.v[0][k], d[k]) : s.v[0][k], mul2(gEu, s.v[1][k]));
    float2 ds[H];
    dsource<R, GM>(m, s.v[1], ds);
    ldchain<NS, R, DM>(ds, xd * fL, gO, gE, nlive, hd, d, s.od);
#pragma unroll
    for (int k = 0; k < H; ++k) {
      s.v[0][k] = m[k];
      s.c[k] = add2(add2(m[k], s.v[1][k]), d[k]);
    }
    s.ds = xc * fL;
    s.oc = s.c[H - 1].y;
    rs = sum2(s.c);
  } else {
    const float2 gU = dup2(gO * fU);
    float2 x[H];
#pragma unroll
    for (int k = 0; k < H; ++k) {
      const float2 p = k == 0 ? make_float2(s.ds, s.v[0][H - 1].x) : s.v[0][k > 0 ? k - 1 : 0];
      d[k] = GM == 1 ? mul2(E[k], mul2(fU2, p)) : mul2(E[k], fma2(fU2, p, st2));
    }
#pragma unroll
    for (int k = 0; k < H; ++k) x[k] = fma2(gU, s.v[0][k], d[k]);
    s.ds = xc * fL;
    col(s.v[0], 0) = fmaf(gO, s.ds, col(x, 0));
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
  // the row sum over columns and states bounds every value of the row (all
  // are >= 0) and is the row's partition term
  s.e = et;
  s.n = floor_frame<GM>(1 - q + sexp(rs));
}

// Rows outside the pair have E = 0 in the outside recursion: the scores there
// are whatever was loaded last, and a lane's state above row 1 enters the
// quiet-chunk test of its warp.
template <int R>
__device__ __forceinline__ void lblank(bool act, float2 (&xs)[R / 2], float2 (&E)[R / 2]) {
#pragma unroll
  for (int j = 0; j < R / 2; ++j) {
    if (!act) { xs[j] = dup2(NEG); E[j] = dup2(0.f); }
  }
}

// Scaled scores and emissions of one step as pairs: clamped at XMAX, NEG
// (E = 0) in columns past the pair.
template <int R, int DM, int GM>
__device__ __forceinline__ void lemit(const float (&sb)[R], float k, int nlive, bool hd, float2 (&xs)[R / 2],
                                      float2 (&E)[R / 2]) {
  constexpr int H = R / 2;
  float x[R];
#pragma unroll
  for (int c = 0; c < R; c += 2) {
    const float2 t = mul2(make_float2(sb[c], sb[c + 1]), dup2(k));
    x[c] = fminf(t.x, score_max<GM>());
    x[c + 1] = fminf(t.y, score_max<GM>());
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
// Affine: one float4 (od, oc, raw frame, normalised frame); linear: one
// float2 (oc, the two frames packed).  A band's records start at the next
// 16-byte boundary of its edge slice (2 NS floats per row hold them with the
// padding; slices start at even offsets).
template <int NS, int GM = 0> struct LEdge {
  static constexpr int BIAS = frame_bias<GM>(), B16 = GM ? (1 << 23) : 0;   // affine; linear
  __device__ static __forceinline__ float* base(float* edge, size_t off) {
    return edge + (NS == 3 ? (off + 3) / 4 * 4 : off);
  }
  __device__ static __forceinline__ void put(float* b, int i, float od, float oc, int e, int n, int rs_exp) {
    if constexpr (NS == 3) {
      reinterpret_cast<float4*>(b)[i - 1] = make_float4(od, oc, __int_as_float(e + BIAS), __int_as_float(n + BIAS));
    } else {
      reinterpret_cast<float2*>(b)[i - 1] = make_float2(oc, __uint_as_float(((unsigned)(e + B16) << 8) | (unsigned)rs_exp));
    }
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
      return is_sentinel(v.x) || is_sentinel(v.y) || is_sentinel(v.z) || is_sentinel(v.w);
    else
      return is_sentinel(v.x) || is_sentinel(v.y);
  }
  // (od, oc, e, n) of a resolved record
  __device__ static __forceinline__ float4 open(const float4& v) {
    if constexpr (NS == 3)
      return make_float4(v.x, v.y, __int_as_float(__float_as_int(v.z) - BIAS), __int_as_float(__float_as_int(v.w) - BIAS));
    const unsigned w = __float_as_uint(v.y);
    const int e = (int)(w >> 8) - B16;
    return make_float4(0.f, v.x, __int_as_float(e), __int_as_float(floor_frame<GM>(e - 126 + (int)(w & 0xffu))));
  }
  // The record that column 0 of a global alignment stands for at row i (a gap
  // of length i), as `open` gives it; column 0 of the other models is empty.
  __device__ static __forceinline__ float4 column0(const LParams& lp, int i) {
    if constexpr (GM != 1) return make_float4(0.f, 0.f, 0.f, 0.f);
    int e;
    const float m = split2(gap_log2<NS>(lp, i), e);
    return make_float4(lp.xgo * m, m, __int_as_float(e), __int_as_float(e));
  }
  // Bounded wait for record i; on expiry the status word and the pair's flag
  // are set and the record reads as 0 (also when the pair is to be run again).
  __device__ static __noinline__ float4 wait(const float* b, int i, uint64_t deadline, unsigned* status,
                                             unsigned* flag) {
    for (int tries = 0;; ++tries) {
      const float4 v = get(b, i, true);
      if (!missing(v)) return v;
      if (GM != 0 && (ld_flag(flag) & PAIR_REDO)) return make_float4(0.f, 0.f, 0.f, 0.f);
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

// ---------------------------------------------------------------------------
// forward band task
// ---------------------------------------------------------------------------

// Score prefetch distance of the tangent kernels' forward (steps).
constexpr int FPF = C_STEPS;
// Score prefetch distance of the sweeps (steps): each row is requested this
// many steps ahead; small batches, whose steps are shorter, look further.
template <bool SPLIT> __host__ __device__ constexpr int fwd_ahead() { return SPLIT ? 8 : 4; }
// Steps per block of the forward: the left band's records are passed a block
// at a time (about 220 cycles a time in a lone warp).
template <bool SPLIT> __host__ __device__ constexpr int fwd_block() { return SPLIT ? 2 * C_STEPS : C_STEPS; }

// Forward wavefront of one band: per-lane partition sums (plain within a
// chunk, Kahan over chunks, in the lane's largest normalised frame), the
// left-to-right edge records and, every C steps, a checkpoint of the lane
// state plus the chunk's largest normalised frame.  The band's partition
// partial is (frame, mantissa sum): Z_band = sum * 2^frame.
//
// The left band's records of a block (WB steps) pass through shared memory,
// where lane 0 reads the one of each step.  They are requested two blocks
// ahead and put there one block ahead, two buffers in turn, so a block whose
// records had been written by then starts without waiting for anything.
//
// DM (see above): 1 also where rows are not 16-byte aligned.
template <int NS, int R, int DM, int GM, bool SPLIT>
__device__ void lfwd_band(const Args& a, const LParams& lp, const Place& w, int lane,
                          uint64_t deadline, float4* sedge) {
  using LD = LDims<NS, R>;
  using LE = LEdge<NS, GM>;
  constexpr int H = R / 2, AH = fwd_ahead<SPLIT>(), WB = fwd_block<SPLIT>();
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
  if (!(L1 > 0 && col0 < L2) || (GM != 0 && redo_set(a, w.p))) {
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
  float2 d[H];
#pragma unroll
  for (int j = 0; j < H; ++j) d[j] = dup2(0.f);
  if constexpr (GM == 1) lstate_row0<NS, R, DM>(s, d, lp, jl, nlive, hd);
  else lstate_zero<NS, R, GM>(s);
  int spread = 0;   // the lane's largest spread so far
  float zm = (band == 0 && lane == 0) ? 1.f : 0.f, zc = 0.f;   // M[0,0]: the empty alignment
  int ze = 0;

  // lane u < WB holds the left band's edge record lane 0 needs at step u of a
  // block: `ea` of the next block, `eb` of the one after
  auto get_edge = [&](int bl) {
    const int ie = bl * WB + lane + 1;
    return LE::get(ein, ie, ein && lane < WB && ie <= L1);
  };
  float4 ea = get_edge(0), eb = get_edge(1);
  bool ready = false;   // this block's records are in shared memory
  [[maybe_unused]] bool stop = false;
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
      if (lane < WB) se[lane] = ein || GM != 1 ? LE::open(ea) : LE::column0(lp, ie);
      __syncwarp();
    }
    // the next block's records, if they are there (fault injection: never)
    ready = __all_sync(FULL, !LE::missing(eb)) && !fault;
    if (ready && lane < WB)
      sedge[((bl + 1) & 1) * WB + lane] = ein || GM != 1 ? LE::open(eb) : LE::column0(lp, (bl + 1) * WB + lane + 1);
    if constexpr (GM != 0) {   // the pair is to be run again in the log domain: leave it
      if (__any_sync(FULL, spread > SPREAD)) flag_redo(a, w.p, lane, PAIR_REDO);
      if (stop) return;
      stop = __any_sync(FULL, lane == 0 && redo_set(a, w.p));
    }
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
        int xe = __shfl_up_sync(FULL, s.e, 1);
        int xn = __shfl_up_sync(FULL, s.n, 1);
        xc = lane == 0 ? e4.y : xc;
        xe = lane == 0 ? __float_as_int(e4.z) : xe;
        xn = lane == 0 ? __float_as_int(e4.w) : xn;
        float2 xs[H], E[H];
        lemit<R, DD, GM>(sb[(h * C_STEPS + cu) % AH], k, nlive, hd, xs, E);
        if constexpr (IN) rows.template fetch<VEC>(src, sb[(h * C_STEPS + cu) % AH]);
        else rows.load(src, i + cu + AH, sb[(h * C_STEPS + cu) % AH]);
        src += rows.ld;
        rsv[cu] = 0.f;
        ev[cu] = 0;
        if (act) {
          lcells<NS, R, DD, GM>(s, xd, xc, xe, xn, E, gO, gE, nlive, hd, d, rsv[cu]);
          if constexpr (GM != 0) {
            float lo;
            if constexpr (NS == 3) lo = min2<DD>(s.c, nlive, hd);
            else lo = min2<DD>(s.v[0], nlive, hd);
            const int x = GM == 2 ? max(sexp(lo), 81 - s.e) : sexp(lo);
            float top = xs[0].x;   // a clamped score (the log domain takes any)
#pragma unroll
            for (int j = 0; j < H; ++j) top = fmaxf(top, fmaxf(xs[j].x, xs[j].y));
            if (top >= score_max<GM>()) spread = 127;
            if (DD == 0 || nlive > 0) spread = max(spread, 127 - x);   // 1 in the row's frame against its least value
          }
          const int rx = sexp(rsv[cu]);
          if constexpr (GM == 2) rsv[cu] = sum2(s.v[0]);   // only M ends an alignment
          ev[cu] = s.e;
          cmx = max(cmx, s.n);
          if (lane == 31) LE::put(eout, i + cu, s.od, s.oc, s.e, s.n, rx);
        }
      }
    };
    bool done = false;
    if constexpr (SPLIT) {
      if (in_block) {
        done = true;
        if (DM != 1 || rows.vec) steps(std::true_type{}, std::true_type{});
        else if constexpr (DM == 1) steps(std::true_type{}, std::false_type{});
      }
    }
    if (!done) steps(std::false_type{}, std::false_type{});
    i += C_STEPS;
    // partition: the chunk's row sums in the frame ze (the largest normalised
    // frame so far), Kahan-compensated from chunk to chunk
    if constexpr (GM != 1) {
      const int zn = max(ze, cmx);
      const float f = p2b(ze - zn + 127);
      float y = 0.f;
#pragma unroll
      for (int cu = 0; cu < C_STEPS; ++cu) y = fmaf(rsv[cu], p2b(ev[cu] - zn + 127), y);
      zm *= f;
      y -= zc * f;
      const float tt = zm + y;
      zc = (tt - zm) - y;
      zm = tt;
      ze = zn;
    }
    if (keep_ck) {
      cmx = __reduce_max_sync(FULL, cmx);
      if (lane == 0 && kc < nch) ckmax[kc] = __int_as_float(cmx);
    }
    }
  }
  if constexpr (GM != 0) {
    if (__any_sync(FULL, spread > SPREAD)) flag_redo(a, w.p, lane, PAIR_REDO);
  }
  if constexpr (GM == 1) {   // the terminal cell (L1, L2): Z of the pair, in its band's partial
    const int q = L2 - 1 - jl;
    if (q >= 0 && q < R) {
      float v = 0.f;
#pragma unroll
      for (int c = 0; c < R; ++c) {
        float x;
        if constexpr (NS == 3) x = col(s.c, c);
        else x = col(s.v[0], c);
        v = c == q ? x : v;
      }
      part[0] = (float)s.e;
      part[1] = v;
    }
  } else {
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
}

#ifndef SWB_LFWD_MINB
#define SWB_LFWD_MINB 4
#endif
template <int NS, int R, int GM, bool SPLIT>
__global__ void __launch_bounds__(128, SWB_LFWD_MINB) lfwd_kernel(Args a) {
  __shared__ float4 s_edge[4][2 * fwd_block<SPLIT>()];   // per warp: the left band's records of two blocks
  const int lane = threadIdx.x & 31;
  const LParams lp = lparams<NS>(a);
  const uint64_t deadline = gtimer() + a.spin_limit_ns;
  const int ntasks = (a.layout == 0) ? a.B * a.nb : a.ntasks;
  while (true) {
    int task = 0;
    if (lane == 0) task = (int)atomicAdd(a.counters + 0, 1u);
    task = __shfl_sync(FULL, task, 0);
    if (task >= ntasks) break;
    const Place w = place_of<NS, R, GM>(a, task, false);
    // a band whose last columns lie past the pair takes the variant that masks them
    float4* se = s_edge[threadIdx.x >> 5];
    if constexpr (!SPLIT) lfwd_band<NS, R, 2, GM, false>(a, lp, w, lane, deadline, se);
    else if ((w.band + 1) * 32 * R > w.pr.L2 || !w.pr.vec) lfwd_band<NS, R, 1, GM, true>(a, lp, w, lane, deadline, se);
    else lfwd_band<NS, R, 0, GM, true>(a, lp, w, lane, deadline, se);
  }
}

// ---------------------------------------------------------------------------
// partition of a pair
// ---------------------------------------------------------------------------

// Z of pair w as (integer frame ze, mantissa zm): Z = zm * 2^ze, combined
// from the band partials in a fixed order (deterministic).
template <int R = 4, int GM = 0>
__device__ __forceinline__ void lpair_z(const Args& a, const Place& w, int lane, int& ze, float& zm) {
  if constexpr (GM == 1) {   // the terminal cell's band holds it
    const float* q = a.part + 2 * (w.slot0 + max(w.pr.L2 - 1, 0) / (32 * R));
    ze = (int)q[0];
    zm = q[1];
  } else {
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
template <int NS, int R, int GM = 0>
__global__ void __launch_bounds__(128) lvalue_kernel(Args a) {
  const int lane = threadIdx.x & 31;
  const int q = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (q >= a.B) return;
  Place w;
  if (a.layout == 0) {
    w = place_of<NS, R, GM>(a, q * a.nb, false);
  } else {
    const long long* pw = a.plan_pairs + (size_t)q * PLAN_PAIR_WORDS;
    w.p = q;
    w.nb = (int)pw[PW_NB];
    w.slot0 = (size_t)pw[PW_SLOT0];
    w.pr.L1 = (int)pw[PW_L1];
    w.pr.L2 = (int)pw[PW_L2];
  }
  if (a.pair_done[w.p] & PAIR_TIMEOUT) {   // a bounded wait of this pair expired
    if (lane == 0) a.value[w.p] = __int_as_float(0x7fc00000);
    return;
  }
  if (GM == 1 && (w.pr.L1 == 0 || w.pr.L2 == 0)) {
    float dgo, dge;
    if (lane == 0) a.value[w.p] = empty_global_value<NS>(a, w.pr.L1 + w.pr.L2, dgo, dge);
    return;
  }
  int ze;
  float zm, Sh, Sl;
  lpair_z<R, GM>(a, w, lane, ze, zm);
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
template <int R, int GM> __device__ __forceinline__ void bstate_zero(BState<R>& s) {
#pragma unroll
  for (int k = 0; k < R / 2; ++k) { s.b[k] = dup2(0.f); s.t[k] = dup2(0.f); }
  s.ht = 0.f; s.ob = 0.f;
  s.fb = zero_frame<GM>(); s.nb = s.fb; s.hn = s.fb;
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

// The gradient sums of a band are formed per segment of kSeg chunks (plain
// sums per lane, then a shuffle tree) and folded over the segments, last one
// first, with compensation: the adjoint of a whole band and the segment
// kernel give the same bits.
constexpr int kSeg = 4;
struct BandSum {
  KSum a, b, m;   // m's compensation goes into the fold as well
  __device__ __forceinline__ void add(float x, float y, float z) {
    if (x != 0.f || y != 0.f || z != 0.f) { a.add(x); b.add(y); m.add(z); }
  }
};

// A pair's outputs from its sums: o = expected gap opens (linear gap: steps),
// e = extensions, m = the sum of posteriors times scaled scores.  Global
// alignments: every path has L1 + L2 gap and twice its match steps, so e comes
// in as the sum of posteriors and the gap counts follow; a path that does not
// start with a match at (1, 1) opens a boundary gap.
// dS/dT is a small difference of large terms, formed in 64 bits.
template <int NS, int GM>
__device__ __forceinline__ void lwrite(const Args& a, const Place& w, float Sh, float Sl, double o, double e, double m,
                                       bool bad, PParams pp) {
  const int p = w.p;
  if (bad) {   // a bounded wait of this pair expired
    const float nan = __int_as_float(0x7fc00000);
    a.value[p] = nan; a.g_open[p] = nan; a.g_T[p] = nan;
    if (a.g_ext) a.g_ext[p] = nan;
    return;
  }
  if constexpr (GM == 1) {
    const int n = w.pr.L1 + w.pr.L2;
    if (w.pr.L1 == 0 || w.pr.L2 == 0) {   // the terminal is a boundary cell
      float dgo, dge;
      a.value[p] = empty_global_value<NS>(a, n, dgo, dge);
      a.g_open[p] = dgo;
      if (a.g_ext) a.g_ext[p] = dge;
      a.g_T[p] = 0.f;
      return;
    }
    const double gaps = (double)n - 2.0 * e;
    if (NS == 3) {
      o += 1.0 - (double)ld_poll(w.pr.m);
      e = gaps - o;
    } else {
      o = gaps;
    }
  }
  const float inv_k = 1.f / pp.k;         // = T * ln 2
  a.value[p] = (Sh + Sl) * inv_k;
  a.g_open[p] = (float)o;
  if (a.g_ext) a.g_ext[p] = NS == 3 ? (float)e : 0.f;
  const double ln2T = 0.69314718055994530942 * (double)pp.T;
  const double S = ((double)Sh + (double)Sl) * ln2T;
  a.g_T[p] = (float)((S - (m * ln2T + o * (double)pp.go + (NS == 3 ? e * (double)pp.ge : 0.0))) / (double)pp.T);
}

// End of a band: its gradient partials; the pair's last band folds them in
// band order, so the result is deterministic.
template <int NS, int GM>
__device__ __forceinline__ void lfinish_band(const Args& a, const Place& w, int lane, float Sh, float Sl,
                                             const BandSum& s, PParams pp) {
  __threadfence();   // the map's first cell (global alignments)
  __syncwarp();
  if (lane != 0) return;
  float* gp = a.gpart + 4 * (w.slot0 + w.band);
  gp[0] = s.a.s; gp[1] = s.b.s; gp[2] = s.m.s; gp[3] = -s.m.c;
  __threadfence();
  const unsigned done = atomicAdd(a.pair_done + w.p, 1u);
  if ((done & ~PAIR_FLAGS) != (unsigned)w.nb - 1) return;
  __threadfence();
  double o = 0.0, e = 0.0, m = 0.0;
  for (int b = 0; b < w.nb; ++b) {
    const float* q = a.gpart + 4 * (w.slot0 + b);
    o += (double)ld_poll(q);
    e += (double)ld_poll(q + 1);
    m += (double)ld_poll(q + 2) + (double)ld_poll(q + 3);
  }
  lwrite<NS, GM>(a, w, Sh, Sl, o, e, m, (done & PAIR_TIMEOUT) != 0, pp);
}

// End of a segment: its gradient partials; the pair's last segment folds them
// (lane l the bands l, l + 32, ...; then the bands in order).
template <int NS, int GM>
__device__ __forceinline__ void lfinish_seg(const Args& a, const Place& w, int lane, int seg, float Sh, float Sl,
                                            float g0, float g1, float ps, PParams pp) {
  __threadfence();   // the map's first cell (global alignments)
  __syncwarp();
  unsigned done = 0;
  if (lane == 0) {
    reinterpret_cast<float4*>(a.spart)[(w.slot0 + w.band) * a.nseg + seg] = make_float4(g0, g1, ps, 0.f);
    __threadfence();
    done = atomicAdd(a.pair_done + w.p, 1u);
  }
  done = __shfl_sync(FULL, done, 0);
  if ((done & ~PAIR_FLAGS) != (unsigned)(w.nb * a.nseg) - 1) return;
  __threadfence();
  double o = 0.0, e = 0.0, m = 0.0;
  for (int b0 = 0; b0 < w.nb; b0 += 32) {
    BandSum s;
    if (b0 + lane < w.nb) {
      const float* x = a.spart + 4 * (w.slot0 + b0 + lane) * a.nseg;
      for (int q = a.nseg - 1; q >= 0; --q) s.add(ld_poll(x + 4 * q), ld_poll(x + 4 * q + 1), ld_poll(x + 4 * q + 2));
    }
    for (int b = 0; b < min(32, w.nb - b0); ++b) {
      o += (double)__shfl_sync(FULL, s.a.s, b);
      e += (double)__shfl_sync(FULL, s.b.s, b);
      m += (double)__shfl_sync(FULL, s.m.s, b) + (double)(-__shfl_sync(FULL, s.m.c, b));
    }
  }
  if (lane == 0) lwrite<NS, GM>(a, w, Sh, Sl, o, e, m, (done & PAIR_TIMEOUT) != 0, pp);
}

// One row of the outside recursion for one lane: (rb, rt, rn) are the right
// lane's beta_D (linear: beta) of its column 0, its t and its normalised
// frame; live: the row is inside the pair (global: it is the last row; term:
// the terminal's column in this lane, or -1).  Returns, in the frame `ft`: vm =
// beta_M (beta), sr = beta_I below + beta_D right and br = beta_D right per
// column.  The state moves on with bfinish.
template <int NS, int R, int DM, int GM>
__device__ __forceinline__ void bcells(const BState<R>& s, float rb, int rn, bool live, int term, float gO, float gE,
                                       float gX, int nlive, bool hd, int& ft, float& fB,
                                       float2 (&vm)[R / 2], float2 (&vi)[R / 2], float2 (&sr)[R / 2],
                                       float2 (&br)[R / 2], float& vd0, float& mx) {
  constexpr int H = R / 2;
  // frames: the row is computed in ft >= every input's normalised frame
  ft = max(max(s.nb, rn), s.hn);
  if constexpr (GM != 0) ft = max(ft - headroom<GM>(), s.fb - 127);
  if (GM == 1 && live && term >= 0) ft = max(ft, 0);
  const int q = 127 - ft;
  fB = p2b(s.fb + q);
  const float fT = p2b(s.nb + q), fR = p2b(rn + q), fH = p2b(s.hn + q);
  const float one = live && (GM != 1 || term >= 0) ? p2b(q) : 0.f;
  // base: the diagonal successor's t, plus 1 where the alignment may end;
  // nom: the same without M's end (Saigo-Vert: only M ends)
  float2 base[H], nom[H];
#pragma unroll
  for (int k = 0; k < H; ++k) {
    float2 oc = dup2(one);
    if constexpr (GM == 1) oc = make_float2(k == term ? one : 0.f, k + H == term ? one : 0.f);
    else if (masks<DM>(hd)) oc = make_float2(k < nlive ? one : 0.f, k + H < nlive ? one : 0.f);
    const float2 f = k == H - 1 ? make_float2(fT, fH) : dup2(fT);
    const float2 t = k == H - 1 ? make_float2(s.t[0].y, s.ht) : s.t[k < H - 1 ? k + 1 : 0];
    base[k] = fma2(f, t, oc);
    nom[k] = GM == 2 ? mul2(f, t) : base[k];
  }
  const float b0 = fR * rb;   // right successor's beta_D (beta) of the last column
  float2 v[H];                // beta_D (beta) per column
  const float2 gEb = dup2(gE * fB), gOb = dup2(gO * fB);
  if constexpr (NS == 3) {
    float2 x[H];              // global: D also goes on to I below
#pragma unroll
    for (int k = 0; k < H; ++k) x[k] = GM == 1 ? fma2(gOb, s.b[k], nom[k]) : nom[k];
    col(v, R - 1) = fmaf(gE, b0, col(x, R - 1));
#pragma unroll
    for (int c = R - 2; c >= 0; --c) col(v, c) = fmaf(gE, col(v, c + 1), col(x, c));
  } else {
    float2 x[H];
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
#pragma unroll
    for (int k = 0; k < H; ++k) {
      vm[k] = fma2(dup2(gO), sr[k], base[k]);
      // I goes on to I below and, but for the local model, to D on the right
      vi[k] = fma2(gEb, s.b[k], GM ? fma2(dup2(gO), br[k], nom[k]) : base[k]);
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

// The state after the row: t = E beta_M in the row's normalised frame.
template <int R, int GM>
__device__ __forceinline__ void bfinish(BState<R>& s, int ft, float mx, const float2 (&vm)[R / 2],
                                        const float2 (&vi)[R / 2], float vd0, const float2 (&E)[R / 2],
                                        float rt, int rn) {
  constexpr int H = R / 2;
  const int nn = floor_frame<GM>(ft - 126 + sexp(mx));
  const float bs = p2b(ft - nn + 127);
#pragma unroll
  for (int k = 0; k < H; ++k) {
    s.t[k] = mul2(mul2(vm[k], dup2(bs)), E[k]);
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
// Global alignments: the only fresh weight is the terminal's, so the 1 counts
// in its chunk alone (own).
template <int R, int GM>
__device__ __forceinline__ bool lquiet(const BState<R>& s, int ckm, const float (&pb)[3], int lane, int zlog,
                                       bool own) {
  int inl = s.hn + fexp(s.ht);
  float mb = 0.f, mt = 0.f;   // largest beta and t of the row below
#pragma unroll
  for (int j = 0; j < R / 2; ++j) {
    mb = fmaxf(mb, fmaxf(s.b[j].x, s.b[j].y));
    mt = fmaxf(mt, fmaxf(s.t[j].x, s.t[j].y));
  }
  inl = max(inl, max(s.fb + fexp(mb), s.nb + fexp(mt)));
  if (lane < C_STEPS) inl = max(inl, __float_as_int(pb[2]) + fexp(fmaxf(pb[0], pb[1])));
  return __all_sync(FULL, ckm + 11 + (GM != 1 || own ? max(inl, 0) : inl) < zlog);
}
// ---- quiet run.  After a quiet chunk only lane 31's held t (pt, pn) and the
// right band's records enter the chunks above, so one round of loads decides
// the next 32 / C chunks: lane l takes chunk kn - l / C at backward step
// l % C (lane 31's row there), checking that record and the one of the row
// below (lane l - 1's; lane 0: the held t).  A record not written yet ends
// the run; that chunk is then decided by lquiet from the same values, so
// results do not depend on timing.  Returns how many chunks from kn down (not
// below k_lo) are quiet; r1, rn: the lane's record's t and frame.  Chunk `own`
// (a global alignment's terminal) ends it too. ----
template <int GM>
__device__ __forceinline__ int lquiet_run(const float* pin, size_t Lm, int L1, const float* ckmax, int kn, int k_lo,
                                          int lane, float pt, int pn, int zlog, int own, float& r1, int& rn) {
  constexpr int RUN = 32 / C_STEPS;
  const int j = lane / C_STEPS, u = lane - j * C_STEPS;
  const int kq = kn - j;
  float r0 = 0.f;
  int cm = -(1 << 30);
  bool written = true;
  r1 = 0.f;
  rn = zero_frame<GM>();
  if (kq >= k_lo) {
    const int ir = kq * C_STEPS + C_STEPS - 1 - u - 30;
    if (pin && ir >= 1 && ir <= L1) {
      r0 = ld_poll(pin + 0 * (Lm + 1) + ir);
      r1 = ld_poll(pin + 1 * (Lm + 1) + ir);
      const float r2 = ld_poll(pin + 2 * (Lm + 1) + ir);
      written = !is_sentinel(r0) && !is_sentinel(r1) && !is_sentinel(r2);
      rn = __float_as_int(r2) - frame_bias<GM>();
    }
    cm = __float_as_int(ckmax[kq]);
  }
  const int lg = written ? rn + fexp(fmaxf(r0, r1)) : 0;
  const int lgu = __shfl_up_sync(FULL, lg, 1);
  const bool wu = __shfl_up_sync(FULL, (int)written, 1) != 0;
  const int lgb = lane == 0 ? pn + fexp(pt) : lgu;
  const bool wb = lane == 0 || wu;
  const bool q = kq >= k_lo && (GM != 1 || kq != own) && written && wb && cm + 11 + (GM == 1 ? max(lg, lgb) : max(max(lg, lgb), 0)) < zlog;
  const unsigned ball = __ballot_sync(FULL, q);
  constexpr unsigned grp = (1u << C_STEPS) - 1u;
  int n = 0;
  while (n < RUN && kn - n >= k_lo && ((ball >> (n * C_STEPS)) & grp) == grp) ++n;
  return n;
}
// Zero records to the left band for the rows of chunk kq (lane 0's).
template <int GM>
__device__ __forceinline__ void zero_push(float* pout, size_t Lm, int L1, int kq, int lane) {
  const int i = kq * C_STEPS + lane + 1;
  if (pout && lane < C_STEPS && i <= L1) {
    pout[0 * (Lm + 1) + i] = 0.f;
    pout[1 * (Lm + 1) + i] = 0.f;
    pout[2 * (Lm + 1) + i] = __int_as_float(zero_frame<GM>() + frame_bias<GM>());
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
template <int NS, int R, bool SPARSE, bool SEG, int GM>
__device__ void lbwd_band(const Args& a, const LParams& lp, const Place& w, int lane, float* sm,
                          uint64_t deadline, int seg) {
  using LD = LDims<NS, R>;
  using LE = LEdge<NS, GM>;
  constexpr int H = R / 2, DM = 2;
  constexpr int CKF = LD::CKF, LREC = LD::LREC, FW = LD::FW, NPF = 3;
  const Pair& pr = w.pr;
  const int L1 = pr.L1, L2 = pr.L2;
  const int band = w.band;
  const int col0 = band * 32 * R;
  int ze;
  float zm, Sh, Sl;
  if (GM != 0 && redo_set(a, w.p)) return;   // run again in the log domain
  lpair_z<R, GM>(a, w, lane, ze, zm);
  lz_log2(ze, zm, Sh, Sl);
  const PParams pp{lp.go, lp.ge, lp.T, lp.k};
  const int nch = band_chunks(L1);
  const int k_lo = SEG ? seg * kSeg : 0, k_hi = SEG ? min(k_lo + kSeg, nch) : nch;
  if (!(L1 > 0 && col0 < L2) || k_lo >= k_hi) {
    if constexpr (SEG) lfinish_seg<NS, GM>(a, w, lane, seg, Sh, Sl, 0.f, 0.f, 0.f, pp);
    else lfinish_band<NS, GM>(a, w, lane, Sh, Sl, BandSum{}, pp);
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
    for (int f = 0; f < NPF; ++f) dst[f] = ld_poll_if(pin + f * (Lm + 1) + i, ok);
    if (GM == 1 && !ok) dst[2] = __int_as_float(zero_frame<GM>() + frame_bias<GM>());
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
  else bstate_zero<R, GM>(bs);
  // global: the terminal's column in this lane, and the chunks with row L1 of its lanes
  const int term = GM == 1 && L2 - 1 - jl >= 0 && L2 - 1 - jl < R ? L2 - 1 - jl : -1;
  const int tl = (L2 - 1 - col0) / R;   // the terminal's lane (32 or more: in another band)
  const int ownc = GM == 1 && tl < 32 ? (L1 - 1 + tl) / C_STEPS : -1;
  [[maybe_unused]] bool lost = false;
  BandSum gsum;
  float cA = 0.f, cB = 0.f;   // the segment's plain sums
  float2 cS = dup2(0.f);
  [[maybe_unused]] float2 cP = dup2(0.f);   // global: posteriors
  auto flush = [&]() {        // at the end of a segment
    float v0 = cA, v1 = GM == 1 ? cP.x + cP.y : cB, v2 = cS.x + cS.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v0 += __shfl_xor_sync(FULL, v0, o);
      v1 += __shfl_xor_sync(FULL, v1, o);
      v2 += __shfl_xor_sync(FULL, v2, o);
    }
    gsum.add(v0, v1, v2);
    cA = 0.f; cB = 0.f; cS = dup2(0.f); cP = dup2(0.f);
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
    pbc[2] = __int_as_float(__float_as_int(pbc[2]) - frame_bias<GM>());
    const bool quiet = lquiet<R, GM>(bs, ckm, pbc, lane, zlog, kc == ownc);
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
        zero_push<GM>(pout, Lm, L1, kq, lane);
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
        const int n = lquiet_run<GM>(pin, Lm, L1, ckmax, kn, k_lo, lane, pt, pn, zlog, ownc, r1, rn);
        for (int m = 0; m < n; ++m) zero_chunk(kn - m);
        if (n > 0) {   // lane 31's held t: the record of its top row of the last zeroed chunk
          pt = __shfl_sync(FULL, r1, n * C_STEPS - 1);
          pn = __shfl_sync(FULL, rn, n * C_STEPS - 1);
        }
        kn -= n;
        if (n < 32 / C_STEPS) break;
      }
      if (!SEG && kc / kSeg != (kn + (kn < 0 ? -kSeg + 1 : 0)) / kSeg) flush();   // the run left the segment
      bstate_zero<R, GM>(bs);
      bs.ht = lane == 31 ? pt : 0.f;
      bs.hn = lane == 31 ? pn : zero_frame<GM>();
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
    lck_restore<NS, R, DM, GM>(stg_ck, lane, st, gO, gE, nlive, hd, d);
    if (lane < C_STEPS) s_eb[lane] = ein || GM != 1 ? LE::open(ebr) : LE::column0(lp, t0 + lane + 1);
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
          float4 er = ein || GM != 1 ? LE::open(get_edge(ka)) : LE::column0(lp, ka * C_STEPS + lane + 1);
#pragma unroll 1
          for (int u0 = 0; u0 < C_STEPS; u0 += PF)
#pragma unroll
          for (int u = 0; u < PF; ++u) {
            const int cu = u0 + u;
            const bool act = (unsigned)(i - 1) < (unsigned)L1;
            float xd = 0.f;
            if constexpr (NS == 3) xd = __shfl_up_sync(FULL, st.od, 1);
            float xc = __shfl_up_sync(FULL, st.oc, 1);
            int xe = __shfl_up_sync(FULL, st.e, 1);
            int xn = __shfl_up_sync(FULL, st.n, 1);
            const float e0 = __shfl_sync(FULL, er.x, cu), e1 = __shfl_sync(FULL, er.y, cu);
            const float e2 = __shfl_sync(FULL, er.z, cu), e3 = __shfl_sync(FULL, er.w, cu);
            if (lane == 0) { xd = e0; xc = e1; xe = __float_as_int(e2); xn = __float_as_int(e3); }
            float2 xs[H], E[H];
            lemit<R, DM, GM>(ab[u], k, nlive, hd, xs, E);
            rows.load(src, i + PF, ab[u]);
            src += rows.ld;
            float rs;
            if (act) lcells<NS, R, DM, GM>(st, xd, xc, xe, xn, E, gO, gE, nlive, hd, d, rs);
            ++i;
          }
        }
      }
    }
#pragma unroll
    for (int cu = 0; cu < C_STEPS; ++cu) {
      const int i = t0 + cu - lane + 1;
      const bool act = (unsigned)(i - 1) < (unsigned)L1;
      float xd = 0.f;
      if constexpr (NS == 3) xd = __shfl_up_sync(FULL, st.od, 1);
      float xc = __shfl_up_sync(FULL, st.oc, 1);
      int xe = __shfl_up_sync(FULL, st.e, 1);
      int xn = __shfl_up_sync(FULL, st.n, 1);
      if (lane == 0) {
        const float4 e4 = s_eb[cu];
        xd = e4.x; xc = e4.y; xe = __float_as_int(e4.z); xn = __float_as_int(e4.w);
      }
      float2 xs[H], E[H];
      lemit<R, DM, GM>(nsb[cu], k, nlive, hd, xs, E);
      lblank<R>(act, xs, E);
      float rs;
      if (act) lcells<NS, R, DM, GM>(st, xd, xc, xe, xn, E, gO, gE, nlive, hd, d, rs);
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
      if constexpr (GM == 0) {
        ent[LD::NF * R * 32 + lane] = __int_as_float(st.e);
      } else {   // the raw frame and the exponent of the row's sum
        float all;
        if constexpr (NS == 3) all = sum2(st.c);
        else all = sum2(st.v[0]);
        ent[LD::NF * R * 32 + lane] = __int_as_float((int)((unsigned)st.e << 8) | sexp(all));
      }
    }
    if (kc > k_lo) {   // prefetch the next chunk's inputs while the outside recursion runs
      load_ck(kc - 1);
      ebr = get_edge(kc - 1);
      load_sb(kc - 1);
      load_pb(kc - 1, pbn);
    }
    if (lane < C_STEPS) s_pb[lane] = make_float4(pbc[0], pbc[1], pbc[2], 0.f);
    __syncwarp();
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
      const int ew = __float_as_int(ent[LD::NF * R * 32 + lane]);
      const int ea = GM == 0 ? ew : ew >> 8;
      float2 fm[H], fd[H], xs[H], E[H];
      get(0, fm);
      get(LD::NF - 2, fd);
      get(LD::NF - 1, xs);
#pragma unroll
      for (int j = 0; j < H; ++j) E[j] = make_float2(ex2(xs[j].x), ex2(xs[j].y));
      int ft;
      float fB, vd0, mx;
      float2 vm[H], vi[H], sr[H], br[H], P[H];
      bcells<NS, R, DM, GM>(bs, rb, rn, GM == 1 ? i == L1 : act, term, gO, gE, gX, nlive, hd, ft, fB, vm, vi, sr, br, vd0, mx);
      // raw alpha (frame ea) times raw beta (frame ft), over Z
      // (with headroom the product's exponent may leave the range of one
      // factor: half goes to each side)
      const int ax = ea + ft - ze;
      const float asc = p2any(GM ? ax >> 1 : ax) * invZ, bsc = GM ? p2any(ax - (ax >> 1)) : 1.f;
      if constexpr (GM != 0) {   // a beta near the end of the range where alpha makes it count
        const int bx = 127 - sexp(min2<DM>(vm, nlive, hd));
        lost = lost || (act && (DM == 0 || nlive > 0) && bx > SPREAD && ea - 126 + (ew & 255) + ft - 81 > zlog + SWB_LQUIET);
      }
      float2 so = dup2(0.f);
#pragma unroll
      for (int j = 0; j < H; ++j) {
        const float2 q = mul2(NS == 3 ? fm[j] : fd[j], dup2(asc));
        const float2 p = mul2(q, GM ? mul2(vm[j], dup2(bsc)) : vm[j]);
        P[j] = make_float2(fminf(p.x, 1.f), fminf(p.y, 1.f));   // a posterior: rounding may pass 1
        if constexpr (GM == 0) so = fma2(fm[j], sr[j], so);
        else if constexpr (NS == 3) so = fma2(q, sr[j], so);   // scaled first: raw values fill the range here
        // (an excluded cell, score -inf, has posterior 0)
        cS = fma2(P[j], GM == 0 ? xs[j] : make_float2(fmaxf(xs[j].x, NEG), fmaxf(xs[j].y, NEG)), cS);
        if constexpr (GM == 1) cP = add2(cP, P[j]);
      }
      if constexpr (GM != 0 && NS == 3) {
        // opens: M to I and D, I to D, and in global alignments D to I (for
        // lane 0 of the first band from column 0 too)
        float2 fi[H];
        get(1, fi);
        float2 sdi = dup2(0.f);
#pragma unroll
        for (int j = 0; j < H; ++j) {
          so = fma2(mul2(fi[j], dup2(asc)), br[j], so);
          if constexpr (GM == 1) sdi = fma2(mul2(fd[j], dup2(asc)), bs.b[j], sdi);
        }
        float o = fmaf(sdi.x + sdi.y, fB, so.x + so.y) * bsc * gO;
        if constexpr (GM == 1) {
          if (band == 0 && lane == 0 && act) {
            const float4 e4 = s_eb[C_STEPS - 1 - cu];
            const int x = __float_as_int(e4.z) + ft - ze;
            o = fmaf(e4.x * (p2any(x >> 1) * invZ), vd0 * p2any(x - (x >> 1)), o);
          }
        }
        if (GM == 2 || act) cA += o;
      } else if constexpr (GM != 1) {
        cA = fmaf((so.x + so.y) * asc, gO, cA);
      }
      if constexpr (NS == 3 && GM != 1) {
        float2 fi[H];
        get(1, fi);
        float2 sxi = dup2(0.f), sxd = dup2(0.f);
#pragma unroll
        for (int j = 0; j < H; ++j) {
          sxi = fma2(GM ? mul2(fi[j], dup2(asc)) : fi[j], bs.b[j], sxi);
          sxd = fma2(GM ? mul2(fd[j], dup2(asc)) : fd[j], br[j], sxd);
        }
        const float x = fmaf(sxi.x + sxi.y, fB, sxd.x + sxd.y);
        cB = fmaf(x * (GM ? bsc : asc), gE, cB);
      }
      bfinish<R, GM>(bs, ft, mx, vm, vi, vd0, E, rt, rn);
      if constexpr (GM == 1 && NS == 3) {
        if (i == 1) {   // the D's of row 0 open into I of row 1
          LState<NS, R> z;
          float2 d0[H], o = dup2(0.f);
#pragma unroll
          for (int j = 0; j < H; ++j) d0[j] = dup2(0.f);
          lstate_row0<NS, R, DM>(z, d0, lp, jl, nlive, hd);
          const int x = z.e + bs.fb - ze;
#pragma unroll
          for (int j = 0; j < H; ++j) o = fma2(mul2(d0[j], dup2(p2any(x >> 1) * invZ)), mul2(bs.b[j], dup2(p2any(x - (x >> 1)))), o);
          cA = fmaf(o.x + o.y, gO, cA);
        }
      }
      if (act) {
        store_pairs<R>(mrow, jl, pr, P);
        if (lane == 0 && pout) {
          pout[0 * (Lm + 1) + i] = bs.ob;
          pout[1 * (Lm + 1) + i] = bs.t[0].x;
          pout[2 * (Lm + 1) + i] = __int_as_float(bs.nb + frame_bias<GM>());
        }
      }
      --i;
      mrow -= pr.ld;
    }
#pragma unroll
    for (int f = 0; f < NPF; ++f) pbc[f] = pbn[f];
    if (!SEG && kc % kSeg == 0) flush();
    __syncwarp();
  }
  if constexpr (GM != 0) {
    if (__any_sync(FULL, lost)) flag_redo(a, w.p, lane, PAIR_LOST);
  }
  if constexpr (SEG) {
    flush();
    lfinish_seg<NS, GM>(a, w, lane, seg, Sh, Sl, gsum.a.s, gsum.b.s, gsum.m.s, pp);
  } else {
    lfinish_band<NS, GM>(a, w, lane, Sh, Sl, gsum, pp);
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

template <int NS, int R, int DM, int GM>
__device__ void lbeta_band(const Args& a, const LParams& lp, const Place& w, int lane, uint64_t deadline,
                           float4* spush) {
  using LD = LDims<NS, R>;
  constexpr int H = R / 2, AH = fwd_ahead<true>(), SUB = AH / C_STEPS, NPF = 3;
  const Pair& pr = w.pr;
  const int L1 = pr.L1, L2 = pr.L2;
  const int band = w.band;
  const int col0 = band * 32 * R;
  if (!(L1 > 0 && col0 < L2)) return;
  int ze;
  float zm;
  if (GM != 0 && redo_set(a, w.p)) return;   // run again in the log domain
  lpair_z<R, GM>(a, w, lane, ze, zm);
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
  bstate_zero<R, GM>(bs);
  const int term = GM == 1 && L2 - 1 - jl >= 0 && L2 - 1 - jl < R ? L2 - 1 - jl : -1;
  const int tl = (L2 - 1 - col0) / R;
  const int ownc = GM == 1 && tl < 32 ? (L1 - 1 + tl) / C_STEPS : -1;
  auto get_push = [&](int kc) {   // lane u < C: the right band's record lane 31 needs at backward step u
    const int i = kc * C_STEPS + C_STEPS - 1 - lane - 30;
    FieldVec<NPF> x;
    const bool ok = pin && lane < C_STEPS && i >= 1 && i <= L1;
#pragma unroll
    for (int f = 0; f < NPF; ++f) x.v[f] = ld_poll_if(pin + f * (Lm + 1) + i, ok);
    if (GM == 1 && !ok) x.v[2] = __int_as_float(zero_frame<GM>() + frame_bias<GM>());
    return x;
  };
  // the state at the top of a segment whose chunks above were quiet
  auto store_zero = [&](int kq, float pt, int pn) {
    BState<R> z;
    bstate_zero<R, GM>(z);
    z.ht = lane == 31 ? pt : 0.f;
    z.hn = lane == 31 ? pn : zero_frame<GM>();
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
    ea.v[2] = __int_as_float(__float_as_int(ea.v[2]) - frame_bias<GM>());
    if (lquiet<R, GM>(bs, ckm, ea.v, lane, zlog, kc == ownc)) {
      zero_push<GM>(pout, Lm, L1, kc, lane);
      float pt = __shfl_sync(FULL, ea.v[1], C_STEPS - 1);
      int pn = __shfl_sync(FULL, __float_as_int(ea.v[2]), C_STEPS - 1);
      int kn = kc - 1;
      while (kn >= 0) {
        float r1;
        int rn;
        const int n = lquiet_run<GM>(pin, Lm, L1, ckmax, kn, 0, lane, pt, pn, zlog, ownc, r1, rn);
        for (int m = 0; m < n; ++m) {
          if ((kn - m + 1) % kSeg == 0) store_zero(kn - m, pt, pn);
          zero_push<GM>(pout, Lm, L1, kn - m, lane);
          pt = __shfl_sync(FULL, r1, m * C_STEPS + C_STEPS - 1);
          pn = __shfl_sync(FULL, rn, m * C_STEPS + C_STEPS - 1);
        }
        kn -= n;
        if (n < 32 / C_STEPS) break;
      }
      bstate_zero<R, GM>(bs);
      bs.ht = lane == 31 ? pt : 0.f;
      bs.hn = lane == 31 ? pn : zero_frame<GM>();
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
        lemit<R, DD, GM>(sb[S0 + cu], k, nlive, hd, xs, E);
        if constexpr (!IN) lblank<R>(act, xs, E);
        if constexpr (IN) rows.template fetch<VEC>(src, sb[S0 + cu]);
        else rows.load(src, i - cu - AH, sb[S0 + cu]);
        src -= rows.ld;
        int ft;
        float fB, vd0, mx;
        float2 vm[H], vi[H], sr[H], br[H];
        bcells<NS, R, DD, GM>(bs, rb, rn, GM == 1 ? i - cu == L1 : act, term, gO, gE, gX, nlive, hd, ft, fB, vm, vi, sr, br, vd0, mx);
        bfinish<R, GM>(bs, ft, mx, vm, vi, vd0, E, rt, rn);
        if (act && lane == 0 && pout) {
          pout[0 * (Lm + 1) + i - cu] = bs.ob;
          pout[1 * (Lm + 1) + i - cu] = bs.t[0].x;
          pout[2 * (Lm + 1) + i - cu] = __int_as_float(bs.nb + frame_bias<GM>());
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

template <int NS, int R, int GM = 0>
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
    const Place w = place_of<NS, R, GM>(a, task, true);
    if ((w.band + 1) * 32 * R > w.pr.L2 || !w.pr.vec)
      lbeta_band<NS, R, 1, GM>(a, lp, w, lane, deadline, s_push[threadIdx.x >> 5]);
    else
      lbeta_band<NS, R, 0, GM>(a, lp, w, lane, deadline, s_push[threadIdx.x >> 5]);
    __syncwarp();
  }
}

// The segments of every band (a.nseg per band): one warp each.
template <int NS, int R, bool SPARSE, int GM = 0>
__global__ void __launch_bounds__(32) lseg_kernel(Args a) {
  extern __shared__ float smem[];
  const int lane = threadIdx.x;
  const LParams lp = lparams<NS>(a);
  const int ntasks = a.B * a.nb * a.nseg;
  for (int task = blockIdx.x; task < ntasks; task += gridDim.x) {
    const int slot = task / a.nseg, seg = task - slot * a.nseg;
    const Place w = place_of<NS, R, GM>(a, slot, false);
    lbwd_band<NS, R, SPARSE, true, GM>(a, lp, w, lane, smem, 0, seg);
    lcp_wait_all();
    __syncwarp();
  }
}

// Pairs flagged for the log domain (GM 1 and 2): their completion counts to 0,
// their cross-band buffers to the sentinel; the task counters to 0.
template <int NS, int R, int GM>
__global__ void __launch_bounds__(128) redo_kernel(Args a) {
  if (blockIdx.x == 0 && threadIdx.x == 0) { a.counters[0] = 0u; a.counters[1] = 0u; }
  if (a.status[1] == 0u) return;
  const float none = __uint_as_float(SENTINEL_BITS);
  for (int p = blockIdx.x; p < a.B; p += gridDim.x) {
    const unsigned f = a.pair_done[p];
    __syncthreads();
    if (!(f & (PAIR_REDO | PAIR_LOST))) continue;
    if (threadIdx.x == 0) a.pair_done[p] = (f & PAIR_TIMEOUT) | PAIR_REDO;
    size_t ed0, bp0, ne, np;
    if (a.layout == 0) {
      ne = (size_t)a.nb * 2 * NS * a.Lmax1;
      np = (size_t)a.nb * push_fields<NS, GM>() * (a.Lmax1 + 1);
      ed0 = p * ne;
      bp0 = p * np;
    } else {
      const long long* q = a.plan_pairs + (size_t)p * PLAN_PAIR_WORDS;
      ne = (size_t)q[PW_NB] * 2 * NS * q[PW_L1];
      np = (size_t)q[PW_NB] * push_fields<NS, GM>() * (q[PW_L1] + 1);
      ed0 = (size_t)q[PW_EDGE0];
      bp0 = (size_t)q[PW_BP0];
    }
    for (size_t x = threadIdx.x; x < ne; x += blockDim.x) a.edge[ed0 + x] = none;
    for (size_t x = threadIdx.x; x < np; x += blockDim.x) a.bpush[bp0 + x] = none;
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
template <int NS, int R, int WARPS, bool SPARSE = false, int GM = 0>
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
    const Place w = place_of<NS, R, GM>(a, task, true);
    lbwd_band<NS, R, SPARSE, false, GM>(a, lp, w, lane, sm, deadline, 0);
  }
}

}  // namespace swb
