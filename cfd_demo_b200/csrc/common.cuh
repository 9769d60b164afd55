// common.cuh — device code shared by every object of libcfd_b200.so: the
// physics, reductions, positivity scaling and the fused stage kernels, plus the
// host templates that launch a stage kernel. The stage kernels' many template
// instantiations (precision x mode x flux x shape) are compiled in six objects
// (stage_inst.cu, one per precision and mode) beside kernels.cu, which holds
// the limiter, adjoint and small kernels and the C ABI.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <atomic>
#include <mutex>

#include "cfd_b200.h"
#include "physics.cuh"
#include "tables.cuh"

namespace cfd {

constexpr int NP = 15;
constexpr int NFP = 5;
constexpr double NEIGHBOR_FACTOR = 1.5;      // limiting.py:22
constexpr double DETECTION_TOLERANCE = 1e-10; // limiting.py:24
// FP32-mixed form: the troubled-cell test compares with ~100 single-precision
// ulps of the average (1e-10 lies far below the state's own round-off there)
constexpr double DETECTION_TOLERANCE_FP32 = 1e-5;
constexpr double POSITIVITY_FLOOR = 1e-13;    // limiting.py:28
constexpr int BISECTION_STEPS = 60;           // limiting.py:29

enum { MODE_RHS = 0, MODE_LIMITED = 1, MODE_UNLIMITED = 2 };
// bits 0-1 decide admissibility; bit 2 marks a NaN CFL step (time_step -> NaN)
enum { FLAG_NONFINITE = 1, FLAG_BAD_AVERAGE = 2, FLAG_NAN_DT = 4, FLAG_ADMISSIBILITY = 3 };

// ---------------------------------------------------------------- helpers ---
// Monotone map double -> uint64 so that unsigned integer order equals float order.
__device__ __forceinline__ unsigned long long dkey(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__host__ __device__ __forceinline__ double dkey_decode(unsigned long long k) {
  const unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  double d;
  memcpy(&d, &b, sizeof(d));
  return d;
}
constexpr unsigned long long KEY_EMPTY = ~0ull;

__device__ __forceinline__ bool finite_(double x) { return isfinite(x); }
__device__ __forceinline__ bool finite_(float x) { return isfinite(x); }

// Face node k of face f, packed 4 bits per entry (tab::FACE_NODES_PACKED).
constexpr unsigned long long FN_PACK = tab::FACE_NODES_PACKED;

// FP32 form: skip the [Dr|Ds] entries that are round-off zeros of the
// construction (|D| < 1e-13: 65 of 225 per matrix). The FP64 form keeps all (but
// for stage_quad.cuh).
template <typename R> __host__ __device__ constexpr bool keep_entry(double v) {
  return sizeof(R) == 8 ? true : (v > 1e-13 || v < -1e-13);
}
__device__ __forceinline__ int face_node_rt(int f, int k) { return (int)((FN_PACK >> (4 * (f * NFP + k))) & 15ull); }


template <typename R> struct GeoPtr;
template <> struct GeoPtr<double> {
  static __device__ __forceinline__ const double* metric(const CfdMesh& m) { return m.metric; }
  static __device__ __forceinline__ const double* face(const CfdMesh& m) { return m.face_geo; }
  static __device__ __forceinline__ const double* cs(const CfdMesh& m) { return m.cs_coef; }
};
template <> struct GeoPtr<float> {
  static __device__ __forceinline__ const float* metric(const CfdMesh& m) { return m.metric32; }
  static __device__ __forceinline__ const float* face(const CfdMesh& m) { return m.face_geo32; }
  static __device__ __forceinline__ const float* cs(const CfdMesh& m) { return m.cs_coef32; }
};

// Per-thread contribution to the per-instance stage reductions.
struct Red {
  double b[4];
  unsigned long long kr, kp, kd;
  int tr, fl;
  __device__ void init() {
    b[0] = b[1] = b[2] = b[3] = 0.0;
    kr = kp = kd = KEY_EMPTY;
    tr = 0;
    fl = 0;
  }
  __device__ void merge(const Red& r) {
#pragma unroll
    for (int c = 0; c < 4; ++c) b[c] += r.b[c];
    kr = min(kr, r.kr);
    kp = min(kp, r.kp);
    kd = min(kd, r.kd);
    tr += r.tr;
    fl |= r.fl;
  }
};

// Appends e to list[] where flag is set, with one atomic per warp on the
// shared counter (when a large share of the elements is listed, per-thread
// atomics on one address serialise), never past list[capacity - 1]. All 32 lanes
// of the warp must call it.
__device__ __forceinline__ void warp_list_append(int* list, int* count, bool flag, int e, int capacity = 0x7fffffff) {
  const unsigned mask = __ballot_sync(0xffffffffu, flag);
  if (!mask) return;
  const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(count, __popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  const unsigned at = base + __popc(mask & ((1u << lane) - 1u));
  if (flag && at < (unsigned)capacity) list[at] = e;
}

__device__ __forceinline__ void commit_one(const Red& r, CfdStageAcc* a) {
#pragma unroll
  for (int c = 0; c < 4; ++c)
    if (r.b[c] != 0.0) atomicAdd(&a->boundary_flux[c], r.b[c]);
  if (r.kr != KEY_EMPTY) atomicMin(&a->min_rho_key, r.kr);
  if (r.kp != KEY_EMPTY) atomicMin(&a->min_p_key, r.kp);
  if (r.kd != KEY_EMPTY) atomicMin(&a->dt_key, r.kd);
  if (r.tr) atomicAdd(&a->troubled, r.tr);
  if (r.fl) atomicOr(&a->flags, r.fl);
}

// Least key of the warp: the high words, then the low words of the lanes that
// hold the least high word (two 32-bit warp reductions).
__device__ __forceinline__ unsigned long long warp_min_key(unsigned long long k) {
  const unsigned hi = (unsigned)(k >> 32), h = __reduce_min_sync(0xffffffffu, hi);
  const unsigned l = __reduce_min_sync(0xffffffffu, hi == h ? (unsigned)k : 0xffffffffu);
  return ((unsigned long long)h << 32) | l;
}

// Block reduction and commit of the minima, the troubled count and the flags
// (no boundary flux) to one stage accumulator. All threads of the block call it.
__device__ __forceinline__ void commit_keys(const Red& r, CfdStageAcc* acc) {
  __shared__ unsigned long long s_key[3];
  __shared__ int s_sum[2];
  if (threadIdx.x < 3) s_key[threadIdx.x] = KEY_EMPTY;
  if (threadIdx.x < 2) s_sum[threadIdx.x] = 0;
  const unsigned long long kr = warp_min_key(r.kr), kp = warp_min_key(r.kp), kd = warp_min_key(r.kd);
  const int tr = __reduce_add_sync(0xffffffffu, r.tr), fl = __reduce_or_sync(0xffffffffu, (unsigned)r.fl);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&s_key[0], kr);
    atomicMin(&s_key[1], kp);
    atomicMin(&s_key[2], kd);
    if (tr) atomicAdd(&s_sum[0], tr);
    if (fl) atomicOr(&s_sum[1], fl);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    Red t;
    t.init();
    // The minima only fall, so a value that is not below the one read here (even
    // a stale one) cannot lower it: the atomic is left out. The limiter's many
    // short blocks commit to the same three words, where atomics serialise. (In a
    // stage kernel the read would only lengthen its block: 1.4 % of a step.)
    const volatile CfdStageAcc* seen = acc;
    const unsigned long long kr0 = seen->min_rho_key, kp0 = seen->min_p_key, kd0 = seen->dt_key;
    t.kr = s_key[0] < kr0 ? s_key[0] : KEY_EMPTY;
    t.kp = s_key[1] < kp0 ? s_key[1] : KEY_EMPTY;
    t.kd = s_key[2] < kd0 ? s_key[2] : KEY_EMPTY;
    t.tr = s_sum[0], t.fl = s_sum[1];
    commit_one(t, acc);
  }
}

// Reduce over the block and commit with one set of atomics when every live
// thread belongs to the same instance (else each thread commits its own).
// `slot(inst)` -> CfdStageAcc*. All threads of the block must call this.
template <int BS>
__device__ __forceinline__ void block_commit(Red r, bool live, int inst, CfdStageAcc* acc, int stride, int offset) {
  __shared__ int s_inst;
  __shared__ double s_b[BS / 32][4];
  __shared__ unsigned long long s_k[BS / 32][3];
  __shared__ int s_i[BS / 32][2];
  if (threadIdx.x == 0) s_inst = live ? inst : -1;
  __syncthreads();
  const int inst0 = s_inst;
  const bool uniform = __syncthreads_and(!live || inst == inst0) && inst0 >= 0;
  if (!uniform) {
    if (live) commit_one(r, acc + inst * stride + offset);
    return;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int c = 0; c < 4; ++c) r.b[c] += __shfl_xor_sync(0xffffffffu, r.b[c], o);
    r.kr = min(r.kr, __shfl_xor_sync(0xffffffffu, r.kr, o));
    r.kp = min(r.kp, __shfl_xor_sync(0xffffffffu, r.kp, o));
    r.kd = min(r.kd, __shfl_xor_sync(0xffffffffu, r.kd, o));
    r.tr += __shfl_xor_sync(0xffffffffu, r.tr, o);
    r.fl |= __shfl_xor_sync(0xffffffffu, r.fl, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
#pragma unroll
    for (int c = 0; c < 4; ++c) s_b[w][c] = r.b[c];
    s_k[w][0] = r.kr;
    s_k[w][1] = r.kp;
    s_k[w][2] = r.kd;
    s_i[w][0] = r.tr;
    s_i[w][1] = r.fl;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    Red t;
    t.init();
    for (int i = 0; i < BS / 32; ++i) {
      for (int c = 0; c < 4; ++c) t.b[c] += s_b[i][c];
      t.kr = min(t.kr, s_k[i][0]);
      t.kp = min(t.kp, s_k[i][1]);
      t.kd = min(t.kd, s_k[i][2]);
      t.tr += s_i[i][0];
      t.fl |= s_i[i][1];
    }
    commit_one(t, acc + inst0 * stride + offset);
  }
}

// Pressure in double of a (possibly float) state: fast form (reciprocal,
// contracted) and the reference's exact operation order (euler.py:21-27).
__device__ __forceinline__ double pressure_d(double q0, double q1, double q2, double q3, double gm1) {
  const double ir = __drcp_rn(q0);
  return gm1 * (q3 - 0.5 * (q1 * (q1 * ir) + q2 * (q2 * ir)));
}
__device__ __forceinline__ double pressure_x(double q0, double q1, double q2, double q3, double gm1) {
  return xmul(gm1, xsub(q3, xmul(0.5, xadd(xmul(q1, xdiv(q1, q0)), xmul(q2, xdiv(q2, q0))))));
}
// The fast form, replaced by the exact one wherever the two could fall on
// different sides of `bound` (they differ by a few ulps of |E| + |m.u|).
__device__ __forceinline__ double pressure_near(double q0, double q1, double q2, double q3, double gm1, double bound) {
  const double ir = __drcp_rn(q0);
  const double k = 0.5 * (q1 * (q1 * ir) + q2 * (q2 * ir));
  const double p = gm1 * (q3 - k);
  const double margin = 1e-13 * (fabs(q3) + fabs(k)) + 1e-300;
  return (p - bound > margin || p != p) ? p : pressure_x(q0, q1, q2, q3, gm1);
}

// Constant-bank operator tables in the arithmetic type (warp-uniform index).
template <typename R> struct tabv;
template <> struct tabv<double> {
  static __device__ __forceinline__ double dr(int i, int j) { return ctab::DR[i][j]; }
  static __device__ __forceinline__ double ds(int i, int j) { return ctab::DS[i][j]; }
  static __device__ __forceinline__ double lift(int i, int j) { return ctab::LIFT[i][j]; }
};
template <> struct tabv<float> {
  static __device__ __forceinline__ float dr(int i, int j) { return ctab::DR32[i][j]; }
  static __device__ __forceinline__ float ds(int i, int j) { return ctab::DS32[i][j]; }
  static __device__ __forceinline__ float lift(int i, int j) { return ctab::LIFT32[i][j]; }
};

// |u| + c of a node (time_integration.py:39-40). The plain form follows the
// reference's operation order exactly (divisions, unfused), so the CFL step
// of a given state is the reference's to the last bit.
template <typename R>
__device__ __forceinline__ double wave_speed(R q0, R q1, R q2, R q3, double gamma) {
  if (sizeof(R) == 8) {
    const double u = xdiv(q1, q0), v = xdiv(q2, q0);
    const double p = xmul(gamma - 1.0, xsub(q3, xmul(0.5, xadd(xmul(q1, u), xmul(q2, v)))));
    return xadd(__dsqrt_rn(xadd(xmul(u, u), xmul(v, v))), __dsqrt_rn(xdiv(xmul(gamma, p), q0)));
  }
  // FP32 form: single precision, except that a pressure lost to cancellation
  // (near vacuum) is recovered in double before the sound speed is taken
  const float ir = rcp<float>((float)q0);
  const float u = (float)q1 * ir, v = (float)q2 * ir;
  const float kin = 0.5f * ((float)q1 * u + (float)q2 * v);
  float p = (float)(gamma - 1.0) * ((float)q3 - kin);
  if (!(p > 1e-4f * (fabsf((float)q3) + kin)))
    p = (float)pressure_x((double)q0, (double)q1, (double)q2, (double)q3, gamma - 1.0);
  return (double)(sqrt_<float>(u * u + v * v) + sqrt_<float>((float)gamma * p * ir));
}

// Exact-order pressure of a node for the positivity test and the minima:
// the fast form unless it lies within rounding of `bound`.
template <typename R>
__device__ __forceinline__ double node_pressure(R q0, R q1, R q2, R q3, double gm1, double bound) {
  if (sizeof(R) == 8) return pressure_near(q0, q1, q2, q3, gm1, bound);
  const float ir = __frcp_rn((float)q0);
  const float k = 0.5f * ((float)q1 * ((float)q1 * ir) + (float)q2 * ((float)q2 * ir));
  const float p = (float)gm1 * ((float)q3 - k);
  const float margin = 1e-5f * (fabsf((float)q3) + fabsf(k));
  return ((double)p - bound > (double)margin || p != p) ? (double)p : pressure_x(q0, q1, q2, q3, gm1);
}

// Pressure target of the positivity limiter: the reference's eps
// (limiting.py:173-176) in the plain form; in the FP32-mixed form eps plus a
// margin covering the rounding of the repaired state to single precision
// (|dp| <= ~2e-7 (gamma-1) |E|), capped at half the average pressure so that
// the average itself stays admissible.
template <typename R>
__device__ __forceinline__ double pressure_target(double eps, double pa, double e_avg, double gm1) {
  if (sizeof(R) == 8) return eps;
  return eps + jmin(2e-6 * gm1 * fabs(e_avg), 0.5 * pa);
}

// Cell average in double, sequential and unfused like NumPy's einsum
// (limiting.py:209, dg.py:168-171).
template <typename R>
__device__ __forceinline__ void cell_average(const R (&q)[NP][4], double a[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    double s = xmul(tab::AVG_W[0], (double)q[0][c]);
#pragma unroll
    for (int i = 1; i < NP; ++i) s = xadd(s, xmul(tab::AVG_W[i], (double)q[i][c]));
    a[c] = s;
  }
}

// Root of the pressure scaling by bisection (limiting.py:183-200): the lower
// end after BISECTION_STEPS halvings of [0, 1] on pressure(a + theta d) >= pt,
// bit for bit, without evaluating the halvings whose outcome is certain.
//
// With positive density at both ends the pressure is concave along the
// segment, so if it exceeds pt by more than the evaluation's rounding at 0 and
// at lo_k, it does so on all of [0, lo_k]; and if it lies below pt by more
// than that at hi_k, it does so on all of [hi_k, 1]. The first k halvings then
// all have the outcome that leads to [lo_k, hi_k], a dyadic interval around
// the root of the quadratic rho (E - pt / (gamma - 1)) - |m|^2 / 2 (every
// midpoint down to 2^-48 is exact). `delta` bounds the rounding of p at any
// point of the segment: the points' own rounding and some ten operations, each
// relative 2^-53, through the pressure's sensitivity to rho, m and E, with the
// velocities bounded by their end values (they are monotone along the
// segment): 5 units, taken twice (the check's own value and the certain one)
// and rounded up to 16. Where a check fails the interval is widened, and in the
// end the loop runs from [0, 1] as written. The remaining halvings go two at a
// time, their three candidate points evaluated together (the loop is one
// serial chain of divisions, 125 cycles each), and end once lo and hi are
// neighbours: the midpoint then rounds to one of them, both known.
__device__ __forceinline__ double pressure_theta(const double a[4], double d0, double d1, double d2, double d3,
                                                 double gm1, double pt) {
  auto at = [&](double th) {
    return pressure_x(xadd(a[0], xmul(th, d0)), xadd(a[1], xmul(th, d1)), xadd(a[2], xmul(th, d2)),
                      xadd(a[3], xmul(th, d3)), gm1);
  };
  double lo = 0.0, hi = 1.0;
  int it = 0;
  const double e0 = a[0] + d0;
  if (a[0] > 0.0 && e0 > 0.0) {
    const double t = a[3] - pt / gm1;
    const double qa = d0 * d3 - 0.5 * (d1 * d1 + d2 * d2), qb = a[0] * d3 + d0 * t - (a[1] * d1 + a[2] * d2);
    const double qc = a[0] * t - 0.5 * (a[1] * a[1] + a[2] * a[2]);
    const double s = sqrt(qb * qb - 4.0 * qa * qc);
    const double root = qb < 0.0 ? 2.0 * qc / (s - qb) : -0.5 * (qb + s) / qa;
    const double ia = 1.0 / a[0], ie = 1.0 / e0;
    const double u = fmax(fabs(a[1] * ia), fabs((a[1] + d1) * ie)), v = fmax(fabs(a[2] * ia), fabs((a[2] + d2) * ie));
    const double delta = 16.0 * 1.1102230246251565e-16 * gm1 *
                         (fabs(a[3]) + fabs(d3) + u * (fabs(a[1]) + fabs(d1)) + v * (fabs(a[2]) + fabs(d2)) +
                          (u * u + v * v) * (fabs(a[0]) + fabs(d0)));
    // 2^-k about 8 delta / |dp/dtheta| at the root, where |d(quadratic)/dtheta| = s
    const double w = 8.0 * delta * (a[0] + root * d0) / (gm1 * s);
    if (root >= 0.0 && root < 1.0 && w > 0.0 && w < 0.0625 && at(0.0) - pt > delta) {
      int k = min(48, -1 - ilogb(w)) & ~1;
#pragma unroll 1
      for (; k >= 4; k -= 4) {
        const double n = ldexp(1.0, k), h = ldexp(1.0, -k);
        const double l = floor(root * n) * h, r = l + h;
        if (r <= 1.0 && (l == 0.0 || at(l) - pt > delta) && pt - at(r) > delta) {
          lo = l;
          hi = r;
          it = k;
          break;
        }
      }
    }
  }
#pragma unroll 1
  for (; it < BISECTION_STEPS; it += 2) {
    const double mid = xmul(0.5, xadd(lo, hi));
    if ((mid == lo || mid == hi) && lo > 0.0 && hi < 1.0) break;
    const double ml = xmul(0.5, xadd(lo, mid)), mr = xmul(0.5, xadd(mid, hi));
    const bool ok = at(mid) >= pt, okl = at(ml) >= pt, okr = at(mr) >= pt;
    const double l = ok ? (okr ? mr : mid) : (okl ? ml : lo);
    hi = ok ? (okr ? hi : mr) : (okl ? mid : ml);
    lo = l;
  }
  return lo;
}

// One face node of the surface term: exterior state, interface flux, lifted
// jump, boundary-flux contribution (dg.py:153-164, boundary: dg.py:119-137).
template <typename R, int FLUX>
__device__ __forceinline__ void face_node_flux(const CfdMesh& m, const R* __restrict__ src, int e, int ld, R gamma,
                                               int n, int kind, int nb, int pn, R nx, R ny, R fs, double bw,
                                               R jump[4], Red& red) {
  R qm[4], qp[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) qm[c] = src[(c * NP + n) * ld + e];
  if (kind == CFD_FACE_INTERIOR) {
#pragma unroll
    for (int c = 0; c < 4; ++c) qp[c] = src[(c * NP + pn) * ld + nb];
  } else if (kind == CFD_FACE_SLIP_WALL) {
    const R mn = qm[1] * nx + qm[2] * ny;
    qp[0] = qm[0];
    qp[1] = qm[1] - R(2) * mn * nx;
    qp[2] = qm[2] - R(2) * mn * ny;
    qp[3] = qm[3];
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c) qp[c] = (R)m.bc_states[nb * 4 + c];
  }
  R fhat[4], fm[4];
  trace_flux<R, FLUX>(qm, qp, nx, ny, gamma, fhat, fm);
#pragma unroll
  for (int c = 0; c < 4; ++c) jump[c] = fs * (fm[c] - fhat[c]);
  if (kind != CFD_FACE_INTERIOR) {
#pragma unroll
    for (int c = 0; c < 4; ++c) red.b[c] += bw * (double)fhat[c];
  }
}

// ----------------------------------------------------------- stage kernel ---
struct StageParams {
  CfdMesh m;
  const CfdControl* ctl;
  const void* x0;
  const void* x1;
  void* stage;
  int stage_idx;  // 1..3; 0 = rhs only
  double gamma;
  double* avg;
  double* aux;
  CfdStageAcc* acc;
  const void* q_in;  // MODE_RHS
  void* q_out;       // MODE_RHS
  double* bflux_out; // MODE_RHS, [instances][4]
  void* tape_src;    // optional: copy of the stage input written here (tiled kernels only)
  void* tape_dst;    // optional: second copy of the stage result (before limiting)
};

template <typename R>
__device__ __forceinline__ void select_buffers(const StageParams& P, int par, const R*& src, const R*& base, R*& dst) {
  const R* cur = (const R*)(par ? P.x1 : P.x0);
  R* nxt = (R*)(par ? P.x0 : P.x1);
  if (P.stage_idx == 1) {
    src = cur;
    base = nullptr;
    dst = nxt;
  } else if (P.stage_idx == 2) {
    src = nxt;
    base = cur;
    dst = (R*)P.stage;
  } else {
    src = (const R*)P.stage;
    base = cur;
    dst = nxt;
  }
}

// SSP-RK3 third stage q = q_n / 3 + 2 (q_2 + dt L(q_2)) / 3 with v = q_2 +
// dt L(q_2) (time_integration.py:64-66). The plain form evaluates it as the
// reference does. In single precision float(1/3) + float(2/3) = 1 + 3e-8,
// which would scale the whole state by that factor every step (a steady
// drift of mass and energy), so the FP32 form uses q_n + (2/3)(v - q_n),
// whose weights sum to one exactly.
template <typename R>
__device__ __forceinline__ R stage3_combine(R b, R v) {
  if (sizeof(R) == 8) return b * (R)(1.0 / 3.0) + (R)(2.0 / 3.0) * v;
  return fma((R)(2.0 / 3.0), v - b, b);
}

#include "stage_pair.cuh"
#include "stage_tile.cuh"
#include "limiter.cuh"
#include "stage_node.cuh"
#include "stage_quad.cuh"
#include "control.cuh"
#include "batch.cuh"

inline unsigned blocks_for(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// Records `msg` as the calling thread's last error (cfd_last_error) and
// returns `code`; defined in kernels.cu.
int cfd_fail(int code, const char* msg);

// ---------------------------------------------------- stage-kernel launches ---
// The differentiable step's shape behind variant 0, at every size: tiles of 32.
// Its gradient takes the branch of |u.n| and of the limiter that round-off picks
// where a region is uniform, so a kernel that rounds differently would change
// the gradient there (1.9e-4 of its norm on a shock tube), not its last bits.
constexpr int SHAPE_TILE32 = -1;
template <typename R, int FLUX, int MODE>
void launch_stage_bs(const StageParams& p, int bs, cudaStream_t st) {
  const unsigned g = blocks_for(p.m.num_elements, bs / 2);  // two threads per element
  if (bs == 64) stage_pair_kernel<R, FLUX, MODE, 64><<<g, 64, 0, st>>>(p);
  else if (bs == 256) stage_pair_kernel<R, FLUX, MODE, 256><<<g, 256, 0, st>>>(p);
  else stage_pair_kernel<R, FLUX, MODE, 128><<<g, 128, 0, st>>>(p);
}
// Whether a form that copies epb elements of every row by 16 bytes at a time may
// serve these buffers: the last block's columns end inside the leading dimension,
// and every row starts at a multiple of 16 bytes (ld a multiple of 4, for the
// int and float rows). Any ld >= num_elements is a valid mesh; the pair and node
// forms read element by element and take all of them.
inline bool staged_fits(const StageParams& p, int precision, int epb) {
  const CfdMesh& m = p.m;
  const bool f64 = precision == CFD_FP64;
  const void* rows[] = {p.q_in, p.x0, p.x1, p.stage, m.face_info, m.neighbor,
                        f64 ? (const void*)m.metric : (const void*)m.metric32,
                        f64 ? (const void*)m.face_geo : (const void*)m.face_geo32};
  for (const void* r : rows)
    if ((uintptr_t)r % 16) return false;
  return m.ld % 4 == 0 && ((long long)m.num_elements + epb - 1) / epb * epb <= m.ld;
}
// The shape that serves a call asking for `variant`: the pair kernel in place of
// a tiled shape that does not fit. (Variant 0 is settled in launch_stage_default.)
inline int staged_variant(const StageParams& p, int precision, int variant) {
  if (variant == 0 || variant == 2) return variant;
  const int epb = variant == 1 || variant == 4 || variant == SHAPE_TILE32 ? 32 : 64;
  return staged_fits(p, precision, epb) ? variant : 2;
}
template <typename R, int FLUX, int MODE, int EPB, bool SB, int MINB = (sizeof(R) == 4 ? 512 : 384) / (2 * EPB),
          bool UF = true, bool PK = true, bool CF = false, bool FJ = false, bool VR = false>
void launch_tile(const StageParams& p, cudaStream_t st) {
  using L = TileLayout<R, EPB, SB, FJ>;
  constexpr bool PACK = PK && sizeof(R) == 4;  // FP64 shares the unpacked instantiation
  constexpr bool CALL = CF && sizeof(R) == 4;
  // opt in to > 48 KB of dynamic shared memory, once per instantiation and
  // device (the attribute belongs to the device's context); setting it twice
  // is harmless, so concurrent first calls need no lock
  constexpr int MAX_DEV = 64;
  static bool configured[MAX_DEV] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= MAX_DEV || !configured[dev]) {
    cudaFuncSetAttribute(stage_tile_kernel<R, FLUX, MODE, EPB, SB, MINB, UF, PACK, CALL, FJ, VR>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES);
    if (dev >= 0 && dev < MAX_DEV) configured[dev] = true;
  }
  const unsigned g = blocks_for(p.m.num_elements, EPB);
  stage_tile_kernel<R, FLUX, MODE, EPB, SB, MINB, UF, PACK, CALL, FJ, VR><<<g, 2 * EPB, L::BYTES, st>>>(p);
}
template <int FLUX, int MODE>
void launch_quad(const StageParams& p, cudaStream_t st) {
  constexpr int BYTES = (int)sizeof(QuadShared) * (QUAD_BS / 32);
  constexpr int MAX_DEV = 64;  // the > 48 KB opt-in, once per instantiation and device (as launch_tile)
  static bool configured[MAX_DEV] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= MAX_DEV || !configured[dev]) {
    cudaFuncSetAttribute(stage_quad_kernel<FLUX, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, BYTES);
    if (dev >= 0 && dev < MAX_DEV) configured[dev] = true;
  }
  stage_quad_kernel<FLUX, MODE><<<blocks_for(p.m.num_elements, QUAD_EPB), QUAD_BS, BYTES, st>>>(p);
}
// Variant 0, by size. One thread per node on small meshes, and where the other
// forms' 16-byte copies do not fit the buffers (staged_fits); above, four lanes per
// element or tiles of 32 elements in FP64 and tiles of 32 in FP32-mixed. One RK3
// attempt (graph replay), us (larger meshes: stage_quad.cuh):
//   elements                  one thread per node   four lanes   tiles of 32   tiles of 64
//   2,000    FP64 / FP32            48 /  41             -         107 /  62     112 /  61
//   8,000    FP64 / FP32           102 /  70            98         105 /  71     105 /  67
//   32,000   FP64 / FP32           330 / 160           167         213 / 106     237 / 101
//   65,522   FP32                                                    112           111
//   125,000  FP32                                                    210           193
//   1.05 M   FP32                                                  1,428         1,286
// What decides in FP64 is waves of resident blocks. The node form holds 2,368
// elements a wave (two blocks of 8 an SM): its third wave ends at 7,104, and the
// fourth makes a stage slower than four lanes (7,938 elements, unlimited, Rusanov /
// Roe / HLLC: 71 / 73 / 81 us an attempt against 66 / 71 / 72); a bare right-hand
// side keeps it up to 8,000 (17 / 18 / 21 us a call against 21 / 22 / 23). Four
// lanes hold 18,944 elements a wave, tiles of 32 hold 23,680 and are the faster
// blocks with Rusanov and Roe fluxes, the slower ones with HLLC and where the last
// tile is ragged. Tiles of 32 over four lanes, time of an unlimited attempt / of a
// right-hand side (of a tube's, Roe, 8,200 and 12,500 elements: 1.12 and 1.16):
//   elements   divisible by 32      Rusanov        Roe           HLLC
//   12,000           yes          0.85 / 0.84   0.87 / 0.88   1.05 / 1.01
//   12,322           no           1.09 / 0.93   1.16 / 0.98   1.41 / 1.17
//   20,000           yes          0.77 / 0.79   0.80 / 0.82   0.89 / 0.87
//   20,402           no           0.93 / 0.86   0.98 / 0.95   1.12 / 1.06
//   24,000           yes          1.16 / 0.99   1.19 / 1.07   1.37 / 1.21
// In FP32-mixed the node form rounds as tiles of 32 do (but for a few sums in
// the limited stages); tiles of 64 with the flux as a call (shape 9) round more of
// them differently, which a run near the slope limiter's thresholds shows: they
// are taken from TILE64_MIN on where the limiter is `unlimited`, and left to the
// autotuner otherwise. A batch may be repacked into a smaller one and keeps its
// kernel then, because another would round differently: in FP64 every batch (flags
// bit 0) takes four lanes, in FP32-mixed a batch repacked from one above NODE_MAX
// (flags bit 1) stays with tiles of 32.
constexpr int NODE_MAX = CFD_NODE_MAX_ELEMENTS, TILE64_MIN = 100000;
constexpr int NODE_WAVE64 = 148 * 2 * NODE_EPB, QUAD_WAVE = 148 * 4 * QUAD_EPB, TILE32_WAVE64 = 148 * 5 * 32;
template <int FLUX, int MODE>
bool tile32_over_quad(int n) {
  if (n > TILE32_WAVE64) return false;
  if (FLUX == FLUX_HLLC) return n % 32 == 0 && n > QUAD_WAVE;
  return n % 32 == 0 || n > QUAD_WAVE || (MODE == MODE_RHS && FLUX == FLUX_RUSANOV);
}
template <typename R, int FLUX, int MODE>
void launch_stage_default(const StageParams& p, cudaStream_t st) {
  const int n = p.m.num_elements, precision = sizeof(R) == 8 ? CFD_FP64 : CFD_FP32_MIXED;
  const int node_max = sizeof(R) == 8 && MODE != MODE_RHS ? 3 * NODE_WAVE64 : NODE_MAX;
  const bool node = n <= node_max && !(p.m.flags & (sizeof(R) == 8 ? 3 : 2));
  if (node || !staged_fits(p, precision, 32))
    stage_node_kernel<R, FLUX, MODE><<<blocks_for(n, NODE_EPB), NODE_BS, 0, st>>>(p);
  else if constexpr (sizeof(R) == 8) {
    if (tile32_over_quad<FLUX, MODE>(n) && !(p.m.flags & 3)) launch_tile<R, FLUX, MODE, 32, false>(p, st);
    else launch_quad<FLUX, MODE>(p, st);
  } else if (MODE == MODE_UNLIMITED && n >= TILE64_MIN && !(p.m.flags & 1) && staged_fits(p, precision, 64))
    launch_tile<R, FLUX, MODE, 64, true, 4, true, true, true>(p, st);
  else launch_tile<R, FLUX, MODE, 32, false>(p, st);
}
static_assert(QUAD_EPB == 32, "launch_stage_default checks the fit of 32 elements a block");
template <typename R, int FLUX, int MODE>
void launch_stage_variant(const StageParams& p, int variant, int bs, cudaStream_t st) {
  if (variant == 2) launch_stage_bs<R, FLUX, MODE>(p, bs, st);
  else if (variant == 1) launch_tile<R, FLUX, MODE, 32, true>(p, st);
  else if (variant == 3) launch_tile<R, FLUX, MODE, 64, false>(p, st);
  else if (variant == 4) launch_tile<R, FLUX, MODE, 32, false, sizeof(R) == 4 ? 10 : 8>(p, st);
  else if (variant == 5) launch_tile<R, FLUX, MODE, 64, false, (sizeof(R) == 4 ? 512 : 384) / 128, false>(p, st);
  // 6 / 7: variants 3 / 5 with scalar FMAs in the contractions (the bitwise reference of the packed form)
  else if (variant == 6) launch_tile<R, FLUX, MODE, 64, false, (sizeof(R) == 4 ? 512 : 384) / 128, true, false>(p, st);
  else if (variant == 7) launch_tile<R, FLUX, MODE, 64, false, (sizeof(R) == 4 ? 512 : 384) / 128, false, false>(p, st);
  else if (variant == 8) launch_tile<R, FLUX, MODE, 64, true>(p, st);
  else if (variant == 9) launch_tile<R, FLUX, MODE, 64, true, (sizeof(R) == 4 ? 512 : 384) / 128, true, true, true>(p, st);
  // 10 / 11: the face-job form (each face's flux once for both sides), without / with staged base rows
  else if (variant == 10)
    launch_tile<R, FLUX, MODE, 64, false, (sizeof(R) == 4 ? 512 : 384) / 128, true, true, true, true>(p, st);
  else if (variant == 11) launch_tile<R, FLUX, MODE, 64, true, sizeof(R) == 4 ? 3 : 2, true, true, true, true>(p, st);
  // 12 / 13: variant 9 with the volume node loop kept rolled, with unrolled / rolled face rounds;
  // 14: variant 5 with the volume node loop kept rolled (smaller code)
  else if (variant == 12)
    launch_tile<R, FLUX, MODE, 64, true, (sizeof(R) == 4 ? 512 : 384) / 128, true, true, true, false, true>(p, st);
  else if (variant == 13)
    launch_tile<R, FLUX, MODE, 64, true, (sizeof(R) == 4 ? 512 : 384) / 128, false, true, true, false, true>(p, st);
  else if (variant == 14)
    launch_tile<R, FLUX, MODE, 64, false, (sizeof(R) == 4 ? 512 : 384) / 128, false, true, false, false, true>(p, st);
  else if (variant == SHAPE_TILE32) launch_tile<R, FLUX, MODE, 32, false>(p, st);
  else launch_stage_default<R, FLUX, MODE>(p, st);
}
// One precision and mode of the stage kernels, every flux and shape; each
// combination is instantiated in its own object (stage_inst.cu).
template <typename R, int MODE>
void launch_stage_part(const StageParams& p, int flux, int variant, int bs, cudaStream_t st) {
  if (flux == 0) launch_stage_variant<R, 0, MODE>(p, variant, bs, st);
  else if (flux == 1) launch_stage_variant<R, 1, MODE>(p, variant, bs, st);
  else launch_stage_variant<R, 2, MODE>(p, variant, bs, st);
}
#define CFD_DECLARE_STAGE_PART(R, MODE) \
  extern template void launch_stage_part<R, MODE>(const StageParams&, int, int, int, cudaStream_t);
CFD_DECLARE_STAGE_PART(double, MODE_RHS)
CFD_DECLARE_STAGE_PART(double, MODE_LIMITED)
CFD_DECLARE_STAGE_PART(double, MODE_UNLIMITED)
CFD_DECLARE_STAGE_PART(float, MODE_RHS)
CFD_DECLARE_STAGE_PART(float, MODE_LIMITED)
CFD_DECLARE_STAGE_PART(float, MODE_UNLIMITED)

}  // namespace cfd
