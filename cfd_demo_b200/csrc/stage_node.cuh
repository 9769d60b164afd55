// stage_node.cuh — the fused DG stage kernel with one thread per node, for
// meshes too small to fill the GPU with one or two threads per element.
//
// A half warp (16 lanes, 15 of them at work) is one element; a block of 128
// threads holds 8. Lane t owns node t of the volume term, face node t of the
// surface term and row t of [Dr|Ds] and LIFT, which it keeps in registers:
//   own node, neighbour trace, metric and table rows are requested together;
//   volume  (dg.py:148-151): the lane forms its node's contravariant fluxes,
//           publishes them to its half warp, and accumulates its row;
//   surface (dg.py:153-164): the lane evaluates its face node's interface flux,
//           publishes the lifted-jump input, and accumulates its LIFT row;
//   combine, averages, node tests: the lane's own node, with reductions over
//           the half warp.
// The values and their operation order are those of stage_tile.cuh, so results
// agree up to the multiply-adds the compiler contracts. (A [Dr|Ds] entry the FP32 form leaves out is a zero row
// entry here: adding 0 x F changes no finite value.)
//
// What bounds a small mesh is the length of one thread's instruction chain: two
// lanes per element leave 63 blocks of two warps on 148 SMs, 19.9 us a stage for
// 2,000 elements in FP64 (hllc); 15 chains of a fifteenth of the work each take
// 7.2 us. The node form issues more instructions in all, so it loses once the
// GPU is full: see launch_stage_default for where.
#pragma once
// Included by common.cuh inside namespace cfd.

// Table rows by lane, [column][lane]: coalesced loads, one row per lane.
template <typename R> struct NodeRows {
  R dr[NP][HALF], ds[NP][HALF], lift[3 * NFP][HALF];
};
template <typename R> constexpr NodeRows<R> make_node_rows() {
  NodeRows<R> t{};
  for (int j = 0; j < NP; ++j)
    for (int i = 0; i < NP; ++i) {
      t.dr[j][i] = keep_entry<R>(tab::DR[i][j]) ? (R)(-tab::DR[i][j]) : R(0);
      t.ds[j][i] = keep_entry<R>(tab::DS[i][j]) ? (R)(-tab::DS[i][j]) : R(0);
      t.lift[j][i] = (R)tab::LIFT[i][j];
    }
  return t;
}
static __device__ const NodeRows<double> NODE_ROWS64 = make_node_rows<double>();
static __device__ const NodeRows<float> NODE_ROWS32 = make_node_rows<float>();
template <typename R> __device__ __forceinline__ const NodeRows<R>& node_rows();
template <> __device__ __forceinline__ const NodeRows<double>& node_rows<double>() { return NODE_ROWS64; }
template <> __device__ __forceinline__ const NodeRows<float>& node_rows<float>() { return NODE_ROWS32; }

constexpr int NODE_BS = 128, NODE_EPB = NODE_BS / HALF;

template <typename R> struct __align__(16) NodeShared {
  R q[NP][4];   // nodal state (the face nodes read it)
  R ft[NP][4];  // contravariant fluxes; later the jumps, then the new state's weighted values
  R gt[NP][4];
};

template <typename R, int FLUX, int MODE>
__global__ void __launch_bounds__(NODE_BS) stage_node_kernel(const StageParams P) {
  __shared__ NodeShared<R> s_el[NODE_EPB];
  __shared__ double s_avg[NODE_EPB][4][NP];
  __shared__ unsigned long long s_key[3][NODE_EPB];
  __shared__ int s_fl[NODE_EPB];
  const CfdMesh& m = P.m;
  const int ld = m.ld;
  const int lane = threadIdx.x & 31, t = lane & (HALF - 1), base_lane = lane & HALF, hw = threadIdx.x / HALF;
  const unsigned hmask = 0xffffu << base_lane;
  const int e = blockIdx.x * NODE_EPB + hw;
  const int i = t < NP ? t : NP - 1;  // lane 15 repeats node 14
  const bool node_lane = t < NP;
  NodeShared<R>& sm = s_el[hw];
  bool live = e < m.num_elements;
  int inst = 0;
  if (m.instance) {
    inst = m.instance[blockIdx.x * NODE_EPB];  // instances start at multiples of 64: uniform in the block
    live = live && inst >= 0 && m.instance[e] == inst;
    inst = inst < 0 ? 0 : inst;
  }
  double b[4] = {0.0, 0.0, 0.0, 0.0};
  unsigned long long kr = KEY_EMPTY, kp = KEY_EMPTY, kd = KEY_EMPTY;
  int fl = 0;
  double dt = 0.0;
  int par = 0;
  bool active = true;
  if (MODE != MODE_RHS) {
    const CfdControl* ctl = P.ctl + inst;
    active = ctl->status == CFD_RUN_ACTIVE;
    dt = ctl->dt;
    par = ctl->parity;
  }
  if (live) {
    const R *src, *base;
    R* dst;
    if (MODE == MODE_RHS) {
      src = (const R*)P.q_in;
      base = nullptr;
      dst = (R*)P.q_out;
    } else {
      select_buffers<R>(P, par, src, base, dst);
    }
    // ---- requests: tables by element and lane, own node, base node
    const int finfo = m.face_info[e];
    const int f = i / NFP, k = i - NFP * f;
    const int nb = m.neighbor[f * ld + e];
    const R* __restrict__ mg = GeoPtr<R>::metric(m);
    const R* __restrict__ fg = GeoPtr<R>::face(m);
    const R rx = mg[e], ry = mg[ld + e], sx = mg[2 * ld + e], sy = mg[3 * ld + e];
    const R nx = fg[(3 * f) * ld + e], ny = fg[(3 * f + 1) * ld + e], fs = fg[(3 * f + 2) * ld + e];
    R q[4], bs[4] = {R(0), R(0), R(0), R(0)};
#pragma unroll
    for (int c = 0; c < 4; ++c) q[c] = src[(size_t)(c * NP + i) * ld + e];
    const bool has_base = MODE != MODE_RHS && P.stage_idx >= 2;
    if (has_base) {
#pragma unroll
      for (int c = 0; c < 4; ++c) bs[c] = base[(size_t)(c * NP + i) * ld + e];
    }
    const NodeRows<R>& rows = node_rows<R>();
    R dr[NP], ds[NP], lf[3 * NFP];
#pragma unroll
    for (int j = 0; j < NP; ++j) dr[j] = rows.dr[j][i], ds[j] = rows.ds[j][i], lf[j] = rows.lift[j][i];
    // ---- the neighbour's trace, needed after the volume term
    const int info = (finfo >> (8 * f)) & 0xff, kind = info & 3;
    R qp[4] = {R(1), R(0), R(0), R(1)};
    if (kind == CFD_FACE_INTERIOR) {
      const int nf = (info >> 2) & 3;
      const int pn = face_node_rt(nf, ((f == 2) != (nf == 2)) ? k : NFP - 1 - k);
#pragma unroll
      for (int c = 0; c < 4; ++c) qp[c] = src[(size_t)(c * NP + pn) * ld + nb];
    } else if (kind != CFD_FACE_SLIP_WALL) {
      // fixed state: one row per face; exact state: one row per face node
      const int row = nb + (kind == CFD_FACE_EXACT_STATE ? k : 0);
#pragma unroll
      for (int c = 0; c < 4; ++c) qp[c] = (R)m.bc_states[row * 4 + c];
    }
    if (MODE != MODE_RHS && !active) live = false;  // a finished instance (uniform in the block)
    if (live) {
      const R gamma = (R)P.gamma, gm1 = gamma - R(1);
      // ---- contravariant fluxes of the own node
      {
        const Prim<R> w = primitive(q, gm1);
        const R ep = q[3] + w.p;
        const R f0 = q[1], f1 = q[1] * w.u + w.p, f2 = q[2] * w.u, f3 = ep * w.u;
        const R g0 = q[2], g1 = q[1] * w.v, g2 = q[2] * w.v + w.p, g3 = ep * w.v;
        R ft[4], gt[4];
        lin_pair<R, true>(rx, ry, f0, f1, g0, g1, ft[0], ft[1]);
        lin_pair<R, true>(rx, ry, f2, f3, g2, g3, ft[2], ft[3]);
        lin_pair<R, true>(sx, sy, f0, f1, g0, g1, gt[0], gt[1]);
        lin_pair<R, true>(sx, sy, f2, f3, g2, g3, gt[2], gt[3]);
        if (sizeof(R) == 4) {  // FP32: differentiate the fluxes less those of node 0 (stage_tile.cuh)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            ft[c] -= __shfl_sync(hmask, ft[c], base_lane);
            gt[c] -= __shfl_sync(hmask, gt[c], base_lane);
          }
        }
        if (node_lane) {
#pragma unroll
          for (int c = 0; c < 4; ++c) sm.q[i][c] = q[c], sm.ft[i][c] = ft[c], sm.gt[i][c] = gt[c];
        }
      }
      __syncwarp(hmask);
      // ---- interface flux of the own face node
      R jump[4];
      {
        const int n = face_node_rt(f, k);
        R qm[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) qm[c] = sm.q[n][c];
        if (kind == CFD_FACE_SLIP_WALL) {  // dg.py:119-126
          const R mn = qm[1] * nx + qm[2] * ny;
          qp[0] = qm[0];
          qp[1] = qm[1] - R(2) * mn * nx;
          qp[2] = qm[2] - R(2) * mn * ny;
          qp[3] = qm[3];
        }
        R fhat[4], fm[4];
        trace_flux<R, FLUX>(qm, qp, nx, ny, gamma, fhat, fm);
        jump_pair<R, true>(fs, fm[0], fm[1], fhat[0], fhat[1], jump[0], jump[1]);
        jump_pair<R, true>(fs, fm[2], fm[3], fhat[2], fhat[3], jump[2], jump[3]);
        if (kind != CFD_FACE_INTERIOR && node_lane) {
          const double bw = ctab::FACE_W[k] * m.face_hlen[(size_t)f * ld + e];
#pragma unroll
          for (int c = 0; c < 4; ++c) b[c] = bw * (double)fhat[c];
        }
      }
      // ---- volume term: the own row of [Dr|Ds]
      R acc[4] = {R(0), R(0), R(0), R(0)};
#pragma unroll
      for (int j = sizeof(R) == 4 ? 1 : 0; j < NP; ++j) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          acc[c] = fma(dr[j], sm.ft[j][c], acc[c]);
          acc[c] = fma(ds[j], sm.gt[j][c], acc[c]);
        }
      }
      __syncwarp(hmask);
      if (node_lane) {
#pragma unroll
        for (int c = 0; c < 4; ++c) sm.ft[i][c] = jump[c];
      }
      __syncwarp(hmask);
      // ---- surface term: the own row of LIFT
#pragma unroll
      for (int j = 0; j < 3 * NFP; ++j) {
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] = fma(lf[j], sm.ft[j][c], acc[c]);
      }
      if (MODE == MODE_RHS) {
        if (node_lane) {
#pragma unroll
          for (int c = 0; c < 4; ++c) dst[(size_t)(c * NP + i) * ld + e] = acc[c];
        }
      } else {
        // ---- SSP-RK3 stage combine (time_integration.py:61-66)
        const R rdt = (R)dt;
        combine_pair<R, true>(P.stage_idx, rdt, q[0], q[1], bs[0], bs[1], acc[0], acc[1]);
        combine_pair<R, true>(P.stage_idx, rdt, q[2], q[3], bs[2], bs[3], acc[2], acc[3]);
        // ---- cell averages in double (FP64: NumPy order, sequential and unfused)
        if (node_lane) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            s_avg[hw][c][i] = sizeof(R) == 8 ? xmul(ctab::AVG_W[i], (double)acc[c]) : (double)acc[c];
        }
        __syncwarp(hmask);
        double a[4];
        {
          const double* col = s_avg[hw][t & 3];
          double s = sizeof(R) == 8 ? col[0] : xmul(tab::AVG_W[0], col[0]);
#pragma unroll
          for (int j = 1; j < NP; ++j) s = sizeof(R) == 8 ? xadd(s, col[j]) : fma(tab::AVG_W[j], col[j], s);
#pragma unroll
          for (int c = 0; c < 4; ++c) a[c] = __shfl_sync(hmask, s, base_lane + c);
          if (MODE == MODE_LIMITED && t < 4) P.avg[t * ld + e] = s;
        }
        const double gm1d = P.gamma - 1.0;
        const double pa = pressure_x(a[0], a[1], a[2], a[3], gm1d);
        const double eps = jmin(POSITIVITY_FLOOR, jmin(a[0], pa));
        const double pt = pressure_target<R>(eps, pa, a[3], gm1d);
        if (!(a[0] > 0.0) || !(pa > 0.0)) fl |= FLAG_BAD_AVERAGE;
        // ---- the own node's tests (stage_epilogue.inc)
        const bool want_lam = P.stage_idx == 3;
        double rmin = (double)acc[0], pmin, lam = -INFINITY;
        bool need, lam_nan = false;
        if (sizeof(R) == 4) {
          const float q0 = (float)acc[0], q1 = (float)acc[1], q2 = (float)acc[2], q3 = (float)acc[3];
          const float ir = rcp<float>(q0);
          const float u = q1 * ir, v = q2 * ir;
          const float kin = 0.5f * (q1 * u + q2 * v);
          float pf = (float)gm1d * (q3 - kin);
          const float margin = 1e-5f * (fabsf(q3) + fabsf(kin));
          bool low = false;
          if (!(pf - (float)pt > margin) && pf == pf) {
            const double px = pressure_x(q0, q1, q2, q3, gm1d);
            low = px < pt;
            pf = (float)px;
          }
          pmin = pf;
          if (want_lam) {
            const float pw = pf > 1e-4f * (fabsf(q3) + kin) ? pf : (float)pressure_x(q0, q1, q2, q3, gm1d);
            const float sp = sqrt_<float>(u * u + v * v) + sqrt_<float>((float)P.gamma * pw * ir);
            lam_nan = sp != sp;
            lam = sp;
          }
          need = low;
        } else {
          pmin = node_pressure<R>(acc[0], acc[1], acc[2], acc[3], gm1d, pt);
          need = pmin < pt;
          if (want_lam) {
            lam = wave_speed<R>(acc[0], acc[1], acc[2], acc[3], P.gamma);
            lam_nan = lam != lam;
          }
        }
        bool finite = finite_(acc[0]) && finite_(acc[1]) && finite_(acc[2]) && finite_(acc[3]);
        if (MODE == MODE_UNLIMITED && __any_sync(hmask, need || (double)acc[0] < eps)) {
          int node;
          double th;
          half_warp_positivity<R>(acc, a, eps, pt, gm1d, i, hmask, th, node);
          rmin = (double)acc[0];
          pmin = node_pressure<R>(acc[0], acc[1], acc[2], acc[3], gm1d, pt);
          finite = finite_(acc[0]) && finite_(acc[1]) && finite_(acc[2]) && finite_(acc[3]);
          if (want_lam) {
            lam = wave_speed<R>(acc[0], acc[1], acc[2], acc[3], P.gamma);
            lam_nan = lam != lam;
          }
        }
        // ---- stores and the element's reductions (NaN ignored in the minima, as fmin does)
        if (node_lane) {
#pragma unroll
          for (int c = 0; c < 4; ++c) dst[(size_t)(c * NP + i) * ld + e] = acc[c];
        }
        rmin = fmin(INFINITY, rmin);
        pmin = fmin(INFINITY, pmin);
#pragma unroll
        for (int o = 1; o < HALF; o <<= 1) {
          rmin = fmin(rmin, __shfl_xor_sync(hmask, rmin, o));
          pmin = fmin(pmin, __shfl_xor_sync(hmask, pmin, o));
        }
        if (!__all_sync(hmask, finite)) fl |= FLAG_NONFINITE;
        if (want_lam) {
          lam = fmax(-INFINITY, lam);
#pragma unroll
          for (int o = 1; o < HALF; o <<= 1) lam = fmax(lam, __shfl_xor_sync(hmask, lam, o));
          if (__any_sync(hmask, lam_nan)) lam = NAN;
        }
        if (t == 0) {
          if (MODE == MODE_LIMITED) {
            P.aux[e] = rmin;
            P.aux[ld + e] = pmin;
            if (want_lam) P.aux[2 * ld + e] = lam;
          } else {
            kr = dkey(rmin);
            kp = dkey(pmin);
            if (want_lam) {
              const double d = m.dt_geo[e] / lam;
              kd = dkey(d);
              if (d != d) fl |= FLAG_NAN_DT;
            }
          }
        }
      }
    }
  }
  // ---- commit: the boundary flux where the block has a boundary face, the
  // keys of the unlimited mode, and the flags
  if (MODE != MODE_RHS && t == 0) {
    s_fl[hw] = fl;
    if (MODE == MODE_UNLIMITED) s_key[0][hw] = kr, s_key[1][hw] = kp, s_key[2][hw] = kd;
  }
  const bool has_b = b[0] != 0.0 || b[1] != 0.0 || b[2] != 0.0 || b[3] != 0.0;
  __syncthreads();
  double* bsum = MODE == MODE_RHS ? P.bflux_out + inst * 4 : P.acc[3 * inst + (P.stage_idx > 0 ? P.stage_idx - 1 : 0)].boundary_flux;
  if (__any_sync(0xffffffffu, has_b)) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) b[c] += __shfl_xor_sync(0xffffffffu, b[c], o);
    }
    if (lane < 4) {
      const double v = lane == 0 ? b[0] : (lane == 1 ? b[1] : (lane == 2 ? b[2] : b[3]));
      if (v != 0.0) atomicAdd(&bsum[lane], v);
    }
  }
  if (MODE != MODE_RHS && threadIdx.x == 0) {
    Red r;
    r.init();
#pragma unroll
    for (int h = 0; h < NODE_EPB; ++h) {
      r.fl |= s_fl[h];
      if (MODE == MODE_UNLIMITED) {
        r.kr = min(r.kr, s_key[0][h]);
        r.kp = min(r.kp, s_key[1][h]);
        r.kd = min(r.kd, s_key[2][h]);
      }
    }
    if (MODE == MODE_UNLIMITED || r.fl) commit_one(r, P.acc + 3 * inst + (P.stage_idx - 1));
  }
}
