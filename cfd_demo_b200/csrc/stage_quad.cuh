// stage_quad.cuh — the fused DG stage kernel with four lanes per element, FP64.
//
// A warp is 8 elements, lane 8 c + s owning conserved variable c of element s:
// its 15 rows of the right-hand side stay in the lane's registers. What needs
// all four variables of a node is dealt out by node instead and passes through
// the warp's own shared memory, so that nothing is computed twice and the warps
// never wait for one another (__syncwarp only):
//   staging  own state and geometry rows (16-byte cp.async) and the neighbours'
//            face traces (one cp.async per value), which arrive under the
//            volume term, as the stage base rows do under the face fluxes;
//   volume   (dg.py:148-151): four rounds; in round r lane c forms the
//            contravariant fluxes of node 4 r + c, publishes them, and every
//            lane accumulates those of its variable at the round's four nodes;
//   surface  (dg.py:153-164): four rounds of face nodes 4 r + c (rolled: one
//            copy of the flux code), each replacing its staged trace by the
//            lifted-jump input; then 15 LIFT columns;
//   combine, average: the lane's variable; node tests: nodes 4 r + c again.
// Shared rows are padded to 8 words past a multiple of 32, which makes the
// accesses by node and by variable both free of bank conflicts. The values are
// the tiled kernel's (stage_tile.cuh) but for the round-off zeros of [Dr|Ds]
// (65 of 225 entries below 1e-13), which a stage leaves out: its result carries a
// non-finite node itself, and the step is rejected for it. A right-hand side is
// handed out as it is: there a sum of zero times every flux carries a non-finite
// one to all rows of its element, as the dense products of the reference do.
//
// What bounds it: instruction issue and the latency of double-precision chains and
// of shared memory (Roe, unlimited, 524,288 elements: the FP64 pipe is 43-45 % busy,
// 52-54 % of the issue slots, 16 warps an SM). Two lanes per element, each forming
// every node's primitives and flux, issue 512 / 527 / 581 warp instructions an
// element (stages 1 / 2 / 3); this form 449 / 474 / 537 (562 in the second before
// the tables were laid out for 16-byte constant loads and the density reciprocals
// were kept from the volume term). One thread per element issues 346 but has 8 warps
// an SM and ran no faster than the tiles. One RK3 attempt (graph replay), us:
//   elements                              tiles of 32   of 64   this form
//   32,000    hllc/van_leer                   213         237       167
//   65,522    roe/unlimited                   296         257       210
//   800,000   hllc/van_leer                 3,260       2,650     2,296
//   1,048,352 roe/unlimited                 3,080       2,890     2,547
#pragma once
// Included by common.cuh inside namespace cfd.

constexpr int QUAD_BS = 128, QUAD_EPW = 8, QUAD_EPB = QUAD_BS / 4;

struct __align__(16) QuadShared {  // of one warp
  using R = double;
  R q[4 * NP][QUAD_EPW];     // own state, row c * 15 + node
  R x[4][17][QUAD_EPW];      // exterior traces, then jumps, then the new state: [variable][face node or node]
  union {
    R f[8][5][QUAD_EPW];     // a round's contravariant fluxes, [F~ of 4, G~ of 4][node of the round]
    R base[4 * NP][QUAD_EPW];  // after the volume term: the stage base rows
  };
  R ir[NP + 1][QUAD_EPW];    // 1 / density of the nodes, for the face nodes' fluxes
  R geo[13][QUAD_EPW];       // rx ry sx sy, (nx ny fs) x 3
};

// The tables by column, one behind another, in the constant bank: read in this
// order two entries come with one 16-byte constant load. (Measured, per FMA:
// 1.7 more instructions with the entries as immediates, which a double operand
// cannot be, 1 with the row-major tables, 0.5 so.)
struct QuadColumns {
  double dr[NP][HALF], ds[NP][HALF], lift[3 * NFP][HALF];
};
constexpr QuadColumns make_quad_columns() {
  QuadColumns t{};
  for (int j = 0; j < NP; ++j)
    for (int i = 0; i < NP; ++i) t.dr[j][i] = -tab::DR[i][j], t.ds[j][i] = -tab::DS[i][j], t.lift[j][i] = tab::LIFT[i][j];
  return t;
}
static __constant__ __align__(16) QuadColumns QUAD_COLUMNS = make_quad_columns();

template <int FLUX, int MODE>
__global__ void __launch_bounds__(QUAD_BS, 4) stage_quad_kernel(const StageParams P) {
  using R = double;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double s_b[4];
  __shared__ unsigned long long s_key[3];
  __shared__ int s_fl;
  constexpr unsigned ALL = 0xffffffffu;
  constexpr int VEC = 16 / (int)sizeof(R);
  const CfdMesh& m = P.m;
  const int ld = m.ld, K = m.num_elements, tid = threadIdx.x, lane = tid & 31;
  const int c = lane >> 3, s = lane & 7;
  QuadShared& sm = reinterpret_cast<QuadShared*>(smem_raw)[tid >> 5];
  const int e0 = blockIdx.x * QUAD_EPB + (tid >> 5) * QUAD_EPW, e = e0 + s;
  // block-uniform instance (instances start at multiples of 64) and loop state
  const int inst = m.instance ? m.instance[blockIdx.x * QUAD_EPB] : 0;
  if (inst < 0) return;  // padding between instances
  double dt = 0.0;
  int par = 0;
  if (MODE != MODE_RHS) {
    const CfdControl* ctl = P.ctl + inst;
    if (ctl->status != CFD_RUN_ACTIVE) return;
    dt = ctl->dt;
    par = ctl->parity;
  }
  if (tid < 4) s_b[tid] = 0.0;
  if (tid < 3) s_key[tid] = KEY_EMPTY;
  if (tid == 0) s_fl = 0;
  __syncthreads();
  unsigned long long kr = KEY_EMPTY, kp = KEY_EMPTY, kd = KEY_EMPTY;
  int fl = 0;
  if (e0 < K) {  // (warp-uniform)
    const bool live = e < K && (m.instance == nullptr || m.instance[e] == inst);
    const R *src, *base;
    R* dst;
    if (MODE == MODE_RHS) {
      src = (const R*)P.q_in;
      base = nullptr;
      dst = (R*)P.q_out;
    } else {
      select_buffers<R>(P, par, src, base, dst);
    }
    const bool has_base = MODE != MODE_RHS && P.stage_idx >= 2;
    // ---- staging: own rows
    {
      constexpr int CPR = QUAD_EPW / VEC;
#pragma unroll
      for (int ch = 0; ch < (60 * CPR + 31) / 32; ++ch) {
        const int k = ch * 32 + lane, row = k / CPR, col = (k - row * CPR) * VEC;
        if (row < 60) cp_async16(&sm.q[row][col], src + (size_t)row * ld + e0 + col);
      }
      const R* __restrict__ mg = GeoPtr<R>::metric(m);
      const R* __restrict__ fg = GeoPtr<R>::face(m);
#pragma unroll
      for (int ch = 0; ch < (13 * CPR + 31) / 32; ++ch) {
        const int k = ch * 32 + lane, row = k / CPR, col = (k - row * CPR) * VEC;
        if (row < 13) cp_async16(&sm.geo[row][col], (row < 4 ? mg + (size_t)row * ld : fg + (size_t)(row - 4) * ld) + e0 + col);
      }
      cp_async_commit();
    }
    const int finfo = live ? m.face_info[e] : 0x010101;  // (a dead lane's faces are walls: no gather)
    int nb[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) nb[f] = m.neighbor[f * ld + e];
    // ---- exterior traces of face nodes 4 r + c
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int sl = 4 * r + c, f = sl / NFP, k = sl - NFP * f;
      const int n = f == 0 ? nb[0] : (f == 1 ? nb[1] : nb[2]);
      const int info = (finfo >> (8 * f)) & 0xff, kind = info & 3;
      if (sl < 3 * NFP && kind == CFD_FACE_INTERIOR) {
        const int nf = (info >> 2) & 3;
        const int pn = face_node_rt(nf, ((f == 2) != (nf == 2)) ? k : NFP - 1 - k);
        const R* p = src + (size_t)pn * ld + n;
#pragma unroll
        for (int v = 0; v < 4; ++v) cp_async_small<sizeof(R)>(&sm.x[v][sl][s], p + (size_t)(v * NP) * ld);
      } else if (sl < 3 * NFP && kind != CFD_FACE_SLIP_WALL) {
        // fixed state: one row per face; exact state: one row per face node
        const int row = n + (kind == CFD_FACE_EXACT_STATE ? k : 0);
#pragma unroll
        for (int v = 0; v < 4; ++v) sm.x[v][sl][s] = (R)m.bc_states[row * 4 + v];
      }
    }
    cp_async_commit();
    if (has_base) {  // the base rows are read in the combine: bring them into L2 now
#pragma unroll
      for (int k = 0; k < 2; ++k)
        if (2 * lane + k < 60) prefetch_l2(base + (size_t)(2 * lane + k) * ld + e0);
    }
    const R gamma = (R)P.gamma, gm1 = gamma - R(1);
    cp_async_wait<1>();
    __syncwarp();
    const R rx = sm.geo[0][s], ry = sm.geo[1][s], sx = sm.geo[2][s], sy = sm.geo[3][s];
    R acc[NP + 1], poison = R(0);
#pragma unroll
    for (int i = 0; i <= NP; ++i) acc[i] = R(0);
    // ---- volume term
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int j = 4 * r + c < NP ? 4 * r + c : NP - 1;
      R q[4], ft[4], gt[4];
#pragma unroll
      for (int v = 0; v < 4; ++v) q[v] = sm.q[v * NP + j][s];
      const Prim<R> w = primitive(q, gm1);
      sm.ir[4 * r + c][s] = w.inv_rho;
      const R ep = q[3] + w.p;
      const R fb = q[1] * w.u + w.p, fc = q[2] * w.u, fd = ep * w.u;
      const R gb = q[1] * w.v, gc = q[2] * w.v + w.p, gd = ep * w.v;
      lin_pair<R, false>(rx, ry, q[1], fb, q[2], gb, ft[0], ft[1]);
      lin_pair<R, false>(rx, ry, fc, fd, gc, gd, ft[2], ft[3]);
      lin_pair<R, false>(sx, sy, q[1], fb, q[2], gb, gt[0], gt[1]);
      lin_pair<R, false>(sx, sy, fc, fd, gc, gd, gt[2], gt[3]);
      if (r) __syncwarp();  // the last round's fluxes have been read
#pragma unroll
      for (int v = 0; v < 4; ++v) sm.f[v][c][s] = ft[v], sm.f[4 + v][c][s] = gt[v];
      __syncwarp();
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const int jj = 4 * r + l;
        if (jj >= NP) break;
        const R x = sm.f[c][l][s], y = sm.f[4 + c][l][s];
        if (MODE == MODE_RHS) poison = fma(R(0), x, fma(R(0), y, poison));
#pragma unroll
        for (int i = 0; i < NP; ++i)
          if (keep_entry<float>(tab::DR[i][jj])) acc[i] = fma(QUAD_COLUMNS.dr[jj][i], x, acc[i]);
#pragma unroll
        for (int i = 0; i < NP; ++i)
          if (keep_entry<float>(tab::DS[i][jj])) acc[i] = fma(QUAD_COLUMNS.ds[jj][i], y, acc[i]);
      }
    }
    cp_async_wait<0>();
    __syncwarp();
    if (has_base) {  // the base rows arrive under the face fluxes
      constexpr int CPR = QUAD_EPW / VEC;
#pragma unroll
      for (int ch = 0; ch < (60 * CPR + 31) / 32; ++ch) {
        const int k = ch * 32 + lane, row = k / CPR, col = (k - row * CPR) * VEC;
        if (row < 60) cp_async16(&sm.base[row][col], base + (size_t)row * ld + e0 + col);
      }
      cp_async_commit();
    }
    // ---- surface term: face node fluxes, one copy of the code
#pragma unroll 1
    for (int r = 0; r < 4; ++r) {
      const int sl = 4 * r + c;
      if (sl >= 3 * NFP) break;
      const int f = sl / NFP, k = sl - NFP * f;
      const int kind = (finfo >> (8 * f)) & 3;
      const R nx = sm.geo[4 + 3 * f][s], ny = sm.geo[5 + 3 * f][s], fs = sm.geo[6 + 3 * f][s];
      const int n = face_node_rt(f, k);
      R qm[4], qp[4];
#pragma unroll
      for (int v = 0; v < 4; ++v) qm[v] = sm.q[v * NP + n][s], qp[v] = sm.x[v][sl][s];
      if (kind == CFD_FACE_SLIP_WALL) {  // dg.py:119-126
        const R mn = qm[1] * nx + qm[2] * ny;
        qp[0] = qm[0];
        qp[1] = qm[1] - R(2) * mn * nx;
        qp[2] = qm[2] - R(2) * mn * ny;
        qp[3] = qm[3];
      }
      R fhat[4], fm[4], jump[4];
      interface_flux<R, FLUX>(qm, qp, primitive(qm, gm1, sm.ir[n][s]), nx, ny, gamma, fhat, fm);
      jump_pair<R, false>(fs, fm[0], fm[1], fhat[0], fhat[1], jump[0], jump[1]);
      jump_pair<R, false>(fs, fm[2], fm[3], fhat[2], fhat[3], jump[2], jump[3]);
      if (kind != CFD_FACE_INTERIOR && live) {
        const double bw = ctab::FACE_W[k] * m.face_hlen[(size_t)f * ld + e];
#pragma unroll
        for (int v = 0; v < 4; ++v) atomicAdd(&s_b[v], bw * (double)fhat[v]);
      }
#pragma unroll
      for (int v = 0; v < 4; ++v) sm.x[v][sl][s] = jump[v];
    }
    __syncwarp();
#pragma unroll
    for (int sl = 0; sl < 3 * NFP; ++sl) {
      const R x = sm.x[c][sl][s];
#pragma unroll
      for (int i = 0; i < NP; ++i) acc[i] = fma(QUAD_COLUMNS.lift[sl][i], x, acc[i]);
    }
    if (MODE == MODE_RHS) {
      if (live) {
#pragma unroll
        for (int i = 0; i < NP; ++i) dst[(size_t)(c * NP + i) * ld + e] = acc[i] + poison;
      }
    } else {
      // ---- SSP-RK3 stage combine (time_integration.py:61-66)
      const R rdt = (R)dt;
      cp_async_wait<0>();
      __syncwarp();
#pragma unroll
      for (int i = 0; i <= NP; i += 2) {
        const int row = c * NP + i, next = i + 1 < NP ? row + 1 : row;
        if (i >= NP) break;
        const R b0 = has_base ? sm.base[row][s] : R(0), b1 = has_base ? sm.base[next][s] : R(0);
        combine_pair<R, false>(P.stage_idx, rdt, sm.q[row][s], sm.q[next][s], b0, b1, acc[i], acc[i + 1]);
      }
      // ---- cell average of the own variable, NumPy order (sequential, unfused)
      double a[4];
      {
        double t = xmul(tab::AVG_W[0], acc[0]);
#pragma unroll
        for (int i = 1; i < NP; ++i)
          t = xadd(t, xmul(tab::AVG_W[i], acc[i]));
        if (MODE == MODE_LIMITED && live) P.avg[c * ld + e] = t;
#pragma unroll
        for (int v = 0; v < 4; ++v) a[v] = __shfl_sync(ALL, t, 8 * v + s);
      }
      const double gm1d = P.gamma - 1.0;
      const double pa = pressure_x(a[0], a[1], a[2], a[3], gm1d);
      const double eps = jmin(POSITIVITY_FLOOR, jmin(a[0], pa));
      const double pt = pressure_target<R>(eps, pa, a[3], gm1d);
      if (live && (!(a[0] > 0.0) || !(pa > 0.0))) fl |= FLAG_BAD_AVERAGE;
      // ---- the new state by node (the jumps have been read)
      __syncwarp();
#pragma unroll
      for (int i = 0; i < NP; ++i) sm.x[c][i][s] = acc[i];
      __syncwarp();
      const bool want_lam = P.stage_idx == 3;
      double rmin = INFINITY, pmin = INFINITY, lam = -INFINITY;
      bool finite = true, lam_nan = false, need_p = false, rho_nan = false;
#pragma unroll 1
      for (int r = 0; r < 4; ++r) {
        const int i = 4 * r + c < NP ? 4 * r + c : NP - 1;  // the last lane repeats node 14
        const R q0 = sm.x[0][i][s], q1 = sm.x[1][i][s], q2 = sm.x[2][i][s], q3 = sm.x[3][i][s];
        finite &= isfinite(q0) && isfinite(q1) && isfinite(q2) && isfinite(q3);
        rmin = fmin(rmin, (double)q0);
        rho_nan |= q0 != q0;
        const double p = node_pressure<R>(q0, q1, q2, q3, gm1d, pt);
        pmin = fmin(pmin, p);
        need_p |= p < pt;
        if (want_lam) {
          const double sp = wave_speed<R>(q0, q1, q2, q3, P.gamma);
          lam_nan |= sp != sp;
          lam = fmax(lam, sp);
        }
      }
      auto join = [&]() {  // the element's values from its four lanes
        unsigned bits = (finite ? 0u : 1u) | (need_p ? 2u : 0u) | (lam_nan ? 4u : 0u) | (rho_nan ? 8u : 0u);
#pragma unroll
        for (int o = 8; o <= 16; o <<= 1) {
          rmin = fmin(rmin, __shfl_xor_sync(ALL, rmin, o));
          pmin = fmin(pmin, __shfl_xor_sync(ALL, pmin, o));
          if (want_lam) lam = fmax(lam, __shfl_xor_sync(ALL, lam, o));
          bits |= __shfl_xor_sync(ALL, bits, o);
        }
        finite = !(bits & 1u), need_p = bits & 2u, lam_nan = bits & 4u, rho_nan = bits & 8u;
      };
      join();
      if (MODE == MODE_UNLIMITED) {
        const bool mine = live && ((!rho_nan && rmin < eps) || need_p);
        if (__any_sync(ALL, mine)) {
          // rare: Zhang-Shu scaling (limiting.py:166-200) of the flagged elements by their four lanes
          const double ac = c == 0 ? a[0] : (c == 1 ? a[1] : (c == 2 ? a[2] : a[3]));
          auto scale = [&](double th) {
#pragma unroll
            for (int i = 0; i < NP; ++i) {
              acc[i] = (R)xadd(ac, xmul(th, xsub((double)acc[i], ac)));
              sm.x[c][i][s] = acc[i];
            }
          };
          if (mine && !rho_nan && rmin < eps) scale(jmin(jmax(xdiv(xsub(a[0], eps), xsub(a[0], rmin)), 0.0), 1.0));
          __syncwarp();
          double th = 1.0;
          if (mine) {
#pragma unroll 1
            for (int i = c; i < NP; i += 4) {
              const double q0 = sm.x[0][i][s], q1 = sm.x[1][i][s], q2 = sm.x[2][i][s], q3 = sm.x[3][i][s];
              if (pressure_near(q0, q1, q2, q3, gm1d, pt) < pt)
                th = jmin(th, pressure_theta(a, xsub(q0, a[0]), xsub(q1, a[1]), xsub(q2, a[2]), xsub(q3, a[3]), gm1d, pt));
            }
          }
          __syncwarp();
          th = fmin(th, __shfl_xor_sync(ALL, th, 8));
          th = fmin(th, __shfl_xor_sync(ALL, th, 16));
          if (mine && th < 1.0) scale(th);
          __syncwarp();
          double rm = INFINITY, pm = INFINITY, lm = -INFINITY;
          bool fin = true, lnan = false;
#pragma unroll 1
          for (int i = c; i < NP; i += 4) {
            const R q0 = sm.x[0][i][s], q1 = sm.x[1][i][s], q2 = sm.x[2][i][s], q3 = sm.x[3][i][s];
            fin &= isfinite(q0) && isfinite(q1) && isfinite(q2) && isfinite(q3);
            rm = fmin(rm, (double)q0);
            pm = fmin(pm, node_pressure<R>(q0, q1, q2, q3, gm1d, pt));
            if (want_lam) {
              const double sp = wave_speed<R>(q0, q1, q2, q3, P.gamma);
              lnan |= sp != sp;
              lm = fmax(lm, sp);
            }
          }
          if (mine) rmin = rm, pmin = pm, lam = lm, finite = fin, lam_nan = lnan;
          join();
        }
      }
      if (lam_nan) lam = NAN;
      // ---- stores and the element's reductions
      if (live) {
#pragma unroll
        for (int i = 0; i < NP; ++i) dst[(size_t)(c * NP + i) * ld + e] = acc[i];
        if (!finite) fl |= FLAG_NONFINITE;
        if (MODE == MODE_LIMITED) {
          if (c < 2) P.aux[c * ld + e] = c == 0 ? rmin : pmin;
          else if (c == 2 && want_lam) P.aux[2 * ld + e] = lam;
        } else if (c == 0) {
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
  // ---- commit: one set of atomics per block
  if (MODE == MODE_UNLIMITED) {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {  // (lanes 0 .. 7 hold the keys)
      kr = min(kr, __shfl_xor_sync(ALL, kr, o));
      kp = min(kp, __shfl_xor_sync(ALL, kp, o));
      if (P.stage_idx == 3) kd = min(kd, __shfl_xor_sync(ALL, kd, o));
    }
    if (lane == 0) {
      atomicMin(&s_key[0], kr);
      atomicMin(&s_key[1], kp);
      atomicMin(&s_key[2], kd);
    }
  }
  if (MODE != MODE_RHS && fl) atomicOr(&s_fl, fl);
  __syncthreads();
  double* bsum = MODE == MODE_RHS ? P.bflux_out + inst * 4 : P.acc[3 * inst + P.stage_idx - 1].boundary_flux;
  if (tid < 4 && s_b[tid] != 0.0) atomicAdd(&bsum[tid], s_b[tid]);
  if (MODE != MODE_RHS && tid == 0) {
    Red r;
    r.init();
    r.fl = s_fl;
    if (MODE == MODE_UNLIMITED) r.kr = s_key[0], r.kp = s_key[1], r.kd = s_key[2];
    if (MODE == MODE_UNLIMITED || r.fl) commit_one(r, P.acc + 3 * inst + (P.stage_idx - 1));
  }
}
