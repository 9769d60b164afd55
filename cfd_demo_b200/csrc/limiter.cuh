// limiter.cuh — the Cockburn-Shu troubled-cell limiter and the Zhang-Shu
// positivity limiter of a stage state (limiting.py:136-216 of CFD-demo), as
// per-element bodies and the kernels that run them.
// Included by common.cuh inside namespace cfd.
#pragma once

// ----------------------------------------------------------- limit kernel ---
struct LimitParams {
  CfdMesh m;
  const CfdControl* ctl;  // null: always active (cfd_limit)
  const void* x0;
  const void* x1;
  void* stage;
  int stage_idx;          // 1..3, or 0 with q = q_io (cfd_limit)
  void* q_io;
  double gamma;
  const double* avg;
  const double* aux;
  CfdStageAcc* acc;       // stage mode
  int32_t* troubled_out;  // cfd_limit mode
  double* pos_out;        // optional [2][ld]: pressure-scaling theta and its critical node
  int* list;              // two launches: the elements to rewrite, and
  int* count;             // [2] their number and a count of blocks, zero before and after the pair
  uint8_t* flags;         // optional [ld]: troubled-cell indicator per element
};

// The stage state the limiter works on, in place.
template <typename R>
__device__ __forceinline__ R* limit_state(const LimitParams& P, int par) {
  return P.stage_idx == 0 ? (R*)P.q_io : P.stage_idx == 2 ? (R*)P.stage : (R*)(par ? P.x0 : P.x1);
}

// Reductions of an element the limiters leave as it is: the stage's minima
// and, in stage 3, its CFL step.
__device__ __forceinline__ void limit_keep(const LimitParams& P, int e, double rmin, double pmin, Red& red) {
  red.kr = dkey(rmin);
  red.kp = dkey(pmin);
  if (P.stage_idx == 3) {
    const double d = P.m.dt_geo[e] / P.aux[2 * P.m.ld + e];
    red.kd = dkey(d);
    if (d != d) red.fl |= FLAG_NAN_DT;
  }
}

constexpr int HALF = 16;  // lanes per element

// Zhang-Shu positivity scaling (limiting.py:166-200) of one element toward its
// average by a half warp, lane t holding node i = min(t, 14)'s values v: density
// scaling, then pressure scaling by the smallest theta of the nodes below the
// target pt. Returns that theta (1 where none is) and its node.
template <typename R>
__device__ __forceinline__ void half_warp_positivity(R (&v)[4], const double a[4], double eps, double pt, double gm1,
                                                     int i, unsigned hmask, double& th, int& node) {
  if (__any_sync(hmask, (double)v[0] < eps)) {
    double rmin = (double)v[0];
#pragma unroll
    for (int o = 1; o < HALF; o <<= 1) rmin = jmin(rmin, __shfl_xor_sync(hmask, rmin, o));
    if (rmin < eps) {  // (a NaN among the nodes leaves the element as it is)
      const double span = xsub(a[0], rmin);
      const double theta = jmin(jmax(xdiv(xsub(a[0], eps), span), 0.0), 1.0);
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = (R)xadd(a[k], xmul(theta, xsub((double)v[k], a[k])));
    }
  }
  const bool low = pressure_near(v[0], v[1], v[2], v[3], gm1, pt) < pt;
  th = 1.0;
  node = -1;
  if (__any_sync(hmask, low)) {
    if (low) {
      const double lo = pressure_theta(a, xsub((double)v[0], a[0]), xsub((double)v[1], a[1]),
                                       xsub((double)v[2], a[2]), xsub((double)v[3], a[3]), gm1, pt);
      if (lo < th) {
        th = lo;
        node = i;
      }
    }
    __syncwarp(hmask);
#pragma unroll
    for (int o = 1; o < HALF; o <<= 1) {
      const double oth = __shfl_xor_sync(hmask, th, o);
      const int onode = __shfl_xor_sync(hmask, node, o);
      if (oth < th || (oth == th && onode >= 0 && (node < 0 || onode < node))) {
        th = oth;
        node = onode;
      }
    }
    if (th < 1.0) {
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = (R)xadd(a[k], xmul(th, xsub((double)v[k], a[k])));
    }
  }
}

// The scan of one element: the troubled-cell test (limiting.py:128-151: the
// scaled neighbour differences from Cockburn-Shu coefficients and neighbour or
// ghost averages, and whether a density or energy trace at a face midpoint
// leaves its minmod bound) and the positivity test on the stage's nodal
// minima. An element the limiters leave as it is contributes its minima (and
// CFL step) to `red`; any other is `listed` for limit_half_warp. Writes the
// troubled flag where asked for.
//
// Bound by memory latency on large meshes (10 of 15 cycles between two
// instructions of a warp went to loads): every load but the neighbours'
// averages is therefore issued before the first value is used, the loop
// state's among them, so that an element takes two round trips.
template <typename R, int PHI>
__device__ __forceinline__ bool limit_scan_one(const LimitParams& P, int e, int inst, Red& red) {
  const CfdMesh& m = P.m;
  const int ld = m.ld;
  const volatile CfdControl* ctl = P.ctl ? P.ctl + inst : nullptr;
  const int status = ctl ? ctl->status : CFD_RUN_ACTIVE, par = ctl ? ctl->parity : 0;
  const double rmin0 = P.aux[e], pmin0 = P.aux[ld + e];
  double a[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) a[c] = P.avg[c * ld + e];
  int finfo = 0, nb[3] = {0, 0, 0};
  R co[6] = {}, tr[3][2] = {};
  if (PHI != LIM_UNLIMITED) {
    finfo = m.face_info[e];
    const R* __restrict__ cs = GeoPtr<R>::cs(m);
#pragma unroll
    for (int f = 0; f < 3; ++f) nb[f] = m.neighbor[f * ld + e];
#pragma unroll
    for (int k = 0; k < 6; ++k) co[k] = cs[k * ld + e];
    const R* __restrict__ q = limit_state<R>(P, par);
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
      for (int k = 0; k < 2; ++k) tr[f][k] = q[(3 * k * NP + tab::MID_NODES[f]) * ld + e];
  }
  if (status != CFD_RUN_ACTIVE) return false;
  bool troubled = false;
  if (PHI != LIM_UNLIMITED) {
    R diff[3][2];  // density and energy: the detection components
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const int kind = (finfo >> (8 * f)) & 3;
      double na[2];
      if (kind == CFD_FACE_INTERIOR) {
        na[0] = P.avg[nb[f]];
        na[1] = P.avg[3 * ld + nb[f]];
      } else if (kind == CFD_FACE_SLIP_WALL) {  // the mirror keeps both
        na[0] = a[0];
        na[1] = a[3];
      } else {
        // the ghost average: the fixed state, or the exact state's row after its node rows
        const int row = nb[f] + (kind == CFD_FACE_EXACT_STATE ? NFP : 0);
        na[0] = m.bc_states[row * 4];
        na[1] = m.bc_states[row * 4 + 3];
      }
      diff[f][0] = (R)xsub(na[0], a[0]);
      diff[f][1] = (R)xsub(na[1], a[3]);
    }
    const double det_tol = sizeof(R) == 8 ? DETECTION_TOLERANCE : DETECTION_TOLERANCE_FP32;
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      const int pf = (finfo >> (8 * f + 4)) & 3;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const double ac = k == 0 ? a[0] : a[3];
        const R pd = pf == 0 ? diff[0][k] : (pf == 1 ? diff[1][k] : diff[2][k]);
        const R sc = xmul((R)NEIGHBOR_FACTOR, xadd(xmul(co[f], diff[f][k]), xmul(co[3 + f], pd)));
        const R t = xsub(tr[f][k], (R)ac);
        troubled |= (double)abs_(xsub(minmod2(t, sc), t)) > xmul(det_tol, fabs(ac));
      }
    }
  }
  if (P.flags) P.flags[e] = troubled ? 1 : 0;
  const double gm1 = P.gamma - 1.0;
  const double pa = pressure_x(a[0], a[1], a[2], a[3], gm1);
  const double eps = jmin(POSITIVITY_FLOOR, jmin(a[0], pa));
  const double pt = pressure_target<R>(eps, pa, a[3], gm1);
  if (troubled || rmin0 < eps || pmin0 < pt) return true;
  limit_keep(P, e, rmin0, pmin0, red);
  return false;
}

// The limiters on element e by the sixteen lanes of a half warp: troubled-cell
// test, reconstruction (limiting.py:136-163) and positivity scaling
// (limiting.py:166-200), in place on the stage state. Every value is formed in
// NumPy's operation order, whichever lane forms it:
//   lane t < 12 owns (face f = t / 4, variable c = t % 4): the scaled
//     neighbour difference, its test, the P1 midpoint value (one sequential sum
//     over the nodes) and its limited delta;
//   lane t < 15 owns node t: the rebuilt state, the positivity scalings, the
//     bisection of its pressure and its statistics (lane 15 repeats node 14).
// Theta and its critical node (the smallest index attaining the minimum, as a
// sequential loop finds it) are order-independent reductions over the lanes;
// each lane's `red` takes its own node.
//
// What bounds this pass is the serial chain of one element, not the count of
// elements: on a shock tube a few hundred of them are rewritten per stage. With
// four lanes an element, one variable each, the node tests and statistics ran
// one node after the other in the warp (15 double divisions, reciprocals and
// square roots in a row): 18.5 us for the 2,000-element tube and 77 us for a
// 40,000-element channel in FP64, at 15 % of the issue slots; a lane per node
// does them at once.
template <typename R> struct LimitShared {
  R v[NP * 4];  // the element's nodal values, [node][variable]
  R d[12];      // limited deltas, [face][variable]
};

template <typename R, int PHI>
__device__ __forceinline__ void limit_half_warp(const LimitParams& P, int e, int inst, int t, unsigned hmask, int base,
                                                LimitShared<R>& sm, bool scanned, Red& red) {
  const CfdMesh& m = P.m;
  const int ld = m.ld;
  const volatile CfdControl* ctl = P.ctl ? P.ctl + inst : nullptr;
  const int status = ctl ? ctl->status : CFD_RUN_ACTIVE, par = ctl ? ctl->parity : 0;
  R* __restrict__ q = limit_state<R>(P, par);
  const double gm1 = P.gamma - 1.0;
  const int i = t < NP ? t : NP - 1;
  const int finfo = m.face_info[e];
  double a[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) a[k] = P.avg[k * ld + e];
  const double rmin0 = P.aux[e], pmin0 = P.aux[ld + e];
  const int f = t < 12 ? t >> 2 : 0, c = t & 3;
  const int nb_ = m.neighbor[f * ld + e];
  R v[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) v[c] = q[(c * NP + i) * ld + e];
  if (status != CFD_RUN_ACTIVE) return;  // a finished instance
  const double ac_d = c == 0 ? a[0] : (c == 1 ? a[1] : (c == 2 ? a[2] : a[3]));
  const R ac = (R)ac_d;
  bool troubled = false;
  R sc = R(0);
  if (PHI != LIM_UNLIMITED) {
    // the scaled neighbour difference of (f, c), as limit_scan_one forms it
    const int kind = (finfo >> (8 * f)) & 3, pf = (finfo >> (8 * f + 4)) & 3;
    const int nb = nb_;
    const R* __restrict__ cs = GeoPtr<R>::cs(m);
    const R al = cs[f * ld + e], be = cs[(3 + f) * ld + e];
    double na;
    if (kind == CFD_FACE_INTERIOR) {
      na = P.avg[c * ld + nb];
    } else if (kind == CFD_FACE_SLIP_WALL) {
      const double nx = m.face_geo[(3 * f) * ld + e], ny = m.face_geo[(3 * f + 1) * ld + e];
      const double mn = xadd(xmul(a[1], nx), xmul(a[2], ny));
      na = (c == 0 || c == 3) ? ac_d : xsub(ac_d, xmul(xmul(2.0, mn), c == 1 ? nx : ny));
    } else {
      na = m.bc_states[(nb + (kind == CFD_FACE_EXACT_STATE ? NFP : 0)) * 4 + c];
    }
    const R diff = (R)xsub(na, ac_d);
    const R pd = __shfl_sync(hmask, diff, base + 4 * pf + c);
    sc = xmul((R)NEIGHBOR_FACTOR, xadd(xmul(al, diff), xmul(be, pd)));
    if (t < NP) {
#pragma unroll
      for (int k = 0; k < 4; ++k) sm.v[4 * t + k] = v[k];
    }
    __syncwarp(hmask);
    const double det_tol = sizeof(R) == 8 ? DETECTION_TOLERANCE : DETECTION_TOLERANCE_FP32;
    const int mid = f == 0 ? tab::MID_NODES[0] : (f == 1 ? tab::MID_NODES[1] : tab::MID_NODES[2]);
    const R tr = xsub(sm.v[4 * mid + c], ac);
    const R ex = abs_(xsub(minmod2(tr, sc), tr));
    troubled = __any_sync(hmask, t < 12 && (c == 0 || c == 3) && (double)ex > xmul(det_tol, fabs(ac_d)));
  }
  if (!scanned && P.flags && t == 0) P.flags[e] = troubled ? 1 : 0;
  const double pa = pressure_x(a[0], a[1], a[2], a[3], gm1);
  const double eps = jmin(POSITIVITY_FLOOR, jmin(a[0], pa));
  const double pt = pressure_target<R>(eps, pa, a[3], gm1);
  const bool need_pos = (rmin0 < eps) || (pmin0 < pt);
  if (!troubled && !need_pos) {
    if (t == 0) limit_keep(P, e, rmin0, pmin0, red);
    return;
  }
  if (troubled) {
    // P1 midpoint values, phi-limited deltas, +/- rescaling, linear rebuild (limiting.py:153-162)
    const double* __restrict__ row = tab::P1MID[f];
    R pr = xmul((R)row[0], sm.v[c]);
#pragma unroll
    for (int j = 1; j < NP; ++j) pr = xadd(pr, xmul((R)row[j], sm.v[4 * j + c]));
    pr = xsub(pr, ac);
    R d = R(0);
    if (pr != R(0)) d = xmul(pr, jmin(R(1), phi<R, PHI>(xdiv(sc, pr))));
    const R d0 = __shfl_sync(hmask, d, base + c), d1 = __shfl_sync(hmask, d, base + 4 + c);
    const R d2 = __shfl_sync(hmask, d, base + 8 + c);
    const R pos = xadd(xadd(jmax(d0, R(0)), jmax(d1, R(0))), jmax(d2, R(0)));
    const R neg = xadd(xadd(jmax(-d0, R(0)), jmax(-d1, R(0))), jmax(-d2, R(0)));
    const R thp = pos > R(0) ? jmin(R(1), xdiv(neg, pos)) : R(0);
    const R thn = neg > R(0) ? jmin(R(1), xdiv(pos, neg)) : R(0);
    if (t < 12) sm.d[t] = xsub(xmul(thp, jmax(d, R(0))), xmul(thn, jmax(-d, R(0))));
    __syncwarp(hmask);
    const R l0 = (R)tab::LINBASIS[i][0], l1 = (R)tab::LINBASIS[i][1], l2 = (R)tab::LINBASIS[i][2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      R x = xmul(l0, sm.d[k]);
      x = xadd(x, xmul(l1, sm.d[4 + k]));
      x = xadd(x, xmul(l2, sm.d[8 + k]));
      v[k] = xadd((R)a[k], x);
    }
    if (t == 0) red.tr += 1;
  }
  double th;
  int node;
  half_warp_positivity<R>(v, a, eps, pt, gm1, i, hmask, th, node);
  if (P.pos_out && t == 0) {
    P.pos_out[e] = th;
    P.pos_out[ld + e] = (double)node;
  }
  if (t < NP) {
#pragma unroll
    for (int k = 0; k < 4; ++k) q[(k * NP + t) * ld + e] = v[k];
  }
  // ---- statistics of the own node; the wave
  // speed only where the CFL step is formed. The minima of the element are left
  // to the block's reduction: dt_geo / speed is monotone, so its least value
  // over the nodes is that of the largest speed.
  red.kr = min(red.kr, dkey(fmin(INFINITY, (double)v[0])));
  red.kp = min(red.kp, dkey(fmin(INFINITY, node_pressure<R>(v[0], v[1], v[2], v[3], gm1, POSITIVITY_FLOOR))));
  if (!(finite_(v[0]) && finite_(v[1]) && finite_(v[2]) && finite_(v[3]))) red.fl |= FLAG_NONFINITE;
  if (P.stage_idx == 3) {
    const double d = m.dt_geo[e] / wave_speed<R>(v[0], v[1], v[2], v[3], P.gamma);
    if (d != d) red.fl |= FLAG_NAN_DT;
    red.kd = min(red.kd, dkey(d));
  }
  __syncwarp(hmask);  // the half warp's next element reuses sm
}

// Adds the reductions of an element of instance i to those of its block, whose
// instance is inst0; an element of another instance (possible where instances are
// not aligned to blocks) commits by itself.
__device__ __forceinline__ void limit_take(const LimitParams& P, const Red& r, int i, int inst0, Red& red) {
  if (i == inst0) red.merge(r);
  else if (P.stage_idx != 0) commit_one(r, P.acc + 3 * i + (P.stage_idx - 1));
  else if (r.tr) atomicAdd(&P.troubled_out[i], r.tr);
}
__device__ __forceinline__ void limit_commit(const LimitParams& P, const Red& red, int inst0) {
  if (P.stage_idx == 0) {
    const int n = __reduce_add_sync(0xffffffffu, red.tr);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(&P.troubled_out[inst0], n);
  } else {
    commit_keys(red, P.acc + 3 * inst0 + (P.stage_idx - 1));
  }
}

// The limiter on the elements e0 .. e0 + EPB - 1 by a block of BS threads.
//   EPB = BS: every thread scans one element, the block lists those the
//     limiters change in shared memory, and its BS / 16 half warps rewrite
//     them. The averages the tests read are the stage's and change no more, so
//     the rewrite needs no other block.
//   EPB = BS / 16: each half warp takes one element directly, no list (smaller
//     meshes, where the scan would only lengthen the chain).
//   GLOBAL (EPB = BS): the scan alone; the listed elements go to P.list, for
//     limit_rewrite_kernel.
//   EXTERNAL: the caller lends the shared memory, BS / 16 LimitShared and EPB ints.
template <typename R, int PHI, int BS, int EPB, bool GLOBAL = false, bool EXTERNAL = false>
__device__ __forceinline__ void limit_block_body(const LimitParams& P, const int e0, LimitShared<R>* lent_half = nullptr,
                                                 int* lent_list = nullptr) {
  constexpr bool SCAN = EPB > BS / HALF;
  __shared__ LimitShared<R> own_half[EXTERNAL ? 1 : BS / HALF];
  __shared__ int own_list[SCAN && !EXTERNAL ? EPB : 1];
  __shared__ int s_count, s_inst;
  LimitShared<R>* const s_half = EXTERNAL ? lent_half : own_half;
  int* const s_list = EXTERNAL ? lent_list : own_list;
  const CfdMesh& m = P.m;
  const int lane = threadIdx.x & 31, t = lane & (HALF - 1), base = lane & HALF;
  const unsigned hmask = 0xffffu << base;
  LimitShared<R>& sm = s_half[threadIdx.x / HALF];
  const int e = e0 + (SCAN ? (int)threadIdx.x : (int)threadIdx.x / HALF);
  bool live = e < m.num_elements && (!SCAN || (int)threadIdx.x < EPB);
  int inst = 0;
  if (live && m.instance) inst = m.instance[e];
  if (inst < 0) {  // padding between instances
    live = false;
    inst = 0;
  }
  if (threadIdx.x == 0) {
    s_count = 0;
    s_inst = 0x7fffffff;
  }
  __syncthreads();
  if (live && m.instance) atomicMin(&s_inst, inst);
  Red red, own;
  red.init();
  own.init();
  if (SCAN) {
    const bool listed = live && limit_scan_one<R, PHI>(P, e, inst, own);
    if (GLOBAL) warp_list_append(P.list, P.count, listed, e, m.num_elements);
    else if (listed) s_list[atomicAdd(&s_count, 1)] = e;
  } else {
    if (live) limit_half_warp<R, PHI>(P, e, inst, t, hmask, base, sm, false, own);
  }
  __syncthreads();
  const int inst0 = m.instance ? s_inst : 0;
  if (live) limit_take(P, own, inst, inst0, red);
  if (SCAN && !GLOBAL) {
    for (int k = threadIdx.x / HALF; k < s_count; k += BS / HALF) {
      const int le = s_list[k];
      const int li = m.instance ? m.instance[le] : 0;
      own.init();
      limit_half_warp<R, PHI>(P, le, li, t, hmask, base, sm, true, own);
      limit_take(P, own, li, inst0, red);
    }
  }
  if (inst0 != 0x7fffffff) limit_commit(P, red, inst0);
}

constexpr int LIMIT_BS = 128;
// Which form: one RK3 attempt (three stages, graph replay) with the same stage
// kernel, us; the channel's elements are nearly all rewritten, the tube's few.
//                                 two launches   direct   scan of 32   of 64   of 128
//   tube,     2,000, FP64              136          104        -          -       -
//   channel,  6,700, FP64 / FP32         -        83/59     116/87        -       -
//   channel,  8,200, FP64 / FP32         -        98/67     127/91        -       -
//   tube,     8,200, FP64 / FP32         -       106/72     113/72        -       -
//   tube,     9,900, FP64 / FP32         -       116/80     110/76        -       -
//   tube,    32,000, FP32              170           -         97         93      93
//   channel, 10,000, FP64               -            -        138        173     218
//   channel, 40,000, FP64              279           -        231        262     321
//   tube,    72,000, FP64               -            -        308        295     289
//   channel, 90,000, FP64               -            -        337        372     439
//   waves,  500,000, FP64               -            -      1,578      1,524   1,564
//   tube,   800,000, FP64               -            -      2,458      2,335   2,280
// (two launches here: a scan of the whole mesh, then a rewrite of a global list with
// four lanes an element.)
// A block that rewrites all it scans takes EPB / 8 rounds of some 4,900 cycles,
// so few elements a block balance better while the blocks fit the GPU at once
// (seven of them an SM at 72 registers); in an attempt the direct form is never
// slower while its blocks of eight elements are one wave (8,288), and on large
// meshes the fixed work of a block counts instead. There a troubled region is a
// long chain in a few blocks, which in FP32-mixed, with its faster stages, made the
// attempt slower than a rewrite of a global list. FP32-mixed meshes above
// LIMIT_SCAN32_MAX therefore scan and rewrite in two launches, the listed elements
// dealt out one by one to the half warps of the grid. One attempt, us (FP32-mixed;
// channel and waves: many troubled elements side by side, tube: few):
//                       four lanes, global list   scan of 32   of 64   of 128   two launches
//   tube,     72,000               219                172        161      155        165
//   channel,  90,000               231                204        226      272        183
//   waves,   180,000               482                431        438      470        371
//   waves,   500,000               942                989        939      976        831
//   tube,    800,000             1,384              1,463      1,325    1,258      1,259
// In FP64 the single launch was nowhere slower than the four-lane rewrite (a limiter
// call on the channels of 72,000 and 90,000 elements: 63 and 82 us against 60 and
// 71) and stays; its line between scans of 32 and of 128 is a compromise.
constexpr int LIMIT_DIRECT_MAX = 148 * 7 * (LIMIT_BS / HALF), LIMIT_SCAN32_MAX = 70000;
constexpr int LIMIT_REWRITE_BLOCKS = 148 * 3;  // 3,552 half warps; seven blocks an SM cost a tube 2 % more
template <typename R, int PHI, int EPB>
__global__ void __launch_bounds__(LIMIT_BS, 7) limit_kernel(const LimitParams P) {
  limit_block_body<R, PHI, LIMIT_BS, EPB>(P, blockIdx.x * EPB);
}

// Least keys and joint flags of a half warp's lanes in each of them.
__device__ __forceinline__ void half_warp_join(Red& r, unsigned hmask) {
#pragma unroll
  for (int o = 1; o < HALF; o <<= 1) {
    r.kr = min(r.kr, __shfl_xor_sync(hmask, r.kr, o));
    r.kp = min(r.kp, __shfl_xor_sync(hmask, r.kp, o));
    r.kd = min(r.kd, __shfl_xor_sync(hmask, r.kd, o));
  }
  r.fl = __reduce_or_sync(hmask, (unsigned)r.fl);
}

// The rewrite of the elements that a GLOBAL scan has listed, dealt out one by one
// to the half warps of the whole grid. The last block to finish zeroes the counters
// for the next pair of launches. (Counters that a caller has not zeroed could make
// it read entries no scan has written: what is no element is left out.)
template <typename R, int PHI>
__global__ void __launch_bounds__(LIMIT_BS, 7) limit_rewrite_kernel(const LimitParams P) {
  constexpr int EPB = LIMIT_BS / HALF;
  __shared__ LimitShared<R> s_half[EPB];
  __shared__ int s_n;
  const CfdMesh& m = P.m;
  auto element = [&](int k) {
    const int e = P.list[k];
    return (unsigned)e < (unsigned)m.num_elements ? e : -1;
  };
  if (threadIdx.x == 0) s_n = min(*(volatile int*)P.count, m.num_elements);
  __syncthreads();
  const int n = s_n, first = blockIdx.x * EPB;
  if (first < n) {
    const int lane = threadIdx.x & 31, t = lane & (HALF - 1), base = lane & HALF;
    const unsigned hmask = 0xffffu << base;
    const int e0 = element(first), inst0 = m.instance && e0 >= 0 ? m.instance[e0] : 0;
    Red red, own;
    red.init();
    for (int k = first + (int)threadIdx.x / HALF; k < n; k += gridDim.x * EPB) {
      const int e = element(k), inst = m.instance && e >= 0 ? m.instance[e] : 0;
      if (e < 0 || inst < 0) continue;
      own.init();
      limit_half_warp<R, PHI>(P, e, inst, t, hmask, base, s_half[threadIdx.x / HALF], true, own);
      if (inst != inst0 && P.stage_idx != 0) {  // a batch's list mixes instances: one commit an element
        half_warp_join(own, hmask);
        if (t != 0) own.init();
      }
      limit_take(P, own, inst, inst0, red);
    }
    limit_commit(P, red, inst0);
  }
  if (threadIdx.x == 0 && atomicAdd(&P.count[1], 1) == (int)gridDim.x - 1) P.count[0] = P.count[1] = 0;
}
template <typename R, int PHI>
__global__ void __launch_bounds__(LIMIT_BS) limit_scan_kernel(const LimitParams P) {
  limit_block_body<R, PHI, LIMIT_BS, LIMIT_BS, true>(P, blockIdx.x * LIMIT_BS);
}
