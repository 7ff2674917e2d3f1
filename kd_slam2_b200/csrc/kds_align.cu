// Fused ICP / CT-ICP linearization and on-device Gauss-Newton.
//
// k_linearize: one launch = one Gauss-Newton iteration for every job (of one kind) of a batch.
// k_linearize_persistent runs all iterations of a batch in one launch, k_align_cluster those of
// a single alignment, with the same tiles and the same step.  A job is one
// alignment (ICP_::compute / CTICP_::compute, kd/icp/tree_aligner_base_.h:100-115)
// or one buildQuadraticForm; it has one moving leaf set and one or more fixed
// entries (the _fixed_forest of kd/icp/icp_impl_.h:55-71).  The grid is a flat list of
// tiles (job, entry, 128 moving leaves); each block:
//   1. runs quadraticTerm for its leaves (kd/icp/icp_impl_.h:102-152,
//      kd/cticp/cticp_impl_.h:105-293): optional CT warp, greedy descent through the
//      fixed tree, gates, symmetric error, Jacobian, robust weight -- the gating path in
//      exact single roundings so matches and masks equal the CPU oracle bit for bit;
//   2. reduces gamma*J^T J and gamma*J^T e over its leaves warp-cooperatively: each
//      lane owns a few of the D(D+1)/2+D entries and sums them over the warp's 32
//      leaves with Kahan compensation; warps are combined in FP64 into one block
//      partial (no per-leaf workspace, replacing ICP_kernel + ~2x14 _reduce1 passes,
//      kd/icp/icp_cuda_impl_.cuh:68-132, kd/cuda/reduce_impl_.cuh:9-78);
//   3. the last block of a job to finish sums the job's partials in tile order (FP64,
//      deterministic: the result of a job does not depend on what else is in the
//      batch), adds the pose prior, solves (H + damping) dx = -b by an FP64 Cholesky
//      factorization, applies X <- expmap(dx) X, v += dx_v, runs the termination test and
//      refreshes the float caches of the next iteration.  No host round trip inside compute().
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "kds_align.cuh"
#include "kds_internal.cuh"
#include "kds_rules.h"

namespace kds {

// Every float operation of the per-leaf path -- gates, errors and Jacobians -- rounds
// once, in the operation order of the CPU oracle (itself the reference's order,
// kd/d3/icp_.h:40-60, kd/d3/cticp_impl_.h:10-73, kd/utils/geometry_3d_impl_.h:143-174):
// 3-term sums as x0 + (x1 + x2), as Eigen reduces a fixed-size-3 dot product.  So the
// per-leaf terms, and with the fixed summation order below H and b, are bit-identical
// to the oracle's.
__device__ __forceinline__ F3 cross3(F3 a, F3 b) {
  return f3(fs(fm(a.y, b.z), fm(a.z, b.y)), fs(fm(a.z, b.x), fm(a.x, b.z)), fs(fm(a.x, b.y), fm(a.y, b.x)));
}

// C = A * B (3x3 row-major), each coefficient a dot3x of a row and a column
__device__ __forceinline__ void mm3(const float* A, const float* B, float* C) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      C[i * 3 + j] = fa(fm(A[i * 3], B[j]), fa(fm(A[i * 3 + 1], B[3 + j]), fm(A[i * 3 + 2], B[6 + j])));
}
__device__ __forceinline__ F3 mv3(const float* A, F3 p) { return mat_vec_x(A, p); }
// column c of a row-major 3x3
__device__ __forceinline__ F3 col3(const float* A, int c) { return f3(A[c], A[3 + c], A[6 + c]); }

// C = A * skew(u): each coefficient's dot3x less its term with a zero factor
__device__ __forceinline__ void mm3_skew(const float* A, F3 u, float* C) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    C[i * 3] = fa(fm(A[i * 3 + 1], u.z), fm(A[i * 3 + 2], -u.y));
    C[i * 3 + 1] = fa(fm(A[i * 3], -u.z), fm(A[i * 3 + 2], u.x));
    C[i * 3 + 2] = fa(fm(A[i * 3], u.y), fm(A[i * 3 + 1], -u.x));
  }
}

// Pieces of dRxp (kd/utils/geometry_3d_impl_.h:143-174) shared by both of its calls:
// with R = rodrigues(w), Q = n n^T + (R^T - I) S / angle, so that
// d(R u)/dw = -R skew(u) Q.  small = angle < 1e-9 (then dR = -skew(u)).
struct DRxp {
  float Q[9];
  bool small;
};
__device__ __forceinline__ void drxp_setup(F3 w, const float* R, DRxp& d) {
  float angle = __fsqrt_rn(dot3x(w, w));
  d.small = angle < 1e-9f;
  if (d.small) {
#pragma unroll
    for (int i = 0; i < 9; ++i) d.Q[i] = 0.f;
    return;
  }
  float inv = __fdiv_rn(1.0f, angle);
  F3 n = f3(fm(w.x, inv), fm(w.y, inv), fm(w.z, inv));
  float RtmI[9] = {fs(R[0], 1.f), R[3], R[6], R[1], fs(R[4], 1.f), R[7], R[2], R[5], fs(R[8], 1.f)};
  float A[9];
  mm3_skew(RtmI, n, A);
  float nn[3] = {n.x, n.y, n.z};
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) d.Q[i * 3 + j] = fa(fm(nn[i], nn[j]), fm(A[i * 3 + j], inv));
}
// out = Ra * d(R u)/dw  (3x3)
__device__ __forceinline__ void ra_drxp(const DRxp& d, const float* R, const float* Ra, F3 u, float* out) {
  float dR[9];
  if (d.small) {
    mm3_skew(Ra, f3(-u.x, -u.y, -u.z), out);
    return;
  }
  float Rs[9];
  mm3_skew(R, u, Rs);
  mm3(Rs, d.Q, dR);
#pragma unroll
  for (int i = 0; i < 9; ++i) dR[i] = -dR[i];
  mm3(Ra, dR, out);
}

// errorAndJacobianVelocityA (kd/d3/cticp_impl_.h:10-39) -> J[0..5].  R = rodrigues(va_w dt);
// pam, nam: the leaf warped by the velocities (applyVelocities).
__device__ __forceinline__ void jac_vel_A(const float* Xm, F3 pa_l, F3 na_l, F3 pam, F3 nam, F3 pb_g, F3 nb_g,
                                          const float* va, const float* R, float dt, float* J) {
  F3 wa = f3(fm(va[3], dt), fm(va[4], dt), fm(va[5], dt));
  DRxp d;
  drxp_setup(wa, R, d);
  float Ra[9] = {Xm[0], Xm[1], Xm[2], Xm[4], Xm[5], Xm[6], Xm[8], Xm[9], Xm[10]};
  F3 pag = add3x(mv3(Ra, pam), f3(Xm[3], Xm[7], Xm[11]));
  F3 nag = mv3(Ra, nam);
  F3 n = add3x(nag, nb_g);
  F3 dp = sub3x(pag, pb_g);
  float A[9], B[9];
  ra_drxp(d, R, Ra, pa_l, A);
  ra_drxp(d, R, Ra, na_l, B);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    J[c] = fm(dot3x(n, col3(Ra, c)), dt);
    J[3 + c] = fm(fa(dot3x(n, col3(A, c)), dot3x(dp, col3(B, c))), dt);
  }
}

// errorAndJacobianVelocityB (kd/d3/cticp_impl_.h:43-73) -> J[0..5]
__device__ __forceinline__ void jac_vel_B(const float* Xf, F3 pa_g, F3 na_g, F3 pb_l, F3 nb_l, const float* vb, float dt,
                                          float* J) {
  F3 wb = f3(fm(vb[3], dt), fm(vb[4], dt), fm(vb[5], dt));
  float R[9];
  F3 pbm, nbm;
  warp_x(vb, dt, pb_l, nb_l, pbm, nbm, R);
  DRxp d;
  drxp_setup(wb, R, d);
  float Rb[9] = {Xf[0], Xf[1], Xf[2], Xf[4], Xf[5], Xf[6], Xf[8], Xf[9], Xf[10]};
  F3 pbg = add3x(mv3(Rb, pbm), f3(Xf[3], Xf[7], Xf[11]));
  F3 nbg = mv3(Rb, nbm);
  F3 n = add3x(na_g, nbg);
  F3 nn = f3(-n.x, -n.y, -n.z);
  F3 dp = sub3x(pa_g, pbg);
  float A[9], B[9];
  ra_drxp(d, R, Rb, pb_l, A);
  ra_drxp(d, R, Rb, nb_l, B);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    J[c] = fm(dot3x(nn, col3(Rb, c)), dt);
    J[3 + c] = fm(fa(dot3x(nn, col3(A, c)), dot3x(dp, col3(B, c))), dt);
  }
}

enum { ST_INLIER = 0, ST_OUTLIER = 1, ST_BAD = 2, ST_ERR_NORMAL = 3, ST_ERR_FN = 4, ST_NONE = 5 };

template <int KIND> struct KindDim;
template <> struct KindDim<0> { static constexpr int D = 6; };
template <> struct KindDim<1> { static constexpr int D = 12; };
template <> struct KindDim<2> { static constexpr int D = 18; };

// The query of one moving leaf: optional CT warp (applyVelocities, its rotation in R) and
// the moving-to-fixed transform Xmf.
template <int KIND>
__device__ __forceinline__ void leaf_query(const CacheF& C, float4 md, float4 nr, F3& m, F3& n, F3& mw, F3& nw,
                                           F3& q, float* R) {
  m = f3(md.x, md.y, md.z);
  n = f3(nr.x, nr.y, nr.z);
  mw = m;
  nw = n;
  if (KIND != 0) warp_x(C.v, md.w, m, n, mw, nw, R);
  q = apply_iso_x(C.Xmf, mw);
}

// Greedy descent (kd/icp/icp_impl_.h:116-121): no backtracking.  idx = the leaf reached,
// or -1 where the descent steps into a pruned child; nd = its record.
__device__ __forceinline__ void descend(const DNode* F, int fnn, const DNode* staged, int nstaged, F3 q, int& idx,
                                        DNode& nd) {
  idx = fnn > 0 ? 0 : -1;
  while (idx >= 0) {
    nd = (idx < nstaged) ? staged[idx] : load_node(F + idx);
    int l = node_left(nd), r = node_right(nd);
    if (l < 0 && r < 0) break;
    bool side = dot3x(node_dir(nd), sub3x(q, node_mean(nd))) > 0.0f;
    idx = side ? l : r;
  }
}

// Two descents through the same tree in lockstep: both chains' node loads are issued
// before either is used, so a thread keeps two dependent load chains in flight.  Each
// chain takes exactly the steps of descend().
__device__ __forceinline__ void descend2(const DNode* F, int fnn, const DNode* staged, int nstaged, bool va, F3 qa,
                                         int& ia, DNode& na, bool vb, F3 qb, int& ib, DNode& nb) {
  ia = (va && fnn > 0) ? 0 : -1;
  ib = (vb && fnn > 0) ? 0 : -1;
  bool ra = ia >= 0, rb = ib >= 0;  // still descending
  while (ra || rb) {
    if (ra) na = (ia < nstaged) ? staged[ia] : load_node(F + ia);
    if (rb) nb = (ib < nstaged) ? staged[ib] : load_node(F + ib);
    if (ra) {
      const int l = node_left(na), r = node_right(na);
      if (l < 0 && r < 0) {
        ra = false;
      } else {
        ia = dot3x(node_dir(na), sub3x(qa, node_mean(na))) > 0.0f ? l : r;
        ra = ia >= 0;
      }
    }
    if (rb) {
      const int l = node_left(nb), r = node_right(nb);
      if (l < 0 && r < 0) {
        rb = false;
      } else {
        ib = dot3x(node_dir(nb), sub3x(qb, node_mean(nb))) > 0.0f ? l : r;
        rb = ib >= 0;
      }
    }
  }
}

// Gates, error, Jacobian and robust weight of one leaf whose descent ended at idx / nd.
template <int KIND>
__device__ __forceinline__ void leaf_math(const CacheF& C, F3 m, F3 n, float dt, F3 mw, F3 nw, const float* R,
                                          int idx, const DNode& nd, const float* fdts, const ParamsF& P, bool stats_mode,
                                          int& status, int& match, float& e_out, float& gamma_out, float* J) {
  constexpr int D = KindDim<KIND>::D;
#pragma unroll
  for (int i = 0; i < D; ++i) J[i] = 0.f;
  e_out = 0.f;
  gamma_out = 0.f;
  match = idx;
  if (idx < 0) { status = ST_BAD; return; }
  F3 pf = node_mean(nd), nf = node_dir(nd);
  F3 pm = apply_iso_x(C.Xm, mw);
  F3 nm = apply_rot_x(C.Xm, nw);
  F3 pfx = apply_iso_x(C.Xf, pf);
  F3 nfx = apply_rot_x(C.Xf, nf);
  // ICP_3D_Traits::errorAndJacobian (kd/d3/icp_.h:40-60)
  if (dot3x(nfx, nm) < P.min_normal_cos) { status = ST_ERR_NORMAL; return; }
  F3 ns = add3x(nm, nfx);
  float e = dot3x(sub3x(pm, pfx), ns);
  if (fabsf(e) > P.max_error) { status = ST_ERR_FN; return; }
  F3 c1 = cross3(pm, nfx), c2 = cross3(pfx, nm);
  J[0] = ns.x; J[1] = ns.y; J[2] = ns.z;
  J[3] = fa(c1.x, c2.x); J[4] = fa(c1.y, c2.y); J[5] = fa(c1.z, c2.z);
  if (KIND != 0) jac_vel_A(C.Xm, m, n, mw, nw, pfx, nfx, C.v, R, dt, J + 6);
  float chi2 = fm(e, e);
  float kt = P.kernel_threshold;
  float gamma;
  if (KIND == 2) {
    gamma = stats_mode ? 0.f : 1.f;
    if (chi2 > kt) { status = ST_OUTLIER; gamma = __fsqrt_rn(__fdiv_rn(kt, chi2)); }
    else status = ST_INLIER;
    jac_vel_B(C.Xf, pm, nm, pf, nf, C.fv, fdts[idx], J + 12);
  } else {
    gamma = 1.f;
    if (chi2 > kt) { status = ST_OUTLIER; gamma = stats_mode ? 0.f : __fsqrt_rn(__fdiv_rn(kt, chi2)); }
    else status = ST_INLIER;
  }
  e_out = e;
  gamma_out = gamma;
}

template <int KIND>
__device__ __forceinline__ void leaf_term(const CacheF& C, const DNode* F, int fnn, const float* fdts,
                                          const DNode* staged, int nstaged, float4 md,
                                          float4 nr, const ParamsF& P, bool stats_mode, int& status, int& match,
                                          float& e_out, float& gamma_out, float* J) {
  F3 m, n, mw, nw, q;
  float R[9];
  leaf_query<KIND>(C, md, nr, m, n, mw, nw, q, R);
  int idx;
  DNode nd;
  descend(F, fnn, staged, nstaged, q, idx, nd);
  leaf_math<KIND>(C, m, n, md.w, mw, nw, R, idx, nd, fdts, P, stats_mode, status, match, e_out, gamma_out, J);
}

// Entry k of the packed D(D+1)/2 + D vector (upper triangle row by row, then J_r e):
// (row, col); col == D means "e".
template <int D>
struct alignas(4) EntryTable {
  static constexpr int M = D * (D + 1) / 2 + D;
  unsigned char rc[M][2];
};
template <int D>
constexpr EntryTable<D> make_entry_table() {
  EntryTable<D> t{};
  int k = 0;
  for (int r = 0; r < D; ++r)
    for (int c = r; c < D; ++c, ++k) {
      t.rc[k][0] = (unsigned char)r;
      t.rc[k][1] = (unsigned char)c;
    }
  for (int r = 0; r < D; ++r, ++k) {
    t.rc[k][0] = (unsigned char)r;
    t.rc[k][1] = (unsigned char)D;
  }
  return t;
}
__device__ const EntryTable<6> g_rc6 = make_entry_table<6>();
__device__ const EntryTable<12> g_rc12 = make_entry_table<12>();
__device__ const EntryTable<18> g_rc18 = make_entry_table<18>();
__device__ __forceinline__ void entry_rc(int D, int k, int& r, int& c) {
  const unsigned char* t = D == 6 ? g_rc6.rc[k] : (D == 12 ? g_rc12.rc[k] : g_rc18.rc[k]);
  const uchar2 v = __ldg(reinterpret_cast<const uchar2*>(t));
  r = v.x;
  c = v.y;
}

constexpr int kBlock = 128;
constexpr int kWarps = kBlock / 32;
// A warp's factors in shared memory: row r (J_0 .. J_{D-1}, e, gamma) holds the 32 leaves' values,
// read four leaves at a time; the row stride of 36 floats spreads the rows over the banks.
constexpr int kFacStride = 36;
constexpr int kMaxFac = 20 * kFacStride;  // floats per warp, D = 18

// One warp's share of a tile partial from its 32 leaves' terms (leaf = lane): stats by
// ballots, chi2 sums by xor butterfly, and gamma J^T J, gamma J^T e as float Kahan sums
// over the lanes (lane k owns packed entries k, k + 32, ...) stored as s - comp in FP64.
// A warp's partial takes STRIDE doubles, its 7 stats at STATS.
template <int KIND, int STRIDE = kPStride, int STATS = kPStats>
__device__ __forceinline__ void tile_reduce(int status, float e, float gamma, const float* J, double* wpart,
                                            float* fac) {
  constexpr int D = KindDim<KIND>::D;
  constexpr int M = D * (D + 1) / 2 + D;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  bool contrib = status == ST_INLIER || status == ST_OUTLIER;
  float* wf = fac + w * (D + 2) * kFacStride;
#pragma unroll
  for (int k = 0; k < D; ++k) wf[k * kFacStride + lane] = contrib ? J[k] : 0.f;
  wf[D * kFacStride + lane] = contrib ? e : 0.f;
  wf[(D + 1) * kFacStride + lane] = contrib ? gamma : 0.f;
  // stats (ICPStats_::pack, kd/icp/icp_stats_.h:57-59)
  unsigned full = 0xffffffffu;
  int c_in = __popc(__ballot_sync(full, status == ST_INLIER));
  int c_out = __popc(__ballot_sync(full, status == ST_OUTLIER));
  int c_bad = __popc(__ballot_sync(full, status == ST_BAD));
  int c_nrm = __popc(__ballot_sync(full, status == ST_ERR_NORMAL));
  int c_fn = __popc(__ballot_sync(full, status == ST_ERR_FN));
  double chi2 = contrib ? (double)fm(e, e) : 0.0;
  double chi2k = contrib ? (double)fm(fm(e, e), gamma) : 0.0;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    chi2 += __shfl_xor_sync(full, chi2, off);
    chi2k += __shfl_xor_sync(full, chi2k, off);
  }
  __syncwarp();
  // Warp-cooperative outer products: lane owns entries lane, lane + 32, ..., all of them summed
  // side by side (one compensated sum is a chain of four dependent operations per leaf).
  constexpr int NE = (M + 31) / 32;
  double* wp = wpart + w * STRIDE;
  const float4 *pr[NE], *pc[NE];
  float s[NE], comp[NE];
#pragma unroll
  for (int k = 0; k < NE; ++k) {
    int r, c;
    entry_rc(D, min(lane + 32 * k, M - 1), r, c);
    pr[k] = reinterpret_cast<const float4*>(wf + r * kFacStride);
    pc[k] = reinterpret_cast<const float4*>(wf + c * kFacStride);
    s[k] = comp[k] = 0.f;
  }
  const float4* pg = reinterpret_cast<const float4*>(wf + (D + 1) * kFacStride);
#pragma unroll 1
  for (int q = 0; q < 8; ++q) {
    const float4 g4 = pg[q];
    const float g[4] = {g4.x, g4.y, g4.z, g4.w};
    float4 r4[NE], c4[NE];
#pragma unroll
    for (int k = 0; k < NE; ++k) {
      r4[k] = pr[k][q];
      c4[k] = pc[k][q];
    }
#pragma unroll
    for (int l = 0; l < 4; ++l)
#pragma unroll
      for (int k = 0; k < NE; ++k) {
        const float rv = l == 0 ? r4[k].x : (l == 1 ? r4[k].y : (l == 2 ? r4[k].z : r4[k].w));
        const float cv = l == 0 ? c4[k].x : (l == 1 ? c4[k].y : (l == 2 ? c4[k].z : c4[k].w));
        float val = fm(fm(rv, cv), g[l]);
        float y = fs(val, comp[k]);
        float t = fa(s[k], y);
        comp[k] = fs(fs(t, s[k]), y);
        s[k] = t;
      }
  }
#pragma unroll
  for (int k = 0; k < NE; ++k)
    if (lane + 32 * k < M) wp[lane + 32 * k] = (double)s[k] - (double)comp[k];
  if (lane == 0) {
    wp[STATS + 0] = c_in;
    wp[STATS + 1] = c_out;
    wp[STATS + 2] = c_bad;
    wp[STATS + 3] = c_nrm;
    wp[STATS + 4] = c_fn;
    wp[STATS + 5] = chi2;
    wp[STATS + 6] = chi2k;
  }
  __syncwarp();  // the warp's rows may be rewritten after this
}

template <int KIND, int STRIDE = kPStride, int STATS = kPStats>
__device__ __forceinline__ void tile_body(const JobIn& Jn, const LinDev& L, const CacheF& C, const TileDev& T,
                                          const DNode* staged, int nstaged,
                                          double* wpart /* [kWarps][STRIDE] */, float* fac /* [kWarps][(D + 2) * kFacStride] */,
                                          int32_t* dbg_match, int32_t* dbg_status) {
  constexpr int D = KindDim<KIND>::D;
  const int i = T.leaf_begin + (threadIdx.x & (kBlock - 1));
  int status = ST_NONE, match = -1;
  float e = 0.f, gamma = 0.f;
  float J[D];
#pragma unroll
  for (int k = 0; k < D; ++k) J[k] = 0.f;
  if (i < T.leaf_end) {
    float4 md = __ldg(Jn.m_md + i);
    float4 nr = __ldg(Jn.m_nrm + i);
    leaf_term<KIND>(C, L.fnodes, L.f_num_nodes, L.fdts, staged, nstaged, md, nr, Jn.P, Jn.stats_mode != 0, status,
                    match, e, gamma, J);
    if (dbg_match) { dbg_match[i] = match; dbg_status[i] = status; }
  }
  tile_reduce<KIND, STRIDE, STATS>(status, e, gamma, J, wpart, fac);
}

// Two tiles of one (job, fixed entry) per block: thread t takes leaf t of both, runs the
// two descents in lockstep, then reduces tile A and tile B one after the other with
// tile_body's arithmetic, so each tile's partial is bit-identical to one-tile blocks.
template <int KIND>
__device__ __forceinline__ void tile_body_pair(const JobIn& Jn, const LinDev& L, const CacheF& C, const TileDev& TA,
                                               const TileDev& TB, bool has_b, const DNode* staged, int nstaged,
                                               double* wpa, double* wpb, float* fac, int32_t* dbg_match,
                                               int32_t* dbg_status) {
  constexpr int D = KindDim<KIND>::D;
  const int ia = TA.leaf_begin + threadIdx.x, ib = TB.leaf_begin + threadIdx.x;
  const bool va = ia < TA.leaf_end, vb = has_b && ib < TB.leaf_end;
  F3 ma, na, mwa, nwa, qa, mb, nb, mwb, nwb, qb;
  float dta = 0.f, dtb = 0.f;
  float R[9];  // recomputed after the descents: two would not fit the registers
  if (va) {
    const float4 md = __ldg(Jn.m_md + ia), nr = __ldg(Jn.m_nrm + ia);
    leaf_query<KIND>(C, md, nr, ma, na, mwa, nwa, qa, R);
    dta = md.w;
  }
  if (vb) {
    const float4 md = __ldg(Jn.m_md + ib), nr = __ldg(Jn.m_nrm + ib);
    leaf_query<KIND>(C, md, nr, mb, nb, mwb, nwb, qb, R);
    dtb = md.w;
  }
  int xa, xb;
  DNode nda, ndb;
  descend2(L.fnodes, L.f_num_nodes, staged, nstaged, va, qa, xa, nda, vb, qb, xb, ndb);
  {
    int status = ST_NONE, match = -1;
    float e = 0.f, gamma = 0.f, J[D];
#pragma unroll
    for (int k = 0; k < D; ++k) J[k] = 0.f;
    if (va) {
      if (KIND != 0) rodrigues_x(f3(fm(C.v[3], dta), fm(C.v[4], dta), fm(C.v[5], dta)), R);
      leaf_math<KIND>(C, ma, na, dta, mwa, nwa, R, xa, nda, L.fdts, Jn.P, Jn.stats_mode != 0, status, match, e, gamma, J);
      if (dbg_match) { dbg_match[ia] = match; dbg_status[ia] = status; }
    }
    tile_reduce<KIND>(status, e, gamma, J, wpa, fac);
  }
  {
    int status = ST_NONE, match = -1;
    float e = 0.f, gamma = 0.f, J[D];
#pragma unroll
    for (int k = 0; k < D; ++k) J[k] = 0.f;
    if (vb) {
      if (KIND != 0) rodrigues_x(f3(fm(C.v[3], dtb), fm(C.v[4], dtb), fm(C.v[5], dtb)), R);
      leaf_math<KIND>(C, mb, nb, dtb, mwb, nwb, R, xb, ndb, L.fdts, Jn.P, Jn.stats_mode != 0, status, match, e, gamma, J);
      if (dbg_match) { dbg_match[ib] = match; dbg_status[ib] = status; }
    }
    tile_reduce<KIND>(status, e, gamma, J, wpb, fac);
  }
}

// ---------------------------------------------------------------------------
// FP64 finalize (one thread) -- ICP_::oneRound / CTICP_::oneRound.
// Pose algebra in FP64 with one rounding per operation and 3-term sums as
// x0 + (x1 + x2), the CPU oracle's order for Eigen's Transform product and inverse.
__device__ __forceinline__ double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double da(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double ds(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double ddot3(double a0, double a1, double a2, double b0, double b1, double b2) {
  return da(dm(a0, b0), da(dm(a1, b1), dm(a2, b2)));
}
// Canonical FP64 sine/cosine (this project's own, shared with the CPU oracle so that the
// pose update is bit-identical there): Cody-Waite reduction by pi/2 with a three-part
// constant (Cody & Waite 1980; parts of 33, 33 and 53 bits, so q * C1 and q * C2 are
// exact for |q| < 2^20), then the Taylor series of sin to r^17 and of cos to r^18 on
// [-pi/4, pi/4] in Horner form (truncation below 1e-19).
__device__ void sincos_canon_d(double x, double* s_out, double* c_out) {
  const double q = rint(dm(x, 0x1.45f306dc9c883p-1));
  const long long j = (long long)q;
  double r = ds(x, dm(q, 0x1.921fb54400000p+0));
  r = ds(r, dm(q, 0x1.0b4611a600000p-34));
  r = ds(r, dm(q, 0x1.3198a2e037073p-69));
  const double r2 = dm(r, r);
  double t = 0x1.952c77030ad4ap-49;             // 1/17!
  t = da(-0x1.ae7f3e733b81fp-41, dm(r2, t));    // 1/15!
  t = da(0x1.6124613a86d09p-33, dm(r2, t));     // 1/13!
  t = da(-0x1.ae64567f544e4p-26, dm(r2, t));    // 1/11!
  t = da(0x1.71de3a556c734p-19, dm(r2, t));     // 1/9!
  t = da(-0x1.a01a01a01a01ap-13, dm(r2, t));    // 1/7!
  t = da(0x1.1111111111111p-7, dm(r2, t));      // 1/5!
  t = da(-0x1.5555555555555p-3, dm(r2, t));     // 1/3!
  const double sn = da(r, dm(r, dm(r2, t)));
  double u = -0x1.6827863b97d97p-53;            // 1/18!
  u = da(0x1.ae7f3e733b81fp-45, dm(r2, u));     // 1/16!
  u = da(-0x1.93974a8c07c9dp-37, dm(r2, u));    // 1/14!
  u = da(0x1.1eed8eff8d898p-29, dm(r2, u));     // 1/12!
  u = da(-0x1.27e4fb7789f5cp-22, dm(r2, u));    // 1/10!
  u = da(0x1.a01a01a01a01ap-16, dm(r2, u));     // 1/8!
  u = da(-0x1.6c16c16c16c17p-10, dm(r2, u));    // 1/6!
  u = da(0x1.5555555555555p-5, dm(r2, u));      // 1/4!
  u = da(-0.5, dm(r2, u));
  const double cs = da(1.0, dm(r2, u));
  switch ((int)(j & 3)) {
    case 0: *s_out = sn; *c_out = cs; break;
    case 1: *s_out = cs; *c_out = -sn; break;
    case 2: *s_out = -sn; *c_out = -cs; break;
    default: *s_out = -cs; *c_out = sn; break;
  }
}

// rodrigues (kd/utils/geometry_3d_impl_.h:37-46) in FP64: I + sin(a) S + (1 - cos(a)) S^2
__device__ __forceinline__ void rodrigues_d(const double* w, double* R) {
  const double a = sqrt(ddot3(w[0], w[1], w[2], w[0], w[1], w[2]));
  if (a < 1e-9) {
    for (int i = 0; i < 9; ++i) R[i] = (i % 4 == 0) ? 1.0 : 0.0;
    return;
  }
  const double inv = 1.0 / a;
  const double n[3] = {dm(w[0], inv), dm(w[1], inv), dm(w[2], inv)};
  const double S[9] = {0, -n[2], n[1], n[2], 0, -n[0], -n[1], n[0], 0};
  double s, c;
  sincos_canon_d(a, &s, &c);
  const double omc = ds(1.0, c);
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      const double s2 = ddot3(S[i * 3], S[i * 3 + 1], S[i * 3 + 2], S[j], S[3 + j], S[6 + j]);
      R[i * 3 + j] = da(da((i == j) ? 1.0 : 0.0, dm(s, S[i * 3 + j])), dm(omc, s2));
    }
}
// Pose prior (posePriorBuildQuadraticForm, kd/icp/tree_aligner_base_.h:139-152, over
// dPoseToPoseError, kd/utils/geometry_3d_impl_.h:125-140, in FP64): adds J^T Omega J and
// J^T Omega e to the pose block.  One warp, an element per lane, with the matrices in t
// (kPriorDoubles of shared memory).  Bound by the chain of an acos, a sine and four small
// products.  A single thread with the matrices in local memory spilled under the 64 registers of
// k_linearize: ten rigid iterations with a prior, launched one by one, took 376 us (290 under
// 128 registers), now 249; without a prior 216.
constexpr int kPriorP = 0, kPriorE = 12, kPriorJ = 18;        // Z X^-1 Xm, error, Jacobian
constexpr int kPriorB = 54, kPriorS = 108;                    // dP's rotation, dlog of it
constexpr int kPriorOJ = kPriorB, kPriorOe = kPriorB + 36;    // Omega J, Omega e: B is done then
constexpr int kPriorDoubles = 135;
__device__ __noinline__ void add_pose_prior(const JobIn& Jn, const double* X, double* H, double* b, int D, double* t,
                                            int lane) {
  const double* A = Jn.prior_ZXi;
  const double* Om = Jn.prior_info;
  if (lane < 12) {
    const int i = lane >> 2, j = lane & 3;
    const double d = ddot3(A[i * 4], A[i * 4 + 1], A[i * 4 + 2], X[j], X[4 + j], X[8 + j]);
    t[kPriorP + lane] = j < 3 ? d : da(d, A[i * 4 + 3]);
  }
  // entry (i, j) of R skew(v), R the rotation of A, v column k of X
  auto rot_skew = [&](int i, int j, int k) {
    double m[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const double v = X[4 * ((6 - r - j) % 3) + k];  // the third index; unused where r == j
      m[r] = A[i * 4 + r] * (r == j ? 0.0 : ((j - r + 3) % 3 == 2 ? v : -v));
    }
    return m[0] + m[1] + m[2];
  };
  for (int e = lane; e < 54; e += 32) {  // rows: P's rotation column by column
    const int r = e / 6, j = e % 6;
    t[kPriorB + e] = j < 3 ? 0.0 : -rot_skew(r % 3, j - 3, r / 3);
  }
  __syncwarp();
  const double* P = t + kPriorP;
  {
    const double ca = fmin(1.0, fmax(-1.0, 0.5 * (P[0] + P[5] + P[10] - 1.0)));
    const double a = acos(ca);
    const bool small = a < 1e-7;
    const double f = small ? 0.5 : a / (2.0 * sin(a));
    auto axis = [&](int i) { return i == 0 ? P[9] - P[6] : (i == 1 ? P[2] - P[8] : P[4] - P[1]); };
    if (lane < 3) t[kPriorE + lane] = P[lane * 4 + 3];
    else if (lane < 6) t[kPriorE + lane] = axis(lane - 3) * f;
    if (lane < 27) {
      const int i = lane / 9, k = lane % 9;
      double v = 0.0;
      if (k == (i == 0 ? 5 : (i == 1 ? 6 : 1))) v = f;
      if (k == (i == 0 ? 7 : (i == 1 ? 2 : 3))) v = -f;
      if (!small && (k & 3) == 0) {
        const double s = sin(a);
        v -= (s - a * cos(a)) / (4.0 * s * s * s) * axis(i);
      }
      t[kPriorS + lane] = v;
    }
  }
  __syncwarp();
  for (int e = lane; e < 36; e += 32) {
    const int i = e / 6, j = e % 6;
    double v = 0.0;
    if (i >= 3) {
      for (int k = 0; k < 9; ++k) v += t[kPriorS + (i - 3) * 9 + k] * t[kPriorB + k * 6 + j];
    } else {
      v = j < 3 ? A[i * 4 + j] : -rot_skew(i, j - 3, 3);
    }
    t[kPriorJ + e] = v;
  }
  __syncwarp();
  const double* J = t + kPriorJ;
  for (int e = lane; e < 42; e += 32) {
    const int i = e < 36 ? e / 6 : e - 36, j = e % 6;
    double v = 0.0;
    for (int k = 0; k < 6; ++k) v += Om[i * 6 + k] * (e < 36 ? J[k * 6 + j] : t[kPriorE + k]);
    t[kPriorOJ + e] = v;
  }
  static_assert(kPriorOe == kPriorOJ + 36 && kPriorOe + 6 <= kPriorS, "Omega e follows Omega J");
  __syncwarp();
  for (int e = lane; e < 42; e += 32) {
    const int i = e < 36 ? e / 6 : e - 36, j = e % 6;
    double v = 0.0;
    for (int k = 0; k < 6; ++k) v += J[k * 6 + i] * (e < 36 ? t[kPriorOJ + k * 6 + j] : t[kPriorOe + k]);
    if (e < 36) H[i * D + j] += v;
    else b[i] += v;
  }
  __syncwarp();
}

// ---------------------------------------------------------------------------
// The last block of a job: FP64 sum of the job's partials in tile order (a thread per entry),
// then warp 0 runs ICP_::oneRound / CTICP_::oneRound (kd/icp/icp_impl_.h:72-89,
// kd/cticp/cticp_impl_.h:67-91): Cholesky of H + damping (SPD) and the triangular solves with
// a row per lane in registers, the pose update, the termination test and the float caches
// of the next iteration.

// Phase stamps (clock64) of the last launch, recorded only when profiling is on:
// [0..3] block 0: entry, staged, tile done, partial published; [8..15] tail block:
// entry, partials summed, state staged, solve start, -, solved, updated, done.
__device__ int g_phase_on;
__device__ unsigned long long g_phase[16];
// Error bits of a k_linearize launch whose caller passed no error slot of its own (the
// served loop): 1 = a bounded wait for the tree-top copy gave up and the block read the
// tree from global memory (results valid); 2 = the copy was still not seen complete when
// the block was about to exit (the CUDA context is suspect).
__device__ int g_kernel_error;
// Polls of the first bounded wait for the tree-top copy (kds_set_tma_wait_limit).  The
// wait a block makes before it exits always allows 2^20 polls.
__device__ int g_wait_spins = 1 << 20;

// Bounded wait for the phase with the given parity of an mbarrier to complete.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, int spins = 1 << 20) {
  for (int i = 0; i < spins; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Shared scratch of a job's step, in doubles.
constexpr int kTailH = 0;                           // H, D x D
constexpr int kTailB = 144;                         // b
constexpr int kTailStats = 156;                     // the 7 stats sums
constexpr int kTailX = 164;                         // dx
constexpr int kTailA = 176;                         // Cholesky factor (transposed read)
constexpr int kTailP = 320;                         // 2 x 12: pose products
constexpr int kTailLin = 344;                       // Xf (12), fv (6) of the first fixed entry
constexpr int kTailJob = 362;                       // the job's inputs
constexpr int kTailState = kTailJob + (int)(sizeof(JobIn) / 8);
constexpr int kTailDoubles = kTailState + (int)(sizeof(JobState) / 8);
static_assert(sizeof(JobIn) % 8 == 0 && sizeof(JobState) % 8 == 0, "staged as 8 B words");
static_assert(kTailDoubles <= kWarps * kPStride, "the step's scratch reuses the warps' partials");
static_assert(kTailX + kPriorDoubles <= kTailP, "the prior's scratch is where dx and the factor come later");
static_assert(sizeof(JobIn) / 8 + sizeof(JobState) / 8 + 18 <= kBlock, "one staged word per thread");

// Sum of v(t) over the nt tiles in tile order over four interleaved accumulators; sixteen
// loads in flight.
template <class Load>
__device__ __forceinline__ double sum_tiles(int nt, Load v) {
  double a4[4] = {0.0, 0.0, 0.0, 0.0};
  int t = 0;
  for (; t + 16 <= nt; t += 16) {
    double x[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) x[u] = v(t + u);
#pragma unroll
    for (int u = 0; u < 16; ++u) a4[u & 3] += x[u];
  }
  for (; t + 4 <= nt; t += 4) {
    double x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = v(t + u);
#pragma unroll
    for (int u = 0; u < 4; ++u) a4[u] += x[u];
  }
  for (; t < nt; ++t) a4[0] += v(t);
  return (a4[0] + a4[1]) + (a4[2] + a4[3]);
}
// Entry e of the sums (e >= M: stats value e - M) to its place: H, b and stats in scr, the
// dual blocks in O.  (r, c): entry_rc of e.
template <int KIND>
__device__ __forceinline__ void tail_place(int e, int r, int c, double v, double* scr, JobOut& O) {
  constexpr int DK = KindDim<KIND>::D;
  constexpr int M = DK * (DK + 1) / 2 + DK;
  constexpr int D = KIND == 0 ? 6 : 12;
  if (e >= M) {
    scr[kTailStats + e - M] = v;
  } else if (c == DK) {
    if (r < D) scr[kTailB + r] = v;
    else O.b_vel_B[r - 12] = v;
  } else if (c < D) {
    scr[kTailH + r * D + c] = v;
    scr[kTailH + c * D + r] = v;
  } else {  // dual blocks, c >= 12
    if (r < 6) O.H_cross_pose_vel_B[r * 6 + (c - 12)] = v;
    else if (r < 12) O.H_cross_vel_AB[(r - 6) * 6 + (c - 12)] = v;
    else { O.H_vel_B[(r - 12) * 6 + (c - 12)] = v; O.H_vel_B[(c - 12) * 6 + (r - 12)] = v; }
  }
}

__device__ __forceinline__ kds_stats tail_stats(const double* scr) {
  kds_stats st;
  st.num_inliers = (int32_t)scr[kTailStats + 0];
  st.num_outliers = (int32_t)scr[kTailStats + 1];
  st.num_bad = (int32_t)scr[kTailStats + 2];
  st.num_err_normal = (int32_t)scr[kTailStats + 3];
  st.num_err_fn = (int32_t)scr[kTailStats + 4];
  st.chi2 = (float)scr[kTailStats + 5];
  st.chi2_kernelized = (float)scr[kTailStats + 6];
  st.pert_pose_norm = 0.f;
  st.pert_vel_norm = 0.f;
  return st;
}

// dx = -(H + damping)^-1 b by one warp: Cholesky by columns (right-looking), lane i with row i
// of the lower triangle and y_i of L y = -b, then L^T x = y by column sweeps.  0 where
// H + damping is not positive definite.  One warp's instructions are what it costs, beside the
// chain of a square root, a division and two shared-memory round trips per pivot: a new
// column is read by broadcast (two shuffles per value otherwise), a row shifts down one
// register per pivot so that the pivots are one short loop (unrolled, the code is fetched
// anew every iteration, at twice the time), and entries above the diagonal are worked on
// unmasked and never read.  5,300 cycles for D = 12, 2,500 for D = 6; with the matrix in
// shared memory, element by element, 11,900 and 4,000.
template <int D>
__device__ __forceinline__ void tail_solve(double* scr, float damping, float velocity_damping, int lane) {
  double a[D];  // columns k, k + 1, ... of row `lane` at pivot k
#pragma unroll
  for (int j = 0; j < D; ++j) {
    a[j] = lane < D ? scr[kTailH + lane * D + j] : 0.0;
    if (lane == j) a[j] += j < 6 ? (double)damping : (double)velocity_damping;
  }
  double y = lane < D ? -scr[kTailB + lane] : 0.0;
  double myinv = 0.0;  // 1 / L(lane, lane)
  bool ok = true;
  double* col = scr + kTailA;  // column k of L, below the diagonal
#pragma unroll 1
  for (int k = 0; k < D; ++k, col += D) {
    const double d = __shfl_sync(0xffffffffu, a[0], k);
    ok = ok && (d > 0.0);
    const double lkk = sqrt(fmax(d, 1e-300));
    const double inv = 1.0 / lkk;
    const double l = a[0] * inv;
    if (lane < D) col[lane] = l;
    const double yk = __shfl_sync(0xffffffffu, y * inv, k);
    myinv = lane == k ? inv : myinv;
    y = lane == k ? yk : (lane > k ? y - l * yk : y);
    __syncwarp();
#pragma unroll
    for (int j = 1; j < D; ++j) a[j - 1] = a[j] - l * col[k + j];
  }
#pragma unroll 1
  for (int k = D - 1; k >= 0; --k) {
    const double lt = lane < k ? scr[kTailA + lane * D + k] : 0.0;
    const double xk = __shfl_sync(0xffffffffu, y * myinv, k);
    y = lane == k ? xk : (lane < k ? y - lt * xk : y);
  }
  if (lane < D) scr[kTailX + lane] = ok ? y : 0.0;
  __syncwarp();
}
static_assert(kTailA + 11 * 12 + 22 < kTailDoubles, "a column is read past its end (values never used)");

// Inverse of the pose Xf (shared memory), an element per lane, into iXf.
__device__ __forceinline__ void tail_inverse(const double* Xf, double* iXf, int lane) {
  if (lane < 12) {
    const int i = lane >> 2, j = lane & 3;
    iXf[lane] = j < 3 ? Xf[j * 4 + i] : -ddot3(Xf[i], Xf[4 + i], Xf[8 + i], Xf[3], Xf[7], Xf[11]);
  }
  __syncwarp();
}
// The float caches of one (job, fixed entry) pair at pose X and velocities v (shared memory)
// by one warp: element e of the caches through put(e, value).  Xf, fv, iXf: the entry's.
template <class Put>
__device__ __forceinline__ void tail_caches(const double* X, const double* v, const double* Xf, const double* fv,
                                            const double* iXf, int lane, Put put) {
  if (lane < 12) {
    const int i = lane >> 2, j = lane & 3;
    double m = ddot3(iXf[i * 4], iXf[i * 4 + 1], iXf[i * 4 + 2], X[j], X[4 + j], X[8 + j]);
    if (j == 3) m = da(m, iXf[i * 4 + 3]);
    put(lane, (float)X[lane]);
    put(12 + lane, (float)Xf[lane]);
    put(24 + lane, (float)m);
  } else if (lane < 18) {
    put(36 + lane - 12, (float)v[lane - 12]);
    put(42 + lane - 12, (float)fv[lane - 12]);
  }
  __syncwarp();
}

// A COMPUTE job's step by one warp, from H, b and the stats in scr: solve, update, test, then
// caches() (unless the job is done) and publish() (the state is final), then the outputs.  Jn
// and S are in shared memory.
template <int KIND, class Caches, class Publish>
__device__ __forceinline__ void tail_step(const JobIn& Jn, JobState& S, JobOut& O, kds_stats* log, double* scr,
                                          int lane, Caches caches, Publish publish) {
  constexpr int D = KIND == 0 ? 6 : 12;
  kds_stats st = tail_stats(scr);
  const int it = S.iter;
  if (st.num_inliers + st.num_outliers < Jn.P.min_good_measurements) {
    __syncwarp();
    if (lane == 0) {
      if (log && it < kMaxLog) log[it] = st;
      O.stats = st;
      O.iterations = it + 1;
      S.done = 1;
      S.result = -it;
      O.result = -it;
      S.arrive = 0u;
    }
    __syncwarp();
    publish();
    return;
  }
  if (g_phase_on && lane == 0) g_phase[11] = clock64();
  tail_solve<D>(scr, Jn.P.damping, Jn.P.velocity_damping, lane);
  if (g_phase_on && lane == 0) g_phase[13] = clock64();
  const double* dx = scr + kTailX;
  double pose = 0.0, vel = 0.0;  // this lane's element of the updated state
  if (lane < 12) pose = S.X[lane];
  else if (lane < 18) vel = S.v[lane - 12];
  if (!Jn.stats_mode) {
    // X <- expmap(dx) X, an element per lane
    double R[9];
    rodrigues_d(dx + 3, R);
    if (lane < 12) {
      const int i = lane >> 2, j = lane & 3;
      const double r0 = i == 0 ? R[0] : (i == 1 ? R[3] : R[6]), r1 = i == 0 ? R[1] : (i == 1 ? R[4] : R[7]);
      const double r2 = i == 0 ? R[2] : (i == 1 ? R[5] : R[8]);
      pose = ddot3(r0, r1, r2, S.X[j], S.X[4 + j], S.X[8 + j]);
      if (j == 3) pose = da(pose, dx[i]);
    } else if (D == 12 && lane < 18) {
      vel += dx[6 + lane - 12];
    }
  }
  bool stop = false;
  auto norms = [&]() {
    double pp = 0.0, pv = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) pp += dx[i] * dx[i];
    st.pert_pose_norm = (float)sqrt(pp);
    if (D == 12) {
#pragma unroll
      for (int i = 6; i < D; ++i) pv += dx[i] * dx[i];
      st.pert_vel_norm = (float)sqrt(pv);
    }
  };
  float score = 0.f;
  if (Jn.P.term_crit) {
    norms();
    // ICPTerminationCriteriaScore_::hasToStop (kd/icp/icp_stats_.h:91-101)
    int nl = st.num_inliers + st.num_outliers + st.num_bad + st.num_err_normal + st.num_err_fn;
    float ratio = nl ? (float)st.num_inliers / (float)nl : 0.f;
    score = ratio / (st.chi2_kernelized / (float)st.num_inliers + 1e-6f);
    if (it > 0) {
      bool pert_ok = st.pert_pose_norm < Jn.P.d_pert;
      float dsc = score - S.prev_score;
      bool score_ok = (dsc > 0.f) && ((double)dsc / ((double)S.prev_score + 1e-6) < (double)Jn.P.d_score);
      if (pert_ok && score_ok) stop = true;
    }
  }
  const bool last = it + 1 >= S.max_iter;
  const int result = stop ? it : (last ? Jn.P.max_iterations : S.result);
  __syncwarp();  // the state was read by every lane
  if (lane < 12) S.X[lane] = pose;
  else if (lane < 18) S.v[lane - 12] = vel;
  if (lane == 0) {
    if (Jn.P.term_crit) S.prev_score = score;
    S.iter = it + 1;
    S.result = result;
    if (stop || last) S.done = 1;
    S.arrive = 0u;
  }
  __syncwarp();
  if (!stop && !last) caches();
  publish();
  if (!Jn.P.term_crit) norms();
  if (lane < D) O.dx[lane] = dx[lane];
  if (lane < 12) O.X[lane] = S.X[lane];
  else if (lane < 18) O.v[lane - 12] = S.v[lane - 12];
  if (lane == 0) {
    if (log && it < kMaxLog) log[it] = st;
    O.stats = st;
    O.iterations = it + 1;
    O.result = result;
  }
  if (g_phase_on && lane == 0) g_phase[14] = clock64();
}

// Threads 0..kBlock-1 of the job's last block.
template <int KIND>
__device__ __noinline__ void job_tail(const JobIn& JnG, JobState& SG, JobOut& O, kds_stats* log, LinDev* lins,
                                      const double* partials, double* scr) {
  constexpr int D = KIND == 0 ? 6 : 12;
  const int tid = threadIdx.x, lane = tid & 31;
  const bool stamp = g_phase_on && tid == 0;
  if (stamp) g_phase[8] = clock64();
  // the job's inputs, state and first fixed entry to shared memory, one word per thread,
  // beside the partials' loads
  typedef unsigned long long u64;
  constexpr int NJ = sizeof(JobIn) / 8, NS = sizeof(JobState) / 8;
  u64 word = 0;
  if (tid < NJ) word = reinterpret_cast<const u64*>(&JnG)[tid];
  else if (tid < NJ + NS) word = reinterpret_cast<const u64*>(&SG)[tid - NJ];
  else if (tid < NJ + NS + 12) word = __double_as_longlong(lins[JnG.lin_begin].Xf[tid - NJ - NS]);
  else if (tid < NJ + NS + 18) word = __double_as_longlong(lins[JnG.lin_begin].fv[tid - NJ - NS - 12]);
  {
    constexpr int DK = KindDim<KIND>::D;
    constexpr int M = DK * (DK + 1) / 2 + DK;
    const double* base = partials + (size_t)JnG.tile_begin * kPStride;
    const int nt = JnG.tile_count;
    for (int e = tid; e < M + 7; e += kBlock) {
      int r = 0, c = 0;
      if (e < M) entry_rc(DK, e, r, c);
      const double* src = base + (e < M ? e : kPStats + (e - M));
      tail_place<KIND>(e, r, c, sum_tiles(nt, [&](int t) { return __ldcg(src + (size_t)t * kPStride); }), scr, O);
    }
  }
  u64* dst = reinterpret_cast<u64*>(scr);
  if (tid < NJ + NS) dst[kTailJob + tid] = word;
  else if (tid < NJ + NS + 18) dst[kTailLin + tid - NJ - NS] = word;
  __syncthreads();
  if (stamp) g_phase[9] = g_phase[10] = clock64();
  const JobIn& Jn = *reinterpret_cast<const JobIn*>(scr + kTailJob);
  JobState& S = *reinterpret_cast<JobState*>(scr + kTailState);
  if (Jn.mode != KDS_JOB_COMPUTE) {
    for (int i = tid; i < D * D; i += kBlock) O.H[i] = scr[kTailH + i];
    if (tid < D) O.b[tid] = scr[kTailB + tid];
    if (tid == 0) {
      O.stats = tail_stats(scr);
      O.result = 0;
      O.iterations = 1;
      SG.done = 1;
      SG.arrive = 0u;
    }
    return;
  }
  if (Jn.prior_enabled) {
    if (tid < 32) add_pose_prior(Jn, S.X, scr + kTailH, scr + kTailB, D, scr + kTailX, lane);
    __syncthreads();
  }
  if (tid >= 32) {
    for (int i = tid - 32; i < D * D; i += kBlock - 32) O.H[i] = scr[kTailH + i];
    if (tid - 32 < D) O.b[tid - 32] = scr[kTailB + tid - 32];
    return;
  }
  tail_step<KIND>(Jn, S, O, log, scr, lane, [&]() {
    for (int l = 0; l < Jn.lin_count; ++l) {
      LinDev& L = lins[Jn.lin_begin + l];
      if (l > 0) {
        if (lane < 12) scr[kTailLin + lane] = L.Xf[lane];
        else if (lane < 18) scr[kTailLin + lane] = L.fv[lane - 12];
        __syncwarp();
      }
      float* c = reinterpret_cast<float*>(&L.cache);
      tail_inverse(scr + kTailLin, scr + kTailP, lane);
      tail_caches(S.X, S.v, scr + kTailLin, scr + kTailLin + 12, scr + kTailP, lane,
                  [&](int e, float x) { c[e] = x; });
    }
  }, []() {});
  __syncwarp();
  if (lane < NS) reinterpret_cast<u64*>(&SG)[lane] = reinterpret_cast<const u64*>(&S)[lane];
  if (stamp) g_phase[15] = clock64();
}

// One Gauss-Newton iteration over the tiles [tile0, tile0 + gridDim.x) of one kind.  A descent is
// a chain of dependent node reads, so a launch with tiles for every SM is bound by the blocks
// that an SM holds until it is bound by issue: 8 (64 registers, where the 12-parameter kind
// spills 56 B a thread; the 18-parameter kind spills too much there and takes 6, with 180 B), with the tree top staged as far as shared memory leaves room
// (stage_room).  4,800 tiles, continuous-time / rigid: 116 / 97 us with 2 blocks and 2,047
// nodes, 74 / 59 with 4 and 1,023, 61 / 46 with 6 and 511, 58 / 42 with 8 and 255.
template <int KIND>
constexpr int kLinBlocks = KIND == 2 ? 6 : 8;
__device__ __forceinline__ void report_error(int32_t* err, int bits) { atomicOr(err ? err : &g_kernel_error, bits); }

template <int KIND>
__global__ void __launch_bounds__(kBlock, kLinBlocks<KIND>) k_linearize(const JobIn* __restrict__ jobs, JobState* states, JobOut* outs,
                                                      kds_stats* logs, LinDev* lins, const TileDev* __restrict__ tiles,
                                                      int tile0, int stage, double* partials, int32_t* dbg_match,
                                                      int32_t* dbg_status, int32_t* err) {
  constexpr int D = KindDim<KIND>::D;
  constexpr int M = D * (D + 1) / 2 + D;
  __shared__ CacheF sC;
  __shared__ __align__(16) float sfac[kWarps * (D + 2) * kFacStride];
  __shared__ double swp[kWarps * kPStride];
  __shared__ int s_last;
  __shared__ __align__(8) unsigned long long s_mbar;
  const bool stamp = g_phase_on && blockIdx.x == 0 && threadIdx.x == 0;
  if (stamp) g_phase[0] = clock64();
  const int tile = tile0 + blockIdx.x;
  const TileDev T = tiles[tile];
  JobState& S = states[T.job];
  if (*(volatile int32_t*)&S.done) return;
  const JobIn& Jn = jobs[T.job];
  const LinDev& L = lins[T.lin];
  // Top of the fixed tree: in BFS order the first nodes are the shallowest levels.
  // One thread issues a TMA bulk copy (cp.async.bulk, no multicast) of them into
  // shared memory while the block loads the rest of its inputs.
  extern __shared__ float4 sDyn[];
  const DNode* sN = reinterpret_cast<const DNode*>(sDyn);
  int nst = min(stage, L.f_num_nodes);
  const uint32_t bytes = (uint32_t)nst * (uint32_t)sizeof(DNode);
  const uint32_t mbar = (uint32_t)__cvta_generic_to_shared(&s_mbar);
  if (threadIdx.x == 0 && bytes > 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(sDyn)),
                 "l"(L.fnodes), "r"(bytes), "r"(mbar)
                 : "memory");
  }
  if (threadIdx.x < (int)(sizeof(CacheF) / 4))
    reinterpret_cast<float*>(&sC)[threadIdx.x] = reinterpret_cast<const float*>(&L.cache)[threadIdx.x];
  __syncthreads();
  if (bytes > 0 && !mbar_wait(mbar, 0u, g_wait_spins)) {
    // copy not observed complete: record it and read the whole tree from global memory
    report_error(err, 1);
    nst = 0;
  }
  // Before the block exits, thread 0 waits (bounded) for the copy to land, so that no
  // bulk copy into this block's shared memory outlives the block.
  auto settle = [&]() {
    if (threadIdx.x == 0 && bytes > 0 && !mbar_wait(mbar, 0u)) report_error(err, 2);
  };
  if (stamp) g_phase[1] = clock64();
  tile_body<KIND>(Jn, L, sC, T, sN, nst, swp, sfac, dbg_match, dbg_status);
  __syncthreads();
  if (stamp) g_phase[2] = clock64();
  double* P = partials + (size_t)tile * kPStride;
  for (int k = threadIdx.x; k < kPStride; k += blockDim.x) {
    if (k >= M && k < kPStats) continue;
    double acc = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) acc += swp[w * kPStride + k];
    P[k] = acc;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned prev = atomicAdd(&S.arrive, 1u);
    s_last = (prev == (unsigned)(Jn.tile_count - 1)) ? 1 : 0;
  }
  __syncthreads();
  if (stamp) g_phase[3] = clock64();
  if (!s_last) {
    settle();
    return;
  }
  __threadfence();
  job_tail<KIND>(Jn, S, outs[T.job], logs ? logs + (size_t)T.job * kMaxLog : nullptr, lins, partials, swp);
  settle();
}

// One Gauss-Newton iteration with two tiles per block: the block list pairs consecutive
// tiles of the same (job, fixed entry) (the second index is -1 for a job's odd last
// tile).  Each thread keeps two descents in flight; the partials, the arrival count and
// the job's step are those of k_linearize.
template <int KIND>
__global__ void __launch_bounds__(kBlock, 4) k_linearize_pair(const JobIn* __restrict__ jobs, JobState* states,
                                                           JobOut* outs, kds_stats* logs, LinDev* lins,
                                                           const TileDev* __restrict__ tiles,
                                                           const int2* __restrict__ pairs, int pair0, int stage,
                                                           double* partials, int32_t* dbg_match, int32_t* dbg_status,
                                                           int32_t* err) {
  constexpr int D = KindDim<KIND>::D;
  constexpr int M = D * (D + 1) / 2 + D;
  __shared__ CacheF sC;
  __shared__ __align__(16) float sfac[kWarps * kMaxFac];
  __shared__ double swp[2][kWarps * kPStride];
  __shared__ int s_last;
  __shared__ __align__(8) unsigned long long s_mbar;
  const int2 pr = pairs[pair0 + blockIdx.x];
  const TileDev TA = tiles[pr.x];
  const bool has_b = pr.y >= 0;
  const TileDev TB = has_b ? tiles[pr.y] : TA;
  JobState& S = states[TA.job];
  if (*(volatile int32_t*)&S.done) return;
  const JobIn& Jn = jobs[TA.job];
  const LinDev& L = lins[TA.lin];
  extern __shared__ float4 sDyn[];
  const DNode* sN = reinterpret_cast<const DNode*>(sDyn);
  int nst = min(stage, L.f_num_nodes);
  const uint32_t bytes = (uint32_t)nst * (uint32_t)sizeof(DNode);
  const uint32_t mbar = (uint32_t)__cvta_generic_to_shared(&s_mbar);
  if (threadIdx.x == 0 && bytes > 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(sDyn)),
                 "l"(L.fnodes), "r"(bytes), "r"(mbar)
                 : "memory");
  }
  if (threadIdx.x < (int)(sizeof(CacheF) / 4))
    reinterpret_cast<float*>(&sC)[threadIdx.x] = reinterpret_cast<const float*>(&L.cache)[threadIdx.x];
  __syncthreads();
  if (bytes > 0 && !mbar_wait(mbar, 0u, g_wait_spins)) {
    report_error(err, 1);  // read the whole tree from global memory
    nst = 0;
  }
  auto settle = [&]() {
    if (threadIdx.x == 0 && bytes > 0 && !mbar_wait(mbar, 0u)) report_error(err, 2);
  };
  tile_body_pair<KIND>(Jn, L, sC, TA, TB, has_b, sN, nst, swp[0], swp[1], sfac, dbg_match, dbg_status);
  __syncthreads();
  for (int h = 0; h < (has_b ? 2 : 1); ++h) {
    double* P = partials + (size_t)(h ? pr.y : pr.x) * kPStride;
    for (int k = threadIdx.x; k < kPStride; k += blockDim.x) {
      if (k >= M && k < kPStats) continue;
      double acc = 0.0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) acc += swp[h][w * kPStride + k];
      P[k] = acc;
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned nt = has_b ? 2u : 1u;
    unsigned prev = atomicAdd(&S.arrive, nt);
    s_last = (prev + nt == (unsigned)Jn.tile_count) ? 1 : 0;
  }
  __syncthreads();
  if (!s_last) {
    settle();
    return;
  }
  __threadfence();
  job_tail<KIND>(Jn, S, outs[TA.job], logs ? logs + (size_t)TA.job * kMaxLog : nullptr, lins, partials, swp[0]);
  settle();
}

// ---------------------------------------------------------------------------
// Persistent form of a batch: one launch runs every Gauss-Newton iteration of every job.
// The work items are (iteration, tile) pairs in iteration-major order, handed out by one
// atomic counter (queue[0]).  Before an item of iteration i runs, its job's iteration
// i - 1 must have finished: the last tile of that iteration ran the job's FP64 step and
// then published ready[job] = i (after a fence).  Items are claimed in order, so every
// earlier item belongs to a running block and every wait ends; the waits are bounded all
// the same (an expired wait sets error bit 4 and queue[1], and every later wait gives up
// at once).  A job that has finished skips its remaining items.  The arithmetic of a
// tile and of the step is k_linearize's, so each job's result is bit-identical to the
// per-iteration launches.  A block re-stages the fixed tree's top only when its next tile
// reads another tree.
constexpr int kWaitPolls = 1 << 22;

template <int KIND>
__device__ __forceinline__ void persistent_tile(const JobIn& Jn, const LinDev& L, const CacheF& C, const TileDev& T,
                                                const DNode* staged, int nst, double* swp, float* sfac, double* P) {
  constexpr int D = KindDim<KIND>::D;
  constexpr int M = D * (D + 1) / 2 + D;
  tile_body<KIND>(Jn, L, C, T, staged, nst, swp, sfac, nullptr, nullptr);
  __syncthreads();
  for (int k = threadIdx.x; k < kPStride; k += blockDim.x) {
    if (k >= M && k < kPStats) continue;
    double acc = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) acc += swp[w * kPStride + k];
    P[k] = acc;
  }
}

__global__ void __launch_bounds__(kBlock, 4) k_linearize_persistent(const JobIn* __restrict__ jobs, JobState* states,
                                                                 JobOut* outs, kds_stats* logs, LinDev* lins,
                                                                 const TileDev* __restrict__ tiles, int num_tiles,
                                                                 int max_iter, int stage, double* partials,
                                                                 int32_t* ready, unsigned int* queue, int32_t* err) {
  __shared__ CacheF sC;
  __shared__ __align__(16) float sfac[kWarps * kMaxFac];
  __shared__ double swp[kWarps * kPStride];
  __shared__ int s_item, s_skip, s_last, s_fail;
  __shared__ __align__(8) unsigned long long s_mbar;
  extern __shared__ float4 sDyn[];
  const DNode* sN = reinterpret_cast<const DNode*>(sDyn);
  const uint32_t mbar = (uint32_t)__cvta_generic_to_shared(&s_mbar);
  const DNode* staged_for = nullptr;  // tree whose top is in shared memory
  int nst = 0;                        // nodes staged (0: read global memory)
  uint32_t phase = 0;                 // parity of the next mbarrier phase
  bool copies = false;                // a copy was issued (settle before exit)
  bool fallback = false;              // a wait gave up: read global memory from here on
  const int items = max_iter * num_tiles;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  for (;;) {
    if (threadIdx.x == 0) {
      s_item = (int)atomicAdd(&queue[0], 1u);
      s_fail = 0;
    }
    __syncthreads();
    const int item = s_item;
    if (item >= items) break;
    const int it = item / num_tiles;
    const int tile = item - it * num_tiles;
    const TileDev T = tiles[tile];
    JobState& S = states[T.job];
    if (threadIdx.x == 0) {
      int skip = 0;
      for (int polls = 0;; ++polls) {
        if (*(volatile int32_t*)&S.done) { skip = 1; break; }
        if (*(volatile int32_t*)&ready[T.job] >= it) {
          __threadfence();
          skip = *(volatile int32_t*)&S.done;  // the step that published may have finished the job
          break;
        }
        if (*(volatile unsigned int*)&queue[1]) { skip = 1; break; }
        if (polls >= kWaitPolls) {
          report_error(err, 4);
          atomicExch(&queue[1], 1u);
          skip = 1;
          break;
        }
        __nanosleep(128);
      }
      s_skip = skip;
    }
    __syncthreads();
    if (s_skip) continue;
    const JobIn& Jn = jobs[T.job];
    const LinDev& L = lins[T.lin];
    const int want = fallback ? 0 : min(stage, L.f_num_nodes);
    if (want > 0 && (L.fnodes != staged_for || want != nst)) {
      const uint32_t bytes = (uint32_t)want * (uint32_t)sizeof(DNode);
      if (threadIdx.x == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(sDyn)),
                     "l"(L.fnodes), "r"(bytes), "r"(mbar)
                     : "memory");
      }
      copies = true;
      if (!mbar_wait(mbar, phase, g_wait_spins)) atomicOr(&s_fail, 1);
      phase ^= 1u;
      __syncthreads();  // one block-wide outcome
      if (s_fail) {
        if (threadIdx.x == 0) report_error(err, 1);
        fallback = true;  // the copy may still land: never stage again, settle at exit
        staged_for = nullptr;
        nst = 0;
      } else {
        staged_for = L.fnodes;
        nst = want;
      }
    } else if (want == 0) {
      nst = 0;
      staged_for = nullptr;
    }
    if (threadIdx.x < (int)(sizeof(CacheF) / 4))
      reinterpret_cast<float*>(&sC)[threadIdx.x] = reinterpret_cast<const float*>(&L.cache)[threadIdx.x];
    __syncthreads();
    double* P = partials + (size_t)tile * kPStride;
    const int use = (L.fnodes == staged_for) ? nst : 0;
    if (Jn.kind == 0) persistent_tile<0>(Jn, L, sC, T, sN, use, swp, sfac, P);
    else if (Jn.kind == 1) persistent_tile<1>(Jn, L, sC, T, sN, use, swp, sfac, P);
    else persistent_tile<2>(Jn, L, sC, T, sN, use, swp, sfac, P);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned prev = atomicAdd(&S.arrive, 1u);
      s_last = (prev == (unsigned)(Jn.tile_count - 1)) ? 1 : 0;
    }
    __syncthreads();
    if (s_last) {
      __threadfence();
      kds_stats* log = logs ? logs + (size_t)T.job * kMaxLog : nullptr;
      if (Jn.kind == 0) job_tail<0>(Jn, S, outs[T.job], log, lins, partials, swp);
      else if (Jn.kind == 1) job_tail<1>(Jn, S, outs[T.job], log, lins, partials, swp);
      else job_tail<2>(Jn, S, outs[T.job], log, lins, partials, swp);
      if (threadIdx.x < 32) {  // every lane that wrote the job's state makes it visible, then publish
        __threadfence();
        __syncwarp();
        if (threadIdx.x == 0) atomicExch(&ready[T.job], it + 1);
      }
    }
  }
  if (threadIdx.x == 0 && copies) {
    // the last copy's phase: wait (bounded) until it has landed before the block exits
    if (!mbar_wait(mbar, phase ^ 1u)) report_error(err, 2);
  }
}

// ---------------------------------------------------------------------------
// One alignment in one launch: a thread-block cluster runs every iteration of a single
// COMPUTE job.  A launch per iteration spends as long around the work as on it: the grid's
// start and end, the tree top staged anew, the partials through global memory with a fence
// and a counter (rigid 16 x 1024 scan, 5 tiles: 11.7 us an iteration, of which the tile takes
// 2.3 and the step 2.8).  Here the tree top is staged once per block, a tile's partial goes
// straight into the first block's shared memory, that block's first warp runs the step, and
// the new caches go back into every block's shared memory; two cluster barriers per
// iteration.  Tiles, partials and the step are those of k_linearize, in the same order, so the
// results are bit-identical.  The inputs are the kernel's parameters and the results go to
// page-locked host memory: no copies around the launch.
// Bound by the chain of one iteration (64 x 1024 CT scan on a 1.45M-node map, 23 tiles in 16
// blocks: 29,000 cycles, of which the tile 12,300 and the step's FP64 chain 13,000).
constexpr int kClusterThreads = 512;
constexpr int kClusterGroups = kClusterThreads / kBlock;  // tiles at a time per block, at most
constexpr int kClusterTiles = 64;

// Shared memory of a block: this, then the warps' partials, the tiles' partials (used in the
// first block) and the factor rows.
struct __align__(16) ClusterSmem {
  double scr[kTailDoubles];  // the first block's
  JobOut out;
  alignas(16) float cache[56];  // a CacheF, in whole 16 B words
  kds_stats log[kMaxLog];
  int32_t done, err;
  unsigned long long mbar;
};

template <int KIND>
__global__ void __launch_bounds__(kClusterThreads, 1)
    k_align_cluster(const __grid_constant__ JobIn job, const __grid_constant__ LinDev lin, int stage, ClusterOut* res) {
  constexpr int DK = KindDim<KIND>::D;
  constexpr int D = DK;
  constexpr int M = D * (D + 1) / 2 + D;
  constexpr int kStride = M + 7;
  extern __shared__ float4 sDyn[];
  const DNode* sN = reinterpret_cast<const DNode*>(sDyn);
  ClusterSmem& sm = *reinterpret_cast<ClusterSmem*>(reinterpret_cast<char*>(sDyn) + (size_t)stage * sizeof(DNode));
  double* wpart = reinterpret_cast<double*>(&sm + 1);
  double* part = wpart + (size_t)(blockDim.x / 32) * kStride;  // the first block's: the tiles' partials
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int rank = (int)cluster.block_rank(), nblk = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, group = tid / kBlock, groups = blockDim.x / kBlock;
  const int nt = job.tile_count;
  float* fac = reinterpret_cast<float*>(part + (size_t)((nt + 1) & ~1) * kStride);
  double* lead_part = cluster.map_shared_rank(part, 0);
  ClusterSmem* lead = cluster.map_shared_rank(&sm, 0);
  // the tree top: one bulk copy per block (this GPU's memory, no multicast)
  int nst = min(stage, lin.f_num_nodes);
  const uint32_t bytes = (uint32_t)nst * (uint32_t)sizeof(DNode);
  const uint32_t mbar = (uint32_t)__cvta_generic_to_shared(&sm.mbar);
  if (tid == 0) {
    sm.done = 0;
    sm.err = 0;
    if (bytes > 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(sDyn)),
                   "l"(lin.fnodes), "r"(bytes), "r"(mbar)
                   : "memory");
    }
  }
  // The first block keeps the job's inputs, state, outputs and log in shared memory.  Every
  // block must have started before another writes its shared memory.
  JobIn& Jn = *reinterpret_cast<JobIn*>(sm.scr + kTailJob);
  JobState& S = *reinterpret_cast<JobState*>(sm.scr + kTailState);
  if (rank == 0) {
    typedef unsigned long long u64;
    for (int k = tid; k < (int)(sizeof(JobIn) / 8); k += blockDim.x)
      reinterpret_cast<u64*>(&Jn)[k] = reinterpret_cast<const u64*>(&job)[k];
    for (int k = tid; k < (int)(sizeof(JobOut) / 8); k += blockDim.x) reinterpret_cast<u64*>(&sm.out)[k] = 0ull;
    __syncthreads();
    if (tid < 12) {
      S.X[tid] = sm.out.X[tid] = job.X0[tid];
      sm.scr[kTailLin + tid] = lin.Xf[tid];
    } else if (tid < 18) {
      S.v[tid - 12] = sm.out.v[tid - 12] = job.v0[tid - 12];
      sm.scr[kTailLin + tid] = lin.fv[tid - 12];
    } else if (tid == 18) {
      S.iter = S.done = S.result = 0;
      S.arrive = 0u;
      S.prev_score = 0.f;
      S.max_iter = job.stats_mode ? 1 : job.P.max_iterations;
      sm.out.result = job.P.max_iterations;
    }
  }
  cluster.sync();
  constexpr int kCacheQuads = (int)(sizeof(ClusterSmem::cache) / 16);
  auto caches = [&]() {  // the first block's first warp: the caches into every block
    float* c = sm.cache;
    tail_caches(S.X, S.v, sm.scr + kTailLin, sm.scr + kTailLin + 12, sm.scr + kTailP, lane,
                [&](int e, float x) { c[e] = x; });
    // two blocks at a time, 16 B a lane
    if (lane < 2 * kCacheQuads) {
      float4* q = reinterpret_cast<float4*>(c) + (lane < kCacheQuads ? lane : lane - kCacheQuads);
      const float4 x = *q;
      for (int b = 1 + (lane >= kCacheQuads ? 1 : 0); b < nblk; b += 2) *cluster.map_shared_rank(q, b) = x;
    }
  };
  const CacheF& C = *reinterpret_cast<const CacheF*>(sm.cache);
  static_assert(sizeof(CacheF) <= sizeof(sm.cache), "cache words");
  // the entry of the sums that this thread of the first block adds up
  int er = 0, ec = 0;
  if (tid < M) entry_rc(DK, tid, er, ec);
  if (rank == 0 && tid < 32) {
    tail_inverse(sm.scr + kTailLin, sm.scr + kTailP, lane);
    caches();
  }
  if (bytes > 0 && !mbar_wait(mbar, 0u, g_wait_spins)) {
    // copy not observed complete: record it and read the whole tree from global memory
    atomicOr(&sm.err, 1);
    nst = 0;
  }
  cluster.sync();
  for (;;) {
    for (int t0 = 0; t0 < nt; t0 += nblk * groups) {
      const int t = t0 + group * nblk + rank;
      if (t < nt) {  // uniform per group
        TileDev T;
        T.job = 0;
        T.lin = 0;
        T.leaf_begin = t * kBlock;
        T.leaf_end = min(T.leaf_begin + kBlock, job.m_num_leaves);
        tile_body<KIND, kStride, M>(job, lin, C, T, sN, nst, wpart, fac, nullptr, nullptr);
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(kBlock) : "memory");
        const int e = tid & (kBlock - 1);
        if (e < kStride) {
          double acc = 0.0;
#pragma unroll
          for (int w = 0; w < kWarps; ++w) acc += wpart[(group * kWarps + w) * kStride + e];
          lead_part[t * kStride + e] = acc;
        }
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(kBlock) : "memory");
      }
    }
    cluster.sync();
    if (rank == 0 && tid < kBlock) {
      if (tid < kStride) {
        const double* src = part + tid;
        const double v = sum_tiles(nt, [&](int t) { return src[t * kStride]; });
        tail_place<KIND>(tid, er, ec, v, sm.scr, sm.out);
      }
      asm volatile("bar.sync %0, %1;" ::"r"(1), "r"(kBlock) : "memory");
      if (tid < 32) {
        if (job.prior_enabled) add_pose_prior(Jn, S.X, sm.scr + kTailH, sm.scr + kTailB, D, sm.scr + kTailX, lane);
        tail_step<KIND>(Jn, S, sm.out, sm.log, sm.scr, lane, caches, [&]() {
          if (S.done && lane < nblk) *cluster.map_shared_rank(&sm.done, lane) = 1;
          __syncwarp();
          cluster.barrier_arrive();  // the others go on while this warp writes the outputs
        });
      }
    }
    if (rank != 0 || tid >= 32) cluster.barrier_arrive();
    cluster.barrier_wait();
    if (sm.done) break;
  }
  // before the blocks exit: the copy has landed, the errors are collected
  if (tid == 0) {
    if (bytes > 0 && !mbar_wait(mbar, 0u)) atomicOr(&sm.err, 2);
    if (rank > 0 && sm.err) atomicOr(&lead->err, sm.err);
  }
  cluster.sync();
  if (rank != 0) return;
  for (int i = tid; i < D * D; i += blockDim.x) sm.out.H[i] = sm.scr[kTailH + i];
  if (tid < D) sm.out.b[tid] = sm.scr[kTailB + tid];
  __syncthreads();
  typedef unsigned long long u64;
  static_assert(sizeof(JobOut) % 8 == 0 && sizeof(kds_stats) % 4 == 0, "copied as words");
  for (int k = tid; k < (int)(sizeof(JobOut) / 8); k += blockDim.x)
    reinterpret_cast<u64*>(&res->out)[k] = reinterpret_cast<const u64*>(&sm.out)[k];
  const int nlog = min(sm.out.iterations, kMaxLog) * (int)(sizeof(kds_stats) / 4);
  for (int k = tid; k < nlog; k += blockDim.x)
    reinterpret_cast<int32_t*>(res->log)[k] = reinterpret_cast<const int32_t*>(sm.log)[k];
  if (tid == 0) res->err = sm.err;
}

// Resets control state, seeds state from the job inputs and writes the first caches: a warp
// per job (a thread per job took 7 us for one job, 20 us for 250: every store a sector of its
// own, the pose algebra one element after the other).
constexpr int kInitWarps = 4;
struct InitScratch {
  double X[12], v[6], Xf[12], fv[6], tmp[12];
};
__device__ __forceinline__ void init_job(int j, const JobIn* jobs, JobState* states, JobOut* outs, LinDev* lins,
                                         InitScratch& C, int lane) {
  const JobIn& Jn = jobs[j];
  JobState& S = states[j];
  JobOut& O = outs[j];
  const int max_iter = Jn.stats_mode ? 1 : Jn.P.max_iterations;
  const bool idle = Jn.tile_count == 0 || max_iter <= 0;
  if (lane < 12) {
    C.X[lane] = S.X[lane] = O.X[lane] = Jn.X0[lane];
  } else if (lane < 18) {
    C.v[lane - 12] = S.v[lane - 12] = O.v[lane - 12] = Jn.v0[lane - 12];
  } else if (lane == 18) {
    S.iter = 0;
    S.done = idle ? 1 : 0;
    S.result = 0;
    S.arrive = 0u;
    S.prev_score = 0.f;
    S.max_iter = max_iter;
    O.result = Jn.P.max_iterations;
    O.iterations = 0;
  }
  __syncwarp();
  if (idle) {
    // no moving leaves: the round sees zero measurements and fails at iteration 0
    for (int i = lane; i < 144; i += 32) O.H[i] = 0.0;
    if (lane < 12) O.b[lane] = O.dx[lane] = 0.0;
    if (lane == 0) {
      kds_stats z;
      memset(&z, 0, sizeof(z));
      O.stats = z;
      O.result = (Jn.mode == KDS_JOB_COMPUTE && max_iter > 0 && Jn.P.min_good_measurements > 0) ? 0
                                                                                                : Jn.P.max_iterations;
      if (Jn.mode != KDS_JOB_COMPUTE) O.result = 0;
    }
    return;
  }
  if (Jn.keep_cache) return;
  for (int l = Jn.lin_begin; l < Jn.lin_begin + Jn.lin_count; ++l) {
    LinDev& L = lins[l];
    if (lane < 12) C.Xf[lane] = L.Xf[lane];
    else if (lane < 18) C.fv[lane - 12] = L.fv[lane - 12];
    __syncwarp();
    float* c = reinterpret_cast<float*>(&L.cache);
    tail_inverse(C.Xf, C.tmp, lane);
    tail_caches(C.X, C.v, C.Xf, C.fv, C.tmp, lane, [&](int e, float x) { c[e] = x; });
  }
}

__global__ void __launch_bounds__(32 * kInitWarps) k_init_jobs(const JobIn* jobs, JobState* states, JobOut* outs,
                                                               LinDev* lins, int num_jobs, int32_t* err,
                                                               int32_t* ready = nullptr,
                                                               unsigned int* queue = nullptr) {
  __shared__ InitScratch scratch[kInitWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = blockIdx.x * kInitWarps + w;
  if (j == 0 && lane == 0) {
    if (err) *err = 0;
    if (queue) { queue[0] = 0u; queue[1] = 0u; }
  }
  if (j >= num_jobs) return;
  if (ready && lane == 0) ready[j] = 0;
  init_job(j, jobs, states, outs, lins, scratch[w], lane);
}

// ---------------------------------------------------------------------------
// Traffic model helper: marks every fixed node that the greedy descents visit.
template <int KIND>
__global__ void k_touch(const JobIn* jobs, const LinDev* lins, uint32_t* bitmap) {
  const JobIn& Jn = jobs[0];
  const LinDev& L = lins[Jn.lin_begin];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= Jn.m_num_leaves || L.f_num_nodes <= 0) return;
  const CacheF& C = L.cache;
  float4 md = Jn.m_md[i], nr = Jn.m_nrm[i];
  F3 m = f3(md.x, md.y, md.z), n = f3(nr.x, nr.y, nr.z);
  F3 mw = m, nw = n;
  if (KIND != 0) warp_x(C.v, md.w, m, n, mw, nw);
  F3 q = apply_iso_x(C.Xmf, mw);
  int idx = 0;
  while (idx >= 0) {
    atomicOr(&bitmap[idx >> 5], 1u << (idx & 31));
    DNode nd = load_node(L.fnodes + idx);
    int l = node_left(nd), r = node_right(nd);
    if (l < 0 && r < 0) break;
    idx = dot3x(node_dir(nd), sub3x(q, node_mean(nd))) > 0.0f ? l : r;
  }
}
__global__ void k_popc(const uint32_t* bitmap, int64_t words, unsigned long long* count) {
  unsigned long long c = 0;
  for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < words; w += (int64_t)gridDim.x * blockDim.x)
    c += __popc(bitmap[w]);
  atomicAdd(count, c);
}

int count_touched(Runner& R, int kind, int64_t fixed_nodes, int64_t* out, cudaStream_t s) {
  *out = 0;
  if (R.num_jobs < 1 || fixed_nodes <= 0) return KDS_OK;
  k_init_jobs<<<1, 32 * kInitWarps, 0, s>>>(R.d_jobs, R.d_states, R.d_outs, R.d_lins, 1, R.d_err); ::kds::count_launch();
  int64_t words = (fixed_nodes + 31) / 32;
  uint32_t* bm = nullptr;
  unsigned long long* cnt = nullptr;
  KDS_CK(cudaMalloc(&bm, words * 4 + 64));
  cnt = reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(bm) + ((words * 4 + 7) & ~7ll));
  cudaMemsetAsync(bm, 0, words * 4 + 64, s);
  int nl = R.h_jobs[0].m_num_leaves;
  int g = (nl + 255) / 256;
  if (g > 0) {
    if (kind == 0) k_touch<0><<<g, 256, 0, s>>>(R.d_jobs, R.d_lins, bm);
    else k_touch<1><<<g, 256, 0, s>>>(R.d_jobs, R.d_lins, bm);
    ::kds::count_launch();
  }
  k_popc<<<64, 256, 0, s>>>(bm, words, cnt); ::kds::count_launch();
  unsigned long long h = 0;
  cudaMemcpyAsync(&h, cnt, 8, cudaMemcpyDeviceToHost, s);
  cudaError_t e = cudaStreamSynchronize(s);
  cudaFree(bm);
  if (e != cudaSuccess) return cuda_status(e, "count_touched", __FILE__, __LINE__);
  *out = (int64_t)h;
  return KDS_OK;
}

// ---------------------------------------------------------------------------
// Host runner
int Runner::reserve(int nj, int nl, int nt) {
  if (nj <= cap_jobs && nl <= cap_lins && nt <= cap_tiles) return KDS_OK;
  // grow by at least half of the old capacity: callers whose job sets vary from call to
  // call (a tracker's frames, served ticks) reallocate -- a device-wide synchronisation in
  // cudaFree -- a logarithmic number of times instead of at every new maximum
  const int oj = cap_jobs, ol = cap_lins, ot = cap_tiles;
  release();
  cap_jobs = std::max({nj, oj + oj / 2, 1});
  cap_lins = std::max({nl, ol + ol / 2, 1});
  cap_tiles = std::max({nt, ot + ot / 2, 1});
  size_t bytes = sizeof(JobIn) * cap_jobs + sizeof(JobState) * cap_jobs + sizeof(JobOut) * cap_jobs +
                 sizeof(kds_stats) * kMaxLog * cap_jobs + sizeof(LinDev) * cap_lins + sizeof(TileDev) * cap_tiles +
                 sizeof(double) * kPStride * cap_tiles + sizeof(int32_t) * cap_jobs + sizeof(int2) * cap_tiles +
                 12 * 256;
  cudaError_t e = cudaMalloc(&block, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    block = nullptr;
    cap_jobs = cap_lins = cap_tiles = 0;
    set_error("cudaMalloc of %zu bytes for the aligner workspace failed", bytes);
    return KDS_ERR_OOM;
  }
  char* p = (char*)block;
  auto carve = [&](size_t sz) {
    char* r = p;
    p += (sz + 255) & ~(size_t)255;
    return (void*)r;
  };
  d_jobs = (JobIn*)carve(sizeof(JobIn) * cap_jobs);
  d_states = (JobState*)carve(sizeof(JobState) * cap_jobs);
  d_outs = (JobOut*)carve(sizeof(JobOut) * cap_jobs);
  d_logs = (kds_stats*)carve(sizeof(kds_stats) * kMaxLog * cap_jobs);
  d_lins = (LinDev*)carve(sizeof(LinDev) * cap_lins);
  d_tiles = (TileDev*)carve(sizeof(TileDev) * cap_tiles);
  d_partials = (double*)carve(sizeof(double) * kPStride * cap_tiles);
  d_err = (int32_t*)carve(sizeof(int32_t));
  d_ready = (int32_t*)carve(sizeof(int32_t) * cap_jobs);
  d_queue = (unsigned int*)carve(2 * sizeof(unsigned int));
  d_pairs = (int2*)carve(sizeof(int2) * cap_tiles);
  return KDS_OK;
}

void Runner::release() {
  drop_graph();
  for (cudaEvent_t e : prof_ev) cudaEventDestroy(e);
  prof_ev.clear();
  if (block) cudaFree(block);
  block = nullptr;
  cap_jobs = cap_lins = cap_tiles = 0;
}

Runner::~Runner() {
  release();
  if (h_cluster) cudaFreeHost(h_cluster);
  for (cudaEvent_t e : fork_ev)
    if (e) cudaEventDestroy(e);
  if (side) cudaStreamDestroy(side);
}

// The second stream and its events, at the priority of s; false where they can't be had.
bool Runner::side_ready(cudaStream_t s) {
  int prio = 0;
  bool ok = cudaStreamGetPriority(s, &prio) == cudaSuccess;
  if (ok && side && prio != side_priority) {
    cudaStreamDestroy(side);  // the work on it was joined, and keeps its resources until it is done
    side = nullptr;
  }
  if (ok && !side) {
    ok = cudaStreamCreateWithPriority(&side, cudaStreamNonBlocking, prio) == cudaSuccess;
    if (!ok) side = nullptr;
    side_priority = prio;
  }
  for (cudaEvent_t& e : fork_ev)
    if (ok && !e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
      e = nullptr;
      ok = false;
    }
  if (!ok) cudaGetLastError();
  return ok;
}

void Runner::drop_graph() {
  if (gexec) cudaGraphExecDestroy(gexec);
  if (graph) cudaGraphDestroy(graph);
  gexec = nullptr;
  graph = nullptr;
  graph_key.clear();
}

// Builds the tile list and device inputs for `jobs` (host descriptions).
int Runner::setup(const std::vector<JobIn>& jobs_in, const std::vector<LinDev>& lins_in, cudaStream_t s) {
  h_jobs = jobs_in;
  h_lins = lins_in;
  h_tiles.clear();
  std::vector<int> order(h_jobs.size());
  for (size_t j = 0; j < order.size(); ++j) order[j] = (int)j;
  if (order_by_size)
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return h_jobs[a].m_num_leaves > h_jobs[b].m_num_leaves; });
  for (int kind = 0; kind < 3; ++kind) {
    kind_begin[kind] = (int)h_tiles.size();
    for (int j : order) {
      JobIn& Jn = h_jobs[j];
      if (Jn.kind != kind) continue;
      Jn.tile_begin = (int32_t)h_tiles.size();
      for (int l = Jn.lin_begin; l < Jn.lin_begin + Jn.lin_count; ++l) {
        for (int b = 0; b < Jn.m_num_leaves; b += kBlock) {
          TileDev t;
          t.job = (int32_t)j;
          t.lin = l;
          t.leaf_begin = b;
          t.leaf_end = std::min(b + kBlock, Jn.m_num_leaves);
          h_tiles.push_back(t);
        }
      }
      Jn.tile_count = (int32_t)h_tiles.size() - Jn.tile_begin;
    }
    kind_count[kind] = (int)h_tiles.size() - kind_begin[kind];
  }
  // blocks of two consecutive tiles of one (job, fixed entry), per kind
  h_pairs.clear();
  for (int kind = 0; kind < 3; ++kind) {
    kind_pair_begin[kind] = (int)h_pairs.size();
    const int e = kind_begin[kind] + kind_count[kind];
    for (int t = kind_begin[kind]; t < e;) {
      const bool two = t + 1 < e && h_tiles[t + 1].job == h_tiles[t].job && h_tiles[t + 1].lin == h_tiles[t].lin;
      h_pairs.push_back(make_int2(t, two ? t + 1 : -1));
      t += two ? 2 : 1;
    }
    kind_pair_count[kind] = (int)h_pairs.size() - kind_pair_begin[kind];
  }
  int rc = reserve((int)h_jobs.size(), (int)h_lins.size(), (int)h_tiles.size());
  if (rc) return rc;
  num_jobs = (int)h_jobs.size();
  num_tiles = (int)h_tiles.size();
  KDS_CK(cudaMemcpyAsync(d_jobs, h_jobs.data(), sizeof(JobIn) * h_jobs.size(), cudaMemcpyHostToDevice, s));
  KDS_CK(cudaMemcpyAsync(d_lins, h_lins.data(), sizeof(LinDev) * h_lins.size(), cudaMemcpyHostToDevice, s));
  if (num_tiles) {
    KDS_CK(cudaMemcpyAsync(d_tiles, h_tiles.data(), sizeof(TileDev) * h_tiles.size(), cudaMemcpyHostToDevice, s));
    if (pair_tiles) KDS_CK(cudaMemcpyAsync(d_pairs, h_pairs.data(), sizeof(int2) * h_pairs.size(), cudaMemcpyHostToDevice, s));
  }
  return KDS_OK;
}

int Runner::max_launches(int kind) const {
  int m = 0;
  for (const JobIn& J : h_jobs) {
    if (kind >= 0 && J.kind != kind) continue;
    int it = (J.mode == KDS_JOB_COMPUTE) ? (J.stats_mode ? 1 : J.P.max_iterations) : 1;
    m = std::max(m, it);
  }
  return m;
}

int phase_stamps(int on, unsigned long long* out16) {
  if (on >= 0) KDS_CK(cudaMemcpyToSymbol(g_phase_on, &on, sizeof(int)));
  if (out16) KDS_CK(cudaMemcpyFromSymbol(out16, g_phase, sizeof(unsigned long long) * 16));
  return KDS_OK;
}

int set_wait_spins(int32_t spins) {
  if (spins < 0) { set_error("kds_set_tma_wait_limit: negative limit %d", spins); return KDS_ERR_INVALID_ARG; }
  KDS_CK(cudaMemcpyToSymbol(g_wait_spins, &spins, sizeof(int32_t)));
  return KDS_OK;
}

int Runner::ensure_events(int n) {
  while ((int)prof_ev.size() < n) {
    cudaEvent_t e;
    KDS_CK(cudaEventCreate(&e));
    prof_ev.push_back(e);
  }
  return KDS_OK;
}

double Runner::profile_mean_ms(int* launches) const {
  double sum = 0.0;
  int n = 0;
  for (int i = 0; i < prof_launches; ++i) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, prof_ev[2 * i], prof_ev[2 * i + 1]) == cudaSuccess) {
      sum += ms;
      ++n;
    } else {
      cudaGetLastError();
    }
  }
  if (launches) *launches = n;
  return n ? sum / n : 0.0;
}

// A profiling event on s: inside a stream capture it becomes an external event node of
// the graph (recorded at every replay); outside one it is a plain record.
static cudaError_t record_profile_event(cudaEvent_t e, cudaStream_t s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaError_t r = cudaStreamIsCapturing(s, &cs);
  if (r != cudaSuccess) return r;
  return cs == cudaStreamCaptureStatusActive ? cudaEventRecordWithFlags(e, s, cudaEventRecordExternal)
                                             : cudaEventRecord(e, s);
}

// Blocks of the persistent kernel: every SM full at its occupancy for `smem` bytes of
// dynamic shared memory, at most one block per work item.
static int persistent_grid(size_t smem, int64_t items) {
  int nsm = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm <= 0)
    nsm = 148;
  int per = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_linearize_persistent, kBlock, smem) != cudaSuccess ||
      per < 1) {
    cudaGetLastError();
    per = 1;
  }
  return (int)std::max<int64_t>(1, std::min<int64_t>(items, (int64_t)nsm * per));
}

// Tree-top nodes that each block of a launch stages, `limit` at most: as many complete levels as
// fit the share of an SM's shared memory that is left to each of the blocks it will hold (of
// fixed_bytes of their own).  One or two blocks per SM stage 2,047 nodes, 3 and 4 1,023; more
// hide the reads of the lower levels better than a staged top saves them (figures at
// k_linearize).
static int stage_room(int limit, int blocks, int most_blocks, size_t fixed_bytes) {
  int nsm = 0, dev = 0, smem = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm <= 0 ||
      cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess || smem <= 0) {
    cudaGetLastError();
    nsm = 148;
    smem = 228 * 1024;
  }
  const int per = std::min(most_blocks, (blocks + nsm - 1) / nsm);
  const size_t share = (size_t)smem / (size_t)std::max(1, per), own = fixed_bytes + 1024;  // 1 KB: the system's
  int n = 2047;
  while (n > 0 && n * sizeof(DNode) + own > share) n >>= 1;
  return std::min(limit, n);
}

// Static shared memory of a block: the pose cache, the leaves' factors, the warps' partials.
template <int KIND>
static constexpr size_t lin_bytes() {
  return sizeof(CacheF) + sizeof(float) * kWarps * (KindDim<KIND>::D + 2) * kFacStride +
         sizeof(double) * kWarps * kPStride + 64;
}
constexpr size_t kPairBytes = sizeof(CacheF) + sizeof(float) * kWarps * kMaxFac + sizeof(double) * 2 * kWarps * kPStride + 64;

// One iteration's launch of one kind.
template <int KIND>
void Runner::enqueue_kind(cudaStream_t s, int32_t* dbg_match, int32_t* dbg_status) {
  if (pair_tiles) {
    const int nb = kind_pair_count[KIND], stage = stage_room(stage_nodes, nb, 4, kPairBytes);
    k_linearize_pair<KIND><<<nb, kBlock, stage * sizeof(DNode), s>>>(d_jobs, d_states, d_outs, d_logs, d_lins, d_tiles,
                                                                     d_pairs, kind_pair_begin[KIND], stage, d_partials,
                                                                     dbg_match, dbg_status, d_err);
  } else {
    const int nb = kind_count[KIND], stage = stage_room(stage_nodes, nb, kLinBlocks<KIND>, lin_bytes<KIND>());
    k_linearize<KIND><<<nb, kBlock, stage * sizeof(DNode), s>>>(d_jobs, d_states, d_outs, d_logs, d_lins, d_tiles,
                                                                kind_begin[KIND], stage, d_partials, dbg_match,
                                                                dbg_status, d_err);
  }
  ::kds::count_launch();
}

int Runner::enqueue(cudaStream_t s, int32_t* dbg_match, int32_t* dbg_status) {
  if (num_jobs == 0) return KDS_OK;
  if (persistent && !dbg_match) {
    k_init_jobs<<<(num_jobs + kInitWarps - 1) / kInitWarps, 32 * kInitWarps, 0, s>>>(
        d_jobs, d_states, d_outs, d_lins, num_jobs, d_err, d_ready, d_queue);
    ::kds::count_launch();
    const int L = max_launches();
    prof_launches = profiling ? 1 : 0;
    if (profiling) {
      int rc = ensure_events(2);
      if (rc) return rc;
    }
    const size_t stage_bytes = (size_t)stage_nodes * sizeof(DNode);
    if (!persistent_attr_set) {
      KDS_CK(cudaFuncSetAttribute((const void*)k_linearize_persistent, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  200 * 1024));
      persistent_attr_set = true;
    }
    if (num_tiles > 0 && L > 0) {
      const int grid = persistent_grid(stage_bytes, (int64_t)num_tiles * L);
      if (profiling) KDS_CK(record_profile_event(prof_ev[0], s));
      k_linearize_persistent<<<grid, kBlock, stage_bytes, s>>>(d_jobs, d_states, d_outs, d_logs, d_lins, d_tiles,
                                                               num_tiles, L, stage_nodes, d_partials, d_ready,
                                                               d_queue, d_err);
      ::kds::count_launch();
      if (profiling) KDS_CK(record_profile_event(prof_ev[1], s));
    }
    KDS_CK(cudaGetLastError());
    return KDS_OK;
  }
  k_init_jobs<<<(num_jobs + kInitWarps - 1) / kInitWarps, 32 * kInitWarps, 0, s>>>(d_jobs, d_states, d_outs, d_lins,
                                                                                   num_jobs, d_err);
  ::kds::count_launch();
  // each kind for the iterations its own jobs can take
  int L[3], nmax = 0, total = 0;
  for (int kind = 0; kind < 3; ++kind) {
    L[kind] = kind_count[kind] ? max_launches(kind) : 0;
    nmax = std::max(nmax, L[kind]);
    total += L[kind];
  }
  prof_launches = profiling ? total : 0;
  if (profiling) {
    int rc = ensure_events(2 * prof_launches);
    if (rc) return rc;
  }
  int ev = 0;
  if (stage_nodes > 0 && !smem_attr_set) {  // static + dynamic shared memory can pass 48 KB
    const void* fs[6] = {(const void*)k_linearize<0>, (const void*)k_linearize<1>, (const void*)k_linearize<2>,
                         (const void*)k_linearize_pair<0>, (const void*)k_linearize_pair<1>,
                         (const void*)k_linearize_pair<2>};
    for (int k = 0; k < 6; ++k) KDS_CK(cudaFuncSetAttribute(fs[k], cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    smem_attr_set = true;
  }
  // The kinds' jobs don't depend on each other: the first kind's iterations run on s, the others'
  // beside them, so that one kind's blocks fill the SMs where the other's last tiles and solves
  // run (a batch of 125 pairs of each kind: 1,735 us one after the other, 1,455 side by side).
  // In order where each launch is timed, for one launch a kind (62 us of kernels give less than
  // the stream costs to create), and where there is no second stream.
  const int first = L[0] ? 0 : (L[1] ? 1 : 2);
  const bool fork = !profiling && total > L[first] && nmax > 1 && side_ready(s);
  if (fork) {
    KDS_CK(cudaEventRecord(fork_ev[0], s));
    KDS_CK(cudaStreamWaitEvent(side, fork_ev[0], 0));
  }
  for (int i = 0; i < nmax; ++i) {
    for (int kind = 0; kind < 3; ++kind) {
      if (i >= L[kind]) continue;
      if (profiling) KDS_CK(record_profile_event(prof_ev[ev++], s));
      const cudaStream_t ks = fork && kind != first ? side : s;
      if (kind == 0) enqueue_kind<0>(ks, dbg_match, dbg_status);
      else if (kind == 1) enqueue_kind<1>(ks, dbg_match, dbg_status);
      else enqueue_kind<2>(ks, dbg_match, dbg_status);
      if (profiling) KDS_CK(record_profile_event(prof_ev[ev++], s));
    }
  }
  const cudaError_t le = cudaGetLastError();
  if (fork) {  // joined also after a failed launch: what did start still uses the batch's buffers
    KDS_CK(cudaEventRecord(fork_ev[1], side));
    KDS_CK(cudaStreamWaitEvent(s, fork_ev[1], 0));
  }
  KDS_CK(le);
  return KDS_OK;
}

// Whether a job runs as one cluster launch: a COMPUTE job of one fixed entry whose tiles fit
// the first block's partials, and no per-launch events asked for.  Against a 1.55M-node map,
// rigid / CT: 128 / 221 us at 1,024 surfels (a launch per iteration: 176 / 295), 140 / 272 at
// 8,192 (188 / 321); beside other streams' work the launches wait once each, the cluster once.
// There the partials end and the blocks begin a second round of tiles,
// while a launch per iteration still has SMs to spare.
bool cluster_fits(const JobIn& J, bool profiling) {
  return !profiling && J.mode == KDS_JOB_COMPUTE && (J.kind == 0 || J.kind == 1) && J.lin_count == 1 &&
         !J.keep_cache && J.m_num_leaves > 0 && J.m_num_leaves <= kClusterTiles * kBlock &&
         (J.stats_mode || J.P.max_iterations > 0);
}

template <int KIND>
static cudaError_t launch_cluster(const JobIn& J, const LinDev& L, int stage, int max_blocks, ClusterOut* res,
                          cudaStream_t s) {
  // as many blocks as tiles, up to the largest cluster that the device schedules: fewer warps
  // per SM to share its issue slots, and more of its L1 per tile for the lower tree levels
  int nblk = 1;
  while (nblk < max_blocks && nblk < J.tile_count) nblk *= 2;
  const int groups = std::min(kClusterGroups, (J.tile_count + nblk - 1) / nblk);
  const int kStride = KIND == 0 ? 34 : 97;
  const size_t smem = (size_t)stage * sizeof(DNode) + sizeof(ClusterSmem) +
                      sizeof(double) * kStride * ((size_t)groups * kWarps + ((J.tile_count + 1) & ~1)) +
                      sizeof(float) * ((KIND == 0 ? 6 : 12) + 2) * kFacStride * groups * kWarps;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nblk);
  cfg.blockDim = dim3((unsigned)(groups * kBlock));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)nblk;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_align_cluster<KIND>, J, L, stage, res);
  if (e == cudaSuccess) count_launch();
  return e;
}

// Sets the cluster kernels' limits (always to the same values: they belong to the process) and
// asks for the largest cluster that this device schedules; 0 for none.
constexpr int kClusterSmemMax = 200 * 1024;  // 172 KB at 64 CT tiles and 2,047 staged nodes
static int cluster_setup() {
  const void* fs[2] = {(const void*)k_align_cluster<0>, (const void*)k_align_cluster<1>};
  for (const void* f : fs)
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kClusterSmemMax) != cudaSuccess ||
        cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
  return largest_cluster([](int blocks) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = kClusterSmemMax;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_align_cluster<1>, &cfg) == cudaSuccess) return n > 0;
    cudaGetLastError();
    return false;
  });
}

bool Runner::cluster_ready() {
  if (cluster_blocks >= 0) return cluster_blocks > 0;
  cluster_blocks = cluster_setup();
  if (cluster_blocks == 0) return false;
  if (cudaHostAlloc((void**)&h_cluster, sizeof(ClusterOut), cudaHostAllocMapped) != cudaSuccess ||
      cudaHostGetDevicePointer((void**)&d_cluster, h_cluster, 0) != cudaSuccess) {
    cudaGetLastError();
    cluster_blocks = 0;
    return false;
  }
  memset(h_cluster, 0, sizeof(ClusterOut));
  return true;
}

bool Runner::run_cluster(JobIn J, const LinDev& L, cudaStream_t s, JobOut* out, std::vector<kds_stats>* log, int* rc) {
  if (!cluster_ready()) return false;
  J.tile_begin = 0;
  J.tile_count = (J.m_num_leaves + kBlock - 1) / kBlock;
  J.lin_begin = 0;
  cudaError_t e = J.kind == 0 ? launch_cluster<0>(J, L, stage_nodes, cluster_blocks, d_cluster, s)
                              : launch_cluster<1>(J, L, stage_nodes, cluster_blocks, d_cluster, s);
  if (e != cudaSuccess) {  // not started; an error of the device itself comes back with the next call
    cudaGetLastError();
    return false;
  }
  e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    *rc = cuda_status(e, "single alignment", __FILE__, __LINE__);
    return true;
  }
  *out = h_cluster->out;
  if (log) log->assign(h_cluster->log, h_cluster->log + kMaxLog);
  *rc = timeout_status(h_cluster->err);
  return true;
}

int Runner::run(cudaStream_t s, bool use_graph, int32_t* dbg_match, int32_t* dbg_status) {
  if (!use_graph || dbg_match) return enqueue(s, dbg_match, dbg_status);
  // graph key: everything the captured launches depend on
  std::vector<int64_t> key;
  key.push_back((int64_t)(uintptr_t)block);
  key.push_back(num_jobs);
  key.push_back(num_tiles);
  for (int k = 0; k < 3; ++k) { key.push_back(kind_begin[k]); key.push_back(kind_count[k]); key.push_back(max_launches(k)); }
  key.push_back(profiling ? 1 : 0);
  key.push_back(stage_nodes);
  key.push_back(order_by_size);
  key.push_back(persistent);
  key.push_back(pair_tiles);
  // two tiles per block: a kind's blocks are not determined by its tiles (3 + 1 tiles of two jobs
  // make three, 2 + 2 make two)
  if (pair_tiles)
    for (int k = 0; k < 3; ++k) { key.push_back(kind_pair_begin[k]); key.push_back(kind_pair_count[k]); }
  if (key != graph_key) {
    // capture only a shape that repeats: a one-off shape (every call of a stream of
    // different scans) costs less launched directly than captured and instantiated
    if (key != last_key) {
      last_key = key;
      return enqueue(s, nullptr, nullptr);
    }
    drop_graph();
    cudaStream_t cs;
    KDS_CK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
    int rc = KDS_OK;
    if (e == cudaSuccess) {
      rc = enqueue(cs, nullptr, nullptr);
      e = cudaStreamEndCapture(cs, &graph);
    }
    cudaStreamDestroy(cs);
    if (e != cudaSuccess || rc) {
      graph = nullptr;
      return rc ? rc : cuda_status(e, "graph capture", __FILE__, __LINE__);
    }
    KDS_CK(cudaGraphInstantiate(&gexec, graph, 0));
    graph_key = key;
  }
  KDS_CK(cudaGraphLaunch(gexec, s));
  return KDS_OK;
}

int Runner::fetch(cudaStream_t s, std::vector<JobOut>& outs, std::vector<kds_stats>* logs) {
  outs.resize(num_jobs);
  if (num_jobs == 0) return KDS_OK;
  KDS_CK(cudaMemcpyAsync(outs.data(), d_outs, sizeof(JobOut) * num_jobs, cudaMemcpyDeviceToHost, s));
  if (logs) {
    logs->resize((size_t)num_jobs * kMaxLog);
    KDS_CK(cudaMemcpyAsync(logs->data(), d_logs, sizeof(kds_stats) * kMaxLog * num_jobs, cudaMemcpyDeviceToHost, s));
  }
  int32_t err = 0;
  KDS_CK(cudaMemcpyAsync(&err, d_err, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  KDS_CK(cudaStreamSynchronize(s));
  return timeout_status(err);
}

// KDS_OK, or KDS_ERR_TIMEOUT with a message for the error bits of a launch sequence.
int timeout_status(int32_t err) {
  if (!err) return KDS_OK;
  if (err & 2)
    set_error("a bounded wait for a tree-top copy gave up and the copy was still not seen complete when its block "
              "exited: the results were computed from global memory, but the CUDA context should be considered "
              "unusable");
  else
    set_error("a bounded wait for a tree-top copy gave up; the results were computed from global memory and are "
              "valid");
  return KDS_ERR_TIMEOUT;
}

// ---------------------------------------------------------------------------
// Served-loop helpers (kds_serve.cu): jobs addressed by slot.
namespace {

__global__ void __launch_bounds__(32 * kInitWarps) k_admit_slots(const int32_t* slots, int n, const JobIn* new_jobs,
                                                                 const LinDev* new_lins, JobIn* jobs,
                                                                 JobState* states, JobOut* outs, LinDev* lins) {
  __shared__ InitScratch scratch[kInitWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = blockIdx.x * kInitWarps + w;
  if (i >= n) return;
  const int slot = slots[i];
  typedef unsigned long long u64;
  static_assert(sizeof(LinDev) % 8 == 0, "copied as 8 B words");
  for (int k = lane; k < (int)(sizeof(JobIn) / 8); k += 32)
    reinterpret_cast<u64*>(jobs + slot)[k] = reinterpret_cast<const u64*>(new_jobs + i)[k];
  for (int k = lane; k < (int)(sizeof(LinDev) / 8); k += 32)
    reinterpret_cast<u64*>(lins + slot)[k] = reinterpret_cast<const u64*>(new_lins + i)[k];
  __syncwarp();
  init_job(slot, jobs, states, outs, lins, scratch[w], lane);
}

__global__ void k_collect(int n, const JobState* states, const JobOut* outs, const unsigned long long* touched,
                          SlotResult* res) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int done = *(const volatile int32_t*)&states[j].done;
  res[j].done = done;
  if (!done) return;
  res[j].touched = touched ? touched[j] : 0ull;
  const JobOut& O = outs[j];
  res[j].result = O.result;
  res[j].iterations = O.iterations;
  res[j].stats = O.stats;
  for (int k = 0; k < 12; ++k) res[j].X[k] = O.X[k];
  for (int k = 0; k < 6; ++k) res[j].v[k] = O.v[k];
}

}  // namespace

static_assert(kBlock == kTileSurfels, "tile size");

int linearize_smem_setup() {
  const int bytes = kStageNodes * (int)sizeof(DNode);
  KDS_CK(cudaFuncSetAttribute((const void*)k_linearize<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  KDS_CK(cudaFuncSetAttribute((const void*)k_linearize<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  KDS_CK(cudaFuncSetAttribute((const void*)k_linearize<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  KDS_CK(cudaFuncSetAttribute((const void*)k_linearize_pair<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  KDS_CK(cudaFuncSetAttribute((const void*)k_linearize_pair<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  KDS_CK(cudaFuncSetAttribute((const void*)k_linearize_pair<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  return KDS_OK;
}

int launch_admit_slots(const int32_t* d_slots, int n, const JobIn* new_jobs, const LinDev* new_lins, JobIn* jobs,
                       JobState* states, JobOut* outs, LinDev* lins, cudaStream_t s) {
  if (n <= 0) return KDS_OK;
  k_admit_slots<<<(n + kInitWarps - 1) / kInitWarps, 32 * kInitWarps, 0, s>>>(d_slots, n, new_jobs, new_lins, jobs, states, outs, lins);
  count_launch();
  KDS_CK(cudaGetLastError());
  return KDS_OK;
}

int launch_linearize_pairs(int kind, int npairs, const JobIn* jobs, JobState* states, JobOut* outs, LinDev* lins,
                           const TileDev* tiles, const int2* pairs, double* partials, cudaStream_t s) {
  if (npairs <= 0) return KDS_OK;
  const size_t stage_bytes = (size_t)kServeStage * sizeof(DNode);
  if (kind == 0)
    k_linearize_pair<0><<<npairs, kBlock, stage_bytes, s>>>(jobs, states, outs, nullptr, lins, tiles, pairs, 0,
                                                            kServeStage, partials, nullptr, nullptr, nullptr);
  else if (kind == 1)
    k_linearize_pair<1><<<npairs, kBlock, stage_bytes, s>>>(jobs, states, outs, nullptr, lins, tiles, pairs, 0,
                                                            kServeStage, partials, nullptr, nullptr, nullptr);
  else
    k_linearize_pair<2><<<npairs, kBlock, stage_bytes, s>>>(jobs, states, outs, nullptr, lins, tiles, pairs, 0,
                                                            kServeStage, partials, nullptr, nullptr, nullptr);
  count_launch();
  KDS_CK(cudaGetLastError());
  return KDS_OK;
}

int launch_collect(int n, const JobState* states, const JobOut* outs, const unsigned long long* touched,
                   SlotResult* res, cudaStream_t s) {
  if (n <= 0) return KDS_OK;
  k_collect<<<(n + 127) / 128, 128, 0, s>>>(n, states, outs, touched, res);
  count_launch();
  KDS_CK(cudaGetLastError());
  return KDS_OK;
}

int launch_touch(int kind, const JobIn* jobs, const LinDev* lins, int slot, int num_leaves, uint32_t* bitmap,
                 int64_t words, unsigned long long* count, cudaStream_t s) {
  KDS_CK(cudaMemsetAsync(bitmap, 0, (size_t)words * 4, s));
  KDS_CK(cudaMemsetAsync(count, 0, sizeof(unsigned long long), s));
  const int g = (num_leaves + 255) / 256;
  if (g > 0) {
    if (kind == 0) k_touch<0><<<g, 256, 0, s>>>(jobs + slot, lins, bitmap);
    else k_touch<1><<<g, 256, 0, s>>>(jobs + slot, lins, bitmap);
    count_launch();
  }
  k_popc<<<64, 256, 0, s>>>(bitmap, words, count);
  count_launch();
  KDS_CK(cudaGetLastError());
  return KDS_OK;
}

// ---------------------------------------------------------------------------
// One linearization (buildQuadraticForm) that allocates nothing.
//
// Some callers cannot allocate device memory when they linearize: a real-time
// odometry or bundle-adjustment loop that reserves all of its memory at start-up and
// must not call cudaMalloc/cudaFree afterwards (they can block on the device and on
// allocator locks), or code that must not touch the allocator while it enqueues work.
// For them the scratch of k_linearize -- the job, state and output records, the
// fixed-entry record, the tile list and one FP64 partial per tile -- lives in one
// file-scope device array.  Every call on a device shares that array: calls that
// overlap on the GPU (other streams, other host threads) race on it, and it keeps the
// last call's contents.  The tile list is rebuilt and the job state reset by every
// call; each tile writes its own partial before the last tile reads them.
namespace {

constexpr int kStaticMaxTiles = 512;  // 512 tiles x 128 = 65,536 moving surfels per call
constexpr int kStaticStage = 2047;    // fixed-tree nodes staged per block (64 KB)

// What the call reads back: the job's outputs and the launch's own error bits.
struct StaticResult {
  JobOut out;
  int32_t err;
  int32_t pad_[3];
};

struct StaticScratch {
  JobIn job;
  JobState state;
  StaticResult res;
  LinDev lin;
  TileDev tiles[kStaticMaxTiles];
  double partials[(size_t)kStaticMaxTiles * kPStride];
};

__device__ __align__(256) unsigned char g_static_scratch[sizeof(StaticScratch)];

std::mutex g_static_mu;
StaticScratch* g_static_ptr[64] = {nullptr};

// Writes the job and fixed-entry records and the tile list into the scratch.
__global__ void k_static_setup(StaticScratch* scr, JobIn job, LinDev lin, int ntiles) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    scr->job = job;
    scr->lin = lin;
    scr->res.err = 0;
  }
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x) {
    TileDev d;
    d.job = 0;
    d.lin = 0;
    d.leaf_begin = t * kBlock;
    d.leaf_end = min((t + 1) * kBlock, job.m_num_leaves);
    scr->tiles[t] = d;
  }
}

// First call on a device, with that device current: resolves the array's device
// address and raises the kernels' dynamic shared-memory limit.
int static_setup(StaticScratch** out) {
  int dev = 0;
  KDS_CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) { set_error("device ordinal %d out of range", dev); return KDS_ERR_INVALID_ARG; }
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (!g_static_ptr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess || p == nullptr) return cuda_status(e, "cudaGetSymbolAddress(g_static_scratch)", __FILE__, __LINE__);
    const int bytes = kStaticStage * (int)sizeof(DNode);
    KDS_CK(cudaFuncSetAttribute((const void*)k_linearize<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    KDS_CK(cudaFuncSetAttribute((const void*)k_linearize<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    g_static_ptr[dev] = reinterpret_cast<StaticScratch*>(p);
  }
  *out = g_static_ptr[dev];
  return KDS_OK;
}

}  // namespace

int linearize_static(const TreeDev& fixed, const TreeDev& moving, int32_t type, const kds_aligner_params& P,
                     const double* X, const double* Xf, const double* v, const double* fv, int32_t stats_mode,
                     cudaStream_t s, double* H, double* b, kds_stats* stats) {
  const int64_t nl = moving.num_leaves;
  const int64_t ntiles = (nl + kBlock - 1) / kBlock;
  if (ntiles > kStaticMaxTiles) {
    set_error("kds_linearize_static: %lld moving leaves exceed the static maximum of %d", (long long)nl,
              kStaticMaxTiles * kBlock);
    return KDS_ERR_CAPACITY;
  }
  StaticScratch* scr = nullptr;
  int rc = static_setup(&scr);
  if (rc) return rc;
  JobIn J;
  memset(&J, 0, sizeof(J));
  J.m_md = moving.leaf_md;
  J.m_nrm = moving.leaf_nrm;
  J.m_num_leaves = (int32_t)nl;
  J.kind = type == KDS_ICP ? 0 : 1;
  J.mode = KDS_JOB_LINEARIZE;
  J.stats_mode = stats_mode;
  J.lin_begin = 0;
  J.lin_count = 1;
  J.tile_begin = 0;
  J.tile_count = (int32_t)ntiles;
  J.P.kernel_threshold = P.kernel_threshold;
  J.P.damping = P.damping;
  J.P.max_error = P.max_error;
  J.P.min_normal_cos = P.min_normal_cos;
  J.P.min_good_measurements = P.min_good_measurements;
  J.P.max_iterations = P.max_iterations;
  J.P.velocity_damping = P.velocity_damping;
  J.P.term_crit = P.term_crit;
  J.P.d_pert = P.d_pert;
  J.P.d_score = P.d_score;
  for (int i = 0; i < 12; ++i) J.X0[i] = X[i];
  for (int i = 0; i < 6; ++i) J.v0[i] = (type == KDS_ICP || !v) ? 0.0 : v[i];
  LinDev L;
  memset(&L, 0, sizeof(L));
  L.fnodes = fixed.nodes;
  L.fdts = fixed.dts_f;
  L.f_num_nodes = (int32_t)fixed.num_nodes;
  L.job = 0;
  for (int i = 0; i < 12; ++i) L.Xf[i] = Xf[i];
  for (int i = 0; i < 6; ++i) L.fv[i] = fv ? fv[i] : 0.0;
  k_static_setup<<<1, 256, 0, s>>>(scr, J, L, (int)ntiles);
  count_launch();
  k_init_jobs<<<1, 32 * kInitWarps, 0, s>>>(&scr->job, &scr->state, &scr->res.out, &scr->lin, 1, &scr->res.err);
  count_launch();
  if (ntiles > 0) {
    const size_t stage_bytes = (size_t)kStaticStage * sizeof(DNode);
    if (J.kind == 0)
      k_linearize<0><<<(unsigned)ntiles, kBlock, stage_bytes, s>>>(&scr->job, &scr->state, &scr->res.out, nullptr,
                                                                  &scr->lin, scr->tiles, 0, kStaticStage,
                                                                  scr->partials, nullptr, nullptr, &scr->res.err);
    else
      k_linearize<1><<<(unsigned)ntiles, kBlock, stage_bytes, s>>>(&scr->job, &scr->state, &scr->res.out, nullptr,
                                                                  &scr->lin, scr->tiles, 0, kStaticStage,
                                                                  scr->partials, nullptr, nullptr, &scr->res.err);
    count_launch();
  }
  KDS_CK(cudaGetLastError());
  // outputs and error bits in one copy on the caller's stream
  StaticResult R;
  KDS_CK(cudaMemcpyAsync(&R, &scr->res, sizeof(StaticResult), cudaMemcpyDeviceToHost, s));
  KDS_CK(cudaStreamSynchronize(s));
  const int D = type == KDS_ICP ? 6 : 12;
  if (H) memcpy(H, R.out.H, sizeof(double) * D * D);
  if (b) memcpy(b, R.out.b, sizeof(double) * D);
  if (stats) *stats = R.out.stats;
  return timeout_status(R.err);
}

}  // namespace kds
