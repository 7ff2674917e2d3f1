// GPU surfel KD-tree build for one or many clouds at once (a forest).  Compiled with
// -fmad=false: every double/float expression rounds each multiply and add separately,
// so the result is bit-identical to the CPU oracle's canonical build.
//
// Replaces TreeGenerator_::makeTree (kd/tree/tree_generator_impl_.h:7-19), which the
// reference runs on the CPU only.  The tree is built level by level for all trees of
// the batch together:
//   * per-node moments [xx,xy,xz,yy,yz,zz,x,y,z] are exact, order-free 128-bit
//     fixed-point sums: floor(v * 2^64) of each product of two floats is formed and added in
//     integers, so warps, blocks and atomics may add them in any order (the stamps' sums,
//     of dt and dt^2, are differences of such prefix sums over the final point order);
//   * FP64 covariance, cyclic Jacobi eigensolver, FlatLeafPolicy_ decision
//     (kd/tree/flat_leaf_policy_.h:52-108) in FP64;
//   * stable partition by Node_::whichSide in float (kd/tree/node_.h:53-56);
//   * children numbered by a scan over the level's split flags: nodes of one level
//     are grouped by tree, so each tree's nodes in global order are its BFS order
//     (kd/tree/tree_cpu_impl_.h:136-158), kept by prune (kd/tree/tree_cpu_.h:172-207).
// Nodes with <= kBig points are processed by one warp each; larger ones by blocks over
// kChunk-point chunks with 128-bit atomics.  The level bounds live in device memory;
// the host checks for completion only every kLevelsPerSync levels.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <utility>
#include <vector>

#include "kds_internal.cuh"
#include "kds_rules.h"

namespace kds {

namespace {

constexpr int kBig = 1024;
constexpr int kRootFrame = 15;  // doubles per root: eigenvalues, eigenvectors, mean (decide)
constexpr int kChunk = 1024;
constexpr int kThreads = 256;
constexpr int kGridBlocks = 148 * 4;
constexpr int kLevelBlocks = 148 * 3;  // k_decide: 3 blocks per SM at its register count
constexpr int kLevelsPerSync = 4;
constexpr int kMaxDepth = 64;
constexpr int kUnroll = 2;  // rounds of 32 points in flight per lane in the warp-per-node partition
constexpr int kScatterPerSM = 2;  // 122 registers: the lanes' 21 64-bit parts and four points in flight
constexpr int kSmallPerSM = 3;
constexpr int kSmallBlocks = 148 * kSmallPerSM * 2;  // two waves: other streams' kernels interleave at block boundaries

// ---------------------------------------------------------------------------
// The build is a chain of short launches on one stream, each reading what the one before
// wrote.  Every kernel may start while its predecessor still runs (programmatic dependent
// launch): it lets its own successor be set up at once and waits here, before it reads
// anything, for its predecessor's end, which includes the predecessor's own wait.  A
// launch then costs its kernel and not the gap before it (an 11,000-point scan, 35 launches: 404 us without, 349 with).
__device__ __forceinline__ void grid_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);  // errors: cudaGetLastError by the callers
  count_launch();
}

// ---------------------------------------------------------------------------
// 128-bit two's complement fixed point (units of 2^-64)
struct U128 {
  unsigned long long lo, hi;
};
__host__ __device__ __forceinline__ U128 u128_zero() { U128 r; r.lo = 0ull; r.hi = 0ull; return r; }
__host__ __device__ __forceinline__ U128 u128_add(U128 a, U128 b) {
  U128 r;
  r.lo = a.lo + b.lo;
  r.hi = a.hi + b.hi + (r.lo < a.lo ? 1ull : 0ull);
  return r;
}
__device__ __forceinline__ void atomic_add_u128(U128* dst, U128 v) {
  unsigned long long old = atomicAdd(&dst->lo, v.lo);
  unsigned long long carry = (old + v.lo < old) ? 1ull : 0ull;
  atomicAdd(&dst->hi, v.hi + carry);
}
__host__ __device__ __forceinline__ U128 u128_sub(U128 a, U128 b) {
  U128 r;
  r.lo = a.lo - b.lo;
  r.hi = a.hi - b.hi - (a.lo < b.lo ? 1ull : 0ull);
  return r;
}
__host__ __device__ __forceinline__ double fx_to_d(U128 q) {
  long long hi = (long long)q.hi;
  return ((double)hi * 0x1p64 + (double)q.lo) * 0x1p-64;
}

// floor(v * 2^64) for v = (-1)^sign * mant * 2^exp2 (exact integer arithmetic)
__device__ __forceinline__ U128 fx_parts(unsigned sign, unsigned long long mant, int exp2) {
  U128 mag = u128_zero();
  bool rem = false;
  if (mant == 0ull) return mag;
  int sh = exp2 + 64;
  if (sh >= 64) {
    mag.hi = mant << (sh - 64);
  } else if (sh > 0) {
    mag.lo = mant << sh;
    mag.hi = mant >> (64 - sh);
  } else if (sh == 0) {
    mag.lo = mant;
  } else {
    int r = -sh;
    if (r >= 64) {
      rem = true;
    } else {
      mag.lo = mant >> r;
      rem = (mant & ((1ull << r) - 1ull)) != 0ull;
    }
  }
  if (!sign) return mag;
  U128 neg;  // -mag - rem: ~mag when rem, else ~mag + 1
  neg.lo = ~mag.lo;
  neg.hi = ~mag.hi;
  if (!rem) {
    neg.lo += 1ull;
    if (neg.lo == 0ull) neg.hi += 1ull;
  }
  return neg;
}
__device__ __forceinline__ void f_parts(float f, unsigned& s, unsigned& m, int& e) {
  unsigned b = __float_as_uint(f);
  s = b >> 31;
  unsigned E = (b >> 23) & 0xffu;
  m = b & 0x7fffffu;
  if (E == 0u) {
    e = -149;
  } else {
    m |= 0x800000u;
    e = (int)E - 150;
  }
}
// floor(a * b * 2^64) of any two floats
__device__ __noinline__ U128 fx_ff(float a, float b) {
  unsigned sa, ma, sb, mb;
  int ea, eb;
  f_parts(a, sa, ma, ea);
  f_parts(b, sb, mb, eb);
  return fx_parts(sa ^ sb, (unsigned long long)ma * (unsigned long long)mb, ea + eb);
}
// floor(d * 2^64) for a double 0 <= d < 2^52 (the stamp terms dt and dt^2: dt >= 0 by
// construction, dt < 2^16 checked): shifts that clamp, no branch.
__device__ __forceinline__ unsigned long long shl_c(unsigned long long v, unsigned n) {
  unsigned long long r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));  // n >= 64 gives 0
  return r;
}
__device__ __forceinline__ unsigned long long shr_c(unsigned long long v, unsigned n) {
  unsigned long long r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));  // n >= 64 gives 0
  return r;
}
__device__ __forceinline__ U128 fx_d_nonneg(double d) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  const unsigned long long m = (b & ((1ull << 52) - 1ull)) | (1ull << 52);  // below 2^-63 all bits are shifted out
  const int sh = (int)(b >> 52) - 1011;                                     // d * 2^64 = m * 2^sh, sh < 64
  U128 r;
  r.lo = shl_c(m, (unsigned)sh) | shr_c(m, (unsigned)(-sh));  // one of them is 0, or both are m
  r.hi = shr_c(m, (unsigned)(64 - sh));
  return r;
}

// ---- exact sums of points --------------------------------------------------------------
// A node's nine sums are floor(v * 2^64) over its points of v = xx, xy, xz, yy, yz, zz, x, y, z:
// products of two of the four numbers x, y, z, 1.
//
// A coordinate that is 0 or at least 2^-17 in magnitude (below 2^15) has no bit below 2^-40:
// x * 2^40 = h * 2^28 + l with |h|, |l| <= 2^27, both exact.  A product is then
// (h h') 2^56 + (h l' + l h') 2^28 + l l' in units of 2^-80; only l l' has bits below 2^-64, and
// clearing its low 16 bits floors the product.  Each part is one multiply-add into a 64-bit
// sum; 64 points, on the grid or off it, stay below 2^63.  The rare point with a nonzero coordinate below 2^-17
// takes fx_ff.
constexpr int kSums = 9;
// the two factors of product c
__device__ __forceinline__ int sum_fa(int c) { return c < 6 ? (c < 3 ? 0 : (c < 5 ? 1 : 2)) : c - 6; }
__device__ __forceinline__ int sum_fb(int c) { return c < 6 ? (c < 3 ? c : (c < 5 ? c - 2 : 2)) : 3; }
__device__ __forceinline__ bool limbs40(float x, int2& w) {
  const float y = x * 4096.0f;  // exact
  w.x = __float2int_rn(y);
  w.y = __float2int_rn((y - (float)w.x) * 0x1p28f);  // the difference is exact
  const float a = fabsf(x);
  return a == 0.0f || a >= 0x1p-17f;
}
// (hh 2^56 + mid 2^28 + ll) / 2^16, ll a multiple of 2^16
__device__ __forceinline__ U128 limb_total(long long hh, long long mid, long long ll) {
  U128 q, m;
  q.lo = (unsigned long long)hh << 40;
  q.hi = (unsigned long long)(hh >> 24);
  m.lo = (unsigned long long)mid << 12;
  m.hi = (unsigned long long)(mid >> 52);
  q = u128_add(q, m);
  m.lo = (unsigned long long)(ll >> 16);
  m.hi = (unsigned long long)(ll >> 63);
  return u128_add(q, m);
}

// Sums of small sets by one warp: the set's points are staged in shared memory as limbs, lane
// c < 27 forms product c % 9 of every third point, so a lane holds one sum, not nine, only
// points of the set cost anything, and the warp total is two exchanges.  Points off the grid
// are staged as they are, from the other end.
constexpr int kStage = 64;  // points staged per warp
struct __align__(16) SumStage {  // a point's first two limb pairs are stored as one 16 B word
  int2 w[kStage][4];  // limbs (h, l) of x, y, z, 1
};
struct WarpSums {
  U128 v;   // lane c < 27: its product's sum
  int cnt;  // points staged as limbs
  int odd;  // and as floats
};
__device__ __forceinline__ void stage_init(SumStage& sg, int lane) {
  for (int k = lane; k < kStage; k += 32) sg.w[k][3] = make_int2(1 << 12, 0);
  __syncwarp();
}
__device__ __forceinline__ void sums_zero(WarpSums& S) {
  S.v = u128_zero();
  S.cnt = S.odd = 0;
}
// Adds the staged points to the lanes' sums (whole warp, staged points visible).
__device__ __forceinline__ void sums_flush(WarpSums& S, const SumStage& sg, int lane) {
  const int c = lane % 9;
  const int2* pa = &sg.w[0][sum_fa(c)];
  const int2* pb = &sg.w[0][sum_fb(c)];
  long long hh = 0, mid = 0, ll = 0;
#pragma unroll 2
  for (int i = lane < 27 ? lane / 9 : S.cnt; i < S.cnt; i += 3) {
    const int2 a = pa[4 * i], b = pb[4 * i];
    hh += (long long)a.x * b.x;
    mid += (long long)a.x * b.y;
    mid += (long long)a.y * b.x;
    ll += ((long long)a.y * b.y) & ~0xffffll;
  }
  S.v = u128_add(S.v, limb_total(hh, mid, ll));
  for (int k = lane < 27 ? lane / 9 : S.odd; k < S.odd; k += 3) {
    const float4 f = *reinterpret_cast<const float4*>(sg.w[kStage - 1 - k]);
    const int a = sum_fa(c), b = sum_fb(c);
    S.v = u128_add(S.v, fx_ff(a == 0 ? f.x : (a == 1 ? f.y : f.z),
                              b == 0 ? f.x : (b == 1 ? f.y : (b == 2 ? f.z : 1.0f))));
  }
  S.cnt = S.odd = 0;
}
// Adds the points p of the lanes with add set (whole warp; room for 32 more staged points is
// the caller's to keep).
__device__ __forceinline__ void sums_add(WarpSums& S, SumStage& sg, bool add, float4 p, int lane) {
  int2 wx, wy, wz;
  const bool ox = limbs40(p.x, wx), oy = limbs40(p.y, wy), oz = limbs40(p.z, wz);
  const bool on = ox && oy && oz;
  const unsigned lt = (1u << lane) - 1u;
  const unsigned bm = __ballot_sync(0xffffffffu, add && on), bo = __ballot_sync(0xffffffffu, add && !on);
  if (add) {
    int2* w = sg.w[on ? S.cnt + __popc(bm & lt) : kStage - 1 - S.odd - __popc(bo & lt)];
    *reinterpret_cast<int4*>(w) = on ? make_int4(wx.x, wx.y, wy.x, wy.y)
                                     : make_int4(__float_as_int(p.x), __float_as_int(p.y), __float_as_int(p.z), 0);
    if (on) w[2] = wz;
  }
  S.cnt += __popc(bm);
  S.odd += __popc(bo);
}
// Flushes if more than `most` points are staged.
__device__ __forceinline__ void sums_room(WarpSums& S, const SumStage& sg, int most, int lane) {
  if (S.cnt + S.odd <= most) return;
  __syncwarp();
  sums_flush(S, sg, lane);
  __syncwarp();
}
// The warp's totals: lane k < 9 returns sum k.  S starts anew.
__device__ __forceinline__ U128 sums_total(WarpSums& S, const SumStage& sg, int lane) {
  __syncwarp();
  sums_flush(S, sg, lane);
  __syncwarp();
  const U128 q = S.v;  // lanes c, c + 9 and c + 18 hold product c
  U128 r, u;
  r.lo = __shfl_down_sync(0xffffffffu, q.lo, 9);
  r.hi = __shfl_down_sync(0xffffffffu, q.hi, 9);
  u.lo = __shfl_down_sync(0xffffffffu, q.lo, 18);
  u.hi = __shfl_down_sync(0xffffffffu, q.hi, 18);
  sums_zero(S);
  return u128_add(q, u128_add(r, u));
}

// Sums of large sets: each lane keeps the three parts of its own points' products (no
// staging, nine independent chains), folded into the warp's totals every kLanePoints points
// per lane at most.
constexpr int kLanePoints = 64;
struct LaneSums {
  long long hh[6], mid[6], ll[6];
  long long s[3];   // x, y, z in units of 2^-40
  unsigned sl[3];   // and what lies below, in units of 2^-64 (points off the grid)
  U128 tot;         // lane k < 9: the warp's sum k
};
__device__ __forceinline__ void lane_zero(LaneSums& S) {
#pragma unroll
  for (int k = 0; k < 6; ++k) S.hh[k] = S.mid[k] = S.ll[k] = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    S.s[k] = 0;
    S.sl[k] = 0u;
  }
}
// Adds the point p of the lanes with add set (whole warp).
__device__ __forceinline__ void lane_add(LaneSums& S, bool add, float4 p, int lane) {
  int2 w[3];
  const bool ox = limbs40(p.x, w[0]), oy = limbs40(p.y, w[1]), oz = limbs40(p.z, w[2]);
  const bool on = ox && oy && oz;
  unsigned odd = __ballot_sync(0xffffffffu, add && !on);
  if (add && on) {
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const int2 a = w[c < 3 ? 0 : (c < 5 ? 1 : 2)], b = w[c < 3 ? c : (c < 5 ? c - 2 : 2)];
      S.hh[c] += (long long)a.x * b.x;
      if (c == 0 || c == 3 || c == 5) {
        S.mid[c] += (long long)a.x * (2 * b.y);
      } else {
        S.mid[c] += (long long)a.x * b.y;
        S.mid[c] += (long long)a.y * b.x;
      }
      S.ll[c] += ((long long)a.y * b.y) & ~0xffffll;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      S.s[k] += (long long)w[k].x * (1 << 28);
      S.s[k] += w[k].y;
    }
  }
  if (!odd) return;
  // Off the grid.  A few points (a map's ground near z = 0): one by one, lane c < 9 forming
  // product c.
  if (__popc(odd) <= 4) {
    while (odd) {
      const int src = __ffs(odd) - 1;
      odd &= odd - 1;
      const float f0 = __shfl_sync(0xffffffffu, p.x, src), f1 = __shfl_sync(0xffffffffu, p.y, src);
      const float f2 = __shfl_sync(0xffffffffu, p.z, src);
      if (lane < 9) {
        const int a = sum_fa(lane), b = sum_fb(lane);
        S.tot = u128_add(S.tot, fx_ff(a == 0 ? f0 : (a == 1 ? f1 : f2),
                                      b == 0 ? f0 : (b == 1 ? f1 : (b == 2 ? f2 : 1.0f))));
      }
    }
    return;
  }
  // Many (a scan's column along an axis brings 128 in a row): the lanes together, whole
  // values split over the same parts.
  if (!add || on) return;
#pragma unroll
  for (int c = 0; c < 6; ++c) {
    const U128 v = fx_ff(c < 3 ? p.x : (c < 5 ? p.y : p.z), c == 0 ? p.x : (c == 1 || c == 3 ? p.y : p.z));
    S.hh[c] += (long long)((v.lo >> 40) | (v.hi << 24));
    S.ll[c] += (long long)((v.lo & 0xffffffffffull) << 16);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const U128 v = fx_ff(k == 0 ? p.x : (k == 1 ? p.y : p.z), 1.0f);
    S.s[k] += (long long)((v.lo >> 24) | (v.hi << 40));
    S.sl[k] += (unsigned)v.lo & 0xffffffu;
  }
}
__device__ __forceinline__ U128 shfl_xor_u128(U128 v, int m) {
  U128 r;
  r.lo = __shfl_xor_sync(0xffffffffu, v.lo, m);
  r.hi = __shfl_xor_sync(0xffffffffu, v.hi, m);
  return r;
}
// Folds the lanes' parts into the warp's totals.  Reduce-scatter: 16 slots (9 used) halved
// over lane bits 4..1, then added with lane ^ 1, so lanes 2k and 2k + 1 hold total k.
__device__ __forceinline__ void lane_fold(LaneSums& S, int lane) {
  U128 v[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = u128_zero();
#pragma unroll
  for (int k = 0; k < 6; ++k) v[k] = limb_total(S.hh[k], S.mid[k], S.ll[k]);
#pragma unroll
  for (int k = 0; k < 3; ++k) {  // x * 2^40 to units of 2^-64
    U128 q;
    q.lo = S.sl[k];
    q.hi = 0ull;
    v[6 + k].lo = (unsigned long long)S.s[k] << 24;
    v[6 + k].hi = (unsigned long long)(S.s[k] >> 40);
    v[6 + k] = u128_add(v[6 + k], q);
  }
  U128 w8[8], w4[4], w2[2];
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4, b1 = lane & 2;
#pragma unroll
  for (int j = 0; j < 8; ++j) w8[j] = u128_add(b4 ? v[8 + j] : v[j], shfl_xor_u128(b4 ? v[j] : v[8 + j], 16));
#pragma unroll
  for (int j = 0; j < 4; ++j) w4[j] = u128_add(b3 ? w8[4 + j] : w8[j], shfl_xor_u128(b3 ? w8[j] : w8[4 + j], 8));
#pragma unroll
  for (int j = 0; j < 2; ++j) w2[j] = u128_add(b2 ? w4[2 + j] : w4[j], shfl_xor_u128(b2 ? w4[j] : w4[2 + j], 4));
  U128 w1 = u128_add(b1 ? w2[1] : w2[0], shfl_xor_u128(b1 ? w2[0] : w2[1], 2));
  w1 = u128_add(w1, shfl_xor_u128(w1, 1));
  U128 q;
  q.lo = __shfl_sync(0xffffffffu, w1.lo, (2 * lane) & 31);
  q.hi = __shfl_sync(0xffffffffu, w1.hi, (2 * lane) & 31);
  if (lane < kSums) S.tot = u128_add(S.tot, q);
  lane_zero(S);
}

// ---------------------------------------------------------------------------
struct __align__(16) BNode {
  int32_t start, end;
  int32_t level;
  int32_t tree;
  int32_t split;      // 1: inner node
  int32_t mid;
  int32_t left, right;
  int32_t has_parent;
  int32_t par_has;    // propagated normal received from the parent
  int32_t has_prop;   // propagated normal handed to the children
  int32_t parent;     // parent node, -1 for a root
  float mean[3], dir[3];
  int32_t big;        // large nodes: ordinal among the level's
  int32_t pad_;
  double prop[3];
  double par_prop[3];
};
static_assert(sizeof(BNode) == 128, "one L1 line");

struct BuildParams {
  int32_t propagate_normal;
  int32_t leaf_min_points;
  int32_t leaf_max_points;
  float leaf_density;
  float leaf_min_normal_incidence;
  float leaf_normal_eigenratio;
  float prune_incidence;
  int32_t max_level;
};

struct LevelState {
  int32_t lb, le;        // node range of the current level
  int32_t cur;           // point buffer holding the current level
  int32_t depth;         // number of levels processed
  int32_t max_size;      // largest node of the current level
  int32_t max_next;      // largest node of the next level (being built)
  int32_t error;         // 1: node capacity, 2: input out of range
  int32_t num_chunks, num_big;
  int32_t pad_;
};

__device__ __forceinline__ double ddot3(const double* a, const double* b) {
  double p0 = a[0] * b[0], p1 = a[1] * b[1], p2 = a[2] * b[2];
  return p0 + (p1 + p2);
}

// Cyclic Jacobi eigensolver for a symmetric 3x3 (Golub & Van Loan, sec. 8.5), fixed
// 8 sweeps; eigenvalues ascending, eigenvectors as columns of V.  Every index is a constant
// once the loops are unrolled, so the matrices stay in registers: with them in local memory
// the decisions of a level of 500,000 nodes took 200 us, now 132.
__device__ __forceinline__ void jacobi3(const double Ain[3][3], double ev[3], double V[3][3]) {
  double a[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) { a[i][j] = Ain[i][j]; V[i][j] = (i == j) ? 1.0 : 0.0; }
#pragma unroll 1
  for (int sweep = 0; sweep < 8; ++sweep) {
    if (a[0][1] == 0.0 && a[0][2] == 0.0 && a[1][2] == 0.0) break;
#pragma unroll
    for (int pq = 0; pq < 3; ++pq) {
      const int p = (pq == 2) ? 1 : 0;
      const int q = (pq == 0) ? 1 : 2;
      const int r = 3 - p - q;
      double apq = a[p][q];
      // negligible off-diagonal: set to zero (same rule in the CPU oracle)
      if (fabs(apq) <= 1e-18 * (fabs(a[p][p]) + fabs(a[q][q]))) {
        a[p][q] = 0.0;
        a[q][p] = 0.0;
        continue;
      }
      double theta = (a[q][q] - a[p][p]) / (2.0 * apq);
      double t = 1.0 / (fabs(theta) + sqrt(theta * theta + 1.0));
      if (theta < 0.0) t = -t;
      double c = 1.0 / sqrt(t * t + 1.0);
      double s = t * c;
      double arp = a[r][p], arq = a[r][q];
      a[p][p] = a[p][p] - t * apq;
      a[q][q] = a[q][q] + t * apq;
      a[p][q] = 0.0;
      a[q][p] = 0.0;
      double nrp = c * arp - s * arq;
      double nrq = s * arp + c * arq;
      a[r][p] = nrp; a[p][r] = nrp;
      a[r][q] = nrq; a[q][r] = nrq;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        double vkp = V[k][p], vkq = V[k][q];
        V[k][p] = c * vkp - s * vkq;
        V[k][q] = s * vkp + c * vkq;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) ev[i] = a[i][i];
  // stable: neighbours change places only where the right one is strictly smaller
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int i = k & 1;
    const bool sw = ev[i + 1] < ev[i];
    const double lo = sw ? ev[i + 1] : ev[i], hi = sw ? ev[i] : ev[i + 1];
    ev[i] = lo;
    ev[i + 1] = hi;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double vl = sw ? V[j][i + 1] : V[j][i], vh = sw ? V[j][i] : V[j][i + 1];
      V[j][i] = vl;
      V[j][i + 1] = vh;
    }
  }
}

// FlatLeafPolicy_::fillMetadata over CountLeafPolicy_ and LabelPolicyBase_
// (kd/tree/flat_leaf_policy_.h:52-108, count_leaf_policy_.h:27-43,
// label_policy_base_impl_.h:12-97) on FP64 statistics.
// Sd: the node's nine moment sums converted to double (fx_to_d of the exact sums).
// root (nullable): for a root node, its frame as TreeCPU_'s constructor stores it
// (kd/tree/tree_cpu_.h:72-86): [0..2] eigenvalues ascending, [3..11] eigenvectors
// column-major (columns 0 and 2 reoriented as in fillMetadata, then column 0 negated if
// the determinant is negative), [12..14] mean; zero where the node has < 3 points.
struct Decision {
  float mean[3], dir[3];
  double prop[3];  // normal handed to the children
  bool has_prop;
  bool split;
};
__device__ __forceinline__ void flip_to_origin(const double* mean, double* e) {
  if (ddot3(mean, e) > 0.0) {
#pragma unroll
    for (int i = 0; i < 3; ++i) e[i] = -e[i];
  }
}
// par_has, par_prop: the normal that the parent handed down, if any (never for a root).
__device__ __forceinline__ Decision decide(const double* Sd, int64_t n, bool par_has, const double* par_prop, int level,
                                           const BuildParams& P, double* root) {
  Decision nd;
  double mean_d[3] = {0, 0, 0};
  double e0[3] = {0, 0, 0}, e2[3] = {0, 0, 0};
  double lam[3] = {0, 0, 0};
  bool is_bad = true;
#pragma unroll
  for (int i = 0; i < 3; ++i) { nd.mean[i] = 0.f; nd.dir[i] = 0.f; nd.prop[i] = 0.0; }
  if (n > 0) {
    double dn = (double)n;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      mean_d[i] = Sd[6 + i] / dn;
      nd.mean[i] = (float)mean_d[i];
    }
    if (n >= 3) {
      double C[3][3];
      C[0][0] = Sd[0] / dn - mean_d[0] * mean_d[0];
      C[0][1] = Sd[1] / dn - mean_d[0] * mean_d[1];
      C[0][2] = Sd[2] / dn - mean_d[0] * mean_d[2];
      C[1][1] = Sd[3] / dn - mean_d[1] * mean_d[1];
      C[1][2] = Sd[4] / dn - mean_d[1] * mean_d[2];
      C[2][2] = Sd[5] / dn - mean_d[2] * mean_d[2];
      C[1][0] = C[0][1];
      C[2][0] = C[0][2];
      C[2][1] = C[1][2];
      double V[3][3];
      jacobi3(C, lam, V);
#pragma unroll
      for (int i = 0; i < 3; ++i) { e0[i] = V[i][0]; e2[i] = V[i][2]; }
      flip_to_origin(mean_d, e0);
      flip_to_origin(mean_d, e2);
      is_bad = false;
      if (root) {
        const double e1[3] = {V[0][1], V[1][1], V[2][1]};
        // det [e0 e1 e2] = e0 . (e1 x e2)
        const double cx = e1[1] * e2[2] - e1[2] * e2[1];
        const double cy = e1[2] * e2[0] - e1[0] * e2[2];
        const double cz = e1[0] * e2[1] - e1[1] * e2[0];
        const double det = e0[0] * cx + (e0[1] * cy + e0[2] * cz);
        const double sg = det < 0.0 ? -1.0 : 1.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          root[i] = lam[i];
          root[3 + i] = sg * e0[i];
          root[6 + i] = e1[i];
          root[9 + i] = e2[i];
        }
      }
    }
  }
  if (root) {
    if (is_bad)
      for (int i = 0; i < 12; ++i) root[i] = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) root[12 + i] = mean_d[i];
  }
  // 0: no direction, 1: e0, 2: e2, 3: the normal handed down
  bool is_node = !is_bad && (float)n > (float)P.leaf_max_points;
  int dir = is_bad ? 0 : (is_node ? 2 : 1);
  bool has_prop = P.propagate_normal && par_has;
  double prop[3] = {0, 0, 0};
  if (P.propagate_normal) {
#pragma unroll
    for (int i = 0; i < 3; ++i) prop[i] = par_prop[i];
  }
  bool is_flat = false;
  bool do_prop = false;
  if (is_bad || (float)n < (float)P.leaf_min_points) {
    do_prop = true;
  } else {
    double eigenratio = lam[0] / lam[2];
    is_flat = eigenratio < (double)P.leaf_normal_eigenratio &&
              fabs(ddot3(mean_d, e0)) > (double)P.leaf_min_normal_incidence;
    if (is_flat) {
      has_prop = true;
#pragma unroll
      for (int i = 0; i < 3; ++i) prop[i] = e0[i];
    }
    if (!is_node) {
      double volume = lam[1] * lam[2];
      double density = (double)n / volume;
      if (density < (double)P.leaf_density) {
        is_node = true;
        dir = 2;
      } else if (is_flat) {
        dir = 1;
      } else {
        do_prop = true;
      }
    }
  }
  if (do_prop && has_prop) dir = 3;
  if (is_node && level >= P.max_level - 1) {
    is_node = false;
    dir = is_flat ? 1 : (has_prop ? 3 : 1);
  }
  double d[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) d[i] = dir == 3 ? prop[i] : (dir == 2 ? e2[i] : (dir == 1 ? e0[i] : 0.0));
  if (dir == 3) flip_to_origin(mean_d, d);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    nd.dir[i] = (float)d[i];
    nd.prop[i] = prop[i];
  }
  nd.split = is_node;
  nd.has_prop = has_prop;
  return nd;
}

__device__ __forceinline__ bool which_side_f(const float* mean, const float* dir, float4 q) {
  F3 d = sub3x(f3(q.x, q.y, q.z), f3(mean[0], mean[1], mean[2]));
  return dot3x(f3(dir[0], dir[1], dir[2]), d) > 0.0f;
}

// block-wide exclusive scan of one int per thread; *total = block sum
__device__ __forceinline__ int block_scan(int v, int* sm, int* total) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
  for (int off = 1; off < 32; off <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) sm[w] = x;
  __syncthreads();
  if (w == 0) {
    int nw = blockDim.x >> 5;
    int y = (lane < nw) ? sm[lane] : 0;
    for (int off = 1; off < 32; off <<= 1) {
      int z = __shfl_up_sync(0xffffffffu, y, off);
      if (lane >= off) y += z;
    }
    if (lane < nw) sm[lane] = y;
  }
  __syncthreads();
  int wprefix = (w > 0) ? sm[w - 1] : 0;
  *total = sm[(blockDim.x >> 5) - 1];
  __syncthreads();
  return wprefix + x - v;
}

// The node range [b, e) of this block when gridDim.x / parts ranges split the current level.
__device__ __forceinline__ void level_range(const LevelState* ls, int& b, int& e, int parts = 1) {
  const int lb = ls->lb, le = ls->le;
  const int nl = le - lb;
  const int ranges = gridDim.x / parts;
  const int per = (nl + ranges - 1) / ranges;
  b = lb + (blockIdx.x / parts) * per;
  e = min(b + per, le);
}

// ---------------------------------------------------------------------------
// Kernels

__global__ void k_ingest(const float* xyz, int64_t n, float4* pts, LevelState* ls) {
  grid_begin();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
    if (!(fabsf(x) < 32768.f && fabsf(y) < 32768.f && fabsf(z) < 32768.f)) ls->error = 2;
    pts[i] = make_float4(x, y, z, __int_as_float((int32_t)i));
  }
}

// Order-preserving map of finite doubles to unsigned 64-bit keys.
__device__ __forceinline__ unsigned long long dkey(double d) {
  unsigned long long b = (unsigned long long)__double_as_longlong(d);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double dkey_inv(unsigned long long k) {
  unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)b);
}

// ts_start of each tree = min stamp (label_policy_base_impl_.h:28-35), as the largest
// complement of its key (tsmin starts at 0); blockIdx.y = tree.
__global__ void k_tree_min(const double* sts, const int64_t* off, unsigned long long* tsmin) {
  grid_begin();
  const int r = blockIdx.y;
  const int64_t b = off[r], e = off[r + 1];
  unsigned long long m = 0ull;
  for (int64_t i = b + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < e; i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, ~dkey(sts[i]));
  for (int off2 = 16; off2 > 0; off2 >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, off2));
  if ((threadIdx.x & 31) == 0 && m != 0ull) atomicMax(&tsmin[r], m);
}

// decodes ts_start, checks every point's stamp and writes its dt; blockIdx.y = tree.
__global__ void k_tree_check(const double* sts, const int64_t* off, const unsigned long long* tsmin, double* ts0,
                             double* dt, LevelState* ls) {
  grid_begin();
  const int r = blockIdx.y;
  const int64_t b = off[r], e = off[r + 1];
  const double t0 = (e > b) ? dkey_inv(~tsmin[r]) : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) ts0[r] = t0;
  for (int64_t i = b + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < e; i += (int64_t)gridDim.x * blockDim.x) {
    const double s = sts[i];
    const double d = s - t0;
    if (!(isfinite(s) && d < 65536.0)) ls->error = 2;
    dt[i] = d;
  }
}

__global__ void k_init_roots(BNode* nodes, const int64_t* off, int R, LevelState* ls) {
  grid_begin();
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < R) {
    BNode nd;
    memset(&nd, 0, sizeof(nd));
    nd.start = (int32_t)off[r];
    nd.end = (int32_t)off[r + 1];
    nd.tree = r;
    nd.left = nd.right = -1;
    nd.parent = -1;
    nodes[r] = nd;
    atomicMax(&ls->max_size, nd.end - nd.start);
  }
  if (r == 0) {
    ls->lb = 0;
    ls->le = R;
    ls->cur = 0;
    ls->depth = 0;
    ls->max_next = 0;
  }
}

// A point moves through the levels as one 16 B record (x, y, z, w = its input index as int
// bits), double-buffered by level parity.  The stamps stay out of the levels: no decision
// needs them, and once the final point order is known every node's dt sums are differences
// of prefix sums over it (k_dt_prefix).
struct PointBufs {
  float4* p[2];
  int32_t* perm;  // final point order (global indices)
};

// Every node's nine exact moment sums are kept in mom[node].  The roots' sums are
// computed from their points; a split node hands its children their sums: the smaller
// child's from one pass over its points after the partition, the other's as the
// parent's minus the smaller's (exact integer arithmetic).  So below the roots each point
// is summed once per level only when it lands in the smaller child of its parent.

// L1 prefetch of the line holding p (no register, no effect on results).
__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// Level 0: warp per root of at most kBig points.
__global__ void __launch_bounds__(kThreads) k_root_moments(const BNode* nodes, int R, PointBufs B, U128* mom) {
  grid_begin();
  const int lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  static_assert(kBig <= 32 * kLanePoints, "a root's points fit the lanes' sums");
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < R; r += nw) {
    const int s = nodes[r].start, e = nodes[r].end;
    if (e - s > kBig) continue;
    LaneSums S;
    lane_zero(S);
    S.tot = u128_zero();
    for (int k0 = s; k0 < e; k0 += 32) {
      const int i = k0 + lane;
      float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i < e) p = B.p[0][i];
      lane_add(S, i < e, p, lane);
    }
    lane_fold(S, lane);
    if (lane < kSums) mom[(size_t)r * kSums + lane] = S.tot;
  }
}

// Accumulators of the large nodes' smaller children: two sets by level parity, so that a
// level's may be read while the next one's are cleared.
struct ChildSums {
  U128* acc[2];
};
// A node whose parent is large has no sums yet: the parent's scatter left the smaller child's
// in the accumulators of its level, the other child's are the parent's minus them.
struct PendingSums {
  const U128* q;    // nullptr: the sums are in mom[i]
  const U128* par;
  bool small;
};
__device__ __forceinline__ PendingSums pending_sums(const BNode* nodes, const U128* mom, const ChildSums& C, int depth,
                                                    int i, int parent) {
  PendingSums r;
  r.q = nullptr;
  r.par = nullptr;
  r.small = false;
  if (parent < 0) return r;
  const BNode& p = nodes[parent];
  const int s = p.start, e = p.end;
  if (e - s <= kBig) return r;
  r.q = C.acc[(depth & 1) ^ 1] + (size_t)p.big * kSums;
  r.par = mom + (size_t)parent * kSums;
  r.small = (p.left == i) == (p.mid - s <= e - p.mid);
  return r;
}
__device__ __forceinline__ U128 pending_value(const PendingSums& r, int k) {
  const U128 q = r.q[k];
  return r.small ? q : u128_sub(r.par[k], q);
}

// Thread per node of the level: the leaf/split decision from its sums.  Block b takes
// the b-th contiguous range of the level's nodes and writes its count of split nodes
// (the children's numbering scans these counts).
__device__ __forceinline__ void level_decide(BNode* nodes, const LevelState* ls, U128* mom, const ChildSums& C,
                                             const BuildParams& P, int32_t* bsum, int32_t* bbig, double* root_frame,
                                             int* sm) {
  int b, e;
  level_range(ls, b, e);
  const int depth = ls->depth;
  int v = 0, nc = 0, nb = 0;
  for (int i = b + threadIdx.x; i < e; i += blockDim.x) {
    BNode& nd = nodes[i];
    const int n = nd.end - nd.start;
    double Sd[kSums];
    const PendingSums r = pending_sums(nodes, mom, C, depth, i, nd.parent);
    if (r.q) {
#pragma unroll
      for (int k = 0; k < kSums; ++k) {
        const U128 q = pending_value(r, k);
        mom[(size_t)i * kSums + k] = q;
        Sd[k] = fx_to_d(q);
      }
    } else {
#pragma unroll
      for (int k = 0; k < kSums; ++k) Sd[k] = fx_to_d(mom[(size_t)i * kSums + k]);
    }
    const double pp[3] = {nd.par_prop[0], nd.par_prop[1], nd.par_prop[2]};
    const Decision q = decide(Sd, n, nd.has_parent && nd.par_has, pp, nd.level, P,
                              depth == 0 ? root_frame + (size_t)nd.tree * kRootFrame : nullptr);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      nd.mean[k] = q.mean[k];
      nd.dir[k] = q.dir[k];
      nd.prop[k] = q.prop[k];
    }
    nd.split = q.split ? 1 : 0;
    nd.has_prop = q.has_prop ? 1 : 0;
    v += q.split ? 1 : 0;
    if (n > kBig) {
      nc += (n + kChunk - 1) / kChunk;
      nb += 1;
    }
  }
  int total, tc, tb;
  block_scan(v, sm, &total);
  block_scan(nc, sm, &tc);
  block_scan(nb, sm, &tb);
  if (threadIdx.x == 0) {
    bsum[blockIdx.x] = total;
    bbig[2 * blockIdx.x] = tc;  // as k_big_sums
    bbig[2 * blockIdx.x + 1] = tb;
  }
}
__global__ void k_decide(BNode* nodes, const LevelState* ls, U128* mom, ChildSums C, BuildParams P, int32_t* bsum,
                         int32_t* bbig, double* root_frame) {
  grid_begin();
  __shared__ int sm[32];
  level_decide(nodes, ls, mom, C, P, bsum, bbig, root_frame, sm);
}

// The level's split count from k_decide's per-block counts, then the next level (one
// whole block).  Children that don't fit the node arrays have no records: the build has failed,
// and the levels to come before the host looks are empty (every kernel takes its nodes from
// [lb, le)).
__device__ void level_advance_block(LevelState* ls, const int32_t* bsum, int nblocks, int32_t cap) {
  __shared__ int sm[32];
  int v = 0;
  for (int k = threadIdx.x; k < nblocks; k += blockDim.x) v += bsum[k];
  int total;
  block_scan(v, sm, &total);
  if (threadIdx.x != 0) return;
  const LevelState x = *ls;  // one round of loads
  if (x.lb >= x.le) return;
  const bool fits = 2 * total <= cap - x.le;
  ls->lb = x.le;
  ls->le = fits ? x.le + 2 * total : x.le;
  ls->cur = x.cur ^ 1;
  ls->depth = x.depth + 1;
  ls->max_size = fits ? x.max_next : 0;
  ls->max_next = 0;
  if (!fits) ls->error = 1;
}

// The last block of the level's last kernel advances the level (done: a counter that
// starts at 0 and is left at 0; nullptr: not the last kernel).  Every block of the
// calling kernel must reach this.
__device__ __forceinline__ void advance_if_last(LevelState* ls, const int32_t* bsum, int nblocks, int32_t cap,
                                                unsigned* done) {
  if (!done) return;
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(done, 1u) == gridDim.x - 1 ? 1 : 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  level_advance_block(ls, bsum, nblocks, cap);
  if (threadIdx.x == 0) *done = 0u;
}

// The first 18 words of a BNode (start .. dir): one coalesced load by lanes 0-17.
constexpr int kNodeHeadWords = 18;
static_assert(offsetof(BNode, dir) + 3 * sizeof(float) == kNodeHeadWords * 4, "BNode head layout");
static_assert(offsetof(BNode, start) == 0 && offsetof(BNode, end) == 4 && offsetof(BNode, tree) == 12 &&
                  offsetof(BNode, split) == 16 && offsetof(BNode, left) == 24 && offsetof(BNode, right) == 28 &&
                  offsetof(BNode, mean) == 48,
              "BNode head layout");

struct __align__(16) Chunk {
  int32_t node;
  int32_t begin;
  int32_t end;
  int32_t big;  // ordinal among the level's large nodes
};

constexpr int kSegs = kThreads / 32;     // 128-point segments per chunk, one per warp of a block
constexpr int kPer = kChunk / kThreads;  // rounds of 32 points per segment
static_assert(kPer * kThreads == kChunk && kSegs == 8, "a chunk is eight segments, its counts one 16 B word");
// Left points of each chunk's eight 128-point segments; a warp per segment, no barrier.
struct __align__(16) SegCounts {
  uint16_t n[kSegs];
};
__device__ __forceinline__ void big_count(const Chunk* chunks, const LevelState* ls, const BNode* nodes,
                                          const PointBufs& B, SegCounts* seg, int block, int blocks) {
  const int nc = ls->num_chunks;
  const float4* pts = B.p[ls->cur];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int ci = block; ci < nc; ci += blocks) {
    const Chunk c = chunks[ci];
    const BNode& nd = nodes[c.node];
    int nl = 0;
    if (nd.split) {
      const int wb = c.begin + w * 32 * kPer;
      float4 pv[kPer];
#pragma unroll
      for (int u = 0; u < kPer; ++u)
        if (wb + u * 32 + lane < c.end) pv[u] = pts[wb + u * 32 + lane];
#pragma unroll
      for (int u = 0; u < kPer; ++u)
        nl += __popc(__ballot_sync(0xffffffffu, wb + u * 32 + lane < c.end && which_side_f(nd.mean, nd.dir, pv[u])));
    }
    if (lane == 0) seg[ci].n[w] = (uint16_t)nl;
  }
}

// Warp per node of at most kBig points, after its children are numbered: stable
// partition by whichSide (or leaf point order), the children's ranges and sums.
// Latency-bound at deep levels (many small nodes per warp), so each node's record
// and sums are fetched in one round of loads, one node ahead.  The staged sums
// (SumStage) leave room for 24 warps per SM: a level of 11.4M points in small nodes takes
// 298 us at most; with eleven 128-bit terms per lane (124 registers, 16 warps) it took 510.
// The first count_blocks blocks count the chunks of the large nodes instead (big_count): neither
// needs the other's results, and a launch less per level takes an 11,000-point scan from 345
// us to 329 and 32 keyframes from 2.46 ms to 2.34 (with the large nodes' lists written by
// k_level_children).
__global__ void __launch_bounds__(kThreads, kSmallPerSM) k_small_part(BNode* nodes, LevelState* ls, PointBufs B,
                                                         U128* mom, const int32_t* bsum, int nblocks, int32_t cap,
                                                         unsigned* done, const Chunk* chunks, SegCounts* seg,
                                                         int count_blocks) {
  grid_begin();
  if ((int)blockIdx.x < count_blocks) {
    big_count(chunks, ls, nodes, B, seg, blockIdx.x, count_blocks);
    return;
  }
  const int blocks = gridDim.x - count_blocks, block = blockIdx.x - count_blocks;
  const int lb = ls->lb, le = ls->le, cur = ls->cur;
  const float4* pin = B.p[cur];
  float4* pout = B.p[cur ^ 1];
  const int lane = threadIdx.x & 31;
  const int nwarps = (blocks * blockDim.x) >> 5;
  const int wslot = (threadIdx.x >> 5) * blocks + block;  // consecutive nodes on different SMs
  const bool sum_lane = lane < kSums;                              // holds sum lane
  __shared__ SumStage stage[kThreads / 32];
  SumStage& sg = stage[threadIdx.x >> 5];
  stage_init(sg, lane);
  WarpSums S;
  sums_zero(S);
  int maxc = 0;
  int word = 0;
  U128 pm = u128_zero();
  auto fetch = [&](int ni) {
    if (ni < le) {
      if (lane < kNodeHeadWords) word = reinterpret_cast<const int*>(nodes + ni)[lane];
      if (sum_lane) pm = mom[(size_t)ni * kSums + lane];
    }
  };
  fetch(lb + wslot);
  for (int ni = lb + wslot; ni < le; ni += nwarps) {
    const int s = __shfl_sync(0xffffffffu, word, 0), e = __shfl_sync(0xffffffffu, word, 1);
    const int split = __shfl_sync(0xffffffffu, word, 4);
    const int li = __shfl_sync(0xffffffffu, word, 6), ri = __shfl_sync(0xffffffffu, word, 7);
    float mean[3], dir[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      mean[k] = __int_as_float(__shfl_sync(0xffffffffu, word, 12 + k));
      dir[k] = __int_as_float(__shfl_sync(0xffffffffu, word, 15 + k));
    }
    const U128 psum = pm;
    fetch(ni + nwarps);  // the next node's record and sums are in flight meanwhile
    if (e - s > kBig) continue;
    if (!split) {
      for (int i = s + lane; i < e; i += 32) B.perm[i] = __float_as_int(pin[i].w);
      if (lane == 0) nodes[ni].mid = e;
      continue;
    }
    const int K = (e - s + 31) >> 5;
    const bool one = K <= kUnroll;  // the whole node fits one round of loads: keep it
    // every round of the node in flight at once (into L1), instead of one dependent
    // round trip per kUnroll rounds
    for (int k = kUnroll; k < K; ++k) {
      const int i = s + (k << 5) + lane;
      if (i < e) prefetch_l1(pin + i);
    }
    unsigned bits = 0u;
    float4 pv[kUnroll];
    for (int k0 = 0; k0 < K; k0 += kUnroll) {
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        int i = s + ((k0 + u) << 5) + lane;
        if (i < e) pv[u] = pin[i];
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        int i = s + ((k0 + u) << 5) + lane;
        if (i < e) {
          if (which_side_f(mean, dir, pv[u])) bits |= 1u << (k0 + u);
        }
      }
    }
    int nl = __popc(bits);
    for (int off = 16; off > 0; off >>= 1) nl += __shfl_xor_sync(0xffffffffu, nl, off);
    const int mid = s + nl;
    // the smaller child is summed while its points move; the other is the parent minus it
    const bool small_left = mid - s <= e - mid;
    const unsigned lt = (1u << lane) - 1u;
    int cl = 0, cr = 0;
    for (int k0 = 0; k0 < K; k0 += kUnroll) {
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        int i = s + ((k0 + u) << 5) + lane;
        if (i < e && !one) pv[u] = pin[i];
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        int i = s + ((k0 + u) << 5) + lane;
        bool valid = i < e;
        bool left = valid && ((bits >> (k0 + u)) & 1u);
        unsigned bl = __ballot_sync(0xffffffffu, left);
        unsigned br = __ballot_sync(0xffffffffu, valid && !left);
        if (valid) {
          int dst = left ? (s + cl + __popc(bl & lt)) : (s + nl + cr + __popc(br & lt));
          pout[dst] = pv[u];
        }
        sums_add(S, sg, valid && left == small_left, pv[u], lane);
        cl += __popc(bl);
        cr += __popc(br);
      }
      sums_room(S, sg, kStage - 32 * kUnroll, lane);
    }
    const U128 q = sums_total(S, sg, lane);
    if (sum_lane) {
      const U128 other = u128_sub(psum, q);
      mom[(size_t)li * kSums + lane] = small_left ? q : other;
      mom[(size_t)ri * kSums + lane] = small_left ? other : q;
    }
    if (lane == 0) {
      nodes[ni].mid = mid;
      nodes[li].start = s;
      nodes[li].end = mid;
      nodes[ri].start = mid;
      nodes[ri].end = e;
      maxc = max(maxc, max(mid - s, e - mid));
    }
  }
  if (lane == 0 && maxc > 0) atomicMax(&ls->max_next, maxc);
  advance_if_last(ls, bsum, nblocks, cap, done);
}

// ---- large nodes ------------------------------------------------------------------
// Large nodes of the level and their kChunk-point chunks, listed in node order by
// kLevelBlocks blocks over contiguous node ranges: per-block counts first, then each
// block writes its list at the prefix of the blocks before it.
__global__ void k_big_sums(const BNode* nodes, const LevelState* ls, int32_t* bbig) {
  grid_begin();
  __shared__ int sm[32];
  if (ls->max_size <= kBig) return;  // no large node on this level
  int b, e;
  level_range(ls, b, e);
  int nc = 0, nb = 0;
  for (int i = b + threadIdx.x; i < e; i += blockDim.x) {
    const int n = nodes[i].end - nodes[i].start;
    if (n > kBig) {
      nc += (n + kChunk - 1) / kChunk;
      nb += 1;
    }
  }
  int tc, tb;
  block_scan(nc, sm, &tc);
  block_scan(nb, sm, &tb);
  if (threadIdx.x == 0) {
    bbig[2 * blockIdx.x] = tc;
    bbig[2 * blockIdx.x + 1] = tb;
  }
}

// acc: the sums to clear for the large nodes listed.  parts: blocks that share one node range
// and write its chunks in turn.
__device__ __forceinline__ void level_plan(BNode* nodes, LevelState* ls, const int32_t* bbig, Chunk* chunks,
                                           int32_t chunk_cap, int32_t* big_list, int32_t* node_chunk0, U128* acc,
                                           int* sm, int part, int parts) {
  if (ls->max_size <= kBig) {  // no large node on this level
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      ls->num_chunks = 0;
      ls->num_big = 0;
    }
    return;
  }
  int b, e;
  level_range(ls, b, e, parts);
  int carry_c, carry_b, all_c, all_b;  // chunks / large nodes of the blocks before this one, of all
  {
    int vc = 0, vb = 0, ac = 0, ab = 0;
    for (int k = threadIdx.x; k < (int)(gridDim.x / parts); k += blockDim.x) {
      if (k < (int)(blockIdx.x / parts)) {
        vc += bbig[2 * k];
        vb += bbig[2 * k + 1];
      }
      ac += bbig[2 * k];
      ab += bbig[2 * k + 1];
    }
    block_scan(vc, sm, &carry_c);
    block_scan(vb, sm, &carry_b);
    block_scan(ac, sm, &all_c);
    block_scan(ab, sm, &all_b);
  }
  // The block's threads share the chunks of its large nodes: chunk by chunk, each thread
  // finds the owner in the block's list.  (A thread per node wrote all of a node's chunks
  // itself before: 261 us for the one 11.4M-point root, 814 us over a map build.)
  __shared__ int s_oc[kThreads];                        // first chunk of the list's nodes, relative
  __shared__ int s_node[kThreads], s_start[kThreads], s_end[kThreads];
  for (int base = b; base < e; base += blockDim.x) {
    int i = base + threadIdx.x;
    int st = 0, en = 0;
    if (i < e) {
      st = nodes[i].start;
      en = nodes[i].end;
    }
    const int n = en - st;
    bool big = n > kBig;
    int nc = big ? (n + kChunk - 1) / kChunk : 0;
    int tc, tb;
    int oc = block_scan(nc, sm, &tc);
    int ob = block_scan(big ? 1 : 0, sm, &tb);
    if (big) {
      s_oc[ob] = oc;
      s_node[ob] = i;
      s_start[ob] = st;
      s_end[ob] = en;
      big_list[carry_b + ob] = i;
      node_chunk0[carry_b + ob] = carry_c + oc;
      nodes[i].big = carry_b + ob;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < tb * kSums; k += blockDim.x) acc[(size_t)carry_b * kSums + k] = u128_zero();
    for (int c = part * blockDim.x + threadIdx.x; c < tc; c += parts * blockDim.x) {
      int lo = 0, hi = tb;  // the last listed node whose first chunk is at or before c
      while (hi - lo > 1) {
        const int m = (lo + hi) >> 1;
        if (s_oc[m] <= c) lo = m;
        else hi = m;
      }
      if (carry_c + c < chunk_cap) {
        const int cb = s_start[lo] + (c - s_oc[lo]) * kChunk;
        Chunk ch;
        ch.node = s_node[lo];
        ch.begin = cb;
        ch.end = min(cb + kChunk, s_end[lo]);
        ch.big = carry_b + lo;
        chunks[carry_c + c] = ch;
      }
    }
    __syncthreads();  // the lists may be rewritten after this
    carry_c += tc;
    carry_b += tb;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ls->num_chunks = min(all_c, chunk_cap);
    ls->num_big = all_b;
    if (all_c > chunk_cap) ls->error = 1;
  }
}

// root: clear the roots' own sums, else the smaller children's of this level.
__global__ void k_big_plan(BNode* nodes, LevelState* ls, const int32_t* bbig, Chunk* chunks, int32_t chunk_cap,
                           int32_t* big_list, int32_t* node_chunk0, U128* root_acc, ChildSums C, int parts) {
  grid_begin();
  __shared__ int sm[32];
  level_plan(nodes, ls, bbig, chunks, chunk_cap, big_list, node_chunk0, root_acc ? root_acc : C.acc[ls->depth & 1], sm,
             (int)blockIdx.x % parts, parts);
}

// Block sum of the warps' sums into one 128-bit accumulator set (any order: exact).
// alone: the block has one chunk only (a small level, where latency counts): each warp adds
// its own.
__device__ __forceinline__ void block_add_sums(LaneSums& S, int lane, U128 (*sm)[kSums], U128* dst, bool alone) {
  lane_fold(S, lane);
  if (alone) {
    if (lane < kSums) atomic_add_u128(&dst[lane], S.tot);
    return;
  }
  if (lane < kSums) sm[threadIdx.x >> 5][lane] = S.tot;
  S.tot = u128_zero();
  __syncthreads();
  if (threadIdx.x < kSums) {
    U128 t = u128_zero();
    for (int ww = 0; ww < (int)(blockDim.x >> 5); ++ww) t = u128_add(t, sm[ww][threadIdx.x]);
    atomic_add_u128(&dst[threadIdx.x], t);
  }
  __syncthreads();
}

constexpr int kFoldChunks = kLanePoints / kPer;

// Level 0: the large roots' sums; a block takes a contiguous range of chunks and adds its
// sums once per root.
__global__ void __launch_bounds__(kThreads, 2) k_big_moments(const Chunk* chunks, const LevelState* ls,
                                                             const PointBufs B, U128* acc) {
  grid_begin();
  __shared__ U128 sm[kSegs][kSums];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  LaneSums S;
  lane_zero(S);
  S.tot = u128_zero();
  const int nc = ls->num_chunks;
  const float4* pts = B.p[ls->cur];
  const int per = (nc + gridDim.x - 1) / gridDim.x;
  const int c0 = blockIdx.x * per, c1 = min(c0 + per, nc);
  int big = -1, held = 0;
  for (int ci = c0; ci < c1; ++ci) {
    const Chunk c = chunks[ci];
    if (c.big != big) {
      if (big >= 0) block_add_sums(S, lane, sm, acc + (size_t)big * kSums, false);
      big = c.big;
      held = 0;
    } else if (++held == kFoldChunks) {
      lane_fold(S, lane);
      held = 0;
    }
    float4 pv[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = c.begin + (w * kPer + u) * 32 + lane;
      if (i < c.end) pv[u] = pts[i];
    }
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int u = 0; u < kPer / 2; ++u)
        lane_add(S, c.begin + (w * kPer + 2 * h + u) * 32 + lane < c.end, h ? pv[2 + u] : pv[u], lane);
    }
  }
  if (big >= 0) block_add_sums(S, lane, sm, acc + (size_t)big * kSums, per == 1);
}

// Level 0: the sums of the large roots, from the chunk accumulators.
__global__ void k_big_to_mom(const LevelState* ls, const int32_t* big_list, const U128* acc, U128* mom) {
  grid_begin();
  const int nb = ls->num_big;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nb * kSums; t += gridDim.x * blockDim.x)
    mom[(size_t)big_list[t / kSums] * kSums + t % kSums] = acc[t];
}

// The eight counts of a chunk, and their sum before segment w (w = 8: of all).
__device__ __forceinline__ int seg_before(const SegCounts& s, int w) {
  int n = 0;
#pragma unroll
  for (int k = 0; k < kSegs; ++k)
    if (k < w) n += s.n[k];
  return n;
}

// Stable scatter by warp ballots: warp w of a block moves segment w of each of its chunks, in
// four rounds of 32 points, so left and right runs are written contiguously.  The points
// that go to the node's smaller child are summed on the way (the sums of the large node's
// smaller child).  A block takes a contiguous range of chunks and its warps keep their sums
// until the range reaches another node: only there do they meet, for one block total and 9
// atomics.  Bound by issue and memory together: a level of 11.4M points takes 110 us (3.3 TB/s
// of records read and written; the node offsets included).  With eleven 128-bit terms per lane,
// reduced per warp and chunk and added with 22 atomics each, it took 235-310 us, and 691 us on
// the root, where every warp hits the same words; three blocks per SM spill and take 118 us.
__global__ void __launch_bounds__(kThreads, kScatterPerSM)
    k_big_scatter(const Chunk* chunks, LevelState* ls, BNode* nodes, PointBufs B, const SegCounts* seg,
                  const int32_t* node_chunk0, ChildSums C, const int32_t* bsum, int nblocks, int32_t cap,
                  unsigned* done) {
  grid_begin();
  __shared__ U128 smm[kSegs][kSums];
  __shared__ int s_pre[kSegs], s_tot[kSegs];
  const int nc = ls->num_chunks, nbig = ls->num_big, cur = ls->cur;
  const float4* pin = B.p[cur];
  float4* pout = B.p[cur ^ 1];
  U128* accl = C.acc[ls->depth & 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  LaneSums S;
  lane_zero(S);
  S.tot = u128_zero();
  const int per = (nc + gridDim.x - 1) / gridDim.x;
  const int c0 = blockIdx.x * per, c1 = min(c0 + per, nc);
  // the current large node (block-uniform); its points' sums are in S
  int big = -1, held = 0;
  float mean[3], dir[3];
  int nstart = 0, nmid = 0;
  int before = 0;  // left points of the node's chunks before this one
  bool split = false, small_left = false;
  for (int ci = c0; ci < c1; ++ci) {
    const Chunk c = chunks[ci];
    const int wb = c.begin + w * 32 * kPer;  // this warp's first point
    float4 pv[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u)
      if (wb + u * 32 + lane < c.end) pv[u] = pin[wb + u * 32 + lane];
    const SegCounts sc = seg[ci];
    if (c.big != big) {
      if (split) block_add_sums(S, lane, smm, accl + (size_t)big * kSums, false);
      big = c.big;
      held = 0;
      BNode& nd = nodes[c.node];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        mean[k] = nd.mean[k];
        dir[k] = nd.dir[k];
      }
      split = nd.split != 0;
      nstart = nd.start;
      // the node's left points, and those before this chunk, from its chunks' counts (every
      // block of the node adds them up itself: no pass of its own over the counts)
      const int n0 = node_chunk0[big], n1 = big + 1 < nbig ? min(node_chunk0[big + 1], nc) : nc;
      const bool few = n1 - n0 <= 64;  // each warp for itself, no barrier
      int pre = 0, tot = 0;
      for (int k = n0 + (few ? lane : (int)threadIdx.x); k < n1; k += few ? 32 : kThreads) {
        const int n = seg_before(seg[k], kSegs);
        tot += n;
        if (k < ci) pre += n;
      }
      pre = __reduce_add_sync(0xffffffffu, pre);
      tot = __reduce_add_sync(0xffffffffu, tot);
      if (!few) {
        if (lane == 0) {
          s_pre[w] = pre;
          s_tot[w] = tot;
        }
        __syncthreads();
        pre = tot = 0;
#pragma unroll
        for (int k = 0; k < kSegs; ++k) {
          pre += s_pre[k];
          tot += s_tot[k];
        }
        __syncthreads();  // they may be rewritten after this
      }
      before = pre;
      nmid = nstart + tot;
      const int nend = nd.end;
      small_left = nmid - nstart <= nend - nmid;
      if (ci == n0 && threadIdx.x == 0) {  // the node's first block: its children's ranges
        nd.mid = split ? nmid : nend;
        if (split) {
          nodes[nd.left].start = nstart;
          nodes[nd.left].end = nmid;
          nodes[nd.right].start = nmid;
          nodes[nd.right].end = nend;
          atomicMax(&ls->max_next, max(nmid - nstart, nend - nmid));
        }
      }
    } else if (++held == kFoldChunks) {
      lane_fold(S, lane);
      held = 0;
    }
    if (!split) {
#pragma unroll
      for (int u = 0; u < kPer; ++u)
        if (wb + u * 32 + lane < c.end) B.perm[wb + u * 32 + lane] = __float_as_int(pv[u].w);
      continue;
    }
    const int loff = before + seg_before(sc, w);  // left points of the node before this segment
    before += seg_before(sc, kSegs);
    int lo = nstart + loff;
    int ro = nmid + min(wb, c.end) - nstart - loff;  // the node's points before this segment, less the left ones
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const bool valid = wb + u * 32 + lane < c.end;
      const bool left = valid && which_side_f(mean, dir, pv[u]);
      const unsigned bl = __ballot_sync(0xffffffffu, left), br = __ballot_sync(0xffffffffu, valid && !left);
      if (valid) pout[left ? lo + __popc(bl & lt) : ro + __popc(br & lt)] = pv[u];
      lane_add(S, valid && left == small_left, pv[u], lane);
      lo += __popc(bl);
      ro += __popc(br);
    }
  }
  if (split) block_add_sums(S, lane, smm, accl + (size_t)big * kSums, per == 1);
  advance_if_last(ls, bsum, nblocks, cap, done);
}

// ---- children ------------------------------------------------------------------------

// Numbers the level's children and writes their records, eight lanes a record (16 B each), so
// that a warp's store is 512 B in a row (a thread per parent writing both of its children's
// records took 100 us for a level of 500,000 nodes, now 63).
__device__ __forceinline__ void level_children(BNode* nodes, LevelState* ls, const int32_t* bsum, int32_t cap, int* sm) {
  __shared__ int s_list[kThreads];  // split nodes of the batch, in order
  int b, e;
  level_range(ls, b, e);
  const int le = ls->le;
  int pre;  // split nodes of the blocks before this one
  {
    int v = 0;
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += blockDim.x) v += bsum[k];
    block_scan(v, sm, &pre);
  }
  int first = le + 2 * pre;  // index of the batch's first child
  for (int base = b; base < e; base += blockDim.x) {
    const int i = base + threadIdx.x;
    bool sp = (i < e) && nodes[i].split;
    int tot;
    const int r = block_scan(sp ? 1 : 0, sm, &tot);
    if (i < e) {
      BNode& nd = nodes[i];
      const int li = first + 2 * r;
      if (sp && li + 1 >= cap) {
        ls->error = 1;
        nd.split = 0;
        sp = false;
      }
      nd.left = sp ? li : -1;
      nd.right = sp ? li + 1 : -1;
      if (sp) s_list[r] = i;
    }
    __syncthreads();
    const int room = min(2 * tot, max(0, (cap - first) & ~1));  // children that fit (all, or the build fails)
    for (int k = threadIdx.x; k < room * 8; k += blockDim.x) {
      const int child = k >> 3, word = k & 7;
      const int par = s_list[child >> 1];
      const BNode& nd = nodes[par];
      int4 w = make_int4(0, 0, 0, 0);  // start and end: set by the partition
      if (word == 0) {
        w.z = nd.level + 1;
        w.w = nd.tree;
      } else if (word == 1) {
        w.z = w.w = -1;  // left, right
      } else if (word == 2) {
        w = make_int4(1, nd.has_prop, 0, par);  // has_parent, par_has, has_prop, parent
      } else if (word == 6) {
        const long long p0 = __double_as_longlong(nd.prop[0]);
        w.z = (int)p0;
        w.w = (int)(p0 >> 32);
      } else if (word == 7) {
        const long long p1 = __double_as_longlong(nd.prop[1]), p2 = __double_as_longlong(nd.prop[2]);
        w = make_int4((int)p1, (int)(p1 >> 32), (int)p2, (int)(p2 >> 32));
      }
      reinterpret_cast<int4*>(nodes + first + child)[word] = w;
    }
    first += 2 * tot;
    __syncthreads();  // the list may be rewritten after this
  }
}
static_assert(offsetof(BNode, level) == 8 && offsetof(BNode, tree) == 12 && offsetof(BNode, left) == 24 &&
                  offsetof(BNode, right) == 28 && offsetof(BNode, has_parent) == 32 && offsetof(BNode, par_has) == 36 &&
                  offsetof(BNode, has_prop) == 40 && offsetof(BNode, parent) == 44 && offsetof(BNode, par_prop) == 104,
              "BNode words as level_children writes them");
__global__ void __launch_bounds__(kThreads) k_level_children(BNode* nodes, LevelState* ls, const int32_t* bsum,
                                                             int32_t cap, int plan, const int32_t* bbig, Chunk* chunks,
                                                             int32_t chunk_cap, int32_t* big_list,
                                                             int32_t* node_chunk0, ChildSums C) {
  grid_begin();
  __shared__ int sm[32];
  level_children(nodes, ls, bsum, cap, sm);
  if (plan) level_plan(nodes, ls, bbig, chunks, chunk_cap, big_list, node_chunk0, C.acc[ls->depth & 1], sm, 0, 1);
}

// A level of at most kThreads nodes: decisions, children and the large nodes' chunks by one
// block in one launch (8 + 2.5 + 3.5 us and two gaps as three kernels, whose later two read
// back what the first wrote).
__global__ void __launch_bounds__(kThreads) k_level_small(BNode* nodes, LevelState* ls, U128* mom, ChildSums C,
                                                          BuildParams P, int32_t* bsum, int32_t* bbig,
                                                          double* root_frame, int32_t cap, Chunk* chunks,
                                                          int32_t chunk_cap, int32_t* big_list, int32_t* node_chunk0,
                                                          int plan) {
  grid_begin();
  __shared__ int sm[32];
  level_decide(nodes, ls, mom, C, P, bsum, bbig, root_frame, sm);
  __syncthreads();
  level_children(nodes, ls, bsum, cap, sm);
  if (!plan) return;
  __syncthreads();
  level_plan(nodes, ls, bbig, chunks, chunk_cap, big_list, node_chunk0, C.acc[ls->depth & 1], sm, 0, 1);
}

// ---- deep levels: whole subtrees in shared memory --------------------------------------
// Once every node of a level is small enough, each of them is the root of a subtree that one
// group of threads builds to the end in shared memory: the points are loaded once, and every
// depth below runs the same steps as the level kernels -- decide (thread per node, from the
// node's exact sums), children numbered by a scan, stable ballot partition by whichSide (a
// warp per node) with the smaller child summed on the way (the other = parent - smaller).  The
// arithmetic and the partition order are those of k_decide / k_small_part, so the nodes are
// bit-identical to a level-by-level build.  Nodes below the roots are written as DeepNode
// records tagged (subtree, depth, rank); k_deep_place then puts them at their breadth-first
// positions: depth by depth, subtree by subtree in the roots' order, by rank inside a subtree
// -- the order in which the level kernels would have numbered them.
//
// Two forms, both for levels that leave most of the machine idle, where a level costs its
// launches and the chain of one decision however few nodes it has:
//  * a block of 16 warps per subtree of at most 2,048 points, while the level has at most
//    kBlockRoots of them: a 12,000-point scan leaves the level kernels after 4 levels (of
//    45 us each) for 91 us here, a 180,000-point one after 8 for 149;
//  * a warp per subtree of at most 256 points, up to 8,192 of them.
// For large forests (hundreds of thousands of tiny subtrees, where a decision runs on a few
// lanes) the level kernels, with a thread per node of the whole level, are faster: the warp
// form on all deep levels of 80 scans took 7.1 ms in place of 4.8.
template <int WARPS>
struct DeepForm;
template <>
struct DeepForm<1> {
  static constexpr int kPoints = 256, kGroups = 4, kPerSM = 4, kRoots = 8192;
};
template <>
struct DeepForm<16> {
  static constexpr int kPoints = 2048, kGroups = 1, kPerSM = 1, kRoots = 296;
};
constexpr int kDeepMax = DeepForm<1>::kPoints;
constexpr int kDeepMaxRoots = DeepForm<1>::kRoots;
constexpr int kBlockMax = DeepForm<16>::kPoints;
constexpr int kBlockRoots = DeepForm<16>::kRoots;
// nodes of one depth: at most two children per split node, which holds at least three points
template <int WARPS>
constexpr int deep_nodes() { return (2 * (DeepForm<WARPS>::kPoints / 3) + 31) / 32 * 32; }

struct DeepNode {
  float mean[3], dir[3];
  double prop[3];
  int32_t start, end;     // point offsets inside the subtree
  int32_t sub;            // subtree ordinal: its root is node lb + sub
  int32_t depth;          // >= 1: levels below the root
  int32_t rank;           // breadth-first position among the subtree's nodes of this depth
  int32_t q;              // split nodes: children ranks 2q, 2q + 1; leaves: -1
  int32_t parent_rank;    // rank of the parent at depth - 1
  int32_t has_prop;
};
static_assert(sizeof(DeepNode) == 80, "DeepNode layout");
static_assert(sizeof(DeepNode) <= kSums * sizeof(U128), "a DeepNode fits the sums slot of one node");

// The sums of a depth's nodes: a subtree of n points has at most max(1, 2 (n / 3)) nodes a depth
// (two children per split node, which holds at least three points).  First slot of the subtree
// that is the sub-th of its level and starts at point `start`; deep_sum_slot(N, roots) in all.
__host__ __device__ __forceinline__ int32_t deep_sum_slot(int64_t start, int32_t sub) {
  return (int32_t)(2 * start / 3) + sub;
}

template <int WARPS>
struct DeepSmem {                             // one group's
  float4 pts[2][DeepForm<WARPS>::kPoints];    // the 16 B point records (w = input index)
  SumStage stage[WARPS];
  uint32_t range[2][deep_nodes<WARPS>()];     // node start | end << 16 (subtree offsets), by depth parity
  int32_t prank[2][deep_nodes<WARPS>()];      // parent's rank, by depth parity
  int32_t list[deep_nodes<WARPS>()];          // q -> rank of the q-th split node of the depth
  int32_t scan[32];
  int32_t base, pad_[3];
  U128 part[WARPS][kSums + 1];                // a node's warps: their sums; [kSums].lo: left points
  // mean and direction of the depth's nodes for the partition (one warp reads its records back:
  // its four groups fill the SM's shared memory).  With the next depth's record slots asked
  // for during the partition, scans of 12,000 and 23,000 points take 322 and 369 us in place of
  // 324 and 377 (both builds alternating in one process).
  float plane[WARPS > 1 ? deep_nodes<WARPS>() : 1][6];
  uint8_t split[deep_nodes<WARPS>()];
};

template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS * DeepForm<WARPS>::kGroups, DeepForm<WARPS>::kPerSM)
    k_deep_build(BNode* nodes, LevelState* ls, PointBufs B, const U128* mom, ChildSums C, BuildParams P,
                 double* root_frame, DeepNode* dn, int32_t dn_cap, int32_t* dn_count, U128* sums, int32_t sum_slots,
                 int32_t group_slots, int32_t* counts, int32_t dcap) {
  grid_begin();
  constexpr int kThreadsG = 32 * WARPS;
  extern __shared__ __align__(16) unsigned char deep_smem_raw[];
  const int lane = threadIdx.x & 31, group = WARPS == 1 ? (int)threadIdx.x >> 5 : 0;
  const int tid = WARPS == 1 ? lane : (int)threadIdx.x, warp = WARPS == 1 ? 0 : (int)threadIdx.x >> 5;
  auto sync = []() {  // the group's threads
    if (WARPS == 1) __syncwarp();
    else __syncthreads();
  };
  DeepSmem<WARPS>& S = reinterpret_cast<DeepSmem<WARPS>*>(deep_smem_raw)[group];
  SumStage& sg = S.stage[warp];
  const int lb = ls->lb, le = ls->le, cur0 = ls->cur, depth0 = ls->depth;
  const int nroots = le - lb;
  const unsigned full = 0xffffffffu, lt = (1u << lane) - 1u;
  const int gw = blockIdx.x * DeepForm<WARPS>::kGroups + group, nw = gridDim.x * DeepForm<WARPS>::kGroups;
  stage_init(sg, lane);
  WarpSums W;
  sums_zero(W);
  const float4* pin = B.p[cur0];
  for (int sub = gw; sub < nroots; sub += nw) {
    const int R = lb + sub;
    const BNode root = nodes[R];
    const int n = root.end - root.start;
    const int pbase = root.start;
    // the subtree's slots for the sums of one depth's nodes, and of the next one's: its own, or
    // (group_slots) the group's, whichever are fewer in all
    U128* const sums0 = sums + (size_t)(group_slots ? gw * group_slots : deep_sum_slot(pbase, sub)) * kSums;
    U128* const sums1 = sums0 + (size_t)sum_slots * kSums;
    for (int i = tid; i < n; i += kThreadsG) S.pts[0][i] = pin[pbase + i];
    if (tid == 0) {
      S.range[0][0] = (uint32_t)n << 16;
      S.prank[0][0] = -1;
    }
    if (tid < kSums) {  // the root's sums
      const PendingSums ps = pending_sums(nodes, mom, C, depth0, R, root.parent);
      sums0[tid] = ps.q ? pending_value(ps, tid) : mom[(size_t)R * kSums + tid];
    }
    sync();
    int cnt = 1, c = 0, base = 0, base_prev = 0;
    for (int d = 0; cnt > 0; ++d, c ^= 1) {
      // ---- decide: thread per node of this depth; record slots for the depth's nodes
      if (d > 0) {
        base_prev = base;
        base = S.base;
        if (base + cnt > dn_cap) {
          if (tid == 0) ls->error = 1;  // out of record slots: the build reports KDS_ERR_CAPACITY
          break;
        }
      }
      const U128* psums = d & 1 ? sums1 : sums0;
      for (int r = tid; r < cnt; r += kThreadsG) {
        const uint32_t rg = S.range[c][r];
        const int st = (int)(rg & 0xffffu), en = (int)(rg >> 16);
        double pp[3];
        bool ph;
        if (d == 0) {
          ph = root.has_parent && root.par_has;
          for (int k = 0; k < 3; ++k) pp[k] = root.par_prop[k];
        } else if (d == 1) {  // the root's decision, written at depth 0
          ph = nodes[R].has_prop != 0;
          for (int k = 0; k < 3; ++k) pp[k] = nodes[R].prop[k];
        } else {
          const DeepNode& pn = dn[base_prev + S.prank[c][r]];
          ph = pn.has_prop != 0;
          for (int k = 0; k < 3; ++k) pp[k] = pn.prop[k];
        }
        double Sd[kSums];
        const U128* ms = psums + (size_t)r * kSums;
#pragma unroll
        for (int k = 0; k < kSums; ++k) Sd[k] = fx_to_d(ms[k]);
        const Decision x = decide(Sd, en - st, ph, pp, root.level + d, P,
                                  root.level + d == 0 ? root_frame + (size_t)root.tree * kRootFrame : nullptr);
        S.split[r] = x.split ? 1 : 0;
        if (WARPS > 1) {
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            S.plane[r][k] = x.mean[k];
            S.plane[r][3 + k] = x.dir[k];
          }
        }
        if (d == 0) {  // left / right follow in k_deep_place
          BNode& o = nodes[R];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            o.mean[k] = x.mean[k];
            o.dir[k] = x.dir[k];
            o.prop[k] = x.prop[k];
          }
          o.split = x.split ? 1 : 0;
          o.has_prop = x.has_prop ? 1 : 0;
        } else {
          DeepNode& o = dn[base + r];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            o.mean[k] = x.mean[k];
            o.dir[k] = x.dir[k];
            o.prop[k] = x.prop[k];
          }
          o.start = st;
          o.end = en;
          o.sub = sub;
          o.depth = d;
          o.rank = r;
          o.q = -1;
          o.parent_rank = S.prank[c][r];
          o.has_prop = x.has_prop ? 1 : 0;
        }
      }
      sync();
      // ---- children numbering: split ranks by a scan in rank order
      int nsplit = 0;
      for (int r0 = 0; r0 < cnt; r0 += kThreadsG) {
        const int r = r0 + tid;
        const bool f = r < cnt && S.split[r];
        int q, total;
        if (WARPS == 1) {
          const unsigned bf = __ballot_sync(full, f);
          q = __popc(bf & lt);
          total = __popc(bf);
        } else {
          q = block_scan(f ? 1 : 0, S.scan, &total);
        }
        if (f) {
          S.list[nsplit + q] = r;
          if (d > 0) dn[base + r].q = nsplit + q;
        }
        nsplit += total;
      }
      if (3 * nsplit > n) {  // cannot happen (split nodes hold >= 3 points); refuse rather than overrun
        if (tid == 0) ls->error = 1;
        break;
      }
      int next_base = 0;  // record slots of the next depth: in flight during the partition
      if (nsplit > 0 && tid == 0) {
        if (d + 1 < dcap) {
          counts[(size_t)(d + 1) * nroots + sub] = 2 * nsplit;
          next_base = atomicAdd(dn_count, 2 * nsplit);
        } else {
          ls->error = 1;
        }
      }
      sync();
      // ---- the leaves' point order (thread per leaf)
      for (int r = tid; r < cnt; r += kThreadsG) {
        if (S.split[r]) continue;
        const uint32_t rg = S.range[c][r];
        const int st = (int)(rg & 0xffffu), en = (int)(rg >> 16);
        for (int i = st; i < en; ++i) B.perm[pbase + i] = __float_as_int(S.pts[c][i].w);
      }
      // ---- partition of the split nodes: several warps per node while there are fewer nodes
      // than warps (one warp takes 20 us for a node of 2,000 points) ...
      int team = 1;  // warps per node
      for (int k = WARPS; k > 1 && nsplit > 0; k /= 2)
        if (2 * team * nsplit <= WARPS) team *= 2;
      if (team > 1) {
        const int q = warp / team, m = warp % team;
        const bool on = q < nsplit;
        int st = 0, en = 0, b = 0, e = 0, r = 0;
        float mean[3], dir[3];
        if (on) {
          r = S.list[q];
          const uint32_t rg = S.range[c][r];
          st = (int)(rg & 0xffffu);
          en = (int)(rg >> 16);
          const int per = (en - st + 32 * team - 1) / (32 * team) * 32;
          b = min(st + m * per, en);
          e = min(b + per, en);
          for (int k = 0; k < 3; ++k) { mean[k] = S.plane[r][k]; dir[k] = S.plane[r][3 + k]; }
          int nl = 0;
          for (int k0 = b; k0 < e; k0 += 32) {
            const int i = k0 + lane;
            nl += __popc(__ballot_sync(full, i < e && which_side_f(mean, dir, S.pts[c][i])));
          }
          if (lane == 0) S.part[warp][kSums].lo = (unsigned long long)nl;
        }
        sync();
        int mid = st, lo = st;
        if (on) {
          for (int k = 0; k < team; ++k) {
            const int nl = (int)S.part[q * team + k][kSums].lo;
            mid += nl;
            if (k < m) lo += nl;
          }
          int ro = mid + (b - st) - (lo - st);
          const bool small_left = mid - st <= en - mid;
          for (int k0 = b; k0 < e; k0 += 32) {
            const int i = k0 + lane;
            const bool valid = i < e;
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
            if (valid) p = S.pts[c][i];
            const bool left = valid && which_side_f(mean, dir, p);
            const unsigned bl = __ballot_sync(full, left), br = __ballot_sync(full, valid && !left);
            if (valid) S.pts[c ^ 1][left ? lo + __popc(bl & lt) : ro + __popc(br & lt)] = p;
            sums_add(W, sg, valid && left == small_left, p, lane);
            sums_room(W, sg, kStage - 32, lane);
            lo += __popc(bl);
            ro += __popc(br);
          }
          const U128 qs = sums_total(W, sg, lane);
          if (lane < kSums) S.part[warp][lane] = qs;
        }
        sync();
        if (on && m == 0) {
          const bool small_left = mid - st <= en - mid;
          if (lane < kSums) {
            U128 qs = u128_zero();
            for (int k = 0; k < team; ++k) qs = u128_add(qs, S.part[warp + k][lane]);
            const U128 other = u128_sub(psums[(size_t)r * kSums + lane], qs);
            U128* nxt = d & 1 ? sums0 : sums1;
            nxt[(size_t)(2 * q) * kSums + lane] = small_left ? qs : other;
            nxt[(size_t)(2 * q + 1) * kSums + lane] = small_left ? other : qs;
          }
          if (lane == 0) {
            S.range[c ^ 1][2 * q] = (uint32_t)st | ((uint32_t)mid << 16);
            S.range[c ^ 1][2 * q + 1] = (uint32_t)mid | ((uint32_t)en << 16);
            S.prank[c ^ 1][2 * q] = r;
            S.prank[c ^ 1][2 * q + 1] = r;
          }
        }
      }
      // ... a warp per node then
      for (int q = team > 1 ? nsplit : warp; q < nsplit; q += WARPS) {
        const int r = S.list[q];
        const uint32_t rg = S.range[c][r];
        const int st = (int)(rg & 0xffffu), en = (int)(rg >> 16);
        float mean[3], dir[3];
        if (WARPS > 1) {
          for (int k = 0; k < 3; ++k) { mean[k] = S.plane[r][k]; dir[k] = S.plane[r][3 + k]; }
        } else if (d == 0) {
          for (int k = 0; k < 3; ++k) { mean[k] = nodes[R].mean[k]; dir[k] = nodes[R].dir[k]; }
        } else {
          const DeepNode& x = dn[base + r];
          for (int k = 0; k < 3; ++k) { mean[k] = x.mean[k]; dir[k] = x.dir[k]; }
        }
        int nl = 0;
        for (int k0 = st; k0 < en; k0 += 32) {
          const int i = k0 + lane;
          const bool left = i < en && which_side_f(mean, dir, S.pts[c][i]);
          nl += __popc(__ballot_sync(full, left));
        }
        const int mid = st + nl;
        const bool small_left = mid - st <= en - mid;
        int cl = 0, cr = 0;
        for (int k0 = st; k0 < en; k0 += 32) {
          const int i = k0 + lane;
          const bool valid = i < en;
          float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
          if (valid) p = S.pts[c][i];
          const bool left = valid && which_side_f(mean, dir, p);
          const unsigned bl = __ballot_sync(full, left);
          const unsigned br = __ballot_sync(full, valid && !left);
          if (valid) {
            const int dst = left ? (st + cl + __popc(bl & lt)) : (mid + cr + __popc(br & lt));
            S.pts[c ^ 1][dst] = p;
          }
          sums_add(W, sg, valid && left == small_left, p, lane);
          sums_room(W, sg, kStage - 32, lane);
          cl += __popc(bl);
          cr += __popc(br);
        }
        const U128 qs = sums_total(W, sg, lane);
        if (lane < kSums) {
          const int k = lane;
          const U128 ps = psums[(size_t)r * kSums + k];
          const U128 other = u128_sub(ps, qs);
          U128* nxt = d & 1 ? sums0 : sums1;
          nxt[(size_t)(2 * q) * kSums + k] = small_left ? qs : other;
          nxt[(size_t)(2 * q + 1) * kSums + k] = small_left ? other : qs;
        }
        if (lane == 0) {
          S.range[c ^ 1][2 * q] = (uint32_t)st | ((uint32_t)mid << 16);
          S.range[c ^ 1][2 * q + 1] = (uint32_t)mid | ((uint32_t)en << 16);
          S.prank[c ^ 1][2 * q] = r;
          S.prank[c ^ 1][2 * q + 1] = r;
        }
      }
      cnt = 2 * nsplit;
      if (d + 1 >= dcap) cnt = 0;
      if (tid == 0) S.base = next_base;
      sync();
    }
    sync();
  }
}

// Deep nodes to their breadth-first positions: node (subtree s, depth d, rank r) goes to
// le + off[d * nroots + s] + r, where off is the exclusive scan of the per-(depth,
// subtree) node counts in depth-major order.  The roots get their children's indices.
__global__ void k_deep_place(BNode* nodes, LevelState* ls, int32_t lb, int32_t le, const DeepNode* dn,
                             const int32_t* dn_count, int32_t dn_cap, const int32_t* off, int32_t dcap,
                             int32_t cap_nodes, int32_t* alive) {
  grid_begin();
  if (ls->error) return;  // the build fails; records may be missing
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ls->le; i += gridDim.x * blockDim.x) alive[i] = 0;
  const int nroots = le - lb;
  const int nd_total = min(*dn_count, dn_cap);
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nroots; i += stride) {
    BNode& rt = nodes[lb + i];
    if (rt.split && dcap > 1) {
      rt.left = le + off[(size_t)1 * nroots + i];
      rt.right = rt.left + 1;
    } else {
      rt.left = rt.right = -1;
    }
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nd_total; i += stride) {
    const DeepNode x = dn[i];
    const int s = x.sub, d = x.depth;
    const BNode& rt = nodes[lb + s];
    BNode o;
    memset(&o, 0, sizeof(o));
    o.start = rt.start + x.start;
    o.end = rt.start + x.end;
    o.level = rt.level + d;
    o.tree = rt.tree;
    o.split = x.q >= 0 ? 1 : 0;
    o.mid = o.end;
    o.left = o.right = -1;
    if (x.q >= 0 && d + 1 < dcap) {
      o.left = le + off[(size_t)(d + 1) * nroots + s] + 2 * x.q;
      o.right = o.left + 1;
    }
    o.has_parent = 1;
    o.has_prop = x.has_prop;
    o.parent = d == 1 ? lb + s : le + off[(size_t)(d - 1) * nroots + s] + x.parent_rank;
    for (int k = 0; k < 3; ++k) {
      o.mean[k] = x.mean[k];
      o.dir[k] = x.dir[k];
      o.prop[k] = x.prop[k];
    }
    const int g = le + off[(size_t)d * nroots + s] + x.rank;
    if (g >= cap_nodes) {
      ls->error = 1;
      continue;
    }
    nodes[g] = o;
  }
}

// One block: the level state after the deep levels (every level done), the depth, and the node capacity check (a thread per depth; one thread for all took
// 11 us of dependent loads).
__device__ __forceinline__ void deep_finish(LevelState* ls, int32_t lb, int32_t le, const int32_t* off, int32_t tot,
                                            int32_t dcap, int32_t cap_nodes) {
  __shared__ int s_dmax;  // deepest local depth holding nodes
  const int depth0 = ls->depth;
  const bool failed = ls->error != 0;
  if (threadIdx.x == 0) s_dmax = 0;
  __syncthreads();
  if (failed) return;
  const int nroots = le - lb;
  for (int d = 1 + threadIdx.x; d < dcap; d += blockDim.x) {
    const int b = off[(size_t)d * nroots];
    const int e = d + 1 < dcap ? off[(size_t)(d + 1) * nroots] : tot;
    if (e > b) atomicMax(&s_dmax, d);
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (le + tot > cap_nodes) ls->error = 1;
  ls->depth = depth0 + s_dmax + 1;
  ls->lb = ls->le = le + tot;
}
__global__ void k_deep_finish(LevelState* ls, int32_t lb, int32_t le, const int32_t* off, const int32_t* total,
                              int32_t dcap, int32_t cap_nodes) {
  grid_begin();
  deep_finish(ls, lb, le, off, *total, dcap, cap_nodes);
}
// The same with the scan of the counts by the one block: up to kDeepScan counts, a run per
// thread (three scan launches and this otherwise).
constexpr int kDeepScan = 16384;
__global__ void __launch_bounds__(1024) k_deep_scan(LevelState* ls, int32_t lb, int32_t le, const int32_t* counts,
                                                    int32_t ncount, int32_t* off, int32_t dcap, int32_t cap_nodes) {
  grid_begin();
  __shared__ int sm[32];
  const int per = (ncount + 1023) / 1024;
  const int b = min((int)threadIdx.x * per, ncount), e = min(b + per, ncount);
  int v = 0;
  for (int i = b; i < e; ++i) v += counts[i];
  int tot;
  int x = block_scan(v, sm, &tot);
  for (int i = b; i < e; ++i) {
    off[i] = x;
    x += counts[i];
  }
  __syncthreads();
  deep_finish(ls, lb, le, off, tot, dcap, cap_nodes);
}

// ---- prune and per-tree compaction -----------------------------------------------------
// Nodes of a finished build, on the device: the host sizes the launches below by what there can
// be and does not wait for the subtree pass (a 180,000-point scan: 937 us with the wait, 866
// without).  A build that failed has none: its records may be incomplete.
__device__ __forceinline__ int built_nodes(const LevelState* ls) { return ls->error ? 0 : ls->le; }

// Prune in one launch (alive[] zeroed before): a leaf lives if it passes
// IsGoodLeafPredicate_ (kd/tree/tree_predicates_.h:18-29, in float), an inner node if
// any child lives, i.e. if a good leaf lies below it (kd/tree/tree_cpu_.h:172-196).  Each
// good leaf marks its ancestors up to the first one already marked: whoever marks a node
// first goes on to its parent, so every ancestor ends marked whatever the order.
__global__ void k_alive(const BNode* nodes, const LevelState* ls, int32_t* alive, float incidence) {
  grid_begin();
  const int total = built_nodes(ls);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const BNode& nd = nodes[i];
    if (nd.left >= 0 || nd.right >= 0) continue;
    F3 d = f3(nd.dir[0], nd.dir[1], nd.dir[2]);
    F3 m = f3(nd.mean[0], nd.mean[1], nd.mean[2]);
    if (!(dot3x(d, d) > 0.0f && fabsf(dot3x(m, d)) > incidence)) continue;
    alive[i] = 1;
    for (int p = nd.parent; p >= 0; p = nodes[p].parent) {
      if (((volatile int32_t*)alive)[p]) break;
      alive[p] = 1;
    }
  }
}

// group = (level, tree); nodes of one group are contiguous in global order
// Counts per (level, tree) group.  A block takes a contiguous range of nodes and keeps its
// counts while they stay in one group (2.1M nodes of one tree: 71 us, 85 with the warps'
// atomics meeting at the same three words); in rows of several groups, lanes with the
// same group combine theirs before one atomic per group and warp.
// flags[i]: x = alive, y = alive leaf.
__global__ void __launch_bounds__(kThreads) k_group_counts(const BNode* nodes, const LevelState* ls,
                                                           const int32_t* alive, int R, int32_t* cnt, int32_t* lcnt,
                                                           int32_t* ucnt, int2* flags) {
  grid_begin();
  const int total = built_nodes(ls);
  const int lane = threadIdx.x & 31;
  const int rows = (total + (int)blockDim.x - 1) / (int)blockDim.x;
  const int per = (rows + (int)gridDim.x - 1) / (int)gridDim.x;
  const int row0 = blockIdx.x * per, row1 = min(row0 + per, rows);
  int hg = -1, ht = 0, hn = 0, hc = 0, hl = 0;  // the group held, its tree, nodes, alive nodes and leaves
  auto put = [&]() {
    if (hg < 0 || threadIdx.x != 0) return;
    atomicAdd(&ucnt[ht], hn);
    if (hc) atomicAdd(&cnt[hg], hc);
    if (hl) atomicAdd(&lcnt[hg], hl);
  };
  for (int row = row0; row < row1; ++row) {
    const int base = row * (int)blockDim.x, i = base + (int)threadIdx.x;
    const bool valid = i < total;
    int tree = -1, g = -1;
    bool al = false, leaf = false;
    if (valid) {
      const BNode& nd = nodes[i];
      tree = nd.tree;
      g = nd.level * R + nd.tree;
      al = alive[i] != 0;
      leaf = al && nd.left < 0 && nd.right < 0;
      flags[i] = make_int2(al ? 1 : 0, leaf ? 1 : 0);
    }
    const int t0 = nodes[base].tree, g0 = nodes[base].level * R + t0;
    if (__syncthreads_and(!valid || g == g0)) {
      const int c = __syncthreads_count(al), l = __syncthreads_count(leaf);
      if (g0 != hg) {
        put();
        hg = g0;
        ht = t0;
        hn = hc = hl = 0;
      }
      hn += min((int)blockDim.x, total - base);
      hc += c;
      hl += l;
      continue;
    }
    const unsigned pt = __match_any_sync(0xffffffffu, tree);
    if (valid && lane == __ffs(pt) - 1) atomicAdd(&ucnt[tree], __popc(pt));
    const unsigned pg = __match_any_sync(0xffffffffu, g);
    const unsigned ba = __ballot_sync(0xffffffffu, al);
    const unsigned bl = __ballot_sync(0xffffffffu, leaf);
    if (valid && lane == __ffs(pg) - 1) {
      const int c = __popc(pg & ba), lc = __popc(pg & bl);
      if (c) atomicAdd(&cnt[g], c);
      if (lc) atomicAdd(&lcnt[g], lc);
    }
  }
  put();
}

// Exclusive scan of the flag pairs (both at once), in place: tiles of kFlagTile pairs, their
// sums by one block, then the prefixes; a single block does it all for small trees.
constexpr int kFlagItems = 4;
constexpr int kFlagTile = 1024 * kFlagItems;
constexpr int kFlagOne = 32768;  // pairs that one block scans by itself
__device__ __forceinline__ int2 pair_add(int2 a, int2 b) { return make_int2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ int2 pair_block_scan(int2 v, int* sm, int2* total) {
  int2 r;
  r.x = block_scan(v.x, sm, &total->x);
  r.y = block_scan(v.y, sm, &total->y);
  return r;
}
__global__ void __launch_bounds__(1024) k_flag_tiles(const int2* flags, const LevelState* ls, int2* tiles) {
  grid_begin();
  const int n = built_nodes(ls);
  __shared__ int sm[32];
  const int base = blockIdx.x * kFlagTile + threadIdx.x * kFlagItems;
  int2 v = make_int2(0, 0), tot;
  for (int k = 0; k < kFlagItems; ++k)
    if (base + k < n) v = pair_add(v, flags[base + k]);
  pair_block_scan(v, sm, &tot);
  if (threadIdx.x == 0) tiles[blockIdx.x] = tot;
}
__global__ void __launch_bounds__(1024) k_flag_top(int2* tiles, int32_t nt) {
  grid_begin();
  __shared__ int sm[32];
  int2 carry = make_int2(0, 0);
  for (int b = 0; b < nt; b += blockDim.x) {
    const int i = b + threadIdx.x;
    int2 tot;
    const int2 ex = pair_block_scan(i < nt ? tiles[i] : make_int2(0, 0), sm, &tot);
    if (i < nt) tiles[i] = pair_add(carry, ex);
    carry = pair_add(carry, tot);
  }
}
// tiles == nullptr: one block, a run of pairs per thread.
__global__ void __launch_bounds__(1024) k_flag_scan(int2* flags, const LevelState* ls, const int2* tiles) {
  grid_begin();
  const int n = built_nodes(ls);
  __shared__ int sm[32];
  const int items = tiles ? kFlagItems : (n + 1023) / 1024;
  const int b = min((int)(blockIdx.x * 1024 + threadIdx.x) * items, n), e = min(b + items, n);
  int2 v = make_int2(0, 0), tot;
  for (int i = b; i < e; ++i) v = pair_add(v, flags[i]);
  int2 x = pair_block_scan(v, sm, &tot);
  if (tiles) x = pair_add(x, tiles[blockIdx.x]);
  for (int i = b; i < e; ++i) {
    const int2 f = flags[i];
    flags[i] = x;
    x = pair_add(x, f);
  }
}

// Exclusive prefix over groups in (level, tree) order (one block, scans with carry),
// and per-tree level offsets (one thread per tree).
__global__ void k_group_tables(const LevelState* state, int R, const int32_t* cnt, const int32_t* lcnt, int32_t* gp, int32_t* lgp,
                               int32_t* to, int32_t* lto, int32_t* tot_nodes, int32_t* tot_leaves) {
  grid_begin();
  __shared__ int sm[32];
  const int depth = state->error ? 0 : state->depth;
  const int G = depth * R;
  int carry = 0, lcarry = 0;
  for (int base = 0; base < G; base += blockDim.x) {
    const int g = base + threadIdx.x;
    const int c = g < G ? cnt[g] : 0, lc = g < G ? lcnt[g] : 0;
    int tc, tl;
    const int o = block_scan(c, sm, &tc);
    const int lo = block_scan(lc, sm, &tl);
    if (g < G) {
      gp[g] = carry + o;
      lgp[g] = lcarry + lo;
    }
    carry += tc;
    lcarry += tl;
  }
  for (int t = threadIdx.x; t < R; t += blockDim.x) {
    int s = 0, ls = 0;
    for (int l = 0; l < depth; ++l) {
      const int g = l * R + t;
      to[g] = s;
      lto[g] = ls;
      s += cnt[g];
      ls += lcnt[g];
    }
    tot_nodes[t] = s;
    tot_leaves[t] = ls;
  }
}

// ---- stamps ----------------------------------------------------------------------------
// Prefix sums of (dt, dt^2) over the final point order, exact: a node's sums are the
// difference at the ends of its point range.  One pass at the end in place of the stamps'
// share of every level (a 32 B sector per summed point and level, two 128-bit terms per
// point, and two more sums to reduce per node).  Tiles of kDtTile points: their sums, the
// scan of those by one block, then every position's exclusive prefix.
struct __align__(16) DtSum {
  U128 d, dd;
};
__host__ __device__ __forceinline__ DtSum dt_add(DtSum a, DtSum b) {
  DtSum r;
  r.d = u128_add(a.d, b.d);
  r.dd = u128_add(a.dd, b.dd);
  return r;
}
constexpr int kDtItems = 8;
constexpr int kDtTile = kThreads * kDtItems;
__device__ __forceinline__ DtSum dt_shfl_up(DtSum v, int off) {
  DtSum r;
  r.d.lo = __shfl_up_sync(0xffffffffu, v.d.lo, off);
  r.d.hi = __shfl_up_sync(0xffffffffu, v.d.hi, off);
  r.dd.lo = __shfl_up_sync(0xffffffffu, v.dd.lo, off);
  r.dd.hi = __shfl_up_sync(0xffffffffu, v.dd.hi, off);
  return r;
}
__device__ __forceinline__ DtSum dt_zero() {
  DtSum r;
  r.d = r.dd = u128_zero();
  return r;
}
// Block-wide exclusive scan (kThreads threads); *total = block sum.
__device__ __forceinline__ DtSum dt_block_scan(DtSum v, DtSum* sm, DtSum* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  DtSum x = v;
  for (int off = 1; off < 32; off <<= 1) {
    const DtSum y = dt_shfl_up(x, off);
    if (lane >= off) x = dt_add(x, y);
  }
  DtSum ex = dt_shfl_up(x, 1);
  if (lane == 0) ex = dt_zero();
  if (lane == 31) sm[w] = x;
  __syncthreads();
  DtSum pre = dt_zero(), tot = dt_zero();
  for (int k = 0; k < kThreads / 32; ++k) {
    if (k == w) pre = tot;
    tot = dt_add(tot, sm[k]);
  }
  __syncthreads();
  *total = tot;
  return dt_add(pre, ex);
}
__device__ __forceinline__ void dt_load(const double* dt, const int32_t* perm, int64_t b, int64_t n, DtSum* t) {
  double d[kDtItems];
#pragma unroll
  for (int k = 0; k < kDtItems; ++k) d[k] = b + k < n ? dt[perm[b + k]] : 0.0;
#pragma unroll
  for (int k = 0; k < kDtItems; ++k) {
    t[k].d = fx_d_nonneg(d[k]);
    t[k].dd = fx_d_nonneg(d[k] * d[k]);
  }
}
__global__ void __launch_bounds__(kThreads) k_dt_tiles(const double* dt, const int32_t* perm, int64_t n, DtSum* tiles) {
  grid_begin();
  __shared__ DtSum sm[kThreads / 32];
  DtSum t[kDtItems], tot;
  dt_load(dt, perm, (int64_t)blockIdx.x * kDtTile + threadIdx.x * kDtItems, n, t);
  DtSum v = t[0];
#pragma unroll
  for (int k = 1; k < kDtItems; ++k) v = dt_add(v, t[k]);
  dt_block_scan(v, sm, &tot);
  if (threadIdx.x == 0) tiles[blockIdx.x] = tot;
}
__global__ void __launch_bounds__(kThreads) k_dt_top(DtSum* tiles, int nt) {
  grid_begin();
  __shared__ DtSum sm[kThreads / 32];
  DtSum carry = dt_zero();
  for (int b = 0; b < nt; b += kThreads) {
    const int i = b + threadIdx.x;
    DtSum tot;
    const DtSum ex = dt_block_scan(i < nt ? tiles[i] : dt_zero(), sm, &tot);
    if (i < nt) tiles[i] = dt_add(carry, ex);
    carry = dt_add(carry, tot);
  }
}
// pre[i] for i in [0, n].  tiles: the tiles' sums, scanned already or (at most kThreads of
// them) not, then each block adds up those before it.
__global__ void __launch_bounds__(kThreads) k_dt_prefix(const double* dt, const int32_t* perm, int64_t n,
                                                        const DtSum* tiles, int scanned, DtSum* pre) {
  grid_begin();
  __shared__ DtSum sm[kThreads / 32];
  const int64_t b = (int64_t)blockIdx.x * kDtTile + threadIdx.x * kDtItems;
  DtSum t[kDtItems], tot;
  dt_load(dt, perm, b, n, t);
  DtSum v = t[0];
#pragma unroll
  for (int k = 1; k < kDtItems; ++k) v = dt_add(v, t[k]);
  DtSum x = dt_block_scan(v, sm, &tot);
  if (scanned) {
    x = dt_add(x, tiles[blockIdx.x]);
  } else if (blockIdx.x > 0) {
    dt_block_scan(threadIdx.x < blockIdx.x ? tiles[threadIdx.x] : dt_zero(), sm, &tot);
    x = dt_add(x, tot);
  }
#pragma unroll
  for (int k = 0; k < kDtItems; ++k) {
    if (b + k <= n) {  // two 16 B stores
      ulonglong2* o = reinterpret_cast<ulonglong2*>(pre + b + k);
      o[0] = make_ulonglong2(x.d.lo, x.d.hi);
      o[1] = make_ulonglong2(x.dd.lo, x.dd.hi);
    }
    x = dt_add(x, t[k]);
  }
}

// pre: prefix sums of the stamps over the point order (nullptr: every dt is 0)
// rank[i]: alive nodes and alive leaves before node i.
__global__ void k_compact_forest(const BNode* nodes, int32_t total, const int32_t* alive, const int2* rank, int R,
                                 const int32_t* gp, const int32_t* lgp, const int32_t* to, const int32_t* lto,
                                 const DtSum* pre, const int64_t* off, TreeDev* trees) {
  grid_begin();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    if (!alive[i]) continue;
    const BNode& nd = nodes[i];
    TreeDev& T = trees[nd.tree];
    if (T.nodes == nullptr) continue;  // rejected tree
    int g = nd.level * R + nd.tree;
    const int2 rk = rank[i];
    int o = to[g] + (rk.x - gp[g]);
    int gc = (nd.level + 1) * R + nd.tree;
    int l = (nd.left >= 0 && alive[nd.left]) ? to[gc] + (rank[nd.left].x - gp[gc]) : -1;
    int r = (nd.right >= 0 && alive[nd.right]) ? to[gc] + (rank[nd.right].x - gp[gc]) : -1;
    DNode d;
    d.a = make_float4(nd.mean[0], nd.mean[1], nd.mean[2], nd.dir[0]);
    d.b = make_float4(nd.dir[1], nd.dir[2], __int_as_float(l), __int_as_float(r));
    T.nodes[o] = d;
    double dts_mean = 0.0, dts_cov = 0.0;
    if (pre && nd.end > nd.start) {
      const double dn = (double)(nd.end - nd.start);
      const DtSum a = pre[nd.start], b = pre[nd.end];
      dts_mean = fx_to_d(u128_sub(b.d, a.d)) / dn;
      dts_cov = fx_to_d(u128_sub(b.dd, a.dd)) / dn - dts_mean * dts_mean;
    }
    T.dts_f[o] = (float)dts_mean;
    T.dts_mean[o] = dts_mean;
    T.dts_cov[o] = dts_cov;
    const int64_t o0 = off[nd.tree];  // ranges are global here
    T.range[2 * o] = nd.start - o0;
    T.range[2 * o + 1] = nd.end - o0;
    T.level[o] = nd.level;
    if (nd.left < 0 && nd.right < 0) {
      const int lf = lto[g] + (rk.y - lgp[g]);
      T.leaf_idx[lf] = o;
      T.leaf_md[lf] = make_float4(nd.mean[0], nd.mean[1], nd.mean[2], (float)dts_mean);
      T.leaf_nrm[lf] = make_float4(nd.dir[0], nd.dir[1], nd.dir[2], 0.f);
    }
  }
}

// tree-relative point order; blockIdx.y = tree
__global__ void k_finish_trees(TreeDev* trees, const int64_t* off, const int32_t* perm_final) {
  grid_begin();
  const int r = blockIdx.y;
  TreeDev& T = trees[r];
  if (T.nodes == nullptr) return;
  const int64_t o0 = off[r], n = T.num_points;
  int32_t* out = T.perm;  // read once: the writes could be to the record itself otherwise
  const int32_t* in = perm_final + o0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride) {
    int32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = in[i + k * stride];
#pragma unroll
    for (int k = 0; k < 4; ++k) out[i + k * stride] = v[k] - (int32_t)o0;
  }
  for (; i < n; i += stride) out[i] = in[i] - (int32_t)o0;
}

inline int nblk(int64_t n, int t) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + t - 1) / t, 1 << 20)); }

template <class T> T* carve(char*& p, size_t count) {
  size_t bytes = (count * sizeof(T) + 255) & ~(size_t)255;
  T* r = reinterpret_cast<T*>(p);
  p += bytes;
  return r;
}
template <class T> size_t carve_size(size_t count) { return (count * sizeof(T) + 255) & ~(size_t)255; }

struct BuildWs {
  void* block = nullptr;
  PointBufs B;
  BNode* nodes;
  int32_t* alive;
  int2 *flags, *flag_tiles;  // (alive, leaf) of every node, then the exclusive prefixes
  Chunk* chunks;
  SegCounts* seg;
  int32_t *big_list, *node_chunk0;
  U128* acc;       // the large roots' sums
  ChildSums accl;  // the smaller children's sums of large nodes, by level parity
  U128* mom;   // exact sums of every node, and room for the subtree passes
  U128* mom_end;
  double* ts0;   // per cloud
  double* dt;    // stamps less ts0, input order
  DtSum* dt_tiles;
  double* root_frame;  // kRootFrame per cloud (k_decide at level 0)
  unsigned long long* tsmin;
  int64_t* off;
  // cleared together at the start: from ls to zero_end
  LevelState* ls;
  unsigned* done;  // last-block counter of the level's last kernel
  char* zero_end;
  int32_t* bsum;
  int32_t* bbig;  // per-block (chunks, large nodes) of the level
  int32_t *cnt, *lcnt, *gp, *lgp, *to, *lto;
  // read back together: tot_nodes, tot_leaves, ucnt (R each), then ts0 and root_frame
  int32_t *tot_nodes, *tot_leaves, *ucnt;
  TreeDev* trees;
  int64_t cap_nodes;
  int32_t chunk_cap;
};

// The subtree passes work in the unused end of the sums array, le slots of which are taken: an
// 80 B record per node to come and two sets of sums of deep_sum_slot(n, roots) nodes (288 B
// each, 192 B a point) or fewer.  The slots left have 144 B a node, so 64 B a point and what the
// roots and the nodes above them take has to be added; 72 B a point do for roots of 52 points or
// more on average (the pass asks the pool where they don't).  A block of the pool beside this
// workspace, one ring of 396 KB per 16-warp group, was up to 59 MB that no reservation counted.
// Words of 16 B.
size_t deep_spare(int64_t n, int R) { return (72 * (size_t)n + 96 * (size_t)R) / 16; }

// Lays the workspace for n points in R clouds out from p (a null base: sizes only); returns its end.
char* ws_layout(BuildWs& w, char* p, int64_t n, int R) {
  w.cap_nodes = 2 * n + 4096 + 4 * (int64_t)R;
  w.chunk_cap = (int32_t)(n / kChunk + n / kBig + 16);
  const int64_t cn = w.cap_nodes;
  const int64_t G = (int64_t)(kMaxDepth + 2) * R;
  const size_t nbig = (size_t)kSums * (n / kBig + 2);
  w.B.p[0] = carve<float4>(p, 2 * n + 2);  // later the n + 1 stamp prefixes of 32 B
  w.B.p[1] = w.B.p[0] + n;
  w.B.perm = carve<int32_t>(p, n);
  w.nodes = carve<BNode>(p, cn);
  w.alive = carve<int32_t>(p, cn);
  w.flags = carve<int2>(p, cn);
  w.flag_tiles = carve<int2>(p, cn / kFlagTile + 2);
  w.chunks = carve<Chunk>(p, w.chunk_cap);
  w.seg = carve<SegCounts>(p, w.chunk_cap);
  w.big_list = carve<int32_t>(p, w.chunk_cap);
  w.node_chunk0 = carve<int32_t>(p, w.chunk_cap);
  w.acc = carve<U128>(p, nbig);
  for (int k = 0; k < 2; ++k) w.accl.acc[k] = carve<U128>(p, nbig);
  w.mom = carve<U128>(p, (size_t)kSums * cn + deep_spare(n, R));
  w.mom_end = w.mom + (size_t)kSums * cn + deep_spare(n, R);
  w.dt = carve<double>(p, n);
  w.dt_tiles = carve<DtSum>(p, n / kDtTile + 1);
  w.off = carve<int64_t>(p, R + 1);
  w.ls = carve<LevelState>(p, 1);
  w.done = carve<unsigned>(p, 1);
  w.cnt = carve<int32_t>(p, G);
  w.lcnt = carve<int32_t>(p, G);
  w.tsmin = carve<unsigned long long>(p, R);
  w.tot_nodes = carve<int32_t>(p, (size_t)3 * R + 1);
  w.tot_leaves = w.tot_nodes + R;
  w.ucnt = w.tot_leaves + R;
  w.ts0 = carve<double>(p, (size_t)(1 + kRootFrame) * R);
  w.root_frame = w.ts0 + R;
  w.zero_end = p;
  w.bsum = carve<int32_t>(p, kLevelBlocks);
  w.bbig = carve<int32_t>(p, 2 * kLevelBlocks);
  w.gp = carve<int32_t>(p, G);
  w.lgp = carve<int32_t>(p, G);
  w.to = carve<int32_t>(p, G);
  w.lto = carve<int32_t>(p, G);
  w.trees = carve<TreeDev>(p, R);
  return p;
}

// Bytes of the build workspace for n points in R clouds.
size_t ws_bytes(int64_t n, int R) {
  BuildWs w;
  return (size_t)(ws_layout(w, nullptr, n, R) - (char*)nullptr) + 256;
}

int ws_alloc(BuildWs& w, int64_t n, int R, cudaStream_t s) {
  const size_t bytes = ws_bytes(n, R);
  cudaError_t e = cudaMallocAsync(&w.block, bytes, s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    w.block = nullptr;
    set_error("cudaMallocAsync of %zu bytes for the tree build workspace failed: %s", bytes, cudaGetErrorString(e));
    return KDS_ERR_OOM;
  }
  ws_layout(w, (char*)w.block, n, R);
  return KDS_OK;
}

}  // namespace

namespace {

// The deep levels of a build whose current level (h, read at the last sync) fits the form:
// k_deep_build, the depth-major scan of the per-(depth, subtree) node counts, k_deep_place and
// k_deep_finish.  n: the build's points.
template <int WARPS>
int deep_pass(BuildWs& w, int64_t n, const BuildParams& P, const LevelState& h, cudaStream_t s) {
  using Form = DeepForm<WARPS>;
  const int lb = h.lb, le = h.le;
  const int nroots = le - lb;
  if (nroots <= 0) return KDS_OK;
  const int dcap = std::max(1, P.max_level - h.depth);
  const int grid = (int)std::min<int64_t>((nroots + Form::kGroups - 1) / Form::kGroups, 148 * Form::kPerSM);
  const int64_t ncount = (int64_t)dcap * nroots;
  if (ncount > INT32_MAX / 2) { set_error("kds_tree_build: too many deep subtrees"); return KDS_ERR_CAPACITY; }
  // Records and sums behind the sums in use, counts and offsets in the prune's flags, both free
  // until the pass is done; a block of the pool in place of what they have no room for.
  const int64_t dn_cap = w.cap_nodes - le;
  const int32_t own_slots = deep_sum_slot(n, nroots), all_groups = grid * Form::kGroups * deep_nodes<WARPS>();
  const int32_t sum_slots = std::min(own_slots, all_groups);
  const int32_t group_slots = all_groups < own_slots ? deep_nodes<WARPS>() : 0;
  DeepNode* dn = reinterpret_cast<DeepNode*>(w.mom + (size_t)le * kSums);
  U128* sums = reinterpret_cast<U128*>(dn + dn_cap);
  const size_t sum_words = (size_t)2 * kSums * sum_slots;
  const bool sums_fit = sums + sum_words <= w.mom_end;
  const size_t bc = carve_size<int32_t>(ncount + 64), bt = carve_size<int32_t>(ncount / 4096 + 2),
               bk = 2 * bc + bt + 256, br = carve_size<U128>(sum_words);
  const bool counts_fit = bk <= sizeof(int2) * (size_t)w.cap_nodes;
  void* blk = nullptr;
  cudaError_t e = cudaSuccess;
  if (!sums_fit || !counts_fit) e = cudaMallocAsync(&blk, (sums_fit ? 0 : br) + (counts_fit ? 0 : bk), s);
  if (e != cudaSuccess) {
    cudaGetLastError();
    set_error("cudaMallocAsync for the deep tree levels failed: %s", cudaGetErrorString(e));
    return KDS_ERR_OOM;
  }
  char* p = (char*)blk;
  if (!sums_fit) sums = carve<U128>(p, sum_words);
  if (counts_fit) p = (char*)w.flags;
  int32_t* counts = carve<int32_t>(p, ncount + 64);  // and dn_count behind them: cleared together
  int32_t* dn_count = counts + ncount;
  int32_t* off = carve<int32_t>(p, ncount + 64);
  int32_t* tiles = carve<int32_t>(p, ncount / 4096 + 2);
  int32_t* total = carve<int32_t>(p, 1);
  int rc = KDS_OK;
  const size_t smem = sizeof(DeepSmem<WARPS>) * Form::kGroups;
  static DeviceSet limits;  // devices with the kernel's limit raised
  int dev = 0;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess && !limits.has(dev)) {
    e = cudaFuncSetAttribute((const void*)k_deep_build<WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) limits.add(dev);
  }
  if (e == cudaSuccess) e = cudaMemsetAsync(counts, 0, sizeof(int32_t) * (ncount + 1), s);
  if (e == cudaSuccess) {
    launch(k_deep_build<WARPS>, grid, 32 * WARPS * Form::kGroups, smem, s, w.nodes, w.ls, w.B, w.mom, w.accl, P, w.root_frame,
                                                                       dn, (int32_t)dn_cap, dn_count, sums, sum_slots, group_slots, counts, dcap);
    if (ncount <= kDeepScan) {
      launch(k_deep_scan, 1, 1024, 0, s, w.ls, lb, le, counts, (int32_t)ncount, off, dcap, (int32_t)w.cap_nodes);
    } else {
      rc = scan_exclusive(counts, off, (int32_t)ncount, tiles, total, s);
      launch(k_deep_finish, 1, 64, 0, s, w.ls, lb, le, off, total, dcap, (int32_t)w.cap_nodes);
    }
    const int pg = (int)std::min<int64_t>(nblk(std::max<int64_t>(w.cap_nodes - le, nroots), kThreads), kGridBlocks * 4);
    launch(k_deep_place, pg, kThreads, 0, s, w.nodes, w.ls, lb, le, dn, dn_count, (int32_t)dn_cap, off, dcap,
           (int32_t)w.cap_nodes, w.alive);
    e = cudaGetLastError();
  }
  if (blk) cudaFreeAsync(blk, s);
  if (e != cudaSuccess) return cuda_status(e, "deep tree levels", __FILE__, __LINE__);
  return rc;
}

}  // namespace

namespace {

// What a finished or abandoned level reports.
int build_error(const LevelState& h) {
  if (h.error == 2) { set_error("kds_tree_build: coordinate >= 32768 m, non-finite stamp or dt >= 65536 s"); return KDS_ERR_RANGE; }
  if (h.error == 1) { set_error("kds_tree_build: node capacity exceeded"); return KDS_ERR_CAPACITY; }
  return KDS_OK;
}

// Blocks that write the chunks of one node range: a thread each for a few thousand chunks (one
// block takes 25 us for 11,000), none but the level's own below.
int chunk_parts(int64_t N) { return (int)std::max<int64_t>(1, std::min<int64_t>(64, N / (1 << 20))); }

int level_blocks(int64_t nodes) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(kLevelBlocks, (nodes + kThreads - 1) / kThreads));
}

// Blocks that take a contiguous range of chunks each: one resident wave, so that no block
// starts when the others are done.
int scatter_blocks(const BuildWs& w) { return std::min<int>(w.chunk_cap, 148 * kScatterPerSM); }

// Level 0: the roots' sums, from their points.
int root_sums(BuildWs& w, int R, int32_t max_size, int64_t N, cudaStream_t s) {
  launch(k_root_moments, (int)std::min<int64_t>(kGridBlocks, (R + 7) / 8), kThreads, 0, s, w.nodes, R, w.B, w.mom);
  if (max_size > kBig) {
    const int nb = level_blocks(R), parts = nb == 1 ? chunk_parts(N) : 1;
    launch(k_big_sums, nb, kThreads, 0, s, w.nodes, w.ls, w.bbig);
    launch(k_big_plan, nb * parts, kThreads, 0, s, w.nodes, w.ls, w.bbig, w.chunks, w.chunk_cap, w.big_list, w.node_chunk0,
                                               w.acc, w.accl, parts);
    launch(k_big_moments, scatter_blocks(w), kThreads, 0, s, w.chunks, w.ls, w.B, w.acc);
    launch(k_big_to_mom, 64, 256, 0, s, w.ls, w.big_list, w.acc, w.mom);
  }
  KDS_CK(cudaGetLastError());
  return KDS_OK;
}

}  // namespace

size_t forest_workspace_bytes(int64_t n, int R) { return ws_bytes(std::max<int64_t>(n, 1), std::max(R, 1)); }

// Builds R trees from R clouds stored back to back (offsets[R+1] on the host).
// out[r] = NULL and status[r] = KDS_ERR_TREE_REJECTED where makeTree returns nullptr.
// Page-locked staging for the build's small device-to-host reads (the level state at each
// host check, the per-tree counts at the end) instead of pageable host memory: one block
// per host thread, grown on demand, released when the thread exits.
struct PinnedStage {
  void* p = nullptr;
  size_t cap = 0;
  ~PinnedStage() {
    if (p) cudaFreeHost(p);
  }
  void* get(size_t bytes) {
    if (bytes > cap) {
      if (p) cudaFreeHost(p);
      p = nullptr;
      cap = 0;
      const size_t c = std::max<size_t>(bytes, 64 * 1024);
      if (cudaMallocHost(&p, c) != cudaSuccess) {
        cudaGetLastError();
        p = nullptr;
        return nullptr;
      }
      cap = c;
    }
    return p;
  }
};

void* pinned_stage(size_t bytes) {
  thread_local PinnedStage st;
  return st.get(bytes);
}

int tree_build_forest(const float* xyz, const double* stamps, const int64_t* offsets, int32_t R, int32_t mem,
                      const kds_tree_params* prm, cudaStream_t s, kds_tree** out, int32_t* status) {
  for (int r = 0; r < R; ++r) { out[r] = nullptr; status[r] = KDS_ERR_TREE_REJECTED; }
  if (R <= 0) { set_error("kds_tree_build: no clouds"); return KDS_ERR_INVALID_ARG; }
  const int64_t N = offsets[R] - offsets[0];
  if (offsets[0] != 0 || N < 0 || N > ((int64_t)1 << 30)) {
    set_error("kds_tree_build: bad point count / offsets");
    return KDS_ERR_INVALID_ARG;
  }
  std::vector<int64_t> off(offsets, offsets + R + 1);
  int32_t max_size = 0;
  for (int r = 0; r < R; ++r) {
    if (off[r + 1] < off[r]) { set_error("kds_tree_build: offsets must be non-decreasing"); return KDS_ERR_INVALID_ARG; }
    max_size = std::max<int32_t>(max_size, (int32_t)(off[r + 1] - off[r]));
  }
  BuildParams P;
  P.propagate_normal = prm->propagate_normal;
  P.leaf_min_points = prm->leaf_min_points;
  P.leaf_max_points = prm->leaf_max_points;
  P.leaf_density = prm->leaf_density;
  P.leaf_min_normal_incidence = prm->leaf_min_normal_incidence;
  P.leaf_normal_eigenratio = prm->leaf_normal_eigenratio;
  P.prune_incidence = prm->prune_min_normal_incidence;
  P.max_level = prm->max_level > 0 ? std::min(prm->max_level, kMaxDepth) : 48;
  if (N == 0) return KDS_OK;  // every cloud rejected (fewer points than leaf_min_points)

  BuildWs w;
  int rc = ws_alloc(w, std::max<int64_t>(N, 1), R, s);
  if (rc) return rc;
  struct Guard {
    BuildWs* w;
    cudaStream_t s;
    void* h_xyz = nullptr;
    void* h_st = nullptr;
    ~Guard() {
      if (w->block) cudaFreeAsync(w->block, s);
      if (h_xyz) cudaFreeAsync(h_xyz, s);
      if (h_st) cudaFreeAsync(h_st, s);
    }
  } guard{&w, s};
  const float* d_xyz = xyz;
  const double* d_st = stamps;
  if (mem == KDS_MEM_HOST) {
    KDS_CK(cudaMallocAsync(&guard.h_xyz, sizeof(float) * 3 * N, s));
    KDS_CK(cudaMemcpyAsync(guard.h_xyz, xyz, sizeof(float) * 3 * N, cudaMemcpyHostToDevice, s));
    d_xyz = (const float*)guard.h_xyz;
    if (stamps) {
      KDS_CK(cudaMallocAsync(&guard.h_st, sizeof(double) * N, s));
      KDS_CK(cudaMemcpyAsync(guard.h_st, stamps, sizeof(double) * N, cudaMemcpyHostToDevice, s));
      d_st = (const double*)guard.h_st;
    }
  }
  KDS_CK(cudaMemsetAsync(w.ls, 0, (size_t)(w.zero_end - (char*)w.ls), s));
  KDS_CK(cudaMemcpyAsync(w.off, off.data(), sizeof(int64_t) * (R + 1), cudaMemcpyHostToDevice, s));
  launch(k_ingest, nblk(N, kThreads), kThreads, 0, s, d_xyz, N, w.B.p[0], w.ls);
  if (d_st) {
    // enough blocks to fill the machine whatever the number of clouds (64 per cloud before:
    // 370 + 200 us over the 11.4M stamps of one map)
    const int64_t gx = std::max<int64_t>(64, (148 * 8 + R - 1) / R);
    dim3 g((unsigned)std::min<int64_t>(std::max<int64_t>((max_size + kThreads - 1) / kThreads, 1), gx), (unsigned)R);
    launch(k_tree_min, g, kThreads, 0, s, d_st, w.off, w.tsmin);
    launch(k_tree_check, g, kThreads, 0, s, d_st, w.off, w.tsmin, w.ts0, w.dt, w.ls);
  }
  launch(k_init_roots, (R + 127) / 128, 128, 0, s, w.nodes, w.off, R, w.ls);
  KDS_CK(cudaGetLastError());

  // pinned: [level state | per-tree nodes, leaves, unpruned nodes | ts0 | root frames]
  const size_t st_ls = (sizeof(LevelState) + 255) & ~(size_t)255;
  const size_t st_cnt = (size_t)((char*)w.ts0 - (char*)w.tot_nodes);
  char* stage = (char*)pinned_stage(st_ls + st_cnt + sizeof(double) * (size_t)(1 + kRootFrame) * R);
  if (!stage) { set_error("kds_tree_build: page-locked staging of the level state failed"); return KDS_ERR_OOM; }
  LevelState& hls = *reinterpret_cast<LevelState*>(stage);
  int32_t* h_cnt = reinterpret_cast<int32_t*>(stage + st_ls);
  double* h_dbl = reinterpret_cast<double*>(stage + st_ls + st_cnt);
  int32_t host_max = max_size;
  const int cb = std::min<int>(w.chunk_cap, kGridBlocks * 2);
  const int sb = scatter_blocks(w);
  // Grids of the level kernels sized to the level: a level has at most twice the nodes
  // of the one before, and the host learns the current level's size at each sync.  The
  // node-range kernels (k_decide, k_level_children, k_big_plan) share
  // one block count per level; every kernel's result is independent of its grid.
  int64_t level_nodes = R;
  int32_t global_levels = -1;  // levels built level by level; -1: no shared-memory pass
  hls.lb = 0;
  hls.le = R;
  hls.depth = 0;
  for (int round = 0; round < kMaxDepth; ++round) {
    const bool by_block = host_max <= kBlockMax && level_nodes <= kBlockRoots;
    if (by_block || (host_max <= kDeepMax && level_nodes <= kDeepMaxRoots)) {
      // every node of the current level fits one group's shared memory: the rest of every
      // subtree is built there; the host reads the final level state with the counts below
      if (round == 0) {  // the roots' sums (roots of 1,025 to 2,048 points by their chunks)
        rc = root_sums(w, R, host_max, N, s);
        if (rc) return rc;
      }
      global_levels = hls.depth;
      rc = by_block ? deep_pass<16>(w, N, P, hls, s) : deep_pass<1>(w, N, P, hls, s);
      if (rc) return rc;
      break;
    }
    // as many levels to the next look at the level state as halvings still separate the
    // largest node from a subtree pass that the level is small enough for (nodes at most
    // double per level), one at a time once it is near
    int nlev = kLevelsPerSync;
    for (int k = 1; k <= kLevelsPerSync; ++k) {
      const bool block_near = (host_max >> k) <= kBlockMax && (level_nodes << k) <= kBlockRoots;
      const bool warp_near = (host_max >> k) <= 2 * kDeepMax && (level_nodes << (k + 1)) <= kDeepMaxRoots;
      if (block_near || warp_near) {
        nlev = k;
        break;
      }
    }
    for (int k = 0; k < nlev; ++k) {
      const bool level0 = round == 0 && k == 0;
      const int64_t nodes_bound = level_nodes << k;
      const int lvl_blocks = level_blocks(nodes_bound);
      const int small_blocks =
          (int)std::max<int64_t>(1, std::min<int64_t>(kSmallBlocks, (nodes_bound + kThreads / 32 - 1) / (kThreads / 32)));
      const int plan_parts = lvl_blocks == 1 ? chunk_parts(N) : 1;
      if (level0) {
        rc = root_sums(w, R, host_max, N, s);
        if (rc) return rc;
      }
      const bool big = host_max > kBig;  // the large-node kernels run after the partition
      if (lvl_blocks == 1) {
        launch(k_level_small, 1, kThreads, 0, s, w.nodes, w.ls, w.mom, w.accl, P, w.bsum, w.bbig, w.root_frame,
                                             (int32_t)w.cap_nodes, w.chunks, w.chunk_cap, w.big_list, w.node_chunk0,
                                             plan_parts == 1 ? 1 : 0);
      } else {
        launch(k_decide, lvl_blocks, kThreads, 0, s, w.nodes, w.ls, w.mom, w.accl, P, w.bsum, w.bbig, w.root_frame);
        launch(k_level_children, lvl_blocks, kThreads, 0, s, w.nodes, w.ls, w.bsum, (int32_t)w.cap_nodes, big ? 1 : 0,
               w.bbig, w.chunks, w.chunk_cap, w.big_list, w.node_chunk0, w.accl);
      }
      if (big && plan_parts > 1) {  // the decisions counted the large nodes per block
        launch(k_big_plan, plan_parts, kThreads, 0, s, w.nodes, w.ls, w.bbig, w.chunks, w.chunk_cap, w.big_list,
               w.node_chunk0, nullptr, w.accl, plan_parts);
      }
      const int count_blocks = big ? cb : 0;
      launch(k_small_part, count_blocks + small_blocks, kThreads, 0, s, w.nodes, w.ls, w.B, w.mom, w.bsum, lvl_blocks,
             (int32_t)w.cap_nodes, big ? nullptr : w.done, w.chunks, w.seg, count_blocks);
      if (big) {
        launch(k_big_scatter, sb, kThreads, 0, s, w.chunks, w.ls, w.nodes, w.B, w.seg, w.node_chunk0, w.accl, w.bsum,
                                              lvl_blocks, (int32_t)w.cap_nodes, w.done);
      }
    }
    KDS_CK(cudaGetLastError());
    KDS_CK(cudaMemcpyAsync(&hls, w.ls, sizeof(LevelState), cudaMemcpyDeviceToHost, s));
    KDS_CK(cudaStreamSynchronize(s));
    if ((rc = build_error(hls))) return rc;
    if (hls.lb >= hls.le) break;
    host_max = hls.max_size;
    level_nodes = hls.le - hls.lb;
  }
  const bool deep = global_levels >= 0;
  if (!deep && hls.lb < hls.le) { set_error("kds_tree_build: depth limit"); return KDS_ERR_CAPACITY; }
  // most nodes there can be: the launches below take their number from the level state
  const int64_t bound = deep ? w.cap_nodes : hls.le;
  const int node_blocks = (int)std::min<int64_t>(nblk(bound, kThreads), kGridBlocks * 4);
  // prune
  if (!deep) KDS_CK(cudaMemsetAsync(w.alive, 0, sizeof(int32_t) * bound, s));
  launch(k_alive, node_blocks, kThreads, 0, s, w.nodes, w.ls, w.alive, P.prune_incidence);
  launch(k_group_counts, node_blocks, kThreads, 0, s, w.nodes, w.ls, w.alive, R, w.cnt, w.lcnt, w.ucnt, w.flags);
  if (bound <= kFlagOne) {
    launch(k_flag_scan, 1, 1024, 0, s, w.flags, w.ls, nullptr);
  } else {
    const int nt = (int)((bound + kFlagTile - 1) / kFlagTile);
    launch(k_flag_tiles, nt, 1024, 0, s, w.flags, w.ls, w.flag_tiles);
    launch(k_flag_top, 1, 1024, 0, s, w.flag_tiles, nt);
    launch(k_flag_scan, nt, 1024, 0, s, w.flags, w.ls, w.flag_tiles);
  }
  launch(k_group_tables, 1, 1024, 0, s, w.ls, R, w.cnt, w.lcnt, w.gp, w.lgp, w.to, w.lto, w.tot_nodes, w.tot_leaves);
  if (deep) KDS_CK(cudaMemcpyAsync(&hls, w.ls, sizeof(LevelState), cudaMemcpyDeviceToHost, s));
  KDS_CK(cudaMemcpyAsync(h_cnt, w.tot_nodes,
                         (size_t)((char*)(w.ts0 + (size_t)(1 + kRootFrame) * R) - (char*)w.tot_nodes),
                         cudaMemcpyDeviceToHost, s));
  KDS_CK(cudaStreamSynchronize(s));
  if (deep && (rc = build_error(hls))) return rc;
  const int depth = hls.depth;
  const int32_t total = hls.le;
  const std::vector<int32_t> tn(h_cnt, h_cnt + R), tl(h_cnt + R, h_cnt + 2 * R), tu(h_cnt + 2 * R, h_cnt + 3 * R);
  const std::vector<double> ts0(h_dbl, h_dbl + R), rf(h_dbl + R, h_dbl + R + (size_t)kRootFrame * R);
  std::vector<TreeDev> td(R);
  std::vector<kds_tree*> made(R, nullptr);
  for (int r = 0; r < R; ++r) {
    int64_t np = off[r + 1] - off[r];
    if (np < prm->leaf_min_points || np == 0 || tl[r] < prm->tree_min_good_leaves) continue;
    kds_tree* t = new kds_tree();
    rc = tree_alloc(t->d, tn[r], tl[r], np, s);
    if (rc) {
      delete t;
      for (int q = 0; q < r; ++q)
        if (made[q]) { tree_release(made[q]->d); delete made[q]; }
      return rc;
    }
    t->d.num_unpruned = tu[r];
    t->d.ts_start = ts0[r];
    t->d.depth = depth;
    t->d.global_levels = global_levels >= 0 ? global_levels : depth;
    const double* f = &rf[(size_t)kRootFrame * r];
    for (int i = 0; i < 3; ++i) {
      t->root_eigenvalues[i] = (float)f[i];
      t->root_mean[i] = (float)f[12 + i];
    }
    for (int i = 0; i < 9; ++i) t->root_eigenvectors[i] = (float)f[3 + i];
    made[r] = t;
    td[r] = t->d;
  }
  KDS_CK(cudaMemcpyAsync(w.trees, td.data(), sizeof(TreeDev) * R, cudaMemcpyHostToDevice, s));
  DtSum* pre = nullptr;
  if (d_st) {  // the point buffers are free now
    pre = reinterpret_cast<DtSum*>(w.B.p[0]);
    const int nt = (int)(N / kDtTile + 1);  // tiles of the N + 1 positions
    if (nt > 1) {
      launch(k_dt_tiles, nt, kThreads, 0, s, w.dt, w.B.perm, N, w.dt_tiles);
    }
    if (nt > kThreads) {
      launch(k_dt_top, 1, kThreads, 0, s, w.dt_tiles, nt);
    }
    launch(k_dt_prefix, nt, kThreads, 0, s, w.dt, w.B.perm, N, w.dt_tiles, nt > kThreads ? 1 : 0, pre);
  }
  launch(k_compact_forest, nblk(total, kThreads), kThreads, 0, s, w.nodes, total, w.alive, w.flags, R, w.gp, w.lgp, w.to,
                                                              w.lto, pre, w.off, w.trees);
  dim3 fg((unsigned)std::min<int64_t>(nblk(max_size, kThreads), std::max<int64_t>(64, 148 * 16 / R)), (unsigned)R);
  launch(k_finish_trees, fg, kThreads, 0, s, w.trees, w.off, w.B.perm);
  cudaError_t e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    for (auto* t : made)
      if (t) { tree_release(t->d); delete t; }
    return cuda_status(e, "tree build", __FILE__, __LINE__);
  }
  for (int r = 0; r < R; ++r) {
    out[r] = made[r];
    status[r] = made[r] ? KDS_OK : KDS_ERR_TREE_REJECTED;
  }
  return KDS_OK;
}

int tree_build(const float* xyz, const double* stamps, int64_t n, int32_t mem, const kds_tree_params* prm,
               cudaStream_t s, kds_tree** out) {
  *out = nullptr;
  if (n < 0 || n > ((int64_t)1 << 30)) {
    set_error("kds_tree_build: bad point count %lld", (long long)n);
    return KDS_ERR_INVALID_ARG;
  }
  if (n < prm->leaf_min_points || n == 0) {
    set_error("kds_tree_build: %lld points < leaf_min_points", (long long)n);
    return KDS_ERR_TREE_REJECTED;
  }
  int64_t off[2] = {0, n};
  int32_t st = 0;
  int rc = tree_build_forest(xyz, stamps, off, 1, mem, prm, s, out, &st);
  if (rc) return rc;
  if (st != KDS_OK) {
    set_error("kds_tree_build: too few good leaves (tree_min_good_leaves %d)", prm->tree_min_good_leaves);
    return KDS_ERR_TREE_REJECTED;
  }
  return KDS_OK;
}

}  // namespace kds
