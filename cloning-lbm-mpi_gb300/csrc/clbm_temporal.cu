// clbm_temporal.cu -- FP32 interval kernel with every clone resident on chip.
//
// One thread-block cluster per clone: the clone's H rows are split into CS
// bands of consecutive rows, given by the launch (an even split, or one
// balanced for the extra cost of the square's rows and the walls), each band
// in one CTA's shared memory.  The T steps of the interval run without
// touching HBM except for the drag terms: P_0 is loaded once, S_T stored once.
//
// In-place update ("AA" pattern): one buffer A holds, alternately,
//   after a local step:  A[n][opp k] = P(n,k)        (post-collision, own node)
//   after a gather step: A[m][k]     = S_next(m,k)   (streamed, natural order)
// Step t with t even is a gather step: S(n,k) = A[n - c_k][opp k], or on a
// bounced slot A[n][k] (= P(n, opp k)); the collided P(n,k) is pushed to
// A[n + c_k][k], or to A[n][opp k] when slot (n, opp k) bounces back.  Step
// t odd is a local step: S(n,k) = A[n][k], P(n,k) -> A[n][opp k].  In both,
// the nine slots a node reads are exactly the nine it writes and no other
// node touches them, so a step needs no barrier inside.  These are the pull
// rules of clbm_step.cu (the reference's collide / push-stream / bounce-back /
// reset / swap sequence, src/mpi_LBM_GK_pops_perturb.cpp:426-443), so results
// are bit-identical to the streaming kernel.  Neighbours across a band edge
// are read and written in the adjacent CTA's shared memory.
//
// A thread takes a pair of nodes, x and x + ceil(W/2) of one row, one in each
// lane of the packed FP32 arithmetic: every neighbour offset is the same for
// both, so a pair's nine slots are nine 64-bit words and the whole collision
// is packed.  Only the pairs at the two ends of a row (the seam: the periodic
// wrap, and between the halves) have their lanes' neighbours in different
// pairs; they are few and take per-lane addresses.  An odd width leaves the
// last pair's lane 1 empty (a column of its own that no node reads).
//
// What bounds it: per 32 pairs 77 packed operations, 2 cycles each on the
// FMA pipe of a scheduler (154), and 36 cycles of the SM's shared memory for
// four schedulers' 18 accesses each (144).  On the 256x64 channel (bands
// 23/18/23, 512 threads) a segment takes about 210 (local step) to 260 cycles;
// 4096 clones run at 0.289 ms per step, where one node per thread with the
// four direction pairs packed took 0.367; 1024 clones of 400x100 (9 bands) at
// 0.196 against 0.353.  What made the difference besides the packing (ms per
// step of the 256x64 case): each warp's share of the deal kept in registers
// instead of worked out in every step (0.344 -> 0.317), whole planes per
// population instead of node records, so that what crosses a band edge goes as
// whole sectors (0.317 -> 0.306; 400x100: 0.265 -> 0.225), planes a constant
// distance apart, so that a pair's slots are constant offsets (0.306 -> 0.297),
// row ends inside the band through plain shared memory and a perimeter update
// of its own (0.298 -> 0.289),
// and the split cluster barrier with the edge rows first (400x100: 0.33 ->
// 0.28).  Random-field steps read two values per pair from L2: loaded one
// segment ahead, 0.343 -> 0.329 ms per step over an interval with 20 of 100
// such steps.
#include <cooperative_groups.h>

#include <algorithm>

#include "clbm_internal.h"
#include "clbm_physics.cuh"
#include "clbm_reseed.cuh"

namespace cg = cooperative_groups;

namespace clbm {

// Distributed shared memory through 32-bit shared::cluster addresses: the
// address of this CTA's shared-memory offset `a` in the CTA of cluster rank
// `rank`, and loads / stores of one float or one pair at such addresses.
__device__ __forceinline__ unsigned cluster_addr(unsigned a, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_cluster(unsigned a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(unsigned a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ f2_t ld_cluster2(unsigned a) {
  f2_t v;
  asm volatile("ld.shared::cluster.b64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster2(unsigned a, f2_t v) {
  asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}

// Geometry of one CTA's band.  NP: the pairs a plane of A has room for, a
// constant, so that the nine slots of a pair lie at constant offsets.
template <int NP>
struct BandT {
  static constexpr int ps = 2 * NP;  // floats per plane
  int cs, rank, clone, W, H, rows, row0;
  int Wh, np;      // pairs per row, pairs of the band
  int rowf;        // floats per row of a plane (2 Wh)
  unsigned div_wh; // ceil(2^32 / Wh)
  int rows_prev;   // rows of the previous band (its last row lies above this band's row 0)
  float *prev, *next;
  unsigned own_c, prev_c, next_c;  // shared::cluster byte addresses of A in this / previous / next CTA
  long long plane;
  const float *src;
  float *dst;
};

// Float offset, within a row of A, of column x's population 0 (population k
// at + k ps): pair x or x - Wh, its lane 0 or 1.
template <class Band>
__device__ __forceinline__ int col_off(const Band &b, int x) { return x < b.Wh ? 2 * x : 2 * (x - b.Wh) + 1; }

// A row of A: in this CTA, or anywhere in the cluster.
struct RowL {
  float *p;
  __device__ __forceinline__ float ld(int o) const { return p[o]; }
  __device__ __forceinline__ void st(int o, float v) const { p[o] = v; }
  __device__ __forceinline__ f2_t ld2(int o) const { return *(const f2_t *)(p + o); }
  __device__ __forceinline__ void st2(int o, f2_t v) const { *(f2_t *)(p + o) = v; }
};
struct RowC {
  unsigned a;
  __device__ __forceinline__ float ld(int o) const { return ld_cluster(a + 4u * o); }
  __device__ __forceinline__ void st(int o, float v) const { st_cluster(a + 4u * o, v); }
  __device__ __forceinline__ f2_t ld2(int o) const { return ld_cluster2(a + 4u * o); }
  __device__ __forceinline__ void st2(int o, f2_t v) const { st_cluster2(a + 4u * o, v); }
};

// ... by a generic pointer, for rows that are in this CTA for some lanes and in
// a neighbour for others (a shared::cluster address of this CTA would go over
// the network between SMs too).
struct RowG {
  float *p;
  __device__ __forceinline__ float ld(int o) const { return p[o]; }
  __device__ __forceinline__ void st(int o, float v) const { p[o] = v; }
  __device__ __forceinline__ f2_t ld2(int o) const { return *(const f2_t *)(p + o); }
  __device__ __forceinline__ void st2(int o, f2_t v) const { *(f2_t *)(p + o) = v; }
};

// Columns of a pair: float offsets of the pair itself (lane 0; lane 1 is one
// further) and of its left (m) and right (p) neighbours, per lane.
struct Cols {
  int o, m0, m1, p0, p1;
};
__device__ __forceinline__ Cols cols_inner(int xh) {
  return Cols{2 * xh, 2 * xh - 2, 2 * xh - 1, 2 * xh + 2, 2 * xh + 3};
}
// any pair: the periodic wrap, and with an odd width lane 1 of the last pair,
// which holds no node: it gets itself for both neighbours (a column of its
// own, periodic over one node, that no node ever reads)
template <class Band>
__device__ __forceinline__ Cols cols_any(const Band &b, int xh) {
  const int x1 = xh + b.Wh;
  Cols c;
  c.o = 2 * xh;
  c.m0 = col_off(b, xh == 0 ? b.W - 1 : xh - 1);
  c.p0 = col_off(b, xh + 1 == b.W ? 0 : xh + 1);
  c.m1 = x1 < b.W ? col_off(b, x1 - 1) : c.o + 1;
  c.p1 = x1 < b.W ? col_off(b, x1 + 1 == b.W ? 0 : x1 + 1) : c.o + 1;
  return c;
}

// The seam: the pairs of a row whose lanes' neighbour columns do not both lie
// at a constant offset -- the first and the last, and with an odd width the
// one before the last (its lane 1 is the last node).  seam_count pairs per
// row; the j-th of them.
template <class Band>
__device__ __forceinline__ bool on_seam(const Band &b, int xh) {
  return xh == 0 || xh >= b.Wh - 1 - (b.W & 1);
}
template <class Band>
__device__ __forceinline__ int seam_count(const Band &b) { return (b.W & 1) && b.Wh > 2 ? 3 : 2; }
template <class Band>
__device__ __forceinline__ int seam_pair(const Band &b, int j) { return j == 0 ? 0 : b.Wh - j; }

// Index p within a row as the segments take its pairs: the pair Wh - 1 first,
// then 0, 1, ..., so that the seam at the two ends falls into one segment.
template <class Band>
__device__ __forceinline__ int pair_of(const Band &b, int p) { return p == 0 ? b.Wh - 1 : p - 1; }

// The random field's values at a pair's nodes (where lane 1 holds no node,
// lane 0's).
template <class Band>
__device__ __forceinline__ f2_t pair_map(const Band &b, const float *map, int y, int xh) {
  const float *m = map + (long long)y * b.W + xh;
  return f2_bits(m[0], m[xh + b.Wh < b.W ? b.Wh : 0]);
}

// The two nodes' force: the run's, or under a random field (while its steps
// last) from its values m at the nodes -- field_beta_f32 and f32_force of both
// nodes in packed arithmetic.
template <bool FIELD>
__device__ __forceinline__ F32Force2 pair_force(const RunDev &R, f2_t m) {
  if (!FIELD) return R.f_force2;
  namespace X = f32x2op;
  const F32FieldOps &o = R.f_field_ops;
  const f2_t beta = X::mul(o.beta, X::fma(o.eps, m, R.f_pairs.one));
  const f2_t fb = X::mul(o.cforce, beta);
  F32Force2 f;
  f.hb = X::mul(o.half, beta);
  f.nfbm3 = X::mul(o.three, fb);
  f.fb9 = X::mul(o.nine, fb);
  f.nfb9 = X::mul(o.mnine, fb);
  f.f2 = X::mul(o.twelfth, fb);
  f.nf2 = X::mul(o.mtwelfth, fb);
  f.nf13 = X::mul(o.mthird, fb);
  return f;
}
template <bool FIELD, class Band>
__device__ __forceinline__ F32Force2 pair_force(const RunDev &R, const Band &b, const float *map, int y, int xh) {
  return pair_force<FIELD>(R, FIELD ? pair_map(b, map, y, xh) : 0ull);
}

// Where a pair's post-collision populations go besides A (checkpoints of the
// adjoint's forward): node (x, y) of plane 0, nullptr for nowhere; lane 1's
// node lies half columns further, if there is one.
struct Keep {
  float *p;
  int half;
};
template <bool STORE>
__device__ __forceinline__ void keep_pair(const RunDev &R, const Keep &kp, const f2_t P[9], bool skip0, bool skip1) {
  if (!STORE || !kp.p) return;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    if (!skip0) kp.p[k * R.plane] = f32x2op::lo(P[k]);
    if (!skip1 && kp.half) kp.p[k * R.plane + kp.half] = f32x2op::hi(P[k]);
  }
}

// One pair of nodes in a gather step.  C, U, D: the pair's row and the rows
// y - 1 and y + 1.  S(n,k) is read from A[n - c_k][opp k] and P(n, opp k)
// goes back to that slot (the pull rules make the two the same).  WALL: 1 =
// the bottom wall y = 0, whose slots 2, 5, 6 are the node's own; 2 = the top
// wall, slots 4, 7, 8 (the row beyond the wall is not touched); 3 = by the
// thread's wb / wt.  UNI: both lanes' neighbour columns lie in one pair, every
// slot pair is one 64-bit access.  PRED: lane h is written only if !skip_h.
template <int ps, bool UNI, int WALL, bool PRED, bool STORE, class RC, class RU, class RD>
__device__ __forceinline__ void gather_pair(const RunDev &R, const RC C, const RU U, const RD D, const Cols &c,
                                            const F32Force2 &f, const Keep &kp, bool &bad, bool skip0 = false, bool skip1 = false,
                                            bool wb = false, bool wt = false) {
  auto ld = [](const auto &row, int a, int b2, int q) {
    return UNI ? row.ld2(a + q) : f2_bits(row.ld(a + q), row.ld(b2 + q));
  };
  f2_t S[9];
  S[0] = C.ld2(c.o);
  S[1] = ld(C, c.m0, c.m1, 3 * ps);
  S[3] = ld(C, c.p0, c.p1, ps);
  // WALL 3: the slot is the thread's own (row C) or the neighbour's, chosen by address
  const bool ob = WALL == 3 && wb, ot = WALL == 3 && wt;
  const int u2 = c.o + (ob ? 2 : 4) * ps, d4 = c.o + (ot ? 4 : 2) * ps;
  const int u5a = ob ? c.o + 5 * ps : c.m0 + 7 * ps, u5b = ob ? c.o + 1 + 5 * ps : c.m1 + 7 * ps;
  const int u6a = ob ? c.o + 6 * ps : c.p0 + 8 * ps, u6b = ob ? c.o + 1 + 6 * ps : c.p1 + 8 * ps;
  const int d7a = ot ? c.o + 7 * ps : c.p0 + 5 * ps, d7b = ot ? c.o + 1 + 7 * ps : c.p1 + 5 * ps;
  const int d8a = ot ? c.o + 8 * ps : c.m0 + 6 * ps, d8b = ot ? c.o + 1 + 8 * ps : c.m1 + 6 * ps;
  if (WALL == 1) {
    S[2] = C.ld2(c.o + 2 * ps);
    S[5] = C.ld2(c.o + 5 * ps);
    S[6] = C.ld2(c.o + 6 * ps);
  } else {
    S[2] = U.ld2(u2);
    S[5] = ld(U, u5a, u5b, 0);
    S[6] = ld(U, u6a, u6b, 0);
  }
  if (WALL == 2) {
    S[4] = C.ld2(c.o + 4 * ps);
    S[7] = C.ld2(c.o + 7 * ps);
    S[8] = C.ld2(c.o + 8 * ps);
  } else {
    S[4] = D.ld2(d4);
    S[7] = ld(D, d7a, d7b, 0);
    S[8] = ld(D, d8a, d8b, 0);
  }
  f2_t P[9];
  const f2_t drho = collide_f32_nodes(S, P, R.f_pairs, f);
  keep_pair<STORE>(R, kp, P, PRED && skip0, PRED && skip1);
  bad |= (!(f32x2op::lo(drho) > -1.0f) && !(PRED && skip0)) || (!(f32x2op::hi(drho) > -1.0f) && !(PRED && skip1));
  auto st = [&](const auto &row, int a, int b2, int q, f2_t v) {
    if (UNI && !PRED) {
      row.st2(a + q, v);
    } else {
      if (!PRED || !skip0) row.st(a + q, f32x2op::lo(v));
      if (!PRED || !skip1) row.st(b2 + q, f32x2op::hi(v));
    }
  };
  auto st2 = [&](const auto &row, int a, f2_t v) {  // a slot pair of one column pair
    if (!PRED) {
      row.st2(a, v);
    } else {
      if (!skip0) row.st(a, f32x2op::lo(v));
      if (!skip1) row.st(a + 1, f32x2op::hi(v));
    }
  };
  st2(C, c.o, P[0]);
  st(C, c.m0, c.m1, 3 * ps, P[3]);
  st(C, c.p0, c.p1, ps, P[1]);
  if (WALL == 1) {
    st2(C, c.o + 2 * ps, P[4]);
    st2(C, c.o + 5 * ps, P[7]);
    st2(C, c.o + 6 * ps, P[8]);
  } else {
    st2(U, u2, P[4]);
    st(U, u5a, u5b, 0, P[7]);
    st(U, u6a, u6b, 0, P[8]);
  }
  if (WALL == 2) {
    st2(C, c.o + 4 * ps, P[2]);
    st2(C, c.o + 7 * ps, P[5]);
    st2(C, c.o + 8 * ps, P[6]);
  } else {
    st2(D, d4, P[2]);
    st(D, d7a, d7b, 0, P[5]);
    st(D, d8a, d8b, 0, P[6]);
  }
}

// One pair of nodes in a local step: S(n,k) = A[n][k], P(n,k) -> A[n][opp k].
template <int ps, bool PRED, bool STORE>
__device__ __forceinline__ void local_pair(const RunDev &R, float *o, const F32Force2 &f, const Keep &kp, bool &bad,
                                           bool skip0 = false, bool skip1 = false) {
  f2_t S[9], P[9];
#pragma unroll
  for (int k = 0; k < 9; k++) S[k] = *(const f2_t *)(o + k * ps);
  const f2_t drho = collide_f32_nodes(S, P, R.f_pairs, f);
  keep_pair<STORE>(R, kp, P, PRED && skip0, PRED && skip1);
  bad |= (!(f32x2op::lo(drho) > -1.0f) && !(PRED && skip0)) || (!(f32x2op::hi(drho) > -1.0f) && !(PRED && skip1));
#pragma unroll
  for (int k = 0; k < 9; k++) {
    if (!PRED) {
      *(f2_t *)(o + opp_of(k) * ps) = P[k];
    } else {
      if (!skip0) o[opp_of(k) * ps] = f32x2op::lo(P[k]);
      if (!skip1) o[opp_of(k) * ps + 1] = f32x2op::hi(P[k]);
    }
  }
}

__device__ __forceinline__ bool in_box(const RunDev &R, int x, int y) {
  return x >= R.xmin && x <= R.xmax && y >= R.ymin && y <= R.ymax;
}

// Node j of the square's perimeter within rows [ylo, yhi]: the left and right
// columns row by row, then the rest of the bottom and top rows.  The count of
// such nodes is perimeter_count.
__device__ __forceinline__ int perimeter_count(const RunDev &R, int ylo, int yhi) {
  if (yhi < ylo) return 0;
  const int nin = R.xmax - R.xmin - 1;
  return 2 * (yhi - ylo + 1) + (ylo == R.ymin ? nin : 0) + (yhi == R.ymax ? nin : 0);
}
__device__ __forceinline__ void perimeter_node(const RunDev &R, int ylo, int yhi, int j, int &x, int &y) {
  const int side = 2 * (yhi - ylo + 1), nin = R.xmax - R.xmin - 1;
  if (j < side) {
    y = ylo + (j >> 1);
    x = (j & 1) ? R.xmax : R.xmin;
  } else {
    const int q = j - side;
    const bool bottom = ylo == R.ymin && q < nin;
    y = bottom ? R.ymin : R.ymax;
    x = R.xmin + 1 + (ylo == R.ymin && !bottom ? q - nin : q);
  }
}

// One node of the square's perimeter, not the last step of the interval:
// bounce-back masks, drag terms.  Gather step: P(n, opp k) goes back to the
// slot S(n,k) came from (never inside the square: every slot across its
// surface bounces back); with the square at a band edge the rows may lie in
// adjacent bands (shared::cluster addresses), else the three are in this CTA
// (plain indexing, which the compiler schedules freely).
template <bool GATHER, bool STORE, class Band>
__device__ __forceinline__ void perimeter_update(const TemporalArgs &a, const Band &b, int x, int y, bool edge,
                                                 const float *map, float feps, float *keep, bool &bad, float *terms, float *A) {
  const RunDev &R = a.rd;
  const bool remote = GATHER && edge;  // a local step stays in A
  const int ly = y - b.row0, rf = b.rowf;
  const int mask = GATHER ? bounce_mask(R, x, y) : 0;
  const int co = col_off(b, x);
  int at[9];  // float offset of slot k's home: in A, or (remote) in the cluster window
  const int rowC = (remote ? (int)(b.own_c >> 2) : 0) + ly * rf;
  if (GATHER) {
    const int cm = col_off(b, x == 0 ? b.W - 1 : x - 1), cp = col_off(b, x == b.W - 1 ? 0 : x + 1);
    const int rowU = remote && ly == 0 ? (int)(b.prev_c >> 2) + (b.rows_prev - 1) * rf : rowC - rf;
    const int rowD = remote && ly == b.rows - 1 ? (int)(b.next_c >> 2) : rowC + rf;
#pragma unroll
    for (int k = 0; k < 9; k++) {  // S(n,k) = A[n - c_k][opp k], or its own slot
      const int cx = cx_of(k), cy = cy_of(k);
      const int row = cy == 1 ? rowU : (cy == -1 ? rowD : rowC), sx = cx == 1 ? cm : (cx == -1 ? cp : co);
      at[k] = (mask >> k) & 1 ? rowC + co + k * b.ps : row + sx + opp_of(k) * b.ps;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 9; k++) at[k] = rowC + co + k * b.ps;
  }
  float S[9], P[9];
  if (remote) {
#pragma unroll
    for (int k = 0; k < 9; k++) S[k] = ld_cluster(4u * (unsigned)at[k]);
  } else {
#pragma unroll
    for (int k = 0; k < 9; k++) S[k] = A[at[k]];
  }
  const float drho = collide_f32_run(R, S, P, map ? map + (long long)y * b.W + x : nullptr, feps);
  bad |= !(drho > -1.0f);
#pragma unroll
  for (int k = 0; k < 9; k++) {
    if (remote)
      st_cluster(4u * (unsigned)at[opp_of(k)], P[k]);
    else
      A[at[opp_of(k)]] = P[k];
  }
  if (STORE && keep) {
#pragma unroll
    for (int k = 0; k < 9; k++) keep[k * b.plane + (long long)y * b.W + x] = P[k];
  }
  store_drag_terms<false>(R, S, x, y, b.clone, terms);
}

// One node of the last step: S_T (and its drag terms), any position.
template <class Band>
__device__ __forceinline__ void store_last(const TemporalArgs &a, const Band &b, const float *A, int x, int ly,
                                           bool gather, float *terms) {
  const RunDev &R = a.rd;
  const int y = b.row0 + ly, rf = b.rowf;
  const bool box = in_box(R, x, y);
  const int mask = (box || y == 0 || y == b.H - 1) ? bounce_mask(R, x, y) : 0;
  const long long n = (long long)y * b.W + x;
  if (mask & 512) {  // inside the square
#pragma unroll
    for (int k = 0; k < 9; k++) b.dst[k * b.plane + n] = 0.0f;
    return;
  }
  const int co = col_off(b, x), cm = col_off(b, x == 0 ? b.W - 1 : x - 1), cp = col_off(b, x == b.W - 1 ? 0 : x + 1);
  const float *rowC = A + ly * rf;
  const float *rowU = ly == 0 ? b.prev + (b.rows_prev - 1) * rf : rowC - rf;
  const float *rowD = ly == b.rows - 1 ? b.next : rowC + rf;
  float S[9], d = 0.f;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const int cx = cx_of(k), cy = cy_of(k);
    const float *row = cy == 1 ? rowU : (cy == -1 ? rowD : rowC);
    const int sx = cx == 1 ? cm : (cx == -1 ? cp : co);
    S[k] = (!gather || ((mask >> k) & 1)) ? rowC[co + k * b.ps] : row[sx + opp_of(k) * b.ps];
  }
  if (box) store_drag_terms<false>(R, S, x, y, b.clone, terms);
#pragma unroll
  for (int k = 0; k < 9; k++) {
    b.dst[k * b.plane + n] = S[k];
    d += S[k];
  }
  if (!(d > -1.0f)) atomicOr(a.err, (unsigned)ERR_BAD_DENSITY);
}

template <class Band>
__device__ __forceinline__ Band make_band(const TemporalArgs &a, float *A, cg::cluster_group &cluster) {
  Band b;
  b.cs = (int)cluster.num_blocks();
  b.rank = (int)cluster.block_rank();
  b.clone = blockIdx.x / b.cs;
  b.W = a.rd.W;
  b.H = a.rd.H;
  b.Wh = (b.W + 1) / 2;
  b.div_wh = a.div_wh;
  b.row0 = a.band_row0[b.rank];
  b.rows = a.band_row0[b.rank + 1] - b.row0;
  b.rows_prev = b.rank > 0 ? b.row0 - a.band_row0[b.rank - 1] : b.rows;
  b.np = b.rows * b.Wh;
  b.rowf = 2 * b.Wh;
  b.prev = b.rank > 0 ? cluster.map_shared_rank(A, b.rank - 1) : A;
  b.next = b.rank + 1 < b.cs ? cluster.map_shared_rank(A, b.rank + 1) : A;
  const unsigned a_cta = (unsigned)__cvta_generic_to_shared(A);
  b.own_c = cluster_addr(a_cta, b.rank);
  b.prev_c = b.rank > 0 ? cluster_addr(a_cta, b.rank - 1) : b.own_c;
  b.next_c = b.rank + 1 < b.cs ? cluster_addr(a_cta, b.rank + 1) : b.own_c;
  b.plane = a.rd.plane;
  const long long cb = a.rd.pop_base + (long long)b.clone * 9 * b.plane;
  b.src = a.src + cb;
  b.dst = a.dst + cb;
  // opaque: held in registers, not worked out again from the lattice width
  asm volatile("" : "+r"(b.rowf), "+r"(b.Wh), "+r"(b.div_wh), "+r"(b.np));
  return b;
}

// P_0 into the "after a local step" layout A[n][opp k].  FUSED: formed here
// from the previous interval's S (parent copy, perturbation, first collision;
// the same per-node function as the reseed kernel, so bit-identical).
// Square-interior nodes get zeros (the fluid at rest).  The empty lane of an odd
// width's last pair gets a fluid of density 2^40 at rest: the force moves it by
// 2^-40 of what it does the others, so that it takes part in the density test at
// no cost (an open column of density one, driven where the square blocks the rest,
// reaches speeds at which FP32 loses its density).
template <int THREADS, bool FUSED, class Band>
__device__ __forceinline__ void load_band(const TemporalArgs &a, const Band &b, float *A) {
  const RunDev &R = a.rd;
#pragma unroll 1
  for (int j = threadIdx.x; j < 2 * b.np; j += THREADS) {
    const int h = j >= b.np, i = h ? j - b.np : j;
    const int ly = (int)__umulhi((unsigned)i, b.div_wh), xh = i - ly * b.Wh, x = xh + h * b.Wh, y = b.row0 + ly;
    float P[9];
    if (x >= b.W) {
#pragma unroll
      for (int k = 0; k < 9; k++) P[k] = 0x1p40f * (float)w_of(k);
    } else if (FUSED && x > R.xmin && x < R.xmax && y > R.ymin && y < R.ymax) {
#pragma unroll
      for (int k = 0; k < 9; k++) P[k] = 0.0f;
    } else if (FUSED) {
      reseed_node<false>(a.rs, R, a.run, b.clone, x, y, y * b.W + x, P);
    } else {
      const long long n = (long long)y * b.W + x;
#pragma unroll
      for (int k = 0; k < 9; k++) P[k] = b.src[k * b.plane + n];
    }
    float *o = A + ly * b.rowf + 2 * xh + h;
#pragma unroll
    for (int k = 0; k < 9; k++) o[opp_of(k) * b.ps] = P[k];
  }
}

__device__ __forceinline__ float field_eps(const TemporalArgs &a, int t) {
  return t + 1 < a.rd.field_steps ? a.rd.f_field_eps : 0.0f;
}

// Shared memory of one CTA: the nine planes, then the segment list, one class
// byte per segment and the ends of the list's ranges.  temporal_smem (a
// function of the nodes alone) is what a shape is accepted by; a plane of
// kPairs takes the largest band of an even width that it accepts (3219
// pairs), one of kPairsHalf lets two CTAs share an SM, one of kPairsQuarter four.
__host__ __device__ inline size_t temporal_smem(int nb) {
  const int nseg = (nb + 31) / 32;
  return sizeof(float) * 9 * (size_t)nb + 2 * (size_t)((nseg + 7) & ~7) + (size_t)((nseg + 15) & ~15) + 32;
}
constexpr int kPairs = 3220, kPairsHalf = 1600, kPairsQuarter = 784;
// segments of 32 pairs: the first and the last row by themselves, then the
// rows between them
__host__ __device__ inline int segment_count(int rows, int Wh) {
  const int spr = (Wh + 31) / 32;
  return rows == 1 ? spr : 2 * spr + ((rows - 2) * Wh + 31) / 32;
}
__host__ __device__ inline size_t pair_smem(int planes_np, int rows, int W) {
  const int nseg = segment_count(rows, (W + 1) / 2);
  return 8 * 9 * (size_t)planes_np + 2 * (size_t)((nseg + 7) & ~7) + (size_t)((nseg + 15) & ~15) + 32;
}

// Segment classes, in the order of the list.
enum : int { SEG_GENERAL = 0, SEG_EDGE, SEG_WALL, SEG_BOX, SEG_PART, SEG_INNER, SEG_CLASSES };

// Split cluster barrier: a thread arrives once it has done its share of what
// the neighbouring bands wait for, and waits before it next touches theirs.
// (A warp that wrote nothing the neighbours read has nothing to release.)
__device__ __forceinline__ void cluster_arrive(bool release) {
  __syncwarp();  // the aligned form takes whole warps
  if (release)
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  else
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// One step of the band (all but the interval's last step).  Work comes in
// warp-sized entries, dealt out in this order:
//   seam    (gather) the seam pairs of the first and the last row, columns and
//           neighbour rows per lane
//   GENERAL segments of a one-row band, or where the square touches a
//           band-edge row: the same path
//   EDGE    a band-edge row, the row across the edge at shared::cluster
//           addresses
//   perimeter  32 nodes of the square's perimeter, one per lane
//           (bounce-back, drag terms)
//   seam    (gather) 32 seam pairs of the rows between, per-lane addresses
//   WALL    a wall row, bounce-back built in
//   BOX     segments with nodes of the square: as INNER, lanes in the square
//           not written
//   PART    as INNER, but partial or with seam pairs (left out) in it
//   INNER   every slot pair one 64-bit access at a constant offset
// In a local step a node touches only its own slots, the seam included.  The
// deal is round robin, except that the warps holding the first kinds, up to
// the perimeter, sit out one round: those wait on the neighbour's memory, or
// take one node per lane through the drag's divisions.
// Neighbouring bands wait only for nodes of the rows at their common edge:
// once a warp's entries up to there are done it arrives at the cluster
// barrier, and it waits for it at the start of the next step, by which time
// the others have long arrived.  Within the CTA a block barrier ends the step.
// The drag terms' global stores come after the arrival, whose release would
// wait for them (unless the square touches an edge row).
// What a warp keeps of the deal between steps, [0] local, [1] gather: its
// first entry after the head (an index into the list; a gather step's inner
// seam entries come before the list, at nedge - einner and up) and the
// distance to its second one, and what the head holds for it.
struct WarpPlan {
  int k[2], dk[2];
  int nbox, npart, nseg;
  unsigned flags;
};
enum : unsigned {
  PLAN_HEAD = 1u,       // entries ahead of the arrival (<< 1: in a gather step)
  PLAN_PERIMETER = 4u,  // perimeter entries (<< 1: in a gather step)
  PLAN_BOX_EDGE = 16u,  // the square touches a row at a band edge
};

// The head of the deal in a step of one kind.
struct Head {
  int ns, nouter, ninner;        // seam pairs per row; of the first and last row, of those between
  int eouter, einner, eper;      // their entries, the perimeter's
  int ylo, yhi, nper;
  bool box_edge;
  template <class Band>
  __device__ __forceinline__ Head(const RunDev &R, const Band &b, bool gather) {
    ns = seam_count(b);
    nouter = gather ? ns * min(b.rows, 2) : 0;
    ninner = gather ? ns * max(b.rows - 2, 0) : 0;
    eouter = (nouter + 31) / 32;
    einner = (ninner + 31) / 32;
    ylo = max(R.ymin, b.row0);
    yhi = min(R.ymax, b.row0 + b.rows - 1);
    nper = perimeter_count(R, ylo, yhi);
    eper = (nper + 31) / 32;
    box_edge = yhi >= ylo &&
               ((ylo == b.row0 && b.rank > 0) || (yhi == b.row0 + b.rows - 1 && b.rank + 1 < b.cs));
  }
};

// The warp's plan, from the class ends of the list.
template <int NW, class Band>
__device__ __forceinline__ WarpPlan warp_plan(const RunDev &R, const Band &b, const int *range, int warp) {
  WarpPlan p;
  p.nbox = range[SEG_BOX];
  p.npart = range[SEG_PART];
  p.nseg = range[SEG_INNER];
  p.flags = 0;
  const int nedge = range[SEG_EDGE];
#pragma unroll
  for (int g = 0; g < 2; g++) {
    const Head h(R, b, g);
    const int lead = h.eouter + nedge, nhead = lead + h.eper;
    // positions NW .. NW + nhead - 1 of the round robin are left out
    const int q = nhead >= NW ? (warp - nhead % NW + NW) % NW : (warp >= nhead ? warp - nhead : 2 * (NW - nhead) + warp);
    p.k[g] = q - h.einner + nedge;
    p.dk[g] = nhead < NW && warp >= nhead ? NW - nhead : NW;
    if (warp < lead) p.flags |= PLAN_HEAD << g;
    if (h.nper > 0 && (warp - lead % NW + NW) % NW < h.eper) p.flags |= PLAN_PERIMETER << g;
    if (h.box_edge) p.flags |= PLAN_BOX_EDGE;
  }
  // opaque: held in registers over the steps, not worked out again in each
#pragma unroll
  for (int g = 0; g < 2; g++) asm volatile("" : "+r"(p.k[g]), "+r"(p.dk[g]));
  asm volatile("" : "+r"(p.nbox), "+r"(p.npart), "+r"(p.nseg), "+r"(p.flags));
  return p;
}

template <int NW, bool GATHER, bool FIELD, bool STORE, class Band>
__device__ __forceinline__ void band_step(const TemporalArgs &a, const Band &b, const WarpPlan &w, float *A,
                                          const unsigned short *list, const int *range, int warp, int lane, int t,
                                          const float *map, bool &bad) {
  const RunDev &R = a.rd;
  const float feps = FIELD ? field_eps(a, t) : 0.0f;
  constexpr int ps = Band::ps;
  const int rf = b.rowf;
  // this step's checkpoint of the clone, if it is one
  float *keep = STORE && a.keep && (t + 1) % a.keep_every == 0
                    ? a.keep + (t + 1) / a.keep_every * a.keep_stride + R.pop_base + (long long)b.clone * 9 * b.plane
                    : nullptr;
  auto keep_at = [&](int y, int xh) {
    return Keep{STORE && keep ? keep + (long long)y * b.W + xh : nullptr, STORE && xh + b.Wh < b.W ? b.Wh : 0};
  };
  // the pair of segment position i: its row and column, inactive past `lim`
#define CLBM_PAIR(lim)                                                                         \
  const int i = list[k] + lane;                                                                \
  if (i >= (lim)) continue;                                                                    \
  const int ly = (int)__umulhi((unsigned)i, b.div_wh), xh = pair_of(b, i - ly * b.Wh), y = b.row0 + ly
  auto general = [&](int ly, int xh) {
    const int y = b.row0 + ly;
    float *C0 = A + ly * rf;
    const bool wb = y == 0, wt = y == b.H - 1;
    const RowL C{C0};
    const RowG U{wb ? C0 : (ly == 0 ? b.prev + (b.rows_prev - 1) * rf : C0 - rf)};
    const RowG D{wt ? C0 : (ly == b.rows - 1 ? b.next : C0 + rf)};
    gather_pair<ps, false, 3, true, STORE>(R, C, U, D, cols_any(b, xh), pair_force<FIELD>(R, b, map, y, xh), keep_at(y, xh), bad,
                                       in_box(R, xh, y), in_box(R, xh + b.Wh, y), wb, wt);
  };
  auto local = [&](int ly, int xh, auto pred) {
    const int y = b.row0 + ly;
    constexpr bool P = decltype(pred)::value;
    local_pair<ps, P, STORE>(R, A + ly * rf + 2 * xh, pair_force<FIELD>(R, b, map, y, xh), keep_at(y, xh), bad, P && in_box(R, xh, y),
                  P && in_box(R, xh + b.Wh, y));
  };
  const bool lead = w.flags & (PLAN_HEAD << GATHER);
  if (b.cs > 1) cluster_wait();
  // ---- what the neighbouring bands wait for
  if (lead) {
    const int nedge = range[SEG_EDGE];
    int e = warp;  // this warp's next entry, counted within the kind at hand
    if (GATHER) {
      const Head h(R, b, true);
#pragma unroll 1
      for (; e < h.eouter; e += NW) {
        const int j = e * 32 + lane;
        if (j >= h.nouter) continue;
        const int last = j >= h.ns;
        general(last ? b.rows - 1 : 0, seam_pair(b, last ? j - h.ns : j));
      }
      e -= h.eouter;
      const int ngen = range[SEG_GENERAL];
#pragma unroll 1
      for (; e < ngen; e += NW) {
        const int k = e;
        CLBM_PAIR(list[k] < b.Wh ? b.Wh : b.np);
        if (!on_seam(b, xh)) general(y - b.row0, xh);
      }
#pragma unroll 1
      for (; e < nedge; e += NW) {
        const int k = e;
        CLBM_PAIR(list[k] < b.Wh ? b.Wh : b.np);
        if (on_seam(b, xh)) continue;
        float *C = A + ly * rf;
        const F32Force2 f = pair_force<FIELD>(R, b, map, y, xh);
        if (ly == 0)  // warp-uniform
          gather_pair<ps, true, 0, false, STORE>(R, RowL{C}, RowC{b.prev_c + 4u * (unsigned)((b.rows_prev - 1) * rf)},
                                             RowL{C + rf}, cols_inner(xh), f, keep_at(y, xh), bad);
        else
          gather_pair<ps, true, 0, false, STORE>(R, RowL{C}, RowL{C - rf}, RowC{b.next_c}, cols_inner(xh), f, keep_at(y, xh), bad);
      }
    } else {
#pragma unroll 1
      for (; e < nedge; e += NW) {
        const int k = e;
        CLBM_PAIR(list[k] < b.Wh ? b.Wh : b.np);
        local(y - b.row0, xh, std::integral_constant<bool, true>());
      }
    }
  }
  // ---- the perimeter before the arrival if it is part of that, else after it
  const bool box_edge = w.flags & PLAN_BOX_EDGE;
  if (b.cs > 1 && !box_edge) cluster_arrive(lead);
  if (w.flags & (PLAN_PERIMETER << GATHER)) {
    const Head h(R, b, GATHER);
    float *terms = a.terms + (long long)t * a.term_slab + R.term_base;
#pragma unroll 1
    for (int e = (warp - (h.eouter + range[SEG_EDGE]) % NW + NW) % NW; e < h.eper; e += NW) {
      const int j = e * 32 + lane;
      if (j >= h.nper) continue;
      int x, y;
      perimeter_node(R, h.ylo, h.yhi, j, x, y);
      perimeter_update<GATHER, STORE>(a, b, x, y, box_edge, FIELD ? map : nullptr, feps, keep, bad, terms, A);
    }
  }
  if (b.cs > 1 && box_edge) cluster_arrive(true);
  // ---- the rest
  int k = w.k[GATHER], dk = w.dk[GATHER];
  auto step = [&]() {
    k += dk;
    dk = NW;
  };
  if (k < w.nbox) {
    const int nwall = range[SEG_WALL], top = b.np - b.Wh;  // first pair of the last row
    if (GATHER) {
      const int ns = seam_count(b), ninner = ns * max(b.rows - 2, 0), nedge = range[SEG_EDGE];
#pragma unroll 1
      for (; k < nedge; step()) {
        const int j = (k - nedge + (ninner + 31) / 32) * 32 + lane;
        if (j >= ninner) continue;
        const int r = ns == 2 ? j >> 1 : j / 3, ly = r + 1, xh = seam_pair(b, j - ns * r), y = b.row0 + ly;
        float *C = A + ly * rf;
        gather_pair<ps, false, 0, true, STORE>(R, RowL{C}, RowL{C - rf}, RowL{C + rf}, cols_any(b, xh),
                                           pair_force<FIELD>(R, b, map, y, xh), keep_at(y, xh), bad, in_box(R, xh, y),
                                           in_box(R, xh + b.Wh, y));
      }
#pragma unroll 1
      for (; k < nwall; step()) {
        CLBM_PAIR(list[k] < b.Wh ? b.Wh : b.np);
        if (on_seam(b, xh)) continue;
        float *C = A + ly * rf;
        const F32Force2 f = pair_force<FIELD>(R, b, map, y, xh);
        if (y == 0)  // warp-uniform
          gather_pair<ps, true, 1, false, STORE>(R, RowL{C}, RowL{C}, RowL{C + rf}, cols_inner(xh), f, keep_at(y, xh), bad);
        else
          gather_pair<ps, true, 2, false, STORE>(R, RowL{C}, RowL{C - rf}, RowL{C}, cols_inner(xh), f, keep_at(y, xh), bad);
      }
#pragma unroll 1
      for (; k < w.nbox; step()) {
        CLBM_PAIR(top);
        if (on_seam(b, xh)) continue;
        float *C = A + ly * rf;
        gather_pair<ps, true, 0, true, STORE>(R, RowL{C}, RowL{C - rf}, RowL{C + rf}, cols_inner(xh),
                                          pair_force<FIELD>(R, b, map, y, xh), keep_at(y, xh), bad, in_box(R, xh, y),
                                          in_box(R, xh + b.Wh, y));
      }
    } else {
#pragma unroll 1
      for (; k < w.nbox; step()) {
        CLBM_PAIR(k < nwall ? (list[k] < b.Wh ? b.Wh : b.np) : top);
        local(y - b.row0, xh, std::integral_constant<bool, true>());
      }
    }
  }
#pragma unroll 1
  for (; k < w.npart; step()) {
    CLBM_PAIR(b.np - b.Wh);
    if (GATHER) {
      if (on_seam(b, xh)) continue;
      float *C = A + ly * rf;
      gather_pair<ps, true, 0, false, STORE>(R, RowL{C}, RowL{C - rf}, RowL{C + rf}, cols_inner(xh),
                                         pair_force<FIELD>(R, b, map, y, xh), keep_at(y, xh), bad);
    } else {
      local(ly, xh, std::integral_constant<bool, false>());
    }
  }
  // (the field's values come from L2, 700 cycles away, a step's worth of them
  // fits no nearer: those of the next segment are loaded ahead of this one)
  auto field_at = [&](int k) -> f2_t {
    if (!FIELD || k >= w.nseg) return 0;
    const int i = list[k] + lane, ly = (int)__umulhi((unsigned)i, b.div_wh);
    return pair_map(b, map, b.row0 + ly, i - ly * b.Wh - 1);
  };
  f2_t ahead = field_at(k);
#pragma unroll 1
  for (; k < w.nseg; step()) {
    float *C = A + 2 * (list[k] + lane - 1);  // the pair itself
    const f2_t m = ahead;
    ahead = field_at(k + dk);
    const F32Force2 f = pair_force<FIELD>(R, m);
    Keep kp{nullptr, 0};
    if (STORE) {
      const int i = list[k] + lane, ly = (int)__umulhi((unsigned)i, b.div_wh);
      kp = keep_at(b.row0 + ly, i - ly * b.Wh - 1);
    }
    if (GATHER)
      gather_pair<ps, true, 0, false, STORE>(R, RowL{C}, RowL{C - rf}, RowL{C + rf}, cols_inner(0), f, kp, bad);
    else
      local_pair<ps, false, STORE>(R, C, f, kp, bad);
  }
#undef CLBM_PAIR
  __syncthreads();
}

// STORE: the adjoint's forward, which keeps checkpoints (TemporalArgs::keep).
template <int THREADS, int MINB, int NP, bool FIELD, bool STORE>
__global__ void __launch_bounds__(THREADS, MINB) k_temporal_f32(TemporalArgs a) {
  // A[k][pair]: a warp's accesses to one population are consecutive 64-bit
  // words, in this CTA (no bank conflicts) and across a band edge (whole
  // sectors on the way to the other SM)
  using Band = BandT<NP>;
  extern __shared__ __align__(16) float A[];
  constexpr int NW = THREADS / 32;
  cg::cluster_group cluster = cg::this_cluster();
  const Band b = make_band<Band>(a, A, cluster);
  const RunDev &R = a.rd;
  if (a.fused)
    load_band<THREADS, true>(a, b, A);
  else
    load_band<THREADS, false>(a, b, A);
  const int nseg = segment_count(b.rows, b.Wh), spr = (b.Wh + 31) / 32;
  unsigned short *list = (unsigned short *)(A + 9 * Band::ps);
  unsigned char *cls = (unsigned char *)(list + ((nseg + 7) & ~7));
  int *range = (int *)(cls + ((nseg + 15) & ~15));
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  // first pair of segment sg: the first row's, the last row's, those between
  auto seg_start = [&](int sg) {
    return sg < spr ? 32 * sg : (sg < 2 * spr ? (b.rows - 1) * b.Wh + 32 * (sg - spr) : b.Wh + 32 * (sg - 2 * spr));
  };
  for (int sg = warp; sg < nseg; sg += NW) {
    const int i = seg_start(sg) + lane;
    const int lim = sg < spr ? b.Wh : (sg < 2 * spr ? b.np : b.np - b.Wh);
    const int ly = (int)__umulhi((unsigned)i, b.div_wh), xh = pair_of(b, i - ly * b.Wh), y = b.row0 + ly;
    const bool in = i < lim;
    const bool any_box = __any_sync(0xffffffffu, in && (in_box(R, xh, y) || in_box(R, xh + b.Wh, y)));
    const bool full = __all_sync(0xffffffffu, in && !on_seam(b, xh));
    int c;
    if (sg < 2 * spr) {
      const bool wall = sg < spr ? b.row0 == 0 : b.row0 + b.rows == b.H;
      c = b.rows == 1 || any_box ? SEG_GENERAL : (wall ? SEG_WALL : SEG_EDGE);
    } else {
      c = any_box ? SEG_BOX : (full ? SEG_INNER : SEG_PART);
    }
    if (lane == 0) cls[sg] = (unsigned char)c;
  }
  __syncthreads();
  if (warp == 0) {  // the list and its ranges' ends
    const unsigned lower = (1u << lane) - 1u;
    int n = 0;
    for (int pass = 0; pass < SEG_CLASSES; pass++) {
      for (int c = 0; c < nseg; c += 32) {
        const bool take = c + lane < nseg && cls[c + lane] == pass;
        const unsigned m = __ballot_sync(0xffffffffu, take);
        if (take) list[n + __popc(m & lower)] = (unsigned short)seg_start(c + lane);
        n += __popc(m);
      }
      if (lane == 0) range[pass] = n;
    }
  }
  __syncthreads();
  const float *map = FIELD ? a.maps + R.map_base + (long long)b.clone * R.nodes : nullptr;
  const WarpPlan plan = warp_plan<NW>(R, b, range, warp);
  bool bad = false;
  cluster.sync();
  if (b.cs > 1) cluster_arrive(true);  // the first step's wait
  // every step but the last
  // (steps past the field's run through the uniform-force path: with eps = 0
  // the field path computes the same beta and constants bit for bit)
#pragma unroll 1
  for (int t = 0; t + 1 < a.steps; t++) {
    const bool field = FIELD && t + 1 < R.field_steps;
    if ((t & 1) == 0) {
      if (field)
        band_step<NW, true, FIELD, STORE>(a, b, plan, A, list, range, warp, lane, t, map, bad);
      else
        band_step<NW, true, false, STORE>(a, b, plan, A, list, range, warp, lane, t, map, bad);
    } else {
      if (field)
        band_step<NW, false, FIELD, STORE>(a, b, plan, A, list, range, warp, lane, t, map, bad);
      else
        band_step<NW, false, false, STORE>(a, b, plan, A, list, range, warp, lane, t, map, bad);
    }
  }
  // the last step stores S_T
  if (b.cs > 1) cluster_wait();
  {
    const int t = a.steps - 1;
    float *terms = a.terms + (long long)t * a.term_slab + R.term_base;
#pragma unroll 1
    for (int j = threadIdx.x; j < 2 * b.np; j += THREADS) {
      const int h = j >= b.np, i = h ? j - b.np : j;
      const int ly = (int)__umulhi((unsigned)i, b.div_wh), x = i - ly * b.Wh + h * b.Wh;
      if (x < b.W) store_last(a, b, A, x, ly, (t & 1) == 0, terms);
    }
  }
  if (bad) atomicOr(a.err, (unsigned)ERR_BAD_DENSITY);
  cluster.sync();  // no CTA leaves while a neighbour may still read its shared memory
}

typedef void (*TemporalFn)(TemporalArgs);

// shared memory a CTA may use
static constexpr size_t kSmemLimit = 227 * 1024;

int temporal_rows_limit(int W) {
  int r = 0;
  while (temporal_smem((r + 1) * W) <= kSmemLimit) r++;
  return r;
}

bool temporal_resident(int W, int rows) {
  return (long long)rows * ((W + 1) / 2) <= kPairs && pair_smem(kPairs, rows, W) <= kSmemLimit;
}

struct TemporalKernel {
  int pairs, threads;  // of a plane, of a block
  TemporalFn fn[3];    // uniform force, random field, checkpoints
};

#define KERNEL(T, M, N) \
  {N, T, {k_temporal_f32<T, M, N, false, false>, k_temporal_f32<T, M, N, true, false>, k_temporal_f32<T, M, N, false, true>}}
// By variant, for bands of up to `pairs`.  (1024 and 512 threads take an SM's
// registers alone: no use for smaller planes.)
static const TemporalKernel kTemporal[][3] = {
    {KERNEL(1024, 1, kPairs)},
    {KERNEL(512, 1, kPairs)},
    {KERNEL(256, 2, kPairs), KERNEL(256, 2, kPairsHalf), KERNEL(128, 4, kPairsQuarter)}};
#undef KERNEL

int temporal_variant_count() { return (int)(sizeof(kTemporal) / sizeof(kTemporal[0])); }

// The kernel of a variant for `blocks` bands of this shape and its shared memory,
// or nullptr when it cannot run it: the smallest planes that hold the band, for as
// many CTAs an SM as they allow, the quarter's only for more blocks than the half
// planes hold at once (its 128 threads take longer over one band).  us a step,
// half and quarter planes: 8192 clones of 24x16 34.8 and 26.4, of 32x24 48.3 and
// 41.5, 4096 of 64x24 32.4 and 30.0 (a kernel of one node a thread, four CTAs an SM
// too, took 35.2, 42.5 and 31.4); 320 clones of 48x32 3.93 and 3.48, 304 (two an
// SM) 2.50 and 2.84, one 1.77 and 2.32.
static const TemporalKernel *temporal_kernel(int variant, int cs, int W, int rows_max, int blocks, size_t *smem) {
  if (variant < 0 || variant >= temporal_variant_count() || cs < 1 || cs > MAX_CLUSTER || rows_max < 1)
    return nullptr;
  if (temporal_smem(rows_max * W) > kSmemLimit) return nullptr;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return nullptr;
  const TemporalKernel *k = kTemporal[variant];
  for (int i = 1; i < (blocks > 2 * sms ? 3 : 2); i++)
    if (kTemporal[variant][i].pairs >= rows_max * ((W + 1) / 2)) k = &kTemporal[variant][i];
  *smem = std::min(pair_smem(k->pairs, rows_max, W), kSmemLimit);
  return k;
}

static cudaLaunchConfig_t temporal_config(int cs, int threads, int nclones, size_t smem, cudaStream_t s,
                                          cudaLaunchAttribute *attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs * nclones);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// (the limit and not a shape's own need: the attribute is the kernel's, and contexts
// in other threads set it for their shapes between this and the launch)
static cudaError_t prepare(TemporalFn fn, int cs) {
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
  if (e == cudaSuccess && cs > 8) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

// Launch one run's interval with cluster size cs over the bands of
// a.band_row0 (every band at least one row).
cudaError_t launch_temporal(const TemporalArgs &a, int cs, int variant, int nclones, int W,
                            cudaStream_t s) {
  const bool field = a.rd.field_mode != 0 && a.maps != nullptr;
  if (cs < 1 || cs > MAX_CLUSTER || a.band_row0[0] != 0 || a.band_row0[cs] != a.rd.H)
    return cudaErrorInvalidConfiguration;
  int rows_max = 0;
  for (int b = 0; b < cs; b++) {
    const int rows = a.band_row0[b + 1] - a.band_row0[b];
    if (rows < 1) return cudaErrorInvalidConfiguration;
    rows_max = std::max(rows_max, rows);
  }
  size_t smem = 0;
  if (field && a.keep) return cudaErrorInvalidConfiguration;
  const TemporalKernel *k = temporal_kernel(variant, cs, W, rows_max, cs * nclones, &smem);
  if (!k || !temporal_resident(W, rows_max) || !square_thick(a.rd) || a.steps < 1)
    return cudaErrorInvalidConfiguration;
  const TemporalFn fn = k->fn[a.keep ? 2 : field];
  cudaError_t e = prepare(fn, cs);
  if (e != cudaSuccess) return e;
  TemporalArgs args = a;
  const unsigned long long wh = (W + 1) / 2;
  args.div_wh = (unsigned)(((1ULL << 32) + wh - 1) / wh);
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = temporal_config(cs, k->threads, nclones, smem, s, attr);
  return cudaLaunchKernelEx(&cfg, fn, args);
}

// Whether the cluster shape can be resident at all (occupancy query, no launch).
int temporal_max_clusters(int cs, int variant, int W, int rows_max, bool field) {
  size_t smem = 0;
  const TemporalKernel *k = temporal_kernel(variant, cs, W, rows_max, 0, &smem);
  if (!k) return 0;
  const TemporalFn fn = k->fn[field];
  if (prepare(fn, cs) != cudaSuccess) return 0;
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = temporal_config(cs, k->threads, 64, smem, nullptr, attr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, (void *)fn, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

}  // namespace clbm
