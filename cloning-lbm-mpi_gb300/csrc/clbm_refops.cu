// clbm_refops.cu -- function-level entry points: the reference's LBM
// functions on one clone in its own FP64 array-of-structures layout
// IDX(x,y,k) = k + 9*(y + Dy*x) (src/lbm_src/global.h:4), on device pointers,
// with the reference's operation order (bit-identical results).
#include <cmath>
#include <cstdio>
#include <mutex>

#include "../../include/clbm.h"
#include "clbm_internal.h"
#include "clbm_physics.cuh"

namespace clbm {

struct GeomDev {
  int nx, ny, xmin, xmax, ymin, ymax;
};

__device__ __forceinline__ long long aos(const GeomDev &g, int x, int y, int k) {
  return k + 9LL * (y + (long long)g.ny * x);
}

// A time step is five small kernels in a row, a perturbation three: each is
// launched with programmatic stream serialisation, so that its blocks take
// their places while the kernel before it drains, and waits here, before it
// touches memory, until that has completed and its writes are visible (a step of
// a 129x129 state 63 -> 51 us, a perturbation of a 257x257 state 65 -> 58.5).
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
static cudaError_t launch_after(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// streamCollCompute.cpp:7-93: collide in place into fin, push to the periodic
// neighbour in fout, macroscopic fields of the pre-collision state.
__global__ void __launch_bounds__(TILE64) k_ref_stream_collide(GeomDev g, double *fin, double *fout, double *rho,
                                     double *ux, double *uy, double beta0, const double *map,
                                     double tau, double eps) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;  // t = y + ny*x
  if (t >= g.nx * g.ny) return;
  const int x = t / g.ny, y = t - x * g.ny;
  const double omega = DDIV(1., tau);
  const double om1 = DSUB(1.0, omega);
  const double cforce = DSUB(1.0, DMUL(0.5, omega));
  double beta = beta0;
  if (map) beta = DMUL(DADD(1.0, DMUL(eps, map[t])), beta0);
  double wcb[9];
#pragma unroll
  for (int k = 0; k < 9; k++) wcb[k] = DMUL(DMUL(w_of(k), cforce), beta);
  double f[9], post[9];
#pragma unroll
  for (int k = 0; k < 9; k++) f[k] = fin[aos(g, x, y, k)];
  double vx, vy;
  __shared__ Node64<TILE64> node;
  const Moments64 m = moments64(node, f);
  collide_ref64(node, m, post, DMUL(0.5, beta), wcb, omega, om1, &vx, &vy);
#pragma unroll
  for (int k = 0; k < 9; k++) {
    fin[aos(g, x, y, k)] = post[k];
    const int tx = (x + cx_of(k) + g.nx) % g.nx;
    const int ty = (y + cy_of(k) + g.ny) % g.ny;
    fout[aos(g, tx, ty, k)] = post[k];
  }
  if (ux) ux[t] = vx;
  if (uy) uy[t] = vy;
  if (rho) rho[t] = m.rho;
}

// domain_noSlipWalls.cpp:6-22
__global__ void k_ref_walls(GeomDev g, double *fout, const double *fin) {
  after_previous();
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= g.nx) return;
  const int top = g.ny - 1;
  const int up[3] = {2, 5, 6}, down[3] = {4, 7, 8};
#pragma unroll
  for (int i = 0; i < 3; i++) {
    fout[aos(g, x, top, down[i])] = fin[aos(g, x, top, opp_of(down[i]))];
    fout[aos(g, x, 0, up[i])] = fin[aos(g, x, 0, opp_of(up[i]))];
  }
}

// square.cpp:24-50 (the live _TEST variant); one thread per perimeter node
__global__ void k_ref_square(GeomDev g, double *fout, const double *fin) {
  after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int sx = g.xmax - g.xmin, sy = g.ymax - g.ymin;
  const int bottom[3] = {7, 4, 8}, top[3] = {5, 2, 6}, left[3] = {6, 3, 7}, right[3] = {8, 1, 5};
  if (i < sx - 1) {
    const int x = g.xmin + 1 + i;
#pragma unroll
    for (int q = 0; q < 3; q++) {
      fout[aos(g, x, g.ymin, bottom[q])] = fin[aos(g, x, g.ymin, opp_of(bottom[q]))];
      fout[aos(g, x, g.ymax, top[q])] = fin[aos(g, x, g.ymax, opp_of(top[q]))];
    }
  } else if (i < sx - 1 + sy - 1) {
    const int y = g.ymin + 1 + (i - (sx - 1));
#pragma unroll
    for (int q = 0; q < 3; q++) {
      fout[aos(g, g.xmin, y, left[q])] = fin[aos(g, g.xmin, y, opp_of(left[q]))];
      fout[aos(g, g.xmax, y, right[q])] = fin[aos(g, g.xmax, y, opp_of(right[q]))];
    }
  } else if (i == sx - 1 + sy - 1) {
    fout[aos(g, g.xmin, g.ymin, 7)] = fin[aos(g, g.xmin, g.ymin, 5)];
    fout[aos(g, g.xmin, g.ymax, 6)] = fin[aos(g, g.xmin, g.ymax, 8)];
    fout[aos(g, g.xmax, g.ymax, 5)] = fin[aos(g, g.xmax, g.ymax, 7)];
    fout[aos(g, g.xmax, g.ymin, 8)] = fin[aos(g, g.xmax, g.ymin, 6)];
  }
}

// pops driver :430-439
__global__ void k_ref_interior(GeomDev g, double *fout) {
  after_previous();
  const int sx = g.xmax - g.xmin - 1, sy = g.ymax - g.ymin - 1;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (sx <= 0 || sy <= 0 || i >= sx * sy) return;
  const int x = g.xmin + 1 + i / sy, y = g.ymin + 1 + i % sy;
#pragma unroll
  for (int k = 0; k < 9; k++) fout[aos(g, x, y, k)] = w_of(k);
}

// force.cpp:8-144: per-node terms in parallel, then each side summed in node
// order by a thread of its own.
__global__ void k_ref_force(GeomDev g, const double *f, double omega, double *out) {
  after_previous();
  extern __shared__ double terms[];
  const int sx = g.xmax - g.xmin + 1, sy = g.ymax - g.ymin + 1;
  const int nterm = 2 * sy + 2 * sx;
  const double third = 1. / 3.;
  const double c = DSUB(1.0, DMUL(.5, omega));
  for (int i = threadIdx.x; i < nterm; i += blockDim.x) {
    int x, y, side;
    if (i < sy) { side = 0; x = g.xmin; y = g.ymin + i; }
    else if (i < 2 * sy) { side = 1; x = g.xmax; y = g.ymin + i - sy; }
    else if (i < 2 * sy + sx) { side = 2; y = g.ymax; x = g.xmin + i - 2 * sy; }
    else { side = 3; y = g.ymin; x = g.xmin + i - 2 * sy - sx; }
    double fn[9];
#pragma unroll
    for (int k = 0; k < 9; k++) fn[k] = f[aos(g, x, y, k)];
    const Moments64 m = moments_ref64(fn);
    const double rho = m.rho;
    double pxx, pxy;
    pi_ref64(fn, m, pxx, pxy);
    double v;
    if (side == 0) v = DADD(DMUL(rho, third), DMUL(c, pxx));
    else if (side == 1) v = DSUB(DMUL(-rho, third), DMUL(c, pxx));
    else if (side == 2) v = DMUL(-c, pxy);
    else v = DMUL(c, pxy);
    terms[i] = v;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    const int s = threadIdx.x, len = s < 2 ? sy : sx, i = s < 2 ? s * sy : 2 * sy + (s - 2) * sx;
    double v = terms[i];
    for (int q = 1; q < len; q++) v = DADD(v, terms[i + q]);
    const double a = __shfl_sync(0xfu, v, 1), b = __shfl_sync(0xfu, v, 2), c4 = __shfl_sync(0xfu, v, 3);
    if (s == 0) *out = DADD(DADD(DADD(v, a), b), c4);
  }
}

// generatePerturbedState.cpp:4-38 in two passes: fixed-order norm reduction,
// then the element-wise update.  A block takes 1024 values, four per thread
// (per value the reduction costs the FP64 pipe, which bounds these kernels,
// 0.5 operations instead of 8, next to the 2 of the squares and the mix's
// 2 nsnap - 1).  mixed
// (nullable): where the mix is kept for the update, which forms it again
// otherwise.
constexpr int PERTURB_BLOCK = 1024;
constexpr int PERTURB_SMALL = 256;  // of small states, one per thread (perturb_block)
struct Prefactors {
  double v[64];
  int place;  // exponent of their sum where snapshot_mix_fx takes them, else NO_PLACE
};
constexpr int NO_PLACE = 1 << 20;
__device__ __forceinline__ double snapshot_mix(const double *snaps, int nsnap, int n, unsigned i,
                                               const Prefactors &pref) {
  double mix = DMUL(pref.v[0], snaps[i]);
  for (int q = 1; q < nsnap; q++) mix = DADD(mix, DMUL(pref.v[q], snaps[(long long)q * n + i]));
  return mix;
}
// The mixes of four values at once (their loads in flight together), the sums
// in fixed point: the FP64 pipe bounds the pass, and the sums are half of its
// operations (clbm_physics.cuh has the method).  At 2^(59 - place) over the
// power of two of the first snapshot's value, room for sums of four times that
// value by the prefactors.  A bit of the result for each value that has a
// negative product, too large a sum or a partial sum of less than 2^-8 of the
// room.  The first product is exact there (mix_place).  Ten snapshots of a
// 257x257 state, from a cold L2: the pass 37 us in FP64, 30 one value at a time,
// 22 four at a time; the whole perturbation 61, 57, 48 us.
__device__ __forceinline__ unsigned snapshot_mix_fx(const double *snaps, int nsnap, int n, const unsigned i[4],
                                                    const Prefactors &pref, double mix[4]) {
  fx_t acc[4];
  int e0[4], bad[4], least[4], most[4];
#pragma unroll
  for (int j = 0; j < 4; j++) acc[j] = 0, least[j] = 0x7fffffff, most[j] = 0;
  for (int q = 0; q < nsnap; q++) {
    const double *snap = snaps + (long long)q * n;
    double p[4];
#pragma unroll
    for (int j = 0; j < 4; j++) p[j] = snap[i[j]];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      if (q == 0) {
        e0[j] = __double2hiint(p[j]) >> 20;
        bad[j] = e0[j] - 900 | 1100 - e0[j];
      }
      p[j] = DMUL(pref.v[q], p[j]);
      const int hi = __double2hiint(p[j]), s = pref.place + e0[j] + 2 - (hi >> 20);
      bad[j] |= hi | s;
      const fxu_t m = (((fxu_t)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(p[j])) << 9;
      const unsigned c = min((unsigned)s, 63u);
      const fxu_t y = m >> c;
      const fx_t v = acc[j] + (fx_t)(y | (fxu_t)((y << c) != m));
      if (q > 0) least[j] = min(least[j], (int)(v >> 32));
      most[j] = max(most[j], (int)(v >> 32));
      acc[j] = q > 0 ? fx_round(v) : v;
    }
  }
  unsigned off = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const double d = fx_double(acc[j]);
    mix[j] = __hiloint2double(__double2hiint(d) + ((pref.place + e0[j] + 2 - 1023) << 20), __double2loint(d));
    off |= (unsigned)!(bad[j] >= 0 && least[j] >= 1 << 22 && most[j] < 1 << 30) << j;
  }
  return off;
}
// The place for the prefactors: none below zero, the first at least 2^-7 and the
// first two together 2^-5 of the sum's power of two, so that few values are
// turned back (ten random prefactors: about 96 of 100 draws); other calls stay
// FP64.
static int mix_place(const double *prefactors, int nsnap) {
  double sum = 0.0;
  for (int q = 0; q < nsnap; q++) {
    if (!(prefactors[q] >= 0.0)) return NO_PLACE;
    sum += prefactors[q];
  }
  if (nsnap < 2 || !(sum > 1e-6 && sum < 1e6)) return NO_PLACE;
  const int e = std::ilogb(sum);
  const bool ok = prefactors[0] >= std::ldexp(1.0, e - 7) && prefactors[0] + 0.5 * prefactors[1] >= std::ldexp(1.0, e - 5);
  return ok ? e : NO_PLACE;
}
template <int PER>
__global__ void __launch_bounds__(256) k_ref_perturb_norms(const double *fin, const double *snaps, int nsnap, int n,
                                                           const Prefactors pref, double *partials, double *mixed) {
  after_previous();
  __shared__ double red[2][256 / 32];
  double n0 = 0.0, n1 = 0.0;
  const unsigned first = blockIdx.x * (256 * PER) + threadIdx.x;
  unsigned i[PER], off = (1u << PER) - 1;
  double mix[PER];
#pragma unroll
  for (int j = 0; j < PER; j++) i[j] = min(first + j * 256, (unsigned)n - 1);
  if constexpr (PER == 4)
    if (pref.place != NO_PLACE) off = snapshot_mix_fx(snaps, nsnap, n, i, pref, mix);
#pragma unroll
  for (int j = 0; j < PER; j++) {
    if (first + j * 256 >= (unsigned)n) break;
    if (off >> j & 1) mix[j] = snapshot_mix(snaps, nsnap, n, i[j], pref);
    if (mixed) mixed[i[j]] = mix[j];
    n0 = __fma_rn(fin[i[j]], fin[i[j]], n0);
    n1 = __fma_rn(mix[j], mix[j], n1);
  }
  for (int o = 16; o > 0; o >>= 1) {
    n0 = DADD(n0, __shfl_down_sync(0xffffffffu, n0, o));
    n1 = DADD(n1, __shfl_down_sync(0xffffffffu, n1, o));
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = n0;
    red[1][threadIdx.x >> 5] = n1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a0 = red[0][0], a1 = red[1][0];
    for (int w = 1; w < 256 / 32; w++) {
      a0 = DADD(a0, red[0][w]);
      a1 = DADD(a1, red[1][w]);
    }
    partials[2 * blockIdx.x] = a0;
    partials[2 * blockIdx.x + 1] = a1;
  }
}

// The two norms summed over the blocks' partials, once, by one block in a fixed
// order (thread t the partials t, t + 256, ..., then a tree; a single thread
// spent 100 us on 2323 pairs): out[0] = |f| / |mix| (the
// mix weight), out[1] = 1 / (1 + eps * sum(pref) * weight)
// (generatePerturbedState.cpp:22-36).
__global__ void __launch_bounds__(256) k_ref_perturb_finalize(const Prefactors pref, int nsnap, const double *partials,
                                                              int nblocks, double eps, double *out) {
  after_previous();
  __shared__ double red[2][256 / 32];
  double a0 = 0.0, a1 = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += 256) {
    a0 = DADD(a0, partials[2 * b]);
    a1 = DADD(a1, partials[2 * b + 1]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    a0 = DADD(a0, __shfl_down_sync(0xffffffffu, a0, o));
    a1 = DADD(a1, __shfl_down_sync(0xffffffffu, a1, o));
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = a0;
    red[1][threadIdx.x >> 5] = a1;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < 256 / 32; w++) {
    a0 = DADD(a0, red[0][w]);
    a1 = DADD(a1, red[1][w]);
  }
  const double weight = DDIV(__dsqrt_rn(a0), __dsqrt_rn(a1));
  double sum = pref.v[0];
  for (int q = 1; q < nsnap; q++) sum = DADD(sum, pref.v[q]);
  out[0] = weight;
  out[1] = DDIV(1., DADD(1.0, DMUL(DMUL(sum, eps), weight)));
}

// f <- (f + eps * mix * weight) / a with (weight, 1/a) from k_ref_perturb_finalize
__global__ void k_ref_perturb_apply(double *fin, const double *snaps, int nsnap, int n,
                                    const Prefactors pref, const double *wa, double eps, const double *mixed) {
  after_previous();
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (unsigned)n) return;
  const double w = wa[0], inv = wa[1];
  const double mix = mixed ? mixed[i] : snapshot_mix(snaps, nsnap, n, i, pref);
  fin[i] = DMUL(DADD(fin[i], DMUL(DMUL(eps, mix), w)), inv);
}

}  // namespace clbm

using namespace clbm;

extern "C" void clbm_set_error(const char *msg);
extern "C" int clbm_status_from_cuda(cudaError_t e);

static int check_geom(const clbm_geom *g) {
  if (!g || g->nx < 3 || g->ny < 3 || g->xmin < 0 || g->xmax >= g->nx || g->xmin > g->xmax ||
      g->ymin < 0 || g->ymax >= g->ny || g->ymin > g->ymax) {
    clbm_set_error("invalid geometry");
    return CLBM_ERR_INVALID;
  }
  return CLBM_OK;
}

// Values a block of the norms takes.  Four per thread where there are blocks for
// all SMs; one per thread up to two such blocks an SM, whose 1024 values kept a
// few SMs' FP64 pipes busy while the others had none.  us a call that allocates
// nothing, one per thread and four: 12x9 with 40 snapshots 34.8 and 48.2, 80x60 with
// 10 28.0 and 29.9, 97x97 33.2 and 32.2, 129x129 37.4 and 34.9.
static int perturb_block(int n) { return n <= 2 * 152 * 256 ? PERTURB_SMALL : PERTURB_BLOCK; }

// The three passes of a perturbation; wa: the weight pair, part: two norm
// partials per block (perturb_block), mixed (nullable): n values (device).
static cudaError_t run_perturb(double *fin, const double *snaps, double eps, int nsnap, int n, const double *prefactors,
                               double *wa, double *part, double *mixed, cudaStream_t st) {
  Prefactors pref = {};
  for (int q = 0; q < nsnap; q++) pref.v[q] = prefactors[q];
  pref.place = mix_place(prefactors, nsnap);
  const int values = perturb_block(n), nb = (n - 1) / values + 1;
  cudaError_t e = launch_after(values == PERTURB_SMALL ? k_ref_perturb_norms<1> : k_ref_perturb_norms<4>, nb, 256, 0, st,
                               fin, snaps, nsnap, n, pref, part, mixed);
  if (e == cudaSuccess) e = launch_after(k_ref_perturb_finalize, 1, 256, 0, st, pref, nsnap, part, nb, eps, wa);
  if (e == cudaSuccess) e = launch_after(k_ref_perturb_apply, (n - 1) / 256 + 1, 256, 0, st, fin, snaps, nsnap, n, pref, wa, eps, mixed);
  return e;
}

static GeomDev to_dev(const clbm_geom *g) {
  return GeomDev{g->nx, g->ny, g->xmin, g->xmax, g->ymin, g->ymax};
}

extern "C" int clbm_ref_stream_collide(const clbm_geom *g, double *fin, double *fout, double *rho,
                                       double *ux, double *uy, double beta, double tau,
                                       void *stream) {
  if (int s = check_geom(g)) return s;
  if (!fin || !fout) return CLBM_ERR_INVALID;
  const int n = g->nx * g->ny;
  return clbm_status_from_cuda(launch_after(k_ref_stream_collide, (n + TILE64 - 1) / TILE64, TILE64, 0,
                                            (cudaStream_t)stream, to_dev(g), fin, fout, rho, ux, uy, beta, (const double *)nullptr, tau, 0.0));
}

extern "C" int clbm_ref_stream_collide_spatial(const clbm_geom *g, double *fin, double *fout,
                                               double *rho, double *ux, double *uy, double beta0,
                                               const double *map, double tau, double eps,
                                               void *stream) {
  if (int s = check_geom(g)) return s;
  if (!fin || !fout || !map) return CLBM_ERR_INVALID;
  const int n = g->nx * g->ny;
  return clbm_status_from_cuda(launch_after(k_ref_stream_collide, (n + TILE64 - 1) / TILE64, TILE64, 0,
                                            (cudaStream_t)stream, to_dev(g), fin, fout, rho, ux, uy, beta0, map, tau, eps));
}

extern "C" int clbm_ref_walls_bb(const clbm_geom *g, double *fout, const double *fin,
                                 void *stream) {
  if (int s = check_geom(g)) return s;
  return clbm_status_from_cuda(launch_after(k_ref_walls, (g->nx + 127) / 128, 128, 0, (cudaStream_t)stream, to_dev(g), fout, fin));
}

extern "C" int clbm_ref_square_bb(const clbm_geom *g, double *fout, const double *fin,
                                  void *stream) {
  if (int s = check_geom(g)) return s;
  const int nthreads = (g->xmax - g->xmin - 1) + (g->ymax - g->ymin - 1) + 1;
  return clbm_status_from_cuda(launch_after(k_ref_square, (nthreads + 127) / 128, 128, 0, (cudaStream_t)stream, to_dev(g), fout, fin));
}

extern "C" int clbm_ref_interior_reset(const clbm_geom *g, double *fout, void *stream) {
  if (int s = check_geom(g)) return s;
  const int sx = g->xmax - g->xmin - 1, sy = g->ymax - g->ymin - 1;
  if (sx <= 0 || sy <= 0) return CLBM_OK;
  return clbm_status_from_cuda(launch_after(k_ref_interior, (sx * sy + 127) / 128, 128, 0, (cudaStream_t)stream, to_dev(g), fout));
}

extern "C" int clbm_ref_force_on_square(const clbm_geom *g, const double *f, double omega,
                                        double *result, void *stream) {
  if (int s = check_geom(g)) return s;
  if (!f || !result) return CLBM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  double *d_out = nullptr;
  cudaError_t e = call_alloc((void **)&d_out, sizeof(double), st);
  if (e != cudaSuccess) return clbm_status_from_cuda(e);
  const int nterm = 2 * (g->xmax - g->xmin + 1) + 2 * (g->ymax - g->ymin + 1);
  e = launch_after(k_ref_force, 1, 256, nterm * sizeof(double), st, to_dev(g), f, omega, d_out);
  if (e == cudaSuccess) e = cudaMemcpyAsync(result, d_out, sizeof(double), cudaMemcpyDeviceToHost, st);
  cudaFreeAsync(d_out, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return clbm_status_from_cuda(e);
}

extern "C" int clbm_ref_perturbed_state(double *fin, const double *snaps, double eps, int nsnap,
                                        int n, const double *prefactors, void *stream) {
  if (!fin || !snaps || !prefactors || nsnap < 1 || nsnap > 64 || n < 1) return CLBM_ERR_INVALID;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t nb = (size_t)(n - 1) / perturb_block(n) + 1, head = 2 + 2 * nb;
  double *d_buf = nullptr;
  // (without room for a further state the mix is formed twice, the same values)
  bool keep = true;
  cudaError_t e = call_alloc((void **)&d_buf, sizeof(double) * (head + n), st);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    keep = false;
    e = call_alloc((void **)&d_buf, sizeof(double) * head, st);
  }
  if (e != cudaSuccess) return clbm_status_from_cuda(e);
  e = run_perturb(fin, snaps, eps, nsnap, n, prefactors, d_buf, d_buf + 2, keep ? d_buf + head : nullptr, st);
  cudaFreeAsync(d_buf, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return clbm_status_from_cuda(e);
}

// ---------------------------------------------------------------------------
// clbm_ref_perturbed_state_noalloc: the same kernels as
// clbm_ref_perturbed_state, with their scratch (two norm partial sums per
// block, the mix weight) in a fixed device array instead of a per-call
// allocation.  It serves callers that must not allocate device memory at all:
// code running under an allocator that already owns the whole device, or
// inside a time-critical loop where an allocation's implicit synchronisation
// is not acceptable.
namespace {
constexpr int NOALLOC_MAX_N = 1 << 20;                     // values per state, 9*Dx*Dy
constexpr int NOALLOC_MAX_BLOCKS = NOALLOC_MAX_N / PERTURB_BLOCK;  // norm partials (pairs; perturb_block: 304 of the small)
constexpr int NOALLOC_PREF = 64;                           // prefactors (nsnap <= 64)
// Shared by every call on a device and kept until the process exits
// (16 KB per device that loads the library): the mix weight and 1/a, then the
// norm partials.  Nothing in it has to start at zero: each call overwrites the
// weight pair and every partial it reads.
static __device__ __align__(256) double g_noalloc_scratch[2 + 2 * NOALLOC_MAX_BLOCKS];

constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mutex;
double *g_noalloc_addr[NOALLOC_MAX_DEVICES] = {};

// The array's device address on the current device, looked up once per
// device with that device current (the host-side symbol is not a device
// address and must never be passed to a kernel).
int noalloc_scratch(double **out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return clbm_status_from_cuda(e);
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
    clbm_set_error("device ordinal beyond the no-alloc scratch table");
    return CLBM_ERR_INVALID;
  }
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_addr[dev]) {
    double *p = nullptr;
    e = cudaGetSymbolAddress((void **)&p, g_noalloc_scratch);
    if (e != cudaSuccess) return clbm_status_from_cuda(e);
    g_noalloc_addr[dev] = p;
  }
  *out = g_noalloc_addr[dev];
  return CLBM_OK;
}
}  // namespace

extern "C" int clbm_ref_perturbed_state_noalloc(double *fin, const double *snaps, double eps,
                                                int nsnap, int n, const double *prefactors,
                                                void *stream) {
  if (!fin || !snaps || !prefactors || nsnap < 1 || nsnap > NOALLOC_PREF || n < 1) {
    clbm_set_error("invalid argument");
    return CLBM_ERR_INVALID;
  }
  if (n > NOALLOC_MAX_N) {
    clbm_set_error("n exceeds the no-alloc scratch limit of 1048576 values (9*Dx*Dy)");
    return CLBM_ERR_INVALID;
  }
  double *scratch = nullptr;
  if (int s = noalloc_scratch(&scratch)) return s;
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = run_perturb(fin, snaps, eps, nsnap, n, prefactors, scratch, scratch + 2, nullptr, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return clbm_status_from_cuda(e);
}
