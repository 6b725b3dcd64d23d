// Mixed-precision multigrid for the tolerance-driven projection solves.
//
// Same discrete operator as the MUDPACK-exact path (dismd2cr's 9-point
// coefficients, periodic x with MUDPACK's ghost columns, Neumann y), a
// different iteration: FP64 iterative refinement around FP32 V-cycles.
//   r = b - A phi            float-float (~48 bits, FP32 pipe), ||r||, ||b||
//   stop if ||r|| <= tol ||b||
//   A e = r                  one FP32 V(1,1) cycle from e = 0 on MUDPACK's
//                            coarse-level operators, alternating-direction
//                            zebra line Gauss-Seidel smoother, MUDPACK's
//                            full-weighting restriction and cubic prolongation
//   phi = phi + e            float-float; phi is widened to FP64 at the end
// GB300 runs FP32 at ~60x its FP64 rate; with float-float refinement the
// solve never touches the FP64 pipe beyond splitting the rhs and widening
// the result, and reaches relative residuals down to ~1e-13.  On a grid stretched in y the strong coupling is
// along y near the wall and along x far from it; line relaxation in both
// directions smooths both regions, so each cycle cuts the residual ~10x
// where MUDPACK's point smoother (W-cycles) gets ~1.3x.
//
// Problems with kx^2 = 0 are singular (periodic x, Neumann y).  They are
// solved as well-posed problems in the same batch: the right-hand side loses
// its component along the operator's left null vector, the tolerance is the
// same as for every other problem, and the solution has zero mean.  Inside
// the FP32 cycle their coarsest-level correction is shifted to zero mean (a
// constant is in the null space at every level and prolongs to a constant).
#include <algorithm>

#include "ek_internal.h"
#include "ek_unet.h"

namespace ek {

namespace {

struct LvF {
  int nx, ny;
  float *e, *r, *cof, *cp;  // e: (0:nx+1,0:ny+1)xP; r: nx*ny*P; cof: 11*nx*ny; cp: line-solve scratch nx*ny*P
  const float4 *cf4;        // cof packed per point (MgLevelF::cf4)
};
struct FastDev {
  int P, ngrid, orth;
  LvF lv[24];
  float *scr;              // finest-size scratch x P (residual / correction)
  double *rhs;              // FP64 finest rhs
  float *phh, *phl;         // float-float finest iterate, with ghosts (buffer 0)
  float *phh2, *phl2;       // buffer 1: problem p's iterate after n corrections is in buffer n & 1
  float *bh, *bl;           // float-float finest rhs
  const float2 *cf2;        // float-float finest coefficients, (hi, lo) interleaved
  int nfx, nfy;
  const double *kx2;
  double *phif;            // output (finest interior, problem fastest)
  double *red;             // 6 per problem: |b|^2, |r|^2, two unused, meas
  int *done, *cycles, *alldone;
  int *iter;               // corrections applied so far
  int *count;              // residual blocks finished (f_check)
  double tol;
};

__device__ __forceinline__ float &E(const LvF &L, int P, int i, int j, int p) {
  return L.e[((size_t)j * (L.nx + 2) + i) * P + p];
}

// Decide per problem after a residual; iter = corrections applied so far
// (the device counter plus incr).  A problem within the tolerance is done
// (1); at iter = maxit the rest stop (2); when none is left, alldone.  In a
// captured step graph the block also sets the condition of the while-node
// that repeats the correction cycle: 1 while any problem is active.
struct CheckF {
  int on, maxit, incr, use_cond;
  cudaGraphConditionalHandle cond;
};
// All threads of one block, after every block's sums have reached g.red.
__device__ __forceinline__ void f_check(const FastDev &g, const CheckF &ck, int tid, int nt) {
  __shared__ int active;
  const int iter = *g.iter + ck.incr;
  const bool last = iter >= ck.maxit;
  if (tid == 0) active = 0;
  __syncthreads();
  for (int p = tid; p < g.P; p += nt) {
    if (g.done[p]) continue;
    g.cycles[p] = iter;
    const double bn = sqrt(__ldcg(&g.red[6 * p]));
    const double meas = (bn > 0.0) ? sqrt(__ldcg(&g.red[6 * p + 1])) / bn : 0.0;
    const bool conv = meas <= g.tol;
    g.red[6 * p + 4] = meas;
    for (int k = 0; k < 4; ++k) g.red[6 * p + k] = 0.0;
    if (conv) g.done[p] = 1;
    else if (last) g.done[p] = 2;
    else atomicAdd(&active, 1);
  }
  __syncthreads();
  if (tid == 0) {
    *g.iter = iter;
    if (active == 0) *g.alldone = 1;
    if (ck.use_cond) cudaGraphSetConditional(ck.cond, active == 0 ? 0u : 1u);
  }
}
__global__ void k_f_check(FastDev g, CheckF ck) {
  if (*g.alldone) {
    if (ck.use_cond && threadIdx.x == 0) cudaGraphSetConditional(ck.cond, 0u);
    return;
  }
  f_check(g, ck, (int)threadIdx.x, (int)blockDim.x);
}

// r = b - A phi at the finest level in float-float (about 48 bits, on the
// FP32 pipe); r32 = r; per-problem |b|^2 and |r|^2.  With `update` the
// correction of the cycle just run is applied first, phi' = phi + e (the
// float-float sum), and written to the other iterate buffer, ghosts
// included; r is then the residual of phi'.  The iterate of problem p is in
// buffer cycles[p] & 1 (corrections applied so far).  Block row j = 1..ny,
// lanes over 32 problems; each warp walks a contiguous run of i with the
// values at i-1, i, i+1 of row j kept in registers.
// On a small grid the time is that of one run, about 1.5 us a point of
// dependent float-float operations, so a row is cut into gridDim.z blocks'
// runs while that fills the SMs (resid_blocks), and with ck.on the last block
// to finish decides per problem, which saves a launch.  64 x 65 x 65, residual
// and decision: 15.4 + 4.5 us -> 12.9.  A grid of several waves
// leaves the decision to k_f_check: there each block's wait for its sums to
// be visible cost more, 277 us -> 285 against 4 on 512 x 385 x 257.
constexpr int kRY = 8;
// (at most 64 registers: four blocks an SM; its loads need the warps)
template <bool UPDATE, bool ORTH>
__global__ void __launch_bounds__(32 * kRY, 4) k_f_resid_ff(FastDev g, CheckF ck) {
  if (*g.alldone) {
    if (ck.on && ck.use_cond && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x | threadIdx.y) == 0)
      cudaGraphSetConditional(ck.cond, 0u);
    return;
  }
  const int P = g.P;
  const int p = blockIdx.x * 32 + threadIdx.x;
  const int ty = threadIdx.y;
  const int nx = g.nfx, ny = g.nfy, j = 1 + (int)blockIdx.y;
  const size_t npt = (size_t)nx * ny;
  float sb = 0.f, sr = 0.f;
  const bool act = (p < P) && !g.done[p];
  if (act) {
    const int par = g.cycles[p] & 1;
    const float *__restrict__ sh = par ? g.phh2 : g.phh;
    const float *__restrict__ sl = par ? g.phl2 : g.phl;
    float *__restrict__ dh = par ? g.phh : g.phh2;
    float *__restrict__ dl = par ? g.phl : g.phl2;
    const float *__restrict__ ef = g.lv[g.ngrid - 1].e;
    const size_t si = P, sj = (size_t)(nx + 2) * P;
    const FF kx2(g.kx2[p]);
    auto V = [&](size_t q) {
      FF v(sh[q], sl[q]);
      if (UPDATE) v = v + FF(ef[q], 0.f);
      return v;
    };
    const int runs = kRY * (int)gridDim.z, per = (nx + runs - 1) / runs;
    const int i0 = 1 + ((int)blockIdx.z * kRY + ty) * per, i1 = min(nx, i0 + per - 1);
    const size_t row = (size_t)j * (nx + 2) * P + p;
    FF wm, wc;
    if (i0 <= i1) {
      wm = V(row + (size_t)(i0 - 1) * si);
      wc = V(row + (size_t)i0 * si);
    }
    for (int i = i0; i <= i1; ++i) {
      const size_t pt = (size_t)(j - 1) * nx + (i - 1);
      const size_t q = row + (size_t)i * si;
      auto CF = [&](int l) {
        const float2 v = g.cf2[l * npt + pt];
        return FF(v.x, v.y);
      };
      const FF wp = V(q + si), wn = V(q + sj), ws = V(q - sj);
      FF s = CF(0) * wp;
      if (!ORTH) s = s + CF(1) * V(q + si + sj);
      s = s + CF(2) * wn;
      if (!ORTH) s = s + CF(3) * V(q + sj - si);
      s = s + CF(4) * wm;
      if (!ORTH) s = s + CF(5) * V(q - si - sj);
      s = s + CF(6) * ws;
      if (!ORTH) s = s + CF(7) * V(q + si - sj);
      const FF c9 = ((-kx2 * CF(10)) - CF(8)) + CF(9);
      s = s + c9 * wc;
      const FF b(g.bh[pt * P + p], g.bl[pt * P + p]);
      const FF r = b - s;
      const float r32 = __fadd_rn(r.hi, r.lo);
      sb = fmaf(b.hi, b.hi, sb);
      sr = fmaf(r32, r32, sr);
      g.lv[g.ngrid - 1].r[pt * P + p] = r32;
      if (UPDATE) {
        dh[q] = wc.hi;
        dl[q] = wc.lo;
        if (i == nx - 1) {
          dh[row] = wc.hi;
          dl[row] = wc.lo;
        }
        if (i == 2) {
          dh[row + (size_t)(nx + 1) * si] = wc.hi;
          dl[row + (size_t)(nx + 1) * si] = wc.lo;
        }
      }
      wm = wc;
      wc = wp;
    }
  }
  __shared__ float red[2][kRY][32];
  red[0][ty][threadIdx.x] = sb;
  red[1][ty][threadIdx.x] = sr;
  __syncthreads();
  if (ty == 0 && act) {
    for (int y = 1; y < kRY; ++y) {
      sb += red[0][y][threadIdx.x];
      sr += red[1][y][threadIdx.x];
    }
    atomicAdd(&g.red[6 * p], (double)sb);
    atomicAdd(&g.red[6 * p + 1], (double)sr);
  }
  if (!ck.on) return;
  __shared__ int mine;
  __threadfence();  // the sums before the count
  __syncthreads();
  const int tid = ty * 32 + (int)threadIdx.x;
  if (tid == 0) mine = atomicAdd(g.count, 1);
  __syncthreads();
  if (mine != (int)(gridDim.x * gridDim.y * gridDim.z) - 1) return;
  __threadfence();
  if (tid == 0) *g.count = 0;
  f_check(g, ck, tid, 32 * kRY);
}

// Learned initial guess: after k_f_resid_ff on the unscaled guess g
// (r = b - A g), <r, b> per problem; then the least-squares factor
// alpha = <A g, b> / |A g|^2 = (|b|^2 - <r,b>) / (|b|^2 - 2<r,b> + |r|^2),
// the residual ratio it leaves, |b - alpha A g| / |b|, in red[6p+5], and the
// accumulators cleared for the iteration.
__global__ void __launch_bounds__(32 * kRY) k_f_guess_rb(FastDev g) {
  const int P = g.P;
  const int p = blockIdx.x * 32 + threadIdx.x;
  const int ty = threadIdx.y;
  const int nx = g.nfx, j = 1 + (int)blockIdx.y;
  const LvF &F = g.lv[g.ngrid - 1];
  float s = 0.f;
  const bool act = (p < P) && !g.done[p];
  if (act)
    for (int i = 1 + ty; i <= nx; i += kRY) {
      const size_t pt = (size_t)(j - 1) * nx + (i - 1);
      s = fmaf(F.r[pt * P + p], g.bh[pt * P + p], s);
    }
  __shared__ float red[kRY][32];
  red[ty][threadIdx.x] = s;
  __syncthreads();
  if (ty == 0 && act) {
    for (int y = 1; y < kRY; ++y) s += red[y][threadIdx.x];
    atomicAdd(&g.red[6 * p + 2], (double)s);
  }
}

__global__ void k_f_guess_alpha(FastDev g, float *alpha) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < g.P; p += gridDim.x * blockDim.x) {
    double a = 0.0;
    if (!g.done[p]) {
      const double bb = g.red[6 * p], rr = g.red[6 * p + 1], rb = g.red[6 * p + 2];
      const double num = bb - rb, den = bb - 2.0 * rb + rr;
      if (den > 0.0) a = num / den;
      const double rho2 = bb > 0.0 ? (bb - a * num) / bb : 0.0;
      g.red[6 * p + 5] = sqrt(fmax(rho2, 0.0));
    }
    alpha[p] = (float)a;
    for (int k = 0; k < 4; ++k) g.red[6 * p + k] = 0.0;
  }
}

__global__ void k_f_guess_scale(FastDev g, const float *alpha) {
  const size_t n = (size_t)(g.nfx + 2) * (g.nfy + 2) * g.P;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
    g.phh[t] *= alpha[t % g.P];
}

// float-float rhs from the FP64 one (once per solve)
__global__ void k_f_split(const double *b, float *bh, float *bl, size_t n) {
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const FF v(b[t]);
    bh[t] = v.hi;
    bl[t] = v.lo;
  }
}

// The solve's statistics on the device (a step run as a graph reads them
// after the step): cycle range, problems stopped at the cap, largest final
// relative residual.  One block.
__global__ void k_f_stats(FastDev g, StepStats *out) {
  __shared__ int smin[256], smax[256], snc[256];
  __shared__ double sres[256];
  int mn = 1 << 30, mx = 0, nc = 0;
  double rs = 0.0;
  for (int p = threadIdx.x; p < g.P; p += blockDim.x) {
    mn = min(mn, g.cycles[p]);
    mx = max(mx, g.cycles[p]);
    nc += (g.done[p] != 1);
    rs = fmax(rs, g.red[6 * p + 4]);
  }
  smin[threadIdx.x] = mn;
  smax[threadIdx.x] = mx;
  snc[threadIdx.x] = nc;
  sres[threadIdx.x] = rs;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      smin[threadIdx.x] = min(smin[threadIdx.x], smin[threadIdx.x + w]);
      smax[threadIdx.x] = max(smax[threadIdx.x], smax[threadIdx.x + w]);
      snc[threadIdx.x] += snc[threadIdx.x + w];
      sres[threadIdx.x] = fmax(sres[threadIdx.x], sres[threadIdx.x + w]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out->min_cycles = smin[0];
    out->max_cycles = smax[0];
    out->n_not_converged = snc[0];
    out->nprob = g.P;
    out->max_residual = sres[0];
  }
}

// Line Gauss-Seidel.  The 9-point operator couples each point to its eight
// neighbours; a line solve takes the three couplings along the line into a
// tridiagonal system and the others from current values.  Zebra order: the
// lines of one colour do not couple to each other, so all of them (for all
// problems) are solved in parallel, one thread per (line, problem).
//
// y-line at column i: c7 e(i,j-1) + c9 e(i,j) + c3 e(i,j+1) = r(i,j) - c1 e(i+1,j)
// - c5 e(i-1,j) [- c2, c4, c6, c8 diagonal terms].  Rows j = 1 and ny have
// c7 = 0 and c3 = 0 after MUDPACK's Neumann folding.  c' is kept in cp, d'
// overwrites e until the back substitution.
constexpr int kChunk = 8;
// zero_nbr: the neighbouring lines hold zero (the first sweep of a cycle
// from e = 0), so their terms are left out and their stale values unread
__device__ __forceinline__ void yline_solve(const LvF &L, int P, int p, int i, float kx2, bool orth,
                                            bool zero_nbr = false) {
  const int nx = L.nx, ny = L.ny;
  const size_t npt = (size_t)nx * ny;
  const size_t si = P, sj = (size_t)(nx + 2) * P;
  const float *cf = L.cof;
  float cprev = 0.f, dprev = 0.f;
  // forward elimination, kChunk rows at a time: every load of a chunk is
  // issued before the recurrence consumes it
  for (int j0 = 1; j0 <= ny; j0 += kChunk) {
    float dv[kChunk], av[kChunk], bv[kChunk], cv[kChunk];
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      const int j = j0 + u;
      if (j > ny) break;
      const size_t pt = (size_t)(j - 1) * nx + (i - 1);
      const float *ep = &L.e[((size_t)j * (nx + 2) + i) * P + p];
      float d = L.r[pt * P + p];
      if (!zero_nbr) {
        d = d - cf[pt] * ep[si] - cf[4 * npt + pt] * ep[-(long)si];
        if (orth == false)
          d = d - cf[npt + pt] * ep[si + sj] - cf[3 * npt + pt] * ep[sj - si] -
              cf[5 * npt + pt] * ep[-(long)(si + sj)] - cf[7 * npt + pt] * ep[si - sj];
      }
      dv[u] = d;
      av[u] = cf[6 * npt + pt];
      cv[u] = cf[2 * npt + pt];
      bv[u] = ((-kx2 * cf[10 * npt + pt]) - cf[8 * npt + pt]) + cf[9 * npt + pt];
    }
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      const int j = j0 + u;
      if (j > ny) break;
      const size_t pt = (size_t)(j - 1) * nx + (i - 1);
      const float m = 1.f / (bv[u] - av[u] * cprev);
      cprev = cv[u] * m;
      dprev = (dv[u] - av[u] * dprev) * m;
      L.cp[pt * P + p] = cprev;
      L.e[((size_t)j * (nx + 2) + i) * P + p] = dprev;
    }
  }
  // back substitution; periodic ghosts written together with their sources
  float x = 0.f;
  for (int j0 = ny; j0 >= 1; j0 -= kChunk) {
    float dv[kChunk], cv[kChunk];
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      const int j = j0 - u;
      if (j < 1) break;
      const size_t pt = (size_t)(j - 1) * nx + (i - 1);
      dv[u] = L.e[((size_t)j * (nx + 2) + i) * P + p];
      cv[u] = L.cp[pt * P + p];
    }
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      const int j = j0 - u;
      if (j < 1) break;
      x = dv[u] - cv[u] * x;
      L.e[((size_t)j * (nx + 2) + i) * P + p] = x;
      if (i == nx - 1) E(L, P, 0, j, p) = x;
      if (i == 2) E(L, P, nx + 1, j, p) = x;
    }
  }
}

// x-line at row j: c5 e(i-1,j) + c9 e(i,j) + c1 e(i+1,j) = r(i,j) - c3 e(i,j+1)
// - c7 e(i,j-1) [- diagonal terms].  The periodic wrap couplings (i = 1 to
// the ghost e(0) = e(nx-1), i = nx to the ghost e(nx+1) = e(2)) are taken
// from the ghosts' current values, so the line system stays tridiagonal.
__device__ __forceinline__ void xline_solve(const LvF &L, int P, int p, int j, float kx2, bool orth) {
  const int nx = L.nx, ny = L.ny;
  const size_t npt = (size_t)nx * ny;
  const size_t si = P, sj = (size_t)(nx + 2) * P;
  const float *cf = L.cof;
  float *erow = &L.e[(size_t)j * (nx + 2) * P + p];  // erow[i * P] = e(i, j)
  float *cprow = &L.cp[(size_t)(j - 1) * nx * P + p];  // cprow[(i-1) * P]
  const size_t rb = (size_t)(j - 1) * nx;
  const float g0 = erow[0], g1 = erow[(size_t)(nx + 1) * si];
  float cprev = 0.f, dprev = 0.f;
  for (int i0 = 1; i0 <= nx; i0 += kChunk) {
    float dv[kChunk], av[kChunk], bv[kChunk], cv[kChunk];
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      const int i = i0 + u;
      if (i > nx) break;
      const size_t pt = rb + (i - 1);
      const float *ep = erow + (size_t)i * si;
      float d = L.r[pt * P + p] - cf[2 * npt + pt] * ep[sj] - cf[6 * npt + pt] * ep[-(long)sj];
      if (orth == false)
        d = d - cf[npt + pt] * ep[si + sj] - cf[3 * npt + pt] * ep[sj - si] - cf[5 * npt + pt] * ep[-(long)(si + sj)] -
            cf[7 * npt + pt] * ep[si - sj];
      float a = cf[4 * npt + pt], c = cf[pt];
      if (i == 1) { d -= a * g0; a = 0.f; }
      if (i == nx) { d -= c * g1; c = 0.f; }
      dv[u] = d;
      av[u] = a;
      cv[u] = c;
      bv[u] = ((-kx2 * cf[10 * npt + pt]) - cf[8 * npt + pt]) + cf[9 * npt + pt];
    }
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      const int i = i0 + u;
      if (i > nx) break;
      const float m = 1.f / (bv[u] - av[u] * cprev);
      cprev = cv[u] * m;
      dprev = (dv[u] - av[u] * dprev) * m;
      cprow[(size_t)(i - 1) * si] = cprev;
      erow[(size_t)i * si] = dprev;
    }
  }
  float x = 0.f;
  for (int i0 = nx; i0 >= 1; i0 -= kChunk) {
    float dv[kChunk], cv[kChunk];
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      const int i = i0 - u;
      if (i < 1) break;
      dv[u] = erow[(size_t)i * si];
      cv[u] = cprow[(size_t)(i - 1) * si];
    }
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      const int i = i0 - u;
      if (i < 1) break;
      x = dv[u] - cv[u] * x;
      erow[(size_t)i * si] = x;
      if (i == nx - 1) erow[0] = x;
      if (i == 2) erow[(size_t)(nx + 1) * si] = x;
    }
  }
}

// y-lines i = i0, i0+istep, ... (ncol of them), all problems
__global__ void __launch_bounds__(64) k_f_yline(FastDev g, int level, int i0, int istep, int ncol, int zero_nbr) {
  if (*g.alldone) return;
  const LvF L = g.lv[level - 1];
  const int P = g.P;
  const long n = (long)ncol * P;
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    const int p = (int)(t % P);
    if (g.done[p]) continue;
    yline_solve(L, P, p, i0 + istep * (int)(t / P), (float)g.kx2[p], g.orth != 0, zero_nbr != 0);
  }
}

// x-lines j = j0, j0+2, ... (nrow of them), all problems
__global__ void __launch_bounds__(64) k_f_xline(FastDev g, int level, int j0, int nrow) {
  if (*g.alldone) return;
  const LvF L = g.lv[level - 1];
  const int P = g.P;
  const long n = (long)nrow * P;
  for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
    const int p = (int)(t % P);
    if (g.done[p]) continue;
    xline_solve(L, P, p, j0 + 2 * (int)(t / P), (float)g.kx2[p], g.orth != 0);
  }
}

// Partitioned line solve: one block per (line, LANES problems), lanes over
// the problems (coalesced, the layout is problem fastest), threadIdx.y over K
// segments of the line.  The line's n rows are K segments of <= SEG interior
// rows separated by K-1 separator rows.  Each thread row eliminates its
// segment in registers, expressing every row as x = delta + gamma X0 -
// beta x(next) with X0, X1 the separators before and after it; the first and
// last rows in terms of (X0, X1) give a tridiagonal system for the
// separators, solved from shared memory by parallel cyclic reduction (one
// thread row per separator, log2(K) combine steps); then every segment
// back-substitutes.
// XL: x-line (along i, the periodic wrap couplings taken from the ghosts'
// current values); else y-line (along j).
enum { SH_A, SH_B, SH_C, SH_D, SH_YF, SH_VF, SH_WF, SH_YL, SH_VL, SH_WL, SH_S, SH_N };
// 4-row segments are capped at 48 registers, so that two or three blocks
// share an SM (their per-thread arrays are half as large)
template <bool XL, bool ORTH, int LANES, int SEG, int REGS = (SEG == 4 ? 48 : 64)>
// zero_e: the first sweep of a cycle from e = 0 (y-lines only): the
// neighbouring lines' terms are left out and their stale values unread.
__global__ void __launch_bounds__(1024) __maxnreg__(REGS) k_f_pline(FastDev g, int level, int l0, int lstep, int mb, int me, int zero_e) {
  constexpr int kSegMax = SEG;
  if (*g.alldone) return;
  extern __shared__ float sh[];
  const int K = blockDim.y;
  auto S = [&](int arr, int seg) -> float & { return sh[(arr * K + seg) * LANES + threadIdx.x]; };
  const LvF L = g.lv[level - 1];
  const int P = g.P;
  const int nx = L.nx, ny = L.ny;
  const int s = threadIdx.y;
  const int p = blockIdx.y * LANES + threadIdx.x;
  const bool act = (p < P) && !g.done[p];
  if (!__syncthreads_or(act)) return;  // every problem of the block converged
  const int pp = act ? p : 0;
  const int line = l0 + lstep * (int)blockIdx.x;
  const int m = mb + (s < me ? 1 : 0);
  const int lo = 1 + s * (mb + 1) + min(s, me);
  // 32-bit offsets: the host checks that (nx+2)(ny+2)P and 11 nx ny fit
  const unsigned npt = (unsigned)nx * (unsigned)ny;
  const unsigned si = (unsigned)P, sj = (unsigned)(nx + 2) * (unsigned)P;
  const float kx2 = (float)g.kx2[pp];
  const float *cf = L.cof;
  // row k of the line: a x(k-1) + b x(k) + c x(k+1) = d
  auto row = [&](int k, float &a, float &b, float &c, float &d) {
    const int i = XL ? k : line, j = XL ? line : k;
    const unsigned pt = (unsigned)((j - 1) * nx + (i - 1));
    const float *ep = L.e + ((unsigned)(j * (nx + 2) + i) * si + (unsigned)pp);
    const float *cp = cf + pt;
    b = ((-kx2 * cp[10 * npt]) - cp[8 * npt]) + cp[9 * npt];
    float dd = L.r[pt * si + (unsigned)pp];
    if (XL) {
      a = cp[4 * npt];
      c = cp[0];
      dd = dd - cp[2 * npt] * ep[sj] - cp[6 * npt] * *(ep - sj);
    } else {
      a = cp[6 * npt];
      c = cp[2 * npt];
      if (!zero_e) dd = dd - cp[0] * ep[si] - cp[4 * npt] * *(ep - si);
    }
    if (!ORTH && !zero_e)
      dd = dd - cp[npt] * ep[si + sj] - cp[3 * npt] * ep[sj - si] - cp[5 * npt] * *(ep - (si + sj)) -
           cp[7 * npt] * *(ep - (sj - si));
    d = dd;
  };
  auto store = [&](int k, float x) {
    const int i = XL ? k : line, j = XL ? line : k;
    float *erow = L.e + (unsigned)(j * (nx + 2)) * si + (unsigned)p;
    erow[(unsigned)i * si] = x;
    if (i == nx - 1) erow[0] = x;
    if (i == 2) erow[(unsigned)(nx + 1) * si] = x;
  };
  // phase 1: every load of the segment (rows past its end repeat its last
  // row, so all addresses are valid and no load waits on arithmetic)
  float av[kSegMax], bv[kSegMax], cv[kSegMax], dv[kSegMax];
#pragma unroll
  for (int u = 0; u < kSegMax; ++u) row(lo + min(u, m - 1), av[u], bv[u], cv[u], dv[u]);
  if (XL) {
    // the periodic wrap of an x-line: i = 1 couples to the ghost e(0) =
    // e(nx-1), i = nx to e(nx+1) = e(2), both taken from current values
    const float *erow = L.e + (unsigned)(line * (nx + 2)) * si + (unsigned)pp;
    if (s == 0) {
      dv[0] -= av[0] * erow[0];
      av[0] = 0.f;
    }
    if (s == K - 1) {
      const float gh = erow[(unsigned)(nx + 1) * si];
#pragma unroll
      for (int u = 0; u < kSegMax; ++u) {
        const bool hit = (u == m - 1);
        dv[u] = hit ? dv[u] - cv[u] * gh : dv[u];
        cv[u] = hit ? 0.f : cv[u];
      }
    }
  }
  // phase 2: elimination in place: cv <- beta, dv <- delta, av <- gamma, where
  // row u of the segment is x = delta + gamma X0 - beta x(next)
  float yl = 0.f, vl = 0.f, wl = 0.f;
  {
    float bprev = 0.f, dprev = 0.f, gprev = 1.f;
#pragma unroll
    for (int u = 0; u < kSegMax; ++u) {
      const float inv = __fdividef(1.f, bv[u] - av[u] * bprev);
      bprev = cv[u] * inv;
      dprev = (dv[u] - av[u] * dprev) * inv;
      gprev = -av[u] * gprev * inv;
      cv[u] = bprev;
      dv[u] = dprev;
      av[u] = gprev;
      const bool last = (u == m - 1);
      yl = last ? dprev : yl;
      vl = last ? gprev : vl;
      wl = last ? -bprev : wl;
    }
  }
  float yf = yl, vf = vl, wf = wl;
#pragma unroll
  for (int u = kSegMax - 2; u >= 0; --u)
    if (u < m - 1) {
      yf = dv[u] - cv[u] * yf;
      vf = av[u] - cv[u] * vf;
      wf = -cv[u] * wf;
    }
  S(SH_YF, s) = yf; S(SH_VF, s) = vf; S(SH_WF, s) = wf;
  S(SH_YL, s) = yl; S(SH_VL, s) = vl; S(SH_WL, s) = wl;
  if (s < K - 1) {
    float a, b, c, d;
    row(lo + m, a, b, c, d);
    S(SH_A, s) = a; S(SH_B, s) = b; S(SH_C, s) = c; S(SH_D, s) = d;
  }
  __syncthreads();
  // the K-1 separator unknowns, A S(t-1) + B S(t) + C S(t+1) = D, by
  // parallel cyclic reduction: thread row t owns separator t; after the
  // steps of stride 1, 2, 4, ... each row couples to nothing and S(t) = D/B
  const int nsep = K - 1;
  float eA = 0.f, eB = 1.f, eC = 0.f, eD = 0.f;
  if (s < nsep) {
    const float a = S(SH_A, s), c = S(SH_C, s);
    eA = (s > 0) ? a * S(SH_VL, s) : 0.f;
    eB = S(SH_B, s) + a * S(SH_WL, s) + c * S(SH_VF, s + 1);
    eC = (s < nsep - 1) ? c * S(SH_WF, s + 1) : 0.f;
    eD = S(SH_D, s) - a * S(SH_YL, s) - c * S(SH_YF, s + 1);
  }
  for (int d = 1; d < nsep; d <<= 1) {
    __syncthreads();
    if (s < nsep) {
      S(SH_A, s) = eA;
      S(SH_B, s) = eB;
      S(SH_C, s) = eC;
      S(SH_D, s) = eD;
    }
    __syncthreads();
    if (s < nsep) {
      float nA = 0.f, nC = 0.f, nB = eB, nD = eD;
      if (s - d >= 0) {
        const float al = __fdividef(eA, S(SH_B, s - d));
        nA = -al * S(SH_A, s - d);
        nB -= al * S(SH_C, s - d);
        nD -= al * S(SH_D, s - d);
      }
      if (s + d < nsep) {
        const float ga = __fdividef(eC, S(SH_B, s + d));
        nC = -ga * S(SH_C, s + d);
        nB -= ga * S(SH_A, s + d);
        nD -= ga * S(SH_D, s + d);
      }
      eA = nA;
      eB = nB;
      eC = nC;
      eD = nD;
    }
  }
  if (s < nsep) S(SH_S, s) = __fdividef(eD, eB);
  __syncthreads();
  if (!act) return;
  const float X0 = (s > 0) ? S(SH_S, s - 1) : 0.f;
  const float X1 = (s < K - 1) ? S(SH_S, s) : 0.f;
  float x = 0.f;
#pragma unroll
  for (int u = kSegMax - 1; u >= 0; --u)
    if (u < m) {
      x = dv[u] + av[u] * X0 - cv[u] * ((u == m - 1) ? X1 : x);
      store(lo + u, x);
    }
  if (s < K - 1) store(lo + m, X1);
}

struct LinePhase {
  int i0, istep, ncol;
};
// y-line colour col (1, 2) of a level with nx columns as one or two ordered
// phases.  With nx odd the colours are odd and even i.  With nx even (only
// possible on the coarsest level) the periodic wrap couples i = 1 to
// i = nx-1 and i = nx to i = 2, so i = 1 and i = nx go in phases of their own.
__host__ __device__ inline int line_phases(int nx, int col, LinePhase *ph) {
  if (nx % 2 == 1) {
    ph[0] = (col == 1) ? LinePhase{1, 2, (nx + 1) / 2} : LinePhase{2, 2, (nx - 1) / 2};
    return 1;
  }
  if (col == 1) {
    ph[0] = LinePhase{3, 2, nx / 2 - 1};
    ph[1] = LinePhase{1, 1, 1};
  } else {
    ph[0] = LinePhase{2, 2, nx / 2 - 1};
    ph[1] = LinePhase{nx, 1, 1};
  }
  return 2;
}

// The coarsest level: `sweeps` alternating-direction sweeps, one thread per
// problem (the level has a few tens of points), in the same order as the
// per-line kernels use.
__global__ void k_f_coarsest(FastDev g, int sweeps) {
  if (*g.alldone) return;
  const LvF L = g.lv[0];
  const int P = g.P;
  const bool orth = g.orth != 0;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
    if (g.done[p]) continue;
    const float kx2 = (float)g.kx2[p];
    for (int sw = 0; sw < sweeps; ++sw) {
      for (int col = 1; col <= 2; ++col) {
        LinePhase ph[2];
        const int nph = line_phases(L.nx, col, ph);
        for (int q = 0; q < nph; ++q)
          for (int c = 0; c < ph[q].ncol; ++c) yline_solve(L, P, p, ph[q].i0 + ph[q].istep * c, kx2, orth);
      }
      for (int col = 1; col <= 2; ++col)
        for (int j = col; j <= L.ny; j += 2) xline_solve(L, P, p, j, kx2, orth);
    }
    if (kx2 == 0.f) {
      // singular: keep the correction at zero mean, ghosts included
      float m = 0.f;
      for (int j = 1; j <= L.ny; ++j)
        for (int i = 1; i <= L.nx; ++i) m += E(L, P, i, j, p);
      m = m / (float)(L.nx * L.ny);
      for (int j = 1; j <= L.ny; ++j)
        for (int i = 0; i <= L.nx + 1; ++i) E(L, P, i, j, p) -= m;
    }
  }
}

// The elementwise multigrid kernels below use one block per grid row (or
// coarse row) and 32 problems: lanes over the problems (coalesced, the
// layout is problem fastest), the block's warps striding along the row.  No
// index needs a division.
constexpr int kRowWarps = 8;

// The level operations below act on one point of one problem: arrays with
// the problem index fastest (stride P, problem p), as the batched kernels
// keep them in global memory, or P = 1, p = 0 for one problem's arrays in
// shared memory (k_f_vtail).  One definition serves both, so a level gives
// the same numbers in either.

// full weighting (res2, mudcom.f:120-257) of the fine residual in scr to the
// coarse rhs at (ic, jc), and e_coarse = 0 there (ghosts included: ic =
// 0..ncx+1, jc = 0..ncy+1)
__device__ __forceinline__ void f_restrict_at(const float *__restrict__ scr, float *__restrict__ ce,
                                              float *__restrict__ cr, int nx, int ny, int ncx, int ncy, int P, int p,
                                              int ic, int jc) {
  const int ix = (ncx == nx) ? 0 : 1, jy = (ncy == ny) ? 0 : 1;
  ce[((size_t)jc * (ncx + 2) + ic) * P + p] = 0.f;
  if (ic < 1 || ic > ncx || jc < 1 || jc > ncy) return;
  const int i = ic + ix * (ic - 1), j = jc + jy * (jc - 1);
  int im1 = i - 1, ip1 = i + 1, jm1 = j - 1, jp1 = j + 1;
  if (ic == 1 || ic == ncx) {
    im1 = max(i - 1, 2);
    ip1 = min(i + 1, nx - 1);
    if (i == 1) im1 = nx - 1;
    if (i == nx) ip1 = 2;
  }
  if (jc == 1 || jc == ncy) {
    jm1 = max(j - 1, 2);
    jp1 = min(j + 1, ny - 1);
  }
  auto R = [&](int a, int b) { return scr[((size_t)b * (nx + 2) + a) * P + p]; };
  cr[((size_t)(jc - 1) * ncx + (ic - 1)) * P + p] =
      (R(im1, jm1) + R(ip1, jm1) + R(im1, jp1) + R(ip1, jp1) + 2.f * (R(im1, j) + R(ip1, j) + R(i, jm1) + R(i, jp1)) +
       4.f * R(i, j)) * .0625f;
}

// residual r - A e of the correction equation at one point (FP32): q0 holds
// the couplings (i+1, j+1, i-1, j-1), q2 the diagonal ones, c9 the centre
__device__ __forceinline__ float f_resid_val(float4 q0, float4 q2, float c9, const float *ep, size_t si, size_t sj,
                                             float rr, bool orth) {
  float s = q0.x * ep[si] + q0.y * ep[sj] + q0.z * ep[-(long)si] + q0.w * ep[-(long)sj];
  if (!orth) s += q2.x * ep[si + sj] + q2.y * ep[sj - si] + q2.z * ep[-(long)(si + sj)] + q2.w * ep[si - sj];
  s += c9 * ep[0];
  return rr - s;
}
// the same from the packed coefficients, at point (i, j) of a level: two or
// three vector loads for seven or eleven scalar ones
__device__ __forceinline__ void f_resid_at4(const float4 *__restrict__ cf4, const float *__restrict__ ee,
                                            const float *__restrict__ rr, float *__restrict__ scr, int nx, int P,
                                            int p, int i, int j, float kx2, bool orth) {
  const size_t si = P, sj = (size_t)(nx + 2) * P;
  const size_t pt = (size_t)(j - 1) * nx + (i - 1), q = ((size_t)j * (nx + 2) + i) * P + p;
  const float4 q0 = cf4[3 * pt], q1 = cf4[3 * pt + 1];
  const float4 q2 = orth ? make_float4(0.f, 0.f, 0.f, 0.f) : cf4[3 * pt + 2];
  const float c9 = ((-kx2 * q1.z) - q1.x) + q1.y;
  scr[q] = f_resid_val(q0, q2, c9, ee + q, si, sj, rr[pt * P + p], orth);
}

// residual of the correction equation at a level (FP32) into the scratch
__global__ void __launch_bounds__(32 * kRowWarps) k_f_resid32(FastDev g, int level) {
  if (*g.alldone) return;
  const LvF L = g.lv[level - 1];
  const int P = g.P;
  const int p = blockIdx.x * 32 + threadIdx.x;
  if (p >= P || g.done[p]) return;
  const int nx = L.nx, j = 1 + (int)blockIdx.y;
  const float kx2 = (float)g.kx2[p];
  const bool orth = g.orth != 0;
#pragma unroll 4
  for (int i = 1 + (int)threadIdx.y; i <= nx; i += kRowWarps)
    f_resid_at4(L.cf4, L.e, L.r, g.scr, nx, P, p, i, j, kx2, orth);
}

// full weighting (res2, mudcom.f:120-257) to the coarse rhs; e_coarse = 0
// (block row jc = 0..ncy+1, ghosts included)
__global__ void __launch_bounds__(32 * kRowWarps) k_f_restrict(FastDev g, int level) {
  if (*g.alldone) return;
  const LvF F = g.lv[level - 1], C = g.lv[level - 2];
  const int P = g.P;
  const int p = blockIdx.x * 32 + threadIdx.x;
  if (p >= P || g.done[p]) return;
  const int jc = (int)blockIdx.y;
#pragma unroll 4
  for (int ic = (int)threadIdx.y; ic <= C.nx + 1; ic += kRowWarps)
    f_restrict_at(g.scr, C.e, C.r, F.nx, F.ny, C.nx, C.ny, P, p, ic, jc);
}

// cubic/linear prolongation (prolon1/prolon2, mudcom.f:261-499) of the
// coarse correction, stage 1: rows given directly by prolon1, into scratch
template <typename F>
__device__ __forceinline__ float prolon1f(int i, int ncx, int nx, bool cubic, F p) {
  if (ncx == nx) return p(i);
  if (!cubic) {
    if (i & 1) return p((i + 1) / 2);
    return 0.5f * (p(i / 2) + p(i / 2 + 1));
  }
  auto q = [&](int ii) { return p((ii + 1) / 2); };
  if (i & 1) return q(i);
  if (i >= 4 && i <= nx - 3) return (-q(i - 3) + 9.f * (q(i - 1) + q(i + 1)) - q(i + 3)) * .0625f;
  if (i == 2) return (-q(nx - 2) + 9.f * (q(1) + q(3)) - q(5)) * .0625f;
  return (-q(nx - 4) + 9.f * (q(nx - 2) + q(nx)) - q(3)) * .0625f;
}

// fine row j = 2 rr + 1 (y coarsened) or rr + 1, point i: stage 1 into scr
__device__ __forceinline__ void f_prolong_x_at(const float *__restrict__ ce, float *__restrict__ scr, int nx, int ny,
                                               int ncx, int ncy, int P, int p, int i, int rr) {
  const bool ycoarse = ncy < ny;
  const bool cubic = ncx >= 4;
  const int j = ycoarse ? 2 * rr + 1 : rr + 1;
  const int jc = ycoarse ? j / 2 + 1 : j;
  auto pc = [&](int ic) { return ce[((size_t)jc * (ncx + 2) + ic) * P + p]; };
  scr[((size_t)j * (nx + 2) + i) * P + p] = prolon1f(i, ncx, nx, cubic, pc);
}

// stage 2 at fine point (i, j): the rows between (cubic or linear in y), then
// e += correction, with the periodic ghosts written together with their
// sources
__device__ __forceinline__ void f_prolong_y_at(const float *__restrict__ scr, float *__restrict__ ef, int nx, int ny,
                                               int ncy, int P, int p, int i, int j) {
  const bool ycoarse = ncy < ny;
  const bool cubic = ncy >= 4;
  const size_t rowj = (size_t)j * (nx + 2) * P + p;
  auto Q = [&](int jj) { return scr[((size_t)jj * (nx + 2) + i) * P + p]; };
  float v;
  if (ycoarse && !(j & 1)) {
    if (!cubic) v = 0.5f * (Q(j - 1) + Q(j + 1));
    else if (j >= 4 && j <= ny - 3) v = (-Q(j - 3) + 9.f * (Q(j - 1) + Q(j + 1)) - Q(j + 3)) * .0625f;
    else if (j == 2) v = (5.f * Q(1) + 15.f * Q(3) - 5.f * Q(5) + Q(7)) * .0625f;
    else v = (5.f * Q(ny) + 15.f * Q(ny - 2) - 5.f * Q(ny - 4) + Q(ny - 6)) * .0625f;
  } else {
    v = Q(j);
  }
  const float ne = ef[rowj + (size_t)i * P] + v;
  ef[rowj + (size_t)i * P] = ne;
  if (i == nx - 1) ef[rowj] = ne;
  if (i == 2) ef[rowj + (size_t)(nx + 1) * P] = ne;
}

// Both stages in one pass: e += the prolonged coarse correction.  What bounds it
// is e's read and write; with stage 1 in a launch of its own, its rows were
// written and read as well.  A thread has one fine column and kProRows
// coarse rows of it: their stage-1 values and those of the rows around, the e
// they go to, then the sums, the same as above one by one.  All loads go out
// together.  Block (32 problems, kProRows coarse rows, every gridDim.z-th
// eight columns).  All transfers of a step: 512 x 385 x 257 8.56 -> 6.93 ms, 256 x
// 193 x 129 2.15 -> 1.68, 128 x 129 x 97 0.94 -> 0.65.  Four rows a thread form
// fewer stage-1 values twice, but hold 51 loads at a time for 27 and leave the
// SMs fewer warps: 7.38, 1.75 and 0.68.
constexpr int kProRows = 2;
__global__ void __launch_bounds__(32 * kRowWarps) k_f_prolong(FastDev g, int level) {
  if (*g.alldone) return;
  const LvF F = g.lv[level - 1], C = g.lv[level - 2];
  const int P = g.P;
  const int p = blockIdx.x * 32 + threadIdx.x;
  if (p >= P || g.done[p]) return;
  const int nx = F.nx, ny = F.ny, ncx = C.nx, ncy = C.ny;
  const int r0 = (int)blockIdx.y * kProRows;  // coarse rows r0 + 1 ..
  constexpr int N = kProRows + 3;
  static_assert(N >= 5, "the first row between takes four stage-1 rows");
  const bool ycoarse = ncy < ny, cubic = ncy >= 4;
  const float *ce = C.e + p;
  float *ef = F.e + p;
  for (int i = 1 + (int)threadIdx.y + kRowWarps * (int)blockIdx.z; i <= nx; i += kRowWarps * (int)gridDim.z) {
    // stage 1's points: one, two or four of a coarse row
    int n = 1, x0 = i, x1 = 0, x2 = 0, x3 = 0;
    if (ncx != nx) {
      x0 = (i + 1) / 2;
      if (!(i & 1) && ncx < 4) {
        n = 2, x0 = i / 2, x1 = i / 2 + 1;
      } else if (!(i & 1)) {
        n = 4;
        const int a = (i == 2) ? nx - 2 : (i == nx - 1) ? nx - 4 : i - 3, d = (i == nx - 1) ? 3 : i + 3;
        x0 = (a + 1) / 2, x1 = i / 2, x2 = i / 2 + 1, x3 = (d + 1) / 2;
      }
    }
    auto row = [&](int r) { return ce + (size_t)(min(max(r, 0), ncy - 1) + 1) * (ncx + 2) * P; };
    auto cub = [](float a, float b, float c, float d) { return (-a + 9.f * (b + c) - d) * .0625f; };
    float e[2 * kProRows], w[N];
    auto fine = [&](int t) { return ycoarse ? 2 * r0 + 1 + t : r0 + 1 + t; };
#pragma unroll
    for (int t = 0; t < 2 * kProRows; ++t)
      if ((ycoarse || t < kProRows) && fine(t) <= ny) e[t] = ef[((size_t)fine(t) * (nx + 2) + i) * P];
    auto stage1 = [&](int r) {
      const float *q = row(r);
      if (n == 1) return q[(size_t)x0 * P];
      if (n == 2) return 0.5f * (q[(size_t)x0 * P] + q[(size_t)x1 * P]);
      return cub(q[(size_t)x0 * P], q[(size_t)x1 * P], q[(size_t)x2 * P], q[(size_t)x3 * P]);
    };
    if (n == 4) {
      float q[N][4];
#pragma unroll
      for (int t = 0; t < N; ++t) {
        const float *qr = row(r0 - 1 + t);
        q[t][0] = qr[(size_t)x0 * P], q[t][1] = qr[(size_t)x1 * P], q[t][2] = qr[(size_t)x2 * P], q[t][3] = qr[(size_t)x3 * P];
      }
#pragma unroll
      for (int t = 0; t < N; ++t) w[t] = cub(q[t][0], q[t][1], q[t][2], q[t][3]);
    } else {
#pragma unroll
      for (int t = 0; t < N; ++t) w[t] = stage1(r0 - 1 + t);
    }
    auto put = [&](int t, float v) {
      float *er = ef + (size_t)fine(t) * (nx + 2) * P;
      const float ne = e[t] + v;
      er[(size_t)i * P] = ne;
      if (i == nx - 1) er[0] = ne;
      if (i == 2) er[(size_t)(nx + 1) * P] = ne;
    };
#pragma unroll
    for (int t = 0; t < kProRows; ++t) {
      const int r = r0 + t;
      if (r >= ncy) break;
      if (!ycoarse) {
        put(t, w[t + 1]);
        continue;
      }
      put(2 * t, w[t + 1]);
      if (r == ncy - 1) break;
      // fine row 2 r + 2, between coarse rows r + 1 and r + 2
      float v;
      if (!cubic) v = 0.5f * (w[t + 1] + w[t + 2]);
      else if (r == 0) v = (5.f * w[1] + 15.f * w[2] - 5.f * w[3] + w[4]) * .0625f;
      else if (r == ncy - 2) v = (5.f * w[t + 2] + 15.f * w[t + 1] - 5.f * w[t] + stage1(r - 2)) * .0625f;
      else v = cub(w[t], w[t + 1], w[t + 2], w[t + 3]);
      put(2 * t + 1, v);
    }
  }
}

// The coarse end of a V(1,1) cycle in one launch: levels ltop, ltop-1, ..., 1
// of one problem per block, with the level arrays in shared memory and the
// (problem-independent) coefficients read through L1.  Each level down: the
// pre-smoothing sweep, the residual, the restriction; the coarsest level's
// `sweeps` alternating sweeps (and, for kx^2 = 0, its zero-mean shift); each
// level up: the prolongation and the post-smoothing sweep -- the operations
// and order of the per-level launches, with every line solved by one thread
// (lines of one colour are independent).  On the coarse levels a per-level
// launch does a few microseconds of work behind a launch and a grid-wide
// dependency; here the levels follow each other behind block barriers.
//
// A line's Thomas factors (m = 1 / (b - a c'), c' = c m, per row) depend on
// the problem's kx^2 and the level coefficients only, so k_f_tail_factors
// computes them once per solve; a sweep then runs the recurrences
// d' = (d - a d') m and x = d' - c' x, with no division on the chain.
// In: the restricted rhs of level ltop (global); out: its correction e,
// ghosts included (global).
//
// Levels lth+1..ltop, above the Thomas ones, solve their lines as k_f_pline
// does, the same segments, separators and operations on the block's shared
// arrays (part_lines), so a level gives the same numbers in either; with
// ltop = ngrid a whole cycle is one launch.
// What bounds it: the serial chain of phases (four colours a sweep, two sweeps
// a level), each a few hundred cycles of dependent arithmetic behind a block
// barrier; a problem's arrays never leave its SM.  Measured, a step:
// 64 x 65 x 65 (a cycle in the block: 163,000 cycles) 4.2 -> 2.6 ms,
// 128 x 129 x 97 sheared 15.4 -> 11.7 ms, 256 x 193 x 129 with LES 23.5 ->
// 22.0 ms.
constexpr int kTailThreads = 128;
constexpr int kTailMax = 12;
constexpr int kTailMost = 512;  // threads of a block
struct TailPlan {
  int ltop, lth, sweeps;
  int nfac;  // factor floats per problem: (c', m) of the y-lines and of the x-lines, every level
  int fac0, scr, total;  // shared-memory offsets (floats): factor block, transfer scratch; total floats
  int nx[kTailMax], ny[kTailMax];
  int e[kTailMax], r[kTailMax];  // shared-memory offsets of e and r of level l + 1
  int f[kTailMax];               // offset of level l + 1's y-line factors in the factor block (x-lines follow)
  int c[kTailMax];               // offset of its coefficients: Thomas levels the lines' lower diagonals (y, x);
                                 // others the planes c1 c3 c5 c7 b (and c2 c4 c6 c8 unless orthogonal)
};

// Segments of a line of n rows in part_lines (k_f_pline's with 8-row segments),
// and the floats of its exchange arrays for a colour's lines of both directions,
// in a block of at most kTailMost threads
constexpr int kPartSeg = 8;
__host__ __device__ inline int part_segments(int n) {
  const int k = (n + kPartSeg + 1) / (kPartSeg + 1);
  return k > 1 ? k : 1;
}
int part_scratch(int nx, int ny) {
  auto lines = [](int n, int colour) { return SH_N * part_segments(n) * std::min(kTailMost / part_segments(n), colour); };
  return std::max(lines(nx, (ny + 1) / 2), lines(ny, (nx + 1) / 2));
}

TailPlan make_tail_plan(const MgPlan &PL, int ltop, int lth) {
  TailPlan t{};
  t.ltop = ltop;
  t.lth = lth;
  t.sweeps = std::max(8, (PL.lv[0].nx + PL.lv[0].ny) / 2);
  int off = 0, fo = 0;
  for (int l = 0; l < ltop; ++l) {
    const int nx = PL.lv[l].nx, ny = PL.lv[l].ny;
    t.nx[l] = nx;
    t.ny[l] = ny;
    t.e[l] = off;
    off += (nx + 2) * (ny + 2);
    t.r[l] = off;
    off += nx * ny;
    t.f[l] = fo;
    if (l < lth) fo += 4 * nx * ny;
  }
  // the transfers' scratch, and part_lines' (the smaller one for every shape
  // with sides of 6 to 700 points, by 11 floats at 7 x 9)
  t.scr = off;
  int scr = (t.nx[ltop - 1] + 2) * (t.ny[ltop - 1] + 2);
  for (int l = lth; l < ltop; ++l) scr = std::max(scr, part_scratch(t.nx[l], t.ny[l]));
  off += scr;
  off = (off + 3) & ~3;  // the factor block is copied as float4
  t.fac0 = off;
  t.nfac = fo;
  off += fo;
  for (int l = 0; l < ltop; ++l) {
    t.c[l] = off;
    off += ((l < lth) ? 2 : PL.orth ? 5 : 9) * t.nx[l] * t.ny[l];
    off = (off + 3) & ~3;
  }
  // tail_chain loads whole chunks of a Thomas line's rows
  t.total = off + kChunk * (t.nx[std::max(lth, 1) - 1] + 2);
  return t;
}

// one level of one problem in shared memory (P = 1, p = 0)
struct TailLv {
  int nx, ny;
  float *e, *r;
  const float2 *fy, *fx;  // (c', m) per point, point (i, j) at (j-1) nx + (i-1)
  const float4 *cf4;      // packed coefficients (MgLevelF::cf4), global
  float *c;               // staged coefficients (TailPlan::c)
};
__device__ __forceinline__ TailLv tail_level_at(const TailPlan &t, const FastDev &g, float *sm, int l) {
  TailLv L;
  L.nx = t.nx[l];
  L.ny = t.ny[l];
  L.e = sm + t.e[l];
  L.r = sm + t.r[l];
  L.fy = reinterpret_cast<const float2 *>(sm + t.fac0 + t.f[l]);
  L.fx = L.fy + (size_t)L.nx * L.ny;
  L.cf4 = g.lv[l].cf4;
  L.c = sm + t.c[l];
  return L;
}

// A Thomas line's two recurrences by one thread, the rows of yline_solve and
// xline_solve: the n right-hand sides at b[k st], replaced by the solution.
// kChunk rows' values are loaded ahead of the recurrence (past the line's end
// too: TailPlan pads the block's arrays for that).  gh, gh2: offsets of the
// ghosts a y-line feeds (0: none).
__device__ __forceinline__ void tail_chain(float *b, int st, const float *a, const float2 *f, int cst, int n, int gh,
                                           int gh2) {
  float prev = 0.f;
  for (int k0 = 0; k0 < n; k0 += kChunk) {
    float dv[kChunk], av[kChunk], mv[kChunk];
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      dv[u] = b[u * st];
      av[u] = a[u * cst];
      mv[u] = f[u * cst].y;
    }
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      prev = (k0 + u < n) ? (dv[u] - av[u] * prev) * mv[u] : prev;
      dv[u] = prev;
    }
#pragma unroll
    for (int u = 0; u < kChunk; ++u)
      if (k0 + u < n) b[u * st] = dv[u];
    b += kChunk * st;
    a += kChunk * cst;
    f += kChunk * cst;
  }
  float x = 0.f;
  for (int k0 = (n - 1) / kChunk * kChunk; k0 >= 0; k0 -= kChunk) {
    float dv[kChunk], cv[kChunk];
    b -= kChunk * st;
    f -= kChunk * cst;
#pragma unroll
    for (int u = 0; u < kChunk; ++u) {
      dv[u] = b[u * st];
      cv[u] = f[u * cst].x;
    }
#pragma unroll
    for (int u = kChunk - 1; u >= 0; --u) {
      x = (k0 + u < n) ? dv[u] - cv[u] * x : x;
      dv[u] = x;
    }
#pragma unroll
    for (int u = 0; u < kChunk; ++u)
      if (k0 + u < n) b[u * st] = dv[u];
    if (gh | gh2)
#pragma unroll
      for (int u = 0; u < kChunk; ++u)
        if (k0 + u < n) {
          if (gh) b[u * st + gh] = dv[u];
          if (gh2) b[u * st + gh2] = dv[u];
        }
  }
}

// `sweeps` alternating-direction zebra sweeps of a Thomas level by the first
// nt threads of the block (a multiple of 32; bar: the named barrier they
// share), in the order of the per-level relax.  A colour goes in two parts:
// every point's right-hand side, one thread a point, into the point's own
// place in e (a line reads only the other colour's lines), then each line's
// recurrences.  A thread keeps its point's coefficients and right-hand side
// over all phases (levels of more points than threads load them again).
__device__ __forceinline__ void tail_relax(const TailLv &L, int nt, int sweeps, bool orth, bool post) {
  const int nx = L.nx, ny = L.ny, sj = nx + 2, npt = nx * ny, tid = threadIdx.x;
  if (tid >= nt) return;
  auto sync = [&]() { asm volatile("bar.sync 1, %0;\n" ::"r"(nt) : "memory"); };
  float *__restrict__ e = L.e;
  struct Pt {
    int i, j, q;
    float r;
    float4 k, k2;
  };
  auto point = [&](int v) {
    Pt t;
    t.j = 1 + v / nx;
    t.i = 1 + v - (t.j - 1) * nx;
    t.q = t.j * sj + t.i;
    t.r = L.r[v];
    t.k = L.cf4[3 * v];
    t.k2 = orth ? t.k : L.cf4[3 * v + 2];
    return t;
  };
  const Pt mine = point(min(tid, npt - 1));
  auto ypoint = [&](const Pt &t) {
    float d = t.r - t.k.x * e[t.q + 1] - t.k.z * e[t.q - 1];
    if (orth == false)
      d = d - t.k2.x * e[t.q + 1 + sj] - t.k2.y * e[t.q + sj - 1] - t.k2.z * e[t.q - 1 - sj] - t.k2.w * e[t.q + 1 - sj];
    e[t.q] = d;
  };
  auto xpoint = [&](const Pt &t) {
    float d = t.r - t.k.y * e[t.q + sj] - t.k.w * e[t.q - sj];
    if (orth == false)
      d = d - t.k2.x * e[t.q + 1 + sj] - t.k2.y * e[t.q + sj - 1] - t.k2.z * e[t.q - 1 - sj] - t.k2.w * e[t.q + 1 - sj];
    if (t.i == 1) d -= t.k.z * e[t.j * sj];
    if (t.i == nx) d -= t.k.x * e[t.j * sj + nx + 1];
    e[t.q] = d;
  };
  for (int sw = 0; sw < sweeps; ++sw) {
    for (int k = 0; k < 2; ++k) {
      const int col = post ? 2 - k : 1 + k;
      // line_phases, without its array: an even nx ends with i = 1 or nx alone
      const bool even = nx % 2 == 0;
      for (int q = 0; q < (even ? 2 : 1); ++q) {
        const int i0 = (q == 1) ? (col == 1 ? 1 : nx) : (even && col == 1) ? 3 : col;
        const int ncol = (q == 1) ? 1 : even ? nx / 2 - 1 : (col == 1) ? (nx + 1) / 2 : (nx - 1) / 2;
        auto in = [&](int i) { return i >= i0 && i < i0 + 2 * ncol && ((i - i0) & 1) == 0; };
        if (tid < npt && in(mine.i)) ypoint(mine);
        for (int v = tid + nt; v < npt; v += nt) {
          const Pt t = point(v);
          if (in(t.i)) ypoint(t);
        }
        sync();
        for (int c = tid; c < ncol; c += nt) {
          const int i = i0 + 2 * c;
          tail_chain(e + sj + i, sj, L.c + (i - 1), L.fy + (i - 1), nx, ny, (i == nx - 1) ? -i : 0, (i == 2) ? nx + 1 - i : 0);
        }
        sync();
      }
    }
    for (int k = 0; k < 2; ++k) {
      const int col = post ? 2 - k : 1 + k;
      if (tid < npt && ((mine.j - col) & 1) == 0) xpoint(mine);
      for (int v = tid + nt; v < npt; v += nt) {
        const Pt t = point(v);
        if (((t.j - col) & 1) == 0) xpoint(t);
      }
      sync();
      for (int j = col + 2 * tid; j <= ny; j += 2 * nt) {
        const int rb = (j - 1) * nx;
        float *erow = e + j * sj;
        tail_chain(erow + 1, 1, L.c + npt + rb, L.fx + rb, 1, nx, 0, 0);
        erow[0] = erow[nx - 1];
        erow[nx + 1] = erow[2];
      }
      sync();
    }
  }
}

// The same sweeps of a level of at most 32 points and N rows and columns (the
// coarsest one: many sweeps of a few points) by one warp, lane = point, e in
// registers.  A line's right-hand sides are gathered by shuffles and every
// lane of the line runs the line's recurrences, with the coefficients of its
// row and column in registers: no shared-memory round trip and no barrier
// stands between the phases.  A ghost column always equals the column it
// copies, and the rows outside the level are zero.
template <int N>
__device__ __forceinline__ void tail_coarse(const TailLv &L, int sweeps, bool orth) {
  const int nx = L.nx, ny = L.ny, sj = nx + 2, npt = nx * ny;
  const unsigned all = 0xffffffffu;
  const int v = min((int)(threadIdx.x & 31), npt - 1);
  const int j = v / nx, i = v - j * nx;  // from 0
  const int vl = v - i + ((i == 0) ? nx - 2 : i - 1), vr = v - i + ((i == nx - 1) ? 1 : i + 1);
  const bool hasn = j < ny - 1, hass = j > 0;
  const int up = hasn ? nx : 0, dn = hass ? -nx : 0;
  const float4 k = L.cf4[3 * v], k2 = orth ? k : L.cf4[3 * v + 2];
  const float r = L.r[v];
  float ay[N], my[N], cy[N], ax[N], mx[N], cx[N];
#pragma unroll
  for (int t = 0; t < N; ++t) {
    const int py = min(t, ny - 1) * nx + i, px = j * nx + min(t, nx - 1);
    ay[t] = L.c[py];
    my[t] = L.fy[py].y;
    cy[t] = L.fy[py].x;
    ax[t] = L.c[npt + px];
    mx[t] = L.fx[px].y;
    cx[t] = L.fx[px].x;
  }
  float e = 0.f;
  auto diag = [&](float d) {
    const float a = __shfl_sync(all, e, vr + up), b = __shfl_sync(all, e, vl + up);
    const float c = __shfl_sync(all, e, vl + dn), f = __shfl_sync(all, e, vr + dn);
    return d - k2.x * (hasn ? a : 0.f) - k2.y * (hasn ? b : 0.f) - k2.z * (hass ? c : 0.f) - k2.w * (hass ? f : 0.f);
  };
  // the line's solution at this lane's place (m) from its right-hand sides
  auto chain = [&](float d, int v0, int st, int n, int m, const float *a, const float *mm, const float *c) {
    float w[N];
#pragma unroll
    for (int t = 0; t < N; ++t) w[t] = __shfl_sync(all, d, v0 + min(t, n - 1) * st);
    float prev = 0.f;
#pragma unroll
    for (int t = 0; t < N; ++t) {
      prev = (w[t] - a[t] * prev) * mm[t];
      w[t] = prev;
    }
    float x = 0.f, mine = 0.f;
#pragma unroll
    for (int t = N - 1; t >= 0; --t) {
      x = (t < n) ? w[t] - c[t] * x : 0.f;
      mine = (t == m) ? x : mine;
    }
    return mine;
  };
  const bool even = nx % 2 == 0;
  for (int sw = 0; sw < sweeps; ++sw) {
    for (int q = 0; q < (even ? 4 : 2); ++q) {
      // the phases of line_phases: columns 1 3 5 .. and 2 4 .. (from 1); an
      // even nx: 3 5 .., 1, 2 4 .. nx-2, nx
      bool in;
      if (!even) in = (i & 1) == q;
      else if (q == 0) in = (i & 1) == 0 && i > 0;
      else if (q == 1) in = i == 0;
      else if (q == 2) in = (i & 1) == 1 && i < nx - 1;
      else in = i == nx - 1;
      const float er = __shfl_sync(all, e, vr), el = __shfl_sync(all, e, vl);
      float d = r - k.x * er - k.z * el;
      if (orth == false) d = diag(d);
      const float x = chain(d, i, nx, ny, j, ay, my, cy);
      e = in ? x : e;
    }
    for (int col = 0; col < 2; ++col) {
      const float en = __shfl_sync(all, e, v + up), es = __shfl_sync(all, e, v + dn);
      const float g0 = __shfl_sync(all, e, v - i + nx - 2), g1 = __shfl_sync(all, e, v - i + 1);
      float d = r - k.y * (hasn ? en : 0.f) - k.w * (hass ? es : 0.f);
      if (orth == false) d = diag(d);
      if (i == 0) d -= k.z * g0;
      if (i == nx - 1) d -= k.x * g1;
      const float x = chain(d, j * nx, 1, nx, i, ax, mx, cx);
      e = ((j & 1) == col) ? x : e;
    }
  }
  float *row = L.e + (j + 1) * sj;
  row[i + 1] = e;
  if (i == nx - 2) row[0] = e;
  if (i == 1) row[nx + 1] = e;
}

// The lines l0, l0 + lstep, ... (nline of them) of one colour by the whole
// block, k_f_pline's partitioned solve operation for operation: thread (s, li)
// owns segment s of line li, G lines at a time, sh the scratch of SH_N arrays
// of K x G (part_scratch).  The level's coefficients and the problem's diagonal are staged in
// shared memory: read from L2, a colour's 110 KB (65 x 65) at an SM's share of
// the L2 bandwidth took longer than the solve.
template <bool XL, bool ORTH>
__device__ __forceinline__ void part_lines(const TailLv &L, float *sh, int l0, int lstep, int nline) {
  constexpr int SEG = kPartSeg;
  const int nx = L.nx, ny = L.ny, n = XL ? nx : ny, sj = nx + 2, npt = nx * ny;
  const int K = part_segments(n);
  const int mb = (n - K + 1) / K, me = (n - K + 1) - mb * K;
  const int G = min((int)blockDim.x / K, nline);
  const int s0 = (int)threadIdx.x / G, li = (int)threadIdx.x - s0 * G;
  const int s = min(s0, K - 1);
  auto S = [&](int arr, int seg) -> float & { return sh[(arr * K + seg) * G + li]; };
  const int m = mb + (s < me ? 1 : 0);
  const int lo = 1 + s * (mb + 1) + min(s, me);
  const int nsep = K - 1;
  for (int g0 = 0; g0 < nline; g0 += G) {
    const bool act = s0 < K && g0 + li < nline;
    const int line = act ? l0 + lstep * (g0 + li) : l0;
    auto row = [&](int k, float &a, float &b, float &c, float &d) {
      const int i = XL ? k : line, j = XL ? line : k;
      const int pt = (j - 1) * nx + (i - 1);
      const float *ep = L.e + (j * sj + i);
      const float *cp = L.c + pt;
      b = cp[4 * npt];
      float dd = L.r[pt];
      if (XL) {
        a = cp[2 * npt];
        c = cp[0];
        dd = dd - cp[npt] * ep[sj] - cp[3 * npt] * ep[-sj];
      } else {
        a = cp[3 * npt];
        c = cp[npt];
        dd = dd - cp[0] * ep[1] - cp[2 * npt] * ep[-1];
      }
      if (!ORTH)
        dd = dd - cp[5 * npt] * ep[1 + sj] - cp[6 * npt] * ep[sj - 1] - cp[7 * npt] * ep[-(1 + sj)] -
             cp[8 * npt] * ep[-(sj - 1)];
      d = dd;
    };
    auto store = [&](int k, float x) {
      const int i = XL ? k : line, j = XL ? line : k;
      float *erow = L.e + j * sj;
      erow[i] = x;
      if (i == nx - 1) erow[0] = x;
      if (i == 2) erow[nx + 1] = x;
    };
    float av[SEG], bv[SEG], cv[SEG], dv[SEG];
    // (threads beyond the group's lines and segments only keep the barriers)
    if (act) {
#pragma unroll
      for (int u = 0; u < SEG; ++u) row(lo + min(u, m - 1), av[u], bv[u], cv[u], dv[u]);
      if (XL) {
        const float *erow = L.e + line * sj;
        if (s == 0) {
          dv[0] -= av[0] * erow[0];
          av[0] = 0.f;
        }
        if (s == K - 1) {
          const float gh = erow[nx + 1];
#pragma unroll
          for (int u = 0; u < SEG; ++u) {
            const bool hit = (u == m - 1);
            dv[u] = hit ? dv[u] - cv[u] * gh : dv[u];
            cv[u] = hit ? 0.f : cv[u];
          }
        }
      }
      float yl = 0.f, vl = 0.f, wl = 0.f;
      {
        float bprev = 0.f, dprev = 0.f, gprev = 1.f;
#pragma unroll
        for (int u = 0; u < SEG; ++u) {
          const float inv = __fdividef(1.f, bv[u] - av[u] * bprev);
          bprev = cv[u] * inv;
          dprev = (dv[u] - av[u] * dprev) * inv;
          gprev = -av[u] * gprev * inv;
          cv[u] = bprev;
          dv[u] = dprev;
          av[u] = gprev;
          const bool last = (u == m - 1);
          yl = last ? dprev : yl;
          vl = last ? gprev : vl;
          wl = last ? -bprev : wl;
        }
      }
      float yf = yl, vf = vl, wf = wl;
#pragma unroll
      for (int u = SEG - 2; u >= 0; --u)
        if (u < m - 1) {
          yf = dv[u] - cv[u] * yf;
          vf = av[u] - cv[u] * vf;
          wf = -cv[u] * wf;
        }
      S(SH_YF, s) = yf; S(SH_VF, s) = vf; S(SH_WF, s) = wf;
      S(SH_YL, s) = yl; S(SH_VL, s) = vl; S(SH_WL, s) = wl;
      if (s < nsep) {
        float a, b, c, d;
        row(lo + m, a, b, c, d);
        S(SH_A, s) = a; S(SH_B, s) = b; S(SH_C, s) = c; S(SH_D, s) = d;
      }
    }
    __syncthreads();
    const bool sep = act && s0 < nsep;
    float eA = 0.f, eB = 1.f, eC = 0.f, eD = 0.f;
    if (sep) {
      const float a = S(SH_A, s), c = S(SH_C, s);
      eA = (s > 0) ? a * S(SH_VL, s) : 0.f;
      eB = S(SH_B, s) + a * S(SH_WL, s) + c * S(SH_VF, s + 1);
      eC = (s < nsep - 1) ? c * S(SH_WF, s + 1) : 0.f;
      eD = S(SH_D, s) - a * S(SH_YL, s) - c * S(SH_YF, s + 1);
    }
    // (the rows go to two sets of arrays in turn, so that a step needs one
    // barrier: a set is written again only after the barrier behind which
    // everyone has read the other; the first set's entries were read by their
    // own thread alone, the second's neighbours before the first barrier)
    int set = 0;
    for (int d = 1; d < nsep; d <<= 1, set ^= 1) {
      const int qA = set ? SH_YF : SH_A, qB = set ? SH_VF : SH_B, qC = set ? SH_WF : SH_C, qD = set ? SH_YL : SH_D;
      if (sep) {
        S(qA, s) = eA;
        S(qB, s) = eB;
        S(qC, s) = eC;
        S(qD, s) = eD;
      }
      __syncthreads();
      if (sep) {
        float nA = 0.f, nC = 0.f, nB = eB, nD = eD;
        if (s - d >= 0) {
          const float al = __fdividef(eA, S(qB, s - d));
          nA = -al * S(qA, s - d);
          nB -= al * S(qC, s - d);
          nD -= al * S(qD, s - d);
        }
        if (s + d < nsep) {
          const float ga = __fdividef(eC, S(qB, s + d));
          nC = -ga * S(qC, s + d);
          nB -= ga * S(qA, s + d);
          nD -= ga * S(qD, s + d);
        }
        eA = nA;
        eB = nB;
        eC = nC;
        eD = nD;
      }
    }
    if (sep) S(SH_S, s) = __fdividef(eD, eB);
    __syncthreads();
    if (act) {
      const float X0 = (s > 0) ? S(SH_S, s - 1) : 0.f;
      const float X1 = (s < nsep) ? S(SH_S, s) : 0.f;
      float x = 0.f;
#pragma unroll
      for (int u = SEG - 1; u >= 0; --u)
        if (u < m) {
          x = dv[u] + av[u] * X0 - cv[u] * ((u == m - 1) ? X1 : x);
          store(lo + u, x);
        }
      if (s < nsep) store(lo + m, X1);
    }
    __syncthreads();
  }
}

// part_lines' zebra sweep at one level (tail_relax's order)
template <bool ORTH>
__device__ __forceinline__ void part_relax(const TailLv &L, float *sh, bool post) {
  for (int k = 0; k < 2; ++k) {
    const int col = post ? 2 - k : 1 + k;
    LinePhase ph[2];
    const int nph = line_phases(L.nx, col, ph);
    for (int q = 0; q < nph; ++q)
      if (ph[q].ncol > 0) part_lines<false, ORTH>(L, sh, ph[q].i0, ph[q].istep, ph[q].ncol);
  }
  for (int k = 0; k < 2; ++k) {
    const int col = post ? 2 - k : 1 + k;
    part_lines<true, ORTH>(L, sh, col, 2, (L.ny - col) / 2 + 1);
  }
}

// Thomas factors of every line of the levels 1..lth, per problem (one block
// per problem), into fac[p * nfac ...] in the shared-memory layout of the
// factor block; the same m and c' as yline_solve / xline_solve compute
__global__ void __launch_bounds__(kTailThreads) k_f_tail_factors(FastDev g, TailPlan t, float *fac) {
  const int p = (int)blockIdx.x;
  if (p >= g.P) return;
  const float kx2 = (float)g.kx2[p];
  float *fb = fac + (size_t)p * t.nfac;
  for (int l = 0; l < t.lth; ++l) {
    const int nx = t.nx[l], ny = t.ny[l], npt = nx * ny;
    const float4 *__restrict__ cf4 = g.lv[l].cf4;
    float2 *fy = reinterpret_cast<float2 *>(fb + t.f[l]);
    float2 *fx = fy + npt;
    // the y-lines on the first threads, the x-lines on the next; a chunk's
    // coefficients are loaded before the divisions run through it
    for (int t0 = threadIdx.x; t0 < nx + ny; t0 += blockDim.x) {
      const bool yl = t0 < nx;
      const int n = yl ? ny : nx, step = yl ? nx : 1, pt0 = yl ? t0 : (t0 - nx) * nx;
      float2 *f = yl ? fy : fx;
      float cprev = 0.f;
      for (int k0 = 0; k0 < n; k0 += kChunk) {
        float bv[kChunk], av[kChunk], cv[kChunk];
#pragma unroll
        for (int u = 0; u < kChunk; ++u) {
          const int k = min(k0 + u, n - 1), pt = pt0 + k * step;
          const float4 q0 = cf4[3 * pt], q1 = cf4[3 * pt + 1];
          bv[u] = ((-kx2 * q1.z) - q1.x) + q1.y;
          av[u] = yl ? q0.w : (k == 0) ? 0.f : q0.z;
          cv[u] = yl ? q0.y : (k == n - 1) ? 0.f : q0.x;
        }
#pragma unroll
        for (int u = 0; u < kChunk; ++u)
          if (k0 + u < n) {
            const float m = 1.f / (bv[u] - av[u] * cprev);
            cprev = cv[u] * m;
            f[pt0 + (k0 + u) * step] = make_float2(cprev, m);
          }
      }
    }
  }
}

template <bool ORTH>
__global__ void __launch_bounds__(kTailMost) k_f_vtail(FastDev g, TailPlan t, const float *fac) {
  if (*g.alldone) return;
  const int p = (int)blockIdx.x;
  if (p >= g.P || g.done[p]) return;
  extern __shared__ __align__(16) float tsh[];
  const int P = g.P;
  const float kx2 = (float)g.kx2[p];
  const int ltop = t.ltop;
  float *const scr = tsh + t.scr;
  {
    // this problem's factors (contiguous), the rhs of level ltop, e = 0 and the
    // coefficients, as asynchronous copies where they move unchanged
    auto cp16 = [](float *dst, const void *src) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                   : "memory");
    };
    auto cp4 = [](float *dst, const void *src) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                   : "memory");
    };
    const float *src = fac + (size_t)p * t.nfac;
    for (int v = threadIdx.x; v < t.nfac / 4; v += blockDim.x) cp16(tsh + t.fac0 + 4 * v, src + 4 * v);
    const TailLv T = tail_level_at(t, g, tsh, ltop - 1);
    const LvF &G = g.lv[ltop - 1];
    const int ne = (T.nx + 2) * (T.ny + 2), nr = T.nx * T.ny;
    for (int v = threadIdx.x; v < nr; v += blockDim.x) cp4(T.r + v, G.r + ((size_t)v * P + p));
    for (int l = t.lth; l < ltop; ++l) {
      const TailLv L = tail_level_at(t, g, tsh, l);
      const int npt = L.nx * L.ny;
      for (int v = threadIdx.x; v < npt; v += blockDim.x) {
        // one plane a coefficient: a line's rows and a colour's lines then
        // read distinct banks (packed float4 rows cost the solves 20%)
        const float *f = reinterpret_cast<const float *>(L.cf4 + 3 * v);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          cp4(L.c + q * npt + v, f + q);
          if (!ORTH) cp4(L.c + (5 + q) * npt + v, f + 8 + q);
        }
      }
    }
    for (int v = threadIdx.x; v < ne; v += blockDim.x) T.e[v] = 0.f;
    for (int l = 0; l < ltop; ++l) {
      const TailLv L = tail_level_at(t, g, tsh, l);
      const int npt = L.nx * L.ny;
      if (l < t.lth) {
        // the lower diagonals of the y-lines and of the x-lines (none at i = 1)
        for (int v = threadIdx.x; v < npt; v += blockDim.x) {
          const float4 q0 = L.cf4[3 * v];
          L.c[v] = q0.w;
          L.c[npt + v] = (v % L.nx == 0) ? 0.f : q0.z;
        }
      } else {
        float *cb = L.c + 4 * npt;
#pragma unroll 8
        for (int v = threadIdx.x; v < npt; v += blockDim.x) {
          const float4 q1 = L.cf4[3 * v + 1];
          cb[v] = ((-kx2 * q1.z) - q1.x) + q1.y;
        }
      }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = (int)blockDim.x >> 5;
  __syncthreads();
  // down the levels ltop..2, the coarsest, and up again (one place for each
  // operation: a second copy of the line solves costs the block its registers)
  for (int st = 0; st < 2 * ltop - 1; ++st) {
    const bool down = st < ltop - 1, up = st >= ltop;
    const int l = down ? ltop - st : up ? st - ltop + 2 : 1;
    const TailLv F = tail_level_at(t, g, tsh, l - 1), C = tail_level_at(t, g, tsh, max(l - 2, 0));
    if (up) {
      const int nrr = (C.ny < F.ny) ? (F.ny + 1) / 2 : F.ny;
      for (int rr = warp; rr < nrr; rr += nw)
        for (int i = 1 + lane; i <= F.nx; i += 32)
          f_prolong_x_at(C.e, scr, F.nx, F.ny, C.nx, C.ny, 1, 0, i, rr);
      __syncthreads();
      for (int j = 1 + warp; j <= F.ny; j += nw)
        for (int i = 1 + lane; i <= F.nx; i += 32) f_prolong_y_at(scr, F.e, F.nx, F.ny, C.ny, 1, 0, i, j);
      __syncthreads();
    }
    // a Thomas level's threads: one a point, whole warps, at most the block
    if (l == 1 && F.nx * F.ny <= 32 && max(F.nx, F.ny) <= 5) {
      if (warp == 0) tail_coarse<5>(F, t.sweeps, ORTH);
    } else if (l > t.lth) part_relax<ORTH>(F, scr, up);
    else tail_relax(F, min((int)blockDim.x, (F.nx * F.ny + 31) & ~31), (l == 1) ? t.sweeps : 1, ORTH, up);
    __syncthreads();
    if (l == 1 && kx2 == 0.f) {
      // singular: keep the correction at zero mean, ghosts included (the
      // sum in k_f_coarsest's order)
      __shared__ float mean;
      if (threadIdx.x == 0) {
        float m = 0.f;
        for (int j = 1; j <= F.ny; ++j)
          for (int i = 1; i <= F.nx; ++i) m += F.e[j * (F.nx + 2) + i];
        mean = m / (float)(F.nx * F.ny);
      }
      __syncthreads();
      for (int v = threadIdx.x; v < F.ny * (F.nx + 2); v += blockDim.x) F.e[(F.nx + 2) + v] -= mean;
      __syncthreads();
    }
    if (down) {
      for (int j = 1 + warp; j <= F.ny; j += nw)
        for (int i = 1 + lane; i <= F.nx; i += 32) {
          if (l > t.lth) {
            const int npt = F.nx * F.ny, v = (j - 1) * F.nx + i - 1, q = j * (F.nx + 2) + i;
            const float *cp = F.c + v;
            const float4 q0 = make_float4(cp[0], cp[npt], cp[2 * npt], cp[3 * npt]);
            const float4 q2 = ORTH ? q0 : make_float4(cp[5 * npt], cp[6 * npt], cp[7 * npt], cp[8 * npt]);
            scr[q] = f_resid_val(q0, q2, cp[4 * npt], F.e + q, 1, (size_t)(F.nx + 2), F.r[v], ORTH);
          } else {
            f_resid_at4(F.cf4, F.e, F.r, scr, F.nx, 1, 0, i, j, kx2, ORTH);
          }
        }
      __syncthreads();
      for (int jc = warp; jc <= C.ny + 1; jc += nw)
        for (int ic = lane; ic <= C.nx + 1; ic += 32)
          f_restrict_at(scr, C.e, C.r, F.nx, F.ny, C.nx, C.ny, 1, 0, ic, jc);
      __syncthreads();
    }
  }
  {
    const TailLv T = tail_level_at(t, g, tsh, ltop - 1);
    const LvF &G = g.lv[ltop - 1];
    const int ne = (T.nx + 2) * (T.ny + 2);
    for (int v = threadIdx.x; v < ne; v += blockDim.x) G.e[(size_t)v * P + p] = T.e[v];
  }
}

// the FP64 solution (finest interior, problem fastest) from the float-float
// iterate, after the last correction
__global__ void __launch_bounds__(32 * kRY) k_f_phif(FastDev g) {
  const int P = g.P;
  const int p = blockIdx.x * 32 + threadIdx.x;
  if (p >= P) return;
  const int nx = g.nfx, j = 1 + (int)blockIdx.y;
  const int par = g.cycles[p] & 1;
  const float *__restrict__ ph = par ? g.phh2 : g.phh;
  const float *__restrict__ pl = par ? g.phl2 : g.phl;
  for (int i = 1 + (int)threadIdx.y; i <= nx; i += kRY) {
    const size_t q = ((size_t)j * (nx + 2) + i) * P + p;
    g.phif[((size_t)(j - 1) * nx + (i - 1)) * P + p] = (double)FF(ph[q], pl[q]);
  }
}


// One partitioned line launch: lines l0, l0+lstep, ... (nline of them) of
// length n at level l, all problems, in the layout (lanes, seg): `lanes`
// problems per block (8, 16 or 32), segments of at most `seg` rows (4 or 8)
// separated by single rows, at most 128 segments and 1024 threads.  Lines
// the layout cannot hold fall back to one thread per line.
// K segments of at most seg rows and K-1 separator rows cover n rows when
// K (seg + 1) >= n + 1
int pline_segments(int n, int seg) { return std::max(1, (n + seg + 1) / (seg + 1)); }
bool pline_fits(int n, int lanes, int seg) {
  const int K = pline_segments(n, seg);
  return K <= 128 && K * lanes <= 1024;
}

// Lines of more rows than this have more than 32 segments of 8: a block of 16
// problems and 64 registers a thread is then alone on its SM.
constexpr int kOneBlockRows = 288;
void launch_pline(const FastDev &g, int l, bool xl, int l0, int lstep, int nline, int n, int lanes, int seg,
                  cudaStream_t s, bool zero_e = false) {
  if (zero_e && xl) throw CudaError("line solve: the zero-neighbour sweep is a y-line sweep");
  const int z = zero_e ? 1 : 0;
  const int K = pline_segments(n, seg);
  // the kernel indexes with 32-bit offsets
  if ((size_t)(g.nfx + 2) * (g.nfy + 2) * g.P >= (1ull << 31) || 11ull * g.nfx * g.nfy >= (1ull << 31))
    throw CudaError("line solve: grid x problems beyond 32-bit offsets");
  if (!pline_fits(n, lanes, seg)) {
    const unsigned b = (unsigned)(((long)nline * g.P + 63) / 64);
    if (xl) k_f_xline<<<b, 64, 0, s>>>(g, l, l0, nline);
    else k_f_yline<<<b, 64, 0, s>>>(g, l, l0, lstep, nline, z);
    return;
  }
  const int mb = (n - K + 1) / K, me = (n - K + 1) % K;
  const dim3 grid((unsigned)nline, (unsigned)((g.P + lanes - 1) / lanes)), blk(lanes, K);
  const size_t smem = sizeof(float) * SH_N * K * lanes;
#define EK_PLINE(W, S)                                                                             \
  do {                                                                                             \
    if (g.orth) {                                                                                  \
      if (xl) k_f_pline<true, true, W, S><<<grid, blk, smem, s>>>(g, l, l0, lstep, mb, me, z);        \
      else k_f_pline<false, true, W, S><<<grid, blk, smem, s>>>(g, l, l0, lstep, mb, me, z);          \
    } else {                                                                                       \
      if (xl) k_f_pline<true, false, W, S><<<grid, blk, smem, s>>>(g, l, l0, lstep, mb, me, z);       \
      else k_f_pline<false, false, W, S><<<grid, blk, smem, s>>>(g, l, l0, lstep, mb, me, z);         \
    }                                                                                              \
  } while (0)
  if (seg == 4) {
    if (lanes == 32) EK_PLINE(32, 4);
    else if (lanes == 16) EK_PLINE(16, 4);
    else EK_PLINE(8, 4);
  } else {
    if (lanes == 32) EK_PLINE(32, 8);
    else if (lanes == 16) EK_PLINE(16, 8);
    // (three blocks of 8 problems and 43 segments an SM for two: default_lanes)
    else if (!xl && g.orth && n > kOneBlockRows) k_f_pline<false, true, 8, 8, 56><<<grid, blk, smem, s>>>(g, l, l0, lstep, mb, me, z);
    else EK_PLINE(8, 8);
  }
#undef EK_PLINE
}

// The layout the solver uses when nothing was tuned: 8-row segments, 16
// problems per block (to 567 rows; 8 beyond).  Over grids of 128 x 129 x 97 to
// 512 x 385 x 257, straight and sheared, 16 problems are as fast as 32 or
// faster at all but one level (129 rows, 21.4 against 20.6 us a sweep; the
// finest x-lines of the largest 213 against 238, of 64 x 225 x 161 21 against
// 27), and 8 gain 2 to 5% on the finest x-lines alone and lose 10 to 25% on
// the short ones.
// Beyond 288 rows a block of 16 is alone on its SM, which waits while that block
// loads, reduces and stores in turn; blocks of 8 share it, three of them for
// the y-lines of an orthogonal grid at 56 registers (at 64 two; shorter lines
// and the sheared kernel, with more to hold, are slower at 56).  A sweep,
// 16 problems against 8: 385 rows of 512 x 385 x 257 314 -> 287 us, 321 rows of
// 128 x 321 x 193 57.6 -> 52.2, x-lines of 321 of a sheared 256 x 65 x 321 49.5 ->
// 42.0; sheared y-lines 414 and 405, 74.0 and 75.5, so these keep 16.  Fewer
// blocks than SMs keep 16 as well (32 x 385 x 129: 20.7 against 24.8).
int default_lanes(const FastDev &g, bool xl, int n, int nline) {
  if (pline_segments(n, 8) > 64) return 8;
  return n > kOneBlockRows && (xl || g.orth) && (long)nline * ((g.P + 15) / 16) > 152 ? 8 : 16;
}

FastDev make_fastdev(Ctx &c, int nprob, const double *kx2_dev) {
  const MgPlan &PL = c.mg;
  MgWork &w = c.mgw;
  FastDev g{};
  g.P = nprob;
  g.ngrid = PL.ngrid;
  g.orth = PL.orth ? 1 : 0;
  for (int l = 0; l < PL.ngrid; ++l) {
    const MgLevelF &F = c.mgf_levels[l];
    g.lv[l] = LvF{PL.lv[l].nx, PL.lv[l].ny, F.e, F.r, F.cof, F.cp, F.cf4};
  }
  g.scr = c.mgf_scratch;
  g.rhs = w.rhs[PL.ngrid - 1];
  g.phh = c.mgf_phh;
  g.phl = c.mgf_phl;
  g.phh2 = c.mgf_phh2;
  g.phl2 = c.mgf_phl2;
  g.bh = c.mgf_bh;
  g.bl = c.mgf_bl;
  g.cf2 = c.mgf_cf2;
  g.nfx = PL.nfx;
  g.nfy = PL.nfy;
  g.kx2 = kx2_dev;
  g.phif = w.phif;
  g.red = w.red;
  g.done = w.done;
  g.cycles = w.cycles;
  g.alldone = w.alldone;
  g.iter = w.iter;
  g.count = w.flags + 2 * w.pmax + 2;
  g.tol = c.p.mg_tol;
  return g;
}

// The levels of k_f_vtail whose lines go one thread each (Thomas factors): the
// largest level below the finest whose iterates, right-hand sides and factors
// fit kTailSmem bytes (0: none fits, k_f_coarsest).
constexpr size_t kTailSmem = 24 * 1024;
int thomas_levels(const MgPlan &PL) {
  int l = 0;
  while (l + 1 < PL.ngrid && l + 1 <= kTailMax && make_tail_plan(PL, l + 1, l + 1).c[0] * sizeof(float) <= kTailSmem)
    ++l;
  return l;
}
constexpr size_t kTailMostSmem = 220 * 1024;
constexpr int kSMs = 152;
size_t tail_bytes_of(const TailPlan &t) { return (size_t)t.total * sizeof(float); }
// Threads of a k_f_vtail block (128 registers each): the whole register file
// while every problem has an SM of its own, half of it when two blocks share
// one.
int tail_threads(const TailPlan &t, int nprob) {
  if (t.ltop == t.lth) return kTailThreads;
  return (nprob <= kSMs) ? kTailMost : kTailMost / 2;
}
// The levels 1..ltop that run as one k_f_vtail launch for nprob problems: the
// largest whose arrays fit one SM's shared memory while every problem has an
// SM of its own, half of it beyond.  With fewer problems than SMs a level's
// batched launches leave the GPU idle between their dependent steps
// (44 problems of 65 x 65: 12 launches a level and cycle of 5-9 us each, 27 us
// in the block); with 342 problems a level of 65 x 97 in the block costs
// 15.2 -> 16.2 ms a batch, and 33 x 49 gains 1% over leaving it out.  A level
// whose line-solve layout was set by hand keeps its launches; a tuned layout
// serves the batches whose level is launched, and moves no level.
bool layout_by_hand(const MgPlan &PL, int l) { return l < (int)PL.by_hand.size() && PL.by_hand[l]; }
int tail_level(const MgPlan &PL, int nprob) {
  const int lth = thomas_levels(PL);
  if (lth == 0) return 0;
  const size_t most = (nprob <= kSMs) ? kTailMostSmem : kTailMostSmem / 2;
  // (k_f_pline takes lines of at most 567 rows at 16 problems a block; longer
  // ones go one thread a line, in another order of operations)
  int top = lth;
  while (top + 1 <= PL.ngrid && top + 1 <= kTailMax && !layout_by_hand(PL, top + 1) && std::max(PL.lv[top].nx, PL.lv[top].ny) <= 567 &&
         tail_bytes_of(make_tail_plan(PL, top + 1, lth)) <= most)
    ++top;
  return top;
}

// Blocks resident at once
constexpr unsigned kResidWave = 4u * 152u;
// A row's blocks: enough to give every SM its four, of runs of two points and
// more.  (64 x 65 x 65: 2 x 65 blocks of nine-point runs become 2 x 65 x 4 of
// three-point ones.)
unsigned resid_blocks(const FastDev &g, unsigned pch) {
  const unsigned fill = kResidWave / (pch * (unsigned)g.nfy), most = (unsigned)g.nfx / (2 * kRY);
  return std::max(1u, std::min(fill, most));
}
void launch_resid_ff(const FastDev &g, bool update, unsigned pch, const CheckF &ck, cudaStream_t s) {
  const dim3 grid(pch, (unsigned)g.nfy, resid_blocks(g, pch)), blk(32, kRY);
  if (update) {
    if (g.orth) k_f_resid_ff<true, true><<<grid, blk, 0, s>>>(g, ck);
    else k_f_resid_ff<true, false><<<grid, blk, 0, s>>>(g, ck);
  } else {
    if (g.orth) k_f_resid_ff<false, true><<<grid, blk, 0, s>>>(g, ck);
    else k_f_resid_ff<false, false><<<grid, blk, 0, s>>>(g, ck);
  }
}

unsigned nb(long n, int bs) {
  long b = (n + bs - 1) / bs;
  if (b < 1) b = 1;
  if (b > 65535L * 32) b = 65535L * 32;
  return (unsigned)b;
}

}  // namespace

int mgfast_tail_levels(const Ctx &c) { return c.mg.ngrid > 0 ? thomas_levels(c.mg) : 0; }

// FP32 copies of the level coefficients and the FP32 work arrays.
void mgfast_alloc(Ctx &c, int pmax) {
  MgPlan &PL = c.mg;
  if (c.mgf_pool) {
    cudaFree(c.mgf_pool);
    c.mgf_pool = nullptr;
  }
  size_t tot = 0;
  std::vector<size_t> off(PL.ngrid);
  for (int l = 0; l < PL.ngrid; ++l) {
    const MgLevel &L = PL.lv[l];
    off[l] = tot;
    tot += (size_t)(L.nx + 2) * (L.ny + 2) * pmax + 2 * (size_t)L.nx * L.ny * pmax + 11 * (size_t)L.nx * L.ny;
  }
  const size_t scr_off = tot;
  const size_t nph = (size_t)(PL.nfx + 2) * (PL.nfy + 2), nf = (size_t)PL.nfx * PL.nfy;
  tot += nph * pmax;
  const size_t ff_off = tot;
  tot += 4 * nph * pmax + 2 * nf * pmax + 22 * nf + 1;
  const int lth = thomas_levels(PL);
  const size_t nfac = lth ? (size_t)make_tail_plan(PL, lth, lth).nfac * pmax : 0;
  tot = (tot + 3) & ~(size_t)3;  // float4 reads of each problem's factor block
  const size_t fac_off = tot;
  tot += nfac;
  EK_CUDA(cudaMalloc(&c.mgf_pool, tot * sizeof(float)));
  c.mgf_levels.assign(PL.ngrid, {});
  // the packed coefficients (3 float4 per point and level)
  if (c.mgf_cf4_pool) {
    cudaFree(c.mgf_cf4_pool);
    c.mgf_cf4_pool = nullptr;
  }
  size_t n4 = 0;
  for (int l = 0; l < PL.ngrid; ++l) n4 += 3 * (size_t)PL.lv[l].nx * PL.lv[l].ny;
  EK_CUDA(cudaMalloc(&c.mgf_cf4_pool, n4 * sizeof(float4)));
  for (int l = 0; l < PL.ngrid; ++l) {
    const MgLevel &L = PL.lv[l];
    float *b = c.mgf_pool + off[l];
    MgLevelF &F = c.mgf_levels[l];
    F.e = b;
    F.r = F.e + (size_t)(L.nx + 2) * (L.ny + 2) * pmax;
    F.cp = F.r + (size_t)L.nx * L.ny * pmax;
    F.cof = F.cp + (size_t)L.nx * L.ny * pmax;
    std::vector<float> cf(PL.cof_host[l].begin(), PL.cof_host[l].end());
    EK_CUDA(cudaMemcpy(F.cof, cf.data(), sizeof(float) * cf.size(), cudaMemcpyHostToDevice));
    {
      const size_t npt = (size_t)L.nx * L.ny;
      size_t o4 = 0;
      for (int q = 0; q < l; ++q) o4 += 3 * (size_t)PL.lv[q].nx * PL.lv[q].ny;
      F.cf4 = c.mgf_cf4_pool + o4;
      std::vector<float4> pk(3 * npt);
      for (size_t pt = 0; pt < npt; ++pt) {
        auto C = [&](int t) { return cf[t * npt + pt]; };
        pk[3 * pt] = make_float4(C(0), C(2), C(4), C(6));
        pk[3 * pt + 1] = make_float4(C(8), C(9), C(10), 0.f);
        pk[3 * pt + 2] = make_float4(C(1), C(3), C(5), C(7));
      }
      EK_CUDA(cudaMemcpy(F.cf4, pk.data(), sizeof(float4) * pk.size(), cudaMemcpyHostToDevice));
    }
  }
  c.mgf_scratch = c.mgf_pool + scr_off;
  c.mgf_phh = c.mgf_pool + ff_off;
  c.mgf_phl = c.mgf_phh + nph * pmax;
  c.mgf_phh2 = c.mgf_phl + nph * pmax;
  c.mgf_phl2 = c.mgf_phh2 + nph * pmax;
  c.mgf_bh = c.mgf_phl2 + nph * pmax;
  c.mgf_bl = c.mgf_bh + nf * pmax;
  // 8-byte aligned for the float2 loads: the address itself decides (the
  // pool holds one float of slack)
  {
    float *cfb = c.mgf_bl + nf * pmax;
    if (reinterpret_cast<uintptr_t>(cfb) & 7) ++cfb;
    c.mgf_cf2 = reinterpret_cast<float2 *>(cfb);
  }
  c.mgf_tailfac = nfac ? c.mgf_pool + fac_off : nullptr;
  c.mgf_tailfac_n = nfac;
  // every context's tail fits kTailMostSmem, so one process-wide limit serves
  // all (set here, never during a stream capture)
  EK_CUDA(cudaFuncSetAttribute(k_f_vtail<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailMostSmem));
  EK_CUDA(cudaFuncSetAttribute(k_f_vtail<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailMostSmem));
  {
    // the finest coefficients split into float-float pairs
    const std::vector<double> &cf = PL.cof_host[PL.ngrid - 1];
    std::vector<float2> hl(cf.size());
    for (size_t t = 0; t < cf.size(); ++t) {
      const float h = (float)cf[t];
      hl[t] = make_float2(h, (float)(cf[t] - (double)h));
    }
    EK_CUDA(cudaMemcpy(c.mgf_cf2, hl.data(), sizeof(float2) * hl.size(), cudaMemcpyHostToDevice));
  }
  c.mgf_pmax = pmax;
}

// Solve with the mixed-precision iteration; the finest rhs must be in
// c.mgw.rhs[ngrid-1] (FP64, problem fastest); the solution is left in
// c.mgw.phif.
int mgfast_solve(Ctx &c, int nprob, const double *kx2_dev, const double *kx2_host, ek_mg_stats *st) {
  MgPlan &PL = c.mg;
  MgWork &w = c.mgw;
  if (nprob > c.mgf_pmax || nprob > w.pmax) return EK_ERR_ARG;
  cudaStream_t s = c.stream;
  const int bs = 256;
  const long npt = (long)PL.nfx * PL.nfy;
  // the kx^2 = 0 problems (well posed by projection; the learned guess and
  // its statistics leave them out)
  std::vector<double> kxh;
  if (!kx2_host) {
    kxh.resize(nprob);
    EK_CUDA(cudaMemcpyAsync(kxh.data(), kx2_dev, sizeof(double) * nprob, cudaMemcpyDeviceToHost, s));
    EK_CUDA(cudaStreamSynchronize(s));
    kx2_host = kxh.data();
  }
  std::vector<char> is_sing(nprob, 0);
  int ns = 0;
  for (int p = 0; p < nprob; ++p)
    if (kx2_host[p] == 0.0) {
      is_sing[p] = 1;
      ++ns;
    }
  if (ns > 0) mg_null_project(c, w.rhs[PL.ngrid - 1], nprob, kx2_dev);
  FastDev g = make_fastdev(c, nprob, kx2_dev);

  {
    KScope ks(c, KC_MG_SETUP, 8.0 * (PL.nfx + 2) * (PL.nfy + 2) * nprob * 2);
    EK_CUDA(cudaMemsetAsync(w.flags, 0, sizeof(int) * (2 * w.pmax + 4), s));
    EK_CUDA(cudaMemsetAsync(w.red, 0, sizeof(double) * (6 * w.pmax + 8), s));
    const size_t nph = (size_t)(PL.nfx + 2) * (PL.nfy + 2) * nprob;
    EK_CUDA(cudaMemsetAsync(g.phh, 0, sizeof(float) * nph, s));
    EK_CUDA(cudaMemsetAsync(g.phl, 0, sizeof(float) * nph, s));
    EK_CUDA(cudaMemsetAsync(g.phh2, 0, sizeof(float) * nph, s));
    EK_CUDA(cudaMemsetAsync(g.phl2, 0, sizeof(float) * nph, s));
    // the finest correction: its ghost rows stay zero from here on, and each
    // cycle's first sweep leaves its other values unread
    EK_CUDA(cudaMemsetAsync(g.lv[PL.ngrid - 1].e, 0, sizeof(float) * nph, s));
    const size_t nf = (size_t)PL.nfx * PL.nfy * nprob;
    k_f_split<<<nb((long)nf, bs), bs, 0, s>>>(g.rhs, g.bh, g.bl, nf);
    after_launch(c);
  }
  const int gx = (nprob + 31) / 32;
  const unsigned pch = (unsigned)gx;  // 32-problem chunks of the row kernels
  // learned initial guess for the kx^2 != 0 problems, scaled by the
  // least-squares factor (a useless guess gets a factor near zero)
  const bool guessed = c.guess.net && c.guess.use && nprob > ns;
  if (guessed) {
    GuessState &G = c.guess;
    KScope ks(c, KC_GUESS, G.net->forward_flops(nprob - ns));
    std::vector<int> nonsing;
    for (int p = 0; p < nprob; ++p)
      if (!is_sing[p]) nonsing.push_back(p);
    guess_predict(c, nprob, g.rhs, kx2_dev, nonsing, g.phh, s);
    if (G.alpha_cap < nprob) {
      cudaFree(G.alpha);
      G.alpha = nullptr;
      G.alpha_cap = 0;
      EK_CUDA(cudaMalloc(&G.alpha, sizeof(float) * nprob));
      G.alpha_cap = nprob;
    }
    launch_resid_ff(g, false, pch, CheckF{}, s);
    after_launch(c);
    k_f_guess_rb<<<dim3(pch, PL.nfy), dim3(32, kRY), 0, s>>>(g);
    after_launch(c);
    k_f_guess_alpha<<<nb(nprob, 128), 128, 0, s>>>(g, G.alpha);
    after_launch(c);
    k_f_guess_scale<<<nb((long)(PL.nfx + 2) * (PL.nfy + 2) * nprob, bs), bs, 0, s>>>(g, G.alpha);
    after_launch(c);
  }

  // one partitioned line launch, in the layout tuned for (level, direction)
  auto pline = [&](int l, bool xl, int l0, int lstep, int nline, int n, bool zero_e) {
    int lanes = default_lanes(g, xl, n, nline), seg = 8;
    const std::vector<int> &tl = xl ? PL.lanes_x : PL.lanes_y;
    const std::vector<int> &ts = xl ? PL.seg_x : PL.seg_y;
    if (l < (int)tl.size() && tl[l] > 0) lanes = tl[l];
    if (l < (int)ts.size() && ts[l] > 0) seg = ts[l];
    launch_pline(g, l, xl, l0, lstep, nline, n, lanes, seg, s, zero_e);
    after_launch(c);
  };


  // one alternating-direction zebra sweep at level l: y-lines (colours
  // 1, 2), then x-lines (rows 1, 3, ... then 2, 4, ...); the post-smoothing
  // sweep takes the colours in the reverse order.  (Post-smoothing with
  // x-lines only needs 8-9 corrections instead of 6-7 on the 256x257x193
  // grid, so it costs more than it saves.)
  // zero_first: e holds stale values that the cycle starts from zero
  // (the finest level, whose e is not cleared between cycles): the first
  // colour's y-lines take their neighbours as zero.  Needs odd nx (one
  // phase per colour, and no line of the first colour reads a line of the
  // same colour), which every level above the coarsest has.
  auto relax = [&](int l, bool post, bool zero_first) {
    const MgLevel &L = PL.lv[l - 1];
    KScope ks(c, KC_MG_RELAX, 4.0 * nprob * L.nx * L.ny * 10);
    for (int k = 0; k < 2; ++k) {
      const int col = post ? 2 - k : 1 + k;
      LinePhase ph[2];
      const int nph = line_phases(L.nx, col, ph);
      for (int q = 0; q < nph; ++q)
        if (ph[q].ncol > 0) pline(l, false, ph[q].i0, ph[q].istep, ph[q].ncol, L.ny, zero_first && k == 0);
    }
    for (int k = 0; k < 2; ++k) {
      const int col = post ? 2 - k : 1 + k;
      pline(l, true, col, 2, (L.ny - col) / 2 + 1, L.nx, false);
    }
  };

  const int maxit = c.p.mg_maxcy;
  // r = b - A phi and the per-problem decision (incr: count one more
  // correction); cond/use_cond: the while-node condition in a graph
  auto check = [&](int incr, cudaGraphConditionalHandle cond, int use_cond) {
    // bytes: b (2), r; phi (2), and with the update e and phi' (2)
    KScope ks(c, KC_MG_CHECK, 4.0 * nprob * npt * (incr ? 8.0 : 5.0));
    const bool one = pch * (unsigned)g.nfy * resid_blocks(g, pch) <= kResidWave;
    const CheckF ck{one ? 1 : 0, maxit, incr, use_cond, cond};
    launch_resid_ff(g, incr != 0, pch, ck, s);
    if (!one) {
      after_launch(c);
      k_f_check<<<1, 256, 0, s>>>(g, ck);
    }
    after_launch(c);
  };
  // the levels 1..ltop run as one k_f_vtail launch
  const int ltop = tail_level(PL, nprob);
  const TailPlan tplan = ltop ? make_tail_plan(PL, ltop, thomas_levels(PL)) : TailPlan{};
  if (ltop) {
    if ((size_t)tplan.nfac * nprob > c.mgf_tailfac_n) throw CudaError("mixed solve: tail factor buffer too small");
    KScope ks(c, KC_MG_SETUP, 4.0 * nprob * tplan.nfac);
    k_f_tail_factors<<<(unsigned)nprob, kTailThreads, 0, s>>>(g, tplan, c.mgf_tailfac);
    after_launch(c);
  }
  // one FP32 V(1,1) cycle on A e = r from e = 0 (phi += e follows in the
  // next check's residual kernel).  The finest e is not cleared: the first
  // sweep reads none of it (odd nx, the MUDPACK grids' rule), else it is
  // cleared here.
  const bool fine_zero = PL.ngrid >= 2 && PL.lv[PL.ngrid - 1].nx % 2 == 1;
  auto correction = [&]() {
    if (!fine_zero) {
      const size_t nph = (size_t)(PL.nfx + 2) * (PL.nfy + 2) * nprob;
      EK_CUDA(cudaMemsetAsync(g.lv[PL.ngrid - 1].e, 0, sizeof(float) * nph, s));
    }
    for (int l = PL.ngrid; l >= 1; --l) {
      const MgLevel &L = PL.lv[l - 1];
      if (l == ltop) {
        // bytes: level ltop's rhs in and its correction out
        KScope ks(c, KC_MG_COARSE, 4.0 * nprob * (L.nx * L.ny + (L.nx + 2.0) * (L.ny + 2)));
        const int nt = tail_threads(tplan, nprob);
        if (g.orth) k_f_vtail<true><<<(unsigned)nprob, nt, tail_bytes_of(tplan), s>>>(g, tplan, c.mgf_tailfac);
        else k_f_vtail<false><<<(unsigned)nprob, nt, tail_bytes_of(tplan), s>>>(g, tplan, c.mgf_tailfac);
        after_launch(c);
        break;
      }
      if (l == 1) {
        const int sweeps = std::max(8, (L.nx + L.ny) / 2);
        KScope ks(c, KC_MG_RELAX, 4.0 * nprob * L.nx * L.ny * 10 * sweeps);
        k_f_coarsest<<<nb(nprob, 64), 64, 0, s>>>(g, sweeps);
        after_launch(c);
        break;
      }
      relax(l, false, l == PL.ngrid && fine_zero);
      const MgLevel &C = PL.lv[l - 2];
      KScope ks(c, KC_MG_TRANSFER, 4.0 * nprob * (4.0 * L.nx * L.ny + 2.0 * (C.nx + 2) * (C.ny + 2)));
      k_f_resid32<<<dim3(pch, L.ny), dim3(32, kRowWarps), 0, s>>>(g, l);
      after_launch(c);
      k_f_restrict<<<dim3(pch, C.ny + 2), dim3(32, kRowWarps), 0, s>>>(g, l);
      after_launch(c);
    }
    for (int l = std::max(2, ltop + 1); l <= PL.ngrid; ++l) {
      const MgLevel &L = PL.lv[l - 1];
      {
        KScope ks(c, KC_MG_TRANSFER, 4.0 * nprob * 4.0 * L.nx * L.ny);
        const unsigned rows = (unsigned)(PL.lv[l - 2].ny + kProRows - 1) / kProRows;
        // columns apart in as many blocks as give every SM four
        const unsigned cols = std::max(1u, std::min(4u * 152u / (pch * rows), nb(L.nx, kRowWarps)));
        k_f_prolong<<<dim3(pch, rows, cols), dim3(32, kRowWarps), 0, s>>>(g, l);
        after_launch(c);
      }
      relax(l, true, false);
    }
  };
  if (c.graph_slot < 0) {
    // eager: the host stops issuing cycles once the done flag it polls is set
    c.poll.init();
    c.poll.reset();
    check(0, 0, 0);
    bool stop = c.poll.after_check(w.alldone, s);
    for (int it = 1; it <= maxit && !stop; ++it) {
      correction();
      check(1, 0, 0);
      stop = c.poll.after_check(w.alldone, s);
    }
  } else {
    // captured: the cycles repeat in a conditional while-node whose
    // condition the check kernel sets, so no host decides between them
    cudaStreamCaptureStatus cs;
    cudaGraph_t cg = nullptr;
    const cudaGraphNode_t *deps = nullptr;
    size_t ndeps = 0;
    EK_CUDA(cudaStreamGetCaptureInfo(s, &cs, nullptr, &cg, &deps, nullptr, &ndeps));
    if (cs != cudaStreamCaptureStatusActive) throw CudaError("mixed solve: step graph capture is not active");
    cudaGraphConditionalHandle cond;
    EK_CUDA(cudaGraphConditionalHandleCreate(&cond, cg, 1u, cudaGraphCondAssignDefault));
    check(0, cond, 1);
    EK_CUDA(cudaStreamGetCaptureInfo(s, &cs, nullptr, &cg, &deps, nullptr, &ndeps));
    cudaGraphNodeParams np = {};
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = cond;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t wnode;
    EK_CUDA(cudaGraphAddNode(&wnode, cg, deps, nullptr, ndeps, &np));
    cudaGraph_t body = np.conditional.phGraph_out[0];
    EK_CUDA(cudaStreamUpdateCaptureDependencies(s, &wnode, nullptr, 1, cudaStreamSetCaptureDependencies));
    const cudaStream_t outer = s;
    s = c.cap_stream2;
    const long long l0 = c.launches;
    try {
      EK_CUDA(cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
      correction();
      check(1, cond, 1);
      cudaGraph_t done_body = nullptr;
      EK_CUDA(cudaStreamEndCapture(s, &done_body));
    } catch (...) {
      cudaGraph_t junk = nullptr;
      cudaStreamEndCapture(c.cap_stream2, &junk);
      s = outer;
      throw;
    }
    s = outer;
    c.graph_body_launches = c.launches - l0;
  }
  {
    KScope ks(c, KC_MG_SETUP, 16.0 * nprob * npt);
    k_f_phif<<<dim3(pch, PL.nfy), dim3(32, kRY), 0, s>>>(g);
    after_launch(c);
  }
  if (ns > 0) mg_null_mean(c, w.phif, nprob, kx2_dev);
  if (c.graph_slot >= 0) {
    // a captured step reads the statistics after the step
    k_f_stats<<<1, 256, 0, s>>>(g, c.step_stats_dev + c.graph_slot);
    after_launch(c);
    return EK_OK;
  }
  std::vector<int> cyc(nprob), done(nprob);
  std::vector<double> meas(6 * nprob);
  EK_CUDA(cudaMemcpyAsync(cyc.data(), w.cycles, sizeof(int) * nprob, cudaMemcpyDeviceToHost, s));
  EK_CUDA(cudaMemcpyAsync(done.data(), w.done, sizeof(int) * nprob, cudaMemcpyDeviceToHost, s));
  EK_CUDA(cudaMemcpyAsync(meas.data(), w.red, sizeof(double) * 6 * nprob, cudaMemcpyDeviceToHost, s));
  EK_CUDA(cudaStreamSynchronize(s));
  ek_mg_stats S{};
  S.nprob = nprob;
  S.min_cycles = nprob ? (1 << 30) : 0;
  double csum = 0.0, rsum = 0.0;
  for (int p = 0; p < nprob; ++p) {
    S.min_cycles = std::min(S.min_cycles, cyc[p]);
    S.max_cycles = std::max(S.max_cycles, cyc[p]);
    if (done[p] != 1) S.n_not_converged++;
    S.max_residual = std::max(S.max_residual, meas[6 * p + 4]);
    if (is_sing[p]) continue;
    csum += cyc[p];
    rsum += guessed ? meas[6 * p + 5] : 1.0;
  }
  c.last_mean_cycles = (nprob > ns) ? csum / (nprob - ns) : 0.0;
  c.guess.last_rho = (nprob > ns) ? rsum / (nprob - ns) : 1.0;
  c.last_stats = S;
  if (st) *st = S;
  return S.n_not_converged ? EK_ERR_NOT_CONVERGED : EK_OK;
}


// Tile-shape autotuner of the line solves: for every level of the mixed
// solver and both line directions, time one full zebra sweep (both colours)
// in each valid layout -- 8, 16 or 32 problems per block, segments of 8 or 4
// rows -- on the solver's own arrays, `reps` times, and keep the fastest.  The level arrays are work
// space that every solve re-initialises, so the timing runs leave no trace.
int mgfast_autotune(Ctx &c, int reps, std::string &report) {
  MgPlan &PL = c.mg;
  MgWork &w = c.mgw;
  const int nprob = 2 * (c.d.NKX + 1);
  if (!c.p.mg_fast || nprob > c.mgf_pmax) return EK_ERR_STATE;
  cudaStream_t s = c.stream;
  FastDev g = make_fastdev(c, nprob, w.kx2);
  EK_CUDA(cudaMemsetAsync(w.flags, 0, sizeof(int) * (2 * w.pmax + 4), s));  // every problem active
  PL.lanes_y.assign(PL.ngrid + 1, 0);
  PL.lanes_x.assign(PL.ngrid + 1, 0);
  PL.seg_y.assign(PL.ngrid + 1, 0);
  PL.seg_x.assign(PL.ngrid + 1, 0);
  PL.by_hand.assign(PL.ngrid + 1, 0);
  cudaEvent_t e0, e1;
  EK_CUDA(cudaEventCreate(&e0));
  EK_CUDA(cudaEventCreate(&e1));
  report = "[";
  bool first = true;
  try {
    // the Thomas levels of k_f_vtail have no line-solve launches to tune; the
    // levels above them that it takes by tail_level's rule are timed as
    // launches, for the larger batches that run them so
    for (int l = std::max(2, thomas_levels(PL) + 1); l <= PL.ngrid; ++l) {
      const MgLevel &L = PL.lv[l - 1];
      for (int dir = 0; dir < 2; ++dir) {
        const bool xl = dir == 1;
        const int n = xl ? L.nx : L.ny;
        auto sweep = [&](int lanes, int seg) {
          if (xl) {
            for (int col = 1; col <= 2; ++col) {
              launch_pline(g, l, true, col, 2, (L.ny - col) / 2 + 1, L.nx, lanes, seg, s);
              after_launch(c);
            }
          } else {
            for (int col = 1; col <= 2; ++col) {
              LinePhase ph[2];
              const int nph = line_phases(L.nx, col, ph);
              for (int q = 0; q < nph; ++q)
                if (ph[q].ncol > 0) {
                  launch_pline(g, l, false, ph[q].i0, ph[q].istep, ph[q].ncol, L.ny, lanes, seg, s);
                  after_launch(c);
                }
            }
          }
        };
        int best = 0, best_seg = 8;
        float best_ms = 0.f;
        std::string row;
        for (int seg : {8, 4})
          for (int lanes : {32, 16, 8}) {
            if (!pline_fits(n, lanes, seg)) continue;
            sweep(lanes, seg);  // warm-up
            EK_CUDA(cudaEventRecord(e0, s));
            for (int r = 0; r < reps; ++r) sweep(lanes, seg);
            EK_CUDA(cudaEventRecord(e1, s));
            EK_CUDA(cudaEventSynchronize(e1));
            float ms = 0.f;
            EK_CUDA(cudaEventElapsedTime(&ms, e0, e1));
            ms /= (float)reps;
            row += (row.empty() ? "" : ", ") + std::string("\"") + std::to_string(lanes) + "x" + std::to_string(seg) +
                   "\": " + std::to_string(1000.0 * ms);
            if (best == 0 || ms < best_ms) {
              best = lanes;
              best_seg = seg;
              best_ms = ms;
            }
          }
        (xl ? PL.lanes_x : PL.lanes_y)[l] = best;
        (xl ? PL.seg_x : PL.seg_y)[l] = best_seg;
        report += std::string(first ? "" : ", ") + "{\"level\": " + std::to_string(l) + ", \"dir\": \"" +
                  (xl ? "x" : "y") + "\", \"n\": " + std::to_string(n) + ", \"us\": {" + row +
                  "}, \"lanes\": " + std::to_string(best) + ", \"seg\": " + std::to_string(best_seg) + "}";
        first = false;
      }
    }
  } catch (...) {
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    throw;
  }
  report += "]";
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  EK_CUDA(cudaStreamSynchronize(s));
  return EK_OK;
}

}  // namespace ek
