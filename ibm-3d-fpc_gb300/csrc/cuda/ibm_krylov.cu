// Restarted, right-preconditioned GMRES for up to kMaxSys independent 7-point
// systems at once, with every scalar kept on the device.
//
// Restates the algorithm of HYPRE_StructGMRESSolve (third-party, called by
// the reference at main.cu:284-286 and 327): Arnoldi with Givens rotations,
// stop when the estimated ||r||/||b|| <= tol, confirm with the true residual
// and restart from it; a cycle whose estimate claimed convergence but whose
// true residual did not decrease stops (stagnation), as HYPRE does.
// Orthogonalisation is classical Gram-Schmidt applied twice, so each pass is
// one sweep over the basis with all dot products batched.
//
// Per Arnoldi step, three streaming kernels:
//   k_arnoldi_spmv : w = A z_j and d1_k = (v_k, w)         (last block: h1, coefficients)
//   k_arnoldi_orth : w -= V c1, d2_k = (v_k, w)              (last block: h2, Hessenberg column)
//   k_arnoldi_next : v_{j+1} = w - V c2, |v_{j+1}|^2          (last block: Givens, stop test)
// Basis vectors are stored unnormalised with their exact norms in nu[].
// Reductions are deterministic: fixed per-warp order inside a block, block
// partials summed in block order by the last block to finish.
#include <algorithm>

#include "ibm_common.cuh"
#include "ibm_krylov.cuh"
#include "ibm_df.cuh"

namespace ibm {

namespace {

constexpr int kLd = kMaxKdim + 2;  // stride of block partials
constexpr int kChunk32 = 8;  // basis vectors whose dot products a thread keeps in registers

// Flat row -> (i, j, k) of a system's box (invariant-divisor division).
__device__ __forceinline__ void sys_ijk(long r, const KSys &S, int &i, int &j, int &k) {
  const unsigned q = fast_div((unsigned)r, S.fdx);
  i = (int)((unsigned)r - q * (unsigned)S.nx);
  const unsigned kk = fast_div(q, S.fdy);
  j = (int)(q - kk * (unsigned)S.ny);
  k = (int)kk;
}

// Slot 0 of row r of Ar and the distance between its slots: the row of the
// row's class, or the planes.
__device__ __forceinline__ const double *ar_row(const KSys &S, long r, long &cs) {
  if (S.cls) { cs = 1; return S.tab + 8 * (long)S.cls[r]; }
  cs = S.n;
  return S.Ar + r;
}
// The same for the Arnoldi operator A (classed only when A is Ar).
__device__ __forceinline__ const double *a_row(const KSys &S, long r, long &cs) {
  if (S.cls && S.A == S.Ar) { cs = 1; return S.tab + 8 * (long)S.cls[r]; }
  cs = S.n;
  return S.A + r;
}
// ... and for Af, the FP32 copy of Ar.
__device__ __forceinline__ const float *af_row(const KSys &S, long r, long &cs) {
  if (S.cls) { cs = 1; return S.tabf + 8 * (long)S.cls[r]; }
  cs = S.n;
  return S.Af + r;
}

// Four class-table rows (8 floats each) as four 16-byte pairs, transposed so
// that cp[s] holds slot s of the four rows.
__device__ __forceinline__ void load_rows4(const float *__restrict__ tab, ushort4 c4, float4 (&cp)[7]) {
  const unsigned short ks[4] = {c4.x, c4.y, c4.z, c4.w};
  float v[4][8];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float4 *p = reinterpret_cast<const float4 *>(tab + 8 * (long)ks[q]);
    const float4 a = __ldg(p), b = __ldg(p + 1);
    v[q][0] = a.x; v[q][1] = a.y; v[q][2] = a.z; v[q][3] = a.w;
    v[q][4] = b.x; v[q][5] = b.y; v[q][6] = b.z; v[q][7] = b.w;
  }
#pragma unroll
  for (int s = 0; s < 7; ++s) cp[s] = make_float4(v[0][s], v[1][s], v[2][s], v[3][s]);
}

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }
__device__ __forceinline__ float f4(const float4 &v, int q) { return q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w; }

// Rows r0 .. r0 + 3 (r0 a multiple of 4) with the values of an FP32 vector
// there and around, 0 outside the box.
struct QuadRows {
  float4 c, w, e, s, n, b, t;  // the rows; their neighbours at x -+ 1, y -+ 1, z -+ 1
};
// LINE: nx is a multiple of 4, the rows are of one line: seven loads instead
// of 28. Else only n is: the rows may go over to the next line (and plane), and
// lines start anywhere, so the y neighbours are single loads.
template <bool LINE>
__device__ __forceinline__ QuadRows load_quad_rows(const KSys &S, const float *z, long r0) {
  int i, j, k;
  sys_ijk(r0, S, i, j, k);
  const int nx = S.nx, ny = S.ny, nz = S.nz;
  const long sy = nx, sz = (long)nx * ny;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  QuadRows q;
  q.c = ld4(z + r0);
  if constexpr (LINE) {
    q.s = j > 0 ? ld4(z + r0 - sy) : z4;
    q.n = j < ny - 1 ? ld4(z + r0 + sy) : z4;
    q.b = k > 0 ? ld4(z + r0 - sz) : z4;
    q.t = k < nz - 1 ? ld4(z + r0 + sz) : z4;
    const float l = i > 0 ? z[r0 - 1] : 0.0f, r = i + 4 < nx ? z[r0 + 4] : 0.0f;
    q.w = make_float4(l, q.c.x, q.c.y, q.c.z);
    q.e = make_float4(q.c.y, q.c.z, q.c.w, r);
  } else {
    const float c[4] = {q.c.x, q.c.y, q.c.z, q.c.w};
    float w[4], e[4], s[4], n[4], b[4], t[4];
    const bool vec = (sz & 3) == 0;
    const bool over = i + 3 >= nx && j == ny - 1;  // the last rows are of the next plane
    const bool below = vec && k > 0, above = vec && (over ? k + 1 : k) < nz - 1;
    if (below) q.b = ld4(z + r0 - sz);
    if (above) q.t = ld4(z + r0 + sz);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool wrap = i + u >= nx;
      const int iu = wrap ? i + u - nx : i + u, j1 = wrap ? j + 1 : j;
      const int ju = j1 == ny ? 0 : j1, ku = j1 == ny ? k + 1 : k;
      const long r = r0 + u;
      w[u] = iu > 0 ? (u > 0 ? c[u > 0 ? u - 1 : 0] : z[r - 1]) : 0.0f;
      e[u] = iu < nx - 1 ? (u < 3 ? c[u < 3 ? u + 1 : 3] : z[r + 1]) : 0.0f;
      s[u] = ju > 0 ? z[r - sy] : 0.0f;
      n[u] = ju < ny - 1 ? z[r + sy] : 0.0f;
      if (!below) b[u] = ku > 0 ? z[r - sz] : 0.0f;
      if (!above) t[u] = ku < nz - 1 ? z[r + sz] : 0.0f;
    }
    q.w = make_float4(w[0], w[1], w[2], w[3]);
    q.e = make_float4(e[0], e[1], e[2], e[3]);
    q.s = make_float4(s[0], s[1], s[2], s[3]);
    q.n = make_float4(n[0], n[1], n[2], n[3]);
    if (!below) q.b = make_float4(b[0], b[1], b[2], b[3]);
    if (!above) q.t = make_float4(t[0], t[1], t[2], t[3]);
  }
  return q;
}
// whether all four codes are `major`
__device__ __forceinline__ bool all_major(ushort4 c, int major) {
  return c.x == major && c.y == major && c.z == major && c.w == major;
}
// A z of one row in FP32, slot order; c[s] the row's slots.
__device__ __forceinline__ float quad_row32(const QuadRows &v, int q, float c0, float c1, float c2, float c3, float c4,
                                            float c5, float c6) {
  float a = 0.0f;
  a = fmaf(c0, f4(v.c, q), a);
  a = fmaf(c1, f4(v.w, q), a);
  a = fmaf(c2, f4(v.e, q), a);
  a = fmaf(c3, f4(v.s, q), a);
  a = fmaf(c4, f4(v.n, q), a);
  a = fmaf(c5, f4(v.b, q), a);
  a = fmaf(c6, f4(v.t, q), a);
  return a;
}
// ... in double-float (hi: slots 0 .. 6, lo: 8 .. 14 of c), widened once.
template <class C>
__device__ __forceinline__ double quad_row_df(const QuadRows &v, int q, const C &c) {
  float ah = 0.0f, al = 0.0f;
  df_fma1(ah, al, c[0], c[8], f4(v.c, q));
  df_fma1(ah, al, c[1], c[9], f4(v.w, q));
  df_fma1(ah, al, c[2], c[10], f4(v.e, q));
  df_fma1(ah, al, c[3], c[11], f4(v.s, q));
  df_fma1(ah, al, c[4], c[12], f4(v.n, q));
  df_fma1(ah, al, c[5], c[13], f4(v.b, q));
  df_fma1(ah, al, c[6], c[14], f4(v.t, q));
  return widen(ah) + widen(al);
}

// Sum block partials of `nd` dot products in block order; one warp per dot.
__device__ void reduce_partials(const double *part, int nblk, int nd, double *out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int k = warp; k < nd; k += kWarps) {
    double s = 0.0;
    for (int b = lane; b < nblk; b += 32) s += part[(long)b * kLd + k];
    s = warp_sum(s);
    if (lane == 0) out[k] = s;
  }
}

// Common tail of the reduction kernels: write this block's sums, and return
// true in the block that finishes last (after all partials are visible).
__device__ bool block_partials_and_last(double *sacc, int nd, double *part, unsigned *ticket) {
  __syncthreads();
  for (int k = threadIdx.x; k < nd; k += blockDim.x) {
    double s = 0.0;
    for (int w = 0; w < kWarps; ++w) s += sacc[k * kWarps + w];
    part[(long)blockIdx.x * kLd + k] = s;
  }
  __threadfence();
  __syncthreads();
  __shared__ int last;
  if (threadIdx.x == 0) last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
  __syncthreads();
  if (last) __threadfence();
  return last != 0;
}

// pc 1 keeps a cycle's preconditioned directions M V_k, as the flexible form
// does, so that the update is x += sum c_k M V_k and not M (V c): one V-cycle
// less per GMRES cycle (six instead of seven for a solve of six iterations; FP64
// step 640x128x128 36.8 -> 34.7 ms, 160x32x32 4.58 -> 4.24). They take no memory of
// their own. The first nlent lie in another solver's basis that is idle meanwhile
// (the momentum systems': with the default restart lengths all of them), from its
// end down, which that solver's own cycles seldom reach; the next ones in the
// vectors of V that the cycle does not reach, from vector kdim + 1 down. A cycle
// longer than nkept iterations has its basis run over these; its later directions
// go to the spare vector kdim + 1 one after the other, and its end takes V c there
// and applies the preconditioner to it, into vector kdim.
__device__ __forceinline__ double *direction_of(const KSys &S, int k, int kdim) {
  if (k < S.nlent) return S.lent - (long)k * S.ldv;
  return S.V + (long)(kdim + 1 - (k < S.nkept ? k - S.nlent : 0)) * S.ldv;
}
// The most directions that a cycle can keep: vectors 0 .. m of V are its basis
// (the last only for m < kdim), m - lent of kdim + 2 above them directions.
int kept_directions(int kdim, int lent) {
  return lent >= kdim - 2 ? kdim : std::min(kdim - 1, (kdim + 1 + lent) / 2);
}
// Whether a system's finished cycle applies the preconditioner at its end.
__device__ __forceinline__ bool end_applies(const KSys &S) { return S.pc == 1 && S.s->i > S.nkept; }
// The next V-cycle: of Arnoldi step i; of a finished cycle's V c.
__device__ __forceinline__ void pc_of_step(const KSys &S, int i, int kdim, int on) {
  if (S.pc != 1) return;
  S.s->pc_in = S.V + (long)i * S.ldv;
  S.s->pc_out = direction_of(S, i, kdim);
  S.s->pc_on = on;
}
__device__ __forceinline__ void pc_of_end(const KSys &S) {
  S.s->pc_in = S.V + (long)(S.s->kdim + 1) * S.ldv;
  S.s->pc_out = S.V + (long)S.s->kdim * S.ldv;
  S.s->pc_on = 2;
}

// r = b - Ar x; V_0 = r; |b|^2, |r|^2. Last block: norms, tolerance, state.
__global__ void __launch_bounds__(kThreads) k_init(const __grid_constant__ KSysPack P) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  __shared__ double sacc[2 * kWarps];
  if (threadIdx.x < 2 * kWarps) sacc[threadIdx.x] = 0.0;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // per-thread sums over all of the thread's rows, one warp reduction at the
  // end (GB300's FP64 pipe is the bound here: no FP64 work per tile)
  double pb = 0.0, pr = 0.0;
  if (S.a32 && S.x_zero) {
    // r = b: the FP32 basis vector from the bits of b (integer split, one FP32
    // add: b rounded to FP32), |b|^2 in FP32 per thread; no FP64 instruction
    float pf = 0.0f;
    for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
#pragma unroll
      for (int t = 0; t < kRowsPerThread; ++t) {
        const long r = t0 + t * kThreads + threadIdx.x;
        if (r < S.n) {
          float bh, bl;
          df_split(S.b[r], bh, bl);
          const float v = __fadd_rn(bh, bl);
          S.Vf[r] = v;
          pf = fmaf(v, v, pf);
        }
      }
    }
    pb = pr = (double)pf;
  } else {
    for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
#pragma unroll
      for (int t = 0; t < kRowsPerThread; ++t) {
        const long r = t0 + t * kThreads + threadIdx.x;
        if (r < S.n) {
          int i, j, k;
          sys_ijk(r, S, i, j, k);
          // with finite coefficients A 0 is +0 in every row, so b - 0 equals b - A x
          // bit for bit: a zero guess takes r = b and |r| = |b|
          const double bv = S.b[r];
          double rv = bv;
          if (!S.x_zero) {
            long cs;
            const double *c0 = ar_row(S, r, cs);
            rv = bv - stencil7_at(c0, cs, S.x, (int)r, i, j, k, S.nx, S.ny, S.nz);
            pr = fma(rv, rv, pr);
          }
          if (S.a32) S.Vf[r] = narrow(rv);
          else S.V[r] = rv;
          if (S.vcur) S.vcur[r] = narrow(rv);
          pb = fma(bv, bv, pb);
        }
      }
    }
    if (S.x_zero) pr = pb;
  }
  pb = warp_sum(pb);
  pr = warp_sum(pr);
  if (lane == 0) { sacc[warp] = pb; sacc[kWarps + warp] = pr; }
  if (!block_partials_and_last(sacc, 2, S.part, &sc->ticket)) return;
  __shared__ double tot[2];
  reduce_partials(S.part, gridDim.x, 2, tot);
  __syncthreads();
  if (threadIdx.x == 0) {
    sc->ticket = 0;
    const double bn = sqrt(tot[0]), rn = sqrt(tot[1]);
    sc->b_norm = bn;
    sc->r_norm = rn;
    sc->eps = sc->tol * (bn > 0.0 ? bn : rn);
    sc->cyc_eps = fmax(sc->eps, sc->cyc_rtol * rn);
    sc->real_old = bn;
    sc->iters = 0;
    sc->i = 0;
    sc->claimed = 0;
    sc->cycle_end = 0;
    sc->nonfinite = !isfinite(rn);
    sc->use64 = 0;
    if (!isfinite(rn)) { sc->status = 2; sc->active = 0; }
    else if (rn == 0.0 || rn <= sc->eps) { sc->status = 1; sc->active = 0; }
    else if (sc->maxit <= 0) { sc->status = 2; sc->active = 0; }
    else { sc->status = 0; sc->active = 1; }
    pc_of_step(S, 0, sc->kdim, sc->active);
    sc->nu[0] = rn;
    sc->inu[0] = 1.0 / rn;
    sc->g[0] = rn;
  }
}

// Closes Arnoldi step j: h(j+1,j) = |v_{j+1}| = hn, the previous rotations
// applied to the new Hessenberg column, a new Givens rotation, the residual
// estimate and the stop tests; at the end of a cycle the back-substitution
// H y = g and the update coefficients y / nu. Called by every thread of the
// last block: what the serial part needs is loaded into shared memory by as
// many threads at once (one memory latency each for the column and, at a
// cycle's end, the triangle), and one thread then works there. One thread
// walking global memory paid a latency per rotation and per matrix entry.
__device__ void arnoldi_finalize(const KSys &S, int j, double hn) {
  KScal *sc = S.s;
  constexpr int K = kMaxKdim;
  __shared__ double col[K + 1], rc[K], rs[K], tri[K * (K + 1) / 2];
  __shared__ int ended;
  const int tid = threadIdx.x;
  const double gj = sc->g[j], eps = sc->eps, cyc_eps = sc->cyc_eps;
  const int kdim = sc->kdim, iters = sc->iters + 1, maxit = sc->maxit, m = j + 1;
  for (int q = tid; q <= j; q += blockDim.x) {
    col[q] = sc->H[q * K + j];
    if (q < j) { rc[q] = sc->cs[q]; rs[q] = sc->sn[q]; }
  }
  __syncthreads();
  if (tid == 32) {
    sc->nu[j + 1] = hn;
    sc->inu[j + 1] = 1.0 / hn;
  }
  if (tid == 0) {
    double a = col[0];
    for (int q = 0; q < j; ++q) {
      const double t = a, h = col[q + 1];
      col[q] = rs[q] * h + rc[q] * t;
      a = -rs[q] * t + rc[q] * h;
    }
    const double b = hn;
    double gam = sqrt(b * b + a * a);
    if (gam == 0.0) gam = 2.220446049250313e-16;
    const double c = a / gam, s = b / gam;
    const double gn = -s * gj;
    const double r_norm = fabs(gn);
    col[j] = s * b + c * a;
    rc[0] = c * gj;  // the rotated g_j
    sc->cs[j] = c;
    sc->sn[j] = s;
    sc->g[j + 1] = gn;
    sc->g[j] = c * gj;
    sc->i = m;
    sc->iters = iters;
    sc->r_norm = r_norm;
    const bool claimed = r_norm <= eps || hn == 0.0;
    const bool cycle_done = r_norm <= cyc_eps;
    if (!isfinite(r_norm)) sc->nonfinite = 1;
    const bool end = claimed || cycle_done || m >= kdim || iters >= maxit || !isfinite(r_norm);
    if (end) {
      sc->claimed = claimed;
      sc->active = 0;
      sc->cycle_end = 1;
    }
    pc_of_step(S, m, kdim, end ? 0 : 1);
    ended = end;
  }
  __syncthreads();
  for (int q = tid; q <= j; q += blockDim.x) sc->H[q * K + j] = col[q];
  if (!ended) return;
  // column c of the triangle at tri[c (c + 1) / 2]; the last column is col
  double *y = rs;  // the rotations' sines are not needed any more
  for (int e = tid; e < j * K; e += blockDim.x) {
    const int c = e / K, q = e - c * K;
    if (q <= c) tri[c * (c + 1) / 2 + q] = sc->H[q * K + c];
  }
  for (int q = tid; q < j; q += blockDim.x) y[q] = sc->g[q];
  if (tid == 0) y[j] = rc[0];
  for (int q = tid; q <= j; q += blockDim.x) tri[j * (j + 1) / 2 + q] = col[q];
  __syncthreads();
  if (tid == 0) {
    for (int q = m - 1; q >= 0; --q) {
      double t = y[q];
      for (int c = q + 1; c < m; ++c) t -= tri[c * (c + 1) / 2 + q] * y[c];
      y[q] = t / tri[q * (q + 1) / 2 + q];
    }
  }
  __syncthreads();
  for (int q = tid; q < m; q += blockDim.x) {
    sc->y[q] = y[q];
    sc->coef[q] = y[q] / sc->nu[q];
  }
}

// The FP64 Arnoldi kernels take their dot products kDots64 basis vectors at a
// time: each stays a per-thread sum over all the thread's rows and is reduced
// across the warp once per kernel. A longer basis takes further passes over
// the rows that read w back (8 bytes a row beside the 64 of the eight basis
// vectors); reducing across the warp for each tile of rows, as a loop over all
// vectors per tile would have to, costs as many FP64 issue slots as the
// products.
constexpr int kDots64 = 8;

// Sums of the N values of pd over the warp: value k in lanes with lane / (32 / N) == k.
// Halves are exchanged, so a lane adds N/2 + N/4 + ... + 1 + log2(32 / N)
// times (9 for N = 8) instead of 5 N: GB300 issues two FP64 operations per
// clock and SM, and eight five-step butterflies in each of 32 warps took 10 us
// of every launch.
template <int N>
__device__ __forceinline__ double warp_sums(double (&pd)[N], int lane) {
  int o = 16;
#pragma unroll
  for (int h = N / 2; h > 0; h >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < h; ++k) {
      const double send = up ? pd[k] : pd[k + h], keep = up ? pd[k + h] : pd[k];
      pd[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double v = pd[0];
  for (; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Adds the block's nd <= kDots64 sums of this pass to sacc[kk * kWarps + warp].
__device__ __forceinline__ void flush_dots64(double (&pd)[kDots64], int nd, double *sacc, int warp, int lane) {
  if (nd == 1) {
    const double v = warp_sum(pd[0]);
    if (lane == 0) sacc[warp] = v;
  } else if (nd <= 4) {
    double q[4] = {pd[0], pd[1], pd[2], pd[3]};
    const double v = warp_sums<4>(q, lane);
    const int k = lane >> 3;
    if ((lane & 7) == 0 && k < nd) sacc[k * kWarps + warp] = v;
  } else {
    const double v = warp_sums<8>(pd, lane);
    const int k = lane >> 2;
    if ((lane & 3) == 0 && k < nd) sacc[k * kWarps + warp] = v;
  }
}

// Row r of w = A z_j. Mode 0: z_j in double-float from the class table; 1: A
// applied to the FP64 vector z times inv_nu (folded Jacobi, or the explicit
// z); 2: A applied to the FP32 direction z_j.
template <int MODE>
__device__ __forceinline__ double spmv_row64(const KSys &S, long r, const double *z, const float *zj, double inv_nu) {
  int i, jj, k;
  sys_ijk(r, S, i, jj, k);
  if constexpr (MODE == 0) {
    // the seven products and their sum in double-float, widened once (two
    // conversions and one FP64 add); a neighbour outside the box reads as 0:
    // its product and sum are exact no-ops, so all seven loads issue together
    const float4 *c4 = reinterpret_cast<const float4 *>(S.tabdf + 16 * (long)S.cls[r]);
    const long sy = S.nx, sz = (long)S.nx * S.ny;
    const float z0 = zj[r], zxm = i > 0 ? zj[r - 1] : 0.0f, zxp = i < S.nx - 1 ? zj[r + 1] : 0.0f,
                zym = jj > 0 ? zj[r - sy] : 0.0f, zyp = jj < S.ny - 1 ? zj[r + sy] : 0.0f,
                zzm = k > 0 ? zj[r - sz] : 0.0f, zzp = k < S.nz - 1 ? zj[r + sz] : 0.0f;
    const float4 h0 = __ldg(c4), h1 = __ldg(c4 + 1), l0 = __ldg(c4 + 2), l1 = __ldg(c4 + 3);
    float ah = 0.0f, al = 0.0f;
    df_fma1(ah, al, h0.x, l0.x, z0);
    df_fma1(ah, al, h0.y, l0.y, zxm);
    df_fma1(ah, al, h0.z, l0.z, zxp);
    df_fma1(ah, al, h0.w, l0.w, zym);
    df_fma1(ah, al, h1.x, l1.x, zyp);
    df_fma1(ah, al, h1.y, l1.y, zzm);
    df_fma1(ah, al, h1.z, l1.z, zzp);
    return widen(ah) + widen(al);
  } else {
    long cs;
    const double *c0 = a_row(S, r, cs);
    if constexpr (MODE == 1) return stencil7_at(c0, cs, z, (int)r, i, jj, k, S.nx, S.ny, S.nz) * inv_nu;
    else return stencil7_at(c0, cs, zj, (int)r, i, jj, k, S.nx, S.ny, S.nz);
  }
}

// The rows of w = A z_j and their dot products with basis vectors c0 ..
// c0 + nd - 1. The rows of a tile are computed before any is stored, so that
// their loads are in flight together (a store between them would hold the
// later ones back); later passes (c0 > 0) read w.
template <int MODE>
__device__ __forceinline__ void spmv_pass64(const KSys &S, const double *z, const float *zj, double inv_nu, int c0,
                                            int nd, double (&pd)[kDots64]) {
  for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
    double wv[kRowsPerThread];
#pragma unroll
    for (int t = 0; t < kRowsPerThread; ++t) {
      const long r = t0 + t * kThreads + threadIdx.x;
      wv[t] = 0.0;
      if (r < S.n) wv[t] = c0 ? S.w[r] : spmv_row64<MODE>(S, r, z, zj, inv_nu);
    }
    if (c0 == 0) {
#pragma unroll
      for (int t = 0; t < kRowsPerThread; ++t) {
        const long r = t0 + t * kThreads + threadIdx.x;
        if (r < S.n) S.w[r] = wv[t];
      }
    }
#pragma unroll
    for (int kk = 0; kk < kDots64; ++kk) {
      if (kk >= nd) break;
      const double *vk = S.V + (long)(c0 + kk) * S.ldv;
#pragma unroll
      for (int t = 0; t < kRowsPerThread; ++t) {
        const long r = t0 + t * kThreads + threadIdx.x;
        if (r < S.n) pd[kk] = fma(vk[r], wv[t], pd[kk]);
      }
    }
  }
}

// spmv_pass64<0> with four consecutive rows per thread (S.quad). The rows of
// most quads are all of the major class: their 14 values come from constant
// memory. Bound: HBM (34 bytes a row at a basis of 2.5 vectors) next to FP64
// issue (one add and nd FMAs a row). One row at a time, with two conversion
// instructions a row, 28 loads for four rows and four 16-byte table loads for
// each, a launch over 3 x 10.5M rows took 371 us, now 353: the v and w rows go
// in quads, and the u rows (an odd number a line) set the time.
__device__ __forceinline__ void spmv_pass64_quad(const KSys &S, const float *zj, int c0, int nd,
                                                 double (&pd)[kDots64]) {
  for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
    const long r0 = t0 + 4 * threadIdx.x;
    if (r0 >= S.n) continue;
    double w[4];
    if (c0 == 0) {
      const ushort4 c4 = __ldcs(reinterpret_cast<const ushort4 *>(S.cls + r0));
      const QuadRows v = load_quad_rows<true>(S, zj, r0);
      if (all_major(c4, S.major)) {
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = quad_row_df(v, q, S.udf);
      } else {
        const unsigned short ks[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 *p = reinterpret_cast<const float4 *>(S.tabdf + 16 * (long)ks[q]);
          const float4 h0 = __ldg(p), h1 = __ldg(p + 1), l0 = __ldg(p + 2), l1 = __ldg(p + 3);
          const float c[16] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w,
                               l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
          w[q] = quad_row_df(v, q, c);
        }
      }
      *reinterpret_cast<double2 *>(S.w + r0) = make_double2(w[0], w[1]);
      *reinterpret_cast<double2 *>(S.w + r0 + 2) = make_double2(w[2], w[3]);
    } else {
      const double2 a = *reinterpret_cast<const double2 *>(S.w + r0), b = *reinterpret_cast<const double2 *>(S.w + r0 + 2);
      w[0] = a.x; w[1] = a.y; w[2] = b.x; w[3] = b.y;
    }
#pragma unroll
    for (int kk = 0; kk < kDots64; ++kk) {
      if (kk >= nd) break;
      const double *vk = S.V + (long)(c0 + kk) * S.ldv + r0;
      const double2 a = *reinterpret_cast<const double2 *>(vk), b = *reinterpret_cast<const double2 *>(vk + 2);
      pd[kk] = fma(a.x, w[0], pd[kk]);
      pd[kk] = fma(a.y, w[1], pd[kk]);
      pd[kk] = fma(b.x, w[2], pd[kk]);
      pd[kk] = fma(b.y, w[3], pd[kk]);
    }
  }
}

// w = A z_j (z_j = M v_j by the system's preconditioner mode), d1_k = (V_k, w).
__global__ void __launch_bounds__(kThreads, 4) k_arnoldi_spmv(const __grid_constant__ KSysPack P) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  if (!sc->active || S.a32) return;
  const int j = sc->i, nd = j + 1;
  const double inv_nu = sc->inu[j];
  __shared__ double sacc[(kMaxKdim + 1) * kWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double *z = S.pc == 1 ? sc->pc_out : S.V + (long)j * S.ldv;
  const float *zj = S.Z + (long)j * S.ldv;
  for (int c0 = 0; c0 < nd; c0 += kDots64) {
    const int ndc = min(nd - c0, kDots64);
    double pd[kDots64];
#pragma unroll
    for (int kk = 0; kk < kDots64; ++kk) pd[kk] = 0.0;
    if (S.df_spmv && S.quad == 1) spmv_pass64_quad(S, zj, c0, ndc, pd);
    else if (S.df_spmv) spmv_pass64<0>(S, z, zj, inv_nu, c0, ndc, pd);
    else if (S.pc != 2) spmv_pass64<1>(S, z, zj, inv_nu, c0, ndc, pd);
    else spmv_pass64<2>(S, z, zj, inv_nu, c0, ndc, pd);
    flush_dots64(pd, ndc, sacc + c0 * kWarps, warp, lane);
  }
  if (!block_partials_and_last(sacc, nd, S.part, &sc->ticket)) return;
  __shared__ double tot[kMaxKdim + 1];
  reduce_partials(S.part, gridDim.x, nd, tot);
  __syncthreads();
  for (int kk = threadIdx.x; kk < nd; kk += blockDim.x) {
    const double h = tot[kk] / sc->nu[kk];
    sc->h1[kk] = h;
    sc->coef[kk] = h / sc->nu[kk];
    if (S.cgs1) sc->H[kk * kMaxKdim + j] = h;  // one pass: the column is the first projection
  }
  if (threadIdx.x == 0) sc->ticket = 0;
}

// w - sum_k cf_k V_k for the rows of one tile of a thread, each row's terms in
// order of k; the rows' loads of a basis vector are in flight together.
__device__ __forceinline__ void orth_rows64(const KSys &S, long t0, const double *cf, int nd,
                                            double (&wv)[kRowsPerThread]) {
#pragma unroll
  for (int t = 0; t < kRowsPerThread; ++t) {
    const long r = t0 + t * kThreads + threadIdx.x;
    wv[t] = r < S.n ? S.w[r] : 0.0;
  }
#pragma unroll 2
  for (int kk = 0; kk < nd; ++kk) {
    const double *vk = S.V + (long)kk * S.ldv;
    const double c = -cf[kk];
#pragma unroll
    for (int t = 0; t < kRowsPerThread; ++t) {
      const long r = t0 + t * kThreads + threadIdx.x;
      if (r < S.n) wv[t] = fma(c, vk[r], wv[t]);
    }
  }
}

// w -= sum_k coef_k V_k (first pass), d2_k = (V_k, w). Last block: the
// second-pass coefficients and the Hessenberg column above the diagonal.
__global__ void __launch_bounds__(kThreads) k_arnoldi_orth(const __grid_constant__ KSysPack P) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  if (!sc->active || S.a32 || S.cgs1) return;
  const int j = sc->i, nd = j + 1;
  __shared__ double sacc[(kMaxKdim + 1) * kWarps];
  __shared__ double cf[kMaxKdim + 1];
  for (int t = threadIdx.x; t < nd; t += blockDim.x) cf[t] = sc->coef[t];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c0 = 0; c0 < nd; c0 += kDots64) {
    const int ndc = min(nd - c0, kDots64);
    double pd[kDots64];
#pragma unroll
    for (int kk = 0; kk < kDots64; ++kk) pd[kk] = 0.0;
    for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
      double wv[kRowsPerThread];
      if (c0 == 0) {
        orth_rows64(S, t0, cf, nd, wv);
#pragma unroll
        for (int t = 0; t < kRowsPerThread; ++t) {
          const long r = t0 + t * kThreads + threadIdx.x;
          if (r < S.n) S.w[r] = wv[t];
        }
      } else {
#pragma unroll
        for (int t = 0; t < kRowsPerThread; ++t) {
          const long r = t0 + t * kThreads + threadIdx.x;
          wv[t] = r < S.n ? S.w[r] : 0.0;
        }
      }
#pragma unroll
      for (int kk = 0; kk < kDots64; ++kk) {
        if (kk >= ndc) break;
        const double *vk = S.V + (long)(c0 + kk) * S.ldv;
#pragma unroll
        for (int t = 0; t < kRowsPerThread; ++t) {
          const long r = t0 + t * kThreads + threadIdx.x;
          if (r < S.n) pd[kk] = fma(vk[r], wv[t], pd[kk]);
        }
      }
    }
    flush_dots64(pd, ndc, sacc + c0 * kWarps, warp, lane);
  }
  if (!block_partials_and_last(sacc, nd, S.part, &sc->ticket)) return;
  __shared__ double tot[kMaxKdim + 1];
  reduce_partials(S.part, gridDim.x, nd, tot);
  __syncthreads();
  for (int kk = threadIdx.x; kk < nd; kk += blockDim.x) {
    const double h2 = tot[kk] / sc->nu[kk];
    sc->coef[kk] = h2 / sc->nu[kk];
    sc->H[kk * kMaxKdim + j] = sc->h1[kk] + h2;
  }
  if (threadIdx.x == 0) sc->ticket = 0;
}

// v_{j+1} = w - sum_k coef_k V_k, stored unnormalised, with its exact norm.
// Last block: Hessenberg column, Givens rotation, stop test, and at the end
// of a cycle the back substitution.
__global__ void __launch_bounds__(kThreads) k_arnoldi_next(const __grid_constant__ KSysPack P) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  if (!sc->active || S.a32) return;
  const int j = sc->i, nd = j + 1;
  __shared__ double cf[kMaxKdim + 1];
  __shared__ double sacc[kWarps];
  for (int t = threadIdx.x; t < nd; t += blockDim.x) cf[t] = sc->coef[t];
  if (threadIdx.x < kWarps) sacc[threadIdx.x] = 0.0;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *vn = S.V + (long)nd * S.ldv;
  const bool store = nd < sc->kdim;  // the last vector of a full cycle is never used
  double p = 0.0;  // per thread over all its rows
  for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
    double wv[kRowsPerThread];
    orth_rows64(S, t0, cf, nd, wv);
#pragma unroll
    for (int t = 0; t < kRowsPerThread; ++t) {
      const long r = t0 + t * kThreads + threadIdx.x;
      if (r < S.n) {
        if (store) {
          vn[r] = wv[t];
          if (S.vcur) S.vcur[r] = narrow(wv[t]);
        }
        p = fma(wv[t], wv[t], p);
      }
    }
  }
  p = warp_sum(p);
  if (lane == 0) sacc[warp] = p;
  if (!block_partials_and_last(sacc, 1, S.part, &sc->ticket)) return;
  __shared__ double tot[1];
  reduce_partials(S.part, gridDim.x, 1, tot);
  __syncthreads();
  if (threadIdx.x == 0) sc->ticket = 0;
  arnoldi_finalize(S, j, sqrt(tot[0]));
}

// Cycle end, solution update. pc 0: x += invd * (V c); pc 1: x += sum of c_k
// times direction k, or where the cycle outgrew them (end_applies) V c is left
// for the preconditioner, and x += M (V c) once that has run; pc 2: x += Z y.
__global__ void __launch_bounds__(kThreads) k_cycle_update(const __grid_constant__ KSysPack P) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  if (!sc->cycle_end) return;
  const int m = sc->i;
  __shared__ double cf[kMaxKdim + 1];
  for (int t = threadIdx.x; t < m; t += blockDim.x) cf[t] = S.pc == 2 ? sc->y[t] : sc->coef[t];
  __syncthreads();
  if (S.a32) {
    // FP32 cycles: the correction sum Z y is formed in FP32 (its rounding is
    // far below what the cycle resolved; the restart measures the true
    // residual of the FP64 x) and added to x in FP64
    __shared__ float cf32[kMaxKdim + 1];
    for (int t = threadIdx.x; t < m; t += blockDim.x) cf32[t] = (float)cf[t];
    __syncthreads();
    if (S.vec4 && m <= kChunk32) {
      // four consecutive rows per thread: 16-byte loads of the directions,
      // every load of the thread in flight together; same sums row by row
      for (long r0 = 4 * ((long)blockIdx.x * blockDim.x + threadIdx.x); r0 < S.n;
           r0 += 4L * gridDim.x * blockDim.x) {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int kk = 0; kk < kChunk32; ++kk) {
          if (kk < m) {
            const float4 z = *reinterpret_cast<const float4 *>(S.Z + (long)kk * S.ldv + r0);
            acc.x = fmaf(cf32[kk], z.x, acc.x);
            acc.y = fmaf(cf32[kk], z.y, acc.y);
            acc.z = fmaf(cf32[kk], z.z, acc.z);
            acc.w = fmaf(cf32[kk], z.w, acc.w);
          }
        }
        const double2 x01 = *reinterpret_cast<const double2 *>(S.x + r0);
        const double2 x23 = *reinterpret_cast<const double2 *>(S.x + r0 + 2);
        const double xn[4] = {x01.x + (double)acc.x, x01.y + (double)acc.y, x23.x + (double)acc.z,
                              x23.y + (double)acc.w};
        *reinterpret_cast<double2 *>(S.x + r0) = make_double2(xn[0], xn[1]);
        *reinterpret_cast<double2 *>(S.x + r0 + 2) = make_double2(xn[2], xn[3]);
        if (S.df_resid) {
          float h[4], l[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) df_split(xn[q], h[q], l[q]);
          *reinterpret_cast<float4 *>(S.xs + r0) = make_float4(h[0], l[0], h[1], l[1]);
          *reinterpret_cast<float4 *>(S.xs + r0 + 2) = make_float4(h[2], l[2], h[3], l[3]);
        }
      }
      return;
    }
    for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < S.n; r += (long)gridDim.x * blockDim.x) {
      float acc = 0.0f;
      for (int kk = 0; kk < m; ++kk) acc = fmaf(cf32[kk], S.Z[(long)kk * S.ldv + r], acc);
      const double xn = S.x[r] + (double)acc;
      S.x[r] = xn;
      if (S.df_resid) {
        float h, l;
        df_split(xn, h, l);
        S.xs[r] = make_float2(h, l);
      }
    }
    return;
  }
  if (S.pc == 2 && S.vec4) {
    // four consecutive rows per thread; the directions widened on the integer
    // pipe (the conversions took as many FP64 issue slots as the sums: 550 us
    // over 3 x 10.5M rows and three to four directions, now 303)
    for (long r0 = 4 * ((long)blockIdx.x * blockDim.x + threadIdx.x); r0 < S.n; r0 += 4L * gridDim.x * blockDim.x) {
      const double2 x01 = *reinterpret_cast<const double2 *>(S.x + r0);
      const double2 x23 = *reinterpret_cast<const double2 *>(S.x + r0 + 2);
      double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
      for (int kk = 0; kk < m; ++kk) {
        const float4 z = ld4(S.Z + (long)kk * S.ldv + r0);
        a[0] = fma(cf[kk], widen(z.x), a[0]);
        a[1] = fma(cf[kk], widen(z.y), a[1]);
        a[2] = fma(cf[kk], widen(z.z), a[2]);
        a[3] = fma(cf[kk], widen(z.w), a[3]);
      }
      *reinterpret_cast<double2 *>(S.x + r0) = make_double2(x01.x + a[0], x01.y + a[1]);
      *reinterpret_cast<double2 *>(S.x + r0 + 2) = make_double2(x23.x + a[2], x23.y + a[3]);
    }
    return;
  }
  const int kdim = sc->kdim;
  if (S.pc == 1 && sc->pc_on == 2) {
    const double *z = sc->pc_out;
    for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < S.n; r += (long)gridDim.x * blockDim.x)
      S.x[r] = S.x[r] + z[r];
    return;
  }
  const bool kept = S.pc == 1 && !end_applies(S);
  // the vectors of the sum: the basis' from V up or the directions in lent
  // memory from its end down, then directions from the spare vector down
  double *const spare = S.V + (long)(kdim + 1) * S.ldv;
  const double *const first = kept ? S.lent : S.V;
  const long step = kept ? -S.ldv : S.ldv;
  const int nfirst = kept ? min(m, S.nlent) : m;
  for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < S.n; r += (long)gridDim.x * blockDim.x) {
    double acc = 0.0;
    if (S.pc == 2) {
      for (int kk = 0; kk < m; ++kk) acc = fma(cf[kk], widen(S.Z[(long)kk * S.ldv + r]), acc);
      S.x[r] = S.x[r] + acc;
    } else {
      for (int kk = 0; kk < nfirst; ++kk) acc = fma(cf[kk], first[(long)kk * step + r], acc);
      for (int kk = nfirst; kk < m; ++kk) acc = fma(cf[kk], spare[r - (long)(kk - nfirst) * S.ldv], acc);
      if (S.pc == 0) S.x[r] = fma(S.invd[r], acc, S.x[r]);
      else if (kept) S.x[r] = S.x[r] + acc;
      else spare[r] = acc;
    }
  }
}

// Relative bound on the double-float residual of one row: |r_df - r| <=
// kDfRowBound * (|b| + sum_s |c_s x_s|). Per row the seven products carry
// about 3 * 2^-47 of their size (split of c and of x, rounded cross terms, the
// dropped lo * lo) and the eight double-float additions 2^-47 of the running
// sum each, about 2^-43.3 in all; 2^-41 leaves a factor of five.
constexpr double kDfRowBound = 4.547473508864641e-13;  // 2^-41

// True residual after a cycle; decide converged / stop / restart (V_0 = r).
// Systems with df_resid compute it in double-float and also the norm M of
// the per-row bounds; a decision closer to the tolerance than
// kDfRowBound * M is taken again from an FP64 residual, and the rest of the
// solve stays in FP64, so convergence is always decided within FP64 rounding.
// Systems whose x waits for the preconditioner are left alone.
__global__ void __launch_bounds__(kThreads) k_cycle_residual(const __grid_constant__ KSysPack P) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  if (!sc->cycle_end || (end_applies(S) && sc->pc_on != 2)) return;
  const bool df = S.df_resid && !sc->use64;
  __shared__ double sacc[2 * kWarps];
  if (threadIdx.x < 2 * kWarps) sacc[threadIdx.x] = 0.0;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (df) {
    // r = b - A x in double-float (about 48 bits) on the FP32 pipe, from the
    // double-float copy of x that the update wrote; |r|^2 and the squared
    // row bounds summed in FP32 per thread and FP64 across threads
    const long sy = S.nx, sz = (long)S.nx * S.ny;
    float pf = 0.0f, mf = 0.0f;  // per thread over all its rows
    for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
#pragma unroll
      for (int t = 0; t < kRowsPerThread; ++t) {
        const long r = t0 + t * kThreads + threadIdx.x;
        if (r < S.n) {
          int i, j, k;
          sys_ijk(r, S, i, j, k);
          const float *c = S.tabdf + 16 * (long)S.cls[r];
          float ah = 0.0f, al = 0.0f, mag = 0.0f;
          auto add = [&](int s, long q) {
            const float2 xv = S.xs[q];
            df_fma(ah, al, c[s], c[8 + s], xv.x, xv.y);
            mag = fmaf(fabsf(c[s]), fabsf(xv.x), mag);
          };
          add(0, r);
          if (i > 0) add(1, r - 1);
          if (i < S.nx - 1) add(2, r + 1);
          if (j > 0) add(3, r - sy);
          if (j < S.ny - 1) add(4, r + sy);
          if (k > 0) add(5, r - sz);
          if (k < S.nz - 1) add(6, r + sz);
          float bh, bl, rh, rl;
          df_split(S.b[r], bh, bl);
          df_sub(bh, bl, ah, al, rh, rl);
          S.Vf[r] = rh;
          pf = fmaf(rh, rh, pf);
          mag = 1.001f * (mag + fabsf(bh));  // the FP32 magnitudes' own rounding
          mf = fmaf(mag, mag, mf);
        }
      }
    }
    const double pr = warp_sum((double)pf), mr = warp_sum((double)mf);
    if (lane == 0) { sacc[warp] = pr; sacc[kWarps + warp] = mr; }
  } else {
  double pr = 0.0;  // per thread over all its rows
  for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
#pragma unroll
    for (int t = 0; t < kRowsPerThread; ++t) {
      const long r = t0 + t * kThreads + threadIdx.x;
      if (r < S.n) {
        int i, j, k;
        sys_ijk(r, S, i, j, k);
        long cs;
        const double *c0 = ar_row(S, r, cs);
        const double rv = S.b[r] - stencil7_at(c0, cs, S.x, (int)r, i, j, k, S.nx, S.ny, S.nz);
        if (S.a32) S.Vf[r] = narrow(rv);
        else S.V[r] = rv;
        if (S.vcur) S.vcur[r] = narrow(rv);
        pr = fma(rv, rv, pr);
      }
    }
  }
  pr = warp_sum(pr);
  if (lane == 0) sacc[warp] = pr;
  }
  if (!block_partials_and_last(sacc, 2, S.part, &sc->ticket)) return;
  __shared__ double tot[2];
  reduce_partials(S.part, gridDim.x, 2, tot);
  __syncthreads();
  if (threadIdx.x == 0) {
    sc->ticket = 0;
    const double rt = sqrt(tot[0]);
    sc->cycle_end = 0;
    sc->pc_on = 0;
    sc->r_norm = rt;
    if (!isfinite(rt)) { sc->nonfinite = 1; sc->status = 2; sc->active = 0; return; }
    if (df) {
      const double bound = kDfRowBound * sqrt(tot[1]);
      if (rt + bound <= sc->eps) { sc->status = 1; sc->active = 0; return; }
      if (rt - bound <= sc->eps) {
        // too close to call: the next cycle end (no update, i = 0) computes the
        // FP64 residual of the same x
        sc->use64 = 1;
        sc->cycle_end = 1;
        sc->i = 0;
        return;
      }
    } else if (rt <= sc->eps) {
      sc->status = 1; sc->active = 0; return;
    }
    if (sc->iters >= sc->maxit) { sc->status = 2; sc->active = 0; return; }
    if (sc->claimed && rt >= sc->real_old) { sc->status = 3; sc->active = 0; return; }
    sc->real_old = rt;
    sc->cyc_eps = fmax(sc->eps, sc->cyc_rtol * rt);
    sc->i = 0;
    pc_of_step(S, 0, sc->kdim, 1);
    sc->claimed = 0;
    sc->nu[0] = rt;
    sc->inu[0] = 1.0 / rt;
    sc->g[0] = rt;
    sc->active = 1;
  }
}

// ---------------------------------------------------------------------------
// FP32 Arnoldi cycles (a32 systems, flexible form only). The same three steps
// on an FP32 basis: the operator is the FP32 copy, products and per-thread
// sums are FP32, sums across threads and blocks and every scalar are FP64.
// A cycle stops once its estimate fell by cyc_rtol; the restart computes the
// true residual in FP64, so the solve still meets the FP64 tolerance.

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void __launch_bounds__(kThreads) k_arnoldi_spmv32(const __grid_constant__ KSysPack P) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  if (!sc->active || !S.a32) return;
  const int j = sc->i, nd = j + 1;
  __shared__ double sacc[(kMaxKdim + 1) * kWarps];
  for (int t = threadIdx.x; t < nd * kWarps; t += blockDim.x) sacc[t] = 0.0;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float *zj = S.Z + (long)j * S.ldv;
  if (nd <= kChunk32 && S.vec4) {
    // four consecutive rows per thread: coefficient planes, w and the basis
    // move as 16-byte vectors; the stencil of each row is stencil7_row_f's
    float acc[kChunk32];
#pragma unroll
    for (int kk = 0; kk < kChunk32; ++kk) acc[kk] = 0.0f;
    const long n = S.n, sy = S.nx, sz = (long)S.nx * S.ny;
    for (long t0 = (long)blockIdx.x * kTile; t0 < n; t0 += (long)gridDim.x * kTile) {
      const long r0 = t0 + 4 * threadIdx.x;
      if (r0 >= n) continue;
      float w[4];
      if (S.quad == 1 && S.cls) {
        // 85 us at 10.5M rows with 28 loads of z and eight of the table per
        // thread, 64 as quads
        const ushort4 c4 = __ldcs(reinterpret_cast<const ushort4 *>(S.cls + r0));
        const QuadRows v = load_quad_rows<true>(S, zj, r0);
        if (all_major(c4, S.major)) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            w[q] = quad_row32(v, q, S.uf[0], S.uf[1], S.uf[2], S.uf[3], S.uf[4], S.uf[5], S.uf[6]);
        } else {
          float4 cp[7];
          load_rows4(S.tabf, c4, cp);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            w[q] = quad_row32(v, q, f4(cp[0], q), f4(cp[1], q), f4(cp[2], q), f4(cp[3], q), f4(cp[4], q), f4(cp[5], q),
                              f4(cp[6], q));
        }
      } else {
      float4 cp[7];
      if (S.cls) {
        load_rows4(S.tabf, __ldcs(reinterpret_cast<const ushort4 *>(S.cls + r0)), cp);
      } else {
#pragma unroll
        for (int q = 0; q < 7; ++q) cp[q] = __ldcs(reinterpret_cast<const float4 *>(S.Af + (long)q * n + r0));
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const long r = r0 + q;
        int i, jj, k;
        sys_ijk(r, S, i, jj, k);
        float a = 0.0f;
        a = fmaf(f4(cp[0], q), zj[r], a);
        a = fmaf(f4(cp[1], q), i > 0 ? zj[r - 1] : 0.0f, a);
        a = fmaf(f4(cp[2], q), i < S.nx - 1 ? zj[r + 1] : 0.0f, a);
        a = fmaf(f4(cp[3], q), jj > 0 ? zj[r - sy] : 0.0f, a);
        a = fmaf(f4(cp[4], q), jj < S.ny - 1 ? zj[r + sy] : 0.0f, a);
        a = fmaf(f4(cp[5], q), k > 0 ? zj[r - sz] : 0.0f, a);
        a = fmaf(f4(cp[6], q), k < S.nz - 1 ? zj[r + sz] : 0.0f, a);
        w[q] = a;
      }
      }
      st4(S.wf + r0, make_float4(w[0], w[1], w[2], w[3]));
#pragma unroll
      for (int kk = 0; kk < kChunk32; ++kk) {
        if (kk < nd) {
          const float4 v = ld4(S.Vf + (long)kk * S.ldv + r0);
          acc[kk] = fmaf(v.x, w[0], acc[kk]);
          acc[kk] = fmaf(v.y, w[1], acc[kk]);
          acc[kk] = fmaf(v.z, w[2], acc[kk]);
          acc[kk] = fmaf(v.w, w[3], acc[kk]);
        }
      }
    }
#pragma unroll
    for (int kk = 0; kk < kChunk32; ++kk) {
      if (kk >= nd) break;
      const float p = warp_sum_f(acc[kk]);
      if (lane == 0) sacc[kk * kWarps + warp] = (double)p;
    }
  } else
  if (nd <= kChunk32) {
    // short basis: every dot product of the thread stays in a register
    // across the whole sweep, one warp reduction per dot at the end
    float acc[kChunk32];
#pragma unroll
    for (int kk = 0; kk < kChunk32; ++kk) acc[kk] = 0.0f;
    for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
#pragma unroll
      for (int t = 0; t < kRowsPerThread; ++t) {
        const long r = t0 + t * kThreads + threadIdx.x;
        if (r < S.n) {
          int i, jj, k;
          sys_ijk(r, S, i, jj, k);
          long cs;
          const float *c0 = af_row(S, r, cs);
          const float w = stencil7_at_f(c0, cs, zj, (int)r, i, jj, k, S.nx, S.ny, S.nz);
          S.wf[r] = w;
#pragma unroll
          for (int kk = 0; kk < kChunk32; ++kk)
            if (kk < nd) acc[kk] = fmaf(S.Vf[(long)kk * S.ldv + r], w, acc[kk]);
        }
      }
    }
#pragma unroll
    for (int kk = 0; kk < kChunk32; ++kk) {
      if (kk >= nd) break;
      const float p = warp_sum_f(acc[kk]);
      if (lane == 0) sacc[kk * kWarps + warp] = (double)p;
    }
  } else
  for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
    float wv[kRowsPerThread];
#pragma unroll
    for (int t = 0; t < kRowsPerThread; ++t) {
      const long r = t0 + t * kThreads + threadIdx.x;
      wv[t] = 0.0f;
      if (r < S.n) {
        int i, jj, k;
        sys_ijk(r, S, i, jj, k);
        long cs;
        const float *c0 = af_row(S, r, cs);
        const float w = stencil7_at_f(c0, cs, zj, (int)r, i, jj, k, S.nx, S.ny, S.nz);
        S.wf[r] = w;
        wv[t] = w;
      }
    }
    for (int kk = 0; kk < nd; ++kk) {
      const float *vk = S.Vf + (long)kk * S.ldv;
      float p = 0.0f;
#pragma unroll
      for (int t = 0; t < kRowsPerThread; ++t) {
        const long r = t0 + t * kThreads + threadIdx.x;
        if (r < S.n) p = fmaf(vk[r], wv[t], p);
      }
      p = warp_sum_f(p);
      if (lane == 0) sacc[kk * kWarps + warp] += (double)p;
    }
  }
  if (!block_partials_and_last(sacc, nd, S.part, &sc->ticket)) return;
  __shared__ double tot[kMaxKdim + 1];
  reduce_partials(S.part, gridDim.x, nd, tot);
  __syncthreads();
  for (int kk = threadIdx.x; kk < nd; kk += blockDim.x) {
    const double h = tot[kk] / sc->nu[kk];
    sc->h1[kk] = h;
    sc->coef[kk] = h / sc->nu[kk];
  }
  if (threadIdx.x == 0) sc->ticket = 0;
}

__global__ void __launch_bounds__(kThreads) k_arnoldi_orth32(const __grid_constant__ KSysPack P) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  if (!sc->active || !S.a32) return;
  const int j = sc->i, nd = j + 1;
  __shared__ double sacc[(kMaxKdim + 1) * kWarps];
  __shared__ float cf[kMaxKdim + 1];
  for (int t = threadIdx.x; t < nd * kWarps; t += blockDim.x) sacc[t] = 0.0;
  for (int t = threadIdx.x; t < nd; t += blockDim.x) cf[t] = (float)sc->coef[t];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (nd <= kChunk32 && S.vec4) {
    float acc[kChunk32];
#pragma unroll
    for (int kk = 0; kk < kChunk32; ++kk) acc[kk] = 0.0f;
    for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
      const long r0 = t0 + 4 * threadIdx.x;
      if (r0 >= S.n) continue;
      float4 v[kChunk32];
#pragma unroll
      for (int kk = 0; kk < kChunk32; ++kk)
        v[kk] = kk < nd ? ld4(S.Vf + (long)kk * S.ldv + r0) : make_float4(0.f, 0.f, 0.f, 0.f);
      float4 w = ld4(S.wf + r0);
#pragma unroll
      for (int kk = 0; kk < kChunk32; ++kk) {
        if (kk < nd) {
          w.x = fmaf(-cf[kk], v[kk].x, w.x);
          w.y = fmaf(-cf[kk], v[kk].y, w.y);
          w.z = fmaf(-cf[kk], v[kk].z, w.z);
          w.w = fmaf(-cf[kk], v[kk].w, w.w);
        }
      }
      st4(S.wf + r0, w);
#pragma unroll
      for (int kk = 0; kk < kChunk32; ++kk) {
        acc[kk] = fmaf(v[kk].x, w.x, acc[kk]);
        acc[kk] = fmaf(v[kk].y, w.y, acc[kk]);
        acc[kk] = fmaf(v[kk].z, w.z, acc[kk]);
        acc[kk] = fmaf(v[kk].w, w.w, acc[kk]);
      }
    }
#pragma unroll
    for (int kk = 0; kk < kChunk32; ++kk) {
      if (kk >= nd) break;
      const float p = warp_sum_f(acc[kk]);
      if (lane == 0) sacc[kk * kWarps + warp] = (double)p;
    }
  } else
  if (nd <= kChunk32) {
    // short basis: each basis value is loaded once for the update and the dots
    float acc[kChunk32];
#pragma unroll
    for (int kk = 0; kk < kChunk32; ++kk) acc[kk] = 0.0f;
    for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
#pragma unroll
      for (int t = 0; t < kRowsPerThread; ++t) {
        const long r = t0 + t * kThreads + threadIdx.x;
        if (r < S.n) {
          float v[kChunk32];
#pragma unroll
          for (int kk = 0; kk < kChunk32; ++kk) v[kk] = kk < nd ? S.Vf[(long)kk * S.ldv + r] : 0.0f;
          float w = S.wf[r];
#pragma unroll
          for (int kk = 0; kk < kChunk32; ++kk)
            if (kk < nd) w = fmaf(-cf[kk], v[kk], w);
          S.wf[r] = w;
#pragma unroll
          for (int kk = 0; kk < kChunk32; ++kk) acc[kk] = fmaf(v[kk], w, acc[kk]);
        }
      }
    }
#pragma unroll
    for (int kk = 0; kk < kChunk32; ++kk) {
      if (kk >= nd) break;
      const float p = warp_sum_f(acc[kk]);
      if (lane == 0) sacc[kk * kWarps + warp] = (double)p;
    }
  } else
  for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
    float wv[kRowsPerThread];
#pragma unroll
    for (int t = 0; t < kRowsPerThread; ++t) {
      const long r = t0 + t * kThreads + threadIdx.x;
      wv[t] = 0.0f;
      if (r < S.n) {
        float w = S.wf[r];
        for (int kk = 0; kk < nd; ++kk) w = fmaf(-cf[kk], S.Vf[(long)kk * S.ldv + r], w);
        S.wf[r] = w;
        wv[t] = w;
      }
    }
    for (int kk = 0; kk < nd; ++kk) {
      float p = 0.0f;
#pragma unroll
      for (int t = 0; t < kRowsPerThread; ++t) {
        const long r = t0 + t * kThreads + threadIdx.x;
        if (r < S.n) p = fmaf(S.Vf[(long)kk * S.ldv + r], wv[t], p);
      }
      p = warp_sum_f(p);
      if (lane == 0) sacc[kk * kWarps + warp] += (double)p;
    }
  }
  if (!block_partials_and_last(sacc, nd, S.part, &sc->ticket)) return;
  __shared__ double tot[kMaxKdim + 1];
  reduce_partials(S.part, gridDim.x, nd, tot);
  __syncthreads();
  for (int kk = threadIdx.x; kk < nd; kk += blockDim.x) {
    const double h2 = tot[kk] / sc->nu[kk];
    sc->coef[kk] = h2 / sc->nu[kk];
    sc->H[kk * kMaxKdim + j] = sc->h1[kk] + h2;
  }
  if (threadIdx.x == 0) sc->ticket = 0;
}

__global__ void __launch_bounds__(kThreads) k_arnoldi_next32(const __grid_constant__ KSysPack P) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  if (!sc->active || !S.a32) return;
  const int j = sc->i, nd = j + 1;
  __shared__ float cf[kMaxKdim + 1];
  __shared__ double sacc[kWarps];
  for (int t = threadIdx.x; t < nd; t += blockDim.x) cf[t] = (float)sc->coef[t];
  if (threadIdx.x < kWarps) sacc[threadIdx.x] = 0.0;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float *vn = S.Vf + (long)nd * S.ldv;
  const bool store = nd < sc->kdim;
  // |w|^2: FP32 per thread (as the dot products of the FP32 cycle), FP64 across threads
  float pt = 0.0f;
  if (nd <= kChunk32 && S.vec4) {
    for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
      const long r0 = t0 + 4 * threadIdx.x;
      if (r0 >= S.n) continue;
      float4 w = ld4(S.wf + r0);
#pragma unroll
      for (int kk = 0; kk < kChunk32; ++kk) {
        if (kk < nd) {
          const float4 v = ld4(S.Vf + (long)kk * S.ldv + r0);
          w.x = fmaf(-cf[kk], v.x, w.x);
          w.y = fmaf(-cf[kk], v.y, w.y);
          w.z = fmaf(-cf[kk], v.z, w.z);
          w.w = fmaf(-cf[kk], v.w, w.w);
        }
      }
      if (store) st4(vn + r0, w);
      pt = fmaf(w.x, w.x, pt);
      pt = fmaf(w.y, w.y, pt);
      pt = fmaf(w.z, w.z, pt);
      pt = fmaf(w.w, w.w, pt);
    }
  } else
  for (long t0 = (long)blockIdx.x * kTile; t0 < S.n; t0 += (long)gridDim.x * kTile) {
#pragma unroll
    for (int t = 0; t < kRowsPerThread; ++t) {
      const long r = t0 + t * kThreads + threadIdx.x;
      if (r < S.n) {
        float w = S.wf[r];
        if (nd <= kChunk32) {
          float v[kChunk32];
#pragma unroll
          for (int kk = 0; kk < kChunk32; ++kk) v[kk] = kk < nd ? S.Vf[(long)kk * S.ldv + r] : 0.0f;
#pragma unroll
          for (int kk = 0; kk < kChunk32; ++kk)
            if (kk < nd) w = fmaf(-cf[kk], v[kk], w);
        } else {
          for (int kk = 0; kk < nd; ++kk) w = fmaf(-cf[kk], S.Vf[(long)kk * S.ldv + r], w);
        }
        if (store) vn[r] = w;
        pt = fmaf(w, w, pt);
      }
    }
  }
  const double ptd = warp_sum((double)pt);
  if (lane == 0) sacc[warp] = ptd;
  if (!block_partials_and_last(sacc, 1, S.part, &sc->ticket)) return;
  __shared__ double tot[1];
  reduce_partials(S.part, gridDim.x, 1, tot);
  __syncthreads();
  if (threadIdx.x == 0) sc->ticket = 0;
  arnoldi_finalize(S, j, sqrt(tot[0]));
}

// Two FP32 Jacobi sweeps from zero in one pass (momentum preconditioner of
// the flexible form): z = D^-1 (2v - A D^-1 v) = D^-1 (v - sum over the
// couplings of (A D^-1)_s v_s), with v = V_j / nu_j; A D^-1 is stored (cjf), so
// the pass reads v, the six scaled couplings and D^-1 once.
template <class VT>
__device__ __forceinline__ void jacobi_two_rows(const KSys &S, const VT *__restrict__ vj, float inv_nu,
                                                float *__restrict__ out) {
  const long n = S.n, sy = S.nx, sz = (long)S.nx * S.ny;
  for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (long)gridDim.x * blockDim.x) {
    int i, jj, k;
    sys_ijk(r, S, i, jj, k);
    // slot s (1..6) of the scaled couplings at cj[s * cs], D^-1 at id
    const float *cj, *id;
    long cs;
    if (S.clsj) { cj = S.tabj + 8 * (long)S.clsj[r]; cs = 1; id = cj; }
    else { cj = S.Ajf + r; cs = n; id = S.invdf + r; }
    float acc = (float)vj[r] * inv_nu;
    if (i > 0) acc = fmaf(-cj[cs], (float)vj[r - 1] * inv_nu, acc);
    if (i < S.nx - 1) acc = fmaf(-cj[2 * cs], (float)vj[r + 1] * inv_nu, acc);
    if (jj > 0) acc = fmaf(-cj[3 * cs], (float)vj[r - sy] * inv_nu, acc);
    if (jj < S.ny - 1) acc = fmaf(-cj[4 * cs], (float)vj[r + sy] * inv_nu, acc);
    if (k > 0) acc = fmaf(-cj[5 * cs], (float)vj[r - sz] * inv_nu, acc);
    if (k < S.nz - 1) acc = fmaf(-cj[6 * cs], (float)vj[r + sz] * inv_nu, acc);
    out[r] = *id * acc;
  }
}

// The same, four consecutive rows per thread (S.quad, classed records): 112 us
// over 3 x 10.5M rows with 28 loads of v and eight of the table per thread;
// 76 so. Lines of an odd number of rows (the u system) take the second form.
template <bool LINE>
__device__ __forceinline__ void jacobi_two_quads(const KSys &S, const float *__restrict__ vj, float inv_nu,
                                                 float *__restrict__ out) {
  auto scaled = [&](float4 &a) { a.x *= inv_nu; a.y *= inv_nu; a.z *= inv_nu; a.w *= inv_nu; };
  for (long r0 = 4 * ((long)blockIdx.x * blockDim.x + threadIdx.x); r0 < S.n; r0 += 4L * gridDim.x * blockDim.x) {
    const ushort4 c4 = __ldcs(reinterpret_cast<const ushort4 *>(S.clsj + r0));
    QuadRows v = load_quad_rows<LINE>(S, vj, r0);
    scaled(v.c); scaled(v.w); scaled(v.e); scaled(v.s); scaled(v.n); scaled(v.b); scaled(v.t);
    auto row = [&](int q, float id, float c1, float c2, float c3, float c4_, float c5, float c6) {
      float acc = f4(v.c, q);
      acc = fmaf(-c1, f4(v.w, q), acc);
      acc = fmaf(-c2, f4(v.e, q), acc);
      acc = fmaf(-c3, f4(v.s, q), acc);
      acc = fmaf(-c4_, f4(v.n, q), acc);
      acc = fmaf(-c5, f4(v.b, q), acc);
      acc = fmaf(-c6, f4(v.t, q), acc);
      return id * acc;
    };
    float z[4];
    if (all_major(c4, S.majorj)) {
#pragma unroll
      for (int q = 0; q < 4; ++q) z[q] = row(q, S.uj[0], S.uj[1], S.uj[2], S.uj[3], S.uj[4], S.uj[5], S.uj[6]);
    } else {
      float4 cp[7];
      load_rows4(S.tabj, c4, cp);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        z[q] = row(q, f4(cp[0], q), f4(cp[1], q), f4(cp[2], q), f4(cp[3], q), f4(cp[4], q), f4(cp[5], q), f4(cp[6], q));
    }
    st4(out + r0, make_float4(z[0], z[1], z[2], z[3]));
  }
}

// Four consecutive rows per thread with 16-byte loads of the coefficient
// planes and stores of z (FP32 basis, n % 4 == 0).
__device__ __forceinline__ void jacobi_two_rows4(const KSys &S, const float *__restrict__ vj, float inv_nu,
                                                 float *__restrict__ out) {
  const long n = S.n, sy = S.nx, sz = (long)S.nx * S.ny;
  for (long r0 = 4 * ((long)blockIdx.x * blockDim.x + threadIdx.x); r0 < n; r0 += 4L * gridDim.x * blockDim.x) {
    float4 cp[7];
    float4 id;
    if (S.clsj) {
      // class records {invdf, Ajf_1..Ajf_6, 0}: slot 0 is D^-1
      load_rows4(S.tabj, __ldcs(reinterpret_cast<const ushort4 *>(S.clsj + r0)), cp);
      id = cp[0];
    } else {
#pragma unroll
      for (int q = 1; q < 7; ++q) cp[q] = __ldcs(reinterpret_cast<const float4 *>(S.Ajf + (long)q * n + r0));
      id = __ldcs(reinterpret_cast<const float4 *>(S.invdf + r0));
    }
    float z[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const long r = r0 + q;
      int i, jj, k;
      sys_ijk(r, S, i, jj, k);
      float acc = vj[r] * inv_nu;
      if (i > 0) acc = fmaf(-f4(cp[1], q), vj[r - 1] * inv_nu, acc);
      if (i < S.nx - 1) acc = fmaf(-f4(cp[2], q), vj[r + 1] * inv_nu, acc);
      if (jj > 0) acc = fmaf(-f4(cp[3], q), vj[r - sy] * inv_nu, acc);
      if (jj < S.ny - 1) acc = fmaf(-f4(cp[4], q), vj[r + sy] * inv_nu, acc);
      if (k > 0) acc = fmaf(-f4(cp[5], q), vj[r - sz] * inv_nu, acc);
      if (k < S.nz - 1) acc = fmaf(-f4(cp[6], q), vj[r + sz] * inv_nu, acc);
      z[q] = f4(id, q) * acc;
    }
    *reinterpret_cast<float4 *>(out + r0) = make_float4(z[0], z[1], z[2], z[3]);
  }
}

__global__ void __launch_bounds__(kThreads) k_jacobi32_two(const __grid_constant__ KSysPack P) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  if (!sc->active || S.pc != 2 || S.pc_cb) return;
  const int j = sc->i;
  const float inv_nu = (float)sc->inu[j];
  float *out = S.Z + (long)j * S.ldv;
  // an FP64 basis is read through its FP32 copy when there is one: the same
  // values ((float) V_j), one conversion per row where the vector is formed
  // instead of one per row and neighbour here
  const float *vf = S.a32 ? S.Vf + (long)j * S.ldv : S.vcur;
  if (vf && S.clsj && S.quad == 1) jacobi_two_quads<true>(S, vf, inv_nu, out);
  else if (vf && S.clsj && S.quad == 2) jacobi_two_quads<false>(S, vf, inv_nu, out);
  else if (vf && S.vec4) jacobi_two_rows4(S, vf, inv_nu, out);
  else if (vf) jacobi_two_rows<float>(S, vf, inv_nu, out);
  else jacobi_two_rows<double>(S, S.V + (long)j * S.ldv, inv_nu, out);
}

// FP32 inner preconditioner for the flexible form: zf = D^-1 v (v = V_j / nu_j),
// then `sweeps-1` Jacobi sweeps zf <- zf + D^-1 (v - A zf); result to Z_j.
__global__ void __launch_bounds__(kThreads) k_jacobi32_first(const __grid_constant__ KSysPack P, int to_z) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  if (!sc->active || S.pc != 2 || S.pc_cb) return;
  const int j = sc->i;
  const double inv_nu = sc->inu[j];
  const double *vj = S.V + (long)j * S.ldv;
  const float *vjf = S.Vf + (long)j * S.ldv;
  float *out = to_z ? S.Z + (long)j * S.ldv : S.zf;
  if (S.vcur) {  // FP64 basis through its FP32 copy: no FP64 instruction
    const float inv_nuf = (float)inv_nu;
    for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < S.n; r += (long)gridDim.x * blockDim.x)
      out[r] = (S.vcur[r] * inv_nuf) * S.invdf[r];
    return;
  }
  for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < S.n; r += (long)gridDim.x * blockDim.x)
    out[r] = (float)((S.a32 ? (double)vjf[r] : vj[r]) * inv_nu) * S.invdf[r];
}

__global__ void __launch_bounds__(kThreads) k_jacobi32_sweep(const __grid_constant__ KSysPack P, int src_is_zf,
                                                             int to_z) {
  const KSys &S = P.s[blockIdx.y];
  KScal *sc = S.s;
  if (!sc->active || S.pc != 2 || S.pc_cb) return;
  const int j = sc->i;
  const double inv_nu = sc->inu[j];
  const double *vj = S.V + (long)j * S.ldv;
  const float *vjf = S.Vf + (long)j * S.ldv;
  const float *src = src_is_zf ? S.zf : S.zf2;
  float *dst = to_z ? S.Z + (long)j * S.ldv : (src_is_zf ? S.zf2 : S.zf);
  const float inv_nuf = (float)inv_nu;
  for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < S.n; r += (long)gridDim.x * blockDim.x) {
    int i, jj, k;
    sys_ijk(r, S, i, jj, k);
    long cs;
    const float *c0 = af_row(S, r, cs);
    const float az = stencil7_at_f(c0, cs, src, (int)r, i, jj, k, S.nx, S.ny, S.nz);
    const float v = S.vcur ? S.vcur[r] * inv_nuf : (float)((S.a32 ? (double)vjf[r] : vj[r]) * inv_nu);
    dst[r] = fmaf(S.invdf[r], v - az, src[r]);
  }
}

__global__ void k_flags(const __grid_constant__ KSysPack P, int nsys, KFlags *out) {
  const int t = threadIdx.x;
  if (t < nsys) {
    KScal *sc = P.s[t].s;
    out[t].active = sc->active;
    out[t].cycle_end = sc->cycle_end;
    out[t].status = sc->status;
    out[t].iters = sc->iters;
    out[t].i = sc->i;
    out[t].nonfinite = sc->nonfinite;
    out[t].rel = sc->b_norm > 0.0 ? sc->r_norm / sc->b_norm : sc->r_norm;
  }
}

// Systems whose finished cycle waits for the preconditioner: the next V-cycle is
// its. (In a launch of its own: the kernels that read the state run in many blocks.)
__device__ void wait_for_pc(const KSys &S) {
  if (S.s->cycle_end && end_applies(S)) pc_of_end(S);
}
__global__ void k_pc_of_end(const __grid_constant__ KSysPack P, int nsys) {
  if ((int)threadIdx.x < nsys) wait_for_pc(P.s[threadIdx.x]);
}

// Loop control of the graph form: WHILE runs while any system is active or
// has a finished cycle to close. Its body is an Arnoldi step and the cycle's
// end, whose kernels return at once for systems with no finished cycle. A cycle
// that waits for the preconditioner takes the next body's V-cycle, in which its
// Arnoldi kernels return at once. count (may be null): bodies run.
__global__ void k_set_while(const __grid_constant__ KSysPack P, int nsys, cudaGraphConditionalHandle hw,
                            unsigned long long *count) {
  const int s = threadIdx.x;  // one warp: a system's flags by a lane each, one memory latency for all
  bool runs = false;
  if (s < nsys) {
    runs = P.s[s].s->active | P.s[s].s->cycle_end;
    wait_for_pc(P.s[s]);
  }
  const unsigned run = __any_sync(0xffffffffu, runs) ? 1u : 0u;
  if (s != 0) return;
  if (count) *count += 1;
  cudaGraphSetConditional(hw, run);
}

}  // namespace

// ---------------------------------------------------------------------------
// Host driver
// ---------------------------------------------------------------------------
void Krylov::configure(int nsys_, const KSysHost *hs, double *lent, size_t lent_n) {
  if (nsys_ < 1 || nsys_ > kMaxSys) throw Error(IBM_ERR_ARG, "Krylov: bad system count");
  nsys = nsys_;
  int maxn = 0;
  for (int s = 0; s < nsys; ++s) {
    if (hs[s].kdim < 1 || hs[s].kdim > kMaxKdim) throw Error(IBM_ERR_ARG, "GMRES restart length must be in [1, 63]");
    maxn = std::max(maxn, hs[s].n);
  }
  nblk = persistent_blocks(maxn, 4);
  // the FP32 SpMV + dots kernel holds 80 registers (three blocks per SM): a
  // grid of as many blocks as stay resident runs in one wave
  {
    int per_sm = 0;
    IBM_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_arnoldi_spmv32, kThreads, 0));
    nblk_spmv32 = std::max(1, std::min(nblk, std::max(1, per_sm) * sm_count()));
  }
  const size_t need_part = (size_t)nblk * (kMaxKdim + 2);
  for (int s = 0; s < nsys; ++s) {
    const KSysHost &h = hs[s];
    Slot &sl = slot[s];
    sl.host = h;
    if (h.a32 && h.pc != 2) throw Error(IBM_ERR_ARG, "Krylov: FP32 cycles need the flexible form");
    if (h.a32) {
      sl.V.release(); sl.w.release();
      sl.Vf.alloc((size_t)(h.kdim + 1) * h.n);
      sl.wf.alloc(h.n);
    } else {
      sl.Vf.release(); sl.wf.release();
      sl.V.alloc((size_t)(h.kdim + (h.pc == 1 ? 2 : 1)) * h.n);  // pc 1: the spare vector (direction_of)
      sl.w.alloc(h.n);
    }
    sl.nlent = h.pc == 1 && nsys == 1 ? (int)std::min((size_t)h.kdim, lent_n / (size_t)h.n) : 0;
    sl.lent = sl.nlent ? lent + (lent_n - (size_t)h.n) : nullptr;
    sl.nkept = h.pc == 1 ? kept_directions(h.kdim, sl.nlent) : 0;
    if (h.a32 && h.cls && h.tabdf && h.df_residual) sl.xs.alloc(h.n);
    else sl.xs.release();
    if (h.pc == 2) {
      sl.Z.alloc((size_t)h.kdim * h.n);
      if (!h.pc_cb) { sl.zf.alloc(h.n); sl.zf2.alloc(h.n); }
    }
    if (h.pc == 2 && !h.pc_cb && !h.a32) sl.vcur.alloc(h.n);
    else sl.vcur.release();
    sl.part.alloc(need_part);
  }
  scal.alloc(nsys);
  dflags.alloc(nsys);
  if (!hflags) IBM_CUDA_TRY(cudaMallocHost((void **)&hflags, sizeof(KFlags) * kMaxSys));
}

double *Krylov::idle(size_t &n) const {
  double *p = nullptr;
  n = 0;
  for (int s = 0; s < nsys; ++s) {
    const size_t v = slot[s].V.n, f = slot[s].Vf.n / 2;
    if (v > n) { n = v; p = slot[s].V.p; }
    if (f > n) { n = f; p = reinterpret_cast<double *>(slot[s].Vf.p); }
  }
  return p;
}

Krylov::~Krylov() {
  if (hflags) cudaFreeHost(hflags);
}

void Krylov::bind(cudaStream_t st, const double *const *b, double *const *x, unsigned mask, bool x_zero) {
  bound_mask = mask;
  bound_x_zero = x_zero;
  memset(&pack, 0, sizeof(pack));
  for (int s = 0; s < nsys; ++s) {
    const KSysHost &h = slot[s].host;
    KSys &k = pack.s[s];
    k.nx = h.nx; k.ny = h.ny; k.nz = h.nz; k.n = ((mask >> s) & 1u) ? h.n : 0;
    k.fdx = make_fastdiv((unsigned)h.nx); k.fdy = make_fastdiv((unsigned)h.ny);
    k.A = h.A; k.Ar = h.Ar; k.invd = h.invd; k.Af = h.Af; k.invdf = h.invdf; k.Ajf = h.Ajf;
    k.cls = h.cls; k.tab = h.tab; k.tabf = h.tabf; k.clsj = h.clsj; k.tabj = h.tabj;
    k.tabdf = h.tabdf;
    k.major = h.major; k.majorj = h.majorj;
    std::copy(h.uf, h.uf + 8, k.uf);
    std::copy(h.udf, h.udf + 16, k.udf);
    std::copy(h.uj, h.uj + 8, k.uj);
    k.quad = h.nx % 4 == 0 ? 1 : h.n % 4 == 0 && h.nx >= 4 ? 2 : 0;
    k.df_resid = (h.a32 && h.cls && h.tabdf && h.df_residual) ? 1 : 0;
    k.df_spmv = (h.pc == 2 && !h.a32 && h.cls && h.tabdf && h.A == h.Ar && h.df_spmv) ? 1 : 0;
    k.xs = slot[s].xs.p;
    k.V = slot[s].V.p; k.ldv = h.n;
    k.Z = slot[s].Z.p;
    k.w = slot[s].w.p;
    k.lent = slot[s].lent; k.nlent = slot[s].nlent; k.nkept = slot[s].nkept;
    k.zf = slot[s].zf.p; k.zf2 = slot[s].zf2.p;
    k.Vf = slot[s].Vf.p; k.wf = slot[s].wf.p; k.a32 = h.a32;
    k.vcur = slot[s].vcur.p;
    k.cgs1 = cgs1(h) ? 1 : 0;
    k.x_zero = x_zero ? 1 : 0;
    k.vec4 = (h.n % 4 == 0) ? 1 : 0;
    k.x = x[s]; k.b = b[s];
    k.part = slot[s].part.p;
    k.nblk = nblk;
    k.pc = h.pc;
    k.pc_cb = h.pc_cb;
    k.s = scal.p + s;
  }
  static KScal init[kMaxSys];
  memset(init, 0, sizeof(init));
  for (int s = 0; s < nsys; ++s) {
    init[s].kdim = slot[s].host.kdim;
    init[s].maxit = slot[s].host.maxit;
    init[s].tol = slot[s].host.tol;
    init[s].cyc_rtol = slot[s].host.a32 ? slot[s].host.cycle_rtol : 0.0;
  }
  IBM_CUDA_TRY(cudaMemcpyAsync(scal.p, init, sizeof(KScal) * nsys, cudaMemcpyHostToDevice, st));
  IBM_CUDA_TRY(cudaStreamSynchronize(st));
}

void Krylov::read_flags(cudaStream_t st) {
  {
    LaunchScope ls(K_GM_UPDATE, st, 0.0);
    k_flags<<<1, 32, 0, st>>>(pack, nsys, dflags.p);
  }
  IBM_CUDA_TRY(cudaMemcpyAsync(hflags, dflags.p, sizeof(KFlags) * nsys, cudaMemcpyDeviceToHost, st));
  IBM_CUDA_TRY(cudaStreamSynchronize(st));
}

// Algorithmic bytes per row (FP64 = 8): the operator's 7 coefficients, the
// vectors each kernel must read or write once, and the basis vectors it
// sweeps. In the graph form the flags are not known on the host and no
// bytes are attributed.
void Krylov::launch_cycle_end(cudaStream_t st, const Precond &pc, const KFlags *fl, unsigned mask) {
  const dim3 grid(nblk, nsys), gridu(nblk * 2, nsys);
  auto rows = [&](int s) { return ((mask >> s) & 1u) ? (double)slot[s].host.n : 0.0; };
  double bu = 0.0, br = 0.0;
  if (fl) {
    for (int s = 0; s < nsys; ++s) {
      if (!fl[s].cycle_end) continue;
      const int m = fl[s].i, pcm = slot[s].host.pc;
      bu += rows(s) * (pcm == 2 ? 4.0 * m + 16.0 : pcm == 1 ? 8.0 * m + (m > slot[s].nkept ? 8.0 : 16.0) : 8.0 * m + 24.0);
      // a classed row is its 2-byte class instead of 7 FP64 coefficients
      if (pcm != 1 || m <= slot[s].nkept)
        br += ((slot[s].host.cls ? 34.0 : 88.0) + (slot[s].vcur.p ? 4.0 : 0.0)) * rows(s);
    }
  }
  auto update = [&](KernelId id, double b_update, double b_resid) {
    {
      LaunchScope ls(id, st, b_update);
      k_cycle_update<<<wave(k_cycle_update), kThreads, 0, st>>>(pack);
    }
    LaunchScope ls(K_GM_RESID, st, b_resid);
    k_cycle_residual<<<wave(k_cycle_residual), kThreads, 0, st>>>(pack);
  };
  update(K_GM_UPDATE, bu, br);
  // cycles that outgrew their stored directions (captured: the next loop body's V-cycle takes them)
  bool applies = false;
  double ba = 0.0, bar = 0.0;
  for (int s = 0; fl && s < nsys; ++s) {
    if (slot[s].host.pc != 1 || !fl[s].cycle_end || fl[s].i <= slot[s].nkept) continue;
    if (!applies) {
      LaunchScope ls(K_GM_UPDATE, st, 0.0);
      k_pc_of_end<<<1, 32, 0, st>>>(pack, nsys);
    }
    apply_explicit(st, pc, s);
    ba += 24.0 * rows(s);
    bar += (slot[s].host.cls ? 34.0 : 88.0) * rows(s);
    applies = true;
  }
  if (applies) update(K_GM_ADDZ, ba, bar);
}

// The V-cycle that a pc 1 system's scalars name (pc_of_step, pc_of_end).
void Krylov::apply_explicit(cudaStream_t st, const Precond &pc, int s) {
  VecRef in;
  in.at = &scal.p[s].pc_in;
  OutRef out;
  out.at = &scal.p[s].pc_out;
  pc.apply(pc.ctx, st, s, in, out, nsys > 1 ? &scal.p[s].pc_on : nullptr);
}

void Krylov::launch_arnoldi(cudaStream_t st, const Precond &pc, const KFlags *fl, unsigned mask) {
  const dim3 grid(nblk, nsys), gridu(nblk * 2, nsys);
  auto rows = [&](int s) { return ((mask >> s) & 1u) ? (double)slot[s].host.n : 0.0; };
  // A single system is active whenever an Arnoldi step runs (the host loop and
  // the graph's WHILE see to that), so its preconditioner needs no gate: one
  // dependent load less at the start of each of its kernels.
  for (int s = 0; s < nsys; ++s) {
    if (!((mask >> s) & 1u) || (fl && !fl[s].active)) continue;
    const KSysHost &h = slot[s].host;
    if (h.pc == 1) {
      apply_explicit(st, pc, s);
    } else if (h.pc == 2 && h.pc_cb) {
      VecRef in;
      if (h.a32) in.basef = slot[s].Vf.p;
      else in.base = slot[s].V.p;
      in.ld = h.n; in.idx = &scal.p[s].i; in.inu = scal.p[s].inu;
      OutRef out;
      out.f = slot[s].Z.p; out.ld = h.n; out.idx = &scal.p[s].i;
      pc.apply(pc.ctx, st, s, in, out, nsys > 1 ? &scal.p[s].active : nullptr);
    }
  }
  int inner_sweeps = 0;
  bool any64 = false, any32 = false, any_orth = false;
  double r32 = 0.0, j32two = 0.0, bsp = 0.0, bor = 0.0, bor_orth = 0.0, bnx = 0.0, bsp32 = 0.0, bor32 = 0.0;
  for (int s = 0; s < nsys; ++s) {
    if (!((mask >> s) & 1u)) continue;
    const bool a32 = slot[s].host.a32 != 0;
    (a32 ? any32 : any64) = true;
    if (!a32 && !cgs1(slot[s].host)) any_orth = true;
    if (slot[s].host.pc == 2 && !slot[s].host.pc_cb && (!fl || fl[s].active))
      inner_sweeps = std::max(inner_sweeps, std::max(1, slot[s].host.inner_sweeps));
    if (!fl || !fl[s].active) continue;
    const double j1 = fl[s].i + 1.0;
    const KSysHost &h = slot[s].host;
    // coefficient bytes of a row: 7 values, or a 2-byte class
    const double c64 = (h.cls && h.A == h.Ar) ? 2.0 : 56.0, c32 = h.cls ? 2.0 : 28.0;
    if (h.pc == 2 && !h.pc_cb) {
      r32 += rows(s) * ((a32 || slot[s].vcur.p) ? 0.75 : 1.0);  // v read as FP32 or FP64
      // two sweeps in one pass: v, z and a 2-byte class instead of 7 FP32 values
      j32two += rows(s) * (h.clsj ? 10.0 : 27.0);  // v read as FP32 (basis or copy)
      if (!a32) bnx += 4.0 * rows(s);                // the copy, written by k_arnoldi_next
    }
    if (a32) {
      bsp32 += rows(s) * (c32 + 8.0 + 4.0 * j1);
      bor32 += rows(s) * (8.0 + 4.0 * j1);
    } else {
      bsp += rows(s) * ((h.pc == 2 ? 12.0 : 16.0) + c64 + 8.0 * j1);
      bor += rows(s) * (16.0 + 8.0 * j1);
      if (!cgs1(h)) bor_orth += rows(s) * (16.0 + 8.0 * j1);
    }
  }
  if (inner_sweeps > 0) {
    if (inner_sweeps == 2) {
      LaunchScope ls(K_GM_JAC32, st, j32two);
      k_jacobi32_two<<<wave(k_jacobi32_two), kThreads, 0, st>>>(pack);
    } else if (inner_sweeps == 1) {
      LaunchScope ls(K_GM_JAC32, st, 16.0 * r32);
      k_jacobi32_first<<<gridu, kThreads, 0, st>>>(pack, 1);
    } else {
      {
        LaunchScope ls(K_GM_JAC32, st, 16.0 * r32);
        k_jacobi32_first<<<gridu, kThreads, 0, st>>>(pack, 0);
      }
      int src_zf = 1;
      for (int q = 1; q < inner_sweeps; ++q) {
        LaunchScope ls(K_GM_JAC32, st, 48.0 * r32);
        k_jacobi32_sweep<<<gridu, kThreads, 0, st>>>(pack, src_zf, q == inner_sweeps - 1);
        src_zf ^= 1;
      }
    }
  }
  if (any64) {
    {
      LaunchScope ls(K_GM_SPMV, st, bsp);
      k_arnoldi_spmv<<<wave(k_arnoldi_spmv), kThreads, 0, st>>>(pack);
    }
    if (any_orth) {
      LaunchScope ls(K_GM_ORTH, st, bor_orth);
      k_arnoldi_orth<<<wave(k_arnoldi_orth), kThreads, 0, st>>>(pack);
    }
    LaunchScope ls(K_GM_NEXT, st, bor + bnx);
    k_arnoldi_next<<<wave(k_arnoldi_next), kThreads, 0, st>>>(pack);
  }
  if (any32) {
    {
      LaunchScope ls(K_GM_SPMV, st, bsp32);
      k_arnoldi_spmv32<<<wave(k_arnoldi_spmv32), kThreads, 0, st>>>(pack);
    }
    {
      LaunchScope ls(K_GM_ORTH, st, bor32);
      k_arnoldi_orth32<<<wave(k_arnoldi_orth32), kThreads, 0, st>>>(pack);
    }
    LaunchScope ls(K_GM_NEXT, st, bor32);
    k_arnoldi_next32<<<wave(k_arnoldi_next32), kThreads, 0, st>>>(pack);
  }
}

// Grid of a grid-stride Krylov kernel: (x, nsys) with x such that all blocks
// stay resident (one wave), at most nblk (the size of the partials).
template <class K>
dim3 Krylov::wave(K kernel) const {
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, 0);
  const int x = std::max(1, std::min(nblk, std::max(1, per_sm) * sm_count() / std::max(1, nsys)));
  return dim3(x, nsys);
}

void Krylov::solve(cudaStream_t st, const double *const *b, double *const *x, const Precond &pc,
                   KResult *res, unsigned mask, bool x_zero) {
  bind(st, b, x, mask, x_zero);
  const dim3 grid(nblk, nsys);
  double init_bytes = 0.0;
  for (int s = 0; s < nsys; ++s)
    if ((mask >> s) & 1u)
      init_bytes += ((x_zero ? 16.0 : slot[s].host.cls ? 26.0 : 80.0) + (slot[s].vcur.p ? 4.0 : 0.0)) * slot[s].host.n;
  {
    LaunchScope ls(K_GM_INIT, st, init_bytes);
    k_init<<<wave(k_init), kThreads, 0, st>>>(pack);
  }
  for (long guard = 0;; ++guard) {
    if (guard > 4L * 1000 * 1000) throw Error(IBM_ERR_CUDA, "GMRES host loop did not terminate");
    read_flags(st);
    bool any_active = false, any_end = false;
    for (int s = 0; s < nsys; ++s) {
      any_active |= hflags[s].active != 0;
      any_end |= hflags[s].cycle_end != 0;
    }
    if (!any_active && !any_end) break;
    if (any_end) launch_cycle_end(st, pc, hflags, mask);
    else launch_arnoldi(st, pc, hflags, mask);
  }
  for (int s = 0; s < nsys; ++s) {
    res[s].iters = hflags[s].iters;
    res[s].rel_res = hflags[s].rel;
    res[s].status = hflags[s].status;
    res[s].nonfinite = hflags[s].nonfinite;
  }
  IBM_CUDA_TRY(cudaGetLastError());
}

namespace {

// Adds a conditional node after the current dependencies of the capture on
// `st` and makes it the new dependency; returns its body graphs.
void add_conditional(cudaStream_t st, cudaGraphConditionalHandle *h, cudaGraphConditionalNodeType type,
                     unsigned size, cudaGraph_t *bodies) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t *deps = nullptr;
  const cudaGraphEdgeData *ed = nullptr;
  size_t nd = 0;
  IBM_CUDA_TRY(cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, &deps, &ed, &nd));
  if (cs != cudaStreamCaptureStatusActive) throw Error(IBM_ERR_STATE, "graph capture not active");
  cudaGraphNodeParams p = {};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.handle = *h;
  p.conditional.type = type;
  p.conditional.size = size;
  cudaGraphNode_t node;
  IBM_CUDA_TRY(cudaGraphAddNode(&node, g, deps, ed, nd, &p));
  for (unsigned i = 0; i < size; ++i) bodies[i] = p.conditional.phGraph_out[i];
  IBM_CUDA_TRY(cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
}

cudaGraph_t capture_graph_of(cudaStream_t st) {
  cudaStreamCaptureStatus cs;
  cudaGraph_t g = nullptr;
  IBM_CUDA_TRY(cudaStreamGetCaptureInfo(st, &cs, nullptr, &g, nullptr, nullptr, nullptr));
  return g;
}

template <class F>
long long capture_body(cudaGraph_t body, cudaStream_t bs, F &&fn) {
  const long long before = launches();
  IBM_CUDA_TRY(cudaStreamBeginCaptureToGraph(bs, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
  fn(bs);
  cudaGraph_t out = nullptr;
  IBM_CUDA_TRY(cudaStreamEndCapture(bs, &out));
  return launches() - before;
}

}  // namespace

Krylov::GraphCounts Krylov::enqueue_graph(cudaStream_t st, cudaStream_t body_st, const Precond &pc,
                                          KFlags *host_flags, unsigned long long *loops) {
  GraphCounts gc;
  const long long t0 = launches();
  const dim3 grid(nblk, nsys);
  const unsigned mask = bound_mask;
  {
    LaunchScope ls(K_GM_INIT, st, 0.0);
    k_init<<<wave(k_init), kThreads, 0, st>>>(pack);
  }
  cudaGraphConditionalHandle hw;
  IBM_CUDA_TRY(cudaGraphConditionalHandleCreate(&hw, capture_graph_of(st), 0, 0));
  {
    LaunchScope ls(K_GM_UPDATE, st, 0.0);
    k_set_while<<<1, 32, 0, st>>>(pack, nsys, hw, nullptr);
  }
  cudaGraph_t wbody;
  add_conditional(st, &hw, cudaGraphCondTypeWhile, 1, &wbody);
  gc.loop = capture_body(wbody, body_st, [&](cudaStream_t b0) {
    // One body for the step and the cycle's end: a SWITCH node and its control
    // kernel cost about 6 us an iteration and a cycle's end an iteration of its
    // own, the three kernels that mostly return at once 1.2 us each. The residual
    // is launched again for systems whose double-float one was too close to the
    // tolerance to call. Steps in us: FP64 160x32x32 3955 -> 3712, 97x33x21
    // 4495 -> 4255, 320x64x64 270 less, twelve channels 38.2 -> 36.9 ms. (A second
    // loop for the ends that apply the preconditioner, inside or beside this one,
    // cost 20 us a solve without any.)
    launch_arnoldi(b0, pc, nullptr, mask);
    launch_cycle_end(b0, pc, nullptr, mask);
    bool df = false;
    for (int s = 0; s < nsys; ++s) df |= pack.s[s].df_resid != 0;
    if (df) {
      LaunchScope ls(K_GM_RESID, b0, 0.0);
      k_cycle_residual<<<wave(k_cycle_residual), kThreads, 0, b0>>>(pack);
    }
    LaunchScope ls(K_GM_UPDATE, b0, 0.0);
    k_set_while<<<1, 32, 0, b0>>>(pack, nsys, hw, loops);
  });
  {
    LaunchScope ls(K_GM_UPDATE, st, 0.0);
    k_flags<<<1, 32, 0, st>>>(pack, nsys, dflags.p);
  }
  IBM_CUDA_TRY(cudaMemcpyAsync(host_flags, dflags.p, sizeof(KFlags) * nsys, cudaMemcpyDeviceToHost, st));
  gc.fixed = (launches() - t0) - gc.loop;
  return gc;
}

}  // namespace ibm
