// tables.cu -- B-spline grid, cell moments, diagonal-cell integrals and the
// assembled R^k / S^k tables, all computed on the device in FP64.
//
// The grid, the Gauss points and the B-splines follow the operation order of the
// reference routines (cited per kernel), with explicit round-to-nearest
// intrinsics where those form a product and then a sum.  The moments, the
// diagonal cells and the tables hold the same sums in another order, as fused
// multiply-adds: a table element whose pairs share no cell is the product of two
// sums of moments, the others take suffix and prefix sums over the cells.  All of
// them agree with the reference's loops within 1e-14 of the largest element.
#include "ff.cuh"
#include "internal.cuh"
#include "pairs.cuh"

#include <algorithm>
#include <cmath>

#define IDX2(i, j, n1) ((size_t)(i) + (size_t)(n1) * (size_t)(j))
#define IDX3(i, j, k, n1, n2) ((size_t)(i) + (size_t)(n1) * ((size_t)(j) + (size_t)(n2) * (size_t)(k)))

// ----------------------------------------------------------------------------
// gauleg on [0,1]: dbsr_lib_zcom.f90:1990-2039 (Newton on the Legendre
// recurrence).  One thread; n is the spline order.
__global__ void k_gauleg(int n, double *x, double *w) {
  const double EPS = 1.0e-14;
  int m = (n + 1) / 2;
  double xm = 0.5, xl = 0.5;
  for (int i = 1; i <= m; i++) {
    double z = cos(__ddiv_rn(__dmul_rn(3.141592654, (i - 0.25)), (n + 0.5)));
    double z1, pp, p1, p2, p3;
    do {
      p1 = 1.0;
      p2 = 0.0;
      for (int j = 1; j <= n; j++) {
        p3 = p2;
        p2 = p1;
        p1 = __ddiv_rn(__dsub_rn(__dmul_rn(__dmul_rn(2.0 * j - 1.0, z), p2),
                                 __dmul_rn(j - 1.0, p3)),
                       (double)j);
      }
      pp = __ddiv_rn(__dmul_rn((double)n, __dsub_rn(__dmul_rn(z, p1), p2)),
                     __dsub_rn(__dmul_rn(z, z), 1.0));
      z1 = z;
      z = __dsub_rn(z1, __ddiv_rn(p1, pp));
    } while (fabs(z - z1) > EPS);
    x[i - 1] = __dsub_rn(xm, __dmul_rn(xl, z));
    x[n - i] = __dadd_rn(xm, __dmul_rn(xl, z));
    w[i - 1] = __ddiv_rn(2.0 * xl, __dmul_rn(__dmul_rn(__dsub_rn(1.0, __dmul_rn(z, z)), pp), pp));
    w[n - i] = w[i - 1];
  }
}

// Gauss points per interval: alloc_DBS_gauss, dbsr_lib_dbs.f90:929-936.
__global__ void k_gauss_points(int nv, int ks, const double *t, const double *gx,
                               const double *gw, double *gr, double *grm, double *grw) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nv * ks) return;
  int iv = q % nv, m = q / nv;  // 0-based
  double tl = t[ks + iv - 1], tr = t[ks + iv];
  double h = __dsub_rn(tr, tl);
  double r = __dadd_rn(__dmul_rn(h, gx[m]), tl);
  gr[q] = r;
  grm[q] = __ddiv_rn(1.0, r);
  grw[q] = __dmul_rn(h, gw[m]);
}

// Knots of a component basis: Def_pbsp / Def_qbsp, dbsr_lib_dbs.f90:997-999.
__global__ void k_sub_knots(int ns, int ks, int kx, int nsx, const double *t, double *tx) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;  // 1-based
  if (i > nsx + kx) return;
  double v;
  if (i <= kx)
    v = t[0];
  else if (i <= nsx)
    v = t[ks + (i - kx) - 1];
  else
    v = t[ns + (i - nsx) - 1];
  tx[i - 1] = v;
}

// B-spline values at the Gauss points, bsp(nv+1,ks,kx): Def_pbsp /
// Def_qbsp (dbsr_lib_dbs.f90:1003-1020); row nv+1 holds the values at the
// last knot in its first column.
__global__ void k_bsp_values(int nv, int ks, int kx, int nsx, const double *tx,
                             const double *gr, double *bsp) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  const int nw = nv + 1;
  if (q >= nw * ks) return;
  int iv = q % nw, m = q / nw;
  double v[DBSRG_MAXK];
  if (iv < nv) {
    bspline_values(tx, kx, kx + iv, gr[IDX2(iv, m, nv)], v);
  } else if (m == 0) {
    bspline_values(tx, kx, nsx, tx[nsx], v);
  } else {
    for (int j = 0; j < kx; j++) v[j] = 0.0;
  }
  for (int j = 0; j < kx; j++) bsp[IDX3(iv, m, j, nw, ks)] = v[j];
}

// Banded Gram matrix ym(i,j) = <B1_i|y|B2_j>: ZINTYM, dbsr_lib_dbs.f90:4472-4497.
// ym has leading dimension ld and is written at offset (off,off).
__global__ void k_gram(int ns, int nv, int ks, int kx, const double *b, const double *ygr,
                       double *ym, int ld, int off) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= ns * ns) return;
  int i = q % ns + 1, j = q / ns + 1;  // 1-based
  const int nw = nv + 1;
  double acc = 0.0;
  int lo = max(max(1, i - kx + 1), j - kx + 1), hi = min(min(nv, i), j);
  for (int iv = lo; iv <= hi; iv++) {
    int ith = i - iv + 1, jth = j - iv + 1;
    double s = 0.0;
    for (int m = 0; m < ks; m++) {
      double p = __dmul_rn(__dmul_rn(ygr[IDX2(iv - 1, m, nv)], b[IDX3(iv - 1, m, ith - 1, nw, ks)]),
                           b[IDX3(iv - 1, m, jth - 1, nw, ks)]);
      s = __dadd_rn(s, p);
    }
    acc = __dadd_rn(acc, s);
  }
  ym[IDX2(off + i - 1, off + j - 1, ld)] = acc;
}

static int build_triang_points(dbsrg_ctx *c);

int build_grid(dbsrg_ctx *c, const double *t_in) {
  DeviceGrid &g = c->g;
  const int ns = g.ns, ks = g.ks, nv = g.nv, nw = nv + 1, ms = g.ms;
  auto alloc = [&](double **p, size_t n) -> cudaError_t {
    return cudaMalloc((void **)p, sizeof(double) * (n > 0 ? n : 1));
  };
  DBSRG_TRY(c, alloc(&g.t, ns + ks));
  DBSRG_TRY(c, alloc(&g.tp, g.nsp + g.ksp));
  DBSRG_TRY(c, alloc(&g.tq, g.nsq + g.ksq));
  DBSRG_TRY(c, alloc(&g.gx, ks));
  DBSRG_TRY(c, alloc(&g.gw, ks));
  DBSRG_TRY(c, alloc(&g.gr, (size_t)nv * ks));
  DBSRG_TRY(c, alloc(&g.grw, (size_t)nv * ks));
  DBSRG_TRY(c, alloc(&g.grm, (size_t)nv * ks));
  DBSRG_TRY(c, alloc(&g.pbsp, (size_t)nw * ks * g.ksp));
  DBSRG_TRY(c, alloc(&g.qbsp, (size_t)nw * ks * g.ksq));
  DBSRG_TRY(c, alloc(&g.fpbs, (size_t)ns * ns));
  DBSRG_TRY(c, alloc(&g.fqbs, (size_t)ns * ns));
  DBSRG_TRY(c, alloc(&g.fppqq, (size_t)ms * ms));
  int rc = copy_in(c, g.t, t_in, sizeof(double) * (ns + ks));
  if (rc) return rc;
  cudaStream_t s = c->stream;
  DBSRG_RUN(c, "k_gauleg", k_gauleg<<<1, 1, 0, s>>>(ks, g.gx, g.gw));
  int nt = nv * ks;
  DBSRG_RUN(c, "k_gauss_points", k_gauss_points<<<(nt + 127) / 128, 128, 0, s>>>(nv, ks, g.t, g.gx, g.gw, g.gr, g.grm, g.grw));
  DBSRG_RUN(c, "k_sub_knots", k_sub_knots<<<(g.nsp + g.ksp + 127) / 128, 128, 0, s>>>(ns, ks, g.ksp, g.nsp, g.t, g.tp));
  DBSRG_RUN(c, "k_sub_knots", k_sub_knots<<<(g.nsq + g.ksq + 127) / 128, 128, 0, s>>>(ns, ks, g.ksq, g.nsq, g.t, g.tq));
  int nb = nw * ks;
  DBSRG_RUN(c, "k_bsp_values", k_bsp_values<<<(nb + 127) / 128, 128, 0, s>>>(nv, ks, g.ksp, g.nsp, g.tp, g.gr, g.pbsp));
  DBSRG_RUN(c, "k_bsp_values", k_bsp_values<<<(nb + 127) / 128, 128, 0, s>>>(nv, ks, g.ksq, g.nsq, g.tq, g.gr, g.qbsp));
  int nn = ns * ns;
  DBSRG_RUN(c, "k_gram", k_gram<<<(nn + 255) / 256, 256, 0, s>>>(ns, nv, ks, g.ksp, g.pbsp, g.grw, g.fpbs, ns, 0));
  DBSRG_RUN(c, "k_gram", k_gram<<<(nn + 255) / 256, 256, 0, s>>>(ns, nv, ks, g.ksq, g.qbsp, g.grw, g.fqbs, ns, 0));
  DBSRG_TRY(c, cudaMemsetAsync(g.fppqq, 0, sizeof(double) * (size_t)ms * ms, s));
  DBSRG_RUN(c, "k_gram", k_gram<<<(nn + 255) / 256, 256, 0, s>>>(ns, nv, ks, g.ksp, g.pbsp, g.grw, g.fppqq, ms, 0));
  DBSRG_RUN(c, "k_gram", k_gram<<<(nn + 255) / 256, 256, 0, s>>>(ns, nv, ks, g.ksq, g.qbsp, g.grw, g.fppqq, ms, ns));
  if ((rc = build_triang_points(c))) return rc;
  DBSRG_TRY(c, cudaStreamSynchronize(s));
  return DBSRG_OK;
}

// ----------------------------------------------------------------------------
// Cell moments <B_i|r^k|B_j> per interval: moment_pp/qq/pq/qp,
// dbsr_lib_dbs.f90:1401-1564.  rkm(ks*ks,nv); pp/qq packed i<=j.
// up to four moment arrays per launch (blockIdx.y): the moments of one cell
// data set
struct MomentSet {
  const double *b1s[4], *b2s[4];
  int k1[4], k2[4], sym[4], k[4];
  double *rkm[4];
};

// One block per cell and array: the weights r^k w(m) and the functions' values
// once in shared memory, a thread per pair.  ns 283, four arrays: 10 us, 16.4
// with a power per thread and point.
__global__ void __launch_bounds__(128) k_moments(int nv, int ks, const MomentSet ms,
                                                 const double *gr, const double *grm,
                                                 const double *grw) {
  __shared__ double w[DBSRG_MAXK], B1[DBSRG_MAXK * DBSRG_MAXK], B2[DBSRG_MAXK * DBSRG_MAXK];
  const int y = blockIdx.y, iv = blockIdx.x, tid = threadIdx.x;
  const double *b1s = ms.b1s[y], *b2s = ms.b2s[y];
  const int k1 = ms.k1[y], k2 = ms.k2[y], sym = ms.sym[y], k = ms.k[y];
  const int nw = nv + 1, kk = ks * ks;
  double *rkm = ms.rkm[y] + (size_t)kk * iv;
  if (tid < ks) {
    double v = grw[IDX2(iv, tid, nv)];
    if (k > 0) v = __dmul_rn(v, ipow_d(gr[IDX2(iv, tid, nv)], k));
    if (k < 0) v = __dmul_rn(v, ipow_d(grm[IDX2(iv, tid, nv)], -k));
    w[tid] = v;
  }
  for (int q = tid; q < ks * k1; q += 128) B1[q] = b1s[IDX3(iv, q % ks, q / ks, nw, ks)];
  for (int q = tid; q < ks * k2; q += 128) B2[q] = b2s[IDX3(iv, q % ks, q / ks, nw, ks)];
  __syncthreads();
  const int npair = sym ? k1 * (k1 + 1) / 2 : k1 * k2;
  for (int ii = tid; ii < kk; ii += 128) {
    double s = 0.0;
    if (ii < npair) {
      int i, j;
      if (sym) {  // invert the packed upper-triangular index
        int r = ii, row = 0;
        while (r >= k1 - row) {
          r -= k1 - row;
          row++;
        }
        i = row;
        j = row + r;
      } else {
        i = ii / k2;
        j = ii % k2;
      }
      for (int m = 0; m < ks; m++) s = fma(B1[m + ks * i], __dmul_rn(B2[m + ks * j], w[m]), s);
    }
    rkm[ii] = s;
  }
}

static void basis_of(const DeviceGrid &g, int which, const double **b1, const double **b2,
                     int *k1, int *k2, int *sym) {
  switch (which) {
    case 0: *b1 = g.pbsp; *b2 = g.pbsp; *k1 = g.ksp; *k2 = g.ksp; *sym = 1; break;
    case 1: *b1 = g.qbsp; *b2 = g.qbsp; *k1 = g.ksq; *k2 = g.ksq; *sym = 1; break;
    case 2: *b1 = g.pbsp; *b2 = g.qbsp; *k1 = g.ksp; *k2 = g.ksq; *sym = 0; break;
    default: *b1 = g.qbsp; *b2 = g.pbsp; *k1 = g.ksq; *k2 = g.ksp; *sym = 0; break;
  }
}

// n (1..4) moment arrays in one launch: basis pair which[i], power k[i]
static int compute_moment_set(dbsrg_ctx *c, int n, const int *which, const int *k,
                              double *const *rkm) {
  const DeviceGrid &g = c->g;
  MomentSet ms{};
  for (int i = 0; i < n; i++) {
    basis_of(g, which[i], &ms.b1s[i], &ms.b2s[i], &ms.k1[i], &ms.k2[i], &ms.sym[i]);
    ms.k[i] = k[i];
    ms.rkm[i] = rkm[i];
  }
  DBSRG_RUN(c, "k_moments", k_moments<<<dim3(g.nv, n), 128, 0, c->stream>>>(g.nv, g.ks, ms, g.gr,
                                                                           g.grm, g.grw));
  return DBSRG_OK;
}

int compute_moments(dbsrg_ctx *c, int which, int k, double *rkm) {
  return compute_moment_set(c, 1, &which, &k, &rkm);
}

// ----------------------------------------------------------------------------
// Diagonal-cell integrals triang_*: dbsr_lib_dbs.f90:2979-3063 (pppp),
// 3151-3245 (pqpq), 3333-3427 (qpqp), 3512-3597 (qqqq), 3682-3767 (ppqq),
// 3852-3936 (pqqp).  One thread block per interval iv.  For each outer
// Gauss point r2 = gr(iv,m) the inner integral of B_j B_jp r^k over
// [t_iv, r2] uses ks Gauss points; B-splines at the inner points come from
// the same de Boor recursion as zbsplvd.
//   type 0 pppp, 1 qqqq: rkd = a + a^T, a(outer pair, inner pair)
//   type 2 pqpq: rkd(P pair, Q pair) = sum bp*INTQ + sum bq*INTP
//   type 3 qpqp: rkd(Q pair, P pair) = the same two sums
//   type 4 ppqq: rkd(inner (P,Q), outer (P,Q))
//   type 5 pqqp: rkd(inner (P,Q), outer (Q,P))
// Inner points of the diagonal cells of every interval iv: for outer point
// r2 = gr(iv,m) the inner Gauss points x = t_iv + (r2 - t_iv) gx(i) on
// [t_iv, r2], their weights (r2 - t_iv) gw(i) and the P and Q B-splines
// there (zbsplvd recursion); one thread per (iv, m, i).
__global__ void k_triang_points(int nv, int ks, int ksp, int ksq, const double *t,
                                const double *tp, const double *tq, const double *gx,
                                const double *gw, const double *gr, double *tri) {
  const int KS2 = ks * ks;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nv * KS2) return;
  const int iv = q / KS2, p = q % KS2, m = p / ks, i = p % ks;
  double *tb = tri + (size_t)iv * KS2 * (2 + ksp + ksq);
  const double xbase = t[iv + ks - 1];
  const double r2 = gr[IDX2(iv, m, nv)];
  const double d = __dsub_rn(r2, xbase);
  const double x = __dadd_rn(__dmul_rn(d, gx[i]), xbase);
  tb[p] = x;
  tb[KS2 + p] = __dmul_rn(d, gw[i]);
  double v[DBSRG_MAXK];
  bspline_values(tp, ksp, iv + ksp, x, v);
  for (int j = 0; j < ksp; j++) tb[2 * KS2 + (size_t)p * ksp + j] = v[j];
  bspline_values(tq, ksq, iv + ksq, x, v);
  for (int j = 0; j < ksq; j++) tb[2 * KS2 + (size_t)KS2 * ksp + (size_t)p * ksq + j] = v[j];
}

// up to three types per launch (blockIdx.y); out: element (pair 1, pair 2; cell)
// at p1 + ld p2 + cell size, no padding where ld is 0 (float-float copy: never
// padded)
struct TriSet {
  int type[3];
  double *rkd[3];
  float2 *rkf[3];
};

// One block per interval and type.  INT (inner integrals) and OB (outer weight
// times two functions) are arrays [pair][outer point] of the type's pairs, of
// odd stride so that a warp's pairs fall on different banks; an element of the
// result is a dot product (types 2 and 3: two) over the outer points.  Bound by
// the FP64 pipe once the integer work per element is small and no padding is
// written: ns 400, R^k (three types) and S^k launches 98 us in the mean with the
// functions' square for INT, the pair's two functions searched for at every
// element and ks^2 x ks^2 results; 69 us here (ns 283: 59 and 50).
__global__ void __launch_bounds__(256) k_triang(int nv, int ks, int ksp, int ksq, const TriSet ts,
                                                int ld, int k, const double *tri,
                                                const double *grm, const double *grw,
                                                const double *pbsp, const double *qbsp) {
  extern __shared__ double sm[];
  const int iv = blockIdx.x;  // 0-based interval
  const int type = ts.type[blockIdx.y];
  float2 *rkf = ts.rkf[blockIdx.y];
  const int nw = nv + 1, KS2 = ks * ks, kr = ks | 1;
  const int ikp = ksp * (ksp + 1) / 2, ikq = ksq * (ksq + 1) / 2, npq = ksp * ksq;
  const bool needP = type != 1, needQ = type != 0;
  // the pairs of the two arrays: 1 for the first family, 2 for the second (types
  // 2 and 3: P and Q)
  const int m1 = type == 1 ? ikq : (type >= 4 ? npq : ikp), m2 = type == 2 || type == 3 ? ikq : 0;
  const double *tb = tri + (size_t)iv * KS2 * (2 + ksp + ksq);  // x | w | BP | BQ
  double *wk = sm;                 // (m,i) inner weight * r^k       [ks*ks]
  double *BP = wk + KS2;           // (m,i,j) P values at inner pts  [ks*ks*ksp]
  double *BQ = BP + KS2 * ksp;     // (m,i,j) Q values               [ks*ks*ksq]
  double *gxo = BQ + KS2 * ksq;    // outer weights                  [ks]
  double *INT1 = gxo + ks;         //                                [m1][kr]
  double *OB1 = INT1 + m1 * kr;    //                                [m1][kr]
  double *INT2 = OB1 + m1 * kr;    //                                [m2][kr]
  double *OB2 = INT2 + m2 * kr;    //                                [m2][kr]
  double *A = OB2 + m2 * kr;       // weighted functions, then types 0/1: a(ii,jj)
  __shared__ unsigned char fn[2][2][DBSRG_MAXK * (DBSRG_MAXK + 1) / 2];  // pairs' functions

  // phase 1: inner points, weights and B-spline values (k_triang_points)
  for (int q = threadIdx.x; q < KS2; q += blockDim.x)
    wk[q] = __dmul_rn(tb[KS2 + q], ipow_d(tb[q], k));
  for (int q = threadIdx.x; q < KS2 * (ksp + ksq); q += blockDim.x)
    BP[q] = tb[2 * KS2 + q];  // BQ follows BP in both layouts
  for (int m = threadIdx.x; m < ks; m += blockDim.x)
    gxo[m] = __dmul_rn(grw[IDX2(iv, m, nv)], ipow_d(grm[IDX2(iv, m, nv)], k + 1));
  for (int q = threadIdx.x; q < ikp + ikq; q += blockDim.x) {
    const int w = q >= ikp, kx = w ? ksq : ksp;
    int r = w ? q - ikp : q, row = 0;
    const int at = r;
    while (r >= kx - row) {
      r -= kx - row;
      row++;
    }
    fn[w][0][at] = (unsigned char)row;
    fn[w][1][at] = (unsigned char)(row + r);
  }
  __syncthreads();
  // phase 2: INT(pair, m) = sum_i (wk*Ba_j)*Bb_jp
  // (the weighted first factors wk*Ba are formed once per call in A, which
  // phase 3 fills only after the last call); w: packed symmetric pairs of P (0)
  // or Q (1), 2: (P, Q) pairs
  auto inner = [&](const double *Ba, int ka, const double *Bb, int kb, int w, int np,
                   double *INT) {
    double *WB = A;
    for (int q = threadIdx.x; q < KS2 * ka; q += blockDim.x) WB[q] = __dmul_rn(wk[q / ka], Ba[q]);
    __syncthreads();
    for (int q = threadIdx.x; q < np * ks; q += blockDim.x) {
      const int pr = q / ks, m = q - pr * ks;
      const int j = w < 2 ? fn[w][0][pr] : pr / kb, jp = w < 2 ? fn[w][1][pr] : pr % kb;
      const double *a = WB + (size_t)m * ks * ka + j, *b = Bb + (size_t)m * ks * kb + jp;
      double s = 0.0;
      for (int i = 0; i < ks; i++) s = fma(a[i * ka], b[i * kb], s);
      INT[pr * kr + m] = s;
    }
    __syncthreads();
  };
  if (type >= 4) {
    inner(BP, ksp, BQ, ksq, 2, npq, INT1);
  } else {
    if (needP) inner(BP, ksp, BP, ksp, 0, ikp, INT1);
    if (needQ) inner(BQ, ksq, BQ, ksq, 1, ikq, type == 1 ? INT1 : INT2);
  }
  // outer products b1(m,i) b2(m,ip) gxo(m) per pair and outer point
  auto ob = [&](const double *b1, int i, const double *b2, int ip, int m) -> double {
    return __dmul_rn(__dmul_rn(b1[IDX3(iv, m, i, nw, ks)], b2[IDX3(iv, m, ip, nw, ks)]), gxo[m]);
  };
  auto outer = [&](int w, int np, double *OB) {
    const double *bs = w ? qbsp : pbsp;
    for (int q = threadIdx.x; q < np * ks; q += blockDim.x) {
      const int pr = q / ks, m = q - pr * ks;
      OB[pr * kr + m] = ob(bs, fn[w][0][pr], bs, fn[w][1][pr], m);
    }
  };
  if (type >= 4) {  // outer (P,Q) pairs ii = i*ksq + ip, or (Q,P) ii = i*ksp + ip
    for (int q = threadIdx.x; q < npq * ks; q += blockDim.x) {
      const int ii = q / ks, m = q - ii * ks;
      OB1[ii * kr + m] = type == 4 ? ob(pbsp, ii / ksq, qbsp, ii % ksq, m)
                                   : ob(qbsp, ii / ksp, pbsp, ii % ksp, m);
    }
  } else {
    if (needP) outer(0, ikp, OB1);
    if (needQ) outer(1, ikq, type == 1 ? OB1 : OB2);
  }
  __syncthreads();
  // element (r, cc) of the result, n1 x n2
  const int n1 = type == 3 ? ikq : m1, n2 = type == 2 ? ikq : m1;
  const int l2 = ld ? ld : n1;
  double *out = ts.rkd[blockIdx.y] + (size_t)(ld ? ld * ld : n1 * n2) * iv;
  if (rkf) rkf += (size_t)n1 * n2 * iv;
  if (type < 2) {
    for (int q = threadIdx.x; q < n1 * n1; q += blockDim.x) {
      const int jj = q / n1, ii = q - jj * n1;
      const double *o = OB1 + ii * kr, *t = INT1 + jj * kr;
      double s = 0.0;
      for (int m = 0; m < ks; m++) s = fma(o[m], t[m], s);
      A[q] = s;
    }
    __syncthreads();
  }
  for (int q = threadIdx.x; q < n1 * n2; q += blockDim.x) {
    const int cc = q / n1, r = q - cc * n1;
    double v;
    if (type < 2) {
      v = __dadd_rn(A[q], A[cc + n1 * r]);
    } else if (type < 4) {
      const int pp = type == 2 ? r : cc, qq = type == 2 ? cc : r;  // P pair, Q pair
      const double *o1 = OB1 + pp * kr, *t2 = INT2 + qq * kr;
      const double *o2 = OB2 + qq * kr, *t1 = INT1 + pp * kr;
      double s1 = 0.0, s2 = 0.0;
      for (int m = 0; m < ks; m++) {
        s1 = fma(o1[m], t2[m], s1);
        s2 = fma(o2[m], t1[m], s2);
      }
      v = __dadd_rn(s1, s2);
    } else {  // rkd(jj,ii): jj inner (P,Q), ii outer
      const double *o = OB1 + cc * kr, *t = INT1 + r * kr;
      v = 0.0;
      for (int m = 0; m < ks; m++) v = fma(o[m], t[m], v);
    }
    out[r + (size_t)l2 * cc] = v;
    if (rkf) rkf[q] = ffa::split(v);
  }
}

static int build_triang_points(dbsrg_ctx *c) {
  DeviceGrid &g = c->g;
  const int KS2 = g.ks * g.ks;
  const size_t n = (size_t)g.nv * KS2 * (2 + g.ksp + g.ksq);
  DBSRG_TRY(c, cudaMalloc((void **)&g.tri, n * sizeof(double)));
  const int nq = g.nv * KS2;
  DBSRG_RUN(c, "k_triang_points",
            k_triang_points<<<(nq + 127) / 128, 128, 0, c->stream>>>(
                g.nv, g.ks, g.ksp, g.ksq, g.t, g.tp, g.tq, g.gx, g.gw, g.gr, g.tri));
  return DBSRG_OK;
}

// n (1..3) types in one launch; ld: as in TriSet
static int compute_diag_set(dbsrg_ctx *c, int n, const TriSet &ts, int k, int ld = 0) {
  const DeviceGrid &g = c->g;
  const size_t ks = g.ks, kr = ks | 1, ikp = g.ksp * (g.ksp + 1) / 2,
               ikq = g.ksq * (g.ksq + 1) / 2, kmax = std::max(g.ksp, g.ksq);
  // the largest type's arrays (k_triang): pairs of both families or the (P,Q)
  // pairs; weighted functions or the square of the larger family's pairs
  const size_t pairs = std::max(ikp + ikq, (size_t)g.ksp * g.ksq);
  const size_t am = std::max(std::max(ikp * ikp, ikq * ikq), ks * ks * kmax);
  const size_t bytes =
      sizeof(double) * (ks * ks * (1 + g.ksp + g.ksq) + ks + 2 * pairs * kr + am);
  int rc = raise_smem_limit(c, (const void *)k_triang, bytes);
  if (rc) return rc;
  DBSRG_RUN(c, "k_triang",
            k_triang<<<dim3(g.nv, n), 256, bytes, c->stream>>>(g.nv, g.ks, g.ksp, g.ksq, ts, ld, k,
                                                               g.tri, g.grm, g.grw, g.pbsp,
                                                               g.qbsp));
  return DBSRG_OK;
}

// one type's cells as ks^2 x ks^2 arrays, zeros past the pairs
int compute_diag_cells(dbsrg_ctx *c, int type, int k, double *rkd) {
  const int kk = c->g.ks * c->g.ks;
  TriSet ts{};
  ts.type[0] = type;
  ts.rkd[0] = rkd;
  DBSRG_TRY(c, cudaMemsetAsync(rkd, 0, sizeof(double) * kk * kk * c->g.nv, c->stream));
  return compute_diag_set(c, 1, ts, k, kk);
}

// ----------------------------------------------------------------------------
// R^k table fill: mrk_pppp/qqqq/pqpq/qpqp, dbsr_lib_dbs.f90:2898-2959,
// 3431-3492, 3067-3131, 3249-3313.  One thread per table element
// rkb(i,j,ip,jp), which gathers its cell contributions (k_fill_r).
__device__ __forceinline__ int tri_index(int h, int hp, int kx) {  // 1-based
  return (h - 1) * kx - ((h - 1) * (h - 2)) / 2 + (hp - h + 1);
}

// Sums over all cells of a function pair's moments, [i + ns ip] for the pair
// (i, i+ip) of one basis ('s', ip = 0..ks-1) or (i, i+ip-ks+1) of two: a table
// element whose two electrons' pairs share no cell is the product of two of them.
// up to four arrays per launch (blockIdx.y)
struct TotalSet {
  int k1[4], k2[4], sym[4];
  const double *M[4];
  double *T[4];
};

__global__ void k_moment_sums(int ns, int ks, int nv, const TotalSet ts) {
  const int y = blockIdx.y, k1 = ts.k1[y], k2 = ts.k2[y], sym = ts.sym[y], kk = ks * ks;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= ns * (sym ? ks : 2 * ks - 1)) return;
  const int i = q % ns + 1, off = q / ns - (sym ? 0 : ks - 1);  // second function i + off
  const double *M = ts.M[y];
  double s = 0.0;
  // (first function's places nine at a time, their loads in flight together)
  for (int h0 = max(1, 1 - off); h0 <= min(k1, k2 - off); h0 += 9) {
    double v[9];
#pragma unroll
    for (int u = 0; u < 9; u++) {
      const int h = h0 + u, iv = i - h + 1;
      const bool ok = h <= min(k1, k2 - off) && iv >= 1 && iv <= nv;
      const int p = sym ? (h - 1) * k1 - ((h - 1) * (h - 2)) / 2 + off : (h - 1) * k2 + h + off - 1;
      v[u] = ok ? M[(size_t)p + (size_t)kk * (iv - 1)] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 9; u++) s += v[u];
  }
  ts.T[y][q] = s;
}

// band > 0: only the elements with |j - i| <= band, stored as
// rkb(i, j-i+band+1, ip, jp) of shape (ns, 2*band+1, ks, ks) -- all that the
// band part of the factored exchange reads.
// Up to three tables per launch (blockIdx.y); tr: rkd has the electron-2 pair
// first.  Bound by the FP64 pipe in the elements whose pairs share cells; the
// others, two thirds of a band and most of a whole table, are one product of
// k_moment_sums' sums.  ns 283, bands of three types 86 -> 44 us (S^k, one type
// 55 -> 33), ns 400 120 -> 59 (77 -> 45), against a loop over the cells each.
struct FillSet {
  int ka[3], kb[3], tr[3];
  const double *lowA[3], *highA[3], *lowB[3], *highB[3], *rkd[3];
  const double *TlowA[3], *ThighA[3], *TlowB[3], *ThighB[3];  // k_moment_sums
  double *rkb[3];
};

__global__ void k_fill_r(int ns, int ks, int nv, const FillSet fs, int band) {
  const int y = blockIdx.y, ka = fs.ka[y], kb = fs.kb[y];
  const double *lowA = fs.lowA[y], *highA = fs.highA[y], *lowB = fs.lowB[y], *highB = fs.highB[y],
               *rkd = fs.rkd[y];
  double *rkb = fs.rkb[y];
  const bool tr = fs.tr[y];
  size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nj = band > 0 ? 2 * band + 1 : ns;
  size_t total = (size_t)ns * nj * ks * ks;
  if (q >= total) return;
  const int kk = ks * ks;
  int i = (int)(q % ns) + 1;
  size_t r = q / ns;
  int j = (int)(r % nj) + 1;
  if (band > 0) j = i + (j - 1) - band;
  r /= nj;
  int ip = (int)(r % ks) + 1;
  int jp = (int)(r / ks) + 1;
  double acc = 0.0;
  if (ip <= ka && jp <= kb && j >= 1 && j <= ns) {
    const int ivlo = max(1, i - ka + ip), ivhi = min(nv, i);
    const int jvlo = max(1, j - kb + jp), jvhi = min(nv, j);
    const int ti = i - 1 + ns * (ip - 1), tj = j - 1 + ns * (jp - 1);
    if (ivhi < jvlo) {
      rkb[q] = fs.TlowA[y][ti] * fs.ThighB[y][tj];
      return;
    }
    if (jvhi < ivlo) {
      rkb[q] = fs.ThighA[y][ti] * fs.TlowB[y][tj];
      return;
    }
    // moment positions of the electron-1 pair in cell iv and the electron-2
    // pair in cell jv
    auto ia = [&](int iv) {
      const int ih = i - iv + 1;
      return (size_t)(tri_index(ih, ih + ip - 1, ka) - 1) + (size_t)kk * (iv - 1);
    };
    auto jb = [&](int jv) {
      const int jh = j - jv + 1;
      return (size_t)(tri_index(jh, jh + jp - 1, kb) - 1) + (size_t)kk * (jv - 1);
    };
    // the separable cells: iv < jv adds lowA(iv) times the sum of highB over
    // the cells jv > iv, iv > jv adds highA(iv) times the sum of lowB over
    // jv < iv.  Both sums are formed by additions only (the moments of
    // B-spline products are positive), suffix sums with iv descending and
    // prefix sums with iv ascending, so every element keeps full relative
    // precision with O(ka + kb) operations instead of O(ka kb).
    const int na = ka * (ka + 1) / 2, nbp = kb * (kb + 1) / 2;
    const size_t n1 = tr ? nbp : na, n2 = tr ? na : nbp;  // pairs of rkd's two indices
    double suf = 0.0;
    for (int jv = jvhi; jv >= max(jvlo, ivhi + 1); jv--) suf += highB[jb(jv)];
    for (int iv = ivhi; iv >= ivlo; iv--) {
      acc = fma(lowA[ia(iv)], suf, acc);
      if (iv >= jvlo && iv <= jvhi) suf += highB[jb(iv)];
    }
    double pre = 0.0;
    for (int jv = jvlo; jv <= min(jvhi, ivlo - 1); jv++) pre += lowB[jb(jv)];
    for (int iv = ivlo; iv <= ivhi; iv++) {
      acc = fma(highA[ia(iv)], pre, acc);
      if (iv >= jvlo && iv <= jvhi) {  // the diagonal cell, then jv = iv joins the prefix
        const int ih = i - iv + 1, jh = j - iv + 1;
        const int ii = tri_index(ih, ih + ip - 1, ka), jj = tri_index(jh, jh + jp - 1, kb);
        const int r1 = tr ? jj : ii, r2 = tr ? ii : jj;
        acc += rkd[(r1 - 1) + n1 * ((r2 - 1) + n2 * (iv - 1))];
        pre += lowB[jb(iv)];
      }
    }
  }
  rkb[q] = acc;
}

// S^k table fill: msk_ppqq / msk_pqqp, dbsr_lib_dbs.f90:3601-3662,
// 3771-3833.  Only cells iv <= jv; band offsets ip = ihp-ih+ks.
__global__ void k_fill_s(int ns, int ks, int nv, int ksp, int ksq, int kj1, int kj2,
                         const double *r1, const double *r2, const double *T1, const double *T2,
                         const double *rkd, double *rkb, int band) {
  const int kb2 = 2 * ks - 1, kk = ks * ks;
  size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int nj = band > 0 ? 2 * band + 1 : ns;
  size_t total = (size_t)ns * nj * kb2 * kb2;
  if (q >= total) return;
  int i = (int)(q % ns) + 1;
  size_t r = q / ns;
  int j = (int)(r % nj) + 1;
  if (band > 0) j = i + (j - 1) - band;
  r /= nj;
  int ip = (int)(r % kb2) + 1;
  int jp = (int)(r / kb2) + 1;
  double acc = 0.0;
  if (j < 1 || j > ns) {
    rkb[q] = 0.0;
    return;
  }
  // electron 1: ih in [1,ksp], ihp = ip+ih-ks in [1,ksq], iv = i-ih+1
  const int ihlo = max(1, ks - ip + 1), ihhi = min(ksp, ks - ip + ksq);
  // electron 2: jh in [1,kj1], jhp = jp+jh-ks in [1,kj2], jv = j-jh+1
  const int jhlo = max(1, ks - jp + 1), jhhi = min(kj1, ks - jp + kj2);
  const int ivlo = max(1, i - ihhi + 1), ivhi = min(nv, i - ihlo + 1);
  const int jvlo = max(1, j - jhhi + 1), jvhi = min(nv, j - jhlo + 1);
  if (ivlo > ivhi || jvlo > jvhi || jvhi < ivlo) {
    rkb[q] = 0.0;
    return;
  }
  if (ivhi < jvlo) {
    rkb[q] = T1[i - 1 + ns * (ip - 1)] * T2[j - 1 + ns * (jp - 1)];
    return;
  }
  auto ia = [&](int iv) {  // (ii - 1) and the cell offset of electron 1
    const int ih = i - iv + 1;
    return (size_t)((ih - 1) * ksq + ip + ih - ks - 1);
  };
  auto jb = [&](int jv) {
    const int jh = j - jv + 1;
    return (size_t)((jh - 1) * kj2 + jp + jh - ks - 1);
  };
  // cells iv < jv: r1(iv) times the suffix sum of r2 over jv > iv (positive
  // moments, additions only, iv descending); the diagonal cells iv = jv
  const size_t npq = (size_t)ksp * ksq;  // pairs of either electron
  double suf = 0.0;
  for (int jv = jvhi; jv >= max(jvlo, ivhi + 1); jv--) suf += r2[jb(jv) + (size_t)kk * (jv - 1)];
  for (int iv = ivhi; iv >= ivlo; iv--) {
    acc = fma(r1[ia(iv) + (size_t)kk * (iv - 1)], suf, acc);
    if (iv >= jvlo && iv <= jvhi) {
      acc += rkd[ia(iv) + npq * (jb(iv) + npq * (iv - 1))];
      suf += r2[jb(iv) + (size_t)kk * (iv - 1)];
    }
  }
  rkb[q] = acc;
}

static int ensure_slot(dbsrg_ctx *c, std::vector<double *> &v, size_t idx) {
  if (v.size() <= idx) v.resize(idx + 1, nullptr);
  return 0;
}

// Cell moments and diagonal-cell integrals of one table (family, type, k),
// kept resident: the table fill and the factored contraction both read
// them (the R^k types of one k share theirs, ensure_r_cells).  R: lo1/hi1 = moments of the electron-1 basis at r^k / r^-(k+1),
// lo2/hi2 the same for electron 2 (mrk_*: rkd1..rkd4).  S: lo1 =
// moments_pq(k) of electron 1, hi2 = moments_pq or moments_qp(-(k+1)) of
// electron 2 (msk_*: rkd1, rkd2); hi1 = lo2 = null (no r1 > r2 cells).
int get_celldata(dbsrg_ctx *c, int family, int type, int k, const CellData **out) {
  const DeviceGrid &g = c->g;
  const int nv = g.nv, kk = g.ks * g.ks;
  const size_t m = (size_t)kk * nv;
  int rc;
  if (family == 0) {
    if ((rc = ensure_r_cells(c, k))) return rc;
    *out = &c->rcell[(size_t)k * 4 + type];
    return DBSRG_OK;
  }
  std::vector<CellData> &v = c->scell;
  const size_t idx = (size_t)k * 2 + type;
  if (v.size() <= idx) v.resize(idx + 1);
  if (v[idx].rkd) {
    *out = &v[idx];
    return DBSRG_OK;
  }
  const TableBases tb = table_bases(g, family, type);
  const size_t f = (size_t)npairs(tb.e1) * npairs(tb.e2) * nv;
  const size_t ts1 = (size_t)g.ns * (2 * g.ks - 1);  // sums of one moment array
  CacheBuffer buf(c, (2 * m + 2 * f + 2 * ts1) * sizeof(double));
  double *base = (double *)buf.p;
  if (!base) return set_err(c, DBSRG_ENOMEM, "cell data allocation failed");
  CellData cd;
  cd.lo1 = base;
  cd.hi2 = base + m;
  cd.rkd = base + 2 * m;
  cd.rkf = (float2 *)(cd.rkd + f);
  const int wh[2] = {2, type == 0 ? 2 : 3}, kp[2] = {k, -(k + 1)};
  double *const mo[2] = {cd.lo1, cd.hi2};
  TriSet ts{};
  ts.type[0] = type == 0 ? 4 : 5;
  ts.rkd[0] = cd.rkd;
  ts.rkf[0] = cd.rkf;
  if ((rc = compute_moment_set(c, 2, wh, kp, mo)) || (rc = compute_diag_set(c, 1, ts, k)))
    return rc;
  buf.keep();
  v[idx] = cd;
  *out = &v[idx];
  return DBSRG_OK;
}

// The R^k tables of one k: the moments of the P and Q pairs (four arrays, one
// launch; every type takes two of each) and the diagonal cells of types 0, 1
// and 2 (one launch; type 3 reads type 2's with the electrons exchanged).  A
// list takes all types of its k, so nothing is built that it does not read.
// ns 283, against a launch per type of the kernels of the day: moments 4 x 18 -> 18 us
// a k (10 now), diagonal cells 4 x 40 -> 95 (50 in the mean of R^k and S^k now), band tables
// (ensure_r_band_tables) 4 x 39 -> 87 (44 now).
int ensure_r_cells(dbsrg_ctx *c, int k) {
  const DeviceGrid &g = c->g;
  const int nv = g.nv, kk = g.ks * g.ks;
  const size_t m = (size_t)kk * nv;
  if ((int)c->rshare.size() <= k) c->rshare.resize(k + 1);
  if (c->rcell.size() < (size_t)(k + 1) * 4) c->rcell.resize((size_t)(k + 1) * 4);
  RCells &r = c->rshare[k];
  if (c->rcell[(size_t)k * 4].rkd) return DBSRG_OK;
  int rc;
  const size_t ts1 = (size_t)g.ns * g.ks;  // sums of one moment array
  if (!r.mom && !(r.mom = (double *)cache_alloc(c, 4 * (m + ts1) * sizeof(double))))
    return set_err(c, DBSRG_ENOMEM, "cell data allocation failed");
  const int wh[4] = {0, 0, 1, 1}, kp[4] = {k, -(k + 1), k, -(k + 1)};
  double *const mo[4] = {r.mom, r.mom + m, r.mom + 2 * m, r.mom + 3 * m};
  if ((rc = compute_moment_set(c, 4, wh, kp, mo))) return rc;
  TriSet ts{};
  for (int i = 0; i < 3; i++) {
    const int t = 2 - i;  // the largest first: the blocks that end the launch are short
    const TableBases tb = table_bases(g, 0, t);
    const size_t f = (size_t)npairs(tb.e1) * npairs(tb.e2) * nv;
    if (!r.diag[t] && !(r.diag[t] = (double *)cache_alloc(c, 2 * f * sizeof(double))))
      return set_err(c, DBSRG_ENOMEM, "cell data allocation failed");
    ts.type[i] = t;
    ts.rkd[i] = r.diag[t];
    ts.rkf[i] = (float2 *)(r.diag[t] + f);
  }
  if ((rc = compute_diag_set(c, 3, ts, k))) return rc;
  for (int t = 0; t < 4; t++) {
    CellData cd;
    const int wa = (t == 0 || t == 2) ? 0 : 1, wb = (t == 0 || t == 3) ? 0 : 1;
    cd.lo1 = r.mom + 2 * wa * m;
    cd.hi1 = cd.lo1 + m;
    cd.lo2 = r.mom + 2 * wb * m;
    cd.hi2 = cd.lo2 + m;
    cd.rkd = r.diag[std::min(t, 2)];
    const TableBases tb = table_bases(g, 0, t);
    cd.rkf = (float2 *)(cd.rkd + (size_t)npairs(tb.e1) * npairs(tb.e2) * nv);
    cd.tr = t == 3;
    c->rcell[(size_t)k * 4 + t] = cd;
  }
  return DBSRG_OK;
}

// the sums of table (family, type, k)'s moments, R^k those of all types of the k;
// entered in the cell data (which marks them as built) once they are launched
int moment_sums(dbsrg_ctx *c, int family, int type, int k) {
  const DeviceGrid &g = c->g;
  TotalSet ts{};
  int n;
  const size_t per = (size_t)g.ns * (family == 0 ? g.ks : 2 * g.ks - 1);
  double *T;
  auto set = [&](int i, const PairSpec &e, const double *M, double *T) {
    ts.k1[i] = e.k1;
    ts.k2[i] = e.k2;
    ts.sym[i] = e.sym;
    ts.M[i] = M;
    ts.T[i] = T;
  };
  if (family == 0) {
    CellData *cd = &c->rcell[(size_t)k * 4];
    if (cd[0].tlo1) return DBSRG_OK;
    n = 4;
    T = c->rshare[k].mom + 4 * (size_t)g.ks * g.ks * g.nv;
    for (int b = 0; b < 2; b++) {  // electron 1 of types 0 and 1: the P and Q pairs
      const PairSpec e = table_bases(g, 0, b).e1;
      set(2 * b, e, cd[b].lo1, T + 2 * b * per);
      set(2 * b + 1, e, cd[b].hi1, T + (2 * b + 1) * per);
    }
  } else {
    CellData &cd = c->scell[(size_t)k * 2 + type];
    if (cd.tlo1) return DBSRG_OK;
    n = 2;
    const TableBases tb = table_bases(g, 1, type);
    T = (double *)(cd.rkf + (size_t)npairs(tb.e1) * npairs(tb.e2) * g.nv);
    set(0, tb.e1, cd.lo1, T);
    set(1, tb.e2, cd.hi2, T + per);
  }
  if (c->stream != c->bstream[0] && c->stream != c->bstream[1]) c->stream_built = true;
  DBSRG_RUN(c, "k_moment_sums",
            k_moment_sums<<<dim3((unsigned)((per + 127) / 128), n), 128, 0, c->stream>>>(
                g.ns, g.ks, g.nv, ts));
  if (family == 0) {
    CellData *cd = &c->rcell[(size_t)k * 4];
    for (int t = 0; t < 4; t++) {
      const bool pa = t == 0 || t == 2, pb = t == 0 || t == 3;
      cd[t].tlo1 = T + (pa ? 0 : 2 * per);
      cd[t].thi1 = cd[t].tlo1 + per;
      cd[t].tlo2 = T + (pb ? 0 : 2 * per);
      cd[t].thi2 = cd[t].tlo2 + per;
    }
  } else {
    CellData &cd = c->scell[(size_t)k * 2 + type];
    cd.tlo1 = T;
    cd.thi2 = T + per;
  }
  return DBSRG_OK;
}

// fills n (1..3) R^k tables of one k, full (band 0) or band-limited
static int fill_r(dbsrg_ctx *c, int n, const int *types, int k, double *const *tab, int band) {
  const DeviceGrid &g = c->g;
  const int nj = band ? 2 * band + 1 : g.ns;
  const size_t nt = (size_t)g.ns * nj * g.ks * g.ks;
  FillSet fs{};
  for (int i = 0; i < n; i++) {
    const CellData *cd;
    int rc = get_celldata(c, 0, types[i], k, &cd);
    if (rc || (rc = moment_sums(c, 0, types[i], k))) return rc;
    const TableBases tb = table_bases(g, 0, types[i]);
    fs.TlowA[i] = cd->tlo1;
    fs.ThighA[i] = cd->thi1;
    fs.TlowB[i] = cd->tlo2;
    fs.ThighB[i] = cd->thi2;
    fs.ka[i] = tb.e1.k1;
    fs.kb[i] = tb.e2.k1;
    fs.tr[i] = cd->tr;
    fs.lowA[i] = cd->lo1;
    fs.highA[i] = cd->hi1;
    fs.lowB[i] = cd->lo2;
    fs.highB[i] = cd->hi2;
    fs.rkd[i] = cd->rkd;
    fs.rkb[i] = tab[i];
  }
  DBSRG_RUN(c, "k_fill_r",
            k_fill_r<<<dim3((unsigned)((nt + 255) / 256), n), 256, 0, c->stream>>>(
                g.ns, g.ks, g.nv, fs, band));
  return DBSRG_OK;
}

int ensure_r_band_tables(dbsrg_ctx *c, int k) {
  const size_t i0 = (size_t)k * 4;
  if (c->rbtab.size() < i0 + 4) c->rbtab.resize(i0 + 4, nullptr);
  const size_t nt = (size_t)c->g.ns * (2 * DBSRG_TABLE_BAND + 1) * c->g.ks * c->g.ks;
  int types[3], n = 0;
  double *tab[3];
  for (int t = 0; t < 3; t++) {
    if (c->rbtab[i0 + t]) continue;
    if (!(tab[n] = (double *)cache_alloc(c, nt * sizeof(double)))) {
      for (int i = 0; i < n; i++) cache_free(c, tab[i]);
      return set_err(c, DBSRG_ENOMEM, "table allocation failed");
    }
    types[n++] = t;
  }
  if (n == 0) return DBSRG_OK;
  const int rc = fill_r(c, n, types, k, tab, DBSRG_TABLE_BAND);
  for (int i = 0; i < n; i++) {
    if (rc)
      cache_free(c, tab[i]);
    else
      c->rbtab[i0 + types[i]] = tab[i];
  }
  return rc;
}

// full (band == 0) or band-limited table of (family, type, k), cached
static int get_table_any(dbsrg_ctx *c, int family, int type, int k, int band,
                         const double **out) {
  const DeviceGrid &g = c->g;
  std::vector<double *> &v = family == 0 ? (band ? c->rbtab : c->rtab) : (band ? c->sbtab : c->stab);
  size_t idx = (size_t)k * (family == 0 ? 4 : 2) + type;
  ensure_slot(c, v, idx);
  if (v[idx]) {
    *out = v[idx];
    return DBSRG_OK;
  }
  const int ns = g.ns, ks = g.ks, nv = g.nv, kb = family == 0 ? ks : 2 * ks - 1;
  const int nj = band ? 2 * band + 1 : ns;
  size_t nt = (size_t)ns * nj * kb * kb;
  const CellData *cd;
  int rc = get_celldata(c, family, type, k, &cd);
  if (rc) return rc;
  CacheBuffer buf(c, nt * sizeof(double));
  double *tab = (double *)buf.p;
  if (!tab) return set_err(c, DBSRG_ENOMEM, "table allocation failed");
  if (family == 0) {
    if ((rc = fill_r(c, 1, &type, k, &tab, band))) return rc;
  } else {
    if ((rc = moment_sums(c, 1, type, k))) return rc;
    const unsigned nb = (unsigned)((nt + 255) / 256);
    int kj1 = type == 0 ? g.ksp : g.ksq, kj2 = type == 0 ? g.ksq : g.ksp;
    DBSRG_RUN(c, "k_fill_s",
              k_fill_s<<<nb, 256, 0, c->stream>>>(ns, ks, nv, g.ksp, g.ksq, kj1, kj2, cd->lo1,
                                                  cd->hi2, cd->tlo1, cd->thi2, cd->rkd, tab,
                                                  band));
  }
  buf.keep();
  v[idx] = tab;
  *out = tab;
  return DBSRG_OK;
}

int get_rtable(dbsrg_ctx *c, int type, int k, const double **out) {
  return get_table_any(c, 0, type, k, 0, out);
}
int get_stable(dbsrg_ctx *c, int type, int k, const double **out) {
  return get_table_any(c, 1, type, k, 0, out);
}
int get_band_table(dbsrg_ctx *c, int family, int type, int k, const double **out) {
  return get_table_any(c, family, type, k, DBSRG_TABLE_BAND, out);
}

// ----------------------------------------------------------------------------
// <a|r^k|b> split by component: quadr (dbsr_lib_dbs.f90:3940-3976), used for
// the asymptotic coefficients (QUADR_PQ at R_data.f90:224, which selects the
// component by atype).  With G(i,j) = sum over cells of the moments <B_i|r^k|B_j>
// and w_b = G p_b -- the far-field vectors of the R^k tables of this k, which
// the exchange lists need as well -- it is p_a . w_b.
// quad[comp][pair]: one warp per pair (a, b), pair = a n + b.  ns 80: 6 us a k;
// as a Gram matrix from the Gauss points, a banded product and 32 x 32 tiles of
// all orbitals (channel ones too) 55 + 8 + 31 us (ns 283: 62 + 10 + 95).
__global__ void k_quad_dot(int n, int ns, const double *P, size_t pstride, const int *b2o,
                           const double *W, size_t wcomp, double *quad) {
  const int q = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x % 32;
  const int comp = blockIdx.y;
  if (q >= n * n) return;
  const int a = q / n, b = q % n;
  const double *p = P + (size_t)(b2o ? b2o[a] - 1 : a) * pstride + (size_t)ns * comp;
  const double *w = W + (size_t)comp * wcomp + (size_t)ns * b;
  double s = 0.0;
#pragma unroll 4
  for (int i = lane; i < ns; i += 32) s = fma(p[i], w[i], s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) quad[(size_t)comp * n * n + q] = s;
}

// bound: over the bound orbitals (pairs as in the factored forms' lists),
// otherwise over all nbf
int get_quad(dbsrg_ctx *c, int k, bool bound, const double **out) {
  std::vector<double *> &v = bound ? c->quadb : c->quad;
  if ((int)v.size() <= k) v.resize(k + 1, nullptr);
  if (v[k]) {
    *out = v[k];
    return DBSRG_OK;
  }
  const DeviceGrid &g = c->g;
  const int n = bound ? c->nbound : c->nbf;
  const size_t m = (size_t)g.ns * n, nq = (size_t)2 * n * n;
  int rc;
  const double *W;
  if (bound && (rc = get_rfar(c, k, &W))) return rc;
  CacheBuffer buf(c, (nq + (bound ? 0 : 4 * m)) * sizeof(double));
  double *q = (double *)buf.p;
  if (!q) return set_err(c, DBSRG_ENOMEM, "quad allocation failed");
  if (!bound) {
    if ((rc = far_vectors_all(c, k, q + nq))) return rc;
    W = q + nq;
  }
  DBSRG_RUN(c, "k_quad_dot",
            k_quad_dot<<<dim3((unsigned)(((size_t)n * n + 7) / 8), 2), 256, 0, c->stream>>>(
                n, g.ns, c->pq, (size_t)2 * g.ns, bound ? c->b2o : nullptr, W, 2 * m, q));
  buf.keep();
  v[k] = q;
  *out = q;
  return DBSRG_OK;
}
