// direct.cu -- the direct cases (convol cases 1/2: R_data itype 3, S_data
// itypes 6/7) of the factored forms, segment by segment: the band density of
// a segment is summed over its entries first and then contracted with the
// cells of the table.
//
//   d_s(i,j)      = sum_e c_e p1_{a_e}(i) p2_{b_e}(j)          (band, 's' or 'n')
//   S_s(iv)       = sum_pair2 M(pair2;iv) d_s(pair2)           moments of a cell
//   Y_s(pair1)    = sum_iv [ lo1(pair1;iv) Suf_s(iv) + hi1(pair1;iv) Pre_s(iv)
//                            + sum_pair2 rkd(pair1,pair2;iv) d_s(pair2) ]
// (case 2 with the electrons exchanged; only the suffix or prefix term for
// S^k, whose tables hold no r1 > r2 cells).  The two PQ types of an R^k list
// that fill the same quadrant are summed in Y.  The work is per segment --
// npo kd multiply-adds a cell, ns ncol an entry -- and there is none per
// orbital pair: factor.cu's pair potentials cost the same whatever the list
// holds, and pay where a list has many segments (direct_by_segment compares the
// two).
//
// Segments lie along the lanes of a warp: every table value is uniform across
// a warp, densities are stored segment-fastest.  In the split form the
// densities and the diagonal cells are float-float (ff.cuh) as the pair
// potentials are; cell moments, their sums over cells and the separable terms
// are FP64 in both forms.
#include <algorithm>
#include <type_traits>

#include "ff.cuh"
#include "internal.cuh"
#include "pairs.cuh"

namespace {

constexpr int NC3 = 3;  // band columns per thread of the density kernel
constexpr int DSL = 8;  // segments per block of the density kernel

// Band densities of every member segment, rho[comp][col*ns + i][nmp].
// blockIdx.z = component set * column groups + column group; lanes are rows i,
// warps are segments.  An entry takes two scaled orbital values and one
// multiply-add per band element (two in the symmetric storage off the
// diagonal); the columns are split over threads because a segment's entries
// are a serial chain.
template <bool FF>
struct DensArgs {
  int ns, ks, nb, nm, nmp, ncol, sym, ngrp;
  const typename Val<FF>::T *P1[2], *P2[2];  // [orbital][ns] per component set
  const int *members, *pairs;
  const SegInfo *info;
  const typename Val<FF>::T *c;
  typename Val<FF>::T *rho;
};

template <bool FF>
__global__ void __launch_bounds__(32 * DSL) k_seg_density(const DensArgs<FF> d) {
  using V = Val<FF>;
  using T = typename V::T;
  __shared__ T out[NC3][32][DSL];
  const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
  const int i = blockIdx.x * 32 + lane, slot = blockIdx.y * DSL + w;
  const int cs = blockIdx.z / d.ngrp, col0 = (blockIdx.z % d.ngrp) * NC3;
  const int off0 = d.sym ? col0 : col0 - (d.ks - 1);
  const int ns = d.ns;
  V acc[NC3];
  if (slot < d.nm && i < ns) {
    const SegInfo si = d.info[d.members[slot]];
    const T *P1 = d.P1[cs] + i, *P2 = d.P2[cs] + i;
    bool ok[NC3];
#pragma unroll
    for (int k = 0; k < NC3; k++)
      ok[k] = col0 + k < d.ncol && i + off0 + k >= 0 && i + off0 + k < ns;
#pragma unroll 4
    for (int e = si.start; e < si.end; e++) {
      const int pr = d.pairs[e], a = pr / d.nb, b = pr - a * d.nb;
      const T *pa = P1 + (size_t)a * ns, *pb = P2 + (size_t)b * ns;
      const T c = d.c[e], ca = V::mul(c, pa[0]);
      if (d.sym) {
        const T cb = V::mul(c, pb[0]);
#pragma unroll
        for (int k = 0; k < NC3; k++) {
          if (!ok[k]) continue;
          acc[k].mac(ca, pb[off0 + k]);
          if (off0 + k > 0) acc[k].mac(cb, pa[off0 + k]);
        }
      } else {
#pragma unroll
        for (int k = 0; k < NC3; k++)
          if (ok[k]) acc[k].mac(ca, pb[off0 + k]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < NC3; k++) out[k][lane][w] = acc[k].get();
  __syncthreads();
  const int s0 = blockIdx.y * DSL;
  for (int q = threadIdx.x; q < NC3 * 32 * DSL; q += 32 * DSL) {
    const int ws = q % DSL, li = (q / DSL) % 32, k = q / (DSL * 32);
    const int ii = blockIdx.x * 32 + li;
    if (ii < ns && col0 + k < d.ncol)
      d.rho[((size_t)cs * d.ncol * ns + (size_t)(col0 + k) * ns + ii) * d.nmp + s0 + ws] =
          out[k][li][ws];
  }
}

// Moments of every cell, S[set][cell][nmp]: set = (component set, moment);
// one warp per (cell, 32 segments)
template <bool FF>
struct CellArgs {
  int ns, nv, ks, kk, nmp, ncol, sym;
  PairSpec ed[4];
  const double *M[4];
  int comp[4];
  const typename Val<FF>::T *rho;
  double *S;
};

constexpr int CW = 8;  // cells per block

template <bool FF>
__global__ void __launch_bounds__(32 * CW) k_seg_cells(const CellArgs<FF> a) {
  const int lane = threadIdx.x % 32, cv = blockIdx.y * CW + threadIdx.x / 32 + 1;
  const int slot = blockIdx.x * 32 + lane, set = blockIdx.z;
  if (cv > a.nv) return;
  const typename Val<FF>::T *rho =
      a.rho + (size_t)a.comp[set] * a.ncol * a.ns * a.nmp + slot;
  const double *M = a.M[set] + (size_t)a.kk * (cv - 1);
  const PairSpec ed = a.ed[set];
  double s = 0.0;
  for (int g1 = 1; g1 <= ed.k1; g1++) {
    const int i = cv + g1 - 2;
    const double *Mr = M;  // the row's moments (pairs are numbered row by row)
    M += a.sym ? ed.k1 - g1 + 1 : ed.k2;
    // the up to nine values of a row loaded together
    typename Val<FF>::T v[9];
    double m[9];
#pragma unroll
    for (int u = 0; u < 9; u++) {
      const int g2 = (a.sym ? g1 : 1) + u, col = a.sym ? u : g2 - g1 + a.ks - 1;
      const bool ok = g2 <= ed.k2 && i < a.ns && cv + g2 - 2 < a.ns;
      v[u] = ok ? rho[((size_t)col * a.ns + i) * a.nmp] : Val<FF>::zero();
      m[u] = ok ? Mr[u] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 9; u++) s = fma(m[u], Val<FF>::dbl(v[u]), s);
  }
  a.S[((size_t)set * a.nv + cv - 1) * a.nmp + slot] = s;
}

// Exclusive sums over the later (bit set in sufmask) or earlier cells, in
// place: eight segments a block, each with sixteen runs of cells
constexpr int SCW = 16, SCL = 8;
__global__ void __launch_bounds__(SCL * SCW) k_seg_scan(int nv, int nmp, unsigned sufmask,
                                                       double *S) {
  __shared__ double tot[SCW][SCL];
  const int lane = threadIdx.x % SCL, w = threadIdx.x / SCL, set = blockIdx.y;
  const bool suf = (sufmask >> set) & 1;
  double *s = S + (size_t)set * nv * nmp + blockIdx.x * SCL + lane;
  const int run = (nv + SCW - 1) / SCW, lo = min(nv, w * run), hi = min(nv, lo + run);
  double t = 0.0;
#pragma unroll 8
  for (int i = lo; i < hi; i++) t += s[(size_t)(suf ? hi - 1 - (i - lo) : i) * nmp];
  tot[w][lane] = t;
  __syncthreads();
  double acc = 0.0;
  if (suf)
    for (int k = SCW - 1; k > w; k--) acc += tot[k][lane];
  else
    for (int k = 0; k < w; k++) acc += tot[k][lane];
  // (loads of eight cells before their stores: the array is overwritten)
  for (int i0 = lo; i0 < hi; i0 += 8) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int i = i0 + u;
      v[u] = i < hi ? s[(size_t)(suf ? hi - 1 - (i - lo) : i) * nmp] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int i = i0 + u;
      if (i >= hi) break;
      s[(size_t)(suf ? hi - 1 - (i - lo) : i) * nmp] = acc;
      acc += v[u];
    }
  }
}

// The potentials: a block forms one row f (the output's first function) for 32
// segments.  Every output pair (h1, h2) of a cell cv = f - h1 + 1 belongs to
// one row, so a row sums its cells' contributions without partial results in
// global memory.  A warp takes the cells of one h1 (symmetric storage: of h1
// and k1 + 1 - h1, ten table rows a warp): a density value read from shared
// memory meets all of the cell's up to nine output pairs, whose sums are nine
// independent chains.  The window of density rows that the cells meet and the
// table values are staged in shared memory; the warps' sums are added there in
// order.  In the split form bound by the twelve FP32 instructions of a
// float-float multiply-add, otherwise by the FP64 pipe.  ns 400, 78 segments,
// R^k (201 M multiply-adds): 274 us; 352 us with one warp per output diagonal.
// A chain is renormalised after each row of up to nine terms: over 30 drawn
// matrices the error against 64 bits is 1.5e-14 in the mean and 3.2e-14 at most
// of a block's norm, 1.7e-14 and 5.5e-14 without (pair potentials 1.6e-14 and
// 3.9e-14).
template <bool FF>
struct ApplyArgs {
  int ns, nv, ks, kk, nm, nmp, ncol, sym;
  int nwin;   // window rows
  int ntype;  // table types summed into one output
  PairSpec eo[2], ed[2][2];  // per output (blockIdx.z) and type
  const typename Val<FF>::T *R[2][2];  // cell integrals: element (po, pd; cell) at
  size_t rcell[2][2];                  // po rpo + pd rpd + cell rcell
  int rpo[2][2], rpd[2][2];
  const double *L1[2][2], *L2[2][2];
  int comp[2][2], set1[2][2], set2[2][2];
  const typename Val<FF>::T *rho;
  const double *S;
  double *Y;  // [output][slot][ns*ncol]
};

constexpr int NRO = 9;  // output pairs of a cell and first function (orders <= 9)

// SYM: the symmetric storage (R^k); its blocks of five warps fit four an SM,
// the eight or nine warps of the other (S^k) two
template <bool FF, bool SYM>
__global__ void __launch_bounds__(SYM ? 160 : 288, SYM ? 4 : 2) k_seg_apply(const ApplyArgs<FF> p) {
  using V = Val<FF>;
  using T = typename V::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  T *win = reinterpret_cast<T *>(smraw);       // [nwin][ncol][32]
  T *Rs = win + (size_t)p.nwin * p.ncol * 32;  // [h1][pd][output pair of h1]
  const int lane = threadIdx.x % 32, w = threadIdx.x / 32, nw = blockDim.x / 32;
  const int slot = blockIdx.y * 32 + lane, out = blockIdx.z;
  const int f = blockIdx.x + 1;  // 1-based
  const int ns = p.ns;
  const PairSpec eo = p.eo[out];
  // first functions of this warp (0: none)
  int h1s[2];
  if (SYM) {
    h1s[0] = 2 * (w + 1) <= eo.k1 + 1 ? w + 1 : 0;
    h1s[1] = 2 * (w + 1) < eo.k1 + 1 ? eo.k1 - w : 0;
  } else {
    h1s[0] = w + 1 <= eo.k1 ? w + 1 : 0;
    h1s[1] = 0;
  }
  // output pairs of the first functions before h1
  auto before = [&](int h1) {
    return SYM ? (h1 - 1) * eo.k1 - (h1 - 1) * (h1 - 2) / 2 : (h1 - 1) * eo.k2;
  };
  V acc[NRO];
  for (int t = 0; t < p.ntype; t++) {
    const PairSpec ed = p.ed[out][t];
    const int kd = npairs(ed);
    if (t > 0) __syncthreads();
    const T *rho = p.rho + (size_t)p.comp[out][t] * p.ncol * ns * p.nmp + blockIdx.y * 32;
#pragma unroll 4
    for (int q = w; q < p.nwin * p.ncol; q += nw) {
      const int i = f - eo.k1 + q / p.ncol, col = q % p.ncol;  // 0-based row
      win[(size_t)q * 32 + lane] =
          i >= 0 && i < ns ? rho[((size_t)col * ns + i) * p.nmp + lane] : V::zero();
    }
    // the warp's own table rows
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int h1 = h1s[k], cv = f - h1 + 1;
      if (h1 == 0 || cv < 1 || cv > p.nv) continue;
      const int nr = SYM ? eo.k1 - h1 + 1 : eo.k2, po0 = before(h1);
      const T *rc = p.R[out][t] + p.rcell[out][t] * (cv - 1) + (size_t)p.rpo[out][t] * po0;
      T *rs = Rs + (size_t)po0 * kd;
      const int rpo = p.rpo[out][t], rpd = p.rpd[out][t];
#pragma unroll 4
      for (int q = lane; q < kd * nr; q += 32) {
        const int pd = q / nr, r = q - pd * nr;
        rs[q] = rc[(size_t)rpo * r + (size_t)rpd * pd];
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int h1 = h1s[k], cv = f - h1 + 1;
      if (h1 == 0 || cv < 1 || cv > p.nv) continue;
      const int nr = SYM ? eo.k1 - h1 + 1 : eo.k2;
      const T *rs = Rs + (size_t)before(h1) * kd;
      const T *wn = win + (size_t)(eo.k1 - h1) * p.ncol * 32 + lane;
      auto cell = [&](auto nrc) {
        constexpr int N = decltype(nrc)::value;
        const T *r = rs;
        for (int g1 = 1; g1 <= ed.k1; g1++) {
          const T *d = wn + ((size_t)(g1 - 1) * p.ncol + (SYM ? 0 : p.ks - g1)) * 32;
          const int n2 = SYM ? ed.k2 - g1 + 1 : ed.k2;
          for (int u = 0; u < n2; u++, r += N) {
            const T dv = d[(size_t)u * 32];
#pragma unroll
            for (int q = 0; q < N; q++) acc[q].mac(r[q], dv);
          }
#pragma unroll
          for (int q = 0; q < N; q++) acc[q].renorm();
        }
      };
      switch (nr) {
        case 1: cell(std::integral_constant<int, 1>()); break;
        case 2: cell(std::integral_constant<int, 2>()); break;
        case 3: cell(std::integral_constant<int, 3>()); break;
        case 4: cell(std::integral_constant<int, 4>()); break;
        case 5: cell(std::integral_constant<int, 5>()); break;
        case 6: cell(std::integral_constant<int, 6>()); break;
        case 7: cell(std::integral_constant<int, 7>()); break;
        case 8: cell(std::integral_constant<int, 8>()); break;
        default: cell(std::integral_constant<int, 9>());
      }
    }
  }
  // the warps' sums to shared memory (over the window): red[warp][q][lane],
  // q = h2 - h1 (symmetric: every warp's first functions alike) or h2 - 1
  __syncthreads();
  T *red = win;
#pragma unroll
  for (int q = 0; q < NRO; q++) red[((size_t)w * NRO + q) * 32 + lane] = acc[q].get();
  __syncthreads();
  // one warp per band column: the separable terms and the sum
  for (int col = w; col < p.ncol; col += nw) {
    const int dl = SYM ? col : col - (p.ks - 1);
    if (f + dl < 1 || f + dl > ns || slot >= p.nm) continue;
    double far = 0.0;
    for (int t = 0; t < p.ntype; t++) {
      const double *s1 = p.S + (size_t)p.set1[out][t] * p.nv * p.nmp + slot;
      const double *s2 = p.S + (size_t)p.set2[out][t] * p.nv * p.nmp + slot;
      const double *L1 = p.L1[out][t], *L2 = p.L2[out][t];
      double a1[NRO], b1[NRO], a2[NRO], b2[NRO];
#pragma unroll
      for (int h = 0; h < NRO; h++) {
        const int h1 = h + 1, cv = f - h1 + 1;
        const bool ok = h1 <= eo.k1 && h1 + dl >= 1 && h1 + dl <= eo.k2 && cv >= 1 && cv <= p.nv;
        const size_t o = ok ? (size_t)pidx(eo, h1, h1 + dl) + (size_t)p.kk * (cv - 1) : 0;
        a1[h] = ok ? L1[o] : 0.0;
        b1[h] = ok ? s1[(size_t)(cv - 1) * p.nmp] : 0.0;
        a2[h] = ok && L2 ? L2[o] : 0.0;
        b2[h] = ok && L2 ? s2[(size_t)(cv - 1) * p.nmp] : 0.0;
      }
#pragma unroll
      for (int h = 0; h < NRO; h++) far = fma(a1[h], b1[h], fma(a2[h], b2[h], far));
    }
    V sum;
    for (int v = 0; v < nw; v++) {
      const int r = SYM ? dl : v + dl;  // h2 - 1 of first function v + 1
      if (r < 0 || r >= NRO || (!SYM && (v + 1 > eo.k1 || r >= eo.k2))) continue;
      sum.add_value(red[((size_t)v * NRO + r) * 32 + lane]);
    }
    p.Y[((size_t)out * p.nm + slot) * ns * p.ncol + (size_t)(f - 1) + (size_t)ns * col] =
        far + sum.value();
  }
}

template <bool FF>
int run(dbsrg_ctx *c, const FactorJob &j) {
  using T = typename Val<FF>::T;
  const DeviceGrid &g = c->g;
  const int ns = g.ns, ks = g.ks, nv = g.nv, kk = ks * ks, nb = c->nbound;
  cudaStream_t st = c->stream;
  const bool sym = j.sym == 's';
  const int ncol = sym ? ks : 2 * ks - 1, nm = j.nm, nmp = (nm + 31) / 32 * 32;
  int rc;
  // outputs: the types that fill one quadrant; component sets of the densities
  int nout = 0, ntype = 0, oii[2], ojj[2], otype[2][2], ncs = 0, c1[2], c2[2], cset[4];
  for (int a = 0; a < j.na; a++) {
    int s = 0;
    while (s < ncs && (c1[s] != j.jp1[a] || c2[s] != j.jp2[a])) s++;
    if (s == ncs) {
      if (ncs == 2) return set_err(c, DBSRG_ECUDA, "direct segments: components");
      c1[ncs] = j.jp1[a];
      c2[ncs++] = j.jp2[a];
    }
    cset[a] = s;
    int o = 0;
    while (o < nout && (oii[o] != j.ii[a] || ojj[o] != j.jj[a])) o++;
    if (o == nout) {
      if (nout == 2) return set_err(c, DBSRG_ECUDA, "direct segments: quadrants");
      oii[nout] = j.ii[a];
      ojj[nout++] = j.jj[a];
      otype[o][0] = a;
      ntype = std::max(ntype, 1);
    } else {
      otype[o][1] = a;
      ntype = 2;
    }
  }
  const CellData *cd[4];
  for (int a = 0; a < j.na; a++)
    if ((rc = get_celldata(c, j.family, j.types[a], j.kpol, &cd[a]))) return rc;
  if (j.prep) return DBSRG_OK;
  // both built before the first list of an assembly is prepared
  const T *rows = FF ? (const T *)c->browsf : (const T *)c->brows;
  const bool two = j.family == 0;  // both fields (r1 < r2 and r1 > r2 cells)
  const int nset = ncs * (two ? 2 : 1);
  const size_t per = (size_t)ns * ncol;
  const size_t rb = (sizeof(T) * ncs * per * nmp + 255) & ~(size_t)255;
  const size_t sb = (sizeof(double) * nset * nv * nmp + 255) & ~(size_t)255;
  if ((rc = ensure_fscratch(c, rb + sb + sizeof(double) * nout * nm * per))) return rc;
  T *rho = (T *)c->fscratch;
  double *S = (double *)((char *)c->fscratch + rb), *Y = (double *)((char *)c->fscratch + rb + sb);
  DensArgs<FF> d{};
  d.ns = ns;
  d.ks = ks;
  d.nb = nb;
  d.nm = nm;
  d.nmp = nmp;
  d.ncol = ncol;
  d.sym = sym;
  d.ngrp = (ncol + NC3 - 1) / NC3;
  for (int s = 0; s < ncs; s++) {
    d.P1[s] = rows + (size_t)(c1[s] - 1) * nb * ns;
    d.P2[s] = rows + (size_t)(c2[s] - 1) * nb * ns;
  }
  d.members = j.members;
  d.pairs = j.pairs;
  d.info = j.info;
  d.c = FF ? (const T *)j.cdf : (const T *)j.cd;
  d.rho = rho;
  // executed work: per entry and band element one multiply-add (two in the
  // symmetric storage); the densities written
  const double df = 2.0 * ncs * (sym ? 2.0 : 1.0) * (double)per * (double)j.nent;
  DBSRG_RUN_W(c, "k_seg_density", 8.0 * ncs * (double)per * nm, df,
              k_seg_density<FF><<<dim3((unsigned)((ns + 31) / 32), (unsigned)(nmp / DSL),
                                       (unsigned)(ncs * d.ngrp)),
                                  32 * DSL, 0, st>>>(d));
  CellArgs<FF> ca{};
  ApplyArgs<FF> p{};
  unsigned sufmask = 0;
  const int nm2 = two ? 2 : 1;  // moments per component set
  int nw = 0, rmax = 0;  // warps of the apply kernel, its table values
  for (int o = 0; o < nout; o++)
    for (int t = 0; t < ntype; t++) {
      const int a = otype[o][t], s = cset[a];
      const CellData &x = *cd[a];
      const TableBases tb = table_bases(g, j.family, j.types[a]);
      // case 1: density on electron 2, result on electron 1; case 2 the other way
      const PairSpec eo = j.icv == 1 ? tb.e1 : tb.e2, ed = j.icv == 1 ? tb.e2 : tb.e1;
      p.eo[o] = eo;
      p.ed[o][t] = ed;
      ca.M[s * nm2] = j.icv == 1 ? x.hi2 : x.lo1;
      if (j.icv == 1) sufmask |= 1u << (s * nm2);
      if (two) ca.M[s * 2 + 1] = x.lo2;
      for (int m = 0; m < nm2; m++) {
        ca.ed[s * nm2 + m] = ed;
        ca.comp[s * nm2 + m] = s;
      }
      // cell integrals (float-float copy or FP64): first pair fastest; it is the
      // second electron's where tr
      const int n1 = npairs(x.tr ? tb.e2 : tb.e1), n2 = npairs(x.tr ? tb.e1 : tb.e2);
      const bool ofirst = (j.icv == 1) != x.tr;
      p.R[o][t] = FF ? (const T *)x.rkf : (const T *)x.rkd;
      p.rcell[o][t] = (size_t)n1 * n2;
      const int r2 = n1;  // stride of the second pair
      p.rpo[o][t] = ofirst ? 1 : r2;
      p.rpd[o][t] = ofirst ? r2 : 1;
      p.L1[o][t] = j.icv == 1 ? x.lo1 : x.hi2;
      p.L2[o][t] = two ? x.hi1 : nullptr;
      p.comp[o][t] = s;
      p.set1[o][t] = s * nm2;
      p.set2[o][t] = s * nm2 + 1;
      p.nwin = std::max(p.nwin, eo.k1 + ed.k1 - 1);
      rmax = std::max(rmax, npairs(eo) * npairs(ed));
      nw = std::max(nw, sym ? (eo.k1 + 1) / 2 : eo.k1);
    }
  ca.ns = p.ns = ns;
  ca.nv = p.nv = nv;
  ca.ks = p.ks = ks;
  ca.kk = p.kk = kk;
  ca.nmp = p.nmp = nmp;
  ca.ncol = p.ncol = ncol;
  ca.sym = p.sym = sym;
  ca.rho = rho;
  ca.S = S;
  DBSRG_RUN(c, "k_seg_cells",
            k_seg_cells<FF><<<dim3((unsigned)(nmp / 32), (unsigned)((nv + CW - 1) / CW),
                                   (unsigned)nset),
                              32 * CW, 0, st>>>(ca));
  DBSRG_RUN(c, "k_seg_scan", k_seg_scan<<<dim3((unsigned)(nmp / SCL), (unsigned)nset), SCL * SCW, 0,
                                          st>>>(nv, nmp, sufmask, S));
  p.nm = nm;
  p.ntype = ntype;
  p.rho = rho;
  p.S = S;
  p.Y = Y;
  // the window is reused for the warps' sums
  p.nwin = std::max(p.nwin, (nw * NRO + ncol - 1) / ncol);
  const size_t smem = sizeof(T) * ((size_t)p.nwin * ncol * 32 + rmax);
  const void *fn = sym ? (const void *)k_seg_apply<FF, true> : (const void *)k_seg_apply<FF, false>;
  if ((rc = raise_smem_limit(c, fn, smem))) return rc;
  // executed work: npo kd multiply-adds a cell, type and segment
  double af = 0.0;
  for (int o = 0; o < nout; o++)
    for (int t = 0; t < ntype; t++) af += 2.0 * nm * nv * npairs(p.eo[o]) * npairs(p.ed[o][t]);
  const dim3 ga((unsigned)ns, (unsigned)(nmp / 32), (unsigned)nout);
  auto apply = [&](auto k) -> int {
    DBSRG_RUN_W(c, "k_seg_apply", 8.0 * nout * nm * (double)per, af,
                k<<<ga, 32 * nw, smem, st>>>(p));
    return DBSRG_OK;
  };
  if ((rc = sym ? apply(k_seg_apply<FF, true>) : apply(k_seg_apply<FF, false>))) return rc;
  return scatter_band(c, nout, oii, ojj, j.sym, ncol, nm, j.members, j.nown, j.own, j.info, Y);
}

}  // namespace

// Multiply-adds of the two ways over a whole list (all its segments, whatever
// the window or chunk, so that a block's result does not depend on them), the
// pair way with the potentials it builds whether or not they are cached.  Per
// cell and lane of 32 segments (used or not) the apply kernel takes npo kd of
// them, counted 1.6 times since its blocks are few (0.7 T/s against the pair
// potentials' 1.2 where both are long), the cell moments about 40 kd (FP64); a pair
// potential about 4000 an output for its small matrix, 120 per second orbital and
// 14 per pair; both ways one an entry and band element.  So pairs up to some 30
// orbitals, segments above unless a list has many.  The direct lists of a matrix
// (R^k k = 0..2 and S^k, 11 lists, ns 300, tables rebuilt), ms by pairs and by
// segment:
//   orbitals               20         28         36         48         64         88
//   split, 16 segments  1.71 1.81  2.14 1.80  3.10 1.83  4.13 1.83  5.94 1.82  10.0 1.89
//          49           1.79 2.28  2.20 2.27  3.22 2.26  4.22 2.29  6.05 2.28  10.0 2.32
//          121          1.85 3.32  2.23 3.31  3.32 3.33  4.30 3.32  6.18 3.34  10.2 3.35
//   FP64,  16 segments  2.23 2.28  2.95 2.32  4.18 2.33  5.94 2.30  9.03 2.34  15.5 2.35
//          121          2.38 5.14  3.08 5.19  4.33 5.24  6.09 5.15  9.15 5.21  15.7 5.14
// (ns 150 and 400 cross at the same counts, 10 to 100 entries a segment too).  The
// rule takes segments from 31 orbitals with up to 32 segments, from some 50 with 49
// and from 70 to 80 with 121, where they are never the slower way.
// The lists of a one-channel matrix (the SCF potentials) hold one segment each
// and come once per orbital, so the pair potentials of an iteration serve all
// of them: 30 orbitals at ns 300 take 29.3 ms by segment, 18.4 by pairs.
bool direct_by_segment(const dbsrg_ctx *c, int family, int icv, int na, const int *types,
                       long long nseg, long long nent) {
  const DeviceGrid &g = c->g;
  if (c->nch == 1) return false;
  const double nb = c->nbound, ns = g.ns, nv = g.nv;
  const double ncol = family == 0 ? g.ks : 2.0 * g.ks - 1.0;
  const double lanes = (double)((nseg + 31) / 32 * 32);
  double seg = 0.0, pair = 0.0;
  for (int a = 0; a < na; a++) {
    const TableBases tb = table_bases(g, family, types[a]);
    const PairSpec eo = icv == 1 ? tb.e1 : tb.e2, ed = icv == 1 ? tb.e2 : tb.e1;
    const double npo = npairs(eo), kd = npairs(ed), np = family == 0 ? nb * (nb + 1) / 2 : nb * nb;
    seg += lanes * nv * kd * (1.6 * npo + 40.0);
    pair += ns * ncol * (4000.0 + 120.0 * nb + 14.0 * np);
    pair += (double)nent * ns * ncol;
  }
  seg += (double)nent * ns * ncol * (na > 1 ? 2.0 : 1.0);
  return seg < pair;
}

int direct_segments(dbsrg_ctx *c, const FactorJob &j) {
  return j.split && j.cdf ? run<true>(c, j) : run<false>(c, j);
}
